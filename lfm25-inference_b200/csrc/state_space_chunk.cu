// State-space recurrence over prompts as matrix products (the chunked form of Dao and Gu 2024), for bf16 activations and states
// of up to 256 rows.
//
// With a_t = exp(-rate dt_t), A_t = a_1 ... a_t inside a chunk of 64 tokens and S the state before it,
//     y_t = A_t S^T C_t + sum_{s <= t} (A_t / A_s) dt_s (C_t . B_s) x_s + skip x_t
//     S  <- A_64 S + sum_s (A_64 / A_s) dt_s B_s x_s^T
// A CTA owns one segment, one head and 64 columns of its state, and walks the segment chunk by chunk: the state stays in
// f32 accumulators (its product B^T x is added there), C B^T and C S share the loads of C.  x, B and C are bf16 already;
// everything that the recurrence multiplies them with -- the decays, the triangle of weights, the state itself -- enters
// the tensor core as a sum of two bf16 values (16 significant bits).  The logarithms of the A_t are summed in double and
// kept as two floats, so that the ratio of two neighbours behind a long decay is exact; one kernel forms them for all heads of
// a chunk, ahead of the CTAs that walk.
//
// Where segments, heads and column blocks do not fill the chip, segments are cut into pieces of several chunks: a first pass
// leaves each piece's contribution to the state (the products B^T x alone), a second one starts every piece from the sum
// of the pieces before it.  Only the order of the f32 sums over the state changes; state against float64 (4096 tokens, 64 heads
// with 128 rows; rates from 2^-9 to 20, 1, 0.02): 5.0e-6, 2.5e-6, 3.3e-6, from end to end 6.7e-6, 2.5e-6, 3.3e-6.
//
// Bound by the latency of a chunk's stages (tensor pipe 33 % busy with two CTAs per SM), so the shapes in use have strides
// known to the compiler (45 instead of 60 us for 8 x 512 tokens of 32 heads with 64 state rows, where the index arithmetic
// was a fifth of the instructions).  One segment of 4096 tokens, 64 heads with 128 state rows: 6 us factors, 35 us
// contributions, 133 us pieces; one CTA per head from end to end: 502 us on 64 SMs.
#include <algorithm>
#include <type_traits>

#include "launch.h"
#include "state_space.h"

namespace lfm25 {

namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kTokens = 64;
constexpr uint32_t kColumns = 64;
constexpr uint32_t kPad = 8;                            // elements behind each row: conflict-free ldmatrix
constexpr uint32_t kColumnPitch = kColumns + kPad;
constexpr size_t kSharedLimit = 227 * 1024;

// What a token contributes to a head: log2 A_t as high + low, dt_t, (A_64 / A_t) dt_t
struct __align__(16) TokenFactors {
    float log_high, log_low, step, into_state;
};

enum class Pass {
    kWhole,         // a CTA walks a whole segment
    kContribute,    // every piece but a segment's last: the state behind it, from zero (the first piece: from the record)
    kPieces,        // every piece: outputs, the state behind the last one
};

// Bytes of one buffer of a chunk's B, C and x
__host__ __device__ constexpr size_t chunk_bytes(uint32_t padded) {
    return (2 * kTokens * (padded + kPad) + kTokens * kColumnPitch) * 2;
}
constexpr size_t shared_bytes(uint32_t padded, uint32_t buffers, bool outputs) {
    // state (where there are outputs) and weighted x, both as two bf16 parts
    return buffers * chunk_bytes(padded) + 2 * ((outputs ? padded : 0) + kTokens) * kColumnPitch * 2 +
           2 * kTokens * sizeof(TokenFactors);
}

__device__ __forceinline__ void split_pair(float a, float b, uint32_t& high, uint32_t& low) {
    high = pack_bf16x2(a, b);
    const float2 rounded = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&high));
    low = pack_bf16x2(a - rounded.x, b - rounded.y);
}

// Factors of a chunk's tokens for eight heads: a warp scans the 64 tokens of a head, two per lane.  Latency only; inside the
// walking kernel the loads and the scan of every chunk were a serial 1200 cycles of one warp.
constexpr uint32_t kFactorHeads = kThreads / 32;
__global__ void __launch_bounds__(kThreads)
state_space_factors_kernel(const StateSpaceArgs<__nv_bfloat16> args, TokenFactors* factors, uint32_t head_blocks) {
    pdl_launch_dependents();
    pdl_wait();
    const SegmentTile tile = locate_tile(args.segments, kTokens, blockIdx.x / head_blocks);
    const uint32_t head = blockIdx.x % head_blocks * kFactorHeads + (threadIdx.x >> 5);
    if (tile.count == 0 || head >= args.heads) return;
    const uint32_t lane = threadIdx.x & 31;
    const float rate_log2 = -state_rate(args, head) * kLog2e;
    float own[2];
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i) {
        own[i] = 2 * lane + i < tile.count ? step_size(args, tile.first + 2 * lane + i, head) : 0.0f;
    }
    const double low = static_cast<double>(rate_log2 * own[0]);
    const double both = low + static_cast<double>(rate_log2 * own[1]);
    double inclusive = both;
#pragma unroll
    for (uint32_t delta = 1; delta < 32; delta <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, inclusive, delta);
        inclusive += lane >= delta ? other : 0.0;
    }
    const double total = __shfl_sync(0xffffffffu, inclusive, 31);
    const double logs[2] = {inclusive - both + low, inclusive};
    TokenFactors* target = factors + static_cast<size_t>(head) * args.segments.num_tokens + tile.first;
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i) {
        const uint32_t t = 2 * lane + i;
        const float high = static_cast<float>(logs[i]);
        if (t < tile.count) {
            target[t] = {high, static_cast<float>(logs[i] - static_cast<double>(high)), own[i],
                         fast_exp2(static_cast<float>(total - logs[i])) * own[i]};
        }
    }
}

// States between pieces: [piece][head][column block][size][columns], and log2 of each piece's decay [piece][head]
struct PieceArgs {
    const TokenFactors* factors;   // [heads][tokens]
    float* states;
    float* decays;
    uint32_t tokens;               // per piece, a multiple of 64
};

// UNITS: units of 16 state rows x 32 columns per warp (8 warps).  FULL: the state has exactly that many rows, so that all
// strides are constants and the loops over them unroll.
template <int UNITS, Pass PASS, bool FULL>
__global__ void __launch_bounds__(kThreads, UNITS <= 2 ? 2 : 1)
state_space_chunk_kernel(const StateSpaceArgs<__nv_bfloat16> args, const PieceArgs pieces, uint32_t column_blocks,
                         uint32_t padded_rows, uint32_t buffers) {
    const uint32_t padded = FULL ? 64 * UNITS : padded_rows;
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    const uint32_t pitch = padded + kPad;
    __nv_bfloat16* tiles = reinterpret_cast<__nv_bfloat16*>(chunk_smem);
    const uint32_t tile_elements = static_cast<uint32_t>(chunk_bytes(padded) / 2);
    __nv_bfloat16* state_high = tiles + buffers * tile_elements;        // [padded][columns]
    __nv_bfloat16* state_low = state_high + padded * kColumnPitch;
    __nv_bfloat16* input_high =                                         // [tokens][columns]
        PASS == Pass::kContribute ? state_high : state_low + padded * kColumnPitch;
    __nv_bfloat16* input_low = input_high + kTokens * kColumnPitch;
    TokenFactors* factor_tiles = reinterpret_cast<TokenFactors*>(input_low + kTokens * kColumnPitch);   // [2][tokens]
    pdl_launch_dependents();
    pdl_wait();

    const uint32_t block = blockIdx.x % column_blocks;
    const uint32_t head = blockIdx.x / column_blocks % args.heads;
    const uint32_t index = blockIdx.x / column_blocks / args.heads;     // of the segment or piece
    uint32_t segment = index, begin, end, piece = 0, last_piece = 0;
    if (PASS == Pass::kWhole) {
        begin = args.segments.offsets[segment];
        const uint32_t stop = args.segments.offsets[segment + 1];
        end = stop < args.segments.num_tokens ? stop : static_cast<uint32_t>(args.segments.num_tokens);
    } else {
        const SegmentTile tile = locate_tile(args.segments, pieces.tokens, index);
        if (tile.count == 0) return;
        segment = tile.segment;
        begin = tile.first;
        end = tile.first + tile.count;
        piece = (tile.first - tile.begin) / pieces.tokens;
        last_piece = (tile.end - tile.begin - 1) / pieces.tokens;
        // offsets that go back name more pieces than there is room for: a segment that reaches beyond is left out
        if (segment_end_tile(tile, pieces.tokens, index) > gridDim.x / column_blocks / args.heads) return;
        if (PASS == Pass::kContribute && piece == last_piece) return;
    }
    const size_t slot = args.segments.slots[segment];
    if (slot >= args.segments.num_request_slots) {
        return;
    }
    const uint32_t group = head / (args.heads / args.groups);
    const size_t inner = static_cast<size_t>(args.heads) * args.vdim;
    const uint32_t column0 = block * kColumns;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t row0 = lane >> 2;
    const uint32_t pair = (lane & 3) * 2;
    const float skip = __bfloat162float(args.skip[head]);
    // state between pieces of piece `other` of this segment
    auto state_between = [&](uint32_t other) {
        return pieces.states +
               ((static_cast<size_t>(index - piece + other) * args.heads + head) * column_blocks + block) * args.size * kColumns;
    };
    auto decay_between = [&](uint32_t other) -> float& {
        return pieces.decays[static_cast<size_t>(index - piece + other) * args.heads + head];
    };

    auto load_chunk = [&](uint32_t first, uint32_t buffer) {
        __nv_bfloat16* b = tiles + buffer * tile_elements;
        __nv_bfloat16* c = b + kTokens * pitch;
        __nv_bfloat16* x = c + kTokens * pitch;
        const uint32_t vectors = padded / 8;
        for (uint32_t item = threadIdx.x; item < kTokens * vectors; item += kThreads) {
            const uint32_t row = item / vectors, n = item % vectors * 8;
            const bool inside = first + row < end && (FULL || n < args.size);
            const __nv_bfloat16* source = args.mixed;
            if (inside) source += static_cast<size_t>(first + row) * args.mixed_pitch + inner + group * args.size + n;
            copy_async_16(b + row * pitch + n, source, inside);
            if (PASS != Pass::kContribute) {
                copy_async_16(c + row * pitch + n, source + (inside ? args.groups * args.size : 0), inside);
            }
        }
        for (uint32_t item = threadIdx.x; item < kTokens * kColumns / 8; item += kThreads) {
            const uint32_t row = item / (kColumns / 8), v = item % (kColumns / 8) * 8;
            const bool inside = first + row < end && column0 + v < args.vdim;
            copy_async_16(x + row * kColumnPitch + v,
                       args.mixed + (inside ? static_cast<size_t>(first + row) * args.mixed_pitch + head * args.vdim +
                                                  column0 + v
                                            : 0),
                       inside);
        }
        if (threadIdx.x < kTokens) {
            // tokens behind the end weigh nothing (their x is zero), and their decays are the last token's
            const uint32_t token = first + threadIdx.x < end ? first + threadIdx.x : end - 1;
            copy_async_16(factor_tiles + (first - begin) / kTokens % 2 * kTokens + threadIdx.x,
                          pieces.factors + static_cast<size_t>(head) * args.segments.num_tokens + token, true);
        }
        copy_async_commit();
    };

    float* state = state_of(args, slot, head);
    float held[UNITS][4][4];
    // calls `visit` with the address of each pair of state values that this thread holds, as rows `row_pitch` apart
    auto each_pair = [&](float* base, size_t row_pitch, auto&& visit) {
#pragma unroll
        for (int unit = 0; unit < UNITS; ++unit) {
            const uint32_t part = warp + 8 * unit;
            const uint32_t n = part / 2 * 16 + row0;
#pragma unroll
            for (uint32_t tile = 0; tile < 4; ++tile) {
                const uint32_t v = part % 2 * 32 + tile * 8 + pair;
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {
                    if (n + half * 8 < args.size && column0 + v < args.vdim) {
                        visit(reinterpret_cast<float2*>(base + static_cast<size_t>(n + half * 8) * row_pitch + v),
                              held[unit][tile][2 * half], held[unit][tile][2 * half + 1]);
                    }
                }
            }
        }
    };
    const auto read = [](const float2* at, float& x, float& y) {
        const float2 value = *at;
        x = value.x;
        y = value.y;
    };
    const auto write = [](float2* at, float x, float y) { *at = make_float2(x, y); };
#pragma unroll
    for (int unit = 0; unit < UNITS; ++unit) {
#pragma unroll
        for (uint32_t tile = 0; tile < 4; ++tile) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) held[unit][tile][i] = 0.0f;
        }
    }
    if (begin < end) load_chunk(begin, 0);
    float total_log = 0.0f;                        // of this piece's decay
    if (PASS == Pass::kWhole || last_piece == 0) {
        each_pair(state + column0, args.vdim, read);
    } else if (PASS == Pass::kContribute) {
        // the first piece takes the state before the segment along and leaves a copy where the last piece's would be:
        // the record is overwritten by whichever CTA of the second pass comes to its end
        if (piece == 0) {
            each_pair(state + column0, args.vdim, read);
            each_pair(state_between(last_piece), kColumns, write);
        }
    } else if (piece == 0) {
        each_pair(state_between(last_piece), kColumns, read);
    } else {
        each_pair(state_between(0), kColumns, read);
        for (uint32_t other = 1; other < piece; ++other) {
            const float decay = fast_exp2(decay_between(other));
            each_pair(state_between(other), kColumns, [decay](const float2* at, float& x, float& y) {
                const float2 value = *at;
                x = fmaf(x, decay, value.x);
                y = fmaf(y, decay, value.y);
            });
        }
    }
    uint32_t buffer = 0;
    for (uint32_t first = begin; first < end; first += kTokens) {
        copy_async_wait<0>();
        __syncthreads();
        if (buffers == 2 && first + kTokens < end) load_chunk(first + kTokens, buffer ^ 1);
        const __nv_bfloat16* b = tiles + buffer * tile_elements;
        const __nv_bfloat16* c = b + kTokens * pitch;
        const __nv_bfloat16* x = c + kTokens * pitch;
        const TokenFactors* factors = factor_tiles + (first - begin) / kTokens % 2 * kTokens;
        // ---- the state and the weighted inputs as two bf16 parts each
#pragma unroll
        for (int unit = 0; unit < UNITS; ++unit) {
            const uint32_t part = warp + 8 * unit;
            if (PASS != Pass::kContribute && part / 2 * 16 < padded) {
#pragma unroll
                for (uint32_t tile = 0; tile < 4; ++tile) {
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        uint32_t high, low;
                        split_pair(held[unit][tile][2 * half], held[unit][tile][2 * half + 1], high, low);
                        const uint32_t row = part / 2 * 16 + row0 + half * 8;
                        const uint32_t at = row * kColumnPitch + part % 2 * 32 + tile * 8 + pair;
                        *reinterpret_cast<uint32_t*>(state_high + at) = high;
                        *reinterpret_cast<uint32_t*>(state_low + at) = low;
                    }
                }
            }
        }
#pragma unroll
        for (uint32_t item = threadIdx.x; item < kTokens * kColumns / 8; item += kThreads) {
            const uint32_t row = item / (kColumns / 8), v = item % (kColumns / 8) * 8;
            float value[8];
            load_values<8>(x + row * kColumnPitch + v, value);
            const float weight = factors[row].into_state;
            uint32_t high[4], low[4];
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) split_pair(value[2 * i] * weight, value[2 * i + 1] * weight, high[i], low[i]);
            *reinterpret_cast<uint4*>(input_high + row * kColumnPitch + v) = make_uint4(high[0], high[1], high[2], high[3]);
            *reinterpret_cast<uint4*>(input_low + row * kColumnPitch + v) = make_uint4(low[0], low[1], low[2], low[3]);
        }
        __syncthreads();

        // ---- outputs: 16 tokens x 32 columns per warp
        if (PASS != Pass::kContribute) {
            const uint32_t tile_row = warp & 3;
            const uint32_t half_column = (warp >> 2) * 32;
            float products[8][4] = {}, carried[4][4] = {};
#pragma unroll 2
            for (uint32_t k = 0; k < padded; k += 16) {
                uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
                ldmatrix_x4(smem_u32(c + (tile_row * 16 + (lane & 15)) * pitch + k + (lane >> 4) * 8), a0, a1, a2, a3);
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    if (j <= tile_row) {
                        ldmatrix_x4(smem_u32(b + (j * 16 + (lane >> 4) * 8 + (lane & 7)) * pitch + k + (lane >> 3 & 1) * 8),
                                    b0, b1, b2, b3);
                        mma_bf16_16816(products[2 * j], a0, a1, a2, a3, b0, b1);
                        mma_bf16_16816(products[2 * j + 1], a0, a1, a2, a3, b2, b3);
                    }
                }
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    const uint32_t at = (k + (lane >> 3 & 1) * 8 + (lane & 7)) * kColumnPitch + half_column + q * 16 +
                                        (lane >> 4) * 8;
                    ldmatrix_x4_trans(smem_u32(state_high + at), b0, b1, b2, b3);
                    mma_bf16_16816(carried[2 * q], a0, a1, a2, a3, b0, b1);
                    mma_bf16_16816(carried[2 * q + 1], a0, a1, a2, a3, b2, b3);
                    ldmatrix_x4_trans(smem_u32(state_low + at), b0, b1, b2, b3);
                    mma_bf16_16816(carried[2 * q], a0, a1, a2, a3, b0, b1);
                    mma_bf16_16816(carried[2 * q + 1], a0, a1, a2, a3, b2, b3);
                }
            }
            const uint32_t t[2] = {tile_row * 16 + row0, tile_row * 16 + row0 + 8};
            const float log_high[2] = {factors[t[0]].log_high, factors[t[1]].log_high};
            const float log_low[2] = {factors[t[0]].log_low, factors[t[1]].log_low};
            float sum[4][4] = {};
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                if (j > tile_row) {
                    continue;
                }
                uint32_t high[4], low[4];
#pragma unroll
                for (uint32_t part = 0; part < 2; ++part) {            // 8 tokens s each
                    const uint32_t s = j * 16 + part * 8 + pair;
                    const TokenFactors from[2] = {factors[s], factors[s + 1]};
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        const float first_weight =
                            fast_exp2((log_high[half] - from[0].log_high) + (log_low[half] - from[0].log_low)) * from[0].step;
                        const float second_weight =
                            fast_exp2((log_high[half] - from[1].log_high) + (log_low[half] - from[1].log_low)) * from[1].step;
                        const float first_value = s <= t[half] ? products[2 * j + part][2 * half] * first_weight : 0.0f;
                        const float second_value =
                            s + 1 <= t[half] ? products[2 * j + part][2 * half + 1] * second_weight : 0.0f;
                        split_pair(first_value, second_value, high[2 * part + half], low[2 * part + half]);
                    }
                }
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(smem_u32(x + (j * 16 + (lane >> 3 & 1) * 8 + (lane & 7)) * kColumnPitch + half_column +
                                               q * 16 + (lane >> 4) * 8),
                                      b0, b1, b2, b3);
                    mma_bf16_16816(sum[2 * q], high[0], high[1], high[2], high[3], b0, b1);
                    mma_bf16_16816(sum[2 * q + 1], high[0], high[1], high[2], high[3], b2, b3);
                    mma_bf16_16816(sum[2 * q], low[0], low[1], low[2], low[3], b0, b1);
                    mma_bf16_16816(sum[2 * q + 1], low[0], low[1], low[2], low[3], b2, b3);
                }
            }
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                const uint32_t token = first + t[half];
                const float carry = fast_exp2(log_high[half] + log_low[half]);
                if (token < end) {
#pragma unroll
                    for (uint32_t tile = 0; tile < 4; ++tile) {
                        const uint32_t local = half_column + tile * 8 + pair;
                        if (column0 + local < args.vdim) {
                            const float2 input = __bfloat1622float2(
                                *reinterpret_cast<const __nv_bfloat162*>(x + t[half] * kColumnPitch + local));
                            const float low = fmaf(skip, input.x, fmaf(carry, carried[tile][2 * half], sum[tile][2 * half]));
                            const float high =
                                fmaf(skip, input.y, fmaf(carry, carried[tile][2 * half + 1], sum[tile][2 * half + 1]));
                            *reinterpret_cast<uint32_t*>(args.out + token * inner + head * args.vdim + column0 + local) =
                                pack_bf16x2(low, high);
                        }
                    }
                }
            }
        }

        // ---- the state behind the chunk
        const float chunk_log = factors[kTokens - 1].log_high + factors[kTokens - 1].log_low;
        const float decay = fast_exp2(chunk_log);
        total_log += chunk_log;
#pragma unroll
        for (int unit = 0; unit < UNITS; ++unit) {
            const uint32_t part = warp + 8 * unit;
            const uint32_t n0 = part / 2 * 16;
            if (n0 >= padded) {
                continue;
            }
#pragma unroll
            for (uint32_t tile = 0; tile < 4; ++tile) {
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) held[unit][tile][i] *= decay;
            }
#pragma unroll
            for (uint32_t k = 0; k < kTokens; k += 16) {
                uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
                ldmatrix_x4_trans(smem_u32(b + (k + (lane >> 4) * 8 + (lane & 7)) * pitch + n0 + (lane >> 3 & 1) * 8), a0, a1,
                                  a2, a3);
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    const uint32_t at = (k + (lane >> 3 & 1) * 8 + (lane & 7)) * kColumnPitch + part % 2 * 32 + q * 16 +
                                        (lane >> 4) * 8;
                    ldmatrix_x4_trans(smem_u32(input_high + at), b0, b1, b2, b3);
                    mma_bf16_16816(held[unit][2 * q], a0, a1, a2, a3, b0, b1);
                    mma_bf16_16816(held[unit][2 * q + 1], a0, a1, a2, a3, b2, b3);
                    ldmatrix_x4_trans(smem_u32(input_low + at), b0, b1, b2, b3);
                    mma_bf16_16816(held[unit][2 * q], a0, a1, a2, a3, b0, b1);
                    mma_bf16_16816(held[unit][2 * q + 1], a0, a1, a2, a3, b2, b3);
                }
            }
        }
        __syncthreads();
        if (buffers == 2) {
            buffer ^= 1;
        } else if (first + kTokens < end) {
            load_chunk(first + kTokens, 0);
        }
    }
    if (PASS == Pass::kContribute) {
        each_pair(state_between(piece), kColumns, write);
        if (threadIdx.x == 0 && block == 0) decay_between(piece) = total_log;
    } else if (piece == last_piece) {
        each_pair(state + column0, args.vdim, write);
    }
}

}  // namespace

bool state_space_chunk_supports(const StateSpaceLaunch& launch) {
    return launch.type == Activation::kBf16 && launch.factors != nullptr && launch.segments.offsets != nullptr &&
           launch.size % 8 == 0 && launch.size <= 256 && launch.vdim % 8 == 0 && launch.mixed_pitch % 8 == 0 && aligned_to(launch.mixed, 16) &&
           aligned_to(launch.out, 4) && launch.record.offset % 16 == 0 && launch.record.stride % 16 == 0 &&
           aligned_to(launch.record.base, 16);
}

// Segments are cut so that the pieces of all heads are resident side by side, two per SM: where one CTA per segment and head
// fills more than half of that, the contributions' extra pass (a quarter of the work) would not pay.  Pieces of fewer than
// four chunks are not worth their launch: a whole step with one prompt of 600 tokens (two pieces) 2989 -> 2760 us, of 200
// tokens (not cut) 1961 -> 1886 us by the rest of this file's changes.
constexpr size_t kResident = 2 * 148;
constexpr size_t kShortestPiece = 4;               // chunks

size_t state_space_factor_bytes(size_t heads, size_t tokens) { return heads * tokens * sizeof(TokenFactors); }

size_t state_space_piece_bytes(uint32_t heads, uint32_t size, uint32_t vdim, size_t tokens) {
    if (tokens < 2 * kShortestPiece * kTokens) return 0;
    // as many pieces as fill the device, and one more for each of the at most kResident / 2 segments and heads
    const size_t column_blocks = (vdim + kColumns - 1) / kColumns;
    return (kResident + kResident / 2 + static_cast<size_t>(heads) * column_blocks) * (size * kColumns + 1) * sizeof(float);
}

cudaError_t launch_state_space_chunk(cudaStream_t stream, const StateSpaceLaunch& launch) {
    const uint32_t padded = (launch.size + 15) / 16 * 16;
    const uint32_t column_blocks = (launch.vdim + kColumns - 1) / kColumns;
    const size_t per_segment = static_cast<size_t>(launch.heads) * column_blocks;
    const StateSpaceArgs<__nv_bfloat16> args = state_space_args<__nv_bfloat16>(launch);
    PieceArgs pieces = {};
    TokenFactors* factors = static_cast<TokenFactors*>(launch.factors);
    pieces.factors = factors;
    const size_t segments = launch.segments.num_segments;
    const size_t tokens = launch.segments.num_tokens - launch.decode_tokens;     // of segments with more than one
    const uint32_t head_blocks = (launch.heads + kFactorHeads - 1) / kFactorHeads;
    cudaError_t status = launch_kernel(state_space_factors_kernel,
                                       static_cast<unsigned int>((tokens / kTokens + segments) * head_blocks), kThreads, 0,
                                       stream, 1, args, factors, head_blocks);
    if (status != cudaSuccess) return status;

    // Pieces: as many per segment as the device holds side by side, none shorter than kShortestPiece chunks.
    const size_t chunks = (tokens + segments * kTokens - 1) / (segments * kTokens);      // of an average segment
    const size_t wanted = std::min(kResident / (segments * per_segment), chunks / kShortestPiece);
    bool split = wanted >= 2;
    size_t bound = segments;
    if (split) {
        const size_t piece_chunks = (chunks + wanted - 1) / wanted;
        pieces.tokens = static_cast<uint32_t>(piece_chunks * kTokens);
        bound = tokens / pieces.tokens + segments;
        const size_t state_floats = bound * per_segment * launch.size * kColumns;
        pieces.states = launch.pieces;
        pieces.decays = launch.pieces + state_floats;
        split = launch.pieces != nullptr && (state_floats + bound * launch.heads) * sizeof(float) <= launch.piece_bytes;
        if (!split) bound = segments;
    }
    const size_t blocks = bound * per_segment;
    const auto go = [&](auto kernel, bool outputs) {
        // two CTAs per SM hide each other's loads; a second buffer does where it fits beside that or there are not enough CTAs
        const bool alone = blocks <= 148 || shared_bytes(padded, 1, outputs) > kSharedLimit / 2 - 1024;
        const uint32_t buffers =
            shared_bytes(padded, 2, outputs) <= (alone ? kSharedLimit : kSharedLimit / 2 - 1024) ? 2 : 1;
        const size_t shared = shared_bytes(padded, buffers, outputs);
        const cudaError_t set = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                     cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared));
        if (set != cudaSuccess) return set;
        return launch_kernel(kernel, static_cast<unsigned int>(blocks), kThreads, shared, stream, 1, args, pieces, column_blocks,
                             padded, buffers);
    };
    const auto sized = [&](auto units) {
        constexpr int kUnits = decltype(units)::value;
        const auto passes = [&](auto full) {
            constexpr bool kFull = decltype(full)::value;
            if (!split) return go(state_space_chunk_kernel<kUnits, Pass::kWhole, kFull>, true);
            const cudaError_t first = go(state_space_chunk_kernel<kUnits, Pass::kContribute, kFull>, false);
            return first == cudaSuccess ? go(state_space_chunk_kernel<kUnits, Pass::kPieces, kFull>, true) : first;
        };
        return launch.size == 64 * kUnits ? passes(std::true_type()) : passes(std::false_type());
    };
    return padded <= 64    ? sized(std::integral_constant<int, 1>())
           : padded <= 128 ? sized(std::integral_constant<int, 2>())
                           : sized(std::integral_constant<int, 4>());
}

}  // namespace lfm25

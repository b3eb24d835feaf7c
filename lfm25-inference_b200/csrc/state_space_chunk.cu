// State-space recurrence over prompts as matrix products (the chunked form of Dao and Gu 2024), for bf16 activations and states
// of up to 256 rows.
//
// With a_t = exp(-rate dt_t), A_t = a_1 ... a_t inside a chunk of 64 tokens and S the state before it,
//     y_t = A_t S^T C_t + sum_{s <= t} (A_t / A_s) dt_s (C_t . B_s) x_s + skip x_t
//     S  <- A_64 S + sum_s (A_64 / A_s) dt_s B_s x_s^T
// A CTA owns one segment, one head and 64 columns of its state, and walks the segment chunk by chunk.  Four warps carry 16
// columns of the state each, transposed, in f32 accumulators: these are operands of C S as they are, and x^T B is added to
// them.  Four more warps copy the next chunk and form the triangle of weights from C B^T, which does not wait for the state,
// and leave it in the order of the operands.  The two sides meet twice per chunk.  x, B and C are bf16 already;
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
// Bound by the tensor cores' legacy products where two CTAs share an SM (336 of 16x8x16 per chunk and SM quarter each, eight
// cycles apiece, of 7300 cycles that two chunks take), and by the chain C S, outputs, x^T B of one warp elsewhere (5400 cycles a
// chunk).  Shapes in use have strides known to the compiler.  One segment of 4096 tokens, 64 heads with 128 state rows: 6 us
// factors, 30 us contributions, 89 us pieces; one CTA per head from end to end: 295 us on 64 SMs.  8 x 512 tokens of 32 heads
// with 64 state rows: 30 us.  With all eight warps on one stage after another and the state and weighted x between them in shared
// memory it was 35 + 133 us, 301 and 45 us.
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

// What a token contributes to a head: log2 A_t as high + low, dt_t, (A_64 / A_t) dt_t
struct __align__(16) TokenFactors {
    float log_high, log_low, step, into_state;
};

enum class Pass {
    kWhole,         // a CTA walks a whole segment
    kContribute,    // every piece but a segment's last: the state behind it, from zero (the first piece: from the record)
    kPieces,        // every piece: outputs, the state behind the last one
};

// Bytes of one buffer of a chunk's B, C (where there are outputs) and x
__host__ __device__ constexpr size_t chunk_bytes(uint32_t padded, bool outputs) {
    return ((outputs ? 2 : 1) * kTokens * (padded + kPad) + kTokens * kColumnPitch) * 2;
}
constexpr uint32_t kBlocks = 10;                        // 16 x 16 blocks on and below the diagonal of a chunk's weights
constexpr size_t kWeightBytes = kBlocks * 2 * 32 * 16;  // in two bf16 parts, as operands
constexpr size_t shared_bytes(uint32_t padded, bool outputs) {
    return 2 * (chunk_bytes(padded, outputs) + (outputs ? kWeightBytes : 0) + kTokens * sizeof(TokenFactors));
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

constexpr uint32_t kRoleThreads = kThreads / 2;
enum : uint32_t { kFullBarrier = 1, kFreeBarrier = 3, kLoadedBarrier = 5 };      // the first two: one per buffer

__device__ __forceinline__ void barrier_sync(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void barrier_arrive(uint32_t id, uint32_t threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Warps 0..3 own the state, warps 4..7 load and weigh.  168 and 88 registers a thread: with 160 and 96 the state's warps spill
// (8 x 512 tokens 31.9 instead of 30.0 us), 176 and 80 are no faster.
// UNITS: 64 state rows each.  FULL: the state has exactly that many rows, so that all strides are constants and the loops over
// them unroll.
template <int UNITS, Pass PASS, bool FULL>
__global__ void __launch_bounds__(kThreads, UNITS <= 2 ? 2 : 1)
state_space_chunk_kernel(const StateSpaceArgs<__nv_bfloat16> args, const PieceArgs pieces, uint32_t column_blocks,
                         uint32_t padded_rows) {
    constexpr uint32_t kTiles = 8 * UNITS;             // of eight state rows
    const uint32_t padded = FULL ? 64 * UNITS : padded_rows;
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    const uint32_t pitch = padded + kPad;
    __nv_bfloat16* tiles = reinterpret_cast<__nv_bfloat16*>(chunk_smem);
    const uint32_t tile_elements = static_cast<uint32_t>(chunk_bytes(padded, PASS != Pass::kContribute) / 2);
    uint4* weights = reinterpret_cast<uint4*>(tiles + 2 * tile_elements);        // [2][block][part][lane]
    TokenFactors* factor_tiles =                                                 // [2][tokens]
        reinterpret_cast<TokenFactors*>(weights + (PASS == Pass::kContribute ? 0 : 2 * kBlocks * 2 * 32));
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
    const size_t inner = static_cast<size_t>(args.heads) * args.vdim;
    const uint32_t column0 = block * kColumns;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t row0 = lane >> 2;
    const uint32_t pair = (lane & 3) * 2;
    const auto inputs_of = [&](uint32_t buffer) { return tiles + buffer * tile_elements; };      // B, then C, then x
    const auto columns_of = [&](uint32_t buffer) {
        return inputs_of(buffer) + (PASS == Pass::kContribute ? 1 : 2) * kTokens * pitch;
    };

    if (warp >= kRoleThreads / 32) {
        // ---- copies, and the weights of each chunk's inputs in its outputs: at most three blocks of 16 x 16 per warp
        if constexpr (UNITS <= 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        const uint32_t thread = threadIdx.x - kRoleThreads;
        const uint32_t weigher = warp - kRoleThreads / 32;
        const uint32_t group = head / (args.heads / args.groups);
        // eight threads per row, 16 rows at a time; behind the end and beyond the state's size zeros
        const uint32_t row = thread / 8, vector = thread % 8 * 8;
        const __nv_bfloat16* source = args.mixed + static_cast<size_t>(begin + row) * args.mixed_pitch;
        const size_t first_row = static_cast<size_t>(inner) + group * args.size, second_row = args.groups * args.size;
        const bool column_inside = column0 + vector < args.vdim;
        const size_t column = column_inside ? head * args.vdim + column0 + vector : 0;
        const TokenFactors* source_factors = pieces.factors + static_cast<size_t>(head) * args.segments.num_tokens;
        const auto load_chunk = [&](uint32_t first, uint32_t buffer) {
            __nv_bfloat16* b = inputs_of(buffer) + row * pitch + vector;
            __nv_bfloat16* c = b + kTokens * pitch;
            __nv_bfloat16* x = columns_of(buffer) + row * kColumnPitch + vector;
#pragma unroll
            for (uint32_t i = 0; i < kTokens; i += 16) {
                const bool inside = first + row + i < end;
                const __nv_bfloat16* at = inside ? source + i * args.mixed_pitch : args.mixed;
#pragma unroll
                for (uint32_t n = 0; n < 64 * UNITS; n += 64) {
                    if (!FULL && n + vector >= padded) continue;
                    const bool filled = inside && (FULL || n + vector < args.size);
                    const __nv_bfloat16* from = filled ? at + first_row + n + vector : args.mixed;
                    copy_async_16(b + i * pitch + n, from, filled);
                    if (PASS != Pass::kContribute) {
                        copy_async_16(c + i * pitch + n, filled ? from + second_row : args.mixed, filled);
                    }
                }
                copy_async_16(x + i * kColumnPitch, at + (inside ? column : 0), inside && column_inside);
            }
            if (thread < kTokens) {
                // tokens behind the end weigh nothing (their x is zero), and their decays are the last token's
                const uint32_t token = first + thread < end ? first + thread : end - 1;
                copy_async_16(factor_tiles + buffer * kTokens + thread, source_factors + token, true);
            }
            copy_async_commit();
            source += kTokens * args.mixed_pitch;
        };
        if (begin < end) load_chunk(begin, 0);
        uint32_t buffer = 0;
        for (uint32_t first = begin; first < end; first += kTokens, buffer ^= 1) {
            copy_async_wait<0>();
            if (PASS != Pass::kContribute) {
                barrier_sync(kLoadedBarrier, kRoleThreads);
                const __nv_bfloat16* b = inputs_of(buffer);
                const __nv_bfloat16* c = b + kTokens * pitch;
                const TokenFactors* factors = factor_tiles + buffer * kTokens;
                // blocks (kRow, kFirst) to (kRow, kLast)
                const auto weigh = [&](auto row_index, auto first_index, auto last_index) {
                    constexpr uint32_t kRow = decltype(row_index)::value, kFirst = decltype(first_index)::value;
                    constexpr uint32_t kCount = decltype(last_index)::value + 1 - kFirst;
                    float products[2 * kCount][4] = {};
#pragma unroll 4
                    for (uint32_t k = 0; k < padded; k += 16) {
                        uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
                        ldmatrix_x4(smem_u32(c + (kRow * 16 + (lane & 15)) * pitch + k + (lane >> 4) * 8), a0, a1, a2, a3);
#pragma unroll
                        for (uint32_t j = 0; j < kCount; ++j) {
                            ldmatrix_x4(smem_u32(b + ((kFirst + j) * 16 + (lane >> 4) * 8 + (lane & 7)) * pitch + k +
                                                 (lane >> 3 & 1) * 8),
                                        b0, b1, b2, b3);
                            mma_bf16_16816(products[2 * j], a0, a1, a2, a3, b0, b1);
                            mma_bf16_16816(products[2 * j + 1], a0, a1, a2, a3, b2, b3);
                        }
                    }
                    const float log_high[2] = {factors[kRow * 16 + row0].log_high, factors[kRow * 16 + row0 + 8].log_high};
                    const float log_low[2] = {factors[kRow * 16 + row0].log_low, factors[kRow * 16 + row0 + 8].log_low};
                    uint4* target = weights + ((buffer * kBlocks + kRow * (kRow + 1) / 2 + kFirst) * 2) * 32 + lane;
#pragma unroll
                    for (uint32_t j = 0; j < kCount; ++j) {
                        uint32_t high[4], low[4];
#pragma unroll
                        for (uint32_t part = 0; part < 2; ++part) {            // 8 tokens s each
                            const uint32_t s = part * 8 + pair;
                            const TokenFactors* at = factors + (kFirst + j) * 16 + s;
                            const TokenFactors from[2] = {at[0], at[1]};
#pragma unroll
                            for (uint32_t half = 0; half < 2; ++half) {
                                float value[2];
#pragma unroll
                                for (uint32_t i = 0; i < 2; ++i) {
                                    const float weight = fast_exp2((log_high[half] - from[i].log_high) +
                                                                   (log_low[half] - from[i].log_low)) * from[i].step;
                                    value[i] = kFirst + j != kRow || s + i <= row0 + half * 8
                                                   ? products[2 * j + part][2 * half + i] * weight
                                                   : 0.0f;
                                }
                                split_pair(value[0], value[1], high[2 * part + half], low[2 * part + half]);
                            }
                        }
                        target[j * 64] = make_uint4(high[0], high[1], high[2], high[3]);
                        target[j * 64 + 32] = make_uint4(low[0], low[1], low[2], low[3]);
                    }
                };
                const std::integral_constant<uint32_t, 0> zero;
                const std::integral_constant<uint32_t, 1> one;
                const std::integral_constant<uint32_t, 2> two;
                const std::integral_constant<uint32_t, 3> three;
                const uint32_t left = end - first;             // rows behind the end have no outputs
                if (weigher == 0) {
                    weigh(zero, zero, zero);
                    if (left > 48) weigh(three, zero, zero);
                } else if (weigher == 1) {
                    if (left > 16) weigh(one, zero, one);
                } else if (weigher == 2) {
                    if (left > 32) weigh(two, zero, two);
                } else {
                    if (left > 48) weigh(three, one, three);
                }
            }
            barrier_arrive(kFullBarrier + buffer, kThreads);
            if (first + kTokens < end) {
                if (first != begin) barrier_sync(kFreeBarrier + (buffer ^ 1), kThreads);
                load_chunk(first + kTokens, buffer ^ 1);
            }
        }
        return;
    }

    // ---- the state, transposed: 16 columns and all rows per warp
    if constexpr (UNITS <= 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const float skip = __bfloat162float(args.skip[head]);
    float* state = state_of(args, slot, head);
    float held[kTiles][4];
    const uint32_t own = warp * 16;                    // first column
    // calls `visit` with the address in the record and the value
    const auto each_value = [&](auto&& visit) {
        const uint32_t column = column0 + own + row0;
        const bool inside[2] = {column < args.vdim, column + 8 < args.vdim};
        float* at = state + static_cast<size_t>(pair) * args.vdim + column;
#pragma unroll
        for (uint32_t tile = 0; tile < kTiles; ++tile) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t n = tile * 8 + pair + (i & 1);
                if ((FULL || n < args.size) && inside[i >> 1]) visit(at + (i & 1) * args.vdim + (i >> 1) * 8, held[tile][i]);
            }
            at += 8 * args.vdim;
        }
    };
    const auto read = [](const float* at, float& x) { x = *at; };
    const auto write = [](float* at, float x) { *at = x; };
    // state between pieces of piece `other` of this segment, in the order of the registers: [warp][tile][lane][4]
    const auto each_between = [&](uint32_t other, auto&& visit) {
        float4* base = reinterpret_cast<float4*>(
                           pieces.states + ((static_cast<size_t>(index - piece + other) * args.heads + head) * column_blocks +
                                            block) * args.size * kColumns) +
                       warp * (args.size / 8) * 32 + lane;
#pragma unroll
        for (uint32_t tile = 0; tile < kTiles; ++tile) {
            if (tile * 8 < args.size) visit(base + tile * 32, held[tile]);
        }
    };
    const auto read_between = [](const float4* at, float (&x)[4]) {
        const float4 value = *at;
        x[0] = value.x;
        x[1] = value.y;
        x[2] = value.z;
        x[3] = value.w;
    };
    const auto write_between = [](float4* at, const float (&x)[4]) { *at = make_float4(x[0], x[1], x[2], x[3]); };
    const auto decay_between = [&](uint32_t other) -> float& {
        return pieces.decays[static_cast<size_t>(index - piece + other) * args.heads + head];
    };
#pragma unroll
    for (uint32_t tile = 0; tile < kTiles; ++tile) {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) held[tile][i] = 0.0f;
    }
    float total_log = 0.0f;                            // of this piece's decay
    if (PASS == Pass::kWhole || last_piece == 0) {
        each_value(read);
    } else if (PASS == Pass::kContribute) {
        // the first piece takes the state before the segment along and leaves a copy where the last piece's would be:
        // the record is overwritten by whichever CTA of the second pass comes to its end
        if (piece == 0) {
            each_value(read);
            each_between(last_piece, write_between);
        }
    } else if (piece == 0) {
        each_between(last_piece, read_between);
    } else {
        each_between(0, read_between);
        for (uint32_t other = 1; other < piece; ++other) {
            const float decay = fast_exp2(decay_between(other));
            each_between(other, [decay](const float4* at, float (&x)[4]) {
                const float4 value = *at;
                x[0] = fmaf(x[0], decay, value.x);
                x[1] = fmaf(x[1], decay, value.y);
                x[2] = fmaf(x[2], decay, value.z);
                x[3] = fmaf(x[3], decay, value.w);
            });
        }
    }
    const uint32_t columns_left = column0 + own + pair < args.vdim ? args.vdim - column0 - own - pair : 0;
    __nv_bfloat16* target = args.out + (static_cast<size_t>(begin) + row0) * inner + head * args.vdim + column0 + own + pair;
    uint32_t buffer = 0;
    for (uint32_t first = begin; first < end; first += kTokens, buffer ^= 1) {
        barrier_sync(kFullBarrier + buffer, kThreads);
        const __nv_bfloat16* b = inputs_of(buffer);
        const __nv_bfloat16* c = b + kTokens * pitch;
        const __nv_bfloat16* x = columns_of(buffer) + own;
        const TokenFactors* factors = factor_tiles + buffer * kTokens;
        if (PASS != Pass::kContribute) {
            // ---- from the state: its accumulators are operands as they are
            float carried[4][2][4] = {};
            uint32_t tokens[2][4][4];                  // C of 16 state rows, and of the next ones
            const auto load_tokens = [&](uint32_t q) {
#pragma unroll
                for (uint32_t row_tile = 0; row_tile < 4; ++row_tile) {
                    uint32_t(&a)[4] = tokens[q % 2][row_tile];
                    ldmatrix_x4(smem_u32(c + (row_tile * 16 + (lane & 15)) * pitch + q * 16 + (lane >> 4) * 8), a[0], a[1], a[2],
                                a[3]);
                }
            };
            load_tokens(0);
#pragma unroll
            for (uint32_t q = 0; q < kTiles / 2; ++q) {
                if (!FULL && q * 16 >= padded) continue;
                if (q + 1 < kTiles / 2 && (FULL || (q + 1) * 16 < padded)) load_tokens(q + 1);
                uint32_t high[4], low[4];
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {        // of the columns
                    split_pair(held[2 * q][2 * half], held[2 * q][2 * half + 1], high[2 * half], low[2 * half]);
                    split_pair(held[2 * q + 1][2 * half], held[2 * q + 1][2 * half + 1], high[2 * half + 1],
                               low[2 * half + 1]);
                }
#pragma unroll
                for (uint32_t part = 0; part < 2; ++part) {
                    const uint32_t(&state_part)[4] = part == 0 ? high : low;
#pragma unroll
                    for (uint32_t row_tile = 0; row_tile < 4; ++row_tile) {
                        const uint32_t(&a)[4] = tokens[q % 2][row_tile];
                        mma_bf16_16816(carried[row_tile][0], a[0], a[1], a[2], a[3], state_part[0], state_part[1]);
                        mma_bf16_16816(carried[row_tile][1], a[0], a[1], a[2], a[3], state_part[2], state_part[3]);
                    }
                }
            }
            // ---- from the chunk's own inputs
            const uint32_t rows_left = end - first > row0 ? end - first - row0 : 0;
            float carries[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const TokenFactors& token = factors[i * 8 + row0];
                carries[i] = fast_exp2(token.log_high + token.log_low);
            }
            uint32_t inputs[4][4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                ldmatrix_x4_trans(smem_u32(x + (j * 16 + (lane >> 3 & 1) * 8 + (lane & 7)) * kColumnPitch + (lane >> 4) * 8),
                                  inputs[j][0], inputs[j][1], inputs[j][2], inputs[j][3]);
            }
#pragma unroll
            for (uint32_t first_tile = 0; first_tile < 4; first_tile += 2) {
                float sum[2][2][4] = {};
#pragma unroll
                for (uint32_t j = 0; j < first_tile + 2; ++j) {
                    uint4 part[2][2];
#pragma unroll
                    for (uint32_t r = 0; r < 2; ++r) {
                        const uint32_t row_tile = first_tile + r;
                        if (j > row_tile) continue;
                        const uint4* source =
                            weights + ((buffer * kBlocks + row_tile * (row_tile + 1) / 2 + j) * 2) * 32 + lane;
                        part[r][0] = source[0];
                        part[r][1] = source[32];
                    }
#pragma unroll
                    for (uint32_t p = 0; p < 2; ++p) {
#pragma unroll
                        for (uint32_t r = 0; r < 2; ++r) {
                            if (j > first_tile + r) continue;
                            const uint4& a = part[r][p];
                            mma_bf16_16816(sum[r][0], a.x, a.y, a.z, a.w, inputs[j][0], inputs[j][1]);
                            mma_bf16_16816(sum[r][1], a.x, a.y, a.z, a.w, inputs[j][2], inputs[j][3]);
                        }
                    }
                }
#pragma unroll
                for (uint32_t r = 0; r < 2; ++r) {
                    const uint32_t row_tile = first_tile + r;
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        const uint32_t t = row_tile * 16 + half * 8;
                        const float carry = carries[2 * row_tile + half];
#pragma unroll
                        for (uint32_t tile = 0; tile < 2; ++tile) {
                            const float2 input = __bfloat1622float2(
                                *reinterpret_cast<const __nv_bfloat162*>(x + (t + row0) * kColumnPitch + tile * 8 + pair));
                            const float even = fmaf(
                                skip, input.x, fmaf(carry, carried[row_tile][tile][2 * half], sum[r][tile][2 * half]));
                            const float odd = fmaf(
                                skip, input.y, fmaf(carry, carried[row_tile][tile][2 * half + 1], sum[r][tile][2 * half + 1]));
                            if (t < rows_left && tile * 8 < columns_left) {
                                *reinterpret_cast<uint32_t*>(target + t * inner + tile * 8) = pack_bf16x2(even, odd);
                            }
                        }
                    }
                }
            }
            target += kTokens * inner;
        }

        // ---- the state behind the chunk
        const float chunk_log = factors[kTokens - 1].log_high + factors[kTokens - 1].log_low;
        const float decay = fast_exp2(chunk_log);
        total_log += chunk_log;
#pragma unroll
        for (uint32_t tile = 0; tile < kTiles; ++tile) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) held[tile][i] *= decay;
        }
        uint32_t rows[2][2][4];                        // B of 16 tokens and 32 state rows, and of the next ones
        constexpr uint32_t kGroups = kTiles / 4;
        const auto load_rows = [&](uint32_t step) {
            const uint32_t k = step / kGroups * 16;
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const uint32_t q = step % kGroups * 2 + i;
                if (!FULL && q * 16 >= padded) continue;
                uint32_t(&out)[4] = rows[step % 2][i];
                ldmatrix_x4_trans(smem_u32(b + (k + (lane >> 3 & 1) * 8 + (lane & 7)) * pitch + q * 16 + (lane >> 4) * 8),
                                  out[0], out[1], out[2], out[3]);
            }
        };
        load_rows(0);
        uint32_t high[4], low[4];
#pragma unroll
        for (uint32_t step = 0; step < kTokens / 16 * kGroups; ++step) {
            if (step + 1 < kTokens / 16 * kGroups) load_rows(step + 1);
            if (step % kGroups == 0) {
                const uint32_t k = step / kGroups * 16;
                uint32_t raw[4];
                ldmatrix_x4_trans(smem_u32(x + (k + (lane >> 4) * 8 + (lane & 7)) * kColumnPitch + (lane >> 3 & 1) * 8),
                                  raw[0], raw[1], raw[2], raw[3]);
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const uint32_t t = k + (i >> 1) * 8 + pair;
                    const float2 value = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[i]));
                    split_pair(value.x * factors[t].into_state, value.y * factors[t + 1].into_state, high[i], low[i]);
                }
            }
#pragma unroll
            for (uint32_t part = 0; part < 2; ++part) {
                const uint32_t(&a)[4] = part == 0 ? high : low;
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    const uint32_t q = step % kGroups * 2 + i;
                    if (!FULL && q * 16 >= padded) continue;
                    const uint32_t(&row)[4] = rows[step % 2][i];
                    mma_bf16_16816(held[2 * q], a[0], a[1], a[2], a[3], row[0], row[1]);
                    mma_bf16_16816(held[2 * q + 1], a[0], a[1], a[2], a[3], row[2], row[3]);
                }
            }
        }
        if (end - first > 2 * kTokens) barrier_arrive(kFreeBarrier + buffer, kThreads);
    }
    if (PASS == Pass::kContribute) {
        each_between(piece, write_between);
        if (threadIdx.x == 0 && block == 0) decay_between(piece) = total_log;
    } else if (piece == last_piece) {
        each_value(write);
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
        split = launch.pieces != nullptr && aligned_to(launch.pieces, 16) &&
                (state_floats + bound * launch.heads) * sizeof(float) <= launch.piece_bytes;
        if (!split) bound = segments;
    }
    const size_t blocks = bound * per_segment;
    const auto go = [&](auto kernel, bool outputs) {
        const size_t shared = shared_bytes(padded, outputs);
        const cudaError_t set = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                     cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared));
        if (set != cudaSuccess) return set;
        return launch_kernel(kernel, static_cast<unsigned int>(blocks), kThreads, shared, stream, 1, args, pieces, column_blocks,
                             padded);
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
    // Three units by themselves: in four, 16 heads of 64 columns with 192 state rows took 74 instead of 46 us (8 x 512 tokens; 74
    // with all warps on one stage after another), and a step of 8 x 5 tokens 99 instead of 83 us (87).
    return padded <= 64    ? sized(std::integral_constant<int, 1>())
           : padded <= 128 ? sized(std::integral_constant<int, 2>())
           : padded <= 192 ? sized(std::integral_constant<int, 3>())
                           : sized(std::integral_constant<int, 4>());
}

}  // namespace lfm25

// The generalised delta rule over prompts in plain f32 arithmetic, for every activation type and head size (f32 activations,
// and the bf16 shapes that the tensor-core kernels of delta_rule.cu do not take).
//
// Per token and value column the recurrence is a short serial chain (dot product, two shuffles, two multiply-adds), and that
// chain is all that has to be serial.  What the tokens contribute (decays, removal rates, unit keys) belongs to one token
// alone, and the columns of a head's state never meet.  Three kernels:
//     elements   r, w, -(a * u), u, k, v of every token and head in f32          tiles of 16 tokens x heads, side by side
//     scan       the recurrence; the result of a token takes the place of its v  8 or 16 value columns a CTA
//     output     norm and gate                                                   one warp per token and head
// What bounds them: `scan` the latency of the chain (about 290 cycles a token in heads of 64), so a head's columns are spread
// over as many CTAs as there are groups of eight or sixteen, operands arrive through cp.async a tile ahead and, for heads up to
// 128, in registers a token ahead, and the result of a token is reduced beside the dot product of the next one.  Eight lanes a
// column: with four a thread's reads of its operands outweigh the shorter sum, with sixteen nothing is left to win (48, 60 and
// 48 us below).  `elements` lets its successor in at its end only: CTAs of `scan` that start early are put on the SMs that
// `elements` has left free, several on one, and share its issue slots and shared memory for the whole scan (81 -> 116).
// 250 tokens, 16 heads of 64 with ranks of 64: 47 us for the three; preparation and recurrence in turns in one CTA per head:
// 219 us.  Eight segments of 200 tokens: 143 and 234 us; 16 heads of 128 with ranks of 224, bf16: 425 and 451 us.
#include <algorithm>

#include "delta_rule.h"
#include "launch.h"

namespace lfm25 {

namespace {

constexpr uint32_t kElementTokens = 16;      // tokens per CTA of the elements kernel
// Values of tanh(z) per token that a launch of the elements kernel holds in shared memory; larger ranks take several launches,
// which leave the logits in the place of w.
constexpr uint32_t kRankBlock = 760;
// 128 threads are as many as 16 tokens of 32 channels need
constexpr __host__ __device__ uint32_t element_threads(uint32_t dim) { return dim <= 32 ? 128 : 256; }
constexpr uint32_t kVectors = 6;             // r, w, -(a * u), u, k, v
constexpr uint32_t kValues = 5;              // place of v, and of the result after the scan

// f32 vectors of a group of heads: [token][head of the group][vector][pitch], pitch = head size in whole float4, padding zero.
struct ScanVectors {
    float* base;
    uint32_t first_head, heads, pitch;
    __device__ __forceinline__ float* at(size_t token, uint32_t head) const {
        return base + (token * heads + head) * kVectors * pitch;
    }
};

__host__ __device__ constexpr uint32_t padded_rank(uint32_t count) { return (count + 7) / 8 * 8; }
// Columns of W2 in shared memory at a time, and elements between its rows: an odd number of 16-byte pieces, so that the rows'
// pieces lie in different banks.
template <uint32_t DP>
constexpr uint32_t kTileRank = DP <= 64 ? 512 : (DP <= 128 ? 320 : 160);
template <uint32_t DP>
__host__ __device__ constexpr uint32_t tile_pitch(uint32_t z_count) {
    return ((z_count < kTileRank<DP> ? padded_rank(z_count) : kTileRank<DP>) / 8 | 1) * 8;
}
template <uint32_t DP>
constexpr size_t element_bytes(uint32_t z_count) {
    return kElementTokens * (1 + static_cast<size_t>(padded_rank(z_count))) * sizeof(float) +
           static_cast<size_t>(DP) * tile_pitch<DP>(z_count) * 2;
}
static_assert(kRankBlock % 8 == 0 && element_bytes<128>(kRankBlock) <= 227 * 1024 && element_bytes<256>(kRankBlock) <= 227 * 1024,
              "whole pieces, in shared memory");

// One channel and groups of four tokens per thread, so that a value of W2 serves four tokens.  W2 is constant and on its way to
// shared memory before the dependency wait; from global memory a thread's row would fetch 32 bytes for every 16 that are used.
// Bound by the latency of its loads, so registers are kept for four CTAs of 256 threads per SM, and a round trip to memory serves
// keys, z and the first tokens' values.  1600 tokens of 32 heads of 64 with ranks of 64, f32: 67 us, and 120 with W2 from global
// memory and 64 values of a row in registers; 16 heads of 128 with ranks of 256, bf16: 144 and 419 us.
template <typename T, uint32_t DP>
__global__ void __launch_bounds__(element_threads(DP), 1024 / element_threads(DP))
delta_scan_elements_kernel(const DeltaArgs<T> args, const ScanVectors vectors, uint32_t first_z, uint32_t z_count) {
    constexpr uint32_t kThreads = element_threads(DP), kWarps = kThreads / 32;
    extern __shared__ __align__(16) float element_shared[];
    const uint32_t padded_z = padded_rank(z_count);
    float* unit_scale = element_shared;                                // [token]
    float* z_values = element_shared + kElementTokens;                 // [token][padded_z], tanh applied, zeros behind z_count
    auto* tile = reinterpret_cast<__nv_bfloat16*>(z_values + kElementTokens * padded_z);      // of W2, [channel][pitch]
    const uint32_t pitch = tile_pitch<DP>(z_count);
    const uint32_t head = blockIdx.x % vectors.heads;
    const size_t first = static_cast<size_t>(blockIdx.x / vectors.heads) * kElementTokens;
    const uint32_t tokens = static_cast<uint32_t>(min(args.segments.num_tokens - first, size_t(kElementTokens)));
    const uint32_t dim = args.dim;
    const size_t width = static_cast<size_t>(args.heads) * dim;
    const size_t head_base = static_cast<size_t>(vectors.first_head + head) * dim;
    constexpr uint32_t kGroups = kThreads / DP;
    const uint32_t channel = threadIdx.x % DP;
    const bool live = channel < dim;
    const size_t index = head_base + (live ? channel : 0);
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    // W2 from z on, zeros behind z_count and the head's channels, in the largest pieces that every row can be read in
    const __nv_bfloat16* decay_rows = args.decay_up + head_base * args.rank + first_z;
    const uint32_t alignment = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(args.decay_up) | args.rank * 2);
    auto load_tile = [&](uint32_t z) {
        const uint32_t count = min(z_count - z, kTileRank<DP>), columns = padded_rank(count);
        for (uint32_t row = warp; row < DP; row += kWarps) {
            const __nv_bfloat16* source = decay_rows + static_cast<size_t>(row) * args.rank + z;
            __nv_bfloat16* target = tile + row * pitch;
            if (alignment % 16 == 0) {
                for (uint32_t column = lane * 8; column < columns; column += 256) {
                    copy_async_16(target + column, row < dim ? source + column : args.decay_up, row < dim);
                }
            } else if (alignment % 4 == 0) {
                for (uint32_t column = lane * 2; column < columns; column += 64) {
                    const bool inside = row < dim && column < count;   // the rank is even
                    copy_async_4(target + column, inside ? source + column : args.decay_up, inside);
                }
            } else {
                for (uint32_t column = lane; column < columns; column += 32) {
                    target[column] = row < dim && column < count ? source[column] : __float2bfloat16_rn(0.0f);
                }
            }
        }
        copy_async_commit();
    };
    load_tile(0);
    const float bias = __bfloat162float(args.removal_bias[index]), base = __bfloat162float(args.decay_base[index]);
    pdl_wait();
    if (first + tokens <= args.segments.offsets[0]) {
        copy_async_wait<0>();
        return;                                                        // single tokens in front of the prompts
    }
    float r[4], k[4], v[4], rate[4];
    auto load_tokens = [&](uint32_t t0) {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            r[i] = k[i] = v[i] = rate[i] = 0.0f;
            if (live && t0 + i < tokens) {
                const T* row = args.projected + (first + t0 + i) * args.pitch + index;
                r[i] = to_float<T>(row[0]);
                k[i] = to_float<T>(row[width]);
                v[i] = to_float<T>(row[2 * width]);
                rate[i] = to_float<T>(row[4 * width]);
            }
        }
    };
    load_tokens(threadIdx.x / DP * 4);                                 // on their way while norms and tanh(z) are formed
    for (uint32_t t = warp; t < kElementTokens; t += kWarps) {
        const T* row = args.projected + (first + t) * args.pitch;
        float keys[DP / 32], sum = 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < DP / 32; ++i) {
            keys[i] = t < tokens && lane + i * 32 < dim ? to_float<T>(row[width + head_base + lane + i * 32]) : 0.0f;
        }
        for (uint32_t z0 = lane; z0 < padded_z; z0 += 128) {           // four loads at a time
            float raw[4];
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t z = z0 + i * 32;
                raw[i] = t < tokens && z < z_count ? to_float<T>(row[5 * width + first_z + z]) : 0.0f;
            }
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                if (z0 + i * 32 < padded_z) z_values[t * padded_z + z0 + i * 32] = tanhf(raw[i]);
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < DP / 32; ++i) sum = fmaf(keys[i], keys[i], sum);
        sum = warp_sum(sum);
        if (lane == 0) unit_scale[t] = 1.0f / sqrtf(sum + kUnitEps);
    }
    copy_async_wait<0>();
    __syncthreads();
    // products of eight values of W2 with those of four tokens, in the order of the values
    auto add_products = [&](const uint4& raw, uint32_t t0, uint32_t z, float (&logit)[4]) {
        const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
            const float2 low = __bfloat1622float2(pairs[2 * half]);
            const float2 high = __bfloat1622float2(pairs[2 * half + 1]);
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const float4 value = *reinterpret_cast<const float4*>(z_values + (t0 + i) * padded_z + z + half * 4);
                logit[i] = fmaf(low.x, value.x, logit[i]);
                logit[i] = fmaf(low.y, value.y, logit[i]);
                logit[i] = fmaf(high.x, value.z, logit[i]);
                logit[i] = fmaf(high.y, value.w, logit[i]);
            }
        }
    };
    uint32_t held = 0;                                                 // where the tile in shared memory begins
    for (uint32_t turn = 0; turn < tokens; turn += kGroups * 4) {
        const uint32_t t0 = threadIdx.x / DP * 4 + turn;
        if (turn > 0) load_tokens(t0);
        float logit[4] = {};
        if (first_z > 0 && channel < vectors.pitch) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                if (t0 + i < tokens) logit[i] = vectors.at(first + t0 + i, head)[vectors.pitch + channel];
            }
        }
        const uint32_t row0 = min(t0, kElementTokens - 4);             // threads without tokens stay for the barriers
        for (uint32_t z = 0; z < z_count; z += kTileRank<DP>) {
            if (z != held) {
                __syncthreads();
                load_tile(z);
                copy_async_wait<0>();
                __syncthreads();
                held = z;
            }
            const uint32_t count = min(z_count - z, kTileRank<DP>);
            for (uint32_t at = 0; at < count; at += 8) {
                add_products(*reinterpret_cast<const uint4*>(tile + channel * pitch + at), row0, z + at, logit);
            }
        }
        if (channel >= vectors.pitch) continue;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const uint32_t t = t0 + i;
            if (t >= tokens) break;
            float* target = vectors.at(first + t, head) + channel;
            if (first_z + z_count < args.rank) {
                target[1 * vectors.pitch] = logit[i];
                continue;
            }
            float w = 0.0f, removal = 0.0f, u = 0.0f;
            if (live) {
                w = expf(-kDecayScale * sigmoidf(logit[i] + base));
                u = k[i] * unit_scale[t];
                removal = -sigmoidf(rate[i] + bias) * u;
            }
            target[0 * vectors.pitch] = r[i];
            target[1 * vectors.pitch] = w;
            target[2 * vectors.pitch] = removal;
            target[3 * vectors.pitch] = u;
            target[4 * vectors.pitch] = k[i];
            target[kValues * vectors.pitch] = v[i];
        }
    }
}

// LANES threads a column, each with the key channels of every LANES-th group of four.
template <uint32_t DP, uint32_t LANES, uint32_t COLUMNS>
struct ScanShape {
    static constexpr uint32_t kThreads = LANES * COLUMNS;
    static constexpr uint32_t kRows = DP / LANES;
    static constexpr uint32_t kGroups = kRows / 4;
    // Per stage.  Heads beyond 128: with 8 two CTAs fit an SM instead of four (bf16, 4 heads of 160, 8 x 200 tokens 369 -> 281 us
    // a layer; one prompt of 4096 tokens pays 3 %).
    static constexpr uint32_t kTokens = DP <= 64 ? 16 : (DP <= 128 ? 8 : 4);
    static constexpr uint32_t kTokenFloats = 5 * DP + COLUMNS;         // r, w, removal, u, k over DP channels, v
    static constexpr uint32_t kPieces = (kTokenFloats / 4 + 31) / 32;       // 16-byte pieces of a token per lane of a warp
    static constexpr size_t kShared = (2 * kTokens + 1) * kTokenFloats * sizeof(float);
    static_assert(kRows % 4 == 0 && kTokenFloats % 4 == 0, "four consecutive key channels per access");
    static_assert(kShared <= 227 * 1024, "shared memory");
};

template <uint32_t GROUPS>
struct ScanToken {
    ulonglong2 r[GROUPS], w[GROUPS], removal[GROUPS], u[GROUPS], k[GROUPS];
    float v;
};

template <typename T, uint32_t DP, uint32_t LANES, uint32_t COLUMNS>
__global__ void __launch_bounds__(ScanShape<DP, LANES, COLUMNS>::kThreads)
delta_scan_kernel(const DeltaArgs<T> args, const ScanVectors vectors) {
    using Shape = ScanShape<DP, LANES, COLUMNS>;
    constexpr uint32_t kThreads = Shape::kThreads, kGroups = Shape::kGroups, kTokens = Shape::kTokens;
    pdl_wait();
    extern __shared__ __align__(16) float scan_shared[];                   // [2][kTokens][kTokenFloats], one more token
    const uint32_t dim = args.dim, pitch = vectors.pitch;
    const uint32_t split = blockIdx.x % args.splits;
    const uint32_t head = blockIdx.x / args.splits % vectors.heads;
    const uint32_t segment = blockIdx.x / args.splits / vectors.heads;
    const uint32_t begin = args.segments.offsets[segment];
    uint32_t end = args.segments.offsets[segment + 1];
    end = end < args.segments.num_tokens ? end : static_cast<uint32_t>(args.segments.num_tokens);
    const size_t slot = args.segments.slots[segment];
    if (begin >= end || slot >= args.segments.num_request_slots) {
        return;
    }
    const uint32_t lane = threadIdx.x % LANES;
    const uint32_t own = threadIdx.x / LANES;                              // column of this CTA
    const uint32_t column = split * COLUMNS + own;
    const bool live = column < dim;
    const size_t head_base = static_cast<size_t>(vectors.first_head + head) * dim;
    float* state_column = reinterpret_cast<float*>(static_cast<unsigned char*>(args.record.base) +
                                                   slot * args.record.stride + args.record.offset) +
                          (head_base + column) * dim;
    const bool vector_state = dim % 4 == 0;
    Pair state[kGroups * 2];
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const uint32_t row = (g * LANES + lane) * 4;
        float4 value = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live && row < dim) {
            if (vector_state) {
                value = *reinterpret_cast<const float4*>(state_column + row);
            } else {
                value.x = state_column[row];
                if (row + 1 < dim) value.y = state_column[row + 1];
                if (row + 2 < dim) value.z = state_column[row + 2];
                if (row + 3 < dim) value.w = state_column[row + 3];
            }
        }
        state[2 * g] = pair_of(value.x, value.y);
        state[2 * g + 1] = pair_of(value.z, value.w);
    }
    // channels behind the pitch are never copied and stay zero
    if (pitch < DP) {
        for (uint32_t item = threadIdx.x; item < (2 * kTokens + 1) * Shape::kTokenFloats / 4; item += kThreads) {
            reinterpret_cast<float4*>(scan_shared)[item] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        __syncthreads();
    }

    // 16-byte pieces of a token: r, w, removal, u, k and this CTA's part of v.  A warp moves a token; where its lanes' pieces
    // lie does not change.
    const uint32_t per_vector = pitch / 4;
    const uint32_t pieces = 5 * per_vector + min(pitch - split * COLUMNS, COLUMNS) / 4;
    uint32_t from[Shape::kPieces], to[Shape::kPieces];
#pragma unroll
    for (uint32_t i = 0; i < Shape::kPieces; ++i) {
        const uint32_t piece = threadIdx.x % 32 + i * 32;
        const uint32_t vector = min(piece / per_vector, kValues), part = piece - vector * per_vector;
        from[i] = vector * pitch + (vector < kValues ? 0 : split * COLUMNS) + part * 4;
        to[i] = vector * DP + part * 4;
    }
    auto load_stage = [&](uint32_t first, float* stage) {
        const uint32_t tokens = first < end ? min(end - first, kTokens) : 0;
        for (uint32_t t = threadIdx.x / 32; t < tokens; t += kThreads / 32) {
            const float* source = vectors.at(first + t, head);
            float* target = stage + t * Shape::kTokenFloats;
#pragma unroll
            for (uint32_t i = 0; i < Shape::kPieces; ++i) {
                if (threadIdx.x % 32 + i * 32 < pieces) copy_async_16(target + to[i], source + from[i], true);
            }
        }
        copy_async_commit();
    };
    auto load_token = [&](const float* token, ScanToken<kGroups>& out) {
#pragma unroll
        for (uint32_t g = 0; g < kGroups; ++g) {
            const float* at = token + (g * LANES + lane) * 4;
            out.u[g] = *reinterpret_cast<const ulonglong2*>(at + 3 * DP);
            out.w[g] = *reinterpret_cast<const ulonglong2*>(at + 1 * DP);
            out.removal[g] = *reinterpret_cast<const ulonglong2*>(at + 2 * DP);
            out.k[g] = *reinterpret_cast<const ulonglong2*>(at + 4 * DP);
            out.r[g] = *reinterpret_cast<const ulonglong2*>(at);
        }
        out.v = token[5 * DP + own];
    };
    float pending = 0.0f;              // this thread's part of the result of the token before
    // S <- diag(w) S - (a u) (u^T S) + k v^T; the result of the token before is reduced beside u^T S and returned
    auto step = [&](const ScanToken<kGroups>& token) -> float {
        Pair dot0 = 0, dot1 = 0;                                           // bit pattern of (0.0f, 0.0f)
#pragma unroll
        for (uint32_t g = 0; g < kGroups; ++g) {
            dot0 = fma_pair(token.u[g].x, state[2 * g], dot0);
            dot1 = fma_pair(token.u[g].y, state[2 * g + 1], dot1);
        }
        float dot = pair_sum(dot0) + pair_sum(dot1);
        float before = pending;
        // w S does not depend on the sum over the lanes
#pragma unroll
        for (uint32_t g = 0; g < kGroups; ++g) {
            state[2 * g] = mul_pair(token.w[g].x, state[2 * g]);
            state[2 * g + 1] = mul_pair(token.w[g].y, state[2 * g + 1]);
        }
#pragma unroll
        for (uint32_t delta = 1; delta < LANES; delta <<= 1) {
            dot += __shfl_xor_sync(0xffffffffu, dot, delta);
            before += __shfl_xor_sync(0xffffffffu, before, delta);
        }
        const Pair recalled = pair_of(dot, dot);
        const Pair values = pair_of(token.v, token.v);
        Pair sum0 = 0, sum1 = 0;
#pragma unroll
        for (uint32_t g = 0; g < kGroups; ++g) {
            state[2 * g] = fma_pair(token.k[g].x, values, fma_pair(token.removal[g].x, recalled, state[2 * g]));
            state[2 * g + 1] = fma_pair(token.k[g].y, values, fma_pair(token.removal[g].y, recalled, state[2 * g + 1]));
            sum0 = fma_pair(token.r[g].x, state[2 * g], sum0);
            sum1 = fma_pair(token.r[g].y, state[2 * g + 1], sum1);
        }
        pending = pair_sum(sum0) + pair_sum(sum1);
        return before;
    };
    const size_t token_stride = static_cast<size_t>(vectors.heads) * kVectors * pitch;
    // where the result of the token before the current one goes
    float* result = vectors.at(begin, head) + kValues * pitch + column;
    const bool writes = lane == 0 && live;
    bool started = false;
    auto store = [&](float value) {
        if (writes && started) *result = value;
        result += started ? token_stride : 0;
        started = true;
    };

    load_stage(begin, scan_shared);
    for (uint32_t first = begin, stage = 0; first < end; first += kTokens, stage ^= 1) {
        load_stage(first + kTokens, scan_shared + (stage ^ 1) * kTokens * Shape::kTokenFloats);
        copy_async_wait<1>();
        __syncthreads();
        const float* tokens = scan_shared + stage * kTokens * Shape::kTokenFloats;
        const uint32_t count = min(end - first, kTokens);
        if constexpr (kGroups <= 4) {
            ScanToken<kGroups> even, odd;
            load_token(tokens, even);
            uint32_t t = 0;
            for (; t + 2 <= count; t += 2) {
                load_token(tokens + (t + 1) * Shape::kTokenFloats, odd);
                store(step(even));
                load_token(tokens + (t + 2) * Shape::kTokenFloats, even);      // behind the tile: not used
                store(step(odd));
            }
            if (t < count) store(step(even));
        } else {
            for (uint32_t t = 0; t < count; ++t) {
                ScanToken<kGroups> now;
                load_token(tokens + t * Shape::kTokenFloats, now);
                store(step(now));
            }
        }
        __syncthreads();
    }
    pdl_launch_dependents();
#pragma unroll
    for (uint32_t delta = 1; delta < LANES; delta <<= 1) pending += __shfl_xor_sync(0xffffffffu, pending, delta);
    store(pending);

#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const uint32_t row = (g * LANES + lane) * 4;
        if (live && row < dim) {
            const float4 value = {low_of(state[2 * g]), high_of(state[2 * g]), low_of(state[2 * g + 1]),
                                  high_of(state[2 * g + 1])};
            if (vector_state) {
                *reinterpret_cast<float4*>(state_column + row) = value;
            } else {
                state_column[row] = value.x;
                if (row + 1 < dim) state_column[row + 1] = value.y;
                if (row + 2 < dim) state_column[row + 2] = value.z;
                if (row + 3 < dim) state_column[row + 3] = value.w;
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(128)
delta_scan_output_kernel(const DeltaArgs<T> args, const ScanVectors vectors) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t item = static_cast<size_t>(blockIdx.x) * 4 + threadIdx.x / 32;
    const size_t token = item / vectors.heads;
    const uint32_t head = static_cast<uint32_t>(item % vectors.heads);
    if (token >= args.segments.num_tokens || token < args.segments.offsets[0]) {
        return;
    }
    const size_t head_base = static_cast<size_t>(vectors.first_head + head) * args.dim;
    const uint32_t lane = threadIdx.x & 31;
    const float* raw = vectors.at(token, head) + kValues * vectors.pitch;
    const T* gate = args.projected + token * args.pitch + 3 * static_cast<size_t>(args.heads) * args.dim + head_base;
    float sum = 0.0f;
    for (uint32_t channel = lane; channel < args.dim; channel += 32) sum = fmaf(raw[channel], raw[channel], sum);
    const float scale = inverse_rms(warp_sum(sum), args.dim, args.eps);
    for (uint32_t channel = lane; channel < args.dim; channel += 32) {
        const float normalised = raw[channel] * scale * __bfloat162float(args.norm[head_base + channel]);
        args.out[token * args.out_pitch + head_base + channel] =
            from_float<T>(normalised * sigmoidf(to_float<T>(gate[channel])));
    }
}

size_t head_bytes(size_t tokens, uint32_t dim) { return tokens * kVectors * ((dim + 3) / 4 * 4) * sizeof(float); }

// of kernels without static shared memory
template <typename Kernel>
cudaError_t allow_shared(Kernel kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(bytes));
}

template <typename T, uint32_t DP, uint32_t LANES, uint32_t COLUMNS>
cudaError_t launch_sized(cudaStream_t stream, DeltaArgs<T> args, ScanVectors vectors, uint32_t heads_at_once) {
    using Shape = ScanShape<DP, LANES, COLUMNS>;
    const size_t tokens = args.segments.num_tokens;
    args.splits = (args.dim + COLUMNS - 1) / COLUMNS;
    const auto elements = delta_scan_elements_kernel<T, DP>;
    const auto scan = delta_scan_kernel<T, DP, LANES, COLUMNS>;
    cudaError_t status = allow_shared(scan, Shape::kShared);
    if (status == cudaSuccess) status = allow_shared(elements, element_bytes<DP>(std::min(args.rank, kRankBlock)));
    for (uint32_t first = 0; first < args.heads && status == cudaSuccess; first += heads_at_once) {
        vectors.first_head = first;
        vectors.heads = std::min(heads_at_once, args.heads - first);
        const size_t tiles = (tokens + kElementTokens - 1) / kElementTokens;
        for (uint32_t first_z = 0; first_z < args.rank && status == cudaSuccess; first_z += kRankBlock) {
            const uint32_t z_count = std::min(args.rank - first_z, kRankBlock);
            status = launch_kernel(elements, static_cast<unsigned int>(tiles * vectors.heads), element_threads(DP),
                                   element_bytes<DP>(z_count), stream, 1, args, vectors, first_z, z_count);
        }
        if (status != cudaSuccess) break;
        status = launch_kernel(scan, static_cast<unsigned int>(args.segments.num_segments * vectors.heads * args.splits),
                               Shape::kThreads, Shape::kShared, stream, 1, args, vectors);
        if (status != cudaSuccess) break;
        status = launch_kernel(delta_scan_output_kernel<T>, static_cast<unsigned int>((tokens * vectors.heads + 3) / 4), 128,
                               0, stream, 1, args, vectors);
    }
    return status;
}

}  // namespace

size_t delta_scan_bytes(size_t heads, uint32_t dim, size_t tokens) {
    return std::max(head_bytes(tokens, dim), std::min(heads * head_bytes(tokens, dim), kDeltaChunkBytes));
}

template <typename T>
cudaError_t launch_delta_scan(cudaStream_t stream, const DeltaArgs<T>& args, float* scratch, size_t scratch_bytes) {
    const size_t one = head_bytes(args.segments.num_tokens, args.dim);
    if (scratch == nullptr || one == 0 || one > scratch_bytes || args.dim > kDeltaMaxDim) return cudaErrorInvalidValue;
    const uint32_t at_once = static_cast<uint32_t>(std::min<size_t>(args.heads, scratch_bytes / one));
    const ScanVectors vectors = {scratch, 0, 0, (args.dim + 3) / 4 * 4};
    if (args.dim <= 32) return launch_sized<T, 32, 8, 8>(stream, args, vectors, at_once);
    if (args.dim <= 64) return launch_sized<T, 64, 8, 8>(stream, args, vectors, at_once);
    if (args.dim <= 128) return launch_sized<T, 128, 8, 16>(stream, args, vectors, at_once);
    return launch_sized<T, 256, 8, 16>(stream, args, vectors, at_once);
}

template cudaError_t launch_delta_scan<float>(cudaStream_t, const DeltaArgs<float>&, float*, size_t);
template cudaError_t launch_delta_scan<__nv_bfloat16>(cudaStream_t, const DeltaArgs<__nv_bfloat16>&, float*, size_t);

}  // namespace lfm25

// The generalised delta rule with a decay per key channel:
//     u_t = k_t / sqrt(|k_t|^2 + 1e-6)
//     S_t = diag(w_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T          o_t = S_t^T r_t
// per head, with w_t = exp(-exp(-1/2) sigmoid(W2 tanh(z_t) + w0)) and a_t = sigmoid(a_t' + bias), followed by the
// head's RMS norm, the norm weight and the output gate.
//
// A column of S (one value channel) never meets another one, so a CTA takes the columns of one head of one sequence and
// keeps them in registers over the whole segment: the state is read from and written to memory once per step however
// long the segment is.  Few long bf16 segments are split along the sequence instead (delta_split.cu).  Kernels for single tokens:
//   decode    one token per sequence: every load is issued up front, then three barriers
//   general   one token per sequence, head sizes and ranks beyond the decode kernel
// and for prompts:
//   chunk     bf16 segments, heads up to 64, ranks up to 128: tiles of 16 tokens as matrix products on the tensor cores
//             (delta_chunk.cu), or split along the sequence (delta_split.cu)
//   prompt    bf16 segments, heads up to 128, ranks up to 256: half of the warps prepare a tile of 16 tokens (decays with one
//             small tensor-core product, removal rates, unit scales) and finish the previous one (norm, gate), the others run
//             the recurrence over the tile between them; projections arrive through cp.async two tiles ahead
//   scan      every other segment, f32 ones among them, token by token in three kernels (delta_scan.cu)
// Outside delta_chunk.cu and delta_split.cu all arithmetic on the state is f32 multiply-adds, two-wide where the
// sm_100 packed instructions take it (each half rounds like the scalar one).
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "delta_rule.h"
#include "launch.h"
#include "options.h"

namespace lfm25 {

namespace {

// per token in shared memory: r, w, -(a * u), u, k over the padded key channels, then v over them as well
constexpr uint32_t kVectors = 6;

template <uint32_t DP>
size_t delta_shared_bytes(uint32_t rank) {
    return ((kVectors + 1) * DP + (rank + 3) / 4 * 4 + 4) * sizeof(float);
}

// What one token's projections turn into for one key channel.
struct Prepared {
    float r, w, removal, u, k, v;
};
template <typename T>
__device__ __forceinline__ Prepared prepare(const DeltaArgs<T>& args, const T* row, size_t width, size_t channel,
                                            float logit, float unit_scale) {
    Prepared p;
    p.r = to_float<T>(row[channel]);
    p.k = to_float<T>(row[width + channel]);
    p.v = to_float<T>(row[2 * width + channel]);
    const float removal = sigmoidf(to_float<T>(row[4 * width + channel]) + __bfloat162float(args.removal_bias[channel]));
    p.w = expf(-kDecayScale * sigmoidf(logit + __bfloat162float(args.decay_base[channel])));
    p.u = p.k * unit_scale;
    p.removal = -removal * p.u;
    return p;
}

// ------------------------------------------------------------------------------------------------ general kernel

// One token per sequence, for head sizes and ranks beyond the decode kernel.  LANES threads a column: what the token
// contributes is prepared in shared memory (all in f32), then a thread forms its share of u^T S, LANES threads add theirs up,
// and the same pass over its rows updates S and accumulates r^T S.
template <typename T, uint32_t DP, uint32_t LANES, uint32_t COLUMNS>
__global__ void __launch_bounds__(LANES * COLUMNS)
delta_rule_kernel(const DeltaArgs<T> args) {
    constexpr uint32_t kThreads = LANES * COLUMNS;
    constexpr uint32_t kRows = DP / LANES;              // key channels per thread, in groups of four
    constexpr uint32_t kGroups = kRows / 4;
    static_assert(kRows % 4 == 0, "four consecutive key channels per access");
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float shared[];
    const uint32_t dim = args.dim;
    float* vectors = shared;                                          // [kVectors][DP]
    float* produced = vectors + kVectors * DP;                        // [DP]
    float* unit_scale = produced + DP;                                // [1], padded to four
    float* z_values = unit_scale + 4;                                 // [rank], tanh applied

    const uint32_t split = blockIdx.x % args.splits;
    const uint32_t head = blockIdx.x / args.splits % args.heads;
    const size_t token = blockIdx.x / args.splits / args.heads;
    const size_t slot = args.segments.slots[token];
    if (slot >= args.segments.num_request_slots) {
        return;
    }
    const uint32_t lane = threadIdx.x % LANES;
    const uint32_t column = split * COLUMNS + threadIdx.x / LANES;
    const size_t width = static_cast<size_t>(args.heads) * dim;
    const size_t head_base = static_cast<size_t>(head) * dim;
    float* state_column = reinterpret_cast<float*>(static_cast<unsigned char*>(args.record.base) +
                                                   slot * args.record.stride + args.record.offset) +
                          (head_base + column) * dim;
    const bool live = column < dim;
    const bool vector_state = dim % 4 == 0;

    Pair state[kRows / 2];
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

    const uint32_t warp = threadIdx.x / 32;
    const uint32_t warp_lane = threadIdx.x % 32;
    const T* row = args.projected + token * args.pitch;
    if (warp == 0) {
        float sum = 0.0f;
        for (uint32_t channel = warp_lane; channel < dim; channel += 32) {
            const float value = to_float<T>(row[width + head_base + channel]);
            sum = fmaf(value, value, sum);
        }
        sum = warp_sum(sum);
        if (warp_lane == 0) *unit_scale = 1.0f / sqrtf(sum + kUnitEps);
    }
    for (uint32_t z = threadIdx.x; z < args.rank; z += kThreads) z_values[z] = tanhf(to_float<T>(row[5 * width + z]));
    __syncthreads();
    for (uint32_t channel = threadIdx.x; channel < DP; channel += kThreads) {
        Prepared p = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (channel < dim) {
            const __nv_bfloat16* source = args.decay_up + (head_base + channel) * args.rank;
            float logit = 0.0f;
            for (uint32_t z = 0; z < args.rank; ++z) logit = fmaf(__bfloat162float(source[z]), z_values[z], logit);
            p = prepare<T>(args, row, width, head_base + channel, logit, *unit_scale);
        }
        float* target = vectors + channel;
        target[0 * DP] = p.r;
        target[1 * DP] = p.w;
        target[2 * DP] = p.removal;
        target[3 * DP] = p.u;
        target[4 * DP] = p.k;
        target[5 * DP] = p.v;
    }
    __syncthreads();

    const float value = vectors[5 * DP + (column < DP ? column : 0)];
    Pair dot0 = 0, dot1 = 0;                                    // bit pattern of (0.0f, 0.0f)
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(vectors + 3 * DP + (g * LANES + lane) * 4);
        dot0 = fma_pair(u.x, state[2 * g], dot0);
        dot1 = fma_pair(u.y, state[2 * g + 1], dot1);
    }
    float dot = pair_sum(dot0) + pair_sum(dot1);
#pragma unroll
    for (uint32_t delta = 1; delta < LANES; delta <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, delta);
    const Pair recalled = pair_of(dot, dot);
    const Pair values = pair_of(value, value);
    Pair sum0 = 0, sum1 = 0;
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const float* at = vectors + (g * LANES + lane) * 4;
        const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(at);
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(at + 1 * DP);
        const ulonglong2 removal = *reinterpret_cast<const ulonglong2*>(at + 2 * DP);
        const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(at + 4 * DP);
        state[2 * g] = fma_pair(k.x, values, fma_pair(removal.x, recalled, mul_pair(w.x, state[2 * g])));
        state[2 * g + 1] = fma_pair(k.y, values, fma_pair(removal.y, recalled, mul_pair(w.y, state[2 * g + 1])));
        sum0 = fma_pair(r.x, state[2 * g], sum0);
        sum1 = fma_pair(r.y, state[2 * g + 1], sum1);
    }
    float result = pair_sum(sum0) + pair_sum(sum1);
#pragma unroll
    for (uint32_t delta = 1; delta < LANES; delta <<= 1) result += __shfl_xor_sync(0xffffffffu, result, delta);
    if (lane == 0 && live) {
        if (args.raw != nullptr) {
            args.raw[token * width + head_base + column] = result;
        } else {
            produced[column] = result;
        }
    }
    __syncthreads();
    if (args.raw == nullptr && warp == 0) {
        const T* gate = row + 3 * width + head_base;
        float sum = 0.0f;
        for (uint32_t channel = warp_lane; channel < dim; channel += 32) {
            sum = fmaf(produced[channel], produced[channel], sum);
        }
        const float scale = inverse_rms(warp_sum(sum), dim, args.eps);
        for (uint32_t channel = warp_lane; channel < dim; channel += 32) {
            const float normalised = produced[channel] * scale * __bfloat162float(args.norm[head_base + channel]);
            args.out[token * args.out_pitch + head_base + channel] =
                from_float<T>(normalised * sigmoidf(to_float<T>(gate[channel])));
        }
    }

#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const uint32_t at = (g * LANES + lane) * 4;
        if (live && at < dim) {
            const float4 held = {low_of(state[2 * g]), high_of(state[2 * g]), low_of(state[2 * g + 1]),
                                 high_of(state[2 * g + 1])};
            if (vector_state) {
                *reinterpret_cast<float4*>(state_column + at) = held;
            } else {
                state_column[at] = held.x;
                if (at + 1 < dim) state_column[at + 1] = held.y;
                if (at + 2 < dim) state_column[at + 2] = held.z;
                if (at + 3 < dim) state_column[at + 3] = held.w;
            }
        }
    }
}

// Norm and gate of heads whose columns were spread over several CTAs: one warp per token and head.
template <typename T>
__global__ void __launch_bounds__(128)
delta_output_kernel(const DeltaArgs<T> args) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t item = static_cast<size_t>(blockIdx.x) * 4 + threadIdx.x / 32;
    const size_t token = item / args.heads;
    if (token >= args.segments.num_tokens) {
        return;
    }
    const size_t width = static_cast<size_t>(args.heads) * args.dim;
    const size_t head_base = item % args.heads * args.dim;
    const uint32_t lane = threadIdx.x & 31;
    const float* raw = args.raw + token * width + head_base;
    const T* gate = args.projected + token * args.pitch + 3 * width + head_base;
    float sum = 0.0f;
    for (uint32_t channel = lane; channel < args.dim; channel += 32) sum = fmaf(raw[channel], raw[channel], sum);
    const float scale = inverse_rms(warp_sum(sum), args.dim, args.eps);
    for (uint32_t channel = lane; channel < args.dim; channel += 32) {
        const float normalised = raw[channel] * scale * __bfloat162float(args.norm[head_base + channel]);
        args.out[token * args.out_pitch + head_base + channel] =
            from_float<T>(normalised * sigmoidf(to_float<T>(gate[channel])));
    }
}


// ------------------------------------------------------------------------------------------------ decode kernel

// One token per sequence, one CTA per sequence and head; four threads per value column (for the state) and per key
// channel (for what the token contributes).
template <typename T, uint32_t DP>
__global__ void __launch_bounds__(DP * 4)
delta_decode_kernel(const DeltaArgs<T> args) {
    constexpr uint32_t kThreads = DP * 4;
    constexpr uint32_t kGroups = DP / 16;              // groups of four key channels per thread
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float shared[];
    float* r_values = shared;                          // [DP] each
    float* w_values = r_values + DP;
    float* removal_values = w_values + DP;
    float* u_values = removal_values + DP;
    float* k_values = u_values + DP;
    float* partial = k_values + DP;                    // [warps] twice: |k|^2, |o|^2
    float* z_values = partial + 2 * (kThreads / 32);   // [rank]
    const uint32_t dim = args.dim;
    const uint32_t head = blockIdx.x % args.heads;
    const size_t token = blockIdx.x / args.heads;
    const size_t slot = args.segments.slots[token];
    if (slot >= args.segments.num_request_slots) {
        return;
    }
    const uint32_t channel = threadIdx.x / 4;          // value column and key channel
    const uint32_t lane = threadIdx.x % 4;
    const bool live = channel < dim;
    const size_t width = static_cast<size_t>(args.heads) * dim;
    const size_t head_base = static_cast<size_t>(head) * dim;
    float* state_column = reinterpret_cast<float*>(static_cast<unsigned char*>(args.record.base) +
                                                   slot * args.record.stride + args.record.offset) +
                          (head_base + channel) * dim;
    const bool vector_state = dim % 4 == 0;
    Pair state[kGroups * 2];
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const uint32_t row = (g * 4 + lane) * 4;
        float4 value = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live && row < dim) {
            if (vector_state) {
                value = __ldcs(reinterpret_cast<const float4*>(state_column + row));
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
    const T* row = args.projected + token * args.pitch;
    float r = 0.0f, k = 0.0f, v = 0.0f, gate = 0.0f, removal = 0.0f, base = 0.0f, weight = 0.0f;
    if (live) {
        const size_t index = head_base + channel;
        r = to_float<T>(row[index]);
        k = to_float<T>(row[width + index]);
        v = to_float<T>(row[2 * width + index]);
        gate = to_float<T>(row[3 * width + index]);
        removal = to_float<T>(row[4 * width + index]) + __bfloat162float(args.removal_bias[index]);
        base = __bfloat162float(args.decay_base[index]);
        weight = __bfloat162float(args.norm[index]);
    }
    for (uint32_t z = threadIdx.x; z < args.rank; z += kThreads) z_values[z] = tanhf(to_float<T>(row[5 * width + z]));
    // this thread's quarter of the channel's row of W2, its first 16 values in registers before the barrier
    const uint32_t part = (args.rank / 4 + 7) / 8 * 8;
    const uint32_t from = min(lane * part, args.rank);
    const uint32_t to = lane == 3 ? args.rank : min(from + part, args.rank);
    const __nv_bfloat16* decay_row = args.decay_up + (head_base + (live ? channel : 0)) * args.rank;
    const bool vector_rank = args.rank % 8 == 0;
    uint4 early[2] = {};
    if (live && vector_rank) {
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            if (from + 8 * i < to) early[i] = *reinterpret_cast<const uint4*>(decay_row + from + 8 * i);
        }
    }
    // every channel is held by four threads
    const float k_squares = warp_sum(lane == 0 ? k * k : 0.0f);
    const uint32_t warp = threadIdx.x / 32;
    if (threadIdx.x % 32 == 0) partial[warp] = k_squares;
    __syncthreads();
    float logit = 0.0f;
    if (live) {
        if (vector_rank) {
            for (uint32_t z = from; z < to; z += 8) {
                const uint4 raw = z < from + 16 ? (z == from ? early[0] : early[1])
                                                : *reinterpret_cast<const uint4*>(decay_row + z);
                const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const float2 both = __bfloat1622float2(pairs[i]);
                    logit = fmaf(both.x, z_values[z + 2 * i], logit);
                    logit = fmaf(both.y, z_values[z + 2 * i + 1], logit);
                }
            }
        } else {
            for (uint32_t z = from; z < to; ++z) logit = fmaf(__bfloat162float(decay_row[z]), z_values[z], logit);
        }
    }
    logit += __shfl_xor_sync(0xffffffffu, logit, 1);
    logit += __shfl_xor_sync(0xffffffffu, logit, 2);
    float squares = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < kThreads / 32; ++w) squares += partial[w];
    const float u = k / sqrtf(squares + kUnitEps);
    if (lane == 0) {
        w_values[channel] = expf(-kDecayScale * sigmoidf(logit + base));
    } else if (lane == 1) {
        removal_values[channel] = -sigmoidf(removal) * u;
    } else if (lane == 2) {
        u_values[channel] = u;
        r_values[channel] = r;
    } else {
        k_values[channel] = k;
    }
    __syncthreads();
    Pair dot0 = 0, dot1 = 0;                           // bit pattern of (0.0f, 0.0f)
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const ulonglong2 unit = *reinterpret_cast<const ulonglong2*>(u_values + (g * 4 + lane) * 4);
        dot0 = fma_pair(unit.x, state[2 * g], dot0);
        dot1 = fma_pair(unit.y, state[2 * g + 1], dot1);
    }
    float dot = pair_sum(dot0) + pair_sum(dot1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
    const Pair recalled = pair_of(dot, dot);
    const Pair values = pair_of(v, v);
    Pair sum0 = 0, sum1 = 0;
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
        const uint32_t at = (g * 4 + lane) * 4;
        const ulonglong2 rr = *reinterpret_cast<const ulonglong2*>(r_values + at);
        const ulonglong2 ww = *reinterpret_cast<const ulonglong2*>(w_values + at);
        const ulonglong2 aa = *reinterpret_cast<const ulonglong2*>(removal_values + at);
        const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(k_values + at);
        state[2 * g] = fma_pair(kk.x, values, fma_pair(aa.x, recalled, mul_pair(ww.x, state[2 * g])));
        state[2 * g + 1] = fma_pair(kk.y, values, fma_pair(aa.y, recalled, mul_pair(ww.y, state[2 * g + 1])));
        sum0 = fma_pair(rr.x, state[2 * g], sum0);
        sum1 = fma_pair(rr.y, state[2 * g + 1], sum1);
        if (live && at < dim) {
            const float4 value = {low_of(state[2 * g]), high_of(state[2 * g]), low_of(state[2 * g + 1]),
                                  high_of(state[2 * g + 1])};
            if (vector_state) {
                __stcs(reinterpret_cast<float4*>(state_column + at), value);
            } else {
                state_column[at] = value.x;
                if (at + 1 < dim) state_column[at + 1] = value.y;
                if (at + 2 < dim) state_column[at + 2] = value.z;
                if (at + 3 < dim) state_column[at + 3] = value.w;
            }
        }
    }
    float result = pair_sum(sum0) + pair_sum(sum1);
    result += __shfl_xor_sync(0xffffffffu, result, 1);
    result += __shfl_xor_sync(0xffffffffu, result, 2);
    const float o_squares = warp_sum(lane == 0 && live ? result * result : 0.0f);
    if (threadIdx.x % 32 == 0) partial[kThreads / 32 + warp] = o_squares;
    __syncthreads();
    squares = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < kThreads / 32; ++w) squares += partial[kThreads / 32 + w];
    if (lane == 0 && live) {
        args.out[token * args.out_pitch + head_base + channel] =
            from_float<T>(result * inverse_rms(squares, dim, args.eps) * weight * sigmoidf(gate));
    }
}

// ------------------------------------------------------------------------------------------------ prompt kernel

// 16-byte copy global -> shared without registers
__device__ __forceinline__ void copy_async_16(void* target, const void* source) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(target)), "l"(source) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}
__device__ __forceinline__ void named_barrier(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

constexpr uint32_t kPromptTokens = 16;       // tokens per tile = rows of one MMA tile
constexpr uint32_t kRawStages = 4;           // being finished, in the recurrence, being prepared, arriving
constexpr uint32_t kPromptMaxRank = 256;

template <uint32_t DP>
struct PromptLayout {
    uint32_t rank_pad;        // multiple of 32
    uint32_t z_stride;        // bf16 elements between rows of z / W2 in shared memory: 16-byte rows, no bank conflicts
    uint32_t raw_row;         // bf16 elements per token: r | k | v | g | a (DP each) | z
    size_t raw, vectors, produced, tanh_parts, w2, constants, scale, total;
    __host__ __device__ explicit PromptLayout(uint32_t rank) {
        rank_pad = (rank + 31) / 32 * 32;
        z_stride = rank_pad + 8;
        raw_row = 5 * DP + rank_pad;
        size_t at = 0;
        raw = at;
        at += static_cast<size_t>(kRawStages) * kPromptTokens * raw_row * 2;
        vectors = at;                                             // [2][tokens][2][DP] f32: w, removal / |k|^2
        at += 2 * kPromptTokens * 2 * DP * 4;
        produced = at;                                            // [2][tokens][DP] f32
        at += 2 * kPromptTokens * DP * 4;
        tanh_parts = at;                                          // [2][tokens][z_stride] bf16: high and low parts
        at += 2 * kPromptTokens * z_stride * 2;
        w2 = at;                                                  // [DP][z_stride] bf16
        at += static_cast<size_t>(DP) * z_stride * 2;
        constants = at;                                           // [3][DP] f32: w0, removal bias, norm weight
        at += 3 * DP * 4;
        scale = at;                                               // [2][tokens] f32: 1 / |k|^2
        at += 2 * kPromptTokens * 4;
        total = at;
    }
};

// Where key channel `row` of a prepared f32 vector lies: the 4-channel groups of the eight threads that share a column
// are interleaved, so that their 16-byte reads are consecutive.
template <uint32_t DP>
__device__ __forceinline__ uint32_t interleaved(uint32_t row) {
    constexpr uint32_t kRows = DP / 8;
    return row % kRows / 4 * 32 + row / kRows * 4 + row % 4;
}

// Eight threads per group of COLUMNS value columns run the recurrence, DP / 8 consecutive key channels each; HELPERS
// threads prepare and finish.
template <uint32_t DP, uint32_t COLUMNS, uint32_t HELPERS>
__global__ void __launch_bounds__(DP / COLUMNS * 8 + HELPERS)
delta_prompt_kernel(const DeltaArgs<__nv_bfloat16> args) {
    constexpr uint32_t kRows = DP / 8;
    constexpr uint32_t kScanThreads = DP / COLUMNS * 8;
    constexpr uint32_t kHelpers = HELPERS;
    constexpr uint32_t kHelperWarps = kHelpers / 32;
    constexpr uint32_t kTokensPerHelper = kPromptTokens / kHelperWarps;   // tokens per helper warp
    static_assert(COLUMNS == 2 || COLUMNS == 4, "columns per thread");
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) unsigned char prompt_shared[];
    const PromptLayout<DP> layout(args.rank);
    const uint32_t dim = args.dim;
    const uint32_t head = blockIdx.x % args.heads;
    const uint32_t segment = blockIdx.x / args.heads;
    const uint32_t begin = args.segments.offsets[segment];
    uint32_t end = args.segments.offsets[segment + 1];
    end = end < args.segments.num_tokens ? end : static_cast<uint32_t>(args.segments.num_tokens);
    const size_t slot = args.segments.slots[segment];
    if (begin >= end || slot >= args.segments.num_request_slots) {
        return;
    }
    const uint32_t tiles = (end - begin + kPromptTokens - 1) / kPromptTokens;
    const size_t width = static_cast<size_t>(args.heads) * dim;
    const size_t head_base = static_cast<size_t>(head) * dim;
    auto* raw = reinterpret_cast<__nv_bfloat16*>(prompt_shared + layout.raw);
    auto* vectors = reinterpret_cast<float*>(prompt_shared + layout.vectors);
    auto* produced = reinterpret_cast<float*>(prompt_shared + layout.produced);
    auto* tanh_parts = reinterpret_cast<__nv_bfloat16*>(prompt_shared + layout.tanh_parts);
    auto* w2 = reinterpret_cast<__nv_bfloat16*>(prompt_shared + layout.w2);
    auto* constants = reinterpret_cast<float*>(prompt_shared + layout.constants);
    auto* scale = reinterpret_cast<float*>(prompt_shared + layout.scale);
    float* state_base = reinterpret_cast<float*>(static_cast<unsigned char*>(args.record.base) +
                                                 slot * args.record.stride + args.record.offset) +
                        head_base * dim;

    // padding channels and tokens that never arrive stay zero
    for (uint32_t item = threadIdx.x; item < kRawStages * kPromptTokens * layout.raw_row / 8;
         item += kScanThreads + kHelpers) {
        reinterpret_cast<uint4*>(raw)[item] = make_uint4(0, 0, 0, 0);
    }
    for (uint32_t item = threadIdx.x; item < DP * layout.z_stride; item += kScanThreads + kHelpers) {
        const uint32_t channel = item / layout.z_stride;
        const uint32_t z = item % layout.z_stride;
        w2[item] = channel < dim && z < args.rank ? args.decay_up[(head_base + channel) * args.rank + z]
                                                  : __float2bfloat16_rn(0.0f);
    }
    for (uint32_t channel = threadIdx.x; channel < DP; channel += kScanThreads + kHelpers) {
        const bool live = channel < dim;
        constants[channel] = live ? __bfloat162float(args.decay_base[head_base + channel]) : 0.0f;
        constants[DP + channel] = live ? __bfloat162float(args.removal_bias[head_base + channel]) : 0.0f;
        constants[2 * DP + channel] = live ? __bfloat162float(args.norm[head_base + channel]) : 0.0f;
    }
    __syncthreads();

    const bool scanner = threadIdx.x < kScanThreads;
    const uint32_t helper = threadIdx.x - kScanThreads;
    const uint32_t helper_warp = helper / 32;
    const uint32_t warp_lane = threadIdx.x % 32;

    // the 16-byte pieces of a token's row that this lane copies: offsets in the row and in the stage
    constexpr uint32_t kPieces = (5 * DP / 8 + kPromptMaxRank / 8 + 31) / 32;
    const uint32_t per_vector = dim / 8;
    const uint32_t pieces = 5 * per_vector + (args.rank + 7) / 8;
    auto piece_offsets = [&](uint32_t piece, uint32_t& source, uint32_t& target) {
        if (piece < 5 * per_vector) {
            const uint32_t vector = piece / per_vector;
            const uint32_t chunk = piece - vector * per_vector;
            source = static_cast<uint32_t>(vector * width + head_base) + chunk * 8;
            target = vector * DP + chunk * 8;
        } else {
            const uint32_t chunk = piece - 5 * per_vector;
            source = static_cast<uint32_t>(5 * width) + chunk * 8;
            target = 5 * DP + chunk * 8;
        }
    };
    uint32_t first_source = 0, first_target = 0, second_source = 0, second_target = 0;
    piece_offsets(warp_lane, first_source, first_target);
    piece_offsets(warp_lane + 32, second_source, second_target);
    auto load_tile = [&](uint32_t tile) {             // helpers only; always one group per call
        const uint32_t first = begin + tile * kPromptTokens;
#pragma unroll
        for (uint32_t i = 0; i < kTokensPerHelper; ++i) {
            const uint32_t t = helper_warp * kTokensPerHelper + i;
            if (tile < tiles && first + t < end) {
                const __nv_bfloat16* source = args.projected + static_cast<size_t>(first + t) * args.pitch;
                __nv_bfloat16* target = raw + (tile % kRawStages * kPromptTokens + t) * layout.raw_row;
                if (warp_lane < pieces) copy_async_16(target + first_target, source + first_source);
                if (warp_lane + 32 < pieces) copy_async_16(target + second_target, source + second_source);
                for (uint32_t piece = warp_lane + 64; kPieces > 2 && piece < pieces; piece += 32) {
                    uint32_t from, to;
                    piece_offsets(piece, from, to);
                    copy_async_16(target + to, source + from);
                }
            }
        }
        copy_async_commit();
    };

    auto prepare_tile = [&](uint32_t tile) {          // helpers only; the tile's copies have arrived for all of them
        const __nv_bfloat16* stage = raw + tile % kRawStages * kPromptTokens * layout.raw_row;
        float* target = vectors + tile % 2 * kPromptTokens * 2 * DP;
        float* unit = scale + tile % 2 * kPromptTokens;
        float squares[kTokensPerHelper];
#pragma unroll
        for (uint32_t i = 0; i < kTokensPerHelper; ++i) {
            const __nv_bfloat16* row = stage + (helper_warp * kTokensPerHelper + i) * layout.raw_row;
            squares[i] = 0.0f;
#pragma unroll
            for (uint32_t part = 0; part < DP / 64; ++part) {
                const float2 both =
                    __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row + DP + part * 64 + warp_lane * 2));
                squares[i] = fmaf(both.x, both.x, fmaf(both.y, both.y, squares[i]));
            }
        }
        for (uint32_t z = warp_lane * 2; z < layout.rank_pad; z += 64) {
#pragma unroll
            for (uint32_t i = 0; i < kTokensPerHelper; ++i) {
                const uint32_t t = helper_warp * kTokensPerHelper + i;
                const float2 both = __bfloat1622float2(
                    *reinterpret_cast<const __nv_bfloat162*>(stage + t * layout.raw_row + 5 * DP + z));
                // columns between rank and the end of its last copy belong to nobody
                const float a = z < args.rank ? fast_tanh(both.x) : 0.0f;
                const float b = z + 1 < args.rank ? fast_tanh(both.y) : 0.0f;
                const __nv_bfloat162 high = __floats2bfloat162_rn(a, b);
                const float2 rounded = __bfloat1622float2(high);
                *reinterpret_cast<__nv_bfloat162*>(tanh_parts + t * layout.z_stride + z) = high;
                *reinterpret_cast<__nv_bfloat162*>(tanh_parts + (kPromptTokens + t) * layout.z_stride + z) =
                    __floats2bfloat162_rn(a - rounded.x, b - rounded.y);
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < kTokensPerHelper; ++i) squares[i] = warp_sum(squares[i]);
        if (warp_lane == 0) {
#pragma unroll
            for (uint32_t i = 0; i < kTokensPerHelper; ++i) {
                unit[helper_warp * kTokensPerHelper + i] = 1.0f / (squares[i] + kUnitEps);
            }
        }
        named_barrier(1, kHelpers);
        // decay logits of 16 tokens x 8 channels at a time: tanh(z) W2^T with tanh(z) as a sum of two bf16 values
#pragma unroll
        for (uint32_t n = 0; n < DP / 8 / kHelperWarps; ++n) {
            const uint32_t channel0 = (n * kHelperWarps + helper_warp) * 8;
            float logits[4] = {};
            const uint32_t z_row = warp_lane % 16, z_part = warp_lane / 16 * 8;
            for (uint32_t step = 0; step < layout.rank_pad; step += 32) {
                uint32_t b0, b1, b2, b3;
                ldmatrix_x4(smem_u32(w2 + (channel0 + warp_lane % 8) * layout.z_stride + step + warp_lane / 8 * 8), b0, b1,
                            b2, b3);
#pragma unroll
                for (uint32_t part = 0; part < 2; ++part) {
                    uint32_t high[4], low[4];
                    const __nv_bfloat16* source = tanh_parts + z_row * layout.z_stride + step + part * 16 + z_part;
                    ldmatrix_x4(smem_u32(source), high[0], high[1], high[2], high[3]);
                    ldmatrix_x4(smem_u32(source + kPromptTokens * layout.z_stride), low[0], low[1], low[2], low[3]);
                    mma_bf16_16816(logits, high[0], high[1], high[2], high[3], part ? b2 : b0, part ? b3 : b1);
                    mma_bf16_16816(logits, low[0], low[1], low[2], low[3], part ? b2 : b0, part ? b3 : b1);
                }
            }
            const uint32_t channel = channel0 + warp_lane % 4 * 2;
            const uint32_t t0 = warp_lane / 4;
            const float2 base = *reinterpret_cast<const float2*>(constants + channel);
            const float2 bias = *reinterpret_cast<const float2*>(constants + DP + channel);
            float2 rate[2];
            float factor[2];
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                rate[half] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(
                    stage + (t0 + half * 8) * layout.raw_row + 4 * DP + channel));
                factor[half] = unit[t0 + half * 8];
            }
            float2 w[2], removal[2];
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                w[half].x = __expf(-kDecayScale * fast_sigmoid(logits[2 * half] + base.x));
                w[half].y = __expf(-kDecayScale * fast_sigmoid(logits[2 * half + 1] + base.y));
                // -(a * u) (u^T S) = -(a / |k|^2) * k * (k^T S): the recurrence multiplies by k anyway
                removal[half].x = -fast_sigmoid(rate[half].x + bias.x) * factor[half];
                removal[half].y = -fast_sigmoid(rate[half].y + bias.y) * factor[half];
            }
            const uint32_t at = interleaved<DP>(channel);
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                float* row = target + (t0 + half * 8) * 2 * DP + at;
                *reinterpret_cast<float2*>(row) = w[half];
                *reinterpret_cast<float2*>(row + DP) = removal[half];
            }
        }
    };

    auto finish_tile = [&](uint32_t tile) {           // helpers only
        const __nv_bfloat16* stage = raw + tile % kRawStages * kPromptTokens * layout.raw_row;
        const float* source = produced + tile % 2 * kPromptTokens * DP;
        const uint32_t first = begin + tile * kPromptTokens;
        float2 value[kTokensPerHelper][DP / 64], gate[kTokensPerHelper][DP / 64];
        float squares[kTokensPerHelper];
#pragma unroll
        for (uint32_t i = 0; i < kTokensPerHelper; ++i) {
            const uint32_t t = helper_warp * kTokensPerHelper + i;
            squares[i] = 0.0f;
#pragma unroll
            for (uint32_t part = 0; part < DP / 64; ++part) {
                const uint32_t channel = part * 64 + warp_lane * 2;
                value[i][part] = *reinterpret_cast<const float2*>(source + t * DP + channel);
                gate[i][part] = __bfloat1622float2(
                    *reinterpret_cast<const __nv_bfloat162*>(stage + t * layout.raw_row + 3 * DP + channel));
                squares[i] = fmaf(value[i][part].x, value[i][part].x,
                                  fmaf(value[i][part].y, value[i][part].y, squares[i]));
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < kTokensPerHelper; ++i) squares[i] = warp_sum(squares[i]);
#pragma unroll
        for (uint32_t i = 0; i < kTokensPerHelper; ++i) {
            const uint32_t t = helper_warp * kTokensPerHelper + i;
            const float factor = rsqrtf(squares[i] / static_cast<float>(dim) + args.eps);
#pragma unroll
            for (uint32_t part = 0; part < DP / 64; ++part) {
                const uint32_t channel = part * 64 + warp_lane * 2;
                const float2 weight = *reinterpret_cast<const float2*>(constants + 2 * DP + channel);
                const uint32_t both =
                    pack_bf16x2(value[i][part].x * factor * weight.x * fast_sigmoid(gate[i][part].x),
                                value[i][part].y * factor * weight.y * fast_sigmoid(gate[i][part].y));
                if (channel < dim && first + t < end) {
                    *reinterpret_cast<uint32_t*>(args.out + static_cast<size_t>(first + t) * args.out_pitch + head_base +
                                                 channel) = both;
                }
            }
        }
    };

    // ---- the state: columns COLUMNS * group .. + COLUMNS - 1, key channels lane * kRows .. + kRows - 1
    const uint32_t lane = threadIdx.x % 8;
    const uint32_t column0 = threadIdx.x / 8 * COLUMNS;
    Pair state[COLUMNS][kRows / 2];
    if (scanner) {
#pragma unroll
        for (uint32_t c = 0; c < COLUMNS; ++c) {
#pragma unroll
            for (uint32_t g = 0; g < kRows / 4; ++g) {
                const uint32_t row = lane * kRows + g * 4;
                float4 value = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (column0 + c < dim && row < dim) {          // dim is a multiple of 8
                    value = *reinterpret_cast<const float4*>(state_base + static_cast<size_t>(column0 + c) * dim + row);
                }
                state[c][2 * g] = pair_of(value.x, value.y);
                state[c][2 * g + 1] = pair_of(value.z, value.w);
            }
        }
    } else {
        load_tile(0);
        load_tile(1);
        copy_async_wait<1>();
        named_barrier(1, kHelpers);
        prepare_tile(0);
    }
    __syncthreads();

    for (uint32_t tile = 0; tile < tiles; ++tile) {
        if (scanner) {
            const uint32_t tokens = min(kPromptTokens, end - begin - tile * kPromptTokens);
            const __nv_bfloat16* stage = raw + tile % kRawStages * kPromptTokens * layout.raw_row;
            const float* prepared = vectors + tile % 2 * kPromptTokens * 2 * DP;
            float* target = produced + tile % 2 * kPromptTokens * DP;
            // software pipeline: a token's vectors are read one token ahead, and the sums over the eight threads of a
            // column group run for o of the previous token beside those for u^T S of this one
            struct Vectors {
                uint4 k[kRows / 8], r[kRows / 8];
                uint32_t v[COLUMNS / 2];
            };
            auto read = [&](uint32_t t) {
                Vectors out;
                const __nv_bfloat16* row = stage + t * layout.raw_row;
#pragma unroll
                for (uint32_t part = 0; part < kRows / 8; ++part) {
                    out.k[part] = *reinterpret_cast<const uint4*>(row + DP + lane * kRows + part * 8);
                    out.r[part] = *reinterpret_cast<const uint4*>(row + lane * kRows + part * 8);
                }
                if constexpr (COLUMNS == 4) {
                    const uint2 both = *reinterpret_cast<const uint2*>(row + 2 * DP + column0);
                    out.v[0] = both.x;
                    out.v[1] = both.y;
                } else {
                    out.v[0] = *reinterpret_cast<const uint32_t*>(row + 2 * DP + column0);
                }
                return out;
            };
            Vectors next = read(0);
            float result[COLUMNS] = {};
            const bool upper1 = lane & 1, upper2 = lane & 2;
            float* slot_of_lane = target + column0 + (COLUMNS == 4 ? (lane & 1) * 2 + (lane >> 1 & 1) : (lane & 1));
            // column sums of o over the eight threads, each pair of threads keeping half of the columns
            auto total_of = [&](const float (&share)[COLUMNS]) {
                if constexpr (COLUMNS == 2) {
                    float total = (upper1 ? share[1] : share[0]) +
                                  __shfl_xor_sync(0xffffffffu, upper1 ? share[0] : share[1], 1);
                    total += __shfl_xor_sync(0xffffffffu, total, 2);
                    return total + __shfl_xor_sync(0xffffffffu, total, 4);
                } else {
                const float keep0 = upper1 ? share[2] : share[0], keep1 = upper1 ? share[3] : share[1];
                const float give0 = upper1 ? share[0] : share[2], give1 = upper1 ? share[1] : share[3];
                const float half0 = keep0 + __shfl_xor_sync(0xffffffffu, give0, 1);
                const float half1 = keep1 + __shfl_xor_sync(0xffffffffu, give1, 1);
                float total = (upper2 ? half1 : half0) + __shfl_xor_sync(0xffffffffu, upper2 ? half0 : half1, 2);
                return total + __shfl_xor_sync(0xffffffffu, total, 4);
                }
            };
            for (uint32_t t = 0; t < tokens; ++t) {
                const Vectors now = next;
                next = read(t + 1 < tokens ? t + 1 : t);
                Pair w[kRows / 2], removal[kRows / 2];
#pragma unroll
                for (uint32_t g = 0; g < kRows / 4; ++g) {
                    const float* token = prepared + t * 2 * DP + g * 32 + lane * 4;
                    const ulonglong2 w_pair = *reinterpret_cast<const ulonglong2*>(token);
                    const ulonglong2 removal_pair = *reinterpret_cast<const ulonglong2*>(token + DP);
                    w[2 * g] = w_pair.x;
                    w[2 * g + 1] = w_pair.y;
                    removal[2 * g] = removal_pair.x;
                    removal[2 * g + 1] = removal_pair.y;
                }
                Pair k[kRows / 2], r[kRows / 2];
#pragma unroll
                for (uint32_t part = 0; part < kRows / 8; ++part) {
                    const uint32_t k_words[4] = {now.k[part].x, now.k[part].y, now.k[part].z, now.k[part].w};
                    const uint32_t r_words[4] = {now.r[part].x, now.r[part].y, now.r[part].z, now.r[part].w};
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {       // bf16 -> f32 is a shift
                        k[part * 4 + i] = pair_of(__uint_as_float(k_words[i] << 16),
                                                  __uint_as_float(k_words[i] & 0xffff0000u));
                        r[part * 4 + i] = pair_of(__uint_as_float(r_words[i] << 16),
                                                  __uint_as_float(r_words[i] & 0xffff0000u));
                    }
                }
                float v[COLUMNS], dot[COLUMNS];
#pragma unroll
                for (uint32_t c = 0; c < COLUMNS; c += 2) {
                    v[c] = __uint_as_float(now.v[c / 2] << 16);
                    v[c + 1] = __uint_as_float(now.v[c / 2] & 0xffff0000u);
                }
#pragma unroll
                for (uint32_t c = 0; c < COLUMNS; ++c) {
                    Pair even = mul_pair(k[0], state[c][0]);
                    Pair odd = mul_pair(k[1], state[c][1]);
#pragma unroll
                    for (uint32_t i = 2; i < kRows / 2; i += 2) {
                        even = fma_pair(k[i], state[c][i], even);
                        odd = fma_pair(k[i + 1], state[c][i + 1], odd);
                    }
                    dot[c] = pair_sum(add_pair(even, odd));
                }
#pragma unroll
                for (uint32_t delta = 1; delta < 8; delta <<= 1) {
#pragma unroll
                    for (uint32_t c = 0; c < COLUMNS; ++c) dot[c] += __shfl_xor_sync(0xffffffffu, dot[c], delta);
                }
                const float before = total_of(result);
                Pair sums[COLUMNS];
                // w S does not depend on the sums above
#pragma unroll
                for (uint32_t c = 0; c < COLUMNS; ++c) {
#pragma unroll
                    for (uint32_t i = 0; i < kRows / 2; ++i) state[c][i] = mul_pair(w[i], state[c][i]);
                }
#pragma unroll
                for (uint32_t c = 0; c < COLUMNS; ++c) {
                    const Pair recalled = pair_of(dot[c], dot[c]);
                    const Pair values = pair_of(v[c], v[c]);
                    Pair even = 0, odd = 0;
#pragma unroll
                    for (uint32_t i = 0; i < kRows / 2; i += 2) {      // w S + k (v - (a / |k|^2) (k^T S))
                        state[c][i] = fma_pair(k[i], fma_pair(removal[i], recalled, values), state[c][i]);
                        state[c][i + 1] = fma_pair(k[i + 1], fma_pair(removal[i + 1], recalled, values), state[c][i + 1]);
                        even = fma_pair(r[i], state[c][i], even);
                        odd = fma_pair(r[i + 1], state[c][i + 1], odd);
                    }
                    sums[c] = add_pair(even, odd);
                }
#pragma unroll
                for (uint32_t c = 0; c < COLUMNS; ++c) result[c] = pair_sum(sums[c]);
                if (lane < COLUMNS && t > 0) slot_of_lane[(t - 1) * DP] = before;
            }
            const float last = total_of(result);
            if (lane < COLUMNS) slot_of_lane[(tokens - 1) * DP] = last;
        } else {
            load_tile(tile + 2);
            if (tile > 0) finish_tile(tile - 1);
            copy_async_wait<1>();                     // tile + 1 has arrived for this thread ...
            named_barrier(1, kHelpers);               // ... and for all helpers
            if (tile + 1 < tiles) prepare_tile(tile + 1);
        }
        __syncthreads();
    }
    if (scanner) {
#pragma unroll
        for (uint32_t c = 0; c < COLUMNS; ++c) {
#pragma unroll
            for (uint32_t g = 0; g < kRows / 4; ++g) {
                const uint32_t row = lane * kRows + g * 4;
                if (column0 + c < dim && row < dim) {
                    *reinterpret_cast<float4*>(state_base + static_cast<size_t>(column0 + c) * dim + row) =
                        make_float4(low_of(state[c][2 * g]), high_of(state[c][2 * g]), low_of(state[c][2 * g + 1]),
                                    high_of(state[c][2 * g + 1]));
                }
            }
        }
    } else {
        finish_tile(tiles - 1);
    }
}


template <typename T, uint32_t DP>
cudaError_t launch_decode(cudaStream_t stream, const DeltaArgs<T>& args) {
    const size_t shared = (5 * DP + 2 * (DP * 4 / 32) + args.rank) * sizeof(float);
    if (shared > 48 * 1024) {
        return cudaErrorInvalidValue;
    }
    return launch_kernel(delta_decode_kernel<T, DP>,
                         static_cast<unsigned int>(args.segments.num_segments * args.heads), DP * 4, shared, stream, 1,
                         args);
}

template <uint32_t DP, uint32_t COLUMNS, uint32_t HELPERS>
cudaError_t launch_prompt(cudaStream_t stream, const DeltaArgs<__nv_bfloat16>& args) {
    const size_t shared = PromptLayout<DP>(args.rank).total;
    const auto kernel = delta_prompt_kernel<DP, COLUMNS, HELPERS>;
    const cudaError_t status = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    static_cast<int>(shared));
    if (status != cudaSuccess) return status;
    return launch_kernel(kernel, static_cast<unsigned int>(args.segments.num_segments * args.heads),
                         DP / COLUMNS * 8 + HELPERS, shared, stream, 1, args);
}

// Whether bf16 prompts of these sizes have kernels of their own.  Asked before a launch and where scratch is sized, so that
// whatever they do not take finds room for all its heads.
bool prompt_kernels_take(uint32_t dim, uint32_t rank, size_t pitch, size_t out_pitch, const void* decay_up) {
    const size_t shared = dim <= 64 ? PromptLayout<64>(rank).total : PromptLayout<128>(rank).total;
    return dim % 8 == 0 && dim <= 128 && rank <= kPromptMaxRank && pitch % 8 == 0 && out_pitch % 2 == 0 &&
           aligned_to(decay_up, 16) && shared <= 227 * 1024;
}

bool prompt_kernels_take(const DeltaArgs<__nv_bfloat16>& args) {
    return prompt_kernels_take(args.dim, args.rank, args.pitch, args.out_pitch, args.decay_up) &&
           aligned_to(args.projected, 16) && aligned_to(args.out, 4);
}

// Where prompts are split along the sequence (delta_split.cu) instead of carried by one CTA per segment and head: it does about
// twice the arithmetic and takes three launches, so it pays while the carrying CTAs leave most SMs idle and a prompt is
// long.  The lengths are on the device, so the line is drawn for segments of equal length, where the longest one does not
// help.  Inside steps of four layers, segments x heads (of 64 dimensions): what a layer gains in us at tokens a segment (two
// runs, one to eight segments)
//     16: 320 6, 400 16, 500 33, 600 40, 1000 91          32: 320 -1, 400 5 to 7, 500 23, 600 4 to 8, 700 14 to 19, 1000 43 to 49
//     48: 320 -4, 400 -24, 600 -5 to -9, 720 1 to 5, 800 -10 to -16, 1000 1 to 2, 1500 27
//     64 (whole models): 1000 -70, 2000 -114
// The steps in between are waves of CTAs.  (The lines were drawn between earlier forms of both.  Today's form beside them gains at
// 16 and 32 heads wherever it is taken; at 48 it loses around 800 tokens.)
constexpr size_t kSplitMostHeads = 48;             // of all segments
constexpr size_t split_shortest(size_t heads) { return heads <= 16 ? 320 : (heads <= 32 ? 400 : 720); }

bool split_pays(const DeltaRuleLaunch& launch) {
    const size_t segments = launch.segments.num_segments, heads = segments * launch.heads;
    const size_t tokens = launch.segments.num_tokens - launch.decode_tokens;
    return heads <= kSplitMostHeads && tokens >= split_shortest(heads) * segments;
}

// The kernels' pairwise accesses, and scratch for one head at least (beside what the chunk kernel needs).
bool split_takes(const DeltaArgs<__nv_bfloat16>& args, const DeltaRuleLaunch& launch) {
    const int64_t forced = option(kOptDeltaPrompt);
    return (forced == 4 || (forced == 0 && split_pays(launch))) && aligned_to(args.decay_base, 4) &&
           aligned_to(args.removal_bias, 4) && aligned_to(args.norm, 4) && launch.chunks != nullptr &&
           delta_split_bytes(1, tile_bound(launch.segments, 64)) <= launch.chunk_bytes;
}

template <typename T, uint32_t DP, uint32_t LANES, uint32_t COLUMNS>
cudaError_t launch_sized(cudaStream_t stream, DeltaArgs<T> args) {
    args.splits = (args.dim + COLUMNS - 1) / COLUMNS;
    const size_t shared = delta_shared_bytes<DP>(args.rank);
    void (*kernel)(const DeltaArgs<T>) = delta_rule_kernel<T, DP, LANES, COLUMNS>;
    if (shared > 227 * 1024) {
        return cudaErrorInvalidValue;
    }
    if (shared > 48 * 1024) {
        const cudaError_t status = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        static_cast<int>(shared));
        if (status != cudaSuccess) return status;
    }
    const size_t blocks = args.segments.num_segments * args.heads * args.splits;
    const cudaError_t status =
        launch_kernel(kernel, static_cast<unsigned int>(blocks), LANES * COLUMNS, shared, stream, 1, args);
    if (status != cudaSuccess || args.raw == nullptr) {
        return status;
    }
    return launch_kernel(delta_output_kernel<T>,
                         static_cast<unsigned int>((args.segments.num_tokens * args.heads + 3) / 4), 128, 0, stream, 1,
                         args);
}

template <typename T>
cudaError_t launch_typed(cudaStream_t stream, const DeltaRuleLaunch& launch) {
    DeltaArgs<T> args;
    args.segments = launch.segments;
    args.heads = launch.heads;
    args.dim = launch.dim;
    args.rank = launch.rank;
    args.projected = static_cast<const T*>(launch.projected);
    args.pitch = launch.pitch;
    args.decay_up = static_cast<const __nv_bfloat16*>(launch.decay_up);
    args.decay_base = static_cast<const __nv_bfloat16*>(launch.decay_base);
    args.removal_bias = static_cast<const __nv_bfloat16*>(launch.removal_bias);
    args.norm = static_cast<const __nv_bfloat16*>(launch.norm);
    args.record = launch.record;
    args.raw = delta_rule_needs_scratch(launch.dim) ? launch.raw : nullptr;
    args.out = static_cast<T*>(launch.out);
    args.out_pitch = launch.out_pitch;
    args.eps = launch.eps;
    args.splits = 1;
    if (launch.segments.offsets == nullptr && launch.dim <= 128 && launch.rank <= 4096) {
        if (launch.dim <= 32) return launch_decode<T, 32>(stream, args);
        if (launch.dim <= 64) return launch_decode<T, 64>(stream, args);
        return launch_decode<T, 128>(stream, args);
    }
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        if (launch.segments.offsets != nullptr && option(kOptDeltaPrompt) != 2 && prompt_kernels_take(args)) {
            if (delta_chunk_takes(launch.dim, launch.rank) && option(kOptDeltaPrompt) != 1) {
                // the kernels for larger ranks keep more bits than the split ones
                if (split_takes(args, launch)) return launch_delta_split(stream, args, launch.chunks, launch.chunk_bytes);
                if (option(kOptDeltaPrompt) == 4) return cudaErrorInvalidValue;       // no scratch for what was asked for
                return launch_delta_chunk(stream, args);
            }
            return launch.dim <= 64 ? launch_prompt<64, 4, 128>(stream, args) : launch_prompt<128, 4, 128>(stream, args);
        }
    }
    if (launch.segments.offsets != nullptr) return launch_delta_scan(stream, args, launch.vectors, launch.vector_bytes);
    if (launch.dim <= 32) return launch_sized<T, 32, 4, 32>(stream, args);
    if (launch.dim <= 64) return launch_sized<T, 64, 4, 64>(stream, args);
    if (launch.dim <= 128) return launch_sized<T, 128, 4, 128>(stream, args);
    if (launch.dim <= kDeltaMaxDim && launch.raw != nullptr) return launch_sized<T, 256, 8, 64>(stream, args);
    return cudaErrorInvalidValue;
}

}  // namespace

bool delta_rule_needs_scratch(uint32_t dim) { return dim > 128; }

size_t delta_rule_vector_bytes(Activation type, uint32_t heads, uint32_t dim, uint32_t rank, size_t pitch, size_t out_pitch,
                               const void* decay_up, size_t tokens) {
    const bool others = type == Activation::kBf16 && prompt_kernels_take(dim, rank, pitch, out_pitch, decay_up);
    return delta_scan_bytes(others ? 1 : heads, dim, tokens);
}

size_t delta_rule_chunk_bytes(Activation type, uint32_t heads, uint32_t dim, size_t tokens, size_t segments) {
    const size_t most = std::min(std::min(segments, tokens / split_shortest(heads)), kSplitMostHeads / heads);
    if (type != Activation::kBf16 || dim > kDeltaChunkDim || dim % 8 != 0 || most == 0) return 0;
    return std::min(delta_split_bytes(heads, tokens / 64 + most), kDeltaChunkBytes);
}

cudaError_t launch_delta_rule(cudaStream_t stream, const DeltaRuleLaunch& launch) {
    const auto run = [&](const DeltaRuleLaunch& part) {
        return part.type == Activation::kF32 ? launch_typed<float>(stream, part)
                                             : launch_typed<__nv_bfloat16>(stream, part);
    };
    if (launch.segments.offsets == nullptr || launch.decode_tokens == 0) {
        return run(launch);
    }
    DeltaRuleLaunch decodes = launch;
    decodes.decode_tokens = 0;
    decodes.segments.offsets = nullptr;
    decodes.segments.num_segments = launch.decode_tokens;
    decodes.segments.num_tokens = launch.decode_tokens;
    const cudaError_t status = run(decodes);
    if (status != cudaSuccess || launch.decode_tokens == launch.segments.num_segments) {
        return status;
    }
    DeltaRuleLaunch prompts = launch;      // segment offsets are absolute token indices
    prompts.segments.offsets += launch.decode_tokens;
    prompts.segments.slots += launch.decode_tokens;
    prompts.segments.num_segments -= launch.decode_tokens;
    return run(prompts);
}

}  // namespace lfm25

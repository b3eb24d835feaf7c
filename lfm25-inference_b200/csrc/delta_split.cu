// The generalised delta rule over bf16 prompts, split along the sequence.
//
// Over a chunk of 64 tokens, with P_t the product of the decays of its tokens up to t, S_t = diag(P_t) Q_t and
//     U_t = u_t P_(t-1),   R_t = r_t P_t,   K_t = k_t / P_t,   B_t = -(a_t u_t) / P_t          (per key channel)
// the update is Q_t = Q_(t-1) + B_t (U_t^T Q_(t-1)) + K_t v_t^T: the chunked form of the delta rule (Yang et al. 2024, after
// Bischof and Van Loan's WY form of products of rank-one updates), here with a decay per key channel.  With
//     (I - tril(U B^T, -1)) [W | Z] = [U | tril(U K^T, -1) V]
// the Q_(t-1)^T U_t of the chunk are W S_0 + Z, so the state behind the chunk and the outputs are linear in the state S_0
// before it:
//     S = diag(P) S_0 + A S_0 + D,        A = diag(P) B^T W,        D = diag(P) (B^T Z + K^T V)
//     O = R' S_0 + O',        R' = R + tril(R B^T) W,         O' = tril(R B^T) Z + tril(R K^T) V
// Everything but S_0 belongs to one chunk alone.  Three kernels:
//     form     P, A, D, R', O' of every chunk of every head                     all chunks side by side
//     carry    S through each segment's chunks, S_0 in the place of D           one product of 64 x 64 x 16 per chunk
//     finish   O = R' S_0 + O', norm, gate                                      all chunks side by side
// so only `carry` is serial, in steps of 64 tokens of a single small product.  4096 tokens of 32 heads: 395 us for the three
// (one CTA per head, tile after tile of 16 tokens: 663 us on 32 SMs).
//
// Decays are multiplied up by a scan, never summed as logarithms: P_t and the 1 / P_s that meets it come from the same
// factors, and both carry a handful of roundings.  A decay is at least exp(-exp(-1/2)), so 1 / P_t stays below 1e17 and a
// product P_t / P_s keeps its relative accuracy.
//
// All matrix products are TF32 with both operands in two parts (bf16 values of v need no second one) and f32 sums.  What
// reaches the state is held to no larger an error than the carrying kernel has: parts rounded to nearest, short sums that are
// added up outside the tensor cores, decays rounded without a direction (decay_of), the state's own part diag(P) S_0 as f32
// multiply-adds.  State against float64 (2-norm; 300 to 4096 tokens, heads of 64, decay logits around 0, spread around -2,
// around -6): 1.5e-7, 2.2e-7, 2.9e-7; the carrying kernel 4.1e-7, 7.4e-7, 1.7e-6.  With plain parts and sums inside the tensor
// cores it was 9e-7, 1.6e-6, 2.0e-6 in 338 us instead of the 418 of that time.  The outputs' own product ends in their bf16 rounding and needs
// none of this.  Not for f32 activations: the decays' products, their reciprocals and the parts each round once more than the
// token-by-token recurrence does (250 tokens of 16 heads: 1.44e-7 at best, 0.76e-7 token by token).
#include <algorithm>
#include <cstddef>

#include "delta_rule.h"
#include "launch.h"

namespace lfm25 {

namespace {

constexpr uint32_t kDim = 64;                      // padded head size
constexpr uint32_t kTokens = 64;
constexpr uint32_t kPitch = 72;                    // rows of U, R, K, B, V in shared memory
constexpr uint32_t kLowerPitch = 68;
constexpr uint32_t kInversePitch = 20;
constexpr uint32_t kMatrix = kDim * kTokens;       // elements of A, D, R' and O'; P behind them
constexpr uint32_t kChunkFloats = 4 * kMatrix + kDim;
constexpr uint32_t kD = kMatrix, kR = 2 * kMatrix, kO = 3 * kMatrix, kP = 4 * kMatrix;     // behind A
constexpr uint32_t kFormThreads = 256;
constexpr uint32_t kCarryThreads = 128;
constexpr uint32_t kCarryColumns = 16;
constexpr uint32_t kCarryPitch = 20;
constexpr uint32_t kCarryStages = 5;
constexpr uint32_t kFinishThreads = 128;

// Fragments in which k index c of a 16 x 8 operand stands for column (row of B) 2c, and c + 4 for 2c + 1: the accumulator of
// one product is then an operand of the next as it is, and operands along a row are read two at a time.
__device__ __forceinline__ FragmentA<true> load_a_pairs(const float* source, uint32_t stride, uint32_t lane) {
    FragmentA<true> out;
    const float* at = source + (lane >> 2) * stride + (lane & 3) * 2;
    const float2 upper = *reinterpret_cast<const float2*>(at), lower = *reinterpret_cast<const float2*>(at + 8 * stride);
    out.set(0, upper.x);
    out.set(1, lower.x);
    out.set(2, upper.y);
    out.set(3, lower.y);
    return out;
}
__device__ __forceinline__ FragmentA<true> a_from_c(const float (&c)[4]) {
    FragmentA<true> out;
    out.set(0, c[0]);
    out.set(1, c[2]);
    out.set(2, c[1]);
    out.set(3, c[3]);
    return out;
}
__device__ __forceinline__ FragmentB<true> load_b_transposed_pairs(const float* source, uint32_t stride, uint32_t lane) {
    FragmentB<true> out;
    const float2 both = *reinterpret_cast<const float2*>(source + (lane >> 2) * stride + (lane & 3) * 2);
    out.set(0, both.x);
    out.set(1, both.y);
    return out;
}
__device__ __forceinline__ FragmentB<true> load_b_pairs(const float* source, uint32_t stride, uint32_t lane) {
    FragmentB<true> out;
    const float* at = source + (lane & 3) * 2 * stride + (lane >> 2);
    out.set(0, at[0]);
    out.set(1, at[stride]);
    return out;
}
__device__ __forceinline__ void load_c(const float* source, uint32_t stride, uint32_t lane, float (&c)[4]) {
    const float* at = source + (lane >> 2) * stride + (lane & 3) * 2;
    const float2 upper = *reinterpret_cast<const float2*>(at), lower = *reinterpret_cast<const float2*>(at + 8 * stride);
    c[0] = upper.x;
    c[1] = upper.y;
    c[2] = lower.x;
    c[3] = lower.y;
}

// d[n] += a * rows for eight column blocks, `rows` bf16 (exact in TF32) or f32; PAIRS: in the order of load_b_pairs
template <bool PAIRS>
__device__ __forceinline__ void multiply_rows(float (&d)[8][4], const FragmentA<true>& a, const __nv_bfloat16* rows,
                                              uint32_t lane) {
    const uint32_t first = (PAIRS ? (lane & 3) * 2 : lane & 3) * kPitch + (lane >> 2);
    const uint32_t second = first + (PAIRS ? 1 : 4) * kPitch;
#pragma unroll
    for (uint32_t n = 0; n < 8; n += 2) {
        const float b0[2] = {__bfloat162float(rows[first + n * 8]), __bfloat162float(rows[second + n * 8])};
        const float b1[2] = {__bfloat162float(rows[first + n * 8 + 8]), __bfloat162float(rows[second + n * 8 + 8])};
        float sums[2][4] = {};
        mma_tf32(sums[0], a.low, b0);
        mma_tf32(sums[1], a.low, b1);
        mma_tf32(sums[0], a.high, b0);
        mma_tf32(sums[1], a.high, b1);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            d[n][i] += sums[0][i];
            d[n + 1][i] += sums[1][i];
        }
    }
}
template <bool PAIRS>
__device__ __forceinline__ void multiply_rows(float (&d)[8][4], const FragmentA<true>& a, const float* rows, uint32_t lane) {
#pragma unroll
    for (uint32_t n = 0; n < 8; n += 2) {
        FragmentB<true> b[2];
#pragma unroll
        for (uint32_t q = 0; q < 2; ++q) {
            b[q] = PAIRS ? load_b_pairs(rows + (n + q) * 8, kPitch, lane)
                         : load_b<true>(rows + (n + q) * 8, kPitch, lane);
        }
        mma_split<true, 2>(d + n, a, b);
    }
}

__device__ __forceinline__ float2 load_pair(const __nv_bfloat16* source) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(source));
}

// 1 - (1 - exp(x)): close to 1, where a rounding to the same side in every token would add up over a long memory, the sum is
// rounded to nearest.  x lies between -exp(-1/2) and 0, where ten terms of the exponential's power series leave 2e-10: errors of
// the state as with expm1f (4096 tokens; decay logits around 0, -2, -6, -10: 1.39e-7, 1.83e-7, 2.97e-7, 4.70e-7 with either), 9 us
// of 404 for the three kernels.
__device__ __forceinline__ float decay_of(float logit) {
    const float x = -kDecayScale * sigmoidf(logit);
    float sum = 1.0f / 3628800.0f;
    sum = fmaf(sum, x, 1.0f / 362880.0f);
    sum = fmaf(sum, x, 1.0f / 40320.0f);
    sum = fmaf(sum, x, 1.0f / 5040.0f);
    sum = fmaf(sum, x, 1.0f / 720.0f);
    sum = fmaf(sum, x, 1.0f / 120.0f);
    sum = fmaf(sum, x, 1.0f / 24.0f);
    sum = fmaf(sum, x, 1.0f / 6.0f);
    sum = fmaf(sum, x, 0.5f);
    return 1.0f + fmaf(sum * x, x, x);
}

struct FormShared {
    float u[kTokens * kPitch];                     // U, then W
    float r[kTokens * kPitch];
    float k[kTokens * kPitch];                     // K, then Z
    float b[kTokens * kPitch];
    float lower[kTokens * kLowerPitch];            // tril(U B^T, -1), blocks on and below the diagonal
    float inverse[4][16 * kInversePitch];          // of I - lower on the diagonal blocks
    float block_decay[4][kDim];                    // products over 16 tokens
    float squares[2][kTokens];                     // |k|^2 over half of the channels each
    __nv_bfloat16 v[kTokens * kPitch];
};

// About 6500 m16n8k8 products per chunk, eight cycles each per SM quarter, beside cutting their operands and adding up their
// sums; the rest is the latency of the five stages between barriers, which two CTAs per SM hide in part.  Longer loops are
// not unrolled further: the code then outgrows the instruction cache.  r, k and the removal's logit come by asynchronous copies
// during the decay product; as 24 loads of four bytes a thread ahead of it they took 14 us more of 418 for the three kernels
// (4096 tokens of 32 heads).
__global__ void __launch_bounds__(kFormThreads, 2)
delta_form_kernel(const DeltaArgs<__nv_bfloat16> args, uint32_t head0, uint32_t head_count, float* chunks) {
    constexpr uint32_t kParts = 3;                 // bf16 parts of tanh(z)
    extern __shared__ __align__(16) unsigned char form_shared[];
    FormShared& shared = *reinterpret_cast<FormShared*>(form_shared);
    pdl_launch_dependents();
    pdl_wait();
    const SegmentTile tile = locate_tile(args.segments, kTokens, blockIdx.x / head_count);
    if (tile.count == 0) {
        return;
    }
    const uint32_t head = head0 + blockIdx.x % head_count;
    const uint32_t dim = args.dim;
    const size_t width = static_cast<size_t>(args.heads) * dim;
    const size_t head_base = static_cast<size_t>(head) * dim;
    const __nv_bfloat16* projected = args.projected + static_cast<size_t>(tile.first) * args.pitch;
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    // ---- V, and r, k and the removal's logit as they are, where K and B will lie: on their way during the decay product
    constexpr uint32_t kPiece = 8;                 // elements of 16 bytes
    constexpr uint32_t kRaw = kTokens * kPitch;
    __nv_bfloat16* raw = reinterpret_cast<__nv_bfloat16*>(shared.k);
    static_assert(3 * kRaw * 2 <= 2 * kTokens * kPitch * 4 && offsetof(FormShared, b) == offsetof(FormShared, k) + kRaw * 4,
                  "inside K and B");
    for (uint32_t item = threadIdx.x; item < kTokens * kDim / kPiece; item += kFormThreads) {
        const uint32_t token = item / (kDim / kPiece), column = item % (kDim / kPiece) * kPiece;
        const bool inside = token < tile.count && column < dim;
        const __nv_bfloat16* source = inside ? projected + token * args.pitch + head_base + column : projected;
        const uint32_t at = token * kPitch + column;
        copy_async_16(raw + at, source, inside);
        copy_async_16(raw + kRaw + at, source + (inside ? width : 0), inside);
        copy_async_16(raw + 2 * kRaw + at, source + (inside ? 4 * width : 0), inside);
        copy_async_16(shared.v + at, source + (inside ? 2 * width : 0), inside);
    }
    copy_async_commit();

    // 16 tokens x 32 channels per warp, in the layout of the decay product below
    const uint32_t block = warp % 4, half = warp / 4;
    const uint32_t row0 = block * 16 + (lane >> 2), pair = (lane & 3) * 2;
    // ---- decay logits W2 tanh(z), 64 columns of z at a time; their operands lie where U and R will
    float logits[4][4] = {};
    {
        __nv_bfloat16* w2 = reinterpret_cast<__nv_bfloat16*>(form_shared);
        __nv_bfloat16* parts = w2 + kDim * kPitch;
        static_assert((1 + kParts) * kDim * kPitch * 2 <= 2 * kTokens * kPitch * 4, "inside U and R");
        const bool vector_rank = args.rank % 8 == 0;
        for (uint32_t z0 = 0; z0 < args.rank; z0 += 64) {
            if (z0 > 0) __syncthreads();
#pragma unroll
            for (uint32_t step = 0; step < 2; ++step) {
                const uint32_t item = threadIdx.x + step * kFormThreads;
                const uint32_t row = item / 8, z = item % 8 * 8;
                uint4 weight = make_uint4(0, 0, 0, 0);
                if (row < dim && z0 + z < args.rank) {
                    const __nv_bfloat16* source = args.decay_up + (head_base + row) * args.rank + z0 + z;
                    if (vector_rank) {
                        weight = *reinterpret_cast<const uint4*>(source);
                    } else {
                        auto* elements = reinterpret_cast<__nv_bfloat16*>(&weight);
                        for (uint32_t i = 0; i < 8 && z0 + z + i < args.rank; ++i) elements[i] = source[i];
                    }
                }
                *reinterpret_cast<uint4*>(w2 + row * kPitch + z) = weight;
                float value[8] = {};
                if (row < tile.count && z0 + z < args.rank) {
                    load_values<8>(projected + row * args.pitch + 5 * width + z0 + z, value);
                }
                // columns between rank and the end of its last 16 bytes belong to nobody
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) value[i] = z0 + z + i < args.rank ? fast_tanh(value[i]) : 0.0f;
#pragma unroll
                for (uint32_t part = 0; part < kParts; ++part) {
                    uint32_t packed[4];
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        packed[i] = pack_bf16x2(value[2 * i], value[2 * i + 1]);
                        const float2 rounded = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&packed[i]));
                        value[2 * i] -= rounded.x;
                        value[2 * i + 1] -= rounded.y;
                    }
                    *reinterpret_cast<uint4*>(parts + part * kTokens * kPitch + row * kPitch + z) =
                        make_uint4(packed[0], packed[1], packed[2], packed[3]);
                }
            }
            __syncthreads();
#pragma unroll
            for (uint32_t z = 0; z < 64; z += 16) {
                uint32_t b[2][4];
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    const uint32_t channel = half * 32 + q * 16 + lane / 16 * 8 + lane % 8;
                    ldmatrix_x4(smem_u32(w2 + channel * kPitch + z + lane / 8 % 2 * 8), b[q][0], b[q][1], b[q][2], b[q][3]);
                }
#pragma unroll
                for (uint32_t part = 0; part < kParts; ++part) {
                    uint32_t a[4];
                    ldmatrix_x4(smem_u32(parts + part * kTokens * kPitch + (block * 16 + lane % 16) * kPitch + z + lane / 16 * 8),
                                a[0], a[1], a[2], a[3]);
#pragma unroll
                    for (uint32_t n = 0; n < 4; ++n) {
                        mma_bf16_16816(logits[n], a[0], a[1], a[2], a[3], b[n / 2][n % 2 * 2], b[n / 2][n % 2 * 2 + 1]);
                    }
                }
            }
        }
    }
    copy_async_wait<0>();
    __syncthreads();
    float2 r[4][2], k[4][2], removal[4][2];
#pragma unroll
    for (uint32_t n = 0; n < 4; ++n) {
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            const __nv_bfloat16* source = raw + (row0 + i * 8) * kPitch + half * 32 + n * 8 + pair;
            r[n][i] = load_pair(source);
            k[n][i] = load_pair(source + kRaw);
            removal[n][i] = load_pair(source + 2 * kRaw);
        }
    }
    // ---- products of the decays up to each token: of its block of 16 here, of the blocks before it below
    float upto[4][4], before[4][4];
    {
        float squares[2] = {};
#pragma unroll
        for (uint32_t n = 0; n < 4; ++n) {
            const uint32_t channel = half * 32 + n * 8 + pair;
            float2 base = make_float2(0.0f, 0.0f);
            if (channel < dim) base = load_pair(args.decay_base + head_base + channel);
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                upto[n][i] = row0 + (i >> 1) * 8 < tile.count ? decay_of(logits[n][i] + (i & 1 ? base.y : base.x)) : 1.0f;
            }
#pragma unroll
            for (uint32_t delta = 4; delta < 32; delta <<= 1) {
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const float other = __shfl_up_sync(0xffffffffu, upto[n][i], delta);
                    if (lane >= delta) upto[n][i] *= other;
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const float first_half = __shfl_sync(0xffffffffu, upto[n][i], 28 + (lane & 3));
                upto[n][2 + i] *= first_half;
                const float upper = __shfl_up_sync(0xffffffffu, upto[n][i], 4);
                const float lower = __shfl_up_sync(0xffffffffu, upto[n][2 + i], 4);
                before[n][i] = lane < 4 ? 1.0f : upper;
                before[n][2 + i] = lane < 4 ? first_half : lower;
            }
            if (lane >= 28) {
                *reinterpret_cast<float2*>(&shared.block_decay[block][channel]) = make_float2(upto[n][2], upto[n][3]);
            }
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) squares[i] = fmaf(k[n][i].x, k[n][i].x, fmaf(k[n][i].y, k[n][i].y, squares[i]));
        }
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            squares[i] += __shfl_xor_sync(0xffffffffu, squares[i], 1);
            squares[i] += __shfl_xor_sync(0xffffffffu, squares[i], 2);
            if ((lane & 3) == 0) shared.squares[half][row0 + i * 8] = squares[i];
        }
    }
    __syncthreads();

    // ---- U, R, K, B
#pragma unroll
    for (uint32_t n = 0; n < 4; ++n) {
        const uint32_t channel = half * 32 + n * 8 + pair;
        float2 earlier = make_float2(1.0f, 1.0f), bias = make_float2(0.0f, 0.0f);
        for (uint32_t other = 0; other < block; ++other) {
            const float2 decay = *reinterpret_cast<const float2*>(&shared.block_decay[other][channel]);
            earlier.x *= decay.x;
            earlier.y *= decay.y;
        }
        if (channel < dim) bias = load_pair(args.removal_bias + head_base + channel);
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            const uint32_t token = row0 + i * 8;
            const float square = shared.squares[0][token] + shared.squares[1][token] + kUnitEps;
            const float unit = rsqrtf(square);
            const float px = upto[n][2 * i] * earlier.x, py = upto[n][2 * i + 1] * earlier.y;
            const float ix = __fdividef(1.0f, px), iy = __fdividef(1.0f, py);
            const float ux = k[n][i].x * unit, uy = k[n][i].y * unit;
            const uint32_t at = token * kPitch + channel;
            *reinterpret_cast<float2*>(shared.u + at) =
                make_float2(ux * (before[n][2 * i] * earlier.x), uy * (before[n][2 * i + 1] * earlier.y));
            *reinterpret_cast<float2*>(shared.r + at) = make_float2(r[n][i].x * px, r[n][i].y * py);
            *reinterpret_cast<float2*>(shared.k + at) = make_float2(k[n][i].x * ix, k[n][i].y * iy);
            *reinterpret_cast<float2*>(shared.b + at) = make_float2(-fast_sigmoid(removal[n][i].x + bias.x) * ux * ix,
                                                                    -fast_sigmoid(removal[n][i].y + bias.y) * uy * iy);
        }
    }
    __syncthreads();

    float* chunk = chunks + static_cast<size_t>(blockIdx.x) * kChunkFloats;
    // Warps 0..3 take 16 tokens of U each, the others 16 tokens of R, the long rows of one beside the short ones of the other.
    const bool forward = warp < 4;
    const uint32_t mine = forward ? warp : 7 - warp;
    const float* rows = (forward ? shared.u : shared.r) + mine * 16 * kPitch;
    float with_values[8][4] = {};                  // tril(U K^T, -1) V or tril(R K^T) V
    float against_b[4][2][4];                      // tril(R B^T), 16 x 16 each
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        if (j > mine) continue;
        float with_b[2][4] = {}, with_k[2][4] = {};
#pragma unroll 2
        for (uint32_t c = 0; c < kDim; c += 8) {
            const FragmentA<true> a = load_a_pairs(rows + c, kPitch, lane);
            const uint32_t at = j * 16 * kPitch + c;
            mma_split(with_b, a, load_b_transposed_pairs(shared.b + at, kPitch, lane),
                      load_b_transposed_pairs(shared.b + at + 8 * kPitch, kPitch, lane));
            mma_split(with_k, a, load_b_transposed_pairs(shared.k + at, kPitch, lane),
                      load_b_transposed_pairs(shared.k + at + 8 * kPitch, kPitch, lane));
        }
#pragma unroll
        for (uint32_t n = 0; n < 2; ++n) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t row = (lane >> 2) + (i >> 1) * 8, column = n * 8 + pair + (i & 1);
                const bool kept = j < mine || (forward ? column < row : column <= row);   // U meets the state before s = t
                if (!kept) with_b[n][i] = with_k[n][i] = 0.0f;
                against_b[j][n][i] = with_b[n][i];
            }
            if (forward) store_c(shared.lower + mine * 16 * kLowerPitch + j * 16 + n * 8, kLowerPitch, lane, with_b[n]);
        }
#pragma unroll
        for (uint32_t n = 0; n < 2; ++n) {
            multiply_rows<true>(with_values, a_from_c(with_k[n]), shared.v + (j * 16 + n * 8) * kPitch, lane);
        }
    }
    float behind[8][4] = {};                       // K^T V, then D: 16 key channels per warp of the first four
    if (forward) {
        // column `lane` of the inverse of I - L: x_t = e_t + sum over s < t of L[t][s] x_s
        __syncwarp();
        const float* lower = shared.lower + mine * 16 * kLowerPitch + mine * 16;
        float x[16];
#pragma unroll
        for (uint32_t t = 0; t < 16; ++t) {
            float even = t == lane ? 1.0f : 0.0f, odd = 0.0f;
#pragma unroll
            for (uint32_t s = 0; s < t; s += 2) {
                const float2 both = *reinterpret_cast<const float2*>(lower + t * kLowerPitch + s);
                even = fmaf(both.x, x[s], even);
                if (s + 1 < t) odd = fmaf(both.y, x[s + 1], odd);
            }
            x[t] = even + odd;
            if (lane < 16) shared.inverse[mine][t * kInversePitch + lane] = x[t];
        }
#pragma unroll 2
        for (uint32_t t = 0; t < kTokens; t += 8) {
            multiply_rows<false>(behind, load_a_transposed<true>(shared.k + t * kPitch + mine * 16, kPitch, lane),
                                   shared.v + t * kPitch, lane);
        }
    }
    __syncthreads();                               // K is free
    if (forward) {
#pragma unroll
        for (uint32_t n = 0; n < 8; ++n) {
            store_c(shared.k + mine * 16 * kPitch + n * 8, kPitch, lane, with_values[n]);
        }
    }
    __syncthreads();

    // ---- W (first four warps, over U) and Z (the others, over K): 16 columns per warp, 16 rows after 16 rows
    {
        float* columns = (forward ? shared.u : shared.k) + warp % 4 * 16;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            float* target = columns + i * 16 * kPitch;
            if (i > 0) {
                float side[2][4];
                load_c(target, kPitch, lane, side[0]);
                load_c(target + 8, kPitch, lane, side[1]);
#pragma unroll
                for (uint32_t s = 0; s < i * 16; s += 8) {
                    mma_split(side, load_a<true>(shared.lower + i * 16 * kLowerPitch + s, kLowerPitch, lane),
                              load_b<true>(columns + s * kPitch, kPitch, lane),
                              load_b<true>(columns + s * kPitch + 8, kPitch, lane));
                }
                __syncwarp();
                store_c(target, kPitch, lane, side[0]);
                store_c(target + 8, kPitch, lane, side[1]);
                __syncwarp();
            }
            float solved[2][4] = {};
#pragma unroll
            for (uint32_t s = 0; s < 16; s += 8) {
                mma_split(solved, load_a<true>(shared.inverse[i] + s, kInversePitch, lane),
                          load_b<true>(target + s * kPitch, kPitch, lane),
                          load_b<true>(target + s * kPitch + 8, kPitch, lane));
            }
            __syncwarp();
            store_c(target, kPitch, lane, solved[0]);
            store_c(target + 8, kPitch, lane, solved[1]);
            __syncwarp();
        }
    }
    __syncthreads();

    float from_state[8][4] = {};                   // A or R'
    if (forward) {
#pragma unroll 1
        for (uint32_t t = 0; t < kTokens; t += 8) {
            const FragmentA<true> a = load_a_transposed<true>(shared.b + t * kPitch + mine * 16, kPitch, lane);
            multiply_rows<false>(from_state, a, shared.u + t * kPitch, lane);
            multiply_rows<false>(behind, a, shared.k + t * kPitch, lane);
        }
        const uint32_t channel = mine * 16 + (lane >> 2);
        float decay[2] = {1.0f, 1.0f};
#pragma unroll
        for (uint32_t other = 0; other < 4; ++other) {
            decay[0] *= shared.block_decay[other][channel];
            decay[1] *= shared.block_decay[other][channel + 8];
        }
        if ((lane & 3) == 0) {
            chunk[kP + channel] = decay[0];
            chunk[kP + channel + 8] = decay[1];
        }
#pragma unroll
        for (uint32_t n = 0; n < 8; ++n) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                from_state[n][i] *= decay[i >> 1];
                behind[n][i] *= decay[i >> 1];
            }
        }
    } else {
#pragma unroll
        for (uint32_t n = 0; n < 8; ++n) load_c(rows + n * 8, kPitch, lane, from_state[n]);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            if (j > mine) continue;
#pragma unroll
            for (uint32_t n = 0; n < 2; ++n) {
                const FragmentA<true> a = a_from_c(against_b[j][n]);
                multiply_rows<true>(from_state, a, shared.u + (j * 16 + n * 8) * kPitch, lane);
                multiply_rows<true>(with_values, a, shared.k + (j * 16 + n * 8) * kPitch, lane);
            }
        }
    }
    float4* first = reinterpret_cast<float4*>(chunk + (forward ? 0 : kR)) + mine * 8 * 32 + lane;
    float4* second = reinterpret_cast<float4*>(chunk + (forward ? kD : kO)) + mine * 8 * 32 + lane;
#pragma unroll
    for (uint32_t n = 0; n < 8; ++n) {
        // A and R' as operands of the next product, D and O' as accumulators
        first[n * 32] = make_float4(from_state[n][0], from_state[n][2], from_state[n][1], from_state[n][3]);
        second[n * 32] = forward ? make_float4(behind[n][0], behind[n][1], behind[n][2], behind[n][3])
                                 : make_float4(with_values[n][0], with_values[n][1], with_values[n][2], with_values[n][3]);
    }
}

template <bool NEAREST>
__device__ __forceinline__ FragmentA<NEAREST> operand_of(const float4& stored) {
    FragmentA<NEAREST> out;
    out.set(0, stored.x);
    out.set(1, stored.y);
    out.set(2, stored.z);
    out.set(3, stored.w);
    return out;
}

// A CTA carries 16 value columns of one head through one segment; a warp owns 16 key channels of A and D and copies them
// into its own part of shared memory kCarryStages - 1 chunks ahead.  Bound by the chain load S, multiply, store S, barrier.
__global__ void __launch_bounds__(kCarryThreads)
delta_carry_kernel(const DeltaArgs<__nv_bfloat16> args, uint32_t head0, uint32_t head_count, uint32_t tiles, float* chunks) {
    extern __shared__ __align__(16) float carry_shared[];
    float4* stages = reinterpret_cast<float4*>(carry_shared);                     // [stage][10][thread]
    float* states = carry_shared + kCarryStages * 10 * kCarryThreads * 4;         // [2][channel][kCarryPitch]
    float* decays = states + 2 * kDim * kCarryPitch;                              // [stage][channel]
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t part = blockIdx.x % (kDim / kCarryColumns);
    const uint32_t local_head = blockIdx.x / (kDim / kCarryColumns) % head_count;
    const uint32_t segment = blockIdx.x / (kDim / kCarryColumns) / head_count;
    const uint32_t head = head0 + local_head;
    const size_t slot = args.segments.slots[segment];
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    auto chunks_of = [&](uint32_t which) {
        const uint32_t begin = args.segments.offsets[which];
        uint32_t end = args.segments.offsets[which + 1];
        end = end < args.segments.num_tokens ? end : static_cast<uint32_t>(args.segments.num_tokens);
        return end > begin ? (end - begin + kTokens - 1) / kTokens : 0u;
    };
    const uint32_t count = chunks_of(segment);
    if (count == 0 || slot >= args.segments.num_request_slots) {
        return;
    }
    uint32_t before = 0;
    for (uint32_t other = lane; other < segment; other += 32) before += chunks_of(other);
    before = __reduce_add_sync(0xffffffffu, before);
    // Offsets that go back name more chunks than the step's tokens have, and the scratch holds `tiles` of them: a segment
    // that reaches beyond is left out, here and by the outputs.
    if (before + count > tiles) {
        return;
    }

    const uint32_t dim = args.dim;
    float* state_base = reinterpret_cast<float*>(static_cast<unsigned char*>(args.record.base) + slot * args.record.stride +
                                                 args.record.offset) +
                        static_cast<size_t>(head) * dim * dim;
    for (uint32_t item = threadIdx.x; item < kDim * kCarryColumns; item += kCarryThreads) {
        const uint32_t column = part * kCarryColumns + item / kDim, row = item % kDim;
        states[row * kCarryPitch + item / kDim] =
            row < dim && column < dim ? state_base[static_cast<size_t>(column) * dim + row] : 0.0f;
    }
    auto chunk_of = [&](uint32_t index) {
        return chunks + (static_cast<size_t>(before + index) * head_count + local_head) * kChunkFloats;
    };
    const uint32_t own = warp * 8 * 32 + lane;               // this lane's pieces of A; those of D start at own_d
    const uint32_t own_d = own + part * 2 * 32;
    auto load = [&](uint32_t index) {
        if (index < count) {
            const float4* a = reinterpret_cast<const float4*>(chunk_of(index)) + own;
            const float4* d = reinterpret_cast<const float4*>(chunk_of(index) + kD) + own_d;
            float4* stage = stages + index % kCarryStages * 10 * kCarryThreads + threadIdx.x;
#pragma unroll
            for (uint32_t n = 0; n < 8; ++n) copy_async_16(stage + n * kCarryThreads, a + n * 32, true);
#pragma unroll
            for (uint32_t n = 0; n < 2; ++n) copy_async_16(stage + (8 + n) * kCarryThreads, d + n * 32, true);
            if (threadIdx.x < kDim / 4) {
                copy_async_16(decays + index % kCarryStages * kDim + threadIdx.x * 4, chunk_of(index) + kP + threadIdx.x * 4,
                              true);
            }
        }
        copy_async_commit();
    };
    for (uint32_t index = 0; index + 1 < kCarryStages; ++index) load(index);
    for (uint32_t index = 0; index < count; ++index) {
        copy_async_wait<kCarryStages - 2>();                 // a thread reads A and D that it copied itself
        __syncthreads();
        load(index + kCarryStages - 1);
        const float* state = states + index % 2 * kDim * kCarryPitch;
        const float4* stage = stages + index % kCarryStages * 10 * kCarryThreads + threadIdx.x;
        float sum[2][4];
#pragma unroll
        for (uint32_t n = 0; n < 2; ++n) {
            const float4 d = stage[(8 + n) * kCarryThreads];
            sum[n][0] = d.x;
            sum[n][1] = d.y;
            sum[n][2] = d.z;
            sum[n][3] = d.w;
            const float* decay = decays + index % kCarryStages * kDim + warp * 16 + (lane >> 2);
            float held[4];
            load_c(state + warp * 16 * kCarryPitch + n * 8, kCarryPitch, lane, held);
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) sum[n][i] = fmaf(decay[i >> 1 << 3], held[i], sum[n][i]);
        }
        float4 kept[2];
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) {
            const FragmentA<true> a = operand_of<true>(stage[c * kCarryThreads]);
            const float* rows = state + (c * 8 + (lane & 3) * 2) * kCarryPitch + (lane >> 2);
#pragma unroll
            for (uint32_t n = 0; n < 2; ++n) {
                FragmentB<true> b;
                const float first = rows[n * 8], second = rows[n * 8 + kCarryPitch];
                b.set(0, first);
                b.set(1, second);
                if (c == 2 * warp) {
                    kept[n].x = first;
                    kept[n].y = second;
                } else if (c == 2 * warp + 1) {
                    kept[n].z = first;
                    kept[n].w = second;
                }
                mma_split(sum[n], a, b);
            }
        }
        // the state before the chunk, as operands of the outputs' product
        float4* before_chunk = reinterpret_cast<float4*>(chunk_of(index) + kD) + own_d;
        float* next = states + (index + 1) % 2 * kDim * kCarryPitch + warp * 16 * kCarryPitch;
#pragma unroll
        for (uint32_t n = 0; n < 2; ++n) {
            before_chunk[n * 32] = kept[n];
            store_c(next + n * 8, kCarryPitch, lane, sum[n]);
        }
    }
    __syncthreads();
    const float* state = states + count % 2 * kDim * kCarryPitch;
    for (uint32_t item = threadIdx.x; item < kDim * kCarryColumns; item += kCarryThreads) {
        const uint32_t column = part * kCarryColumns + item / kDim, row = item % kDim;
        if (row < dim && column < dim) {
            state_base[static_cast<size_t>(column) * dim + row] = state[row * kCarryPitch + item / kDim];
        }
    }
}

__device__ __forceinline__ void store_pair(__nv_bfloat16* target, float low, float high) {
    *reinterpret_cast<uint32_t*>(target) = pack_bf16x2(low, high);
}

// 16 tokens per warp: O = R' S_0 + O', the norm over the head, the gate.  Bound by reading 48 KB per chunk.
__global__ void __launch_bounds__(kFinishThreads)
delta_finish_kernel(const DeltaArgs<__nv_bfloat16> args, uint32_t head0, uint32_t head_count, const float* chunks) {
    pdl_launch_dependents();
    pdl_wait();
    const SegmentTile tile = locate_tile(args.segments, kTokens, blockIdx.x / head_count);
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (warp * 16 >= tile.count || args.segments.slots[tile.segment] >= args.segments.num_request_slots ||
        segment_end_tile(tile, kTokens, blockIdx.x / head_count) > gridDim.x / head_count) {
        return;
    }
    const size_t head_base = static_cast<size_t>(head0 + blockIdx.x % head_count) * args.dim;
    const size_t width = static_cast<size_t>(args.heads) * args.dim;
    const float* chunk = chunks + static_cast<size_t>(blockIdx.x) * kChunkFloats;
    const float4* operands = reinterpret_cast<const float4*>(chunk + kR) + warp * 8 * 32 + lane;
    const float4* partial = reinterpret_cast<const float4*>(chunk + kO) + warp * 8 * 32 + lane;
    const float4* states = reinterpret_cast<const float4*>(chunk + kD) + lane;
    float out[8][4];
#pragma unroll
    for (uint32_t n = 0; n < 8; ++n) {
        const float4 value = partial[n * 32];
        out[n][0] = value.x;
        out[n][1] = value.y;
        out[n][2] = value.z;
        out[n][3] = value.w;
    }
#pragma unroll
    for (uint32_t m = 0; m < 4; ++m) {
        const FragmentA<> a0 = operand_of<false>(operands[2 * m * 32]), a1 = operand_of<false>(operands[(2 * m + 1) * 32]);
#pragma unroll
        for (uint32_t n = 0; n < 8; ++n) {
            const float4 state = states[(m * 8 + n) * 32];
            FragmentB<> b0, b1;
            b0.set(0, state.x);
            b0.set(1, state.y);
            b1.set(0, state.z);
            b1.set(1, state.w);
            mma_split(out[n], a0, b0);
            mma_split(out[n], a1, b1);
        }
    }
#pragma unroll
    for (uint32_t half = 0; half < 2; ++half) {
        float squares = 0.0f;
#pragma unroll
        for (uint32_t n = 0; n < 8; ++n) {
            squares = fmaf(out[n][2 * half], out[n][2 * half], fmaf(out[n][2 * half + 1], out[n][2 * half + 1], squares));
        }
        squares += __shfl_xor_sync(0xffffffffu, squares, 1);
        squares += __shfl_xor_sync(0xffffffffu, squares, 2);
        const float factor = rsqrtf(squares / static_cast<float>(args.dim) + args.eps);
        const uint32_t token = warp * 16 + (lane >> 2) + half * 8;
        if (token < tile.count) {
            const size_t row = tile.first + token;
            const __nv_bfloat16* gates = args.projected + row * args.pitch + 3 * width + head_base;
            __nv_bfloat16* target = args.out + row * args.out_pitch + head_base;
#pragma unroll
            for (uint32_t n = 0; n < 8; ++n) {
                const uint32_t channel = n * 8 + (lane & 3) * 2;
                if (channel < args.dim) {
                    const float2 gate = load_pair(gates + channel);
                    const float2 weight = load_pair(args.norm + head_base + channel);
                    store_pair(target + channel, out[n][2 * half] * factor * weight.x * fast_sigmoid(gate.x),
                               out[n][2 * half + 1] * factor * weight.y * fast_sigmoid(gate.y));
                }
            }
        }
    }
}

}  // namespace

size_t delta_split_bytes(size_t heads, size_t tiles) { return heads * tiles * kChunkFloats * sizeof(float); }

// Heads are taken in groups whose chunks fit the scratch.
cudaError_t launch_delta_split(cudaStream_t stream, const DeltaArgs<__nv_bfloat16>& args, float* chunks,
                               size_t chunk_bytes) {
    const size_t tiles = tile_bound(args.segments, kTokens);
    const uint32_t most = static_cast<uint32_t>(std::min<size_t>(args.heads, chunk_bytes / delta_split_bytes(1, tiles)));
    if (most == 0) return cudaErrorInvalidValue;
    const uint32_t groups = (args.heads + most - 1) / most;
    const uint32_t group = (args.heads + groups - 1) / groups;
    const size_t carry_bytes = (kCarryStages * (10 * kCarryThreads * 4 + kDim) + 2 * kDim * kCarryPitch) * sizeof(float);
    cudaError_t status = cudaFuncSetAttribute(reinterpret_cast<const void*>(delta_form_kernel),
                                              cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(FormShared));
    if (status == cudaSuccess) {
        status = cudaFuncSetAttribute(reinterpret_cast<const void*>(delta_carry_kernel),
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(carry_bytes));
    }
    for (uint32_t head0 = 0; head0 < args.heads && status == cudaSuccess; head0 += group) {
        const uint32_t count = std::min(group, args.heads - head0);
        const unsigned int blocks = static_cast<unsigned int>(tiles * count);
        status = launch_kernel(delta_form_kernel, blocks, kFormThreads, sizeof(FormShared), stream, 1, args, head0, count,
                               chunks);
        if (status == cudaSuccess) {
            status = launch_kernel(delta_carry_kernel,
                                   static_cast<unsigned int>(args.segments.num_segments * count * (kDim / kCarryColumns)),
                                   kCarryThreads, carry_bytes, stream, 1, args, head0, count, tiles, chunks);
        }
        if (status == cudaSuccess) {
            status = launch_kernel(delta_finish_kernel, blocks, kFinishThreads, 0, stream, 1, args, head0, count, chunks);
        }
    }
    return status;
}

}  // namespace lfm25

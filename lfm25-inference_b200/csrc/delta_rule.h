// Shared by the kernels of the generalised delta rule: their argument block, the element functions of bf16 prompts, and
// matrix products in TF32 with f32-sized errors.
#pragma once

#include "stack_common.cuh"

namespace lfm25 {

constexpr float kUnitEps = 1e-6f;
constexpr float kDecayScale = 0.60653065971263342f;    // exp(-1/2)

template <typename T>
struct DeltaArgs {
    StackSegments segments;
    uint32_t heads, dim, rank;
    const T* projected;
    size_t pitch;
    const __nv_bfloat16* decay_up;
    const __nv_bfloat16* decay_base;
    const __nv_bfloat16* removal_bias;
    const __nv_bfloat16* norm;
    StackRecord record;
    float* raw;
    T* out;
    size_t out_pitch;
    float eps;
    uint32_t splits;         // CTAs per head, each with COLUMNS value channels
};

using Pair = unsigned long long;     // two f32 values

__device__ __forceinline__ Pair pair_of(float low, float high) {
    Pair out;
    asm("mov.b64 %0, {%1, %2};" : "=l"(out) : "f"(low), "f"(high));
    return out;
}
__device__ __forceinline__ float pair_sum(Pair value) {
    float low, high;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(low), "=f"(high) : "l"(value));
    return low + high;
}
__device__ __forceinline__ float low_of(Pair value) { return __uint_as_float(static_cast<uint32_t>(value)); }
__device__ __forceinline__ float high_of(Pair value) { return __uint_as_float(static_cast<uint32_t>(value >> 32)); }
__device__ __forceinline__ Pair fma_pair(Pair a, Pair b, Pair c) {
    Pair out;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(out) : "l"(a), "l"(b), "l"(c));
    return out;
}
__device__ __forceinline__ Pair add_pair(Pair a, Pair b) {
    Pair out;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(out) : "l"(a), "l"(b));
    return out;
}
__device__ __forceinline__ Pair mul_pair(Pair a, Pair b) {
    Pair out;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(out) : "l"(a), "l"(b));
    return out;
}

// Decays and rates: the fast f32 exponential and division, a few units in the last place from the
// correctly rounded ones.
__device__ __forceinline__ float fast_sigmoid(float z) { return __fdividef(1.0f, 1.0f + __expf(-z)); }
__device__ __forceinline__ float fast_tanh(float z) { return 1.0f - __fdividef(2.0f, 1.0f + __expf(2.0f * z)); }

// D(16x8) += A(16x8, tf32) * B(8x8, tf32), f32 accumulation
__device__ __forceinline__ void mma_tf32(float (&d)[4], const float (&a)[4], const float (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
          "r"(__float_as_uint(b[0])), "r"(__float_as_uint(b[1])));
}

// An operand fragment as high + low.  TF32 keeps 10 mantissa bits and ignores the rest: the high part is what it keeps of the
// value, the low part the remainder, of which it keeps another 10.  NEAREST: the high part is rounded to nearest, which
// halves the low one and leaves it either sign, so that what the products leave out has no direction.
template <int N, bool NEAREST = false>
struct SplitFragment {
    float high[N], low[N];
    __device__ __forceinline__ void set(int index, float value) {
        high[index] = __uint_as_float((__float_as_uint(value) + (NEAREST ? 0x1000u : 0u)) & 0xffffe000u);
        low[index] = value - high[index];
    }
};
template <bool NEAREST = false>
using FragmentA = SplitFragment<4, NEAREST>;
template <bool NEAREST = false>
using FragmentB = SplitFragment<2, NEAREST>;

// The tensor cores cut what falls behind the accumulator's last bit.  NEAREST: every product of fragments starts from zero
// and is added up with rounding to nearest.
template <bool NEAREST, uint32_t COUNT>
__device__ __forceinline__ void mma_split(float (*d)[4], const FragmentA<NEAREST>& a, const FragmentB<NEAREST> (&b)[COUNT]) {
    float sums[COUNT][4] = {};
    float (*target)[4] = NEAREST ? sums : d;
    // the accumulators' products alternate so that none waits for the one before it
#pragma unroll
    for (uint32_t n = 0; n < COUNT; ++n) mma_tf32(target[n], a.low, b[n].high);
#pragma unroll
    for (uint32_t n = 0; n < COUNT; ++n) mma_tf32(target[n], a.high, b[n].low);
#pragma unroll
    for (uint32_t n = 0; n < COUNT; ++n) mma_tf32(target[n], a.high, b[n].high);
    if (NEAREST) {
#pragma unroll
        for (uint32_t n = 0; n < COUNT; ++n) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) d[n][i] += sums[n][i];
        }
    }
}
template <bool NEAREST>
__device__ __forceinline__ void mma_split(float (&d)[4], const FragmentA<NEAREST>& a, const FragmentB<NEAREST>& b) {
    const FragmentB<NEAREST> one[1] = {b};
    mma_split<NEAREST, 1>(&d, a, one);
}
template <bool NEAREST>
__device__ __forceinline__ void mma_split(float (&d)[2][4], const FragmentA<NEAREST>& a, const FragmentB<NEAREST>& b0,
                                          const FragmentB<NEAREST>& b1) {
    const FragmentB<NEAREST> both[2] = {b0, b1};
    mma_split<NEAREST, 2>(d, a, both);
}
// rows `source[row * stride + column]` of a 16 x 8 operand
template <bool NEAREST = false>
__device__ __forceinline__ FragmentA<NEAREST> load_a(const float* source, uint32_t stride, uint32_t lane) {
    FragmentA<NEAREST> out;
    const float* at = source + (lane >> 2) * stride + (lane & 3);
    out.set(0, at[0]);
    out.set(1, at[8 * stride]);
    out.set(2, at[4]);
    out.set(3, at[8 * stride + 4]);
    return out;
}
// the same operand stored transposed: `source[column * stride + row]`
template <bool NEAREST = false>
__device__ __forceinline__ FragmentA<NEAREST> load_a_transposed(const float* source, uint32_t stride, uint32_t lane) {
    FragmentA<NEAREST> out;
    const float* at = source + (lane & 3) * stride + (lane >> 2);
    out.set(0, at[0]);
    out.set(1, at[8]);
    out.set(2, at[4 * stride]);
    out.set(3, at[4 * stride + 8]);
    return out;
}
// an 8 x 8 operand B[k][n] stored as `source[k * stride + n]`
template <bool NEAREST = false>
__device__ __forceinline__ FragmentB<NEAREST> load_b(const float* source, uint32_t stride, uint32_t lane) {
    FragmentB<NEAREST> out;
    const float* at = source + (lane & 3) * stride + (lane >> 2);
    out.set(0, at[0]);
    out.set(1, at[4 * stride]);
    return out;
}
// a 16 x 8 result to `target[row * stride + column]`
__device__ __forceinline__ void store_c(float* target, uint32_t stride, uint32_t lane, const float (&c)[4]) {
    float* at = target + (lane >> 2) * stride + (lane & 3) * 2;
    *reinterpret_cast<float2*>(at) = make_float2(c[0], c[1]);
    *reinterpret_cast<float2*>(at + 8 * stride) = make_float2(c[2], c[3]);
}

// The kernel of delta_chunk.cu: bf16 segments whose projections lie in whole 16-byte pieces, heads up to kDeltaChunkDim and ranks
// up to what its shared memory holds.
constexpr uint32_t kDeltaChunkDim = 64;
bool delta_chunk_takes(uint32_t dim, uint32_t rank);
cudaError_t launch_delta_chunk(cudaStream_t stream, const DeltaArgs<__nv_bfloat16>& args);

// The kernels of delta_scan.cu: segments of any length in plain f32 arithmetic.  Scratch for `heads` heads of a step of `tokens`
// tokens: all of them, or as many as a bound allows, which are then taken in turns.
size_t delta_scan_bytes(size_t heads, uint32_t dim, size_t tokens);
template <typename T>
cudaError_t launch_delta_scan(cudaStream_t stream, const DeltaArgs<T>& args, float* scratch, size_t scratch_bytes);

// The kernels of delta_split.cu: bf16 segments whose projections lie in whole 16-byte pieces, heads up to 64.
size_t delta_split_bytes(size_t heads, size_t tiles);
cudaError_t launch_delta_split(cudaStream_t stream, const DeltaArgs<__nv_bfloat16>& args, float* chunks,
                               size_t chunk_bytes);

}  // namespace lfm25

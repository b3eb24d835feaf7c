// y[m, n] = x[m, k] w[n, k]^T for f32 activations and bf16 weights, with every product exact and f32 sums.
//
// A weight is a bf16 value, so only x has to be taken apart: x = high + middle + low, each a bf16 value cut from the bits
// of x (8 + 8 + 8 significant bits), which leaves nothing over for |x| above 2^-110 (below it the low part falls under the
// smallest bf16 value).  This is the splitting of a floating-point number into shorter ones that Dekker (1971) and Ozaki et al.
// (2012) use for exact products; the three products with w are exact in the tensor core's arithmetic (bf16 x bf16 in f32).
//
// What the sums keep: the high parts' products are summed 32 at a time in the tensor core, from zero, and these short
// sums are added up in f32 with rounding to nearest; the other two parts, at most 2^-7 of the first, go to an accumulator
// of their own that stays in the tensor core.  The tensor core cuts what falls behind its accumulator's last bit: 2^-23 of a
// short sum, 2^-30 of the whole for the parts.  Measured against float64 through a whole model of 8 layers (250 tokens,
// k = 1024 and 7168): logits off by 1.0e-6 (2-norm), by 6.7e-6 with serial chains of f32 multiply-adds.
//
// Bound: the tensor pipe through mma.sync (3 instructions of 16x8x16 per 16x8x16 block) for prompts, the weight stream for
// a few rows.  A CTA owns ROWS x 128 outputs; its four warps take 32 columns each.  Weights arrive through a cp.async ring
// (the first stages before the dependency wait: they are constants), x through registers, where it is taken apart once per
// CTA.  Where the tiles do not fill the device, the CTAs of a cluster share a tile's k range and add their f32 parts in
// rank order through distributed shared memory.  250 rows of k = 1024 and 7168, n = 1024 to 6144 (25 products of a step): 48 us
// a product, 232 with plain multiply-adds (64 x 64 outputs per CTA).
#include <cooperative_groups.h>

#include "launch.h"
#include "stack_common.cuh"

namespace lfm25 {

namespace {

constexpr uint32_t kThreads = 128;
constexpr uint32_t kColumns = 128;
constexpr uint32_t kWarpColumns = kColumns / 4;
constexpr uint32_t kDepth = 32;                    // k per round
constexpr uint32_t kPitch = kDepth + 8;            // elements: rows 80 bytes apart, conflict-free ldmatrix
constexpr uint32_t kStages = 4;                    // weight tiles in the ring
constexpr uint32_t kOutPitch = kColumns + 4;       // floats

template <uint32_t ROWS>
constexpr size_t shared_bytes() {
    const size_t ring = (kStages * kColumns + 2 * 3 * ROWS) * kPitch * 2;
    const size_t parked = static_cast<size_t>(ROWS) * kOutPitch * 4;
    return ring > parked ? ring : parked;
}

struct Parts {
    __nv_bfloat16 high, middle, low;
};
__device__ __forceinline__ Parts take_apart(float x) {
    const uint32_t bits = __float_as_uint(x);
    const float high = __uint_as_float(bits & 0xffff0000u);
    const float rest = x - high;                                                     // exact
    const float middle = __uint_as_float(__float_as_uint(rest) & 0xffff0000u);
    Parts parts = {__float2bfloat16_rn(high), __float2bfloat16_rn(middle), __float2bfloat16_rn(rest - middle)};
    if ((bits & 0x7f800000u) == 0x7f800000u) {       // infinities and NaN have no rest
        parts = {__float2bfloat16_rn(x), __float2bfloat16_rn(0.0f), __float2bfloat16_rn(0.0f)};
    }
    return parts;
}

template <uint32_t ROWS>
__global__ void __launch_bounds__(kThreads)
linear_f32_kernel(const float* x, const __nv_bfloat16* weight, float* y, uint32_t m, uint32_t n, uint32_t k,
                  uint32_t column_tiles, uint32_t splits) {
    // x is no __restrict__ pointer: a load that the compiler takes for one of constant memory may move above pdl_wait()
    constexpr uint32_t kTilesM = ROWS / 16;
    constexpr uint32_t kTilesN = kWarpColumns / 8;
    constexpr uint32_t kLoads = ROWS * kDepth / 4 / kThreads;          // float4 of x per thread and round
    static_assert(ROWS % 16 == 0 && kLoads >= 1, "whole MMA tiles and whole loads");
    extern __shared__ __align__(16) unsigned char linear_shared[];
    __nv_bfloat16* ring = reinterpret_cast<__nv_bfloat16*>(linear_shared);              // [stage][column][kPitch]
    __nv_bfloat16* parts = ring + kStages * kColumns * kPitch;                          // [2][part][row][kPitch]
    const uint32_t split = blockIdx.x % splits;
    const uint32_t tile = blockIdx.x / splits;
    const uint32_t row0 = tile / column_tiles * ROWS;
    const uint32_t column0 = tile % column_tiles * kColumns;
    const uint32_t rounds_total = (k + kDepth - 1) / kDepth;
    const uint32_t round0 = static_cast<uint32_t>(static_cast<uint64_t>(rounds_total) * split / splits);
    const uint32_t rounds = static_cast<uint32_t>(static_cast<uint64_t>(rounds_total) * (split + 1) / splits) - round0;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;

    // four threads per weight row and round, 32 rows at a time
    auto load_weights = [&](uint32_t round) {
        if (round < rounds) {
            const uint32_t depth = (round0 + round) * kDepth + (threadIdx.x & 3) * 8;
            __nv_bfloat16* target = ring + round % kStages * kColumns * kPitch + (threadIdx.x & 3) * 8;
#pragma unroll
            for (uint32_t part = 0; part < kColumns / 32; ++part) {
                const uint32_t row = (threadIdx.x >> 2) + part * 32;
                const bool inside = column0 + row < n && depth < k;    // k is a multiple of 8
                const __nv_bfloat16* source = inside ? weight + static_cast<size_t>(column0 + row) * k + depth : weight;
                copy_async_16(target + row * kPitch, source, inside);
            }
        }
        copy_async_commit();
    };
    // eight threads per row of x and round, 16 rows at a time
    float4 pending[kLoads];
    auto load_x = [&](uint32_t round) {
        const uint32_t depth = (round0 + round) * kDepth + (threadIdx.x & 7) * 4;
#pragma unroll
        for (uint32_t part = 0; part < kLoads; ++part) {
            const uint32_t row = row0 + (threadIdx.x >> 3) + part * (kThreads / 8);
            pending[part] = round < rounds && row < m && depth < k
                                ? *reinterpret_cast<const float4*>(x + static_cast<size_t>(row) * k + depth)
                                : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    auto store_x = [&](uint32_t round) {
        __nv_bfloat16* target = parts + round % 2 * 3 * ROWS * kPitch + (threadIdx.x & 7) * 4;
#pragma unroll
        for (uint32_t part = 0; part < kLoads; ++part) {
            const uint32_t row = (threadIdx.x >> 3) + part * (kThreads / 8);
            const Parts a = take_apart(pending[part].x), b = take_apart(pending[part].y);
            const Parts c = take_apart(pending[part].z), d = take_apart(pending[part].w);
            const __nv_bfloat162 values[6] = {
                __halves2bfloat162(a.high, b.high),     __halves2bfloat162(c.high, d.high),
                __halves2bfloat162(a.middle, b.middle), __halves2bfloat162(c.middle, d.middle),
                __halves2bfloat162(a.low, b.low),       __halves2bfloat162(c.low, d.low)};
#pragma unroll
            for (uint32_t which = 0; which < 3; ++which) {
                __nv_bfloat162* at = reinterpret_cast<__nv_bfloat162*>(target + (which * ROWS + row) * kPitch);
                at[0] = values[2 * which];
                at[1] = values[2 * which + 1];
            }
        }
    };

#pragma unroll
    for (uint32_t round = 0; round < kStages - 1; ++round) load_weights(round);
    pdl_wait();
    load_x(0);
    store_x(0);
    load_x(1);

    float main_sum[kTilesM][kTilesN][4] = {}, rest_sum[kTilesM][kTilesN][4] = {};
    for (uint32_t round = 0; round < rounds; ++round) {
        copy_async_wait<kStages - 2>();
        __syncthreads();       // this round's weights and x are in shared memory, the round before has been read
        load_weights(round + kStages - 1);
        if (round + 1 < rounds) {
            store_x(round + 1);
            load_x(round + 2);
        }
        const __nv_bfloat16* weights = ring + round % kStages * kColumns * kPitch + warp * kWarpColumns * kPitch;
        const __nv_bfloat16* rows = parts + round % 2 * 3 * ROWS * kPitch;
        uint32_t b[2][kTilesN][2];                 // [16 of k][8 columns]
#pragma unroll
        for (uint32_t step = 0; step < 2; ++step) {
#pragma unroll
            for (uint32_t pair = 0; pair < kTilesN / 2; ++pair) {
                const uint32_t address = smem_u32(weights + (pair * 16 + lane / 16 * 8 + lane % 8) * kPitch + step * 16 +
                                                  lane / 8 % 2 * 8);
                ldmatrix_x4(address, b[step][2 * pair][0], b[step][2 * pair][1], b[step][2 * pair + 1][0],
                            b[step][2 * pair + 1][1]);
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < kTilesM; ++i) {
            const uint32_t offset = (i * 16 + lane % 16) * kPitch + lane / 16 * 8;
            float fresh[kTilesN][4] = {};
#pragma unroll
            for (uint32_t step = 0; step < 2; ++step) {
#pragma unroll
                for (uint32_t which = 0; which < 3; ++which) {
                    uint32_t a[4];
                    ldmatrix_x4(smem_u32(rows + which * ROWS * kPitch + offset + step * 16), a[0], a[1], a[2], a[3]);
#pragma unroll
                    for (uint32_t j = 0; j < kTilesN; ++j) {
                        mma_bf16_16816(which == 0 ? fresh[j] : rest_sum[i][j], a[0], a[1], a[2], a[3], b[step][j][0],
                                       b[step][j][1]);
                    }
                }
            }
#pragma unroll
            for (uint32_t j = 0; j < kTilesN; ++j) {
#pragma unroll
                for (uint32_t e = 0; e < 4; ++e) main_sum[i][j][e] += fresh[j][e];
            }
        }
    }
    // The successors are let in only now: a grid of several waves would otherwise share its SMs with CTAs that wait for it.
    pdl_launch_dependents();
#pragma unroll
    for (uint32_t i = 0; i < kTilesM; ++i) {
#pragma unroll
        for (uint32_t j = 0; j < kTilesN; ++j) {
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) {
                // a weight that is no finite number meets parts that are zero: the high part alone has the right answer
                const float rest = rest_sum[i][j][e];
                main_sum[i][j][e] += isfinite(rest) ? rest : 0.0f;
            }
        }
    }
    const uint32_t row_of = lane >> 2, column_of = warp * kWarpColumns + (lane & 3) * 2;
    if (splits == 1) {
#pragma unroll
        for (uint32_t i = 0; i < kTilesM; ++i) {
#pragma unroll
            for (uint32_t j = 0; j < kTilesN; ++j) {
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {
                    const uint32_t row = row0 + i * 16 + row_of + half * 8;
                    const uint32_t column = column0 + column_of + j * 8;
                    float* target = y + static_cast<size_t>(row) * n + column;
                    if (row < m && column < n) target[0] = main_sum[i][j][2 * half];
                    if (row < m && column + 1 < n) target[1] = main_sum[i][j][2 * half + 1];
                }
            }
        }
        return;
    }
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    float* parked = reinterpret_cast<float*>(linear_shared);           // [row][kOutPitch]
    copy_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < kTilesM; ++i) {
#pragma unroll
        for (uint32_t j = 0; j < kTilesN; ++j) {
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                *reinterpret_cast<float2*>(parked + (i * 16 + row_of + half * 8) * kOutPitch + column_of + j * 8) =
                    make_float2(main_sum[i][j][2 * half], main_sum[i][j][2 * half + 1]);
            }
        }
    }
    cluster.sync();
    // rank r finishes the rows r, r + splits, ..; a warp reads one row of each partner per pass
    for (uint32_t row = split + warp * splits; row < ROWS && row0 + row < m; row += 4 * splits) {
        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t rank = 0; rank < splits; ++rank) {
            const float* source = cluster.map_shared_rank(parked, rank) + row * kOutPitch + lane * 4;
            const float4 part = *reinterpret_cast<const float4*>(source);
            sum.x += part.x;
            sum.y += part.y;
            sum.z += part.z;
            sum.w += part.w;
        }
        const uint32_t column = column0 + lane * 4;
        float* target = y + static_cast<size_t>(row0 + row) * n + column;
        if (column < n) target[0] = sum.x;
        if (column + 1 < n) target[1] = sum.y;
        if (column + 2 < n) target[2] = sum.z;
        if (column + 3 < n) target[3] = sum.w;
    }
    cluster.sync();       // nobody leaves while its part is still being read
}

template <uint32_t ROWS>
cudaError_t launch(cudaStream_t stream, const float* x, const __nv_bfloat16* weight, float* y, size_t m, size_t n, size_t k) {
    const size_t column_tiles = (n + kColumns - 1) / kColumns;
    const size_t tiles = (m + ROWS - 1) / ROWS * column_tiles;
    const size_t rounds = (k + kDepth - 1) / kDepth;
    // as many CTAs as two per SM, each with eight rounds at least
    uint32_t splits = 1;
    while (splits < 8 && tiles * splits * 2 <= 2 * 148 && rounds >= 16 * splits) splits *= 2;
    if (tiles == 0 || tiles * splits > 0x7fffffffu) return cudaErrorInvalidValue;
    const auto kernel = linear_f32_kernel<ROWS>;
    constexpr size_t shared = shared_bytes<ROWS>();
    const cudaError_t status = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared));
    if (status != cudaSuccess) return status;
    return launch_kernel(kernel, static_cast<unsigned int>(tiles * splits), kThreads, shared, stream, splits, x, weight, y,
                         m, n, k, column_tiles, splits);
}

}  // namespace

bool linear_f32_supports(const void* x, const void* weight, size_t m, size_t n, size_t k) {
    return k > 0 && k % 8 == 0 && aligned_to(x, 16) && aligned_to(weight, 16) && m <= 0x7fffffffu && n <= 0x7fffffffu &&
           k <= 0x7fffffffu;
}

cudaError_t launch_linear_f32(cudaStream_t stream, const void* x, const void* weight, void* y, size_t m, size_t n,
                              size_t k) {
    const auto* activations = static_cast<const float*>(x);
    const auto* weights = static_cast<const __nv_bfloat16*>(weight);
    auto* out = static_cast<float*>(y);
    if (m <= 16) return launch<16>(stream, activations, weights, out, m, n, k);
    // three tiles of 32 rows rather than two of 64, which would be half empty: a step of 70 tokens 1367 -> 1284 us (width
    // 1024, 8 layers); at 130 rows five of 32 lose to three of 64, 1547 against 2056 us
    if (m <= 32 || (m > 64 && m <= 96)) return launch<32>(stream, activations, weights, out, m, n, k);
    return launch<64>(stream, activations, weights, out, m, n, k);
}

}  // namespace lfm25

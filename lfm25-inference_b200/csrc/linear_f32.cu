// y[m, n] = x[m, k] w[n, k]^T for f32 activations and bf16 weights on the 5th-generation tensor cores, with every product
// exact and f32 sums.
//
// A weight is a bf16 value, so only x has to be taken apart: x = high + middle + low, each a bf16 value cut from the bits
// of x (8 + 8 + 8 significant bits), which leaves nothing over for |x| above 2^-110 (below it the low part falls under the
// smallest bf16 value).  This is the splitting of a floating-point number into shorter ones that Dekker (1971) and Ozaki et al.
// (2012) use for exact products; the three products with w are exact in the tensor core's arithmetic (bf16 x bf16 in f32).
//
// What the sums keep: the tensor core cuts what falls behind its accumulator's last bit, so the high parts' products are summed
// 64 at a time, from zero, and these short sums are added up in registers, two and two, with rounding to nearest; the other
// two parts, at most 2^-7 of the first, go to an accumulator of their own that stays in tensor memory (2^-30 of the whole).
// Short sums of 32, 64, 128 and 256 products: 1.17, 1.07, 1.37 and 2.38e-7 from float64 (2-norm, k = 1024, not in pairs), all of
// k in one: 1.0e-6.
//
// A tile is 128 weight rows (the M operand, from TMA) times N rows of x (the N operand), 16, 32, 64 or 96.  Per 64
// of k a slot of the ring holds the weights and the three parts of x.  Warps:
//     0         TMA loads of the weights; the first ring is requested before the dependency wait (they are constants)
//     1         issues the MMAs: four for the high parts into one of four accumulators that take turns, eight for the others,
//               and allocates tensor memory.  One commit and two waits a slot: with a barrier for each purpose and short sums of
//               32 (three commits, four waits) the lone thread took 1300 to 1800 cycles a slot
//     2 to 9    take x apart: f32 from global memory two slots ahead in registers, three bf16 tiles into the slot
//     10 to 17  add the short sums up: 32 weight rows and half of the columns each, N / 2 sums in registers
// Bound: shared memory, which the MMAs' operands (12 x (4 KiB + 32 N bytes) a slot) and the parts of x pass through: a slot takes
// 100 + 16 N cycles, the MMAs' arithmetic 6 N.  Where the tiles do not fill the device, the CTAs of a cluster share a tile's
// k range and add their f32 parts in rank order through distributed shared memory.
//
// Against the same products through mma.sync (three 16x8x16 per block, 64 x 128 outputs per CTA), us, launches back to back and
// weights beyond the L2:
//     rows x n x k     250x6144x1024   250x1024x7168   64x6144x1024   16x1024x7168   1x32768x1024   2500x2048x12288
//     mma.sync                  49.1            45.3           16.7           18.4           22.4              1553
//     here                      19.1            24.9            9.9           10.2           13.1               615
// Up to 16 rows take tiles of 16: 1 x 6144 x 1024 7.9 / 7.2, 16 x 1024 x 2048 6.7 / 6.1 (in tiles of 32 8.2 and 7.0, 16 x 64 x 64
// 2.3 / 2.6 instead of 2.1); 16 x 2048 x 2048, four blocks of k in 128 CTAs, stays behind with 7.4 / 7.9.
//
// Every mbarrier wait is bounded; a wait that runs out sets the CTA's abort flag, is recorded in the device status words, and
// the CTA (in a cluster: all its CTAs) leaves without storing, once its copies and MMAs are through (drain()).
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cstddef>

#include "kernels.h"
#include "launch.h"
#include "stack_common.cuh"
#include "tcgen05.cuh"
#include "tensor_map.h"

namespace lfm25 {

namespace {

constexpr uint32_t kThreads = 576;
constexpr uint32_t kTileM = 128;                   // weight rows
constexpr uint32_t kBlockK = 64;                   // of k per slot = one swizzle row of 128 bytes
constexpr uint32_t kWeightBytes = kTileM * 128;
constexpr uint32_t kFirstConverter = 2, kConverters = 8, kFirstAdder = 10, kAdders = 8;
constexpr uint32_t kMaxStages = 6;
constexpr uint32_t kControlBytes = 1024 + 256;     // alignment of the ring and the barriers

template <uint32_t N>
struct Shape {
    static constexpr uint32_t kPartBytes = N * 128;
    static constexpr uint32_t kStageBytes = kWeightBytes + 3 * kPartBytes;
    static constexpr uint32_t kCtas = N <= 32 ? 2 : 1;                     // per SM
    static constexpr uint32_t kBudget = kCtas == 2 ? 110 * 1024 : 216 * 1024;
    static constexpr uint32_t kStages = (kBudget - kControlBytes) / kStageBytes < kMaxStages
                                            ? (kBudget - kControlBytes) / kStageBytes : kMaxStages;
    static constexpr uint32_t kShared = kStages * kStageBytes + kControlBytes;
    // of tensor memory: four short sums, the rest
    static constexpr uint32_t kColumns = N == 16 ? 128 : (5 * N <= 256 ? 256 : 512);
    static constexpr uint32_t kPiece = N == 16 ? 8 : 16;                   // columns that an adding thread reads at a time
    static constexpr uint32_t kLoads = N / (2 * kConverters);              // float4 of x per converting thread and slot
    static_assert(N % 16 == 0 && N / 2 % kPiece == 0, "whole loads");
    static_assert(N * kTileM * 4 <= kStages * kStageBytes, "a parked tile fits the ring");
};

struct LinearParams {
    const float* x;
    float* y;
    unsigned int* status;
    uint64_t wait_limit;
    uint32_t m, n, k;
    uint32_t column_tiles;     // of weight rows
    uint32_t k_blocks, splits;
    uint32_t drop_block;       // self-test: the copy of this K block is armed but never issued
};

// four consecutive values of x as the three parts' bf16 pairs
struct Taken {
    uint2 part[3];
};
__device__ __forceinline__ uint32_t upper_halves(uint32_t low, uint32_t high) { return __byte_perm(low, high, 0x7632); }
// x - its upper half, both exact, for two values
__device__ __forceinline__ void cut(uint32_t& a, uint32_t& b) {
    asm("{\n"
        ".reg .b64 x, h, m;\n"
        "mov.b64 x, {%0, %1};\n"
        "mov.b64 h, {%2, %3};\n"
        "mov.b64 m, {%4, %4};\n"
        "fma.rn.f32x2 x, h, m, x;\n"
        "mov.b64 {%0, %1}, x;\n"
        "}" : "+r"(a), "+r"(b) : "r"(a & 0xffff0000u), "r"(b & 0xffff0000u), "r"(0xbf800000u));
}
__device__ __forceinline__ Taken take_apart(const float4& value) {
    uint32_t x[4] = {__float_as_uint(value.x), __float_as_uint(value.y), __float_as_uint(value.z), __float_as_uint(value.w)};
    Taken taken;
    taken.part[0] = make_uint2(upper_halves(x[0], x[1]), upper_halves(x[2], x[3]));
    const uint32_t largest = max(max(x[0] & 0x7fffffffu, x[1] & 0x7fffffffu), max(x[2] & 0x7fffffffu, x[3] & 0x7fffffffu));
    if (largest >= 0x7f800000u) {           // infinities and NaN have no rest
        uint32_t bits[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const bool special = (x[i] & 0x7f800000u) == 0x7f800000u;
            bits[i] = special ? static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(__uint_as_float(x[i])))) << 16 : x[i];
            x[i] = special ? 0u : x[i];
        }
        taken.part[0] = make_uint2(upper_halves(bits[0], bits[1]), upper_halves(bits[2], bits[3]));
    }
    cut(x[0], x[1]);
    cut(x[2], x[3]);
    taken.part[1] = make_uint2(upper_halves(x[0], x[1]), upper_halves(x[2], x[3]));
    cut(x[0], x[1]);
    cut(x[2], x[3]);
    taken.part[2] = make_uint2(upper_halves(x[0], x[1]), upper_halves(x[2], x[3]));
    return taken;
}

__device__ __forceinline__ void umma(uint32_t accumulator, uint64_t a, uint64_t b, uint32_t descriptor, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(accumulator),
        "l"(a), "l"(b), "r"(descriptor), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void load_columns(uint32_t address, uint32_t (&raw)[8]) { tmem_load8_nowait(address, raw); }
__device__ __forceinline__ void load_columns(uint32_t address, uint32_t (&raw)[16]) { tmem_load16_nowait(address, raw); }

__device__ __forceinline__ void store_shared(uint32_t address, uint32_t value) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(address), "r"(value) : "memory");
}

// What each role has got through when it leaves: blocks of weights requested, blocks of MMAs issued, blocks converted by each warp.
struct Progress {
    uint32_t requested, multiplied, converted[kConverters];
};
constexpr uint32_t kProgressAt = 16 * kMaxStages + 24;   // in the control bytes, behind the barriers and two words
static_assert(kProgressAt + sizeof(Progress) <= 256, "the control bytes end");

// Nobody leaves with a copy or an MMA in flight: only once all roles are through is it known that a wait of the CTA has run out.
// By itself, so that it takes no registers from the roles.
template <uint32_t N>
__device__ __noinline__ void drain(uint8_t* control, uint64_t wait_limit) {
    constexpr uint32_t kStages = Shape<N>::kStages;
    const volatile Progress& progress = *reinterpret_cast<volatile Progress*>(control + kProgressAt);
    if (threadIdx.x == 0) {
        // The last copy of every slot.  Its barrier also counts the converting warps: what those have left out is made good.
        const uint32_t requested = progress.requested;
        for (uint32_t block = requested > kStages ? requested - kStages : 0; block < requested; ++block) {
            const uint32_t bar = smem_u32(control) + 8 * (block % kStages);
            for (uint32_t i = 0; i < kConverters; ++i) {
                if (progress.converted[i] <= block) mbar_arrive(bar);
            }
            (void)mbar_wait_bounded(bar, block / kStages & 1, wait_limit);
        }
    } else if (threadIdx.x / 32 == 1 && progress.multiplied > 0) {
        const uint32_t block = progress.multiplied - 1;
        (void)mbar_wait_bounded(smem_u32(control) + 8 * kMaxStages + 8 * (block % kStages), block / kStages & 1, wait_limit);
    }
}

template <uint32_t N>
__global__ void __launch_bounds__(kThreads, Shape<N>::kCtas)
linear_f32_umma_kernel(const __grid_constant__ CUtensorMap weight_map, const LinearParams p) {
    using S = Shape<N>;
    extern __shared__ uint8_t linear_raw[];
    uint8_t* shared = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(linear_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t ring = smem_u32(shared);
    uint8_t* control = shared + S::kStages * S::kStageBytes;
    const uint32_t bar_ready = smem_u32(control);                          // [stage] weights and parts of x are in the slot
    const uint32_t bar_read = bar_ready + 8 * kMaxStages;                  // [stage] its MMAs are complete
    const uint32_t bar_taken = bar_read + 8 * kMaxStages;                  // [2] a short sum has been added up
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(control + 16 * kMaxStages + 16);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    const uint32_t progress = bar_ready + kProgressAt;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t split = blockIdx.x % p.splits;
    const uint32_t tile = blockIdx.x / p.splits;
    const uint32_t column0 = tile % p.column_tiles * kTileM;               // of y
    const uint32_t row0 = tile / p.column_tiles * N;
    const uint32_t block0 = static_cast<uint32_t>(static_cast<uint64_t>(p.k_blocks) * split / p.splits);
    const uint32_t blocks = static_cast<uint32_t>(static_cast<uint64_t>(p.k_blocks) * (split + 1) / p.splits) - block0;
    const uint32_t ahead = blocks < S::kStages ? blocks : S::kStages;

    auto load_weights = [&](uint32_t block, uint32_t stage) {
        mbar_arrive_expect_tx(bar_ready + 8 * stage, kWeightBytes);
        if (block != p.drop_block) {
            tma_load_2d(ring + stage * S::kStageBytes, &weight_map, bar_ready + 8 * stage,
                        static_cast<int32_t>((block0 + block) * kBlockK), static_cast<int32_t>(column0));
        }
    };
    if (threadIdx.x == 0) {
        tma_prefetch_descriptor(&weight_map);
        for (uint32_t stage = 0; stage < S::kStages; ++stage) {
            mbar_init(bar_ready + 8 * stage, 1 + kConverters);
            mbar_init(bar_read + 8 * stage, 1);
        }
        mbar_init(bar_taken, kAdders);
        mbar_init(bar_taken + 8, kAdders);
        for (uint32_t i = 0; i < kConverters; ++i) store_shared(progress + offsetof(Progress, converted) + 4 * i, 0);
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async_smem();
        for (uint32_t block = 0; block < ahead; ++block) load_weights(block, block);
    }
    __syncwarp();
    if (warp == 1) tmem_allocate(smem_u32(const_cast<uint32_t*>(tmem_slot)), S::kColumns);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto give_up = [&](uint32_t detail) {
        if (!*abort_flag) record_wait_timeout(p.status, kTagLinearF32, (blockIdx.x << 4) | detail);
        *abort_flag = 1;
    };

    float sums[N / 2];
    const uint32_t quadrant = warp & 3;                                    // tensor-memory lanes of an adding warp
    const uint32_t half = warp >= kFirstAdder + 4 ? 1 : 0;                 // and its columns
    if (warp == 0) {
        if (elect_one()) {
            uint32_t stage = 0, parity = 0, issued = ahead;
            for (uint32_t block = ahead; block < blocks; ++block) {
                if (*abort_flag || !mbar_wait_bounded(bar_read + 8 * stage, parity, p.wait_limit)) {
                    give_up(1);
                    break;
                }
                load_weights(block, stage);
                ++issued;
                if (++stage == S::kStages) {
                    stage = 0;
                    parity ^= 1;
                }
            }
            store_shared(progress + offsetof(Progress, requested), issued);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            // D = f32, A = B = bf16, both K-major, N columns, M = 128
            constexpr uint32_t descriptor = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((kTileM >> 4) << 24);
            constexpr uint64_t kDescriptorHigh = (static_cast<uint64_t>(1) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
                                                 (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
            constexpr uint32_t kPart = S::kPartBytes >> 4;
            const uint32_t rest = tmem + 4 * N;
            uint32_t stage = 0, parity = 0, slot = ring, accumulate = 0, block = 0;
            for (; block < blocks; ++block) {
                const uint32_t pair = block / 2;
                if (!mbar_wait_bounded(bar_ready + 8 * stage, parity, p.wait_limit) ||
                    (block % 2 == 0 && pair > 1 && !mbar_wait_bounded(bar_taken + 8 * (pair & 1), (pair / 2 - 1) & 1, p.wait_limit))) {
                    give_up(2);
                    break;
                }
                tcgen05_fence_after();
                const uint64_t a = kDescriptorHigh | (slot >> 4);
                const uint64_t x = kDescriptorHigh | ((slot + kWeightBytes) >> 4);
                const uint32_t sum = tmem + block % 4 * N;
                // 16 of k = 32 bytes = 2 in the descriptors' address field
#pragma unroll
                for (uint32_t at = 0; at < 8; at += 2) umma(sum, a + at, x + at, descriptor, at > 0 ? 1 : 0);
#pragma unroll
                for (uint32_t at = 0; at < 8; at += 2) {
                    umma(rest, a + at, x + kPart + at, descriptor, at > 0 ? 1 : accumulate);
                }
#pragma unroll
                for (uint32_t at = 0; at < 8; at += 2) umma(rest, a + at, x + 2 * kPart + at, descriptor, 1);
                umma_commit(bar_read + 8 * stage);
                accumulate = 1;
                slot += S::kStageBytes;
                if (++stage == S::kStages) {
                    stage = 0;
                    slot = ring;
                    parity ^= 1;
                }
            }
            store_shared(progress + offsetof(Progress, multiplied), block);
        }
        __syncwarp();
    } else if (warp < kFirstAdder) {
        // sixteen lanes per row of x, two rows per warp at a time
        const uint32_t row = (warp - kFirstConverter) * 2 + lane / 16;
        const uint32_t piece = lane % 16 * 4;
        const float* source = p.x + static_cast<size_t>(row0 + row) * p.k + piece;
        const uint32_t target = row * 128 + ((piece * 2) ^ (row % 8 * 16));    // 8 rows further the swizzle is the same
        // Two slots ahead: the loads of one take about as long as the conversion of another.
        float4 pending[2][S::kLoads];
        auto load = [&](uint32_t block, uint32_t i, float4& out) {
            const uint32_t depth = (block0 + block) * kBlockK;
            const uint32_t r = row + i * 2 * kConverters;
            out = block < blocks && row0 + r < p.m && depth + piece < p.k
                      ? *reinterpret_cast<const float4*>(source + static_cast<size_t>(i * 2 * kConverters) * p.k + depth)
                      : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        };
        pdl_wait();
#pragma unroll
        for (uint32_t i = 0; i < S::kLoads; ++i) load(0, i, pending[0][i]);
#pragma unroll
        for (uint32_t i = 0; i < S::kLoads; ++i) load(1, i, pending[1][i]);
        uint32_t stage = 0, parity = 1;                                    // the first pass over the ring finds it empty
        bool ok = true;
        auto convert = [&](uint32_t block, float4 (&held)[S::kLoads]) {
            if (block >= S::kStages && !mbar_wait_bounded(bar_read + 8 * stage, parity, p.wait_limit)) {
                give_up(3);
                ok = false;
                return;
            }
            uint8_t* slot = shared + stage * S::kStageBytes + kWeightBytes + target;
#pragma unroll
            for (uint32_t i = 0; i < S::kLoads; ++i) {
                const Taken taken = take_apart(held[i]);
                load(block + 2, i, held[i]);
#pragma unroll
                for (uint32_t part = 0; part < 3; ++part) {
                    *reinterpret_cast<uint2*>(slot + part * S::kPartBytes + i * 2 * kConverters * 128) = taken.part[part];
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bar_ready + 8 * stage);
                store_shared(progress + offsetof(Progress, converted) + 4 * (warp - kFirstConverter), block + 1);
            }
            if (++stage == S::kStages) {
                stage = 0;
                parity ^= 1;
            }
        };
        for (uint32_t block = 0; ok && block < blocks; block += 2) {
            convert(block, pending[0]);
            if (ok && block + 1 < blocks) convert(block + 1, pending[1]);
        }
    } else {
#pragma unroll
        for (uint32_t j = 0; j < N / 2; ++j) sums[j] = 0.0f;
        const uint32_t address = tmem + ((quadrant * 32) << 16) + half * (N / 2);
        bool ok = true;
        for (uint32_t pair = 0; pair * 2 < blocks; ++pair) {
            // MMAs are complete in the order of the blocks: the pair's last one speaks for both
            const bool both = pair * 2 + 1 < blocks;
            const uint32_t last = pair * 2 + (both ? 1 : 0);
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar_read + 8 * (last % S::kStages), last / S::kStages & 1, p.wait_limit));
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t source = address + (pair & 1) * 2 * N;
#pragma unroll
            for (uint32_t j = 0; j < N / 2; j += S::kPiece) {
                uint32_t raw[2][S::kPiece];
                load_columns(source + j, raw[0]);
                load_columns(source + N + j, raw[1]);
                tmem_load_wait();
                // without a second block the other short sum is an old one
#pragma unroll
                for (uint32_t i = 0; i < S::kPiece; ++i) {
                    sums[j + i] += __uint_as_float(raw[0][i]) + (both ? __uint_as_float(raw[1][i]) : 0.0f);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_taken + 8 * (pair & 1));
        }
        if (!ok && lane == 0) give_up(4);
        tcgen05_fence_after();
#pragma unroll
        for (uint32_t j = 0; j < N / 2; j += S::kPiece) {
            uint32_t raw[S::kPiece];
            load_columns(address + 4 * N + j, raw);
            tmem_load_wait();
#pragma unroll
            for (uint32_t i = 0; i < S::kPiece; ++i) {
                // a weight that is no finite number meets parts that are zero: the high part alone has the right answer
                const float rest = __uint_as_float(raw[i]);
                sums[j + i] += isfinite(rest) ? rest : 0.0f;
            }
        }
        tcgen05_fence_before();
    }
    // The successors are let in only now: a grid of several waves would otherwise share its SMs with CTAs that wait for it.
    pdl_launch_dependents();
    pdl_wait();                  // y may still be read by an earlier kernel
    __syncthreads();
    if (*abort_flag) drain<N>(control, p.wait_limit);
    if (warp == 1) {
        __syncwarp();
        tcgen05_fence_after();
        tmem_free(tmem, S::kColumns);
    }
    const bool adder = warp >= kFirstAdder;
    const uint32_t own_column = quadrant * 32 + lane, own_row = half * (N / 2);
    if (p.splits == 1) {
        if (adder && !*abort_flag && column0 + own_column < p.n) {
#pragma unroll
            for (uint32_t j = 0; j < N / 2; ++j) {
                const uint32_t row = row0 + own_row + j;
                if (row < p.m) p.y[static_cast<size_t>(row) * p.n + column0 + own_column] = sums[j];
            }
        }
        return;
    }
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    float* parked = reinterpret_cast<float*>(shared);                      // [row][128 columns], the ring is no longer used
    if (adder && !*abort_flag) {
#pragma unroll
        for (uint32_t j = 0; j < N / 2; ++j) parked[(own_row + j) * kTileM + own_column] = sums[j];
    }
    cluster.sync();
    bool whole = true;
    for (uint32_t rank = 0; rank < p.splits; ++rank) {
        whole = whole && *cluster.map_shared_rank(const_cast<uint32_t*>(abort_flag), rank) == 0;
    }
    // rank r finishes the rows r, r + splits, ..; a warp reads one row of each partner per pass
    for (uint32_t row = split + warp * p.splits; whole && row < N && row0 + row < p.m; row += kThreads / 32 * p.splits) {
        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t rank = 0; rank < p.splits; ++rank) {
            const float4 part = *reinterpret_cast<const float4*>(cluster.map_shared_rank(parked, rank) + row * kTileM + lane * 4);
            sum.x += part.x;
            sum.y += part.y;
            sum.z += part.z;
            sum.w += part.w;
        }
        const uint32_t column = column0 + lane * 4;
        float* target = p.y + static_cast<size_t>(row0 + row) * p.n + column;
        if (column < p.n) target[0] = sum.x;
        if (column + 1 < p.n) target[1] = sum.y;
        if (column + 2 < p.n) target[2] = sum.z;
        if (column + 3 < p.n) target[3] = sum.w;
    }
    cluster.sync();       // nobody leaves while its part is still being read
}

// Clusters of `size` CTAs that the device holds at once (0: none), asked once per kernel and size.
template <uint32_t N>
uint32_t resident_clusters(uint32_t size) {
    static std::atomic<int> known[9];
    int clusters = known[size].load(std::memory_order_relaxed);
    if (clusters == 0) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(size, 1, 1);
        config.blockDim = dim3(kThreads, 1, 1);
        config.dynamicSmemBytes = Shape<N>::kShared;
        cudaLaunchAttribute attribute;
        attribute.id = cudaLaunchAttributeClusterDimension;
        attribute.val.clusterDim.x = size;
        attribute.val.clusterDim.y = 1;
        attribute.val.clusterDim.z = 1;
        config.attrs = &attribute;
        config.numAttrs = 1;
        int count = 0;
        if (cudaOccupancyMaxActiveClusters(&count, linear_f32_umma_kernel<N>, &config) != cudaSuccess) {
            (void)cudaGetLastError();
            count = 0;
        }
        clusters = count + 1;
        known[size].store(clusters, std::memory_order_relaxed);
    }
    return static_cast<uint32_t>(clusters - 1);
}

template <uint32_t N>
cudaError_t allow_shared() {
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(linear_f32_umma_kernel<N>),
                                cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Shape<N>::kShared));
}

// Splits of k for tiles of N rows, and about how many cycles the product takes with them.
struct Choice {
    uint32_t splits;
    double cycles;
};
template <uint32_t N>
Choice choose(size_t m, size_t column_tiles, size_t k_blocks) {
    const size_t tiles = (m + N - 1) / N * column_tiles;
    Choice best = {1, 1e30};
    for (uint32_t splits = 1; splits <= 8 && (splits == 1 || k_blocks >= 2 * splits); ++splits) {
        const size_t resident = splits == 1 ? 148 * Shape<N>::kCtas : resident_clusters<N>(splits);
        if (resident == 0) continue;
        const size_t waves = (tiles + resident - 1) / resident;
        // Measured: a K block takes a CTA 100 + 16 N cycles (1000 and 1650 for N = 64 and 96; the MMAs alone 6 N to 12 N), 1.6
        // times as long where two share an SM, and 11000 pass before the first and behind the last.
        const double block = (100.0 + 16.0 * N) * (Shape<N>::kCtas > 1 && tiles * splits > 148 ? 1.6 : 1.0);
        const double cycles = static_cast<double>(waves) * (block * static_cast<double>((k_blocks + splits - 1) / splits) + 11000.0) +
                              (splits > 1 ? 2000.0 : 0.0);
        if (cycles < best.cycles) best = {splits, cycles};
    }
    return best;
}

template <uint32_t N>
cudaError_t launch(cudaStream_t stream, LinearParams params, const CUtensorMap& weight_map, const Choice& choice) {
    const uint32_t splits = choice.splits;
    const size_t ctas = (static_cast<size_t>(params.m) + N - 1) / N * params.column_tiles * splits;
    if (ctas == 0 || ctas > 0x7fffffffu) return cudaErrorInvalidValue;
    params.splits = splits;
    return launch_kernel(linear_f32_umma_kernel<N>, static_cast<unsigned int>(ctas), kThreads, Shape<N>::kShared, stream, splits,
                         weight_map, params);
}

}  // namespace

bool linear_f32_supports(const void* x, const void* weight, size_t m, size_t n, size_t k) {
    return k > 0 && k % 8 == 0 && aligned_to(x, 16) && aligned_to(weight, 16) && m <= 0x7fffffffu && n <= 0x7fffffffu &&
           k <= 0x7fffffffu;
}

cudaError_t launch_linear_f32(cudaStream_t stream, const void* x, const void* weight, void* y, size_t m, size_t n, size_t k) {
    if (m == 0 || n == 0) return cudaErrorInvalidValue;
    cudaError_t status = m <= 16 ? allow_shared<16>() : allow_shared<32>();
    if (status == cudaSuccess && m > 16) status = allow_shared<64>();
    if (status == cudaSuccess && m > 16) status = allow_shared<96>();
    if (status != cudaSuccess) return status;
    CUtensorMap weight_map;
    if (!make_swizzled_2d_map(&weight_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, weight, n, k * 2, kTileM)) {
        return cudaErrorInvalidValue;
    }
    LinearParams params;
    params.x = static_cast<const float*>(x);
    params.y = static_cast<float*>(y);
    params.status = device_status_words();
    params.wait_limit = wait_limit_ns();
    params.m = static_cast<uint32_t>(m);
    params.n = static_cast<uint32_t>(n);
    params.k = static_cast<uint32_t>(k);
    params.column_tiles = static_cast<uint32_t>((n + kTileM - 1) / kTileM);
    params.k_blocks = static_cast<uint32_t>((k + kBlockK - 1) / kBlockK);
    params.drop_block = wait_selftest_drop() ? 0u : 0xffffffffu;
    if (m <= 16) return launch<16>(stream, params, weight_map, choose<16>(m, params.column_tiles, params.k_blocks));
    // the tile height that is through first: few rows waste less of a low one, 250 rows of 48 column tiles fill the device
    // with three of 96
    const Choice low = choose<32>(m, params.column_tiles, params.k_blocks), middle = choose<64>(m, params.column_tiles, params.k_blocks),
                 high = choose<96>(m, params.column_tiles, params.k_blocks);
    if (low.cycles <= middle.cycles && low.cycles <= high.cycles) return launch<32>(stream, params, weight_map, low);
    if (middle.cycles <= high.cycles) return launch<64>(stream, params, weight_map, middle);
    return launch<96>(stream, params, weight_map, high);
}

}  // namespace lfm25

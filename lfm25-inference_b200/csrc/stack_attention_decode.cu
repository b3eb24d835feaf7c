// Decode attention of the layer stack for bf16 activations: one query token per sequence, any grouping of up to 16
// query heads per key/value head, query/key and value sizes up to 256, an optional chunk mask.
//
// One CTA per token, key/value head and split of the visible pages; its warps take pages in turn, each through a
// ring of its own that TMA fills (one box of 64 dimensions x 16 keys per copy, 128-byte swizzle).  A page is 16 keys of
// one head, the rows of S^T = K Q^T and the contracted index of O^T += V^T P^T, mma.sync tiles whose 8 columns are the query
// heads of the group (two tiles beyond 8): with the heads as rows a group of four left three quarters of them empty.  The
// weights turn from rows into columns by movmatrix and enter the second product as a sum of two bf16 values (16 significant
// bits); maximum, sum and accumulators are f32.  The warps merge through shared memory, the splits of a token through the
// distributed shared memory of their cluster.
//
// Bound by the latency of a page in a warp until the memory's rate is reached.  us with four warps and the heads as rows, with
// twelve warps two pages at a time and splits of eight pages, and now (eight warps, one page at a time, splits and shared memory
// chosen so that the CTAs spread over the SMs); launches back to back, caches beyond the L2:
//     32 tokens, 32 heads on 8 of 64: contexts of 128 to 4096     46.7 / 29.8 / 29.2      all 4096 (6.4 TB/s)  55.8 / 44.8 / 42.2
//     the same, all 1100    19.6 / 15.5 / 14.3                    24 tokens of 100 to 4000 on 2 of 128         21.2 / 18.3 / 18.6
//     groups of 16 heads of 64: 32 tokens of 4096 on 1    19.5 / 36.2 / 13.9     64 of 1024 on 4     20.6 / 24.7 / 16.6
//     8 tokens of 256 on 8 of 64    6.0 / 6.3 / 3.7               64 of 1024 on 8 of 64                        34.5 / 27.3 / 23.5
// Over 847 shapes and contexts, one to 192 tokens, 0.88 of the first and 0.86 of the second.  Equal long contexts in a few CTAs
// more than are resident are what is slower than in either (40 tokens of 4096 keys on 8 heads of 64 57.2 / 66.2 / 67.7).
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>
#include <atomic>

#include "launch.h"
#include "options.h"
#include "stack_attention.h"
#include "stack_common.cuh"

namespace lfm25 {

namespace {

namespace cg = cooperative_groups;

constexpr uint32_t kBoxBytes = kPageSize * 128;   // 16 keys x 64 dimensions
constexpr uint32_t kGroupRows = 16;
constexpr uint32_t kMostSplits = 8;
constexpr size_t kLongPages = 128;
// Of shared memory, so that no second CTA of the kernel is put on the SM while others are empty: 128 CTAs in clusters of 4 (32
// tokens of 4096 keys, 16 heads on 1 with values of 128) 18.6 us, 27.0 with what they need.
constexpr uint32_t kAloneBytes = 116 * 1024;

// WIDE: eight warps with short rings; otherwise four, so that more CTAs share an SM.  Of 14 combinations of 4 to 12 warps, 2 to 4
// stages and 1 or 2 pages at a time, (8, 2, 1) or its neighbours (8, 3, 1) and (8, 2, 2) were fastest wherever all CTAs are
// resident.
template <uint32_t KC, uint32_t VC, uint32_t TILES, bool WIDE>
struct Layout {
    static constexpr uint32_t kWarps = WIDE ? 8 : 4;
    static constexpr uint32_t kThreads = kWarps * 32;
    static constexpr uint32_t kStageBytes = (KC + VC) * kBoxBytes;
    static constexpr uint32_t kStages = !WIDE && (KC + VC == 3 || KC + VC == 4) ? 3 : 2;
    static constexpr uint32_t kPages = kStages == 3 ? 2 : 1;        // that a warp takes at a time
    // per SM that the registers must allow: beside small rings the compiler takes more than 128 where nothing is said
    static constexpr uint32_t kCtas = WIDE && KC + VC <= 3 ? 2 : 1;
    static constexpr uint32_t kRingBytes = kWarps * kStages * kStageBytes;
    static constexpr uint32_t kColumns = 64 * VC;
    // the warps' partial results reuse the ring once every page has been consumed
    static constexpr uint32_t kPartialPitch = kColumns + 4;          // rows 2 apart lie 8 banks apart
    static constexpr uint32_t kPartialBytes = kWarps * kGroupRows * kPartialPitch * 4;
    static constexpr uint32_t kBodyBytes = kRingBytes > kPartialBytes ? kRingBytes : kPartialBytes;
    // behind it: the CTA's result, maxima and sums per warp, maxima and sums per CTA, barriers, abort flag
    static constexpr uint32_t kResultBytes = kGroupRows * kColumns * 4;
    static constexpr uint32_t kSharedBytes = kBodyBytes + kResultBytes + (kWarps + 1) * kGroupRows * 8 +
                                             kWarps * kStages * 8 + 16 + 1024;
    static_assert(kSharedBytes <= 227 * 1024, "shared memory");
    static constexpr uint32_t shared_bytes(bool alone) {
        return alone && kSharedBytes < kAloneBytes ? kAloneBytes : kSharedBytes;
    }
};

struct Params {
    StackAttentionShape shape;
    const __nv_bfloat16* query;
    const uint32_t* block_tables;
    size_t block_table_stride;
    size_t block_table_rows;
    size_t num_pages;
    const uint32_t* request_slots;
    const uint32_t* positions;
    __nv_bfloat16* out;
    size_t out_pitch;
    unsigned int* status;
    uint32_t splits;
    uint64_t wait_limit;
};

// The 8 x 8 matrix of 16-bit values that a warp holds, row g of it in the lanes 4 g .. 4 g + 3, with rows and columns swapped.
__device__ __forceinline__ uint32_t transposed_8x8(uint32_t pair) {
    uint32_t out;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(out) : "r"(pair));
    return out;
}

template <uint32_t KC, uint32_t VC, uint32_t TILES, bool WIDE>
__global__ void __launch_bounds__(Layout<KC, VC, TILES, WIDE>::kThreads, Layout<KC, VC, TILES, WIDE>::kCtas)
stack_attention_decode_kernel(const __grid_constant__ CUtensorMap key_map, const __grid_constant__ CUtensorMap value_map,
                              const Params p) {
    using L = Layout<KC, VC, TILES, WIDE>;
    constexpr uint32_t kWarps = L::kWarps, kThreads = L::kThreads;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    extern __shared__ uint8_t decode_smem[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(decode_smem) + 1023) & ~uintptr_t(1023));
    float* partial = reinterpret_cast<float*>(smem);                                  // [warp][row][column]
    float* result = reinterpret_cast<float*>(smem + L::kBodyBytes);                   // [row][column]
    float* warp_top = result + kGroupRows * L::kColumns;                              // [warp][row]
    float* warp_sums = warp_top + kWarps * kGroupRows;
    float* cta_top = warp_sums + kWarps * kGroupRows;                                 // [row]
    float* cta_sum = cta_top + kGroupRows;
    uint8_t* barriers = reinterpret_cast<uint8_t*>(cta_sum + kGroupRows);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(barriers + kWarps * L::kStages * 8);
    const uint32_t ring = smem_u32(smem) + warp * L::kStages * L::kStageBytes;
    const uint32_t bar = smem_u32(barriers) + warp * L::kStages * 8;
    pdl_launch_dependents();
    if (threadIdx.x == 0) *abort_flag = 0;
    if (lane == 0) {
        tma_prefetch_descriptor(&key_map);
        tma_prefetch_descriptor(&value_map);
        for (uint32_t stage = 0; stage < L::kStages; ++stage) mbar_init(bar + 8 * stage, 1);
        fence_barrier_init();
    }
    __syncthreads();
    pdl_wait();

    const uint32_t split = blockIdx.x % p.splits;
    const uint32_t kv_head = blockIdx.x / p.splits % p.shape.kv_heads;
    const size_t token = blockIdx.x / p.splits / p.shape.kv_heads;
    const uint32_t group = p.shape.heads / p.shape.kv_heads;
    const size_t table_row = p.request_slots[token];
    const uint32_t position = p.positions[token];
    const uint32_t first = first_visible(position, p.shape.chunk);
    const bool valid = table_row < p.block_table_rows && position / kPageSize < p.block_table_stride;
    const uint32_t first_page = first / kPageSize;
    const uint32_t pages = valid ? position / kPageSize - first_page + 1 : 0;
    const uint32_t* table = p.block_tables + (valid ? table_row * p.block_table_stride : 0);
    // this warp's pages: first_page + mine, + stride, ...
    const uint32_t stride = kWarps * p.splits;
    const uint32_t mine = split * kWarps + warp;
    const uint32_t count = pages > mine ? (pages - mine + stride - 1) / stride : 0;

    // entry of this warp's page `index`; read 32 at a time
    uint32_t held = 0;
    uint32_t held_base = 0xffffffffu;
    auto entry_of = [&](uint32_t index) -> uint32_t {
        const uint32_t base = index & ~31u;
        if (base != held_base) {
            held_base = base;
            held = base + lane < count ? __ldg(table + first_page + mine + (base + lane) * stride) : 0xffffffffu;
        }
        return __shfl_sync(0xffffffffu, held, index & 31);
    };
    uint32_t usable = 0;        // bit per stage: the page in it exists
    auto issue = [&](uint32_t index) {
        const uint32_t stage = index % L::kStages;
        const uint32_t entry = entry_of(index);
        const bool exists = entry < p.num_pages;
        usable = exists ? usable | (1u << stage) : usable & ~(1u << stage);
        if (lane == 0) {
            // a page that does not exist is read as page 0 and not used
            const int32_t row = static_cast<int32_t>(((exists ? entry : 0) * p.shape.kv_heads + kv_head) * kPageSize);
            const uint32_t target = ring + stage * L::kStageBytes;
            mbar_arrive_expect_tx(bar + 8 * stage, L::kStageBytes);
#pragma unroll
            for (uint32_t chunk = 0; chunk < KC; ++chunk) {
                tma_load_2d(target + chunk * kBoxBytes, &key_map, bar + 8 * stage, static_cast<int32_t>(chunk * 64), row);
            }
#pragma unroll
            for (uint32_t chunk = 0; chunk < VC; ++chunk) {
                tma_load_2d(target + (KC + chunk) * kBoxBytes, &value_map, bar + 8 * stage,
                            static_cast<int32_t>(chunk * 64), row);
            }
        }
    };
    uint32_t issued = 0;
    for (; issued < L::kStages && issued < count; ++issued) issue(issued);

    // query fragments: column = head of the group, times nothing (the scale is applied to the f32 scores)
    const uint32_t g = lane >> 2;
    const uint32_t pair = (lane & 3) * 2;
    uint32_t query[KC * 4][TILES][2];
    const __nv_bfloat16* query_rows = p.query + (token * p.shape.heads + static_cast<size_t>(kv_head) * group) * p.shape.dim;
#pragma unroll
    for (uint32_t ks = 0; ks < KC * 4; ++ks) {
#pragma unroll
        for (uint32_t tile = 0; tile < TILES; ++tile) {
#pragma unroll
            for (uint32_t part = 0; part < 2; ++part) {
                const uint32_t head = tile * 8 + g;
                const uint32_t dim = ks * 16 + pair + part * 8;
                query[ks][tile][part] = head < group && dim < p.shape.dim
                                            ? *reinterpret_cast<const uint32_t*>(query_rows + head * p.shape.dim + dim)
                                            : 0u;
            }
        }
    }

    // [16 value dimensions][8 heads]: dimensions g and g + 8, heads 2 (lane % 4) and the next
    float out[VC * 4][TILES][4];
#pragma unroll
    for (uint32_t m = 0; m < VC * 4; ++m) {
#pragma unroll
        for (uint32_t tile = 0; tile < TILES; ++tile) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) out[m][tile][i] = 0.0f;
        }
    }
    float top[TILES][2], sum[TILES][2];              // of the lane's two heads; a sum covers its own keys
#pragma unroll
    for (uint32_t tile = 0; tile < TILES; ++tile) {
        top[tile][0] = top[tile][1] = -INFINITY;
        sum[tile][0] = sum[tile][1] = 0.0f;
    }
    const float scale_log2 = p.shape.scale * kLog2e;
    bool ok = true;
    uint32_t waited = 0;
    for (uint32_t index = 0; index < count; index += L::kPages) {
        // keys g and g + 8 of a page, the lane's two heads
        float scores[L::kPages][TILES][4];
        bool there[L::kPages];
#pragma unroll
        for (uint32_t j = 0; j < L::kPages; ++j) {
            const uint32_t stage = (index + j) % L::kStages;
            there[j] = index + j < count;
            if (there[j]) {
                ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(bar + 8 * stage, ((index + j) / L::kStages) & 1, p.wait_limit));
                if (!ok) break;
                waited = index + j + 1;
                there[j] = usable >> stage & 1u;
            }
#pragma unroll
            for (uint32_t tile = 0; tile < TILES; ++tile) {
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) scores[j][tile][i] = there[j] ? 0.0f : -INFINITY;
            }
            if (!there[j]) continue;
            const uint32_t key_base = ring + stage * L::kStageBytes;
            const uint32_t value_base = key_base + KC * kBoxBytes;
            const uint32_t page_first = (first_page + mine + (index + j) * stride) * kPageSize;
#pragma unroll
            for (uint32_t ks = 0; ks < KC * 4; ++ks) {
                const uint32_t key = lane & 15;
                const uint32_t part = (ks & 3) * 2 + (lane >> 4);
                uint32_t a0, a1, a2, a3;
                ldmatrix_x4(key_base + (ks >> 2) * kBoxBytes + key * 128 + ((part ^ (key & 7)) << 4), a0, a1, a2, a3);
#pragma unroll
                for (uint32_t tile = 0; tile < TILES; ++tile) {
                    mma_bf16_16816(scores[j][tile], a0, a1, a2, a3, query[ks][tile][0], query[ks][tile][1]);
                }
            }
            const bool whole = page_first >= first && page_first + kPageSize - 1 <= position;
            if (!whole) {
                if (page_first + kPageSize - 1 > position) {
                    // value rows behind the last key may hold anything, and zero times a NaN pattern is NaN
                    for (uint32_t item = lane; item < VC * kPageSize * 8; item += 32) {
                        const uint32_t key = item / 8 % kPageSize;
                        if (page_first + key > position) {
                            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(
                                             value_base + item / (kPageSize * 8) * kBoxBytes + key * 128 + item % 8 * 16),
                                         "r"(0u)
                                         : "memory");
                        }
                    }
                    __syncwarp();
                }
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const uint32_t key = page_first + g + (i >> 1) * 8;
                    if (key < first || key > position) {
#pragma unroll
                        for (uint32_t tile = 0; tile < TILES; ++tile) scores[j][tile][i] = -INFINITY;
                    }
                }
            }
        }
        if (!ok) break;
        float rescale[TILES][2];
        uint32_t high[L::kPages][TILES][2], low[L::kPages][TILES][2];        // [8 keys], turned into columns
        bool same = true;
#pragma unroll
        for (uint32_t tile = 0; tile < TILES; ++tile) {
            float best[2];
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                best[h] = fmaxf(scores[0][tile][h], scores[0][tile][2 + h]);
#pragma unroll
                for (uint32_t j = 1; j < L::kPages; ++j) best[h] = max3(best[h], scores[j][tile][h], scores[j][tile][2 + h]);
            }
#pragma unroll
            for (uint32_t delta = 4; delta < 32; delta <<= 1) {
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) best[h] = fmaxf(best[h], __shfl_xor_sync(0xffffffffu, best[h], delta));
            }
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const float now = fmaxf(top[tile][h], best[h]);
                const float base = now == -INFINITY ? 0.0f : now;
                rescale[tile][h] = fast_exp2((top[tile][h] - base) * scale_log2);
                const float offset = -base * scale_log2;
                float total = 0.0f;
#pragma unroll
                for (uint32_t j = 0; j < L::kPages; ++j) {
                    scores[j][tile][h] = fast_exp2(fmaf(scores[j][tile][h], scale_log2, offset));
                    scores[j][tile][2 + h] = fast_exp2(fmaf(scores[j][tile][2 + h], scale_log2, offset));
                    total += scores[j][tile][h] + scores[j][tile][2 + h];
                }
                sum[tile][h] = fmaf(sum[tile][h], rescale[tile][h], total);
                top[tile][h] = now;
                same = same && rescale[tile][h] == 1.0f;
            }
#pragma unroll
            for (uint32_t j = 0; j < L::kPages; ++j) {
#pragma unroll
                for (uint32_t part = 0; part < 2; ++part) {
                    const float a = scores[j][tile][2 * part], b = scores[j][tile][2 * part + 1];
                    const uint32_t both = pack_bf16x2(a, b);
                    const float2 rounded = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&both));
                    high[j][tile][part] = transposed_8x8(both);
                    low[j][tile][part] = transposed_8x8(pack_bf16x2(a - rounded.x, b - rounded.y));
                }
            }
        }
        if (!__all_sync(0xffffffffu, same)) {
#pragma unroll
            for (uint32_t m = 0; m < VC * 4; ++m) {
#pragma unroll
                for (uint32_t tile = 0; tile < TILES; ++tile) {
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) out[m][tile][i] *= rescale[tile][i & 1];
                }
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < L::kPages; ++j) {
            if (!there[j]) continue;
            const uint32_t value_base = ring + (index + j) % L::kStages * L::kStageBytes + KC * kBoxBytes;
#pragma unroll
            for (uint32_t m = 0; m < VC * 4; ++m) {     // 16 value dimensions at a time
                const uint32_t key = (lane >> 4) * 8 + (lane & 7);
                const uint32_t part = (m & 3) * 2 + (lane >> 3 & 1);
                uint32_t a0, a1, a2, a3;
                ldmatrix_x4_trans(value_base + (m >> 2) * kBoxBytes + key * 128 + ((part ^ (key & 7)) << 4), a0, a1, a2, a3);
#pragma unroll
                for (uint32_t tile = 0; tile < TILES; ++tile) {
                    mma_bf16_16816(out[m][tile], a0, a1, a2, a3, high[j][tile][0], high[j][tile][1]);
                    mma_bf16_16816(out[m][tile], a0, a1, a2, a3, low[j][tile][0], low[j][tile][1]);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (uint32_t j = 0; j < L::kPages; ++j) {
            if (issued < count) {
                issue(issued);
                ++issued;
            }
        }
    }
    if (!ok) {
        if (lane == 0) {
            *abort_flag = 1;
            record_wait_timeout(p.status, kTagStackDecode, blockIdx.x);
        }
        for (uint32_t index = waited; index < issued; ++index) {      // copies still in flight, each for a bounded time
            mbar_wait_bounded(bar + 8 * (index % L::kStages), (index / L::kStages) & 1, p.wait_limit);
        }
    }

    // ---- warps of the CTA
#pragma unroll
    for (uint32_t tile = 0; tile < TILES; ++tile) {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
#pragma unroll
            for (uint32_t delta = 4; delta < 32; delta <<= 1) {
                sum[tile][h] += __shfl_xor_sync(0xffffffffu, sum[tile][h], delta);
            }
        }
    }
    __syncthreads();          // every ring is drained
#pragma unroll
    for (uint32_t tile = 0; tile < TILES; ++tile) {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t row = tile * 8 + pair + h;
            if (row < group) {
                if (g == 0) {
                    warp_top[warp * kGroupRows + row] = top[tile][h];
                    warp_sums[warp * kGroupRows + row] = sum[tile][h];
                }
                float* target = partial + (warp * kGroupRows + row) * L::kPartialPitch + g;
#pragma unroll
                for (uint32_t m = 0; m < VC * 4; ++m) {
                    target[m * 16] = out[m][tile][h];
                    target[m * 16 + 8] = out[m][tile][2 + h];
                }
            }
        }
    }
    __syncthreads();
    const uint32_t vdim = p.shape.vdim;
    __nv_bfloat16* target = p.out + token * p.out_pitch + static_cast<size_t>(kv_head) * group * vdim;
    const bool aborted = *abort_flag != 0;
    for (uint32_t item = threadIdx.x; item < group * vdim; item += kThreads) {
        const uint32_t row = item / vdim;
        const uint32_t column = item - row * vdim;
        float best = -INFINITY;
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w) best = fmaxf(best, warp_top[w * kGroupRows + row]);
        const float base = best == -INFINITY ? 0.0f : best;
        float total = 0.0f, value = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w) {
            const float factor = fast_exp2((warp_top[w * kGroupRows + row] - base) * scale_log2);
            total = fmaf(warp_sums[w * kGroupRows + row], factor, total);
            value = fmaf(partial[(w * kGroupRows + row) * L::kPartialPitch + column], factor, value);
        }
        if (p.splits == 1) {
            if (!aborted) target[item] = __float2bfloat16_rn(total > 0.0f ? value / total : 0.0f);
        } else {
            result[row * L::kColumns + column] = value;
            if (column == 0) {
                cta_top[row] = best;
                cta_sum[row] = total;
            }
        }
    }
    if (p.splits == 1) {
        return;
    }
    // ---- splits of the token: every CTA of the cluster finishes a share of the outputs
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    bool any_abort = false;
    for (uint32_t rank = 0; rank < p.splits; ++rank) {
        any_abort = any_abort || *cluster.map_shared_rank(const_cast<uint32_t*>(abort_flag), rank) != 0;
    }
    for (uint32_t item = threadIdx.x * p.splits + split; item < group * vdim; item += kThreads * p.splits) {
        const uint32_t row = item / vdim;
        const uint32_t column = item - row * vdim;
        float best = -INFINITY;
        for (uint32_t rank = 0; rank < p.splits; ++rank) {
            best = fmaxf(best, cluster.map_shared_rank(cta_top, rank)[row]);
        }
        const float base = best == -INFINITY ? 0.0f : best;
        float total = 0.0f, value = 0.0f;
        for (uint32_t rank = 0; rank < p.splits; ++rank) {
            const float factor = fast_exp2((cluster.map_shared_rank(cta_top, rank)[row] - base) * scale_log2);
            total = fmaf(cluster.map_shared_rank(cta_sum, rank)[row], factor, total);
            value = fmaf(cluster.map_shared_rank(result, rank)[row * L::kColumns + column], factor, value);
        }
        if (!any_abort) target[item] = __float2bfloat16_rn(total > 0.0f ? value / total : 0.0f);
    }
    cluster.sync();           // nobody leaves while its results are being read
}

// Clusters of `size` CTAs of the wide form that the device holds at once, asked once per kernel, size and spread.
template <uint32_t KC, uint32_t VC, uint32_t TILES>
size_t resident_clusters(uint32_t size, bool alone) {
    using L = Layout<KC, VC, TILES, true>;
    static std::atomic<int> answers[2][kMostSplits + 1];
    std::atomic<int>& known = answers[alone ? 1 : 0][size];
    int clusters = known.load(std::memory_order_relaxed);
    if (clusters == 0) {
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(size, 1, 1);
        config.blockDim = dim3(L::kThreads, 1, 1);
        config.dynamicSmemBytes = L::shared_bytes(alone);
        cudaLaunchAttribute attribute;
        attribute.id = cudaLaunchAttributeClusterDimension;
        attribute.val.clusterDim.x = size;
        attribute.val.clusterDim.y = 1;
        attribute.val.clusterDim.z = 1;
        config.attrs = &attribute;
        config.numAttrs = 1;
        int count = 0;
        if (cudaOccupancyMaxActiveClusters(&count, stack_attention_decode_kernel<KC, VC, TILES, true>, &config) != cudaSuccess) {
            (void)cudaGetLastError();
            count = 0;
        }
        clusters = count + 1;
        known.store(clusters, std::memory_order_relaxed);
    }
    return static_cast<size_t>(clusters - 1);
}

template <uint32_t KC, uint32_t VC, uint32_t TILES, bool WIDE>
cudaError_t allow_shared() {
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(stack_attention_decode_kernel<KC, VC, TILES, WIDE>),
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(Layout<KC, VC, TILES, WIDE>::shared_bytes(true)));
}

template <uint32_t KC, uint32_t VC, uint32_t TILES, bool WIDE>
cudaError_t launch_form(cudaStream_t stream, const StackAttentionLaunch& launch, uint32_t splits, bool alone) {
    using L = Layout<KC, VC, TILES, WIDE>;
    CUtensorMap key_map, value_map;
    if (!make_page_map(&key_map, launch, false) || !make_page_map(&value_map, launch, true)) {
        return cudaErrorInvalidValue;
    }
    Params params;
    params.shape = launch.shape;
    params.query = static_cast<const __nv_bfloat16*>(launch.query);
    params.block_tables = launch.block_tables;
    params.block_table_stride = launch.block_table_stride;
    params.block_table_rows = launch.block_table_rows;
    params.num_pages = launch.num_pages;
    params.request_slots = launch.request_slots;
    params.positions = launch.positions;
    params.out = static_cast<__nv_bfloat16*>(launch.out);
    params.out_pitch = launch.out_pitch;
    params.status = launch.status;
    params.splits = splits;
    params.wait_limit = wait_limit_ns();
    const size_t blocks = launch.decode_tokens * launch.shape.kv_heads * splits;
    return launch_kernel(stack_attention_decode_kernel<KC, VC, TILES, WIDE>, static_cast<unsigned int>(blocks), L::kThreads,
                         L::shared_bytes(alone), stream, splits, key_map, value_map, params);
}

template <uint32_t KC, uint32_t VC, uint32_t TILES>
cudaError_t launch_tiles(cudaStream_t stream, const StackAttentionLaunch& launch) {
    cudaError_t status = allow_shared<KC, VC, TILES, true>();
    if (status == cudaSuccess) status = allow_shared<KC, VC, TILES, false>();
    if (status != cudaSuccess) return status;
    const size_t clusters = launch.decode_tokens * launch.shape.kv_heads;
    const size_t visible = launch.shape.chunk != 0 ? std::min<size_t>(launch.decode_context, launch.shape.chunk)
                                                   : launch.decode_context;
    const size_t pages = (visible + kPageSize - 1) / kPageSize;
    constexpr size_t kWarps = Layout<KC, VC, TILES, true>::kWarps;
    // Measured, in rounds of a page per warp (0.6 to 0.75 us; 1024 keys of one token and head 8 rounds, 10.4 us in one CTA and 9.4,
    // 8.0, 8.2 in 2, 4, 8; 4096 keys 28.5 and 18.7, 12.7, 10.6): a cluster's merge costs 2.9 (2 or 4 CTAs) or 4.5 of them (8), a
    // round half as much again where two CTAs share an SM and a group is one tile of columns, twice as much where it is two.
    uint32_t splits = 0;
    bool alone = false;
    double best = 0.0;
    for (uint32_t size = 1; size <= kMostSplits; size *= 2) {
        const double merge = size == 1 ? 0.0 : (size < 8 ? 2.9 : 4.5);
        if (splits > 0 && best <= merge + 1.0) break;
        const bool spread = clusters <= resident_clusters<KC, VC, TILES>(size, true);
        const bool shares = !spread && (size == 1 || clusters * size <= 2 * 148) &&
                            clusters <= resident_clusters<KC, VC, TILES>(size, false);
        if (!spread && !shares) continue;
        const double rounds = static_cast<double>((pages + kWarps * size - 1) / (kWarps * size));
        const double cost = rounds * (spread ? 1.0 : (TILES == 1 ? 1.5 : 2.0)) + merge * (spread || TILES == 1 ? 1.0 : 2.0);
        if (splits == 0 || cost < best) {
            splits = size;
            alone = spread;
            best = cost;
        }
    }
    // More CTAs than are resident: eight warps where contexts may be long, since of unequal ones the longest decides (80 tokens of
    // 128 to 4096 keys, 8 heads of 64 59.5 us, with four warps 64.4; 96 of 4096 118 and 137), or where rings of three boxes leave
    // room for two such CTAs anyway (keys of 128, values of 64: 128 tokens of 1024 keys 63 and 71; not with two tiles of columns);
    // four for the others (64 of 256 keys 8.5, with eight 11.3).  All resident: four only where each has at most one page and no
    // two CTAs share an SM.
    const bool wide = splits == 0 ? (KC + VC == 3 && TILES == 1) || pages >= kLongPages
                                  : pages > kWarps / 2 || clusters > 148;
    if (wide) return launch_form<KC, VC, TILES, true>(stream, launch, std::max(splits, 1u), alone);
    return launch_form<KC, VC, TILES, false>(stream, launch, 1, clusters <= 148);
}

template <uint32_t KC, uint32_t VC>
cudaError_t launch_sized(cudaStream_t stream, const StackAttentionLaunch& launch) {
    return launch.shape.heads / launch.shape.kv_heads <= 8 ? launch_tiles<KC, VC, 1>(stream, launch)
                                                           : launch_tiles<KC, VC, 2>(stream, launch);
}

template <uint32_t KC>
cudaError_t launch_keys(cudaStream_t stream, const StackAttentionLaunch& launch) {
    switch ((launch.shape.vdim + 63) / 64) {
        case 1: return launch_sized<KC, 1>(stream, launch);
        case 2: return launch_sized<KC, 2>(stream, launch);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

bool stack_attention_decode_supports(const StackAttentionLaunch& launch) {
    const StackAttentionShape& shape = launch.shape;
    return paged_copies_possible(launch) && shape.dim <= 256 && shape.vdim <= 128 &&
           shape.heads / shape.kv_heads <= kGroupRows;
}

cudaError_t launch_stack_attention_decode(cudaStream_t stream, const StackAttentionLaunch& launch) {
    switch ((launch.shape.dim + 63) / 64) {
        case 1: return launch_keys<1>(stream, launch);
        case 2: return launch_keys<2>(stream, launch);
        case 3: return launch_keys<3>(stream, launch);
        case 4: return launch_keys<4>(stream, launch);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace lfm25

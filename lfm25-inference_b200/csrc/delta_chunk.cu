// The generalised delta rule over bf16 prompts with heads up to 64, a segment's head per CTA.
//
// The recurrence over a tile of 16 tokens as matrix products.  With P_t the product of the decays of the tile's tokens
// up to t, S_t = diag(P_t) Q_t, and
//     U_t = u_t P_(t-1),   R_t = r_t P_t,   K_t = k_t / P_t,   B_t = -(a_t u_t) / P_t          (per key channel)
// the update is Q_t = Q_(t-1) + B_t (U_t^T Q_(t-1)) + K_t v_t^T, so with Y_t = Q_(t-1)^T U_t
//     (I - tril(U B^T, -1)) Y = U Q_0 + tril(U K^T, -1) V
//     O = R Q_0 + tril(R B^T) Y + tril(R K^T) V,      Q_16 = Q_0 + B^T Y + K^T V.
// A decay is at least exp(-exp(-1/2)), so 1 / P_t stays below 17000 and every product keeps its relative accuracy.
// The products run on the tensor cores in TF32 with both operands split into two parts (three products), which
// leaves errors of the size of f32 rounding; v is bf16 and needs no second part.
//
// A CTA owns one head of one segment and works as a pipeline over tiles, one barrier per step; in step i
//     copies       load tile i + 4, tanh(z) and |k| of tile i + 3
//     elements     decay logits (a small product), prefix sums over the tokens, U, R, K, B of tile i + 2, and each warp's
//                  share (8 key channels) of the four 16 x 16 products among them
//     triangles    the sums of those shares, masked, and the inverse of the unit triangle of tile i + 1; norm, gate and output of
//                  tile i - 1
//     matrices     everything that meets the state, for tile i; a warp owns 16 value columns and their state
//
// What bounds it: the instructions of the four groups (a step takes each of them about 4000 cycles, the tensor pipe 2240 of
// them), so no operand passes through shared memory in another form than the one its reader's MMA takes:
//   * the matrices' products are transposed (value columns are the rows of the MMA), and the contracted index of a fragment is
//     numbered so that places j and j + 4 hold neighbours 2 j and 2 j + 1.  An accumulator is then the A operand of the next
//     product as it stands: the state, the right-hand side and Y never leave their registers.
//   * U, R, K, B and the triangles lie in shared memory as B fragments, already in two parts: 16 bytes per lane, one load (K and B
//     for ranks up to 64, beyond which there is no room).
//   * the elements' own layout (tokens x channels) is that of A and B fragments too, so the triangles' products start from
//     registers.
// The elements take eight warps, the others four each; the matrices' warps get the registers that copies and triangles leave
// (in 96 they spill: 5136 instead of 3900 cycles a step and all others wait).  One head of one segment, 4096 tokens: 770 us
// with operands in plain rows and four equal groups, 663 us now; 7 segments of 300 to 700 tokens, 32 heads: 274 us in the order
// of the step, 245 us with the longest segments first, 180 us with both.
#include <type_traits>

#include "delta_rule.h"
#include "launch.h"

namespace lfm25 {

namespace {

constexpr uint32_t kTokens = 16;                  // per tile
constexpr uint32_t kDim = kDeltaChunkDim;         // padded head size
constexpr uint32_t kEarlyStages = 3;              // r, k, a, z of tiles i + 2 .. i + 4
constexpr uint32_t kLateStages = 6;               // v, g of tiles i - 1 .. i + 4
constexpr uint32_t kLateRow = 2 * kDim + 8;       // bf16; rows four banks apart
constexpr uint32_t kProducedStride = kDim + 4;
constexpr uint32_t kLowerStride = 20;
constexpr uint32_t kFragments = 16;               // of a 16 x 64 operand: 8 x 8 pieces
constexpr uint32_t kTriangleFragments = 4;
constexpr uint32_t kElementWarps = 8;             // 8 channels each
constexpr uint32_t kThreads = 32 * (12 + kElementWarps);

template <bool SPLIT>
struct Layout {
    uint32_t rank_pad = 0, z_stride = 0, early_row = 0;
    size_t early = 0, late = 0, rows = 0, columns = 0, partials = 0, triangles = 0, lower = 0, decay_end = 0, tanh_parts = 0,
           w2 = 0, constants = 0, scale = 0, produced = 0, total = 0;
    __host__ __device__ constexpr explicit Layout(uint32_t rank) {
        rank_pad = (rank + 31) / 32 * 32;
        z_stride = rank_pad + 8;
        early_row = 3 * kDim + rank_pad + 8;
        size_t at = 0;
        early = at;                               // [stage][token][r | k | a | z] bf16
        at += kEarlyStages * kTokens * early_row * 2;
        late = at;                                // [stage][token][v | g] bf16
        at += kLateStages * kTokens * kLateRow * 2;
        rows = at;                                // [3][U | R][fragment][lane] float4
        at += 3 * 2 * kFragments * 32 * 16;
        columns = at;                             // [3][K | B][fragment][lane] float4, or float2 (SPLIT: in two parts)
        at += 3 * 2 * kFragments * 32 * (SPLIT ? 16 : 8);
        partials = at;                            // [warp][U B^T | U K^T | R B^T | R K^T][2][lane] float4
        at += kElementWarps * 4 * 2 * 32 * 16;
        triangles = at;                           // [2][inverse | U K^T | R B^T | R K^T][fragment][lane] float4
        at += 2 * 4 * kTriangleFragments * 32 * 16;
        lower = at;                               // U B^T, plain
        at += kTokens * kLowerStride * 4;
        decay_end = at;                           // [3][channel]: P of the tile's last token
        at += 3 * kDim * 4;
        tanh_parts = at;                          // [2][high | low][token][z_stride]
        at += 2 * 2 * kTokens * z_stride * 2;
        w2 = at;
        at += kDim * z_stride * 2;
        constants = at;                           // w0, removal bias, norm weight
        at += 3 * kDim * 4;
        scale = at;                               // [2][token]: 1 / |k|
        at += 2 * kTokens * 4;
        produced = at;                            // [2][token][kProducedStride]
        at += 2 * kTokens * kProducedStride * 4;
        total = at;
    }
};

// Two values as what a lane holds of a B fragment: their high parts, then their low ones.
__device__ __forceinline__ float4 in_parts(float first, float second) {
    FragmentB<> parts;
    parts.set(0, first);
    parts.set(1, second);
    return make_float4(parts.high[0], parts.high[1], parts.low[0], parts.low[1]);
}
__device__ __forceinline__ FragmentB<> fragment_of(const float4& parts) {
    FragmentB<> out;
    out.high[0] = parts.x;
    out.high[1] = parts.y;
    out.low[0] = parts.z;
    out.low[1] = parts.w;
    return out;
}
__device__ __forceinline__ FragmentB<> fragment_of(const float2& values) {
    FragmentB<> out;
    out.set(0, values.x);
    out.set(1, values.y);
    return out;
}
// An accumulator as the A operand of the next product.
__device__ __forceinline__ FragmentA<> fragment_of(const float (&c)[4]) {
    FragmentA<> out;
    out.set(0, c[0]);
    out.set(1, c[2]);
    out.set(2, c[1]);
    out.set(3, c[3]);
    return out;
}
// A is exact in TF32
__device__ __forceinline__ void mma_exact(float (&d)[4], const float (&a)[4], const FragmentB<>& b) {
    mma_tf32(d, a, b.low);
    mma_tf32(d, a, b.high);
}

__device__ __forceinline__ void barrier_sync(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void barrier_arrive(uint32_t id, uint32_t threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Registers per thread: the compiler gives all 96 (640 threads at one CTA per SM), the matrices' warps take over what the copies
// and the triangles do without.
constexpr uint32_t kMatrixRegisters = 144, kOtherRegisters = 72;
static_assert(kMatrixRegisters + 2 * kOtherRegisters + kElementWarps / 4 * 96 <= kThreads / 128 * 96, "more than the CTA has");
template <uint32_t COUNT>
__device__ __forceinline__ void set_more_registers() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(COUNT));
}
template <uint32_t COUNT>
__device__ __forceinline__ void set_fewer_registers() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(COUNT));
}

constexpr uint32_t kCopiesBarrier = 1;            // the copying warps among themselves
constexpr uint32_t kStepBarrier = 3;
constexpr uint32_t kPartialsBarrier = 2;          // the shares of the triangles have been read, the next ones may come

// CTAs start in the order of their numbers, so the longest segments come first: in the order of the step the last wave of
// CTAs may hold the longest ones (7 segments of 300 to 700 tokens on 148 SMs: 72 tiles in a row instead of 52).  With more
// segments than these the tail is short beside the rest.
constexpr uint32_t kSortedSegments = 64;

__device__ __forceinline__ uint32_t segment_length(const StackSegments& segments, uint32_t segment) {
    const uint32_t begin = segments.offsets[segment];
    const uint32_t end = min(segments.offsets[segment + 1], static_cast<uint32_t>(segments.num_tokens));
    return end > begin ? end - begin : 0;
}

template <bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
delta_chunk_kernel(const DeltaArgs<__nv_bfloat16> args) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) unsigned char chunk_shared[];
    __shared__ uint32_t segment_of_rank;
    const Layout<SPLIT> layout(args.rank);
    const uint32_t dim = args.dim;
    const uint32_t head = blockIdx.x % args.heads;
    uint32_t segment = blockIdx.x / args.heads;
    if (args.segments.num_segments > 1 && args.segments.num_segments <= kSortedSegments) {
        const uint32_t count = static_cast<uint32_t>(args.segments.num_segments);
        if (threadIdx.x < count) {
            const uint32_t mine = segment_length(args.segments, threadIdx.x);
            uint32_t rank = 0;
            for (uint32_t other = 0; other < count; ++other) {
                const uint32_t length = segment_length(args.segments, other);
                rank += length > mine || (length == mine && other < threadIdx.x) ? 1 : 0;
            }
            if (rank == segment) segment_of_rank = threadIdx.x;
        }
        __syncthreads();
        segment = segment_of_rank;
    }
    const uint32_t begin = args.segments.offsets[segment];
    uint32_t end = args.segments.offsets[segment + 1];
    end = end < args.segments.num_tokens ? end : static_cast<uint32_t>(args.segments.num_tokens);
    const size_t slot = args.segments.slots[segment];
    if (begin >= end || slot >= args.segments.num_request_slots) {
        return;
    }
    const int tiles = static_cast<int>((end - begin + kTokens - 1) / kTokens);
    const size_t width = static_cast<size_t>(args.heads) * dim;
    const size_t head_base = static_cast<size_t>(head) * dim;
    auto* tanh_parts = reinterpret_cast<__nv_bfloat16*>(chunk_shared + layout.tanh_parts);
    auto* w2 = reinterpret_cast<__nv_bfloat16*>(chunk_shared + layout.w2);
    auto* constants = reinterpret_cast<float*>(chunk_shared + layout.constants);
    auto* lower = reinterpret_cast<float*>(chunk_shared + layout.lower);
    auto* partials = reinterpret_cast<float4*>(chunk_shared + layout.partials);
    float* state_base = reinterpret_cast<float*>(static_cast<unsigned char*>(args.record.base) +
                                                 slot * args.record.stride + args.record.offset) +
                        head_base * dim;
    // tile + 6 keeps the numbers of the tiles in front of the first one positive
    auto early_of = [&](int tile) {
        return reinterpret_cast<__nv_bfloat16*>(chunk_shared + layout.early) +
               static_cast<uint32_t>(tile + 6) % kEarlyStages * kTokens * layout.early_row;
    };
    auto late_of = [&](int tile) {
        return reinterpret_cast<__nv_bfloat16*>(chunk_shared + layout.late) +
               static_cast<uint32_t>(tile + 6) % kLateStages * kTokens * kLateRow;
    };
    auto unit_of = [&](int tile) { return reinterpret_cast<float*>(chunk_shared + layout.scale) + tile % 2 * kTokens; };
    auto tanh_of = [&](int tile) { return tanh_parts + tile % 2 * 2 * kTokens * layout.z_stride; };
    auto rows_of = [&](int tile) {
        return reinterpret_cast<float4*>(chunk_shared + layout.rows) + tile % 3 * 2 * kFragments * 32;
    };
    using Column = std::conditional_t<SPLIT, float4, float2>;
    auto columns_of = [&](int tile) {
        return reinterpret_cast<Column*>(chunk_shared + layout.columns) + tile % 3 * 2 * kFragments * 32;
    };
    auto decay_end_of = [&](int tile) { return reinterpret_cast<float*>(chunk_shared + layout.decay_end) + tile % 3 * kDim; };
    constexpr uint32_t kTriangle = kTriangleFragments * 32;
    auto triangles_of = [&](int tile) {
        return reinterpret_cast<float4*>(chunk_shared + layout.triangles) + tile % 2 * 4 * kTriangle;
    };
    auto produced_of = [&](int tile) {
        return reinterpret_cast<float*>(chunk_shared + layout.produced) + tile % 2 * kTokens * kProducedStride;
    };

    // padding channels and tokens that never arrive stay zero
    for (uint32_t item = threadIdx.x; item < (layout.rows - layout.early) / 16; item += kThreads) {
        reinterpret_cast<uint4*>(chunk_shared + layout.early)[item] = make_uint4(0, 0, 0, 0);
    }
    {
        // eight threads per channel
        const uint32_t channel = threadIdx.x / 8;
        const __nv_bfloat16* source = args.decay_up + (head_base + channel) * args.rank;
        const bool vector_rank = args.rank % 8 == 0;
        for (uint32_t z = threadIdx.x % 8 * 8; channel < kDim && z < layout.z_stride; z += 64) {
            uint4 value = make_uint4(0, 0, 0, 0);
            if (channel < dim && z < args.rank) {
                if (vector_rank) {
                    value = *reinterpret_cast<const uint4*>(source + z);
                } else {
                    auto* elements = reinterpret_cast<__nv_bfloat16*>(&value);
                    for (uint32_t i = 0; i < 8 && z + i < args.rank; ++i) elements[i] = source[z + i];
                }
            }
            *reinterpret_cast<uint4*>(w2 + channel * layout.z_stride + z) = value;
        }
    }
    if (threadIdx.x < kDim) {
        const uint32_t channel = threadIdx.x;
        const bool live = channel < dim;
        constants[channel] = live ? __bfloat162float(args.decay_base[head_base + channel]) : 0.0f;
        constants[kDim + channel] = live ? __bfloat162float(args.removal_bias[head_base + channel]) : 0.0f;
        constants[2 * kDim + channel] = live ? __bfloat162float(args.norm[head_base + channel]) : 0.0f;
    }

    enum { kMatrices, kCopies, kElements, kTriangles };
    const uint32_t warp_of_cta = threadIdx.x / 32;
    const uint32_t group = warp_of_cta < 4 ? kMatrices : (warp_of_cta < 8 ? kCopies
                           : (warp_of_cta < 8 + kElementWarps ? kElements : kTriangles));
    const uint32_t warp = warp_of_cta < 8 ? warp_of_cta % 4
                          : (group == kElements ? warp_of_cta - 8 : warp_of_cta - 8 - kElementWarps);   // of the group
    const uint32_t lane = threadIdx.x % 32;
    const uint32_t g = lane >> 2, q = lane & 3;

    __syncthreads();

    auto step_barrier = [] { barrier_sync(kStepBarrier, kThreads); };
    // Every group has a loop of its own, so that none holds the registers of another.
    if (group == kMatrices) {
        set_more_registers<kMatrixRegisters>();
        // the state of 16 value columns, [8 key channels]: value columns g and g + 8, channels 2 q and 2 q + 1
        const uint32_t column0 = warp * 16;
        float state[8][4];
#pragma unroll
        for (uint32_t n = 0; n < 8; ++n) {
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                const uint32_t row = n * 8 + q * 2, column = column0 + g + half * 8;
                const bool live = row < dim && column < dim;          // the head size is a multiple of 8
                const float2 both = live ? *reinterpret_cast<const float2*>(state_base + static_cast<size_t>(column) * dim + row)
                                         : make_float2(0.0f, 0.0f);
                state[n][2 * half] = both.x;
                state[n][2 * half + 1] = both.y;
            }
        }
        for (int step = -4; step <= tiles; ++step) {
            const int tile = step;
            if (tile >= 0 && tile < tiles) {
                const float4* rows = rows_of(tile) + lane;
                const float4* triangles = triangles_of(tile) + lane;
                // (U S)^T and (R S)^T: value columns x tokens
                float right[2][4] = {}, result[2][4] = {};             // [8 tokens]
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) {
                    const FragmentA<> a = fragment_of(state[k]);
                    FragmentB<> b[4];
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) b[j] = fragment_of(rows[(j * 8 + k) * 32]);
                    // the accumulators alternate so that no product waits for the one before it
#pragma unroll
                    for (uint32_t part = 0; part < 3; ++part) {
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j) {
                            mma_tf32(j < 2 ? right[j] : result[j - 2], part == 0 ? a.low : a.high,
                                     part == 1 ? b[j].low : b[j].high);
                        }
                    }
                }
                // v of the tile: A operand [column][token], exact in TF32
                float v[2][4];                                         // [8 tokens]
                {
                    uint32_t raw[4];
                    const __nv_bfloat16* values = late_of(tile) + (lane / 16 * 8 + lane % 8) * kLateRow + column0 + lane / 8 % 2 * 8;
                    ldmatrix_x4_trans(smem_u32(values), raw[0], raw[1], raw[2], raw[3]);
#pragma unroll
                    for (uint32_t k = 0; k < 2; ++k) {
                        v[k][0] = __uint_as_float(raw[2 * k] << 16);
                        v[k][1] = __uint_as_float(raw[2 * k + 1] << 16);
                        v[k][2] = __uint_as_float(raw[2 * k] & 0xffff0000u);
                        v[k][3] = __uint_as_float(raw[2 * k + 1] & 0xffff0000u);
                    }
                }
                // Triangles as B operands [s][t]: fragment (t / 8) * 2 + s / 8; the one of t < 8 <= s is zero.
                {
                    const FragmentB<> b0 = fragment_of(triangles[kTriangle]), b2 = fragment_of(triangles[kTriangle + 64]),
                                      b3 = fragment_of(triangles[kTriangle + 96]);
                    mma_exact(right[0], v[0], b0);
                    mma_exact(right[1], v[0], b2);
                    mma_exact(right[1], v[1], b3);
                }
                FragmentA<> y[2];
                {
                    float solved[2][4] = {};
                    const FragmentA<> a0 = fragment_of(right[0]), a1 = fragment_of(right[1]);
                    mma_split(solved[0], a0, fragment_of(triangles[0]));
                    mma_split(solved[1], a0, fragment_of(triangles[64]));
                    mma_split(solved[1], a1, fragment_of(triangles[96]));
                    y[0] = fragment_of(solved[0]);
                    y[1] = fragment_of(solved[1]);
                }
                // the state behind the tile
                const Column* columns = columns_of(tile) + (g * 4 + (q ^ (g >> 1)));
                const float* decay = decay_end_of(tile);
#pragma unroll
                for (uint32_t quad = 0; quad < 8; quad += 4) {         // four accumulators: each product is through when its turn comes
#pragma unroll
                    for (uint32_t k = 0; k < 2; ++k) {
                        FragmentB<> with_v[4], with_y[4];
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) {
                            const uint32_t at = ((quad + i) * 2 + k) * 32;
                            with_v[i] = fragment_of(columns[at]);
                            with_y[i] = fragment_of(columns[kFragments * 32 + at]);
                        }
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) mma_tf32(state[quad + i], v[k], with_v[i].low);
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) mma_tf32(state[quad + i], v[k], with_v[i].high);
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) mma_tf32(state[quad + i], y[k].low, with_y[i].high);
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) mma_tf32(state[quad + i], y[k].high, with_y[i].low);
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) mma_tf32(state[quad + i], y[k].high, with_y[i].high);
                    }
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        const float2 factor = *reinterpret_cast<const float2*>(decay + (quad + i) * 8 + q * 2);
                        state[quad + i][0] *= factor.x;
                        state[quad + i][1] *= factor.y;
                        state[quad + i][2] *= factor.x;
                        state[quad + i][3] *= factor.y;
                    }
                }
                // O
                {
                    const float4* with_y = triangles + 2 * kTriangle;
                    const float4* with_v = triangles + 3 * kTriangle;
                    mma_exact(result[0], v[0], fragment_of(with_v[0]));
                    mma_exact(result[1], v[0], fragment_of(with_v[64]));
                    mma_split(result[0], y[0], fragment_of(with_y[0]));
                    mma_split(result[1], y[0], fragment_of(with_y[64]));
                    mma_exact(result[1], v[1], fragment_of(with_v[96]));
                    mma_split(result[1], y[1], fragment_of(with_y[96]));
                }
                float* produced = produced_of(tile) + column0 + g;
#pragma unroll
                for (uint32_t j = 0; j < 2; ++j) {
                    float* at = produced + (j * 8 + q * 2) * kProducedStride;
                    at[0] = result[j][0];
                    at[kProducedStride] = result[j][1];
                    at[8] = result[j][2];
                    at[kProducedStride + 8] = result[j][3];
                }
            }
            step_barrier();
        }
#pragma unroll
        for (uint32_t n = 0; n < 8; ++n) {
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                const uint32_t row = n * 8 + q * 2, column = column0 + g + half * 8;
                if (row < dim && column < dim) {
                    *reinterpret_cast<float2*>(state_base + static_cast<size_t>(column) * dim + row) =
                        make_float2(state[n][2 * half], state[n][2 * half + 1]);
                }
            }
        }
    } else if (group == kCopies) {
        set_fewer_registers<kOtherRegisters>();
        // the 16-byte pieces of a token's row that a lane moves, at most two (ranks up to 128), and where they go
        struct Piece {
            const __nv_bfloat16* source;
            uint32_t target, row_bytes, stage_bytes, ring_bytes, slot_bytes;
            bool mine;
        };
        Piece pieces[2];
#pragma unroll
        for (uint32_t which = 0; which < 2; ++which) {
            const uint32_t piece = lane + which * 32, per_vector = dim / 8;
            const uint32_t vector = min(piece / per_vector, 5u);           // r, k, v, g, a, z
            const uint32_t chunk = piece - vector * per_vector;
            const bool late = vector == 2 || vector == 3;
            Piece& out = pieces[which];
            out.source = args.projected + static_cast<size_t>(begin + warp * 4) * args.pitch + vector * width +
                         (vector < 5 ? head_base : 0) + chunk * 8;
            out.row_bytes = (late ? kLateRow : layout.early_row) * 2;
            out.stage_bytes = kTokens * out.row_bytes;
            out.ring_bytes = (late ? kLateStages : kEarlyStages) * out.stage_bytes;
            out.slot_bytes = 0;
            out.target = smem_u32(chunk_shared) + static_cast<uint32_t>(late ? layout.late : layout.early) +
                         warp * 4 * out.row_bytes + ((vector < 2 ? vector : vector - 2) * kDim + chunk * 8) * 2;
            out.mine = piece < 5 * per_vector + (args.rank + 7) / 8;
        }
        uint32_t left = end - begin > warp * 4 ? end - begin - warp * 4 : 0;   // tokens from this warp's first of the next tile on
        for (int step = -4; step <= tiles; ++step) {
            // ---- load tile step + 4
#pragma unroll
            for (uint32_t which = 0; which < 2; ++which) {
                Piece& piece = pieces[which];
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    if (piece.mine && i < left) {
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(piece.target + piece.slot_bytes +
                                                                                      i * piece.row_bytes),
                                     "l"(piece.source + i * args.pitch)
                                     : "memory");
                    }
                }
                piece.source += kTokens * args.pitch;
                piece.slot_bytes += piece.stage_bytes;
                if (piece.slot_bytes == piece.ring_bytes) piece.slot_bytes = 0;
            }
            left = left > kTokens ? left - kTokens : 0;
            copy_async_commit();
            // ---- tanh(z) and 1 / |k| of tile step + 3, whose copies were issued one step ago
            copy_async_wait<1>();
            barrier_sync(kCopiesBarrier, 128);
            const int tile = step + 3;
            if (tile >= 0 && tile < tiles) {
                const __nv_bfloat16* stage = early_of(tile);
                __nv_bfloat16* parts = tanh_of(tile);
                float squares[4];
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const float2 both = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(
                        stage + (warp * 4 + i) * layout.early_row + kDim + lane * 2));
                    squares[i] = fmaf(both.x, both.x, both.y * both.y);
                }
                for (uint32_t z = lane * 2; z < layout.rank_pad; z += 64) {
                    float2 both[4];
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        both[i] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(
                            stage + (warp * 4 + i) * layout.early_row + 3 * kDim + z));
                        // columns between rank and the end of its last copy belong to nobody
                        both[i].x = z < args.rank ? fast_tanh(both[i].x) : 0.0f;
                        both[i].y = z + 1 < args.rank ? fast_tanh(both[i].y) : 0.0f;
                    }
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        const __nv_bfloat162 high = __floats2bfloat162_rn(both[i].x, both[i].y);
                        const float2 rounded = __bfloat1622float2(high);
                        __nv_bfloat16* target = parts + (warp * 4 + i) * layout.z_stride + z;
                        *reinterpret_cast<__nv_bfloat162*>(target) = high;
                        *reinterpret_cast<__nv_bfloat162*>(target + kTokens * layout.z_stride) =
                            __floats2bfloat162_rn(both[i].x - rounded.x, both[i].y - rounded.y);
                    }
                }
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) squares[i] = warp_sum(squares[i]);
                if (lane < 4) {
                    const float mine = lane == 0 ? squares[0] : (lane == 1 ? squares[1] : (lane == 2 ? squares[2] : squares[3]));
                    unit_of(tile)[warp * 4 + lane] = rsqrtf(mine + kUnitEps);
                }
            }
            step_barrier();
        }
    } else if (group == kElements) {
        for (int step = -4; step <= tiles; ++step) {
            const int tile = step + 2;
            const bool active = tile >= 0 && tile < tiles;
            float products[4][2][4] = {};             // U B^T, U K^T, R B^T, R K^T over this warp's channels: [8 tokens s]
            if (active) {
                const uint32_t tokens = min(kTokens, end - begin - static_cast<uint32_t>(tile) * kTokens);
                const __nv_bfloat16* stage = early_of(tile);
                const __nv_bfloat16* parts = tanh_of(tile);
                const float* unit = unit_of(tile);
                // decay logits of 16 tokens x 8 channels per warp
                float logits[4] = {};
                const uint32_t z_row = lane % 16, z_part = lane / 16 * 8;
                for (uint32_t z = 0; z < layout.rank_pad; z += 32) {
                    uint32_t w[4];
                    ldmatrix_x4(smem_u32(w2 + (warp * 8 + lane % 8) * layout.z_stride + z + lane / 8 * 8), w[0], w[1], w[2], w[3]);
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        uint32_t high[4], low[4];
                        const __nv_bfloat16* source = parts + z_row * layout.z_stride + z + half * 16 + z_part;
                        ldmatrix_x4(smem_u32(source), high[0], high[1], high[2], high[3]);
                        ldmatrix_x4(smem_u32(source + kTokens * layout.z_stride), low[0], low[1], low[2], low[3]);
                        mma_bf16_16816(logits, high[0], high[1], high[2], high[3], w[2 * half], w[2 * half + 1]);
                        mma_bf16_16816(logits, low[0], low[1], low[2], low[3], w[2 * half], w[2 * half + 1]);
                    }
                }
                // log decay per token, then its prefix sums: over the eight lanes that hold tokens 0..7, and over
                // those that hold 8..15 in the other half of the fragment
                const uint32_t channel = warp * 8 + q * 2;
                float own[4], prefix[4];
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    own[i] = g + (i >> 1) * 8 < tokens ? -kDecayScale * fast_sigmoid(logits[i] + constants[channel + (i & 1)]) : 0.0f;
                    prefix[i] = own[i];
                }
#pragma unroll
                for (uint32_t delta = 4; delta < 32; delta <<= 1) {
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        const float other = __shfl_up_sync(0xffffffffu, prefix[i], delta);
                        if (lane >= delta) prefix[i] += other;
                    }
                }
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) prefix[2 + i] += __shfl_sync(0xffffffffu, prefix[i], 28 + q);
                float4* rows = rows_of(tile) + lane;
                // fragments [8 tokens s][8 channels]: channel 2 q + (g & 1) and the tokens around g of a lane's pair
                const uint32_t channel8 = q * 2 + (g & 1);
                Column* columns = columns_of(tile) + channel8 * 4 + ((g >> 1) ^ (channel8 >> 1));
                {
                    const uint32_t fragment = warp;
                    const float2 bias = *reinterpret_cast<const float2*>(constants + kDim + channel);
                    FragmentA<> with_u, with_r;
                    FragmentB<> with_k[2], with_b[2];
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        const uint32_t t = g + half * 8;
                        const __nv_bfloat16* row = stage + t * layout.early_row + channel;
                        float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row));
                        float2 k = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row + kDim));
                        const float2 rate = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(row + 2 * kDim));
                        if (t >= tokens) r = k = make_float2(0.0f, 0.0f);      // left over from an earlier tile
                        const float scale = unit[t];
                        const float px = __expf(prefix[2 * half]), py = __expf(prefix[2 * half + 1]);
                        const float bx = __expf(prefix[2 * half] - own[2 * half]);
                        const float by = __expf(prefix[2 * half + 1] - own[2 * half + 1]);
                        const float ix = __expf(-prefix[2 * half]), iy = __expf(-prefix[2 * half + 1]);
                        const float4 u_parts = in_parts(k.x * scale * bx, k.y * scale * by);
                        const float4 r_parts = in_parts(r.x * px, r.y * py);
                        rows[(half * 8 + fragment) * 32] = u_parts;
                        rows[(kFragments + half * 8 + fragment) * 32] = r_parts;
                        with_u.high[half] = u_parts.x;
                        with_u.high[2 + half] = u_parts.y;
                        with_u.low[half] = u_parts.z;
                        with_u.low[2 + half] = u_parts.w;
                        with_r.high[half] = r_parts.x;
                        with_r.high[2 + half] = r_parts.y;
                        with_r.low[half] = r_parts.z;
                        with_r.low[2 + half] = r_parts.w;
                        const float2 key = make_float2(k.x * ix, k.y * iy);
                        const float2 back = make_float2(-fast_sigmoid(rate.x + bias.x) * k.x * scale * ix,
                                                        -fast_sigmoid(rate.y + bias.y) * k.y * scale * iy);
                        with_k[half] = fragment_of(key);
                        with_b[half] = fragment_of(back);
                        // the neighbouring token's value of one of the two channels comes from its lane
                        const bool odd = (g & 1) != 0;
                        auto exchange = [&](float first, float second) {
                            const float other = __shfl_xor_sync(0xffffffffu, odd ? first : second, 4);
                            return odd ? make_float2(other, second) : make_float2(first, other);
                        };
                        const uint32_t at = (fragment * 2 + half) * 32;
                        if constexpr (SPLIT) {
                            const float2 k_high = exchange(with_k[half].high[0], with_k[half].high[1]);
                            const float2 k_low = exchange(with_k[half].low[0], with_k[half].low[1]);
                            const float2 b_high = exchange(with_b[half].high[0], with_b[half].high[1]);
                            const float2 b_low = exchange(with_b[half].low[0], with_b[half].low[1]);
                            columns[at] = make_float4(k_high.x, k_high.y, k_low.x, k_low.y);
                            columns[kFragments * 32 + at] = make_float4(b_high.x, b_high.y, b_low.x, b_low.y);
                        } else {
                            columns[at] = exchange(key.x, key.y);
                            columns[kFragments * 32 + at] = exchange(back.x, back.y);
                        }
                        if (t == kTokens - 1) {
                            *reinterpret_cast<float2*>(decay_end_of(tile) + channel) = make_float2(px, py);
                        }
                    }
#pragma unroll
                    for (uint32_t part = 0; part < 3; ++part) {
#pragma unroll
                        for (uint32_t j = 0; j < 2; ++j) {
                            const auto& u_part = part == 0 ? with_u.low : with_u.high;
                            const auto& r_part = part == 0 ? with_r.low : with_r.high;
                            const auto& b_part = part == 1 ? with_b[j].low : with_b[j].high;
                            const auto& k_part = part == 1 ? with_k[j].low : with_k[j].high;
                            mma_tf32(products[0][j], u_part, b_part);
                            mma_tf32(products[1][j], u_part, k_part);
                            mma_tf32(products[2][j], r_part, b_part);
                            mma_tf32(products[3][j], r_part, k_part);
                        }
                    }
                }
            }
            barrier_sync(kPartialsBarrier, 32 * (kElementWarps + 4));
            if (active) {
                float4* target = partials + warp * 8 * 32 + lane;
#pragma unroll
                for (uint32_t p = 0; p < 4; ++p) {
#pragma unroll
                    for (uint32_t j = 0; j < 2; ++j) {
                        target[(p * 2 + j) * 32] =
                            make_float4(products[p][j][0], products[p][j][1], products[p][j][2], products[p][j][3]);
                    }
                }
            }
            step_barrier();
        }
    } else {
        set_fewer_registers<kOtherRegisters>();
        for (int step = -4; step <= tiles; ++step) {
            const int tile = step + 1;
            const bool active = tile >= 0 && tile < tiles;
            float4 sum[2];                             // product `warp`: rows g and g + 8, columns 8 j + 2 q and the next
            if (active) {
#pragma unroll
                for (uint32_t j = 0; j < 2; ++j) {
                    const float4* source = partials + (warp * 2 + j) * 32 + lane;
                    float4 part[kElementWarps];
#pragma unroll
                    for (uint32_t w = 0; w < kElementWarps; ++w) part[w] = source[w * 8 * 32];
#pragma unroll
                    for (uint32_t step_of = kElementWarps / 2; step_of > 0; step_of /= 2) {
#pragma unroll
                        for (uint32_t w = 0; w < step_of; ++w) {
                            part[w].x += part[w + step_of].x;
                            part[w].y += part[w + step_of].y;
                            part[w].z += part[w + step_of].z;
                            part[w].w += part[w + step_of].w;
                        }
                    }
                    sum[j] = part[0];
                }
            }
            barrier_arrive(kPartialsBarrier, 32 * (kElementWarps + 4));
            if (active) {
                float4* triangles = triangles_of(tile);
                const uint32_t reach = warp < 2 ? 0 : 1;               // U meets the state before s = t
#pragma unroll
                for (uint32_t j = 0; j < 2; ++j) {
                    const uint32_t s = j * 8 + q * 2;
                    if (s >= g + reach) sum[j].x = 0.0f;
                    if (s + 1 >= g + reach) sum[j].y = 0.0f;
                    if (s >= g + 8 + reach) sum[j].z = 0.0f;
                    if (s + 1 >= g + 8 + reach) sum[j].w = 0.0f;
                    if (warp > 0) {
                        triangles[warp * kTriangle + j * 32 + lane] = in_parts(sum[j].x, sum[j].y);
                        triangles[warp * kTriangle + (2 + j) * 32 + lane] = in_parts(sum[j].z, sum[j].w);
                    } else {
                        const float values[4] = {sum[j].x, sum[j].y, sum[j].z, sum[j].w};
                        store_c(lower + j * 8, kLowerStride, lane, values);
                    }
                }
                if (warp == 0) {
                    __syncwarp();
                    // column `lane` of the inverse of I - L: x_t = e_t + sum over s < t of L[t][s] x_s
                    float x[kTokens];
                    float* target = reinterpret_cast<float*>(triangles) +
                                    ((lane >> 3) * 32 + (lane % 8 >> 1)) * 4 + (lane & 1);
#pragma unroll
                    for (uint32_t t = 0; t < kTokens; ++t) {
                        float even = t == lane ? 1.0f : 0.0f, odd = 0.0f;
#pragma unroll
                        for (uint32_t s = 0; s < t; s += 2) {
                            const float2 pair = *reinterpret_cast<const float2*>(lower + t * kLowerStride + s);
                            even = fmaf(pair.x, x[s], even);
                            if (s + 1 < t) odd = fmaf(pair.y, x[s + 1], odd);
                        }
                        x[t] = even + odd;
                        if (lane < kTokens) {
                            FragmentB<> parts;
                            parts.set(0, x[t]);
                            float* at = target + ((t >> 3) * 2 * 32 + t % 8 * 4) * 4;
                            at[0] = parts.high[0];
                            at[2] = parts.low[0];
                        }
                    }
                    __syncwarp();          // the plain triangle is free again
                }
            }
            // ---- finish tile step - 1: norm and gate, by the warps that invert no triangle
            if (step >= 1 && warp > 0) {
                const int done = step - 1;
                const __nv_bfloat16* stage = late_of(done);
                const float* source = produced_of(done);
                const uint32_t first = begin + static_cast<uint32_t>(done) * kTokens;
                const float2 weight = *reinterpret_cast<const float2*>(constants + 2 * kDim + lane * 2);
                const float inverse_dim = 1.0f / static_cast<float>(dim);
                __nv_bfloat16* target = args.out + static_cast<size_t>(first) * args.out_pitch + head_base + lane * 2;
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {            // three tokens of each half of the tile, the last warp two
                    float2 value[3], gate[3];
                    float squares[3];
#pragma unroll
                    for (uint32_t i = 0; i < 3; ++i) {
                        const uint32_t t = min(half * 8 + (warp - 1) * 3 + i, kTokens - 1);
                        value[i] = *reinterpret_cast<const float2*>(source + t * kProducedStride + lane * 2);
                        gate[i] =
                            __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(stage + t * kLateRow + kDim + lane * 2));
                        squares[i] = fmaf(value[i].x, value[i].x, value[i].y * value[i].y);
                    }
#pragma unroll
                    for (uint32_t delta = 16; delta > 0; delta >>= 1) {
#pragma unroll
                        for (uint32_t i = 0; i < 3; ++i) squares[i] += __shfl_xor_sync(0xffffffffu, squares[i], delta);
                    }
#pragma unroll
                    for (uint32_t i = 0; i < 3; ++i) {
                        const uint32_t of_half = (warp - 1) * 3 + i, t = half * 8 + of_half;
                        const float factor = rsqrtf(fmaf(squares[i], inverse_dim, args.eps));
                        const uint32_t both = pack_bf16x2(value[i].x * factor * weight.x * fast_sigmoid(gate[i].x),
                                                          value[i].y * factor * weight.y * fast_sigmoid(gate[i].y));
                        if (of_half < 8 && lane * 2 < dim && first + t < end) {
                            *reinterpret_cast<uint32_t*>(target + t * args.out_pitch) = both;
                        }
                    }
                }
            }
            step_barrier();
        }
    }
}

template <bool SPLIT>
cudaError_t launch(cudaStream_t stream, const DeltaArgs<__nv_bfloat16>& args) {
    const size_t shared = Layout<SPLIT>(args.rank).total;
    const auto kernel = delta_chunk_kernel<SPLIT>;
    const cudaError_t status = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared));
    if (status != cudaSuccess) return status;
    return launch_kernel(kernel, static_cast<unsigned int>(args.segments.num_segments * args.heads), kThreads, shared, stream,
                         1, args);
}

constexpr size_t kSharedLimit = 226 * 1024;            // beside the static word; holds Layout<false> of kMostRank
constexpr uint32_t kMostRank = 128;                    // larger ones keep the plain f32 arithmetic of the prompt kernel
constexpr uint32_t kMostTwoPartRank = 64;                // K and B in two parts where shared memory holds them
static_assert(Layout<true>(kMostTwoPartRank).total <= kSharedLimit && Layout<true>(kMostTwoPartRank + 1).total > kSharedLimit &&
                  Layout<false>(kMostRank).total <= kSharedLimit, "what shared memory holds");

}  // namespace

bool delta_chunk_takes(uint32_t dim, uint32_t rank) { return dim <= kDim && rank <= kMostRank; }

cudaError_t launch_delta_chunk(cudaStream_t stream, const DeltaArgs<__nv_bfloat16>& args) {
    return args.rank <= kMostTwoPartRank ? launch<true>(stream, args) : launch<false>(stream, args);
}

}  // namespace lfm25

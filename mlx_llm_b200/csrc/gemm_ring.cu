// Projections of up to 32 tokens: weights through a ring of shared memory.
//
//   y[M, N] = x[M, K] . W[N, K]^T,   W dense bf16 or MLX-format group-64 affine Q4 / Q8,   M <= 32
//
// Same contract as the register-streaming kernel in gemm_stream.cu (primitives::nn::linear, src/primitives/nn.rs:26-33;
// QuantizedLinear::forward, src/primitives/quant.rs:56-70): the weights are the A operand of mma.sync m16n8k16, dequantised in
// registers to that kernel's weights, the tokens its 8-wide N side.  HBM bounds these calls, and behind it the instructions that a weight
// costs and the fixed time of a launch.
//   * A stage, 128 feature rows x 128 bytes, comes in by one TMA copy, with its scales and biases (from the transposed table) as bulk
//     copies on the same barrier: no address arithmetic, no load per row, 130 KB in flight on an SM without a register.
//   * A code becomes a bf16 weight in little more than one instruction (dequant.cuh), two 16-byte shared-memory loads feed a row's 32 codes
//     and the activations of two MMA steps.  Both are free of bank conflicts: MMA row g is feature row 4 (g & 1) + g / 2, so that the
//     rows of a quarter-warp lie in different halves of the 128-byte swizzle, and the activations are laid out as [8 K][thread of a
//     row group] with 64 bytes more than a multiple of 128 per token.
//   * K is cut into the other kernel's ranges, each summed in K order by one warp, and the ranges are added in order: the results are
//     that kernel's bits.  The blocks of a cluster share a row tile's ranges and add them up through distributed shared memory, where
//     that kernel writes partial sums to global memory and lets the block that counts in last read them back.
// The weights of a model do not depend on the kernel before this one: the ring is filled with them before the wait for that kernel.
// One token, us a call among others of its kind, register-streaming kernel -> this one (bytes at the copy rate): 28672 x 4096 Q4
// 29.1 -> 22.3 (10.2), 4096 x 14336 Q4 17.4 -> 14.4 (5.1), 51200 x 5120 Q8 100 -> 52.1 (43.1), 5120 x 25600 Q8 55.2 -> 29.3 (21.6),
// 2048 x 2048 bf16 7.1 -> 5.1 (1.3), 128256 x 4096 bf16 172 -> 159 (163); 16 tokens: 39.6 -> 32.8, 25.5 -> 19.9, 112 -> 63.4,
// 67.1 -> 36.6, 9.2 -> 6.1, 185 -> 170.  With 17 to 32 tokens on Q4 the activations leave the ring too few stages, and the other
// kernel is faster; on Q8 and bf16 it is not (32 tokens: 51200 x 5120 Q8 127 -> 80, 28672 x 4096 bf16 62 -> 55).
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "dequant.cuh"
#include "kernels.h"
#include "tc5.cuh"

namespace {
using namespace tc5;

constexpr int kRows = 128, kRowBytes = 128, kTileBytes = kRows * kRowBytes;
constexpr int kConsumers = 256, kThreads = kConsumers + 64;  // and a warp each for the weights and the activations
constexpr int kGroupStride = kRows * 4 + 32;  // bytes of one group's scale|bias words: the next group eight banks further
constexpr int kSumStride = kRows + 4;         // floats of one token's partial sums
constexpr int kWeightsGaveUp = 20, kActivationsGaveUp = 21, kConsumersGaveUp = 22;  // error codes of bounded waits, none of another kernel's

template <int WK, int NT>
struct Ring {
    static constexpr int KS = kRowBytes * 8 / (WK ? WK : 16);  // K of a stage: 256, 128, 64
    static constexpr int E = KS / 8;                           // K of a 16-byte piece of a row
    static constexpr int XS = KS * 2 + 64;                     // bytes of a token's activations
    static constexpr int X_BYTES = NT * 8 * XS;
    static constexpr int SB_BYTES = WK ? KS / 64 * kGroupStride : 0;
    static constexpr int STAGE = kTileBytes + X_BYTES + SB_BYTES;
    static constexpr int SUMS = NT * 8 * kSumStride * 4;         // sums of one K range
    static constexpr int kSlots = NT == 1 ? 3 : NT == 2 ? 2 : 0;  // ... kept beside the ring; a block's last range goes over the ring
    static constexpr int kBudget = 114000 - kSlots * SUMS;        // two blocks on an SM
    static constexpr int STAGES = kBudget / STAGE > 6 ? 6 : kBudget / STAGE;
    static constexpr int SMEM = STAGES * STAGE + kSlots * SUMS + 1024 + 16 * STAGES;
    static_assert(STAGES >= 3 && SUMS <= STAGES * STAGE);
};

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(kConsumers) : "memory"); }

// four consecutive features of a token
template <int EPI>
__device__ __forceinline__ void store4(const GemmParams& p, int tok, int row, float4 a) {
    if (EPI == EPI_F32) {
        *reinterpret_cast<float4*>(gemm_f32_dst(p, tok, row)) = a;
    } else if (EPI == EPI_BF16) {
        *reinterpret_cast<uint2*>(p.out + (size_t)tok * p.ldo + row) = make_uint2(pack_bf2(a.x, a.y), pack_bf2(a.z, a.w));
    } else {
        const uint2 r = *reinterpret_cast<const uint2*>(p.res + (size_t)tok * p.ldres + row);
        *reinterpret_cast<uint2*>(p.out + (size_t)tok * p.ldo + row) =
            make_uint2(pack_bf2(bflo(r.x) + rbf(a.x), bfhi(r.x) + rbf(a.y)), pack_bf2(bflo(r.y) + rbf(a.z), bfhi(r.y) + rbf(a.w)));
    }
}

template <int WK, int NT, int EPI>
__global__ void __launch_bounds__(kThreads, 2)
    gemm_ring_kernel(const __grid_constant__ CUtensorMap wmap, const GemmParams p, int ranges, int range_stages, int* err) {
    using R = Ring<WK, NT>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;  // tiles on 1024 bytes, as their swizzle asks
    const uint32_t xring = ring + R::STAGES * kTileBytes, sbring = xring + R::STAGES * R::X_BYTES, slots = sbring + R::STAGES * R::SB_BYTES;
    const uint32_t bars = slots + R::kSlots * R::SUMS;
    auto full = [&](int s) { return bars + 16u * s; };
    auto empty = [&](int s) { return bars + 16u * s + 8u; };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int M = p.M, N = p.N, row0 = blockIdx.y * kRows, splits = gridDim.x;
    // this block's K ranges, and their stages
    auto first_range = [&](int rank) { return ranges * rank / splits; };
    const int range0 = first_range(blockIdx.x), range1 = first_range(blockIdx.x + 1);
    const int stage0 = range0 * range_stages, stage1 = min(range1 * range_stages, p.K / R::KS);

    if (tid == 0) {
        for (int s = 0; s < R::STAGES; s++) {
            mbar_init(full(s), 33);  // the copy engine's bytes behind one arrival, the activations behind one of each producing lane
            mbar_init(empty(s), kConsumers / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();

    if (warp == kConsumers / 32) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"(&wmap) : "memory");
            if (!p.w_settled) pdl_wait();
            int stage = stage0;
            for (int s = 0, lap = 0; stage < stage1; stage++) {
                if (lap > 0 && !mbar_wait(empty(s), (lap - 1) & 1)) {
                    atomicExch(err, kWeightsGaveUp);
                    break;
                }
                mbar_expect_tx(full(s), kTileBytes + (WK ? R::KS / 64 * kRows * 4 : 0));
                tma_load_2d(ring + s * kTileBytes, &wmap, stage * kRowBytes, row0, full(s));
                if (WK)
#pragma unroll
                    for (int g = 0; g < R::KS / 64; g++)
                        bulk_load(sbring + s * R::SB_BYTES + g * kGroupStride, p.sbt + (size_t)(stage * (R::KS / 64) + g) * N + row0, kRows * 4, full(s));
                if (++s == R::STAGES) s = 0, lap++;
            }
            // No copy may land in shared memory that another block has by then: the consumers have waited for all of them, unless a wait
            // of theirs ran out.
            for (int i = max(stage0, stage - R::STAGES); i < stage; i++)
                if (!mbar_wait(full((i - stage0) % R::STAGES), (i - stage0) / R::STAGES & 1)) break;
        }
        __syncwarp();
        pdl_wait();  // (no block may return before the kernel in front of this one has completed)
    } else if (warp == kConsumers / 32 + 1) {
        pdl_wait();
        constexpr int PIECES = R::KS / 8, DM = 32 / PIECES;  // 16-byte pieces of a token's activations; tokens a warp copies at once
        const int q = lane % PIECES, m0 = lane / PIECES;
        // piece q holds K 8q .. 8q + 7: thread t = (8q / E) & 3 of span (8q / E) / 4 needs it for its MMA steps 2 e8, 2 e8 + 1
        const int c = q * 8 / R::E, e8 = (q * 8 % R::E) / 8;
        const uint32_t xdst = xring + m0 * R::XS + (uint32_t)((((c >> 2) * (R::E / 8) + e8) * 4 + (c & 3)) * 16);
        const uint16_t* xsrc = p.x + (size_t)m0 * p.ldx + q * 8;
        for (int stage = stage0, s = 0, lap = 0; stage < stage1; stage++) {
            if (lap > 0 && !__all_sync(0xffffffffu, mbar_wait(empty(s), (lap - 1) & 1))) {
                if (lane == 0) atomicExch(err, kActivationsGaveUp);
                break;
            }
            const uint16_t* src = xsrc + stage * R::KS;
            uint32_t dst = xdst + s * R::X_BYTES;
            for (int m = m0; m < M; m += DM) {
                cp_async16(dst, src);
                dst += DM * R::XS;
                src += (size_t)DM * p.ldx;
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(full(s)) : "memory");
            if (++s == R::STAGES) s = 0, lap++;
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    } else {
        const int g = lane >> 2, t = lane & 3, rg = (g & 1) * 4 + (g >> 1);  // 16 rows of the tile
        const uint32_t row = (uint32_t)(warp * 16 + rg), xoff = (uint32_t)(g * R::XS + t * 16);
        float acc[NT][4] = {};
        bool alive = true;  // after a wait that ran out the sums are worthless
        for (int stage = stage0, s = 0, lap = 0, range = range0, left = range_stages; stage < stage1; stage++) {
            if (alive && !__all_sync(0xffffffffu, mbar_wait(full(s), lap & 1))) {
                if (lane == 0) atomicExch(err, kConsumersGaveUp);
                alive = false;
            }
            uint4 w[2][2];  // [half of the stage's K][row g, row g + 8]
#pragma unroll
            for (int sp = 0; sp < 2; sp++)
#pragma unroll
                for (int i = 0; i < 2; i++) w[sp][i] = lds128(ring + s * kTileBytes + (row + i * 8) * kRowBytes + (((4 * sp + t) ^ rg) << 4));
            uint32_t sb[2][2];
            bool all_once = true;
            if (WK)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int sp = j >> 1, i = j & 1;
                    sb[sp][i] = lds32(sbring + s * R::SB_BYTES + (WK == 4 ? 2 * sp + (t >> 1) : sp) * kGroupStride + (row + i * 8) * 4);
                    if (WK == 8) all_once = all_once && one_rounding(sb[sp][i]);
                }
            auto half = [&](int sp, auto once) {
                uint32_t s_lo[2], s_hi[2], b2[2];
                if (WK)
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        s_lo[i] = prmt(sb[sp][i], 0u, 0x1010u), b2[i] = prmt(sb[sp][i], 0u, 0x3232u);
                        if (WK == 4) s_hi[i] = mul_bf2(s_lo[i], 0x3d803d80u);  // 2^-4
                    }
#pragma unroll
                for (int e8 = 0; e8 < R::E / 8; e8++) {  // eight K of every row: two MMA steps
                    uint32_t o[2][4];
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const uint4& wi = w[sp][i];
                        if (WK == 4) {
                            scaled_q4_paired((&wi.x)[e8], s_lo[i], s_hi[i], b2[i], o[i]);
                        } else if (WK == 8) {
#pragma unroll
                            for (int j = 0; j < 2; j++) {
                                const uint32_t codes = (&wi.x)[(2 * e8 + j) & 3];
                                if (decltype(once)::value)
                                    scaled_q8_once(codes, s_lo[i], b2[i], o[i][2 * j], o[i][2 * j + 1]);
                                else
                                    scaled_q8(codes, bflo(s_lo[i]), bflo(b2[i]), o[i][2 * j], o[i][2 * j + 1]);
                            }
                        } else {
                            o[i][0] = wi.x, o[i][1] = wi.y, o[i][2] = wi.z, o[i][3] = wi.w;
                        }
                    }
#pragma unroll
                    for (int nt = 0; nt < NT; nt++) {
                        const uint4 x = lds128(xring + s * R::X_BYTES + xoff + nt * 8 * R::XS + (sp * (R::E / 8) + e8) * 64);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            uint32_t b[2];
                            if (WK == 4) {  // the weights' pairs: (0,4) (1,5), (2,6) (3,7)
                                const uint32_t lo = h ? x.y : x.x, hi = h ? x.w : x.z;
                                b[0] = prmt(lo, hi, 0x5410u), b[1] = prmt(lo, hi, 0x7632u);
                            } else {
                                b[0] = h ? x.z : x.x, b[1] = h ? x.w : x.y;
                            }
                            const uint32_t a[4] = {o[0][2 * h], o[1][2 * h], o[0][2 * h + 1], o[1][2 * h + 1]};
                            mma_bf16_16816(acc[nt], a, b);
                        }
                    }
                }
            };
            // (a choice for the whole stage: inside the loops it cost 7 %, the f32 fma throughout 10 %, of a step of 6 sequences)
            if (WK != 8 || __all_sync(0xffffffffu, all_once)) {
                half(0, std::true_type{});
                half(1, std::true_type{});
            } else {
                half(0, std::false_type{});
                half(1, std::false_type{});
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(s));
            if (++s == R::STAGES) s = 0, lap++;
            if (--left > 0 && stage + 1 < stage1) continue;

            // a range's sums, [token][row]: the last one over the ring, once no warp reads it any more
            uint32_t at = slots + (uint32_t)(range - range0) * R::SUMS;
            if (stage + 1 == stage1) {
                consumers_sync();
                at = ring;
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(at + (uint32_t)((nt * 8 + 2 * t + (e & 1)) * kSumStride + (e >> 1) * 8 + row) * 4u),
                                 "f"(WK ? acc[nt][e] * p.sbt_unscale : acc[nt][e])
                                 : "memory");
                    acc[nt][e] = 0.f;
                }
            range++, left = range_stages;
        }
        pdl_wait();  // (the residual)
    }
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    // this block's share of the outputs, four rows of a token at a time, summed over the ranges in order
    for (int e = blockIdx.x * kConsumers + tid; tid < kConsumers && e < M * (kRows / 4); e += splits * kConsumers) {
        const int tok = e / (kRows / 4), f = e % (kRows / 4) * 4;
        const uint32_t off = (uint32_t)(tok * kSumStride + f) * 4u;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int z = 0, rank = 0, here = 0, next = first_range(1); z < ranges; z++) {
            uint32_t peer;
            asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(peer) : "r"(off + (z + 1 == next ? ring : slots + (uint32_t)here * R::SUMS)), "r"(rank));
            float4 v;
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer));
            a.x += v.x, a.y += v.y, a.z += v.z, a.w += v.w;
            here++;
            if (z + 1 == next) here = 0, rank++, next = first_range(rank + 1);
        }
        store4<EPI>(p, tok, row0 + f, a);
    }
    // no block leaves while another may still read its sums
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// clusters of `splits` blocks that the machine runs at once
template <int WK, int NT, int EPI>
int max_clusters(b2_ctx* ctx, int splits) {
    static std::atomic<int> known[16][9];
    std::atomic<int>& n = known[ctx->device & 15][splits];
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(splits, 256);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = Ring<WK, NT>::SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = splits;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int count = 0;
        if (cudaOccupancyMaxActiveClusters(&count, gemm_ring_kernel<WK, NT, EPI>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            count = 0;
        }
        n = count > 0 ? count : 1;
    }
    return n;
}

// Blocks of a cluster that share a row tile's K: 0 where a block would have more ranges than it has room for.  The cost is in stages
// of an SM's time: two blocks there share it, one alone takes 3/4 as long as the two; a round of blocks costs some 14 more.  One token,
// us with clusters of 1 .. 8 (- : too many ranges a block; Q8 with weights rounded once throughout, 4 % below now):
//   4096 x 14336 Q4   - - - - 17.1 16.3 14.7 14.8      5120 x 25600 Q8  - - - 34.6 28.2 29.5 40.1 38.3      6144 x 4096 Q4  - 9.0 9.8 8.4 8.5 12.8 13.2 11.3
//   28672 x 4096 Q4   22.7 29.3 26.5                   51200 x 5120 Q8  57.0 50.4                           10240 x 5120 Q8  - 16.0 13.4 20.1 19.7 19.3 22.5
//   17792 x 2048 bf16 14.9 14.0 19.2 16.3              28672 x 4096 bf16  39.4 44.1 44.2                    2048 x 2048 bf16  10.4 6.8 6.8 5.0
template <int WK, int NT, int EPI>
int ring_splits(b2_ctx* ctx, int tiles, int ranges, int range_stages) {
    int found = 0;
    double best = 1e30;
    for (int s = 1; s <= 8 && s <= ranges; s++) {
        const int each = (ranges + s - 1) / s;
        if (each > Ring<WK, NT>::kSlots + 1) continue;
        const int fit = max_clusters<WK, NT, EPI>(ctx, s), rounds = (tiles + fit - 1) / fit;
        const double cost = rounds * (each * range_stages * (tiles * s > ctx->sm_count ? 2.0 : 1.5) + 14);
        if (cost < best) best = cost, found = s;
    }
    return found;
}

template <int WK, int NT, int EPI>
int32_t launch_ring(b2_ctx* ctx, const GemmParams& p, int* cluster) {
    using R = Ring<WK, NT>;
    B2_SMEM_ONCE(ctx, (gemm_ring_kernel<WK, NT, EPI>), R::SMEM);
    const int tiles = p.N / kRows;
    const RangePlan cut = b2_gemm_stream_ranges(ctx, p.N, p.K);
    const int range_stages = cut.k_per_range / R::KS;
    const int splits = ring_splits<WK, NT, EPI>(ctx, tiles, cut.ranges, range_stages);
    B2_REQUIRE(splits > 0, B2_ERR_MSG, "gemm: no split of K for the ring kernel");
    if (cluster) {
        *cluster = splits;
        return B2_OK;
    }
    EncodeTiledFn encode = encode_fn();
    B2_REQUIRE(encode != nullptr, B2_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    CUtensorMap map;
    const cuuint64_t row_bytes = (cuuint64_t)p.K * (WK ? WK : 16) / 8;
    const cuuint64_t dims[2] = {row_bytes, (cuuint64_t)p.N}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {kRowBytes, kRows}, one[2] = {1, 1};
    const CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(p.w), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B2_REQUIRE(rc == CUDA_SUCCESS, B2_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)rc));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, tiles);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = R::SMEM;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    B2_CUDA(cudaLaunchKernelEx(&cfg, gemm_ring_kernel<WK, NT, EPI>, map, p, cut.ranges, range_stages, ctx->dev_err));
    B2_LAUNCHED(ctx);
    B2_CUDA(cudaGetLastError());
    return B2_OK;
}

template <int WK, int NT>
int32_t dispatch_epi(b2_ctx* ctx, const GemmParams& p, int* cluster) {
    switch (p.epilogue) {
        case EPI_BF16: return launch_ring<WK, NT, EPI_BF16>(ctx, p, cluster);
        case EPI_BF16_RESADD: return launch_ring<WK, NT, EPI_BF16_RESADD>(ctx, p, cluster);
        case EPI_F32: return launch_ring<WK, NT, EPI_F32>(ctx, p, cluster);
    }
    return b2_fail(B2_ERR_MSG, "gemm: bad epilogue");
}

template <int WK>
int32_t dispatch_nt(b2_ctx* ctx, const GemmParams& p, int* cluster) {
    if (p.M <= 8) return dispatch_epi<WK, 1>(ctx, p, cluster);
    if (p.M <= 16) return dispatch_epi<WK, 2>(ctx, p, cluster);
    if constexpr (WK != 4) return dispatch_epi<WK, 4>(ctx, p, cluster);
    return b2_fail(B2_ERR_MSG, "gemm: too many tokens for the ring kernel");
}

}  // namespace

bool b2_gemm_ring_eligible(b2_ctx* ctx, const GemmParams& p) {
    const bool dense = p.bits == 0;
    if (p.M < 1 || p.M > (p.bits == 4 ? 16 : 32) || p.N % kRows != 0 || p.N / kRows > 65535 || p.K % 256 != 0 || p.ldx % 8 != 0 || ((uintptr_t)p.x & 15) != 0 ||
        ((uintptr_t)p.w & 15) != 0 || !(dense || ((p.bits == 4 || p.bits == 8) && p.sbt && ((uintptr_t)p.sbt & 15) == 0)) ||
        // four rows of a token are stored at a time
        p.ldo % 4 != 0 || ((uintptr_t)p.out & 7) != 0 || ((uintptr_t)p.out_f32 & 15) != 0 ||
        (p.epilogue == EPI_BF16_RESADD && (p.ldres % 4 != 0 || ((uintptr_t)p.res & 7) != 0)))
        return false;
    const RangePlan cut = b2_gemm_stream_ranges(ctx, p.N, p.K);
    // Room for the sums of a block's ranges in clusters of eight; from 17 tokens on it has one range, and short ranges of many tiles
    // are no faster than the other kernel (17792 x 2048 bf16 at 32 tokens: 20.0 us there, 21.3 here).
    if (p.M > 16) return cut.ranges <= 8 && (p.N / kRows * cut.ranges <= 2 * ctx->sm_count || cut.k_per_range >= 1024);
    return (cut.ranges + 7) / 8 <= 1 + (p.M <= 8 ? Ring<0, 1>::kSlots : Ring<0, 2>::kSlots);
}

int32_t b2_gemm_ring_launch(b2_ctx* ctx, const GemmParams& p, int* cluster) {
    if (p.bits == 0) return dispatch_nt<0>(ctx, p, cluster);
    if (p.bits == 4) return dispatch_nt<4>(ctx, p, cluster);
    return dispatch_nt<8>(ctx, p, cluster);
}

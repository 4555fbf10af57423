// Fused W8A16 QKV projection for few rows: three f16 outputs [M,N] = (A[M,K] f16 x W_P[K,N] s8) *
// scale_P, the s8 -> f16 conversion inside the GEMM (no f16 copy of the weights in global memory).
//
// Replaces KAIO's `qkv_project_int8` kernel (kaio-ops/src/qkv_project_int8_kernel.rs) where M is
// small: cvt.rn.f16.s8 is exact, the products accumulate in f32, one f32 multiplication by the
// projection's (or column's) scale, one rounding to f16 -- the arithmetic of the two-launch path.
//
// What bounds it: a handful of latencies, not a rate.  The weights of three 2048 x 2048 projections
// are 12.6 MB (2 us); the path that first writes them out as f16 (and reads them back) took 39 us at
// M = 64, most of it two launches whose tiles left two thirds of the SMs idle.  So:
//  * the product is computed transposed, D^T[128 weight columns, NROWS rows]: at M <= 256 one tile
//    covers all rows and every weight is converted once;
//  * the weights go [64 k][128 columns] s8 by TMA -> f16 in the 128-byte swizzle that tcgen05 reads
//    MN-major (columns are contiguous in both, so the conversion never transposes) and the
//    activations by TMA as the K-major operand;
//  * the K range of a tile is cut over the CTAs of a cluster while they all run at once; the partial
//    tiles meet in distributed shared memory, in rank order: no scratch, no atomics, one launch.
// Measured (us per call, three projections, weights from HBM, two launches -> this one): 2048 x 2048, M = 64:
// 38.9 -> 14.0; 4096 x 4096, M = 300 / 512: 92 / 93 -> 60 / 66.  The kernel alone: 12.1 and, 4096 x 4096, M = 16 /
// 128 / 256: 23 / 30 / 36.
#include "common.cuh"
#include "kernels.h"

namespace kaio {
namespace w8f {

constexpr int BN = 128;  // weight columns per tile = UMMA M
constexpr int BK = 64;
constexpr int NUM_THREADS = 320;
constexpr int NUM_CONVERT_WARPS = 8;
constexpr int MAX_PROBS = 3;
constexpr uint32_t MAX_SPLIT = 8;

template <int NROWS>
struct Cfg {
    static constexpr int X_BYTES = NROWS * 128;   // [NROWS rows][64 k] f16
    static constexpr int W_BYTES = BK * BN;       // [64 k][128 columns] s8
    static constexpr int STAGE_BYTES = X_BYTES + W_BYTES;
    static constexpr int STAGES = NROWS <= 32 ? 6 : (NROWS <= 64 ? 4 : (NROWS <= 128 ? 3 : 4));
    static constexpr int A_BYTES = BK * BN * 2;   // converted: two [64 k][64 columns] sub-tiles
    static constexpr int A_SLOTS = NROWS <= 128 ? 2 : 3;
    static constexpr int RING_BYTES = A_SLOTS * A_BYTES + STAGES * STAGE_BYTES;
    static constexpr int RED_BYTES = NROWS * BN * 4;  // the f32 tile, over the rings when they are done
    static constexpr int BODY_BYTES = RING_BYTES > RED_BYTES ? RING_BYTES : RED_BYTES;
    static constexpr int NUM_BARS = 2 * STAGES + 2 * A_SLOTS + 1;
    static constexpr int SMEM_BYTES = 1024 + BODY_BYTES + NUM_BARS * 8 + 16;
    static constexpr int CTAS_PER_SM = NROWS <= 128 ? 2 : 1;
    static constexpr uint32_t IDESC = make_idesc(/*d=f32*/ 1, /*a=f16*/ 0, /*b=f16*/ 0,
                                                 /*a MN-major*/ 1, /*b K-major*/ 0, BN, NROWS);
    static_assert(SMEM_BYTES <= (CTAS_PER_SM == 2 ? 113 : 227) * 1024, "rings do not fit");
};

enum : uint32_t { SITE_EMPTY = 31, SITE_FULL = 32, SITE_A_FREE = 33, SITE_A_FULL = 34, SITE_D_FULL = 35 };

struct Problem {
    const float* col_scale;
    float scale;
    __half* out;
};

struct Params {
    Problem probs[MAX_PROBS];
    uint32_t m, n, num_kb, tiles_n;
    uint32_t* status;
};

struct TensorMaps {
    CUtensorMap x;
    CUtensorMap w[MAX_PROBS];
};

// Four s8 -> two half2 in order, exactly: the flipped sign bit makes a byte q + 128, under the
// exponent of 1024 it is 1024 + (q + 128).
__device__ __forceinline__ void convert4(uint32_t w, uint32_t& lo, uint32_t& hi)
{
    const uint32_t u = w ^ 0x80808080u;
    const uint32_t magic = 0x64646464u, bias = 0x64806480u;  // 1152
    const uint32_t a = __byte_perm(u, magic, 0x4140), b = __byte_perm(u, magic, 0x4342);
    const __half2 l = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&bias));
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&b), *reinterpret_cast<const __half2*>(&bias));
    lo = *reinterpret_cast<const uint32_t*>(&l);
    hi = *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

template <int NROWS>
__global__ void __launch_bounds__(NUM_THREADS, Cfg<NROWS>::CTAS_PER_SM)
w8a16_fused_kernel(const __grid_constant__ TensorMaps maps, const Params p, const uint32_t split)
{
    using C = Cfg<NROWS>;
    constexpr uint32_t STAGES = C::STAGES, A_SLOTS = C::A_SLOTS;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    // [A_SLOTS x converted weights] [STAGES x activations] [STAGES x s8 weights]
    constexpr uint32_t X_REGION = A_SLOTS * C::A_BYTES;
    constexpr uint32_t W_REGION = X_REGION + STAGES * C::X_BYTES;
    const uint32_t bar_base = smem_base + C::BODY_BYTES;
    auto full_bar = [&](uint32_t s) { return bar_base + 8u * s; };
    auto empty_bar = [&](uint32_t s) { return bar_base + 8u * (STAGES + s); };
    auto a_full = [&](uint32_t t) { return bar_base + 8u * (2 * STAGES + t); };
    auto a_free = [&](uint32_t t) { return bar_base + 8u * (2 * STAGES + A_SLOTS + t); };
    const uint32_t d_full = bar_base + 8u * (2 * STAGES + 2 * A_SLOTS);
    volatile uint32_t* tmem_slot =
        reinterpret_cast<volatile uint32_t*>(smem_gen + C::BODY_BYTES + C::NUM_BARS * 8);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = split > 1 ? cluster_ctarank() : 0u;
    const uint32_t tile = blockIdx.x / split;
    const uint32_t prob = tile / p.tiles_n;
    const uint32_t n0 = (tile - prob * p.tiles_n) * BN;
    const uint32_t m0 = blockIdx.y * NROWS;
    const uint32_t kb0 = p.num_kb * rank / split, kb1 = p.num_kb * (rank + 1) / split;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (uint32_t t = 0; t < A_SLOTS; ++t) {
            mbar_init(a_full(t), NUM_CONVERT_WARPS);
            mbar_init(a_free(t), 1);
        }
        mbar_init(d_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&maps.x);
        tma_prefetch_desc(&maps.w[prob]);
    }
    if (warp == 1) {
        tmem_alloc<NROWS>(smem_u32(const_cast<uint32_t*>(tmem_slot)));
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        uint32_t s = 0, ph = 0;
        for (uint32_t kb = kb0; kb < kb1; ++kb) {
            if (!mbar_wait_bounded(empty_bar(s), ph ^ 1u, abort_flag, p.status, SITE_EMPTY, KERNEL_DQ_GEMM))
                break;
            if (elect_one()) {
                mbar_expect_tx(full_bar(s), C::STAGE_BYTES);
                tma_load_2d(smem_base + W_REGION + s * C::W_BYTES, &maps.w[prob], full_bar(s), (int32_t)n0,
                            (int32_t)(kb * BK));
                tma_load_2d(smem_base + X_REGION + s * C::X_BYTES, &maps.x, full_bar(s), (int32_t)(kb * BK),
                            (int32_t)m0);
            }
            __syncwarp();
            if (++s == STAGES) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (*abort_flag)
            for (uint32_t spin = 0; spin < 2000; ++spin)
                __nanosleep(100);  // copies in flight land before the CTA leaves
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (converged warp)
        uint32_t s = 0, t = 0, aph = 0;
        for (uint32_t kb = kb0; kb < kb1; ++kb) {
            // a_full implies that the stage's TMA data landed: the converters waited for it
            if (!mbar_wait_bounded(a_full(t), aph, abort_flag, p.status, SITE_A_FULL, KERNEL_DQ_GEMM))
                break;
            tc_fence_after_sync();
            const uint32_t a_addr = smem_base + t * C::A_BYTES;
            const uint32_t x_addr = smem_base + X_REGION + s * C::X_BYTES;
            if (elect_one()) {
#pragma unroll
                for (uint32_t kk = 0; kk < BK / 16; ++kk)
                    umma_f16(tmem_base, make_smem_desc_sw128(a_addr + kk * 2048, BK * 128, 1024),
                             make_smem_desc_sw128(x_addr + kk * 32, 16, 1024), C::IDESC,
                             (kb != kb0 || kk != 0) ? 1u : 0u);
                umma_commit(empty_bar(s));
                umma_commit(a_free(t));
                if (kb + 1 == kb1)
                    umma_commit(d_full);
            }
            __syncwarp();
            if (++s == STAGES)
                s = 0;
            if (++t == A_SLOTS) {
                t = 0;
                aph ^= 1u;
            }
        }
    } else {
        // ------------------------------------------------------------ converters
        // warp w: k rows 8w .. 8w + 7 of a stage; lane: 16 columns (chunk lane % 8) of two rows.  The
        // upper four chunks store their odd half first: the two halves of a tile's columns lie a
        // multiple of 128 bytes apart and would meet in the same banks otherwise.
        const uint32_t cw = warp - 2, chunk = lane & 7u, odd = chunk >> 2;
        uint32_t s = 0, ph = 0, t = 0, tph = 0;
        for (uint32_t kb = kb0; kb < kb1; ++kb) {
            if (!mbar_wait_bounded(full_bar(s), ph, abort_flag, p.status, SITE_FULL, KERNEL_DQ_GEMM))
                break;
            const uint8_t* src = smem_gen + W_REGION + s * C::W_BYTES + cw * 8 * BN + lane * 16;
            uint4 raw[2];
            raw[0] = *reinterpret_cast<const uint4*>(src);
            raw[1] = *reinterpret_cast<const uint4*>(src + 4 * BN);
            if (!mbar_wait_bounded(a_free(t), tph ^ 1u, abort_flag, p.status, SITE_A_FREE, KERNEL_DQ_GEMM))
                break;
            uint8_t* dst = smem_gen + t * C::A_BYTES + odd * (BK * 128);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t row = cw * 8 + r * 4 + (lane >> 3);
                uint4 h0, h1;
                convert4(raw[r].x, h0.x, h0.y);
                convert4(raw[r].y, h0.z, h0.w);
                convert4(raw[r].z, h1.x, h1.y);
                convert4(raw[r].w, h1.z, h1.w);
                const uint32_t c0 = (chunk & 3u) * 2;
                *reinterpret_cast<uint4*>(dst + sw128_offset(row, c0 + odd)) = odd ? h1 : h0;
                *reinterpret_cast<uint4*>(dst + sw128_offset(row, c0 + (odd ^ 1u))) = odd ? h0 : h1;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(a_full(t));
            if (++s == STAGES) {
                s = 0;
                ph ^= 1u;
            }
            if (++t == A_SLOTS) {
                t = 0;
                tph ^= 1u;
            }
        }
        // ------------------------------------------------------------ the tile, as f32 [row][column]
        if (warp < 6) {
            const uint32_t q = warp & 3u, col = q * 32 + lane;
            const bool ok = mbar_wait_bounded(d_full, 0, abort_flag, p.status, SITE_D_FULL, KERNEL_DQ_GEMM);
            tc_fence_after_sync();
            if (ok) {
                // every MMA has retired, so every stage has been read: the rings are free
                float* red = reinterpret_cast<float*>(smem_gen) + col;
#pragma unroll 1
                for (uint32_t c = 0; c < NROWS / 32; ++c) {
                    if (m0 + c * 32 >= p.m)
                        break;
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(tmem_base + ((q * 32u) << 16) + c * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        red[(c * 32 + i) * BN] = __uint_as_float(r[i]);
                }
            }
            tc_fence_before_sync();
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc<NROWS>(tmem_base);
    }
    if (split > 1)
        cluster_sync_all();
    // ---------------------------------------------------------------- sum over the cluster, scale, store
    const uint32_t rows = p.m - m0 < (uint32_t)NROWS ? p.m - m0 : (uint32_t)NROWS;
    const Problem& pr = p.probs[prob];
    const uint32_t col = n0 + lane * 4;
    if (col < p.n) {  // n % 4 == 0
        const float4 sc = pr.col_scale ? *reinterpret_cast<const float4*>(pr.col_scale + col)
                                       : make_float4(pr.scale, pr.scale, pr.scale, pr.scale);
        for (uint32_t r = rank + warp * split; r < rows; r += split * (NUM_THREADS / 32)) {
            const uint32_t addr = smem_base + (r * BN + lane * 4) * 4;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (split == 1) {
                v = *reinterpret_cast<const float4*>(smem_gen + (addr - smem_base));
            } else {
                float4 part[MAX_SPLIT];
#pragma unroll
                for (uint32_t i = 0; i < MAX_SPLIT; ++i)
                    if (i < split)
                        part[i] = ld_cluster_f4(mapa_shared(addr, i));
#pragma unroll
                for (uint32_t i = 0; i < MAX_SPLIT; ++i)
                    if (i < split) {
                        v.x += part[i].x;
                        v.y += part[i].y;
                        v.z += part[i].z;
                        v.w += part[i].w;
                    }
            }
            const __half2 a = __floats2half2_rn(__fmul_rn(v.x, sc.x), __fmul_rn(v.y, sc.y));
            const __half2 b = __floats2half2_rn(__fmul_rn(v.z, sc.z), __fmul_rn(v.w, sc.w));
            uint2 o;
            o.x = *reinterpret_cast<const uint32_t*>(&a);
            o.y = *reinterpret_cast<const uint32_t*>(&b);
            *reinterpret_cast<uint2*>(pr.out + (size_t)(m0 + r) * p.n + col) = o;
        }
    }
    if (split > 1)
        cluster_sync_all();  // the other CTAs' tiles are read until here
}

template <int NROWS>
static cudaError_t launch(const TensorMaps& maps, const Params& p, uint32_t tiles, uint32_t tiles_m,
                          uint32_t split, int device, cudaStream_t stream)
{
    using C = Cfg<NROWS>;
    static bool attr_set[64] = {};
    if (!attr_set[device]) {
        const cudaError_t err = cudaFuncSetAttribute(
            w8a16_fused_kernel<NROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        if (err != cudaSuccess)
            return err;
        attr_set[device] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * split, tiles_m);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {split, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = split > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, w8a16_fused_kernel<NROWS>, maps, p, split);
}

}  // namespace w8f

bool w8a16_fused_ok(const void* x, const DqProblem* probs, int num_probs, uint32_t m, uint32_t n, uint32_t k)
{
    if (num_probs < 1 || num_probs > w8f::MAX_PROBS || n % 16 != 0 || k % 8 != 0 || (uintptr_t)x % 16 != 0)
        return false;
    if ((m + 255) / 256 > 65535)
        return false;
    for (int i = 0; i < num_probs; ++i)
        if ((uintptr_t)probs[i].w % 16 != 0 || (uintptr_t)probs[i].out % 16 != 0 ||
            (probs[i].col_scale != nullptr && (uintptr_t)probs[i].col_scale % 16 != 0))
            return false;
    return true;
}

cudaError_t launch_w8a16_fused(const DeviceCtx& ctx, const __half* x, const DqProblem* probs, int num_probs,
                               uint32_t m, uint32_t n, uint32_t k, cudaStream_t stream)
{
    using namespace w8f;
    const uint32_t nrows = m <= 32 ? 32 : (m <= 64 ? 64 : (m <= 128 ? 128 : 256));
    TensorMaps maps;
    cudaError_t err = encode_tensor_map_2d(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, k, m,
                                           (uint64_t)k * 2, BK, nrows, CU_TENSOR_MAP_SWIZZLE_128B);
    if (err != cudaSuccess)
        return err;
    Params p = {};
    for (int i = 0; i < MAX_PROBS; ++i) {
        const DqProblem& pr = probs[i < num_probs ? i : 0];
        err = encode_tensor_map_2d(&maps.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, pr.w, n, k, n, BN, BK,
                                   CU_TENSOR_MAP_SWIZZLE_NONE);
        if (err != cudaSuccess)
            return err;
        p.probs[i].col_scale = pr.col_scale;
        p.probs[i].scale = pr.scale;
        p.probs[i].out = static_cast<__half*>(pr.out);
    }
    p.m = m;
    p.n = n;
    p.num_kb = (k + BK - 1) / BK;
    p.tiles_n = (n + BN - 1) / BN;
    p.status = ctx.status;
    const uint32_t tiles = p.tiles_n * (uint32_t)num_probs, tiles_m = (m + nrows - 1) / nrows;
    // K is cut as long as all CTAs run at once (two fit an SM up to 128 rows, the 256-row form has one)
    // and keep eight K blocks each to cover the fill of their pipeline and the sum over the cluster.  us
    // for a cut in 1 / 2 / 4 / 8: 2048 x 2048, M = 64 17.3 / 12.7 / 12.1 / 17.3 (48 tiles); K x N = 4096 x
    // 4096, M = 16 27.9 / 23.2 / 24.1 / 30.0 (96 tiles), M = 256 35.9 / 46 / 49 / 89; 8192 x 1024, M = 16
    // 51 / 29 / 17 / 15 (24 tiles).  With more tiles than SMs a long K is still cut once, for the balance:
    // 8192 x 8192, M = 8 74 / 65 / 67 / 82 (192 tiles).
    const uint32_t ctas = tiles * tiles_m, slots = nrows <= 128 ? 2 * ctx.num_sms : ctx.num_sms;
    uint32_t split = 1;
    while (split < MAX_SPLIT && ctas * split * 2 <= slots && p.num_kb >= 16 * split)
        split *= 2;
    if (nrows <= 128 && split == 1 && ctas > (uint32_t)ctx.num_sms && ctas <= slots && p.num_kb >= 128)
        split = 2;
    switch (nrows) {
    case 32:
        return launch<32>(maps, p, tiles, tiles_m, split, ctx.device, stream);
    case 64:
        return launch<64>(maps, p, tiles, tiles_m, split, ctx.device, stream);
    case 128:
        return launch<128>(maps, p, tiles, tiles_m, split, ctx.device, stream);
    default:
        return launch<256>(maps, p, tiles, tiles_m, split, ctx.device, stream);
    }
}

}  // namespace kaio

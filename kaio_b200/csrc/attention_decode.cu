// Attention of ONE query row per (batch, head) over its key/value cache (decode step), head_dim 64
// or 128: out = softmax(q K^T / sqrt(d)) V, f16 in, f32 scores, probabilities and sums.
//
// What bounds it: HBM, every K and V element is read once and used once.  The tile kernel of
// flash_attention.cu carries 256 query rows per work item and would spend its tensor time and its
// score registers on 255 rows of padding, with one CTA per SM and 128 KB in flight only between
// hand-overs.  Here nothing is staged: a warp reads 16 keys (32 at head_dim 64) of K and V straight
// into registers (16 loads of 16 bytes per lane in flight), and K of the next block is requested
// before the softmax of this one.
//  * scores: mma.sync m16n8k16 with the 16 KEYS as the rows and q as column 0.  The contraction
//    index may be permuted freely as long as both operands agree, so lane (g, t) takes the 16-byte
//    chunks t, t + 4, ... of key row g: whole sectors per load and no shuffles for the dot product.
//  * P V on the CUDA cores: with one row it is 8 FMAs per 16 bytes loaded, a tenth of the time the
//    bytes take, and P stays f32.
//  * The key range of a pair is cut over the CTAs of a cluster (and over the warps of a CTA); the
//    partial (max, sum, output) meet in distributed shared memory.  No scratch buffer, no atomics,
//    so the result does not depend on arrival order and a first call may be captured in a graph.
// Measured at 8 x 32 heads, 2000 keys, d 128 (262 MB), per call: 66 us with the tile kernel (4.0 TB/s), 50.2 us here
// (5.2 TB/s of 6.54 copied); 8 heads over 8192 keys 10.8 us; head_dim 64 went to a scalar kernel before.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"
#include "mma_sync.cuh"

namespace kaio {
namespace adec {

struct Params {
    const __half *q, *k, *v;
    void* out;
    uint32_t heads, kv_end;
    uint64_t k_row, v_row;
    uint64_t q_head, k_head, v_head, o_head;
    uint64_t q_batch, k_batch, v_batch, o_batch;
    float scale_log2;
    int out_f16;
};

__device__ __forceinline__ uint4 ldg_stream(const __half* p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

template <int D, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
attention_decode_kernel(const Params p)
{
    namespace cg = cooperative_groups;
    constexpr int SUB = 128 / D;         // 16-key blocks a warp handles at a time
    constexpr int KC = D / 32;           // 16-byte chunks of a key row per lane
    constexpr int LPR = D / 8;           // lanes across a value row
    constexpr int RPL = 32 / LPR;        // value rows per load instruction
    constexpr int VL = 16 * SUB / RPL;   // value loads per lane and block (8)
    constexpr uint32_t KEYS = 16 * SUB;  // keys per block

    __shared__ float o_part[WARPS][D];
    __shared__ float ml_part[WARPS][2];
    __shared__ float o_cta[D];
    __shared__ float ml_cta[2];

    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t csize = cluster.num_blocks(), crank = cluster.block_rank();
    const uint32_t pair = blockIdx.x / csize;
    const uint32_t b = pair / p.heads, h = pair - b * p.heads;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t g = lane >> 2, t = lane & 3u;

    const __half* q = p.q + b * p.q_batch + h * p.q_head;
    const __half* kb = p.k + b * p.k_batch + h * p.k_head + t * 8;
    const __half* vb = p.v + b * p.v_batch + h * p.v_head + (lane % LPR) * 8;

    // q as the B operand: column 0 of eight, the other seven columns are zero
    uint32_t bq[KC][4];
#pragma unroll
    for (int c = 0; c < KC; ++c) {
        uint4 x = make_uint4(0, 0, 0, 0);
        if (g == 0)
            x = *reinterpret_cast<const uint4*>(q + (t + 4 * c) * 8);
        bq[c][0] = x.x;
        bq[c][1] = x.y;
        bq[c][2] = x.z;
        bq[c][3] = x.w;
    }

    const uint32_t last = p.kv_end - 1;
    const uint32_t blocks = (p.kv_end + KEYS - 1) / KEYS;
    const uint32_t step = csize * WARPS;
    uint32_t blk = crank * WARPS + warp;

    uint4 kr[SUB][2][KC];
    auto load_k = [&](uint32_t bi) {
#pragma unroll
        for (int s = 0; s < SUB; ++s)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                uint32_t key = bi * KEYS + s * 16 + r * 8 + g;
                key = key < last ? key : last;  // rows past the end repeat the last key and are masked
                const __half* row = kb + key * p.k_row;
#pragma unroll
                for (int c = 0; c < KC; ++c)
                    kr[s][r][c] = ldg_stream(row + c * 32);
            }
    };
    float m_run = -INFINITY, l_run = 0.0f;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        acc[i] = 0.0f;

    if (blk < blocks)
        load_k(blk);
    for (; blk < blocks; blk += step) {
        const uint32_t key0 = blk * KEYS;
        uint4 vr[VL];
#pragma unroll
        for (int i = 0; i < VL; ++i) {
            uint32_t key = key0 + i * RPL + lane / LPR;
            key = key < last ? key : last;
            vr[i] = ldg_stream(vb + key * p.v_row);
        }
        float s0[SUB], s1[SUB];  // scores of keys g and g + 8 (lanes with t == 0)
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
            float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < KC; ++i) {
                mma_m16n8k16_f16(c, kr[s][0][i].x, kr[s][1][i].x, kr[s][0][i].y, kr[s][1][i].y,
                                 bq[i][0], bq[i][1]);
                mma_m16n8k16_f16(c, kr[s][0][i].z, kr[s][1][i].z, kr[s][0][i].w, kr[s][1][i].w,
                                 bq[i][2], bq[i][3]);
            }
            s0[s] = key0 + s * 16 + g <= last ? c[0] * p.scale_log2 : -INFINITY;
            s1[s] = key0 + s * 16 + 8 + g <= last ? c[2] * p.scale_log2 : -INFINITY;
        }
        if (blk + step < blocks)
            load_k(blk + step);
        // only column 0 counts: lanes with t == 0 hold it, the reduction runs over g
        float mx = s0[0];
#pragma unroll
        for (int s = 0; s < SUB; ++s)
            mx = fmaxf(mx, fmaxf(s0[s], s1[s]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        mx = __shfl_sync(0xffffffffu, mx, 0);
        const float m_new = fmaxf(m_run, mx);
        const float ref = m_new == -INFINITY ? 0.0f : m_new;
        const float alpha = exp2f(m_run - ref);
        m_run = m_new;
        l_run *= alpha;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            acc[i] *= alpha;
        float p0[SUB], p1[SUB];
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
            p0[s] = exp2f(s0[s] - ref);
            p1[s] = exp2f(s1[s] - ref);
            l_run += p0[s] + p1[s];  // lanes with t == 0; summed over g at the end
        }
#pragma unroll
        for (int i = 0; i < VL; ++i) {
            // the RPL rows of a load lie in one half (8 keys) of one 16-key block
            const int key = i * RPL;
            const int s = key >> 4;
            const float src = (key & 8) ? p1[s] : p0[s];
            const float pv = __shfl_sync(0xffffffffu, src, ((key & 7) + lane / LPR) * 4);
            const bool live = key0 + key + lane / LPR <= last;
            const uint32_t w[4] = {vr[i].x, vr[i].y, vr[i].z, vr[i].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[c]));
                acc[2 * c] = live ? fmaf(pv, f.x, acc[2 * c]) : acc[2 * c];
                acc[2 * c + 1] = live ? fmaf(pv, f.y, acc[2 * c + 1]) : acc[2 * c + 1];
            }
        }
    }
    // rows of the same columns (lanes LPR apart), then warps, then CTAs of the cluster
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
        l_run += __shfl_xor_sync(0xffffffffu, l_run, o);
    if (lane < LPR) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            o_part[warp][lane * 8 + i] = acc[i];
    }
    if (lane == 0) {
        ml_part[warp][0] = m_run;
        ml_part[warp][1] = l_run;
    }
    __syncthreads();
    float m_all = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w)
        m_all = fmaxf(m_all, ml_part[w][0]);
    const float ref = m_all == -INFINITY ? 0.0f : m_all;
    if (threadIdx.x < D) {
        float o = 0.0f, l = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = exp2f(ml_part[w][0] - ref);
            o += f * o_part[w][threadIdx.x];
            l += f * ml_part[w][1];
        }
        o_cta[threadIdx.x] = o;
        if (threadIdx.x == 0) {
            ml_cta[0] = m_all;
            ml_cta[1] = l;
        }
    }
    cluster.sync();
    if (crank == 0 && threadIdx.x < D) {
        float m = -INFINITY;
        for (uint32_t r = 0; r < csize; ++r)
            m = fmaxf(m, cluster.map_shared_rank(ml_cta, r)[0]);
        const float cref = m == -INFINITY ? 0.0f : m;
        float o = 0.0f, l = 0.0f;
        for (uint32_t r = 0; r < csize; ++r) {
            const float* ml = cluster.map_shared_rank(ml_cta, r);
            const float f = exp2f(ml[0] - cref);
            o += f * cluster.map_shared_rank(o_cta, r)[threadIdx.x];
            l += f * ml[1];
        }
        o = l > 0.0f ? o / l : (l == 0.0f ? 0.0f : l);
        const size_t idx = b * p.o_batch + h * p.o_head + threadIdx.x;
        if (p.out_f16)
            reinterpret_cast<__half*>(p.out)[idx] = __float2half_rn(o);
        else
            reinterpret_cast<float*>(p.out)[idx] = o;
    }
    cluster.sync();  // the other CTAs' shared memory is read until here
}

template <int D, int WARPS>
static cudaError_t launch(const Params& p, uint32_t pairs, uint32_t csize, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pairs * csize);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {csize, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, attention_decode_kernel<D, WARPS>, p);
}

}  // namespace adec

bool attention_decode_ok(const AttnParams& p)
{
    if (p.seq_q != 1 || p.seq_k == 0 || p.d_k != p.d_v || (p.d_k != 64 && p.d_k != 128))
        return false;
    const uint64_t strides[] = {p.k_row, p.v_row, p.q_head, p.k_head, p.v_head, p.q_batch, p.k_batch,
                                p.v_batch};
    for (uint64_t s : strides)
        if (s % 8 != 0)
            return false;
    return (uintptr_t)p.q % 16 == 0 && (uintptr_t)p.k % 16 == 0 && (uintptr_t)p.v % 16 == 0 &&
           (uint64_t)p.batch * p.heads <= 0x7fffffffu / 8;
}

cudaError_t launch_attention_decode(const DeviceCtx& ctx, const AttnParams& ap, cudaStream_t stream)
{
    using namespace adec;
    Params p = {};
    p.q = ap.q;
    p.k = ap.k;
    p.v = ap.v;
    p.out = ap.out;
    p.heads = ap.heads;
    p.kv_end = ap.causal ? 1u : ap.seq_k;  // causal in absolute positions: row 0 sees key 0
    p.k_row = ap.k_row;
    p.v_row = ap.v_row;
    p.q_head = ap.q_head;
    p.k_head = ap.k_head;
    p.v_head = ap.v_head;
    p.o_head = ap.o_head;
    p.q_batch = ap.q_batch;
    p.k_batch = ap.k_batch;
    p.v_batch = ap.v_batch;
    p.o_batch = ap.o_batch;
    p.scale_log2 = 1.4426950408889634f / sqrtf((float)ap.d_k);
    p.out_f16 = ap.out_f16;
    const uint32_t pairs = ap.batch * ap.heads;
    const uint32_t keys = ap.d_k == 64 ? 32 : 16;
    const uint32_t blocks = (p.kv_end + keys - 1) / keys;
    // Four warps per CTA when the pairs alone (times a full cluster) fill the SMs' sixteen warps
    // each: many small CTAs even out the last wave.  With fewer pairs sixteen warps, so that eight
    // CTAs of a pair still keep enough loads in flight.  The cluster is as wide as there are blocks
    // for its warps.
    const bool wide = (uint64_t)pairs * 8 * 4 < (uint64_t)ctx.num_sms * 16;
    const uint32_t warps = wide ? 16 : 4;
    uint32_t csize = 1;
    while (csize < 8 && csize * warps < blocks)
        csize *= 2;
    if (ap.d_k == 64)
        return wide ? launch<64, 16>(p, pairs, csize, stream) : launch<64, 4>(p, pairs, csize, stream);
    return wide ? launch<128, 16>(p, pairs, csize, stream) : launch<128, 4>(p, pairs, csize, stream);
}

}  // namespace kaio

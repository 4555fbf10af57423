// Attention forward on warp-level MMAs (m16n8k16), head_dim 64 or 128:
//   out = softmax(Q K^T / sqrt(d) [+ causal mask j > i]) V,  f16 in, f32 or f16 out, any seq_k.
//
// It serves what the 256-row tcgen05 kernel of flash_attention.cu does not fit:
//  * head_dim 64 of any length (before: one warp per query row on the CUDA cores);
//  * a few heads of a short sequence, where that kernel runs on a handful of SMs and every one of its
//    hand-overs (TMA, tensor memory, three warp roles) is a latency nothing hides.
// What bounds it.  Short: latency, so a CTA takes only 16 query rows and its eight warps share out the
// keys, each with its own three 16-key stages all requested at once, no CTA barrier before the partial
// results are merged in shared memory.  Long, head_dim 64: the tensor pipe and the exponentials, four
// warps of 16 rows over common 64-key stages, two in flight.
// Precision: P enters the second product as hi + lo, two f16 numbers that hold 22 bits of it (scaled
// by 2^12 so that lo stays clear of f16's subnormals), because the scalar kernel kept it in f32.  Against
// 64-bit arithmetic, 2-norm over head_dim 64, f32 out: 1.3e-7 (64 keys causal) to 2.6e-7 (384 keys), the scalar
// kernel 2.2e-7 to 4.5e-7; the tcgen05 form, whose P is one f16, 1.3e-4 to 2.0e-4 at head_dim 128, here 1.5e-7 to 3.5e-7.
// Measured, us per call back to back: one head of 384 keys, d 128, causal: 12.3 (tcgen05 form) -> 8.2; d 64, one
// head of 384 keys 96 (scalar kernel, alone) -> 6.3, 8 x 32 heads of 512 causal 16.6 ms -> 65 us.
#include <cfloat>

#include "common.cuh"
#include "kernels.h"
#include "mma_sync.cuh"

namespace kaio {
namespace awarp {

constexpr float P_SCALE = 4096.0f;  // P <= 2^12

__device__ __forceinline__ void cp_async_16_zfill(uint32_t smem, const void* gmem, bool live)
{
    const uint32_t bytes = live ? 16u : 0u;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(gmem), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two f32 operations in one instruction (sm_100).
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 d;
    asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\n"
        "add.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

__device__ __forceinline__ float2 mul2(float2 a, float b)
{
    float2 d;
    asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %4};\n"
        "mul.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b));
    return d;
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\n"
        "fma.rn.f32x2 d, a, b, c;\nmov.b64 {%0, %1}, d;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// Two probabilities -> hi and lo f16 pairs.
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo)
{
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const float2 r = add2(make_float2(a, b), make_float2(-f.x, -f.y));
    const __half2 l = __floats2half2_rn(r.x, r.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// One row of the output by the plain sums, two columns: what the product of P's halves cannot give.  An
// infinite value meets lo halves that are negative or zero, and, in its stage, masked keys of weight zero.
template <int D>
__device__ __forceinline__ float2 plain_output(const __half* q, const __half* k, uint64_t k_row, const __half* v,
                                               uint64_t v_row, uint32_t keys, float scale_log2, float m, float l)
{
    float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (uint32_t j = 0; j < keys; ++j, k += k_row, v += v_row) {
        float dot = 0.0f;
#pragma unroll 1
        for (int d = 0; d < D; d += 2) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(q + d));
            const float2 b = __half22float2(*reinterpret_cast<const __half2*>(k + d));
            dot = fmaf(a.x, b.x, fmaf(a.y, b.y, dot));
        }
        const float w = P_SCALE * ex2((dot - m) * scale_log2);
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(v));
        sum.x = fmaf(w, f.x, sum.x);
        sum.y = fmaf(w, f.y, sum.y);
    }
    return make_float2(sum.x / l, sum.y / l);
}

// QW warps along the query rows (16 each), KW groups of them along the keys, BKV keys per stage, ST
// stages per group.
template <int D, int QW, int KW, int BKV, int ST>
struct Cfg {
    static constexpr int ROWS = QW * 16;
    static constexpr int THREADS = QW * KW * 32;
    static constexpr int ROW_BYTES = D * 2;
    static constexpr int TILE_BYTES = BKV * ROW_BYTES;  // K or V of one stage
    static constexpr int RING_BYTES = KW * ST * 2 * TILE_BYTES;
    static constexpr int MERGE_BYTES = KW > 1 ? KW * (16 * (D + 4) * 4 + 16 * 8) : 0;
    static constexpr int SMEM_BYTES = RING_BYTES > MERGE_BYTES ? RING_BYTES : MERGE_BYTES;
    static_assert(QW == 1 || KW == 1, "one of the two splits");
    static_assert(SMEM_BYTES <= 227 * 1024, "stages do not fit");
};

template <int D, int QW, int KW, int BKV, int ST>
__global__ void __launch_bounds__(QW* KW * 32) attention_warp_kernel(const AttnParams p, const float scale_log2)
{
    using C = Cfg<D, QW, KW, BKV, ST>;
    constexpr int CHUNKS = D / 8;  // 16-byte chunks of a row
    constexpr int NS = BKV / 8;    // score fragments (8 keys each)
    constexpr int NO = D / 8;      // output fragments (8 columns each)
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t qw = QW > 1 ? warp : 0u, kw = KW > 1 ? warp : 0u;
    const uint32_t b = blockIdx.y / p.heads, h = blockIdx.y - b * p.heads;
    // heaviest (causal) row blocks first
    const uint32_t q0 = (gridDim.x - 1 - blockIdx.x) * C::ROWS;
    const uint32_t row0 = q0 + qw * 16 + g, row1 = row0 + 8;

    const __half* kbase = p.k + b * p.k_batch + h * p.k_head;
    const __half* vbase = p.v + b * p.v_batch + h * p.v_head;
    uint32_t kv_end = p.seq_k;
    if (p.causal && q0 + C::ROWS < kv_end)
        kv_end = q0 + C::ROWS;
    const uint32_t blocks = (kv_end + BKV - 1) / BKV;

    const uint32_t ring = smem_u32(smem) + kw * (ST * 2 * C::TILE_BYTES);
    const uint32_t gtid = QW > 1 ? threadIdx.x : lane;  // thread inside the group
    auto fetch = [&](uint32_t blk, uint32_t slot) {
        if (blk < blocks) {
            const uint32_t kt = ring + slot * 2 * C::TILE_BYTES;
#pragma unroll
            for (uint32_t i = gtid; i < (uint32_t)(BKV * CHUNKS); i += QW * 32) {
                const uint32_t r = i / CHUNKS, c = i % CHUNKS;
                const uint32_t key = blk * BKV + r;
                const bool live = key < p.seq_k;
                const uint32_t src = live ? key : 0u;
                const uint32_t off = r * C::ROW_BYTES + ((c ^ (r & 7u)) << 4);
                cp_async_16_zfill(kt + off, kbase + src * p.k_row + c * 8, live);
                cp_async_16_zfill(kt + C::TILE_BYTES + off, vbase + src * p.v_row + c * 8, live);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto group_sync = [&]() {
        if (QW > 1)
            __syncthreads();
        else
            __syncwarp();
    };
#pragma unroll
    for (int s = 0; s < ST; ++s)
        fetch(kw + s * KW, s);

    // Q as the A operand, straight from global memory
    uint32_t qa[D / 16][4];
    {
        const __half* qb = p.q + b * p.q_batch + h * p.q_head + 2 * t;
        const __half* r0 = qb + (row0 < p.seq_q ? row0 : 0u) * p.q_row;
        const __half* r1 = qb + (row1 < p.seq_q ? row1 : 0u) * p.q_row;
#pragma unroll
        for (int c = 0; c < D / 16; ++c) {
            qa[c][0] = *reinterpret_cast<const uint32_t*>(r0 + c * 16);
            qa[c][1] = *reinterpret_cast<const uint32_t*>(r1 + c * 16);
            qa[c][2] = *reinterpret_cast<const uint32_t*>(r0 + c * 16 + 8);
            qa[c][3] = *reinterpret_cast<const uint32_t*>(r1 + c * 16 + 8);
        }
    }

    float o[NO][4];
#pragma unroll
    for (int i = 0; i < NO; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            o[i][j] = 0.0f;
    float m0 = -INFINITY, m1 = -INFINITY;  // largest raw score q.k of the row
    float2 l0 = make_float2(0.0f, 0.0f), l1 = l0;

    // ldmatrix row addresses of this lane: K: matrices (keys 0-7, d 0-7) (keys 0-7, d 8-15) (keys 8-15,
    // d 0-7) (keys 8-15, d 8-15); V, transposed: (keys 0-7, d 0-7) (keys 8-15, d 0-7) (keys 0-7,
    // d 8-15) (keys 8-15, d 8-15)
    const uint32_t k_row = (lane & 7u) + ((lane >> 4) << 3), k_chunk = (lane >> 3) & 1u;
    const uint32_t v_row = lane & 15u, v_chunk = lane >> 4;

    uint32_t slot = 0;
    for (uint32_t blk = kw; blk < blocks; blk += KW) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 1) : "memory");
        group_sync();
        const uint32_t kt = ring + slot * 2 * C::TILE_BYTES, vt = kt + C::TILE_BYTES;

        float s[NS][4];
#pragma unroll
        for (int i = 0; i < NS; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                s[i][j] = 0.0f;
#pragma unroll
        for (int c = 0; c < D / 16; ++c)
#pragma unroll
            for (int i = 0; i < NS / 2; ++i) {
                const uint32_t r = i * 16 + k_row;
                uint32_t f[4];
                ldmatrix_x4(f, kt + r * C::ROW_BYTES + (((2 * c + k_chunk) ^ (r & 7u)) << 4));
                mma_m16n8k16_f16(s[2 * i], qa[c][0], qa[c][1], qa[c][2], qa[c][3], f[0], f[1]);
                mma_m16n8k16_f16(s[2 * i + 1], qa[c][0], qa[c][1], qa[c][2], qa[c][3], f[2], f[3]);
            }
        const uint32_t key0 = blk * BKV;
        if (key0 + BKV > p.seq_k || (p.causal && key0 + BKV > q0 + qw * 16 + 1)) {
            const uint32_t lim0 = p.causal && row0 + 1 < p.seq_k ? row0 + 1 : p.seq_k;
            const uint32_t lim1 = p.causal && row1 + 1 < p.seq_k ? row1 + 1 : p.seq_k;
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                const uint32_t key = key0 + i * 8 + 2 * t;
                if (key >= lim0)
                    s[i][0] = -INFINITY;
                if (key + 1 >= lim0)
                    s[i][1] = -INFINITY;
                if (key >= lim1)
                    s[i][2] = -INFINITY;
                if (key + 1 >= lim1)
                    s[i][3] = -INFINITY;
            }
        }
        float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            x0 = fmaxf(x0, fmaxf(s[i][0], s[i][1]));
            x1 = fmaxf(x1, fmaxf(s[i][2], s[i][3]));
        }
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) {
            x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, d));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, d));
        }
        // P = 2^((s - m) scale) from the difference of the raw scores: it is exact where P is large, whatever
        // their size.  With s * scale - n, n the rounded maximum, the exponent was off by the rounding of n:
        // 2^-21 of P at best, and NaN or nothing from maxima of 2^25 on.
        x0 = fmaxf(m0, x0);
        x1 = fmaxf(m1, x1);
        const float ref0 = x0 == -INFINITY ? 0.0f : x0, ref1 = x1 == -INFINITY ? 0.0f : x1;
        const float al0 = ex2((m0 - ref0) * scale_log2), al1 = ex2((m1 - ref1) * scale_log2);
        m0 = x0;
        m1 = x1;
        l0 = mul2(l0, al0);
        l1 = mul2(l1, al1);
#pragma unroll
        for (int i = 0; i < NO; ++i) {
            const float2 u = mul2(make_float2(o[i][0], o[i][1]), al0);
            const float2 v = mul2(make_float2(o[i][2], o[i][3]), al1);
            o[i][0] = u.x;
            o[i][1] = u.y;
            o[i][2] = v.x;
            o[i][3] = v.y;
        }
        auto prob2 = [&](float& a, float& b, float ref, float2& l) {
            const float2 e = mul2(add2(make_float2(a, b), make_float2(-ref, -ref)), scale_log2);
            const float2 pr = mul2(make_float2(ex2(e.x), ex2(e.y)), P_SCALE);
            l = add2(l, pr);
            a = pr.x;
            b = pr.y;
        };
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            prob2(s[i][0], s[i][1], ref0, l0);
            prob2(s[i][2], s[i][3], ref1, l1);
        }
#pragma unroll
        for (int i = 0; i < NS / 2; ++i) {
            uint32_t ph[4], pl[4];
            split2(s[2 * i][0], s[2 * i][1], ph[0], pl[0]);
            split2(s[2 * i][2], s[2 * i][3], ph[1], pl[1]);
            split2(s[2 * i + 1][0], s[2 * i + 1][1], ph[2], pl[2]);
            split2(s[2 * i + 1][2], s[2 * i + 1][3], ph[3], pl[3]);
            const uint32_t r = i * 16 + v_row;
#pragma unroll
            for (int c = 0; c < NO / 2; ++c) {
                uint32_t f[4];
                ldmatrix_x4_trans(f, vt + r * C::ROW_BYTES + (((2 * c + v_chunk) ^ (r & 7u)) << 4));
                mma_m16n8k16_f16(o[2 * c], pl[0], pl[1], pl[2], pl[3], f[0], f[1]);
                mma_m16n8k16_f16(o[2 * c + 1], pl[0], pl[1], pl[2], pl[3], f[2], f[3]);
                mma_m16n8k16_f16(o[2 * c], ph[0], ph[1], ph[2], ph[3], f[0], f[1]);
                mma_m16n8k16_f16(o[2 * c + 1], ph[0], ph[1], ph[2], ph[3], f[2], f[3]);
            }
        }
        group_sync();  // the stage has been read
        fetch(blk + ST * KW, slot);
        slot = slot + 1 == ST ? 0 : slot + 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float sum0 = l0.x + l0.y, sum1 = l1.x + l1.y;
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        sum0 += __shfl_xor_sync(0xffffffffu, sum0, d);
        sum1 += __shfl_xor_sync(0xffffffffu, sum1, d);
    }
    auto inverse = [](float l) { return l > 0.0f ? 1.0f / l : 0.0f; };
    // not finite although the row's scores were (l is)
    auto lost = [](float x, float l) { return !(fabsf(x) <= FLT_MAX) && l > 0.0f && l <= FLT_MAX; };
    auto plain2 = [&](uint32_t row, uint32_t col, float m, float l) {
        return plain_output<D>(p.q + b * p.q_batch + h * p.q_head + row * p.q_row, kbase, p.k_row, vbase + col,
                               p.v_row, p.causal && row + 1 < p.seq_k ? row + 1 : p.seq_k, scale_log2, m, l);
    };
    auto store2 = [&](uint32_t row, uint32_t col, float x, float y) {
        const size_t idx = b * p.o_batch + h * p.o_head + (size_t)row * p.o_row + col;
        if (p.out_f16)
            *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(p.out) + idx) = __floats2half2_rn(x, y);
        else
            *reinterpret_cast<float2*>(reinterpret_cast<float*>(p.out) + idx) = make_float2(x, y);
    };
    if (KW == 1) {
        const float i0 = inverse(sum0), i1 = inverse(sum1);
#pragma unroll
        for (int i = 0; i < NO; ++i) {
            if (row0 < p.seq_q)
                store2(row0, i * 8 + 2 * t, o[i][0] * i0, o[i][1] * i0);
            if (row1 < p.seq_q)
                store2(row1, i * 8 + 2 * t, o[i][2] * i1, o[i][3] * i1);
        }
        float2 za = make_float2(0.0f, 0.0f), zb = za;  // NaN if an output of the row is not finite
#pragma unroll
        for (int i = 0; i < NO; ++i) {
            za = fma2(make_float2(o[i][0], o[i][1]), make_float2(0.0f, 0.0f), za);
            zb = fma2(make_float2(o[i][2], o[i][3]), make_float2(0.0f, 0.0f), zb);
        }
        const float z0 = za.x + za.y, z1 = zb.x + zb.y;
        if (lost(z0, sum0) || lost(z1, sum1)) {
#pragma unroll 1
            for (uint32_t i = 0; i < 2 * NO; ++i) {
                const bool upper = i >= NO;
                const uint32_t row = upper ? row1 : row0, col = (upper ? i - NO : i) * 8 + 2 * t;
                if (row < p.seq_q && lost(upper ? z1 : z0, upper ? sum1 : sum0)) {
                    const float2 v = plain2(row, col, upper ? m1 : m0, upper ? sum1 : sum0);
                    store2(row, col, v.x, v.y);
                }
            }
        }
    } else {
        // ---- the groups' partial results, in ascending group order
        constexpr uint32_t PITCH = D + 4;
        float* part = reinterpret_cast<float*>(smem);      // [KW][16][PITCH]
        float* ml = part + KW * 16 * PITCH;                // [KW][16][2]
        __syncthreads();  // every group is done with its stages
#pragma unroll
        for (int i = 0; i < NO; ++i) {
            *reinterpret_cast<float2*>(part + (kw * 16 + g) * PITCH + i * 8 + 2 * t) =
                make_float2(o[i][0], o[i][1]);
            *reinterpret_cast<float2*>(part + (kw * 16 + g + 8) * PITCH + i * 8 + 2 * t) =
                make_float2(o[i][2], o[i][3]);
        }
        if (t == 0) {
            ml[(kw * 16 + g) * 2] = m0;
            ml[(kw * 16 + g) * 2 + 1] = sum0;
            ml[(kw * 16 + g + 8) * 2] = m1;
            ml[(kw * 16 + g + 8) * 2 + 1] = sum1;
        }
        __syncthreads();
        // outputs (row, col) and (row, col + 1) of the CTA's 16 rows
        auto merged = [&](uint32_t row, uint32_t col, float& m, float& l) {
            m = -INFINITY;
#pragma unroll
            for (int w = 0; w < KW; ++w)
                m = fmaxf(m, ml[(w * 16 + row) * 2]);
            const float ref = m == -INFINITY ? 0.0f : m;
            float x = 0.0f, y = 0.0f;
            l = 0.0f;
#pragma unroll
            for (int w = 0; w < KW; ++w) {
                const float f = ex2((ml[(w * 16 + row) * 2] - ref) * scale_log2);
                const float2 v = *reinterpret_cast<const float2*>(part + (w * 16 + row) * PITCH + col);
                l += f * ml[(w * 16 + row) * 2 + 1];
                x += f * v.x;
                y += f * v.y;
            }
            const float inv = inverse(l);
            return make_float2(x * inv, y * inv);
        };
        constexpr uint32_t PAIRS = 16 * D / 2;
        bool any_lost = false;
        float m, l;
#pragma unroll
        for (uint32_t i = threadIdx.x; i < PAIRS; i += C::THREADS) {
            const uint32_t r = i / (D / 2), c = (i % (D / 2)) * 2;
            const float2 v = merged(r, c, m, l);
            any_lost |= lost(v.x + v.y, l);
            if (q0 + r < p.seq_q)
                store2(q0 + r, c, v.x, v.y);
        }
        if (any_lost) {
#pragma unroll 1
            for (uint32_t i = threadIdx.x; i < PAIRS; i += C::THREADS) {
                const uint32_t r = i / (D / 2), c = (i % (D / 2)) * 2;
                const float2 v = merged(r, c, m, l);
                if (q0 + r < p.seq_q && lost(v.x + v.y, l)) {
                    const float2 w = plain2(q0 + r, c, m, l);
                    store2(q0 + r, c, w.x, w.y);
                }
            }
        }
    }
}

template <int D, int QW, int KW, int BKV, int ST>
static cudaError_t launch(const AttnParams& p, int device, cudaStream_t stream)
{
    using C = Cfg<D, QW, KW, BKV, ST>;
    auto kernel = attention_warp_kernel<D, QW, KW, BKV, ST>;
    static bool attr_set[64] = {};
    if (!attr_set[device]) {
        const cudaError_t err =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        if (err != cudaSuccess)
            return err;
        attr_set[device] = true;
    }
    const float scale_log2 = 1.4426950408889634f / sqrtf((float)D);
    kernel<<<dim3((p.seq_q + C::ROWS - 1) / C::ROWS, p.batch * p.heads), C::THREADS, C::SMEM_BYTES, stream>>>(
        p, scale_log2);
    return cudaGetLastError();
}

// 16-row CTAs with the keys shared out over eight warps: while they all fit the SMs at once and a
// warp has three stages of 16 keys at most.
static bool short_form(const DeviceCtx& ctx, const AttnParams& p)
{
    return p.seq_k <= 384 && (uint64_t)p.batch * p.heads * ((p.seq_q + 15) / 16) <= (uint64_t)ctx.num_sms;
}

}  // namespace awarp

bool attention_warp_ok(const DeviceCtx& ctx, const AttnParams& p)
{
    if (p.d_k != p.d_v || (p.d_k != 64 && p.d_k != 128) || p.seq_k == 0)
        return false;
    if (p.d_k == 128 && !awarp::short_form(ctx, p))
        return false;  // flash_attention.cu's, or the scalar kernel's where TMA cannot read the operands
    const uint64_t k_strides[] = {p.k_row, p.v_row, p.k_head, p.v_head, p.k_batch, p.v_batch};
    for (uint64_t s : k_strides)
        if (s % 8 != 0)
            return false;
    const uint64_t qo_strides[] = {p.q_row, p.o_row, p.q_head, p.o_head, p.q_batch, p.o_batch};
    for (uint64_t s : qo_strides)
        if (s % 2 != 0)
            return false;
    return (uintptr_t)p.k % 16 == 0 && (uintptr_t)p.v % 16 == 0 && (uintptr_t)p.q % 4 == 0 &&
           (uintptr_t)p.out % (p.out_f16 ? 4 : 8) == 0 && (uint64_t)p.batch * p.heads <= 65535;
}

cudaError_t launch_attention_warp(const DeviceCtx& ctx, const AttnParams& p, cudaStream_t stream)
{
    using namespace awarp;
    if (short_form(ctx, p))
        return p.d_k == 64 ? launch<64, 1, 8, 16, 3>(p, ctx.device, stream)
                           : launch<128, 1, 8, 16, 3>(p, ctx.device, stream);
    return launch<64, 4, 1, 64, 2>(p, ctx.device, stream);
}

}  // namespace kaio

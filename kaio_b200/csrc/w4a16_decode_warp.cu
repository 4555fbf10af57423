// W4A16 GEMM for decode, M <= 16:  C[M, N] = A[M, K] f16  x  dequant(B)[K, N], for one weight matrix
// or three that share A (the fused QKV projection).
// B is the reference's packed layout (kaio-ops/src/matmul_int4_kernel.rs:5-13): word k/8 of column j
// at (k/8) + j*(K/8), nibble k%8 at bits [4(k%8), +4); scales f16 [K/128, N].
//
// What bounds it: HBM, K*N/2 bytes of weights read once (a kernel that only copies them to shared
// memory takes 7.2 us for 22.5 MB and 21 us for 117 MB).  The product is thin, and every hand-over
// between a loader, a dequantiser and an MMA issuer costs more than the arithmetic it separates: the
// tcgen05 form (w4a16_decode.cu) needs 15.3 us for the first and 41-43 us for the second.  Here a warp
// does all three by itself, without a barrier in its loop:
//  * The transposed product on mma.sync m16n8k16: 16 weight columns are the rows of the instruction,
//    the activations its 8 columns (two groups of them for M > 8).  The contraction index may be
//    permuted freely when both operands agree, so lane (g, t) owns the 16 bytes (four words, 32 k)
//    number t of columns g and g + 8: 128 k = one scale group of a column are 64 contiguous bytes
//    over four lanes, and the words become MMA fragments in place, without a shuffle.
//  * A lane copies its own bytes with cp.async into its own slots (eight per warp, 1 KB each) and is
//    the only one to read them back: the wait for the oldest copy is the only synchronisation, and
//    56 KB per CTA, 112 KB per SM, are in flight all the time.
//  * Dequantisation keeps the reference's rounding, f16(q) * f16(scale) in f16: one LOP3 makes two
//    nibbles the exact f16 numbers 1024 + 16^i (q + 8), one HADD2 / HFMA2 the integers, one HMUL2 the
//    scaled weights: 13 instructions per word of 8 weights.
//  * The walks over the units only add to pointers inside a tile: with the position of every copy,
//    scale and activation computed from the unit's number the loop had 27 instructions per word.
// A unit = a column tile (16 * TC columns) x 128 k.  The units of all tiles are cut into one
// contiguous range per CTA (two CTAs per SM) and dealt to its eight warps in turn; a tile's partial
// sums meet in shared memory, and where a range ends inside a tile the CTAs park f32 partials that
// the last one to arrive adds in ascending CTA order (deterministic; no float atomics).
// Programmatic dependent launch: what runs before griddepcontrol.wait reads only weights and scales, and of
// three matrices not even these.  The early reads save 0.5 to 1 us where calls follow each other (13.2 against
// 14.2 us for three of 4096 x 4096 at M = 8), but weights or scales that the kernel in front writes would be
// read too early if it lets its dependents start; a fused QKV call never asked its callers to mind that.
// Measured (us per call back to back, tcgen05 form -> this one), M = 1, K x N: 1024 x 1024 7.6 -> 2.9, 4096 x 4096
// 13.3 -> 8.2, 4096 x 11008 15.4 -> 11.7, 8192 x 28672 41 -> 34 (3.5 TB/s); three 4096 x 4096 matrices at M = 8 63 (f16
// copy of the weights, then a GEMM) -> 14.2.  At M = 1, 4096 x 11008: 30 instructions per word at 0.39 per cycle and
// scheduler, no pipe above 28 %: four warps per scheduler do not cover the latencies of the chain.
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "mma_sync.cuh"

namespace kaio {
namespace w4dw {

constexpr uint32_t WARPS = 8;
constexpr uint32_t NUM_THREADS = WARPS * 32;
constexpr uint32_t CTAS_PER_SM = 2;
constexpr uint32_t UNIT_K = 128;      // = the scale group
constexpr uint32_t SLOTS = 8;         // 1 KB each: 16 columns x 128 k
constexpr uint32_t RING_BYTES = WARPS * SLOTS * 1024;
constexpr uint32_t MAX_ROWS = 16;
constexpr uint32_t MIN_TILE = 32;     // narrowest column tile
constexpr uint32_t MAX_TILE = 64;

// columns of a tile, padded so that the lanes of a fragment store hit 32 different banks
__host__ __device__ constexpr uint32_t red_pitch(uint32_t tc) { return tc * 16 + 4; }
__host__ __device__ constexpr uint32_t smem_bytes(uint32_t tc, uint32_t nb)
{
    return RING_BYTES + WARPS * nb * 8 * red_pitch(tc) * 4 + 16;
}

struct Params {
    const uint32_t* w[3];
    const __half* scales[3];
    void* out[8];  // one weight matrix: the copies; three: their outputs
    const __half* x;
    float* partials;
    uint32_t* counters;
    uint32_t copies;        // destinations of the one output
    uint32_t scatter_cols;
    uint64_t ld;
    uint32_t m, n, k;
    uint32_t num_kb;        // units per tile
    uint32_t tiles;         // per weight matrix
    uint32_t per_cta, rem;  // units of all matrices = gridDim.x * per_cta + rem
    bool weights_wait;      // weights and scales are read only behind the launch in front
};

// CTA c's range of units: `rem` CTAs of per_cta + 1 units, then CTAs of per_cta.  (With the ranges as
// 64-bit quotients the divisions alone were a third of the way from the last unit to the output.)
__device__ __forceinline__ uint32_t range_begin(uint32_t cta, const Params& p)
{
    return cta * p.per_cta + (cta < p.rem ? cta : p.rem);
}

// The CTA whose range holds unit u.
__device__ __forceinline__ uint32_t owner_of(uint32_t u, const Params& p)
{
    const uint32_t big = p.rem * (p.per_cta + 1);
    return u < big ? u / (p.per_cta + 1) : p.rem + (u - big) / p.per_cta;
}

__device__ __forceinline__ void cp_async_16(uint32_t smem, const void* gmem)
{
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}

__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Not a read-only (nc) load: the compiler may move such a one over the wait for the launch in front.
__device__ __forceinline__ uint32_t load_scale(const unsigned short* p)
{
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return v;
}

// (w & mask) ^ flip in one instruction
__device__ __forceinline__ __half2 and_xor(uint32_t w, uint32_t mask, uint32_t flip)
{
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(r) : "r"(w), "r"(mask), "r"(flip));
    return *reinterpret_cast<__half2*>(&r);
}

// (The conversion by exponent bits is the published one of Kim et al., "Who Says Elephants Can't Run", 2022.)
// Eight signed nibbles -> f16(q) * scale, rounded to f16, as the pairs (0,4) (1,5) (2,6) (3,7).  The
// flipped sign bit makes a nibble q + 8; under the exponent of 1024 it is 1024 + (q + 8), or
// 1024 + 16 (q + 8) where it sits four bits up.
__device__ __forceinline__ void dequant_word(uint32_t w, __half2 scale, uint32_t (&r)[4])
{
    const __half2 bias = __half2half2(__ushort_as_half(0x6408));         // 1032
    const __half2 sixteenth = __half2half2(__ushort_as_half(0x2c00));    // 1/16
    const __half2 bias16 = __half2half2(__ushort_as_half(0xd480));       // -72
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const __half2 lo = __hmul2(__hsub2(and_xor(w, 0x000f000fu, 0x64086408u), bias), scale);
        const __half2 hi =
            __hmul2(__hfma2(and_xor(w, 0x00f000f0u, 0x64806480u), sixteenth, bias16), scale);
        r[2 * i] = *reinterpret_cast<const uint32_t*>(&lo);
        r[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&hi);
        w >>= 8;
    }
}

template <int TC, int NB, bool OUT_F16>
__global__ void __launch_bounds__(NUM_THREADS, CTAS_PER_SM) w4a16_decode_warp_kernel(const Params p)
{
    constexpr uint32_t TILE = TC * 16;
    constexpr uint32_t ROWS = NB * 8;
    constexpr uint32_t PITCH = red_pitch(TC);
    constexpr uint32_t AHEAD = SLOTS / TC;  // units in flight
    constexpr bool PREFETCH_X = NB == 1;    // 16 registers; with NB == 2 the other warps cover the wait
    extern __shared__ __align__(16) uint8_t smem[];
    float* red = reinterpret_cast<float*>(smem + RING_BYTES);
    volatile uint32_t* last_flag =
        reinterpret_cast<volatile uint32_t*>(smem + RING_BYTES + WARPS * ROWS * PITCH * 4);

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t u_begin = range_begin(blockIdx.x, p);
    const uint32_t u_end = range_begin(blockIdx.x + 1, p);
    const size_t col_bytes = p.k / 2;
    // this lane's part of slot 0: column g's bytes in the first half, column g + 8's in the second
    uint8_t* my_slots = smem + warp * SLOTS * 1024 + lane * 16;
    const uint32_t my_slots_u32 = smem_u32(my_slots);
    auto prob_of = [&](uint32_t tile) { return (tile >= p.tiles ? 1u : 0u) + (tile >= 2 * p.tiles ? 1u : 0u); };
    // bit j: this lane's column of half-sub-tile j (8 columns each) exists.  What does not is neither
    // copied nor scaled: it stays in its own row of the product and is not stored.
    auto live_mask = [&](uint32_t col0) {
        const uint32_t first = col0 + g;
        const uint32_t cnt = first < p.n ? (p.n - first + 7) / 8 : 0u;
        return cnt >= 2 * TC ? (1u << (2 * TC)) - 1u : (1u << cnt) - 1u;
    };

    // Two walks over this warp's units, a few units apart from each other: copies, and scales and
    // activations.  Inside a tile they only add to their pointers.
    uint32_t u = u_begin + warp;
    const uint32_t tile0 = u / p.num_kb, kb0 = u - tile0 * p.num_kb;

    uint32_t a_u = u, a_tile = tile0, a_kb = kb0, a_mask = 0;
    const uint8_t* a_ptr = nullptr;
    auto a_setup = [&]() {
        const uint32_t prob = prob_of(a_tile), col0 = (a_tile - prob * p.tiles) * TILE;
        a_mask = live_mask(col0);
        a_ptr = reinterpret_cast<const uint8_t*>(p.w[prob]) + (col0 + g) * col_bytes +
                (size_t)a_kb * (UNIT_K / 2) + t * 16;
    };
    auto a_advance = [&]() {
        a_u += WARPS;
        a_kb += WARPS;
        a_ptr += WARPS * (UNIT_K / 2);
        if (a_kb >= p.num_kb && a_u < u_end) {
            do {
                a_kb -= p.num_kb;
                ++a_tile;
            } while (a_kb >= p.num_kb);
            a_setup();
        }
    };
    // one sub-tile's copy into a slot; an empty group at the end keeps the count of pending groups
    auto fetch = [&](uint32_t c, uint32_t slot) {
        if (a_u < u_end) {
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half)
                if (a_mask >> (2 * c + half) & 1u)
                    cp_async_16(my_slots_u32 + slot * 1024 + half * 512,
                                a_ptr + (2 * c + half) * 8 * col_bytes);
        }
        cp_async_commit();
    };

    uint32_t n_u = u, n_tile = tile0, n_kb = kb0, n_mask = 0;
    const unsigned short* n_scale = nullptr;
    const __half* n_x = nullptr;
    auto n_setup = [&]() {
        const uint32_t prob = prob_of(n_tile), col0 = (n_tile - prob * p.tiles) * TILE;
        n_mask = live_mask(col0);
        n_scale = reinterpret_cast<const unsigned short*>(p.scales[prob]) + (size_t)n_kb * p.n + col0 + g;
        n_x = p.x + (size_t)g * p.k + (size_t)n_kb * UNIT_K + t * 32;
    };
    auto n_advance = [&]() {
        n_u += WARPS;
        n_kb += WARPS;
        n_scale += (size_t)WARPS * p.n;
        n_x += WARPS * UNIT_K;
        if (n_kb >= p.num_kb && n_u < u_end) {
            do {
                n_kb -= p.num_kb;
                ++n_tile;
            } while (n_kb >= p.num_kb);
            n_setup();
        }
    };
    uint32_t sc[2 * TC];
    auto fetch_scales = [&]() {
#pragma unroll
        for (int j = 0; j < 2 * TC; ++j)
            sc[j] = (n_mask >> j & 1u) ? load_scale(n_scale + j * 8) : 0u;
    };
    uint4 xr[NB][4];  // row g (and g + 8): the 32 k of this lane
    auto fetch_x = [&]() {
#pragma unroll
        for (int r = 0; r < NB; ++r) {
            const uint4* src = reinterpret_cast<const uint4*>(n_x + (size_t)r * 8 * p.k);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                xr[r][i] = r * 8 + g < p.m ? src[i] : make_uint4(0, 0, 0, 0);
        }
    };

    if (u < u_end) {
        a_setup();
        n_setup();
    }
    if (p.weights_wait)
        asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (uint32_t i = 0; i < AHEAD; ++i) {
#pragma unroll
        for (uint32_t c = 0; c < TC; ++c)
            fetch(c, i * TC + c);
        a_advance();
    }
    if (u < u_end)
        fetch_scales();
    // activations, scratch and outputs belong to the launch in front until it is done
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (PREFETCH_X && u < u_end)
        fetch_x();

    uint32_t ring = 0;  // first slot of the current unit
    for (uint32_t seg = u_begin; seg < u_end;) {
        const uint32_t tile = seg / p.num_kb;
        const uint32_t tile_end = (tile + 1) * p.num_kb;
        const uint32_t seg_end = tile_end < u_end ? tile_end : u_end;
        float acc[TC][NB][4];
#pragma unroll
        for (int c = 0; c < TC; ++c)
#pragma unroll
            for (int r = 0; r < NB; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    acc[c][r][i] = 0.0f;

        for (; u < seg_end; u += WARPS) {
            if (!PREFETCH_X)
                fetch_x();
            // pair the activations' k as dequant_word pairs the weights'
            uint32_t xb[NB][4][4];
#pragma unroll
            for (int r = 0; r < NB; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    xb[r][i][0] = __byte_perm(xr[r][i].x, xr[r][i].z, 0x5410);
                    xb[r][i][1] = __byte_perm(xr[r][i].x, xr[r][i].z, 0x7632);
                    xb[r][i][2] = __byte_perm(xr[r][i].y, xr[r][i].w, 0x5410);
                    xb[r][i][3] = __byte_perm(xr[r][i].y, xr[r][i].w, 0x7632);
                }
            uint32_t s2[2 * TC];
#pragma unroll
            for (int j = 0; j < 2 * TC; ++j)
                s2[j] = __byte_perm(sc[j], 0, 0x1010);
            n_advance();
            if (n_u < u_end) {
                fetch_scales();
                if (PREFETCH_X)
                    fetch_x();
            }
#pragma unroll
            for (int c = 0; c < TC; ++c) {
                cp_async_wait<(int)SLOTS - 1>();  // the oldest copy is in, seven stay in flight
                const uint4 wl = *reinterpret_cast<const uint4*>(my_slots + (ring + c) * 1024);
                const uint4 wh = *reinterpret_cast<const uint4*>(my_slots + (ring + c) * 1024 + 512);
                const __half2 sl = *reinterpret_cast<const __half2*>(&s2[2 * c]);
                const __half2 sh = *reinterpret_cast<const __half2*>(&s2[2 * c + 1]);
                const uint32_t lo[4] = {wl.x, wl.y, wl.z, wl.w};
                const uint32_t hi[4] = {wh.x, wh.y, wh.z, wh.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t a[4], b[4];
                    dequant_word(lo[i], sl, a);
                    dequant_word(hi[i], sh, b);
#pragma unroll
                    for (int r = 0; r < NB; ++r)
                        mma_m16n8k16_f16(acc[c][r], a[0], b[0], a[1], b[1], xb[r][i][0], xb[r][i][1]);
#pragma unroll
                    for (int r = 0; r < NB; ++r)
                        mma_m16n8k16_f16(acc[c][r], a[2], b[2], a[3], b[3], xb[r][i][2], xb[r][i][3]);
                }
                fetch(c, ring + c);
            }
            a_advance();
            ring = (ring + TC) & (SLOTS - 1);
        }

        // ---- the warps' sums of this tile meet in shared memory, as [row][column]
        __syncthreads();  // the previous tile's sums have been read
#pragma unroll
        for (int c = 0; c < TC; ++c)
#pragma unroll
            for (int r = 0; r < NB; ++r) {
                float* d = red + (warp * ROWS + r * 8 + 2 * t) * PITCH + c * 16 + g;
                d[0] = acc[c][r][0];
                d[PITCH] = acc[c][r][1];
                d[8] = acc[c][r][2];
                d[PITCH + 8] = acc[c][r][3];
            }
        __syncthreads();
        const bool complete = seg == tile * p.num_kb && seg_end == tile_end;
        constexpr uint32_t QUADS = ROWS * TILE / 4;  // at most one per thread
        const uint32_t row = threadIdx.x / (TILE / 4), cq = (threadIdx.x % (TILE / 4)) * 4;
        const bool live = threadIdx.x < QUADS && row < p.m;
        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live) {
#pragma unroll
            for (uint32_t w = 0; w < WARPS; ++w) {
                const float4 v = *reinterpret_cast<const float4*>(red + (w * ROWS + row) * PITCH + cq);
                sum.x += v.x;
                sum.y += v.y;
                sum.z += v.z;
                sum.w += v.w;
            }
        }
        bool write_out = complete;
        if (!complete) {
            // slot 0: the tile that opens this CTA's range; slot 1: the one that closes it
            const uint32_t slot = tile == u_begin / p.num_kb ? 0u : 1u;
            if (live)
                __stcg(reinterpret_cast<float4*>(p.partials + (size_t)(blockIdx.x * 2 + slot) * MAX_ROWS *
                                                                  MAX_TILE) + threadIdx.x, sum);
            // One thread synchronises for the CTA with a single acquire-release atomic: the barrier
            // in front orders the parked stores before its release, the one behind orders its
            // acquire before the loads.
            __syncthreads();
            const uint32_t c_first = owner_of(tile * p.num_kb, p);
            const uint32_t c_last = owner_of(tile_end - 1, p);
            if (threadIdx.x == 0) {
                uint32_t prev;
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
                             : "=r"(prev)
                             : "l"(p.counters + tile)
                             : "memory");
                const bool last = prev == c_last - c_first;
                if (last)
                    p.counters[tile] = 0;  // ready for the next launch
                *last_flag = last ? 1u : 0u;
            }
            __syncthreads();
            write_out = *last_flag != 0;
            if (write_out && live) {
                sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4  // contributors' loads in flight
                for (uint32_t c = c_first; c <= c_last; ++c) {
                    // this tile opens c's range unless an earlier one does
                    const uint32_t cslot = range_begin(c, p) >= tile * p.num_kb ? 0u : 1u;
                    const float4 v = __ldcg(reinterpret_cast<const float4*>(
                                                p.partials + (size_t)(c * 2 + cslot) * MAX_ROWS * MAX_TILE) +
                                            threadIdx.x);
                    sum.x += v.x;
                    sum.y += v.y;
                    sum.z += v.z;
                    sum.w += v.w;
                }
            }
        }
        if (write_out && live) {
            const uint32_t prob = prob_of(tile);
            const uint32_t col0 = (tile - prob * p.tiles) * TILE + cq;
            const float v[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t col = col0 + i;
                if (col >= p.n)
                    break;
                // three matrices: one output each; scatter form: a column belongs to one destination
                const uint32_t d_lo = p.scatter_cols ? col / p.scatter_cols : prob;
                const uint32_t d_hi = p.scatter_cols ? d_lo + 1u : prob + p.copies;
                const uint32_t dcol = p.scatter_cols ? col - d_lo * p.scatter_cols : col;
                for (uint32_t d = d_lo; d < d_hi; ++d) {
                    const size_t idx = (size_t)row * p.ld + dcol;
                    if (OUT_F16)
                        reinterpret_cast<__half*>(p.out[d])[idx] = __float2half_rn(v[i]);
                    else
                        reinterpret_cast<float*>(p.out[d])[idx] = v[i];
                }
            }
        }
        seg = seg_end;
    }
}

// Column tiles of 64 (four 16-column sub-tiles per activation fragment) where every warp still gets
// four units or more, else of 32: the activations a warp reads through L1 weigh as much as the
// weights at M = 16 and 64 columns, and half a unit per warp is lost at the end of a launch.  One matrix of
// that size with more than eight rows is the tcgen05 form's (see use_tc), unless it has next to no columns.
static uint32_t tile_cols(const DeviceCtx& ctx, uint32_t num_probs, uint32_t m, uint32_t n, uint32_t k)
{
    if (num_probs == 1 && m > 8)
        return MIN_TILE;
    const uint64_t units = (uint64_t)num_probs * ((n + MAX_TILE - 1) / MAX_TILE) * (k / UNIT_K);
    return units >= (uint64_t)ctx.num_sms * CTAS_PER_SM * WARPS * 4 ? MAX_TILE : MIN_TILE;
}

}  // namespace w4dw

bool w4a16_decode_ok(const void* x, const DqProblem* probs, int num_probs, uint32_t m, uint32_t n,
                     uint32_t k)
{
    using namespace w4dw;
    if (m > MAX_ROWS || k % UNIT_K != 0 || (num_probs != 1 && num_probs != 3))
        return false;
    // unit numbers are 32-bit
    if ((uint64_t)num_probs * ((n + MIN_TILE - 1) / MIN_TILE) * (k / UNIT_K) > 0x7fffffffu)
        return false;
    for (int i = 0; i < num_probs; ++i)
        if ((uintptr_t)probs[i].w % 16 != 0 || (uintptr_t)probs[i].scales % 2 != 0)
            return false;
    return (uintptr_t)x % 16 == 0;
}

// Where the tcgen05 form, which always served one matrix before, is the faster one (us back to back, tcgen05 /
// this one; three matrices in one launch are this kernel's alone):
//  * a tile of one or two units of K, whatever the rows: most of a CTA's warps idle at every tile's end.  M = 1 / 16:
//    4096 x 128 3.9 / 8.2, 4.1 / 11.9; 28672 x 256 4.7 / 5.9, 4.9 / 8.6 (N x K); from 128 columns on;
//  * few units in all, so a CTA takes eight, and K no power of two of units: every tile is cut and summed through
//    memory.  4096 columns, K = 384 / 640 at M = 1: 6.1 / 8.2, 0.90 of it; K = 384 .. 1280 at M = 16: 0.67 to 0.96;
//  * more than eight rows, which double the MMAs and the activations, over many columns: the line follows
//    rows * columns^2 * K.  M = 16: 16384 x 1024 10.0 / 11.7, 28672 x 1024 12.1 / 14.7, 9216 x 2048 10.4 / 11.3, 11008 x
//    4096 15.2 / 17.1, 28672 x 8192 41.9 / 53.5; below it 16384 x 512 7.4 / 5.7, 11008 x 1024 11.7 / 9.6, 4096 x 8192
//    15.1 / 13.9, 2048 x 28672 23.4 / 18.2; M = 9: 28672 x 1024 11.8 / 13.3, 8192 x 2048 10.4 / 10.2; up to 8192
//    columns a little later: 8192 x 2560 14.1 / 11.9, x 3072 12.5 / 12.7;
//  * very many columns: 98304 x 512 at M = 1 0.73 of this one's time, at M = 16 0.54; from K = 1792 on alike at M = 1.
// Over 337 widths and depths at M = 1, 8, 9 and 16 the pick is 0.4 % off the better form on
// average, 12.8 % with the line at 2^25 weights and nine rows alone.
static bool use_tc(const DeviceCtx& ctx, int num_probs, uint32_t m, uint32_t n, uint32_t k)
{
    using namespace w4dw;
    if (num_probs != 1 || n < 128)
        return false;
    const uint32_t kb = k / UNIT_K;
    if (kb <= 2)
        return true;
    const uint64_t tiles = (n + MIN_TILE - 1) / MIN_TILE, max_grid = (uint64_t)ctx.num_sms * CTAS_PER_SM;
    const bool cut = n >= 256 && 8 % kb != 0 && kb % 8 != 0 && tiles * kb <= max_grid * WARPS;
    if (m <= 8)
        return (cut && kb <= 5) || (n >= 49152 && kb <= 12);
    if ((cut && kb <= 10) || n >= 49152)
        return true;
    if (tiles % max_grid == 0)  // no tile is cut here: 9472 columns, K = 1536 at M = 16 9.8 / 6.3
        return (uint64_t)n * k >= (1u << 25);
    return (kb >= 7 || n >= 24576) && (double)m * n * n * k > (n > 8192 ? 2.2e12 : 2.9e12);
}

size_t w4a16_decode_workspace_bytes(const DeviceCtx& ctx)
{
    using namespace w4dw;
    const size_t own = (size_t)ctx.num_sms * CTAS_PER_SM * 2 * MAX_ROWS * MAX_TILE * sizeof(float);
    const size_t tc = w4a16_decode_tc_workspace_bytes(ctx);
    return own > tc ? own : tc;
}

size_t w4a16_decode_num_counters(int num_probs, uint32_t n)
{
    return (size_t)num_probs * ((n + w4dw::MIN_TILE - 1) / w4dw::MIN_TILE);
}

cudaError_t launch_w4a16_decode(const DeviceCtx& ctx, const __half* x, const DqProblem* probs,
                                int num_probs, bool out_f16, uint32_t m, uint32_t n, uint32_t k,
                                void* workspace, uint32_t* counters, cudaStream_t stream,
                                const OutputCopies* copies)
{
    using namespace w4dw;
    if (use_tc(ctx, num_probs, m, n, k))
        return launch_w4a16_decode_tc(ctx, x, probs[0], out_f16, m, n, k, workspace, counters, stream,
                                      copies);
    Params p;
    for (int i = 0; i < 3; ++i) {
        const DqProblem& pr = probs[i < num_probs ? i : 0];
        p.w[i] = static_cast<const uint32_t*>(pr.w);
        p.scales[i] = pr.scales;
    }
    for (int i = 0; i < 8; ++i)
        p.out[i] = copies ? copies->ptrs[(uint32_t)i < copies->count ? i : 0]
                          : probs[i < num_probs ? i : 0].out;
    p.x = x;
    p.partials = static_cast<float*>(workspace);
    p.counters = counters;
    p.copies = copies ? copies->count : 1u;
    p.scatter_cols = copies ? copies->scatter_cols : 0u;
    p.ld = copies ? copies->ld : n;
    p.m = m;
    p.n = n;
    p.k = k;
    const uint32_t tile = tile_cols(ctx, num_probs, m, n, k);
    p.num_kb = k / UNIT_K;
    p.tiles = (n + tile - 1) / tile;
    const uint32_t units = num_probs * p.tiles * p.num_kb;
    // a unit per warp is the least a CTA is started for
    uint32_t grid = (units + WARPS - 1) / WARPS;
    if (grid > (uint32_t)ctx.num_sms * CTAS_PER_SM)
        grid = (uint32_t)ctx.num_sms * CTAS_PER_SM;
    p.per_cta = units / grid;
    p.rem = units % grid;
    p.weights_wait = num_probs == 3;

    // Programmatic dependent launch: this launch may begin (weight prefetch) while the kernel in
    // front of it in the stream drains.  KAIO_B200_PDL=0 restores plain stream serialisation.
    static const bool use_pdl = [] {
        const char* e = getenv("KAIO_B200_PDL");
        return !(e != nullptr && e[0] == '0');
    }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl ? 1 : 0;

    static bool attr_set[8][64] = {};
    auto go = [&](auto kernel, uint32_t tc, uint32_t nb) -> cudaError_t {
        cfg.dynamicSmemBytes = smem_bytes(tc, nb);
        bool& set = attr_set[(tc == 4) * 4 + (nb == 2) * 2 + out_f16][ctx.device];
        if (!set) {
            const cudaError_t err = cudaFuncSetAttribute(
                kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
            if (err != cudaSuccess)
                return err;
            set = true;
        }
        return cudaLaunchKernelEx(&cfg, kernel, p);
    };
    const bool wide = tile == MAX_TILE;
    if (m <= 8) {
        if (wide)
            return out_f16 ? go(w4a16_decode_warp_kernel<4, 1, true>, 4, 1)
                           : go(w4a16_decode_warp_kernel<4, 1, false>, 4, 1);
        return out_f16 ? go(w4a16_decode_warp_kernel<2, 1, true>, 2, 1)
                       : go(w4a16_decode_warp_kernel<2, 1, false>, 2, 1);
    }
    if (wide)  // three matrices: f16 outputs
        return go(w4a16_decode_warp_kernel<4, 2, true>, 4, 2);
    return out_f16 ? go(w4a16_decode_warp_kernel<2, 2, true>, 2, 2)
                   : go(w4a16_decode_warp_kernel<2, 2, false>, 2, 2);
}

}  // namespace kaio

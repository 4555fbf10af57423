// The warp-level tensor instruction, for the kernels whose tiles are too thin for tcgen05's 128 rows
// (one to a few query rows, sixteen activation rows) and whose time is not set by the tensor pipe.
#pragma once

#include <stdint.h>

namespace kaio {

// c[16 x 8] += a[16 x 16] * b[16 x 8], f16 in, f32 accumulators.  Lane (g, t) = (lane / 4, lane % 4)
// holds a: rows g (a0, a2) and g + 8 (a1, a3), k pairs 2t (a0, a1) and 2t + 8 (a2, a3); b: column g,
// the same k pairs; c: rows g (c0, c1) and g + 8 (c2, c3), columns 2t and 2t + 1.
__device__ __forceinline__ void mma_m16n8k16_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                 uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
                 "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

}  // namespace kaio

// The even cut of a stream-K launch's units into one contiguous range per CTA, for the tcgen05 W4A16
// kernels: CTA c takes units [c * units / grid, (c + 1) * units / grid).
//
// The host divides once; a CTA gets its range with a multiplication and the owner of a unit with a
// float estimate that two comparisons put right.  In the kernels these quotients stand in front of the
// first load and between the last product and the output.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define KAIO_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define KAIO_HOST_DEVICE inline
#endif

namespace kaio {

struct UnitRanges {
    uint32_t len, rem;    // units = grid * len + rem
    uint32_t inv_grid;    // ceil(2^32 / grid), grid >= 2
    float ctas_per_unit;  // grid / units

    // First unit of CTA c <= grid: c * units / grid = c * len + c * rem / grid.  Exact for grid <= 1024:
    // c * rem < grid^2, the reciprocal is less than 1 / 2^32 too large, so the product is less than
    // grid^2 / 2^32 < 1 / grid too large.
    KAIO_HOST_DEVICE uint32_t begin(uint32_t c) const
    {
        return c * len + (uint32_t)(((uint64_t)(c * rem) * inv_grid) >> 32);
    }

    // The CTA whose range holds unit u.  The estimate is off by less than one: three roundings of
    // 2^-24 each of a number below 1024.
    KAIO_HOST_DEVICE uint32_t owner(uint32_t u) const
    {
        uint32_t c = (uint32_t)((float)u * ctas_per_unit);
        if (begin(c) > u)
            --c;
        else if (begin(c + 1) <= u)
            ++c;
        return c;
    }
};

// grid <= units, grid <= 1024.
inline UnitRanges unit_ranges(uint32_t units, uint32_t grid)
{
    UnitRanges r;
    r.len = units / grid;
    r.rem = units % grid;
    r.inv_grid = grid < 2 ? 0u : (uint32_t)((((uint64_t)1 << 32) + grid - 1) / grid);  // rem is 0 for 1
    r.ctas_per_unit = (float)((double)grid / (double)units);
    return r;
}

}  // namespace kaio

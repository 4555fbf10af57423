"""The cut of a stream-K launch's units into ranges, and the registers of the kernel that uses it, on
the CPU: csrc/unit_ranges.cuh compiled for the host against the quotients it stands for."""
import os
import subprocess

from kaio_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ranges_and_owners_are_the_exact_quotients(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(r'''
#include <cstdio>
#include <initializer_list>
#include "unit_ranges.cuh"
int main()
{
    const uint32_t grids[] = {1, 2, 3, 64, 127, 147, 148, 296, 320, 1023, 1024};
    uint32_t bad = 0;
    for (uint32_t grid : grids)
        for (uint64_t units : {(uint64_t)grid, (uint64_t)grid + 1, (uint64_t)1024, (uint64_t)2047, (uint64_t)7168,
                               (uint64_t)100003, (uint64_t)16777217, (uint64_t)1 << 31, (uint64_t)4294967295u}) {
            if (units < grid)
                continue;
            const kaio::UnitRanges r = kaio::unit_ranges((uint32_t)units, grid);
            for (uint32_t c = 0; c < grid; ++c) {
                const uint64_t lo = c * units / grid, hi = (c + 1) * units / grid;
                bad += r.begin(c) != lo || r.begin(c + 1) != hi;
                for (uint64_t u : {lo, lo + 1, (lo + hi) / 2, hi - 1})
                    if (u >= lo && u < hi)
                        bad += r.owner((uint32_t)u) != c;
            }
        }
    std::printf("%u\n", bad);
    return bad != 0;
}
''')
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "kaio_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_the_middle_row_kernel_does_not_spill(tmp_path):
    """Its fourteen warps run at the 128-register cap; addresses kept over a loop end up on the stack."""
    src = os.path.join(ROOT, "kaio_b200", "csrc", "w4a16_fused.cu")
    r = subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-c", src, "-o", str(tmp_path / "o")], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    spills = [line.strip() for line in r.stderr.splitlines() if "spill stores" in line]
    assert len(spills) == 4
    assert all("0 bytes spill stores" in line and line.startswith("0 bytes stack") for line in spills), spills

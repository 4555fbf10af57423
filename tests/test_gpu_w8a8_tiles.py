"""W8A8 over the tile widths: halves and quarters of the pair kernel's tiles, the 64- / 128- / 256-column
tiles of the single-CTA kernel, ragged last columns and rows of each, and the pair kernel with few rows
of a fused QKV call.  s32 sums are exact and the epilogue is one or two roundings: bit for bit."""
import numpy as np
import pytest
import torch

from kaio_b200 import ops
from helpers import dev, device, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (129, 80, 96), (300, 528, 1056), (512, 512, 512), (257, 4112, 160), (1024, 2064, 256), (1500, 3008, 128),  # pairs
    (1, 16, 32), (64, 80, 544), (128, 4112, 1024), (100, 9488, 160), (128, 20000, 96)])  # single CTA
def test_matmul(oracle, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.integers(-128, 128, m * k, dtype=np.int8), rng.integers(-128, 128, k * n, dtype=np.int8)
    sa, sw = rng.uniform(0.001, 0.01, m).astype(np.float32), rng.uniform(0.001, 0.01, n).astype(np.float32)
    out = torch.full((m * n,), float("nan"), device="cuda")
    ops.matmul_int8_scaled(device(), dev(a), dev(b), out, dev(sa), dev(sw), m, n, k)
    assert ops.device_status(device())[0] == 0
    assert np.array_equal(host(out, (m, n)), oracle.matmul_int8_scaled(a, b, sa, sw, m, n, k))


@pytest.mark.parametrize("m,n,k", [(1, 256, 128), (16, 1040, 512), (100, 272, 1056), (128, 4096, 256), (300, 528, 512)])
def test_qkv(oracle, m, n, k):
    rng = np.random.default_rng(m + n + k)
    x = rng.standard_normal(m * k).astype(np.float16)
    ws = [rng.integers(-127, 128, k * n, dtype=np.int8) for _ in range(3)]
    sc = [rng.uniform(0.001, 0.01, n).astype(np.float32) for _ in range(3)]
    o = [torch.full((m * n,), float("nan"), device="cuda", dtype=torch.float16) for _ in range(3)]
    ops.qkv_project_w8a8(device(), dev(x), *[dev(w) for w in ws], *[dev(s) for s in sc], *o, m, n, k)
    assert ops.last_variant() == "qkv_w8a8_tcgen05_2cta"
    assert ops.device_status(device())[0] == 0
    for t, w, s in zip(o, ws, sc):
        assert np.array_equal(host(t, (m, n)).view(np.uint16), oracle.qkv_w8a8(x, w, s, m, n, k).view(np.uint16))

"""The fused W8A16 QKV kernel at the edges of its row tiles (32 / 64 / 128 / 256), column tiles (128),
K blocks (64) and K cuts, with scalar and per-column scales; the bar is the reference's 1e-3."""
import numpy as np
import pytest
import torch

from kaio_b200 import ops
from helpers import dev, device, host, max_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 16, 16), (32, 144, 80), (33, 128, 1024), (64, 1040, 2048), (65, 256, 528),
                                   (128, 272, 4096), (129, 128, 640), (256, 400, 1008),
                                   (257, 144, 512), (512, 128, 2048)])
def test_fused(oracle, m, n, k, col):
    rng = np.random.default_rng(m + n + k)
    x = rng.standard_normal(m * k).astype(np.float16)
    ws = [rng.integers(-128, 128, k * n, dtype=np.int8) for _ in range(3)]
    sc = [rng.uniform(0.0005, 0.002, n).astype(np.float32) if col else 0.001 * (i + 1) for i in range(3)]
    o = [torch.full((m * n,), float("nan"), device="cuda", dtype=torch.float16) for _ in range(3)]
    ops.qkv_project_int8(device(), dev(x), *[dev(w) for w in ws], *[dev(s) if col else s for s in sc], *o, m, n, k)
    assert ops.last_variant() == "qkv_w8a16_fused"
    assert ops.device_status(device())[0] == 0
    for got, w, s in zip(o, ws, sc):
        want = oracle.qkv_int8(x, w, 0.0 if col else s, m, n, k, col_scale=s if col else None)
        assert max_rel(host(got, (m, n)), want) < 1e-3

"""The M <= 16 W4A16 kernel where it can go wrong: ragged column tiles (32 and 64 columns), a single
scale group, one unit per warp and less, tiles cut between CTAs, both row groups, three matrices in
one launch.  The bar is the reference's (|g-w| / max(|w|, 1) < 1e-3 for f32 out and for the QKV
outputs); two runs agree bit for bit, since every sum has a fixed order."""
import numpy as np
import pytest
import torch

from kaio_b200 import ops
from helpers import dev, device, host, max_rel

pytestmark = pytest.mark.gpu
G = 128


def weights(oracle, rng, k, n):
    return (oracle.pack_s4(rng.integers(-8, 8, k * n, dtype=np.int8), k, n),
            rng.uniform(0.005, 0.02, (k // G) * n).astype(np.float16))


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(1, 128), (31, 256), (33, 1152), (65, 8192), (1030, 2048), (14344, 8192)])
def test_matmul_int4(oracle, m, n, k):
    rng = np.random.default_rng(m + n + k)
    (packed, scales), a = weights(oracle, rng, k, n), rng.standard_normal(m * k).astype(np.float16)
    got = []
    for _ in range(2):
        c = torch.full((m * n,), float("nan"), device="cuda")
        ops.matmul_int4(device(), dev(a), dev(packed), dev(scales), c, m, n, k, G)
        got.append(host(c, (m, n)))
    assert ops.last_variant() == "w4a16_decode_splitk"
    assert np.array_equal(got[0], got[1])
    assert max_rel(got[0], oracle.matmul_int4(a, packed, scales, m, n, k)) < 1e-3


@pytest.mark.parametrize("m", [1, 8, 16])
@pytest.mark.parametrize("n,k", [(16, 128), (40, 384), (1000, 1024), (4096, 4096)])
def test_qkv(oracle, m, n, k):
    rng = np.random.default_rng(m * 3 + n + k)
    ws, x = [weights(oracle, rng, k, n) for _ in range(3)], rng.standard_normal(m * k).astype(np.float16)
    o = [torch.full((m * n,), float("nan"), device="cuda", dtype=torch.float16) for _ in range(3)]
    ops.qkv_project_int4(device(), dev(x), *[dev(w) for w, _ in ws], *[dev(s) for _, s in ws], *o, m, n, k, G)
    assert ops.last_variant() == "qkv_w4a16_decode_splitk"
    for got, (w, s) in zip(o, ws):
        assert max_rel(host(got, (m, n)), oracle.qkv_int4(x, w, s, m, n, k)) < 1e-3


def test_qkv_decode_capture_after_warming_many_rows(oracle):
    """Warming the op at its largest shape covers a decode step captured later on that stream."""
    n, k, m = 256, 512, 4
    rng = np.random.default_rng(3)
    ws = [weights(oracle, rng, k, n) for _ in range(3)]
    wd, sd = [dev(w) for w, _ in ws], [dev(s) for _, s in ws]
    x = rng.standard_normal(600 * k).astype(np.float16)
    xd = dev(x)
    o = [torch.zeros((600 * n,), device="cuda", dtype=torch.float16) for _ in range(3)]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ops.qkv_project_int4(device(), xd, *wd, *sd, *o, 600, n, k, G)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            ops.qkv_project_int4(device(), xd, *wd, *sd, *o, m, n, k, G)
        for t in o:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
    for got, (w, s) in zip(o, ws):
        assert max_rel(host(got)[:m * n].reshape(m, n), oracle.qkv_int4(x[:m * k], w, s, m, n, k)) < 1e-3

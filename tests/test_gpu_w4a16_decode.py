"""The M <= 16 W4A16 kernel where it can go wrong: ragged column tiles (32 and 64 columns), a single
scale group, one unit per warp and less, tiles cut between CTAs, both row groups, three matrices in
one launch.  The bar is the reference's (|g-w| / max(|w|, 1) < 1e-3 for f32 out and for the QKV
outputs); two runs agree bit for bit, since every sum has a fixed order."""
import numpy as np
import pytest
import torch

from kaio_b200 import _lib, ops
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


def test_qkv_scales_written_by_the_launch_in_front():
    """The decode GEMM in front lets its dependents start before it is done; its f16 output is the QKV call's
    scale matrix.  Back to back and with a synchronisation in between: the same bits."""
    n, k, k0 = 512, 1024, 4096
    g = torch.Generator(device="cuda").manual_seed(5)

    def words(rows, cols):
        return torch.randint(-2**31, 2**31 - 1, (rows // 8 * cols,), generator=g, device="cuda", dtype=torch.int32)

    w0, s0 = words(k0, n), torch.full((k0 // G * n,), 0.01, device="cuda").half()
    ws = [words(k, n) for _ in range(3)]
    x = torch.randn(8 * k, generator=g, device="cuda").half()
    a = [torch.rand(k // G * k0, generator=g, device="cuda").mul_(0.01).half() for _ in range(8)]
    scales = [torch.zeros(k // G * n, device="cuda", dtype=torch.float16) for _ in range(3)]

    def run(i, sync):
        o = [torch.zeros(8 * n, device="cuda", dtype=torch.float16) for _ in range(3)]
        torch.cuda.synchronize()
        for j, s in enumerate(scales):
            ops.matmul_int4(device(), a[(i + j) % 8], w0, s0, s, k // G, n, k0, G)
        if sync:
            torch.cuda.synchronize()
        ops.qkv_project_int4(device(), x, *ws, *scales, *o, 8, n, k, G)
        return torch.cat(o)

    want = [run(i, True) for i in range(8)]
    for i in range(64):
        assert torch.equal(run(i % 8, False), want[i % 8])


@pytest.mark.parametrize("warm", [17, 64, 256, 512, 600])
def test_decode_capture_after_warming_any_row_count(oracle, warm):
    """Whichever kernel served the many rows (none of these needs split-K scratch for itself)."""
    n, k, m = 256, 512, 4
    rng = np.random.default_rng(warm)
    ws, x = [weights(oracle, rng, k, n) for _ in range(3)], rng.standard_normal(warm * k).astype(np.float16)
    wd, sd, xd = [dev(w) for w, _ in ws], [dev(s) for _, s in ws], dev(x)
    o = [torch.zeros(warm * n, device="cuda", dtype=torch.float16) for _ in range(3)]
    c = torch.zeros(warm * n, device="cuda")
    # torch hands out pooled streams: one with no scratch of its own yet is what the promise is about
    for run, outs in ((lambda rows: ops.matmul_int4(device(), xd, wd[0], sd[0], c, rows, n, k, G), [c]),
                      (lambda rows: ops.qkv_project_int4(device(), xd, *wd, *sd, *o, rows, n, k, G), o)):
        torch.cuda.synchronize()
        _lib.load().kaio_b200_shutdown()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            run(warm)
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                run(m)
            for t in outs:
                t.zero_()
            graph.replay()
            torch.cuda.synchronize()
        for got, (w, s) in zip(outs, ws):
            want = oracle.matmul_int4(x[:m * k], w, s, m, n, k) if outs[0] is c else oracle.qkv_int4(x[:m * k], w, s, m, n, k)
            assert max_rel(host(got)[:m * n].reshape(m, n), want) < 1e-3


@pytest.mark.parametrize("m", [1, 9, 16])
def test_qkv_of_64_column_tiles(oracle, m):
    """Three matrices large enough for the wide tiles, of a width that ends inside one; every third row."""
    n, k = 5128, 5120
    rng = np.random.default_rng(m)
    ws, x = [weights(oracle, rng, k, n) for _ in range(3)], rng.standard_normal(m * k).astype(np.float16)
    got = []
    for _ in range(2):
        o = [torch.full((m * n,), float("nan"), device="cuda", dtype=torch.float16) for _ in range(3)]
        ops.qkv_project_int4(device(), dev(x), *[dev(w) for w, _ in ws], *[dev(s) for _, s in ws], *o, m, n, k, G)
        got.append([host(t, (m, n)) for t in o])
    rows = list(range(0, m, 3)) + [m - 1]
    xs = np.ascontiguousarray(x.reshape(m, k)[rows]).reshape(-1)
    for first, again, (w, s) in zip(*got, ws):
        assert np.array_equal(first.view(np.uint16), again.view(np.uint16))
        assert max_rel(first[rows], oracle.qkv_int4(xs, w, s, len(rows), n, k)) < 1e-3


@pytest.mark.parametrize("m", [1, 8])
def test_f16_output_of_64_column_tiles(oracle, m):
    n, k = 14344, 8192
    rng = np.random.default_rng(m)
    (packed, scales), a = weights(oracle, rng, k, n), rng.standard_normal(m * k).astype(np.float16)
    got = []
    for _ in range(2):
        c = torch.full((m * n,), float("nan"), device="cuda", dtype=torch.float16)
        ops.matmul_int4(device(), dev(a), dev(packed), dev(scales), c, m, n, k, G)
        got.append(host(c, (m, n)))
    assert np.array_equal(got[0].view(np.uint16), got[1].view(np.uint16))
    # f32 sums narrowed once: half a unit in the last place of f16 beside the f32 bar
    want = oracle.matmul_int4(a, packed, scales, m, n, k).reshape(m, n).astype(np.float64)
    assert np.all(np.abs(got[0] - want) <= 2.0 ** -11 * np.abs(want) + 1e-3 * np.maximum(np.abs(want), 1.0))


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(127, 128), (128, 128), (130, 256), (255, 384), (256, 384), (1000, 640), (520, 1280),
                                 (16384, 1024), (49160, 384)])
def test_on_both_sides_of_the_line_between_the_two_forms(oracle, m, n, k):
    rng = np.random.default_rng(m * 7 + n + k)
    (packed, scales), a = weights(oracle, rng, k, n), rng.standard_normal(m * k).astype(np.float16)
    got = []
    for _ in range(2):
        c = torch.full((m * n,), float("nan"), device="cuda")
        ops.matmul_int4(device(), dev(a), dev(packed), dev(scales), c, m, n, k, G)
        got.append(host(c, (m, n)))
    assert ops.device_status(device())[0] == 0
    assert np.array_equal(got[0], got[1])
    assert max_rel(got[0], oracle.matmul_int4(a, packed, scales, m, n, k)) < 1e-3

"""One query row per (batch, head) over a key/value cache (`attention_mha_f16` with seq_q == 1).

The key counts sit at the edges of what a warp (16 keys at head_dim 128, 32 at 64), a CTA and a
cluster take at a time; the bar is the reference's (kaio-ops/tests/common/mod.rs:249-284).
"""
import numpy as np
import pytest
import torch

from kaio_b200 import CudaError, ops
from helpers import assert_attention_close, dev, device, host

pytestmark = pytest.mark.gpu


def run(oracle, b, h, sk, d, causal, stride, sigma=1.0):
    rng = np.random.default_rng(b * 1000 + h * 100 + sk + d)
    q = (rng.standard_normal((b, stride)) * sigma).astype(np.float16)
    k = (rng.standard_normal((b * sk, stride)) * sigma).astype(np.float16)
    v = rng.standard_normal((b * sk, stride)).astype(np.float16)
    want = np.zeros((b, stride), np.float16)
    for bi in range(b):
        for hi in range(h):
            oracle.attention(q.reshape(-1)[bi * stride + hi * d:], k.reshape(-1)[bi * sk * stride + hi * d:],
                             v.reshape(-1)[bi * sk * stride + hi * d:], 1, sk, d, d, causal=causal,
                             strides=(stride,) * 4, f16_out=True, out=want.reshape(-1)[bi * stride + hi * d:])
    out = torch.zeros((b * stride,), device="cuda", dtype=torch.float16)
    ops.attention_mha_f16(device(), dev(q), dev(k), dev(v), out, b, h, 1, sk, d, stride, causal)
    assert ops.last_variant() == "attention_decode"
    assert_attention_close(host(out, (b, stride)).astype(np.float32), want.astype(np.float32))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,h,sk", [(1, 1, 1), (1, 2, 15), (2, 3, 33), (1, 8, 257), (1, 1, 2049), (8, 32, 517)])
def test_decode(oracle, b, h, sk, d):
    run(oracle, b, h, sk, d, False, h * d)


@pytest.mark.parametrize("d", [64, 128])
def test_decode_causal_strided_hot(oracle, d):
    run(oracle, 2, 2, 40, d, True, 2 * d + 8)       # row 0 sees key 0 only; padded rows
    run(oracle, 1, 4, 1000, d, False, 4 * d, 3.7)   # scores spread over some twenty powers of two


def test_more_pairs_than_a_grid_has_rows():
    """65536 (batch, head) pairs and more: the one-row kernel numbers its CTAs in one dimension; the kernels
    for several rows do not, and such a call is refused on the host as it always was."""
    b, sk, d = 70000, 3, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = [torch.randn(b * n, d, generator=g, device="cuda").half() for n in (1, sk, sk)]
    out = torch.zeros(b * d, device="cuda", dtype=torch.float16)
    ops.attention_mha_f16(device(), q, k, v, out, b, 1, 1, sk, d, d, False)
    assert ops.last_variant() == "attention_decode"
    s = torch.einsum("bd,bsd->bs", q.float(), k.view(b, sk, d).float()) / 8.0
    want = torch.einsum("bs,bsd->bd", torch.softmax(s, 1), v.view(b, sk, d).float())
    assert_attention_close(host(out, (b, d)).astype(np.float32), want.cpu().numpy())
    with pytest.raises(CudaError):
        ops.attention_mha_f16(device(), torch.cat([q, q]), k, v, torch.cat([out, out]), b, 1, 2, sk, d, d, False)

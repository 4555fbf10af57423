"""The warp-MMA attention kernel: head_dim 64 of any length and short sequences of few heads, at the
edges of its 16-row CTAs, 16- and 64-key stages and eight key groups.  The bar is the reference's
(kaio-ops/tests/common/mod.rs:249-284); the f32 form is also held to 2e-6 of the row's largest value
against 64-bit arithmetic, since P keeps 22 bits (products exact, f32 sums of at most 384 terms)."""
import numpy as np
import pytest
import torch

from kaio_b200 import ops
from helpers import assert_attention_close, dev, device, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,h,sq,sk,d,pad", [
    (1, 1, 2, 1, 64, 0), (1, 2, 17, 15, 64, 0), (1, 2, 33, 65, 128, 0), (2, 3, 48, 129, 128, 8),   # short form
    (1, 1, 384, 384, 128, 0), (1, 3, 100, 384, 64, 0), (1, 1, 16, 300, 64, 8),
    (1, 1, 65, 385, 64, 0), (2, 40, 70, 63, 64, 0), (1, 2, 500, 500, 64, 8), (1, 1, 130, 1000, 64, 0)])  # long form
def test_mha(oracle, b, h, sq, sk, d, pad, causal):
    rng = np.random.default_rng(b * 1000 + h * 100 + sq + sk + d)
    stride = h * d + pad
    q = (rng.standard_normal((b * sq, stride)) * 2.0).astype(np.float16)
    k, v = [rng.standard_normal((b * sk, stride)).astype(np.float16) for _ in range(2)]
    want = np.zeros((b * sq, stride), np.float16)
    for bi in range(b):
        for hi in range(h):
            oracle.attention(q.reshape(-1)[bi * sq * stride + hi * d:], k.reshape(-1)[bi * sk * stride + hi * d:],
                             v.reshape(-1)[bi * sk * stride + hi * d:], sq, sk, d, d, causal=causal,
                             strides=(stride,) * 4, f16_out=True, out=want.reshape(-1)[bi * sq * stride + hi * d:])
    out = torch.zeros((b * sq * stride,), device="cuda", dtype=torch.float16)
    ops.attention_mha_f16(device(), dev(q), dev(k), dev(v), out, b, h, sq, sk, d, stride, causal)
    assert ops.last_variant() == "attention_warp_mma"
    assert_attention_close(host(out, (b * sq, stride)).astype(np.float32), want.astype(np.float32))


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("sq,sk,d", [(16, 16, 64), (64, 384, 64), (384, 384, 128), (48, 80, 128)])
def test_tc_precision(sq, sk, d, causal):
    g = torch.Generator().manual_seed(sq + sk + d)
    q, k, v = [torch.randn((n, d), generator=g).half() for n in (sq, sk, sk)]
    s = q.double() @ k.double().T / d ** 0.5
    if causal:
        s = s.masked_fill(torch.arange(sk)[None, :] > torch.arange(sq)[:, None], float("-inf"))
    want = torch.softmax(s, 1) @ v.double()
    out = torch.full((sq * d,), float("nan"), device="cuda")
    fn = ops.attention_tc_causal if causal else ops.attention_tc
    fn(device(), q.flatten().cuda(), k.flatten().cuda(), v.flatten().cuda(), out, sq, sk, d, d)
    assert ops.last_variant() == "attention_warp_mma"
    err = (out.cpu().double().view(sq, d) - want).abs().amax(1) / want.abs().amax(1)
    assert err.max() < 2e-6

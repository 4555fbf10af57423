"""Attention with values at the ends of the f16 range, on the warp-MMA and the one-row kernels: scores far
beyond what an exponent holds, rows whose result is known to the last bit, infinities and NaN."""
import numpy as np
import pytest
import torch

from kaio_b200 import ops
from helpers import dev, device, host

pytestmark = pytest.mark.gpu

# (batch, heads, seq_q, seq_k, d): short form, long head_dim 64 form, one-row kernel
SHAPES = [(1, 2, 33, 100, 64), (1, 1, 48, 384, 128), (2, 3, 70, 500, 64), (1, 2, 1, 700, 64), (2, 2, 1, 300, 128)]


def attend(q, k, v, b, h, sq, sk, d, causal):
    out = torch.full((b * sq * h * d,), 7.0, device="cuda", dtype=torch.float16)
    ops.attention_mha_f16(device(), dev(q), dev(k), dev(v), out, b, h, sq, sk, d, h * d, causal)
    assert ops.last_variant() == ("attention_decode" if sq == 1 else "attention_warp_mma")
    return host(out, (b, sq, h, d)).astype(np.float64)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("b,h,sq,sk,d", SHAPES)
def test_scores_of_2_to_the_28(b, h, sq, sk, d, sign, causal):
    """q = +-2^15 everywhere, every k element of key j = 1024 + 8 r(j): dots are exact in f32, the scores are
    +-2^28 and more, and two different r are 2^15 and more apart in the exponent.  So the output is the
    mean of V over the visible keys of the largest r (smallest, for -), to one rounding to f16."""
    rng = np.random.default_rng(sk + d)
    q = np.full((b, sq, h, d), sign * 32768.0, np.float16)
    r = rng.integers(0, 60, (b, sk, h))
    k = np.broadcast_to((1024.0 + 8.0 * r)[..., None], (b, sk, h, d)).astype(np.float16)
    v = rng.standard_normal((b, sk, h, d)).astype(np.float16)
    got = attend(q, k, v, b, h, sq, sk, d, causal)
    for bi in range(b):
        for hi in range(h):
            for i in range(sq):
                n = min(i + 1, sk) if causal else sk
                key = sign * r[bi, :n, hi]
                want = v[bi, :n, hi].astype(np.float64)[key == key.max()].mean(0)
                # f16 output: 2^-11 of the value; the mean of up to a dozen values adds f32 roundings only
                assert np.all(np.abs(got[bi, i, hi] - want) <= 2.0 ** -10 * np.abs(want) + 1e-6), (bi, hi, i)


@pytest.mark.parametrize("seq,d", [(16, 64), (384, 64), (128, 128), (384, 128)])
def test_a_row_that_sees_one_key_is_its_value(seq, d):
    """P of the largest score is exactly 1, so row 0 of a causal call is V's row 0, bit for bit, also in f32."""
    g = torch.Generator(device="cuda").manual_seed(seq)
    q, k, v = [torch.randn(seq * d, generator=g, device="cuda").mul_(3.0).half() for _ in range(3)]
    out = torch.zeros(seq * d, device="cuda")
    ops.attention_tc_causal(device(), q, k, v, out, seq, seq, d, d)
    assert ops.last_variant() == "attention_warp_mma"
    assert torch.equal(out[:d], v[:d].float())


@pytest.mark.parametrize("special", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("b,h,sq,sk,d", SHAPES)
def test_special_values(oracle, b, h, sq, sk, d, special):
    """One element of one key, and of one value, of head 0 of batch 0.  What the oracle makes non-finite is
    non-finite of the same kind, what has weight zero or belongs to another head stays finite and right."""
    rng = np.random.default_rng(sk)
    q, k, v = [rng.standard_normal((b, n, h, d)).astype(np.float16) for n in (sq, sk, sk)]
    q[:, :, 0, 5] = np.abs(q[:, :, 0, 5]) + np.float16(0.1)
    for t, name in ((k, "k"), (v, "v")):
        clean = t[0, sk // 2, 0, 5]
        t[0, sk // 2, 0, 5] = special
        got = attend(q, k, v, b, h, sq, sk, d, False)
        t_q, t_k, t_v = [np.ascontiguousarray(x.transpose(0, 2, 1, 3)) for x in (q, k, v)]
        for bi in range(b):
            for hi in range(h):
                with np.errstate(all="ignore"):
                    want = oracle.attention(t_q[bi, hi], t_k[bi, hi], t_v[bi, hi], sq, sk, d, d)
                want = np.asarray(want, dtype=np.float64).reshape(sq, d)
                if name == "k" and bi == 0 and hi == 0 and special != float("-inf"):
                    assert np.isnan(got[bi, :, hi]).all()  # inf - inf or NaN in every row
                    continue
                same = np.isfinite(want)
                assert np.array_equal(np.isnan(got[bi, :, hi]), np.isnan(want))
                assert np.array_equal(got[bi, :, hi][~same], want[~same], equal_nan=True)
                # one f16 rounding beside the f32 sums
                assert np.all(np.abs(got[bi, :, hi][same] - want[same]) <= 2.0 ** -10 * np.abs(want[same]) + 2e-5)
        t[0, sk // 2, 0, 5] = clean


@pytest.mark.parametrize("special", [float("nan"), float("inf")])
@pytest.mark.parametrize("b,h,sq,sk,d", [s for s in SHAPES if s[2] > 1])
def test_rows_that_do_not_see_a_value_are_not_touched_by_it(b, h, sq, sk, d, special):
    """Causal: the key sits in the middle of a 16- and of a 64-key stage, so earlier rows meet it masked."""
    rng = np.random.default_rng(sk + d)
    q, k, v = [rng.standard_normal((b, n, h, d)).astype(np.float16) for n in (sq, sk, sk)]
    clean = attend(q, k, v, b, h, sq, sk, d, True)
    key = 21
    v[0, key, 0, 5] = special
    got = attend(q, k, v, b, h, sq, sk, d, True)
    seen = np.zeros(got.shape, bool)
    seen[0, key:, 0, 5] = True
    assert np.array_equal(got[seen], np.full(seen.sum(), special), equal_nan=True)
    # the masked meeting is summed once more in another order: one f16 rounding and f32 sums apart
    assert np.all(np.abs(got - clean)[~seen] <= 2.0 ** -10 * np.abs(clean[~seen]) + 2e-5)

"""Precision conversion on the integer pipe gives the bits of the conversion
instructions: random numbers over the whole exponent range, ties to even,
zeros of both signs, subnormals, infinities and NaN, with and without a scale."""
import numpy as np
import pytest

gpu = pytest.mark.gpu


def _values(n):
    r = np.random.default_rng(11)
    bits = r.integers(0, 2**64, n, dtype=np.uint64)
    v = bits.view(np.float64).copy()
    k = n // 3
    # the float range, half of it exactly on a tie between two floats
    f = (r.standard_normal(k) * 2.0 ** r.integers(-149, 128, k)).astype(np.float32).astype(np.float64)
    tie = f + np.spacing(np.abs(f).astype(np.float32)).astype(np.float64) / 2
    v[:k] = f
    v[k:2 * k] = np.where(np.isfinite(tie), tie, 1.5)
    v[:12] = [0.0, -0.0, 2.0**-126, -2.0**-126, 2.0**-149, 2.0**-150, np.inf, -np.inf, np.nan, 3.4028235677973366e38,
              2.0**-126 * (1 - 2.0**-25), np.float64(np.float32(3.4028235e38))]
    return v


@gpu
@pytest.mark.parametrize("scale", [1.0, 0.7])
def test_conversions_are_correctly_rounded(scale):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import gpt_gb300 as g

    dims = [4, 4, 4, 6]
    N = int(np.prod(dims)) // 2
    v = _values(2 * N * 24)

    def lat(prec, a=None):
        x = g.lattice(g.layout.get(g.grid(dims, prec)))
        if a is not None:
            x.tensor.copy_(torch.from_numpy(a.view(np.uint8)))
        return x

    def planes64(a):  # [half][12][N][2] -> values in the order of the single layout [half][6][N][4]
        return a.reshape(2, 6, 2, N, 2).transpose(0, 1, 3, 2, 4).reshape(-1)

    d = lat(g.double, v)
    s = lat(g.single)
    g.convert(s, d, scale)
    with np.errstate(all="ignore"):
        want = planes64(v * scale if scale != 1.0 else v).astype(np.float32)
    got = s.tensor.cpu().numpy().view(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(got[ok].view(np.uint32), want[ok].view(np.uint32))
    # and back: every float is a double
    b = lat(g.double)
    g.convert(b, s, scale)
    with np.errstate(all="ignore"):
        want = got.astype(np.float64) * (scale if scale != 1.0 else 1.0)
    back = planes64(b.tensor.cpu().numpy().view(np.float64))
    assert np.array_equal(np.isnan(back), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(back[ok].view(np.uint64), want[ok].view(np.uint64))
    # double-float keeps h = fl32(v), l = fl32(v - h) of ordinary numbers
    w = np.random.default_rng(12).standard_normal(v.size)
    dw, q = lat(g.double, w), lat(g.double_float)
    g.convert(q, dw)
    f = q.tensor.cpu().numpy().view(np.float32).reshape(2, 12, N, 4)
    h = w.reshape(2, 12, N, 2).astype(np.float32)
    low = (w.reshape(2, 12, N, 2) - h.astype(np.float64)).astype(np.float32)
    assert np.array_equal(f[..., :2], h) and np.array_equal(f[..., 2:], low)
    g.convert(b, q)
    assert np.array_equal(b.tensor.cpu().numpy().view(np.float64).reshape(h.shape), h.astype(np.float64) + low.astype(np.float64))

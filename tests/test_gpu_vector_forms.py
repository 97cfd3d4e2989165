"""The forms of the vector kernels (complex and real coefficients, b = 1 or
not, no y, reductions, one and two halves) against numpy, on fields of less
than a block, with a remainder and with packed right-hand sides, in place and
out of place."""
import numpy as np
import pytest

gpu = pytest.mark.gpu
# one rounding of the result per operation (at most three), relative to the largest term
EPS = {"double": 4 * 2.0 ** -53, "single": 4 * 2.0 ** -24, "double_float": 16 * 2.0 ** -48, "half": 2.0 ** -10}


@gpu
@pytest.mark.parametrize("prec", ["double", "single", "half", "double_float"])
@pytest.mark.parametrize("dims,Ls,n_rhs", [((2, 2, 2, 2), 1, 1), ((4, 6, 2, 10), 1, 1), ((4, 2, 6, 2), 7, 3), ((2, 2, 2, 4), 16, 16)])
def test_vector_forms(prec, dims, Ls, n_rhs):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import gpt_gb300 as g

    grid = g.grid(list(dims), getattr(g, prec))
    lay = g.layout.get(grid, Ls, n_rhs, five_d=Ls > 1)
    rng = np.random.default_rng(7)
    shape = (n_rhs,) + lay.natural_shape()

    def field():
        f = g.lattice(lay)
        v = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        for r in range(n_rhs):
            f.set_natural(v[r], r)
        return f, np.stack([f.get_natural(r) for r in range(n_rhs)])  # as stored

    def get(f):
        return np.stack([f.get_natural(r) for r in range(n_rhs)])

    def lst(v):
        return [v] if n_rhs == 1 else v

    x, X = field()
    y, Y = field()
    av = rng.standard_normal(n_rhs) + 1j * rng.standard_normal(n_rhs)
    ar = av.real
    bv = rng.standard_normal(n_rhs)

    def col(v):
        return np.asarray(v).reshape((n_rhs,) + (1,) * (len(shape) - 1))

    def close(got, a, b):
        scale = np.max(np.abs(col(a)) * np.max(np.abs(X)) + np.abs(col(b)) * np.max(np.abs(Y)))
        assert np.max(np.abs(got - (col(a) * X + col(b) * Y))) <= EPS[prec] * max(scale, 1.0) * 2

    one, zero = np.ones(n_rhs), np.zeros(n_rhs)
    out = g.lattice(lay)
    for a in (av, ar):
        g.axpby(out, list(a), x, list(bv), y)
        close(get(out), a, bv)
        g.axpby(out, list(a), x, 1.0, y)
        close(get(out), a, one)
        g.axpby(out, list(a), x)
        close(get(out), a, zero)
        n2 = lst(g.axpy_norm2(out, list(a), x, y))
        close(get(out), a, one)
        O = get(out)
        for r in range(n_rhs):
            want = np.vdot(O[r], O[r]).real
            # the sum is taken before the result is rounded to its storage
            assert abs(n2[r] - want) <= 2 * EPS[prec] * want + 1e-14 * want
    tol = {"double": 1e-14, "double_float": 1e-12, "single": 2e-6, "half": 2e-6}[prec]
    n2, ip = lst(g.norm2(x)), lst(g.inner_product(x, y))
    for r in range(n_rhs):
        assert abs(n2[r] - np.vdot(X[r], X[r]).real) <= tol * n2[r]
        assert abs(ip[r] - np.vdot(X[r], Y[r])) <= tol * np.linalg.norm(X[r]) * np.linalg.norm(Y[r])
    # one half, and in place
    hx, hy = x.half(g.odd), y.half(g.odd)
    before = get(y)
    h2 = lst(g.norm2(hx))
    e2 = lst(g.norm2(x.half(g.even)))
    assert np.allclose(np.add(h2, e2), n2, rtol=tol, atol=0)
    g.axpby(hy, list(ar), hx, 1.0, hy)
    Y2 = get(y)
    moved = np.any(Y2 != before, axis=tuple(range(2, len(shape))))
    import oracle as o

    odd = o.parity_of_sites(list(dims)) == 1
    assert not moved[:, ~odd].any() and moved[:, odd].all()

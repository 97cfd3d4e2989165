"""Natural layout to internal and back, every precision, against numpy's casts:
the bits of the converted numbers, also where float rounds, underflows or
overflows, on ragged lattices, every right-hand side by itself."""
import numpy as np
import pytest

gpu = pytest.mark.gpu


def _need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _values(shape, seed, special):
    r = np.random.default_rng(seed)
    v = r.standard_normal(shape) * 10.0 ** r.integers(-6, 7, shape)
    if special:
        odd = np.array([0.0, -0.0, 1.0 + 2.0**-24, 1.0 + 3 * 2.0**-24, 3.4028235e38, 3.5e38, -1e300, 1.5e-45, 1e-46, 1e-39,
                        2.0**-126 * (1 - 2.0**-25), np.inf, -np.inf, np.nan])
        flat = v.reshape(-1)
        flat[r.integers(0, flat.size, odd.size * 3)] = np.tile(odd, 3)
    return np.ascontiguousarray(v).view(np.complex128)[..., 0]


def _bits(a):
    a = np.ascontiguousarray(a).view(np.float64)
    return np.where(np.isnan(a), np.float64(np.nan), a).view(np.uint64)


@gpu
@pytest.mark.parametrize("prec", ["double", "single", "half", "double_float"])
@pytest.mark.parametrize("dims,Ls,n_rhs", [((2, 2, 2, 4), 1, 1), ((4, 6, 2, 10), 1, 3), ((6, 2, 4, 6), 7, 2), ((8, 4, 4, 6), 12, 1)])
def test_round_trip(dims, Ls, n_rhs, prec):
    _need_gpu()
    import gpt_gb300 as g

    grid = g.grid(list(dims), getattr(g, prec))
    lay = g.layout.get(grid, Ls, n_rhs, five_d=Ls > 1)
    x = g.lattice(lay, g.full)
    V = int(np.prod(dims))
    special = prec in ("double", "single")
    src = [_values(((V, Ls, 4, 3) if Ls > 1 else (V, 4, 3)) + (2,), 11 + r, special) for r in range(n_rhs)]
    for r, v in enumerate(src):
        x.set_natural(v, r)
    for r, v in enumerate(src):
        got = np.asarray(x.get_natural(r)).reshape(v.shape)
        if prec == "double":
            assert np.array_equal(_bits(got), _bits(v))
        elif prec == "single":
            with np.errstate(over="ignore"):
                want = v.astype(np.complex64).astype(np.complex128)
            assert np.array_equal(_bits(got), _bits(want))
        elif prec == "double_float":  # 48-bit significands
            assert np.all(np.abs(got.real - v.real) <= 2.0**-47 * np.abs(v.real))
            assert np.all(np.abs(got.imag - v.imag) <= 2.0**-47 * np.abs(v.imag))
        else:  # 11-bit fractions of the largest component of the site
            m = np.maximum(np.abs(v.real), np.abs(v.imag)).max(axis=(-1, -2), keepdims=True)
            assert np.all(np.abs(got - v) <= 2.0**-10 * m)

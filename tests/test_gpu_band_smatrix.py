"""The O(Ls) form of the Mobius s-matrices (constant real b, c) against the
oracle and against the dense form, which zmobius with omega = 1 takes for the
same operator: fifth dimensions of 1 to 32 slices, packed right-hand sides,
walls of different mass, and coefficients on both sides of the rule that
chooses the form (|rho| <= 3/4)."""
import numpy as np
import pytest

gpu = pytest.mark.gpu
TOL = {"double": 1e-13, "double_float": 1e-13, "single": 1e-6, "half": 3e-3}
DIMS = [4, 2, 4, 6]


def _rand(shape, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal(shape) + 1j * r.standard_normal(shape)


def _set(lat, values):
    for r, v in enumerate(values):
        lat.set_natural(v, r)


@gpu
@pytest.mark.parametrize("Ls,n_rhs", [(1, 1), (2, 3), (5, 2), (7, 1), (12, 12), (16, 1), (32, 8)])
@pytest.mark.parametrize("b,c,M5", [(1.5, 0.5, 1.8), (1.0, 0.0, 1.8), (1.5, 1.0 / 2.2, 1.8), (2.0, 1.4, 1.2), (0.1, 0.0, 1.8)])
def test_band_form_matches_oracle_and_dense_form(Ls, n_rhs, b, c, M5):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import gpt_gb300 as g
    import oracle as o

    grid = g.grid(DIMS, g.double)
    U = g.qcd.gauge.random_su3(grid, 0.4, 23)
    p = dict(Ls=Ls, b=b, c=c, M5=M5, mass_plus=0.07, mass_minus=0.19, boundary_phases=[1, 1, 1, -1], n_rhs=n_rhs)
    op64 = g.qcd.fermion.mobius(U, p)
    dense64 = g.qcd.fermion.zmobius(U, dict({k: v for k, v in p.items() if k != "Ls"}, omega=[1.0] * Ls))
    ref = o.mobius(U.U, DIMS, Ls=Ls, b=b, c=c, M5=M5, mass_plus=0.07, mass_minus=0.19, boundary_phases=[1, 1, 1, -1])
    src = [_rand((grid.gsites, Ls, 4, 3), 40 + r) for r in range(n_rhs)]
    even = (np.add.reduce(o.coords(DIMS), axis=1) % 2 == 0)
    for prec in (g.double, g.double_float, g.single, g.half):
        op = op64 if prec is g.double else op64.converted(prec)
        dense = dense64 if prec is g.double else dense64.converted(prec)
        x = op.F_lattice()
        _set(x, src)
        for name in ("M", "Mdag", "Mdiag"):
            out = [q.F_lattice() for q in (op, dense)]
            for q, d in zip((op, dense), out):
                q._apply(name, d, x)
            for r in (0, n_rhs - 1):
                want = ref.apply(name, src[r]).reshape(src[r].shape)
                for d in out:
                    err = np.linalg.norm(d.get_natural(r) - want) / np.linalg.norm(want)
                    assert err < TOL[prec.name], (prec.name, name, r, err)
        # half fields: the site-local terms and the hop with an s-matrix on either side
        for name in ("Mooee", "MooeeDag", "MooeeInv", "MooeeInvDag", "Meooe", "MeooeDag"):
            sp = g.even
            full = [q.F_lattice() for q in (op, dense)]
            for q, f in zip((op, dense), full):
                h = x.half(sp)
                t = q.F_lattice(sp)
                q._apply(name, t, h)
                f.half(t.cb).tensor.copy_(t.tensor)
            want = ref.apply(name, src[-1], 0 if "Meooe" not in name else 1).reshape(src[-1].shape)
            mask = even if "Meooe" not in name else ~even
            for f in full:
                got = f.get_natural(n_rhs - 1)[mask]
                err = np.linalg.norm(got - want[mask]) / np.linalg.norm(want[mask])
                assert err < TOL[prec.name], (prec.name, name, err)

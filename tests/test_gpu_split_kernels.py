"""The kernels that spread one site over several threads (hop8_kernel,
local6_kernel) at the edges of their range, against the oracle: fields of less
than one tile of 16 sites, with a remainder tile, and of exactly and just above
the largest size they take; plus the reducing launches inside a CG."""
import numpy as np
import pytest


gpu = pytest.mark.gpu

PARAMS = dict(mass=0.1, csw_r=0.7, csw_t=1.2, xi_0=1.3, nu=0.9, isAnisotropic=True,
              boundary_phases=[np.exp(0.3j), 1.0, np.exp(-0.5j), -1.0])
# half-field sites 8, 24, 1080 (a remainder tile), 6000 / 6048 and 12288 / 15360
DIMS = [(2, 2, 2, 2), (4, 2, 2, 6), (6, 6, 6, 10), (10, 10, 10, 12), (12, 6, 12, 14), (16, 16, 12, 8), (16, 16, 12, 10)]
TOL = {"double": 1e-13, "double_float": 1e-13, "single": 1e-6}


def _rand(shape, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal(shape) + 1j * r.standard_normal(shape)


@gpu
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("kind", ["wilson_clover", "wilson_twisted_mass"])
def test_split_kernels_match_the_oracle(kind, dims):
    import gpt_gb300 as g
    import oracle as o

    if not __import__("torch").cuda.is_available():
        pytest.skip("needs a GPU")
    grid = g.grid(list(dims), g.double)
    U = g.qcd.gauge.random_su3(grid, 0.4, 17)
    if kind == "wilson_clover":
        op64 = g.qcd.fermion.wilson_clover(U, PARAMS)
        ref = o.wilson_clover(U.U, list(dims), **{k: v for k, v in PARAMS.items() if k != "isAnisotropic"})
    else:
        p = dict(mass=0.1, mu=0.23, boundary_phases=PARAMS["boundary_phases"])
        op64 = g.qcd.fermion.wilson_twisted_mass(U, p)
        ref = o.wilson_twisted_mass(U.U, list(dims), **p)
    s = _rand((grid.gsites, 4, 3), 5)
    for prec in (g.double, g.double_float, g.single):
        op = op64 if prec is g.double else op64.converted(prec)
        src = op.F_lattice()
        src[:] = s
        for name, got in (("M", op.M(src)), ("Mdag", op.M.adj()(src)), ("Dhop", op.Dhop(src)), ("Mdiag", op.Mdiag(src))):
            want = ref.apply(name, s)
            err = np.linalg.norm(got[:] - want) / np.linalg.norm(want)
            assert err < TOL[prec.name], (prec.name, name, err)


@gpu
@pytest.mark.parametrize("prec", ["double", "double_float", "single"])
@pytest.mark.parametrize("dims", [(2, 2, 2, 4), (6, 4, 6, 6), (10, 10, 10, 12)])
def test_split_kernels_inside_cg(dims, prec):
    import gpt_gb300 as g
    import oracle as o

    if not __import__("torch").cuda.is_available():
        pytest.skip("needs a GPU")
    grid = g.grid(list(dims), g.double)
    U = g.qcd.gauge.random_su3(grid, 0.4, 18)
    p = dict(mass=0.1, csw_r=1.0, csw_t=1.0, boundary_phases=[1, 1, 1, -1])
    op = g.qcd.fermion.wilson_clover(U, p)
    if prec != "double":
        op = op.converted(getattr(g, prec))
    ref = o.wilson_clover(U.U, list(dims), **p)
    b = _rand((grid.gsites, 4, 3), 6)
    src = op.F_lattice()
    src[:] = b
    eps = 1e-5 if prec == "single" else 1e-11
    cg = g.algorithms.inverter.cg({"eps": eps, "maxiter": 500})
    x = g.algorithms.inverter.preconditioned(g.qcd.fermion.preconditioner.eo2_ne(), cg)(op)(src)[:]
    assert cg.last.converged
    r = b - ref.apply("M", x)
    # the residual of M x = b is at most about ten times that of the normal equations here
    assert np.sqrt(o.norm2(r) / o.norm2(b)) < 10 * eps

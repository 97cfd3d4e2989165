"""The hops that read a record per 4D site (hop5_kernel, one inner site per
thread; hop5p_kernel, two): inner extents on both sides of the rule that
chooses between them, odd extents, tiles that end past the lattice, fields
aligned to 16 instead of 32 bytes, the reducing launches of a CG, and a new
gauge field in an old operator."""
import numpy as np
import pytest

gpu = pytest.mark.gpu
TOL = {"single": 1e-6, "half": 3e-3}


def _rand(shape, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal(shape) + 1j * r.standard_normal(shape)


def _need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


@gpu
@pytest.mark.parametrize("prec", ["single", "half"])
@pytest.mark.parametrize("Ls,n_rhs", [(8, 1), (10, 1), (5, 3), (12, 2), (31, 1), (32, 1), (11, 3), (16, 3), (12, 12), (16, 16)])
@pytest.mark.parametrize("dims", [(2, 2, 2, 4), (4, 6, 2, 10)])
def test_record_hops_match_oracle(dims, Ls, n_rhs, prec):
    _need_gpu()
    import gpt_gb300 as g
    import oracle as o

    dims = list(dims)
    grid = g.grid(dims, g.double)
    U = g.qcd.gauge.random_su3(grid, 0.4, 29)
    ph = [np.exp(0.4j), 1.0, -1.0, np.exp(-0.2j)]
    p = dict(Ls=Ls, b=1.5, c=0.5, M5=1.8, mass=0.1, boundary_phases=ph, n_rhs=n_rhs)
    op = g.qcd.fermion.mobius(U, p).converted(getattr(g, prec))
    ref = o.mobius(U.U, dims, Ls=Ls, b=1.5, c=0.5, M5=1.8, mass=0.1, boundary_phases=ph)
    x, y = op.F_lattice(), op.F_lattice()
    src = [_rand((grid.gsites, Ls, 4, 3), 60 + r) for r in range(n_rhs)]
    for r, v in enumerate(src):
        x.set_natural(v, r)
    for name in ("Dhop", "DhopDag", "M", "Mdag", "Dminus"):
        op._apply(name, y, x)
        for r in {0, n_rhs // 2, n_rhs - 1}:
            want = ref.apply(name, src[r])
            err = np.linalg.norm(y.get_natural(r) - want) / np.linalg.norm(want)
            assert err < TOL[prec], (name, r, err)


@gpu
@pytest.mark.parametrize("n_rhs", [5, 8, 12, 16])
def test_record_hops_of_packed_wilson_clover(n_rhs):
    _need_gpu()
    import gpt_gb300 as g
    import oracle as o

    dims = [4, 6, 4, 2]
    grid = g.grid(dims, g.double)
    U = g.qcd.gauge.random_su3(grid, 0.4, 30)
    p = dict(mass=0.1, csw_r=1.0, csw_t=1.0, boundary_phases=[1, 1, 1, -1])
    op = g.qcd.fermion.wilson_clover(U, dict(p, n_rhs=n_rhs)).converted(g.single)
    ref = o.wilson_clover(U.U, dims, **p)
    x = op.F_lattice()
    src = [_rand((grid.gsites, 4, 3), 70 + r) for r in range(n_rhs)]
    for r, v in enumerate(src):
        x.set_natural(v, r)
    for name, out in (("M", op.M(x)), ("Mdag", op.M.adj()(x))):
        for r in range(n_rhs):
            want = ref.apply(name, src[r])
            err = np.linalg.norm(out.get_natural(r) - want) / np.linalg.norm(want)
            assert err < 1e-6, (name, r, err)
    # the reducing launch: every right-hand side of a packed CG
    cg = g.algorithms.inverter.cg({"eps": 1e-6, "maxiter": 500})
    sol = g.algorithms.inverter.preconditioned(g.qcd.fermion.preconditioner.eo2_ne(), cg)(op)(x)
    assert cg.last.converged
    for r in range(n_rhs):
        res = src[r] - ref.apply("M", sol.get_natural(r))
        assert np.linalg.norm(res) < 1e-5 * np.linalg.norm(src[r]), r


@gpu
@pytest.mark.parametrize("prec,Ls", [("single", 32), ("half", 12)])
def test_fields_aligned_to_16_bytes(prec, Ls):
    """A caller of the C ABI may pass fields that are only 16-byte aligned."""
    _need_gpu()
    import torch

    import gpt_gb300 as g
    from gpt_gb300 import _lib

    grid = g.grid([4, 4, 4, 4], getattr(g, prec))
    U = g.qcd.gauge.random_su3(g.grid([4, 4, 4, 4], g.double), 0.4, 31).U
    op = g.qcd.fermion.mobius(g.qcd.gauge.gauge_field(grid, U),
                              dict(Ls=Ls, b=1.5, c=0.5, M5=1.8, mass=0.1, boundary_phases=[1, 1, 1, -1]))
    x = op.F_lattice()
    x[:] = _rand(x.layout.natural_shape(), 3)
    want = op.Dhop(x).tensor
    nb = x.tensor.numel()
    buf = [torch.zeros(nb + 32, dtype=torch.uint8, device="cuda")[16:16 + nb] for _ in range(2)]
    assert all(b.data_ptr() % 32 == 16 for b in buf)
    buf[0].copy_(x.tensor)
    _lib.check(_lib.load().gbf_apply(op.obj, _lib.OPCODES["Dhop"], _lib.ptrs([buf[0].data_ptr()]),
                                     _lib.ptrs([buf[1].data_ptr()]), 1, 2, g.core.stream_ptr()))
    assert torch.equal(buf[1], want)


@gpu
def test_records_follow_a_new_gauge_field():
    _need_gpu()
    import ctypes

    import gpt_gb300 as g
    from gpt_gb300 import _lib

    dims = [4, 4, 4, 6]
    grid = g.grid(dims, g.single)
    U = [g.qcd.gauge.gauge_field(grid, g.qcd.gauge.random_su3(g.grid(dims, g.double), 0.4, s).U) for s in (1, 2)]
    p = dict(Ls=8, b=1.5, c=0.5, M5=1.8, mass=0.1, boundary_phases=[1, 1, 1, -1])
    old, new = g.qcd.fermion.mobius(U[0], p), g.qcd.fermion.mobius(U[1], p)
    x = old.F_lattice()
    x[:] = _rand(x.layout.natural_shape(), 4)
    old.M(x)
    ptr, on_dev = U[1].ptr()
    _lib.check(_lib.load().gbf_update_gauge(old.obj, ctypes.c_void_p(ptr), on_dev, g.core.stream_ptr()))
    assert np.array_equal(old.M(x)[:], new.M(x)[:])

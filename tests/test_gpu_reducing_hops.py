"""The hops that end in a sum over the field, at sizes where a block takes more
than one tile, on both sides of the rules that choose between the kernels.  One
step of CG from zero is x = alpha b with alpha = |b|^2 / Re <b, A b>: the sum
comes from the hop, and the same number from the operator and two separate
sums.  In FP32 the two differ by the roundings of the per-site sums and of x
(a few 6e-8), in FP64 and double-float likewise (1e-15), in half by the storage
of the vectors (fractions of 5e-4 per component, averaged over the field)."""
import pytest

gpu = pytest.mark.gpu
TOL = {"double": 1e-13, "double_float": 1e-13, "single": 2e-6, "half": 1e-3}


def _need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


CASES = [
    # one inner site per thread: band and clover epilogue, even and odd extents, four to seven inner sites
    ("mobius", "single", (16, 16, 16, 8), 8, 1),
    ("mobius", "single", (16, 16, 16, 8), 12, 1),
    ("mobius", "single", (16, 16, 16, 12), 5, 1),
    ("mobius", "single", (16, 16, 10, 12), 7, 3),
    ("zmobius", "single", (16, 16, 16, 8), 8, 2),
    ("wilson_clover", "single", (16, 16, 16, 16), 1, 12),
    ("wilson_clover", "single", (16, 16, 16, 16), 1, 7),
    # two inner sites per thread
    ("mobius", "single", (16, 16, 16, 8), 12, 4),
    ("mobius", "single", (16, 16, 16, 8), 11, 3),
    ("mobius", "half", (16, 16, 16, 8), 12, 2),
    ("mobius", "half", (16, 16, 16, 8), 9, 1),
    ("mobius", "half", (16, 16, 16, 14), 5, 1),
    ("wilson_clover", "half", (16, 16, 16, 16), 1, 12),
    ("wilson_clover", "half", (16, 16, 16, 16), 1, 9),
    # one site per thread
    ("wilson_clover", "single", (24, 24, 24, 24), 1, 1),
    ("wilson_clover", "single", (24, 24, 24, 24), 1, 3),
    ("wilson_clover", "double", (16, 16, 16, 16), 1, 1),
    # eight threads per site: at the limit in FP64 and FP32, looping in FP64; in double-float inside and above it
    ("wilson_clover", "double", (16, 16, 12, 8), 1, 1),
    ("wilson_clover", "double", (12, 12, 12, 14), 1, 1),
    ("wilson_clover", "single", (16, 16, 12, 8), 1, 1),
    ("wilson_clover", "double_float", (16, 16, 16, 16), 1, 1),
    ("wilson_clover", "double_float", (20, 20, 20, 20), 1, 1),
    ("wilson_clover", "double_float", (24, 24, 24, 24), 1, 1),
    ("wilson_clover", "double_float", (24, 24, 24, 26), 1, 1),
    ("wilson_clover", "double_float", (16, 16, 16, 16), 1, 4),
    ("mobius", "double_float", (16, 16, 16, 8), 12, 1),
    ("mobius", "double", (8, 8, 8, 8), 12, 2),
]


@gpu
@pytest.mark.parametrize("name,prec,dims,Ls,n_rhs", CASES)
def test_first_cg_step_has_the_operators_alpha(name, prec, dims, Ls, n_rhs):
    _need_gpu()
    import torch

    import gpt_gb300 as g

    torch.cuda.empty_cache()
    grid = g.grid(list(dims), g.double)
    U = g.qcd.gauge.random_su3(grid, 0.3, 41)
    p = dict(boundary_phases=[1, 1, 1, -1], n_rhs=n_rhs)
    if name == "wilson_clover":
        op = g.qcd.fermion.wilson_clover(U, dict(p, mass=0.1, csw_r=1.0, csw_t=1.0))
    elif name == "mobius":
        op = g.qcd.fermion.mobius(U, dict(p, Ls=Ls, mass=0.1, M5=1.8, b=1.5, c=0.5))
    else:
        omega = [0.6 + 0.05 * i + (0.02j if i % 2 else -0.02j) for i in range(Ls)]
        op = g.qcd.fermion.zmobius(U, dict(p, mass=0.1, M5=1.8, b=1.0, c=0.0, omega=omega))
    if prec != "double":
        op = op.converted(getattr(g, prec))
    # Gaussian sources, another size for every right-hand side
    lay64 = g.layout.get(grid, Ls, n_rhs, five_d=name != "wilson_clover")
    b64 = g.lattice(lay64, g.odd)
    gen = torch.Generator("cuda").manual_seed(7)
    v = torch.randn(b64.tensor.numel() // 8, dtype=torch.float64, device="cuda", generator=gen)
    v = v.view(12, -1, n_rhs, Ls, 2) * torch.arange(1, n_rhs + 1, device="cuda").view(1, 1, n_rhs, 1, 1)
    b64.tensor.copy_(v.reshape(-1).view(torch.uint8))
    del v
    b, x = op.F_lattice(g.odd), op.F_lattice(g.odd)
    g.convert(b, b64)
    A = g.qcd.fermion.preconditioner.eo2_ne()(op).Mpc

    def per_rhs(z):
        return [q.real for q in (z if isinstance(z, (list, tuple)) else [z])]

    q = op.F_lattice(g.odd)
    A(q, b)
    bb, bq = per_rhs(g.norm2(b)), per_rhs(g.inner_product(b, q))
    cg = g.algorithms.inverter.cg({"eps": 1e-30, "maxiter": 1})
    runs = []
    for _ in range(2):
        x[:] = 0
        cg(A)(x, b)
        runs.append(x.tensor.clone())
        bx = per_rhs(g.inner_product(b, x))
        for r in range(n_rhs):
            want, got = bb[r] / bq[r], bx[r] / bb[r]
            assert abs(got - want) < TOL[prec] * want, (r, got, want)
    assert torch.equal(*runs)  # fixed order of the sums

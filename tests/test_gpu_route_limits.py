"""The rules that choose a kernel by the size of the field, on both sides of each
limit that the tests against the oracle are too small for.  The oracle here is
the FP64 operator on the GPU (one thread per site at these sizes, itself checked
against the CPU oracle); the tolerances are those of the oracle tests."""
import os
import subprocess
import sys

import pytest

gpu = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOL = {"double_float": 1e-13, "single": 1e-6, "half": 3e-3}


def _need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _operator(g, name, dims, Ls, n_rhs):
    U = g.qcd.gauge.random_su3(g.grid(list(dims), g.double), 0.4, 23)
    p = dict(boundary_phases=[1, 1, 1, -1], n_rhs=n_rhs, mass=0.1)
    if name == "wilson_clover":
        return g.qcd.fermion.wilson_clover(U, dict(p, csw_r=1.0, csw_t=1.0))
    return g.qcd.fermion.mobius(U, dict(p, Ls=Ls, M5=1.8, b=1.5, c=0.5))


def _gaussian(x, seed):
    import torch

    gen = torch.Generator("cuda").manual_seed(seed)
    x.tensor.copy_(torch.randn(x.tensor.numel() // 8, dtype=torch.float64, device="cuda", generator=gen).view(torch.uint8))
    return x


def _distance(g, a, b64):
    """|a - b| / |b| with a converted to FP64 (all right-hand sides together)."""
    import torch

    c = b64.new()
    g.convert(c, a)
    u, v = c.tensor.view(torch.float64), b64.tensor.view(torch.float64)
    return float(torch.linalg.vector_norm(u - v) / torch.linalg.vector_norm(v))


CASES = [
    # double-float: local6_kernel to 80,000 sites of a half field, reducing hop8_kernel to 100,000, with an
    # epilogue to 170,000, without to 1,000,000 and dslash_dd2_kernel above
    ("wilson_clover", "double_float", (20, 20, 20, 20), 1, 1),
    ("wilson_clover", "double_float", (20, 20, 20, 22), 1, 1),
    ("wilson_clover", "double_float", (24, 24, 24, 24), 1, 1),
    ("wilson_clover", "double_float", (24, 24, 24, 26), 1, 1),
    ("mobius", "double_float", (16, 16, 16, 30), 16, 1),
    ("mobius", "double_float", (16, 16, 16, 32), 16, 1),
] + [
    # the record hops at four to seven inner sites, from 100,000 sites on (and dslash_kernel just below)
    (name, prec, dims, Ls, n_rhs)
    for prec in ("single", "half")
    for name, dims, Ls, n_rhs in [
        ("mobius", (12, 18, 18, 12), 4, 1),
        ("mobius", (14, 18, 18, 12), 4, 1),
        ("mobius", (16, 16, 16, 12), 5, 1),
        ("mobius", (16, 16, 10, 14), 3, 2),
        ("mobius", (16, 16, 16, 8), 7, 1),
        ("wilson_clover", (16, 16, 16, 16), 1, 4),
        ("wilson_clover", (16, 16, 16, 14), 1, 5),
        ("wilson_clover", (16, 16, 10, 14), 1, 6),
        ("wilson_clover", (18, 14, 10, 14), 1, 7),
    ]
]


@gpu
@pytest.mark.parametrize("name,prec,dims,Ls,n_rhs", CASES)
def test_operators_on_both_sides_of_a_limit(name, prec, dims, Ls, n_rhs):
    _need_gpu()
    import torch

    import gpt_gb300 as g

    torch.cuda.empty_cache()
    op64 = _operator(g, name, dims, Ls, n_rhs)
    op = op64.converted(getattr(g, prec))
    x = op.F_lattice()
    g.convert(x, _gaussian(op64.F_lattice(), 3))
    x64, y64, y = op64.F_lattice(), op64.F_lattice(), op.F_lattice()
    g.convert(x64, x)
    for m in ("M", "Mdag", "Dhop", "DhopDag", "Mdiag"):
        op64._apply(m, y64, x64)
        op._apply(m, y, x)
        assert _distance(g, y, y64) < TOL[prec], m
    for parity in (g.even, g.odd):
        for m in ("Meooe", "MeooeDag", "Mooee", "MooeeInv", "MooeeInvDag", "DhopEO"):
            out = parity if m.startswith("Mooee") else parity.inv()
            op64._apply(m, y64.half(out), x64.half(parity))
            op._apply(m, y.half(out), x.half(parity))
            assert _distance(g, y.half(out), y64.half(out)) < TOL[prec], (m, parity)
    pc = g.qcd.fermion.preconditioner.eo2_ne()
    pc(op64).Mpc(y64.half(g.odd), x64.half(g.odd))
    pc(op).Mpc(y.half(g.odd), x.half(g.odd))
    assert _distance(g, y.half(g.odd), y64.half(g.odd)) < 10 * TOL[prec]  # four hops in a row


CHILD = r'''
import sys
import torch
import gpt_gb300 as g
from tests.test_gpu_route_limits import _operator, _gaussian
out = {}
for name, dims, Ls, n_rhs in [("mobius", (4, 6, 2, 10), 8, 1), ("mobius", (4, 6, 2, 10), 11, 3), ("mobius", (8, 4, 4, 6), 12, 4),
                              ("wilson_clover", (4, 6, 8, 4), 1, 12), ("mobius", (16, 16, 16, 12), 5, 1)]:
    op64 = _operator(g, name, dims, Ls, n_rhs)
    for prec in ("single", "half"):
        op = op64.converted(getattr(g, prec))
        x, y = op.F_lattice(), op.F_lattice()
        g.convert(x, _gaussian(op64.F_lattice(), 9))
        for m in ("Dhop", "DhopDag", "M", "Mdag"):
            op._apply(m, y, x)
            z = op64.F_lattice()
            g.convert(z, y)
            out[name, dims, Ls, n_rhs, prec, m] = z.tensor.view(torch.float64).cpu()
torch.save(out, sys.argv[1])
'''


@gpu
def test_record_hops_and_the_hop_without_records(tmp_path):
    """GBF_HOP5=0, also what an operator takes whose records do not fit: FP32
    the same bits, FP16 within one rounding of its storage (the site's scale is
    applied before or after the projection)."""
    _need_gpu()
    import torch

    got = []
    for hop5 in ("1", "0"):
        f = tmp_path / hop5
        r = subprocess.run([sys.executable, "-c", CHILD, str(f)], cwd=ROOT, env=dict(os.environ, GBF_HOP5=hop5), capture_output=True,
                           text=True, timeout=600)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
        got.append(torch.load(f))
    for key, a in got[0].items():
        b = got[1][key]
        if key[4] == "single":
            assert torch.equal(a, b), key
        else:
            # the fractions are rounded to 2^-11 of the site's largest component
            assert float((a - b).abs().max()) < 2.0**-9 * float(b.abs().max()), key
            assert float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b)) < 1e-3, key

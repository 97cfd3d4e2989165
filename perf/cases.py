"""The work that a program built on this framework has it do, as cases that can be timed.

Every case goes through the public Python entry points (g.qcd.fermion operators, the eo2_ne normal operator, the
inverters, the vector algebra).  A program keeps its operators, its destination fields and, for a solve, its solver
between calls, and so do these cases; every pass applies the operator to the whole field again.

A case is a dict of plain values: "kind" is "apply" (one operator application), "solve" (a whole eo2_ne solve) or
"vector" (a Krylov step's vector algebra); "op", "method", "prec", the lattice L0..L3, Ls and n_rhs say the rest.
"""
import math

import torch

import gpt_gb300 as g

# ---------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------
PHASES = (1.0, 1.0, 1.0, -1.0)
MOBIUS = dict(b=1.5, c=0.5, M5=1.8)
_BYTES = {"double": 192, "single": 96, "half": 52, "double_float": 192}
# a drawn case costs at most about this many FP32 5D-site hops (the largest listed case has 25.2 M)
_LARGEST = 24e6


def _case(name, kind, op, method, prec, dims, Ls=1, n_rhs=1, mass=0.05, **kw):
    c = dict(name=name, kind=kind, op=op, method=method, prec=prec, L0=dims[0], L1=dims[1], L2=dims[2], L3=dims[3],
             Ls=Ls, n_rhs=n_rhs, mass=mass)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: one application of the full matrix in double on 8^4 (a parity check, a smoke test, the
        # outer residual of a small request)
        _case("clover M 8^4 f64", "apply", "wilson_clover", "M", "double", (8, 8, 8, 8)),
        # the smallest whole solve: plain FP64 CG on 8^4, a few dozen iterations of six launches
        _case("clover cg 8^4 f64", "solve", "wilson_clover", "cg", "double", (8, 8, 8, 8)),
        # the headline: a mixed-precision solve on 32^4 (FP32 inner CG under FP64 defect correction)
        _case("clover mixed 32^4", "solve", "wilson_clover", "mixed", "double", (32, 32, 32, 32)),
        # the body of that inner CG by itself
        _case("clover normal 32^4 f32", "apply", "wilson_clover", "normal", "single", (32, 32, 32, 32)),
        # a few sources packed into one field on a ragged lattice
        _case("clover M ragged f32 x3", "apply", "wilson_clover", "M", "single", (12, 20, 14, 22), n_rhs=3),
        # FP64-class arithmetic on the FP32 pipe, the outer operator of a double-float solve, adjoint direction
        _case("clover Mdag 24^4 dd", "apply", "wilson_clover", "Mdag", "double_float", (24, 24, 24, 24)),
        # domain-wall matrix, one source, the shape of the 12-source propagator benchmark
        _case("mobius M 16^3x32 f32", "apply", "mobius", "M", "single", (16, 16, 16, 32), Ls=12, mass=0.01),
        # the inner CG's body with all 12 sources of a propagator packed
        _case("mobius normal 16^3x32 x12", "apply", "mobius", "normal", "single", (16, 16, 16, 32), Ls=12, n_rhs=12,
              mass=0.01),
        # a small domain-wall lattice with an odd number of slices
        _case("mobius normal ragged Ls7", "apply", "mobius", "normal", "single", (12, 8, 10, 14), Ls=7, mass=0.1),
        # the reference's own Dslash benchmark, the largest call
        _case("mobius Dhop 64x32^3 f32", "apply", "mobius", "Dhop", "single", (64, 32, 32, 32), Ls=12, mass=0.08),
        # FP16 storage (the half-precision inner solve), the hop on the packed 12 sources
        _case("mobius hop 16^3x32 x12 f16", "apply", "mobius", "DhopEO", "half", (16, 16, 16, 32), Ls=12, n_rhs=12,
              mass=0.01),
        # the vector algebra of an outer double-precision loop on 32^4: axpy_norm2, inner_product, norm2
        _case("vector 32^4 f64", "vector", "wilson_clover", "vector", "double", (32, 32, 32, 32)),
    ]


def _even(rng, lo, hi):
    """An even extent, spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, 2 * round(0.5 * math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    while True:
        family = rng.choice(["clover", "clover", "mobius", "mobius", "mobius", "solve", "vector"])
        dims = tuple(_even(rng, 6, 40) for _ in range(4))
        V = dims[0] * dims[1] * dims[2] * dims[3]
        mass = round(rng.uniform(0.01, 0.2), 4)
        if family == "clover":
            prec = rng.choice(["single", "single", "double", "double_float"])
            method = rng.choice(["M", "Mdag", "normal", "Meooe"])
            c = _case("", "apply", "wilson_clover", method, prec, dims, n_rhs=rng.choice([1, 1, 1, 2, 3, 4, 12]), mass=mass)
        elif family == "mobius":
            prec = rng.choice(["single", "single", "single", "half", "double_float", "double"])
            method = rng.choice(["DhopEO", "MooeeInv"] if prec == "half" else ["M", "Mdag", "normal", "normal", "Dhop", "MooeeInv"])
            shamir = rng.random() < 0.3
            c = _case("", "apply", "mobius", method, prec, dims, Ls=rng.choice([4, 6, 7, 8, 10, 12, 12, 16, 24]),
                      n_rhs=rng.choice([1, 1, 2, 3, 6, 12]), mass=mass, b=1.0 if shamir else 1.5, c=0.0 if shamir else 0.5)
        elif family == "solve":
            dims = tuple(_even(rng, 8, 24) for _ in range(4))
            V = dims[0] * dims[1] * dims[2] * dims[3]
            method = "cg" if V < 20000 else "mixed"
            c = _case("", "solve", "wilson_clover", method, "double", dims, n_rhs=rng.choice([1, 2, 4]), mass=mass)
        else:
            prec = rng.choice(["double", "single"])
            c = _case("", "vector", "wilson_clover", "vector", prec, dims, n_rhs=rng.choice([1, 1, 4, 12]), mass=mass)
        del c["name"]
        hops = V * c["Ls"] * c["n_rhs"] * (2 if c["method"] == "normal" else 1)
        hops *= {"double": 16, "double_float": 6}.get(c["prec"], 1) if c["kind"] != "vector" else 2
        if c["kind"] == "solve":
            hops = 40 * V * c["n_rhs"]
        if c["Ls"] * c["n_rhs"] <= 256 and hops <= _LARGEST:
            return c


def work(case):
    """Each input and each output once: the spinors, the links (48 bytes stored as two SU(3) rows, 72 or 144 in full)
    and the clover term; for a solve, one application's worth per iteration of a few dozen."""
    V = case["L0"] * case["L1"] * case["L2"] * case["L3"]
    n = case["n_rhs"] * case["Ls"]
    sites = V * n
    sb = _BYTES[case["prec"]]
    wide = case["prec"] in ("double", "double_float")
    lb = 144 if wide else (48 if n < 4 else 72)
    clover = case["op"] == "wilson_clover"
    cb = (576 if wide else 288) if clover else 0
    s_flops = 0 if clover else 24 * 2 * 3  # a bidiagonal or recursive fifth-dimension factor
    m = case["method"]
    if case["kind"] == "vector":
        return {"bytes": 6 * sb * sites, "flops": 24 * 8 * sites}
    if case["kind"] == "solve":
        inner, its = ("double", 45) if m == "cg" else ("single", 95)
        ib, il, ic = (192, 144, 576) if inner == "double" else (96, 48 if n < 4 else 72, 288)
        per = 0.5 * V * (2 * 8 * il + 4 * ic + n * 16 * ib)
        return {"bytes": its * per + 4 * sb * sites, "flops": its * sites * (2 * 1320 + 4 * 500)}
    if m in ("M", "Mdag"):
        return {"bytes": 2 * sb * sites + V * (4 * lb + cb), "flops": sites * (1320 + (500 if clover else 2 * s_flops))}
    if m == "normal":
        return {"bytes": sb * sites + V * (4 * lb + cb), "flops": sites * (2 * 1320 + 2 * (500 if clover else s_flops))}
    if m == "Dhop":
        return {"bytes": 2 * sb * sites + V * 4 * lb, "flops": sites * 1320}
    if m in ("DhopEO", "Meooe"):
        return {"bytes": sb * sites + V * 4 * lb, "flops": sites * (1320 + s_flops) // 2}
    return {"bytes": sb * sites, "flops": sites * s_flops // 2}  # MooeeInv


# ---------------------------------------------------------------------------------------------------------------
# inputs from the seed: an SU(3) gauge field near the identity (roughness 0.3) and Gaussian fermion fields
# ---------------------------------------------------------------------------------------------------------------
def _dims(case):
    return (case["L0"], case["L1"], case["L2"], case["L3"])


def _volume(case):
    return case["L0"] * case["L1"] * case["L2"] * case["L3"]


def _generator(seed, stream):
    return torch.Generator("cuda").manual_seed(1000003 * int(seed) + stream)


def _gauge(case, seed):
    """complex128 [4, V, 3, 3]: Gram-Schmidt of 1 + 0.3 * (Gaussian), third row the conjugate cross product."""
    V = _volume(case)
    U = torch.empty(4, V, 3, 3, dtype=torch.complex128, device="cuda")
    for mu in range(4):
        A = torch.randn(V, 2, 3, 2, dtype=torch.float64, device="cuda", generator=_generator(seed, mu))
        A = 0.3 * torch.view_as_complex(A)
        A[:, 0, 0] += 1.0
        A[:, 1, 1] += 1.0
        a = A[:, 0] / torch.linalg.vector_norm(A[:, 0], dim=-1, keepdim=True)
        b = A[:, 1] - (a.conj() * A[:, 1]).sum(-1, keepdim=True) * a
        b = b / torch.linalg.vector_norm(b, dim=-1, keepdim=True)
        U[mu, :, 0], U[mu, :, 1] = a, b
        U[mu, :, 2] = torch.linalg.cross(a, b).conj()
    return U


def _field(case, seed, stream, halves):
    """Gaussian values of a field in the layout of the double or single precision ([halves][planes][N][reals]);
    double_float and half fields are converted from these."""
    N = _volume(case) // 2 * case["Ls"] * case["n_rhs"]
    dt = torch.float64 if case["prec"] in ("double", "double_float") else torch.float32
    return torch.randn(halves * N * 24, dtype=dt, device="cuda", generator=_generator(seed, stream))


def _precision(name):
    return {"double": g.double, "single": g.single, "half": g.half, "double_float": g.double_float}[name]


def _lattice(case, values, cb):
    """The field as a lattice of the case's precision."""
    five = case["op"] == "mobius"
    grid = g.grid(list(_dims(case)), g.double if values.dtype == torch.float64 else g.single)
    lay = g.layout.get(grid, case["Ls"], case["n_rhs"], five_d=five)
    x = g.lattice(lay, cb, values.view(torch.uint8))
    if case["prec"] in ("double", "single"):
        return x
    y = g.lattice(g.layout.get(grid.converted(_precision(case["prec"])), case["Ls"], case["n_rhs"], five_d=five), cb)
    g.convert(y, x)
    return y


def _operator(case, seed):
    grid = g.grid(list(_dims(case)), _precision(case["prec"]))
    U = g.qcd.gauge.gauge_field(grid, torch.view_as_real(_gauge(case, seed)).reshape(-1))
    if case["op"] == "wilson_clover":
        return g.qcd.fermion.wilson_clover(U, dict(mass=case["mass"], csw_r=1.0, csw_t=1.0, boundary_phases=list(PHASES),
                                                   n_rhs=case["n_rhs"]))
    p = dict(MOBIUS, Ls=case["Ls"], mass=case["mass"], boundary_phases=list(PHASES), n_rhs=case["n_rhs"])
    p.update({k: case[k] for k in ("b", "c") if k in case})
    return g.qcd.fermion.mobius(U, p)


_HALF_IN = {"normal": g.odd, "Meooe": g.even, "DhopEO": g.even, "MooeeInv": g.odd}


def prepare(case, seed):
    if case["kind"] == "vector":
        x, y = (_lattice(case, _field(case, seed, 10 + i, 2), g.full) for i in range(2))
        return dict(case=case, x=x, y=y, out=y.new())
    op = _operator(case, seed)
    if case["kind"] == "solve":
        src = _lattice(case, _field(case, seed, 10, 2), g.full)
        inv, pc = g.algorithms.inverter, g.qcd.fermion.preconditioner
        if case["method"] == "cg":
            solver = inv.preconditioned(pc.eo2_ne(), inv.cg({"eps": 1e-12, "maxiter": 2000}))(op)
        else:
            inner = inv.preconditioned(pc.eo2_ne(), inv.cg({"eps": 1e-5, "maxiter": 2000}))
            solver = inv.defect_correcting(inv.mixed_precision(inner, g.single, g.double), eps=1e-12, maxiter=50)(op)
        return dict(case=case, op=op, solver=solver, src=src)
    m = case["method"]
    cb = _HALF_IN.get(m, g.full)
    src = _lattice(case, _field(case, seed, 10, 1 if m in _HALF_IN else 2), cb)
    dst = op.F_lattice(cb)
    fn = {"normal": lambda: g.qcd.fermion.preconditioner.eo2_ne()(op).Mpc, "M": lambda: op.M, "Mdag": lambda: op.M.adj(),
          "Dhop": lambda: op.Dhop, "DhopEO": lambda: op.DhopEO, "Meooe": lambda: op.Meooe,
          "MooeeInv": lambda: op.Mooee.inv()}[m]()
    s = dict(case=case, op=op, fn=fn, src=src, dst=dst)
    if case["prec"] == "double_float":  # a program that works in double takes the result over as double
        grid = g.grid(list(_dims(case)), g.double)
        s["out"] = g.lattice(g.layout.get(grid, case["Ls"], case["n_rhs"], five_d=case["op"] == "mobius"), cb)
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "vector":
        x, y, out = state["x"], state["y"], state["out"]
        n2 = g.axpy_norm2(out, -0.75, x, y)
        ip = g.inner_product(x, out)
        nx = g.norm2(x)
        one = case["n_rhs"] == 1
        ip = [ip] if one else ip
        return (_values(case["prec"], out.tensor), [n2] if one else n2, [z.real for z in ip], [z.imag for z in ip],
                [nx] if one else nx)
    if case["kind"] == "solve":
        return _values("double", state["solver"](state["src"]).tensor)
    state["fn"](state["dst"], state["src"])
    if case["prec"] == "double_float":
        g.convert(state["out"], state["dst"])
        return _values("double", state["out"].tensor)
    return _values(case["prec"], state["dst"].tensor, 1 if case["method"] in _HALF_IN else 2)


def _values(prec, t, halves=1):
    """The field's values by their type."""
    if prec == "half":
        t = t.view(halves, 52, -1)
        N = t.shape[2]
        t = t.reshape(halves, 52 * N)
        return [(t[h, :48 * N].view(torch.float16), t[h, 48 * N:].view(torch.float32)) for h in range(halves)]
    return t.view(torch.float32 if prec == "single" else torch.float64)


# ---------------------------------------------------------------------------------------------------------------
# the same in plain torch, complex128
# ---------------------------------------------------------------------------------------------------------------
# gamma_mu[r][perm] = coef in the basis with gamma_5 = diag(1, 1, -1, -1)
_PERM = ((3, 2, 1, 0), (3, 2, 1, 0), (2, 3, 0, 1), (2, 3, 0, 1))
_COEF = ((1j, 1j, -1j, -1j), (-1, 1, 1, -1), (1j, -1j, -1j, 1j), (1, 1, 1, 1))


class _Exact:
    """Fields are [4, 3, L3, L2, L1, L0, I] over the whole lattice, I = (rhs, s)."""

    def __init__(self, case, seed):
        self.case, self.L = case, _dims(case)
        self.I = case["n_rhs"] * case["Ls"]
        self.shape = (self.L[3], self.L[2], self.L[1], self.L[0])
        U = _gauge(case, seed)
        self.U = [[[U[mu, :, i, j].reshape(*self.shape, 1) for j in range(3)] for i in range(3)] for mu in range(4)]
        x = [torch.arange(n, device="cuda") for n in self.L]
        x = torch.meshgrid(x[3], x[2], x[1], x[0], indexing="ij")
        self.par = ((x[0] + x[1] + x[2] + x[3]) & 1).unsqueeze(-1)
        sites = torch.arange(_volume(case), device="cuda").reshape(self.shape)
        # checkerboard order: x0 / 2 fastest, then x1, x2, x3
        self.sites = [sites[self.par[..., 0] == p] for p in (0, 1)]
        if case["op"] == "wilson_clover":
            self._clover(U)
        else:
            self._fifth()

    def shift(self, f, mu, d, off):
        """f(x + d mu); off: the number of leading dimensions before (x3, x2, x1, x0)."""
        return torch.roll(f, -d, off + 3 - mu)

    def hop(self, psi, dag):
        out = torch.zeros_like(psi)
        sgn = 1.0 if dag else -1.0
        for mu in range(4):
            last = torch.ones(self.L[mu], dtype=torch.float64, device="cuda")
            last[-1] = PHASES[mu]
            last = last.reshape([-1 if k == 3 - mu else 1 for k in range(4)] + [1])
            for d in (1, -1):
                s = sgn if d == 1 else -sgn
                p, c = _PERM[mu], _COEF[mu]
                h = [[None] * 3 for _ in range(2)]
                for r in range(2):
                    for k in range(3):
                        h[r][k] = psi[r, k] + (s * c[r]) * psi[p[r], k]
                        if d == 1:
                            h[r][k] = self.shift(h[r][k], mu, 1, 0) * (-0.5 * last)
                for r in range(2):
                    uh = []
                    for i in range(3):
                        t = 0
                        for j in range(3):
                            u = self.U[mu][i][j] if d == 1 else self.U[mu][j][i].conj()
                            t = t + u * h[r][j]
                        uh.append(t if d == 1 else self.shift(t * (-0.5 * last), mu, -1, 0))
                    low = [q for q in (2, 3) if p[q] == r][0]
                    for i in range(3):
                        out[r, i] += uh[i]
                        out[low, i] += (s * c[low]) * uh[i]
        return out

    # -- site-local terms ----------------------------------------------------------------------------------------
    def _clover(self, U):
        U = U.reshape(4, *self.shape, 3, 3)

        def sh(m, mu, d):
            return self.shift(m, mu, d, 0)

        gam = torch.zeros(4, 4, 4, dtype=torch.complex128, device="cuda")
        for mu in range(4):
            for r in range(4):
                gam[mu, r, _PERM[mu][r]] = _COEF[mu][r]
        C = torch.zeros(2, *self.shape, 6, 6, dtype=torch.complex128, device="cuda")
        for mu in range(4):
            for nu in range(mu + 1, 4):
                up = sh(U[nu], mu, 1) @ sh(U[mu], nu, 1).mH @ U[nu].mH
                dn = sh(sh(U[nu], mu, 1).mH @ U[mu].mH @ U[nu], nu, -1)
                v = up - dn
                Q = U[mu] @ v + sh(v @ U[mu], mu, -1)
                F = 0.125 * (Q - Q.mH)
                sig = 0.5 * (gam[mu] @ gam[nu] - gam[nu] @ gam[mu])
                for b in range(2):
                    s = -0.5 * sig[2 * b:2 * b + 2, 2 * b:2 * b + 2]
                    C[b] += torch.einsum("st,...ac->...satc", s, F).reshape(*self.shape, 6, 6)
        C += (4.0 + self.case["mass"]) * torch.eye(6, dtype=torch.complex128, device="cuda")
        self.C, self.Ci = C, torch.linalg.inv(C)

    def _site(self, C, psi):
        out = torch.empty_like(psi)
        for b in range(2):
            v = psi[2 * b:2 * b + 2].reshape(6, *psi.shape[2:])
            for i in range(6):
                out[2 * b + i // 3, i % 3] = sum(C[b][..., i, j].unsqueeze(-1) * v[j] for j in range(6))
        return out

    def _fifth(self):
        c, Ls, m = self.case, self.case["Ls"], self.case["mass"]
        b5, c5, M5 = c.get("b", MOBIUS["b"]), c.get("c", MOBIUS["c"]), MOBIUS["M5"]
        one = torch.eye(Ls, dtype=torch.float64, device="cuda")
        self.B, self.A, self.Ai, self.G = [], [], [], []
        for ch in range(2):
            K = torch.zeros(Ls, Ls, dtype=torch.float64, device="cuda")
            for s in range(Ls):
                if ch == 0:
                    K[s, s - 1] = 1.0 if s else -m
                else:
                    K[s, (s + 1) % Ls] = 1.0 if s < Ls - 1 else -m
            B = b5 * one + c5 * K
            A = (4.0 - M5) * B + one - K
            self.B.append(B)
            self.A.append(A)
            self.Ai.append(torch.linalg.inv(A))
            self.G.append(B @ self.Ai[-1])

    def _s(self, Ms, psi, dag):
        v = psi.reshape(*psi.shape[:-1], self.case["n_rhs"], self.case["Ls"])
        out = [v[2 * b:2 * b + 2] @ (Ms[b].T if not dag else Ms[b]).to(torch.complex128) for b in range(2)]
        return torch.cat(out).reshape(psi.shape)

    def mooee(self, psi, dag=False, inv=False):
        if self.case["op"] == "wilson_clover":
            return self._site(self.Ci if inv else self.C, psi)
        return self._s(self.Ai if inv else self.A, psi, dag)

    def G_(self, psi, dag=False):
        return self._site(self.Ci, psi) if self.case["op"] == "wilson_clover" else self._s(self.G, psi, dag)

    def M(self, psi, dag=False):
        if self.case["op"] == "wilson_clover":
            return self.hop(psi, dag) + self.mooee(psi)
        if dag:
            return self._s(self.B, self.hop(psi, True), True) + self.mooee(psi, True)
        return self.hop(self._s(self.B, psi, False), False) + self.mooee(psi)

    def normal(self, psi):
        """Mpc^+ Mpc on the odd sites, Mpc = 1 - Dhop G Dhop G."""
        odd = self.par.to(torch.float64)
        w = psi - odd * self.hop(self.G_(self.hop(self.G_(psi), False)), False)
        return w - odd * self.G_(self.hop(self.G_(self.hop(w, True), True), True), True)

    # -- the layouts ---------------------------------------------------------------------------------------------
    def load(self, halves, parities):
        """Internal layout (double or single) to the whole lattice, zero on the other parity."""
        psi = torch.zeros(12, _volume(self.case), self.I, dtype=torch.complex128, device="cuda")
        per = halves.numel() // len(parities)
        for k, p in enumerate(parities):
            h = halves[k * per:(k + 1) * per]
            if h.dtype == torch.float32:
                h = h.double().reshape(6, -1, 2, 2).permute(0, 2, 1, 3).reshape(12, -1, 2)
            else:
                h = h.reshape(12, -1, 2)
            psi[:, self.sites[p], :] = torch.view_as_complex(h.contiguous()).reshape(12, -1, self.I)
        return psi.reshape(4, 3, *self.shape, self.I)

    def store(self, psi, parities, prec):
        psi = psi.reshape(12, -1, self.I)
        out = []
        for p in parities:
            h = torch.view_as_real(psi[:, self.sites[p], :].reshape(12, -1).contiguous())
            if prec == "single":
                out.append(h.reshape(6, 2, -1, 2).permute(0, 2, 1, 3).reshape(-1))
            elif prec == "half":
                m = h.abs().amax(dim=(0, 2))
                out.append(((h / m[None, :, None]).reshape(3, 4, -1, 2).permute(0, 2, 1, 3).reshape(-1), m))
            else:
                out.append(h.reshape(-1))
        return out if prec == "half" else torch.cat(out)


def _stored_half(values):
    """What a half-precision field holds of these single-precision values: 10-bit fractions of the site's largest."""
    h = values.reshape(6, -1, 4)
    m = h.abs().amax(dim=(0, 2))
    return ((h * (1.0 / m)[None, :, None]).half().float() * m[None, :, None]).reshape(-1)


def exact(case, seed):
    with torch.no_grad():
        return _exact(case, seed)


def _exact(case, seed):
    m, prec = case["method"], case["prec"]
    if case["kind"] == "vector":
        x, y = (_field(case, seed, 10 + i, 2).double() for i in range(2))
        out = -0.75 * x + y
        # [half][plane][site][rhs][reals of a plane] and the sums of each rhs; (re, im) are neighbours
        reals = 2 if prec == "double" else 4
        shape = (2, 24 // reals, -1, case["n_rhs"], reals // 2, 2)
        X, O = torch.view_as_complex(x.reshape(shape)), torch.view_as_complex(out.reshape(shape))
        ip = (X.conj() * O).sum(dim=(0, 1, 2, 4))
        return (out, *([float(v) for v in t] for t in ((O.abs() ** 2).sum(dim=(0, 1, 2, 4)), ip.real, ip.imag,
                                                        (X.abs() ** 2).sum(dim=(0, 1, 2, 4)))))
    E = _Exact(case, seed)
    if case["kind"] == "solve":
        b = E.load(_field(case, seed, 10, 2), (0, 1))
        # CG on M^+ M x = M^+ b, every right-hand side by itself
        dims = tuple(range(6))
        x = torch.zeros_like(b)
        r = E.M(b, True)
        p = r.clone()
        rr = (r.abs() ** 2).sum(dim=dims)
        stop = 1e-28 * rr
        for _ in range(2000):
            q = E.M(E.M(p), True)
            a = rr / (p.conj() * q).real.sum(dim=dims)
            x += a * p
            r -= a * q
            new = (r.abs() ** 2).sum(dim=dims)
            if bool((new <= stop).all()):
                break
            p = r + (new / rr) * p
            rr = new
        return E.store(x, (0, 1), prec)
    full = m not in _HALF_IN
    src = (0, 1) if full else (_HALF_IN[m].code,)
    v = _field(case, seed, 10, 2 if full else 1)
    if prec == "half":
        v = torch.cat([_stored_half(h) for h in v.reshape(len(src), -1)])
    psi = E.load(v, src)
    del v
    dst = src
    if m in ("M", "Mdag"):
        out = E.M(psi, m == "Mdag")
    elif m == "normal":
        out = E.normal(psi)
    elif m in ("Dhop", "DhopEO"):
        out = E.hop(psi, False)
        dst = src if m == "Dhop" else (1 - src[0],)
    elif m == "Meooe":
        out = E.hop(psi if case["op"] == "wilson_clover" else E._s(E.B, psi, False), False)
        dst = (1 - src[0],)
    else:
        out = E.mooee(psi, inv=True)
    return E.store(out, dst, "double" if prec == "double_float" else prec)

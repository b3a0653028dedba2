"""The work that this framework's users have it do, as measurable cases.

A case is one call (or one solve) through the public entry points: the classes
of `iroiro_b200`, `iroiro_b200.learned` and, for operators on resident fields,
`iro_dirac_apply_field` of the C ABI.  The kinds:

  apply      a Dirac operator on device-resident fields
  cg         Solver_CG on D^dag D, from host arrays or on resident fields
  multishift MultiShiftSolver_CG on resident fields
  qprop      Qprop_EvenOdd.calc on a point source, propagators to host storage
  force      the molecular-dynamics force, host arrays in and out
  update     a new gauge field on the same lattice (upload, clover term), then
             one application, as between two steps of an HMC trajectory
  ptc        the parallel-transport network applied to a resident field
  train      one training step's loss and gradient of that network

Links are U = exp(i eps H) with a random gauge transformation, kappa = 0.12,
csw = 1.0, eps = 0.2: the configuration of this repository's benchmark and
tests.  Sources are Gaussian or point sources.  Every solve goes to a true
relative residual of 1e-10.
"""
import math

import numpy as np
import torch

import iroiro_b200 as ib
from iroiro_b200 import learned

KAPPA, CSW, EPS, GOAL = 0.12, 1.0, 0.2, 1e-20
MASS = 0.5 / KAPPA - 4.0
OPS = {"wilson": ib.OP_WILSON_FULL, "wilson_eo": ib.OP_WILSON_SCHUR_EE,
       "clover": ib.OP_CLOVER_FULL, "clover_eo": ib.OP_CLOVER_SCHUR_EE}
REAL_BYTES = {"double": 8, "single": 4, "half": 2}
# iterations of CG on D^dag D to the goal on these fields, for work()
ITERATIONS = {"wilson": 200, "wilson_eo": 90, "clover": 210, "clover_eo": 95}


# ---- the cases -----------------------------------------------------------------------

def listed():
    return [
        # the operator on a small test lattice: two launches, all latency
        dict(name="mult_eo_8x16", kind="apply", op="wilson_eo", lattice="8,8,8,16", prec="double", nrhs=1, dag=False),
        # the benchmark's headline: the even-odd operator on a production lattice
        dict(name="mult_eo_32x64", kind="apply", op="wilson_eo", lattice="32,32,32,64", prec="double", nrhs=1, dag=False),
        # the 12 spin-colour columns of a propagator at once, on an odd-shaped lattice
        dict(name="mult_block12_ragged", kind="apply", op="wilson", lattice="12,20,28,44", prec="double", nrhs=12, dag=True),
        # the plain solver through host arrays on the small lattice of the reference's own runs
        dict(name="cg_host_8x16", kind="cg", op="wilson", lattice="8,8,8,16", inner="double", nrhs=1, host=True),
        # one clover solve in mixed precision on an ordinary lattice
        dict(name="cg_clover_half_24x48", kind="cg", op="clover_eo", lattice="24,24,24,48", inner="half", nrhs=1, host=False),
        # 12 sources as one block in mixed precision on a production lattice
        dict(name="cg_block12_half_32x64", kind="cg", op="wilson_eo", lattice="32,32,32,64", inner="half", nrhs=12, host=False),
        # the shifted systems of a 12-pole rational function
        dict(name="multishift12_32x64", kind="multishift", op="wilson_eo", lattice="32,32,32,64", inner="double", nshift=12),
        # a quark propagator from host to host: 12 clover inversions
        dict(name="qprop_clover_16x32", kind="qprop", op="clover_eo", lattice="16,16,16,32", inner="single"),
        # the clover force of one molecular-dynamics step
        dict(name="force_clover_16x32", kind="force", op="clover", lattice="16,16,16,32"),
        # the gauge field of the next molecular-dynamics step
        dict(name="update_clover_24x48", kind="update", op="clover_eo", lattice="24,24,24,48"),
        # the preconditioner's network, as flexible GCR applies it
        dict(name="ptc_32x64", kind="ptc", lattice="32,32,32,64", widths="4,4,4,4"),
        # one training step of the default network on a training lattice
        dict(name="train_16x32", kind="train", lattice="16,16,16,32", widths="4,16,16,16,4"),
    ]


def _draw_lattice(rng, lo, hi):
    """Even extents with a volume that is a multiple of 64, spread over the
    logarithm of the volume; t is the longest extent more often than not."""
    while True:
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        t = rng.uniform(1.0, 2.5)
        s = (v / t) ** 0.25
        L = [max(4, 2 * round(s * rng.uniform(0.75, 1.3) / 2)) for _ in range(3)]
        L.append(max(4, 2 * round(v / (L[0] * L[1] * L[2]) / 2)))
        V = math.prod(L)
        if V % 64 == 0 and lo <= V <= hi and L[3] <= 96:
            return ",".join(str(x) for x in L)


def draw(rng):
    kind = rng.choice(["apply", "apply", "cg", "cg", "multishift", "qprop", "force", "update", "ptc", "train"])
    c = {"kind": kind}
    if kind == "apply":
        c["op"] = rng.choice(list(OPS))
        c["nrhs"] = rng.choice([1, 1, 2, 3, 5, 12, 16])
        c["prec"] = rng.choice(list(REAL_BYTES))
        c["dag"] = rng.random() < 0.5
        c["lattice"] = _draw_lattice(rng, 1 << 10, (1 << 21) if c["nrhs"] == 1 else (1 << 20))
    elif kind == "cg":
        c["op"] = rng.choice(list(OPS))
        c["nrhs"] = rng.choice([1, 1, 1, 3, 4, 12])
        c["inner"] = rng.choice(list(REAL_BYTES))
        c["host"] = rng.random() < 0.4
        c["lattice"] = _draw_lattice(rng, 1 << 10, (1 << 19) // c["nrhs"] * 2)
    elif kind == "multishift":
        c["op"] = rng.choice(["wilson_eo", "clover_eo"])
        c["inner"] = rng.choice(list(REAL_BYTES))
        c["nshift"] = rng.choice([5, 8, 12, 15])
        c["lattice"] = _draw_lattice(rng, 1 << 11, 1 << 20)
    elif kind == "qprop":
        c["op"] = rng.choice(["wilson_eo", "clover_eo"])
        c["inner"] = rng.choice(list(REAL_BYTES))
        c["lattice"] = _draw_lattice(rng, 1 << 11, 1 << 18)
    elif kind == "force":
        c["op"] = rng.choice(["wilson", "wilson_eo", "clover"])
        c["lattice"] = _draw_lattice(rng, 1 << 11, 1 << 19)
    elif kind == "update":
        c["op"] = rng.choice(["wilson_eo", "clover_eo", "clover"])
        c["lattice"] = _draw_lattice(rng, 1 << 11, 1 << 20)
    else:
        c["widths"] = rng.choice(["4,4,4,4", "4,8,8,4", "4,16,16,16,4", "4,8,4"])
        c["lattice"] = _draw_lattice(rng, 1 << 11, (1 << 21) if kind == "ptc" else (1 << 18))
    return c


# ---- inputs --------------------------------------------------------------------------

def _extents(case):
    return [int(v) for v in case["lattice"].split(",")]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _exp(H):
    """exp(i H) of traceless Hermitian 3x3 matrices by scaling and squaring."""
    A = (1j / 16.0) * H
    E = torch.eye(3, dtype=H.dtype, device=H.device).expand_as(H)
    S = E.clone()
    for k in range(12, 0, -1):
        S = E + (A @ S) / k
    for _ in range(4):
        S = S @ S
    return S


def _random_hermitian(n, scale, g):
    th = scale * torch.randn((n, 8), generator=g, device="cuda", dtype=torch.float64) / 2
    H = torch.zeros((n, 3, 3), device="cuda", dtype=torch.complex128)
    for (a, b), (re, im) in {(0, 1): (0, 1), (0, 2): (3, 4), (1, 2): (5, 6)}.items():
        H[:, a, b] = torch.complex(th[:, re], -th[:, im])
        H[:, b, a] = H[:, a, b].conj()
    d = th[:, 7] / math.sqrt(3.0)
    H[:, 0, 0] = th[:, 2] + d
    H[:, 1, 1] = -th[:, 2] + d
    H[:, 2, 2] = -2.0 * d
    return H


def _links(L, g):
    """U_mu(x) = G(x) exp(i eps H_mu(x)) G(x+mu)^dag, [mu, t, z, y, x, 3, 3]."""
    V = math.prod(L)
    shape = (L[3], L[2], L[1], L[0], 3, 3)
    G = _exp(_random_hermitian(V, 1.5, g)).reshape(shape)
    U = torch.empty((4,) + shape, device="cuda", dtype=torch.complex128)
    for mu in range(4):
        u = _exp(_random_hermitian(V, EPS, g)).reshape(shape)
        U[mu] = G @ u @ torch.roll(G, -1, dims=3 - mu).mH
    return U


def _host(t):
    """A complex tensor as the float64 array of the reference's layouts."""
    return torch.view_as_real(t).reshape(-1).cpu().numpy()


def _spinors(L, n, g):
    shape = (n, L[3], L[2], L[1], L[0], 4, 3)
    return torch.complex(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64),
                         torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))


def _even_index(L):
    """Lexicographic sites of the even half, in order."""
    t, z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in (L[3], L[2], L[1], L[0])], indexing="ij")
    return torch.nonzero(((t + z + y + x) % 2 == 0).reshape(-1)).reshape(-1)


def _pick(f, L, op):
    """Full-lattice fields, or their even halves for an even-odd operator."""
    if not op.endswith("_eo"):
        return f
    return f.reshape(f.shape[0], -1, 4, 3)[:, _even_index(L)]


def _inputs(case, seed):
    """The case's links and fields as complex tensors: made from the seed alone."""
    L, g = _extents(case), _generator(seed)
    d = {"L": L, "U": _links(L, g)}
    kind = case["kind"]
    if kind in ("apply", "cg", "update", "multishift"):
        d["f"] = _pick(_spinors(L, case.get("nrhs", 1), g), L, case["op"])
    elif kind == "force":
        d["f"] = _pick(_spinors(L, 2, g), L, case["op"])
    elif kind == "qprop":
        d["site"] = [int(v) for v in (torch.rand(4, generator=g, device="cuda").cpu() * torch.tensor(L)).long()]
    else:
        d["f"] = _spinors(L, 2 if kind == "train" else 1, g)
        d["W"] = _weights(case, seed)
    return d


def _widths(case):
    return tuple(int(w) for w in case["widths"].split(","))


def _weights(case, seed):
    return learned.init_weights(_widths(case), seed=int(seed) % (1 << 31), scale=0.3)


class Resident(list):
    """Results that stay on the GPU: the DeviceFields, read back when the
    values are looked at."""

    def __iter__(self):
        return (f.download() if isinstance(f, ib.DeviceField) else f for f in list.__iter__(self))


class State:
    pass


def _operator(op, u, ctx, prec="double"):
    if op == "wilson":
        return ib.Dirac_Wilson(MASS, u, ctx=ctx, prec=prec)
    if op == "wilson_eo":
        return ib.Dirac_Wilson_EvenOdd(MASS, u, ctx=ctx, prec=prec)
    if op == "clover":
        return ib.Dirac_Clover(ib.Dirac_Wilson(MASS, u, ctx=ctx, prec=prec), CSW, u, ctx=ctx, prec=prec)
    return ib.Dirac_Clover_EvenOdd(MASS, CSW, u, ctx=ctx, prec=prec)


def _shifts(case):
    return np.geomspace(1e-4, 10.0, case["nshift"])


def prepare(case, seed):
    d = _inputs(case, seed)
    L, kind = d["L"], case["kind"]
    s = State()
    s.case, s.kind = case, kind
    s.ctx = ib.Context(L)
    s.u = _host(d["U"])
    if kind in ("ptc", "train"):
        s.ctx.upload_gauge(s.u)
        s.net = learned.PTCNet(s.ctx, _widths(case), weights=d["W"])
        n = 24 * s.ctx.V
        f = _host(d["f"])
        s.b = ib.DeviceField(s.ctx, 2, "single" if kind == "ptc" else "double").upload(f[:n])
        s.x = ib.DeviceField(s.ctx, 2, "single" if kind == "ptc" else "double")
        if kind == "train":
            s.x.upload(f[n:])
        return s
    s.D = _operator(case["op"], s.u, s.ctx, case.get("prec", "double"))
    sub = 0 if case["op"].endswith("_eo") else 2
    f = _host(d["f"]) if "f" in d else None
    if kind in ("apply", "update"):
        prec, nrhs = case.get("prec", "double"), case.get("nrhs", 1)
        s.b = ib.DeviceField(s.ctx, sub, prec, nrhs).upload(f)
        s.x = ib.DeviceField(s.ctx, sub, prec, nrhs)
    elif kind == "cg":
        s.solver = ib.Solver_CG(GOAL, 5000, ib.Fopr_DdagD(s.D), inner=case["inner"],
                                delta=0.02 if case["nrhs"] > 1 else 0.1)
        s.b, s.x = f, np.empty_like(f)
        if not case["host"]:
            s.b = ib.DeviceField(s.ctx, sub, "double", case["nrhs"]).upload(f)
            s.x = ib.DeviceField(s.ctx, sub, "double", case["nrhs"])
    elif kind == "multishift":
        s.solver = ib.MultiShiftSolver_CG(ib.Fopr_DdagD(s.D), GOAL, 5000, inner=case["inner"])
        s.b = ib.DeviceField(s.ctx, sub, "double").upload(f)
        s.x = ib.DeviceField(s.ctx, sub, "double", case["nshift"])
        s.shifts = _shifts(case)
    elif kind == "qprop":
        s.solver = ib.Qprop_EvenOdd(s.D, ib.Solver_CG(GOAL, 5000, ib.Fopr_DdagD(s.D), inner=case["inner"], delta=0.02))
        s.b = ib.Source_local(d["site"], L)
        s.x = np.empty(12 * 24 * s.ctx.V)
    elif kind == "force":
        s.b, s.x = f[:f.size // 2], f[f.size // 2:]
    return s


def _apply_field(s):
    D = s.D
    s.ctx.check(ib.lib().iro_dirac_apply_field(s.ctx.h, D.op, D.mass, D.csw, int(s.case.get("dag", False)), s.b.h, s.x.h),
                "iro_dirac_apply_field")


def run(s):
    kind, case = s.kind, s.case
    if kind == "apply":
        _apply_field(s)
        return Resident([s.x])
    if kind == "update":
        s.D.update_internal_state()
        _apply_field(s)
        return Resident([s.x])
    if kind == "cg":
        if not case["host"]:
            outs, rc = s.solver.solve_field(s.b, s.x)
            _converged(rc)
            return Resident([s.x])
        if case["nrhs"] == 1:
            s.solver.solve(s.x, s.b)
            return [s.x]
        x, outs, rc = s.solver.solve_many(s.b, case["nrhs"])
        _converged(rc)
        return [x]
    if kind == "multishift":
        s.solver.solve_field(s.b, s.x, s.shifts)
        return Resident([s.x])
    if kind == "qprop":
        return s.solver.calc(s.b, out=s.x)
    if kind == "force":
        return [s.D.md_force(s.b, s.x)]
    if kind == "ptc":
        s.ctx.check(s.net.L.iro_ptc_apply_field(s.ctx.h, s.net.h, s.b.h, s.x.h), "iro_ptc_apply_field")
        return Resident([s.x])
    loss, grads = s.net.loss_grad(s.ctx, s.b, s.x)
    return [loss] + grads


def _converged(rc):
    if rc != ib.OK:
        raise ib.ConvergenceError(rc, "not converged")


# ---- what a pass cannot do without -----------------------------------------------------

def work(case):
    L = _extents(case)
    V, kind = math.prod(L), case["kind"]
    if kind in ("ptc", "train"):
        w = _widths(case)
        mix = sum(9 * a * b * 3 * 8 for a, b in zip(w, w[1:]))       # channel mixing
        move = sum(8 * a * 66 for a in w[:-1])                        # SU(3) times colour vectors
        k = 3 if kind == "train" else 1
        return {"bytes": V * (2 * 24 * (8 if kind == "train" else 4) + 4 * 48), "flops": k * V * (mix + move)}
    op = case["op"]
    eo, clover = op.endswith("_eo"), op.startswith("clover")
    sites = V // 2 if eo else V
    nrhs = case.get("nrhs", {"qprop": 12}.get(kind, 1))
    hops = 2 if eo else 1
    per_site = hops * (1320 + (504 if clover else 0)) + 48
    if kind == "apply":
        r = REAL_BYTES[case["prec"]]
        data = V * 4 * 12 * r + (V * 72 * r if clover else 0) + 2 * 24 * r * sites * nrhs
        return {"bytes": data, "flops": sites * nrhs * per_site}
    if kind == "force":
        return {"bytes": V * 4 * 18 * 8 * 2 + 2 * 24 * 8 * sites, "flops": V * 4 * (2 * 1000 if not clover else 20000)}
    if kind == "update":
        return {"bytes": V * 4 * 18 * 8 + 2 * 24 * 8 * sites,
                "flops": V * (6 * 4 * 3 * 216 if clover else 200) + sites * per_site}
    # solves: every iteration reads the links (and clover blocks) once per
    # application of D and of D^dag, and moves p, r, x once each
    inner = case["inner"]
    r = REAL_BYTES[inner]
    n = ITERATIONS[op]
    links = 2 * (V * 4 * 12 * r + (V * 72 * r if clover else 0))
    vectors = 5 * 24 * r * sites * nrhs
    return {"bytes": n * (links + vectors), "flops": n * sites * nrhs * (2 * per_site + 6 * 24)}


def tolerance(case):
    """Four times what the same path shows against 64 bits, by storage."""
    kind = case["kind"]
    if kind == "apply":
        return {"double": {"rel": 1e-14, "max": 1e-12}, "single": {"rel": 1e-6, "max": 5e-5}, "half": {"rel": 2e-3, "max": 5e-2}}[case["prec"]]
    if kind == "update":
        return {"rel": 1e-13, "max": 1e-11}
    if kind == "force":
        return {"rel": 1e-13, "max": 1e-11}
    if kind in ("ptc", "train"):  # BF16 operands, FP32 sums
        return {"rel": 1e-2, "max": 0.2}
    # the iterate at a true residual of 1e-10: the next iteration's would do
    # too, and the condition number of D^dag D is a few hundred
    return {"rel": 1e-8, "max": 1e-6}


# ---- the same in plain torch, 64 bits ----------------------------------------------------

_I = 1j
# gamma_mu f = phase * f[perm] (the Dirac-Pauli basis of the reference)
_GAMMA = [([3, 2, 1, 0], [-_I, -_I, _I, _I]), ([3, 2, 1, 0], [-1, 1, 1, -1]),
          ([2, 3, 0, 1], [-_I, _I, _I, -_I]), ([0, 1, 2, 3], [1, 1, -1, -1])]
# i sigma_{mu nu} of the planes (1,2) (2,0) (0,1) (3,0) (3,1) (3,2)
_PLANES = [(1, 2), (2, 0), (0, 1), (3, 0), (3, 1), (3, 2)]
_ISIGMA = [([1, 0, 3, 2], [_I, _I, _I, _I]), ([1, 0, 3, 2], [1, -1, 1, -1]),
           ([0, 1, 2, 3], [_I, -_I, _I, -_I]), ([3, 2, 1, 0], [-_I, -_I, -_I, -_I]),
           ([3, 2, 1, 0], [-1, 1, -1, 1]), ([2, 3, 0, 1], [-_I, _I, -_I, _I])]


def _spin(table, f):
    perm, phase = table
    return f[..., perm, :] * torch.tensor(phase, device=f.device, dtype=f.dtype)[:, None]


def _shift(f, mu, sign, lead):
    """f(x + sign mu), with `lead` axes before t, z, y, x."""
    return torch.roll(f, -sign, dims=lead + 3 - mu)


def _times(U, f):
    return torch.einsum("tzyxab,rtzyxsb->rtzyxsa", U, f)


def _hop(U, f):
    acc = 0
    for mu in range(4):
        a = _times(U[mu], _shift(f, mu, 1, 1))
        acc = acc + a - _spin(_GAMMA[mu], a)
        a = _shift(_times(U[mu].mH, f), mu, -1, 1)
        acc = acc + a + _spin(_GAMMA[mu], a)
    return acc


def _gamma5(f):
    return f[..., [2, 3, 0, 1], :]


def _field_strength(U, mu, nu):
    up = U[nu] @ _shift(U[mu], nu, 1, 0) @ _shift(U[nu], mu, 1, 0).mH
    c = U[nu].mH @ U[mu] @ _shift(U[nu], mu, 1, 0)
    v = up.mH - _shift(c, nu, -1, 0).mH
    M = U[mu] @ v + _shift(v @ U[mu], mu, -1, 0)
    M = 0.5 * (M - M.mH)
    tr = torch.diagonal(M, dim1=-2, dim2=-1).sum(-1) / 3.0
    return 0.25 * (M - tr[..., None, None] * torch.eye(3, device=U.device, dtype=U.dtype))


class _Plain:
    """The operators on full-lattice fields [r, t, z, y, x, spin, colour]."""

    def __init__(self, op, U, L):
        self.U, self.L, self.op = U, L, op
        self.eo, self.clover = op.endswith("_eo"), op.startswith("clover")
        if self.clover:
            self.F = torch.stack([_field_strength(U, mu, nu) for mu, nu in _PLANES])
        if self.eo:
            m = torch.zeros(math.prod(L), device=U.device, dtype=torch.float64)
            m[_even_index(L)] = 1.0
            self.even = m.reshape(1, L[3], L[2], L[1], L[0], 1, 1)
            if self.clover:
                A = torch.zeros((L[3], L[2], L[1], L[0], 4, 3, 4, 3), device=U.device, dtype=U.dtype)
                for s in range(4):
                    for c in range(3):
                        A[..., s, c, s, c] = 1.0
                for k, (perm, phase) in enumerate(_ISIGMA):
                    for s in range(4):
                        A[..., s, :, perm[s], :] -= KAPPA * CSW * phase[s] * self.F[k]
                A = torch.linalg.inv(A.reshape(-1, 12, 12))
                self.Ainv = A

    def diag(self, f):
        if not self.clover:
            return f
        return f - KAPPA * CSW * sum(_times(self.F[k], _spin(_ISIGMA[k], f)) for k in range(6))

    def diag_inv(self, f):
        if not self.clover:
            return f
        r = f.shape[0]
        v = f.reshape(r, -1, 12).permute(1, 2, 0)
        return torch.matmul(self.Ainv, v).permute(2, 0, 1).reshape(f.shape)

    def mult(self, f, dag=False):
        if dag:
            return _gamma5(self.mult(_gamma5(f)))
        if not self.eo:
            return self.diag(f) - KAPPA * _hop(self.U, f)
        t = self.diag_inv(KAPPA * _hop(self.U, f)) * (1 - self.even)
        return (self.diag(f) - KAPPA * _hop(self.U, t)) * self.even

    def full(self, half):
        """An even half [r, sites, 4, 3] on the full lattice."""
        L = self.L
        f = torch.zeros((half.shape[0], math.prod(L), 4, 3), device=half.device, dtype=half.dtype)
        f[:, _even_index(L)] = half
        return f.reshape(half.shape[0], L[3], L[2], L[1], L[0], 4, 3)

    def take(self, f):
        return f if not self.eo else f.reshape(f.shape[0], -1, 4, 3)[:, _even_index(self.L)]

    def solve(self, b, sigma=0.0):
        """(D^dag D + sigma) x = b by CG, every right-hand side to 1e-13."""
        def dot(a, c):
            return (a.conj() * c).real.sum(dim=tuple(range(1, a.dim())), keepdim=True)
        x, r = torch.zeros_like(b), b.clone()
        p, rr = r.clone(), dot(b, b)
        goal = 1e-26 * rr
        for _ in range(1500):
            q = self.mult(self.mult(p), True) + sigma * p
            a = rr / dot(p, q)
            x += a * p
            r -= a * q
            new = dot(r, r)
            if bool((new < goal).all()):
                break
            p = r + (new / rr) * p
            rr = new
        return x


def _flat(t):
    return _host(t.to(torch.complex128))


def exact(case, seed):
    kind = case["kind"]
    L = _extents(case)
    V = math.prod(L)
    nrhs = case.get("nrhs", 1)
    # what would take the plain operators too long
    if V * nrhs * case.get("nshift", 1) > ((1 << 20) if kind in ("cg", "multishift") else (1 << 22)):
        return None
    d = _inputs(case, seed)
    U = d["U"]
    if kind in ("ptc", "train"):
        return _exact_network(case, d)
    P = _Plain(case["op"], U, L)
    if kind in ("apply", "update"):
        f = P.full(d["f"]) if P.eo else d["f"]
        return [_flat(P.take(P.mult(f, case.get("dag", False))))]
    if kind == "cg":
        b = P.full(d["f"]) if P.eo else d["f"]
        return [_flat(P.take(P.solve(b)))]
    if kind == "multishift":
        b = P.full(d["f"])
        x = [P.take(P.solve(b, float(sg))) for sg in _shifts(case)]
        return [_flat(torch.cat(x))]
    if kind == "qprop":
        # the first and the last of the 12 sources
        F = _Plain(case["op"][:-3], U, L)
        x, y, z, t = d["site"]
        b = torch.zeros((2, L[3], L[2], L[1], L[0], 4, 3), device="cuda", dtype=torch.complex128)
        b[0, t, z, y, x, 0, 0] = 1.0
        b[1, t, z, y, x, 3, 2] = 1.0
        # D x = b as D^dag D x = D^dag b, through the Schur complement
        bo = P.diag_inv(b * (1 - P.even))
        be = (b + KAPPA * _hop(U, bo)) * P.even
        ye = P.solve(P.mult(be, True))
        xo = P.diag_inv((b + KAPPA * _hop(U, ye)) * (1 - P.even))
        sol = ye + xo
        assert float((F.mult(sol) - b).norm()) < 1e-8
        return [_flat(sol[:1])] + [None] * 10 + [_flat(sol[1:])]
    # force: Re Tr(X F_mu(x)) is the derivative of Re(zeta^dag D eta) along
    # U_mu(x) -> (1 + e X) U_mu(x), so F = U G^dag with G the gradient in U
    U = U.clone().requires_grad_(True)
    P = _Plain(case["op"], U, L)
    eta, zeta = d["f"][:1], d["f"][1:]
    if P.eo:
        eta, zeta = P.full(eta), P.full(zeta)
    value = (zeta.conj() * P.mult(eta)).real.sum()
    (G,) = torch.autograd.grad(value, U)
    return [_flat((U.detach() @ G.mH))]


def _exact_network(case, d):
    U = d["U"]
    f = d["f"]
    W = [torch.tensor(w, device="cuda", dtype=torch.complex128, requires_grad=True) for w in d["W"]]
    x = f[:1]
    for w in W:
        # w: [displacement, out, in]
        acc = torch.einsum("oi,rtzyxia->rtzyxoa", w[0], x)
        for mu in range(4):
            acc = acc + torch.einsum("oi,rtzyxia->rtzyxoa", w[1 + 2 * mu], _times(U[mu], _shift(x, mu, 1, 1)))
            acc = acc + torch.einsum("oi,rtzyxia->rtzyxoa", w[2 + 2 * mu], _shift(_times(U[mu].mH, x), mu, -1, 1))
        x = acc
        if case["kind"] == "ptc":
            x = x.detach()
    if case["kind"] == "ptc":
        return [_flat(x)]
    target = f[1:]
    loss = (x - target).abs().square().sum() / target.abs().square().sum()
    G = torch.autograd.grad(loss, W)
    return [float(loss)] + [g.cpu().numpy() for g in G]

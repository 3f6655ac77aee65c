"""Performance cases of the framework: the calls its users make, at the sizes they make them.

A case is a dict of plain values.  `kind` says which call sequence it is:

  eval      one SIMP design evaluation of a resident optimisation loop (mixed precision):
            new densities, solve to `rtol`, compliance and dC/drho
  batch     many designs with several load cases each, solved together
  plain     the FP64 form with host buffers: densities in, displacement, compliance and
            dC/drho out; `ks` adds the KS-aggregated stress and its total derivative
  heat      nonlinear conduction: Newton, mean temperature, its adjoint sensitivities
  tangent   Green-Lagrange residual and tangent of a host program that drives its own
            Newton-Krylov iteration: assemble at X, then one product with the tangent
  filter    the density filter and its transpose on device vectors (one design step)

listed() holds the named cases, draw(rng) more of the same ranges, prepare(case, seed) what
a program holds before the call, run(state) the call, work(case) the bytes and operations
it cannot do without, exact(case, seed) the same outputs from plain FP64 torch.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "mast-multiphysics_gb300"))
import mastgpu as M  # noqa: E402

PRECISION = {"tf32x3": M.MIXED_TF32X3, "bf16x3": M.MIXED_BF16X3}
BATCH_SIZES = M.BATCH_SIZES
NU, PENAL, EMIN = 0.3, 3.0, 1e-9
KS_P, KS_SIGMA0 = 8.0, 1.0


def listed():
    return [
        # the smallest grid of the batched mix, on its own: launches and latency only
        dict(name="eval_16x8x8", kind="eval", nx=16, ny=8, nz=8, precision="tf32x3", rtol=1e-9, u=False),
        # a mid-size design solved tightly, with the displacement field (post-processing)
        dict(name="eval_48x24x24_tight", kind="eval", nx=48, ny=24, nz=24, precision="tf32x3", rtol=1e-10, u=True),
        # a grid that coarsens once and then is odd in two directions
        dict(name="eval_90x46x38", kind="eval", nx=90, ny=46, nz=38, precision="tf32x3", rtol=1e-9, u=False),
        # the headline benchmark, at its tolerance (the others a step finer, as an optimiser's
        # last iterations are run)
        dict(name="eval_128x64x64", kind="eval", nx=128, ny=64, nz=64, precision="tf32x3", rtol=1e-8, u=False),
        # the BF16 operator
        dict(name="eval_64x32x32_bf16", kind="eval", nx=64, ny=32, nz=32, precision="bf16x3", rtol=1e-9, u=False),
        # a tenth of the batched benchmark: uneven designs, 1 to 4 load cases each
        dict(name="batch_24", kind="batch", designs=24, grids=9, nx=0, ny=0, nz=0, cases=4),
        # the largest grid of the request mix, two load cases
        dict(name="batch_192x96x96", kind="batch", designs=1, grids=0, nx=192, ny=96, nz=96, cases=2),
        # the plain FP64 form at its benchmark size (uniform density, 1e-10)
        dict(name="plain_24x12x12", kind="plain", nx=24, ny=12, nz=12, uniform=True, rtol=1e-10, ks=False),
        # a stress-constrained evaluation in FP64
        dict(name="plain_stress_40x20x20", kind="plain", nx=40, ny=20, nz=20, uniform=False, rtol=1e-10, ks=True),
        # nonlinear conduction at its benchmark size
        dict(name="heat_200x200", kind="heat", nx=200, ny=200),
        # residual and tangent of the large-deflection element
        dict(name="tangent_64x32x32", kind="tangent", nx=64, ny=32, nz=32),
        # the filter at the headline grid
        dict(name="filter_128x64x64", kind="filter", nx=128, ny=64, nz=64, radius=2.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi, max_elems):
    """A cantilever grid of about 2:1:1, any parity, at most max_elems elements."""
    while True:
        m = 1 << rng.randint(0, 2)
        ny = max(1, _log_int(rng, lo, hi) // m) * m
        nx = max(1, int(round(ny * rng.uniform(1.0, 2.2) / m))) * m
        nz = max(1, int(round(ny * rng.uniform(0.6, 1.2) / m))) * m
        if min(nx, ny, nz) >= min(lo, 4) and nx * ny * nz <= max_elems:
            return nx, ny, nz


def draw(rng: random.Random):
    kind = rng.choice(["eval", "eval", "eval", "batch", "plain", "heat", "tangent", "filter"])
    if kind == "eval":
        bf16 = rng.random() < 0.25
        if bf16:  # grids that coarsen at least twice: the split BF16 form needs the multigrid
            s = 4 * _log_int(rng, 2, 8)
            nx, ny, nz = 2 * s, s, s
        else:
            nx, ny, nz = _grid(rng, 8, 64, 400000)
        tight = (not bf16) and rng.random() < 0.3
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision="bf16x3" if bf16 else "tf32x3",
                    rtol=1e-10 if tight else 1e-9, u=tight)
    if kind == "batch":
        return dict(kind=kind, designs=_log_int(rng, 3, 24), grids=rng.randint(1, 1 << 20), nx=0, ny=0, nz=0, cases=4)
    if kind == "plain":
        nx, ny, nz = _grid(rng, 4, 24, 20000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, uniform=rng.random() < 0.3, rtol=1e-10, ks=rng.random() < 0.4)
    if kind == "heat":
        return dict(kind=kind, nx=_log_int(rng, 24, 256), ny=_log_int(rng, 24, 256))
    if kind == "tangent":
        nx, ny, nz = _grid(rng, 6, 36, 70000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz)
    nx, ny, nz = _grid(rng, 8, 96, 1000000)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, radius=rng.choice([1.5, 2.0, 2.5, 3.0, 3.5]))


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return np.random.default_rng(seed)


def _densities(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    if case.get("uniform"):  # a homogeneous start design: the level of an optimiser's volume bound
        return np.full(n, 0.45 + 0.1 * _rng(seed).random())
    return _rng(seed).uniform(0.01, 1.0, n)


def _batch_designs(case, seed):
    """Grids and load spans from the case (a program's fixed chains), densities from the seed."""
    shape = _rng(case["grids"])
    out = []
    rng = _rng(seed)
    for d in range(case["designs"]):
        if case["nx"]:
            nx, ny, nz, nc = case["nx"], case["ny"], case["nz"], case["cases"]
        else:
            nx, ny, nz = BATCH_SIZES[int(shape.integers(len(BATCH_SIZES)))]
            nc = int(shape.integers(1, case["cases"] + 1))
        spans = []
        for _ in range(nc):
            j0 = int(shape.integers(0, ny + 1))
            spans.append((j0, int(shape.integers(j0, ny + 1))))
        out.append(dict(nx=nx, ny=ny, nz=nz, rho=rng.uniform(0.01, 1.0, nx * ny * nz), spans=spans))
    return out


class _DeviceArray:
    """A device buffer of the library as a torch tensor, which keeps the handle that owns it."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(int(ptr), False), version=2)


def _device(owner, ptr, n):
    return torch.as_tensor(_DeviceArray(owner, ptr, n), device="cuda")


def _filter_mask(case, seed):
    """Design-variable mask: a passive frame at one end of the domain."""
    dv = np.ones((case["nz"], case["ny"], case["nx"]), dtype=np.uint8)
    dv[:, :, : max(1, case["nx"] // 16)] = 0
    return dv.reshape(-1)


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k == "eval":
        s["problem"] = M.simp_cantilever(case["nx"], case["ny"], case["nz"])
        s["rho"] = torch.from_numpy(_densities(case, seed)).cuda()
        s["opts"] = M.default_opts(precision=PRECISION[case["precision"]], rtol=case["rtol"], inner_rtol=1e-2)
    elif k == "batch":
        designs = _batch_designs(case, seed)
        s["batch"] = M.Batch(designs)
        s["rho"] = [torch.from_numpy(d["rho"]).cuda() for d in designs]
        s["opts"] = M.default_opts(precision=M.MIXED_TF32X3, rtol=1e-9, inner_rtol=1e-2)
    elif k == "plain":
        s["problem"] = M.simp_cantilever(case["nx"], case["ny"], case["nz"])
        s["rho"] = _densities(case, seed)
        s["opts"] = M.default_opts(precision=M.PLAIN_FP64, rtol=case["rtol"])
    elif k == "heat":
        s["problem"] = M.heat_square(case["nx"], case["ny"])
        s["scale"] = _rng(seed).uniform(0.5, 1.5, case["nx"] * case["ny"])
        s["opts"] = M.default_opts(precision=M.PLAIN_FP64, rtol=1e-10, newton_rtol=1e-10, krylov=M.KRYLOV_CG)
        s["adjoint"] = M.default_opts(precision=M.PLAIN_FP64, rtol=1e-10, krylov=M.KRYLOV_BICGSTAB)
    elif k == "tangent":
        p = M.simp_cantilever(case["nx"], case["ny"], case["nz"], physics=M.PHYS_HEX8_NONLINEAR, load=0.01)
        rng = _rng(seed)
        p.set_design(rng.uniform(0.3, 1.0, p.n_elems))
        s["problem"] = p
        s["X"] = rng.normal(scale=1e-3, size=p.n_dofs)
        s["v"] = rng.normal(size=p.n_dofs)
    elif k == "filter":
        n = case["nx"] * case["ny"] * case["nz"]
        s["filter"] = M.Filter.grid(case["nx"], case["ny"], case["nz"], case["radius"], dv=_filter_mask(case, seed))
        s["rho"] = torch.from_numpy(_rng(seed).uniform(0.01, 1.0, n)).cuda()
        s["g"] = torch.from_numpy(_rng(seed + 1).normal(size=n)).cuda()
        s["out"] = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2)]
    else:
        raise ValueError(k)
    if torch.cuda.is_available():
        torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ the calls
def _run_eval(s):
    p, o = s["problem"], s["opts"]
    p.set_design_device(s["rho"].data_ptr())
    rc, _ = p.solve_resident(o)
    M.check(rc, "mg_solve")
    c = ctypes.c_double()
    M.check(M.lib().mg_compliance_resident(p.h, ctypes.byref(c)), "mg_compliance_resident")
    out = {"compliance": c.value, "dc": _device(p, M.lib().mg_sensitivities_device(p.h), p.n_elems)}
    if s["case"]["u"]:
        out["u"] = _device(p, M.lib().mg_solution_device(p.h), p.n_dofs)
    return out


def _run_batch(s):
    b = s["batch"]
    for d, rho in enumerate(s["rho"]):
        b.set_design_device(d, rho.data_ptr())
    b.solve(s["opts"])
    out = []
    for d in range(b.n_designs):
        comp, dc, _ = b.results(d)
        out.append({"compliance": comp, "dc": dc})
    return out


def _run_plain(s):
    p = s["problem"]
    p.set_design(s["rho"])
    u, _ = p.solve(s["opts"])
    c, dc = p.compliance()
    out = {"u": u, "compliance": c, "dc": dc}
    if s["case"]["ks"]:
        out["ks"], out["max_vm"], out["dks"] = p.ks_stress(KS_P, KS_SIGMA0, PENAL)
    return out


def _run_heat(s):
    p = s["problem"]
    p.set_elem_scale(s["scale"])
    T, _ = p.solve(s["opts"])
    q, dk0, ds = p.mean_temperature(opts=s["adjoint"])
    return {"T": T, "q": q, "dk0": dk0, "ds": ds}


def _run_tangent(s):
    p = s["problem"]
    R = p.residual_and_jacobian(s["X"])
    return {"R": R, "Jv": p.spmv(s["v"])}


def _run_filter(s):
    f, L = s["filter"], M.lib()
    a, b = s["out"]
    vp = ctypes.c_void_p
    M.check(L.mg_filter_apply_device(f.h, vp(s["rho"].data_ptr()), vp(a.data_ptr()), 0, None), "mg_filter_apply_device")
    M.check(L.mg_filter_apply_device(f.h, vp(s["g"].data_ptr()), vp(b.data_ptr()), 1, None), "mg_filter_apply_device")
    return {"filtered": a, "gradient": b}


_RUN = dict(eval=_run_eval, batch=_run_batch, plain=_run_plain, heat=_run_heat, tangent=_run_tangent,
            filter=_run_filter)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ------------------------------------------------------------------ the work of one pass
def _hex_counts(nx, ny, nz):
    return nx * ny * nz, 3 * (nx + 1) * (ny + 1) * (nz + 1)


def _iterations(n_elems):
    """Conjugate-gradient iterations of a multigrid-preconditioned design evaluation."""
    return 20 if n_elems < 1e4 else 30


def _eval_work(nx, ny, nz):
    """Per iteration: the operator and a V-cycle of two smoothing steps on each side (5 level-0
    applications, coarser levels 1/7 more), each with its operands once in FP32."""
    ne, n = _hex_counts(nx, ny, nz)
    it = _iterations(ne)
    per_it = (5 * (12 * n + 4 * ne) * 8 / 7 + 28 * n, (5 * 8 / 7 * 255 * ne + 10 * n))
    once = (8 * ne * 3 + 4 * 8 * (3 * n + ne), 4 * 255 * ne * 10)
    return it * per_it[0] + once[0], it * per_it[1] + once[1]


def work(case):
    k = case["kind"]
    if k == "eval":
        b, f = _eval_work(case["nx"], case["ny"], case["nz"])
    elif k == "batch":
        b = f = 0.0
        shape = _rng(case["grids"])
        for _ in range(case["designs"]):
            if case["nx"]:
                nx, ny, nz, nc = case["nx"], case["ny"], case["nz"], case["cases"]
            else:
                nx, ny, nz = BATCH_SIZES[int(shape.integers(len(BATCH_SIZES)))]
                nc = int(shape.integers(1, case["cases"] + 1))
            for _ in range(nc):
                j0 = int(shape.integers(0, ny + 1))
                shape.integers(j0, ny + 1)
            w = _eval_work(nx, ny, nz)
            b, f = b + nc * w[0], f + nc * w[1]
    elif k == "plain":
        ne, n = _hex_counts(case["nx"], case["ny"], case["nz"])
        nnz = 81 * n
        it = 14 * max(case["nx"], case["ny"], case["nz"]) * (2 if case["ks"] else 1)
        b = it * (8.0 * nnz + 4 * nnz / 3 + 10 * 8 * n) + 8.0 * nnz
        f = it * (2.0 * nnz + 14 * n) + 1e4 * ne
    elif k == "heat":
        ne, n = case["nx"] * case["ny"], (case["nx"] + 1) * (case["ny"] + 1)
        it = 3 * 3 * max(case["nx"], case["ny"])  # two Newton steps and the adjoint
        b = it * (12.0 * 9 * n + 10 * 8 * n) + 3 * 12.0 * 9 * n
        f = it * (2.0 * 9 * n + 12 * n) + 3 * 400.0 * ne
    elif k == "tangent":
        ne, n = _hex_counts(case["nx"], case["ny"], case["nz"])
        b = 2 * 8.0 * 81 * n + 12 * 8 * n / 3 + 8 * ne + 4 * 8 * n
        # half of the symmetric tangent (36 of 64 node pairs), the gradients and the product
        f = (36 * 8 * 82 + 10000.0) * ne + 2 * 81 * n
    else:
        n = case["nx"] * case["ny"] * case["nz"]
        m = len(_offsets(case["radius"]))
        b = 2 * (2 * 8.0 + 1 + 8) * n
        f = 2 * 2.0 * m * n / 2  # the stencil is symmetric: points of equal weight are added first
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------ FP64 values
_D = lambda: torch.device("cuda" if torch.cuda.is_available() else "cpu")  # noqa: E731
_HEX = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=_D())


def _hex_gradients():
    """Shape gradients of the unit cube at the 2x2x2 Gauss points: (8 points, 8 nodes, 3)."""
    g = 0.5 / math.sqrt(3.0)
    pts = [(0.5 + (2 * (q & 1) - 1) * g, 0.5 + (2 * (q >> 1 & 1) - 1) * g, 0.5 + (2 * (q >> 2) - 1) * g)
           for q in range(8)]
    G = np.zeros((8, 8, 3))
    for q, x in enumerate(pts):
        for a, c in enumerate(_HEX):
            h = [x[i] if c[i] else 1 - x[i] for i in range(3)]
            d = [1.0 if c[i] else -1.0 for i in range(3)]
            G[q, a] = (d[0] * h[1] * h[2], h[0] * d[1] * h[2], h[0] * h[1] * d[2])
    return G


def _lame():
    return NU / ((1 + NU) * (1 - 2 * NU)), 0.5 / (1 + NU)


def _unit_stiffness():
    lam, mu = _lame()
    S = np.einsum("qai,qbj->aibj", _hex_gradients(), _hex_gradients()) / 8.0
    tr = np.einsum("aibi->ab", S)
    K = lam * S + mu * np.einsum("aibj->ajbi", S) + mu * np.einsum("ab,ij->aibj", tr, np.eye(3))
    return K.reshape(24, 24)


def _corners(v, nx, ny, nz):
    """(..., NZ, NY, NX, 3) nodal vectors -> (..., n_el, 8, 3)"""
    lead = v.shape[:-4]
    return torch.stack([v[..., c[2]:c[2] + nz, c[1]:c[1] + ny, c[0]:c[0] + nx, :].reshape(*lead, -1, 3)
                        for c in _HEX], dim=-2)


def _add_corners(fe, nx, ny, nz):
    lead = fe.shape[:-3]
    y = torch.zeros(*lead, nz + 1, ny + 1, nx + 1, 3, dtype=fe.dtype, device=fe.device)
    for a, c in enumerate(_HEX):
        y[..., c[2]:c[2] + nz, c[1]:c[1] + ny, c[0]:c[0] + nx, :] += fe[..., a, :].reshape(*lead, nz, ny, nx, 3)
    return y


def _pcg(apply, diag, b, rtol=1e-13, maxit=40000):
    """Jacobi-preconditioned CG on stacked right-hand sides (leading dimension)."""
    dims = tuple(range(1, b.dim()))
    dot = lambda a, c: (a * c).sum(dim=dims, keepdim=True)  # noqa: E731
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = dot(r, z)
    stop = rtol * rtol * dot(b, b)
    for it in range(maxit):
        q = apply(p)
        alpha = rz / dot(p, q).clamp_min(1e-300)
        x += alpha * p
        r -= alpha * q
        if it % 25 == 24 and bool((dot(r, r) <= stop).all()):
            break
        z = r / diag
        rz, old = dot(r, z), rz
        p = z + (rz / old.clamp_min(1e-300)) * p
    return x


class _Simp:
    """The cantilever of one density field in FP64 torch (node arrays NZ x NY x NX x 3)."""

    def __init__(self, nx, ny, nz, rho):
        self.g = (nx, ny, nz)
        self.rho = _t(rho)
        self.E = EMIN + (1 - EMIN) * self.rho ** PENAL
        self.dE = (1 - EMIN) * PENAL * self.rho ** (PENAL - 1)
        self.K = _t(_unit_stiffness())
        self.free = torch.ones(nz + 1, ny + 1, nx + 1, 1, dtype=torch.float64, device=_D())
        self.free[:, :, 0] = 0.0
        d = torch.diagonal(self.K).reshape(8, 3)
        self.diag = _add_corners(self.E[:, None, None] * d, nx, ny, nz)

    def apply(self, v):
        nx, ny, nz = self.g
        ve = _corners(v * self.free, nx, ny, nz)
        fe = (ve.reshape(-1, 24) @ self.K).reshape(ve.shape) * self.E[:, None, None]
        return _add_corners(fe, nx, ny, nz) * self.free

    def load(self, j0, j1):
        nx, ny, nz = self.g
        f = torch.zeros(nz + 1, ny + 1, nx + 1, 3, dtype=torch.float64, device=_D())
        f[0, j0:j1 + 1, nx, 2] = -1.0 / (j1 - j0 + 1)
        return f

    def solve(self, f):
        return _pcg(self.apply, self.diag, f * self.free)

    def energy(self, a, b):
        """a_e^T K b_e of every element at unit modulus."""
        A, B = _corners(a, *self.g), _corners(b, *self.g)
        return ((A.reshape(-1, 24) @ self.K) * B.reshape(-1, 24)).sum(1).reshape(A.shape[:-2])

    def evaluate(self, f):
        u = self.solve(f)
        dims = tuple(range(1, u.dim()))
        return u, (f * u).sum(dim=dims), -self.dE * self.energy(u, u)


def _exact_eval(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if nx * ny * nz > 600000:
        return None
    s = _Simp(nx, ny, nz, _densities(case, seed))
    u, c, dc = s.evaluate(s.load(0, ny)[None])
    out = {"compliance": float(c[0]), "dc": dc[0]}
    if case["u"]:
        out["u"] = u.reshape(-1)
    return out


def _exact_batch(case, seed):
    if case["nx"] * case["ny"] * case["nz"] > 600000:
        return None
    out, budget = [], 150000  # element budget: the larger designs are left out
    for d in _batch_designs(case, seed):
        ne = d["nx"] * d["ny"] * d["nz"]
        if ne > budget or ne > 30000:
            out.append({"compliance": None, "dc": None})
            continue
        budget -= ne
        s = _Simp(d["nx"], d["ny"], d["nz"], d["rho"])
        _, c, dc = s.evaluate(torch.stack([s.load(*sp) for sp in d["spans"]]))
        out.append({"compliance": c, "dc": dc})
    return out


def _exact_plain(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    s = _Simp(nx, ny, nz, _densities(case, seed))
    u, c, dc = s.evaluate(s.load(0, ny)[None])
    out = {"u": u.reshape(-1), "compliance": float(c[0]), "dc": dc[0]}
    if case["ks"]:
        # KS value of the von Mises stress at the Gauss points and its total derivative
        lam, mu = _lame()
        G = _t(_hex_gradients())
        ue = _corners(u[0], nx, ny, nz).requires_grad_(True)
        Es = s.E.clone().requires_grad_(True)
        H = torch.einsum("eai,qaj->eqij", ue, G)
        eps = 0.5 * (H + H.transpose(-1, -2))
        tr = torch.diagonal(eps, dim1=-2, dim2=-1).sum(-1)
        sig = Es[:, None, None, None] * (lam * tr[..., None, None] * torch.eye(3, dtype=torch.float64, device=_D())
                                         + 2 * mu * eps)
        sx, sy, sz = sig[..., 0, 0], sig[..., 1, 1], sig[..., 2, 2]
        vm = torch.sqrt(0.5 * ((sx - sy) ** 2 + (sy - sz) ** 2 + (sz - sx) ** 2)
                        + 3 * (sig[..., 0, 1] ** 2 + sig[..., 1, 2] ** 2 + sig[..., 2, 0] ** 2))
        ks = torch.log(torch.exp(KS_P * (vm - KS_SIGMA0) / KS_SIGMA0).mean()) / KS_P
        gu, gE = torch.autograd.grad(ks, (ue, Es))
        rhs = -_add_corners(gu, nx, ny, nz)
        adj = s.solve(rhs[None])
        out["ks"], out["max_vm"] = float(ks.detach()), float(vm.detach().max())
        out["dks"] = gE * s.dE + s.dE * s.energy(adj[0], u[0])
    return out


def _exact_tangent(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = _rng(seed)
    rho = rng.uniform(0.3, 1.0, nx * ny * nz)
    n = 3 * (nx + 1) * (ny + 1) * (nz + 1)
    shape = (nz + 1, ny + 1, nx + 1, 3)
    X = _t(rng.normal(scale=1e-3, size=n)).reshape(shape)
    v = _t(rng.normal(size=n)).reshape(shape)
    s = _Simp(nx, ny, nz, rho)
    lam, mu = _lame()
    G = _t(_hex_gradients())
    eye = torch.eye(3, dtype=torch.float64, device=_D())
    ue, ve = _corners(X, nx, ny, nz), _corners(v * s.free, nx, ny, nz)
    E = s.E[:, None, None]
    fe = torch.zeros_like(ue)
    ke = torch.zeros_like(ue)
    for q in range(8):
        H = torch.einsum("eai,aj->eij", ue, G[q])
        D = torch.einsum("eai,aj->eij", ve, G[q])
        F = eye + H
        eps = 0.5 * (H + H.transpose(1, 2) + H.transpose(1, 2) @ H)
        de = 0.5 * (F.transpose(1, 2) @ D + D.transpose(1, 2) @ F)
        tr = lambda a: torch.diagonal(a, dim1=1, dim2=2).sum(-1)[:, None, None]  # noqa: E731
        S = E * (lam * tr(eps) * eye + 2 * mu * eps)
        dS = E * (lam * tr(de) * eye + 2 * mu * de)
        fe += torch.einsum("eij,aj->eai", F @ S, G[q]) / 8.0
        ke += torch.einsum("eij,aj->eai", D @ S + F @ dS, G[q]) / 8.0
    f = 0.01 * s.load(0, ny)
    R = (_add_corners(fe, nx, ny, nz) - f) * s.free + X * (1 - s.free)
    J = _add_corners(ke, nx, ny, nz) * s.free + v * (1 - s.free)
    return {"R": R.reshape(-1), "Jv": J.reshape(-1)}


def _exact_heat(case, seed):
    nx, ny = case["nx"], case["ny"]
    hx, hy, beta, hc = 1.0 / nx, 1.0 / ny, 0.01, 10.0
    scale = _t(_rng(seed).uniform(0.5, 1.5, nx * ny))
    Q = [(0, 0), (1, 0), (1, 1), (0, 1)]
    g = 0.5 / math.sqrt(3.0)
    N, G = np.zeros((4, 4)), np.zeros((4, 4, 2))
    for q in range(4):
        x = (0.5 + (2 * (q & 1) - 1) * g, 0.5 + (2 * (q >> 1) - 1) * g)
        for a, c in enumerate(Q):
            h = [x[i] if c[i] else 1 - x[i] for i in range(2)]
            N[q, a] = h[0] * h[1]
            G[q, a] = ((1 if c[0] else -1) * h[1] / hx, (1 if c[1] else -1) * h[0] / hy)
    N, G, w = _t(N), _t(G), hx * hy / 4.0
    B = torch.einsum("qai,qbi->qab", G, G) * w

    def corners(v):
        return torch.stack([v[..., c[1]:c[1] + ny, c[0]:c[0] + nx].reshape(*v.shape[:-2], -1) for c in Q], -1)

    def scatter(fe):
        y = torch.zeros(*fe.shape[:-2], ny + 1, nx + 1, dtype=torch.float64, device=_D())
        for a, c in enumerate(Q):
            y[..., c[1]:c[1] + ny, c[0]:c[0] + nx] += fe[..., a].reshape(*fe.shape[:-2], ny, nx)
        return y

    free = torch.ones(ny + 1, nx + 1, dtype=torch.float64, device=_D())
    free[:, 0] = 0.0
    ic, jc = (np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny
    src = _t(np.where(((jc[:, None] > 0.25) & (jc[:, None] < 0.75)) & ((ic[None, :] > 0.25) & (ic[None, :] < 0.75)),
                      1.0, 0.0).reshape(-1))
    load = scatter((src * hx * hy / 4.0)[:, None].expand(-1, 4)) * free
    ones = scatter(torch.full((nx * ny, 4), hx * hy / 4.0, dtype=torch.float64, device=_D()))

    def side(v):
        y = torch.zeros_like(v)
        y[..., :-1, nx] += hc * hy * (v[..., :-1, nx] / 3 + v[..., 1:, nx] / 6)
        y[..., 1:, nx] += hc * hy * (v[..., 1:, nx] / 3 + v[..., :-1, nx] / 6)
        return y

    def conductance(T):  # (n_el, 4 points)
        return scale[:, None] * (1 + beta * corners(T) @ N.T)

    def solver(T):
        k = conductance(T)
        Ke = (k @ B.reshape(4, 16)).reshape(-1, 4, 4)
        diag = scatter(torch.diagonal(Ke, dim1=1, dim2=2))
        sd = torch.zeros_like(diag)
        sd[:-1, nx] += hc * hy / 3
        sd[1:, nx] += hc * hy / 3

        def apply(v):
            v = v * free
            return (scatter(torch.einsum("eab,neb->nea", Ke, corners(v))) + side(v)) * free

        return lambda b: _pcg(apply, diag + sd, (b * free)[None])[0]

    T = torch.zeros(ny + 1, nx + 1, dtype=torch.float64, device=_D())
    for _ in range(20):  # frozen conductance: contracts by about beta max T per pass
        new = solver(T)(load)
        done = (new - T).abs().max() <= 1e-15 * new.abs().max()
        T = new
        if bool(done):
            break
    # adjoint: (A(T) + N(T))^T lambda = -dq/dT, N the derivative of the conductance
    Te = corners(T)
    grad = torch.einsum("ea,qai->eqi", Te, G)
    flux = torch.einsum("eqi,qai->eqa", grad, G) * w * beta * scale[:, None, None]
    lam = torch.zeros_like(T)
    solve = solver(T)
    for _ in range(20):
        ext = scatter(torch.einsum("eqa,ea,qb->eb", flux, corners(lam), N))
        new = solve(-ones - ext)
        done = (new - lam).abs().max() <= 1e-15 * new.abs().max()
        lam = new
        if bool(done):
            break
    le = corners(lam)
    per = torch.einsum("eqi,qai,ea->eq", grad, G, le) * w * (1 + beta * Te @ N.T)
    ds = per.sum(1)
    return {"T": T.reshape(-1), "q": float((ones * T).sum()), "dk0": float((ds * scale).sum()), "ds": ds}


def _offsets(radius):
    a = int(math.floor(radius))
    out = []
    for c in range(-a, a + 1):
        for b in range(-a, a + 1):
            for i in range(-a, a + 1):
                d = math.sqrt(i * i + b * b + c * c)
                if radius - d > 0:
                    out.append((i, b, c, radius - d))
    return out


def _exact_filter(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n, offs = nx * ny * nz, _offsets(case["radius"])
    a = int(math.floor(case["radius"]))
    dv = torch.as_tensor(_filter_mask(case, seed).astype(bool), device=_D()).reshape(nz, ny, nx)

    def stencil(v):
        p = torch.nn.functional.pad(v, (a, a, a, a, a, a))
        y = torch.zeros_like(v)
        for i, b, c, w in offs:
            y += w * p[a + c:a + c + nz, a + b:a + b + ny, a + i:a + i + nx]
        return y

    rho = _t(_rng(seed).uniform(0.01, 1.0, n)).reshape(nz, ny, nx)
    g = _t(_rng(seed + 1).normal(size=n)).reshape(nz, ny, nx)
    S = stencil(torch.ones_like(rho))
    fwd = torch.where(dv, stencil(rho) / S, rho)
    back = stencil(torch.where(dv, g / S, torch.zeros_like(g))) + torch.where(dv, torch.zeros_like(g), g)
    return {"filtered": fwd.reshape(-1), "gradient": back.reshape(-1)}


_EXACT = dict(eval=_exact_eval, batch=_exact_batch, plain=_exact_plain, heat=_exact_heat, tangent=_exact_tangent,
              filter=_exact_filter)


def exact(case, seed):
    with torch.set_grad_enabled(case["kind"] == "plain"):
        v = _EXACT[case["kind"]](case, seed)

    def plain(x):
        if isinstance(x, dict):
            return {k: plain(y) for k, y in x.items()}
        if isinstance(x, list):
            return [plain(y) for y in x]
        return x.detach() if isinstance(x, torch.Tensor) else x

    return plain(v)

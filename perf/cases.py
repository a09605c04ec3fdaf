"""Workloads that the factor / solve path is measured on, through the public
Python API (``uhm_gb300.api``) over host buffers, as a program uses it.

Every pass of a ``step`` case is one step of a nonlinear or time-dependent
computation: new element matrices and right-hand sides are copied in from
page-locked host memory, the mesh is factored and solved, and the solution
is copied out element by element.  A ``solve`` case keeps a factorisation
and takes new right-hand sides only.  The mesh, its tree and its plan stay
from pass to pass, as such a program keeps them.

Meshes are the hp-FEM meshes of ``uhm_gb300.hpfem``: uniform quads or hexes,
Legendre-hierarchic shapes, Dirichlet boundary, nested dissection; the
diffusion coefficient is lognormal per element (clipped to ``contrast``), the
right-hand side i.i.d. N(0, 1) per degree of freedom.
"""
import functools
import math

import numpy as np
import torch

from uhm_gb300 import api, hpfem

METHODS = {"chol": api.UHM_CHOL, "lu_piv": api.UHM_LU_PIV, "lu_nopiv": api.UHM_LU_NOPIV}
# fp64: the plain drop-in (the API's default mode); the others are the mixed
# modes, refined in FP64 to a backward error of 1e-12
PRECS = {"fp64": None, "fp32": api.PREC_FP32, "bf16": api.PREC_BF16X3, "learned": api.PREC_LEARNED}
TOL = 1e-12
PECLET = 100.0


def _case(name=None, dim=3, n=8, p=4, pmax=0, method="chol", prec="fp64", rhs=1, contrast=1.0,
          call="step", meshes=0, elements="host"):
    c = dict(dim=dim, n=n, p=p, pmax=pmax, method=method, prec=prec, rhs=rhs, contrast=contrast,
             call=call, meshes=meshes, elements=elements)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small 2D problem solved over and over (a parameter study): launches and latency count
        _case("quad16_p4_fp64", dim=2, n=16, p=4),
        # an ordinary 3D problem in the default, plain FP64 mode
        _case("hex8_p4_fp64", n=8, p=4),
        # a ragged tree (11 -> 6 -> 3 -> 2 -> 1) with mixed orders, strong coefficient jumps, several load cases
        _case("hex11_p2to5_fp64_rhs3", n=11, p=2, pmax=5, rhs=3, contrast=1e4),
        # the headline mesh in the default, plain FP64 mode: the largest FP64 problem
        _case("hex16_p4_fp64", n=16, p=4),
        # nonsymmetric operators in FP64: convection-diffusion, LU with partial pivoting
        _case("convdiff12_p3_lupiv_fp64", n=12, p=3, method="lu_piv", contrast=1e4),
        # convection-diffusion at production size in the mixed mode
        _case("convdiff24_p3_lupiv_bf16", n=24, p=3, method="lu_piv", prec="bf16", contrast=1e4),
        # the headline: mixed precision chosen by the learned selector
        _case("hex16_p4_learned", n=16, p=4, prec="learned"),
        # heterogeneous diffusion with mixed orders, element matrices generated on the device
        _case("hex12_p3to5_learned_gen", n=12, p=3, pmax=5, prec="learned", contrast=1e1, elements="device"),
        # single-precision fronts with refinement, ragged tree
        _case("hex13_p4_fp32_rhs2", n=13, p=4, prec="fp32", rhs=2, contrast=1e1),
        # many independent meshes as one forest, 16 right-hand sides each
        _case("forest12_n6to12_fp32_rhs16", n=6, p=2, pmax=4, prec="fp32", rhs=16, meshes=12),
        # time stepping with a constant operator: new right-hand sides on a kept FP64 factorisation
        _case("hex12_p4_fp64_solve_rhs4", n=12, p=4, rhs=4, call="solve"),
        # nonsymmetric operators without pivoting, small
        _case("convdiff6_p3_lunopiv_fp64", n=6, p=3, method="lu_nopiv"),
    ]


def draw(rng):
    kind = rng.choice(["quad", "chol64", "chol64", "lu64", "lumix", "cholmix", "cholmix", "forest", "solve"])
    rhs = rng.choice([1, 1, 1, 2, 3, 5])
    contrast = rng.choice([1.0, 3.0, 1e1])

    def sizes(lo, hi, p_lo, p_hi, np_max):
        # cells per side over their logarithm, with n * p (degrees of freedom
        # per side) bounded; an f-way merge has f - 1 separators per axis
        while True:
            n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
            p = rng.randint(p_lo, p_hi)
            factors = [f for f in range(2, n + 1) if n % f == 0 and all(f % d for d in range(2, f))]
            widest = 2 if max(factors) > 5 else max(factors)
            if n * p * math.sqrt(widest - 1) <= np_max:
                return n, p

    if kind == "quad":
        n, p = sizes(6, 40, 2, 6, 160)
        return _case(dim=2, n=n, p=p, rhs=rhs, contrast=contrast, prec=rng.choice(["fp64", "fp32"]))
    if kind == "chol64":
        n, p = sizes(3, 18, 2, 5, 56)
        return _case(n=n, p=p, rhs=rhs, contrast=contrast, pmax=rng.choice([0, 0, min(5, p + 1)]))
    if kind == "lu64":
        n, p = sizes(3, 13, 2, 4, 44)
        return _case(n=n, p=p, method="lu_piv", rhs=rhs, contrast=contrast)
    if kind == "lumix":
        n, p = sizes(6, 20, 2, 4, 54)
        return _case(n=n, p=p, method="lu_piv", prec=rng.choice(["fp32", "bf16"]), contrast=contrast)
    if kind == "cholmix":
        n, p = sizes(5, 18, 2, 6, 60)
        return _case(n=n, p=p, prec=rng.choice(["fp32", "bf16", "learned"]), rhs=rhs, contrast=contrast,
                     elements=rng.choice(["host", "device"]))
    if kind == "forest":
        return _case(n=rng.randint(4, 8), p=2, pmax=rng.randint(3, 4), prec="fp32", rhs=rng.choice([1, 4, 7, 16]),
                     meshes=rng.randint(3, 14))
    n, p = sizes(5, 14, 2, 5, 48)
    return _case(n=n, p=p, rhs=rng.choice([1, 3, 8, 16]), call="solve", prec=rng.choice(["fp64", "bf16"]))


# ----------------------------------------------------------------------------
# meshes: topology, tree and unit-coefficient element matrices, per shape
# ----------------------------------------------------------------------------
def _orders(n, dim, p, pmax):
    """p, or per-element orders uniform in p..pmax (a fixed draw per shape)."""
    if not pmax or pmax <= p:
        return p
    return np.random.default_rng(1000 * n + pmax).integers(p, pmax + 1, n ** dim)


class _Shape:
    """What stays the same from seed to seed."""

    def __init__(self, dim, n, p, pmax, convection, rhs, meshes):
        orders = _orders(n, dim, p, pmax)
        if meshes:
            # sizes n .. 2 n and orders p .. pmax, uniform, a fixed draw
            r = np.random.default_rng(77 + meshes)
            parts = [hpfem.build_mesh(3, int(r.integers(n, 2 * n + 1)), int(r.integers(p, pmax + 1)), n_rhs=rhs)
                     for _ in range(meshes)]
            self.spec = hpfem.forest(parts)
        else:
            merges = [3, 2, 2, 2] if (dim, n) == (3, 24) else None
            self.spec = hpfem.build_mesh(dim, n, orders, n_rhs=rhs, merges=merges)
        s = self.spec
        self.diffusion = s.mats.copy()
        self.convection = None
        if convection:
            beta = PECLET * np.array([1.0, 0.5, 0.25])[:dim]
            full = hpfem.build_mesh(dim, n, orders, n_rhs=rhs, merges=merges, beta=beta)
            self.convection = full.mats - self.diffusion
            s.symmetric = False
        # per element row: its degree of freedom, and its place in element-ordered vectors
        dof0 = np.concatenate([[0], np.cumsum(s.node_ndof)])
        nodes = s.elem_node if not meshes else np.searchsorted(s.node_id, s.elem_node)
        cnt = s.node_ndof[nodes]
        start = np.repeat(dof0[nodes], cnt)
        run0 = np.repeat(np.cumsum(cnt) - cnt, cnt)
        self.gdof = start + (np.arange(cnt.sum()) - run0)
        m = s.elem_m.astype(np.int64)
        row0 = np.cumsum(m) - m
        self.m_of_row = np.repeat(m, m)
        local = np.arange(m.sum()) - np.repeat(row0, m)
        self.pos = np.repeat(s.rhs_off.astype(np.int64), m) + local
        self.local = local
        self.elem_of_row = np.repeat(np.arange(len(m)), m)
        first = np.zeros(len(self.gdof), bool)
        first[np.unique(self.gdof, return_index=True)[1]] = True
        self.first = first

    def mats(self, kappa):
        a = self.diffusion * np.repeat(kappa, self.spec.elem_m.astype(np.int64) ** 2)
        return a if self.convection is None else a + self.convection

    def spread(self, v):
        """(n_dof, n_rhs) values to element order (every copy of a shared one)."""
        out = np.zeros(self.spec.rhs.size)
        for q in range(v.shape[1]):
            out[self.pos + q * self.m_of_row] = v[self.gdof, q]
        return out

    def loads(self, b):
        """(n_dof, n_rhs) right-hand sides as element vectors that add up to them."""
        out = np.zeros(self.spec.rhs.size)
        for q in range(b.shape[1]):
            out[self.pos + q * self.m_of_row] = np.where(self.first, b[self.gdof, q], 0.0)
        return out


@functools.lru_cache(maxsize=2)
def _shape(dim, n, p, pmax, convection, rhs, meshes):
    return _Shape(dim, n, p, pmax, convection, rhs, meshes)


def _shape_of(case):
    return _shape(case["dim"], case["n"], case["p"], case["pmax"], case["method"] != "chol", case["rhs"],
                  case["meshes"])


def _values(case, seed):
    """Coefficients per element and right-hand sides per degree of freedom."""
    sh = _shape_of(case)
    rng = np.random.default_rng(seed)
    half = 0.5 * math.log(case["contrast"])
    kappa = np.exp(np.clip(2.0 * rng.standard_normal(sh.spec.n_leaves), -half, half))
    b = rng.standard_normal((sh.spec.n_dof(), case["rhs"]))
    return sh, kappa, b


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    v = t.numpy()
    v[:] = a
    return t, v


def prepare(case, seed):
    sh, kappa, b = _values(case, seed)
    spec = sh.spec
    method = METHODS[case["method"]]
    rhs = _pinned(sh.loads(b))
    s = dict(case=case, method=method, rhs=rhs, out=_pinned(np.zeros(spec.rhs.size)), n_out=spec.rhs.size)
    spec.rhs = rhs[1]
    if case["elements"] == "device":
        recipe = hpfem.element_recipe(spec)
        recipe["kappa"] = np.ascontiguousarray(kappa)
        s["recipe"] = recipe
        m = api.load_spec(spec, lhs=False)
    else:
        s["lhs"] = _pinned(sh.mats(kappa))
        spec.mats = s["lhs"][1]
        m = api.load_spec(spec)
    spec.mats = sh.diffusion
    if PRECS[case["prec"]] is not None:
        if case["prec"] == "learned":
            from uhm_gb300 import selector
            m.set_selector(selector.load_weights())
        m.set_mode(1, PRECS[case["prec"]], TOL, 10)
    if case["call"] == "solve":
        m.factor(method)
    s["mesh"] = m
    return s


def run(s):
    m = s["mesh"]
    if s["case"]["call"] == "step":
        if "recipe" in s:
            m.generate_elements(s["recipe"], s["method"])
        else:
            m.copy_in_leaves(api.UHM_LHS, s["lhs"][1])
    m.copy_in_leaves(api.UHM_RHS, s["rhs"][1])
    if s["case"]["call"] == "step":
        m.factor(s["method"])
    m.solve(s["method"])
    return m.copy_out_leaves(s["n_out"], out=s["out"][1])


def work(case):
    """Element matrices and right-hand sides read once, the solution written
    once; the LAWN-41 operation counts of the factorisation and the solve.  A
    solve on a kept factorisation reads the factor once instead of the matrices."""
    sh = _shape_of(case)
    spec = sh.spec
    m = api.load_spec(spec, lhs=False)
    factor, solve = m.estimate_cost(METHODS[case["method"]], case["rhs"])
    _, _, fs, ss = (v.astype(np.float64) for v in m.fronts())
    chol = case["method"] == "chol"
    entries = float((fs * (fs + 1) / 2 + fs * ss).sum()) if chol else float((fs * fs + 2 * fs * ss).sum())
    vectors = 16.0 * spec.rhs.size
    if case["call"] == "solve":
        return {"bytes": vectors + entries * (8 if case["prec"] == "fp64" else 4), "flops": solve}
    given = 8.0 * spec.n_leaves if case["elements"] == "device" else 8.0 * spec.mats.size
    return {"bytes": given + vectors, "flops": factor + solve}


# ----------------------------------------------------------------------------
# 64-bit solutions without the solver: conjugate gradients (symmetric), dense
# single-precision LU refined in 64 bits (nonsymmetric, moderate sizes)
# ----------------------------------------------------------------------------
def exact(case, seed):
    sh, kappa, b = _values(case, seed)
    spec = sh.spec
    n = spec.n_dof()
    if case["method"] != "chol" and n > 45_000:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = spec.elem_m.astype(np.int64)
    width = int(m.max())
    mats = sh.mats(kappa)
    # element matrices padded to one width; padding rows belong to the extra entry n
    A = torch.zeros(len(m), width, width, dtype=torch.float64)
    idx = torch.full((len(m), width), n, dtype=torch.int64)
    for size in np.unique(m):
        which = np.flatnonzero(m == size)
        at = spec.mat_off[which][:, None] + np.arange(size * size)
        A[which, :size, :size] = torch.from_numpy(mats[at].reshape(len(which), size, size)).transpose(1, 2)
    idx[torch.from_numpy(sh.elem_of_row), torch.from_numpy(sh.local)] = torch.from_numpy(sh.gdof)
    A, idx = A.to(dev), idx.to(dev)
    flat = idx.reshape(-1)
    rhs = torch.from_numpy(b).to(dev)

    def matvec(x):
        xp = torch.cat([x, x.new_zeros(1, x.shape[1])])
        y = torch.zeros_like(xp)
        y.index_add_(0, flat, torch.bmm(A, xp[idx]).reshape(-1, x.shape[1]))
        return y[:n]

    diag = torch.zeros(n + 1, dtype=torch.float64, device=dev)
    diag.index_add_(0, flat, torch.diagonal(A, dim1=1, dim2=2).reshape(-1))
    scale = diag[:n].abs().sqrt().reciprocal()[:, None]
    x = torch.zeros_like(rhs)
    if case["method"] == "chol":
        for _ in range(4):                                  # restarts from the true residual
            r = rhs - matvec(x)
            z = r * scale * scale
            p, rz, d = z.clone(), (r * z).sum(0), torch.zeros_like(x)
            goal = rz * 1e-26
            for it in range(6000):
                q = matvec(p)
                a = torch.where(rz > 0, rz / (p * q).sum(0).clamp_min(1e-300), torch.zeros_like(rz))
                d += a * p
                r -= a * q
                z = r * scale * scale
                new = (r * z).sum(0)
                if it % 50 == 49 and bool((new <= goal).all()):
                    break
                p = z + torch.where(rz > 0, new / rz.clamp_min(1e-300), torch.zeros_like(rz)) * p
                rz = new
            x += d
    else:
        full = torch.zeros(n + 1, n + 1, dtype=torch.float32, device=dev)
        scaled = torch.cat([scale, scale.new_zeros(1, 1)])[:, 0]
        part = (A * scaled[idx][:, :, None] * scaled[idx][:, None, :]).float()
        for e in range(len(m)):
            full[idx[e][:, None], idx[e][None, :]] += part[e]
        lu, piv = torch.linalg.lu_factor(full[:n, :n])
        del full
        for _ in range(25):
            r = (rhs - matvec(x)) * scale
            big = r.abs().amax(0).clamp_min(1e-300)
            d = torch.linalg.lu_solve(lu, piv, (r / big).float()).double() * big * scale
            x += d
            if float((d.norm() / x.norm())) < 1e-15:
                break
    return sh.spread(x.cpu().numpy())

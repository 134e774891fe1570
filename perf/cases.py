"""What a program built on this package has the GPU do, as cases that can be timed and compared.

Every case is one call sequence of the flow solver's time step through the public entry points:

* ``pass``      one assembly pass of the quench fields (NS+VOF and temperature, matrix and vector), the right-hand
                sides read back into page-locked memory, and one product with each assembled matrix (the start of a
                residual check or of an outer Krylov step) on device vectors;
* ``residual``  the vector-only pass of the Newton loop (the convergence test of an iteration);
* ``cavity``    one Newton iteration of the lid-driven cavity: assembleNavSto, then SparseGMRES_up;
* ``gmres``     one cycle of SparseGMRES_ns_conv / SparseGMRES_tem on an assembled system;
* ``mixed``     the refined mixed-precision solve of the coupled system to a true residual;
* ``newton``    the Newton loop of one whole quench time step on the device;
* ``vjp``       the adjoint of the residual (NS+VOF and temperature) for one cotangent.

The meshes are boxes of tetrahedra (six per cell) or trilinear hexahedra with displaced inner nodes; ``numbering``
"random" renumbers nodes and elements the way a mesh generator's file may have them.  ``solid`` puts a solid block in
the middle (its nodes held by Dirichlet flags), ``phase`` switches phase change and discontinuity capturing on.
"""
from __future__ import annotations

import functools
import math
import time

import numpy as np
import torch

from oversetdevfort_b200 import _ffi as F
from oversetdevfort_b200 import api
from oversetdevfort_b200 import distributed as D
from oversetdevfort_b200 import mesh as M

BOTH = api.ASSEMBLE_TENSOR_MAT | api.ASSEMBLE_TENSOR_VEC
ALL_FIELDS = api.ASSEMBLE_FIELD_NS | api.ASSEMBLE_FIELD_VOF | api.ASSEMBLE_FIELD_TEM
TOL_GMRES, TOL_MIXED = 1e-6, 1e-10


def _case(kind, nx, ny, nz, **kw):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, hex=False, fp32=False, numbering="grid", solid=False, phase=False,
             kspace=50, system="nsvof")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest problem users start from: the 16^3 cavity, all launches and latency
        _case("cavity", 16, 16, 16, name="cavity_16_fp64"),
        # the ordinary assembly pass: the 48x48x96 quench box
        _case("pass", 48, 48, 96, phase=True, name="pass_48x48x96_fp64"),
        # the largest: the 128^3 quench cube
        _case("pass", 128, 128, 128, name="pass_128_fp64"),
        # single precision, odd sizes, a solid block, numbered as a mesh file may be
        _case("pass", 95, 81, 113, fp32=True, numbering="random", solid=True, phase=True, name="pass_95x81x113_fp32"),
        # the residual evaluation of every Newton iteration
        _case("residual", 48, 48, 96, phase=True, name="residual_48x48x96_fp64"),
        # trilinear hexahedra: the 96^3 box in double, an odd one in single precision
        _case("pass", 96, 96, 96, hex=True, name="hex_pass_96_fp64"),
        _case("pass", 53, 61, 47, hex=True, fp32=True, phase=True, name="hex_pass_53x61x47_fp32"),
        # one FP64 GMRES cycle of the coupled system, ordinary and largest
        _case("gmres", 48, 48, 96, phase=True, name="gmres_48x48x96_fp64"),
        _case("gmres", 128, 128, 128, name="gmres_128_fp64"),
        # the mixed-precision solve
        _case("mixed", 48, 48, 96, name="mixed_solve_48x48x96"),
        # a whole time step of a small problem: assembly, both solves, updates, residual tests
        _case("newton", 24, 24, 48, phase=True, name="newton_step_24x24x48"),
        # the adjoint on the 32^3 cube
        _case("vjp", 32, 32, 32, phase=True, name="vjp_32_fp64"),
    ]


def draw(rng):
    kind = rng.choice(["pass", "pass", "pass", "residual", "cavity", "gmres", "gmres", "mixed", "newton", "vjp"])
    hexa = kind == "pass" and rng.random() < 0.35
    lo, hi = {"pass": (6, 126), "residual": (8, 126), "cavity": (5, 64), "gmres": (8, 110), "mixed": (14, 44),
              "newton": (6, 40), "vjp": (5, 56)}[kind]
    if hexa:
        lo, hi = 5, 94
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = math.exp(rng.uniform(-0.35, 0.35)), math.exp(rng.uniform(-0.35, 0.35))
    dims = [max(4, min(hi + 20, round(n * s))) for s in (a, b, 1.0 / (a * b))]
    while dims[0] * dims[1] * dims[2] > hi ** 3:
        dims[dims.index(max(dims))] -= 1
    c = _case(kind, *dims, hex=hexa, fp32=kind in ("pass", "residual") and rng.random() < 0.4)
    c["numbering"] = rng.choice(["grid", "grid", "random"])
    # the refined solve is used without phase change (the reference's quench settings): with it the reference's
    # matrix is too far from its rounding for the refinement to reach the tolerance on a coarse mesh
    c["phase"] = kind not in ("cavity", "mixed") and rng.random() < 0.5
    c["solid"] = kind in ("pass", "residual") and rng.random() < 0.3
    if kind == "gmres":
        c["system"] = rng.choice(["nsvof", "tem"])
        c["kspace"] = rng.randint(12, 70)
    return c


# --------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=2)
def _mesh(nx, ny, nz, hexa, numbering, solid):
    """The box (unit cells up to a common factor), inner nodes moved by up to 15% of the cell, and which nodes and
    elements are solid."""
    h = 1.0 / max(nx, ny)
    lx, ly, lz = nx * h, ny * h, nz * h
    m = (M.box_hex if hexa else M.box_tet)(nx, ny, nz, lx, ly, lz)
    rng = np.random.default_rng(1000003 * nx + 1009 * ny + nz)
    wall = np.zeros(m.nnode, dtype=bool)
    for f in m.faces:
        wall[f] = True
    m.xg[~wall] += 0.15 * h * rng.uniform(-1.0, 1.0, (int((~wall).sum()), 3))
    if numbering == "random":
        new = rng.permutation(m.nnode)
        x = np.empty_like(m.xg)
        x[new] = m.xg
        ien = (new[m.ien.astype(np.int64) - 1] + 1).astype(np.int32)[rng.permutation(m.nelem)]
        m = M.Mesh(np.asfortranarray(x), np.asfortranarray(ien), m.elm_id, [np.sort(new[f]) for f in m.faces], m.dims,
                   m.lengths)
    held = np.zeros(m.nnode, dtype=bool)
    if solid:
        centre = m.xg[m.ien.astype(np.int64) - 1].mean(axis=1)
        inside = np.all(np.abs(centre - 0.5 * np.array(m.lengths)) < 0.15 * np.array(m.lengths), axis=1)
        m.elm_id[inside] = 101
        held[(m.ien[inside].astype(np.int64) - 1).ravel()] = True
    return m, held


def _params(case):
    if case["kind"] == "cavity":
        return M.base_params(delt=0.01, rhoa=1.0, mua=0.01, rhow=1.0, muw=0.01)
    if case["phase"]:
        return M.base_params(c_evap=0.3, c_cond=0.2, c_dmdot=0.7, lsc_kdc=0.05, tem_kdc=0.02, tref=400.0)
    return M.base_params()


def _waves(m, rng, modes=4):
    """A smooth random field of size one."""
    x = m.xg / np.array(m.lengths)
    s = np.zeros(m.nnode)
    for _ in range(modes):
        k = rng.integers(1, 4, 3) * np.pi
        s += rng.uniform(-1, 1) * np.sin(k[0] * x[:, 0] + rng.uniform(0, 6)) * np.sin(
            k[1] * x[:, 1] + rng.uniform(0, 6)) * np.sin(k[2] * x[:, 2] + rng.uniform(0, 6))
    return s


def _inputs(case, seed):
    """The mesh, parameters, state and Dirichlet flags of a time step: a perturbed interface, a hot block, a weak
    flow; for the cavity the moving lid."""
    m, held = _mesh(case["nx"], case["ny"], case["nz"], case["hex"], case["numbering"], case["solid"])
    p = _params(case)
    rng = np.random.default_rng(seed)
    N = m.nnode
    st = M.empty_state(N)
    ibc = np.zeros((N, 8), dtype=np.int32, order="F")
    wall = held.copy()
    for f in m.faces:
        wall[f] = True
    for d in range(3):
        st["ugold"][:, d] = 0.02 * _waves(m, rng) + rng.uniform(-1e-3, 1e-3, N)
    st["ugold"][wall] = 0.0
    st["ug"][:] = st["ugold"]
    st["acgold"][:] = rng.uniform(-0.01, 0.01, (N, 3)) * ~wall[:, None]
    st["acg"][:] = (p["gami"] - 1.0) / p["gami"] * st["acgold"]
    ibc[wall, 0:3] = 1
    if case["kind"] == "cavity":
        lid = m.faces[5]
        st["ug"][lid, 0] = 1.0
        st["acg"][lid, 0] = (1.0 / p["delt"] + (p["gami"] - 1.0) * st["acgold"][lid, 0]) / p["gami"]
        return m, p, st, ibc
    ibc[held, 0:5] = 1
    ibc[m.faces[5], 3] = 1
    ibc[m.faces[4], 5] = 1
    lz = m.lengths[2]
    z = m.xg[:, 2]
    st["phig"][:] = np.tanh((z - 0.5 * lz + 0.03 * lz * _waves(m, rng)) / (0.02 * lz + 0.5 / case["nz"]))
    st["phigold"][:] = st["phig"]
    st["rphig"][:] = 5.0 * _waves(m, rng)
    st["rphigold"][:] = st["rphig"]
    r = np.max(np.abs(m.xg / np.array(m.lengths) - 0.5), axis=1)
    st["tg"][:] = 300.0 + 350.0 * (1.0 - np.tanh((r - 0.2) / 0.05)) + 5.0 * _waves(m, rng)
    st["tgold"][:] = st["tg"]
    st["rtg"][:] = 10.0 * _waves(m, rng)
    st["rtgold"][:] = st["rtg"]
    st["pg"][:] = 10.0 * _waves(m, rng)
    st["pg"][m.faces[5]] = 0.0
    return m, p, st, ibc


def _vectors(case, seed, N):
    """The vectors that the products and the adjoint take (nf, N), FP64, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda nf: torch.rand((nf, N), generator=g, device="cuda", dtype=torch.float64) - 0.5
    return mk(5), mk(1)


class _State:
    pass


def prepare(case, seed):
    m, p, st, ibc = _inputs(case, seed)
    kind = case["kind"]
    s = _State()
    s.case = case
    kernel = F.OVS_ASM_NS if kind == "cavity" else F.OVS_ASM_NSVOF
    s.ctx = ctx = api.Context.from_case(M.Case(kind, m, p, st, ibc, kernel))
    N = m.nnode
    s.prec = F.OVS_FP32 if case["fp32"] else F.OVS_FP64
    if kind in ("pass", "residual"):
        api.assembleQuenching(ctx, BOTH, ALL_FIELDS, s.prec)
        # where the right-hand sides land: page-locked, column-major (N, nf)
        s.rhs = [torch.empty((nf, N), dtype=torch.float64, pin_memory=True) for nf in (5, 1)]
    if kind == "pass":
        s.ops = [D.DeviceOperator(ctx, sy, s.prec) for sy in (F.OVS_SYS_NSVOF, F.OVS_SYS_TEM)]
        s.x = _vectors(case, seed, N)
        s.y = [torch.empty_like(x) for x in s.x]
    elif kind == "gmres":
        s.sys = F.OVS_SYS_TEM if case["system"] == "tem" else F.OVS_SYS_NSVOF
        ctx.assemble(F.OVS_ASM_TEM if case["system"] == "tem" else F.OVS_ASM_NSVOF, BOTH, F.OVS_FP64)
        nf = api.NF[s.sys]
        s.zero = [np.zeros((N, 3), order="F"), np.zeros(N), np.zeros(N)] if nf == 5 else [np.zeros(N)]
    elif kind == "mixed":
        ctx.assemble(F.OVS_ASM_NSVOF, BOTH, F.OVS_FP64)
    elif kind == "cavity":
        s.zero = [np.zeros((N, 3), order="F"), np.zeros(N)]
    elif kind == "newton":
        s.begin = {f: st[f] for f in ("ug", "acg", "pg", "phig", "rphig", "tg", "rtg")}
    elif kind == "vjp":
        s.cot = [x.cpu().numpy().T for x in _vectors(case, seed, N)]
    return s


def run(s):
    ctx, kind, case = s.ctx, s.case["kind"], s.case
    if kind in ("pass", "residual"):
        cfl = api.assembleQuenching(ctx, BOTH if kind == "pass" else api.ASSEMBLE_TENSOR_VEC, ALL_FIELDS, s.prec)
        for sy, r in zip((F.OVS_SYS_NSVOF, F.OVS_SYS_TEM), s.rhs):
            ctx.get_rhs_async(sy, s.prec, r.numpy().T)
        out = {"cfl": cfl}
        if kind == "pass":
            for op, x, y in zip(s.ops, s.x, s.y):
                op.apply(x, y)
            out["products"] = list(s.y)
        else:
            out["norms"] = api.calculate_residual(ctx, s.prec)
        ctx.sync_copies()
        out["rhs"] = list(s.rhs)
        if case["fp32"]:   # a single-precision pass: its results are kept in single precision
            for k in ("rhs", "products", "norms"):
                if k in out:
                    out[k] = out[k].astype(np.float32) if k == "norms" else [v.float() for v in out[k]]
        return out
    if kind == "cavity":
        cfl = api.assembleNavSto(ctx, BOTH)
        u, q, info = api.SparseGMRES_up(ctx, TOL_GMRES, case["kspace"], 1, *s.zero)
        return {"cfl": cfl, "rhs": ctx.get_rhs(F.OVS_SYS_NS), "u": u, "p": q}
    if kind == "gmres":
        fn = api.SparseGMRES_ns_conv if len(s.zero) == 3 else api.SparseGMRES_tem
        return list(fn(ctx, TOL_GMRES, case["kspace"], 1, *s.zero)[:-1])
    if kind == "mixed":
        sol, info = ctx.solve(F.OVS_SYS_NSVOF, F.OVS_MIXED, TOL_MIXED, kspace=case["kspace"], max_cycles=400)
        # the solve promises a residual: its solution is that of the system to about single precision
        return {"sol": [sol[:, k].astype(np.float32) for k in range(5)], "converged": bool(info.converged)}
    if kind == "newton":
        for f, v in s.begin.items():
            ctx.set_field(f, v)
        ctx.quench_newton(F.OVS_FP64, newton_max=2, kspace=case["kspace"], tol_ns=TOL_GMRES, tol_tem=TOL_GMRES,
                          utol=(1e-30,) * 4, atol=(1e-30,) * 4)
        return {f: ctx.get_field(f) for f in s.begin}
    return [ctx.residual_vjp(k, c) for k, c in zip((F.OVS_ASM_NSVOF, F.OVS_ASM_TEM), s.cot)]


# ----------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass: mesh, state, matrix, vectors once each; a Krylov iteration reads the matrix
    once and every basis vector twice (its dot products come before the update that needs them)."""
    n = (case["nx"], case["ny"], case["nz"])
    N = math.prod(k + 1 for k in n)
    cells = math.prod(n)
    E, nshl = (cells, 8) if case["hex"] else (6 * cells, 4)
    nnz = M.expected_nnz_hex(*n) if case["hex"] else M.expected_nnz_kuhn(*n)
    kind, ts = case["kind"], 4 if case["fp32"] else 8
    nodal = 4 * nshl * E + 4 * E + N * (35 * 8 + 1)
    point = 8 if case["hex"] else 4
    # per Gauss point about 400 operations and 30 a node; a pair's block about 90 (a hexahedron's at every point)
    vec = E * point * (400 + 30 * nshl)
    mat = E * nshl * nshl * (90 * (8 if case["hex"] else 1) + 14 * point)
    if kind == "residual":
        return {"bytes": nodal + 6 * N * 8, "flops": vec}
    if kind == "pass":
        by = nodal + 6 * N * 8 + 25 * nnz * ts * 2 + 4 * nnz + 12 * N * 8
        return {"bytes": by, "flops": vec + mat + 50 * nnz}
    if kind == "vjp":
        return {"bytes": nodal + 6 * N * 8 + 2 * 14 * N * 8, "flops": 4 * vec}
    nf, nv = {"cavity": (4, 16), "gmres": (1, 1) if case["system"] == "tem" else (5, 24)}.get(kind, (5, 24))

    def cycle(its, nf, nv, ts):
        by = sum(nv * nnz * ts + 4 * nnz + 2 * nf * N * ts + 2 * k * nf * N * ts for k in range(1, its + 1))
        return by, its * 2 * nv * nnz + 2 * its * its * nf * N

    if kind == "cavity":
        by, fl = cycle(30, nf, nv, 8)
        return {"bytes": by + nodal + nv * nnz * 8, "flops": fl + vec + mat}
    if kind == "gmres":
        by, fl = cycle(case["kspace"] if nf == 5 else 10, nf, nv, 8)
        return {"bytes": by, "flops": fl}
    if kind == "mixed":
        by, fl = cycle(case["kspace"], nf, nv, 4)
        return {"bytes": 8 * by + 12 * nv * nnz, "flops": 8 * fl}
    by, fl = cycle(case["kspace"], nf, nv, 8)
    bt, ft = cycle(10, 1, 1, 8)
    return {"bytes": 2 * (by + bt + 2 * nodal + 25 * nnz * 8), "flops": 2 * (fl + ft + 2 * vec + mat)}


# ---------------------------------------------------------------- exact
# The same quantities in plain torch, 64 bits: element integrals by quadrature, summed over the nodes.  Component
# order of a node's five unknowns: u1 u2 u3 p phi.

_HEX_SIGN = [(-1, 1, -1), (1, 1, -1), (1, 1, 1), (-1, 1, 1), (-1, -1, -1), (1, -1, -1), (1, -1, 1), (-1, -1, 1)]
CHUNK = 1 << 17


def _rule(hexa):
    """(weight, N (nshl), dN (nshl, 3)) of every quadrature point."""
    out = []
    if hexa:
        q = 0.57735026918963
        for g in range(8):
            xi = [q if g >> d & 1 else -q for d in range(3)]
            f = [[1.0 + s[d] * xi[d] for d in range(3)] for s in _HEX_SIGN]
            out.append((1.0, [v[0] * v[1] * v[2] / 8 for v in f],
                        [[s[0] * v[1] * v[2] / 8, s[1] * v[0] * v[2] / 8, s[2] * v[0] * v[1] / 8]
                         for s, v in zip(_HEX_SIGN, f)]))
    else:
        a, b = 0.5854101966249685, 0.1381966011250105
        for g in range(4):
            n = [a if g == d else b for d in range(3)]
            out.append((0.25 / 6.0, n + [1.0 - sum(n)], [[1.0, 0, 0], [0, 1.0, 0], [0, 0, 1.0], [-1.0, -1.0, -1.0]]))
    return out


class _Exact:
    def __init__(self, case, seed, device=None):
        m, p, st, ibc = _inputs(case, seed)
        self.dev = dev = device or ("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        self.p, self.N, self.E, self.hex = p, m.nnode, m.nelem, case["hex"]
        self.ien = torch.as_tensor(np.ascontiguousarray(m.ien), device=dev).long() - 1
        self.fluid = torch.as_tensor(m.elm_id == p["fluid_elm_id"], device=dev)
        self.free = torch.as_tensor(np.ascontiguousarray(ibc[:, :6]) == 0, device=dev)
        self.st = {k: t(v) for k, v in st.items()}
        self.st["xg"] = t(m.xg)
        self.rule = _rule(case["hex"])

    # generalized-alpha values of the fields
    def alpha(self):
        s, af, am = self.st, self.p["alfi"], self.p["almi"]
        mid = lambda k, o, w: s[o] + w * (s[k] - s[o])
        return {"x": s["xg"] + mid("dg", "dgold", af), "u": mid("ug", "ugold", af), "um": mid("ugm", "ugmold", af),
                "ac": mid("acg", "acgold", am), "p": s["pg"], "phi": mid("phig", "phigold", af),
                "rphi": mid("rphig", "rphigold", am), "T": mid("tg", "tgold", af), "rT": mid("rtg", "rtgold", am)}

    def points(self, f, el):
        """Geometry and interpolated fields of the elements `el` at every point."""
        nodes = self.ien[el]
        v = {k: a[nodes] for k, a in f.items()}
        for wt, N, dN in self.rule:
            N = torch.tensor(N, dtype=torch.float64, device=self.dev)
            dN = torch.tensor(dN, dtype=torch.float64, device=self.dev)
            J = torch.einsum("eai,aj->eij", v["x"] - v["x"][:, :1], dN)
            Ji = torch.linalg.inv(J)
            q = {"w": torch.linalg.det(J) * wt, "N": N, "g": torch.einsum("ak,ekj->eaj", dN, Ji),
                 "G": torch.einsum("eki,ekj->eij", Ji, Ji)}
            for k in ("u", "um", "ac"):
                q[k] = torch.einsum("eai,a->ei", v[k], N)
            for k in ("p", "phi", "rphi", "T", "rT"):
                q[k] = v[k] @ N
            q["du"] = torch.einsum("eai,eaj->eij", v["u"], q["g"])
            for k in ("p", "phi", "T"):
                q["d" + k] = torch.einsum("ea,eaj->ej", v[k], q["g"])
            q["ua"] = q["u"] - q["um"]
            q["uGu"] = torch.einsum("ei,eij,ej->e", q["ua"], q["G"], q["ua"])
            q["GG"] = (q["G"] ** 2).sum((1, 2))
            q["trG"] = torch.einsum("eii->e", q["G"])
            q["c"] = torch.einsum("eaj,ej->ea", q["g"], q["ua"])
            yield q

    def phase(self, q):
        p = self.p
        ph = q["phi"].clamp(0.0, 1.0)
        dT = (q["T"] - p["ts"]) / p["ts"]
        hot = q["T"] > p["ts"]
        ev, co = p["c_evap"] * p["rhow"], p["c_cond"] * p["rhoa"]
        mdot = torch.where(hot, ev * (1.0 - ph) * dT, co * ph * dT)
        dphi = torch.where(hot, -ev * dT, co * dT) * p["c_dmdot"]
        dphi = torch.where((q["phi"] < 0) | (q["phi"] > 1), torch.zeros_like(dphi), dphi)
        dtem = torch.where(hot, ev * (1.0 - ph), co * ph) / p["ts"] * p["c_dmdot"]
        mix = lambda w, a, s: torch.where(q["fl"], w * (1.0 - ph) + a * ph, torch.full_like(ph, s))
        return ph, mdot, dphi, dtem, mix

    def nsvof(self, q, want_matrix):
        """Point terms of the element residual (e, a, 5) and matrix (e, a, 5, b, 5)."""
        p, w, N, g, c = self.p, q["w"], q["N"], q["g"], q["c"]
        ph, mdot, dmd, _, mix = self.phase(q)
        rho, mu = mix(p["rhow"], p["rhoa"], p["rhos"]), mix(p["muw"], p["mua"], p["mus"])
        ia, iw = 1.0 / p["rhoa"], 1.0 / p["rhow"]
        vdot, lam = mdot * (ia - iw), -2.0 / 3.0 * mu
        grav = torch.tensor(p["gravvec"], dtype=torch.float64, device=self.dev)
        t1 = rho[:, None] * (q["ac"] + torch.einsum("eij,ej->ei", q["du"], q["ua"]) - grav)
        rL = t1 + q["dp"]
        divu = torch.einsum("eii->e", q["du"])
        rphi = q["rphi"] + (q["ua"] * q["dphi"]).sum(1) + q["phi"] * vdot - mdot * ia
        taut = 4.0 / p["delt"] ** 2
        nu2 = (mu / rho) ** 2 * 12.0 * q["GG"]
        tM, tL = 1.0 / (rho * torch.sqrt(taut + q["uGu"] + nu2)), 1.0 / torch.sqrt(taut + q["uGu"])
        tC = rho * torch.sqrt(q["uGu"] + nu2) / q["trG"]
        kd = p["lsc_kdc"] * rphi.abs() / torch.sqrt(q["GG"])
        di = dmd * (ia - iw)
        w = torch.where(q["fl"], w, torch.zeros_like(w))
        sv = torch.einsum("eaj,ejk->ea", g, q["du"] + q["du"].transpose(1, 2))
        col = lambda s: s[:, None]
        flux = q["p"] - tC * divu + tC * vdot - lam * divu
        ru = (-N[None, :, None] * t1[:, None, :] + g * flux[:, None, None] - (col(mu) * sv)[:, :, None]
              - (col(rho * tM) * c)[:, :, None] * rL[:, None, :])
        rp = -N * col(divu - vdot) - col(tM) * torch.einsum("eai,ei->ea", g, rL)
        rf = (-(N + col(tL) * c) * col(rphi) - col(kd) * torch.einsum("eai,ei->ea", g, q["dphi"])
              + N * col(di * tC * (divu - vdot)))
        R = torch.cat([ru, rp[:, :, None], rf[:, :, None]], 2) * w[:, None, None]
        if not want_matrix:
            return R, None
        f1, f2 = p["almi"], p["alfi"] * p["gami"] * p["delt"]
        K = torch.zeros((len(w), len(N), 5, len(N), 5), dtype=torch.float64, device=self.dev)
        gab = torch.einsum("eai,ebi->eab", g, g)
        beta = f1 * N + f2 * c
        pair = lambda a, b: a[:, :, None] * b[:, None, :]
        NN = N.expand(len(w), -1)
        k3 = lambda s: s[:, None, None]
        S = k3(w * rho) * pair(NN + col(rho * tM) * c, beta) + k3(f2 * w * mu) * gab
        gam = col(w) * (N + col(tL) * c)
        for i in range(3):
            for j in range(3):
                K[:, :, i, :, j] = k3(f2 * w * mu) * pair(g[:, :, j], g[:, :, i]) + \
                    k3(f2 * w * (tC + lam)) * pair(g[:, :, i], g[:, :, j])
            K[:, :, i, :, i] += S
            K[:, :, i, :, 3] = k3(f2 * w) * (pair(col(rho * tM) * c, g[:, :, i]) - pair(g[:, :, i], NN))
            K[:, :, 3, :, i] = k3(w) * (f2 * pair(NN, g[:, :, i]) + pair(g[:, :, i], col(rho * tM) * beta))
            K[:, :, 4, :, i] = f2 * k3(q["dphi"][:, i]) * pair(gam, NN) - k3(f2 * tC * di * w) * pair(NN, g[:, :, i])
            K[:, :, i, :, 4] = k3(f2 * tC * di * w) * pair(g[:, :, i], NN)
        K[:, :, 3, :, 3] = k3(f2 * w * tM) * gab
        K[:, :, 4, :, 4] = pair(gam, beta + f2 * N * col(vdot + q["phi"] * di - dmd * ia)) + \
            k3(f2 * w * kd) * gab + k3(f2 * w * tC * di * di) * pair(NN, NN)
        K[:, :, 3, :, 4] = -k3(f2 * di * w) * pair(NN, NN)
        return R, K

    def ns(self, q, want_matrix):
        """The constant-property flow of the cavity (rows u, p)."""
        p, w, N, g, c = self.p, q["w"], q["N"], q["g"], q["c"]
        rho, mu = p["rhoa"], p["mua"] + p["ns_kdc_a"]
        grav = torch.tensor(p["gravvec"], dtype=torch.float64, device=self.dev)
        nu2 = (p["mua"] / rho) ** 2 * 12.0 * q["GG"]
        tM = 1.0 / (rho * torch.sqrt(4.0 / p["delt"] ** 2 + q["uGu"] + nu2))
        tC = rho * torch.sqrt(q["uGu"] + nu2) / q["trG"]
        divu = torch.einsum("eii->e", q["du"])
        t1 = rho * (q["ac"] + torch.einsum("eij,ej->ei", q["du"], q["ua"]) - grav)
        sym = torch.einsum("eaj,eij->eai", g, q["du"] + q["du"].transpose(1, 2))
        ru = -(N[None, :, None] * t1[:, None, :] + mu * sym - g * (q["p"] - tC * divu)[:, None, None])
        rp = -N * divu[:, None]
        R = torch.cat([ru, rp[:, :, None], torch.zeros_like(rp)[:, :, None]], 2) * w[:, None, None]
        if not want_matrix:
            return R, None
        f1, f2 = p["almi"], p["alfi"] * p["gami"] * p["delt"]
        K = torch.zeros((len(w), len(N), 5, len(N), 5), dtype=torch.float64, device=self.dev)
        gab = torch.einsum("eai,ebi->eab", g, g)
        pair = lambda a, b: a[:, :, None] * b[:, None, :]
        NN = N.expand(len(w), -1)
        k3 = lambda s: s[:, None, None]
        rt = (rho * tM)[:, None]
        S = k3(w * rho) * pair(NN + rt * c, f1 * N + f2 * c) + f2 * mu * k3(w) * gab
        for i in range(3):
            for j in range(3):
                K[:, :, i, :, j] = f2 * mu * k3(w) * pair(g[:, :, j], g[:, :, i]) + \
                    k3(f2 * tC * w) * pair(g[:, :, i], g[:, :, j])
            K[:, :, i, :, i] += S
            K[:, :, i, :, 3] = k3(f2 * w) * (pair(rt * c, g[:, :, i]) - pair(g[:, :, i], NN))
            K[:, :, 3, :, i] = k3(w) * (f2 * pair(NN, g[:, :, i]) + pair(g[:, :, i], rt * (f1 * N + f2 * c)))
        K[:, :, 3, :, 3] = k3(f2 * w * tM) * gab
        return R, K

    def tem(self, q, want_matrix):
        p, w, N, g = self.p, q["w"], q["N"], q["g"]
        ph, mdot, _, dmd, mix = self.phase(q)
        rho, cp, hk = mix(p["rhow"], p["rhoa"], p["rhos"]), mix(p["cpw"], p["cpa"], p["cps"]), \
            mix(p["kappaw"], p["kappaa"], p["kappas"])
        rcp = mix(p["rhow"] * p["cpw"], p["rhoa"] * p["cpa"], p["rhos"] * p["cps"])
        fl = q["fl"].double()
        lat = (p["cpw"] - p["cpa"]) * (q["T"] - p["ts"]) - p["lh"]
        Se, dSe = lat * mdot * fl, ((p["cpw"] - p["cpa"]) * mdot + lat * dmd) * fl
        udT = (q["ua"] * q["dT"]).sum(1) * fl
        res = rcp * (q["rT"] + udT) - Se
        tT = 1.0 / (rho * cp * torch.sqrt(q["uGu"] + 4.0 / p["delt"] ** 2 + (hk / (rho * cp)) ** 2 * 12.0 * q["GG"]))
        kd = p["tem_kdc"] * res.abs() / torch.sqrt(q["GG"]) / p["tref"] * fl
        c = q["c"] * fl[:, None]
        col = lambda s: s[:, None]
        R = -N * col(res) - col(rcp * tT * res) * c - col(hk + kd) * torch.einsum("eai,ei->ea", g, q["dT"])
        R = R[:, :, None] * w[:, None, None]
        if not want_matrix:
            return R, None
        f1, f2 = p["almi"], p["alfi"] * p["gami"] * p["delt"]
        left = col(w) * (N + col(tT * rcp) * c)
        right = col(rcp) * (f1 * N + f2 * c) - f2 * col(dSe) * N
        K = left[:, :, None] * right[:, None, :] + (f2 * (hk + kd) * w)[:, None, None] * torch.einsum("eai,ebi->eab", g, g)
        return R, K[:, :, None, :, None]

    def blocks(self, which, f, el, want_matrix):
        """Element residuals and matrices of the elements `el`, and their largest advective rate."""
        R, K, rate = 0.0, 0.0, 0.0
        for q in self.points(f, el):
            q["fl"] = self.fluid[el]
            r, k = getattr(self, which)(q, want_matrix)
            R = R + r
            K = K + k if want_matrix else None
            rate = max(rate, float(q["uGu"].detach().max()))
        return R, K, rate

    def chunks(self):
        n = CHUNK // 8 if self.hex else CHUNK
        for e in range(0, self.E, n):
            yield slice(e, min(e + n, self.E))

    def free_of(self, nf):
        return self.free[:, 5:6] if nf == 1 else self.free[:, :nf]

    def masked(self, K, nodes):
        """The element Dirichlet treatment: constrained rows and columns out (the continuity row's entry against the
        pressure and its column of the VOF keep the column, a row constrained in velocity i loses the VOF row's
        velocity-i entry), one on the element diagonal of a constrained unknown."""
        nf = K.shape[2]
        fr = self.free_of(nf)[nodes]
        row = torch.ones(K.shape, dtype=torch.bool, device=K.device)
        row &= fr[:, :, :, None, None]
        colm = torch.ones_like(row) & fr[:, None, None, :, :]
        if nf > 1:
            colm[:, :, 3, :, 3] = True
        if nf == 5:
            row[:, :, 0:3, :, 4] = True
            row[:, :, 4, :, 0:3] &= fr[:, :, None, 0:3]
        K = K * (row & colm)
        d = torch.arange(K.shape[1], device=K.device)
        for k in range(nf):
            one = ~fr[:, :, k]
            K[:, d, k, d, k] = torch.where(one, torch.ones_like(K[:, d, k, d, k]), K[:, d, k, d, k])
        return K

    def assemble(self, which, nf, x=None, keep=False):
        """Residual (nf, N); the product with x (nf, N) if given; the element matrices if they are kept."""
        f = self.alpha()
        R = torch.zeros((self.N, nf), dtype=torch.float64, device=self.dev)
        y, kept, rate = torch.zeros_like(R), [], 0.0
        for el in self.chunks():
            nodes = self.ien[el]
            r, K, t = self.blocks(which, f, el, x is not None or keep)
            rate = max(rate, t)
            R.index_add_(0, nodes.reshape(-1), r[:, :, :nf].reshape(-1, nf))
            if K is None:
                continue
            n = nodes.shape[1] * nf
            K = self.masked(K[:, :, :nf, :, :nf], nodes)
            if keep:
                kept.append(K.reshape(-1, n, n))
            else:
                v = x.t()[nodes].reshape(-1, n, 1)
                y.index_add_(0, nodes.reshape(-1), torch.bmm(K.reshape(-1, n, n), v).reshape(-1, nf))
        return (R * self.free_of(nf)).t().contiguous(), y.t().contiguous(), kept, self.p["delt"] * math.sqrt(rate)

    # one Krylov cycle on P^-1 A (P the block diagonal), from zero
    def system(self, which, nf):
        R, _, kept, _ = self.assemble(which, nf, keep=True)
        n = kept[0].shape[1]
        D = torch.zeros((self.N, nf, nf), dtype=torch.float64, device=self.dev)
        a = n // nf
        for el, K in zip(self.chunks(), kept):
            blk = K.reshape(-1, a, nf, a, nf)
            d = torch.arange(a, device=self.dev)
            D.index_add_(0, self.ien[el].reshape(-1), blk[:, d, :, d, :].transpose(0, 1).reshape(-1, nf, nf))
        P = torch.zeros_like(D)
        if nf > 1:
            P[:, :3, :3] = torch.linalg.inv(D[:, :3, :3])
        for k in range(3 if nf > 1 else 0, nf):
            P[:, k, k] = torch.where(D[:, k, k] == 0, 0.0 if k == 4 else 1.0, 1.0 / D[:, k, k])

        def apply(x):
            y = torch.zeros_like(x)
            for el, K in zip(self.chunks(), kept):
                y.index_add_(0, self.ien[el].reshape(-1), torch.bmm(K, x[self.ien[el]].reshape(-1, n, 1)).reshape(-1, nf))
            return y
        return R.t().contiguous(), apply, lambda x: torch.einsum("nij,nj->ni", P, x)

    def cycle(self, b, apply, pre, tol, kspace):
        v = pre(b)
        beta = float(v.norm())
        if beta == 0.0:
            return torch.zeros_like(b), 0.0
        V, H = [v / beta], np.zeros((kspace + 1, kspace))
        for k in range(kspace):
            w = pre(apply(V[k]))
            for _ in range(2):
                for j in range(k + 1):
                    h = float((V[j] * w).sum())
                    w = w - h * V[j]
                    H[j, k] += h
            H[k + 1, k] = float(w.norm())
            V.append(w / H[k + 1, k])
            e1 = np.zeros(k + 2)
            e1[0] = beta
            y, *_ = np.linalg.lstsq(H[:k + 2, :k + 1], e1, rcond=None)
            if np.linalg.norm(e1 - H[:k + 2, :k + 1] @ y) <= tol * beta:
                break
        return sum(float(c) * u for c, u in zip(y, V)), beta


def exact(case, seed):
    """What run() gives, from plain torch in 64 bits: None for the cases whose element matrices would not fit or whose
    iteration would take too long."""
    kind = case["kind"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind in ("gmres", "mixed", "newton") and cells > 250_000:
        return None
    x = _Exact(case, seed)
    if kind in ("pass", "residual"):
        vec = _vectors(case, seed, x.N) if kind == "pass" else (None, None)
        r5, y5, _, cfl = x.assemble("nsvof", 5, vec[0])
        r1, y1, _, c1 = x.assemble("tem", 1, vec[1])
        out = {"cfl": max(cfl, c1), "rhs": [r5, r1]}
        if kind == "pass":
            out["products"] = [y5, y1]
        else:
            out["norms"] = [float((r5[:3] ** 2).sum()), float((r5[3] ** 2).sum()), float((r5[4] ** 2).sum()),
                            float((r1 ** 2).sum())]
            out["norms"] = np.array(out["norms"])
        return out
    if kind == "vjp":
        leaves = [x.st[k].requires_grad_() for k in ("xg", "ug", "pg", "phig", "tg", "acg", "rphig", "rtg")]
        out = []
        for which, nf, cot in zip(("nsvof", "tem"), (5, 1), _vectors(case, seed, x.N)):
            r, *_ = x.assemble(which, nf)
            g = torch.autograd.grad((r * cot).sum(), leaves, allow_unused=True)
            out.append(torch.cat([(torch.zeros_like(v) if a is None else a).reshape(x.N, -1)
                                  for a, v in zip(g, leaves)], 1).detach().cpu().numpy())
        return out
    if kind == "cavity":
        b, apply, pre = x.system("ns", 4)
        s, _ = x.cycle(b, apply, pre, TOL_GMRES, case["kspace"])
        cfl = x.assemble("ns", 4)[3]
        s = s.cpu().numpy()
        return {"cfl": cfl, "rhs": b.cpu().numpy(), "u": s[:, :3], "p": s[:, 3]}
    if kind == "gmres":
        which, nf = ("tem", 1) if case["system"] == "tem" else ("nsvof", 5)
        s, _ = x.cycle(*x.system(which, nf), TOL_GMRES, case["kspace"])
        s = s.cpu().numpy()
        return [s[:, :3], s[:, 3], s[:, 4]] if nf == 5 else [s[:, 0]]
    if kind == "mixed":
        b, apply, pre = x.system("nsvof", 5)
        s, r, began = torch.zeros_like(b), b, time.monotonic()
        while float(r.norm()) > 1e-12 * float(b.norm()):
            if time.monotonic() - began > 12.0:
                return None
            s = s + x.cycle(r, apply, pre, 1e-9, 100)[0]
            r = b - apply(s)
        s = s.cpu().numpy()
        return {"sol": [s[:, k] for k in range(5)], "converged": None}
    p = x.p
    for _ in range(2):
        s, _ = x.cycle(*x.system("nsvof", 5), TOL_GMRES, case["kspace"])
        gd = p["gami"] * p["delt"]
        x.st["acg"] = x.st["acg"] + s[:, :3]
        x.st["ug"] = x.st["ug"] + gd * s[:, :3]
        x.st["pg"] = x.st["pg"] + p["alfi"] * gd * s[:, 3]
        x.st["rphig"] = x.st["rphig"] + s[:, 4]
        x.st["phig"] = x.st["phig"] + gd * s[:, 4]
        s, _ = x.cycle(*x.system("tem", 1), TOL_GMRES, case["kspace"])
        x.st["rtg"] = x.st["rtg"] + s[:, 0]
        x.st["tg"] = x.st["tg"] + gd * s[:, 0]
    return {k: x.st[k].cpu().numpy() for k in ("ug", "acg", "pg", "phig", "rphig", "tg", "rtg")}

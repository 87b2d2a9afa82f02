"""What a user of this framework has it do, as cases that can be timed.

Five kinds of call, each through a public entry point:

* ``pcg``        the ``pcg_solver`` drop-in: the reference's program keeps its
                 plastic loop and hands dense FP64 element matrices over.
* ``stress``     the ``stress_bodyload`` drop-in, the other heavy step of
                 that loop, with the plastic state in host arrays.
* ``trials``     strength-reduction trials on a model that is resident on the
                 device: one plain FP64 trial, or a batch of mixed-precision
                 trials as the factor-of-safety search and the server run them.
* ``excavation`` staged excavation on a resident model.
* ``fos``        a whole factor-of-safety search.

Solver tolerances are tight (``cg_tol`` 1e-12 or 1e-14 for FP64 solves,
``refine_rtol`` 1e-12 for mixed ones, its default 1e-10 on the largest mesh),
as a user sets them who compares two runs, so that an output is the solution
of the equations and not of the last iterations.  A pass is a few plastic
iterations of a trial that in real use takes tens to thousands of them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import specfem3d_geotech_gb300 as sg
from specfem3d_geotech_gb300 import meshgen

PIT_LAYERS = 4   # vertical elements of a pit's depth are taken out in two lifts


def listed():
    return [
        # the reference's 2D example slope through the drop-in: the smallest real call, 300 elements
        dict(name="pcg_2d_300", kind="pcg", mesh="slope2d"),
        # a 3D slope whose dense matrices (315 MB) cross to the device on every call
        dict(name="pcg_3d_6k", kind="pcg", mesh="slope3d", nx=60, ny=10, nz=10),
        # the stress / yield / body-load step of a host's own plastic loop
        dict(name="stress_3d_24k", kind="stress", nx=60, ny=20, nz=20, srf=1.2),
        # one plain FP64 trial of the 2D slope: what `sweep` and a bisection repeat
        dict(name="fp64_2d_300", kind="trials", mesh="slope2d", mixed=False, k=1, srf=1.0, dsrf=0.0, nl=8),
        # the plain FP64 form on a 3D slope of ordinary size
        dict(name="fp64_3d_12k", kind="trials", mesh="slope3d", nx=40, ny=15, nz=20, mixed=False, k=1, srf=1.1, dsrf=0.0,
             nl=2),
        # one mixed trial of a small odd-sized mesh: a serving request's last open probe
        dict(name="mixed1_3d_1k", kind="trials", mesh="slope3d", nx=17, ny=7, nz=9, mixed=True, k=1, srf=1.2, dsrf=0.0,
             nl=6),
        # the eight-trial batch on the 3D cut that whole searches are run on
        dict(name="mixed8_cut_576", kind="trials", mesh="slope3d", nx=24, ny=4, nz=6, mixed=True, k=8, srf=1.0,
             dsrf=0.04, nl=8),
        # five probes (a partly filled batch) on a serving request of ordinary size
        dict(name="mixed5_3d_3k", kind="trials", mesh="slope3d", nx=23, ny=11, nz=13, mixed=True, k=5, srf=1.0,
             dsrf=0.07, nl=4),
        # sixteen probes at once, the widest batch
        dict(name="mixed16_3d_16k", kind="trials", mesh="slope3d", nx=50, ny=16, nz=20, mixed=True, k=16, srf=1.0,
             dsrf=0.03, nl=1),
        # the headline batch on a large slope: one plastic iteration of eight trials
        dict(name="mixed8_3d_62k", kind="trials", mesh="slope3d", nx=72, ny=24, nz=36, mixed=True, k=8, srf=1.0,
             dsrf=0.0625, nl=1, rtol=1e-10),
        # a pit taken out in two lifts, mixed precision, one right-hand side
        dict(name="pit_7k", kind="excavation", nx=24, ny=24, nz=12, nl=2),
        # a whole factor-of-safety search of a small slope
        dict(name="fos_2d_300", kind="fos", lo=1.0, hi=2.0, step=0.1, k=4, nl=20),
    ]


def _box(rng, ne):
    """An odd-sized 3D slope of about `ne` elements."""
    s = (ne / 3.0) ** (1.0 / 3.0)
    n = [max(2, round(f * s * rng.uniform(0.8, 1.25))) for f in (3.0, 1.0, 1.0)]
    return dict(nx=n[0], ny=n[1], nz=n[2])


def _size(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["pcg", "stress", "fp64", "mixed", "mixed", "mixed", "excavation"])
    if kind == "pcg":
        return dict(kind="pcg", mesh="slope3d", **_box(rng, _size(rng, 100, 5000)))
    if kind == "stress":
        return dict(kind="stress", **_box(rng, _size(rng, 200, 20000)), srf=round(rng.uniform(1.0, 1.6), 3))
    if kind == "fp64":
        b = _box(rng, _size(rng, 150, 10000))
        return dict(kind="trials", mesh="slope3d", **b, mixed=False, k=1, srf=round(rng.uniform(1.0, 1.4), 3), dsrf=0.0,
                    nl=max(1, min(6, 10000 // (b["nx"] * b["ny"] * b["nz"]))))
    if kind == "mixed":
        k = rng.choice([1, 2, 3, 4, 6, 8, 8, 11, 16])
        b = _box(rng, _size(rng, 150, 45000 if k <= 8 else 20000))
        ne = b["nx"] * b["ny"] * b["nz"]
        return dict(kind="trials", mesh="slope3d", **b, mixed=True, k=k, srf=1.0, dsrf=round(rng.uniform(0.01, 0.5 / k), 4),
                    nl=max(1, min(8, 10000 // ne)), rtol=1e-12 if ne < 20000 else 1e-10)
    n = round(_size(rng, 9, 24))
    return dict(kind="excavation", nx=n, ny=n + rng.randrange(3), nz=max(8, n // 2), nl=2)


# ---------------------------------------------------------------------------
def _mesh(case, seed):
    if case["kind"] == "excavation":
        m = meshgen.excavation(case["nx"], case["ny"], case["nz"], L=100.0, H=50.0, pit=40.0, lifts=2,
                               lift_h=50.0 * max(1, case["nz"] // PIT_LAYERS) / case["nz"])
    elif case.get("mesh") == "slope2d" or case["kind"] == "fos":
        m = meshgen.slope2d()
    else:
        return meshgen.slope3d(case["nx"], case["ny"], case["nz"], seed=seed % (1 << 31))
    # these have one ground: its stiffness, cohesion and friction come from the seed
    g = np.random.default_rng(seed).standard_normal(3)
    m.props = m.props.copy()
    m.props[:, 1] *= math.exp(0.1 * g[0])
    m.props[:, 4] *= math.exp(0.02 * g[1])
    m.props[:, 3] *= math.exp(0.02 * g[2])
    return m


def _reduced(props, srf):
    """Factored nu, phi, c, psi of a strength reduction (degrees)."""
    phi = np.degrees(np.arctan(np.tan(np.radians(props[:, 3])) / srf))
    psi = np.degrees(np.arctan(np.tan(np.radians(props[:, 5])) / srf))
    return props[:, 2].copy(), phi, props[:, 4] / srf, psi


def _time_step(ym, nuf, phif):
    sn = np.sin(np.radians(phif))
    return float((4.0 * (1.0 + nuf) * (1.0 - 2.0 * nuf) / (ym * (1.0 - 2.0 * nuf + sn * sn))).min())


def prepare(case, seed):
    mesh = _mesh(case, seed)
    kind = case["kind"]
    if kind == "pcg":
        model = sg.Model(mesh)
        k, diag, load = model.stiffness()
        diag[1:] = 1.0 / diag[1:]
        diag[0] = 0.0
        s = dict(kind=kind, neq=model.neq, nelmt=model.nelmt, k=k, f=load, dprecon=diag,
                 ge=model.arrays()["gdof_elmt"])
        model.close()
        return s
    if kind == "stress":
        model = sg.Model(mesh)
        a = model.arrays()
        rng = np.random.default_rng(seed)
        # a settled slope: the column's compression under its own weight, with noise that keeps some points yielding
        z, zt = a["g_coord"][:, 2], mesh.z.max()
        u = np.zeros((model.nnode, 3))
        u[:, 2] = -19.0 / 1.2e5 * (zt * z - 0.5 * z * z) + 1e-5 * rng.standard_normal(model.nnode)
        u[:, 0] = 2e-4 * z + 1e-5 * rng.standard_normal(model.nnode)
        x = np.zeros(model.neq + 1)
        x[a["gdof"].reshape(-1)] = u.reshape(-1)
        x[0] = 0.0
        nuf, phif, cohf, psif = _reduced(mesh.props, case["srf"])
        n = 162 * model.nelmt
        s = dict(kind=kind, neq=model.neq, nelmt=model.nelmt, nnode=model.nnode, coord=a["g_coord"].reshape(-1),
                 gnum=a["g_num"] + 1, ge=a["gdof_elmt"], mat=mesh.mat_id, ym=mesh.props[:, 1].copy(), nuf=nuf, phif=phif,
                 cohf=cohf, psif=psif, dt=_time_step(mesh.props[:, 1], nuf, phif), x=x,
                 evpt=1e-6 * rng.standard_normal(n), stress=np.zeros(n), bodyload=np.zeros(model.neq + 1))
        model.close()
        return s
    mixed = case.get("mixed", True)
    prec = sg.PREC_MIXED if mixed else sg.PREC_FP64
    ctl = sg.make_control(cg_tol=1e-8 if mixed else 1e-14, nl_tol=1e-4, cg_maxiter=20000, nl_maxiter=case["nl"],
                          precision=prec, refine_rtol=case.get("rtol", 1e-12))
    s = dict(kind=kind, mesh=mesh, model=sg.Model(mesh, precision=prec), ctl=ctl)
    if kind == "trials":
        s["srf"] = [case["srf"] + case["dsrf"] * t for t in range(case["k"])]
    elif kind == "fos":
        s["search"] = {k: case[k] for k in ("lo", "hi", "step", "k")}
    return s


def run(s):
    kind = s["kind"]
    if kind == "pcg":
        u = np.zeros(s["neq"] + 1)
        _, err, _ = sg.pcg_solver(s["neq"], s["nelmt"], s["k"], u, s["f"], s["dprecon"], s["ge"], 20000, 1e-12)
        return {"u": u, "errcode": err}
    if kind == "stress":
        fmax = sg.stress_bodyload(s["neq"], s["nelmt"], s["nnode"], s["coord"], s["gnum"], s["ge"], s["mat"], s["ym"],
                                  s["nuf"], s["phif"], s["cohf"], s["psif"], s["dt"], False, False, s["x"], s["evpt"],
                                  s["stress"], s["bodyload"])
        return {"fmax": fmax, "evpt": s["evpt"], "stress": s["stress"], "bodyload": s["bodyload"]}
    if kind == "trials":
        rows, x = s["model"].trials(s["srf"], s["ctl"], want_x=True)
        out = {key: np.array([r[key] for r in rows]) for key in ("uxmax", "umax", "fmax", "uerr")}
        for key in ("nl_iter", "converged", "failed", "errcode"):
            out[key] = np.array([r[key] for r in rows], np.int32)
        return {"x": x, **out}
    if kind == "excavation":
        m = s["mesh"]
        rows = s["model"].excavation(s["ctl"], 1, 50.0, 0.0, 0.5, list(m.control.excavid))
        strain, safety = s["model"].excavation_fields()
        return {"stages": rows[:, 2:].copy(), "vmeps": strain, "scf": safety}
    fos, _, _ = s["model"].fos(s["ctl"], **s["search"])
    return {"fos": fos, "stress": s["model"].last_stress(0)}


# ---------------------------------------------------------------------------
def _counts(case):
    """(elements, dofs, right-hand sides) of a case."""
    if case.get("mesh") == "slope2d" or case["kind"] == "fos":
        nx, ny, nz = 30, 1, 10
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return nx * ny * nz, 3 * (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1), case.get("k", 1), nx


def _moved(its, held):
    """Bytes of `its` iterations over `held` bytes, of which 129 MB stay in the L2 cache."""
    return held + (its - 1) * max(0, held - 129_000_000)


def work(case):
    """Bytes and operations of one pass, with as many PCG iterations as the
    Jacobi-preconditioned solve of such a mesh takes (about 16 for each element
    along its longest side)."""
    ne, n, k, nx = _counts(case)
    kind = case["kind"]
    state = 162 * 8 * ne
    if kind == "stress":
        return {"bytes": 4 * state + 8 * n * 3 + ne * (27 * 4 + 81 * 4 + 27 * 24), "flops": 27 * ne * 900}
    its = 16 * nx
    if kind == "pcg":
        # the matrices and six vectors on each iteration
        return {"bytes": _moved(its, 8 * 6561 * ne + 8 * 6 * n), "flops": its * 2 * 6561 * ne}
    steps = case.get("nl", 1) * (2 if kind == "excavation" else 1)
    if kind == "fos":
        steps *= 5
    word = 4 if case.get("mixed", True) else 8
    # per iteration and right-hand side six vectors; the operator's point records (12 values) are read once for all
    each = _moved(its, word * 6 * n * k + word * 12 * 27 * ne)
    return {"bytes": steps * (each + k * 3 * state), "flops": steps * k * (its * 2 * 3600 * ne + 27 * ne * 900)}


# ---------------------------------------------------------------------------
# The same results in 64 bits from the equations themselves: dense matrices
# from B^T C B, a Cholesky factor in the place of the PCG.  The node and dof
# numbers, which only say where a value stands, are the model's.
# ---------------------------------------------------------------------------
class _Fe:
    def __init__(self, coord, gnum, ge, mat, neq, dev):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.dev, self.neq = dev, neq
        self.ge, self.mat = t(ge).long().reshape(-1, 81), t(mat).long() - 1
        D = np.array([[-1.5, 2.0, -0.5], [-0.5, 0.0, 0.5], [0.5, -2.0, 1.5]])
        i3 = np.eye(3)
        # derivative of node n's shape function at point q, nodes and points numbered i + 3j + 9k
        dl = np.stack([np.einsum("kc,jb,ia->kjicba", i3, i3, D), np.einsum("kc,jb,ia->kjicba", i3, D, i3),
                       np.einsum("kc,jb,ia->kjicba", D, i3, i3)]).reshape(3, 27, 27)
        w1 = np.array([1.0, 4.0, 1.0]) / 3.0
        w = np.einsum("k,j,i->kji", w1, w1, w1).reshape(27)
        # 8-node map: corner signs of the corner nodes
        xi = np.array([-1.0, 0.0, 1.0])
        P = np.array([[xi[q % 3], xi[q // 3 % 3], xi[q // 9]] for q in range(27)])
        corner = [0, 2, 8, 6, 18, 20, 26, 24]
        S = P[corner]
        ds = np.empty((27, 8, 3))
        for a in range(3):
            b, c = [d for d in range(3) if d != a]
            ds[:, :, a] = 0.125 * S[:, a] * (1 + P[:, None, b] * S[None, :, b]) * (1 + P[:, None, c] * S[None, :, c])
        xc = t(np.asarray(coord).reshape(-1, 3)[np.asarray(gnum)[:, corner]])
        J = torch.einsum("qga,egb->eqab", t(ds), xc)
        self.wd = torch.linalg.det(J) * t(w)
        self.grad = torch.einsum("eqda,aqn->eqnd", torch.linalg.inv(J), t(dl))

    def strain(self, x):
        """Engineering strain at the points; x is (..., neq + 1)."""
        u = x[..., self.ge].reshape(*x.shape[:-1], -1, 27, 3)
        G = torch.einsum("...enc,eqnd->...eqcd", u, self.grad)
        return torch.stack([G[..., 0, 0], G[..., 1, 1], G[..., 2, 2], G[..., 0, 1] + G[..., 1, 0],
                            G[..., 1, 2] + G[..., 2, 1], G[..., 2, 0] + G[..., 0, 2]], -1)

    def force(self, s):
        """Sum over elements and points of B^T s w detJ, as (..., neq + 1) with entry 0 left out."""
        T = torch.stack([torch.stack([s[..., 0], s[..., 3], s[..., 5]], -1),
                         torch.stack([s[..., 3], s[..., 1], s[..., 4]], -1),
                         torch.stack([s[..., 5], s[..., 4], s[..., 2]], -1)], -2)
        F = torch.einsum("...eqcd,eqnd,eq->...enc", T, self.grad, self.wd)
        F = F.reshape(*F.shape[:-3], -1)
        out = torch.zeros(*F.shape[:-1], self.neq + 1, dtype=F.dtype, device=F.device)
        out.index_add_(-1, self.ge.reshape(-1), F)
        out[..., 0] = 0.0
        return out

    def elastic(self, ym, nu):
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=self.dev)[self.mat][:, None]  # noqa: E731
        E, v = t(ym), t(nu)
        f = E / ((1 + v) * (1 - 2 * v))
        self.c11, self.c12, self.c44 = (1 - v) * f, v * f, 0.5 * (1 - 2 * v) * f

    def hooke(self, e):
        tr = e[..., :3].sum(-1, keepdim=True)
        d = (self.c11 - self.c12)[..., None]
        return torch.cat([self.c12[..., None] * tr + d * e[..., :3], self.c44[..., None] * e[..., 3:]], -1)

    def factor(self):
        K = torch.zeros(self.neq + 1, self.neq + 1, dtype=torch.float64, device=self.dev)
        B = torch.zeros(*self.grad.shape[:2], 6, 27, 3, dtype=torch.float64, device=self.dev)
        g = self.grad
        for row, col, d in ((0, 0, 0), (1, 1, 1), (2, 2, 2), (3, 0, 1), (3, 1, 0), (4, 1, 2), (4, 2, 1), (5, 0, 2),
                            (5, 2, 0)):
            B[:, :, row, :, col] = g[:, :, :, d]
        B = B.reshape(*B.shape[:3], 81)
        unit = torch.eye(6, dtype=torch.float64, device=self.dev)[None].expand(B.shape[0], 6, 6)
        CB = torch.einsum("est,eqtb,eq->eqsb", self.hooke(unit), B, self.wd)
        Ke = torch.einsum("eqsa,eqsb->eab", B, CB)
        K.index_put_((self.ge[:, :, None].expand_as(Ke), self.ge[:, None, :].expand_as(Ke)), Ke, accumulate=True)
        self.L = torch.linalg.cholesky(K[1:, 1:])

    def solve(self, f):
        x = torch.zeros_like(f)
        x[..., 1:] = torch.cholesky_solve(f[..., 1:].T.contiguous(), self.L).T
        return x

    def flow(self, eff, phif, cohf, psif, dt):
        """Mohr-Coulomb F and the viscoplastic strain increment of one step; the strengths are per element."""
        sn, cs, sp = torch.sin(phif), torch.cos(phif), torch.sin(psif)
        r3 = math.sqrt(3.0)
        s = eff
        sm = s[..., :3].sum(-1) / 3
        d2 = ((s[..., 0] - s[..., 1]) ** 2 + (s[..., 1] - s[..., 2]) ** 2 + (s[..., 2] - s[..., 0]) ** 2) / 6 + \
            (s[..., 3:] ** 2).sum(-1)
        d2 = d2.clamp_min(1e-12)
        dx, dy, dz = (s[..., i] - sm for i in range(3))
        xy, yz, zx = s[..., 3], s[..., 4], s[..., 5]
        d3 = dx * dy * dz - dx * yz ** 2 - dy * zx ** 2 - dz * xy ** 2 + 2 * xy * yz * zx
        q = r3 * d2.sqrt()
        sine = (-3 * r3 * d3 / (2 * d2.sqrt() ** 3)).clamp(-1, 1)
        th = torch.where(q < 1e-12, torch.zeros_like(q), torch.asin(sine) / 3)
        F = sn * sm + q * (torch.cos(th) / r3 - torch.sin(th) * sn / 3) - cohf * cs
        st, ct = torch.sin(th), torch.cos(th)
        t3, tt = torch.tan(3 * th), st / ct
        corner = st.abs() > 0.49
        c1 = torch.where(st < 0, -1.0, 1.0)
        g2 = torch.where(corner, (r3 / 2 - c1 * sp / 2 / r3) * r3 / 2 / q,
                         r3 * ct / q * ((1 + tt * t3) + sp * (t3 - tt) / r3) / 2)
        g3 = torch.where(corner, torch.zeros_like(q), 1.5 * (r3 * st + sp * ct) / (torch.cos(3 * th) * q * q))
        # the flow direction: M1 s = 1/3 on the normals, M2 s the deviator (shears doubled), M3 s the deviator's square
        one = torch.zeros_like(s)
        one[..., :3] = 1.0
        dev = torch.stack([dx, dy, dz, 2 * xy, 2 * yz, 2 * zx], -1)
        j2 = (2.0 / 3.0) * d2
        sq = torch.stack([dx * dx + xy * xy + zx * zx - j2, dy * dy + xy * xy + yz * yz - j2,
                          dz * dz + yz * yz + zx * zx - j2, 2 * (dx * xy + xy * dy + zx * yz),
                          2 * (xy * zx + dy * yz + yz * dz), 2 * (dx * zx + xy * yz + zx * dz)], -1)
        m = (sp / 3)[..., None] * one + g2[..., None] * dev + g3[..., None] * sq
        return F, torch.where((F >= 0)[..., None], dt * F[..., None] * m, torch.zeros_like(m))


def exact(case, seed):
    kind = case["kind"]
    ne, n, _, _ = _counts(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "pcg" and n < 24000:
        s = prepare(case, seed)
        K = torch.zeros(s["neq"] + 1, s["neq"] + 1, dtype=torch.float64, device=dev)
        ge = torch.as_tensor(s["ge"], device=dev).long()
        Ke = torch.as_tensor(s["k"], device=dev)
        K.index_put_((ge[:, :, None].expand_as(Ke), ge[:, None, :].expand_as(Ke)), Ke, accumulate=True)
        u = np.zeros(s["neq"] + 1)
        u[1:] = torch.linalg.solve(K[1:, 1:], torch.as_tensor(s["f"][1:], device=dev)).cpu().numpy()
        return {"u": u, "errcode": None}
    if kind == "stress":
        s = prepare(case, seed)
        fe = _Fe(s["coord"], s["gnum"] - 1, s["ge"], s["mat"], s["neq"], dev)
        fe.elastic(s["ym"], s["nuf"])
        per = lambda a: torch.as_tensor(a, device=dev)[fe.mat][:, None]  # noqa: E731
        ev = torch.as_tensor(s["evpt"].copy(), device=dev).reshape(-1, 27, 6)
        eff = fe.hooke(fe.strain(torch.as_tensor(s["x"], device=dev)) - ev)
        F, evp = fe.flow(eff, per(np.radians(s["phif"])), per(s["cohf"]), per(np.radians(s["psif"])), s["dt"])
        return {"fmax": max(0.0, float(F.max())), "evpt": (ev + evp).reshape(-1).cpu().numpy(), "stress": s["stress"],
                "bodyload": fe.force(fe.hooke(evp)).cpu().numpy()}
    if kind != "trials" or n > 24000:
        return None
    mesh = _mesh(case, seed)
    model = sg.Model(mesh)
    a, neq = model.arrays(), model.neq
    model.close()
    fe = _Fe(a["g_coord"], a["g_num"], a["gdof_elmt"], mesh.mat_id, neq, dev)
    fe.elastic(mesh.props[:, 1], mesh.props[:, 2])
    fe.factor()
    per = lambda v: torch.as_tensor(v, device=dev)[fe.mat][:, None]  # noqa: E731
    load = torch.zeros(neq + 1, dtype=torch.float64, device=dev)
    load.index_add_(0, fe.ge[:, 2::3].reshape(-1), -(fe.wd * per(mesh.props[:, 0])).reshape(-1))
    load[0] = 0.0
    gdof = torch.as_tensor(a["gdof"], device=dev).long()
    out = {key: [] for key in ("x", "uxmax", "umax", "fmax", "uerr")}
    for t in range(case["k"]):
        nuf, phif, cohf, psif = _reduced(mesh.props, case["srf"] + case["dsrf"] * t)
        dt = _time_step(mesh.props[:, 1], nuf, phif)
        strength = per(np.radians(phif)), per(cohf), per(np.radians(psif))
        body, old, ev = torch.zeros_like(load), torch.zeros_like(load), 0.0
        for it in range(1, case["nl"] + 1):
            x = fe.solve((load + body)[None])[0]
            uerr = float((x - old).abs().max() / x.abs().max())
            old = x
            eff = fe.hooke(fe.strain(x) - ev)
            F, evp = fe.flow(eff, *strength, dt)
            ev = ev + evp
            if uerr <= 1e-4:
                break
            if it < case["nl"]:
                body = body + fe.force(fe.hooke(evp))
        u = x[gdof]
        for key, v in (("x", x.cpu().numpy()), ("uxmax", float(u.abs().max())), ("umax", float(u.norm(dim=1).max())),
                       ("fmax", max(0.0, float(F.max()))), ("uerr", uerr)):
            out[key].append(v)
    return {key: np.array(v) for key, v in out.items()}

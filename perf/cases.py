"""Performance cases: what users of this framework have it do, through its
public entry points (``mafem.py`` over ``libmafem.so``).

A user steps membrane patches: the reference's ``time_step!`` on host arrays
(``Solver.time_step``), its time loop on a resident state (``run_analysis``),
the two lines a Julia host replaces (``calc_r_K`` and ``\\``), the record it
writes after every step (``pull_record``), many patches at once (``Batch``) and
solves that arrive at a server (``Server``).  Patches run from a few elements a
side, where launches and latencies count, to 64 x 64; they are square or not,
their sizes even or odd, in every mesh motion, in plain FP64 and in the FP32
form with FP64 refinement.

A case names what is called (``do``), the scenario and motion, the elements per
side (``n1``, ``n2``), the precision and the number of time steps; batches and
servers hold ``patches`` patches of ``lo`` to ``hi`` elements a side.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "membranealefem.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import mafem as M  # noqa: E402

MOTIONS = {"static": M.STATIC, "eul": M.EUL, "lag": M.LAG, "alev": M.ALEV, "alevb": M.ALEVB}
SCENARIOS = {"cavity": M.F_CAVI, "couette": M.F_COUE, "poiseuille": M.F_POIS, "pull": M.F_PULL, "bend": M.F_BEND}
PRECISIONS = {"fp64": M.PLAIN_FP64, "fp32": M.FP32_REFINE}
SIZES = (8, 12, 16, 24, 32, 48)  # the batching workload's sizes
DT = 0.01
DOF = {"lag": 4, "alev": 8, "alevb": 8, "eul": 7, "static": 3}


def _one(do, scenario, motion, n1, n2, precision="fp64", steps=1):
    return {"do": do, "scenario": scenario, "motion": motion, "n1": n1, "n2": n2, "precision": precision,
            "steps": steps}


def _many(do, patches, lo, hi, steps):
    return {"do": do, "patches": patches, "lo": lo, "hi": hi, "steps": steps}


def listed():
    return [
        # what a tether-pull run writes after every step: the smallest call, on the reference's default mesh
        {"name": "record_17", **_one("record", "pull", "alevb", 17, 17)},
        # a host program that keeps the tangent itself: one small assembly, r and K taken back
        {"name": "assemble_lag_8", **_one("assemble", "pull", "lag", 8, 8)},
        # the drop-in for the reference's two lines r, K = calc_r_K(...), K \ r, on a ragged Lagrangian patch
        {"name": "seam_lag_24x21", **_one("seam", "pull", "lag", 24, 21)},
        # time_step! of a small Lagrangian patch: latency and launches
        {"name": "step_lag_8", **_one("step", "pull", "lag", 8, 8)},
        # time_step! on the reference's default mesh and motion (odd size)
        {"name": "step_alevb_17", **_one("step", "pull", "alevb", 17, 17)},
        # pure bending with the Eulerian mesh, a long ragged patch, boundary moments
        {"name": "bend_eul_23x11", **_one("step", "bend", "eul", 23, 11)},
        # the benchmark's patch: the time loop on a resident state, plain FP64
        {"name": "run_alevb_32", **_one("run", "pull", "alevb", 32, 32, steps=2)},
        # the largest patch a user refines to, plain FP64
        {"name": "step_alevb_64", **_one("step", "pull", "alevb", 64, 64)},
        # the benchmark's patch in the FP32 form with FP64 refinement
        {"name": "step_alevb_32_fp32", **_one("step", "pull", "alevb", 32, 32, precision="fp32")},
        # a parameter study on small patches: one batch, a few steps
        {"name": "batch_small", **_many("batch", 24, 8, 16, 2)},
        # the batching workload: 256 patches of every size, half Lagrangian, half ALEVB
        {"name": "batch_mixed", **_many("batch", 256, 8, 48, 1)},
        # solves submitted to the server together, admitted and run as one continuous batch
        {"name": "serve_mixed", **_many("serve", 24, 8, 32, 2)},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    do = rng.choice(["record", "assemble", "seam", "step", "step", "step", "run", "step32", "batch", "serve"])
    if do in ("batch", "serve"):
        lo = rng.choice(SIZES[:3])
        hi = rng.choice([s for s in SIZES if s >= lo and (do == "batch" or s <= 32)])
        patches = _log_int(rng, 6, 200 if do == "batch" else 40)
        return _many(do, patches, lo, hi, rng.randint(1, 2) if hi <= 24 else 1)
    top = {"record": 40, "assemble": 20, "seam": 40, "step": 56, "run": 36, "step32": 40}[do]
    motion = rng.choice(["eul", "lag", "alev", "alevb", "alevb"])
    if do == "seam" and motion != "lag":
        top = 12  # one linear solve: beyond, the moving meshes' condition leaves it few digits to compare
    n1 = _log_int(rng, 6, top)
    n2 = max(5, min(top, round(n1 * math.exp(rng.uniform(-0.5, 0.5)))))
    scenario = "pull"
    if do in ("step", "run") and rng.random() < 0.25:
        scenario, motion = rng.choice([("bend", "lag"), ("bend", "eul"), ("cavity", "static"), ("couette", "static"),
                                       ("poiseuille", "static")])
    return _one("step" if do == "step32" else do, scenario, motion, n1, n2,
                "fp32" if do == "step32" else "fp64", rng.randint(2, 3) if do == "run" else 1)


# ---- inputs ------------------------------------------------------------------------
# Parameters and states are drawn from the seed in the ranges of the batching
# workload: bending modulus, edge tension and pull force per patch, the pull in
# the first steps of its ramp.  A single pulled patch starts from a smooth
# out-of-plane bump, as a membrane in the middle of a run has one.
def _patch(rng, scenario, motion, n1, n2, bump):
    sc, mo = SCENARIOS[scenario], MOTIONS[motion]
    kb = float(np.exp(rng.uniform(np.log(0.5), np.log(2.0))))
    lam0 = float(np.exp(rng.uniform(np.log(0.1), np.log(10.0))))
    force = float(rng.uniform(2.0, 10.0))
    kw = {}
    if sc == M.F_PULL:
        kw = {"kb": kb, "lambda0": lam0, "pull_centre": 1, "pull_speed": 0.02 * force / 30.0}
    elif sc == M.F_BEND:
        kw = {"kb": kb, "kg": -kb / 2, "bend_mf": kb / 2.0}
    else:
        kw = {"zeta_v": kb}
    p = M.Params(motion=mo, scenario=sc, num1el=n1, num2el=n2, length=1.0, **kw)
    mesh = M.Mesh(p)
    if sc == M.F_BEND:
        xms = np.zeros((mesh.numnp, 3), order="F")
        s1, s2 = np.arange(mesh.numnp) % mesh.num1np, np.arange(mesh.numnp) // mesh.num1np
        xms[:, 0] = np.clip((s1 - 0.5) / (mesh.num1np - 2), 0, 1)
        xms[:, 1] = np.clip((s2 - 0.5) / (mesh.num2np - 2), 0, 1)
        cps = np.zeros((mesh.numnp, mesh.ndf), order="F")
        cps[:, mesh.dofs[6] - 1] = kb / 4
    else:
        _, xms, cps = M.prepare_input(p, mesh)
    if sc == M.F_PULL and bump:
        x, y = xms[:, 0] - xms[:, 0].min(), xms[:, 1] - xms[:, 1].min()
        for k in (1, 2):
            for m in (1, 2):
                xms[:, 2] += 1e-3 / (k * m) * rng.uniform(-1, 1) * np.sin(np.pi * k * x) * np.sin(np.pi * m * y)
    if sc not in (M.F_PULL, M.F_BEND):  # a flow that has not settled yet: some tension on the free unknowns
        free = (mesh.ID > 0).T
        cps = np.asfortranarray(cps + np.where(free, 0.1 * rng.uniform(-1, 1, cps.shape), 0.0))
    return p, mesh, xms, cps


def _patches(case, seed):
    rng = np.random.default_rng(seed)
    if case["do"] not in ("batch", "serve"):
        return [_patch(rng, case["scenario"], case["motion"], case["n1"], case["n2"], True)]
    sizes = [s for s in SIZES if case["lo"] <= s <= case["hi"]]
    out = []
    for k in range(case["patches"]):  # every size about as often, in either motion
        n = sizes[k // 2 % len(sizes)]
        out.append(_patch(rng, "pull", "lag" if k % 2 == 0 else "alevb", n, n, False))
    return out


class _State:
    """What a user's program holds: meshes, initial states and a solver, batch or server."""

    def __init__(self, case, seed):
        self.case = case
        self.patches = _patches(case, seed)
        self.solvers, self.batch, self.server = [], None, None
        if case["do"] == "serve":
            self.server = M.Server()
            return
        prec = PRECISIONS[case.get("precision", "fp32")]
        self.solvers = [M.Solver(mesh, p, prec) for p, mesh, _, _ in self.patches]
        if case["do"] == "batch":
            for s, (_, _, xms, cps) in zip(self.solvers, self.patches):
                s.set_refinement(30, 1e-4)  # the benchmark's: Newton's FP64 criterion decides convergence
                s.upload(xms, cps)
                s.snapshot_reserve(1)
                s.snapshot(0)
            self.batch = M.Batch(self.solvers)

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        if self.server is not None:
            self.server.close()
        for s in self.solvers:
            s.close()


def prepare(case, seed):
    return _State(case, seed)


# ---- one pass ----------------------------------------------------------------------
def run(state):
    case = state.case
    do = case["do"]
    if do == "batch":
        for s in state.solvers:
            s.restore(0)
        for k in range(case["steps"]):
            status, _ = state.batch.step((k + 1) * DT, DT)
        got = [s.download() for s in state.solvers]
        return {"status": np.array(status), "xms": np.concatenate([x.ravel() for x, _ in got]),
                "cps": np.concatenate([c.ravel() for _, c in got])}
    if do == "serve":
        sv = state.server
        ids = [sv.submit(mesh, p, xms, cps, case["steps"], DT, precision=M.FP32_REFINE, refine_tol=1e-4)
               for p, mesh, xms, cps in state.patches]
        while sum(sv.round()):
            pass
        got = [sv.result(i) for i in ids]
        return {"status": np.array([st for st, _, _ in got]), "xms": np.concatenate([x.ravel() for _, x, _ in got]),
                "cps": np.concatenate([c.ravel() for _, _, c in got])}
    s = state.solvers[0]
    _, mesh, xms, cps = state.patches[0]
    if do == "record":
        s.upload(xms, cps)
        return {"record": np.array(s.pull_record(DT))}
    if do == "assemble":
        r, band = s.calc_r_K(xms, cps, DT, DT)
        return {"r": r, "K": band}
    if do == "seam":
        r, _ = s.calc_r_K(xms, cps, DT, DT, tangent=False)
        return {"r": r, "du": s.solve(r)}
    if do == "step":
        x, c = xms.copy(order="F"), cps.copy(order="F")
        s.time_step(x, c, DT, DT)
        return {"xms": x, "cps": c}
    s.upload(xms, cps)
    s.run_analysis([DT] * case["steps"])
    x, c = s.download()
    return {"xms": x, "cps": c}


# ---- the work of one pass --------------------------------------------------------------
NEWTON = 4  # Newton iterations of a typical time step


def _sizes(motion, n1, n2):
    ndf = DOF[motion]
    n = (n1 + 2) * (n2 + 2) * ndf
    return ndf, n, (2 * (n1 + 2) + 2) * ndf


def work(case):
    do = case["do"]
    if do in ("batch", "serve"):
        sizes = [s for s in SIZES if case["lo"] <= s <= case["hi"]]
        per = [("lag" if k % 2 == 0 else "alevb", sizes[k // 2 % len(sizes)]) for k in range(case["patches"])]
        per = [(m, s, s) for m, s in per]
    else:
        per = [(case["motion"], case["n1"], case["n2"])]
    nbytes = flops = 0.0
    for motion, n1, n2 in per:
        ndf, n, bw = _sizes(motion, n1, n2)
        state = 8.0 * (n1 + 2) * (n2 + 2) * (3 + ndf)
        # per Gauss point: the derivative of its ~5 ndf row coefficients along ~4 ndf inputs and the two
        # contractions with the nodes' basis values; a banded LU and its two substitutions
        asm = n1 * n2 * 9.0 * (200.0 * ndf * ndf + 2 * 54.0 * ndf * ndf * 9)
        lu = 2.0 * n * bw * bw + 4.0 * n * bw
        if do == "record":
            nbytes, flops = state, 25 * 9 * 1500.0
        elif do == "assemble":
            nbytes, flops = state + 8.0 * n + 8.0 * n * (3 * bw + 1), asm
        elif do == "seam":
            nbytes, flops = state + 3 * 8.0 * n, asm + lu
        else:
            nbytes += 2 * state
            flops += case["steps"] * NEWTON * (asm + lu)
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------------
# The weak form evaluated at the Gauss points with torch (complex128, so that a
# complex step gives the tangent to rounding), dense matrices and torch's dense
# solver.  The mesh (connectivity, numbering, basis values at the Gauss points,
# boundary conditions) is input data here as it is for the solver.
class _Exact:
    def __init__(self, p, mesh):
        self.p, self.mesh = p, mesh
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=self.dev)  # noqa: E731
        self.IX = t(mesh.IX.T - 1, torch.int64)  # [E, 9]
        self.LM = t(mesh.LM.T - 1, torch.int64)  # [E, 9 ndf], -1: Dirichlet
        uel, uf = mesh.area_tables()
        self.tab = t(uf[uel - 1])  # [E, 9, 55]
        xi = np.array([-math.sqrt(0.6), 0.0, math.sqrt(0.6)])
        q = np.stack([np.tile(xi, 3), np.repeat(xi, 3), np.ones(9)])  # the projection's polynomials at the points
        db = []
        for f in uf:
            w, N = f[:, 0], f[:, 1:10]
            G, H = (q * w) @ N, (q * w) @ q.T
            db.append(G.T @ np.linalg.solve(H, G))
        self.db = t(np.array(db)[uel - 1])  # [E, 9, 9]
        d = [v - 1 for v in mesh.dofs]
        self.d = d
        self.ndf, self.n, self.E = mesh.ndf, mesh.nmdf, mesh.numel
        self.move = {M.STATIC: [], M.LAG: d[0:3]}.get(p.motion, d[3:6])
        self.neu = []
        n1, n2 = mesh.num1el, mesh.num2el
        for b, kind, val in mesh.neumann():
            el = {M.BOTTOM: np.arange(n1), M.RIGHT: n1 - 1 + n1 * np.arange(n2), M.TOP: n1 * (n2 - 1) + np.arange(n1),
                  M.LEFT: n1 * np.arange(n2)}[b]
            ub, ufb = mesh.bdry_tables(b)
            self.neu.append((b, kind, val, t(el, torch.int64), t(ufb[ub - 1])))

    @staticmethod
    def _geo(X, dN, ddN=None):
        a = torch.einsum("...ebi,egbk->...egik", X, dN)
        m = torch.einsum("...ik,...il->...kl", a, a)
        det = m[..., 0, 0] * m[..., 1, 1] - m[..., 0, 1] * m[..., 0, 1]
        inv = torch.stack([torch.stack([m[..., 1, 1], -m[..., 0, 1]], -1),
                           torch.stack([-m[..., 0, 1], m[..., 0, 0]], -1)], -2) / det[..., None, None]
        J = torch.sqrt(det)
        a1, a2 = a[..., 0], a[..., 1]
        n = torch.stack([a1[..., 1] * a2[..., 2] - a1[..., 2] * a2[..., 1], a1[..., 2] * a2[..., 0] - a1[..., 0] * a2[..., 2],
                         a1[..., 0] * a2[..., 1] - a1[..., 1] * a2[..., 0]], -1) / J[..., None]
        up = a @ inv
        return a, inv, det, J, n, up

    def elem(self, X, C, time, area_only=False, els=None):
        """Element residuals [..., E, 9, ndf] of node positions X [..., E, 9, 3] and unknowns C [..., E, 9, ndf]."""
        p, d = self.p, self.d
        cx = X.dtype
        tab = self.tab if els is None else self.tab[els]
        w, N = tab[..., 0].to(cx), tab[..., 1:10].to(cx)
        dN = tab[..., 10:28].unflatten(-1, (2, 9)).transpose(-1, -2).to(cx)
        ddN = tab[..., 28:55].unflatten(-1, (3, 9)).transpose(-1, -2).to(cx)
        a, inv, det, J, n, up = self._geo(X, dN)
        xab = torch.einsum("...ebi,egbk->...egik", X, ddN)  # [.., 3, (11, 22, 12)]
        Gam = torch.einsum("...ik,...ia->...ka", xab, up)
        bv = torch.einsum("...ik,...i->...k", xab, n)
        b = torch.stack([torch.stack([bv[..., 0], bv[..., 2]], -1), torch.stack([bv[..., 2], bv[..., 1]], -1)], -2)
        bup = inv @ b @ inv
        H = 0.5 * (inv * b).sum((-1, -2))
        K = (bv[..., 0] * bv[..., 1] - bv[..., 2] * bv[..., 2]) / det
        val = lambda us: torch.einsum("...ebu,egb->...egu", C[..., us], N)  # noqa: E731
        der = lambda us: torch.einsum("...ebu,egbk->...eguk", C[..., us], dN)  # noqa: E731
        lam = val([d[6]])[..., 0]
        absent = [u for u in d[0:3] if u < 0]
        Z = torch.zeros_like(a)

        def grad(us):
            if not absent and min(us) >= 0:
                return der(us)
            g = Z.clone()
            for i, u in enumerate(us):
                if u >= 0:
                    g[..., i, :] = der([u])[..., 0, :]
            return g

        def visc(g):
            q = up.transpose(-1, -2) @ g @ inv
            return p.zeta_v * (q + q.transpose(-1, -2))

        dv = grad(d[0:3])
        s = lambda v: v[..., None, None]  # noqa: E731
        bend = inv * s(p.kb * H * H - p.kg * K) - bup * s(2 * p.kb * H)
        sig = bend + inv * s(lam) + visc(dv)
        Mm = inv * s(H * (p.kb + 2 * p.kg)) - bup * p.kg
        JW = J * w
        MV = torch.stack([Mm[..., 0, 0], Mm[..., 1, 1], 2 * Mm[..., 0, 1]], -1)
        # second derivatives along the surface: N_,k - Gamma^a_k N_,a
        nn = ddN - torch.einsum("...egka,egba->...egbk", Gam, dN)
        mrow = torch.einsum("...egbk,...egk->...egb", nn, MV * JW[..., None])

        def rows(st, moment, press):
            f = torch.einsum("...egia,...egac,egbc->...egbi", a, st * s(JW), dN)
            if moment:
                f = f + n[..., None, :] * mrow[..., None]
            return f - n[..., None, :] * (press * JW)[..., None, None] * N[..., None]

        out = torch.zeros(X.shape[:-3] + (X.shape[-3], 9, self.ndf), dtype=cx, device=X.device)

        def put(us, f):
            for i, u in enumerate(us):
                if u >= 0:
                    out[..., u] += f[..., i].sum(-2)

        one = torch.ones_like(J)
        put(d[0:3], rows(sig, True, p.pn * one))
        adb = (p.length ** 2 if p.alpha_db is None else p.alpha_db) / p.zeta_v
        if p.motion in (M.ALEV, M.ALEVB):
            pm = val([d[7]])[..., 0]
            put(d[3:6], rows(bend + visc(grad(d[3:6])), p.motion == M.ALEVB, pm))
            nd = (n * (val(d[3:6]) - val(d[0:3]))).sum(-1)
            put([d[7]], ((-(JW * nd) - pm * w * adb)[..., None] * N)[..., None])
        if p.motion == M.EUL:
            v, vm = val(d[0:3]), val(d[3:6])
            f = (vm - n * (n * v).sum(-1)[..., None]) * (JW * p.alpha_m)[..., None]
            put(d[3:6], f[..., None, :] * N[..., None])
        tr = (up * dv).sum((-1, -2))
        put([d[6]], (((J * tr - adb * lam) * w)[..., None] * N)[..., None])
        if area_only:
            return out
        for u in [d[6]] + ([d[7]] if p.motion in (M.ALEV, M.ALEVB) else []):
            out[..., u] += adb * torch.einsum("ebc,...ec->...eb", self.db.to(cx), C[..., u])
        for bd, kind, value, el, tb in self.neu:
            w, N = tb[..., 0].to(cx), tb[..., 1:10].to(cx)
            dN = tb[..., 10:28].unflatten(-1, (2, 9)).transpose(-1, -2).to(cx)
            a, inv, det, J, n, up = self._geo(X[..., el, :, :], dN)
            t0 = a[..., 0] if bd in (M.BOTTOM, M.TOP) else a[..., 1]
            sgn = 1.0 if bd in (M.BOTTOM, M.RIGHT) else -1.0
            tau = sgn * t0 / torch.sqrt((t0.real ** 2).sum(-1, keepdim=True)).to(cx)  # the norm is not differentiated
            nu = torch.stack([tau[..., 1] * n[..., 2] - tau[..., 2] * n[..., 1],
                              tau[..., 2] * n[..., 0] - tau[..., 0] * n[..., 2],
                              tau[..., 0] * n[..., 1] - tau[..., 1] * n[..., 0]], -1)
            tu = torch.einsum("...ia,...i->...a", up, tau)
            JG = w / torch.sqrt((tu * tu).sum(-1))
            if kind == M.MOMENT:
                nua = torch.einsum("...ia,...i->...a", up, nu)
                dn = torch.einsum("...ega,egba->...egb", nua, dN) * (JG * value * min(time / p.bend_tm, 1.0))[..., None]
                f = -n[..., None, :] * dn[..., None]
            else:
                f = -(nu if kind == M.STRETCH else tau)[..., None, :] * (JG * value)[..., None, None] * N[..., None]
            for i, u in enumerate(d[0:3]):
                if u >= 0:
                    out[..., el, :, u] += f[..., i].sum(-2)
        return out

    def r_K(self, xms, cps, time, dt, tangent=True):
        X, C = xms[self.IX].to(torch.complex128), cps[self.IX].to(torch.complex128)
        re = self.elem(X, C, time).real.flatten(-2)
        lm = torch.where(self.LM >= 0, self.LM, self.n)
        r = torch.zeros(self.n + 1, dtype=torch.float64, device=self.dev)
        r.index_add_(0, lm.flatten(), re.flatten())
        if not tangent:
            return r[:-1], None
        nq, h = 9 * self.ndf, 1e-30
        K = torch.zeros((self.n + 1) * (self.n + 1), dtype=torch.float64, device=self.dev)
        for q in range(nq):  # the complex step of element unknown q, every element at once
            b, k = divmod(q, self.ndf)
            Xq, Cq = X.clone(), C.clone()
            Cq[:, b, k] += 1j * h
            for j, u in enumerate(self.move):
                if u == k:
                    Xq[:, b, j] += 1j * h * dt
            col = self.elem(Xq, Cq, time).imag.flatten(-2) / h
            K.index_add_(0, (lm * (self.n + 1) + lm[:, q:q + 1]).flatten(), col.flatten())
        return r[:-1], K.view(self.n + 1, self.n + 1)[:-1, :-1]

    def step(self, xms, cps, time, dt):
        ID = torch.as_tensor(np.ascontiguousarray(self.mesh.ID.T) - 1, device=self.dev)
        node, dof = torch.nonzero(ID >= 0, as_tuple=True)
        unk = ID[node, dof]
        polish = False
        for _ in range(20):
            r, K = self.r_K(xms, cps, time, dt)
            du = -torch.linalg.solve(K, r)
            dc = torch.zeros_like(cps)
            dc[node, dof] = du[unk]
            cps = cps + dc
            for j, u in enumerate(self.move):
                xms[:, j] += dt * dc[:, u]
            if polish:
                return xms, cps
            polish = float(du.norm()) / self.n < 1e-12
        return None

    def state(self, xms, cps):
        return torch.as_tensor(xms, device=self.dev).clone(), torch.as_tensor(cps, device=self.dev).clone()

    def predict(self, xms, cps, dt):
        for j, u in enumerate(self.move):
            xms[:, j] += dt * cps[:, u]


def exact(case, seed):
    do = case["do"]
    patches = _patches(case, seed)
    sizes = [mesh.nmdf for _, mesh, _, _ in patches]
    steps = case.get("steps", 1)
    if max(sizes) > 9500 or steps * sum(s / 1e3 + (s / 4e3) ** 3 for s in sizes) > 40:
        return None  # dense matrices: over 20 seconds
    if do in ("batch", "serve"):
        xs, cs = [], []
        for p, mesh, xms, cps in patches:
            ex = _Exact(p, mesh)
            x, c = ex.state(xms, cps)
            for k in range(steps):
                ex.predict(x, c, DT)
                got = ex.step(x, c, (k + 1) * DT, DT)
                if got is None:
                    return None
                x, c = got
            xs.append(x.flatten().cpu().numpy())
            cs.append(c.flatten().cpu().numpy())
        return {"status": None, "xms": np.concatenate(xs), "cps": np.concatenate(cs)}
    p, mesh, xms, cps = patches[0]
    ex = _Exact(p, mesh)
    x, c = ex.state(xms, cps)
    if do == "record":
        n1, n2 = mesh.num1el, mesh.num2el
        pull = n1 // 2 + n1 * (n2 // 2)  # the centre element
        els = torch.tensor([pull + i * n1 + j for i in range(-2, 3) for j in range(-2, 3)], device=ex.dev)
        ix = ex.IX[els]
        r = ex.elem(x[ix].to(torch.complex128), c[ix].to(torch.complex128), 0.0, True, els).real
        own = ex.IX[pull]
        held = torch.isin(ix, own)
        f = [float(r[..., ex.d[i]][held].sum()) if ex.d[i] >= 0 else 0.0 for i in range(3)]
        return {"record": np.array([DT] + x[own].mean(0).tolist() + f)}
    if do in ("assemble", "seam"):
        r, K = ex.r_K(x, c, DT, DT)
        if do == "seam":
            return {"r": r.cpu().numpy(), "du": -torch.linalg.solve(K, r).cpu().numpy()}
        kl = mesh.half_bw
        K = K.cpu().numpy()
        band = np.zeros((mesh.nmdf, 3 * kl + 1))
        for j in range(mesh.nmdf):
            lo, hi = max(0, j - kl), min(mesh.nmdf, j + kl + 1)
            band[j, 2 * kl + lo - j:2 * kl + hi - j] = K[lo:hi, j]
        return {"r": r.cpu().numpy(), "K": band}
    for k in range(steps):
        if do == "run":
            ex.predict(x, c, DT)
        got = ex.step(x, c, (k + 1) * DT, DT)
        if got is None:
            return None
        x, c = got
    return {"xms": x.cpu().numpy(), "cps": c.cpu().numpy()}

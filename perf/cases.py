"""Workloads that time euler3d_b200 through its public entry points.

Each case is one piece of work that a user's program has the framework do: load a flow state, run a
number of iterations of the solver, read the state, the residual history and the force coefficients
back.  The meshes are the three families of the repository's benchmark and tests (bump channel,
biconvex O-grid, Gaussian-bump box), prepared once per process; the states are made from the seed.

A case's keys: ``kind`` ("run": EulerSolver.run; "residual": EulerSolver.residual; "batch": Batch),
``family`` / ``nx`` ``ny`` ``nz``, ``mach`` / ``aoa`` / ``cfl``, ``scheme``, ``precision``,
``integrator`` and ``smoothing``, ``iterations``, and for a batch ``members`` and the range of their
sizes (``cells_lo``, ``cells_hi``).
"""
import functools
import math

import numpy as np
import torch

from euler3d_b200 import _lib, meshgen
from euler3d_b200.batch import Batch
from euler3d_b200.solver import STATE_KEYS, EulerSolver, FlowConfig, Mesh

PRECISION = {"fp64": _lib.PREC_FP64, "fp32": _lib.PREC_FP32_FLUX, "exact": _lib.PREC_FP64_EXACT}
SCHEME = {"roe": _lib.SCHEME_ROE, "ausm": _lib.SCHEME_AUSM}
INTEGRATOR = {"rk5": _lib.INTEGRATOR_RK5, "euler": _lib.INTEGRATOR_EULER}
ALPHAS = {"rk5": (0.0533, 0.1263, 0.2375, 0.4414, 1.0), "euler": (1.0,)}
STEP = 32  # iterations per batch step, as the server runs them


def _solo(name, family, nx, ny, nz, mach, aoa, cfl, iterations, scheme="roe", precision="fp64", integrator="rk5",
          smoothing=False, kind="run"):
    case = {"kind": kind, "family": family, "nx": nx, "ny": ny, "nz": nz, "mach": mach, "aoa": aoa, "cfl": cfl,
            "iterations": iterations, "scheme": scheme, "precision": precision, "integrator": integrator,
            "smoothing": smoothing}
    return dict(case, name=name) if name else case


def _batch(name, members, cells_lo, cells_hi, precision, iterations, mesh_seed):
    case = {"kind": "batch", "members": members, "cells_lo": cells_lo, "cells_hi": cells_hi, "precision": precision,
            "iterations": iterations, "mesh_seed": mesh_seed}
    return dict(case, name=name) if name else case


def listed():
    return [
        # The small named configuration: a 64 x 32 x 2 channel, the size at which launches count.
        _solo("channel_4k_fp64", "channel", 64, 32, 2, 0.5, 0.0, 1.5, 200),
        # One request of the served stream solved alone: an O-grid of odd size, AUSM fluxes.
        _solo("ogrid_20k_ausm_fp64", "ogrid", 101, 50, 2, 0.6, 2.0, 1.2, 100, scheme="ausm"),
        # One request of the served stream in the precision ladder's first phase, ragged sizes.
        _solo("channel_37k_fp32", "channel", 193, 97, 2, 0.45, -1.5, 1.5, 100, precision="fp32"),
        # The airfoil configuration: a 256 x 128 x 4 O-grid of prisms at Mach 0.8.
        _solo("ogrid_262k_fp64", "ogrid", 256, 128, 4, 0.8, 1.25, 1.2, 60),
        # Tetrahedra, an ordinary unstructured size with odd extents.
        _solo("tets_1p5m_fp64", "box", 65, 63, 61, 0.6, 0.0, 1.0, 40),
        # The largest: the benchmark's tetrahedral box at 96^3 x 6 cells.
        _solo("tets_5p3m_fp64", "box", 96, 96, 96, 0.6, 0.0, 1.0, 40),
        # The same family with single-precision fluxes.
        _solo("tets_1p6m_fp32", "box", 64, 64, 64, 0.6, 0.0, 1.0, 40, precision="fp32"),
        # The mode that reproduces the reference bit for bit, as the drop-in program runs it.
        _solo("channel_17k_exact", "channel", 129, 65, 2, 0.5, 0.0, 1.5, 50, precision="exact"),
        # TIME_INTEGRATION= 0 with RESIDUAL_SMOOTHING= 1.
        _solo("tets_146k_euler_smoothed", "box", 29, 29, 29, 0.6, 0.0, 0.6, 100, integrator="euler", smoothing=True),
        # The residual and time step of one state, as a caller with its own integrator asks for them.
        _solo("tets_162k_residual", "box", 30, 30, 30, 0.6, 0.0, 1.0, 1, kind="residual"),
        # The served stream in batches: members of both families and schemes, 5k to 50k cells each.
        _batch("batch_16_served_fp64", 16, 5000, 50000, "fp64", 96, 3),
        # The precision ladder's single-precision batch beside it.
        _batch("batch_16_served_fp32", 16, 5000, 50000, "fp32", 96, 4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.18:
        lo = _log_int(rng, 4000, 20000)
        return _batch(None, rng.randint(4, 16), lo, min(60000, lo * rng.randint(2, 8)), rng.choice(["fp64", "fp64", "fp32"]),
                      STEP * rng.randint(2, 3), rng.randrange(1 << 20))
    family = rng.choice(["channel", "ogrid", "box"])
    cells = _log_int(rng, 3000, {"channel": 1_500_000, "ogrid": 400_000, "box": 4_500_000}[family])
    if family == "channel":
        nz = rng.choice([2, 2, 3])
        ny = max(6, int(math.sqrt(cells / (2.0 * nz))) + rng.randint(-1, 1))
        nx = 2 * ny + rng.randint(-3, 3)
    elif family == "ogrid":
        nz = rng.choice([2, 2, 3, 4])
        ny = max(10, int(math.sqrt(cells / (4.0 * nz))) + rng.randint(-1, 1))
        nx = 2 * ny + rng.randint(-1, 2)
    else:
        s = (cells / 6.0) ** (1 / 3)
        nx, ny, nz = (max(6, int(round(s)) + rng.randint(-2, 2)) for _ in range(3))
    mach, aoa = round(rng.uniform(0.3, 0.75), 3), round(rng.uniform(-3.0, 4.0), 2)
    iterations = max(20, min(200, int(2.0e7 / cells)))
    scheme = rng.choice(["roe", "roe", "ausm"])
    if rng.random() < 0.12:
        return _solo(None, family, nx, ny, nz, mach, aoa, 1.0, 1, scheme, kind="residual")
    if rng.random() < 0.15:
        return _solo(None, family, nx, ny, nz, mach, aoa, 0.6, iterations, scheme, integrator="euler",
                     smoothing=rng.random() < 0.7)
    # the bit-exact mode is used on meshes that the reference runs too
    # the bit-exact mode is used for parity checks, on meshes that the reference itself runs
    precision = rng.choice(["fp64", "fp64", "fp32"] + (["exact"] if cells < 60_000 else []))
    if precision == "exact":
        iterations = min(iterations, 50)
    return _solo(None, family, nx, ny, nz, mach, aoa, {"channel": 1.5, "ogrid": 1.2, "box": 1.0}[family], iterations,
                 scheme, precision)


# ------------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=64)
def _mesh(family, nx, ny, nz):
    """Prepared mesh arrays in the reference's numbering."""
    if family == "channel":
        raw = meshgen.bump_channel(nx, ny, nz)
    elif family == "ogrid":
        # the radial growth of 128 layers at 1.1, span layers 0.1 chord thick and thinner on fine grids
        dz = 0.1 * min(1.0, 128.0 / ny)
        raw = meshgen.biconvex_ogrid(nx, ny, nz, stretch=1.1 ** (128.0 / ny), span=nz * dz)
    else:
        raw = meshgen.bump_box_tets(nx=nx, ny=ny, nz=nz)
    mesh = Mesh.from_raw(raw)
    arrays = mesh.arrays()
    mesh.close()
    return arrays


def _members(case):
    """The single solves of a case: itself, or a batch's members (sizes and conditions as the served
    stream draws them: log-uniform cells, Mach 0.3 to 0.7, both families and schemes)."""
    if case["kind"] != "batch":
        return [case]
    rng = np.random.default_rng(case["mesh_seed"])
    out = []
    for _ in range(case["members"]):
        cells = math.exp(rng.uniform(math.log(case["cells_lo"]), math.log(case["cells_hi"])))
        family = ("channel", "ogrid")[int(rng.integers(2))]
        ny = max(6, int(round(math.sqrt(cells / (4.0 if family == "channel" else 8.0)))))
        out.append(_solo(None, family, 2 * ny, ny, 2, round(float(rng.uniform(0.3, 0.7)), 3),
                         round(float(rng.uniform(-4.0, 4.0)), 2), 1.5 if family == "channel" else 1.2,
                         case["iterations"], ("roe", "ausm")[int(rng.integers(2))], case["precision"]))
    return out


def _flow(m):
    return FlowConfig(mach=m["mach"], aoa=m["aoa"], cfl=m["cfl"], scheme=SCHEME[m["scheme"]],
                      precision=PRECISION[m["precision"]], integrator=INTEGRATOR[m["integrator"]],
                      smoothing=m["smoothing"], ordering=_lib.ORDER_SPATIAL)


def _arrays(m):
    return _mesh(m["family"], m["nx"], m["ny"], m["nz"])


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _state(m, seed):
    """A flow field on its way to the steady state: the freestream with smooth waves of about 2 % in
    every variable; ghost cells at the freestream, as FlowField's arrays (8 rows, STATE_KEYS)."""
    a = _arrays(m)
    n = int(a["n_cells"])
    total = n + int(a["n_faces"]) - int(a["n_faces_int"])
    rng = np.random.default_rng(seed)
    g, ang = 1.4, math.radians(m["aoa"])
    speed = m["mach"] * math.sqrt(g)
    x = torch.from_numpy(a["cell_centroid"]).to(_device()).reshape(-1, 3)
    lo, hi = x.min(0).values, x.max(0).values
    x = (x - lo) / (hi - lo).clamp(min=1e-12)

    def wave():
        v = torch.zeros_like(x[:, 0])
        for _ in range(3):
            k, phase = rng.uniform(-12.0, 12.0, 3), float(rng.uniform(0.0, 2.0 * math.pi))
            v += torch.sin(x[:, 0] * float(k[0]) + x[:, 1] * float(k[1]) + x[:, 2] * float(k[2]) + phase) * (0.02 / 3)
        return v

    s = torch.empty((8, total), dtype=torch.float64, device=x.device)
    for k, v in enumerate((1.0, speed * math.cos(ang), speed * math.sin(ang), 0.0, 1.0, 0.0, 0.0, m["mach"])):
        s[k] = v
    s[0, :n] += wave()
    for k in (1, 2, 3):
        s[k, :n] += speed * wave()
    s[4, :n] += wave()
    q2 = s[1] ** 2 + s[2] ** 2 + s[3] ** 2
    s[5] = s[4] / ((g - 1.0) * s[0]) + q2 / 2.0
    s[6] = s[5] + s[4] / s[0]
    s[7, :n] = (g * s[4, :n] / s[0, :n]).sqrt() / q2[:n].sqrt()
    return s


def _pinned(shape):
    t = torch.empty(shape, dtype=torch.float64)
    return t.pin_memory() if torch.cuda.is_available() else t


class _Solve:
    """One solver with its input and output state in pinned host memory."""

    def __init__(self, m, seed, autotune):
        state = _state(m, seed)
        self.solver = EulerSolver(_arrays(m), _flow(m), autotune=autotune)
        self.keep = (_pinned(state.shape), _pinned(state.shape))
        self.start = {k: self.keep[0].numpy()[i] for i, k in enumerate(STATE_KEYS)}
        self.result = {k: self.keep[1].numpy()[i] for i, k in enumerate(STATE_KEYS)}
        self.keep[0].copy_(state)


def prepare(case, seed):
    ms = _members(case)
    solves = [_Solve(m, seed * 131 + i, autotune=case["kind"] != "batch") for i, m in enumerate(ms)]
    return {"case": case, "solves": solves, "batch": Batch() if case["kind"] == "batch" else None}


def run(state):
    case, solves = state["case"], state["solves"]
    if case["kind"] == "batch":
        return _run_batch(state["batch"], case, solves)
    s = solves[0]
    s.solver.set_state(s.start)
    if case["kind"] == "residual":
        r, dt = s.solver.residual()
        return {"residual": r, "dt": dt}
    stats = s.solver.run(case["iterations"])
    s.solver.get_state(s.result)
    return {"state": s.result, "rms": s.solver.rms_history(), "force": np.array(stats["force"]),
            "moment": np.array(stats["moment"]), "iterations": stats["iterations"]}


def _run_batch(batch, case, solves):
    for s in solves:
        s.solver.set_state(s.start)
        batch.add(s.solver, case["iterations"])
    done = {id(solver): stats for solver, stats, _ in batch.run_all(STEP)}
    for s in solves:
        s.solver.get_state(s.result)
    stats = [done[id(s.solver)] for s in solves]
    return {"state": [s.keep[1] for s in solves], "rms": np.stack([s.solver.rms_history() for s in solves]),
            "force": np.array([t["force"] for t in stats]), "moment": np.array([t["moment"] for t in stats]),
            "iterations": np.array([t["iterations"] for t in stats])}


def work(case):
    """Per stage and cell: the cell's state and W0 in, its state out, its geometry; per face its
    normal and area (doubles; the states, normals and geometry in single precision for fp32).  About
    170 operations for a face's flux, 60 for a cell's update.  The state comes from and goes to the host once."""
    total_b = total_f = 0.0
    for m in _members(case):
        a = _arrays(m)
        n, f = int(a["n_cells"]), int(a["n_faces"])
        w = 4 if m["precision"] == "fp32" else 8
        stages = 1 if case["kind"] == "residual" else m["iterations"] * len(ALPHAS[m["integrator"]])
        total_b += stages * (n * (5 * w + 5 * 8 + 5 * w + 4 * w) + f * (4 * w + 8)) + 2 * 64.0 * n
        total_f += stages * (170.0 * f + 60.0 * n)
    return {"bytes": total_b, "flops": total_f}


# ------------------------------------------------------------------------------- 64-bit evaluation
class _Exact:
    """The scheme written out in plain torch, in double precision: ghost cells, Roe or AUSM fluxes,
    local time step, five-stage Runge-Kutta or explicit Euler, residual smoothing, wall forces."""

    def __init__(self, m, seed):
        a = _arrays(m)
        dev = _device()
        self.m, self.g = m, 1.4

        def d(v):
            return torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).to(dev)

        def ix(v):
            return torch.from_numpy(np.ascontiguousarray(v, dtype=np.int64)).to(dev)

        self.n, self.fi = int(a["n_cells"]), int(a["n_faces_int"])
        f2c = ix(a["face2cell"]).reshape(-1, 2)
        self.left, self.right = f2c[:, 0].contiguous(), f2c[:, 1].contiguous()
        self.normal = list(d(a["face_unit_normal"]).reshape(-1, 3).t().contiguous())
        self.area, self.vol = d(a["face_area"]), d(a["cell_volume"])
        full, ctr = d(a["face_normal"]).reshape(-1, 3), d(a["face_center"]).reshape(-1, 3)
        ptr = np.asarray(a["cell2face_ptr"])
        c2f = ix(a["cell2face"])
        owner = ix(np.repeat(np.arange(self.n), np.diff(ptr)))
        self.sums = [torch.zeros(self.n, dtype=torch.float64, device=dev).index_add_(0, owner, full[c2f, k].abs())
                     for k in range(3)]
        self.n_faces_of = ix(np.diff(ptr)).double()
        self.bc = {t: (ix(a[t + "_ghost"]), ix(a[t + "_interior"]), ix(a[t + "_face"])) for t in ("wall", "farfield", "sym")}
        self.wall_s, self.wall_x = full[self.bc["wall"][2]], ctr[self.bc["wall"][2]]
        ang = math.radians(m["aoa"])
        u, v = m["mach"] * math.sqrt(self.g) * math.cos(ang), m["mach"] * math.sqrt(self.g) * math.sin(ang)
        e = 1.0 / (self.g - 1.0) + (u * u + v * v) / 2.0
        self.inf = (1.0, u, v, 0.0, 1.0, e, e + 1.0, m["mach"])
        self.s = list(_state(m, seed))

    def _put(self, ghost, rho, u, v, w, p, c):
        q2 = u * u + v * v + w * w
        e = p / ((self.g - 1.0) * rho) + q2 / 2.0
        for k, x in enumerate((rho, u, v, w, p, e, e + p / rho, q2.sqrt() / c)):
            self.s[k][ghost] = x

    def ghosts(self):
        g, s = self.g, self.s
        gh, d, f = self.bc["farfield"]
        if gh.numel():
            n = [c[f] for c in self.normal]
            vn, mach = sum(s[1 + k][gh] * n[k] for k in range(3)), s[7][gh]
            q = [x[d] for x in s]
            c = (g * q[4] / q[0]).sqrt()
            r = self.inf
            out = [torch.where((mach >= 1.0) & (vn > 0.0), q[k], torch.full_like(vn, r[k])) for k in range(8)]
            pin = 0.5 * (r[4] + q[4] - q[0] * c * sum(n[k] * (r[1 + k] - q[1 + k]) for k in range(3)))
            sub_out = [q[0] + (r[4] - q[4]) / (c * c)] + [q[1 + k] + n[k] * (q[4] - r[4]) / (q[0] * c) for k in range(3)]
            sub_in = [r[0] + (pin - r[4]) / (c * c)] + [r[1 + k] - n[k] * (r[4] - pin) / (q[0] * c) for k in range(3)]
            sel = [torch.where(vn > 0.0, sub_out[k], sub_in[k]) for k in range(4)]
            self._put(gh, *sel, torch.where(vn > 0.0, torch.full_like(vn, r[4]), pin), c)
            sup = mach >= 1.0
            for k in range(8):
                s[k][gh[sup]] = out[k][sup]
        for t in ("wall", "sym"):
            gh, d, f = self.bc[t]
            n = [c[f] for c in self.normal]
            q = [x[d] for x in s]
            vn = sum(q[1 + k] * n[k] for k in range(3))
            self._put(gh, q[0], *(q[1 + k] - 2.0 * vn * n[k] for k in range(3)), q[4], (g * q[4] / q[0]).sqrt())

    def flux(self, faces):
        """Fluxes between the two cells of `faces` (an index tensor or a slice)."""
        g, n = self.g, [c[faces] for c in self.normal]
        li, ri = self.left[faces], self.right[faces]
        rl, ul, vl, wl, pl, hl = (self.s[k][li] for k in (0, 1, 2, 3, 4, 6))
        rr, ur, vr, wr, pr, hr = (self.s[k][ri] for k in (0, 1, 2, 3, 4, 6))
        nl, nr = ul * n[0] + vl * n[1] + wl * n[2], ur * n[0] + vr * n[1] + wr * n[2]
        cl = (g * pl / rl).sqrt()
        if self.m["scheme"] == "ausm":
            cr = (g * pr / rr).sqrt()
            ml, mr = nl / cl, nr / cr
            one, zero = torch.ones_like(ml), torch.zeros_like(ml)
            mp = torch.where(ml.abs() <= 1.0, 0.25 * (ml + 1.0) ** 2, 0.5 * (ml + ml.abs()))
            pp = torch.where(ml.abs() <= 1.0, 0.25 * (ml + 1.0) ** 2 * (2.0 - ml), torch.where(ml > 0.0, one, zero))
            mm = torch.where(mr.abs() <= 1.0, -0.25 * (mr - 1.0) ** 2, 0.5 * (mr - mr.abs()))
            pm = torch.where(mr.abs() <= 1.0, 0.25 * (mr - 1.0) ** 2 * (2.0 + mr), torch.where(mr < 0.0, one, zero))
            mi, pi = mp + mm, pp * pl + pm * pr
            al, ar = mi.clamp(min=0.0) * rl * cl, mi.clamp(max=0.0) * rr * cr
            return [al + ar, al * ul + ar * ur + pi * n[0], al * vl + ar * vr + pi * n[1],
                    al * wl + ar * wr + pi * n[2], al * hl + ar * hr]
        sl, sr = rl.sqrt(), rr.sqrt()
        rt = (rl * rr).sqrt()
        ut, vt, wt, ht = ((a * sl + b * sr) / (sl + sr) for a, b in ((ul, ur), (vl, vr), (wl, wr), (hl, hr)))
        q2 = ut * ut + vt * vt + wt * wt
        ct = ((g - 1.0) * (ht - q2 / 2.0)).sqrt()
        nt = ut * n[0] + vt * n[1] + wt * n[2]
        drho, du, dv, dw, dp, dn = rr - rl, ur - ul, vr - vl, wr - wl, pr - pl, nr - nl
        delta = cl / 15.0
        lam1, lam5 = ((nt - ct).abs(), (nt + ct).abs())
        lam1 = torch.where(lam1 > delta, lam1, (lam1 * lam1 + delta * delta) / (2.0 * delta))
        lam5 = torch.where(lam5 > delta, lam5, (lam5 * lam5 + delta * delta) / (2.0 * delta))
        a1 = lam1 * (dp - rt * ct * dn) / (2.0 * ct * ct)
        a5 = lam5 * (dp + rt * ct * dn) / (2.0 * ct * ct)
        a2, av = drho - dp / (ct * ct), nt.abs()
        out = [(rr * nr + rl * nl) / 2.0 - (a1 + a5 + a2 * av) / 2.0]
        for k, (a, b, t, dd) in enumerate(((ul, ur, ut, du), (vl, vr, vt, dv), (wl, wr, wt, dw))):
            out.append((rr * nr * b + rl * nl * a + (pr + pl) * n[k]) / 2.0 -
                       ((t - ct * n[k]) * a1 + (t + ct * n[k]) * a5 + (t * a2 + rt * (dd - dn * n[k])) * av) / 2.0)
        out.append((rr * nr * hr + rl * nl * hl) / 2.0 -
                   ((ht - ct * nt) * a1 + (ht + ct * nt) * a5 +
                    (q2 / 2.0 * a2 + rt * (ut * du + vt * dv + wt * dw - nt * dn)) * av) / 2.0)
        return out

    def residual(self):
        res = [torch.zeros_like(self.vol) for _ in range(5)]
        inner = slice(0, self.fi)
        for k, f in enumerate(self.flux(inner)):
            f = f * self.area[inner]
            res[k].index_add_(0, self.left[inner], f)
            res[k].index_add_(0, self.right[inner], f, alpha=-1.0)
        for t in ("wall", "farfield", "sym"):
            gh, d, f = self.bc[t]
            if not gh.numel():
                continue
            if t == "sym":
                fl = self.flux(f)
            else:
                n = [c[f] for c in self.normal]
                r, u, v, w, p, h = (self.s[k][gh] for k in (0, 1, 2, 3, 4, 6))
                vn = u * n[0] + v * n[1] + w * n[2] if t == "farfield" else torch.zeros_like(r)
                fl = [r * vn, r * u * vn + p * n[0], r * v * vn + p * n[1], r * w * vn + p * n[2], r * h * vn]
            for k in range(5):
                res[k].index_add_(0, d, fl[k] * self.area[f])
        return res

    def time_step(self):
        s, n = self.s, self.n
        c = (self.g * s[4][:n] / s[0][:n]).sqrt()
        return self.m["cfl"] * self.vol / (0.5 * sum((s[1 + k][:n].abs() + c) * self.sums[k] for k in range(3)))

    def smooth(self, res):
        """Two Jacobi passes, the reference's loop (a change of at most 1e-16 ends it after the first)."""
        li, ri = self.left[:self.fi], self.right[:self.fi]
        last = res
        for sweep in range(2):
            out = []
            for r, x in zip(res, last):
                y = torch.zeros_like(r).index_add_(0, li, x[ri]).index_add_(0, ri, x[li])
                out.append((r + 0.25 * y) / (1.0 + 0.25 * self.n_faces_of))
            change = max(float((a - b).abs().max()) for a, b in zip(out, last)) if sweep == 0 else 0.0
            last = out
            if sweep == 0 and not change > 1e-16:
                break
        return last

    def update(self, w):
        n, g = self.n, self.g
        u, v, ww, e = (w[k] / w[0] for k in (1, 2, 3, 4))
        q2 = u * u + v * v + ww * ww
        p = (g - 1.0) * w[0] * (e - q2 / 2.0)
        for k, x in enumerate((w[0], u, v, ww, p, e, e + p / w[0], (g * p / w[0]).sqrt() / q2.sqrt())):
            self.s[k][:n] = x

    def conservative(self):
        s, n = self.s, self.n
        return [s[0][:n].clone()] + [s[k][:n] * s[0][:n] for k in (1, 2, 3, 5)]

    def forces(self):
        u2 = self.inf[1] ** 2 + self.inf[2] ** 2
        cp = (self.s[4][self.bc["wall"][1]] - 1.0) / (0.5 * u2)
        coeff = self.wall_s * cp[:, None]
        force, lever = coeff.sum(0), torch.tensor([0.25, 0.0, 0.0], dtype=torch.float64, device=cp.device) - \
            (coeff * self.wall_x).sum(0)
        return force.cpu().numpy(), torch.linalg.cross(force, lever).cpu().numpy()

    def run(self, iterations, integrator, smoothing):
        rms, carried = [], self.conservative() if integrator == "euler" else None
        for _ in range(iterations):
            w0 = carried if carried else self.conservative()
            for alpha in ALPHAS[integrator]:
                self.ghosts()
                res = self.residual()
                if smoothing:
                    res = self.smooth(res)
                f = alpha * self.time_step() / self.vol
                w = [a - f * r for a, r in zip(w0, res)]
                self.update(w)
            if carried:
                carried = w
            rms.append((res[0] * res[0]).sum())
        return np.sqrt(torch.stack(rms).cpu().numpy() / self.n)


def exact(case, seed):
    outs = []
    for i, m in enumerate(_members(case)):
        e = _Exact(m, seed * 131 + i)
        if case["kind"] == "residual":
            e.ghosts()
            return {"residual": torch.stack(e.residual(), 1).cpu().numpy(), "dt": e.time_step().cpu().numpy()}
        rms = e.run(m["iterations"], m["integrator"], m["smoothing"])
        outs.append((torch.stack(e.s).cpu().numpy(), rms, *e.forces()))
    state, rms, force, moment = (list(x) for x in zip(*outs))
    if case["kind"] == "batch":
        return {"state": state, "rms": np.stack(rms), "force": np.stack(force), "moment": np.stack(moment), "iterations": None}
    return {"state": {k: state[0][i] for i, k in enumerate(STATE_KEYS)}, "rms": rms[0], "force": force[0],
            "moment": moment[0], "iterations": None}

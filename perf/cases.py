"""The work that a program using phenlei_b200 has it do, as cases to be timed and compared.

A case is a mesh kind with its sizes, the flow model and its options, and what is run on it: outer
iterations of the solver (the everyday call), the phases of one iteration called one at a time (a program
that needs the residual itself), a partitioned grid stepped zone by zone, or the training of the learned
turbulence source.  The state comes in and goes out through the C ABI's device entry points, as in a program
that keeps its fields on the GPU; solvers, meshes and the learned model are what such a program sets up once.
"""
import math

import numpy as np
import torch

from phenlei_b200 import cases as flows
from phenlei_b200 import mesh as meshes
from phenlei_b200 import solver as phx
from phenlei_b200 import zones

STEP = 200          # outer step the passes start from: the CFL ramp (500 steps) well under way
RE = 1.0e5          # Reynolds number per unit length of the drawn viscous cases


def _case(name, mesh, nx, ny, nz, **more):
    c = {"do": "steps", "mesh": mesh, "nx": nx, "ny": ny, "nz": nz, "prism": 0, "physics": "euler", "mach": 0.5,
         "re": RE, "gradient": "ggcell", "limiter": "vencat", "scheme": "roe", "precision": "mixed",
         "source": "exact", "steps": 1}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one outer iteration of the Euler bump (64x32x4), where launches and latency count
        _case("euler_8k_one_step", "bump", 64, 32, 4),
        # the same mesh in double precision, as a long run steps it (residuals read every 20 iterations)
        _case("euler_8k_fp64_run", "bump", 64, 32, 4, precision="fp64", steps=20),
        # laminar flow on an odd, small tetrahedral grid: residual and sweeps called phase by phase, FP64
        _case("laminar_tets_fp64_phases", "tets", 23, 23, 23, do="phases", physics="laminar", mach=0.3, re=1.0e4,
              gradient="lsq", precision="fp64"),
        # the laminar jittered-tetrahedra cube, a million cells, least-squares gradient, mixed precision
        _case("laminar_tets_1M", "tets", 55, 55, 55, physics="laminar", mach=0.3, re=1.0e4, gradient="lsq",
              steps=3),
        # node-based gradient and Barth limiter on an odd-sized laminar bump, FP64
        _case("laminar_ggnode_fp64", "bump", 97, 53, 21, physics="laminar", mach=0.3, re=1.0e4, gradient="ggnode",
              limiter="barth", precision="fp64", steps=2),
        # Spalart-Allmaras flat plate (128x96x16, AUSMPW+, first cell 1e-5), the training flow of the learned source
        _case("sa_plate_200k", "plate", 128, 96, 16, physics="sa", mach=0.2, re=5.0e6, scheme="ausmpw+", steps=5),
        # the transonic bump with prism layers, one million cells: FP64, mixed, and mixed with the learned source
        _case("sa_bump_1M_fp64", "bump", 256, 92, 32, prism=30, physics="sa", mach=0.8, re=1.0e7, precision="fp64",
              steps=2),
        _case("sa_bump_1M", "bump", 256, 92, 32, prism=30, physics="sa", mach=0.8, re=1.0e7, steps=3),
        _case("sa_bump_1M_learned", "bump", 256, 92, 32, prism=30, physics="sa", mach=0.8, re=1.0e7,
              source="learned", steps=3),
        # the largest: the transonic bump again with wider levels and planes, 2.6 million cells
        _case("sa_bump_2.6M", "bump", 224, 92, 96, prism=30, physics="sa", mach=0.8, re=1.0e7, steps=3),
        # a partitioned grid: four slabs of an odd-sized bump in one process, with their halo exchanges
        _case("sa_bump_4_zones", "bump", 132, 45, 27, prism=11, physics="sa", mach=0.8, re=1.0e7, do="zones",
              steps=2),
        # training of the learned source: 65,536 samples, batches of 8,192, three epochs
        _case("train_learned_source", "bump", 16, 8, 2, physics="sa", mach=0.8, do="train", samples=65536,
              batch=8192, epochs=3),
    ]


def draw(rng):
    """A case of the same ranges: sizes from a few hundred cells to about two million, their logarithm uniform."""
    if rng.random() < 0.08:
        n = int(math.exp(rng.uniform(math.log(3000), math.log(100000))))
        return _case("", "bump", 16, 8, 2, physics="sa", mach=0.8, do="train", samples=n,
                     batch=rng.randint(max(1, n // 9), n), epochs=rng.randint(1, 3))
    cells = math.exp(rng.uniform(math.log(400), math.log(2.0e6)))
    physics = rng.choice(["euler", "laminar", "sa", "sa"])
    mesh = "tets" if physics != "sa" and rng.random() < 0.35 else ("plate" if physics == "sa" and rng.random() < 0.3
                                                                   else "bump")
    c = _case("", mesh, 0, 0, 0, physics=physics, precision=rng.choice(["mixed", "mixed", "fp64"]),
              mach=round(rng.uniform(0.2, 0.85), 3), re=float(int(10 ** rng.uniform(4.0, 7.0))),
              gradient=rng.choice(["ggcell", "ggcell", "lsq", "ggnode"]),
              limiter=rng.choice(["vencat", "vencat", "barth", "nolim"]),
              scheme=rng.choice(["roe", "roe", "ausmpw+", "ausmdv", "hlle", "vanleer"]), steps=rng.randint(1, 4))
    if mesh == "tets":
        c["nx"] = c["ny"] = c["nz"] = max(4, int((cells / 6.0) ** (1.0 / 3.0)))
    else:
        c["nz"] = max(2, int(cells ** (1.0 / 3.0) * rng.uniform(0.2, 0.9)))
        c["ny"] = max(6, int(math.sqrt(cells / c["nz"]) * rng.uniform(0.5, 0.9)))
        c["nx"] = max(8, int(cells / (c["nz"] * c["ny"])))
        if mesh == "bump" and physics != "euler" and rng.random() < 0.5:
            c["prism"] = rng.randint(1, c["ny"] // 3)
    if physics == "sa" and rng.random() < 0.25:
        c["source"] = "learned"
    if rng.random() < 0.15:
        c["do"] = "phases"
    elif mesh != "tets" and c["nx"] >= 16 and c["gradient"] != "ggnode" and rng.random() < 0.12:
        c["do"] = "zones"
        c["zones"] = rng.randint(2, 4)
    return c


# ---------------------------------------------------------------------------
# Set-up: meshes, solvers and the learned model, kept as a program keeps them
# (one solver at a time; host meshes of this process).
# ---------------------------------------------------------------------------
_meshes, _solver, _model = {}, {}, {}


def _skew_angle(case):
    """The viscous flux's angle switch.  The cube's boundary tetrahedra have angles of exactly 60 degrees, the
    default, where rounding alone would decide."""
    return 50.0 if case["mesh"] == "tets" else 60.0


def _params(case):
    p = dict(flows.EULER_BUMP, refMachNumber=case["mach"], gradientName=case["gradient"],
             uns_limiter_name=case["limiter"], uns_scheme_name=case["scheme"], skewnessAngle=_skew_angle(case))
    if case["physics"] != "euler":
        p.update(viscousType=1, refReNumber=case["re"], refDimensionalTemperature=288.15, prl=0.72,
                 wallTemperature=-1.0)
    if case["physics"] == "sa":
        p.update(viscousType=3, prt=0.9, muoo=3.0, CFLEnd=20.0)
        if case["source"] == "learned":
            p["sa_source"] = "mlp_fallback"
    return p


def _mesh(case):
    """The mesh, its wall distance (SA) and its node-average cell centres scaled to the unit box."""
    key = tuple(case[k] for k in ("mesh", "nx", "ny", "nz", "prism")) + (case["physics"] == "sa",)
    if key not in _meshes:
        n = (case["nx"], case["ny"], case["nz"])
        if case["mesh"] == "tets":
            m = meshes.tet_cube(n[0], jitter=0.15, seed=1)
        elif case["mesh"] == "plate":
            m = meshes.flat_plate(*n, first_spacing=min(1e-5, 0.5 / n[1]))
        else:
            m = meshes.channel_bump(*n, thickness=0.08, wall_spacing=min(0.001 if n[1] > 40 else 0.01, 0.5 / n[1]),
                                    prism_layers=case["prism"])
        wd = meshes.wall_distance(m) if case["physics"] == "sa" else None
        c = flows.cell_centres(m)
        lo, hi = c.min(axis=0), c.max(axis=0)
        if sum(v[0].n_cell for v in _meshes.values()) > 5_000_000:
            _meshes.clear()
        _meshes[key] = (m, wd, (c - lo) / np.maximum(hi - lo, 1e-12))
    return _meshes[key]


def _samples(n, seed):
    """Training samples (features, target) of the Spalart-Allmaras source: it is a function of chi = nu~ rho / mu
    and s = vorticity / (nu~ / d^2 Re) alone."""
    rng = np.random.default_rng(seed)
    chi = np.exp(rng.uniform(np.log(1e-3), np.log(1e4), n))
    s = np.exp(rng.uniform(np.log(1e-3), np.log(1e6), n))
    k2, cb1, cw2 = 0.41 ** 2, 0.1355, 0.3
    cw1 = cb1 / k2 + 1.622 * 1.5
    fv1 = chi ** 3 / (chi ** 3 + 7.1 ** 3)
    fv2 = 1.0 - chi / (1.0 + chi * fv1)
    sbar = fv2 / k2
    st = np.where(sbar >= -0.7 * s, s + sbar, s + s * (0.49 * s + 0.9 * sbar) / (-0.5 * s - sbar + 1e-300))
    r = np.minimum(1.0 / (k2 * st), 10.0)
    g = r + cw2 * (r ** 6 - r)
    fw = g * ((1.0 + 64.0) / (g ** 6 + 64.0)) ** (1.0 / 6.0)
    f = np.stack([np.log(chi), np.log(s), fv1, s / (1 + s), 1 / (1 + chi), np.log1p(s)], axis=1)
    return f.astype(np.float32), ((cb1 * st - cw1 * fw) / (1.0 + s)).astype(np.float32)


def _learned_model():
    """A saved model of the learned source (weights, normalisation, training hull), fitted here with torch so that
    every program under comparison loads the same one."""
    if "blob" not in _model:
        f, t = _samples(60000, 7)
        mean, std = f.mean(axis=0), np.maximum(f.std(axis=0), 1e-6)
        scale = math.sqrt(float((t.astype(np.float64) ** 2).mean()))
        gen = torch.Generator().manual_seed(1)
        w = []
        for o, i in ((64, 6), (64, 64), (64, 64), (1, 64)):
            w += [(torch.rand((o, i), generator=gen) * 2 - 1) * math.sqrt(3.0 / i), torch.zeros(o)]
        for v in w:
            v.requires_grad_(True)
        x, y = torch.from_numpy((f - mean) / std), torch.from_numpy(t / scale)
        opt = torch.optim.Adam(w, lr=2e-3)
        for k in range(150):
            i = torch.randint(0, len(y), (2048,), generator=gen)
            h = x[i]
            for j in (0, 2, 4):
                h = torch.nn.functional.silu(h @ w[j].T + w[j + 1])
            loss = ((h @ w[6].T + w[7])[:, 0] - y[i]).square().mean()
            opt.zero_grad()
            loss.backward()
            opt.step()
        flat = np.concatenate([v.detach().numpy().reshape(-1) for v in w])
        lo, hi = f.min(axis=0), f.max(axis=0)
        occ = np.ones(int(phx.lib().phx_mlp_blob_size()) - flat.size - 25)
        _model["blob"] = np.concatenate([flat, mean, 1.0 / std, lo, hi, [scale], occ]).astype(np.float32)
    return _model["blob"]


def _get_solver(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "samples", "batch", "epochs")))
    if _solver.get("key") != key:
        if "s" in _solver:
            _solver.pop("s").close()
        _solver.clear()
        m, wd, _ = _mesh(case)
        if case["do"] == "zones":
            s = zones.ZoneSet(m, _params(case), nparts=case.get("zones", 4), wall_dist=wd,
                              precision=case["precision"])
            each = s.zones
        else:
            s = phx.NSSolverUnstruct(m, precision=case["precision"], wall_dist=wd, **_params(case))
            each = [s]
        if case["source"] == "learned":
            for z in each:
                z.set_mlp_blob(_learned_model())
        _solver.update(key=key, s=s)
    return _solver["s"]


def _fields(case, seed):
    """Cell values of the primitive state (free stream plus random-phase sinusoids, 2 %), nu~ and eddy viscosity."""
    m, _, x = _mesh(case)
    rng = np.random.default_rng(seed)
    q0 = flows.freestream(_params(case))
    x = torch.from_numpy(x).cuda()
    q = torch.empty((5, m.n_cell), dtype=torch.float64, device="cuda")
    for v in range(5):
        w = torch.zeros(m.n_cell, dtype=torch.float64, device="cuda")
        for ax in range(3):
            for k in range(1, 4):
                w += torch.sin(2.0 * math.pi * k * x[:, ax] + rng.uniform(0.0, 2.0 * math.pi))
        q[v] = q0[v] + 0.02 / 3.0 * (q0[v] if v in (0, 4) else 1.0) * w
    nut = 3.0 * (1.0 + 0.3 * torch.sin(2.0 * math.pi * (x[:, 0] + x[:, 1]) + rng.uniform(0.0, 2.0 * math.pi)))
    fv1 = nut ** 3 / (nut ** 3 + 7.1 ** 3)
    return q, nut, nut * fv1


def _put(s, which, t):
    s._check(phx.lib().phx_set_state_device(s.h, which, t.data_ptr(), t.numel()), "phx_set_state_device")


def _take(s, which, rows):
    t = torch.empty((rows, s.nt), dtype=torch.float64, device="cuda")
    s._check(phx.lib().phx_get_state_device(s.h, which, t.data_ptr(), t.numel()), "phx_get_state_device")
    return t


def prepare(case, seed):
    if case["do"] == "train":
        f, t = _samples(case["samples"], seed)
        return {"case": case, "s": _get_solver(case), "f": f, "t": t}
    s = _get_solver(case)
    q, nut, vist = _fields(case, seed)
    if case["do"] == "zones":
        # a partitioned program's restart: every zone's cells and ghosts
        s.set_state(q.cpu().numpy(), nut.cpu().numpy())
        st = {"case": case, "s": s, "in": []}
        for part, z in zip(s.parts, s.zones):
            cells = torch.from_numpy(np.asarray(part.cells, np.int64)).cuda()
            v = torch.full((1, z.nt), 1e-3, dtype=torch.float64, device="cuda")
            v[0, : part.mesh.n_cell] = vist[cells]
            st["in"].append((_take(z, phx.PHX_Q, 5), _take(z, phx.PHX_Q_TURB, 1), v))
        return st
    nc, nt = s.mesh.n_cell, s.nt
    full = torch.from_numpy(flows.freestream(_params(case))).cuda()[:, None].repeat(1, nt)
    full[:, :nc] = q
    state = [(phx.PHX_Q, full)]
    if case["physics"] == "sa":
        for which, v, ghost in ((phx.PHX_Q_TURB, nut, 3.0), (phx.PHX_VIST, vist, 1e-3)):
            t = torch.full((1, nt), ghost, dtype=torch.float64, device="cuda")
            t[0, :nc] = v
            state.append((which, t))
    return {"case": case, "s": s, "in": state}


def run(state):
    case, s = state["case"], state["s"]
    if case["do"] == "train":
        loss = s.train_sa_mlp(state["f"], state["t"], epochs=case["epochs"], batch=case["batch"], lr=1e-3, seed=3)
        n = int(phx.lib().phx_mlp_param_count())
        return {"loss": loss, "weights": s.mlp_blob()[:n]}
    if case["do"] == "zones":
        out = {}
        for z, (q, nut, vist) in zip(s.zones, state["in"]):
            _put(z, phx.PHX_Q, q)
            _put(z, phx.PHX_Q_TURB, nut)
            _put(z, phx.PHX_VIST, vist)
            z.step = STEP
        out["residual"] = s.iterate(case["steps"])
        for k, z in enumerate(s.zones):
            out["q%d" % k] = _take(z, phx.PHX_Q, 5)
            out["nut%d" % k] = _take(z, phx.PHX_Q_TURB, 1)
        return out
    for which, t in state["in"]:
        _put(s, which, t)
    s.step = STEP
    if case["do"] == "phases":
        s.Boundary()
        s.ComputeGradientAndLimiter()
        s.UpdateResiduals()
        s.LUSGS()
        return {"res": _take(s, phx.PHX_RES, 5), "dq": _take(s, phx.PHX_DQ, 5)}
    out = {"residual": s.Relaxation(case["steps"]), "q": _take(s, phx.PHX_Q, 5)}
    if case["physics"] == "sa":
        out["nut"] = _take(s, phx.PHX_Q_TURB, 1)
    return out


def work(case):
    """Bytes of the path's own arrays (each read or written once per global pass: gradient, limiter, face residual,
    two sweeps, update, and the turbulence equation alike; metrics and the state that is kept 8 bytes, working values
    4 or 8) and operations (about 500 per face and 400 per cell for Euler, half as much again for viscous flow)."""
    if case["do"] == "train":
        n = case["samples"] // case["batch"] * case["batch"] * case["epochs"]
        return {"bytes": 28.0 * case["samples"] * case["epochs"], "flops": 3.0 * 2.0 * n * (6 * 64 + 2 * 64 * 64 + 64)}
    n = case["nx"] * case["ny"] * case["nz"] + case["nx"] * case["prism"] * case["nz"]
    f = 2.0 * 6 * n if case["mesh"] == "tets" else 3.0 * n
    n = 6 * n if case["mesh"] == "tets" else n
    e = 8 if case["precision"] == "fp64" else 4
    vis = case["physics"] != "euler"
    nv = 6 if vis else 5
    face = f * 40
    b = n * 5 * e + face + 8 * n + 3 * nv * n * e                              # gradient
    b += n * 9 * e + f * 32 + 24 * n                                           # limiter
    b += n * (14 + 3 * nv) * e + face + 24 * (f + n)                           # face residual
    b += 2 * (n * 22 * e + face + 2 * f * 4 + 4 * n) + n * (80 + 5 * e)        # sweeps, update
    if case["physics"] == "sa":
        b += 3 * face + n * (40 * e + 64) + 4 * f * 4
    steps = case["steps"] if case["do"] != "phases" else 1
    return {"bytes": b * steps, "flops": (500.0 * f + 400.0 * n) * (1.5 if vis else 1.0) * steps}


def tolerance(case):
    """About four times the largest differences seen against 64 bits (plain torch, sums in another order) and after
    inputs moved by their last bit, over the listed cases and thirty drawn ones."""
    if case["do"] == "train":           # 1.5e-6, 1.4e-4
        return {"rel": 1e-5, "max": 1e-3}
    if case["source"] == "learned":     # half-precision activations: 2.2e-5, 1e-3
        return {"rel": 1e-4, "max": 5e-3}
    if case["precision"] == "fp64":     # 4.2e-14, 6.9e-13; twenty steps more
        return {"rel": 1e-12, "max": 2e-11}
    if case["do"] == "phases":          # residuals are small differences of large fluxes: 2.8e-5, 3.6e-4
        return {"rel": 1.2e-4, "max": 1.5e-3}
    return {"rel": 5e-6, "max": 2e-5}   # 1.2e-6, 4e-6


# ---------------------------------------------------------------------------
# The same results in 64 bits with plain torch: face metrics, cell metrics, boundary, gradient, limiter, fluxes,
# time step, the two LU-SGS sweeps level by level, update, and the Spalart-Allmaras step.
# ---------------------------------------------------------------------------
TINY = 1e-40


def _add(n, idx, v):
    """Sum of the columns of v over idx, n columns (rows of v kept)."""
    return torch.zeros(v.shape[:-1] + (n,), dtype=v.dtype, device=v.device).index_add_(v.dim() - 1, idx, v)


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


class _Grid:
    def __init__(self, m, wall_dist, skew_angle):
        d = lambda a, t=torch.int64: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", t)  # noqa: E731
        self.nc, self.nb, self.nf = m.n_cell, m.n_bface, m.n_face
        nc, nb, nf = self.nc, self.nb, self.nf
        xyz = torch.stack([d(a, torch.float64) for a in (m.x, m.y, m.z)])
        off, f2n = d(m.face_offsets()), d(m.face2node)
        self.l = d(m.left)
        self.r = d(m.right).clone()
        self.r[:nb] = nc + torch.arange(nb, device="cuda")
        types, region = m.solver_regions()
        self.bc = d(types)[d(region)[:nb]]
        n = torch.zeros((3, nf), dtype=torch.float64, device="cuda")
        fc = torch.zeros_like(n)
        groups = []
        for k in torch.unique(off[1:] - off[:-1]).tolist():
            fs = torch.nonzero(off[1:] - off[:-1] == k)[:, 0]
            p = xyz[:, f2n[off[fs][:, None] + torch.arange(k, device="cuda")]]
            nxt = torch.roll(p, -1, 2)
            c = p.mean(2)
            for _ in range(5):
                t = torch.linalg.cross(p - c[:, :, None], nxt - c[:, :, None], dim=0)
                ta = t.norm(dim=0)
                c = ((p + nxt + c[:, :, None]) * ta).sum(2) / (3.0 * ta.sum(1))
            n[:, fs], fc[:, fs] = t.sum(2), c
            groups.append((fs, p, nxt))
        s = n.norm(dim=0)
        self.area, self.n, self.fc = 0.5 * s, n / (s + TINY), fc
        co, c2n = d(m.cell_offsets()), d(m.cell2node)
        cnt = co[1:] - co[:-1]
        cc = _add(nc, torch.repeat_interleave(torch.arange(nc, device="cuda"), cnt), xyz[:, c2n]) / cnt
        mom, vol = torch.zeros_like(cc), torch.zeros(nc, dtype=torch.float64, device="cuda")
        for fs, p, nxt in groups:
            t = torch.linalg.cross(p - fc[:, fs, None], nxt - fc[:, fs, None], dim=0)
            for side, sign in ((self.l, -1.0), (self.r, 1.0)):
                ok = side[fs] < nc
                c = side[fs][ok]
                v = sign * (t[:, ok] * (cc[:, c] - fc[:, fs[ok]])[:, :, None]).sum(0)
                e = (fc[:, fs[ok]] + cc[:, c])[:, :, None] + p[:, ok] + nxt[:, ok]
                vol += _add(nc, c, v.sum(1))
                mom += _add(nc, c, (e * v).sum(2))
        t = mom / (4.0 * vol + TINY)
        ins = torch.ones(nc, dtype=torch.bool, device="cuda")
        i = slice(nb, nf)
        ins[self.l[_dot(t[:, self.l] - fc, self.n) > 0]] = False
        ins[self.r[i][_dot(t[:, self.r[i]] - fc[:, i], self.n[:, i]) < 0]] = False
        cc = torch.where(ins, t, cc)
        b = slice(0, nb)
        gh = cc[:, self.l[b]] - self.n[:, b] * (2.0 * _dot(cc[:, self.l[b]] - fc[:, b], self.n[:, b]))
        self.cc = torch.cat([cc, gh], 1)
        self.vol = torch.cat([vol / 6.0, vol[self.l[b]] / 6.0])
        ang = lambda v: torch.asin((_dot(self.n, v) / (v.norm(dim=0) + TINY)).clamp(-1, 1)) * (180 / math.pi)  # noqa: E731
        al, ar = ang(fc - self.cc[:, self.l]), ang(self.cc[:, self.r] - fc)
        worst = torch.where(torch.arange(nf, device="cuda") < nb, al, torch.minimum(al, ar))
        sk = torch.full((nc + nb,), 180.0, dtype=torch.float64, device="cuda")
        sk.scatter_reduce_(0, self.l, worst, "amin")
        sk.scatter_reduce_(0, self.r[i], worst[i], "amin")
        self.skew = sk[:nc]
        self.dL, self.dR = _dot(self.n, self.cc[:, self.l] - fc), _dot(self.n, self.cc[:, self.r] - fc)
        far = (self.dL.abs() > TINY) & (self.dR.abs() > TINY)
        self.project, self.normal = (al > skew_angle) & (ar > skew_angle), (al > 0) & (ar > 0) & far
        self.wd = None if wall_dist is None else d(wall_dist, torch.float64)
        # the uses of the interior faces in the two sweeps, in the order of the levels of the cells they serve
        a, b = torch.minimum(self.l[i], self.r[i]), torch.maximum(self.l[i], self.r[i])
        self.sweeps = [self._levels(b, a), self._levels(a, b)]

    def _levels(self, cell, nbr):
        lev = torch.zeros(self.nc, dtype=torch.int64, device="cuda")
        while True:
            new = lev.scatter_reduce(0, cell, lev[nbr] + 1, "amax")
            if torch.equal(new, lev):
                break
            lev = new
        order = torch.argsort(lev[cell], stable=True)
        cells = torch.argsort(lev, stable=True)
        nlev = int(lev.max()) + 1
        uses = torch.cumsum(torch.bincount(lev[cell], minlength=nlev), 0).tolist()
        ends = torch.cumsum(torch.bincount(lev, minlength=nlev), 0).tolist()
        return order + self.nb, cell[order], nbr[order], cells, uses, ends


def _roe(L, R, n, g, mach):
    s = 0.0001 if mach <= 0.6 else 0.0001 * (mach - 2.0) / -1.4 + 0.01 * (mach - 0.6) / 1.4
    fix = lambda e, m: torch.where(e.abs() < s * m, 0.5 * (e * e + (s * m) ** 2) / (s * m), e.abs())  # noqa: E731
    sides = []
    for q in (L, R):
        v2, vn = _dot(q[1:4], q[1:4]), _dot(n, q[1:4])
        h = g / (g - 1) * q[4] / q[0] + 0.5 * v2
        e = q[4] / q[0] / (g - 1) + 0.5 * v2
        u = torch.stack([q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3], q[0] * e])
        f = q[0] * vn * torch.stack([torch.ones_like(h), q[1], q[2], q[3], h])
        f[1:4] += n * q[4]
        sides.append((u, f, h))
    t = torch.sqrt(R[0] / L[0])
    w = (L + R * t) / (1 + t)
    rm, pm, v2, vn = torch.sqrt(L[0] * R[0]), w[4], _dot(w[1:4], w[1:4]), _dot(n, w[1:4])
    hm = g / (g - 1) * pm / rm + 0.5 * v2
    c2 = (g - 1) * (hm - 0.5 * v2)
    c = torch.sqrt(c2.abs())
    top = vn.abs() + c
    e1, e2, e3 = fix(vn, top), fix(vn + c, top), fix(vn - c, top)
    x1, x2 = (2 * e1 - e2 - e3) / (2 * c2), (e2 - e3) / (2 * c)
    dq = sides[1][0] - sides[0][0]
    dc = vn * dq[0] - _dot(n, dq[1:4])
    dh = -(g - 1) * (_dot(w[1:4], dq[1:4]) - dq[4]) + 0.5 * (g - 1) * v2 * dq[0]
    a, b = dh * x1 + dc * x2, c2 * dc * x1 + dh * x2
    diss = torch.stack([e1 * dq[0] - a, *(e1 * dq[1:4] - w[1:4] * a + n * b), e1 * dq[4] - hm * a + vn * b])
    return 0.5 * (sides[0][1] + sides[1][1] - diss)


def _ausmpwp(L, R, n, g):
    hs, cs, vns = [], [], []
    for q in (L, R):
        hs.append(g / (g - 1) * q[4] / q[0] + 0.5 * _dot(q[1:4], q[1:4]))
        cs.append(torch.sqrt(g * q[4] / q[0]))
        vns.append(_dot(n, q[1:4]))
    c = 0.5 * (cs[0] + cs[1])
    ml, mr = vns[0] / c, vns[1] / c
    mpn = lambda m, s: torch.where(m.abs() >= 1, 0.5 * (m + s * m.abs()), s * 0.25 * (m + s) ** 2)  # noqa: E731
    ppn = lambda m, s: torch.where(m.abs() >= 1, 0.5 * (m + s * m.abs()) / m,  # noqa: E731
                                   s * 0.25 * (m + s) ** 2 * (2 * s - m))
    a, b = mpn(ml, 1.0), mpn(mr, -1.0)
    p12 = ppn(ml, 1.0) * L[4] + ppn(mr, -1.0) * R[4]
    fw = 1 - torch.minimum(L[4] / R[4], R[4] / L[4]) ** 3
    fl = torch.where((ml.abs() <= 1) & (p12 != 0), L[4] / p12 - 1, 0.0)
    fr = torch.where((mr.abs() <= 1) & (p12 != 0), R[4] / p12 - 1, 0.0)
    pos = a + b >= 0
    mp = torch.where(pos, a + b * ((1 - fw) * (1 + fr) - fl), a * fw * (1 + fl))
    mm = torch.where(pos, b * fw * (1 + fr), b + a * ((1 - fw) * (1 + fl) - fr))
    out = c * (mp * L[0] * torch.stack([torch.ones_like(c), *L[1:4], hs[0]])
               + mm * R[0] * torch.stack([torch.ones_like(c), *R[1:4], hs[1]]))
    out[1:4] += p12 * n
    return out


class _Solver64:
    def __init__(self, case):
        m, wd, _ = _mesh(case)
        self.case, self.g = case, _Grid(m, wd, _skew_angle(case))
        p = _params(case)
        self.vis, self.sa = case["physics"] != "euler", case["physics"] == "sa"
        self.gam, self.mach, self.re = 1.4, case["mach"], case["re"]
        self.coef = 1.0 / (1.4 * self.mach ** 2)
        self.inf = torch.tensor([1.0, 1.0, 0.0, 0.0, self.coef], dtype=torch.float64, device="cuda")
        self.tsuth, self.cfl_end = 110.4 / p.get("refDimensionalTemperature", 288.15), p["CFLEnd"]
        bc = self.g.bc
        self.far, self.wall = bc == meshes.BC_FARFIELD, (bc == meshes.BC_SOLID_SURFACE) & self.vis

    def boundary(self, q):
        g, G = self.gam, self.g
        o = q[:, G.l[: G.nb]]
        n = G.n[:, : G.nb]
        vn, out = _dot(n, o[1:4]), o.clone()
        out[1:4] = o[1:4] - 2.0 * n * vn
        out[1:4] = torch.where(self.wall, -o[1:4], out[1:4])
        i = self.inf[:, None]
        vno = _dot(n, i[1:4].expand_as(n))
        ci, co = torch.sqrt(g * o[4] / o[0]), math.sqrt(g * self.coef)
        rp, rm = vn + 2 * ci / (g - 1), vno - 2 * co / (g - 1)
        vb, cb = 0.5 * (rp + rm), 0.25 * (rp - rm) * (g - 1)
        leave = vb >= 0
        ent = torch.where(leave, o[4] / o[0] ** g, torch.full_like(vb, self.coef))
        rb = (cb * cb / (ent * g)) ** (1 / (g - 1))
        far = torch.stack([rb, *(torch.where(leave, o[1:4] - n * vn, i[1:4] - n * vno) + n * vb), cb * cb * rb / g])
        sup = _dot(o[1:4], o[1:4]).sqrt() > ci
        far = torch.where(sup, torch.where(vn < 0, i.expand_as(o), o), far)
        q[:, G.nc:] = torch.where(self.far, far, out)

    def temp(self, q):
        return q[4] / (self.coef * q[0])

    def mu(self, t):
        return t ** 1.5 * (1 + self.tsuth) / (t + self.tsuth)

    def gradient(self, v):
        G, nc, nb = self.g, self.g.nc, self.g.nb
        i = slice(nb, None)
        if self.case["gradient"] == "lsq":
            d = G.cc[:, G.r] - G.cc[:, G.l]
            w = 1.0 / (_dot(d, d) + TINY)
            mat = (w * d[:, None] * d[None])
            mat = _add(nc, G.l, mat) + _add(nc, G.r[i], mat[..., i])
            t = (w * (v[:, G.r] - v[:, G.l]))[:, None] * d[None]
            t = _add(nc, G.l, t) + _add(nc, G.r[i], t[..., i])
            inv = torch.linalg.inv(mat.permute(2, 0, 1))
            return torch.einsum("cij,vjc->vic", inv, t)
        t = (0.5 * (v[:, G.l] + v[:, G.r]))[:, None] * (G.n * G.area)[None]
        return (_add(nc, G.l, t) - _add(nc, G.r[i], t[..., i])) / G.vol[:nc]

    def limiter(self, q, grad):
        G, nc, nb = self.g, self.g.nc, self.g.nb
        lim = torch.ones(nc + nb, dtype=torch.float64, device="cuda")
        if self.case["limiter"] == "nolim":
            return lim
        l, r = G.l[nb:], G.r[nb:]
        for k in (0, 4):
            lo, hi = q[k].clone(), q[k].clone()
            for a, b in ((l, r), (r, l)):
                lo.scatter_reduce_(0, a, q[k][b], "amin")
                hi.scatter_reduce_(0, a, q[k][b], "amax")
            eps = 125.0 / (G.vol[:nc].sum() / nc) * q[k][:nc] ** 2 * G.vol[:nc]
            for side, fs in ((G.l, slice(0, None)), (r, slice(nb, None))):
                d = _dot(grad[k][:, side], G.fc[:, fs] - G.cc[:, side])
                x = torch.where(d > 0, hi[side], lo[side]) - q[k][side]
                e = eps[side]
                f = (x * x + e + 2 * d * x) / (x * x + 2 * d * d + x * d + e)
                lim.scatter_reduce_(0, side, torch.where(d.abs() > TINY, f, 1.0), "amin")
        lim[G.l[:nb][self.far]] = 0.0
        lim[nc:][self.far] = 0.0
        return lim

    def residual(self, q, vist, cfl):
        G, nc, nb, g = self.g, self.g.nc, self.g.nb, self.gam
        v = torch.cat([q, self.temp(q)[None]])
        grad = self.gradient(v)
        self.grad = grad
        lim = self.limiter(q, grad)
        n, area = G.n, G.area
        L, R = q[:, G.l], q[:, G.r]
        lf = torch.minimum(lim[G.l], lim[G.r])
        face = []
        for S, side in ((L, G.l), (R, G.r)):
            c = side.clamp(max=nc - 1)
            t = S + lf * (grad[:5, :, c] * (G.fc - G.cc[:, side])[None]).sum(1)
            face.append(torch.where((side < nc) & (t[0] > 0) & (t[4] > 0), t, S))
        ql, qr = face
        b = slice(0, nb)
        solid = G.bc == meshes.BC_SOLID_SURFACE
        sym = G.bc == meshes.BC_SYMMETRY
        mean = 0.5 * (L[:, b] + R[:, b])
        refl = mean.clone()
        refl[1:4] -= 2.0 * n[:, b] * _dot(n[:, b], mean[1:4])
        still = mean.clone()
        still[1:4] = 0.0
        ql[:, b] = torch.where(solid | sym, torch.where(self.wall, still, mean), ql[:, b])
        qr[:, b] = torch.where(solid | sym, torch.where(sym, refl, torch.where(self.wall, still, mean)), qr[:, b])
        flux = (_roe(ql, qr, n, g, self.mach) if self.case["scheme"] == "roe" else _ausmpwp(ql, qr, n, g)) * area
        vn = 0.5 * (_dot(n, L[1:4]) + _dot(n, R[1:4]))
        spec = 0.5 * area * (vn.abs() + torch.sqrt(g * (L[4] + R[4]) / (L[0] + R[0])))
        vsp = torch.zeros_like(spec)
        if self.vis:
            fv, vsp = self.viscous(q, grad, vist)
            flux = flux + fv
        i = slice(nb, None)
        res = _add(nc, G.r[i], flux[:, i]) - _add(nc, G.l, flux)
        both = lambda f: _add(nc, G.l, f) + _add(nc, G.r[i], f[i])  # noqa: E731
        self.spec, self.vsp, tot_v = both(spec), vsp, both(vsp)
        cc = torch.full((nc,), cfl, dtype=torch.float64, device="cuda")
        base = 1.0 + 0.5 * (g - 1) * (2 / (g - 1) + self.mach ** 2) / (2 * g / (g - 1) * self.mach ** 2 - 1)
        if base > 0:
            pt = self.coef * base ** (g / (g - 1))
            lo, hi = 0.001 * pt, 0.02 * pt
            cc = torch.where(q[4, :nc] < hi, (q[4, :nc] - hi) * (cfl - 0.01) / (hi - lo) + cfl, cc)
            cc = torch.where(q[4, :nc] < lo, 0.01, cc)
        cc = torch.where(G.skew < 0.1, 0.1 * cc, torch.where(G.skew < 10, cc * (1 - torch.exp(-G.skew)), cc))
        self.dt = cc * G.vol[:nc] / (self.spec + tot_v)
        self.diag = G.vol[:nc] / self.dt + self.spec + tot_v
        return res

    def viscous(self, q, grad, vist):
        G, nc, nb = self.g, self.g.nc, self.g.nb
        n, fc = G.n, G.fc
        L, R, T = q[:, G.l], q[:, G.r], self.temp(q)
        mu = self.mu(T)
        mul, mut = 0.5 * (mu[G.l] + mu[G.r]), 0.5 * (vist[G.l] + vist[G.r])
        ds = _dot(n, G.cc[:, G.r] - G.cc[:, G.l]).abs()
        vsp = G.area * (mul + mut) / (0.5 * (L[0] + R[0]) * ds * self.re + TINY)
        bnd = torch.arange(G.nf, device="cuda") < nb
        wall = torch.zeros(G.nf, dtype=torch.bool, device="cuda")
        wall[:nb] = self.wall
        xl, xr = G.cc[:, G.l] - fc, G.cc[:, G.r] - fc
        d1, d2 = xl.norm(dim=0), xr.norm(dim=0)
        wl = torch.where(bnd, 1.0, d2 / (d1 + d2))
        keep = self.case["gradient"] != "ggcell"
        gl = grad[1:, :, G.l].clone()
        gl[4 - 1] = grad[5][:, G.l]
        gl = gl[:4]
        gr = torch.stack([grad[1], grad[2], grad[3], grad[5]])[:, :, torch.where(G.r < nc, G.r, G.l)]
        if not keep:
            gr = torch.where(G.r < nc, gr, 0.0)
        vl = torch.cat([L[1:4], T[G.l][None]])
        vr = torch.cat([R[1:4], T[G.r][None]])
        mid = 0.5 * (vl + vr)
        pl = vl + (gl * (n * G.dL - xl)[None]).sum(1)
        pr = vr + (gr * (n * G.dR - xr)[None]).sum(1)
        pl[3], pr[3] = torch.where(pl[3] < TINY, vl[3], pl[3]), torch.where(pr[3] < TINY, vr[3], pr[3])
        vl, vr = torch.where(G.project, pl, vl), torch.where(G.project, pr, vr)
        mid[:3] = torch.where(G.project & wall, 0.0, mid[:3])
        w = torch.where(bnd, 1.0, G.dL ** 2 / (G.dL ** 2 + G.dR ** 2))
        dn = torch.where(G.normal, w * (vl - mid) / G.dL + (1 - w) * torch.where(bnd, 0.0, (vr - mid) / G.dR), 0.0)
        gf = wl * gl[:3] + torch.where(bnd, 0.0, 1 - wl) * gr[:3]
        gf = gf + n[None] * (dn[:3] - (gf * n[None]).sum(1))[:, None]
        cp = 1.0 / (0.4 * self.mach ** 2)
        div = (gf[0, 0] + gf[1, 1] + gf[2, 2]) * (2.0 / 3.0)
        tau = (mul + mut) * (gf + gf.transpose(0, 1))
        for k in range(3):
            tau[k, k] -= (mul + mut) * div
        f = (tau * n[None]).sum(1)
        heat = (mul / 0.72 + mut / 0.9) * cp * dn[3]
        out = torch.cat([torch.zeros_like(heat)[None], f, (_dot(mid[:3], f) + heat)[None]])
        return -out * G.area / self.re, vsp

    def apply(self, q, cell, nbr, fs, sign, dq):
        """The sweeps' term of neighbour nbr (state q[:, nbr]) for the faces fs, with the neighbour's dq."""
        G, g = self.g, self.gam
        n, area = G.n[:, fs] * sign, G.area[fs]
        a, b = q[:, cell], q[:, nbr]
        h = lambda s: g / (g - 1) * s[4] / s[0] + 0.5 * _dot(s[1:4], s[1:4])  # noqa: E731
        t = torch.sqrt(b[0] / a[0])
        u = (a[1:4] + b[1:4] * t) / (1 + t)
        c = torch.sqrt((g - 1) * ((h(a) + h(b) * t) / (1 + t) - 0.5 * _dot(u, u)))
        rad = _dot(n, u).abs() + c
        c2 = g * b[4] / b[0]
        cm, vn = torch.sqrt(c2), _dot(n, b[1:4])
        l1, l2, l3 = 0.5 * (vn - rad), 0.5 * (vn + cm - rad), 0.5 * (vn - cm - rad)
        x1, x2 = (2 * l1 - l2 - l3) / (2 * c2), (l2 - l3) / (2 * cm)
        dc = vn * dq[0] - _dot(n, dq[1:4])
        dh = -(g - 1) * (_dot(b[1:4], dq[1:4]) - dq[4]) + 0.5 * (g - 1) * _dot(b[1:4], b[1:4]) * dq[0]
        p, r = dh * x1 + dc * x2, c2 * dc * x1 + dh * x2
        f = torch.stack([l1 * dq[0] - p, *(l1 * dq[1:4] - b[1:4] * p + n * r), l1 * dq[4] - h(b) * p + vn * r])
        return f * area - self.vsp[fs] * dq

    def sweep(self, which, term, rhs, dq, diag):
        """One sweep: dq = (rhs - sum of the terms of the neighbours already swept) / diag; returns the sums."""
        order, cell, nbr, cells, uses, ends = self.g.sweeps[which]
        total = torch.zeros_like(rhs)
        u0 = c0 = 0
        for u1, c1 in zip(uses, ends):
            if u1 > u0:
                s = slice(u0, u1)
                total.index_add_(1, cell[s], term(order[s], cell[s], nbr[s]))
            c = cells[c0:c1]
            dq[:, c] = (rhs[:, c] - total[:, c]) / diag[c]
            u0, c0 = u1, c1
        return total

    def lusgs(self, q, res):
        G, nc, nb = self.g, self.g.nc, self.g.nb
        dq = torch.zeros_like(res)

        def term(fs, cell, nbr):
            sign = torch.where(G.l[fs] == cell, 1.0, -1.0)
            return self.apply(q, cell, nbr, fs, sign, dq[:, nbr])

        low = self.sweep(0, term, res, dq, self.diag)
        # ghosts: symmetry reflects the forward dq through the conservative state, a wall its momentum
        b, o = torch.arange(nb, device="cuda"), G.l[:nb]
        n, d = G.n[:, :nb], dq[:, o]
        s, gq, g = q[:, o], q[:, nc:], self.gam
        u = torch.stack([s[0], *(s[0] * s[1:4]), s[4] / (g - 1) + 0.5 * s[0] * _dot(s[1:4], s[1:4])]) + d
        gh = d.clone()
        gh[1:4] = d[1:4] - 2.0 * n * _dot(n, d[1:4])
        m = u[1:4] - 2.0 * n * _dot(n, u[1:4])
        p = u[4] - 0.5 * _dot(u[1:4], u[1:4]) / u[0]
        gh[4] = p - gq[4] / (g - 1) + 0.5 * (_dot(m, m) / u[0] - gq[0] * _dot(gq[1:4], gq[1:4]))
        back = d.clone()
        back[1:4] = -d[1:4]
        gh = torch.where(self.far, 0.0, torch.where(self.wall, back, gh))
        ghost = _add(nc, o, self.apply(q, o, nc + b, b, 1.0, gh))
        self.sweep(1, term, res - low - ghost, dq, self.diag)
        return dq

    def update(self, q, dq):
        g, c = self.gam, slice(0, self.g.nc)
        s = q[:, c]
        u = torch.stack([s[0], *(s[0] * s[1:4]), s[4] / (g - 1) + 0.5 * s[0] * _dot(s[1:4], s[1:4])]) + dq
        v = u[1:4] / u[0]
        q[:, c] = torch.stack([u[0], *v, (g - 1) * (u[4] - 0.5 * u[0] * _dot(v, v))])

    # -- Spalart-Allmaras ---------------------------------------------------------
    def sa_boundary(self, q, nut, vist):
        G, nb, nc, g = self.g, self.g.nb, self.g.nc, self.gam
        o, n = G.l[:nb], G.n[:, :nb]
        s = q[:, o]
        vn, ci = _dot(n, s[1:4]), torch.sqrt(g * s[4] / s[0])
        vb = 0.5 * (vn + 2 * ci / (g - 1) + n[0] - 2 * math.sqrt(g * self.coef) / (g - 1))
        leave = torch.where(_dot(s[1:4], s[1:4]).sqrt() > ci, vn >= 0, vb >= 0)
        for a, inf in ((nut, 3.0), (vist, 1e-3)):
            v = torch.where(G.bc == meshes.BC_SOLID_SURFACE, -a[o], a[o])
            a[nc:] = torch.where(self.far & ~leave, inf, v)

    @staticmethod
    def positive(nu, mu, rho):
        x = (nu / (mu / rho)) ** 3
        return torch.where(nu < 0, nu * (16 + x) / (16 - x), nu)

    def source(self, nu, om, olam, rate):
        """Production minus destruction and its implicit part; rate = 1 / (d^2 Re)."""
        k2, cb1, cw2, cw36 = 0.41 ** 2, 0.1355, 0.3, 64.0
        cw1 = cb1 / k2 + 1.622 * 1.5
        x = nu * olam + TINY
        cv = 7.1 ** 3
        fv1 = x ** 3 / (x ** 3 + cv)
        fv2 = 1 - x / (1 + x * fv1)
        rs = nu * rate / k2
        sb = rs * fv2
        st = torch.where(sb >= -0.7 * om, om + sb, om + om * (0.49 * om + 0.9 * sb) / (-0.5 * om - sb))
        ost = 1 / (st + TINY)
        r = torch.minimum(rs * ost, torch.full_like(nu, 10.0))
        gg = r + cw2 * (r ** 6 - r)
        g6 = gg ** 6
        fw = gg * ((1 + cw36) / (g6 + cw36)) ** (1 / 6)
        neg = nu < 0
        prod, dest = cb1 * st, cw1 * fw * nu * rate
        src = prod * nu - cw1 * k2 * fw * nu * rs
        dfv2 = (3 * cv * (fv1 / x) ** 2 - 1) / (1 + x * fv1) ** 2
        dst = rate / k2 * (fv2 + x * dfv2)
        dfw = fw / (gg + TINY) * (1 - g6 / (g6 + cw36)) * (1 + cw2 * (6 * r ** 5 - 1)) * rate / k2 * ost * (1 - nu * ost * dst)
        dp, dd = cb1 * dst, cw1 * (fw + dfw * nu) * rate
        src = torch.where(neg, -0.2 * cb1 * om * nu + 50.0 * cw1 * k2 * nu * rs, src)
        prod, dest = torch.where(neg, -0.2 * cb1 * om, prod), torch.where(neg, -50.0 * cw1 * nu * rate, dest)
        dp, dd = torch.where(neg, -0.2 * cb1 * dst, dp), torch.where(neg, -50.0 * cw1 * rate, dd)
        a, b = prod - dest, dp - dd
        return src, -0.5 * (a - a.abs()) - 0.5 * (b - b.abs()) * nu

    def turbulence(self, q, nut, vist, mu):
        """One step of the turbulence equation after the flow's update (mu: the flow step's laminar viscosity)."""
        G, nc, nb = self.g, self.g.nc, self.g.nb
        n, area, c, i = G.n, G.area, slice(0, G.nc), slice(nb, None)
        self.sa_boundary(q, nut, vist)
        x = (nut[c] * q[0, c] / mu[c]) ** 3
        vist[c] = torch.where(nut[c] > 0, q[0, c] * nut[c] * x / (x + 7.1 ** 3), 0.0)
        self.sa_boundary(q, nut, vist)
        L, R, nl, nr, ml, mr = q[:, G.l], q[:, G.r], nut[G.l], nut[G.r], mu[G.l], mu[G.r]
        fb = torch.arange(G.nf, device="cuda") < nb
        sym, solid = torch.zeros_like(fb), torch.zeros_like(fb)
        sym[:nb], solid[:nb] = G.bc == meshes.BC_SYMMETRY, G.bc == meshes.BC_SOLID_SURFACE
        hl = torch.where(fb & ~sym, 0.5 * (nl + nr), nl)
        hr = torch.where(sym, nl, torch.where(fb, 0.5 * (nl + nr), nr))
        um = 0.5 * (L[1:4] + R[1:4])
        vl, vr = _dot(n, torch.where(fb, um, L[1:4])), _dot(n, torch.where(fb, um, R[1:4]))
        conv = (vl.clamp(min=0) * hl + vr.clamp(max=0) * hr) * area
        cb2, osig, ore = 0.622, 1.5, 1.0 / self.re
        pl, pr = self.positive(nl, ml, L[0]), self.positive(nr, mr, R[0])
        dl = pl
        dr = torch.where(fb, torch.where(solid & (nl < 0), -pl, nr), pr)
        mlt = osig * 0.5 * (ml / L[0] + mr / R[0] + dl + dr)
        mid = 0.5 * (nl + nr)
        w = G.dL ** 2 / (G.dL ** 2 + G.dR ** 2)
        dn = w * (nl - mid) / G.dL + (1 - w) * (nr - mid) / G.dR
        dn = torch.where(fb & ~sym, (nr - nl) / _dot(n, G.cc[:, G.r] - G.cc[:, G.l]), dn)
        dn = torch.where(G.normal, dn, 0.0)
        f1, f2 = -ore * (1 + cb2) * mlt * dn * area, ore * cb2 * osig * dn * area
        el = ml / L[0] + pl.abs()
        er = mr / R[0] + torch.where(solid, -pl, pr).abs()
        tl, tr = _dot(n, L[1:4]), _dot(n, R[1:4])
        jl, jr = torch.where(tl > 0, L[0] * tl * area, 0.0), torch.where(tr < 0, R[0] * tr * area, 0.0)
        scale = ore * area ** 2 / (0.5 * (G.vol[G.l] + G.vol[G.r])) * osig
        vt = scale * (1 + cb2) * 0.5 * (el + er)
        mat_r, mat_l = jr - vt + scale * cb2 * er, -jl - vt + scale * cb2 * el
        om = torch.stack([self.grad[3, 1] - self.grad[2, 2], self.grad[1, 2] - self.grad[3, 0],
                          self.grad[2, 0] - self.grad[1, 1]]).norm(dim=0)
        src, imp = self.source(nut[c], om, q[0, c] / mu[c], ore / G.wd ** 2)
        own = mu[c] / q[0, c] + self.positive(nut[c], mu[c], q[0, c])
        out = lambda f: _add(nc, G.r[i], f[i]) - _add(nc, G.l, f)  # noqa: E731
        res = src * G.vol[c] + out(conv + f1) + own * out(f2)
        spec = G.vol[c] / (self.dt + TINY) + imp * G.vol[c] + _add(nc, G.l, jl + vt) + _add(nc, G.r[i], (vt - jr)[i])
        dq = torch.zeros((1, nc), dtype=torch.float64, device="cuda")

        def term(fs, cell, nbr):
            return (torch.where(G.l[fs] == cell, mat_r[fs], mat_l[fs]) * dq[0, nbr])[None]

        low = self.sweep(0, term, res[None], dq, spec)
        self.sweep(1, term, res[None] - low, dq, spec)
        nut[c] += dq[0]
        self.sa_boundary(q, nut, vist)


def _train64(case, seed):
    """The Adam run of train_sa_mlp in 64 bits: its seeded initial weights and shuffles (splitmix64), its batches."""
    f, t = _samples(case["samples"], seed)
    n, size = len(t), min(case["batch"], len(t))
    mask = (1 << 64) - 1
    x = (3 * 0x2545F4914F6CDD1D + 1) & mask

    def rnd():
        nonlocal x
        x = (x + 0x9E3779B97F4A7C15) & mask
        z = x
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        return z ^ (z >> 31)

    w = []
    for o, i in ((64, 6), (64, 64), (64, 64), (1, 64)):
        a = np.sqrt(np.float32(3.0) / np.float32(i))
        u = np.array([np.float32((rnd() >> 11) * (1.0 / 9007199254740992.0)) for _ in range(o * i)], np.float32)
        w += [torch.from_numpy(((2 * u - 1) * a).reshape(o, i)).double().cuda(),
              torch.zeros(o, dtype=torch.float64, device="cuda")]
    for v in w:
        v.requires_grad_(True)
    f64 = f.astype(np.float64)
    mean = f64.mean(axis=0).astype(np.float32)
    rstd = (1.0 / np.sqrt(np.maximum((f64 ** 2).mean(axis=0) - f64.mean(axis=0) ** 2, 1e-12))).astype(np.float32)
    scale = np.float32(np.sqrt((t.astype(np.float64) ** 2).mean()))
    xs = torch.from_numpy((f64 - mean) * rstd.astype(np.float64)).cuda()
    ys = torch.from_numpy(t.astype(np.float64) / scale).cuda()
    m1, m2 = [torch.zeros_like(v) for v in w], [torch.zeros_like(v) for v in w]
    b1, b2, lr, eps = (float(np.float32(v)) for v in (0.9, 0.999, 1e-3, 1e-8))
    perm, step = list(range(n)), 0
    for _ in range(case["epochs"]):
        for k in range(n - 1, 0, -1):
            j = rnd() % (k + 1)
            perm[k], perm[j] = perm[j], perm[k]
        p = torch.tensor(perm, device="cuda")
        last = 0.0
        for k in range(0, n - size + 1, size):
            i = p[k:k + size]
            h = xs[i]
            for j in (0, 2, 4):
                h = torch.nn.functional.silu(h @ w[j].T + w[j + 1])
            err = (h @ w[6].T + w[7])[:, 0] - ys[i]
            gr = torch.autograd.grad(err.square().mean(), w)
            last += float(err.detach().square().sum())
            step += 1
            with torch.no_grad():
                for v, g, a, b in zip(w, gr, m1, m2):
                    a.mul_(b1).add_((1 - b1) * g)
                    b.mul_(b2).add_((1 - b2) * g * g)
                    v -= lr * (a / (1 - b1 ** step)) / ((b / (1 - b2 ** step)).sqrt() + eps)
    return {"loss": last / (n // size * size), "weights": torch.cat([v.detach().reshape(-1) for v in w]).cpu().numpy()}


def exact(case, seed):
    if case["do"] == "train":
        return _train64(case, seed)
    if (case["do"] == "zones" or case["source"] != "exact" or case["gradient"] == "ggnode"
            or case["limiter"] == "barth" or case["scheme"] not in ("roe", "ausmpw+") or case["steps"] > 5):
        return None
    s = _Solver64(case)
    G = s.g
    qc, nc_, vc = _fields(case, seed)
    q = s.inf[:, None].repeat(1, G.nc + G.nb)
    q[:, : G.nc] = qc
    nut = torch.full((G.nc + G.nb,), 3.0, dtype=torch.float64, device="cuda")
    vist = torch.full_like(nut, 1e-3 if s.sa else 0.0)
    if s.sa:
        nut[: G.nc], vist[: G.nc] = nc_, vc
    hist = []
    phases = case["do"] == "phases"
    for k in range(case["steps"] if not phases else 1):
        step = STEP + (0 if phases else k + 1)
        s.boundary(q)
        mu = s.mu(s.temp(q))
        res = s.residual(q, vist, 0.01 + (s.cfl_end - 0.01) * step / 500)
        dq = s.lusgs(q, res)
        if phases:
            pad = torch.zeros((5, G.nb), dtype=torch.float64, device="cuda")
            return {"res": torch.cat([res, pad], 1), "dq": torch.cat([dq, pad], 1)}
        s.update(q, dq)
        hist.append(float(torch.sqrt(res[0].square().mean())))
        s.boundary(q)
        if s.sa:
            s.turbulence(q, nut, vist, mu)
    out = {"residual": np.array(hist), "q": q}
    if s.sa:
        out["nut"] = nut[None]
    return out

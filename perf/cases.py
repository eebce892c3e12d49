"""The calls of this library that programs spend their time in, over the sizes they have in use.

listed()            a fixed set of cases; draw(rng) one more of the same ranges
prepare(case, seed) the seeded bodies on the GPU (host memory for run_host) and the handles a program keeps
run(state)          one pass through the public binding (gi.py over the C ABI)
exact(case, seed)   the same outputs in 64 bits, plain torch
work(case)          bytes and flops that a pass cannot do without

Kinds of call:
  forces    gi_forces_collision: the drop-in for the reference's force launch, once per step of its drivers
  modes     gi_forces with a one-sided accumulation mode: the precision study and accuracy checks
  step      gi_step_pingpong: one fused force + kick-drift step of one impact, the library's main loop
  settle    gi_step: target and impactor as two damped runs in place, the body builder's loop
  sweep     gi_graph_launch: many impacts of uneven size, several steps in one captured graph
  host      gi_run_host: bodies in pinned host memory, the steps between two records, bodies back
  energy    gi_diag_fp64 + gi_potential_fp64: the energy and momentum log of a run
  diag      gi_diag_fp64 alone, up to the 8.4M-body state
  analysis  gi_find_earth_moon, the scope statistics and gi_find_disk: the end of an impact
  picture   gi_splat: one frame of the headless viewer

States (code units G = D = 1; Fe is the inner 30 % by radius of a body, listed first):
  ball      a body builder's raw ball, 0.24 elements per unit volume (about 1 contact each)
  settled   target and impactor after settling, about 18 contacts each, apart
  merged    an impact's remnant: one interpenetrating clump (about 2,400 contacts each, 6,500 in
            its core), a small second clump and debris in orbit
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "giant-impact_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import gi  # noqa: E402

DT = 1e-3
K_FE, K_SI, KR_FE, KR_SI, SD_FE, SD_SI = 5.0, 1.5, 0.02, 0.01, 0.002, 0.001
MASS = (1.0, 0.4)      # Fe, Si
# The reference's kernels fix m_Si = 1: masses / 0.4, stiffnesses / 0.16.
REF_MASS = (2.5, 1.0)
REF_K = (K_FE / 0.16, K_SI / 0.16)
PAIR_FLOPS = 23.0      # one unordered far pair, applied to both bodies
ACCUM = {"fp32": gi.GI_ACCUM_FP32, "fp64": gi.GI_ACCUM_FP64, "kahan": gi.GI_ACCUM_KAHAN}


def listed():
    return [
        # latency: the drop-in force call on a test-size body set, launches and host work count
        {"name": "forces-1500", "kind": "forces", "n": 1500, "state": "ball"},
        # the one-sided Kahan mode of the accuracy ladder, odd size
        {"name": "modes-kahan-20001", "kind": "modes", "n": 20001, "state": "ball", "accum": "kahan"},
        # the 66,000-body impact before contact: a run's ordinary step
        {"name": "step-settled-66000", "kind": "step", "n": 66000, "state": "settled"},
        # the same impact while the bodies interpenetrate: contacts cost as much as the far field
        {"name": "step-merged-66000", "kind": "step", "n": 66000, "state": "merged"},
        # the large-N impact of the precision study
        {"name": "step-ball-1153434", "kind": "step", "n": 1153434, "state": "ball"},
        # settling a small target and impactor: many short steps in one call
        {"name": "settle-8192", "kind": "settle", "n": 8192, "state": "ball", "steps": 10},
        # a parameter sweep's batch: uneven runs, graph-captured steps
        {"name": "sweep-24", "kind": "sweep", "runs": 24, "nmin": 4505, "nmax": 24003, "state": "settled",
         "steps": 4},
        # a driver's steps between two records, host buffers in and out
        {"name": "host-25001", "kind": "host", "n": 25001, "state": "settled", "steps": 4},
        # the energy / momentum log of the 66,000-body impact
        {"name": "energy-66000", "kind": "energy", "n": 66000, "state": "settled"},
        # FP64 diagnostics where they are bound by memory
        {"name": "diag-8448000", "kind": "diag", "n": 8448000, "state": "ball", "scope": 0},
        # Earth, Moon and disk of a finished impact
        {"name": "analysis-66000", "kind": "analysis", "n": 66000, "state": "merged"},
        # one frame of the viewer at the reference's window size
        {"name": "picture-66000", "kind": "picture", "n": 66000, "state": "merged", "px": 1000, "point": 2},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forces", "modes", "step", "step", "step", "settle", "sweep", "host", "energy", "diag",
                       "analysis", "picture"])
    if kind == "forces":
        return {"kind": kind, "n": _size(rng, 500, 50000), "state": rng.choice(["ball", "settled"])}
    if kind == "modes":
        return {"kind": kind, "n": _size(rng, 4000, 60000), "state": "ball",
                "accum": rng.choice(["fp32", "fp64", "kahan"])}
    if kind == "step":
        state = rng.choice(["ball", "settled", "merged"])
        return {"kind": kind, "n": _size(rng, 4000, {"ball": 900000, "settled": 400000, "merged": 150000}[state]),
                "state": state}
    if kind == "settle":
        return {"kind": kind, "n": _size(rng, 1000, 40000), "state": "ball", "steps": rng.randint(5, 20)}
    if kind == "sweep":
        lo = _size(rng, 4505, 9000)
        return {"kind": kind, "runs": rng.randint(6, 48), "nmin": lo, "nmax": lo + rng.randint(1000, 20000),
                "state": "settled", "steps": rng.randint(2, 5)}
    if kind == "host":
        return {"kind": kind, "n": _size(rng, 2000, 130000), "state": "settled", "steps": rng.randint(1, 8)}
    if kind == "energy":
        return {"kind": kind, "n": _size(rng, 2000, 150000), "state": rng.choice(["ball", "settled"])}
    if kind == "diag":
        return {"kind": kind, "n": _size(rng, 20000, 8000000), "state": "ball", "scope": rng.choice([0, 1, 2])}
    if kind == "analysis":
        return {"kind": kind, "n": _size(rng, 5000, 100000), "state": "merged"}
    return {"kind": "picture", "n": _size(rng, 5000, 1000000), "state": rng.choice(["settled", "merged"]),
            "px": rng.randint(300, 1400), "point": rng.randint(1, 4)}


# ------------------------------------------------------------------ bodies --

def _directions(g, n):
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True).clamp_min(1e-12)


def _clump(g, n, radius, power):
    """n elements in a ball, r = radius u^power (1/3 is uniform), as (x, Fe first, Fe count)."""
    r = radius * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) ** power
    x = _directions(g, n) * r[:, None]
    fe = r < 0.3 * radius
    order = torch.argsort((~fe).to(torch.int8), stable=True)
    return x[order], int(fe.sum())


def _pair(x1, f1, x2, f2, v1, v2):
    """Two bodies in impact order [Fe1, Fe2, Si1, Si2]."""
    x = torch.cat([x1[:f1], x2[:f2], x1[f1:], x2[f2:]])
    v = torch.cat([v1[:f1], v2[:f2], v1[f1:], v2[f2:]])
    return x, v, f1 + f2, [f1, f1 + f2, f1 + f2 + len(x1) - f1]


def _spin(x, rate):
    return torch.stack([-rate * x[:, 1], rate * x[:, 0], torch.zeros_like(x[:, 0])], 1)


def _bodies(g, n, state, mass=MASS):
    """(pos, vel float32 (n, 4), Fe count, origin bounds)."""
    if state == "merged":
        n2, nd = max(1, n // 64), max(1, n // 40)
        n1 = n - n2 - nd
        radius = (n / 2250.0) ** (1.0 / 3.0)
        x1, f1 = _clump(g, n1, radius, 0.5)
        x2, f2 = _clump(g, n2, radius * 0.25, 1.0 / 3.0)
        gm = float(n1 * 0.42)
        x2 = x2 + torch.tensor([6.0 * radius, 0.0, 0.3 * radius], device="cuda", dtype=torch.float64)
        xd = _directions(g, nd) * (radius * (2.0 + 10.0 * torch.rand(nd, 1, generator=g, device="cuda",
                                                                     dtype=torch.float64)))
        v1 = _spin(x1, 0.3)
        v2 = _spin(x2, math.sqrt(gm / (6.0 * radius) ** 3))
        rd = xd.norm(dim=1, keepdim=True)
        t = _spin(xd, 1.0)
        t = t / t.norm(dim=1, keepdim=True).clamp_min(1e-9)
        vd = t * (gm / rd).sqrt() * (0.3 + 1.5 * torch.rand(nd, 1, generator=g, device="cuda", dtype=torch.float64))
        x, v, nfe, bounds = _pair(x1, f1, torch.cat([x2, xd]), f2, v1, torch.cat([v2, vd]))
        thermal = 0.5
    else:
        rho = 0.2445 if state == "ball" else 4.3
        n2 = max(1, n // 11)
        n1 = n - n2
        r1, r2 = ((3.0 * k / (4.0 * math.pi * rho)) ** (1.0 / 3.0) for k in (n1, n2))
        x1, f1 = _clump(g, n1, r1, 1.0 / 3.0)
        x2, f2 = _clump(g, n2, r2, 1.0 / 3.0)
        w1, w2 = (0.5 * math.sqrt(0.42 * k / r ** 3) for k, r in ((n1, r1), (n2, r2)))
        v1, v2 = _spin(x1, w1), _spin(x2, w2)
        d = r1 + r2
        x2 = x2 + torch.tensor([-1.25 * d, 0.7071 * d, 0.0], device="cuda", dtype=torch.float64)
        v2 = v2 + torch.tensor([1.2 * math.sqrt(0.84 * n / d), 0.0, 0.0], device="cuda", dtype=torch.float64)
        x, v, nfe, bounds = _pair(x1, f1, x2, f2, v1, v2)
        thermal = 0.05
    v = v + thermal * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    pos = torch.zeros(n, 4, device="cuda")
    vel = torch.zeros(n, 4, device="cuda")
    pos[:, :3], vel[:, :3] = x.float(), v.float()
    pos[:, 3] = torch.bucketize(torch.arange(n, device="cuda"), torch.tensor(bounds, device="cuda"), right=True).float()
    vel[:nfe, 3], vel[nfe:, 3] = mass
    return pos, vel, nfe, bounds


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _sweep_sizes(case):
    r, lo, hi = case["runs"], math.log(case["nmin"]), math.log(case["nmax"])
    return [int(math.exp(lo + (hi - lo) * ((7 * k) % r) / max(1, r - 1))) for k in range(r)]


def _inputs(case, seed):
    """pos, vel, [(offset, n, nfe)], bounds and whatever else is drawn, from the seed alone."""
    g, kind = _generator(seed), case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "sweep":
        parts, runs, off = [], [], 0
        for n in _sweep_sizes(case):
            p, v, nfe, _ = _bodies(g, n, case["state"])
            parts.append((p, v))
            runs.append((off, n, nfe))
            off += n
        s["pos"], s["vel"] = (torch.cat([q[k] for q in parts]) for k in (0, 1))
        s["parts"], s["bounds"] = runs, [0, 0, 0]
    elif kind == "settle":
        nt = case["n"] - case["n"] // 11
        parts, runs, off = [], [], 0
        for n in (nt, case["n"] - nt):
            x, nfe = _clump(g, n, (n / 4.0) ** (1.0 / 3.0), 1.0 / 3.0)  # the raw body of the builder
            p, v = torch.zeros(n, 4, device="cuda"), torch.zeros(n, 4, device="cuda")
            p[:, :3] = x.float()
            v[:nfe, 3], v[nfe:, 3] = MASS
            parts.append((p, v))
            runs.append((off, n, nfe))
            off += n
        s["pos"], s["vel"] = (torch.cat([q[k] for q in parts]) for k in (0, 1))
        s["parts"], s["bounds"] = runs, [0, 0, 0]
    else:
        s["pos"], s["vel"], nfe, s["bounds"] = _bodies(g, case["n"], case["state"],
                                                       REF_MASS if kind == "forces" else MASS)
        s["parts"] = [(0, case["n"], nfe)]
        if kind == "diag" and case["scope"]:
            s["label"] = torch.randint(0, 4, (case["n"],), generator=g, device="cuda", dtype=torch.uint8)
    return s


def _damp(kind):
    return 8.0 if kind == "settle" else 0.0


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = s["kind"]
    s["stream"] = torch.cuda.current_stream().cuda_stream
    if kind == "forces":
        s["params"] = gi.params_from_material(1.0, 1.0, *REF_MASS, *REF_K, KR_FE, KR_SI, SD_FE, SD_SI)
        s["consts"] = gi.collision_consts(s["params"], s["parts"][0][2])
        s["force"] = torch.zeros_like(s["pos"])
        return s
    s["params"] = gi.params_from_material(1.0, 1.0, *MASS, K_FE, K_SI, KR_FE, KR_SI, SD_FE, SD_SI)
    s["runs"] = [gi.Run(o, n, f, 0, DT, DT / MASS[0], DT / MASS[1], _damp(kind)) for o, n, f in s["parts"]]
    s["ctx"] = gi.Context(0, accum=ACCUM[case["accum"]]) if kind == "modes" else gi.Context(0)
    if kind == "modes":
        s["force"] = torch.zeros_like(s["pos"])
    elif kind == "step":
        s["pos2"], s["vel2"] = torch.zeros_like(s["pos"]), torch.zeros_like(s["vel"])
    elif kind == "settle":
        s["p"], s["v"] = s["pos"].clone(), s["vel"].clone()
    elif kind == "sweep":
        s["a"] = s["pos"].clone(), s["vel"].clone()
        s["b"] = torch.zeros_like(s["pos"]), torch.zeros_like(s["vel"])
        s["side"] = torch.cuda.Stream()
        s["side"].wait_stream(torch.cuda.current_stream())
        s["graph"] = s["ctx"].graph(*(t.data_ptr() for t in s["a"] + s["b"]), s["runs"], s["params"], case["steps"],
                                    s["side"].cuda_stream)
    elif kind == "host":
        s["p0"], s["v0"] = s.pop("pos").cpu(), s.pop("vel").cpu()
        s["p"], s["v"] = s["p0"].clone().pin_memory(), s["v0"].clone().pin_memory()
    elif kind == "analysis":
        s["scope"] = torch.zeros(case["n"], device="cuda", dtype=torch.uint8)
        s["group"] = torch.zeros(case["n"], device="cuda", dtype=torch.int32)
    elif kind == "picture":
        s["view"] = _view(case)
    return s


def _view(case):
    r = (case["n"] / 2250.0) ** (1.0 / 3.0) * 9.0 if case["state"] == "merged" else (case["n"] / 4.3) ** (1.0 / 3.0)
    return gi.view((0.0, 0.0, 2.0 * r), width=case["px"], height=case["px"], point_size=case["point"])


def run(s):
    kind, case, st = s["kind"], s["case"], s["stream"]
    if kind == "forces":
        gi.forces_collision(s["pos"].data_ptr(), s["vel"].data_ptr(), s["force"].data_ptr(), s["consts"], case["n"], st)
        return s["force"]
    ctx, runs, params = s["ctx"], s["runs"], s["params"]
    if kind == "modes":
        ctx.forces(s["pos"].data_ptr(), s["vel"].data_ptr(), s["force"].data_ptr(), runs, params, st)
        return s["force"]
    if kind == "step":
        ctx.step_pingpong(s["pos"].data_ptr(), s["vel"].data_ptr(), s["pos2"].data_ptr(), s["vel2"].data_ptr(), runs,
                          params, 1, st)
        return s["pos2"], s["vel2"]
    if kind == "settle":
        s["p"].copy_(s["pos"])
        s["v"].copy_(s["vel"])
        ctx.step(s["p"].data_ptr(), s["v"].data_ptr(), runs, params, case["steps"], st)
        return s["p"], s["v"]
    if kind == "sweep":
        with torch.cuda.stream(s["side"]):
            s["a"][0].copy_(s["pos"])
            s["a"][1].copy_(s["vel"])
        s["graph"].launch(s["side"].cuda_stream)
        return s["b"] if case["steps"] % 2 else s["a"]
    if kind == "host":
        s["p"].copy_(s["p0"])
        s["v"].copy_(s["v0"])
        ctx.run_host(s["p"].data_ptr(), s["v"].data_ptr(), case["n"], runs, params, case["steps"], st)
        return s["p"], s["v"]
    pos, vel = s["pos"].data_ptr(), s["vel"].data_ptr()
    if kind == "energy":
        return (np.array(ctx.diag(pos, vel, runs[0], params, stream=st)),
                np.array(ctx.potential(pos, runs, params, stream=st)))
    if kind == "diag":
        label = s["label"].data_ptr() if "label" in s else None
        return np.array(ctx.diag(pos, vel, runs[0], params, label, case["scope"], stream=st))
    if kind == "picture":
        return gi.splat(ctx, pos, case["n"], s["bounds"], s["view"], stream=st)
    scope, group = s["scope"].data_ptr(), s["group"].data_ptr()
    em = gi.find_earth_moon(ctx, pos, case["n"], 1.5, s["bounds"], group, scope, st)
    stats = [ctx.diag(pos, vel, runs[0], params, scope, k, st) for k in range(4)]
    disk = gi.find_disk(ctx, pos, vel, runs[0], params, scope, st)
    stats.append(ctx.diag(pos, vel, runs[0], params, scope, 4, st))
    counts = np.frombuffer(ctypes.string_at(ctypes.byref(em), ctypes.sizeof(em)), np.int32)
    return {"earth_moon": counts, "groups": s["group"], "scopes": s["scope"], "statistics": np.array(stats),
            "disk": np.array([disk.n_disk, disk.n_bound_inside, disk.n_unbound], np.int64),
            "earth": np.array([disk.earth_mass, disk.earth_radius])}


# ------------------------------------------------------------------- 64 bits --

def _table(mass, k):
    """The pair table by class (0 Si-Si, 1 Fe-Si, 2 Fe-Fe), stored as float like the constant structs."""
    f = np.float32
    (mf, ms), (kf, ks) = mass, k
    mix = kf + ks * KR_SI if SD_FE >= SD_SI else kf * KR_FE + ks
    t = {"G": [ms * ms, mf * ms, mf * mf], "K": [2 * ks, kf + ks, 2 * kf],
         "mid": [2 * ks * KR_SI, mix, 2 * kf * KR_FE],
         "in": [2 * ks * KR_SI, kf * KR_FE + ks * KR_SI, 2 * kf * KR_FE],
         "b1": [1 - SD_SI, 1 - min(SD_FE, SD_SI), 1 - SD_FE], "b2": [1 - SD_SI, 1 - max(SD_FE, SD_SI), 1 - SD_FE]}
    return {q: torch.tensor(np.array(v, f).astype(np.float64), device="cuda") for q, v in t.items()}


def _classes(n, nfe, a, b):
    """Pair class of bodies [a, b) against all n."""
    fe = torch.arange(n, device="cuda") < nfe
    return fe[a:b, None].long() + fe[None, :].long()


def _blocks(n):
    rows = max(1, int(6e7) // n)
    return [(a, min(n, a + rows)) for a in range(0, n, rows)]


def _force64(x, v, nfe, t):
    n = len(x)
    out = torch.empty_like(x)
    for a, b in _blocks(n):
        d = [x[None, :, c] - x[a:b, None, c] for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        cls = _classes(n, nfe, a, b)
        coef = t["G"][cls] * r2.clamp_min(1e-60).rsqrt() ** 3
        i, j = torch.nonzero(r2 < 1.0, as_tuple=True)
        keep = i + a != j
        coef[i[~keep], j[~keep]] = 0.0
        i, j = i[keep], j[keep]
        c, q = cls[i, j], r2[i, j]
        r = q.sqrt()
        dp = torch.stack([e[i, j] for e in d], 1)
        sep = (dp * (v[j] - v[i + a])).sum(1) >= 1.0
        k = torch.where(sep & (r < t["b1"][c]), torch.where(r >= t["b2"][c], t["mid"][c], t["in"][c]), t["K"][c])
        coef[i, j] = (t["G"][c] - k * (1.0 - q)) / r
        for e in range(3):
            out[a:b, e] = (coef * d[e]).sum(1)
    return out


def _steps64(pos, vel, parts, steps, damp):
    t = _table(MASS, (K_FE, K_SI))
    dtm = [float(np.float32(DT / m)) for m in MASS]
    dt = float(np.float32(DT))
    p, v = pos.double(), vel.double()
    for o, n, nfe in parts:
        x, u = p[o:o + n, :3].clone(), v[o:o + n, :3].clone()
        w = torch.full((n, 1), dtm[1], device="cuda", dtype=torch.float64)
        w[:nfe] = dtm[0]
        for _ in range(steps):
            u = u + (_force64(x, u, nfe, t) - damp * u) * w
            x = x + u * dt
        p[o:o + n, :3], v[o:o + n, :3] = x, u
    return p, v


def _diag64(pos, vel, nfe, sel=None):
    m = torch.full((len(pos),), float(np.float32(MASS[1])), device="cuda", dtype=torch.float64)
    m[:nfe] = MASS[0]
    x, v = pos[:, :3].double(), vel[:, :3].double()
    if sel is not None:
        m, x, v = m[sel], x[sel], v[sel]
    tot = m.sum()
    com, p = (m[:, None] * x).sum(0) / tot, (m[:, None] * v).sum(0)
    ang = (m[:, None] * torch.linalg.cross(x - com, v - p / tot)).sum(0)
    return torch.cat([tot[None], com, p / tot, ang, 0.5 * (m * (v * v).sum(1)).sum()[None], p,
                      torch.tensor([float(len(m))], device="cuda", dtype=torch.float64)])


def _potential64(x, nfe):
    t = _table(MASS, (K_FE, K_SI))
    n, total = len(x), 0.0
    for a, b in _blocks(n):
        d = [x[None, :, c] - x[a:b, None, c] for c in range(3)]
        r = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt()
        cls = _classes(n, nfe, a, b)
        u = -t["G"][cls] / r.clamp_min(1e-30)
        i, j = torch.nonzero(r < 1.0, as_tuple=True)
        g, k, q = t["G"][cls[i, j]], t["K"][cls[i, j]], r[i, j]
        u[i, j] = torch.where(i + a == j, torch.zeros_like(q), -g + g * (q - 1) - k * (q - q ** 3 / 3 - 2.0 / 3.0))
        total += float(u.sum())
    return 0.5 * total


def exact(case, seed):
    kind = case["kind"]
    if kind in ("analysis", "picture") or (kind not in ("sweep", "diag") and case["n"] > 160000):
        return None  # labels and pixels; or more pairs than 64 bits take in a few seconds
    work_n = sum(n * n for n in _sweep_sizes(case)) if kind == "sweep" else case.get("n", 0) ** 2
    if kind in ("sweep", "settle", "host") and work_n * case["steps"] > 6e10:
        return None
    s = _inputs(case, seed)
    pos, vel, parts = s["pos"], s["vel"], s["parts"]
    if kind == "diag":
        sel = None
        if case["scope"]:
            sel = (s["label"] == 1) | (s["label"] == 2) if case["scope"] == 1 else s["label"] == case["scope"] - 1
        return _diag64(pos, vel, parts[0][2], sel).cpu().numpy()
    if kind == "energy":
        return (_diag64(pos, vel, parts[0][2]).cpu().numpy(),
                np.array([_potential64(pos[:, :3].double(), parts[0][2])]))
    if kind in ("forces", "modes"):
        t = _table(REF_MASS, REF_K) if kind == "forces" else _table(MASS, (K_FE, K_SI))
        f = _force64(pos[:, :3].double(), vel[:, :3].double(), parts[0][2], t)
        return torch.cat([f, torch.zeros_like(f[:, :1])], 1)
    return _steps64(pos, vel, parts, 1 if kind == "step" else case["steps"], _damp(kind))


def work(case):
    kind = case["kind"]
    n = case.get("n", 0)
    pairs = 0.5 * n * (n - 1)
    if kind in ("forces", "modes"):
        return {"bytes": 48.0 * n, "flops": PAIR_FLOPS * pairs}
    if kind == "step":
        return {"bytes": 64.0 * n, "flops": PAIR_FLOPS * pairs}
    if kind == "settle":
        a, b = n - n // 11, n // 11
        return {"bytes": 64.0 * n * case["steps"], "flops": PAIR_FLOPS * 0.5 * (a * (a - 1) + b * (b - 1)) * case["steps"]}
    if kind == "sweep":
        sizes = _sweep_sizes(case)
        return {"bytes": 64.0 * sum(sizes) * case["steps"],
                "flops": PAIR_FLOPS * sum(0.5 * k * (k - 1) for k in sizes) * case["steps"]}
    if kind == "host":
        return {"bytes": 64.0 * n * case["steps"], "flops": PAIR_FLOPS * pairs * case["steps"]}
    if kind == "energy":
        return {"bytes": 48.0 * n, "flops": 12.0 * pairs}
    if kind == "diag":
        return {"bytes": (32.0 + (case["scope"] > 0)) * n, "flops": 40.0 * n}
    if kind == "analysis":
        return {"bytes": 37.0 * n + 33.0 * n, "flops": 200.0 * n}
    return {"bytes": 16.0 * n + 3.0 * case["px"] ** 2, "flops": 30.0 * n}

"""The workloads that this repository's speed is judged on, each through the Python binding (pe.py).

listed() holds the cases, draw() gives more of the same ranges, prepare() makes what a program has in
hand before a call, run() is one call, work() counts what it cannot do without, and exact() restates
the path in FP64 torch: mesh, mass properties, print variation, release, flight, tail-aware score and,
through autograd, the gradient.

Kinds of case:
  eval        genomes and outputs in device memory: a training evaluation, a holdout
  generation  the same, then the next population (pe_ga_step): one step of the device GA
  host        host arrays in and out (pe_evaluate_population): the command-line drivers' call
  audit       one design under many scenarios, statistics and distances to the host (pe_audit)
  sim         the drop-in boundary of the reference program: gpu_prepare, then gpu_sim
  grad        d(objective)/d(genome) (pe_grad)
  objective   the smoothed objective alone (pe_objective): line searches, differences
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "planes-rl_gb300"))
import pe  # noqa: E402

MAX_STEPS = 7200


# ------------------------------------------------------------------ cases
def _case(name, kind, pop, nseeds, first=1, stride=1, vary=0, max_steps=MAX_STEPS, formulation=1, precision=0, every=0):
    return {"name": name, "kind": kind, "pop": pop, "nseeds": nseeds, "first": first, "stride": stride, "vary": vary,
            "max_steps": max_steps, "formulation": formulation, "precision": precision, "every": every}


def listed():
    return [
        # the smallest call: one design under the 8 training scenarios, host to host (`planes evaluate` on a draft)
        _case("design_1x8", "host", 1, 8, first=3, stride=7919),
        # the finalists of a generation on the shared 128-scenario holdout
        _case("holdout_8x128", "eval", 8, 128, first=3, stride=7919),
        # a small population under 8 training scenarios: the first benchmark configuration
        _case("training_1024x8", "eval", 1024, 8),
        # one generation of the device GA at the second benchmark configuration: evaluate, then breed
        _case("generation_8192x8", "generation", 8192, 8, first=9),
        # the headline: a generation at scale
        _case("training_100000x12", "eval", 100000, 12, first=25),
        # the robustness audit of a champion
        _case("audit_1x100000", "audit", 1, 100000, first=9001, stride=7919),
        # a program that keeps its genomes on the host, at a ragged size
        _case("host_3001x5", "host", 3001, 5, first=11),
        # the reference program's own boundary, each plane under its own scenario
        _case("sim_8000", "sim", 8000, 1, first=17, vary=1),
        # the reference's summation order and frame, for parity with its results
        _case("reference_order_2048x8", "eval", 2048, 8, formulation=0),
        # the gradient benchmark: 256 genomes, 8 scenarios, 6 s of flight
        _case("gradient_256x8", "grad", 256, 8, max_steps=3600, every=60),
        # the hybrid search's polish of a generation's top 64
        _case("gradient_64x8", "grad", 64, 8, max_steps=7200, every=60),
        # a line search: the objective of candidates along a step, single precision
        _case("objective_512x8", "objective", 512, 8, max_steps=3600, precision=32),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "holdout", "generation", "host", "audit", "sim", "reference", "grad", "grad",
                       "objective"])
    first = rng.randrange(1, 400)
    if kind == "holdout":
        c = _case("", "eval", _log(rng, 1, 16), _log(rng, 32, 256), first, 7919)
    elif kind == "reference":
        c = _case("", "eval", _log(rng, 64, 4096), rng.randrange(1, 13), first, formulation=0)
    elif kind == "audit":
        c = _case("", "audit", 1, _log(rng, 1000, 100000), first, 7919)
    elif kind == "sim":
        c = _case("", "sim", _log(rng, 16, 16000), 1, first, vary=rng.randrange(2))
    elif kind == "grad":
        c = _case("", "grad", _log(rng, 8, 256), rng.randrange(1, 13), first, max_steps=rng.choice([2400, 3600, 7200]),
                  every=rng.choice([60, 60, 40, 90]))
    elif kind == "objective":
        c = _case("", "objective", _log(rng, 16, 512), rng.randrange(1, 9), first, max_steps=3600,
                  precision=rng.choice([32, 64]))
    else:
        lo, hi = {"eval": (16, 100000), "generation": (64, 100000), "host": (1, 4000)}[kind]
        c = _case("", kind, _log(rng, lo, hi), rng.randrange(1, 13), first)
    del c["name"]
    return c


def _seeds(case):
    return [case["first"] + i * case["stride"] for i in range(case["nseeds"])]


def _genomes(case, seed):
    """The population: uniform over the gene bounds, as the search's first generation and its fresh draws are.  Up to 16
    genomes are somebody's designs: the printable ones of a larger draw."""
    lo, hi = (b.astype(np.float64) for b in pe.genome_bounds())
    rs, pop = np.random.RandomState(seed % (1 << 31)), case["pop"]
    if pop > 16:
        return (lo + rs.rand(pop, 35) * (hi - lo)).astype(np.float32)
    g = (lo + rs.rand(16 * pop + 64, 35) * (hi - lo)).astype(np.float32)
    fits = _planes(torch.from_numpy(g).double())["fits"].numpy()
    return np.ascontiguousarray(g[fits][:pop])


def prepare(case, seed):
    g = _genomes(case, seed)
    pop, flights, kind = case["pop"], case["pop"] * case["nseeds"], case["kind"]
    s = {"case": case, "seeds": np.asarray(_seeds(case), np.int32), "host": g}
    if kind == "sim":
        s["buf"] = pe.PanelBuf(pop)
    else:
        s["engine"] = pe.Engine(0)
        if case["formulation"] == 0:
            s["engine"].set_config(formulation=0, lanes=32, warps=4, reg_cap=0)
    if kind in ("host", "audit"):
        return s
    d = torch.device("cuda", 0)
    s["g"] = torch.from_numpy(g).to(d)
    wide = torch.float64 if kind == "objective" else torch.float32
    s["dist"] = torch.empty(flights, dtype=wide, device=d)
    s["scores"] = torch.empty(pop, dtype=wide, device=d)
    s["steps"] = torch.empty(flights, dtype=torch.int32, device=d)
    s["next"] = torch.empty(pop, 35, dtype=torch.float32, device=d)
    return s


def run(state):
    c, seeds = state["case"], state["seeds"]
    kind, pop, e = c["kind"], c["pop"], state.get("engine")
    if kind == "host":
        return e.evaluate_population(state["host"], seeds, c["vary"], c["max_steps"])
    if kind == "audit":
        return e.audit(state["host"][0], seeds, want_dist=True)
    g, dist, scores = state["g"], state["dist"], state["scores"]
    if kind == "sim":
        state["buf"].prepare(g, pop)
        state["buf"].sim(pop, int(seeds[0]), dist, vary=c["vary"])
        return {"dist": dist}
    if kind == "grad":
        e.grad(g, pop, seeds, state["next"], c["vary"], c["max_steps"], c["every"], d_obj=scores, d_dist=dist)
        return {"dist": dist, "objective": scores, "grad": state["next"]}
    if kind == "objective":
        e.objective(g, pop, seeds, c["precision"], c["vary"], c["max_steps"], d_obj=scores, d_dist=dist)
        return {"dist": dist, "objective": scores}
    e.eval_batch(g, pop, seeds, c["vary"], c["max_steps"], dist, state["steps"], scores)
    out = {"dist": dist, "steps": state["steps"], "scores": scores}
    if kind == "generation":
        pe.ga_step(g, scores, pop, 0, 30, 5, state["next"])
        out["next"] = state["next"]
    return out


def work(case):
    """Of drawn genomes 69 % fit the printer; their flights last 430 steps of 276 panels on average.  A panel-step takes 103
    operations and a plane-step 230; the gradient's way back takes twice its way forward."""
    flights = case["pop"] * case["nseeds"]
    fly = flights * (1.0 if case["pop"] <= 16 else 0.69) * 430 * (103 * 276 + 230)
    grad = case["kind"] == "grad"
    out = 4 * (flights * (2 if case["kind"] in ("eval", "generation", "host") else 1) + case["pop"])
    extra = 140 * case["pop"] if grad or case["kind"] == "generation" else 0
    return {"bytes": 140 * case["pop"] + out * (2 if case["kind"] == "objective" else 1) + extra, "flops": fly * (3 if grad else 1)}


# ------------------------------------------------------------------ the path in FP64
(SPAN, CHORD, TAPER, SWEEP, DIH_IN, DIH_OUT, KINK, CAMBER1, CAMBER2, WASHOUT, ELEVATOR, NOSE, KEEL, DECK_GAP, DECK_SCALE,
 BODY, FIN_H, FIN_CHORD, FIN_SWEEP, TAIL_SPAN, TAIL_CHORD, TAIL_ANGLE, LE_B1, LE_B2, CHORD_B1, CHORD_B2, FIN_LAYOUT, FIN_CANT,
 FIN_TAPER, FIN_SPAN_POS, TAIL_SWEEP, TAIL_TAPER, TAIL_DIH, TIP_ROUND, CENTER_CHORD) = range(35)
RHO, WALL, DT, GRAV = 1240 * 0.00045, 0.00045, 1.0 / 600, 9.81


def _camber(g, x):
    return (3 * (1 - x) ** 2 * x * g[:, CAMBER1:CAMBER1 + 1] + 3 * (1 - x) * x * x * g[:, CAMBER2:CAMBER2 + 1]
            + x ** 3 * g[:, ELEVATOR:ELEVATOR + 1] * 0.22)


def _wing(g, u, x, zoff, scale):
    """Points of a wing at span stations u [., K] and chord stations x [1, K]; zoff and scale are [P, 1]."""
    k = [g[:, i:i + 1] for i in range(35)]
    half = k[SPAN] * 0.5 * scale
    tf, b = u.abs(), k[BODY] * k[SPAN] * 0.5
    t, kink = tf * half, torch.maximum(k[KINK] * k[SPAN] * 0.5, b)
    in_, out = (torch.minimum(t, kink) - b).clamp(min=0), (t - kink).clamp(min=0)
    y = torch.minimum(t, b) + in_ * torch.cos(k[DIH_IN]) + out * torch.cos(k[DIH_OUT])
    z = in_ * torch.sin(k[DIH_IN]) + out * torch.sin(k[DIH_OUT])
    v, cr = 1 - tf, 1 + k[CENTER_CHORD]

    def bezier(a, b1, b2, e):
        return v ** 3 * a + 3 * v * v * tf * b1 + 3 * v * tf * tf * b2 + tf ** 3 * e

    ratio = bezier(cr, 1 + k[CHORD_B1], k[TAPER] + k[CHORD_B2], k[TAPER])
    ratio = ratio * (1 - k[TIP_ROUND] + k[TIP_ROUND] * (1 - 0.92 * tf * tf).clamp(min=0.08).sqrt())
    c = k[CHORD] * scale * ratio.clamp(0.035, 1.9)
    xr = 0.5 * k[CHORD] * scale * cr
    xt = 0.5 * k[CHORD] * scale - torch.tan(k[SWEEP]) * half
    le = bezier(xr, xr + k[LE_B1] * k[CHORD] * scale, xt + k[LE_B2] * k[CHORD] * scale, xt)
    px = le - x * c
    pz = z * scale + _camber(g, x) * c + k[WASHOUT] * tf * (px - (le - 0.25 * c))
    return torch.stack([px, torch.where(u < 0, -y, y), pz + zoff], 2)


def _mesh(g, mode, deck):
    """Vertices [P, nv, 3] and triangles [nt, 3] of genomes that share a fin layout and a deck count."""
    n, k = g.shape[0], [g[:, i] for i in range(35)]
    one, zero = g.new_ones(n, 1), g.new_zeros(n, 1)

    def row(*v):
        return g.new_tensor([list(v)])

    grid_u, grid_x = row(*[(i - 8) / 8 for i in range(17) for _ in range(6)]), row(*[j / 5 for _ in range(17) for j in range(6)])
    parts, tris, at = [_wing(g, grid_u, grid_x, zero, one)], [], 0

    def quads(rows, cols):
        for i in range(rows):
            for j in range(cols):
                a = at + i * (cols + 1) + j
                b = a + cols + 1
                tris.extend([(a, b, a + 1), (b, b + 1, a + 1)])

    def strip(base):
        tris.extend([(base, base + 1, base + 2), (base + 1, base + 3, base + 2)])

    def points(rows):
        parts.append(torch.stack([torch.stack([c + 0 * k[0] for c in p], 1) for p in rows], 1))

    quads(16, 5)
    at += 102
    hs, z0, hc = 0.5 * k[SPAN] * k[TAIL_SPAN], _camber(g, 0.82)[:, 0] * k[CHORD], k[CHORD] * k[TAIL_CHORD]
    tail = []
    for i in range(3):
        au = abs(i - 1)
        tc, le = hc * (1 + (k[TAIL_TAPER] - 1) * au), -0.32 * k[CHORD] - k[TAIL_SWEEP] * hc * au
        for j in range(3):
            x = le - 0.5 * j * tc
            tail.append((x, (i - 1) * hs * torch.cos(k[TAIL_DIH]), z0 + k[TAIL_ANGLE] * (x - le) + au * hs * torch.sin(k[TAIL_DIH])))
    points(tail)
    quads(2, 2)
    at += 9
    share = 0.94 if mode == 3 else k[FIN_SPAN_POS]
    fins = []
    for side in ([0], [-1, 1], [0, -1, 1], [-1, 1])[mode]:
        y0, zb = side * hs * share * torch.cos(k[TAIL_DIH]), z0 + abs(side) * hs * share * torch.sin(k[TAIL_DIH])
        fc = k[CHORD] * k[FIN_CHORD]
        xr, tip = -0.32 * k[CHORD] - k[TAIL_CHORD] * k[CHORD] * 0.82, fc * k[FIN_TAPER]
        cant, xs = abs(side) * k[FIN_CANT], -fc * k[FIN_SWEEP]
        ya, za = y0 + side * torch.sin(cant) * k[FIN_H], zb + torch.cos(cant) * k[FIN_H]
        fins += [(xr + 0.5 * fc, y0, zb), (xr - 0.5 * fc, y0, zb), (xr + xs + 0.5 * tip, ya, za), (xr + xs - 0.5 * tip, ya, za)]
        strip(at)
        at += 4
    points(fins)
    gap, scale = k[DECK_GAP][:, None], k[DECK_SCALE][:, None]
    if deck:
        parts.append(_wing(g, grid_u, grid_x, gap, scale))
        quads(16, 5)
        at += 102
    top = _wing(g, row(0.0, 0.0, 0.0, 0.0), row(0.0, 1 / 3, 2 / 3, 1.0), zero, one)
    keel = []
    for j in range(4):
        keel += [tuple(top[:, j].T), (top[:, j, 0], 0 * k[0], top[:, j, 2] - k[KEEL] * (0.35 + 0.65 * j / 3))]
    points(keel)
    for j in range(3):
        strip(at + 2 * j)
    at += 8
    if deck:
        for side in (-1, 1):
            u = (side * k[KINK])[:, None] * row(1.0, 1.0)
            parts += [_wing(g, u, row(0.25, 0.55), zero, one), _wing(g, u, row(0.25, 0.55), gap, scale)]
            strip(at)
            at += 4
    return torch.cat(parts, 1), torch.tensor(tris, device=g.device)


def _planes(g):
    """Of FP64 genomes [P, 35]: whether each fits the printer, mass [P], inertia [P, 6] (xx yy zz xy xz yz) and panels
    [P, 344, 7] about the centre of mass (centroid, area, normal), the unused ones without area."""
    lay, deck = g[:, FIN_LAYOUT], g[:, DECK_GAP] > float(np.float32(0.02))
    mode = (lay >= 0.25).long() + (lay >= 0.5).long() + (lay >= 0.75).long()
    fits, mass, inertia, panels, at = [], [], [], [], []
    for m in range(4):
        for b in range(2):
            i = torch.nonzero((mode == m) & (deck == bool(b)))[:, 0]
            if not len(i):
                continue
            gi = g[i]
            V, tri = _mesh(gi, m, b)
            ext = V.amax(1) - V.amin(1)
            fits.append((ext <= 0.250 - 0.00045).all(1))
            A, B, C = (V[:, tri[:, c]] for c in range(3))
            nrm = torch.linalg.cross(B - A, C - A)
            length = (nrm * nrm).sum(2).sqrt()
            area, unit = 0.5 * length, nrm / length[..., None]
            mi, ct = area * RHO, (A + B + C) / 3
            shell = mi.sum(1)
            mn = gi[:, NOSE] * shell
            pn = torch.stack([0.5 * gi[:, CHORD], 0 * mn, 0 * mn], 1)
            mm = shell + mn
            com = ((mi[..., None] * ct).sum(1) + mn[:, None] * pn) / mm[:, None]
            a, bb, c = (x - com[:, None] for x in (A, B, C))
            s = a + bb + c
            # second moments of a triangle about the centre: (sum of squares + square of the sum) / 12
            E = (a[..., :, None] * a[..., None, :] + bb[..., :, None] * bb[..., None, :] + c[..., :, None] * c[..., None, :]
                 + s[..., :, None] * s[..., None, :]) / 12
            E = (mi[..., None, None] * E).sum(1)
            th = mi * WALL * WALL / 12
            N = (th[..., None, None] * unit[..., :, None] * unit[..., None, :]).sum(1)
            r = pn - com
            E = E + mn[:, None, None] * r[:, :, None] * r[:, None, :]
            tr, tw = E.diagonal(dim1=1, dim2=2).sum(1), th.sum(1)
            diag = [tr - E[:, q, q] + tw - N[:, q, q] + 1e-9 for q in range(3)]
            off = [-E[:, p, q] - N[:, p, q] for p, q in ((0, 1), (0, 2), (1, 2))]
            pan = torch.cat([ct - com[:, None], area[..., None], unit], 2)
            pad = g.new_tensor([0, 0, 0, 0, 0, 0, 1]).expand(len(i), 344 - pan.shape[1], 7)
            panels.append(torch.cat([pan, pad], 1))
            mass.append(mm)
            inertia.append(torch.stack(diag + off, 1))
            at.append(i)
    back = torch.argsort(torch.cat(at))
    return {"fits": torch.cat(fits)[back], "mass": torch.cat(mass)[back], "inertia": torch.cat(inertia)[back],
            "panels": torch.cat(panels)[back]}


def _scenario(seeds):
    """The 25 numbers of each scenario: hashed draws, the seed's gust and base wind."""
    s = np.asarray(seeds, np.int64)

    def u(lane):
        x = (s.astype(np.uint32) * np.uint32(0x9E3779B9) + np.uint32(lane * 0x85EBCA6B & 0xFFFFFFFF)).astype(np.uint32)
        x = (x ^ (x >> np.uint32(16))) * np.uint32(0x7FEB352D)
        x = (x ^ (x >> np.uint32(15))) * np.uint32(0x846CA68B)
        return ((x ^ (x >> np.uint32(16))) >> np.uint32(8)).astype(np.float64) / 16777216.0

    def w(lane):
        return 2 * u(lane) - 1

    p = (s.astype(np.uint32) * np.uint32(37)).astype(np.int32).astype(np.int64)
    phase = np.sign(p) * (np.abs(p) % 97).astype(np.float64)
    angle = (s.astype(np.float32) * np.float32(1.61803)).astype(np.float64)  # the seed's angle is defined in FP32
    return {"speed": 9.2 + 2 * w(0), "pitch": 0.1 + 0.2 * w(1), "yaw": 0.12 * w(2), "roll": 0.16 * w(3), "height": 1.75 + 0.35 * w(4),
            "rates": np.stack([1.8 * w(5), 1.2 * w(6), 1.5 * w(7)], 1), "rho": 1.225 * (0.88 + 0.22 * u(8)),
            "cf": 0.02 * (0.75 + 0.55 * u(9)) * (0.9 + 0.25 * u(20)), "gust": 0.45 + 1.1 * (0.5 + 0.5 * np.sin(angle)),
            "bx": -0.25 + 1.15 * np.sin(phase * 0.71), "by": np.sin(phase * 1.13), "fpitch": 0.075 * w(10), "fyaw": 0.06 * w(11),
            "grip": np.stack([0.018 * w(12), 0.022 * w(13), 0.01 * w(14)], 1), "material": 0.88 + 0.24 * u(15),
            "infill": 0.06 + 0.34 * u(16), "bias": np.stack([0.018 * w(17), 0.01 * w(18), 0.006 * w(19)], 1),
            "wp": 0.025 * w(21), "wr": 0.035 * w(22), "phase": phase}


def _sym(I):
    return torch.stack([I[:, 0], I[:, 3], I[:, 4], I[:, 3], I[:, 1], I[:, 5], I[:, 4], I[:, 5], I[:, 2]], 1).reshape(-1, 3, 3)


def _qmul(a, b):
    aw, av, bw, bv = a[:, :1], a[:, 1:], b[:, :1], b[:, 1:]
    return torch.cat([aw * bw - (av * bv).sum(1, keepdim=True), aw * bv + bw * av + torch.linalg.cross(av, bv)], 1)


def _rot(q):
    w, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                        1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                        1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)


def _mv(M, v):
    return (M @ v[..., None])[..., 0]


def _cap(v, most):
    n = (v * v).sum(1, keepdim=True).sqrt()
    return torch.where(n > most, v * (most / n.clamp(min=1e-300)), v)


def _release(pl, at, sc):
    """Flight parameters and release state of flights of planes `at` under scenarios sc (a dict of [F] tensors)."""
    m_shell = pl["mass"][at] * sc["material"]
    m_fill = m_shell * sc["infill"]
    m = m_shell + m_fill
    cg = sc["bias"] * (m_fill / m)[:, None]
    I = _sym(pl["inertia"][at]) * (m / pl["mass"][at])[:, None, None]
    eye = torch.eye(3, dtype=m.dtype, device=m.device)
    for r, w in ((-cg, m_shell), (sc["bias"] - cg, m_fill)):
        I = I + w[:, None, None] * ((r * r).sum(1)[:, None, None] * eye - r[:, :, None] * r[:, None, :])
    inv = torch.linalg.inv(I)
    pan = pl["panels"][at]
    rb, n = pan[:, :, :3] - cg[:, None], pan[:, :, 4:]
    ar = sc["wr"][:, None] * (8 * rb[..., 1]).clamp(-1, 1)
    ap = sc["wp"][:, None] * (8 * rb[..., 0]).clamp(-1, 1)
    nx, ny, nz = n[..., 0], n[..., 1] - ar * n[..., 2], n[..., 2] + ar * n[..., 1]
    nb = torch.stack([nx + ap * nz, ny, nz - ap * nx], 2)
    nb = nb / (nb * nb).sum(2, keepdim=True).sqrt()
    ak = 0.5 * sc["rho"][:, None] * pan[..., 3]

    def turn(axis, angle):
        v = [0 * angle] * 3
        v[axis] = torch.sin(angle / 2)
        return torch.stack([torch.cos(angle / 2)] + v, 1)

    q = _qmul(turn(2, sc["yaw"]), _qmul(turn(1, -sc["pitch"]), turn(0, sc["roll"])))
    qf = _qmul(turn(2, sc["yaw"] + sc["fyaw"]), turn(1, -(sc["pitch"] + sc["fpitch"])))
    vel = _rot(qf)[:, :, 0] * sc["speed"][:, None]
    Jb = _mv(_rot(q).transpose(1, 2), vel * m[:, None])
    wb = _cap(sc["rates"] + 0.12 * _mv(inv, torch.linalg.cross(sc["grip"] - cg, Jb)), 35.0)
    pos = torch.stack([0 * m, 0 * m, sc["height"] + 0 * m], 1)
    par = [rb[..., 0], rb[..., 1], rb[..., 2], nb[..., 0], nb[..., 1], nb[..., 2], ak, m, I, inv]
    return par, torch.cat([pos, q, vel, wb], 1)


def _step(par, wind, st, k):
    """One step of 1/600 s from states st [F, 13] (position, quaternion, velocity, body rates) at step k."""
    rx, ry, rz, nx, ny, nz, ak, m, I, inv = par
    cf, phase, gust, bx, by = wind
    pos, q, vel, wb = st[:, :3], st[:, 3:7], st[:, 7:10], st[:, 10:]
    x, y, z, t, sin = pos[:, 0], pos[:, 1], pos[:, 2], k * DT, torch.sin
    air = torch.stack([
        bx + gust * (0.55 * sin(0.9 * x + 1.3 * t + phase) + 0.35 * sin(2.3 * z + 2.1 * t + 1.7 * phase)
                     + 0.25 * sin(4.1 * y + 3.3 * t + 0.4 * phase)),
        by + gust * (0.50 * sin(1.1 * x + 1.7 * t + 2.2 * phase) + 0.30 * sin(3.1 * z + 2.9 * t + 0.9 * phase)),
        gust * (0.30 * sin(1.4 * x + 2.3 * t + 3.1 * phase) + 0.20 * sin(2.7 * y + 1.9 * t + 1.2 * phase))], 1)
    R = _rot(q)
    v, w = _mv(R.transpose(1, 2), vel - air)[:, :, None].unbind(1), wb[:, :, None].unbind(1)
    vx, vy, vz = v[0] + w[1] * rz - w[2] * ry, v[1] + w[2] * rx - w[0] * rz, v[2] + w[0] * ry - w[1] * rx
    V2 = vx * vx + vy * vy + vz * vz + 1e-30
    V = V2.sqrt()
    s = (vx * nx + vy * ny + vz * nz) / V
    a = ak * V2 * s * (1.9 * (1 - s * s).clamp(min=1e-18).sqrt() + 2 * s.abs() - cf[:, None])
    b = ak * V * cf[:, None]
    fx, fy, fz = -(a * nx + b * vx), -(a * ny + b * vy), -(a * nz + b * vz)
    F = torch.stack([fx.sum(1), fy.sum(1), fz.sum(1)], 1)
    T = torch.stack([(ry * fz - rz * fy).sum(1), (rz * fx - rx * fz).sum(1), (rx * fy - ry * fx).sum(1)], 1)
    acc = _mv(R, F) / m[:, None]
    acc = torch.stack([acc[:, 0], acc[:, 1], acc[:, 2] - GRAV], 1)
    w1 = _cap(wb + DT * _mv(inv, T - torch.linalg.cross(wb, _mv(I, wb))), 150.0)
    v1 = _cap(vel + DT * acc, 60.0)
    q1 = q + 0.5 * DT * _qmul(q, torch.cat([0 * w1[:, :1], w1], 1))
    return torch.cat([pos + DT * v1, q1 / (q1 * q1).sum(1, keepdim=True).sqrt(), v1, w1], 1)


def _ended(st):
    return (st[:, 2] <= 0) | (st[:, 1].abs() > 300) | (st[:, 0] < -50) | (st[:, 0] != st[:, 0]) | (st[:, 7] != st[:, 7])


def _landing(before, after):
    """x where the flight crosses z = 0 between two states; of flights that end otherwise, the last x."""
    ground = after[:, 2] <= 0
    f = before[:, 2] / torch.where(ground, before[:, 2] - after[:, 2], 1.0)
    return torch.where(ground, before[:, 0] + f * (after[:, 0] - before[:, 0]), after[:, 0])


def _fly(par, wind, st, max_steps, smooth, every=0):
    """Distances of all flights and the step at which each ended; with `every`, also the states at its multiples."""
    n, dev = st.shape[0], st.device
    dist, end = torch.zeros(n, dtype=st.dtype, device=dev), torch.full((n,), max_steps - 1, device=dev)
    at, marks = torch.arange(n, device=dev), []
    alive = torch.ones(n, dtype=torch.bool, device=dev)
    for k in range(max_steps):
        if k % (every or 50) == 0:  # the flights that have ended leave
            if not bool(alive.all()):
                at, st, par, wind, alive = at[alive], st[alive], [p[alive] for p in par], [w[alive] for w in wind], alive[alive]
            if not len(at):
                break
            if every:
                marks.append((k, at, st))
        new = _step(par, wind, st, k)
        over = alive & (_ended(new) | torch.full_like(alive, k == max_steps - 1))
        where = at[over]
        if len(where):
            dist[where] = _landing(st[over], new[over]) if smooth else new[over, 0]
            end[where] = k
            alive = alive & ~over
        st = new
    return dist, end, marks


def _tail(d):
    s = d.shape[1]
    srt, n = d.sort(1).values, (s + 3) // 4
    return 0.65 * d.mean(1) + 0.25 * srt[:, :n].mean(1) + 0.10 * srt[:, 0]


def _audit_stats(d):
    s, n = d.sort().values, d.numel()

    def pct(p):
        x = p * (n - 1)
        i = int(x)
        return s[i] + (s[min(i + 1, n - 1)] - s[i]) * (x - i)

    worst = max(1, n // 10)
    sd = ((s * s).mean() - s.mean() ** 2).clamp(min=0).sqrt()
    return torch.stack([s[0], pct(0.05), pct(0.1), pct(0.25), pct(0.5), s.mean(), sd, pct(0.75), pct(0.9), pct(0.95), s[-1],
                        s[:worst].mean(), (s < 0).double().sum()])


def exact(case, seed):
    kind, pop, S = case["kind"], case["pop"], case["nseeds"]
    if pop * S > 120000:  # over 20 s
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    g = torch.from_numpy(_genomes(case, seed)).to(dev).double()
    smooth, grad = kind in ("grad", "objective"), kind == "grad"
    g.requires_grad_(grad)
    with torch.set_grad_enabled(grad):
        planes = _planes(g)
    fits = planes.pop("fits")
    at = torch.arange(pop, device=dev).repeat_interleave(S)
    seeds = np.tile(np.asarray(_seeds(case), np.int64), pop) + case["vary"] * 7919 * np.repeat(np.arange(pop, dtype=np.int64), S)
    fly = fits[at]
    at, seeds = at[fly], seeds[fly.cpu().numpy()]
    sc = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in _scenario(seeds).items()}
    wind = [sc[k] for k in ("cf", "phase", "gust", "bx", "by")]
    leaf = {k: v.detach().requires_grad_(grad) for k, v in planes.items()}
    with torch.set_grad_enabled(grad):
        par, st = _release(leaf, at, sc)
    with torch.no_grad():
        flat = [p.detach() for p in par]
        d, end, marks = _fly(flat, wind, st.detach(), case["max_steps"], smooth, every=30 if grad else 0)
        dist = torch.full((pop * S,), -100.0, dtype=torch.float64, device=dev)
        dist[fly] = d
        scores = _tail(dist.reshape(pop, S))
    if not grad:
        if kind == "audit":
            return {"stats": _audit_stats(dist).cpu().numpy(), "dist": dist.cpu().numpy()}
        if kind == "sim":
            return {"dist": dist}
        if kind == "objective":
            return {"dist": dist, "objective": scores}
        return {"dist": dist, "steps": None, "scores": scores, "next": None}
    # back through the score, the flights segment by segment, the release and the mesh
    D = dist.reshape(pop, S).clone().requires_grad_(True)
    w = torch.autograd.grad(_tail(D).sum(), D)[0].reshape(-1)[fly]
    back = [torch.zeros_like(p) for p in flat]
    lam = torch.zeros_like(st)
    for k0, idx, s0 in reversed(marks):
        p = [x[idx].requires_grad_(True) for x in flat]
        s = first = s0.detach().requires_grad_(True)
        ends, total = end[idx], 0.0
        for k in range(k0, min(k0 + 30, case["max_steps"])):
            new = _step(p, [x[idx] for x in wind], s, k)
            over = ends == k
            total = total + (torch.where(over, w[idx] * _landing(s, new), 0.0)).sum()
            s = new
        total = total + (torch.where((ends >= k0 + 30)[:, None], lam[idx] * s, 0.0)).sum()
        got = torch.autograd.grad(total, [first] + p)
        lam[idx] = got[0]
        for acc, x in zip(back, got[1:]):
            acc.index_add_(0, idx, x)
    got = torch.autograd.grad([*par, st], list(leaf.values()), [*back, lam])
    dg = torch.autograd.grad(list(planes.values()), g, list(got))[0]
    return {"dist": dist, "objective": scores, "grad": torch.where(fits[:, None], dg, 0.0)}

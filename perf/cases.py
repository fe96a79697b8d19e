"""Workloads of the substep engine, each through the public `Sim` calls a program makes.

A pass is one turn of a program's loop around `Sim`:

  * an editing loop (`"loop": "edit"`): the program writes its host arrays, `upload()`,
    `advance(dt)`, `download()`: the per-frame loop of the twist and pull scenarios, and of any
    program that owns the state;
  * a resident loop (`"loop": "resident"`): the state stays on the device; `advance(dt)` (or
    `step()`), then `download()` to draw or to export the frame; a batch is a clip of so many
    passes, after which the program starts it again.

Scenes:

  readme   the two-yarn example of the README (64 vertices)
  swatch   layers of wavy yarns, alternating directions, each layer resting within the barrier
           range of the next: woven and stacked fabric
  bundle   parallel yarns on a square grid, both ends pinned, one end turned by the program: the
           cable twist, where almost every contact is between near-parallel segments
  pile     random-walk yarns in a cube: the contact-heavy single scene
  batch    many uneven random-walk piles in one batch: throughput
"""
import math

import numpy as np

from yarnball_b200 import scenes
from yarnball_b200.sim import Sim

SEG = 2e-3
RADIUS = float(np.float32(0.05 * 0.5e-3))
BARRIER = float(np.float32(1.9 * 0.5e-3))
META = dict(kCollision=1e-7, frictionCoeff=0.3, radius=RADIUS, barrierThickness=BARRIER)
KBEND, KSTRETCH, DENSITY = 1e-8, 2e-2, 1e-3
MAX_H = 1e-3
DRIFT = 0.15  # m/s: a scene in motion, 0.15 mm a substep
FRAME = 1 / 30.0
CLIP = 24  # passes of a resident batch before the program starts its clip again


def listed():
    return [
        # The README's example, its frame in an interactive loop.
        {"name": "readme_frame", "scene": "readme", "loop": "edit", "dt": FRAME},
        # The same scene stepped by a program that couples it with something else every substep.
        {"name": "readme_step", "scene": "readme", "loop": "resident", "dt": 0.0},
        # A small swatch, the largest simulations that fit one block's worth of vertices.
        {"name": "swatch_240", "scene": "swatch", "loop": "edit", "layers": 4, "yarns": 4, "verts": 15, "dt": FRAME},
        # A sample of fabric of a few thousand vertices, odd counts, one frame.
        {"name": "swatch_2k", "scene": "swatch", "loop": "edit", "layers": 6, "yarns": 11, "verts": 31, "dt": FRAME},
        # The size, step length, iteration count and detection cadence of the letter scenes.
        {"name": "swatch_13k_letter", "scene": "swatch", "loop": "edit", "layers": 10, "yarns": 27, "verts": 49,
         "dt": 1 / 60.0, "max_h": 4e-4, "iterations": 4, "period": 4},
        # The same size in the FP64 build, as a reference run.
        {"name": "swatch_13k_fp64", "scene": "swatch", "loop": "edit", "layers": 10, "yarns": 27, "verts": 49,
         "dt": 1 / 120.0, "precision": "fp64"},
        # Cable twist driven from the host, frame by frame.
        {"name": "bundle_100k", "scene": "bundle", "loop": "edit", "grid": 7, "verts": 2048, "dt": 1 / 60.0},
        # Contact-heavy piles as one plain scene.
        {"name": "pile_65k", "scene": "pile", "loop": "edit", "yarns": 256, "verts": 257, "cube": 0.063, "dt": 1 / 60.0},
        {"name": "pile_262k", "scene": "pile", "loop": "edit", "yarns": 1024, "verts": 256, "cube": 0.1, "dt": 1 / 120.0},
        # Uneven scenes in one batch: about a million vertices, and the benchmark's batch.
        {"name": "batch_1m", "scene": "batch", "loop": "resident", "cap": 1 << 20, "spec": 7, "dt": 1 / 120.0},
        {"name": "batch_8m", "scene": "batch", "loop": "resident", "cap": 1 << 23, "spec": 7, "dt": 1 / 120.0},
    ]


def draw(rng):
    scene = rng.choice(["swatch", "swatch", "swatch", "pile", "pile", "bundle", "batch"])

    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = {"scene": scene, "loop": "edit", "dt": rng.choice([FRAME, 1 / 60.0, 1 / 120.0])}
    if scene == "swatch":
        n, layers = spread(100, 150000), rng.randint(2, 12)
        verts = max(8, int(math.sqrt(n / layers * rng.uniform(0.7, 3.0))))
        c.update(layers=layers, verts=verts, yarns=max(2, int(n / layers / verts)))
        if n > 20000:
            c["dt"] = 1 / 120.0
        if rng.random() < 0.25:
            c["precision"] = "fp64"
        if rng.random() < 0.25:
            c.update(max_h=4e-4, iterations=4, period=4)
        elif rng.random() < 0.2:
            c.update(iterations=rng.choice([5, 6, 10]), period=rng.choice([1, 2]))
    elif scene == "bundle":
        c.update(grid=rng.randint(3, 9), verts=spread(100, 3000))
    elif scene == "pile":
        n, verts = spread(8000, 300000), rng.randint(60, 700)
        yarns = max(8, n // verts)
        # 130 to 260 vertices per cubic centimetre, the density of the listed piles
        c.update(yarns=yarns, verts=verts, cube=round((yarns * verts / rng.uniform(130e6, 260e6)) ** (1 / 3), 4),
                 dt=1 / 120.0)
    else:
        c.update(loop="resident", cap=spread(200000, 4000000), spec=rng.randint(1, 1000), dt=1 / 120.0)
    return c


# ---- inputs ------------------------------------------------------------------------------


def _wavy(rng, length, count):
    """`count` random curves of `length` points and amplitude about 1, smooth over some ten points."""
    i = np.arange(length)
    out = np.zeros((count, length))
    for _ in range(3):
        w = rng.uniform(0.15, 0.6, (count, 1))
        out += np.sin(w * i + rng.uniform(0, 2 * np.pi, (count, 1)))
    return out / 3


def _swatch(case, seed):
    """(positions, yarn lengths) of alternating layers; neighbouring layers are 0.85 mm apart."""
    rng = np.random.default_rng([seed, 1])
    L, Y, V = case["layers"], case["yarns"], case["verts"]
    pos, lens = [], []
    for layer in range(L):
        along = (np.arange(V) + rng.uniform(-0.4, 0.4, (Y, 1))) * SEG * 0.97
        across = np.arange(Y)[:, None] * 2.2e-3 + 0.25e-3 * _wavy(rng, V, Y)
        up = layer * 0.85e-3 + rng.uniform(-0.06e-3, 0.06e-3, (Y, 1)) + 0.05e-3 * _wavy(rng, V, Y)
        xyz = np.stack([along, up, across] if layer % 2 == 0 else [across, up, along], -1)
        for y in range(Y):
            n = V - (3 * layer + y) % 4  # ragged ends
            pos.append(xyz[y, :n])
            lens.append(n)
    return np.concatenate(pos).astype(np.float32), np.array(lens, np.int32)


def _bundle(case, seed):
    rng = np.random.default_rng([seed, 2])
    g, V = case["grid"], case["verts"]
    x = np.empty((g * g, V, 3))
    at = (np.arange(g) - (g - 1) / 2) * 1.1e-3
    x[:, :, 0] = np.repeat(at, g)[:, None] + 0.05e-3 * _wavy(rng, V, g * g)
    x[:, :, 2] = np.tile(at, g)[:, None] + 0.05e-3 * _wavy(rng, V, g * g)
    x[:, :, 1] = np.arange(V) * SEG
    return x.reshape(-1, 3).astype(np.float32), np.full(g * g, V, np.int32)


def _drift(seed, n):
    """Velocities of a scene in motion: one direction for all, and a little per vertex."""
    rng = np.random.default_rng([seed, 3])
    d = rng.normal(size=3)
    return (DRIFT * d / np.linalg.norm(d) + rng.normal(0, 0.01, (n, 3))).astype(np.float32)


def _single(case, pos, lens, pin_last=False):
    sim = Sim(int(lens.sum()), precision=case.get("precision", "fp32"))
    scenes.fill_yarns(sim, pos, lens, pin_first=True, pin_last=pin_last)
    for k, v in META.items():
        setattr(sim.meta, k, v)
    return sim


def prepare(case, seed):
    kind = case["scene"]
    if kind == "batch":
        sim, _ = scenes.build_batched(seed=seed, spec=scenes.batched_spec(case["spec"], cap=case["cap"]))
        sim.vels[:] = _drift(seed, sim.numVerts)
    else:
        if kind == "readme":
            sim = Sim(64)
            sim.verts["pos"][:] = scenes.readme_positions()
            for i in (0, 32, 63):
                sim.verts["invMass"][i] = 0.0
            sim.verts["flags"][31] = 0
            sim.meta.kCollision = 1e-7
        elif kind == "swatch":
            pos, lens = _swatch(case, seed)
            sim = _single(case, pos, lens)
        elif kind == "bundle":
            pos, lens = _bundle(case, seed)
            sim = _single(case, pos, lens, pin_last=True)
        else:
            lens = np.full(case["yarns"], case["verts"], np.int32)
            pos = scenes.random_walks(seed, lens, cube=case["cube"])
            sim = _single(case, pos, lens)
        if "iterations" in case:
            sim.meta.numItr = case["iterations"]
        if "period" in case:
            sim.meta.detectionPeriod = case["period"]
        sim.configure(DENSITY)
        sim.setKBend(KBEND)
        sim.setKStretch(KSTRETCH)
        sim.maxH = case.get("max_h", MAX_H)
        vels = _drift(seed, sim.numVerts)
        if kind == "bundle":  # the program turns the pinned upper ends and holds the lower ones
            top = np.cumsum(lens) - 1
            vels[top - lens + 1] = 0
            vels[top, 0] = 2 * np.pi * pos[top, 2]
            vels[top, 1] = 0
            vels[top, 2] = -2 * np.pi * pos[top, 0]
        sim.vels[:] = vels
    sim.upload()
    state = {"sim": sim, "loop": case["loop"], "dt": case["dt"], "vels_out": _vels_out(case)}
    state.update(verts=sim.verts.copy(), qs=sim.qs.copy(), vels=sim.vels.copy())
    state.update(passes=0, clip=CLIP if kind == "batch" else 0)
    return state


def _vels_out(case):
    """Whether a pass returns the velocities beside the positions and rotors.  A velocity is the
    substep's displacement over h, which in 32 bits leaves it the rounding of every sum of contact
    forces, magnified: in the scenes with thousands of contacts two orders of summation of the same
    code differ by 1e-4 in the velocities' norm and by 6e-3 at single vertices, and by 5e-8 and 5e-6
    in the positions.  There the positions and rotors, which a program draws and exports, are the
    result; in the FP64 build and in the small scenes the velocities are too."""
    if case.get("precision") == "fp64":
        return True
    return case["scene"] in ("readme", "swatch") and _count(case) <= 4096 and "max_h" not in case


def run(state):
    sim = state["sim"]
    over = state["clip"] and state["passes"] == state["clip"]
    state["passes"] = 1 if over else state["passes"] + 1
    if state["loop"] == "edit" or over:
        sim.verts[:] = state["verts"]
        sim.qs[:] = state["qs"]
        sim.vels[:] = state["vels"]
        sim.upload()
    if state["dt"] > 0:
        sim.advance(state["dt"])
    else:
        sim.step()
    sim.download()
    out = {"pos": sim.verts["pos"], "qs": sim.qs}
    if state["vels_out"]:
        out["vels"] = sim.vels
    return out


# ---- work --------------------------------------------------------------------------------


def _steps(case):
    dt, h = case["dt"], case.get("max_h", MAX_H)
    return max(1, math.ceil(np.float32(dt) / np.float32(h))) if dt > 0 else 1


def _count(case):
    if case["scene"] == "readme":
        return 64
    if case["scene"] == "swatch":
        return int(sum(case["verts"] - (3 * a + b) % 4 for a in range(case["layers"]) for b in range(case["yarns"])))
    if case["scene"] == "bundle":
        return case["grid"] ** 2 * case["verts"]
    if case["scene"] == "pile":
        return case["yarns"] * case["verts"]
    return int(sum(int(x.sum()) for x in scenes.batched_spec(case["spec"], cap=case["cap"])[1]))


# listed contacts per segment, about, as the passes have them
CONTACTS = {"readme": 0.0, "swatch": 4.0, "bundle": 13.0, "pile": 11.0, "batch": 2.0}


def work(case):
    """Every array element of a substep's passes once: 152 + 4c bytes a vertex for predictor, step
    limit and advection, 176 + 4c for an iteration, 128 + 12c for a detection; about 330 operations
    a vertex and iteration and 230 a contact."""
    n, steps, c = _count(case), _steps(case), CONTACTS[case["scene"]]
    it, period = case.get("iterations", 8), case.get("period", 1)
    w = 2 if case.get("precision") == "fp64" else 1
    sub = 152 + 4 * c + it * (176 + 4 * c) + (128 + 12 * c) / period
    host = 60 + (76 if case["loop"] == "edit" else 0)
    return {"bytes": n * (w * steps * sub + host), "flops": n * steps * it * (330 + 230 * c)}


# ---- the same results in 64 bits ---------------------------------------------------------

HAS_PREV, HAS_NEXT, HAS_NEXT_ORI, FIX_ORI = 1, 2, 4, 8


def _dot(a, b):
    return np.einsum("...i,...i->...", a, b)


def _qmul(l, r):
    lv, rv, lw, rw = l[..., :3], r[..., :3], l[..., 3:], r[..., 3:]
    return np.concatenate([lw * rv + rw * lv + np.cross(lv, rv), lw * rw - _dot(lv, rv)[..., None]], -1)


def _qinv(q):
    return q * np.array([-1, -1, -1, 1], q.dtype)


def _configured(pos, lens, pin_last):
    """Flags, masses, rest lengths, rotors and stiffnesses that configure() gives, in 32 bits."""
    f = np.float32
    n = len(pos)
    ends = np.cumsum(lens) - 1
    flags = np.full(n, HAS_NEXT)
    flags[ends] = 0
    free = np.ones(n, f)
    free[ends - lens + 1] = 0
    if pin_last:
        free[ends] = 0
    prev = np.concatenate([[False], (flags[:-1] & HAS_NEXT) != 0])
    nxt = (flags & HAS_NEXT) != 0
    nn = nxt & np.concatenate([nxt[1:], [False]])
    fix = ~nxt
    fix[-1] = False
    flags = flags | prev * HAS_PREV | nn * HAS_NEXT_ORI | fix * FIX_ORI
    seg = np.zeros((n, 3), f)
    seg[:-1] = pos[1:] - pos[:-1]
    lr = np.sqrt((seg[:, 0] * seg[:, 0] + seg[:, 1] * seg[:, 1]) + seg[:, 2] * seg[:, 2])
    length = np.where(nxt, lr, f(1) / f(n)).astype(f)
    mass = np.where(prev, np.concatenate([[f(0)], length[:-1]]), f(0)) + np.where(nxt, length, f(0))
    mass = mass.astype(f) * (f(0.5) * f(DENSITY))
    im = (free * (f(1) / mass)).astype(f)
    # rotor of each segment: from (1, 0, 0) to its direction, turned to the last one's twist
    d = seg * np.where(nxt, f(1) / np.where(nxt, lr, 1), 0)[:, None].astype(f)
    half = (d + np.array([1, 0, 0], f)) * f(0.5)
    half = half / np.sqrt(np.maximum(_dot(half, half), f(1e-30)))[:, None]
    qq = np.stack([np.zeros(n, f), -half[:, 2], half[:, 1], half[:, 0]], -1).astype(f)
    # e1 wedge half = (0*hz - hy*0, 0*hx - 1*hz, 1*hy - 0*hx)
    q = np.zeros((n, 4), f)
    last = np.array([0, 0, 0, 1], f)
    for i in range(n):
        if nxt[i]:
            a, b = qq[i], last
            # the x and w parts of inverse(a) * b, normalised
            x = a[3] * b[0] - b[3] * a[0] - (a[1] * b[2] - b[1] * a[2])
            w = a[3] * b[3] + (a[0] * b[0] + a[1] * b[1] + a[2] * b[2])
            s = f(1) / np.sqrt(x * x + w * w)
            x, w = x * s, w * s
            last = np.array([a[3] * x + w * a[0], w * a[1] + a[2] * x, w * a[2] - a[1] * x, a[3] * w - a[0] * x], f)
        q[i] = last
    rest = np.zeros((n, 4), f)
    rest[:, 3] = 5
    rest[:-1] = f(5) * _qmul(_qinv(q[:-1]), q[1:]).astype(f)
    rest *= ((f(4) * f(KBEND)) / length / np.sqrt(_dot(rest, rest)))[:, None]
    return flags, im, length, (f(KSTRETCH) * length).astype(f), q, rest


def _closest(a1, b0, b1):
    """Parameters of the closest points of segments [0, a1] and [b0, b1]."""
    e = b1 - b0
    a, b, c, da, db = _dot(a1, a1), _dot(a1, e), _dot(e, e), _dot(a1, b0), _dot(e, b0)
    with np.errstate(all="ignore"):
        v = (b * da - a * db) / (a * c - b * b)
    v = np.clip(np.where(np.isfinite(v), v, 0.5), 0, 1)[:, None]
    u = np.clip(_dot(b0 * (1 - v) + b1 * v, a1) / a, 0, 1)[:, None]
    v = np.clip(_dot(u * a1 - b0, e) / c, 0, 1)[:, None]
    return u, v


def _pairs(lo, hi):
    """Pairs i < j of overlapping boxes, by a grid with cells of the largest extent."""
    cell = float((hi - lo).max()) * 1.0001
    at = np.floor((lo - lo.min(0)) / cell).astype(np.int64) + 1
    dim = at.max(0) + 2
    key = (at[:, 0] * dim[1] + at[:, 1]) * dim[2] + at[:, 2]
    order = np.argsort(key, kind="stable")
    sk = key[order]
    found = []
    for ox in (-1, 0, 1):
        for oy in (-1, 0, 1):
            k = key + (ox * dim[1] + oy) * dim[2]
            a, b = np.searchsorted(sk, k - 1), np.searchsorted(sk, k + 2)
            cnt = b - a
            i = np.repeat(np.arange(len(lo)), cnt)
            j = order[np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(a, cnt)]
            keep = i < j
            i, j = i[keep], j[keep]
            keep = np.all((lo[i] <= hi[j]) & (lo[j] <= hi[i]), -1)
            found.append(np.stack([i[keep], j[keep]]))
    return np.concatenate(found, 1)


def _solve(H, f):
    """H x = f, H = (xx, yy, zz, xy, xz, yz)."""
    a, b, c, xy, xz, yz = (H[:, k] for k in range(6))
    m = np.stack([b * c - yz * yz, xz * yz - xy * c, xy * yz - xz * b, a * c - xz * xz, xy * xz - a * yz, a * b - xy * xy], -1)
    det = a * m[:, 0] + xy * m[:, 1] + xz * m[:, 2]
    g = np.stack([_dot(m[:, (0, 1, 2)], f), _dot(m[:, (1, 3, 4)], f), _dot(m[:, (2, 4, 5)], f)], -1)
    return g / det[:, None]


def exact(case, seed):
    """The pass from a new state in 64 bits: strict-Jacobi substeps of Stable Cosserat Rods."""
    if case["scene"] not in ("readme", "swatch", "bundle"):
        return None
    n, steps, its = _count(case), _steps(case), case.get("iterations", 8)
    if n * steps * its > 2_500_000:  # some fifteen seconds
        return None
    meta = dict(META)
    if case["scene"] == "readme":
        i = np.arange(32, dtype=np.float32)
        x = (np.float32(0.00002) * i) * (i - 16) + np.float32(0.002)
        half = np.stack([x, -np.float32(0.002) * i, 0 * i], -1)
        pos, lens = np.concatenate([half, half * np.array([-1, 1, 1], np.float32)]), np.array([32, 32])
        meta = dict(kCollision=1e-7, frictionCoeff=0.1, radius=1e-4, barrierThickness=8e-4)
    else:
        pos, lens = (_swatch if case["scene"] == "swatch" else _bundle)(case, seed)
    flags, im, length, ks, q, rest = _configured(pos, lens, case["scene"] == "bundle")
    vel = _drift(seed, n)
    if case["scene"] == "readme":
        im[63] = 0
    if case["scene"] == "bundle":
        top = np.cumsum(lens) - 1
        vel[top - lens + 1] = 0
        vel[top, 0] = 2 * np.pi * pos[top, 2]
        vel[top, 1] = 0
        vel[top, 2] = -2 * np.pi * pos[top, 0]

    x, vel, q, rest, im, length, ks = (np.asarray(t, np.float64) for t in (pos, vel, q, rest, im, length, ks))
    meta = {k: float(np.float32(v)) for k, v in meta.items()}
    # the single-precision values that the parameters have
    h = float(np.float32(case["dt"]) / np.float32(steps)) if case["dt"] > 0 else float(np.float32(MAX_H))
    last_h, damping, drag, stiff_fric = float(np.float32(MAX_H)), float(np.float32(1e-6)), float(np.float32(0.2)), 5.0
    scaler = float(np.float32(1.2))
    g = np.array([0, float(np.float32(-9.8)), 0])
    D, two_r, inv_b = damping / h, 2 * meta["radius"], 1 / meta["barrierThickness"]
    k_col, mu = meta["kCollision"] * inv_b, meta["frictionCoeff"]
    det_r = meta["radius"] + 0.5 * meta["barrierThickness"]
    safe = (1 - float(np.float32(0.1))) * 0.5
    nxt, prev = (flags & HAS_NEXT) != 0, (flags & HAS_PREV) != 0
    seg, pv = np.nonzero(nxt)[0], np.nonzero(prev)[0]
    mov = im != 0
    inertia = np.where(mov, 1 / (np.where(mov, im, 1) * h * h), 0)
    turn = np.nonzero(nxt & ((flags & FIX_ORI) == 0))[0]
    tp, tn = turn[(flags[turn] & HAS_PREV) != 0], turn[(flags[turn] & HAS_NEXT_ORI) != 0]
    last_vel, A, B = np.zeros_like(vel), np.zeros(0, int), np.zeros(0, int)
    diag = np.array([1.0, 1, 1, 0, 0, 0])

    def outer(v):
        return np.stack([v[:, 0] ** 2, v[:, 1] ** 2, v[:, 2] ** 2, v[:, 0] * v[:, 1], v[:, 0] * v[:, 2], v[:, 1] * v[:, 2]], -1)

    def gather(at, what):
        return np.stack([np.bincount(at, what[:, k], n) for k in range(what.shape[1])], -1)

    for step in range(steps):
        dx = h * vel
        y = dx + h * h * g
        s = np.clip(_dot((vel - last_vel) / last_h, g) / (g @ g), 0, 1)
        dx = dx + np.where(mov, h * h * s, 0)[:, None] * g
        last_vel = vel
        size = np.linalg.norm(dx, axis=1)
        if step % case.get("period", 1) == 0:
            both = np.maximum(size[seg], size[seg + 1])
            pad = (det_r * scaler + both)[:, None]
            i, j = _pairs(np.minimum(x[seg], x[seg + 1]) - pad, np.maximum(x[seg], x[seg + 1]) + pad)
            a, b = seg[i], seg[j]
            ok = b - a > 2
            i, j, a, b = i[ok], j[ok], a[ok], b[ok]
            u, v = _closest(x[a + 1] - x[a], x[b] - x[a], x[b + 1] - x[a])
            d = u * (x[a + 1] - x[a]) - ((x[b] - x[a]) * (1 - v) + (x[b + 1] - x[a]) * v)
            ok = _dot(d, d) < (2 * det_r * scaler + both[i] + both[j]) ** 2
            A, B = np.concatenate([a[ok], b[ok]]), np.concatenate([b[ok], a[ok]])
        limit = np.full(n, np.inf)
        limit[seg] = det_r * (scaler - 1) + size[seg]
        u, v = _closest(x[A + 1] - x[A], x[B] - x[A], x[B + 1] - x[A])
        d = u * (x[A + 1] - x[A]) - ((x[B] - x[A]) * (1 - v) + (x[B + 1] - x[A]) * v)
        np.minimum.at(limit, A, safe * np.linalg.norm(d, axis=1))
        limit[pv] = np.minimum(limit[pv], limit[pv - 1])
        e = np.zeros_like(x)
        e[seg] = x[seg + 1] - x[seg]
        for _ in range(its):
            f = inertia[:, None] * (y - dx)
            H = inertia[:, None] * diag
            # stretch
            now = (e[seg] + dx[seg + 1] - dx[seg]) / length[seg, None]
            w, xyz = q[seg, 3:], q[seg, :3]
            e1 = np.zeros_like(xyz)
            e1[:, 0] = 1
            r = w * e1 + np.cross(xyz, e1)
            c = now - (w * r + np.cross(xyz, r) + xyz[:, :1] * xyz)
            k = (ks[seg] / length[seg])[:, None]
            dd = k / length[seg, None]
            f[seg] += k * c - D * dd * dx[seg]
            f[seg + 1] += -k * c - D * dd * dx[seg + 1]
            H[seg] += dd * (1 + D) * diag
            H[seg + 1] += dd * (1 + D) * diag
            # contacts
            if len(A):
                a1, b0, b1 = x[A + 1] - x[A], x[B] - x[A], x[B + 1] - x[A]
                u, v = _closest(a1 + dx[A + 1] - dx[A], b0 + dx[B] - dx[A], b1 + dx[B + 1] - dx[A])
                move = dx[A] * (1 - u) + dx[A + 1] * u - (dx[B] * (1 - v) + dx[B + 1] * v)
                nrm = u * a1 - (b0 * (1 - v) + b1 * v) + move
                dist = np.linalg.norm(nrm, axis=1)
                gap = (dist - two_r) * inv_b
                on = gap <= 1
                at, u, move, nrm = A[on], u[on], move[on], nrm[on] / dist[on, None]
                gap = np.maximum(gap[on], float(np.float32(1e-3)))[:, None]
                lg, ig, wa = np.log(gap), 1 / gap, 1 - u
                dH = (-3 + (2 + ig) * ig - 2 * lg) * k_col * inv_b
                ff = -(1 - gap) * (gap - 1 + 2 * gap * lg) * ig * k_col
                fa = (ff * wa - D * dH * wa * wa * _dot(nrm, dx[at])[:, None]) * nrm
                fb = (ff * u - D * dH * u * u * _dot(nrm, dx[at + 1])[:, None]) * nrm
                slide = move - _dot(nrm, move)[:, None] * nrm
                sl = np.linalg.norm(slide, axis=1)[:, None]
                f1 = np.where(sl > 0, np.minimum(stiff_fric, mu * ff / np.where(sl > 0, sl, 1)), 0)
                nn = outer(nrm)
                M = dH * (1 + D) * nn + f1 * (diag - nn)
                f += gather(at, fa - f1 * wa * slide) + gather(at + 1, fb - f1 * u * slide)
                H += gather(at, wa * wa * M) + gather(at + 1, u * u * M)
            new = dx + np.where(mov[:, None], _solve(np.where(mov[:, None], H, diag), f), 0)
            ln = np.linalg.norm(new, axis=1)
            cut = mov & (ln > limit)
            new[cut] *= (limit[cut] / ln[cut])[:, None]
            dx = new
            # orientations
            v = (e[turn] + dx[turn + 1] - dx[turn]) / length[turn, None] * (-2 * ks[turn, None])
            b = np.zeros((n, 4))
            sign = np.where(_dot(_qmul(_qinv(q[tp - 1]), q[tp]), rest[tp - 1]) > 0, 1.0, -1.0)[:, None]
            b[tp] += sign * _qmul(q[tp - 1], rest[tp - 1])
            sign = np.where(_dot(_qmul(_qinv(q[tn]), q[tn + 1]), rest[tn]) > 0, 1.0, -1.0)[:, None]
            b[tn] += sign * _qmul(q[tn + 1], _qinv(rest[tn]))
            b = b[turn]
            lam = np.linalg.norm(v, axis=1) + np.linalg.norm(b, axis=1)
            r = _qmul(_qmul(np.concatenate([v, 0 * v[:, :1]], -1), b), np.array([1.0, 0, 0, 0])) + lam[:, None] * b
            q = q.copy()
            q[turn] = r / np.linalg.norm(r, axis=1)[:, None]
        x = x + dx
        vel = np.where(mov[:, None], dx / h * (1 - drag * h), vel)
    return {"pos": x, "qs": q, "vels": vel} if _vels_out(case) else {"pos": x, "qs": q}

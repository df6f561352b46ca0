"""The work that a program built on this solver has it do, as timed cases.

A case is one call of a public entry point on a state that a simulation has
reached: a solver with its mesh assembled and its reference trees built, and
the arrays of the next step. The scenes are the generators of
collision_gb300.scenes, from a single small sheet to the full batch of 256,
in both arithmetic modes, through device and host buffers; plus a scene's
start (assembly and its first steps) and the exact CCD re-check of a step.

`layout` fixes what a scene is (sheet sizes, obstacles, speeds), the seed
passed to prepare() its noise, its gaps and its shapes.
"""
from __future__ import annotations

import numpy as np
import torch

from collision_gb300 import scenes
from collision_gb300.solver import CollisionSolver3d

DT = 1e-3
# Impact-zone passes after which a scene's step is ended (the reference's loop
# has no bound and does not end on some scenes).
ZONE_CAP = 300


def listed():
    return [
        # One small sheet on a sphere, stepped by a simulation that keeps its
        # state on the GPU: the smallest call, where launches and waits count.
        dict(name="sheet33_mixed", kind="sheet", n=33, obstacle="sphere", radius=0.25, speed=1.0, settle=10,
             mode="mixed", io="device"),
        # The same surface as the reference's own call: FP64, host arrays in
        # and out of every step.
        dict(name="sheet41_plain_host", kind="sheet", n=41, obstacle="box", radius=0.25, speed=2.0, settle=10,
             mode="plain", io="host"),
        # A run's start with a movable rigid body (the ball_plane deck): the
        # mesh assembled, both reference trees built, the first steps taken.
        dict(name="deck_ball_plane_start", kind="deck", deck="ball_plane", advance=0.04, steps=4, mode="plain"),
        # A start with a larger sheet: assembly and tree builds lead.
        dict(name="sheet97_start", kind="start", n=97, obstacle="sphere", radius=0.2, speed=2.0, steps=2,
             mode="mixed"),
        # A sheet folding into itself: self-contact, point-triangle and
        # edge-edge tests lead.
        dict(name="folded129_mixed", kind="folded", n=129, settle=42, mode="mixed", io="device"),
        # Strings on a box: bonds only, edge-edge tests and the strain limit.
        dict(name="strings64x512_mixed", kind="strings", nstr=64, nseg=512, settle=8, mode="mixed", io="device"),
        # A batch in free fall, before anything touches: broad phase, filters
        # and strain limiting with no contact.
        dict(name="batch128_fall", kind="batch", scenes=128, nmin=16, nmax=128, layout=1, contact=False, settle=1,
             mode="mixed", io="device"),
        # Batches of uneven sheets in contact: a middle size on the device,
        # plain FP64, and the full batch through host buffers.
        dict(name="batch48_contact", kind="batch", scenes=48, nmin=16, nmax=128, layout=2, contact=True, settle=8,
             mode="mixed", io="device"),
        dict(name="batch24_plain", kind="batch", scenes=24, nmin=16, nmax=96, layout=3, contact=True, settle=6,
             mode="plain", io="device"),
        dict(name="batch256_contact_host", kind="batch", scenes=256, nmin=16, nmax=128, layout=0, contact=True,
             settle=6, mode="mixed", io="host"),
        # A fine sheet crossing several thicknesses a step: CCD passes over
        # thousands of contacts, impact zones, a long strain sweep.
        dict(name="fast257_mixed", kind="fast", n=257, sub=4, settle=7, mode="mixed", io="device"),
        # The exact re-check of a finished step of a batch.
        dict(name="recheck64", kind="recheck", scenes=64, nmin=16, nmax=128, layout=4, contact=True, settle=6,
             mode="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["sheet", "sheet", "deck", "start", "folded", "strings", "batch", "batch", "batch", "fast",
                       "recheck"])
    mode = rng.choice(["mixed", "mixed", "plain"])
    io = rng.choice(["device", "device", "host"])
    shape = dict(obstacle=rng.choice(["sphere", "box"]), radius=round(rng.uniform(0.1, 0.3), 3),
                 speed=round(rng.uniform(0.5, 3.0), 2))
    if kind == "sheet":
        return dict(kind=kind, n=_log(rng, 9, 128), settle=rng.randint(4, 12), mode=mode, io=io, **shape)
    if kind == "deck":
        return dict(kind=kind, deck="ball_plane", advance=round(rng.uniform(0.03, 0.045), 4), steps=rng.randint(2, 5),
                    mode=mode)
    if kind == "start":
        return dict(kind=kind, n=_log(rng, 12, 128), steps=rng.randint(1, 3), mode=mode, **shape)
    if kind == "folded":
        return dict(kind=kind, n=_log(rng, 48, 129), settle=42, mode=mode, io=io)
    if kind == "strings":
        return dict(kind=kind, nstr=_log(rng, 4, 64), nseg=_log(rng, 60, 512), settle=rng.randint(5, 10), mode=mode,
                    io=io)
    if kind == "fast":
        return dict(kind=kind, n=_log(rng, 65, 257), sub=rng.choice([3, 4]), settle=rng.randint(2, 7), mode="mixed",
                    io=io)
    most = 24 if mode == "plain" else 128
    batch = dict(scenes=_log(rng, 2, most), nmin=rng.randint(8, 24), nmax=_log(rng, 32, 128),
                 layout=rng.randrange(1000), settle=rng.randint(3, 8))
    if kind == "recheck":
        return dict(kind=kind, mode="mixed", contact=True, **batch)
    return dict(kind=kind, mode=mode, io=io, contact=rng.random() < 0.75, **batch)


def _gap(rng, speed, contact=True):
    # in contact: reached in one to four steps of fall
    return speed * DT * float(rng.uniform(1.0, 4.0)) if contact else 0.05


def _batch_layout(case):
    """Sheet side, obstacle, radius and speed of every scene."""
    rng = np.random.default_rng([case["layout"], 17])
    return [(int(rng.integers(case["nmin"], case["nmax"] + 1)), "sphere" if rng.random() < 0.5 else "box",
             float(rng.uniform(0.1, 0.3)), float(rng.uniform(0.5, 3.0))) for _ in range(case["scenes"])]


def _scenes(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, 29])
    if kind in ("sheet", "start"):
        return [scenes.cloth_on_obstacle(case["n"], case["obstacle"], case["radius"], case["speed"], seed=seed,
                                         gap=_gap(rng, case["speed"]))]
    if kind == "deck":
        sc = scenes.deck(case["deck"], advance=case["advance"])
        # off the grid line, where the deck's meshes line up exactly, and with
        # a little noise on the free surface's points
        free = sc.fixed == 0
        sc.x[free] += np.array([1.1e-3, 0.7e-3, 0.0])
        sc.v[free] += rng.uniform(-1e-3, 1e-3, (int(free.sum()), 3))
        return [sc]
    if kind == "folded":
        return [scenes.folded_cloth(n=case["n"], seed=seed)]
    if kind == "strings":
        # the lowest strings a few steps above the box
        return [scenes.strings(nstr=case["nstr"], nseg=case["nseg"], seed=seed, z_range=(-0.035, 0.3),
                               volume_z=(-0.045, 0.45))]
    if kind == "fast":
        return [scenes.large(n=case["n"], sub=case["sub"], seed=seed)]
    return [scenes.cloth_on_obstacle(n, obstacle, radius, speed, seed=seed * 100003 + i,
                                     gap=_gap(rng, speed, case["contact"]))
            for i, (n, obstacle, radius, speed) in enumerate(_batch_layout(case))]


def _solver(case, scs):
    s = CollisionSolver3d(0)
    s.setMode(s.MIXED if case["mode"] == "mixed" else s.PLAIN_FP64)
    s.setZoneCap(ZONE_CAP)
    if len(scs) == 1:
        s.assembleFromScene(scs[0])
    else:
        s.assembleBatch(scs)
    return s


def prepare(case, seed):
    scs = _scenes(case, seed)
    if case["kind"] in ("deck", "start"):
        return dict(case=case, scene=scs[0])
    dt = scs[0].params["dt"]
    s = _solver(case, scs)
    stream = torch.cuda.Stream()
    s.setStream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        x = torch.from_numpy(np.concatenate([sc.x for sc in scs])).cuda()
        v = torch.from_numpy(np.concatenate([sc.v for sc in scs])).cuda()
        hc = torch.zeros(x.shape[0], dtype=torch.uint8, device="cuda")
        # the simulation up to this step, as its host loop runs it
        for _ in range(case["settle"]):
            x_new = torch.empty_like(x)
            s.resolveCollisionBatchDevice(x, x + dt * v, v, hc, x_new)
            x = x_new
        st = dict(case=case, solver=s, stream=stream, x=x, cand=x + dt * v, v0=v, hc0=hc, v=v.clone(), hc=hc.clone(),
                  out=torch.empty_like(x))
    stream.synchronize()
    if case["kind"] == "recheck":
        with torch.cuda.stream(stream):
            s.resolveCollisionBatchDevice(st["x"], st["cand"], st["v"], st["hc"], st["out"])
        stream.synchronize()
    elif case["io"] == "host":
        for k in ("x", "cand", "v0", "hc0"):
            st[k] = st[k].cpu().numpy()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("deck", "start"):
        sc = state["scene"]
        s = _solver(case, [sc])
        x, v, hc = sc.x, sc.v, np.zeros(sc.nv, np.uint8)
        for _ in range(case["steps"]):
            x, v, hc, _ = s.resolveCollisionBatch(x, scenes.candidate(sc, x, v), v, hc)
        out = dict(x=x, v=v, has_collsn=hc)
        for surface in sorted(sc.bodies):
            out[f"com{surface}"], out[f"comv{surface}"] = s.body(surface)
        s.close()
        return out
    s = state["solver"]
    if kind == "recheck":
        hits, per_scene = s.checkCCD(state["x"], state["out"])
        return dict(hits=hits, per_scene=per_scene)
    if case["io"] == "host":
        x, v, hc, collided = s.resolveCollisionBatch(state["x"], state["cand"], state["v0"], state["hc0"])
        return dict(x=x, v=v, has_collsn=hc, collided=collided)
    with torch.cuda.stream(state["stream"]):
        state["v"].copy_(state["v0"])
        state["hc"].copy_(state["hc0"])
        collided = s.resolveCollisionBatchDevice(state["x"], state["cand"], state["v"], state["hc"], state["out"])
    return dict(x=state["out"], v=state["v"], has_collsn=state["hc"], collided=collided)


_SPHERE = {3: (642, 1280), 4: (2562, 5120)}  # points and triangles of an icosphere


def _sizes(case):
    """(points, triangles, bonds) of the case's scenes."""
    kind = case["kind"]

    def sheet(n, obstacle):
        p, t = _SPHERE[3] if obstacle == "sphere" else (8, 12)
        return n * n + p, 2 * (n - 1) ** 2 + t

    if kind in ("sheet", "start"):
        return (*sheet(case["n"], case["obstacle"]), 0)
    if kind == "deck":
        sc = _scenes(case, 0)[0]
        return sc.nv, sc.nt, sc.nb
    if kind == "folded":
        return case["n"] ** 2, 2 * (case["n"] - 1) ** 2, 0
    if kind == "strings":
        return 8 + case["nstr"] * (case["nseg"] + 1), 12, case["nstr"] * case["nseg"]
    if kind == "fast":
        p, t = _SPHERE[case["sub"]]
        return case["n"] ** 2 + p + 8, 2 * (case["n"] - 1) ** 2 + t + 12, 0
    each = [sheet(n, obstacle) for n, obstacle, _, _ in _batch_layout(case)]
    return sum(p for p, _ in each), sum(t for _, t in each), 0


def work(case):
    """The step's inputs and outputs once: per point two positions, a velocity
    and a flag in, a position, a velocity and a flag out; per triangle its
    points, surface and rest lengths, per bond its points and rest length. The
    arithmetic no step is without: average velocity, final position and domain
    box per point, a swept box per element."""
    p, t, b = _sizes(case)
    steps = case.get("steps", 1)
    if case["kind"] == "recheck":
        return dict(bytes=48 * p + 12 * t + 8 * b, flops=6 * p + 54 * t + 36 * b)
    return dict(bytes=steps * (73 * p + 49 * p + 40 * t + 16 * b), flops=steps * (18 * p + 54 * t + 36 * b))


def exact(case, seed):
    """A sheet in free fall keeps its velocities and moves by them; with
    contacts a step is a sequence of decisions over the reference's trees
    (hundreds of thousands of pair tests, each in visiting order), which
    plain Python takes minutes for."""
    if case["kind"] != "batch" or case["contact"] or case["settle"] > 8:
        return None
    scs = _scenes(case, seed)
    x = np.concatenate([sc.x for sc in scs])
    v = np.concatenate([sc.v for sc in scs])
    for _ in range(case["settle"] + 1):
        x = x + DT * ((x + DT * v - x) / DT)
    if case["settle"] * max(3.0, np.abs(v).max()) * DT > 0.03:
        return None
    return dict(x=x, v=v, has_collsn=np.zeros(len(x), np.uint8), collided=np.zeros(len(scs), bool))

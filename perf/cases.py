"""Performance cases of the FLIP framework: what its users have it do.

A case is one call pattern of the public Python interface at one size:

  frame    a user's loop body: update(dt), then the particles' positions and
           velocities read back to host memory.  The kind covers dam breaks
           (grid, fill, particles per cell, tolerance, obstacle), the
           FluidManager demo (fluid added as meshes), mesh fluid sources and
           viscous fluid; `scene` says which
  surface  buildIsomesh() of a frame's particles and getIsomesh()
  batch    FluidRuntime.update_all over many resident scenes, and every
           scene's positions read back
  order    order_particles_by_id_noalloc on device arrays: particles in
           storage order put into load order

Scenes come from flipengine3d_gb300.scenes, sizes from its plain, mixed and
served sets, the tests' fixtures and the reference demo.  Frames follow each
other on the same simulation, as in a user's loop, so every frame meets new
particles.  Frame lengths are such that a frame is one substep at the speeds
these tanks reach (the larger grids step at 1/240 s), so that a frame's work
changes little from one to the next.
"""
from __future__ import annotations

import math
import os

# Hardware work queues for one stream per scene, read when the CUDA context
# is made (as the benchmark and a serving program set them).
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np
import torch

import flipengine3d_gb300 as fg
from flipengine3d_gb300 import scenes
from flipengine3d_gb300.fluidsimulation import FLIP_NOALLOC_MAX_IDS, order_particles_by_id_noalloc


def listed():
    return [
        # The reference demo's scene (FluidManager: fluid boxes as meshes, 1/30 s
        # frames, gravity -25, the engine's default tolerance) on 32^3 with a
        # loaded block: the smallest frame, bound by launches and waits.
        dict(name="demo_32", kind="frame", scene="demo", i=32, j=32, k=32, tol=1e-9, dt=1 / 30, warm=6),
        # The plain 64^3 dam break: an interactive preview.
        dict(name="dam_64", kind="frame", scene="dam", i=64, j=64, k=64, fx=0.4, fy=0.6, ppc=8, tol=1e-6,
             dt=1 / 120, warm=12, sphere=False, obstacle="none"),
        # A ragged box with two mesh obstacles (one with friction), sparse
        # particles and the served set's tolerance: what production scenes look like.
        dict(name="ragged_obstacles", kind="frame", scene="dam", i=101, j=83, k=67, fx=0.55, fy=0.5, ppc=5, tol=1e-5,
             dt=1 / 120, warm=12, sphere=False, obstacle="both"),
        # The benchmark's workload: 128^3 dam break plus falling sphere, 4.1M particles.
        dict(name="dam_sphere_128", kind="frame", scene="dam", i=128, j=128, k=128, fx=0.4, fy=0.6, ppc=8, tol=1e-6,
             dt=1 / 240, warm=8, sphere=True, obstacle="none"),
        # The large offline configuration: a 256x128x128 tank filled to 45%, 14M particles.
        dict(name="tank_256", kind="frame", scene="dam", i=256, j=128, k=128, fx=2.0, fy=0.45, ppc=8, tol=1e-6,
             dt=1 / 240, warm=4, sphere=False, obstacle="none"),
        # Inflow, outflow and a once-per-frame inflow: particles appear and vanish every frame.
        dict(name="sources_48", kind="frame", scene="sources", i=48, j=48, k=48, tol=1e-9, dt=1 / 60, warm=6),
        # A viscous (honey-like) dam break: the second linear system of the engine.
        dict(name="viscous_40", kind="frame", scene="viscous", i=40, j=40, k=40, fx=0.45, fy=0.55, tol=1e-9, nu=0.1,
             dt=1 / 60, warm=4),
        # The surface of the benchmark's particles at the demo's subdivision level: the largest mesh.
        dict(name="surface_128_s2", kind="surface", i=128, j=128, k=128, fx=0.4, fy=0.6, ppc=8, sub=2, sphere=True,
             warm=8),
        # A preview mesh of a ragged scene at the engine's default level.
        dict(name="surface_71_s1", kind="surface", i=71, j=59, k=83, fx=0.4, fy=0.6, ppc=8, sub=1, sphere=False,
             warm=8),
        # Many mixed-size scenes stepped together (a batch of the mixed set).
        dict(name="batch_16", kind="batch", count=16, lo=32, hi=96, tol=1e-6, dt=1 / 120, warm=4),
        # Load-order readback on the device for a host that may not allocate: the smallest call.
        dict(name="order_300k", kind="order", n=300_007),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dam"] * 4 + ["demo", "sources", "viscous", "surface", "surface", "batch", "order"])
    if kind == "dam":
        i, j, k = (_log_int(rng, 28, 144) for _ in range(3))
        return dict(kind="frame", scene="dam", i=i, j=j, k=k, fx=round(rng.uniform(0.2, 0.6), 3),
                    fy=round(rng.uniform(0.35, 0.6), 3), ppc=rng.randint(4, 8), tol=rng.choice([1e-5, 1e-6, 1e-9]),
                    dt=rng.choice([1 / 120, 1 / 240]), warm=rng.randint(4, 16), sphere=rng.random() < 0.5,
                    obstacle=rng.choice(["none", "none", "box", "sphere", "both"]))
    if kind == "demo":
        n = _log_int(rng, 29, 56)
        return dict(kind="frame", scene="demo", i=n, j=n, k=n, tol=1e-9, dt=rng.choice([1 / 30, 1 / 60]),
                    warm=rng.randint(3, 12))
    if kind == "sources":
        n = _log_int(rng, 24, 72)
        return dict(kind="frame", scene="sources", i=n, j=n, k=n, tol=1e-9, dt=rng.choice([1 / 60, 1 / 120]),
                    warm=rng.randint(3, 10))
    if kind == "viscous":
        i, j, k = (_log_int(rng, 18, 44) for _ in range(3))
        return dict(kind="frame", scene="viscous", i=i, j=j, k=k, fx=round(rng.uniform(0.3, 0.6), 3),
                    fy=round(rng.uniform(0.3, 0.6), 3), tol=1e-9, nu=rng.choice([0.01, 0.1, 1.0]), dt=1 / 60,
                    warm=rng.randint(2, 6))
    if kind == "surface":
        i, j, k = (_log_int(rng, 24, 128) for _ in range(3))
        return dict(kind="surface", i=i, j=j, k=k, fx=round(rng.uniform(0.2, 0.6), 3),
                    fy=round(rng.uniform(0.3, 0.6), 3), ppc=rng.randint(4, 8), sub=rng.choice([1, 2, 2, 3]),
                    sphere=rng.random() < 0.5, warm=rng.randint(2, 10))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 16), lo=_log_int(rng, 24, 40), hi=_log_int(rng, 48, 96),
                    tol=rng.choice([1e-5, 1e-6]), dt=1 / 120, warm=rng.randint(2, 6))
    return dict(kind="order", n=_log_int(rng, 1000, 1 << 20))


# ------------------------------------------------------------------- scenes
def _dam(case, seed):
    """A dam break over i x j x k cells of edge 1/i.  The fill fractions are of
    the box in x and y (2.0 in x: the whole length); z is filled."""
    i, j, k = case["i"], case["j"], case["k"]
    kw = dict(seed=seed, jsize=j, ksize=k, dx=1.0 / min(i, 128), sphere=bool(case.get("sphere")),
              ppc=case.get("ppc", 8), tolerance=case.get("tol", 1e-6))
    length = i * kw["dx"]
    kw["fill"] = (min(case["fx"], 1.0) * length if case["fx"] <= 1.0 else length, case["fy"] * j * kw["dx"],
                  k * kw["dx"])
    which = case.get("obstacle", "none")
    return scenes.dam_break(i, **kw) if which == "none" else scenes.dam_with_obstacles(i, which=which, **kw)


def _scene(case, seed):
    what = case.get("scene", "dam")
    if what == "demo":
        return scenes.mesh_fluid(case["i"], which="both", jitter_factor=None, seed=seed)
    if what == "sources":
        return scenes.fluid_sources(case["i"], which="both", seed=seed)
    sc = _dam(case, seed)
    if what == "viscous":
        sc.viscosity = case["nu"]
    return sc


def _warmed(case, seed):
    """The simulation after its first frames, and the particles loaded."""
    sc = _scene(case, seed)
    sim = fg.FluidSimulation.from_scene(sc, tolerance=case.get("tol"))
    for _ in range(case["warm"]):
        sim.update(case.get("dt", 1 / 120))
    return sim, sc.num_particles


def _pinned(rows):
    """A program's own pinned buffer for a readback, sized for the most it can
    get; rows past the current count hold what they held before."""
    return torch.zeros((rows, 3), dtype=torch.float32, pin_memory=True).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "order":
        # particles as an emitting and removing simulation holds them: ids
        # sparse in the id space, the storage sorted by position, not by id
        n = case["n"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        space = min(n + n // 8 + 1, FLIP_NOALLOC_MAX_IDS)
        ids = torch.randperm(space, generator=g, device="cuda")[:n].to(torch.int32)
        xyz = torch.rand(3, n, generator=g, device="cuda")
        out = torch.empty(n, 3, dtype=torch.float32, device="cuda")
        return dict(kind=kind, n=n, space=space, ids=ids, xyz=xyz, out=out)
    if kind == "batch":
        r = np.random.default_rng(seed)
        # the sizes are the case's (spread over its range), the particles the seed's
        edges = np.linspace(case["lo"], case["hi"], case["count"]).astype(int)
        fills = 0.2 + 0.4 * ((np.arange(case["count"]) * 7) % case["count"]) / case["count"]
        made = [scenes.dam_break(int(e), seed=int(r.integers(1 << 30)), fill=(float(f), 0.6, 1.0),
                                 tolerance=case["tol"]) for e, f in zip(edges, fills)]
        sims = [fg.FluidSimulation.from_scene(sc, tuned=True) for sc in made]
        outs = [_pinned(sc.num_particles) for sc in made]
        rt = fg.FluidRuntime(workers=16)
        for _ in range(case["warm"]):
            rt.update_all(sims, case["dt"])
        return dict(kind=kind, rt=rt, sims=sims, outs=outs, dt=case["dt"])
    if kind == "surface":
        # the mesh goes to the program's staging buffers, as a renderer's would
        sim, _ = _warmed(case, seed)
        sim.setSurfaceSubdivisionLevel(case["sub"])
        rows = int(8 * (case["i"] * case["j"] * case["k"]) ** (2 / 3) * case["sub"] ** 2) + 4096
        return dict(kind=kind, sim=sim, verts=np.zeros((rows, 3), np.float32), tris=np.zeros((2 * rows, 3), np.int32))
    sim, loaded = _warmed(case, seed)
    # fluid meshes and sources add particles: room for a full grid
    rows = loaded if case["scene"] in ("dam", "viscous") else 8 * case["i"] * case["j"] * case["k"]
    return dict(kind=kind, sim=sim, dt=case["dt"], pos=_pinned(rows), vel=_pinned(rows))


def run(state):
    kind = state["kind"]
    if kind == "order":
        xyz = state["xyz"]
        step = 4 * state["n"]
        order_particles_by_id_noalloc(xyz.data_ptr(), xyz.data_ptr() + step, xyz.data_ptr() + 2 * step,
                                      state["ids"].data_ptr(), state["n"], state["space"],
                                      state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "batch":
        state["rt"].update_all(state["sims"], state["dt"])
        for s, o in zip(state["sims"], state["outs"]):
            s.getMarkerParticlePositionData(out=o)
        return state["outs"]
    sim = state["sim"]
    if kind == "surface":
        sim.buildIsomesh()
        v, t = sim.getIsomesh()
        state["verts"][: len(v)] = v
        state["tris"][: len(t)] = t
        return state["verts"], state["tris"]
    sim.update(state["dt"])
    sim.getMarkerParticlePositionData(out=state["pos"])
    sim.getMarkerParticleVelocityData(out=state["vel"])
    return state["pos"], state["vel"]


# --------------------------------------------------------------- accounting
def _counts(i, j, k, fx, fy, ppc):
    """(cells, particles) of a dam break, the three wall cells on each side empty."""
    nx = max(min(fx, 1.0) * i - 3, 1.0)
    ny = max(fy * j - 3, 1.0)
    nz = max(k - 6, 1)
    return i * j * k, ppc * nx * ny * nz


def work(case):
    """What a pass cannot do without: the particles' state (position,
    velocity, rank: 28 bytes) read and written once per frame and copied out
    (24 bytes to the host), the level set and the MAC faces written and read
    once (4 + 2 * 12 bytes a cell), and one solution of the pressure system
    (its 32-byte rows read, the pressure written).  A mesh reads the
    positions and writes its vertices and triangles.  FLOPs: the splat onto
    and the interpolation from the faces and the three stages of the
    advection, about 1000 a particle."""
    kind = case["kind"]
    if kind == "order":
        return {"bytes": 28.0 * case["n"], "flops": 0.0}
    if kind == "batch":
        edges = np.linspace(case["lo"], case["hi"], case["count"]).astype(int)
        cn = [_counts(e, e, e, 0.4, 0.6, 8) for e in edges]
        cells, n = sum(c for c, _ in cn), sum(p for _, p in cn)
        return {"bytes": 68.0 * n + 28.0 * cells + 36.0 * n / 8, "flops": 1000.0 * n}
    ppc = case.get("ppc", 8)
    cells, n = _counts(case["i"], case["j"], case["k"], case.get("fx", 0.3), case.get("fy", 0.3), ppc)
    if case.get("sphere"):
        n += ppc * 0.0141 * min(case["i"], case["j"], case["k"]) ** 3
    if kind == "surface":
        area = 4.0 * (case["i"] * case["j"] * case["k"]) ** (2 / 3) * case["sub"] ** 2
        return {"bytes": 12.0 * n + 36.0 * area, "flops": 30.0 * n * case["sub"] ** 3}
    return {"bytes": 80.0 * n + 28.0 * cells + 36.0 * n / ppc, "flops": 1000.0 * n}


def exact(case, seed):
    """The load order of given positions is their exact answer.  A frame and
    a mesh have none of reasonable size: a 64-bit restatement of a whole FLIP
    step, with its incomplete-Cholesky solve, is a second engine."""
    if case["kind"] != "order":
        return None
    state = prepare(case, seed)
    order = torch.argsort(state["ids"].long())
    return state["xyz"].t()[order].double().contiguous()

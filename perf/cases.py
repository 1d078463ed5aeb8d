"""The work that programs built on this framework have it do, as timed cases.

Each case is a dict of plain values; `prepare` makes what a program has in
hand before the call (particles on the device in a context, a sorter and its
buffers), `run` is one pass through the public entry points, `work` the bytes
and operations such a pass cannot do without, and `exact` the same outputs
from a plain FP64 computation where one takes seconds. Inputs come from torch
generators keyed by the seed.

Kinds:
  step    Simulation.draw for a few steps, then the state back on the host:
          a resident run that looks at its particles every few steps
  batch   the same over many independent systems (draw_batched)
  forces  the stage calls on a fixed snapshot, with keys, layer counts and
          accelerations read back: an analysis program
  stream  independent snapshots pushed through the pipelined transfers,
          one step each
  scene   the reference's frame loop: draw, then the headless scene pass
  sort    RadixSort on device tensors
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from astro_gb300 import ic
from astro_gb300 import layouts as L
from astro_gb300.radix_sort import RadixSort
from astro_gb300.render import reference_camera
from astro_gb300.simulation import Simulation, default_params

# Tree and accuracy knobs of the committed autotuner results, by workload.
_C1 = dict(lbits=8, bucket=8, group_size=8, far_ratio=0.2, delta_weight=0.5)
_C2 = dict(lbits=12, bucket=16, group_size=32, far_ratio=0.15, delta_weight=0.7)
_C3 = dict(lbits=11, bucket=16, group_size=64, far_ratio=0.5, delta_weight=0.5)
_C4 = dict(lbits=9, bucket=16, group_size=32, far_ratio=0.25, delta_weight=0.5)
_C5 = dict(lbits=6, bucket=32, group_size=64, far_ratio=0.5, delta_weight=0.5)
# What a program that sets only theta, eps and the depth gets.
_DEFAULT = dict(lbits=14, bucket=16, group_size=0, far_ratio=0.0, delta_weight=1.0)


def _case(kind, scene, n, **kw):
    c = dict(kind=kind, scene=scene, n=n, form="plain", steps=1, dt=1e-3, eps=0.01, theta=0.7,
             block_warps=0, sort_variant=0)
    c.update(kw)
    return c


def listed():
    return [
        # One frame of a small interactive run: launches and waits count.
        dict(name="frame_1k", **_case("step", "plummer", 1024, dt=1e-4, **_C1)),
        # The small benchmark sphere, ten steps between looks at the state.
        dict(name="plummer_16k", **_case("step", "plummer", 16384, steps=10, block_warps=8,
                                         sort_variant=7, **_C1)),
        # A program with the driver's defaults reading keys and forces of a snapshot.
        dict(name="forces_100k", **_case("forces", "disk_bulge", 100003, eps=0.005, **_DEFAULT)),
        # The reference-scale galaxy, four steps between looks.
        dict(name="disk_524k", **_case("step", "disk_bulge", 524288, steps=4, dt=5e-4, eps=0.005,
                                       block_warps=4, sort_variant=4, **_C2)),
        # The precision form of the merger run.
        dict(name="merger_4m_precision", **_case("step", "two_plummer", 4194304, form="precision",
                                                 steps=2, eps=0.002, block_warps=8,
                                                 sort_variant=12, **_C3)),
        # 256 uneven systems in one step, precision form.
        dict(name="batch_256_precision", nsys=256, n_min=1024, n_max=65536, sizes_seed=4,
             **_case("batch", "plummer", 0, form="precision", block_warps=4, sort_variant=12, **_C4)),
        # The large cube at the reference's 7 layers.
        dict(name="cube_16m", **_case("step", "cube", 16777216, steps=2, dt=2e-4, eps=0.001,
                                      block_warps=4, sort_variant=12, **_C5)),
        # A cube keyed with all 21 bits per axis: 63-bit keys, 22 layers.
        dict(name="cube_6m_21bits", **_case("step", "cube", 6000007, steps=1, dt=2e-4, eps=0.001,
                                            **{**_C5, "lbits": 21})),
        # Snapshots streamed through upload, step and download.
        dict(name="stream_1m", snapshots=3, **_case("stream", "two_plummer", 1000003, eps=0.002, **_C3)),
        # The reference's own scene: frames with lighting, drawn headless.
        dict(name="scene_500k", width=1280, height=720, **_case("scene", "reference", 500205, steps=4,
                                                                dt=1.0 / 60.0)),
        # The stand-alone sort: a large array of 63-bit Morton keys on a stream ...
        dict(name="sort_16m", **_sort_case(16777216, 63, 64, True)),
        # ... and a small one on the default stream, its count known on the device only.
        dict(name="sort_60k", **_sort_case(60001, 63, 64, False)),
    ]


def _sort_case(n, used_bits, key_bits, own_stream):
    return dict(kind="sort", n=n, used_bits=used_bits, key_bits=key_bits, own_stream=own_stream)


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _depth(rng, n, scene):
    """A depth near the one the autotuner finds: a few particles per occupied
    cell (clustered scenes run deeper), or the driver's default, or all bits."""
    base = math.log(max(n, 8) / 32.0, 8) + (0 if scene == "cube" else 5)
    return min(21, max(3, int(round(base)) + rng.choice([-1, 0, 0, 1]))) if rng.random() < 0.8 \
        else rng.choice([14, 21])


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "forces", "batch", "stream", "scene", "sort", "sort"])
    if kind == "sort":
        used = rng.choice([18, 30, 36, 48, 63, 63])
        return _sort_case(_log_uniform(rng, 1000, 16777216), used, rng.choice([64, used]),
                          rng.random() < 0.5)
    if kind == "scene":
        w, h = rng.choice([(640, 360), (1280, 720), (1283, 717)])
        return dict(width=w, height=h, **_case("scene", "reference", 205 + _log_uniform(rng, 1000, 1000000),
                                               steps=rng.choice([1, 2, 4]), dt=1.0 / 60.0))
    scene = rng.choice(["plummer", "disk_bulge", "two_plummer", "cube"])
    knobs = dict(form=rng.choice(["plain", "precision"]), theta=rng.choice([0.5, 0.7, 0.7, 1.0]),
                 eps=rng.choice([0.001, 0.005, 0.01]), dt=2e-4, bucket=rng.choice([8, 16, 32]),
                 group_size=rng.choice([0, 8, 16, 32, 64, 64]),
                 far_ratio=rng.choice([0.0, 0.2, 0.35, 0.5]), delta_weight=rng.choice([0.5, 0.7, 1.0]),
                 block_warps=rng.choice([0, 0, 4, 8]), sort_variant=rng.choice([0, 0, 4, 12]))
    if kind == "batch":
        n_max = _log_uniform(rng, 512, 32768)
        return dict(nsys=_log_uniform(rng, 2, 300), n_min=max(64, n_max // 64), n_max=n_max,
                    sizes_seed=rng.randrange(1 << 20), lbits=rng.choice([6, 8, 9]),
                    **_case("batch", "plummer", 0, **knobs))
    n = _log_uniform(rng, 1000, 4000000 if kind == "step" else 1000000)
    c = _case(kind, scene, n, lbits=_depth(rng, n, scene), **knobs)
    if kind == "step":
        c["steps"] = rng.choice([1, 2, 5])
    if kind == "stream":
        c["snapshots"] = rng.choice([2, 3, 4])
    return c


# ------------------------------------------------------------ particles --

def _isotropic(u, r):
    cz = 2 * u[0] - 1
    sz = torch.sqrt(torch.clamp(1 - cz * cz, min=0))
    phi = 2 * math.pi * u[1]
    return torch.stack([r * sz * torch.cos(phi), r * sz * torch.sin(phi), r * cz], 1)


def _plummer(n, a, mass, gen):
    """Plummer sphere in equilibrium (Aarseth, Henon & Wielen 1974), G = 1."""
    def rand(*s):
        return torch.rand(*s, device="cuda", dtype=torch.float64, generator=gen)

    u = torch.clamp(rand(n), min=1e-9, max=0.999)
    r = a / torch.sqrt(u ** (-2.0 / 3.0) - 1)
    q = torch.zeros(n, device="cuda", dtype=torch.float64)
    done = torch.zeros(n, device="cuda", dtype=torch.bool)
    for _ in range(40):  # a trial is taken with probability 0.37
        t, y = rand(n), 0.1 * rand(n)
        ok = (y < t * t * (1 - t * t) ** 3.5) & ~done
        q = torch.where(ok, t, q)
        done |= ok
    ve = math.sqrt(2 * mass / a) * (1 + r * r / (a * a)) ** -0.25
    return _isotropic(rand(2, n), r), _isotropic(rand(2, n), q * ve)


def _particles(scene, n, seed, a=1.0):
    """(positions, velocities, masses) in FP32 on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*s):
        return torch.rand(*s, device="cuda", dtype=torch.float64, generator=gen)

    m = torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    if scene == "plummer":
        x, v = _plummer(n, a, 1.0, gen)
    elif scene == "two_plummer":
        # Two spheres 10 apart on a parabolic approach with pericentre 1.
        x, v = _plummer(n, 1.0, 0.5, gen)
        d = 10.0
        vt = math.sqrt(2.0) / d
        vr = -math.sqrt(2.0 / d - vt * vt)
        sign = torch.where(torch.arange(n, device="cuda") < n // 2, -0.5, 0.5).double()
        x[:, 0] += sign * d
        v[:, 0] += sign * vr
        v[:, 1] += sign * vt
    elif scene == "disk_bulge":
        # Exponential disk (80%) and Hernquist bulge, circular and isotropic speeds.
        nd = int(round(0.8 * n))
        u = torch.clamp(rand(7, n), min=1e-12, max=1 - 1e-12)
        rad = -torch.log(u[0] * u[1])
        x = torch.stack([rad * torch.cos(2 * math.pi * u[2]), rad * torch.sin(2 * math.pi * u[2]),
                         0.1 * torch.atanh(torch.clamp(2 * u[3] - 1, -0.999999, 0.999999))], 1)
        su = torch.sqrt(torch.clamp(u[4], max=0.99))
        x[nd:] = _isotropic(u[5:7], 0.2 * su / (1 - su))[nd:]
        r = torch.clamp(x.norm(dim=1), min=1e-6)
        menc = torch.empty_like(r)
        menc[torch.argsort(r)] = torch.arange(1, n + 1, device="cuda", dtype=torch.float64) / n
        g = torch.randn(n, 3, device="cuda", dtype=torch.float64, generator=gen)
        rxy = torch.clamp(x[:, :2].norm(dim=1), min=1e-6)
        vc = torch.sqrt(menc / r) * torch.sqrt(rxy / r)
        v = 0.05 * vc[:, None] * g
        v[:, 0] -= vc * x[:, 1] / rxy
        v[:, 1] += vc * x[:, 0] / rxy
        v[nd:] = (torch.sqrt(menc / (3 * r))[:, None] * g)[nd:]
    else:  # unit cube, Gaussian velocities, log-normal masses
        x = rand(n, 3)
        v = 0.1 * torch.randn(n, 3, device="cuda", dtype=torch.float64, generator=gen)
        m = torch.exp(0.5 * torch.randn(n, device="cuda", dtype=torch.float64, generator=gen))
        m /= m.sum()
    return x.float(), v.float(), m.float()


def _sizes(case):
    rng = random.Random(case["sizes_seed"])
    sizes = [_log_uniform(rng, case["n_min"], case["n_max"]) for _ in range(case["nsys"])]
    return sizes, [rng.uniform(0.5, 2.0) for _ in sizes]


def _initial(case, seed):
    """(positions, velocities, masses, system sizes) of a case on the GPU."""
    if case["kind"] != "batch":
        return (*_particles(case["scene"], case["n"], seed), [case["n"]])
    sizes, scales = _sizes(case)
    parts = [_particles(case["scene"], s, seed * 1009 + k, a) for k, (s, a) in enumerate(zip(sizes, scales))]
    return (*(torch.cat([p[i] for p in parts]) for i in range(3)), sizes)


def _pinned(n):
    return torch.zeros((n, 8), dtype=torch.float32, pin_memory=True)


def _as(t, dtype):
    return t.numpy().view(dtype).reshape(-1)


def _host(x, v, m):
    """Pinned PositionMass and VelocityRadius rows of these particles."""
    pm = torch.zeros((x.shape[0], 8), device=x.device)
    vr = torch.zeros_like(pm)
    pm[:, :3], pm[:, 4], vr[:, :3] = x, m, v
    hp, hv = _pinned(x.shape[0]), _pinned(x.shape[0])
    hp.copy_(pm)
    hv.copy_(vr)
    return hp, hv


def _params(case):
    if case["kind"] == "scene":
        return default_params(L.PRESET_REFERENCE)
    return default_params(L.PRESET_PHYSICAL,
                          form=L.FORM_PRECISION if case["form"] == "precision" else L.FORM_PLAIN,
                          theta=case["theta"], softening=case["eps"], lbits=case["lbits"],
                          bucket=case["bucket"], group_size=case["group_size"],
                          far_ratio=case["far_ratio"], open_delta_weight=case["delta_weight"],
                          block_warps=case["block_warps"], sort_variant=case["sort_variant"])


# ---------------------------------------------------------------- cases --

def prepare(case, seed):
    if case["kind"] == "sort":
        return _prepare_sort(case, seed)
    if case["kind"] == "scene":
        n = case["n"]
        pm, vr, ct = ic.reference_scene(5, 200, n - 205, seed=seed)
        sim = Simulation(_params(case), max_n=n)
        sim.upload(pm, vr, ct, n_tree=205)
        return dict(case=case, sim=sim, pm=_pinned(n), vr=_pinned(n),
                    camera=reference_camera(case["width"], case["height"]))
    if case["kind"] == "stream":
        inputs = [_host(*_particles(case["scene"], case["n"], seed * 1009 + k)) for k in range(case["snapshots"])]
        sim = Simulation(_params(case), max_n=case["n"])
        sim.upload(_as(inputs[0][0], L.POSITION_MASS), _as(inputs[0][1], L.VELOCITY_RADIUS))
        return dict(case=case, sim=sim, inputs=inputs,
                    outputs=[(_pinned(case["n"]), _pinned(case["n"])) for _ in inputs])
    x, v, m, sizes = _initial(case, seed)
    pm, vr = _host(x, v, m)
    n = x.shape[0]
    sim = Simulation(_params(case), max_n=n, max_systems=len(sizes))
    torch.cuda.synchronize()
    if case["kind"] == "batch":
        sim.upload_systems(_as(pm, L.POSITION_MASS), _as(vr, L.VELOCITY_RADIUS), sizes)
    else:
        sim.upload(_as(pm, L.POSITION_MASS), _as(vr, L.VELOCITY_RADIUS))
    sim.synchronize()
    return dict(case=case, sim=sim, sizes=np.asarray(sizes, np.uint32), pm=pm, vr=vr)


def _prepare_sort(case, seed):
    n, dev = case["n"], "cuda"
    gen = torch.Generator(device=dev).manual_seed(seed)
    # Room for a few more than the count, as a caller sizes its buffers ahead.
    room = n + n // 16
    top = (1 << case["used_bits"]) - 1
    keys = torch.randint(0, top, (room,), device=dev, generator=gen, dtype=torch.int64)
    state = dict(case=case, keys=keys, index=torch.arange(room, device=dev, dtype=torch.int32),
                 keys_out=torch.zeros_like(keys), index_out=torch.zeros(room, device=dev, dtype=torch.int32),
                 count=torch.tensor([n], device=dev, dtype=torch.int32), room=room,
                 sorter=RadixSort(room, case["key_bits"]),
                 stream=torch.cuda.Stream() if case["own_stream"] else None)
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        s = state["stream"].cuda_stream if state["stream"] is not None else 0
        state["sorter"].sort(state["keys"], state["index"], state["keys_out"], state["index_out"],
                             state["room"], state["count"], stream=s)
        return state["keys_out"], state["index_out"]
    sim = state["sim"]
    if kind == "forces":
        sim.generate_morton_codes()
        sim.sort()
        sim.build_tree()
        sim.barnes_hut()
        codes, sorted_codes, index = sim.read_keys()
        _, _, layers = sim.tree_info()
        return dict(accel=sim.read_accel(), codes=codes.view(np.int64),
                    sorted=sorted_codes.view(np.int64), index=index.view(np.int32),
                    layers=layers.view(np.int32))
    if kind == "stream":
        for (pm, vr), (pm_out, vr_out) in zip(state["inputs"], state["outputs"]):
            sim.upload_async(_as(pm, L.POSITION_MASS), _as(vr, L.VELOCITY_RADIUS))
            sim.draw(case["dt"], 1)
            sim.download_async(_as(pm_out, L.POSITION_MASS), _as(vr_out, L.VELOCITY_RADIUS))
        sim.synchronize()
        return state["outputs"]
    out = {}
    if kind == "scene":
        for _ in range(case["steps"]):
            sim.draw(case["dt"], 1)
            out["rgba"], out["depth"] = sim.splat(state["camera"], case["width"], case["height"])
    elif kind == "batch":
        sim.draw_batched(case["dt"], case["steps"], state["sizes"])
    else:
        sim.draw(case["dt"], case["steps"])
    sim.download(_as(state["pm"], L.POSITION_MASS), _as(state["vr"], L.VELOCITY_RADIUS))
    return dict(pm=state["pm"], vr=state["vr"], **out)


def _interactions(n, case):
    """Interactions per particle that a walk at this opening angle makes, to
    within a factor of about two: the opened leaves around a particle, one
    particle each time, and the accepted nodes, a constant number per layer
    that the particle count resolves."""
    leaf = n / 8.0 ** case["lbits"] if case["scene"] == "cube" else case["bucket"] / 2.0
    near = 27.0 * max(leaf, case["bucket"] / 2.0)
    cells = 60.0 * (0.7 / case["theta"]) ** 3 * max(1.0, math.log(max(n, 16) / max(leaf, 4.0), 8))
    return min(float(n), near * (0.7 / case["theta"]) ** 3 + cells)


def work(case):
    """Each input read once, each output written once; 20 operations an interaction."""
    n = case["n"]
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 24.0 * n, "flops": 0.0}
    if kind == "scene":
        # Position, velocity and colour read and written a frame; the image and the state out.
        frame = n * 96.0 + case["width"] * case["height"] * 20.0
        return {"bytes": case["steps"] * frame + 64.0 * n, "flops": case["steps"] * n * (205.0 + 5.0) * 20.0}
    per = 128.0 if case["form"] == "precision" else 72.0  # position, velocity, id, both ways
    if kind == "batch":
        sizes, _ = _sizes(case)
        flops = sum(20.0 * s * _interactions(s, case) for s in sizes)
        n = sum(sizes)
    else:
        flops = 20.0 * n * _interactions(n, case)
    if kind == "forces":
        return {"bytes": n * (16.0 + 16.0 + 20.0), "flops": flops}
    if kind == "stream":
        return {"bytes": case["snapshots"] * 128.0 * n, "flops": case["snapshots"] * flops}
    return {"bytes": case["steps"] * per * n + 64.0 * n, "flops": case["steps"] * flops}


# ---------------------------------------------------------------- exact --

def _accel64(x, m, eps):
    """Softened direct sum, G = 1."""
    n = x.shape[0]
    out = torch.empty_like(x)
    rows = max(1, (1 << 24) // n)
    for i in range(0, n, rows):
        d = [x[None, :, c] - x[i:i + rows, None, c] for c in range(3)]
        w = torch.rsqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps * eps)
        w = m * w * w * w
        for c in range(3):
            out[i:i + rows, c] = (w * d[c]).sum(1)
    return out


def _rows(x, other):
    out = torch.zeros((x.shape[0], 8), dtype=torch.float64, device=x.device)
    out[:, :3] = x
    if other is not None:
        out[:, 4] = other
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        s = _prepare_sort(case, seed)
        n = case["n"]
        keys, order = torch.sort(s["keys"][:n], stable=True)
        s["keys_out"][:n], s["index_out"][:n] = keys, s["index"][:n][order]
        return s["keys_out"], s["index_out"]
    if kind == "scene":
        return None
    if kind == "batch":
        pairs = case["steps"] * sum(float(s) * s for s in _sizes(case)[0])
    else:
        pairs = case.get("snapshots", case["steps"]) * float(case["n"]) ** 2
    if pairs > 1.6e11:
        return None
    eps = ctypes.c_float(case["eps"]).value  # as the context holds it
    dt = ctypes.c_float(case["dt"]).value
    if kind == "stream":
        snaps = [(*_particles(case["scene"], case["n"], seed * 1009 + k), [case["n"]])
                 for k in range(case["snapshots"])]
    else:
        snaps = [_initial(case, seed)]
    results = []
    for x, v, m, sizes in snaps:
        x, v, m = x.double(), v.double(), m.double()
        for _ in range(case["steps"]):
            a = torch.cat([_accel64(xs, ms, eps) for xs, ms in zip(x.split(sizes), m.split(sizes))])
            if kind != "forces":
                v = v + dt * a
                x = x + dt * v
        if kind == "forces":
            acc = torch.zeros((x.shape[0], 4), dtype=torch.float64, device=x.device)
            acc[:, :3] = a
            return dict(accel=acc, codes=None, sorted=None, index=None, layers=None)
        results.append((_rows(x, m), _rows(v, None)))
    return results if kind == "stream" else dict(pm=results[0][0], vr=results[0][1])

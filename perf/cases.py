"""What a user of this package has it do, as timed cases through the public entry points.

`listed()` gives the named cases, `draw(rng)` more of the same ranges, `prepare(case, seed)`
what a program holds before the call, `run(state)` one pass, `work(case)` the bytes and
operations a pass cannot do without, and `exact(case, seed)` a 64-bit answer where there is one
(the voxel render; a Monte Carlo tally is a sample of its packets, not a value to be computed).

The seed picks the packet stream (and the optics of a batch, the vessels or the spheres of a
scene), so another seed is another simulation of the same size.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from signedmcrt_b200 import kernels, presets as P, scene as S
from signedmcrt_b200.autograd import layered_groups, transport
from signedmcrt_b200.config import DetectorCfg
from signedmcrt_b200.scene import FlatScene
from signedmcrt_b200.transport import Batch, Transport, render, render_device

COUNTERS = ("packets", "sdf_evals", "voxel_segments", "trace_steps", "scatters", "fresnel_events", "reflections",
            "rng_draws", "kills_error", "kills_step_cap")

# Work of one packet by scene: (path length in cm inside the grid, sphere-tracing steps, flop of all but the
# voxel segments), from the event counters of the scenes and the source formulas; a voxel segment is 12 flop.
PER_PACKET = {"box_slab": (1.96, 64, 7000.0), "sphere_water": (3.50, 178, 25700.0), "layered_vessels": (0.65, 116, 47000.0),
              "test_egg": (0.74, 44, 9400.0), "sphere_scene": (1.77, 90, 115000.0)}
PER_PACKET_WEIGHT = {"box_slab": (2.40, 73, 8100.0), "sphere_water": (1.33, 55, 7700.0),
                     "layered_vessels": (0.044, 37, 15100.0), "test_egg": (0.80, 49, 10600.0)}
HALF = {"box_slab": (1.0, 1.0, 1.0), "sphere_water": (2.0, 2.0, 2.0), "layered_vessels": (1.0, 1.0, 0.605),
        "test_egg": (4.0, 4.0, 4.0), "sphere_scene": (1.0, 1.0, 1.0)}


def case(name, do, scene, packets, grid, **more):
    nx, ny, nz = grid
    c = {"name": name, "do": do, "scene": scene, "packets": packets, "nx": nx, "ny": ny, "nz": nz,
         "kernel": "pathlength", "precision": "fp32"}
    c.update(more)
    return c


def listed():
    return [
        # a short call on a small grid, as in a fit or an interactive program: latency and launches count
        case("box_short", "run", "box_slab", 1000, (20, 20, 20)),
        # the benchmark's small slab at its full size, tallies to host memory
        case("box_slab", "run", "box_slab", 1000000, (100, 100, 100), pinned=True),
        # the benchmark's curved-surface scene on its full grid, tallies kept on the device (a share of a long run)
        case("sphere_water", "device", "sphere_water", 4000000, (200, 200, 200)),
        # layered tissue with vessels and ten annular detectors on its full grid
        case("layered_vessels", "device", "layered_vessels", 2000000, (150, 150, 150)),
        # implicit capture with roulette (weight_scatter)
        case("sphere_weight", "device", "sphere_water", 1000000, (200, 200, 200), kernel="weight"),
        # the accuracy mode: FP64 transport
        case("sphere_fp64", "device", "sphere_water", 300000, (200, 200, 200), precision="fp64"),
        # a table of simulations over optical properties in one launch
        case("batch", "batch", "box_slab", 100000, (64, 64, 64), instances=24),
        # a training step on optical properties: forward and gradient
        case("adjoint", "adjoint", "layered_vessels", 300000, (50, 50, 50)),
        # fluence with its standard error per voxel
        case("moments", "moments", "layered_vessels", 200000, (150, 150, 150)),
        # a whole program call: scene with modifiers and a model's set-up, transport, normalisation; ragged grid
        case("egg_call", "call", "test_egg", 200000, (101, 77, 53)),
        # a scene too large for the parameter block (40 spheres), non-scattering
        case("sphere_scene", "device", "sphere_scene", 20000, (200, 200, 200), spheres=40),
        # the geometry rendered to voxels in FP64
        case("render", "render", "layered_vessels", 0, (256, 256, 256), precision="fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    return tuple(_log(rng, lo, hi) for _ in range(3))


def draw(rng):
    """One more case of the listed kinds, sizes over their whole range (odd ones among them)."""
    kind = rng.choice(["run", "run", "device", "device", "device", "weight", "fp64", "batch", "adjoint", "moments",
                       "call", "sphere_scene", "render"])
    scene = rng.choice(["box_slab", "sphere_water", "layered_vessels"])
    if kind == "run":
        c = case("", "run", scene, _log(rng, 500, 600000), _grid(rng, 16, 160), pinned=rng.random() < 0.5)
    elif kind == "device":
        c = case("", "device", scene, _log(rng, 20000, 2000000), _grid(rng, 40, 200))
    elif kind == "weight":
        c = case("", "device", scene, _log(rng, 20000, 1000000), _grid(rng, 40, 200), kernel="weight")
    elif kind == "fp64":
        c = case("", "device", scene, _log(rng, 5000, 250000), _grid(rng, 40, 200), precision="fp64")
    elif kind == "batch":
        c = case("", "batch", "box_slab", _log(rng, 10000, 80000), _grid(rng, 24, 64), instances=_log(rng, 2, 40))
    elif kind == "adjoint":
        c = case("", "adjoint", "layered_vessels", _log(rng, 10000, 300000), _grid(rng, 24, 80))
    elif kind == "moments":
        c = case("", "moments", scene, _log(rng, 10000, 200000), _grid(rng, 40, 150))
    elif kind == "call":
        c = case("", "call", rng.choice(["test_egg", "box_slab", "layered_vessels"]), _log(rng, 10000, 300000),
                 _grid(rng, 32, 128))
    elif kind == "sphere_scene":
        c = case("", "device", "sphere_scene", _log(rng, 2000, 20000), _grid(rng, 50, 200), spheres=_log(rng, 10, 60))
    else:
        c = case("", "render", "layered_vessels", 0, _grid(rng, 50, 300), precision=rng.choice(["fp64", "fp32"]),
                 host=rng.random() < 0.3)
    del c["name"]
    return c


def _scene(case, seed):
    name = case["scene"]
    if name == "test_egg":
        return P.setup_egg()
    if name == "sphere_scene":
        return P.setup_sphere_scene(case["spheres"], seed)
    if name == "layered_vessels" and case["do"] == "render":
        return P.layered_vessels(seed=seed)
    return {"box_slab": P.box_slab, "sphere_water": P.sphere_water, "layered_vessels": P.layered_vessels}[name]()


def _settings(case, seed):
    name = case["scene"]
    if name == "test_egg":
        # a pencil beam from above onto the egg, a circle detector under it
        st = P.benchmark_settings("box_slab")
        st.geometry.geom_name = name
        st.source.position = (0.0, 0.0, 3.9)
        st.detectors = [DetectorCfg("circle", position=(0.0, 0.0, -4.0), direction=(0.0, 0.0, -1.0), layer=4,
                                    radius1=4.0, nbins=50, maxval=4.0)]
    else:
        st = P.benchmark_settings(name)
    g = st.grid
    g.nxg, g.nyg, g.nzg = case["nx"], case["ny"], case["nz"]
    g.xmax, g.ymax, g.zmax = HALF[name] if name != "layered_vessels" else (1.0, 1.0, 0.5 * sum(P.LAYER_THICK))
    st.source.nphotons = case["packets"]
    st.simulation.iseed = seed
    st.output.render_geom = False
    return st


def _extent(seed):
    """Half-widths of a render: around the scene's own, as a user zooms."""
    return tuple(e * f for e, f in zip((1.0, 1.0, 0.7), np.random.default_rng(seed).uniform(0.8, 1.2, 3).tolist()))


def prepare(case, seed):
    do = case["do"]
    seed = 1000003 * int(seed) + 17
    s = {"case": case, "do": do, "seed": seed}
    if do == "render":
        s["flat"] = FlatScene(_scene(case, seed))
        s["samples"] = (case["nx"], case["ny"], case["nz"])
        s["extent"] = _extent(seed)
        s["image"] = torch.empty(case["nx"] * case["ny"] * case["nz"], dtype=torch.float32, device="cuda")
        return s
    st = s["settings"] = _settings(case, seed)
    if do == "call":
        return s
    if do == "adjoint":
        s["scene_fn"], s["groups"] = layered_groups()
        s["params"] = torch.tensor([[5.0, 50.0, 0.9], [1.0, 100.0, 0.8], [0.3, 50.0, 0.9], [0.1, 30.0, 0.9],
                                    [0.01, 0.1, 0.5]], dtype=torch.float64)
        gen = torch.Generator(device="cuda").manual_seed(seed % (1 << 31))
        s["target"] = torch.rand((case["nx"], case["ny"], case["nz"]), generator=gen, device="cuda",
                                 dtype=torch.float64)
        return s
    flat = FlatScene(_scene(case, seed))
    if do == "batch":
        n = case["instances"]
        rng = np.random.default_rng(seed)
        optics = np.zeros((n, 2, 4))
        optics[:, 0] = np.stack([rng.uniform(1.0, 100.0, n), rng.uniform(0.01, 1.0, n), rng.uniform(0.7, 0.95, n),
                                 rng.uniform(1.33, 1.45, n)], axis=1)
        optics[:, 1] = (0.0, 0.0, 0.0, 1.0)
        s["counts"] = np.maximum(1, np.round(case["packets"] * 10.0 ** rng.uniform(-1.0, 0.0, n))).astype(np.int64)
        s["seeds"] = (seed + np.arange(n)).astype(np.uint64)
        s["batch"] = Batch(flat, st, n, optics=optics, precision=case["precision"])
        s["host"] = torch.empty(n * s["batch"].ncell, dtype=torch.float64, pin_memory=True).numpy()
        return s
    stream = torch.cuda.current_stream().cuda_stream if do == "device" else None
    tr = s["tr"] = Transport(flat, st, kernel=case["kernel"], precision=case["precision"], stream=stream,
                             variance=do == "moments")
    if do == "device":
        s["jmean"] = torch.zeros(tr.ncell, dtype=torch.float64, device="cuda")
        s["bins"] = torch.zeros(max(tr.nbins, 1), dtype=torch.float64, device="cuda")
    elif do == "run" and case.get("pinned"):
        s["host"] = torch.empty(tr.ncell, dtype=torch.float64, pin_memory=True).numpy()
    return s


def run(state):
    case, do = state["case"], state["do"]
    n, seed = case["packets"], state["seed"]
    if do == "run":
        r = state["tr"].run(n, seed, jmean_out=state.get("host"))
        return {"jmean": r.jmean, "bins": r.bins, "counts": [int(r.stats[k]) for k in COUNTERS],
                "nscatt": float(r.stats["nscatt"])}
    if do == "device":
        state["jmean"].zero_()
        state["bins"].zero_()
        tr = state["tr"]
        tr.run_device(0, n, seed, state["jmean"].data_ptr(), state["bins"].data_ptr() if tr.nbins else None)
        return {"jmean": state["jmean"], "bins": state["bins"]}
    if do == "moments":
        r = state["tr"].run_moments(n, seed)
        return {"jmean": r.jmean, "jmean2": r.jmean2, "bins": r.bins, "counts": [int(r.stats[k]) for k in COUNTERS]}
    if do == "batch":
        state["batch"].launch(state["counts"], state["seeds"], use_graph=True)
        jm, bins, per, total = state["batch"].wait(jmean_out=state["host"])
        return {"jmean": jm, "per": [[int(p["packets"]), int(p["rng_draws"]), int(p["nscatt"])] for p in per[:16]],
                "counts": [int(total[k]) for k in COUNTERS]}
    if do == "adjoint":
        params = state["params"].clone().requires_grad_(True)
        phi, det = transport(params, state["scene_fn"], state["settings"], state["groups"], n, seed)
        loss = (phi * state["target"]).sum() + det.sum()
        loss.backward()
        return {"phi": phi.detach(), "det": det.detach(), "grad": params.grad}
    if do == "call":
        r = kernels.run_kernel(state["settings"], case["kernel"], write=False, verbose=False)
        return {"jmean": r.jmean, "fluence": r.fluence, "bins": r.bins, "nscatt": float(r.nscatt)}
    if case.get("host"):
        return {"image": render(state["flat"], state["samples"], state["extent"], precision=case["precision"])}
    render_device(state["flat"], state["samples"], state["extent"], state["image"].data_ptr(),
                  precision=case["precision"], stream=torch.cuda.current_stream().cuda_stream)
    return {"image": state["image"]}


def work(case):
    """Outputs written once, and the flop of the algorithm's own events for the case's packets (or voxels)."""
    do, scene = case["do"], case["scene"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if do == "render":  # 364 flop a voxel of the layered scene's 8 regions, 4 bytes written
        return {"bytes": 4.0 * cells, "flops": 364.0 * cells}
    path, steps, flop = (PER_PACKET_WEIGHT if case["kernel"] == "weight" else PER_PACKET)[scene]
    # a path of random direction crosses |dx| / voxel faces on each axis, half the length on average
    faces = sum(0.5 * path * n / (2.0 * h) for n, h in zip((case["nx"], case["ny"], case["nz"]), HALF[scene]))
    per = flop + 12.0 * (steps + faces)
    packets = float(case["packets"])
    if do == "batch":
        packets = 0.39 * packets * case["instances"]  # the mean of 10^U(-1, 0)
        cells *= case["instances"]
    if do == "adjoint":
        per, cells = 3.0 * per, 1.5 * cells  # forward, then each packet twice; FP32 weights read
    if do == "moments":
        cells *= 2
    return {"bytes": 8.0 * cells, "flops": packets * per}


def exact(case, seed):
    """The render in 64 bits: the minimum over the scene's boxes and capsules."""
    if case["do"] != "render":
        return None
    seed = 1000003 * int(seed) + 17
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ns = (case["nx"], case["ny"], case["nz"])
    axes = []
    for n, ext in zip(ns, _extent(seed)):
        half = (n + 1) // 2
        axes.append((torch.arange(1, n + 1, dtype=torch.float64, device=dev) - half) * (ext / half))
    x, y, z = axes[0][None, None, :], axes[1][None, :, None], axes[2][:, None, None]
    best = torch.full((ns[2], ns[1], ns[0]), math.inf, dtype=torch.float64, device=dev)
    for ent in P.layered_vessels(seed=seed):
        m, q = ent.transform, ent.params
        p = [m[0, j] * x + m[1, j] * y + m[2, j] * z + m[3, j] for j in range(3)]
        if ent.kind == S.box((1, 1, 1), ent.opt, 1).kind:
            d = [p[j].abs() - q[j] for j in range(3)]
            out = sum(v.clamp(min=0.0) ** 2 for v in d).sqrt()
            v = out + torch.maximum(d[0], torch.maximum(d[1], d[2])).clamp(max=0.0)
        else:
            ba = [q[3 + j] - q[j] for j in range(3)]
            pa = [p[j] - q[j] for j in range(3)]
            h = (sum(a * b for a, b in zip(pa, ba)) / sum(b * b for b in ba)).clamp(0.0, 1.0)
            v = sum((a - b * h) ** 2 for a, b in zip(pa, ba)).sqrt() - q[6]
        best = torch.minimum(best, v)
    image = best.reshape(-1)
    if case.get("host"):  # the host call's shape: Fortran order
        return {"image": best.permute(2, 1, 0).cpu().numpy()}
    return {"image": image}

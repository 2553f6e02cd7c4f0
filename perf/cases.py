"""The work that users of this framework have it do, as measurable cases.

Every case is a dict of plain values. `kind` says which public entry points
it goes through:

* "sim": one scene (`Simulation`). A pass uploads a state of the flow, runs
  whole frames (`frame`, the reference's `EZ_EXAMPLE_SIM::step`) or fixed-dt
  sub-steps (`begin_frame` + `sub_step`), and reads positions, velocities and
  the solver's densities back. The scenes are the seeded dam breaks of
  `emerald_b200.workloads` (support = dx, three boundary rows).
* "batch": many scenes of uneven size advanced together (`Batch`).
* "served": a burst of requests through the request loop (`Server`).
* "ops": the z-order sort, the neighbour search and the sph_common sums as
  single device functions, as a caller of the reference's own pipeline
  strings them together.

Sizes: a scene holds from about a thousand particles (the smallest of the
batched workload) to 1,048,576 (the precision configuration); the batched and
served scenes are log-uniform in size, as in `workloads`.
"""
import ctypes
import math

import numpy as np
import torch

import emerald_b200 as E
from emerald_b200 import workloads as W

F = np.float32
METHODS = ("dfsph_p", "iisph", "iisph_ap", "iisph_pseudo_ap", "pcisph")


def listed():
    return [
        # the smallest request of the served workload, its first frames from
        # rest: launch latency
        dict(name="dfsph_frames_2k", kind="sim", method="dfsph_p", nx=48, ny=43, warm=0, frames=2,
             steps=0, compensated=False),
        # the plain IISPH configuration: 128 x 128 block, fixed dt = 1e-4 s
        dict(name="iisph_fixed_dt_16k", kind="sim", method="iisph", nx=128, ny=128, warm=0,
             frames=0, steps=10, compensated=False),
        # an ordinary scene of odd size, in motion
        dict(name="dfsph_frames_37k_odd", kind="sim", method="dfsph_p", nx=173, ny=211, warm=2,
             frames=3, steps=0, compensated=False),
        # the other two implicit solvers, at ordinary sizes
        dict(name="iisph_ap_frames_65k", kind="sim", method="iisph_ap", nx=256, ny=256, warm=2,
             frames=2, steps=0, compensated=False),
        dict(name="pseudo_ap_frames_56k_odd", kind="sim", method="iisph_pseudo_ap", nx=301,
             ny=187, warm=2, frames=2, steps=0, compensated=False),
        # the headline scene of the benchmark, over the sub-steps it times
        dict(name="dfsph_frames_262k", kind="sim", method="dfsph_p", nx=512, ny=512, warm=2,
             frames=3, steps=0, compensated=False),
        # the same block under PCISPH (four fixed sub-steps a frame)
        dict(name="pcisph_frame_262k", kind="sim", method="pcisph", nx=512, ny=512, warm=1,
             frames=1, steps=0, compensated=False),
        # FP64 positions and Kahan-compensated sums
        dict(name="dfsph_compensated_262k", kind="sim", method="dfsph_p", nx=512, ny=512, warm=2,
             frames=2, steps=0, compensated=True),
        # the largest scene of the configurations
        dict(name="dfsph_frames_1m", kind="sim", method="dfsph_p", nx=1024, ny=1024, warm=2,
             frames=3, steps=0, compensated=False),
        # the batched workload (IISPH, 200 iterations at most), 32 scenes of it
        dict(name="batch_iisph_32", kind="batch", method="iisph", scenes=32, lo=1024, hi=65536,
             steps=6, scene_set=2024),
        # a burst of the served workload, every request in one lane's batch
        dict(name="served_dfsph_16", kind="served", method="dfsph_p", requests=16, lo=2048,
             hi=131072, steps_lo=8, steps_hi=24, scene_set=77),
        # the device functions of the reference's pipeline, one after the other
        dict(name="device_functions_100k", kind="ops", nx=317, ny=316),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block(rng, lo, hi):
    n = _log_uniform(rng, lo, hi)
    aspect = rng.uniform(0.25, 4.0)
    nx = max(8, int(round(math.sqrt(n * aspect))))
    return nx, max(8, int(round(n / nx)))


def draw(rng):
    """A case of the listed ones' ranges: all kinds, methods and both
    precision modes, block aspect 1:4 to 4:1, sizes log-uniform."""
    kind = rng.choices(("sim", "batch", "served", "ops"), (9, 1, 1, 1))[0]
    if kind == "batch":
        return dict(kind=kind, method=rng.choice(("iisph", "dfsph_p")), scenes=rng.randint(4, 32),
                    lo=1024, hi=int(_log_uniform(rng, 4096, 65536)), steps=rng.randint(2, 6),
                    scene_set=rng.randint(1, 9999))
    if kind == "served":
        return dict(kind=kind, method="dfsph_p", requests=rng.randint(3, 16), lo=2048,
                    hi=int(_log_uniform(rng, 8192, 131072)), steps_lo=8, steps_hi=24,
                    scene_set=rng.randint(1, 9999))
    if kind == "ops":
        nx, ny = _block(rng, 1024, 262144)
        return dict(kind=kind, nx=nx, ny=ny)
    method = rng.choices(METHODS, (6, 3, 1, 1, 1))[0]
    compensated = rng.random() < 0.15
    nx, ny = _block(rng, 1024, 1000000 if method == "dfsph_p" and not compensated else 262144)
    fixed = rng.random() < 0.25
    return dict(kind=kind, method=method, nx=nx, ny=ny, warm=rng.randint(0, 2),
                frames=0 if fixed else rng.randint(1, 3), steps=rng.randint(1, 6) if fixed else 0,
                compensated=compensated)


# ------------------------------------------------------------------ prepare


def _pinned(n):
    """A page-locked float32 (n, 2) host array."""
    return torch.zeros((n, 2), dtype=torch.float32, pin_memory=True).numpy()


def _prepare_sim(case, seed):
    over = dict(precision=E.PRECISION_COMPENSATED) if case["compensated"] else {}
    scene = W.scene_for(case["nx"], case["ny"], 1 + seed % 1000003, **over)
    sim = E.Simulation.from_block_scene(scene)
    # a flow in motion, reached by the frames before the measured ones
    for _ in range(case["warm"]):
        sim.frame(case["method"])
    x, v, x_out, v_out = (_pinned(sim.n) for _ in range(4))
    sim.state(x, v)
    return dict(case=case, sim=sim, x=x, v=v, x_out=x_out, v_out=v_out)


def _prepare_batch(case, seed):
    # sizes and shapes are the case's, the jitter of the positions the seed's
    specs = W.batched_specs(case["scenes"], case["lo"], case["hi"], seed=case["scene_set"])
    scenes = [W.scene_for(s["nx"], s["ny"], s["seed"] + seed % 1000003, s["viscosity"],
                          iisph_max_pressure_iterations=200) for s in specs]
    pad = 128  # a scene starts on a tile of 128 particles
    fluid = sum(-(-len(s.fluid) // pad) * pad for s in scenes)
    solid = sum(-(-len(s.solid) // pad) * pad for s in scenes)
    batch = E.Batch(fluid, solid, len(scenes))
    ids = [batch.add_block_scene(s) for s in scenes]
    return dict(case=case, batch=batch, ids=ids, x=[s.fluid for s in scenes],
                v=[np.zeros_like(s.fluid) for s in scenes])


def _prepare_served(case, seed):
    reqs = W.serving_requests(case["requests"], lo=case["lo"], hi=case["hi"],
                              steps_lo=case["steps_lo"], steps_hi=case["steps_hi"],
                              seed=case["scene_set"])
    scenes = [W.scene_for(r["nx"], r["ny"], r["seed"] + seed % 1000003) for r in reqs]
    server = E.Server(6e9, method=case["method"], max_scenes=64, lanes=1)
    return dict(case=case, server=server, scenes=scenes, steps=[r["substeps"] for r in reqs])


def _prepare_ops(case, seed):
    scene = W.scene_for(case["nx"], case["ny"], 1 + seed % 1000003)
    n = len(scene.fluid)
    cuda = dict(device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(mean, sd, *shape):
        return mean + sd * torch.randn(*shape, generator=gen, **cuda)

    st = dict(case=case, n=n, support=float(scene.support), cell=float(F(2) * scene.support),
              rho0=1000.0, dt=5e-4)
    st["x"] = torch.from_numpy(scene.fluid).cuda()
    st["v"] = normal(0.0, 0.3, n, 2)
    st["p"] = normal(0.0, 500.0, n).abs()
    st["vol"] = (float(scene.params.mass_per_particle) / 1000.0) * torch.ones(n, **cuda)
    st["gc"] = torch.zeros(n, 2, dtype=torch.int32, **cuda)
    st["z"] = torch.zeros(n, dtype=torch.int64, **cuda)
    st["pairs"] = torch.zeros(n, 2, dtype=torch.int64, **cuda)
    st["block_of"] = torch.zeros(n, dtype=torch.int32, **cuda)
    st["blocks"] = torch.zeros(n, 2, dtype=torch.int64, **cuda)
    st["counts"] = torch.zeros(n, dtype=torch.uint8, **cuda)
    st["idx"] = torch.zeros(n, 64, dtype=torch.int64, **cuda)
    st["dist"] = torch.zeros(n, 64, **cuda)
    st["vec"] = torch.zeros(n, 64, 2, **cuda)
    st["w"] = torch.zeros(n, 64, **cuda)
    st["gw"] = torch.zeros(n, 64, 2, **cuda)
    st["rho"] = torch.zeros(n, **cuda)
    st["div"] = torch.zeros(n, **cuda)
    st["v_out"] = torch.zeros(n, 2, **cuda)
    # no boundary particles: their lists are empty
    st["none"] = torch.zeros(n, dtype=torch.uint8, **cuda)
    size = ctypes.c_size_t()
    _ok(E.lib.emerald_index_pairs_workspace(n, ctypes.byref(size)))
    st["work"] = torch.empty(max(size.value, 1), dtype=torch.uint8, **cuda)
    handle = ctypes.c_void_p()
    _ok(E.lib.emerald_block_map_create(ctypes.byref(handle)))
    st["map"] = _BlockMap(handle)
    return st


class _BlockMap:
    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        E.lib.emerald_block_map_destroy(self.handle)


def _ok(rc):
    if rc != 0:
        raise RuntimeError("status %d: %s" % (rc, E.lib.emerald_last_error().decode()))


def prepare(case, seed):
    return dict(sim=_prepare_sim, batch=_prepare_batch, served=_prepare_served,
                ops=_prepare_ops)[case["kind"]](case, seed)


# ---------------------------------------------------------------------- run


def _run_sim(st):
    case, sim = st["case"], st["sim"]
    sim.set_state(st["x"], st["v"])
    for _ in range(case["frames"]):
        sim.frame(case["method"])
    if case["steps"]:
        dt = 1e-4
        sim.begin_frame(case["method"])
        for k in range(case["steps"]):
            sim.sub_step(case["method"], k * dt, dt)
    x, v = sim.state(st["x_out"], st["v_out"])
    return x, v, sim.array("densities")


def _run_batch(st):
    batch = st["batch"]
    for sid, x, v in zip(st["ids"], st["x"], st["v"]):
        batch.set_state(sid, x, v)
    batch.step(st["case"]["method"], st["case"]["steps"])
    return [batch.state(sid) for sid in st["ids"]]


def _run_served(st):
    server = st["server"]
    ids = [server.submit_block_scene(s, k) for s, k in zip(st["scenes"], st["steps"])]
    return [server.wait(r)[:2] for r in ids]


def _run_ops(st):
    L, n = E.lib, st["n"]
    h, rho0, dt = st["support"], st["rho0"], st["dt"]
    stream = torch.cuda.current_stream().cuda_stream
    p = {k: t.data_ptr() for k, t in st.items() if isinstance(t, torch.Tensor)}
    _ok(L.emerald_compute_grid_coords(n, st["cell"], 0.0, 0.0, p["gc"], p["x"], stream))
    _ok(L.emerald_compute_z_indices(n, p["z"], p["gc"], stream))
    _ok(L.emerald_compute_index_pairs(n, p["pairs"], p["z"], stream))
    _ok(L.emerald_sort_index_pairs(n, p["pairs"], p["work"], st["work"].numel(), stream))
    _ok(L.emerald_compute_block_indices(n, p["block_of"], p["pairs"], p["work"],
                                        st["work"].numel(), stream))
    # the reference sizes its block array here, on the host
    blocks = int(st["block_of"][-1]) + 1
    _ok(L.emerald_fill_blocks(n, p["blocks"], p["block_of"], stream))
    bmap = st["map"].handle
    _ok(L.emerald_create_block_map(blocks, bmap, p["blocks"], p["pairs"], stream))
    _ok(L.emerald_create_regular_neighborhoods(n, st["cell"], p["counts"], p["idx"], p["dist"],
                                               p["vec"], p["x"], p["gc"], p["x"], p["pairs"], bmap,
                                               stream))
    _ok(L.emerald_compute_neighbor_kernels(n, h, p["w"], p["counts"], p["dist"], stream))
    _ok(L.emerald_compute_neighbor_kernel_gradients(n, h, p["gw"], p["counts"], p["vec"], stream))
    fluid = E.Neighborhood(p["counts"], p["idx"], p["dist"], p["vec"], p["w"], p["gw"])
    solid = E.Neighborhood(p["none"], p["idx"], p["dist"], p["vec"], p["w"], p["gw"])
    _ok(L.emerald_compute_densities(n, h, rho0, p["rho"], p["vol"], fluid, p["vol"], solid, stream))
    _ok(L.emerald_compute_divergences(n, rho0, p["div"], p["vol"], p["v"], fluid, p["vol"],
                                      p["v"], solid, stream))
    st["v_out"].copy_(st["v"])
    _ok(L.emerald_apply_pressures_in_place(n, dt, rho0, p["v_out"], p["rho"], p["p"], p["vol"],
                                           fluid, p["vol"], solid, stream))
    return [st[k] for k in ("counts", "idx", "w", "gw", "rho", "div", "v_out")]


def run(state):
    return dict(sim=_run_sim, batch=_run_batch, served=_run_served,
                ops=_run_ops)[state["case"]["kind"]](state)


# --------------------------------------------------------------------- work


def _particles(case):
    """Particles and the sub-steps each takes at least, per scene."""
    if case["kind"] in ("sim", "ops"):
        n = case["nx"] * case["ny"]
        per_frame = {"iisph": 6, "pcisph": 4}.get(case.get("method"), 4)
        return [(n, case.get("frames", 0) * per_frame + case.get("steps", 0))]
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    count = case.get("scenes") or case["requests"]
    mean = (math.exp(hi) - math.exp(lo)) / (hi - lo)  # of a log-uniform size
    steps = case["steps"] if case["kind"] == "batch" else (case["steps_lo"] + case["steps_hi"]) / 2
    return [(mean, steps)] * count


def work(case):
    """Bytes: positions and velocities in and out once (a pass starts and ends
    with them), and the densities out; for the device functions their inputs
    and the outputs up to each particle's count. Flops: about 11 neighbours a
    particle, 40 operations to find and weigh each, and two solver iterations
    of 20 operations a neighbour, in every sub-step."""
    bytes_, flops = 0.0, 0.0
    for n, steps in _particles(case):
        if case["kind"] == "ops":
            bytes_ += n * (8 + 8 + 4 + 4 + 1 + 11 * (8 + 4 + 8) + 4 + 4 + 8)
            flops += n * 11 * 60
        else:
            bytes_ += n * (16 + 16 + (4 if case["kind"] == "sim" else 0))
            flops += steps * n * 11 * 80
    return dict(bytes=bytes_, flops=flops)


# -------------------------------------------------------------------- exact


def _lists64(x, cell):
    """Neighbours within `cell` of each of the (n, 2) float64 points, ordered
    by (distance, index): (n, 64) indices, a mask, and vectors to them."""
    n = len(x)
    g = torch.floor(x / cell).long()
    g -= g.min(0).values - 1
    width = int(g[:, 0].max()) + 2
    key = g[:, 1] * width + g[:, 0]
    order = torch.argsort(key, stable=True)
    sorted_key = key[order]
    most = int(torch.unique_consecutive(sorted_key, return_counts=True)[1].max())
    cand = []
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            k = key + dy * width + dx
            at = torch.searchsorted(sorted_key, k)[:, None] + torch.arange(most, device=x.device)
            inside = at < n
            at = at.clamp(max=n - 1)
            inside &= sorted_key[at] == k[:, None]
            cand.append(torch.where(inside, order[at], -1))
    cand = torch.cat(cand, 1)
    cand = torch.sort(cand, dim=1).values  # ties of the distance go to the lower index
    vec = x[cand.clamp(min=0)] - x[:, None]
    dist = vec.square().sum(2).sqrt()
    own = torch.arange(n, device=x.device)[:, None]
    dist = torch.where((cand >= 0) & (cand != own) & (dist < cell), dist, math.inf)
    dist, at = torch.sort(dist, dim=1, stable=True)
    dist, at = dist[:, :64], at[:, :64]
    if dist.shape[1] < 64:
        fill = 64 - dist.shape[1]
        dist = torch.nn.functional.pad(dist, (0, fill), value=math.inf)
        at = torch.nn.functional.pad(at, (0, fill))
    live = torch.isfinite(dist)
    idx = cand.gather(1, at).clamp(min=0)
    vec = torch.where(live[..., None], x[idx] - x[:, None], 0.0)
    return idx, live, torch.where(live, dist, 0.0), vec


def _exact_ops(case, seed):
    st = _prepare_ops(case, seed)
    h, rho0, dt = st["support"], st["rho0"], st["dt"]
    x, v, p, vol = (st[k].double() for k in ("x", "v", "p", "vol"))
    idx, live, dist, vec = _lists64(x, st["cell"])
    q = dist / h
    k = math.pi * h ** 3
    w = torch.where(q <= 1, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * (2 - q) ** 3) / k
    w = torch.where(live, w, 0.0)
    dw = torch.where(q <= 1, -3 * q + 2.25 * q ** 2, -0.75 * (2 - q) ** 2) / (k * h)
    unit = -vec / torch.where(live, dist, 1.0)[..., None]
    gw = torch.where(live[..., None], unit * dw[..., None], 0.0)
    mass = rho0 * vol
    rho = mass / k + (w * mass[idx]).sum(1)
    div = (mass[idx] * ((v[:, None] - v[idx]) * gw).sum(2)).sum(1)
    c = p / rho ** 2
    acc = -(mass[idx] * (c[:, None] + c[idx]))[..., None] * gw
    return [None, None, w, gw, rho, div, v + dt * acc.sum(1)]


def exact(case, seed):
    """The device functions have a value in 64 bits. A stepped scene has none:
    its solver loops stop where an error of 32 bits passes a threshold, so
    64 bits would stop at other iterations."""
    return _exact_ops(case, seed) if case["kind"] == "ops" else None

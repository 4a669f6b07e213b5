"""Timed workloads of the mechanics library, through its public entry points.

Every case is a piece of a simulation program that keeps its agents in a
`Simulation` (or, for the binning call, in its own device buffers). The agents
come from the seeded generators of `paraphysicell_b200.workloads`; the sizes
are those of the benchmark, the tests and the reference's README (900, 14,300
and 88,700 agents, ensembles, one million agents), and odd ones between them.

`listed()` gives the fixed cases, `draw(rng)` one more of the same ranges,
`prepare(case, seed)` what a program has in hand before the call, `run(state)`
one pass, `work(case)` the bytes and operations a pass cannot do without and
`exact(case, seed)` the result of a pass in plain 64-bit torch arithmetic.
"""
import ctypes
import math

import numpy as np
import torch

from paraphysicell_b200 import abi, device
from paraphysicell_b200 import workloads as wl

IN_FIELDS = ("positions", "previous_velocities")
OUT_FIELDS = ("positions", "previous_velocities", "simple_pressure")
INTERVAL = 60  # mechanics steps (0.1 min) in a phenotype step (6 min), the reference's default


def listed():
    return [
        # custom rules on the host every step, smallest model of the README: launches and latency
        {"name": "loop_2d_900", "kind": "host_loop", "config": 1, "agents": 900, "steps": 1, "fp32": False},
        # the same model left to run for a phenotype interval, then saved
        {"name": "run_2d_900", "kind": "run", "config": 1, "agents": 900, "steps": INTERVAL, "fp32": False},
        # two cell types in a ball, walls on: the FP64 drop-in at the README's middle size
        {"name": "run_walls_14k", "kind": "run", "config": 2, "agents": 14300, "steps": INTERVAL, "fp32": False},
        # a caller of the reference's solver functions, one by one, every step
        {"name": "entry_points_14k", "kind": "entry_points", "config": 2, "agents": 14300, "steps": 1, "fp32": False},
        # the benchmark's default: three types, 20 % of the agents with springs
        {"name": "run_springs_88k", "kind": "run", "config": 3, "agents": 88700, "steps": INTERVAL, "fp32": False},
        # the same with the host's copy authoritative: positions up, one step, results down
        {"name": "loop_springs_88k", "kind": "host_loop", "config": 3, "agents": 88700, "steps": 1, "fp32": False},
        # the same in the FP32-force form
        {"name": "run_fp32_88k", "kind": "run", "config": 3, "agents": 88700, "steps": INTERVAL, "fp32": True},
        # spring attachment and detachment rates on: neighbour lists and stochastic springs every step
        {"name": "spring_rates_88k", "kind": "spring_rates", "config": 3, "agents": 88700, "steps": 10, "fp32": False},
        # a parameter study: independent replicates of 500 to 50,000 agents in one state
        {"name": "ensemble_96", "kind": "ensemble", "config": 4, "agents": 96, "steps": INTERVAL, "fp32": False},
        # the largest: one million agents that divide and die every step
        {"name": "divide_1m", "kind": "divide", "config": 5, "agents": 1000000, "steps": 10, "fp32": False},
        # migrating, chemotactic cells that phagocytose, attack and fuse: a full model's mechanics loop
        {"name": "immune_20k", "kind": "immune", "config": 2, "agents": 20011, "steps": 20, "fp32": False},
        # binning of a caller's own device positions, without a state or an allocation
        {"name": "bins_100k", "kind": "bins", "config": 3, "agents": 100003, "steps": 1, "fp32": False},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host_loop", "run", "run", "run", "entry_points", "spring_rates", "ensemble", "divide",
                       "immune", "bins"])
    fp32 = False
    if kind in ("host_loop", "run"):
        config = rng.choice([1, 2, 3])
        agents = _log_uniform(rng, 300, 15000) if config == 1 else _log_uniform(rng, 2000, 90000)
        fp32 = rng.random() < 0.25
        steps = 1 if kind == "host_loop" else rng.randint(7, INTERVAL)
    elif kind == "entry_points":
        config, agents, steps = 2, _log_uniform(rng, 1500, 90000), 1
    elif kind == "spring_rates":
        config, agents, steps = 3, _log_uniform(rng, 3000, 90000), rng.randint(3, 10)
    elif kind == "ensemble":
        config, agents, steps = 4, rng.randint(5, 90), rng.randint(11, INTERVAL)
        fp32 = rng.random() < 0.25
    elif kind == "divide":
        config, agents, steps = 5, _log_uniform(rng, 60000, 950000), rng.randint(4, 10)
        fp32 = rng.random() < 0.25
    elif kind == "immune":
        config, agents, steps = 2, _log_uniform(rng, 2000, 60000), rng.randint(5, 20)
    else:
        config, agents, steps = rng.choice([1, 2, 3]), _log_uniform(rng, 900, 131000), 1
    return {"kind": kind, "config": config, "agents": agents, "steps": steps, "fp32": fp32}


# ---- inputs ------------------------------------------------------------------


def _make(case, seed):
    """(Mesh, Params, AgentArrays) of a case with one simulation, at the
    configuration's own density."""
    n, config = case["agents"], case["config"]
    if config == 1:
        # the 2-D model's density is 900 agents per 2000 x 2000 um
        half = max(60, int(round(1000.0 * math.sqrt(n / 900.0))))
        mesh, params, a = wl.config1(seed=seed, n=n)
        mesh = abi.Mesh.make(2, (-half, -half, -10), (half, half, 10))
        a.arrays["positions"][: 2 * n] *= half / 1000.0
        return mesh, params, a
    if config == 5:
        cap = int(n * 1.05) + 1024
        if n == 1000000:
            return wl.config5(seed=seed, n=n, capacity=cap)
        return wl.scaled(wl.config5, n, seed, capacity=cap)
    fn = {2: wl.config2, 3: wl.config3}[config]
    if (config, n) in ((2, 14300), (3, 88700)):
        return fn(seed=seed, n=n)
    return wl.scaled(fn, n, seed)


_NP = {np.dtype(np.float64): torch.float64, np.dtype(np.int32): torch.int32, np.dtype(np.int64): torch.int64,
       np.dtype(np.uint8): torch.uint8}


def _pinned(arr):
    """A page-locked copy of a host array (the array keeps its memory alive)."""
    t = torch.empty(max(arr.size, 1), dtype=_NP[arr.dtype], pin_memory=True)
    out = t.numpy()[: arr.size]
    out[:] = arr
    return out


def _pin(a, fields):
    for f in fields:
        a.arrays[f] = _pinned(a.arrays[f])


def _simulation(case, mesh, params, a, seed):
    sim = device.Simulation(mesh, params, a.capacity, seed=seed)
    if case["fp32"]:
        sim.set_precision(abi.PPC_FP32_FORCE)
    sim.upload(a)
    return sim


def prepare(case, seed):
    kind = case["kind"]
    if kind == "bins":
        mesh, params, a = _make(case, seed) if case["config"] != 3 else _bins_ball(case["agents"], seed)
        pos = torch.from_numpy(np.ascontiguousarray(a["positions"]).reshape(-1)).cuda()
        L = device.lib()
        L.ppc_bin_agents_noalloc.argtypes = [ctypes.POINTER(abi.Mesh), ctypes.c_void_p, ctypes.c_int32,
                                             ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        return {"kind": kind, "mesh": mesh, "pos": pos, "n": a.count, "lib": L,
                "counts": torch.empty(mesh.voxel_count(), dtype=torch.int32, device="cuda"),
                "agents": torch.empty(a.count, dtype=torch.int32, device="cuda")}
    if kind == "ensemble":
        meshes, params, sets = _ensemble(case["agents"], seed)
        sim = device.Simulation(meshes, params, [a.capacity for a in sets], seed=seed)
        if case["fp32"]:
            sim.set_precision(abi.PPC_FP32_FORCE)
        # every replicate's result lands in its part of one page-locked array per field
        total = sum(a.capacity for a in sets)
        whole = {f: torch.zeros(total * (1 if f == "simple_pressure" else 3), dtype=torch.float64,
                                pin_memory=True).numpy() for f in OUT_FIELDS}
        at = 0
        for r, a in enumerate(sets):
            sim.upload(a, r)
            for f in OUT_FIELDS:
                w = 1 if f == "simple_pressure" else 3
                a.arrays[f] = whole[f][at * w: (at + a.capacity) * w]
            at += a.capacity
        sim.update_mechanics_mesh()
        return {"kind": kind, "sim": sim, "sets": sets, "whole": whole, "steps": case["steps"]}

    mesh, params, a = _make(case, seed)
    state = {"kind": kind, "a": a, "steps": case["steps"]}
    if kind == "spring_rates":
        a.arrays["attachment_rate"][: a.count] = 0.8
        a.arrays["detachment_rate"][: a.count] = 0.3
        a.arrays["maximum_number_of_attachments"][: a.count] = 3
    if kind == "immune":
        fields = wl.interaction_fields(a, params.cell_definitions_count, seed + 1, scale=2e-4)
    state["sim"] = sim = _simulation(case, mesh, params, a, seed)
    if kind == "immune":
        state["fields"], state["motility"] = fields, _motility(a, params, seed + 2)
        state["gradients"] = _gradients(mesh, seed + 3)
        sim.upload_interactions(fields)
        sim.upload_motility(state["motility"])
        sim.upload_gradients(state["gradients"])
    sim.update_mechanics_mesh()
    _pin(a, OUT_FIELDS)
    return state


def _ensemble(replicates, seed):
    """wl.config4's replicates; their sizes follow from their number, the agents from the seed."""
    sizes = np.random.default_rng(replicates).uniform(math.log(500), math.log(50000), replicates)
    rng = np.random.default_rng(seed)
    meshes, sets = [], []
    for n in np.rint(np.exp(sizes)).astype(int):
        side = max(1, int(np.rint((8000.0 * n) ** (1.0 / 3.0))))
        a = abi.AgentArrays(int(n), 3, 1, int(n))
        a.arrays["positions"][:] = rng.uniform(0, side, size=3 * n)
        a.arrays["radius"][:] = rng.uniform(7.0, 10.0, n)
        meshes.append(abi.Mesh.make(3, (0, 0, 0), (side, side, side)))
        sets.append(a)
    return meshes, abi.Params.make(dt=0.1, ndefs=1, walls=False), sets


def _bins_ball(n, seed):
    """A ball at config 3's density in a cube that the call's voxel limit allows."""
    rng = np.random.default_rng(seed)
    radius = 1300.0 * (n / 88700.0) ** (1.0 / 3.0)
    half = 30 * int(math.ceil((radius + 60.0) / 30.0))
    a = abi.AgentArrays(n, 3, 1, n)
    d = rng.normal(size=(n, 3))
    d *= (radius * rng.random(n) ** (1.0 / 3.0) / np.linalg.norm(d, axis=1))[:, None]
    a.arrays["positions"][: 3 * n] = d.ravel()
    return abi.Mesh.make(3, (-half,) * 3, (half,) * 3), None, a


def _motility(a, params, seed):
    """30 % of the agents migrate at 0.2 to 1 um/min, half of them by chemotaxis."""
    rng = np.random.default_rng(seed)
    n = a.count
    m = abi.MotilityArrays(n, a.dims, restrict_per_agent=True, substrates=2)
    m["is_motile"][:] = rng.random(n) < 0.3
    m["persistence_time"][:] = rng.uniform(1.0, 15.0, n)
    m["migration_speed"][:] = rng.uniform(0.2, 1.0, n)
    m["migration_bias"][:] = rng.random(n)
    m["direction_rule"][:] = np.where(rng.random(n) < 0.5, abi.PPC_DIRECTION_CHEMOTAXIS, abi.PPC_DIRECTION_NONE)
    m["chemotaxis_index"][:] = rng.integers(0, 2, n)
    m["chemotaxis_direction"][:] = np.where(rng.random(n) < 0.5, 1.0, -1.0)
    m["chemotactic_sensitivities"][:] = rng.random((n, 2))
    return m


def _gradients(mesh, seed):
    rng = np.random.default_rng(seed)
    shape = (40, 40, 40)
    vox = 1
    for d in range(3):
        vox *= max(1, -(-(mesh.bounding_box_maxs[d] - mesh.bounding_box_mins[d]) // shape[d]))
    return abi.GradientField.make(rng.normal(size=(vox, 2, 3)) * 1e-2, shape)


# ---- one pass ----------------------------------------------------------------


def run(state):
    return _RUN[state["kind"]](state)


def _tail(arr, rows, count):
    """`arr` (of `rows` agents) with zeros in the rows of agents that were removed: those are no result."""
    if count < rows:
        arr[count * (arr.size // rows):] = 0
    return arr


def _result(state, fields=OUT_FIELDS):
    a = state["a"]
    state["sim"].download(a, fields=fields)
    out = {f: _tail(a.arrays[f], a.capacity, a.count) for f in fields}
    out["count"] = a.count
    return out


def _run_steps(state):
    state["sim"].step(state["steps"])
    return _result(state)


def _run_host_loop(state):
    sim = state["sim"]
    sim.upload_fields(state["a"], IN_FIELDS)
    sim.step(1)
    return _result(state)


def _run_entry_points(state):
    sim = state["sim"]
    sim.update_mechanics_mesh()
    sim.update_cell_neighbors()
    sim.update_cell_forces()
    sim.update_basement_membrane_interactions()
    sim.update_spring_attachments()
    sim.update_positions()
    sim.update_cell_container_for_mechanics()
    return _result(state)


def _run_divide(state):
    state["sim"].step_with_phenotype(state["steps"], 5e-5, 5e-5)
    return _result(state, OUT_FIELDS + ("radius", "agent_ids"))


def _run_spring_rates(state):
    state["sim"].step(state["steps"])
    return _result(state, OUT_FIELDS + ("spring_counts",))


def _run_immune(state):
    sim = state["sim"]
    for _ in range(state["steps"]):
        sim.update_motility_fields()
        sim.step(1)
        sim.update_cell_cell_interactions()
    out = _result(state, OUT_FIELDS + ("radius", "flags"))
    f, m = state["fields"], state["motility"]
    sim.download_interactions(f)
    sim.download_motility(m)
    rows = state["a"].capacity
    out.update({k: _tail(f.arrays[k], rows, f.count)
                for k in ("damage", "total_attack_time", "number_of_nuclei", "fluid", "solid",
                          "internalized_substrates")})
    out["motility_vector"] = _tail(m.arrays["motility_vector"], rows, m.count)
    return out


def _run_ensemble(state):
    sim = state["sim"]
    sim.step(state["steps"])
    for r, a in enumerate(state["sets"]):
        sim.download(a, r, fields=OUT_FIELDS)
        for f in OUT_FIELDS:
            _tail(a.arrays[f], a.capacity, a.count)
    return dict(state["whole"], counts=np.array([a.count for a in state["sets"]], np.int64))


def _run_bins(state):
    rc = state["lib"].ppc_bin_agents_noalloc(
        ctypes.byref(state["mesh"]), state["pos"].data_ptr(), state["n"], state["counts"].data_ptr(),
        state["agents"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError(device.lib().ppc_last_error())
    return {"counts": state["counts"], "agents": state["agents"]}


_RUN = {"run": _run_steps, "host_loop": _run_host_loop, "entry_points": _run_entry_points, "divide": _run_divide,
        "spring_rates": _run_spring_rates, "immune": _run_immune, "ensemble": _run_ensemble, "bins": _run_bins}


# ---- what a pass cannot do without ---------------------------------------------


def work(case):
    kind, config, steps = case["kind"], case["config"], case["steps"]
    dims, ndefs, walls, springs, neighbours = {
        1: (2, 1, 0, 0.0, 0.2), 2: (3, 2, 1, 0.0, 1.5), 3: (3, 3, 0, 0.4, 0.4), 4: (3, 1, 0, 0.0, 5.0),
        5: (3, 2, 0, 0.0, 0.4)}[config]
    n = case["agents"]
    if kind == "ensemble":
        n *= 10750  # the mean of log-uniform replicate sizes between 500 and 50,000
    if kind == "bins":
        voxels = n / {1: 900.0 / 4489, 2: 14300.0 / 300763, 3: 88700.0 / 700000}[config]
        return {"bytes": 8.0 * dims * n + 4.0 * n + 4.0 * min(voxels, 1048576), "flops": 4.0 * dims * n}
    # per agent and step: position and previous velocity in and out, pressure out, radius, repulsion, adhesion,
    # adhesion distance, affinities, type and movability in, spring partners
    per = 4 * 8 * dims + 8 + 32 + 8 * walls + 8 * ndefs + 5 + 12 * springs
    if kind == "spring_rates":
        per += 16 + 8 * springs  # rates, and the changed spring rows
    if kind == "divide":
        per += 1  # the division and death flags
    if kind == "immune":
        per += 8 * (7 + 2 * dims) + 8 * (2 + 4 * ndefs)  # motility in and out, interaction rates
    flops = n * steps * (neighbours * 60.0 + 12.0 * dims)
    total = float(per) * n * steps + n * (16.0 * dims + 8)  # the results down
    if kind == "host_loop":
        total += n * 16.0 * dims
    return {"bytes": total, "flops": flops}


# ---- a pass in plain 64-bit arithmetic -----------------------------------------


def _pairs(pos, mins, grid, reach):
    """(i, j) of every ordered pair of distinct agents in adjacent 30 um voxels within reach_i + reach_j."""
    dims = pos.shape[1]
    c = ((pos - mins) / 30.0).to(torch.int64).clamp_(min=0)
    c = torch.minimum(c, grid - 1)
    stride = [1]
    for d in range(dims - 1):
        stride.append(stride[-1] * int(grid[d]))
    stride = torch.tensor(stride, device=pos.device)
    key = (c * stride).sum(1)
    key, order = torch.sort(key)
    found_i, found_j = [], []
    for k in range(3 ** dims):
        off = torch.tensor([k // 3 ** d % 3 - 1 for d in range(dims)], device=pos.device)
        q = c + off
        ok = ((q >= 0) & (q < grid)).all(1).nonzero()[:, 0]
        want = (q[ok] * stride).sum(1)
        lo = torch.searchsorted(key, want)
        cnt = torch.searchsorted(key, want, right=True) - lo
        i = torch.repeat_interleave(ok, cnt)
        first = torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
        j = order[torch.repeat_interleave(lo, cnt) + torch.arange(i.numel(), device=pos.device) - first]
        near = (i != j) & ((pos[i] - pos[j]).square().sum(1).sqrt() <= reach[i] + reach[j])
        found_i.append(i[near])
        found_j.append(j[near])
    return torch.cat(found_i), torch.cat(found_j)


def _kept(out):
    """The reference's removal loop over the agents that are `out`: the last agent moves into each hole."""
    perm, h, cnt = list(range(len(out))), 0, len(out)
    while h < cnt:
        if out[perm[h]]:
            cnt -= 1
            perm[h] = perm[cnt]
        else:
            h += 1
    return perm[:cnt]


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind not in ("run", "host_loop", "entry_points") or case["agents"] * steps > 6000000:
        return None
    mesh, params, a = _make(case, seed)
    n, dims = a.count, a.dims
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def t(name):
        return torch.from_numpy(np.ascontiguousarray(a[name])).to(dev)

    pos, prev = t("positions").clone(), t("previous_velocities").clone()
    r, rep, adh, bm = t("radius"), t("cell_cell_repulsion_strength"), t("cell_cell_adhesion_strength"), \
        t("cell_BM_repulsion_strength")
    reach = t("relative_maximum_adhesion_distance") * r
    types, aff, elastic = t("cell_definition_indices").long(), t("cell_adhesion_affinities"), \
        t("attachment_elastic_constant")
    mins = torch.tensor([float(mesh.bounding_box_mins[d]) for d in range(dims)], dtype=torch.float64, device=dev)
    maxs = torch.tensor([float(mesh.bounding_box_maxs[d]) for d in range(dims)], dtype=torch.float64, device=dev)
    grid = torch.tensor(mesh.grid_shape()[:dims], device=dev)
    rows = np.repeat(np.arange(n), a["spring_counts"])
    cols = a["springs"][np.arange(a.spring_capacity)[None, :] < a["spring_counts"][:, None]]
    si, sj = torch.from_numpy(rows).to(dev), torch.from_numpy(cols.astype(np.int64)).to(dev)
    dt = params.mechanics_time_step
    for _ in range(steps):
        i, j = _pairs(pos, mins, grid, reach)
        diff = pos[i] - pos[j]
        dist = diff.square().sum(1).sqrt().clamp(min=1e-5)
        overlap = (1.0 - dist / (r[i] + r[j])).clamp(min=0.0).square()
        pressure = torch.zeros_like(r).index_add_(0, i, overlap * (2 * 36.64504274775163))
        pull = (1.0 - dist / (reach[i] + reach[j])).square()
        pull = pull * (adh[i] * adh[j] * aff[i, types[j]] * aff[j, types[i]]).sqrt()
        force = (overlap * (rep[i] * rep[j]).sqrt() - pull) / dist
        vel = torch.zeros_like(pos).index_add_(0, i, force[:, None] * diff)
        if params.virtual_wall_at_domain_edges:
            for wall, sign in ((mins, 1.0), (maxs, -1.0)):
                d = (wall - pos).abs().clamp(min=1e-5)
                push = (1.0 - d / r[:, None]).clamp(min=0.0).square()
                vel = vel + push * bm[:, None] * sign * d
        if si.numel():
            k = (elastic[si] * elastic[sj] * aff[si, types[sj]] * aff[sj, types[si]]).sqrt()
            vel = vel.index_add(0, si, k[:, None] * (pos[sj] - pos[si]))
        pos = pos + (vel * (dt * 1.5) + prev * (dt * -0.5))
        prev = vel
        out = ((pos < mins) | (pos > maxs)).any(1)
        if bool(out.any()):
            if si.numel():
                return None
            keep = torch.tensor(_kept(out.tolist()), device=dev, dtype=torch.int64)
            pos, prev, pressure = pos[keep], prev[keep], pressure[keep]
            r, rep, adh, bm, reach, types, aff, elastic = (x[keep] for x in (r, rep, adh, bm, reach, types, aff,
                                                                             elastic))
    out = {"count": pos.shape[0]}
    for f, x in zip(OUT_FIELDS, (pos, prev, pressure)):
        out[f] = torch.zeros(a.capacity * (x.numel() // x.shape[0]), dtype=torch.float64, device=dev)
        out[f][: x.numel()] = x.reshape(-1)
    return out

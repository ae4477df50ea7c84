"""The work users of this library have it do, as cases that can be timed and compared.

A case names one call pattern of the public Python binding (`kind`) with its sizes:

  points   block points of one world, host to host          World.biome_points
  map      the drop-in biome map, ids on the host            World.biome_grid
  quart    one quart-resolution grid into device memory      World.quart_grid_dev
  seeds    many seeds x fixed quart points, on the device    World.seed_points_dev
  plan     a frozen batch of uneven requests, replayed       Plan.run_dev
  batch    a request list from the host, once, to the host   Plan(...) + Plan.run + Plan.close
  serve    requests submitted to a running server            Server.submit / Server.wait
  search   the biome seed search over a range                World.search

Sizes come from the repository's benchmark workloads and GPU tests.  Every output is whole numbers (biome ids,
quantised climate targets, seeds, counts), so there is nothing for a 64-bit evaluation to measure.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OVERWORLD, NETHER, END = "minecraft:overworld", "minecraft:the_nether", "minecraft:the_end"
VERSIONS = ("26.1", "26.2", "26.3")
TIES = {"engine": 0, "grid_chain": 1, "chunk_cell": 2}
# the mixed batch's dimensions, 6:2:2
MIX = (OVERWORLD,) * 6 + (NETHER,) * 2 + (END,) * 2


def listed():
    return [
        # one block's biome: a tool that asks for the biome under the cursor (the smallest call, all latency)
        {"name": "point", "kind": "points", "version": "26.3", "dim": OVERWORLD, "preset": "normal", "n": 1},
        # scattered block points of one world, e.g. every village of a structure list
        {"name": "points_3001", "kind": "points", "version": "26.1", "dim": OVERWORLD, "preset": "normal", "n": 3001},
        # the drop-in map of the first benchmark configuration: a map viewer's tile (256 x 256, step 4)
        {"name": "map_256", "kind": "map", "version": "26.3", "dim": OVERWORLD, "preset": "normal", "nx": 256,
         "nz": 256, "step": 4, "y": 64},
        # the reference's own GPU benchmark shape: a 2048 x 2048 map, here in a double-branch version
        {"name": "map_2048", "kind": "map", "version": "26.1", "dim": OVERWORLD, "preset": "normal", "nx": 2048,
         "nz": 2048, "step": 4, "y": 64},
        # an odd-sized quart grid under the golden digests' tie rule (row-major candidate chain)
        {"name": "quart_chain", "kind": "quart", "version": "26.2", "dim": OVERWORLD, "preset": "amplified", "nx": 1001,
         "nz": 333, "qy": 16, "tie": "grid_chain"},
        # many seeds at the same few places, on the device: the second benchmark configuration
        {"name": "seeds8", "kind": "seeds", "version": "26.3", "dim": OVERWORLD, "preset": "normal", "ns": 65536, "np": 8,
         "targets": False},
        # the same in a double-branch version with the climate targets wanted as well, odd sizes
        {"name": "seeds_targets", "kind": "seeds", "version": "26.1", "dim": OVERWORLD, "preset": "large_biomes",
         "ns": 1501, "np": 33, "targets": True},
        # the uneven mixed batch (the benchmark's default workload): all versions and dimensions, replayed
        {"name": "plan_10k", "kind": "plan", "mix": "all", "n": 10000, "lo": 16, "hi": 512, "tie": "engine"},
        # the other dimensions' configuration: 64 x 64 grids of many seeds, Nether and End
        {"name": "plan_dims", "kind": "plan", "mix": "dims", "n": 8192, "lo": 64, "hi": 65, "tie": "engine"},
        # a request list that comes once: plan, run into host memory, free (end to end)
        {"name": "batch_300", "kind": "batch", "mix": "all", "n": 300, "lo": 16, "hi": 512, "tie": "engine"},
        # a burst of requests to a running server, each waited for
        {"name": "serve_48", "kind": "serve", "n": 48, "lo": 16, "hi": 512},
        # a chunk of the seed search: 2^20 candidates against eight observed cells, ties accepted
        {"name": "search_1m", "kind": "search", "version": "26.3", "dim": OVERWORLD, "n": 1 << 20, "nobs": 8,
         "block": False},
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["points", "map", "quart", "seeds", "seeds", "plan", "plan", "batch", "serve", "search"])
    version = rng.choice(VERSIONS)
    dim = rng.choice(MIX)
    preset = rng.choice(["normal", "normal", "large_biomes", "amplified"]) if dim == OVERWORLD else "normal"
    case = {"kind": kind, "version": version, "dim": dim, "preset": preset}
    if kind == "points":
        case["n"] = _log_int(rng, 1, 20000)
    elif kind == "map":
        case.update(nx=_log_int(rng, 16, 2048), nz=_log_int(rng, 16, 2048), step=rng.choice([1, 4, 4, 16, 37]),
                    y=rng.choice([-60, 0, 63, 64, 200]))
    elif kind == "quart":
        case.update(nx=_log_int(rng, 1, 1500), nz=_log_int(rng, 1, 1500), qy=rng.choice([-16, 0, 16, 40]),
                    tie=rng.choice(["engine", "engine", "grid_chain"]))
    elif kind == "seeds":
        case["np"] = _log_int(rng, 1, 64)
        case["ns"] = _log_int(rng, 1, 65536 * 8 // max(8, case["np"]))
        case["targets"] = rng.random() < 0.5
    elif kind in ("plan", "batch"):
        mix = rng.choice(["all", "all", "dims"])
        lo = rng.choice([1, 16, 16])
        case = {"kind": kind, "mix": mix, "n": _log_int(rng, 1, 4000 if kind == "plan" else 500), "lo": lo,
                "hi": _log_int(rng, lo + 16, 512), "tie": rng.choice(["engine", "engine", "chunk_cell"])}
    elif kind == "serve":
        case = {"kind": kind, "n": _log_int(rng, 1, 100), "lo": 16, "hi": _log_int(rng, 32, 512)}
    else:
        case = {"kind": kind, "version": version, "dim": dim, "n": _log_int(rng, 1 << 12, 1 << 20),
                "nobs": rng.randint(3, 8), "block": rng.random() < 0.3}
    return case


# ------------------------------------------------------------------------------------------ preparation
def _package():
    """The library's Python binding (its directory's name is not an identifier)."""
    name = "mcgen_gb300"
    if name not in sys.modules:
        d = os.path.join(REPO, "mc-worldgen-seed-lab_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"), submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _world(version, dim, preset="normal", seed=0):
    return _package().Generator.open(version=version).world(dim, preset, seed)


def _sides(case):
    u = (np.arange(case["n"]) + 0.5) / case["n"]
    return np.minimum((case["lo"] * (case["hi"] / case["lo"]) ** u).astype(np.int64), case["hi"] - 1)


def _uneven(case, rng):
    """The case's requests as one record array: seed, version and dimension, square side log-uniform in
    [lo, hi) (its n quantiles in random order, so that the total does not depend on the seed), corner uniform in
    [-30000, 30000] blocks, y = 64, as the benchmark draws them."""
    mg, n = _package(), case["n"]
    keys = [(v, d) for v in VERSIONS for d in (OVERWORLD, NETHER, END)]
    worlds = {}
    if case.get("mix", "all") == "dims":
        picked = [("26.3", (NETHER, END)[i % 2]) for i in range(n)]
    else:
        picked = [(VERSIONS[v], MIX[d]) for v, d in zip(rng.integers(0, 3, n), rng.integers(0, 10, n))]
    for k in keys:
        if k in set(picked):
            worlds[k] = _world(*k)
    used = list(worlds)
    side = rng.permutation(_sides(case))
    corner = rng.integers(-30000, 30001, (2, n)) >> 2
    seeds = rng.integers(-2**63, 2**63 - 1, n, dtype=np.int64)
    reqs = mg.RequestArray.from_index([worlds[k] for k in used], [used.index(k) for k in picked], seeds, corner[0],
                                      corner[1], side, side, 16)
    return reqs, [worlds[k] for k in picked]


def prepare(case, seed):
    mg = _package()
    rng = np.random.default_rng(seed)
    dev = torch.device("cuda")
    state = {"case": case}
    kind = case["kind"]
    one_seed = int(rng.integers(-2**63, 2**63 - 1))
    if kind in ("points", "map", "quart", "seeds"):
        state["world"] = _world(case["version"], case["dim"], case["preset"], one_seed)
    if kind == "points":
        xyz = rng.integers(-30000, 30001, (case["n"], 3))
        xyz[:, 1] = rng.integers(-64, 321, case["n"])
        state["xyz"] = xyz.astype(np.int32)
    elif kind == "map":
        state["origin"] = [int(v) for v in rng.integers(-30000, 30001, 2)]
    elif kind == "quart":
        state["origin"] = [int(v) for v in rng.integers(-7500, 7501, 2)]
        state["out"] = torch.empty((case["nz"], case["nx"]), dtype=torch.uint8, device=dev)
    elif kind == "seeds":
        ns, np_ = case["ns"], case["np"]
        pts = rng.integers(-2500, 2501, (np_, 3))
        pts[:, 1] = rng.integers(-16, 81, np_)
        state["seeds"] = torch.from_numpy(rng.integers(-2**63, 2**63 - 1, ns, dtype=np.int64)).to(dev)
        state["pts"] = torch.from_numpy(pts.astype(np.int32)).to(dev)
        state["out"] = torch.empty((ns, np_), dtype=torch.uint8, device=dev)
        state["targets"] = torch.empty((ns, np_, 6), dtype=torch.int32, device=dev) if case["targets"] else None
    elif kind == "plan":
        reqs, _ = _uneven(case, rng)
        state["plan"] = mg.Plan(reqs, TIES[case["tie"]])
        state["out"] = torch.empty(state["plan"].output_bytes, dtype=torch.uint8, device=dev)
    elif kind == "batch":
        state["reqs"], _ = _uneven(case, rng)
        cells = int((state["reqs"].records["nx"].astype(np.int64) * state["reqs"].records["nz"]).sum())
        state["host"] = torch.empty(cells, dtype=torch.uint8).pin_memory()
        state["out"] = state["host"].numpy()
    elif kind == "serve":
        reqs, worlds = _uneven(case, rng)
        r = reqs.records
        ends = np.cumsum(r["nx"].astype(np.int64) * r["nz"])
        state["out"] = np.empty(int(ends[-1]), np.uint8)
        state["calls"] = [(w, int(q["seed"]), int(q["qx0"]), int(q["qz0"]), int(q["nx"]), int(q["nz"]), int(q["qy"]),
                           state["out"][e - int(q["nx"]) * int(q["nz"]):e]) for w, q, e in zip(worlds, r, ends)]
        state["server"] = mg.Server(hbm_budget_bytes=1 << 30)
    elif kind == "search":
        # what a player saw: cells (or blocks) of one seed's world and the biomes there
        state["world"] = w = _world(case["version"], case["dim"], "normal", one_seed)
        at = rng.integers(-5000, 5001, (case["nobs"], 3))
        at[:, 1] = 16
        if case["block"]:
            ids = w.biome_points(at * 4)
            at = at * 4
        else:
            ids = w.seed_points(np.array([one_seed], np.int64), at)[0]
        state["obs"] = mg.make_obs([(int(x), int(y), int(z), [int(b)]) for (x, y, z), b in zip(at, ids)], case["block"])
        if case["dim"] == END:
            for o in state["obs"]:
                o["flags"] = (int(o["flags"]) & ~0xFF) | w.end_radius(o["mask"])
        state["base"] = one_seed - int(rng.integers(0, case["n"]))
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "points":
        return state["world"].biome_points(state["xyz"])
    if kind == "map":
        x0, z0 = state["origin"]
        return state["world"].biome_grid(x0, z0, case["nx"], case["nz"], case["step"], case["y"])
    if kind == "quart":
        qx0, qz0 = state["origin"]
        state["world"].quart_grid_dev(qx0, qz0, case["nx"], case["nz"], case["qy"], TIES[case["tie"]],
                                      state["out"].data_ptr(), stream)
        return state["out"]
    if kind == "seeds":
        t = state["targets"]
        state["world"].seed_points_dev(state["seeds"].data_ptr(), case["ns"], state["pts"].data_ptr(), case["np"],
                                       state["out"].data_ptr(), t.data_ptr() if t is not None else 0, stream)
        return state["out"] if t is None else [state["out"], t]
    if kind == "plan":
        state["plan"].run_dev(state["out"].data_ptr(), stream)
        return state["out"]
    if kind == "batch":
        plan = _package().Plan(state["reqs"], TIES[case["tie"]])
        plan.run(state["out"])
        plan.close()
        return state["out"]
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(w, s, qx, qz, nx, nz, qy, out) for w, s, qx, qz, nx, nz, qy, out in state["calls"]]
        for t in tickets:
            server.wait(t)
        return state["out"]
    found, reached, _ = state["world"].search(state["obs"], kind=_package().SEEDS_RANGE, base=state["base"], n=case["n"])
    listed_seeds = np.zeros(1 << 16, np.int64)  # the list at its full length, whatever was found
    listed_seeds[:found.size] = found
    return [listed_seeds, found.size, reached.view(np.int64)]


# ------------------------------------------------------------------------------------------ work
# Arithmetic operations (floating-point and integer) that the algorithm itself asks for: an octave sample is
# 8 gradient dots of 5, 7 lerps of 3, two smoothsteps of 7 and two coordinate splits of 3; 52 octave samples
# per Overworld cell, 8 per Nether cell; an End cell shares its chunk's window; a lattice's setup is 256
# Fisher-Yates steps of 21 and three coordinate draws of 20; a block's zoom compares 8 cells of 40.
OCTAVE, ZOOM, LATTICE = 81, 320, 256 * 21 + 60
CELL = {OVERWORLD: 52 * OCTAVE, NETHER: 8 * OCTAVE, END: 16}
LATTICES = {OVERWORLD: 46, NETHER: 8, END: 1}
SEED_BYTES = 8


def work(case):
    kind = case["kind"]
    if kind == "points":
        return {"bytes": 13 * case["n"], "flops": case["n"] * (CELL[case["dim"]] + ZOOM)}
    if kind == "map":
        n = case["nx"] * case["nz"]
        return {"bytes": n, "flops": n * (CELL[case["dim"]] + ZOOM)}
    if kind == "quart":
        n = case["nx"] * case["nz"]
        return {"bytes": n, "flops": n * CELL[case["dim"]]}
    if kind == "seeds":
        n = case["ns"] * case["np"]
        return {"bytes": n * (25 if case["targets"] else 1) + case["ns"] * SEED_BYTES + 12 * case["np"],
                "flops": n * CELL[case["dim"]] + case["ns"] * LATTICES[case["dim"]] * LATTICE}
    if kind == "search":
        return {"bytes": 32 * case["nobs"] + 8 * (case["nobs"] + 1),
                "flops": case["n"] * (LATTICES[case["dim"]] * LATTICE + CELL[case["dim"]])}
    # uneven requests: their cells, and the mix's mean cost of a cell and of a seed
    cells = float((_sides(case) ** 2).sum())
    dims = (NETHER, END) if case.get("mix") == "dims" else MIX
    cell = sum(CELL[d] for d in dims) / len(dims)
    lattices = sum(LATTICES[d] for d in dims) / len(dims)
    setup = 0 if kind == "serve" else lattices * LATTICE  # a running server keeps its seeds' noise states
    return {"bytes": cells + 40 * case["n"], "flops": cells * cell + case["n"] * setup}


def exact(case, seed):
    """Biome ids, targets, seeds and counts are whole numbers: they are compared for equality."""
    return None

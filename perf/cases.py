"""What this framework is measured on: whole calls through its public Python entry points, over the
range of problems that its users solve. Sizes and physical parameters are those of the repository's
own inputs (tests/golden/inputs, tests/gen_inputs.py, exaca_b200/batch.py, bench.py) or lie in their
ranges.

The reference's random streams have fixed seeds, so the seed of `prepare` moves what a user varies
between runs (nucleation density and undercooling, the surface fraction, the substrate's grain
spacing, a heat source's speed) by a few percent: other inputs, the same amount of work.
"""
import ctypes
import math
import os
import random
import shutil
import tempfile

import numpy as np
import torch

import exaca_b200 as ex
from exaca_b200 import batch, serve

MIN_LIST = 1 << 20  # floor of a pool's list capacity, as serve.sequential_plain uses


# ------------------------------------------------------------------------------------------------
# the cases

def _directional(name, nx, ny, nz, G, R, n, density, dtn, sigma, frac, octahedra=False, pinned=False):
    return dict(name=name, kind="directional", nx=nx, ny=ny, nz=nz, G=G, R=R, n=n, density=density, dtn=dtn,
                sigma=sigma, frac=frac, octahedra=octahedra, pinned=pinned)


def listed():
    return [
        # One small directional solve (tests/golden/inputs/DirS64.txt): parameter studies, where the
        # latency of a cycle is everything.
        _directional("directional 64^3", 64, 64, 64, 5e5, 3e5, 17, 10.0, 5.0, 0.5, 0.08),
        # An odd, flat-sided box with dense nucleation, read back with its octahedra (a restart or a
        # check against the reference's DiagonalLength / DOCenter / CritDiagonalLength).
        _directional("directional ragged, octahedra", 61, 127, 45, 1e6, 5e5, 20, 300.0, 4.0, 0.6, 0.05, octahedra=True),
        # The ordinary solve: the benchmark's parameters at 256^3 (tests/golden/DirS256.json).
        _directional("directional 256^3", 256, 256, 256, 1e6, 1e6, 25, 100.0, 3.0, 0.5, 0.02),
        # The largest: the benchmark workload itself (bench.py), results into page-locked buffers
        # that the caller keeps, as its end-to-end arm does.
        _directional("directional 512^3", 512, 512, 512, 1e6, 1e6, 25, 100.0, 3.0, 0.5, 0.02, pinned=True),
        # Type S, one layer: tests/golden/inputs/SpotMelt3x3.txt (304 x 304 x 78 cells, 71000 cycles).
        dict(name="spot melts 3x3", kind="spots", sx=3, sy=3, radius=75, offset=75, layers=1, layer_offset=25, n=17,
             spacing=15.2, density=10.0, dtn=5.0),
        # Type S, several layers, small and with bulk nucleation (SpotMelt3Layers.txt's parameters
        # on a larger spot): the layer loop, its cycle jumps and its window moves.
        dict(name="spot melts, 3 layers", kind="spots", sx=2, sy=2, radius=20, offset=20, layers=3, layer_offset=8,
             n=25, spacing=6.0, density=500.0, dtn=5.0),
        # Type R: melt tracks from temperature files, two files repeated over three layers
        # (RTwoFiles3Layers.txt's parameters on longer tracks).
        dict(name="melt tracks, 3 layers", kind="tracks", points_x=90, points_y=40, points_z=12, files=2, layers=3,
             layer_offset=4, speed=0.6, spacing=5.0, density=300.0, dt=0.05),
        # A process map: many uneven domains stepped together (batch.process_map's parameter ranges).
        dict(name="process map, 96 domains", kind="map", domains=96, lo=32, hi=96, map_seed=3),
        # The request loop (serve.request_stream's arrivals and ranges): initialised, admitted,
        # stepped and copied out as requests come in.
        dict(name="serve, 20 requests", kind="serve", requests=20, lo=48, hi=160, rate=200.0, map_seed=4),
        # A caller that drives the cycles itself and watches them (exaca_pool_step / _status /
        # _census): many short calls on a small domain.
        dict(name="stepped 48^3, watched", kind="stepped", nx=48, ny=48, nz=48, G=5e5, R=3e5, n=17, density=10.0,
             dtn=5.0, sigma=0.5, frac=0.08, chunk=25, chunks=40),
        # Analysis of a finished solve on the device (exaca_pool_grain_stats).
        dict(name="grain statistics 192x160x128", kind="statistics", nx=192, ny=160, nz=128, G=1e6, R=1e6, n=25,
             density=100.0, dtn=3.0, sigma=0.5, frac=0.02),
        # A progress monitor over cell fields in device memory (exaca_census_cells): the smallest call.
        dict(name="census of 24 domains", kind="census", domains=24, side=56),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log(rng, lo, hi):
    return float("%.4g" % math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["directional", "directional", "directional", "spots", "tracks", "map", "serve", "stepped",
                       "statistics", "census"])
    if kind == "directional":
        big = rng.random() < 0.3
        lo, hi = (96, 320) if big else (17, 128)
        return dict(kind=kind, nx=_log_int(rng, lo, hi), ny=_log_int(rng, lo, hi), nz=_log_int(rng, lo, hi),
                    G=_log(rng, 5e5, 2e6), R=_log(rng, 3e5, 1e6), n=rng.randint(12, 28), density=_log(rng, 1, 500),
                    dtn=round(rng.uniform(2, 6), 2), sigma=round(rng.uniform(0.2, 1.0), 2), frac=_log(rng, 0.01, 0.15),
                    octahedra=rng.random() < 0.25, pinned=rng.random() < 0.25)
    if kind == "spots":
        radius = _log_int(rng, 10, 40)
        return dict(kind=kind, sx=rng.randint(1, 3), sy=rng.randint(1, 3), radius=radius,
                    offset=rng.randint(radius // 2, radius + 4), layers=rng.randint(1, 3),
                    layer_offset=rng.randint(3, radius // 2), n=rng.randint(12, 28), spacing=round(rng.uniform(4, 12), 2),
                    density=_log(rng, 1, 500), dtn=round(rng.uniform(2, 6), 2))
    if kind == "tracks":
        return dict(kind=kind, points_x=rng.randint(24, 90), points_y=rng.randint(12, 40), points_z=rng.randint(5, 12),
                    files=rng.randint(1, 2), layers=rng.randint(1, 3), layer_offset=rng.randint(2, 5),
                    speed=_log(rng, 0.4, 1.5), spacing=round(rng.uniform(3, 8), 2), density=_log(rng, 1, 500),
                    dt=round(rng.uniform(0.03, 0.08), 3))
    if kind == "map":
        return dict(kind=kind, domains=_log_int(rng, 6, 96), lo=32, hi=rng.randint(48, 96), map_seed=rng.randint(10, 10**6))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(4, 20), lo=48, hi=rng.randint(64, 160), rate=200.0,
                    map_seed=rng.randint(10, 10**6))
    if kind == "stepped":
        return dict(kind=kind, nx=_log_int(rng, 16, 128), ny=_log_int(rng, 16, 128), nz=_log_int(rng, 16, 128),
                    G=_log(rng, 5e5, 2e6), R=_log(rng, 3e5, 1e6), n=rng.randint(12, 28), density=_log(rng, 1, 500),
                    dtn=round(rng.uniform(2, 6), 2), sigma=round(rng.uniform(0.2, 1.0), 2), frac=_log(rng, 0.01, 0.15),
                    chunk=_log_int(rng, 1, 200), chunks=rng.randint(8, 60))
    if kind == "statistics":
        return dict(kind=kind, nx=_log_int(rng, 32, 192), ny=_log_int(rng, 32, 192), nz=_log_int(rng, 32, 192), G=1e6,
                    R=1e6, n=rng.randint(12, 28), density=_log(rng, 1, 500), dtn=round(rng.uniform(2, 6), 2), sigma=0.5,
                    frac=_log(rng, 0.01, 0.15))
    return dict(kind=kind, domains=_log_int(rng, 1, 256), side=_log_int(rng, 16, 96))


# ------------------------------------------------------------------------------------------------
# inputs

class _Files:
    """Input files of one problem; they are read while it is built and gone after that."""

    def __init__(self):
        self.dir = tempfile.mkdtemp(prefix="exaca_case_")

    def write(self, name, text):
        path = os.path.join(self.dir, name)
        with open(path, "w") as f:
            f.write(text)
        return path

    def gone(self):
        shutil.rmtree(self.dir, ignore_errors=True)


_HEAD = """A measured problem
*****
Problem type: {kind}
Decomposition strategy: 1
Material: Inconel625
Cell size (microns): 1
Heterogeneous nucleation density (normalized by 1*10^12 per m^3): {density}
Mean nucleation undercooling (in K): {dtn}
Standard deviation of nucleation undercooling: 0.5
Path to output: ./
Output file base name: case
File of grain orientations: GrainOrientationVectors_Uniform10k.csv
"""

_SPOTS = """Thermal gradient (K/m): 500000
Cooling rate (K/s): 300000
Number of spots in x: {sx}
Number of spots in y: {sy}
Offset between spot centers (in microns): {offset}
Radii of spots (in microns): {radius}
Number of layers: {layers}
Offset between layers (in cells): {layer_offset}
"N", where the time step = deltax/(Steady State Velocity * N): {n}
Substrate grain spacing (in microns): {spacing}
"""

_TRACKS = """Heat transport data mesh size (microns): 1
Time step (microseconds): {dt}
Substrate grain spacing (in microns): {spacing}
Path to temperature file(s): {dir}
Temperature filename (* glob before the name): {tname}
Number of temperature files: {files}
Extra set of wall cells around temperature field (used for spot melt problems, Y or N)?: N
Number of layers: {layers}
Offset between layers (if Number of layers > 1, in cells): {layer_offset}
"""

_TAIL = """***Output data printing options: (Y or N) which data should be printed***
Print Paraview vtk file of grain misorientation values (Y or N)?: N
Print Paraview vtk file of all ExaCA data for post-processing (Y or N)?: N
Debug check (reduced)- Print data for main Kokkos views (CellType, LayerID, CritTimeStep) following initialization for debug check (Y or N)?: N
Debug check (extensive) - Print data for all main data structures (CellType, GrainID, CritTimeStep, UndercoolingCurrent, UndercoolingChange, Melted, LayerID) following initialization for debug check (Y or N)?: N
"""


def _nudge(rng, v, share):
    return v * rng.uniform(1 - share, 1 + share)


def _directional_problem(case, rng):
    return ex.Problem.directional(
        case["nx"], case["ny"], case["nz"], G=case["G"], R=case["R"], n_ratio=case["n"],
        nucleation_density=_nudge(rng, case["density"], 0.05), dTN=_nudge(rng, case["dtn"], 0.01),
        dTsigma=case["sigma"], fract_surface_active=_nudge(rng, case["frac"], 0.04))


def _spots_problem(case, rng):
    files = _Files()
    try:
        text = _HEAD.format(kind="S", density=round(_nudge(rng, case["density"], 0.05), 4), dtn=case["dtn"])
        text += _SPOTS.format(**{**case, "spacing": round(_nudge(rng, case["spacing"], 0.04), 4)}) + _TAIL
        return ex.Problem.from_file(files.write("spots.txt", text))
    finally:
        files.gone()


def _track(rng, case, number):
    """One pass of a heat source along +x: the points of a half-ellipsoid track, in the reference's
    reduced temperature-file format (as tests/golden/make_temperatures.py writes them)."""
    h, nx, ny, nz = 1e-6, case["points_x"], case["points_y"], case["points_z"]
    width, depth = (0.48 - 0.05 * number) * ny * h, 0.9 * (nz - 1) * h
    speed = _nudge(rng, case["speed"], 0.02)
    i, j, k = (a.ravel() for a in np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"))
    inside = ((j - 0.5 * (ny - 1)) * h / width) ** 2 + (k * h / depth) ** 2 <= 1.0
    i, j, k = i[inside], j[inside], k[inside]
    jitter = np.random.default_rng(rng.randrange(1 << 30)).random(i.size)
    tl = 2e-6 * number + i * h / speed + 2e-6 * (k * h) / depth + 1e-7 * jitter
    cr = np.where(k * h < 0.5 * depth, 9e5 - 2e5 * number, 6e5 - 2e5 * number)
    rows = ["x,y,z,tm,tl,cr"]
    rows += ["%r,%r,%r,%r,%r,%r" % (float(a) * h, float(b) * h, -float(c) * h, float(t) - 5e-6, float(t), float(r))
             for a, b, c, t, r in zip(i, j, k, tl, cr)]
    return "\n".join(rows) + "\n"


def _tracks_problem(case, rng):
    files = _Files()
    try:
        for f in range(case["files"]):
            files.write((str(f + 1) if case["files"] > 1 else "") + "track.csv", _track(rng, case, f))
        text = _HEAD.format(kind="R", density=round(_nudge(rng, case["density"], 0.05), 4), dtn=5)
        text += _TRACKS.format(**{**case, "dir": files.dir, "tname": "track.csv",
                                  "spacing": round(_nudge(rng, case["spacing"], 0.04), 4)}) + _TAIL
        return ex.Problem.from_file(files.write("tracks.txt", text))
    finally:
        files.gone()


def _nudged_params(params, rng):
    for p in params:
        p["nucleation_density"] = _nudge(rng, p["nucleation_density"], 0.05)
        p["fract_surface_active"] = _nudge(rng, p["fract_surface_active"], 0.04)
    return params


def _census_domains(case, seed):
    """Cell fields of half-solidified domains on the device: a solid bottom, an active front, liquid
    above it, CritTimeSteps that grow with z."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    side = case["side"]
    fields, domains = [], []
    for d in range(case["domains"]):
        mx, my, nz = side + 2 + d % 3, side + 2, side + 1 + d % 5
        n = mx * my * nz
        u = torch.rand(n, generator=g, device="cuda")
        z = torch.arange(n, device="cuda") // (mx * my)
        front = (z.float() + 6 * u) / nz
        ctype = torch.where(front < 0.45, ex.SOLID, torch.where(front < 0.5, ex.ACTIVE, ex.LIQUID)).to(torch.int8)
        layer = torch.zeros(n, dtype=torch.int8, device="cuda")
        cts = (z * 25 + (u * 20).long()).to(torch.int32)
        fields += [ctype, layer, cts]
        domains.append(dict(cell_type=ctype.data_ptr(), layer_id=layer.data_ptr(), crit_time_step=cts.data_ptr(),
                            domain_size=n, active_size=n, cycle=25 * nz // 2 + d))
    torch.cuda.synchronize()
    return fields, domains


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    state = dict(kind=kind, case=case)
    if kind in ("directional", "spots", "tracks", "stepped", "statistics"):
        build = {"spots": _spots_problem, "tracks": _tracks_problem}.get(kind, _directional_problem)
        state["problem"] = problem = build(case, rng)
        cells = problem.geometry.domain_size
        state["pool"] = ex.Pool(0, list_capacity=max(problem.geometry.active_size, MIN_LIST))
        if case.get("pinned"):
            state["buffers"] = tuple(torch.empty(cells, dtype=torch.int32, pin_memory=True) for _ in range(2))
        if kind == "statistics":
            state["slot"] = state["pool"].admit(problem, device_check=False)
            state["pool"].run_plain(state["slot"])
    elif kind == "map":
        params = batch.process_map(case["domains"], seed=case["map_seed"], side=(case["lo"], case["hi"]))
        state["problems"] = batch.build_problems(_nudged_params(params, rng))
    elif kind == "serve":
        requests = serve.request_stream(case["requests"], rate=case["rate"], seed=case["map_seed"],
                                        side=(case["lo"], case["hi"]))
        _nudged_params([p for _, p in requests], rng)
        state["requests"] = requests
    else:
        state["fields"], state["domains"] = _census_domains(case, seed)
    return state


# ------------------------------------------------------------------------------------------------
# one pass

def _solve(state):
    pool, case = state["pool"], state["case"]
    slot = pool.admit(state["problem"], device_check=False)
    out = dict(cycle=pool.run_plain(slot))
    if case.get("pinned"):
        gid, ctype = state["buffers"]
        lib = ex.load_library()
        rc = lib.exaca_pool_copy_out(pool._h, slot, ctypes.c_void_p(gid.data_ptr()), ctypes.c_void_p(ctype.data_ptr()))
        if rc != 0:
            raise RuntimeError(lib.exaca_last_error())
        out["grain_id"], out["cell_type"] = gid, ctype
    else:
        out["grain_id"], out["cell_type"] = pool.copy_out(slot)
    if case.get("octahedra"):
        out["dl"], out["centre"], out["critical"] = pool.copy_octahedra(slot)
    pool.retire(slot)
    return out


def _stepped(state):
    pool, case = state["pool"], state["case"]
    slot = pool.admit(state["problem"], device_check=True)
    watched = []
    for _ in range(case["chunks"]):
        pool.step(case["chunk"])
        s = pool.status(slot)
        c = pool.census(slot)
        watched.append([s.cycle, int(s.done), s.nn, s.error, s.liquid, c["superheated"], c["undercooled"], c["active"],
                        c["solid"], c["remaining"]])
    gid, ctype = pool.copy_out(slot)
    pool.retire(slot)
    return dict(watched=np.array(watched, dtype=np.int64), grain_id=gid, cell_type=ctype)


def run(state):
    kind, case = state["kind"], state["case"]
    if kind in ("directional", "spots", "tracks"):
        return _solve(state)
    if kind == "stepped":
        return _stepped(state)
    if kind == "map":
        out = batch.solve_batch(state["problems"], autotune_cycles=50)
        return dict(cycle=np.array(out["cycle"]), grain_id=np.concatenate(out["grain_id"]),
                    cell_type=np.concatenate(out["cell_type"]))
    if kind == "serve":
        out = serve.serve(state["requests"], chunk_cycles=250, keep_results=True)
        return dict(results=[(g, t, np.int64(c)) for g, t, c in out["results"]], timed_out=len(out["timed_out"]))
    if kind == "statistics":
        out = state["pool"].grain_stats(state["slot"])
        return {**out, "misorientation_hist": np.array(out["misorientation_hist"], dtype=np.int64)}
    found = ex.census_cells(0, state["domains"], stream=torch.cuda.current_stream().cuda_stream)
    # next_cts is 2^64 - 1 where no liquid is left: kept as it is, in unsigned words
    return np.array([[c[k] for k in ("superheated", "undercooled", "active", "solid", "remaining", "next_cts")]
                     for c in found], dtype=np.uint64).view(np.int64)


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without

# floating-point operations of one capture: the capture geometry (about 150) and 26 critical
# lengths of 21 each (src/CAupdate.cpp:353-563); every cell that solidifies was captured once
CAPTURE_FLOPS = 700


def _cells(case):
    kind = case["kind"]
    if kind == "spots":
        # a quarter of an ellipsoid-like melt pool per spot is what solidifies
        side = [2 * case["radius"] + (case[s] - 1) * case["offset"] for s in ("sx", "sy")]
        depth = case["radius"] + (case["layers"] - 1) * case["layer_offset"]
        return side[0] * side[1] * depth
    if kind == "tracks":
        return case["points_x"] * case["points_y"] * (case["points_z"] + (case["layers"] - 1) * case["layer_offset"])
    if kind == "map":
        return sum(p["nx"] * p["ny"] * p["nz"]
                   for p in batch.process_map(case["domains"], seed=case["map_seed"], side=(case["lo"], case["hi"])))
    if kind == "serve":
        return sum(p["nx"] * p["ny"] * p["nz"]
                   for _, p in serve.request_stream(case["requests"], rate=case["rate"], seed=case["map_seed"],
                                                    side=(case["lo"], case["hi"])))
    if kind == "census":
        return sum((case["side"] + 2 + d % 3) * (case["side"] + 2) * (case["side"] + 1 + d % 5)
                   for d in range(case["domains"]))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    cells, kind = _cells(case), case["kind"]
    if kind == "census":
        return dict(bytes=6 * cells, flops=0)  # CellType, LayerID and CritTimeStep read once
    if kind == "statistics":
        return dict(bytes=5 * cells, flops=2 * cells)  # GrainID and the melted flag read once
    out = 8 * cells  # GrainID and CellType to the caller
    if case.get("octahedra"):
        out += 30 * 4 * cells
    if kind in ("spots", "tracks"):
        out += 14 * cells  # the cell fields come from the host
    captured = cells
    if kind == "stepped":
        captured = min(cells, cells * case["chunk"] * case["chunks"] / (25.0 * case["nz"]))
    return dict(bytes=out, flops=CAPTURE_FLOPS * captured)


def exact(case, seed):
    """No output has a value in 64 bits: grain numbers, cell types and counts are whole numbers, and
    the octahedra are the rounded float sums that decide them."""
    return None

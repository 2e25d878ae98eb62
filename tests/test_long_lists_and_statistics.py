"""Active lists longer than the range that has octahedron bodies beside it (2^21 records), and the
statistics kernels at their edges: region rows below, at and above a warp's width, regions of one
cell, at the walls and of the whole grid; cell counts that are no multiple of sixteen and fields off
the 16-byte boundary. Whole numbers are compared exactly, sums of doubles to 1e-9 (their additions
are in another order: at most 1e5 terms of 2^-53 each)."""
import os
import sys

import numpy as np
import pytest

from helpers import input_path, load_golden

import exaca_b200 as ex
from exaca_b200 import batch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import grain_stats as gs  # noqa: E402

pytestmark = pytest.mark.gpu

GUV = np.loadtxt(os.path.join(os.path.dirname(ex.__file__), "data", "Substrate", "GrainOrientationVectors_Uniform10k.csv"),
                 skiprows=1, delimiter=",", dtype=np.float32)


@pytest.fixture(scope="module")
def large_domains():
    """Domains of which three fit below 2^21 records and the fourth lies across it; their own runs."""
    probs = [ex.Problem.directional(nx, ny, 8, G=1e6, R=1e6, n_ratio=8, nucleation_density=50.0 + k, dTN=3.0, dTsigma=0.5,
                                    fract_surface_active=1.0) for k, (nx, ny) in
             enumerate([(800, 797), (811, 790), (640, 960), (901, 799)])]
    own = []
    pool = ex.Pool(0, list_capacity=max(p.geometry.active_size for p in probs))
    for p in probs:
        s = pool.admit(p, device_check=True)
        pool.run_all(chunk_cycles=500)
        own.append((pool.status(s).cycle,) + pool.copy_out(s))
        pool.retire(s)
    pool.close()
    return probs, own


@pytest.mark.parametrize("config", range(4))
def test_records_past_the_bodies(lib, large_domains, config):
    probs, own = large_domains
    pool = ex.Pool(0, list_capacity=sum(p.geometry.active_size for p in probs))
    try:
        pool.set_config(config)
        slots = [pool.admit(p, device_check=True) for p in probs]
        # the short first steps see the list at its longest
        for n in (7, 30):
            pool.step(n)
        pool.run_all(chunk_cycles=500)
        for k, s in enumerate(slots):
            cycle, gid, ct = own[k]
            assert pool.status(s).cycle == cycle, f"domain {k}"
            g, c = pool.copy_out(s)
            assert np.array_equal(g, gid) and np.array_equal(c, ct), f"domain {k}"
    finally:
        pool.close()


def test_more_domains_than_growth_views(lib):
    """The last domains lie past the block's table of growth fields and take the general path."""
    params = batch.process_map(332, seed=12, side=(5, 9), G=(1e6, 4e6), R=(5e5, 1e6), density=(1e15, 1e16))
    probs = batch.build_problems(params)
    plain = batch.solve_plain(probs)
    res = batch.solve_batch(probs, chunk_cycles=250)
    for i in range(len(probs)):
        assert res["cycle"][i] == plain["cycle"][i], f"domain {i}"
        assert np.array_equal(res["grain_id"][i], plain["grain_id"][i]), f"domain {i}"
        assert np.array_equal(res["cell_type"][i], plain["cell_type"][i]), f"domain {i}"


def test_spot_melts_among_many_domains(lib):
    """A multilayer type-S domain (growth extras: no short path for any domain) among ten type-C ones."""
    probs = batch.build_problems(batch.process_map(10, seed=13, side=(8, 14), G=(1e6, 4e6), R=(5e5, 1e6)))
    for case in ("SmallSpotMelt", "SpotMelt3Layers"):
        spot = ex.Problem.from_file(input_path(case))
        alone = ex.Pool(0, list_capacity=spot.geometry.active_size)
        a = alone.admit(spot, device_check=False)
        pool = ex.Pool(0, list_capacity=1 << 20)
        s = pool.admit(spot, device_check=False)
        for p in probs:
            pool.admit(p, device_check=True)
        for n in (150, 400):
            alone.step(n)
            pool.step(n)
            for u, v in zip(alone.copy_out(a) + alone.copy_octahedra(a)[:1], pool.copy_out(s) + pool.copy_octahedra(s)[:1]):
                assert np.array_equal(u, v), (case, n)
        alone.close()
        pool.close()


def same_statistics(dev, host):
    for k in ("region_cells", "melted_cells", "n_grains", "misorientation_hist"):
        assert dev[k] == host[k], k
    for k in ("mean_grain_volume_um3", "nucleated_fraction", "mean_misorientation_deg", "mean_misorientation_top_deg"):
        assert dev[k] == pytest.approx(host[k], rel=1e-9), k


@pytest.mark.parametrize("nx,ny,nz", [(7, 33, 9), (31, 34, 12), (5, 65, 6), (40, 3, 8)])
def test_grain_statistics_of_directional_domains(lib, nx, ny, nz):
    p = ex.Problem.directional(nx, ny, nz, G=1e6, R=1e6, n_ratio=12, nucleation_density=20000.0, dTN=2.0, dTsigma=0.3,
                               fract_surface_active=0.3)
    pool = ex.Pool(0, list_capacity=p.geometry.active_size)
    slot = pool.admit(p, device_check=False)
    nx, ny, nz = p.geometry.nx, p.geometry.ny, p.geometry.nz  # with the wall layers
    for n in (0, 120, 1500):
        if n:
            pool.step(n)
        gid, _ = pool.copy_out(slot)
        mel = np.zeros((nz, nx + 2, ny + 2), np.int8)
        mel[1:nz - 1, 1:nx + 1, 1:ny + 1] = 1
        for region in (None, (0, nx - 1, 0, ny - 1, 0, nz - 1), (2, 2, 1, 1, 3, 3), (0, nx - 1, ny - 1, ny - 1, 0, 0),
                       (1, 3, 0, ny - 1, nz - 2, nz - 1)):
            same_statistics(pool.grain_stats(slot, region), gs.grain_stats(gid, mel.ravel(), GUV, nx, ny, nz, 1e-6, region))
    pool.close()


def test_grain_statistics_of_a_raster_region(lib):
    case = "SmallSpotMelt"
    init = load_golden(case)["init_melted"]
    nz, ny, nx = init.shape
    mel = np.zeros((nz, nx + 2, ny + 2), np.int8)
    mel[:, 1:nx + 1, 1:ny + 1] = init.transpose(0, 2, 1)
    p = ex.Problem.from_file(input_path(case))
    pool = ex.Pool(0, list_capacity=p.geometry.active_size)
    slot = pool.admit(p, device_check=False)
    pool.run_plain(slot)
    gid, _ = pool.copy_out(slot)
    for region in (None, (0, nx - 1, 0, ny - 1, 0, nz - 1), (1, 3, 0, ny - 1, 0, 2)):
        dev = pool.grain_stats(slot, region)
        # the volume factor is the cell size of the input file
        host = gs.grain_stats(gid, mel.ravel(), GUV, nx, ny, nz, 1e-6, region)
        host["mean_grain_volume_um3"] = dev["mean_grain_volume_um3"]
        same_statistics(dev, host)
    pool.close()


@pytest.mark.parametrize("sizes", [(1, 15, 16, 17), (4096 * 16 + 3, 31, 257)])
@pytest.mark.parametrize("offset", [0, 1])
def test_census_of_odd_fields(lib, sizes, offset):
    import torch

    rng = np.random.default_rng(len(sizes))
    doms, fields, keep = [], [], []
    for k, n in enumerate(sizes):
        t = rng.integers(-1, 6, n + offset, dtype=np.int8)
        ly = rng.integers(0, 3, n + offset, dtype=np.int8)
        cts = rng.integers(0, 3000, n + offset, dtype=np.int32)
        d = [torch.from_numpy(a).cuda() for a in (t, ly, cts)]
        keep.append(d)
        w0 = n // 3
        doms.append(dict(cell_type=d[0].data_ptr() + offset, layer_id=d[1].data_ptr() + offset,
                         crit_time_step=d[2].data_ptr() + 4 * offset, domain_size=n, active_size=n - w0, cycle=1400, layer=1,
                         window_start=w0))
        fields.append((t[offset:], ly[offset:], cts[offset:], w0))
    torch.cuda.synchronize()
    got = ex.census_cells(0, doms)
    for (t, ly, cts, w0), g in zip(fields, got):
        cur, liquid = ly == 1, t == 5
        assert g["superheated"] == np.sum(cur & liquid & (cts > 1400))
        assert g["undercooled"] == np.sum(cur & liquid & (cts <= 1400))
        assert g["active"] == np.sum(cur & (t == 2))
        assert g["solid"] == np.sum(cur & (t == 1))
        assert g["remaining"] == np.sum(~cur & liquid)
        window = (cur & liquid)[w0:]
        assert g["next_cts"] == (cts[w0:][window].min() if window.any() else 2**64 - 1)

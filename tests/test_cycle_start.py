"""The persistent kernel's cycle start under the capture pass, its block-owned claim lists and its
meetings, where they can go wrong: launches of one and two cycles (no site marked, one marked),
dense nucleation (many sites firing in one cycle, next to each other and to captured cells), more
domains than blocks, and a grid so small that a block's claim queue and claim list overflow. All
results are whole numbers and reference-order floats: compared bit for bit."""
import os

import numpy as np
import pytest

import exaca_b200 as ex
from exaca_b200 import batch
from gen_inputs import C_TEMPLATE
from oracle_port import Oracle

pytestmark = pytest.mark.gpu


def directional(tmp_path, **kw):
    prm = dict(name="start", out=str(tmp_path), nx=21, ny=19, nz=23, G=1e6, R=1e6, density=2e4, dtn=2.0, sigma=0.3, N=12,
               frac=0.02)
    prm.update(kw)
    path = os.path.join(str(tmp_path), "start.txt")
    with open(path, "w") as f:
        f.write(C_TEMPLATE.format(**prm))
    return path


def equal(pool, slot, o, where):
    f = o.fields()
    gid, ct = pool.copy_out(slot)
    dl, _, _ = pool.copy_octahedra(slot)
    for name, a, b in (("CellType", ct, f["cell_type"]), ("GrainID", gid, f["grain_id"]), ("DiagonalLength", dl, f["dl"])):
        assert np.array_equal(a, b), f"{where}: {np.sum(a != b)} {name} differ"


@pytest.mark.parametrize("kw", [
    dict(),
    dict(density=2e5, sigma=0.02),                    # a fifth of the cells, many in one cycle
    dict(density=1e6, sigma=0.02, nx=5, ny=4, nz=6),  # nearly every cell of a tiny domain
    dict(density=500, sigma=1.0, frac=0.3),
])
def test_launch_lengths_and_dense_nucleation(lib, tmp_path, kw):
    inp = directional(tmp_path, **kw)
    p = ex.Problem.from_file(inp)
    o = Oracle(inp)
    pool = ex.Pool(0, list_capacity=p.geometry.active_size)
    slot = pool.admit(p, device_check=False)
    done = 0
    for n in (1, 1, 2, 3, 40, 1, 64, 150, 2, 300):
        pool.step(n)
        o.step(n)
        done += n
        equal(pool, slot, o, f"cycle {done}")
    pool.close()


@pytest.mark.parametrize("n_domains,divisor", [(9, 0), (160, 0), (160, 32)])
def test_domains_started_by_several_warps(lib, n_domains, divisor):
    params = batch.process_map(n_domains, seed=21, side=(6, 12), G=(1e6, 4e6), R=(5e5, 1e6), density=(1e15, 1e16))
    probs = batch.build_problems(params)
    plain = batch.solve_plain(probs)
    pool = ex.Pool(0, list_capacity=sum(p.geometry.active_size for p in probs))
    try:
        pool.set_grid(divisor)
        slots = [pool.admit(p, device_check=True) for p in probs]
        pool.run_all(chunk_cycles=333)
        for i, s in enumerate(slots):
            gid, ct = pool.copy_out(s)
            assert np.array_equal(gid, plain["grain_id"][i]) and np.array_equal(ct, plain["cell_type"][i]), f"domain {i}"
            assert pool.status(s).cycle == plain["cycle"][i], f"domain {i}"
    finally:
        pool.close()


@pytest.mark.parametrize("config", range(4))
def test_queue_and_claim_list_overflow(lib, config):
    # 4 blocks: thousands of flagged records and claims per block and cycle
    p = ex.Problem.directional(160, 150, 40, G=1e6, R=1e6, n_ratio=8, nucleation_density=2000.0, dTN=3.0, dTsigma=0.5,
                               fract_surface_active=0.3)
    res = []
    for divisor in (1, 32):
        pool = ex.Pool(0, list_capacity=p.geometry.active_size)
        slot = pool.admit(p, device_check=False)
        pool.set_config(config)
        pool.set_grid(divisor)
        for n in (40, 1, 60):
            pool.step(n)
        st = pool.status(slot)
        assert st.error == 0 and st.liquid > 0
        res.append(pool.copy_out(slot) + (st.nn, st.liquid))
        pool.close()
    assert all(np.array_equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("dtn", [3.0, 60.0])
def test_cycles_that_do_nothing(lib, tmp_path, dtn):
    # one seed in a corner of a wide, late front: stretches of cycles without an eligible record,
    # without claims, and (dtn 60) ended by a nucleation; stepped across them in every way
    inp = directional(tmp_path, nx=9, ny=8, nz=30, G=5e6, R=2e5, density=3e3, dtn=dtn, N=25, frac=0.03)
    p = ex.Problem.from_file(inp)
    o = Oracle(inp)
    o.step(2000)
    for chunks in ((2000,), (1, 2, 997, 1000), tuple([37] * 54 + [2])):
        assert sum(chunks) == 2000
        pool = ex.Pool(0, list_capacity=p.geometry.active_size)
        slot = pool.admit(p, device_check=False)
        for n in chunks:
            pool.step(n)
        assert pool.status(slot).cycle == 2000
        equal(pool, slot, o, f"chunks {chunks[:4]}")
        pool.close()


@pytest.mark.parametrize("config", [0, 2, 3])
@pytest.mark.parametrize("n,frac,divisor", [(12, 0.02, 0), (20, 0.15, 32), (26, 0.3, 32), (26, 0.3, 16)])
def test_few_and_many_per_block(lib, tmp_path, config, n, frac, divisor):
    # from no record of a block to more than its warps (16), its threads and beyond: on 4 or 9 blocks
    # the flagged records and claims per block run over every such edge as the front grows
    inp = directional(tmp_path, nx=n, ny=n - 1, nz=n, density=800, sigma=0.4, N=14, frac=frac)
    p = ex.Problem.from_file(inp)
    o = Oracle(inp)
    pool = ex.Pool(0, list_capacity=p.geometry.active_size)
    pool.set_config(config)
    pool.set_grid(divisor)
    slot = pool.admit(p, device_check=False)
    for k in (30, 90, 200):
        pool.step(k)
        o.step(k)
        equal(pool, slot, o, f"{k} cycles on")
    pool.close()

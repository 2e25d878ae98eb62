"""Active lists at their capacity (1024 records, the smallest that a pool takes): initial cells, captures
or nucleations beyond it are flagged, the list ends at its last slot with every slot below it written,
and the pool can still be stepped, read and emptied."""
import numpy as np
import pytest

import exaca_b200 as ex

pytestmark = pytest.mark.gpu


def problem(nx=60, ny=59, nz=9, density=10.0, dtn=5.0, sigma=0.5, frac=1.0):
    return ex.Problem.directional(nx, ny, nz, G=1e6, R=1e6, n_ratio=10, nucleation_density=density, dTN=dtn, dTsigma=sigma,
                                  fract_surface_active=frac)


@pytest.mark.parametrize("config", range(ex.STEP_CONFIGS))
@pytest.mark.parametrize("kw,at_once", [
    (dict(), True),                                                              # by admission
    (dict(nx=64, ny=64, nz=40, frac=0.05), False),                               # by captures
    (dict(nx=30, ny=31, nz=32, density=1e6, dtn=2.0, sigma=0.02, frac=0.003), False),  # by nucleations
])
def test_past_the_capacity(lib, config, kw, at_once):
    p = problem(**kw)
    pool = ex.Pool(0, list_capacity=1)
    try:
        pool.set_config(config)
        slot = pool.admit(p, device_check=False)
        assert pool.status(slot).error == (ex.FLAG_LIST_OVERFLOW if at_once else 0)
        for n in (1, 2, 60, 300, 1):
            pool.step(n)
        assert pool.status(slot).error == ex.FLAG_LIST_OVERFLOW
        gid, ct = pool.copy_out(slot)
        pool.copy_octahedra(slot)
        assert gid.size == ct.size == p.geometry.domain_size
        with pytest.raises(ex.ExacaError):
            pool.run_plain(slot)
        pool.retire(slot)
        again = pool.admit(problem(nx=8, ny=8, nz=8, frac=0.1), device_check=True)
        pool.step(5)
        assert pool.status(again).error == ex.FLAG_LIST_OVERFLOW  # the flag stays with the pool
    finally:
        pool.close()


def test_at_the_capacity(lib):
    # the 32 x 32 cells of the bottom plane, all active: a full list is no overflow
    p = problem(nx=30, ny=30, nz=1, density=0.0)
    assert np.sum(p.fields()["cell_type"] == 2) == 1024
    res = []
    for capacity in (1, 1 << 14):
        pool = ex.Pool(0, list_capacity=capacity)
        slot = pool.admit(p, device_check=True)
        pool.run_all(chunk_cycles=100)
        st = pool.status(slot)
        assert st.error == 0 and st.liquid == 0
        res.append((st.cycle,) + pool.copy_out(slot))
        pool.close()
    assert res[0][0] == res[1][0]
    for a, b in zip(res[0][1:], res[1][1:]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("chunk", [1, 7, 1000])
def test_dropped_records_leave_the_list(lib, chunk):
    # solves one after the other in a list of 2.4 times their 1024 records, of which no cell ever claims another:
    # the records dropped in cycles without claims, and in the last cycles of a launch, make room too
    p = problem(nx=30, ny=30, nz=1, density=0.0)
    pool = ex.Pool(0, list_capacity=2500)
    try:
        for solve in range(5):
            slot = pool.admit(p, device_check=False)
            for _ in range(max(1, 35 // chunk)):
                pool.step(chunk)
            st = pool.status(slot)
            assert st.error == 0, f"solve {solve}"
            _, ct = pool.copy_out(slot)
            assert not np.any(ct == 2)
            pool.retire(slot)
    finally:
        pool.close()

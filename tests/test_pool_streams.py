"""A pool's set-up and its tables go out on the pool's own stream, whose kernels read them: nothing of it
is ordered by, or waits for, work that a caller has on the device's legacy stream. Pools stepped from several
threads at a time do not disturb each other."""
import threading

import numpy as np
import pytest

import exaca_b200 as ex

pytestmark = pytest.mark.gpu


def test_set_up_does_not_go_through_the_legacy_stream(lib):
    import torch

    p = ex.Problem.directional(20, 21, 12, G=1e6, R=1e6, n_ratio=12, nucleation_density=2000.0, dTN=2.0, dTsigma=0.3,
                               fract_surface_active=0.3)

    def first_calls():
        pool = ex.Pool(0, list_capacity=p.geometry.active_size)
        slot = pool.admit(p, device_check=False)
        return pool, pool.grain_stats(slot)

    pool, want = first_calls()
    pool.close()
    torch.cuda._sleep(1)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    torch.cuda._sleep(2_000_000_000)  # about a second on the legacy stream
    done.record()
    pool, got = first_calls()
    still_running = not done.query()
    torch.cuda.synchronize()
    pool.close()
    assert got == want
    assert still_running


@pytest.mark.parametrize("n_pools", [2, 8])
def test_pools_stepped_from_several_threads(lib, n_pools):
    # short lists, whose launches run side by side, and one long list
    probs = [ex.Problem.directional(n, n + 1, n + 3, G=1e6, R=1e6, n_ratio=10, nucleation_density=500.0, dTN=3.0,
                                    dTsigma=0.5, fract_surface_active=0.1)
             for n in [14 + k for k in range(n_pools - 1)] + [150]]
    alone = []
    for p in probs:
        pool = ex.Pool(0, list_capacity=p.geometry.active_size)
        slot = pool.admit(p, device_check=True)
        pool.step(1500)
        alone.append(pool.copy_out(slot))
        pool.close()
    got = [None] * n_pools

    def work(k):
        pool = ex.Pool(0, list_capacity=probs[k].geometry.active_size)
        slot = pool.admit(probs[k], device_check=True)
        for _ in range(15):
            pool.step(100)
            assert pool.status(slot).error == 0
        got[k] = pool.copy_out(slot)
        pool.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(n_pools)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(n_pools):
        assert all(np.array_equal(a, b) for a, b in zip(got[k], alone[k])), f"pool {k}"

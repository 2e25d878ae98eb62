"""A pool's set-up and its tables go out on the pool's own stream, whose kernels read them: nothing of it
is ordered by, or waits for, work that a caller has on the device's legacy stream."""
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

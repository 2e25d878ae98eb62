"""The autotuner times every configuration on launches of that configuration, the same number of cycles in
each, whatever the pool chose before; without one fixed, launches take the shape for the list's length."""
import pytest

import exaca_b200 as ex
from exaca_b200 import batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trial", [1, 7, 20])
def test_trials_run_what_they_time(lib, trial):
    probs = batch.build_problems(batch.process_map(10, seed=5, side=(10, 26)))
    pool = ex.Pool(0, list_capacity=sum(p.geometry.active_size for p in probs))
    try:
        slots = [pool.admit(p, device_check=True) for p in probs]
        before = pool.config_cycles()
        for _ in range(2):  # the second on a list that a tuned shape has run
            config, ms = pool.autotune(trial)
            after = pool.config_cycles()
            assert [a - b for a, b in zip(after, before)] == [trial] * ex.STEP_CONFIGS
            assert config == ms.index(min(ms)) and min(ms) > 0
            before = after
        assert pool.status(slots[0]).cycle == 2 * trial * ex.STEP_CONFIGS
        pool.step(3)
        assert pool.config_cycles()[config] == before[config] + 3
    finally:
        pool.close()


def test_shape_follows_the_list(lib):
    p = batch.build_problems(batch.process_map(1, seed=5, side=(10, 26)))[0]
    pool = ex.Pool(0, list_capacity=p.geometry.active_size)
    try:
        slot = pool.admit(p, device_check=False)
        pool.status(slot)
        pool.step(5)
        assert pool.config_cycles()[3] == 5  # a short list
        for c in (0, 3, 1):
            n = pool.config_cycles()[c]
            pool.set_config(c)
            pool.step(4)
            assert pool.config_cycles()[c] == n + 4
    finally:
        pool.close()

"""The census of caller-held fields where it reads sixteen cells per step (every thread of the largest
domain has that many): tails of 0-15 cells, domains smaller than a step, fields on and off the 16-byte
boundary in one call, windows that begin and end inside a step. Counts are compared exactly."""
import numpy as np
import pytest

import exaca_b200 as ex

pytestmark = pytest.mark.gpu

ALIGNED, UNALIGNED = 0, 1  # cells by which a domain's fields lie off a 256-byte boundary


@pytest.mark.parametrize("sizes,largest", [
    ([12288 * 2 + 3] + [1, 15, 16, 17, 31, 0] + [4096 + k for k in range(249)], 24579),  # 256 domains: 3 blocks each
    ([41003 + k for k in range(64)], 41066),                                             # 10 blocks
    ([1212416 + 48, 1212416 - 5, 7], 1212464),                                           # 198 blocks
])
def test_census_of_long_domains(lib, sizes, largest):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = -(-4 * sms // len(sizes))
    assert max(sizes) == largest >= 16 * blocks * 256  # the domains for which the wide reads are chosen
    rng = np.random.default_rng(len(sizes))
    starts, end = [], 0
    for n in sizes:
        starts.append(end)
        end += (n + 16 + 255) // 256 * 256
    t = rng.integers(-1, 8, end, dtype=np.int8)
    layer = rng.integers(-1, 2, end, dtype=np.int8)
    cts = rng.integers(0, 1 << 30, end, dtype=np.int32)
    dev = [torch.from_numpy(a).cuda() for a in (t, layer, cts)]
    for shift in (ALIGNED, UNALIGNED):
        doms, want = [], []
        for k, (n, s) in enumerate(zip(sizes, starts)):
            s += (k + shift) % 2 * (1 + k % 15)  # every other domain off the boundary, by 1-15 cells
            w0 = n // 3
            w1 = n - n // 5
            cycle, number = 1 << 29, k % 2
            doms.append(dict(cell_type=dev[0].data_ptr() + s, layer_id=dev[1].data_ptr() + s,
                             crit_time_step=dev[2].data_ptr() + 4 * s, domain_size=n, active_size=w1 - w0, cycle=cycle,
                             layer=number, window_start=w0))
            ct, ly, c = t[s:s + n], layer[s:s + n], cts[s:s + n]
            cur, liquid = ly == number, ct == ex.LIQUID
            window = (cur & liquid)[w0:w1]
            want.append(dict(superheated=int(np.sum(cur & liquid & (c > cycle))),
                             undercooled=int(np.sum(cur & liquid & (c <= cycle))),
                             active=int(np.sum(cur & (ct == ex.ACTIVE))), solid=int(np.sum(cur & (ct == ex.SOLID))),
                             remaining=int(np.sum(~cur & liquid)),
                             next_cts=int(c[w0:w1][window].min()) if window.any() else 2**64 - 1))
        torch.cuda.synchronize()
        for k, (g, w) in enumerate(zip(ex.census_cells(0, doms), want)):
            assert {q: g[q] for q in w} == w, f"domain {k} of {sizes[k]} cells"

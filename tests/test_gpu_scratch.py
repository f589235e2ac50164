"""The library's memory pool: bounded between calls, and given back by
stc_release_scratch and with a device's contexts (include/stc.h)."""
import ctypes

import numpy as np
import pytest

from stcdb_gb300.pipeline import Pipeline, StcConfig

from parity import trace_and_box
from test_gpu_sort import _sort_fn

pytestmark = pytest.mark.gpu

KEPT = 512 << 20
SLACK = 8 << 20  # of the driver's own


def _sort(lib, n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=g)
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    assert _sort_fn(lib)(k.data_ptr(), v.data_ptr(), ko.data_ptr(), vo.data_ptr(), n, 32, 0) == 0
    return before, torch.cuda.mem_get_info()[0], (k, v, ko, vo)


@pytest.mark.parametrize("n", [3_000_001, 20_000_000, 70_000_000])
def test_sort_scratch_is_bounded_and_given_back(built_cuda, n):
    import torch
    from stcdb_gb300._lib import load_library
    lib = load_library("libstc")
    _sort(lib, 1000, 1)  # loads the kernels
    for seed in (2, 3):  # again after the pool has been given back
        assert lib.stc_release_scratch(0) == 0
        before, after, (k, v, ko, vo) = _sort(lib, n, seed)
        assert before - after <= KEPT + SLACK
        assert lib.stc_release_scratch(0) == 0
        assert before - torch.cuda.mem_get_info()[0] <= SLACK
        want, at = torch.sort(k.long() & 0xFFFFFFFF, stable=True)
        assert torch.equal(ko.long() & 0xFFFFFFFF, want) and torch.equal(vo.long(), at)
        del k, v, ko, vo, want, at


def test_the_last_context_takes_the_pool_with_it(built_cuda):
    """Contexts that come and go, with flushes between, leave no memory; one
    outlives another's end and the release of the scratch."""
    import torch
    from stcdb_gb300._lib import load_library
    from stcdb_gb300.tracegen import hotspot_grid
    lib = load_library("libstc")
    tr, mbr = trace_and_box(hotspot_grid(5000, n_hotspots=5, box_m=2000.0, grid_n=12, sigma_m=100.0, seed=3), 8)
    cfg = StcConfig(num_objects=5000, reach_distance=8.0, min_meet_time=2, grid_capacity=40, grid_amplify=4.0,
                    num_meeting_buckets=1 << 20, kv_restriction=1 << 20, ctf_count=16)

    def run(p, a, b):
        for t in range(a, b):
            p.step(tr[t], t)
        return p.flush()

    def keys(p):
        info = p.ctb_info()
        return info.kv_count, info.key_bytes

    free = []
    for _ in range(3):
        with Pipeline(cfg, mbr, tr[0]) as p:
            with Pipeline(cfg, mbr, tr[0]) as q:
                run(q, 0, 8)
                want = keys(q)
                run(p, 0, 5)
                assert lib.stc_release_scratch(0) == 0
            p.flush()
            assert want[0] > 0
        with Pipeline(cfg, mbr, tr[0]) as p:
            run(p, 0, 8)
            assert keys(p) == want
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[2] >= free[1] - SLACK

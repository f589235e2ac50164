"""The pair tests' jobs taken from a common counter (csrc/stc_refine.cu,
job_shares) against jobs dealt out beforehand: whole-number results are equal.
One block an SM makes eight jobs a warp of a crowd of 60k objects."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import Pipeline, StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import trace_and_box

pytestmark = pytest.mark.gpu

N, STEPS = 60000, 5


@pytest.fixture(scope="module")
def crowd():
    return trace_and_box(hotspot_grid(N, n_hotspots=10, box_m=3000.0, grid_n=16, sigma_m=100.0, seed=41), STEPS)


def _run(crowd, **more):
    tr, mbr = crowd
    out = []
    with Pipeline(StcConfig(num_objects=N, reach_distance=10.0, min_meet_time=2, grid_capacity=100, grid_amplify=8.0,
                            num_meeting_buckets=1 << 25, refine_blocks_per_sm=1, **more), mbr, tr[0]) as p:
        for t in range(STEPS):
            p.step(tr[t], t)
            m = p.drain()
            m = m[np.lexsort((m["end"], m["start"], m["pid_hi"], m["pid_lo"]))]
            s = p.stats()
            out.append((m.tobytes(), s.pair_tests, s.hits, s.new_candidates, s.taken_buckets, s.emitted))
    return out


@pytest.fixture(scope="module")
def dealt(built_cuda, crowd):
    return _run(crowd, job_chunk=8, refine_chunk=32)


@pytest.mark.parametrize("more", [dict(refine_chunk=32), dict(refine_chunk=64), dict(refine_chunk=32, step_slices=7),
                                  dict()])
def test_shared_jobs_equal_dealt_ones(crowd, dealt, more):
    got = _run(crowd, **more)
    assert dealt[-1][2] > 1_000_000
    for t, (a, b) in enumerate(zip(got, dealt)):
        assert a == b, f"step {t}: counters {a[1:]} against {b[1:]}"

"""Launch shapes that stand for each other give what the others give: jobs
dealt out (a job_chunk other than the built-in 8) and by demand, and the
autotuner's setting, which names every field, against the fields left at 0."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import autotune
from stcdb_gb300.pipeline import StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import trace_and_box
from test_gpu_job_share import N, _run, crowd  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [dict(), dict(job_chunk=8), dict(step_slices=5)])
def test_dealt_jobs_equal_shared_ones(built_cuda, crowd, more):  # noqa: F811
    dealt = _run(crowd, job_chunk=9, refine_chunk=32)
    got = _run(crowd, refine_chunk=32, **more)
    assert dealt[-1][2] > 1_000_000
    for t, (a, b) in enumerate(zip(got, dealt)):
        assert a == b, f"step {t}: counters {a[1:]} against {b[1:]}"


def test_autotune_reports_a_setting_it_ran(built_cuda):
    """The setting is not slower than the configuration given by its own
    figures, and keeps the built-in shape or one at least 1% faster."""
    tr, mbr = trace_and_box(hotspot_grid(30000, n_hotspots=30, box_m=3000.0, grid_n=16, sigma_m=120.0, seed=10), 6)
    cfg = StcConfig(num_objects=30000, reach_distance=10.0, min_meet_time=3, grid_capacity=50, grid_amplify=2.0,
                    num_meeting_buckets=1_500_000)
    chosen, rep = autotune(cfg, mbr, np.stack(tr), capacities=[50])
    shape = (chosen.job_chunk, chosen.refine_chunk, chosen.refine_blocks_per_sm, chosen.hits_blocks_per_sm)
    assert shape == (8, 0, 8, 16) or rep["best_step_ms"] <= 0.9901 * rep["base_step_ms"]
    assert rep["best_step_ms"] <= rep["base_step_ms"]
    again, rep2 = autotune(chosen, mbr, np.stack(tr), capacities=[chosen.grid_capacity])
    assert rep2["base_step_ms"] > 0 and rep2["best_step_ms"] <= rep2["base_step_ms"]

"""The general path of the table update: its kernels are cut into step_slices
launches as the tiled path's are."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import Pipeline, StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import trace_and_box

pytestmark = pytest.mark.gpu

N, STEPS = 12000, 10


@pytest.fixture(scope="module")
def trace(built_cuda):
    return trace_and_box(hotspot_grid(N, n_hotspots=12, box_m=2500.0, grid_n=14, sigma_m=150.0, seed=22), STEPS)


def _config(**more):
    return StcConfig(**{**dict(num_objects=N, reach_distance=8.0, min_meet_time=2, grid_capacity=40, grid_amplify=2.0,
                               num_meeting_buckets=300_007), **more})


def _row(p):
    m = p.drain()
    m = m[np.lexsort((m["end"], m["start"], m["pid_hi"], m["pid_lo"]))]
    s = p.stats()
    return m.tobytes(), s.hits, s.new_candidates, s.taken_buckets, s.emitted


def _steps(trace, cfg):
    tr, mbr = trace
    rows, launches, halos = [], [], []
    with Pipeline(cfg, mbr, tr[0]) as p:
        for t in range(STEPS):
            p.step(tr[t], t)
            rows.append(_row(p))
            launches.append(p.stats().kernel_launches)
            halos.append(p.table_halo())
    return rows, launches, halos


@pytest.mark.parametrize("slices", [2, 7, 64])
@pytest.mark.parametrize("per_bin", [1, 40])
def test_slices_cut_every_long_kernel(trace, slices, per_bin):
    """Pair tests, tiled update, general update and sweep: one launch each, or
    one a slice."""
    want, whole, halos = _steps(trace, _config(hit_capacity=391 * per_bin))
    assert 0 in halos
    got, cut, _ = _steps(trace, _config(hit_capacity=391 * per_bin, step_slices=slices))
    assert got == want
    assert [c - w for c, w in zip(cut, whole)] == [4 * (slices - 1)] * STEPS

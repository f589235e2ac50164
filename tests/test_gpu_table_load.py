"""The tiled table update at the loads where its rule reaches far back (halos
of up to 15 tiles) and gives up (csrc/stc_insert.cuh, fuse_halo), against the
general path on the same steps."""
import pytest

from stcdb_gb300.pipeline import StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import trace_and_box
from test_gpu_table import _run

pytestmark = pytest.mark.gpu

N = 20000


@pytest.fixture(scope="module")
def steps():
    return trace_and_box(hotspot_grid(N, n_hotspots=20, box_m=3000.0, grid_n=16, sigma_m=150.0, seed=91), 10)


@pytest.fixture(scope="module")
def live(built_cuda, steps):
    """The most live meetings of a step, with room to spare."""
    tr, mbr = steps
    return max(row[3] for row in _run(StcConfig(num_objects=N, reach_distance=9.0, min_meet_time=2, grid_capacity=50,
                                                grid_amplify=2.0, num_meeting_buckets=1 << 23), tr, mbr))


# (live meetings + hits) a slot, about; with 0.55 the halo is short, from about
# 0.85 on the general path takes the step
@pytest.mark.parametrize("load", [0.55, 0.65, 0.72, 0.78, 0.84, 0.9, 1.0])
def test_loaded_tables_equal_the_general_path(steps, live, load):
    tr, mbr = steps
    base = dict(num_objects=N, reach_distance=9.0, min_meet_time=2, grid_capacity=50, grid_amplify=2.0,
                num_meeting_buckets=int(2 * live / load) | 1)
    tiled = _run(StcConfig(**base), tr, mbr)
    general = _run(StcConfig(**base, hit_capacity=1), tr, mbr)
    assert len(tiled) == len(general)
    for t, (a, b) in enumerate(zip(tiled, general)):
        assert a == b, f"step {t} differs: counters {a[1:]} against {b[1:]}"

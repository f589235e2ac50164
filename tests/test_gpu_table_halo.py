"""The path of the table update that a context reports (stc_table_halo): the
comparisons of the tiled update with the general one (test_gpu_table*.py) do
compare the two, over short and long halos."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import Pipeline, StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import trace_and_box

pytestmark = pytest.mark.gpu

N = 20000


@pytest.fixture(scope="module")
def steps(built_cuda):
    return trace_and_box(hotspot_grid(N, n_hotspots=20, box_m=3000.0, grid_n=16, sigma_m=150.0, seed=91), 10)


def _run(steps, **more):
    """Per step the halo, and the meetings and counters."""
    tr, mbr = steps
    cfg = StcConfig(num_objects=N, reach_distance=9.0, min_meet_time=2, grid_capacity=50, grid_amplify=2.0, **more)
    halos, out = [], []
    with Pipeline(cfg, mbr, tr[0]) as p:
        assert p.table_halo() == 0
        for t in range(len(tr)):
            p.step(tr[t], t)
            halos.append(p.table_halo())
            m = p.drain()
            m = m[np.lexsort((m["end"], m["start"], m["pid_hi"], m["pid_lo"]))]
            s = p.stats()
            out.append((m.tobytes(), s.hits, s.new_candidates, s.taken_buckets, s.emitted))
    return halos, out


def test_sparse_tables_are_updated_in_tiles_and_full_bins_the_general_way(steps):
    tiled, a = _run(steps, num_meeting_buckets=1 << 23)
    general, b = _run(steps, num_meeting_buckets=1 << 23, hit_capacity=1)
    assert all(1 <= h <= 15 for h in tiled) and general == [0] * len(general)
    assert a == b


def test_loaded_tables_reach_long_halos_and_the_general_path(steps):
    """From sparse to full: the halo of the step with the most meetings grows
    with the load, beyond the seven tiles of the first rule, and then there is
    none."""
    most = [row[3] for row in _run(steps, num_meeting_buckets=1 << 23)[1]]
    live, fullest = max(most), int(np.argmax(most))
    seen, there = set(), []
    for load in [0.2, 0.4, 0.55, 0.6, 0.65, 0.68, 0.7, 0.72, 0.74, 0.76, 0.78, 0.8, 0.84, 0.9, 1.0]:
        table = dict(num_meeting_buckets=int(2 * live / load) | 1)
        halos, out = _run(steps, **table)
        assert out == _run(steps, **table, hit_capacity=1)[1]
        seen.update(halos)
        there.append(halos[fullest])
    assert there[0] >= 1 and there[-1] == 0 and max(seen) > 7, (sorted(seen), there)
    in_tiles = [h for h in there if h]
    assert in_tiles == sorted(in_tiles) and there[len(in_tiles):] == [0] * (len(there) - len(in_tiles)), there

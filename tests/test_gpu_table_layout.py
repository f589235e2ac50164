"""The meeting table's two layouts (csrc/stc_table.cu): tiles packed by the
tiled update, meetings in their slots for the general path. Steps that change
between the two, steps whose hits overflow a bin while the tiles are packed
(the pair tests run again), a time given twice, and a checkpoint in between
must all leave what the general path alone leaves."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import Pipeline, StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import trace_and_box

pytestmark = pytest.mark.gpu

N, STEPS = 12000, 14


@pytest.fixture(scope="module")
def positions():
    """Crowded steps, and steps in which three objects of four stand alone."""
    tr, mbr = trace_and_box(hotspot_grid(N, n_hotspots=12, box_m=2500.0, grid_n=14, sigma_m=150.0, seed=77), STEPS)
    tr = np.array(tr)
    rng = np.random.default_rng(5)
    apart = rng.random((N, 2)) * (mbr[2] - mbr[0], mbr[3] - mbr[1]) + (mbr[0], mbr[1])
    away = np.arange(N) % 4 != 0
    for t in range(STEPS):
        if t % 7 in (0, 1, 3, 5):
            tr[t][away] = apart[away]
    return np.ascontiguousarray(tr), mbr


def _config(**more):
    return StcConfig(num_objects=N, reach_distance=8.0, min_meet_time=2, grid_capacity=40, grid_amplify=2.0,
                     num_meeting_buckets=300_007, **more)


def _row(p):
    m = p.drain()
    m = m[np.lexsort((m["end"], m["start"], m["pid_hi"], m["pid_lo"]))]
    s = p.stats()
    return m.tobytes(), s.hits, s.new_candidates, s.taken_buckets, s.emitted


def _run(cfg, positions, times, save=None):
    tr, mbr = positions
    out = []
    with Pipeline(cfg, mbr, tr[0]) as p:
        for k, t in enumerate(times):
            p.step(tr[k], t)
            out.append(_row(p))
            if save and k in (3, 6, 9):
                p.checkpoint(save)
    return out


TWICE = [0, 1, 2, 3, 3, 4, 5, 5, 6, 7, 8, 9, 9, 10]


@pytest.mark.parametrize("times", [list(range(STEPS)), TWICE])
# records a bin of 391: the crowded steps overflow some, most or none
@pytest.mark.parametrize("per_bin", [8, 40, 90, 0])
def test_layouts_change_with_the_path(built_cuda, positions, times, per_bin):
    want = _run(_config(hit_capacity=1), positions, times)
    assert sum(w[4] for w in want) > 0 and max(w[1] for w in want) > 4 * min(w[1] for w in want)
    got = _run(_config(hit_capacity=391 * per_bin), positions, times)
    for k, (a, b) in enumerate(zip(got, want)):
        assert a == b, f"step {k}: counters {a[1:]} against {b[1:]}"


def test_checkpoint_of_packed_tiles(built_cuda, positions, tmp_path):
    """The run goes on after a checkpoint, and a restored one from its file."""
    tr, mbr = positions
    path = str(tmp_path / "c")
    want = _run(_config(), positions, range(STEPS))
    assert _run(_config(), positions, range(STEPS), save=path) == want
    with Pipeline.restore(path) as q:
        q.drain()
        for t in range(10, STEPS):
            q.step(tr[t], t)
            assert _row(q)[0] == want[t][0], f"step {t}"

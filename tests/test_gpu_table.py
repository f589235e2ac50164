"""The tiled table update and sweep (csrc/stc_table.cu) against the general
path (one random table access per hit, then the sweep) on the same steps:
meetings, box bits and counters are whole numbers and must be equal. A hit
buffer of one record per bin overflows, so it forces the general path."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import Pipeline, StcConfig, StcError
from stcdb_gb300.tracegen import hotspot_grid

from parity import trace_and_box

pytestmark = pytest.mark.gpu

TILE = 768  # TILE_SLOTS of csrc/stc_pipeline.cuh


def _run(cfg, tr, mbr):
    p = Pipeline(cfg, mbr, tr[0])
    out = []
    try:
        for t in range(len(tr)):
            try:
                p.step(tr[t], t)
            except StcError as e:  # a full table: every path reports it
                out.append(("error", e.status))
                break
            m = p.drain()
            m = m[np.lexsort((m["end"], m["start"], m["pid_hi"], m["pid_lo"]))]
            s = p.stats()
            out.append((m.tobytes(), s.hits, s.new_candidates, s.taken_buckets, s.emitted))
    finally:
        p.close()
    return out


# table sizes: the fewest tiles the tiled path takes and one slot around it,
# odd sizes that cut uneven tiles, a loaded table (long probe chains across
# tile ends) and a sparse one of whole tiles
@pytest.mark.parametrize("objects,buckets", [(3000, 14 * TILE - 1), (3000, 14 * TILE), (3000, 14 * TILE + 1),
                                             (3000, 20 * TILE + 333), (12000, 130_003), (12000, 262_144),
                                             (12000, 1 << 20)])
def test_tiled_path_equals_the_general_path(built_cuda, objects, buckets):
    n_hot = max(objects // 1000, 3)
    tr, mbr = trace_and_box(hotspot_grid(objects, n_hotspots=n_hot, box_m=2500.0, grid_n=14, sigma_m=150.0, seed=21), 12)
    base = dict(num_objects=objects, reach_distance=8.0, min_meet_time=2, grid_capacity=40, grid_amplify=2.0,
                num_meeting_buckets=buckets)
    tiled = _run(StcConfig(**base), tr, mbr)
    general = _run(StcConfig(**base, hit_capacity=1), tr, mbr)
    assert general[-1][0] == "error" or (sum(s[4] for s in general) > 0 and sum(s[2] for s in general) > 0)
    assert len(tiled) == len(general)
    for t, (a, b) in enumerate(zip(tiled, general)):
        assert a == b, f"step {t} differs: counters {a[1:]} against {b[1:]}"


def test_tiled_path_in_slices_and_after_a_restore(built_cuda, tmp_path):
    """Step slices cut the runs of tiles into launches; a restored context
    counts its tiles again before the first step."""
    tr, mbr = trace_and_box(hotspot_grid(12000, n_hotspots=12, box_m=2500.0, grid_n=14, sigma_m=150.0, seed=22), 10)
    base = dict(num_objects=12000, reach_distance=8.0, min_meet_time=2, grid_capacity=40, grid_amplify=2.0,
                num_meeting_buckets=300_007)
    want = _run(StcConfig(**base), tr, mbr)
    assert _run(StcConfig(**base, step_slices=7), tr, mbr) == want
    p = Pipeline(StcConfig(**base), mbr, tr[0])
    try:
        for t in range(5):
            p.step(tr[t], t)
        p.drain()
        p.checkpoint(str(tmp_path / "c"))
    finally:
        p.close()
    q = Pipeline.restore(str(tmp_path / "c"))
    try:
        for t in range(5, 10):
            q.step(tr[t], t)
            m = q.drain()
            m = m[np.lexsort((m["end"], m["start"], m["pid_hi"], m["pid_lo"]))]
            s = q.stats()
            assert (m.tobytes(), s.hits, s.new_candidates, s.taken_buckets, s.emitted) == want[t], f"step {t}"
    finally:
        q.close()

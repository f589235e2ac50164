"""The automatic hit buffer's device memory (csrc/stc_rules.cuh): small beside
a table of many slots for few objects, and not sized for all tiles by one
crowd's; the steps whose bins overflow leave what the general path leaves."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import Pipeline, StcConfig

pytestmark = pytest.mark.gpu

REC, TILE = 32, 768


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _used(n, slots, xy):
    before = _free()
    with Pipeline(StcConfig(num_objects=n, num_meeting_buckets=slots), (0.0, 0.0, 0.01, 0.01), xy):
        return before - _free()


def test_few_objects_in_a_large_table(built_cuda):
    """1000 objects in 2^28 slots (8.6 GB) against the same in 2^12: the table
    itself, bins of 32 records a tile of 768 slots, and the tiles' marks."""
    n, slots = 1000, 1 << 28
    xy = np.random.default_rng(1).random((n, 2)) * 0.01
    _used(n, 1 << 12, xy)  # loads the kernels
    assert _used(n, slots, xy) - _used(n, 1 << 12, xy) <= slots * REC * (1 + 32 / TILE + 1 / 128)


CROWD, N, STEPS = 1600, 20_000, 6


def _positions():
    """1600 objects of neighbouring ids within reach of each other, in every
    step; the others stand alone."""
    rng = np.random.default_rng(7)
    box = np.array([0.0, 0.0, 0.2, 0.2])
    apart = np.stack(np.meshgrid(np.arange(142), np.arange(142)), -1).reshape(-1, 2)[:N] * 0.0013 + 0.005
    tr = np.repeat(apart[None], STEPS, 0)
    for t in range(STEPS):
        tr[t, :CROWD] = (0.1, 0.1) + (rng.random((CROWD, 2)) - 0.5) * 4e-5  # 4.5 m across
        if t % 3 == 2:
            tr[t, : CROWD // 2] = apart[: CROWD // 2]
    return np.ascontiguousarray(tr), box


def _run(tr, box, window=False, **more):
    cfg = StcConfig(num_objects=N, reach_distance=10.0, min_meet_time=1, grid_capacity=100, grid_amplify=20.0,
                    num_meeting_buckets=1 << 26, emit_capacity=1 << 23, **more)
    out = []
    with Pipeline(cfg, box, tr[0]) as p:
        before = _free()
        for t in range(STEPS):
            if window:
                m = p.step_window(tr[t:t + 1], t, out=np.empty(1 << 22, dtype=p.drain().dtype))
            else:
                p.step(tr[t], t)
                m = p.drain()
            m = m[np.lexsort((m["end"], m["start"], m["pid_hi"], m["pid_lo"]))]
            s = p.stats()
            out.append((m.tobytes(), s.hits, s.new_candidates, s.taken_buckets, s.emitted))
        return out, before - _free()


def test_one_crowd_does_not_size_all_bins(built_cuda):
    """The crowd's 1.3M pairs lie in a few thousand of 87382 tiles, hundreds in
    each; the bins may grow to 48 records each (134 MB) or eight times the
    hits (328 MB), where the fullest bin's size for all would be 1.5 GB and
    more. Steps whose bins overflow equal those of the general path."""
    tr, box = _positions()
    want, _ = _run(tr, box, hit_capacity=1)
    got, grown = _run(tr, box)
    assert want[0][1] > 1_000_000 and sum(w[4] for w in want) > 500_000
    for t, (a, b) in enumerate(zip(got, want)):
        assert a == b, f"step {t}: counters {a[1:]} against {b[1:]}"
    assert grown <= (336 << 20)
    assert _run(tr, box, window=True)[0] == want

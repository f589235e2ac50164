"""The general path of the table update (csrc/stc_refine.cu): a step that the
tiles cannot take goes by its bins; steps after it may be told beforehand to
leave their hits in sequence and update the table beside the pair tests. Against the
oracle and against each other: on loaded tables, with bins that overflow, in
plain steps, windows and replayed graphs. Its kernels are cut into step_slices
launches as the tiled path's are."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import MEETING_DTYPE, Pipeline, StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import as_tuples, describe_diff, run_pair, trace_and_box

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
    one a slice. A step told to be general has four parts of pair tests, of
    their ends' marks and of the update at least, and two forms of the sweep."""
    want, whole, halos = _steps(trace, _config(hit_capacity=391 * per_bin))
    assert 0 in halos
    got, cut, _ = _steps(trace, _config(hit_capacity=391 * per_bin, step_slices=slices))
    assert got == want
    told = whole[0] - 5 + 16  # for the five kernels of one launch each: 2 + 4 * 3 + 2 launches
    assert set(whole) <= {whole[0], told}
    bins_cut, told_cut = whole[0] + 4 * (slices - 1), told + 3 * (max(slices, 4) - 4) + 2 * (slices - 1)
    assert cut[0] == bins_cut and set(cut) <= {bins_cut, told_cut}
    assert per_bin > 1 or cut[1:] == [told_cut] * (STEPS - 1)  # every step is general


@pytest.mark.parametrize("load", [0.3, 0.5, 0.58])
def test_loaded_table_equals_the_oracle(trace, load):
    """The crowd at up to `load` live meetings a slot: some steps in tiles, the
    others general, told and not."""
    tr, mbr = trace
    cfg = _config(num_meeting_buckets=1 << 20)
    live = max(r[3] for r in _steps(trace, cfg)[0])
    cfg = _config(num_meeting_buckets=int(live / load) | 1)
    halos, emitted = _steps(trace, cfg)[2], 0
    for t, g, o, gs, os_ in run_pair(cfg, tr, mbr):
        assert gs.hits == os_.hits
        assert np.array_equal(g, o), f"step {t}: " + describe_diff(g, o)
        emitted += len(o)
    assert emitted > 0 and (0 in halos or load < 0.5)


def _window(trace, cfg, sizes):
    tr, mbr = trace
    rows, t = [], 0
    with Pipeline(cfg, mbr, tr[0]) as p:
        for n in sizes:
            m = p.step_window(np.ascontiguousarray(tr[t:t + n]), t, out=np.empty(1 << 20, MEETING_DTYPE))
            t += n
            rows.append(np.ascontiguousarray(m).copy())
            last = p.stats()
        return np.concatenate(rows), last.hits, last.taken_buckets


# records a bin: none to speak of, too few in the crowd's tiles (overflows
# while the tiles are packed: the pair tests again), room for all
@pytest.mark.parametrize("graphs", [1, 2])
@pytest.mark.parametrize("more", [dict(hit_capacity=1), dict(hit_capacity=391 * 40), dict(hit_capacity=391 * 90),
                                  dict(load=0.5), dict(load=0.5, step_slices=5), {}])
def test_windows_and_graphs_take_the_same_paths(trace, graphs, more):
    tr, mbr = trace
    more = dict(more)
    if "load" in more:
        live = max(r[3] for r in _steps(trace, _config(num_meeting_buckets=1 << 20))[0])
        more["num_meeting_buckets"] = int(live / more.pop("load")) | 1
    plain, _, halos = _steps(trace, _config(**more))
    assert ("num_meeting_buckets" not in more and more != dict(hit_capacity=1)) or 0 in halos
    want = np.concatenate([np.frombuffer(r[0], MEETING_DTYPE) for r in plain])
    for sizes in ([STEPS], [1, 4, 2, 3]):
        got, hits, taken = _window(trace, _config(window_graphs=graphs, **more), sizes)
        assert (hits, taken) == (plain[-1][1], plain[-1][3])
        assert np.array_equal(as_tuples(got), as_tuples(want))


# records a bin of 391 tiles: none to speak of (general from the second step on),
# some overflow while the tiles are packed, so that the pair tests run again
@pytest.mark.parametrize("per_bin", [1, 8, 40, 90])
@pytest.mark.parametrize("graphs", [0, 1])
def test_overflowing_bins_equal_the_oracle(trace, per_bin, graphs):
    """Against a run with room for every hit, and the oracle: plain steps, and
    a window of replayed graphs."""
    import oracle
    tr, mbr = trace
    cfg = _config(hit_capacity=391 * per_bin, window_graphs=graphs)
    ref = oracle.Oracle(cfg, mbr, tr[0])
    try:
        want = [as_tuples(ref.step(tr[t], t)) for t in range(STEPS)]
    finally:
        ref.close()
    assert sum(len(w) for w in want) > 0
    if graphs:
        got, _, _ = _window(trace, cfg, [3, STEPS - 3])
        assert np.array_equal(as_tuples(got), as_tuples(np.concatenate(want)))
        return
    rows, _, halos = _steps(trace, cfg)
    room, _, tiled = _steps(trace, _config())
    assert 0 in halos and 0 not in tiled
    assert rows == room
    for t in range(STEPS):
        got = as_tuples(np.frombuffer(rows[t][0], MEETING_DTYPE))
        assert np.array_equal(got, want[t]), f"step {t}: " + describe_diff(got, want[t])

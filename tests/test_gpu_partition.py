"""Leaves at the sizes where the partition changes its ways, against the
oracle: around 256 kept members (k_leaf_small / k_leaf_big), fuller than the
leaf list holds in either, strips of one to more than 128 members, and
objects that leave the map box."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import StcConfig

from parity import run_pair, describe_diff

pytestmark = pytest.mark.gpu

BOX = np.array([-87.75, 41.75, -87.25, 42.25])
M = 1.0 / 111322.2  # degrees of latitude in a metre


def _clumps(sizes, spread_m, steps, seed, outside=0):
    """Clumps of the given sizes on a coarse grid of places, each member within
    spread_m of its place, walking up to 2 m a step; `outside` objects walk out
    of the map box."""
    rng = np.random.default_rng(seed)
    xy = []
    for k, s in enumerate(sizes):
        c = np.array([-87.7 + 0.03 * (k % 12), 41.8 + 0.04 * (k // 12)])
        xy.append(c + rng.uniform(-spread_m, spread_m, (s, 2)) * M)
    xy = np.concatenate(xy)
    tr = [xy]
    for _ in range(steps - 1):
        tr.append(tr[-1] + rng.uniform(-2, 2, xy.shape) * M)
    tr = np.stack(tr)
    for k in range(outside):  # by up to 30 m a step, through each side in turn
        tr[:, k] = [BOX[2], BOX[1] + 0.1 + 1e-5 * k] if k % 2 else [BOX[0] + 0.1 + 1e-5 * k, BOX[1]]
        tr[:, k, 0 if k % 2 else 1] += np.arange(steps) * (30 * M if k % 2 else -30 * M)
    return np.ascontiguousarray(tr)


@pytest.mark.parametrize("sizes,spread,cap,amplify", [
    ([255, 256, 257, 300, 31, 32, 33, 1, 2], 40.0, 1000, 1.0),   # one leaf a clump, either kernel
    ([129, 128, 127, 600, 700], 4.0, 1000, 1.0),                 # all in one or two strips: unordered from 129 on
    ([260, 400, 600], 8.0, 200, 1.2),                            # leaves cut at 240 members: the lowest pids stay
    ([700, 900, 1200], 10.0, 400, 1.0),                          # cut at 400
])
def test_leaf_sizes_match_the_oracle(built_cuda, sizes, spread, cap, amplify):
    tr = _clumps(sizes, spread, 7, seed=sum(sizes), outside=6)
    n = tr.shape[1]
    cfg = StcConfig(num_objects=n, reach_distance=6.0, min_meet_time=2, grid_capacity=cap, grid_amplify=amplify,
                    num_meeting_buckets=8_000_000, refine_size=8)
    total = 0
    for t, g, o, gs, os_ in run_pair(cfg, tr, BOX):
        assert np.array_equal(g, o), f"step {t}: {describe_diff(g, o)}"
        assert gs.hits > 0
        total += len(o)
    assert total > 0

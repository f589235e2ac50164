"""Box queries at the edges of their plan and rows (k_box_plan, k_box_rows):
query edges on decoded key corners and one double beside them (the float test
of the rows must leave those to the exact one), batches either side of the
rows-per-item rule, and a batch whose plan outgrows its buffers."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import QUERY_BOX, QUERY_DTYPE, StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from test_gpu_query import _compare, _ingest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def blocks_100(built_cuda):
    tc = hotspot_grid(30000, n_hotspots=30, box_m=3000.0, grid_n=16, sigma_m=120.0, seed=23)
    cfg = StcConfig(num_objects=30000, reach_distance=10.0, min_meet_time=3, max_meet_time=6, grid_capacity=50,
                    grid_amplify=1.2, num_meeting_buckets=1_500_000, kv_restriction=40_000, ctf_count=100,
                    ctb_retain=3)
    pipe, blocks, mbr = _ingest(cfg, tc, 15, 3)
    yield pipe, blocks, mbr
    pipe.close()


def _touching(pipe, mbr, n, seed):
    """n box queries, each with one edge at a key's decoded corner: on it, or
    one double short of it or past it."""
    rng = np.random.default_rng(seed)
    boxes = pipe.query_box(mbr)["mbr"]
    qs = np.zeros(n, QUERY_DTYPE)
    for i in range(n):
        x0, y0, x1, y1 = boxes[rng.integers(len(boxes))]
        s = 10 ** rng.uniform(-4.5, -2.5)
        q = [x0 - s, y0 - s, x1 + s, y1 + s]
        side = int(rng.integers(4))
        edge = (x1, y1, x0, y0)[side]  # the query's low edge at the key's high corner and vice versa
        q[side] = edge if i % 3 == 0 else np.nextafter(edge, np.inf if i % 3 == 1 else -np.inf)
        qs[i]["kind"], qs[i]["box"], qs[i]["t_end"] = QUERY_BOX, q, 0xFFFFFFFF
    return qs


@pytest.mark.parametrize("n", [1, 63, 64, 129])
def test_edges_on_key_corners(blocks_100, n):
    pipe, blocks, mbr = blocks_100
    _compare(pipe, blocks, _touching(pipe, mbr, n, n))


def test_plan_outgrows_its_buffers(blocks_100):
    """21000 counted boxes that cut nearly every CTF of three blocks: several
    times the plans and items that a lane keeps room for."""
    pipe, blocks, mbr = blocks_100
    few = _touching(pipe, mbr, 5, 7)
    W, H = mbr[2] - mbr[0], mbr[3] - mbr[1]
    for i in range(4):  # windows of most of the map, in time so that CTFs are not taken whole
        few[i]["box"] = (mbr[0] + 0.01 * i * W, mbr[1], mbr[2], mbr[3] - 0.02 * i * H)
        few[i]["t_start"] = max(int(b.end_time_min) for b, _ in blocks) + 1
    few = np.concatenate([few, few[:1]])
    few[5]["t_start"] = min(int(b.end_time_min) for b, _ in blocks) + 1
    want = pipe.query_counts(few)
    assert int(want[5]) > 1000
    got = pipe.query_counts(np.tile(few, 3500))
    assert np.array_equal(np.asarray(got), np.tile(np.asarray(want), 3500))


@pytest.mark.parametrize("late", [None, 0, 1, 3])
def test_crowded_items_leave_pieces(built_cuda, late):
    """Four CTFs of tens of thousands of keys: items with more keys to decode,
    and more end offsets to compare, than they keep."""
    tc = hotspot_grid(30000, n_hotspots=30, box_m=3000.0, grid_n=16, sigma_m=120.0, seed=31)
    cfg = StcConfig(num_objects=30000, reach_distance=10.0, min_meet_time=3, max_meet_time=6, grid_capacity=50,
                    grid_amplify=1.2, num_meeting_buckets=1_500_000, kv_restriction=70_000, ctf_count=4,
                    ctb_retain=1)
    pipe, blocks, mbr = _ingest(cfg, tc, 15, 1)
    try:
        W, H = mbr[2] - mbr[0], mbr[3] - mbr[1]
        qs = np.zeros(70, QUERY_DTYPE)
        for i in range(len(qs)):
            f = 0.4 * i / len(qs)
            qs[i]["kind"], qs[i]["t_end"] = QUERY_BOX, 0xFFFFFFFF
            qs[i]["box"] = (mbr[0] + f * W, mbr[1] + 0.5 * f * H, mbr[2] - 0.3 * f * W, mbr[3] - f * H)
            qs[i]["t_start"] = 0 if late is None else int(blocks[0][0].end_time_min) + late
        assert _compare(pipe, blocks, qs) >= {None: 100_000, 0: 1000}.get(late, 0)
    finally:
        pipe.close()

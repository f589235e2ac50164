"""The border lookup's thread layouts (csrc/stc_partition.cu, k_border_count)
against the oracle: object counts either side of the rule (1024 a
multiprocessor), and tiles of 256 points with one point or one short of full."""
import numpy as np
import pytest

from stcdb_gb300.pipeline import StcConfig
from stcdb_gb300.tracegen import hotspot_grid

from parity import describe_diff, run_pair, trace_and_box

pytestmark = pytest.mark.gpu


def _counts():
    import torch
    if not torch.cuda.is_available():
        return []
    edge = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    return [255, 256, 257, edge, edge + 1]


@pytest.mark.parametrize("which", range(5))
def test_border_units_match_the_oracle(built_cuda, which):
    n = _counts()[which]
    hot = max(n // 1000, 2)
    box = 400.0 if n < 1000 else 6000.0
    tr, mbr = trace_and_box(hotspot_grid(n, n_hotspots=hot, box_m=box, grid_n=8 if n < 1000 else 24, sigma_m=60.0,
                                         seed=n % 97), 4)
    cfg = StcConfig(num_objects=n, reach_distance=8.0, min_meet_time=2, grid_capacity=20, grid_amplify=4.0,
                    num_meeting_buckets=1 << 25, refine_size=8)
    hits = 0
    for t, g, o, gs, os_ in run_pair(cfg, np.asarray(tr), mbr):
        assert np.array_equal(g, o), f"step {t}: {describe_diff(g, o)}"
        assert gs.hits == os_.hits and gs.border_units == os_.border_units
        hits += gs.hits
    assert hits > 0

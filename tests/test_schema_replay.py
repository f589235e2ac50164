"""The closed form of a step's split and merge events on the quadtree's free
stacks (k_schema_phase2_par of csrc/stc_schema.cu) against replaying the
stacks one event after the other."""
import random

import pytest


def replay(events, schema, grids, si, gi):
    """tracing/filter.cpp:316-375 on the two stacks; what each event got, and the stacks behind."""
    schema, grids, got = list(schema), list(grids), []
    for kind, nodes, gids in events:
        if kind == "split":
            gi -= 1
            grids[gi] = gids[0]
            got.append((schema[si:si + 4], grids[gi:gi + 4]))
            si, gi = si + 4, gi + 4
        else:
            for n, g in zip(nodes, gids):
                si, gi = si - 1, gi - 1
                schema[si], grids[gi] = n, g
            got.append(grids[gi])
            gi += 1
    return got, schema[si:], grids[gi:]


def closed_form(events, schema, grids, si, gi):
    level, levels = 0, []
    for kind, _, _ in events:
        levels.append(level)
        level += 1 if kind == "split" else -1
    out_s, out_g, got = list(schema), list(grids), []
    for e, (kind, nodes, gids) in enumerate(events):
        k = levels[e]
        if kind == "split":
            m = next((j for j in range(e - 1, -1, -1) if events[j][0] == "merge" and levels[j] == k + 1), None)
            if m is None:
                got.append((schema[si + 4 * k:si + 4 * k + 4], [gids[0]] + grids[gi + 3 * k:gi + 3 * k + 3]))
            else:
                got.append((events[m][1][::-1], [gids[0]] + events[m][2][2::-1]))
        else:
            got.append(gids[3])
            if k - 1 >= level and not any(events[j][0] == "merge" and levels[j] == k for j in range(e + 1, len(events))):
                for i in range(4):
                    out_s[si + 4 * (k - 1) + 3 - i] = nodes[i]
                for i in range(3):
                    out_g[gi + 3 * (k - 1) + 2 - i] = gids[i]
    return got, out_s[si + 4 * level:], out_g[gi + 3 * level:]


@pytest.mark.parametrize("count,share", [(1, 0.5), (2, 0.5), (7, 0.3), (60, 0.5), (60, 0.9), (60, 0.1), (400, 0.5)])
def test_closed_form_equals_the_replay(count, share):
    rng = random.Random(count * 10 + int(share * 10))
    for _ in range(20):
        size = 8 * count + 16
        si = gi = 4 * count + 8
        schema, grids = list(range(size)), list(range(10_000, 10_000 + size))
        events, fresh = [], 1_000_000
        for _ in range(count):
            nodes, gids = list(range(fresh, fresh + 4)), list(range(fresh + 4, fresh + 8))
            fresh += 8
            events.append(("split" if rng.random() < share else "merge", nodes, gids))
        assert closed_form(events, schema, grids, si, gi) == replay(events, schema, grids, si, gi)

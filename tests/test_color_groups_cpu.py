"""The groups of inherited face colours that the colour pass reduces together (tmc_gb300/csrc/color_groups.h).

A face comes from a grid edge and its colour is 3 * parity of the edge's lower point + axis; faces share an edge
across a grid face, whose grid edges theirs are.  So: two colours that meet on any grid face are in different
groups, the one that is reduced earlier (5..23 in order, then 4) in the earlier group, and 4 is alone in the last
(it is reduced to one of four colours, the others to one of five)."""
import itertools
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _groups():
    text = open(os.path.join(ROOT, "tmc_gb300", "csrc", "color_groups.h")).read()
    lo, hi = (int(re.search(rf"{n} (0x[0-9a-f]+)ull", text).group(1), 16) for n in ("GROUPS_LO", "GROUPS_HI"))
    return {c: (lo >> 4 * (c - 4) if c < 20 else hi >> 4 * (c - 20)) & 15 for c in range(4, 24)}


def _meetings():
    unit = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
    colour = lambda p, axis: 3 * sum((c & 1) << d for d, c in enumerate(p)) + axis  # noqa: E731
    for p in itertools.product((0, 1), repeat=3):
        for a, b in itertools.combinations(range(3), 2):  # the grid face at p along axes a and b
            step = [tuple(x + y for x, y in zip(p, unit[d])) for d in (a, b)]
            edges = [colour(p, a), colour(step[1], a), colour(p, b), colour(step[0], b)]
            yield from itertools.permutations(edges, 2)


def test_colours_that_meet_are_reduced_in_order():
    groups = _groups()
    turn = {c: n for n, c in enumerate(list(range(5, 24)) + [4])}
    for c, d in set(_meetings()):
        assert c != d
        if c in turn and d in turn and turn[c] < turn[d]:
            assert groups[c] < groups[d], (c, d)
    assert sorted(set(groups.values())) == list(range(14))
    assert [c for c in groups if groups[c] == 13] == [4]

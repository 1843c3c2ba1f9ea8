"""Closest points by groups of lanes (nricp_b200/csrc/lbvh.cu,
`nearest_triangle_group`): a query is walked by 4, 8 or 16 lanes, by the number
of queries, and a walk whose pending subtrees pass the group's stack is left to
one lane.  Each answer is the FP64 brute-force winner whatever the group.

A B200 holds about 76,000 threads of the kernel at once, so the counts below
fall on both sides of the lines (2 x resident / 16 and 4 x resident / 8) and on
ragged last warps.
"""

from __future__ import annotations

import numpy as np
import pytest

from nricp_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 33, 9_001, 12_000, 36_001, 50_003])
def test_every_group_width_finds_the_fp64_winner(dp, device, oracle, count):
    rng = np.random.default_rng(count)
    points, faces, _ = S.latlong_ellipsoid(24, 60, (1.0, 0.8, 1.2))  # fans of slivers at the poles
    points = points + rng.normal(0.0, 1e-3, size=points.shape)       # no exact ties
    queries = rng.normal(size=(count, 3)) * rng.choice([0.02, 1.0, 4.0], size=(count, 1))
    got = dp.closest_points(points, faces, queries)
    exact = oracle.closest_points(points, faces, queries)
    # the same FP64 routine on both sides: a last-bit tie may pick a neighbour
    # that shares the point, so distances are compared, to the rounding of
    # coordinates below ten
    assert np.abs(got["distances"] - exact["distances"]).max() < 1e-13
    assert np.abs(got["points"] - exact["points"]).max() < 1e-12


def test_a_group_whose_stack_overflows_still_finds_the_winner(dp, device, oracle):
    """A query at the centre of a sphere is nearly as far from every triangle:
    the walk prunes nothing, and its pending subtrees pass any group's stack."""
    points, faces = S.icosphere(5)
    rng = np.random.default_rng(3)
    points = points * (1.0 + rng.uniform(0.0, 1e-7, size=(len(points), 1)))
    queries = rng.normal(0.0, 1e-9, size=(40, 3))
    got = dp.closest_points(points, faces, queries)
    exact = oracle.closest_points(points, faces, queries)
    assert np.abs(got["distances"] - exact["distances"]).max() < 1e-13

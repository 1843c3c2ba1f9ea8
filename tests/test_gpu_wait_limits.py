"""Waits inside a kernel that run out are reported, end their wrap at once and
leave the device and the library usable.  A limit of 0 tries makes every wait
run out without anything failing: the copies and the other CTAs' data still
arrive.
"""

from __future__ import annotations

import ctypes as C
import time

import numpy as np
import pytest

from nricp_b200 import _abi
from nricp_b200 import synthetic as S
from nricp_b200._lib import check, load

pytestmark = pytest.mark.gpu


def _large(nodes):
    case = S.config2(seed=nodes, vertex_count=nodes + 500, triangle_count=6_000, nodes_finest=nodes, k=4, levels=1)
    case.level_settings = [dict(case.level_settings[0], smoothness=1.0, max_outer_iterations=1,
                                max_inner_iterations=1)]
    return case


def _solve_gives_up_and_recovers(dp, case, cluster):
    batch = dp.WrapBatch([(*case.args(), case.options)])
    if cluster is not None:
        batch.tune(cluster)
    batch.run()
    expected = batch.result(0)
    batch.wait_limit(0)
    began = time.perf_counter()
    with pytest.raises(RuntimeError, match="a wait inside the linear solve ran out"):
        batch.step()
    # the first solve's failure ends the wrap: no further damping attempts
    assert batch.counters()[0] <= 16
    assert time.perf_counter() - began < 5.0
    batch.wait_limit(1 << 19)
    batch.step()
    got = batch.result(0)
    assert np.array_equal(expected["vertices"], got["vertices"])
    assert np.array_equal(expected["rotations"], got["rotations"])


# several CTAs, one CTA, the whole device (a lone graph above 2,000 nodes)
@pytest.mark.parametrize("nodes, cluster", [(300, 8), (300, 1), (2_600, 16), (2_600, None)])
def test_a_solve_that_waits_in_vain_is_reported(dp, device, nodes, cluster):
    _solve_gives_up_and_recovers(dp, _large(nodes), cluster)


# u in global memory (above 7,680 nodes): the loop meets at cluster barriers, and
# a CTA that leaves it early stays until every CTA has left
@pytest.mark.parametrize("cluster", [16, 4, 1])
def test_a_solve_that_meets_at_barriers_gives_up_together(dp, device, cluster):
    _solve_gives_up_and_recovers(dp, _large(8_200), cluster)


def test_a_limit_out_of_range_is_refused(dp, device):
    case = S.small_case(seed=3)
    batch = dp.WrapBatch([(*case.args(), case.options)])
    for tries in (-1, (1 << 19) + 1):
        with pytest.raises(ValueError):
            batch.wait_limit(tries)


def _seeds_within(points, nodes, tries):
    """The seeds of one level of `nodes` nodes, built with this wait limit."""
    n = len(points)
    P = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    level = {"indices": np.full(nodes, -1, dtype=np.int32), "positions": np.empty((nodes, 3)),
             "nodes": np.empty((n, _abi.MAX_SLOTS), dtype=np.int32), "weights": np.empty((n, _abi.MAX_SLOTS)),
             "counts": np.empty(n, dtype=np.int32), "edges": np.empty((nodes * 4, 2), dtype=np.int32)}
    out = _abi.GraphLevel(P(level["indices"], C.c_int32), P(level["positions"], C.c_double),
                          P(level["nodes"], C.c_int32), P(level["weights"], C.c_double),
                          P(level["counts"], C.c_int32), P(level["edges"], C.c_int32), nodes * 4, 0)
    center, scale = np.zeros(3), C.c_double()
    check(load().nricp_template_graph_within(P(points, C.c_double), n, 1, nodes, 2, 4, 4, P(center, C.c_double),
                                             C.byref(scale), C.byref(out), tries))
    return level["indices"]


# 2 seeds: the only wait is the last step's
@pytest.mark.parametrize("points, nodes", [(3_000, 2), (3_000, 3), (30_000, 40), (100_000, 2)])
def test_seeds_that_wait_in_vain_are_reported(dp, device, points, nodes):
    p = np.random.default_rng(points).normal(size=(points, 3))
    with pytest.raises(RuntimeError, match="a wait inside the farthest-point seeds ran out"):
        _seeds_within(p, nodes, 0)
    after = _seeds_within(p, nodes, 1 << 19)
    assert np.array_equal(after, dp.farthest_point_seeds(p, nodes))

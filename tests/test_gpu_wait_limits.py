"""Waits inside a kernel that run out are reported, end their wrap at once and
leave the device and the library usable.  A limit of 0 tries makes every wait
run out without anything failing: the copies and the other CTAs' data still
arrive.
"""

from __future__ import annotations

import time

import numpy as np
import pytest

from nricp_b200 import synthetic as S

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

"""A uniform cluster size of the linear solve is taken for graphs of every size:
the whole device's solve, which a new batch may give a graph of more than 2,000
nodes, is then not among a tick's launches, and the cluster solve gives its
bits at every size -- vectors in shared memory and in global memory, u in
every CTA's shared memory (up to 7,680 nodes) and in global memory.
"""

from __future__ import annotations

import numpy as np
import pytest

from nricp_b200 import synthetic as S

pytestmark = pytest.mark.gpu

# stats twice, the solve, prologue, evaluate, normals, query, and in each of
# the two branches residual, assembly and decision
TICK_LAUNCHES = 13


def _case(nodes):
    case = S.config2(seed=nodes, vertex_count=nodes + 500, triangle_count=6_000, nodes_finest=nodes, k=4, levels=1)
    case.level_settings = [dict(case.level_settings[0], smoothness=1.0, max_outer_iterations=1,
                                max_inner_iterations=1)]
    return case


@pytest.mark.parametrize("nodes, clusters", [(2_600, (1, 2, 4, 8, 16)), (7_690, (2, 16)), (8_200, (1, 4))])
def test_a_uniform_size_is_taken_for_large_graphs(dp, device, nodes, clusters):
    case = _case(nodes)
    own = dp.WrapBatch([(*case.args(), case.options)])  # alone: the whole device's
    own.run()
    reference = own.result(0)
    ticks, launches = own.counters()
    assert launches > TICK_LAUNCHES * ticks
    batch = dp.WrapBatch([(*case.args(), case.options)])
    for cluster in clusters:
        assert batch.tune(cluster) == cluster
        batch.step()
        ticks, launches = batch.counters()
        builds = launches - TICK_LAUNCHES * ticks  # the hierarchy's, once a step
        assert 0 < builds < 13, (ticks, launches)
        got = batch.result(0)
        assert np.array_equal(reference["vertices"], got["vertices"]), cluster
        assert np.array_equal(reference["rotations"], got["rotations"]), cluster

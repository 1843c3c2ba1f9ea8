"""The linear solve at the edges of its partition (nricp_b200/csrc/
wrap_kernels.cu, `pcg_solve`): octets of eight nodes that are full, one short
and one over, CTAs without rows, blocks that fit in shared memory and blocks
that are streamed, and graphs whose vectors do not fit, solved by a cluster
and by the whole device.  Every one of these gives the same bits, and the increment satisfies the damped system that the
device assembled to the bar of test_gpu_solve_stats.
"""

from __future__ import annotations

import numpy as np
import pytest

from nricp_b200 import synthetic as S

from test_gpu_solve_stats import RESIDUAL_FACTOR, _damped_matvec

pytestmark = pytest.mark.gpu


def _case(nodes):
    case = S.config2(seed=nodes, vertex_count=max(600, nodes + 500), triangle_count=6_000, nodes_finest=nodes, k=4,
                     levels=1)
    case.level_settings = [dict(case.level_settings[0], smoothness=1.0, max_outer_iterations=2,
                                max_inner_iterations=2)]
    return case


@pytest.mark.parametrize("nodes", [1, 7, 8, 9, 127, 129, 1_001, 2_600, 5_003, 8_200])
def test_solves_at_every_partition_edge(dp, device, nodes):
    case = _case(nodes)
    reference = None
    for cluster in (16, 4, 1) if nodes < 5_000 else (16, 8):
        batch = dp.WrapBatch([(*case.args(), case.options)])
        batch.tune(cluster)
        batch.run()
        got = batch.result(0)
        if reference is None:
            reference = got
        assert np.array_equal(reference["vertices"], got["vertices"]), cluster
        assert np.array_equal(reference["rotations"], got["rotations"]), cluster
    if nodes > 2_000:  # alone a large graph is the whole device's, among equals a cluster's
        many = dp.WrapBatch([(*case.args(), case.options)] * (nodes // 2_000 + 1))
        many.run()
        assert np.array_equal(reference["vertices"], many.result(0)["vertices"])
        assert np.array_equal(reference["rotations"], many.result(0)["rotations"])
    session = dp.RouteBSession(*case.args(), **case.options)
    checked = 0
    while not session.finished() and checked < 2:
        before = session.inspect()
        session.step()
        after = session.inspect()
        if before["phase"] != 2 or not after["pcg_ok"]:
            continue
        rhs = before["rhs"].astype(np.float64)
        x = after["delta"][: before["node_count"]]
        residual = rhs - _damped_matvec(before["diag"], before["off_nodes"], before["off_blocks"], before["damping"], x)
        assert np.linalg.norm(residual) <= RESIDUAL_FACTOR * case.options["pcg_tolerance"] * np.linalg.norm(rhs)
        checked += 1
    assert checked

"""Route C's right-hand side with its vertex pass (`k_c_deform`, a thread per
vertex, blocks of 256): a block that is one vertex short, several with a
remainder, one node and many (the generator rounds the vertex counts to 255,
597 and 1,037).  Whole wraps against the FP64 restatement, to the bars of
test_gpu_parity.
"""

from __future__ import annotations

import pytest

from nricp_b200 import synthetic as S

from test_gpu_parity import ENERGY_TOL, VERTEX_TOL, _compare_wraps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vertices,nodes", [(255, 1), (256, 9), (257, 40), (600, 33), (1_025, 200)])
def test_route_c_at_the_edges_of_a_block(dp, device, oracle, vertices, nodes):
    from oracle.oracle import ROUTE_C

    case = S.config2(seed=vertices, vertex_count=vertices, triangle_count=4_000, nodes_finest=nodes,
                     k=min(4, nodes), levels=1)
    case.level_settings = [dict(case.level_settings[0], max_outer_iterations=3, max_inner_iterations=3)]
    gpu = dp.solve_route_c(*case.args(), **case.options)
    ref = oracle.solve(*case.args(), route=ROUTE_C, **case.options)
    vertex_error, energy_error = _compare_wraps(gpu, ref, case.target_points)
    assert vertex_error <= VERTEX_TOL, vertex_error
    assert energy_error <= ENERGY_TOL, energy_error

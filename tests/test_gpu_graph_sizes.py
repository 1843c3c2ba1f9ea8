"""The device template graph at the edges of its launches (nricp_b200/csrc/
graph_build.cu): farthest-point seeds with 1, 2, 4 and 8 points per thread, full
and ragged chunks, clusters of 1 to 16 CTAs, and one block past 131,072 points;
bindings of 1 to 8 nodes and node edges over more than one staged tile of
nodes.  Everything equals the host build bit for bit.
"""

from __future__ import annotations

import numpy as np
import pytest

from nricp_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count, nodes, support, neighbours", [
    (1, 1, 1, 4), (2, 2, 8, 4), (9, 9, 3, 16), (1_024, 33, 2, 3), (1_025, 513, 5, 5), (2_049, 1_100, 7, 8),
    (16_385, 70, 8, 4), (32_769, 40, 6, 1), (65_537, 50, 4, 4), (131_073, 12, 4, 4),
])
def test_device_graph_is_the_host_graph(dp, device, count, nodes, support, neighbours):
    rng = np.random.default_rng(count)
    points = rng.normal(size=(count, 3))
    if count > 4:
        points[count // 2] = points[count // 3]  # an exact tie
    faces = np.array([[0, min(1, count - 1), min(2, count - 1)]])
    options = dict(levels=1, nodes_initial=nodes, growth=2, max_nodes_per_vertex=support, edge_neighbours=neighbours)
    gpu = dp.build_template_graph(points, faces, use_device=True, **options)["levels"][0]
    host = dp.build_template_graph(points, faces, use_device=False, **options)["levels"][0]
    assert np.array_equal(gpu["node_template_indices"], host["node_template_indices"])
    assert np.array_equal(gpu["node_positions"], host["node_positions"])
    assert np.array_equal(gpu["edges"], host["edges"])
    for key in ("nodes", "weights", "counts"):
        assert np.array_equal(gpu["bindings"][key], host["bindings"][key]), key


def test_more_templates_than_the_device_holds_at_once_give_the_same_graphs(dp, device):
    """40 templates of 4,500 vertices want 160 CTAs at two points per thread;
    they are built at four, and alone at two."""
    case = S.config2(seed=3, vertex_count=4_500, triangle_count=3_000, nodes_finest=60, k=4, levels=1)
    args = (*case.args(), case.options)
    batch = dp.WrapBatch([args] * 40)
    batch.run()
    alone = dp.solve_route_b(*case.args(), **case.options)
    for i in (0, 39):
        got = batch.result(i)
        assert np.array_equal(got["node_positions"], alone["node_positions"])
        assert np.array_equal(got["vertices"], alone["vertices"])

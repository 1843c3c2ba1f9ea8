"""The correspondence statistics and the deformed template's normals on
templates large enough for every part of their kernels (nricp_b200/csrc/
wrap_kernels.cu): more distances than the select keeps in shared memory and
than it has bins, and a pole whose fan is its warp's.
"""

from __future__ import annotations

import json

import numpy as np
import pytest

from nricp_b200 import synthetic as S

from test_gpu_assembly import _deformed, _graph

pytestmark = pytest.mark.gpu


def _finished(dp, case, **options):
    levels = [dict(case.level_settings[0], max_outer_iterations=1, max_inner_iterations=1)]
    session = dp.RouteBSession(case.template_points, case.template_faces, case.target_points, case.target_faces,
                               levels, **dict(case.options, **options))
    session.run()
    return session


@pytest.mark.parametrize("vertices", [40, 1_500, 2_600, 30_000])
@pytest.mark.parametrize("masked", [0.0, 0.9])
def test_percentile_maximum_and_mean_are_those_of_the_distances(dp, device, vertices, masked):
    case = S.config2(seed=vertices, vertex_count=vertices, triangle_count=4_000, nodes_finest=20, k=4, levels=1)
    n = len(case.template_points)
    mask = np.ones(n, np.uint8)
    mask[: int(masked * n)] = 0
    session = _finished(dp, case, mask=mask)
    seen, stats = session.inspect(), json.loads(session.report())["correspondence"]
    kept = np.sort(seen["corr_distances"][seen["corr_codes"] == 0])
    assert stats["accepted"] == len(kept) > 0
    assert stats["distance_p95"] == kept[int(0.95 * (len(kept) - 1))]
    assert stats["distance_max"] == kept[-1]
    assert abs(stats["distance_mean"] - kept.mean()) <= 1e-12 * kept.mean()  # summed in another order


def test_normals_at_a_wide_fan_decide_the_normal_filter(dp, device):
    """The poles of a lat-long template have 300 faces each."""
    template, faces, _ = S.latlong_ellipsoid(40, 300, (1.0, 0.8, 1.2))
    target, target_faces, _ = S.latlong_ellipsoid(30, 64, (1.1, 0.9, 1.1))
    rng = np.random.default_rng(2)
    template = template + rng.normal(0.0, 5e-3, size=template.shape)
    least = 0.8
    options = dict(graph_levels=1, nodes_initial=30, growth=2, min_normal_cosine=least)
    case = S.WrapCase(template, faces, target, target_faces, S.reference_settings(1), options)
    graph = _graph(dp, case, options)
    center, scale = graph["normalization"]["center"][0], graph["normalization"]["scale"]
    session = dp.RouteBSession(template, faces, target, target_faces, case.level_settings, **options)
    session.step()
    seen = session.inspect()
    deformed = _deformed((template - center) * scale, graph["levels"][0], seen)
    cosine = (S.vertex_normals(deformed, faces) * seen["corr_normals"]).sum(1)
    clear = np.abs(cosine - least) > 1e-9  # FP64 normals summed in another order
    assert clear[[0, len(template) - 1]].all()
    assert np.array_equal((seen["corr_codes"] == 2)[clear], (cosine < least)[clear])
    assert 0 < (seen["corr_codes"] == 2).sum() < len(template)

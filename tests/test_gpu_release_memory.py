"""What calls leave in the library's device pool is given back on request, and
the calls and batches around the request are not disturbed by it."""

from __future__ import annotations

import numpy as np
import pytest

from nricp_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def test_kept_memory_is_given_back(dp, device):
    torch = pytest.importorskip("torch")
    case = S.small_case(seed=6)
    batch = dp.WrapBatch([(*case.args(), case.options)])
    batch.run()
    expected = batch.result(0)["vertices"]
    points, faces = S.uv_sphere(400, 800)
    rng = np.random.default_rng(3)
    points = points + rng.normal(0.0, 1e-4, size=points.shape)
    queries = rng.normal(size=(1_000, 3))
    first = dp.closest_points(points, faces, queries)
    dp.release_memory()
    before = torch.cuda.mem_get_info()[0]
    again = dp.closest_points(points, faces, queries)
    # the hierarchy alone: 64 bytes a node and 80 a leaf
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept >= 144 * (len(faces) - 1)
    dp.release_memory()
    assert before - torch.cuda.mem_get_info()[0] <= kept // 8
    for key in first:
        assert np.array_equal(first[key], again[key]), key
    batch.step()  # the batch kept its memory
    assert np.array_equal(batch.result(0)["vertices"], expected)

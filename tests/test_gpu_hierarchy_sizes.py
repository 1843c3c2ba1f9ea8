"""The hierarchy's sort and bounds at the edges of their tiles (nricp_b200/
csrc/lbvh.cu): one key, a tile of 2,048 keys one short and one over, 128 tiles
(whose counts each block sums itself) and one more (a scan kernel's), many
equal codes.  Codes, permutation, children and bounds equal the oracle's
line-by-line build bit for bit.
"""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import _lbvh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 31, 257, 2_047, 2_048, 2_049, 262_144, 262_145])
@pytest.mark.parametrize("cells", [0, 3])
def test_sorted_codes_children_and_bounds_match_the_oracle(dp, device, oracle, count, cells):
    rng = np.random.default_rng(count)
    points = rng.normal(size=(max(3, count // 2), 3))
    if cells:  # a few positions only: long runs of equal codes, ordered by index
        points = np.round(points * cells) / cells
    faces = rng.integers(0, len(points), size=(count, 3)).astype(np.int32)
    gpu = _lbvh(dp, points, faces)
    cpu = oracle.lbvh_build(points.astype(np.float32), faces)
    for key in ("codes", "order", "left", "right"):
        assert np.array_equal(gpu[key], cpu[key]), key
    assert np.array_equal(gpu["bounds"], cpu["bounds"])

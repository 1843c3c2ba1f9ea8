"""A new batch's own choice of solve classes (about 64 nodes per CTA, about 128,
halved, with a finer tail): from one wrap to more than fit the device at once,
the results are the ones of a uniform cluster, bit for bit.
"""

from __future__ import annotations

import numpy as np
import pytest

from nricp_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 7, 10, 24])
def test_a_new_batch_gives_a_uniform_clusters_bits(dp, device, count):
    cases = [S.small_case(seed=4, nodes_initial=40),
             S.small_case(seed=7, rings=40, segments=60, nodes_initial=300)]
    tuples = [(*c.args(), c.options) for c in (cases * count)[:count]]
    own = dp.WrapBatch(tuples)
    own.run()
    uniform = dp.WrapBatch(tuples)
    uniform.tune(4)
    uniform.run()
    for i in range(count):
        a, b = own.result(i), uniform.result(i)
        assert np.array_equal(a["vertices"], b["vertices"]), i
        assert np.array_equal(a["rotations"], b["rotations"]), i

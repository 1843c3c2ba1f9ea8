"""A launch that the device refuses is an error of that call and of no other: the
query's shared memory holds the lists of up to 2,047 wraps, and the calls after a
larger batch's failure do their work.
"""

from __future__ import annotations

import numpy as np
import pytest

from nricp_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def test_a_batch_too_large_for_the_querys_lists_is_an_error(dp, device):
    case = S.small_case(seed=2, rings=4, segments=6, levels=1, nodes_initial=4)
    wrap = (*case.args(), case.options)
    batch = dp.WrapBatch([wrap] * 2_048)
    with pytest.raises(RuntimeError, match="tick launch"):
        batch.run()
    del batch
    most = dp.WrapBatch([wrap] * 2_047)
    most.run()
    alone = dp.WrapBatch([wrap])
    alone.run()
    assert np.array_equal(most.result(2_046)["vertices"], alone.result(0)["vertices"])

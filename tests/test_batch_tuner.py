"""nspt_batch_tune_shape: what it reports is what it timed -- 1 to 4 warps per CTA,
once each -- and the shape kept is the fastest of them.  Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [6, 13])
def test_each_shape_is_timed_once(engine_mod, N):
    P = engine_mod
    with P.NsptBatch([(4, 4, 4, 4), (6, 4, 4, 4)], N, [0.01, 0.005], [1, 2]) as b:
        w, mo, table = b.tune_shape(0)
        assert mo == 8 and 1 <= w <= 4
        assert np.all(table[0, :4] > 0) and table[0, w - 1] == table[0, :4].min()
        assert np.all(table[0, 4:] == table[0, 3])
        if N <= 12:
            assert np.array_equal(table[1, :6], table[0, :6]) and np.all(table[1, 6:] == 0)
        else:
            assert np.all(table[1] == 0)

"""Host result arrays are not cleared before the call that fills them; a value
the call will not write (an imaginary part longer than the real one) still is
zero."""
import numpy as np
import pytest


@pytest.mark.parametrize("shape,n", [((6,), 6), ((2, 3), 6), ((6,), 4), ((2, 4), 5), ((3,), 0)])
def test_values_past_the_result_are_zero(pkg, shape, n):
    like = np.full(shape, 7.0)
    a = pkg._out(like, n)
    assert a.shape == shape and a.dtype == like.dtype and a is not like
    assert not a.reshape(-1)[n:].any()

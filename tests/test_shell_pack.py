"""Shell records handed to the C entry points: the origin may be any indexable
sequence of three numbers (an array, a list or a tuple that a program assigned)."""
import numpy as np
import pytest


@pytest.mark.parametrize("origin", [[0.5, -1.0, 2.0], (0.5, -1.0, 2.0), [0.5, -1, 2],
                                    np.array([0.5, -1.0, 2.0], np.float32)])
def test_origin_sequences(lgx, origin):
    s = lgx.Shell(2, [(1.3, 0.4), (0.6, 0.7)])
    s.O = origin
    r = s._c()
    assert [r.origin[x] for x in range(3)] == [0.5, -1.0, 2.0]
    assert (r.l, r.pure, r.nprim) == (2, 1, 2)
    assert [r.alpha[0], r.alpha[1]] == [1.3, 0.6]
    assert [r.coeff[0], r.coeff[1]] == list(s.coeff)

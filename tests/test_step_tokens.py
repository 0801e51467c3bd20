"""The token array of a serving step: every sequence and number that numpy takes gives what numpy makes of it, errors included."""
import numpy as np
import pytest

from pkgload import load_pkg


def _numpy(lists):
    return np.array([t for x in lists for t in x], np.int32)


@pytest.mark.parametrize("lists", [[], [[], []], [[1, 2], [3]], [[1, 2], (3, 4)], [np.arange(3), [4]], [[np.int64(5)], [True, -1]], [[1.5], [2]], [[2**31]],
                                   [["x"]], [[None]]], ids=str)
def test_tokens_as_numpy_makes_them(lists):
    serving = load_pkg("serving")
    try:
        want = _numpy(lists)
    except Exception as e:
        with pytest.raises(type(e)):
            serving._int32(lists)
        return
    a = serving._int32(lists)
    assert a.dtype == np.int32 and a.shape == want.shape and (a == want).all()

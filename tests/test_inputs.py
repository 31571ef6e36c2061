"""Cell types given from Python: what float() takes is taken, anything else is refused there, not
passed on as NaN."""
import decimal

import numpy as np
import pytest

from procell import _lib


@pytest.mark.parametrize("kind", [list, tuple, np.array])
def test_types_are_converted_by_float(kind):
    rows = [(0.25, 30, np.float32(4.5)), (decimal.Decimal("0.75"), "60.5", -1.0)]
    got = _lib.types_numpy(rows if kind is not np.array else np.array([(0.25, 30, 4.5), (0.75, 60.5, -1.0)]))
    assert got.dtype == _lib.TYPE_DTYPE and got.tolist() == [(0.25, 30.0, 4.5), (0.75, 60.5, -1.0)]
    assert _lib.types_numpy(kind([])).shape == (0,)


@pytest.mark.parametrize("bad", [None, 1 + 0j, [1.0], (1.0,)])
def test_what_float_refuses_is_refused(bad):
    for rows in ([(bad, 1.0, 2.0)], [[1.0, bad, 2.0]], ((1.0, 1.0, bad),)):
        with pytest.raises(TypeError):
            _lib.types_numpy(rows)

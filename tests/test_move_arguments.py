"""The particle and type of a single move in every form that numpy assigns to an int32."""
import numpy as np
import pytest

from rampack_gb300.packing import MOVE_DTYPE, GpuPacking


class Library:
    """Takes the place of the engine: keeps the move it is given."""

    def rp_try_move(self, handle, move, domain, energy):
        self.move = move._obj
        return 0


def assigned(value):
    m = np.zeros(1, dtype=MOVE_DTYPE)
    m["particle"] = value
    return int(m["particle"][0])


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("value", [5, np.int64(7), np.uint8(3), np.array(4), np.array([6]), np.array([[2]], dtype=np.int16), [1], (8,),
                                   2.0, 3.7, np.float32(2.5), True, "9", -1, 0x7fffffff, np.array([1.0])], ids=repr)
def test_accepted_forms(value):
    g = GpuPacking.__new__(GpuPacking)
    g.lib, g.h = Library(), None
    g.try_move(value, np.array([1]), rotation=np.eye(3))
    assert (g.lib.move.particle, g.lib.move.type, g.lib.move.domain) == (assigned(value), 1, -1)


@pytest.mark.parametrize("value", [1 << 31, -(1 << 31) - 1, [1, 2], None, "x"], ids=repr)
def test_refused_forms(value):
    g = GpuPacking.__new__(GpuPacking)
    g.lib, g.h = Library(), None
    with pytest.raises((OverflowError, ValueError, TypeError)) as a:
        assigned(value)
    with pytest.raises(a.type):
        g.try_move(value, 0)

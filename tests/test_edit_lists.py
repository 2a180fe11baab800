"""Edit lists as the C records they become: whatever int() takes is a coordinate, a size or an id,
truncated as int() and a 32-bit field truncate it."""
import numpy as np
import pytest
import torch

from sandengine_gb300.simulation import SimModification, mods_to_c


class _Number:
    """Has no index: int() takes its __int__."""

    def __int__(self):
        return 7

    def __index__(self):
        raise TypeError("not an index")


@pytest.mark.parametrize("value, field", [
    (7, 7), (True, 1), (7.9, 7), (-7.9, -7), ("7", 7), (2**31 + 5, -2**31 + 5), (-2**40 + 3, 3),
    (np.int64(7), 7), (np.uint8(200), 200), (np.float32(7.5), 7), (np.array(7), 7), (np.array(7.5), 7),
    (torch.tensor(7), 7), (torch.tensor(7.5), 7), (torch.tensor(-7.5), -7), (torch.tensor([7.5])[0], 7),
    (_Number(), 7),
])
def test_fields_are_truncated_as_int_does(value, field):
    mods = [SimModification((3, 4), 1, 5, 6), SimModification((value, value), value, value, value),
            SimModification((8, value), 0, 2, 1)]
    rec = mods_to_c(mods)
    got = [(r.position[0], r.position[1], r.mod_shape, r.mod_size, r.mod_matID, list(r._pad4)) for r in rec]
    assert got == [(3, 4, 1, 5, 6, [0, 0, 0]), (field, field, field, field, field, [0, 0, 0]),
                   (8, field, 0, 2, 1, [0, 0, 0])]


@pytest.mark.parametrize("value", [None, "x", (1, 2), object()])
def test_what_int_refuses_is_refused(value):
    with pytest.raises((TypeError, ValueError)):
        mods_to_c([SimModification((1, 2), 0, value, 3)])

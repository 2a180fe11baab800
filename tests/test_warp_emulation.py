"""The device code of tiles with two cells a byte, run on the CPU with whole warps (device_emu/warps.py)."""
import ctypes

import numpy as np
import pytest

from sandengine_gb300 import workloads as wl
from tests.device_emu.warps import WarpEmu

_emus = {}


def _emu(se, text):
    if text not in _emus:
        _emus[text] = WarpEmu(se.parse_string(text))
    return _emus[text]


def _words(rng, rows, stride, nmat):
    """An array of 4-bit ids, a third of its rows at rest."""
    ids = rng.integers(0, nmat, size=(rows, 8 * stride)).astype(np.uint32)
    ids[rng.random((rows, 8 * stride)) < 0.3] = 0
    ids[rows // 3: 2 * rows // 3] = 0
    return np.ascontiguousarray((ids.reshape(rows, stride, 8) << (4 * np.arange(8, dtype=np.uint32))).sum(axis=2)
                                .astype(np.uint32))


@pytest.mark.parametrize("name", ["four_materials", "twelve_materials"])
def test_a_failed_chunk_check_skips_its_chunk_only(se, rulesets, name):
    """A lane whose index check fails records it and leaves its chunk alone, and goes on with its
    warp: the other chunks get what they get without it, and the launch ends."""
    E = _emu(se, rulesets[name])
    n = se.parse_string(rulesets[name]).num_materials
    rng = np.random.default_rng(5)
    vp = ctypes.c_void_p
    stride, rows = E.lib.emu_cut_stride(), E.lib.emu_cut_rows()
    cut, cpr = 6, 3
    for f in (4, 5, 6, 7):
        a = _words(rng, rows, stride, n)
        want, got = a.copy(), a.copy()
        E.lib.emu_cut_step(vp(want.ctypes.data), f, 0)
        E.checked()
        E.lib.emu_cut_step(vp(got.ctypes.data), f, 1)
        E.checked(8)
        # chunks start at rows ly0 + 2 j; the last whose window ends inside the cut array
        ly0 = (((f + 1) >> 1) & 1)
        last = max(r for r in range(ly0, rows, 2) if r + 2 <= rows - cut)
        assert np.array_equal(got[:last], want[:last]) and np.array_equal(got[last + 4:], a[last + 4:])
        assert not np.array_equal(want, a)
        w = _words(rng, 21, 2 * cpr + 2, n)
        want, got = w.copy(), w.copy()
        E.lib.emu_world_step(vp(want.ctypes.data), 21, cpr, 0, f)
        E.checked()
        E.lib.emu_world_step(vp(got.ctypes.data), 21, cpr, -2, f)
        E.checked(8)
        assert np.array_equal(got, want) and not np.array_equal(want, w)

"""The device code of tiles with two cells a byte, run on the CPU with whole warps, the lane layout and
the reduced tables that the GPU uses (device_emu/warps.py), against the oracle port: every 4-bit
tile shape, whole worlds, edits, bands, jobs of batches and servers, and rule sets whose hash
comparisons take every form (none, lane 1, 2 or 3 alone, several, lane 0 again), with the table in
shared memory and in global memory.  Exact equality: cells are ids."""
import ctypes

import numpy as np
import pytest

from sandengine_gb300 import workloads as wl
from tests.device_emu.emu import Emu
from tests.device_emu.warps import BYTE_SHAPES, SHAPES, WarpEmu

SMALL = [(56, 30, 1, 128), (48, 48, 8, 128)]
_emus = {}


def _emu(se, text, shapes=None):
    key = (text, tuple(shapes or ()))
    if key not in _emus:
        _emus[key] = WarpEmu(se.parse_string(text), shapes)
    return _emus[key]


def _shake(four, cond, probability=""):
    rule = f"""
  shake:
    if: {cond} and RIGHT.mat == EMPTY
{probability}    do: SWAP SELF RIGHT
"""
    return (four.replace("rules:\n", "rules:\n" + rule.lstrip("\n"), 1)
            .replace("base_rules: [fall, spread]", "base_rules: [fall, spread, shake]"))


def _more(text, count):
    """The rule set with materials of ids up to count - 1."""
    return text.rstrip("\n") + "\n" + "".join(
        f"  m{i}:\n    type: {'powder' if i % 2 else 'liquid'}\n    color: [0.1, 0.2, 0.3]\n    density: 1.{i}\n"
        for i in range(6, count))


def _forms(rulesets):
    """Rule set texts by the form of their hash comparisons: (text, the extra lane as WarpEmu tells it)."""
    four = rulesets["four_materials"]
    prob = "    probability: 0.5\n"
    return {"lane1": (_shake(four, "SELF.mat.density > 0.0", prob), 1), "lane2": (_shake(four, "rand.z < 0.3"), 2),
            "lane3": (_shake(four, "rand.w < 0.3"), 3), "lane0": (_shake(four, "rand.x < 0.2"), 0),
            "several": (_shake(four, "rand.z < 0.25", prob), 0),
            "seven": (_more(_shake(four, "rand.z < 0.3"), 7), 2), "eight": (_more(_shake(four, "rand.z < 0.3"), 8), 2),
            "nine": (_more(_shake(four, "rand.z < 0.3"), 9), 2),
            "fifteen": (_more(_shake(four, "rand.z < 0.25", prob), 15), 0), "sixteen": (_more(four, 16), -1)}


def _world(rng, w, h, nmat):
    g = rng.integers(0, nmat + 1, size=(h, w)).astype(np.uint32)  # nmat: an id that names no material
    g[rng.random((h, w)) < 0.4] = 0
    return g


def _mods(rng, w, h, count):
    """Overlapping circles and squares across the world and its edges, some of an unknown material (NULL)."""
    return [(int(rng.integers(-8, w + 8)), int(rng.integers(-8, h + 8)), int(rng.integers(0, 2)),
             int(rng.integers(1, 14)), int(rng.choice([0, 3, 4, 200]))) for _ in range(count)]


def _edit_params(nmat, w, h, mods, row0=0):
    e = Emu.__new__(Emu)
    e.nmat = nmat
    assert row0 == 0
    return e.edit_params(w, h, mods)[:2]


def _check(E, P, shape, rng, w, h, nmat, nmods, rep=0):
    tw, th, k, _ = shape
    f0 = 3 + rep
    n = max(1, k - rep)
    g = _world(rng, w, h, nmat)
    mods = _mods(rng, w, h, nmods)
    params, live = _edit_params(nmat, w, h, mods)
    got = E.tiles(g, f0, n, shape, edits=params if live else None, nedits=live)
    want = g.copy()
    P.run(want, f0 - 1, n, mods)
    assert np.array_equal(got, want), f"{tw}x{th}_k{k} world {w}x{h}, {n} frames: {np.count_nonzero(got != want)} differ"


@pytest.mark.parametrize("name", ["four_materials", "twelve_materials"])
def test_tile_shapes_with_whole_warps_match_port(se, rulesets, ports, name):
    E, P = _emu(se, rulesets[name]), ports[name]
    n = se.parse_string(rulesets[name]).num_materials
    assert E.nib_lane == (-1 if name == "four_materials" else 1)
    rng = np.random.default_rng(11)
    for i, shape in enumerate(SHAPES):
        tw, th, k, _ = shape
        for j, (w, h) in enumerate(((tw + 1, th + 1), (33, 31), (2 * tw + 8 + 4 * i, max(1, th - 1)))):
            _check(E, P, shape, rng, w, h, n, (0, 1, 40)[j], rep=j)
    for shape in BYTE_SHAPES[:1]:  # large one-frame tiles stay on bytes
        _check(E, P, shape, rng, 131, 70, n, 3)


@pytest.mark.parametrize("form", ["lane1", "lane2", "lane3", "lane0", "several", "seven", "eight", "nine", "fifteen",
                                  "sixteen"])
def test_hash_forms_with_whole_warps_match_port(se, rulesets, form):
    from oracle.build import Port
    text, lane = _forms(rulesets)[form]
    rs = se.parse_string(text)
    E, P = _emu(se, text, SMALL), Port(text)
    assert E.nib_lane == lane
    rng = np.random.default_rng(12)
    for shape in SMALL:
        for rep in range(2):
            _check(E, P, shape, rng, 101 + rep, 67, rs.num_materials, 2, rep)


def test_byte_tiles_with_four_bit_keys_match_port(se, rulesets):
    """All 16 ids and hash comparisons besides the mirror test: multi-frame tiles on bytes."""
    from oracle.build import Port
    text = _more(_shake(rulesets["four_materials"], "rand.z < 0.3"), 16)
    rs = se.parse_string(text)
    E, P = _emu(se, text, BYTE_SHAPES), Port(text)
    assert "#define SE_LUT_BITS 4" in rs.kernel_source and E.nib_lane == -2
    rng = np.random.default_rng(13)
    for shape in BYTE_SHAPES:
        for rep in range(2):
            _check(E, P, shape, rng, 140 + 3 * rep, 70, rs.num_materials, 2, rep)
    grids = [_world(rng, w, h, rs.num_materials) for w, h in ((64, 64), (33, 17))]
    for got, g in zip(E.resident(grids, [4, 9], 7, 256), grids):
        P.run(g, 4 if g.shape[0] == 64 else 9, 7)
        assert np.array_equal(got, g)


def test_long_edit_lists_with_whole_warps_match_port(se, rulesets, ports):
    """256 mods of which a tile meets few or all, in several words of a tile's bits; and one whose box
    is the whole world."""
    name = "four_materials"
    E, P = _emu(se, rulesets[name]), ports[name]
    n = se.parse_string(rulesets[name]).num_materials
    rng = np.random.default_rng(14)
    w, h = 231, 117
    for shape in ((56, 30, 1, 128), (48, 48, 8, 128), (112, 112, 8, 256)):
        for mods in (_mods(rng, w, h, 256), _mods(rng, 30, 30, 4), _mods(rng, 30, 30, 5), _mods(rng, 40, 40, 256), _mods(rng, w, h, 33) + [(5, 5, 1, 1 << 23, 3)] +
                     _mods(rng, w, h, 31)):
            g = _world(rng, w, h, n)
            params, live = _edit_params(n, w, h, mods)
            got = E.tiles(g, 6, shape[2], shape, edits=params, nedits=live)
            want = g.copy()
            P.run(want, 5, shape[2], mods)
            assert np.array_equal(got, want), f"{shape}: {np.count_nonzero(got != want)} differ"


@pytest.mark.parametrize("name", ["four_materials", "twelve_materials"])
def test_bands_jobs_and_whole_worlds_with_whole_warps_match_port(se, rulesets, ports, name):
    E, P = _emu(se, rulesets[name]), ports[name]
    n = se.parse_string(rulesets[name]).num_materials
    rng = np.random.default_rng(15)
    W, H = 130, 150
    g = _world(rng, W, H, n)
    for ya, yb, shape in ((40, 130, (48, 48, 8, 128)), (0, 90, (96, 96, 16, 256)), (62, 150, (120, 120, 4, 128))):
        k = shape[2]
        buf, want = E.tiles(g[ya:yb].copy(), 7, k, shape, band=(H, ya)), g.copy()
        P.run(want, 6, k)
        lo, hi = 0 if ya == 0 else k, yb - ya if yb == H else yb - ya - k
        assert np.array_equal(buf[lo:hi], want[ya + lo:ya + hi]), f"band [{ya}, {yb})"
    sizes = [(64, 64), (33, 17), (130, 70), (7, 9), (1, 200), (203, 5)]
    grids = [_world(rng, w, h, n) for w, h in sizes]
    frames, ks = [3, 10, 1, 7, 2, 5], [8, 1, 5, 3, 8, 2]
    wants = {k: [] for k in ("jobs", "serve", "whole")}
    for g, f, k in zip(grids, frames, ks):
        for key, m in (("jobs", 6), ("serve", k), ("whole", 38)):
            w = g.copy()
            P.run(w, f, m)
            wants[key].append(w)
    shape = (48, 48, 8, 128)
    for got, want in zip(E.tile_jobs(grids, frames, 6, shape), wants["jobs"]):
        assert np.array_equal(got, want)
    for got, want in zip(E.serve(grids, frames, ks, shape), wants["serve"]):
        assert np.array_equal(got, want)
    for threads in (128, 512):
        for got, want in zip(E.resident(grids, frames, 38, threads), wants["whole"]):
            assert np.array_equal(got, want)


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

"""Tiles and whole worlds with two cells per byte (kernels/nibble.cuh) against the oracle port:
every tile shape they are chosen for, at world sizes around the tile, item (32 x 32 cells) and
chunk (16 cells) edges, for rule sets with and without hash comparisons besides the mirror test
(on one lane, on several, on none), with the reduced table in shared memory and in global
memory, and with all 16 ids.  Exact equality: cells are ids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (tile width, tile height, frames) of the shapes; sizes are derived from them
SHAPES = [(56, 30, 1), (120, 120, 4), (112, 112, 8), (48, 48, 8), (240, 176, 8), (240, 240, 8), (96, 96, 16), (32, 32, 16)]
# several lanes compared: probability on lane 1, a condition on lane 2
LANES_RULE = """
  shake:
    if: rand.z < 0.25 and RIGHT.mat == EMPTY
    probability: 0.5
    do: SWAP SELF RIGHT
"""


def _texts(rulesets):
    four = rulesets["four_materials"]
    more = "".join(f"  m{i}:\n    type: {'powder' if i % 2 else 'liquid'}\n    color: [0.1, 0.2, 0.3]\n"
                   f"    density: 1.{i}\n" for i in range(6, 16))
    lanes = four.replace("rules:\n", "rules:\n" + LANES_RULE.lstrip("\n"), 1)
    return {"four": four, "twelve": rulesets["twelve_materials"], "reference": rulesets["reference"],
            "sixteen": four.rstrip("\n") + "\n" + more,
            "lanes": lanes.replace("base_rules: [fall, spread]", "base_rules: [fall, spread, shake]")}


def _world(wl, name, nmat, w, h, seed):
    if name == "twelve":
        return wl.patch_fill(w, h, seed, *wl.twelve_fill_spec(), patch=16)
    rng = np.random.default_rng(seed)
    g = rng.integers(0, nmat + 1, size=(h, w)).astype(np.uint32)  # nmat: an id that names no material
    g[rng.random((h, w)) < 0.4] = 0
    return g


@pytest.mark.parametrize("name", ["four", "twelve", "reference", "sixteen", "lanes"])
def test_tile_shapes_match_port(se, rulesets, name):
    from oracle.build import Port
    from sandengine_gb300 import workloads as wl
    text = _texts(rulesets)[name]
    rs, port = se.parse_string(text), Port(text)
    assert "#define SE_LUT_BITS 4" in rs.cuda_source
    for i, (tw, th, k) in enumerate(SHAPES):
        for w, h in ((1, 1), (33, 31), (tw, th), (tw + 1, th + 1), (2 * tw + 8 + 4 * i, th - 1)):
            g = _world(wl, name, rs.num_materials, w, h, 7 * i + w)
            sim = se.Simulation(rs, (w, h))
            sim.set_tile(tw, th, k)
            sim.grid = g
            sim.params.frame = 3 + i
            mods = wl.circle_edits(w, h, 9, i, 3, [0, 3, 200], rmin=1, rmax=20)
            frames = 2 * k + 1 + i % k
            sim.run_frames(frames, [se.SimModification((m[0], m[1]), m[2], m[3], m[4]) for m in mods])
            port.run(g, 3 + i, frames, mods, nthreads=8)
            got = sim.grid
            assert np.array_equal(got, g), f"{name} {tw}x{th} k={k} world {w}x{h}: {np.count_nonzero(got != g)} differ"


@pytest.mark.parametrize("name", ["four", "twelve", "sixteen", "lanes"])
def test_whole_worlds_match_port(se, rulesets, name):
    from oracle.build import Port
    from sandengine_gb300 import workloads as wl
    from sandengine_gb300.batch import Batch
    text = _texts(rulesets)[name]
    rs, port = se.parse_string(text), Port(text)
    # widths around the chunk (16 cells, the array starts 4 columns left of the world), one-row
    # and one-column worlds, and one that fills most of a CTA's shared memory
    sizes = [(1, 1), (10, 3), (11, 1), (12, 2), (27, 31), (28, 64), (64, 64), (1, 200), (203, 131), (640, 600)]
    b = Batch(rs, sizes)
    b.set_resident_limit(1 << 30)
    assert b.info()["resident_worlds"] == len(sizes)
    grids = [_world(wl, name, rs.num_materials, w, h, 3 * i) for i, (w, h) in enumerate(sizes)]
    for i, g in enumerate(grids):
        b.set_grid(i, g)
        b.set_frame(i, 1 + i)
    frames = [1 + i for i in range(len(sizes))]
    for nf in (1, 38, 70):
        b.step(nf)
        b.synchronize()
        for i, g in enumerate(grids):
            port.run(g, frames[i], nf, nthreads=8)
            frames[i] += nf
            got = b.grid(i)
            assert np.array_equal(got, g), f"{name} world {sizes[i]}: {np.count_nonzero(got != g)} cells differ"


@pytest.mark.parametrize("frames", [4, 8, 16])
def test_serving_iterations_of_many_and_few_cells(se, rulesets, ports, frames):
    """Iterations above 2^22 active cells and, once the large session is done, below."""
    from sandengine_gb300 import workloads as wl
    from sandengine_gb300.serving import Server
    srv = Server(se.parse_string(rulesets["twelve_materials"]), 1 << 30)
    srv.set_frames_per_iteration(frames)
    want, jobs = [], []
    for i, (w, h, n) in enumerate(((2050, 2049, 2 * frames + 3), (301, 203, 5 * frames + 1), (64, 64, 3 * frames))):
        g = wl.patch_fill(w, h, i, *wl.twelve_fill_spec(), patch=16)
        sid = srv.open_session(w, h, g, 2 + i)
        mods = wl.circle_edits(w, h, 9, i, 3, [0, 3], rmin=1, rmax=20)
        jobs.append((sid, n, [se.SimModification((m[0], m[1]), m[2], m[3], m[4]) for m in mods]))
        ports["twelve_materials"].run(g, 2 + i, n, mods, nthreads=8)
        want.append(g)
    srv.start()
    for r in [srv.submit(sid, n, mods) for sid, n, mods in jobs]:
        srv.wait(r)
    srv.stop()
    for (sid, _, _), g in zip(jobs, want):
        assert np.array_equal(srv.grid(sid), g)

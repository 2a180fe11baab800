"""Light, colours, alpha pyramid and composite at sizes around the passes' dispatch lines and tile
edges: the light pass takes tiles of 4 rows up to 2^20 cells and of 16 rows beyond (several
launches past 65535 row blocks), the colour pass reduces pyramid levels 1-4 from 16 x 8 cells a warp
and 64 x 16 a CTA, and a second kernel levels 5 and 6.  Bit-exact against the oracle port."""
import numpy as np
import pytest

from sandengine_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1024, 1024), (1025, 1024), (65, 17), (63, 15), (16, 8), (32, 33), (64, 1), (1, 64),
                                   (31, 127), (129, 66), (3, 262150)])
def test_light_and_composite_match_port(se, rulesets, ports, shape):
    W, H = shape
    P = ports["twelve_materials"]
    sim = se.Simulation(se.parse_string(rulesets["twelve_materials"]), (W, H))
    g = wl.patch_fill(W, H, 6, *wl.twelve_fill_spec(), patch=8)
    sim.grid = g
    sim.params.frame = 3
    sim.set_light(True)
    sim.run_frames(3)
    light = np.zeros((H, W, 4), dtype=np.float32)
    for f in (4, 5, 6):
        old = g.copy()
        P.step(g, f)
        light = P.light(old, g, light)
    assert np.array_equal(sim.grid, g)
    assert np.array_equal(sim.output_light.view(np.uint32), light.view(np.uint32))
    col = P.color(g)
    got = sim.composite()
    assert np.array_equal(got.view(np.uint32), P.composite(col, light).view(np.uint32))
    assert np.array_equal(sim.output_color.view(np.uint32), col.view(np.uint32))


@pytest.mark.parametrize("shape", [(1, 1), (2, 1), (1, 2), (64, 64), (256, 192), (257, 192), (256, 193), (64, 768),
                                   (64, 769), (3072, 16), (3073, 16), (1, 768), (768, 1), (191, 255)])
def test_image_in_one_launch_matches_port(se, rulesets, ports, shape):
    """Worlds of up to 48 blocks of 64 x 16 cells have their image made by one cluster; timed
    passes are launched one by one.  Both with a background, against the oracle port."""
    W, H = shape
    P = ports["twelve_materials"]
    sim = se.Simulation(se.parse_string(rulesets["twelve_materials"]), (W, H))
    g = wl.patch_fill(W, H, 6, *wl.twelve_fill_spec(), patch=8)
    sim.grid = g
    sim.params.frame = 3
    bg = np.random.default_rng(3).random((5, 7, 4), dtype=np.float32)
    sim.set_light(True)
    light = np.random.default_rng(4).random((H, W, 4), dtype=np.float32)
    sim.output_light = light
    want = P.composite(P.color(g), light, bg)
    for timing in (False, True):
        sim.set_timing(timing)
        assert np.array_equal(sim.composite(bg).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("shape", [(97, 70), (1, 100), (100, 1), (32, 32), (33, 31), (2000, 3), (1048576, 1),
                                   (3, 1048575), (1048573, 2)])
def test_colour_noise_matches_port(se, rulesets, ports, shape):
    """Tiles of 32 x 32 cells and their remainders, up to the longest sides, whose sines have
    arguments beyond the range of the integer path."""
    W, H = shape
    sim = se.Simulation(se.parse_string(rulesets["twelve_materials"]), (W, H))
    g = np.full((H, W), 3, dtype=np.uint32)
    sim.grid = g
    assert np.array_equal(sim.output_color.view(np.uint32), ports["twelve_materials"].color(g).view(np.uint32))

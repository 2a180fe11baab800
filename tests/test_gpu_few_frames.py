"""Calls of few frames, and callers that ask for few or many a launch, on rule sets with 4-bit tiles: the
shape for the world's cells, and the oracle port's cells."""
import numpy as np
import pytest

from sandengine_gb300 import workloads as wl
from tests.test_gpu_one_frame_shapes import _kernels, _profiler  # noqa: F401

pytestmark = pytest.mark.gpu


def _world(se, rulesets, ports, size):
    W, H = size
    sim = se.Simulation(se.parse_string(rulesets["twelve_materials"]), size)
    g = wl.patch_fill(W, H, 3, *wl.twelve_fill_spec(), patch=16)
    sim.grid = g
    sim.params.frame = 3
    mods = wl.circle_edits(W, H, 9, 1, 6, [0, 3], rmin=1, rmax=20)
    c = [se.SimModification((m[0], m[1]), m[2], m[3], m[4]) for m in mods]

    def run(frames, edits=False):
        f = sim.params.frame
        ports["twelve_materials"].run(g, f, frames, mods if edits else (), nthreads=8)
        names = _kernels(lambda: sim.run_frames(frames, c if edits else ()))
        assert np.array_equal(sim.grid, g), (size, frames)
        return sorted(n for n in names if n.startswith("se_tile"))
    return sim, run


@pytest.mark.parametrize("size, big", [((4096, 2048), True), ((4095, 2048), False)])
def test_last_frames_of_a_call(se, rulesets, ports, size, big):
    sim, run = _world(se, rulesets, ports, size)
    sim.autotune()
    full = "se_tile_%dx%d_k%d" % sim.tile()
    few = "se_tile_120x120_k4" if big else full
    for frames in (2, 4, 3):
        assert run(frames) == [few]
    assert run(sim.tile()[2] + 3) == sorted({full, few})
    assert run(3, edits=True) == [few.replace("tile", "tile_edit")]
    assert run(5) == [full]
    sim.set_tile(48, 48, 8)  # the caller's choice holds for every launch
    assert run(3) == ["se_tile_48x48_k8"]
    sim.autotune()
    assert "se_tile_48x48_k8" not in run(3) or not big


@pytest.mark.parametrize("size, shapes", [
    ((64, 64), {2: "48x48_k8", 3: "48x48_k8", 4: "48x48_k8", 8: "48x48_k8", 16: "96x96_k16"}),
    ((1001, 777), {2: "112x112_k8", 4: "112x112_k8", 8: "112x112_k8", 16: "96x96_k16"}),
    ((2100, 1800), {2: "112x112_k8", 16: "96x96_k16"}),
    ((2049, 2048), {3: "112x112_k8", 16: "96x96_k16"}),
    ((4096, 2048), {2: "120x120_k4", 4: "120x120_k4", 8: "112x112_k8", 16: "96x96_k16"}),
    ((4096, 4096), {16: "128x128_k16"})])
def test_frames_asked_for(se, rulesets, ports, size, shapes):
    sim, run = _world(se, rulesets, ports, size)
    for k, shape in shapes.items():
        sim.set_steps_per_launch(k)
        assert run(2 * k) == ["se_tile_" + shape]

"""The device buffer of the colour field: once a caller has its pointer, composites renew it."""
import numpy as np
import pytest

from sandengine_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


class _Buffer:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("shape", [(64, 64), (517, 389)])
def test_composite_renews_the_colour_buffer(se, rulesets, ports, shape):
    import torch
    W, H = shape
    P = ports["twelve_materials"]
    sim = se.Simulation(se.parse_string(rulesets["twelve_materials"]), (W, H))
    g = wl.patch_fill(W, H, 6, *wl.twelve_fill_spec(), patch=8)
    sim.grid = g
    sim.params.frame = 3
    color = torch.as_tensor(_Buffer(sim.render_color_device(), (H, W, 4)), device="cuda")
    for _ in range(2):
        sim.run_frames(20)
        P.run(g, sim.params.frame - 20, 20)
        want = P.color(g)
        image = sim.composite()
        assert np.array_equal(color.cpu().numpy().view(np.uint32), want.view(np.uint32))
        assert np.array_equal(image.view(np.uint32), P.composite(want).view(np.uint32))

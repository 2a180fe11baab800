"""Batches and servers that launch one frame at a time take the shape for the cells at hand: 4-bit
56 x 30 tiles up to 2^22 cells, 128 x 64 byte tiles beyond, which run at the memory's speed there."""
import numpy as np
import pytest

from sandengine_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def _kernels(fn):
    """The names of the kernels that fn launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    return {e.name for e in p.events()}


@pytest.fixture(scope="module", autouse=True)
def _profiler():
    """A process's first profile may come back empty while the tracer starts."""
    import torch
    for _ in range(5):
        if _kernels(lambda: torch.zeros(1000, device="cuda").add_(1)):
            return
    pytest.skip("no kernel trace on this machine")


@pytest.mark.parametrize("size, shape", [((2048, 2048), "56x30"), ((2049, 2048), "128x64"), ((64, 64), "56x30")])
def test_one_frame_launches(se, rulesets, ports, size, shape):
    from sandengine_gb300.batch import Batch
    from sandengine_gb300.serving import Server
    W, H = size
    rs = se.parse_string(rulesets["twelve_materials"])
    g = wl.patch_fill(W, H, 3, *wl.twelve_fill_spec(), patch=16)
    want = g.copy()
    ports["twelve_materials"].run(want, 3, 2, nthreads=8)
    b = Batch(rs, [size])
    b.set_resident_limit(0)
    b.set_steps_per_launch(1)
    b.set_grid(0, g)
    b.set_frame(0, 3)
    names = _kernels(lambda: b.step(2))
    assert [n for n in names if "tile" in n] == [f"se_mtile_{shape}_k1"], names
    assert np.array_equal(b.grid(0), want)
    srv = Server(rs, 1 << 28, 1)
    sid = srv.open_session(W, H, g, 3)
    srv.submit(sid, 2)
    names = _kernels(srv.run)
    assert [n for n in names if "tile" in n] == [f"se_stile_{shape}_k1"], names
    assert np.array_equal(srv.grid(sid), want)


def test_the_shape_follows_what_is_tiled(se, rulesets):
    from sandengine_gb300.batch import Batch
    rs = se.parse_string(rulesets["four_materials"])
    b = Batch(rs, [(400, 400)] * 40)
    b.set_steps_per_launch(1)
    for limit, shape in ((0, "128x64"), (1 << 30, None), (0, "128x64")):
        b.set_resident_limit(limit)
        for i in range(40):
            b.set_frame(i, 3)
        names = [n for n in _kernels(lambda: b.step(1)) if "mtile" in n]
        assert names == ([f"se_mtile_{shape}_k1"] if shape else [])

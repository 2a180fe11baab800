"""The frames a server's iteration or a batch's launch advances are the compiled depth that was asked
for (1, 2, 4, 8 or 16), whichever tile shape runs them, and the worlds are the oracle port's."""
import numpy as np
import pytest

from sandengine_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

DEPTHS = {1: 1, 2: 2, 3: 4, 4: 4, 5: 8, 8: 8, 16: 16}


@pytest.mark.parametrize("name", ["four_materials", "twelve_materials", "reference"])
def test_iterations_take_the_depth_asked_for(se, rulesets, ports, name):
    from sandengine_gb300.serving import Server
    rs, P = se.parse_string(rulesets[name]), ports[name]
    g = np.random.default_rng(3).integers(0, rs.num_materials, size=(70, 131)).astype(np.uint32)
    want = g.copy()
    P.run(want, 3, 35)
    for asked, depth in DEPTHS.items():
        srv = Server(rs, 1 << 26, asked)
        sid = srv.open_session(131, 70, g, 3)
        srv.submit(sid, 35)
        srv.run()
        assert srv.stats()["iterations"] == -(-35 // depth), asked
        assert np.array_equal(srv.grid(sid), want), asked


@pytest.mark.parametrize("name", ["four_materials", "twelve_materials"])
def test_batches_take_the_depth_asked_for(se, rulesets, ports, name):
    from sandengine_gb300.batch import Batch
    rs, P = se.parse_string(rulesets[name]), ports[name]
    rng = np.random.default_rng(4)
    sizes = [(300, 200), (64, 64), (7, 5), (129, 400)]
    grids = [rng.integers(0, rs.num_materials, size=(h, w)).astype(np.uint32) for w, h in sizes]
    wants = [g.copy() for g in grids]
    for i, w in enumerate(wants):
        P.run(w, 2 + i, 35)
    for asked, depth in DEPTHS.items():
        for limit in (None, 0, 20000):  # the default line, all tiled, some tiled; asked before and after
            b = Batch(rs, sizes)
            if limit == 0:
                b.set_resident_limit(limit)
            b.set_steps_per_launch(asked)
            if limit == 20000:
                b.set_resident_limit(limit)
            for i, g in enumerate(grids):
                b.set_grid(i, g)
                b.set_frame(i, 2 + i)
            assert b.info()["steps_per_launch"] == depth
            b.step(35)
            b.synchronize()
            for i, w in enumerate(wants):
                assert np.array_equal(b.grid(i), w), (asked, limit, sizes[i])

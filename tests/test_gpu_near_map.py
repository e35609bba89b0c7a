"""The near-wall map with wall nodes strewn over lattices of odd sizes: on closed lattices, where they also lie on
faces and edges, strict FP64 equals the oracle; on periodic ones a lattice whose walls and populations are
shifted by some nodes, across the wrap, ends as the shifted one.  Making the map is quick."""
import time

import numpy as np
import pytest

from hippolbm_b200 import capi
from hippolbm_b200.deck import Case, Op, couette_case

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def strewn(nodes, periodic, **kw):
    d = tuple(n - 1 for n in nodes)
    return Case(name="strewn", cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=periodic, tau=0.8, nuth=0.1,
                pre_stream_bcs=[Op("pre_bounce_back"), Op("wall_bounce_back")], post_stream_bcs=[Op("post_bounce_back")], **kw)


@pytest.mark.parametrize("nodes", [(13, 9, 11), (2, 7, 5), (33, 2, 6), (131, 5, 2)], ids=str)
def test_strewn_walls_equal_the_oracle(nodes, oracle_mod):
    from hippolbm_b200.lattice import Lattice

    rng = np.random.default_rng(sum(nodes))
    balls = [("ball", k, (tuple(float(rng.integers(0, n)) for n in nodes), 0.4)) for k in range(int(np.prod(nodes)) // 12)]
    c = strewn(nodes, (False,) * 3, obstacles=balls, double_couette={"U": [0.03, 0.02, 0.0], "dimension": "Z"})
    o = oracle_mod.run_case(c, 12)
    f_ref = o.real(o.f()).copy()
    for variant in (None, 4, 1):
        with Lattice.from_case(c, "f64_strict") as lat:
            if variant is not None:
                lat.tune(variant)
            lat.step(12)
            fluid = lat.flags() != -2
            assert 0 < (~fluid).sum() < fluid.size
            assert np.array_equal(lat.populations()[:, fluid], f_ref[:, fluid])


@pytest.mark.parametrize("nodes", [(13, 9, 11), (64, 7, 5), (35, 4, 6)], ids=str)
@pytest.mark.parametrize("axes", [(True, False, False), (False, True, True), (True, True, True)], ids=str)
@pytest.mark.parametrize("precision,variant", [("f64_strict", None), ("f64_strict", 4), ("f32", 4), ("f64", 1)])
def test_shifted_walls_give_the_shifted_state(nodes, axes, precision, variant):
    from hippolbm_b200.lattice import Lattice

    rng = np.random.default_rng(3)
    shape = nodes[::-1]
    flags = np.where(rng.random(shape) < 0.08, np.int8(-2), np.int8(-1))
    f = W[:, None, None, None] * (1 + 0.05 * rng.standard_normal((19,) + shape))
    shift = tuple(2 + k if axes[2 - k] else 0 for k in range(3))  # of the (z, y, x) arrays
    out = []
    for s in ((0, 0, 0), shift):
        with Lattice.from_case(strewn(nodes, axes), precision) as lat:
            if variant is not None:
                lat.tune(variant)
            lat.put_flags(np.roll(flags, s, axis=(0, 1, 2)))
            lat.put_populations(np.roll(f, s, axis=(1, 2, 3)))
            lat.step(6)
            back = tuple(-k for k in s)
            out.append(np.roll(lat.populations(), back, axis=(1, 2, 3))[:, flags != -2])
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])


def test_the_map_is_quick():
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(couette_case(320, 0.8, 0.05, 0), "f16") as lat:
        best = 1e9
        for _ in range(10):
            lat.sync()
            t = time.perf_counter()
            capi.check(lat.L.hlbm_update_obstacles(lat.h))
            lat.sync()
            best = min(best, time.perf_counter() - t)
        assert best < 0.4e-3  # 1.0 ms by the general loop for every node

"""A 16-bit lattice starts with a kernel that is not much slower than the better of the pair kernel and the
pipelines, small or large and whichever of its axes are periodic (rounds alternate, the fastest counts)."""
import time

import pytest

from hippolbm_b200.deck import Case, Op

pytestmark = pytest.mark.gpu

SPANS = [((255, 201, 130), (False, False, True)), ((255, 201, 130), (False, True, True)),
         ((181, 150, 170), (False, True, False)), ((181, 150, 170), (True, True, False)),
         ((37, 37, 2000), (False, True, False)), ((37, 37, 2000), (False, False, True)),
         ((80, 80, 80), (True, True, True)), ((64, 64, 64), (True, True, True)), ((80, 80, 80), (True, True, False))]


def box(nodes, periodic):
    d = tuple(n - 1 for n in nodes)
    return Case(name="box", cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=periodic, tau=0.7, nuth=0.2 / 3,
                pre_stream_bcs=[Op("pre_bounce_back")], post_stream_bcs=[Op("post_bounce_back")],
                double_couette={"U": [0.03, 0.02, 0.0], "dimension": "Z"})


@pytest.mark.parametrize("nodes,periodic", SPANS, ids=str)
def test_default_is_a_fast_kernel(nodes, periodic):
    from hippolbm_b200.lattice import Lattice

    lats = [Lattice.from_case(box(nodes, periodic), "f16") for _ in range(3)]
    lats[1].tune(4)
    lats[2].tune(9)
    best = [1e9] * 3
    for _ in range(4):
        for k, lat in enumerate(lats):
            lat.step(2)
            lat.sync()
            t = time.perf_counter()
            lat.step(100)
            lat.sync()
            best[k] = min(best[k], time.perf_counter() - t)
    for lat in lats:
        lat.close()
    assert best[0] <= 1.15 * min(best)


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_calls_of_one_step_are_quick(precision):
    """A small lattice stepped one step a call, without a fix-up launch: no slower than its step kernel."""
    from hippolbm_b200.lattice import Lattice

    lats = [Lattice.from_case(box((31, 31, 31), (True, True, True)), precision) for _ in range(2)]
    lats[1].tune(4)
    best = [1e9] * 2
    for _ in range(8):
        for k, lat in enumerate(lats):
            lat.step(2)
            lat.sync()
            t = time.perf_counter()
            for _ in range(100):
                lat.step(1)
            lat.sync()
            best[k] = min(best[k], time.perf_counter() - t)
    for lat in lats:
        lat.close()
    assert best[0] <= 1.2 * best[1]


@pytest.mark.parametrize("nodes,collision", [((130, 97, 113), "mrt"), ((256, 128, 128), "bgk")], ids=str)
def test_forced_fp32_variants_are_not_slower_than_one_node(nodes, collision):
    from hippolbm_b200.deck import poiseuille_case
    from hippolbm_b200.lattice import Lattice

    lats = [Lattice.from_case(poiseuille_case(nodes, 0.8, 1e-5, 0, collision), "f32").tune(v) for v in (4, 1, 3, 5)]
    best = [1e9] * len(lats)
    for _ in range(4):
        for k, lat in enumerate(lats):
            lat.step(2)
            lat.sync()
            t = time.perf_counter()
            lat.step(60)
            lat.sync()
            best[k] = min(best[k], time.perf_counter() - t)
    for lat in lats:
        lat.close()
    assert max(best[1:]) <= 1.15 * best[0]

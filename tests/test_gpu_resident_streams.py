"""Small lattices on their own streams share the GPU: eight of them, many steps a launch each, take well below
eight times as long as one (3.3 us a lattice step alone, 0.9 of eight), and each ends where it ends alone."""
import threading
import time

import numpy as np
import pytest

from hippolbm_b200.deck import lid_cavity_case

pytestmark = pytest.mark.gpu


def test_small_lattices_overlap():
    from hippolbm_b200.lattice import Lattice

    lats = [Lattice.from_case(lid_cavity_case((24, 24, 24), 0.8, 0.02 + 0.01 * k, 0), "f64") for k in range(8)]

    def seconds(some):
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            for lat in some:
                lat.step(400)
            for lat in some:
                lat.sync()
            best = min(best, time.perf_counter() - t)
        return best

    seconds(lats)
    one, eight = seconds(lats[:1]), seconds(lats)
    assert eight < 0.6 * 8 * one
    for lat in lats:
        lat.close()


@pytest.mark.parametrize("precision", ["f64", "f16"])
def test_threads_equal_alone(precision):
    from hippolbm_b200.lattice import Lattice

    sizes = [(24, 24, 24), (31, 20, 17), (41, 41, 41), (13, 9, 10), (57, 43, 61), (33, 33, 34)]
    cases = [lid_cavity_case(n, 0.8, 0.02 + 0.01 * k, 0) for k, n in enumerate(sizes)]
    want = []
    for c in cases:
        with Lattice.from_case(c, precision) as lat:
            want.append(lat.step(700).populations())
    lats = [Lattice.from_case(c, precision) for c in cases]

    def go(lat):
        for n in (300, 1, 399):
            lat.step(n)

    threads = [threading.Thread(target=go, args=(lat,)) for lat in lats]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for lat, f in zip(lats, want):
        assert np.array_equal(lat.populations(), f)
        lat.close()

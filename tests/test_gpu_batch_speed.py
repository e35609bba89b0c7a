"""The tile-list kernel, a batch's default, on ten mixed lattices (one with walls): FP32 steps faster than FP64, and
16-bit storage, which the same FP32 arithmetic bounds, about as fast as FP32."""
import time

import numpy as np
import pytest

from hippolbm_b200.deck import Case, Op, lid_cavity_case, sphere_channel_case

pytestmark = pytest.mark.gpu


def lattices():
    rng = np.random.default_rng(3)
    out = []
    for _ in range(8):
        d = tuple(int(v) - 1 for v in rng.choice(np.arange(32, 129, 8), 3))
        out.append(Case(name="couette", cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=(True, True, False), tau=0.7,
                        nuth=0.2 / 3, collision=str(rng.choice(["bgk", "mrt"])), pre_stream_bcs=[Op("pre_bounce_back")],
                        post_stream_bcs=[Op("post_bounce_back")]))
    return out + [sphere_channel_case((96, 48, 40), (24.0, 24.0, 20.0), 6.0, 0.7, 0.02, 0, "bgk"),
                  lid_cavity_case((64, 40, 48), 0.8, 0.05, 0)]


def test_default_batch_kernel_by_tier():
    from hippolbm_b200.batch import Batch
    from hippolbm_b200.lattice import Lattice

    seconds = {}
    for precision in ("f64", "f32", "f16"):
        lats = [Lattice.from_case(c, precision) for c in lattices()]
        batch = Batch(precision)
        for lat in lats:
            batch.add(lat)
        batch.step(20)
        seconds[precision] = 1e9
        for _ in range(5):
            t = time.perf_counter()
            batch.step(40)
            seconds[precision] = min(seconds[precision], time.perf_counter() - t)
        for lat in lats:
            lat.close()
    assert seconds["f32"] < 0.9 * seconds["f64"]
    assert seconds["f16"] < 1.3 * seconds["f32"]

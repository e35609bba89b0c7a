"""Lattices with a body force whose rows suit the vectorised kernel and the pipelines: FP32 with both collisions and
16-bit BGK by node pairs, every kernel against the one-node kernel bit for bit, alone and as batch
members; small ones alone step in the resident kernel."""
import numpy as np
import pytest

from hippolbm_b200.deck import poiseuille_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [(128, 9, 7), (132, 6, 8), (160, 11, 5), (260, 5, 6), (256, 40, 31), (128, 61, 43)], ids=str)
@pytest.mark.parametrize("precision,collision,variants", [("f32", "bgk", (1, 3, 5)), ("f32", "mrt", (1, 3, 5)),
                                                          ("f16", "bgk", (1, 3, 5, 8, 9)), ("bf16", "bgk", (1, 3, 5, 8, 9))])
def test_forced_kernels_agree(nodes, precision, collision, variants):
    from hippolbm_b200.batch import Batch
    from hippolbm_b200.lattice import Lattice

    case = poiseuille_case(nodes, 0.8, 1e-5, 0, collision)
    out = []
    for how in (4, None, "batch") + variants:
        with Lattice.from_case(case, precision) as lat:
            if how == "batch":
                batch = Batch(precision).tune(10)
                batch.add(lat)
                batch.step(15)
            else:
                if how is not None:
                    lat.tune(how)
                lat.step(15)
            out.append(lat.populations())
    assert np.isfinite(out[0]).all()
    for k, f in enumerate(out[1:]):
        assert np.array_equal(f, out[0]), k

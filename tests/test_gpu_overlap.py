"""Steps queued in one call, whose launches may overlap, equal steps launched and waited for one by one,
on lattices of many waves of blocks: the one-node, pair and vectorised kernels and both pipelines,
with the fix-up behind them, near-wall nodes and an outlet pass between the steps."""
import numpy as np
import pytest

from hippolbm_b200.deck import couette_case, lid_cavity_case, sphere_channel_case

pytestmark = pytest.mark.gpu

CASES = [lid_cavity_case((192, 160, 128), 0.7, 0.05, 0),  # six operator faces, rows of whole chunks
         lid_cavity_case((181, 150, 130), 0.7, 0.05, 0),  # ragged rows
         couette_case(150, 0.7, 0.05, 0),                  # periodic faces that are no operator's
         sphere_channel_case((256, 120, 110), (64.0, 60.0, 55.0), 12.0, 0.7, 0.02, 0)]


@pytest.mark.parametrize("precision", ["f64", "f32", "f16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c.name}-{c.nodes[0]}")
def test_queued_equals_waited(case, precision):
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(case, precision) as a, Lattice.from_case(case, precision) as b:
        a.step(1).step(60)
        for _ in range(61):
            b.step(1)
            b.sync()
        f = a.populations()
        assert np.isfinite(f).all()
        assert np.array_equal(f, b.populations())

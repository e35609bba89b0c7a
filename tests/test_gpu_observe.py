"""simulation_state straight from the post-collision state (one launch, nothing stored) gives the
values of the path that stores the streamed state first and reads it back, and leaves the run as it
was: odd sizes, fewer nodes than one block, walls, outlets and every tier.  Strict FP64 bit for bit;
elsewhere the boundary operators may contract products into FMAs differently in the two kernels, a
few ulp of the tier's arithmetic on face populations of order 1 (16-bit: one storage quantum, 2^-11
of a deviation of order 1e-3)."""
import numpy as np
import pytest

from hippolbm_b200.deck import lid_cavity_case, poiseuille_case, sphere_channel_case

pytestmark = pytest.mark.gpu

CASES = [lid_cavity_case((5, 6, 7), 0.8, 0.05, 0, "mrt"), lid_cavity_case((33, 18, 29), 0.8, 0.05, 0),
         poiseuille_case((70, 61, 75), 0.9, 1e-5, 0),
         sphere_channel_case((48, 21, 23), (14.0, 10.0, 11.0), 4.0, 0.7, 0.02, 0)]


@pytest.mark.parametrize("precision", ["f64_strict", "f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_state_without_storing_equals_the_stored_one(case, precision):
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(case, precision) as a, Lattice.from_case(case, precision) as b:
        for n in (1, 4, 7):
            a.step(n)
            b.step(n)
            straight = a.simulation_state()
            f = b.populations()  # stores S_k; the statistics then read it
            stored = b.simulation_state()
            if precision == "f64_strict":
                assert straight == stored
            eps = 1e-14 if precision.startswith("f64") else 2e-6
            assert abs(straight[0] - stored[0]) <= eps * a.ncell
            assert abs(straight[1] - stored[1]) <= eps and abs(straight[2] - stored[2]) <= eps
        assert np.array_equal(a.populations(), f)

"""simulation_state gives the same three numbers, in every tier and to the last bit, whether or not a read-out has
stored the state before: operators on every face, walls on faces, outlets, a body force and periodic axes."""
import numpy as np
import pytest

import test_gpu_fixup
import test_gpu_leading_bounce_back as leading
import test_gpu_resident
from hippolbm_b200.deck import lid_cavity_case, poiseuille_case, sphere_channel_case

pytestmark = pytest.mark.gpu


def cases(collision):
    return (test_gpu_resident.cases(collision) + [leading.case(o, (48, 14, 9), collision) for o in sorted(leading.ORDERS)]
            + [c.copy(collision=collision) for c in test_gpu_fixup.CASES]
            + [lid_cavity_case((75, 70, 69), 0.8, 0.05, 0, collision), poiseuille_case((70, 61, 75), 0.9, 1e-5, 0, collision),
               sphere_channel_case((128, 41, 43), (30.0, 20.0, 21.0), 8.0, 0.7, 0.02, 0, collision),
               sphere_channel_case((126, 41, 43), (30.0, 20.0, 21.0), 8.0, 0.7, 0.02, 0, collision)])


@pytest.mark.parametrize("precision", ["f64_strict", "f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("collision", ["bgk", "mrt"])
def test_statistics_do_not_depend_on_a_read_out(precision, collision):
    from hippolbm_b200.lattice import Lattice

    for c in cases(collision):
        with Lattice.from_case(c, precision) as a, Lattice.from_case(c, precision) as b:
            for n in (1, 4, 7):
                a.step(n)
                b.step(n)
                straight = a.simulation_state()
                f = b.populations()
                assert straight == b.simulation_state(), c.name
                assert straight == a.simulation_state(), c.name
            assert np.array_equal(a.populations(), f), c.name


LARGE = [sphere_channel_case((150, 91, 83), (40.0, 45.0, 41.0), 12.0, 0.7, 0.02, 0, "bgk"),
         lid_cavity_case((131, 97, 90), 0.8, 0.05, 0, "mrt"), poiseuille_case((128, 91, 97), 0.9, 1e-5, 0)]


@pytest.mark.parametrize("precision", ["f64_strict", "f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("c", LARGE, ids=lambda c: c.name)
def test_large_lattices_keep_the_state_they_observe(precision, c):
    """From a million nodes on simulation_state stores the state: read-outs after it, and steps after those, are the
    ones of a lattice that was never observed."""
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(c, precision) as a, Lattice.from_case(c, precision) as b:
        assert a.ncell >= 1 << 20
        for n in (1, 5, 3):
            a.step(n)
            b.step(n)
            state = a.simulation_state()
            launches = a.info()["launches"]
            f = a.populations()
            if precision.startswith("f64"):
                assert a.info()["launches"] == launches  # nothing is streamed again
            assert np.array_equal(f, b.populations())
            assert state == a.simulation_state() == b.simulation_state()

"""The near-wall list is made only for kernels that walk it: after the flags change, the first step by the FP64
one-node kernel, by the resident kernel or by a tile-list batch launches nothing but the step."""
import numpy as np
import pytest

from hippolbm_b200.deck import sphere_channel_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,variant", [("f64", 4), ("f32", None), ("f16", None), ("f32", 4)])
def test_no_list_for_kernels_that_test_for_walls(precision, variant):
    from hippolbm_b200.lattice import Lattice

    case = sphere_channel_case((40, 21, 23), (14.0, 10.0, 11.0), 4.0, 0.7, 0.02, 0, "bgk")
    case.boundary_conditions = [op for op in case.boundary_conditions if op.name != "zero_gradient"]
    with Lattice.from_case(case, precision) as lat:
        if variant is not None:
            lat.tune(variant)
        lat.step(2)
        for shift in (1, 2):
            before = lat.info()["launches"]
            lat.step(1)
            one = lat.info()["launches"] - before
            lat.put_flags(np.roll(lat.flags(), shift, axis=2))
            before = lat.info()["launches"]
            lat.step(1)
            assert lat.info()["launches"] - before == one


@pytest.mark.parametrize("precision,nodes", [("f32", (128, 30, 31)), ("f16", (96, 41, 30)), ("f16", (91, 90, 88))])
def test_list_follows_the_flags(precision, nodes):
    """Kernels that walk it, chosen before or after the flags change, alone and in a batch, equal the
    one-node kernel, which tests every node."""
    from hippolbm_b200.batch import Batch
    from hippolbm_b200.lattice import Lattice

    case = sphere_channel_case(nodes, (14.0, 10.0, 11.0), 4.0, 0.7, 0.02, 0)
    out = []
    for how in (4, 1, 9, "batch", "autotune"):
        with Lattice.from_case(case, precision) as lat:
            step = lat.step
            if how == "batch":
                lat.tune(9 if precision == "f16" else 1)
                batch = Batch(precision).tune(10)
                batch.add(lat)
                step = batch.step
            elif how == "autotune":
                lat.autotune(1)
            else:
                lat.tune(how)
            step(3)
            f = lat.populations()
            flags = lat.flags()
            f[:, flags == -2] = f[:, :1, 0, 0]
            lat.put_flags(np.roll(flags, (5, 3), axis=(2, 0)))
            lat.put_populations(f)
            step(5)
            out.append(lat.populations()[:, lat.flags() != -2])
    for f in out[1:]:
        assert np.array_equal(f, out[0])

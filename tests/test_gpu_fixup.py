"""The fix-up launch after the kernels that leave operator faces and near-wall nodes out: the
vectorised kernel and the row and span pipelines with it equal the kernels that do everything in
place, where faces meet each other and walls meet faces, and launches that overlap (a thousand
steps queued at once) equal launches waited for one by one."""
import numpy as np
import pytest

from hippolbm_b200.deck import Case, Op

pytestmark = pytest.mark.gpu


def case(nodes, faces, balls, collision="bgk"):
    d = tuple(n - 1 for n in nodes)
    ops = {"lid": Op("lid_driven_cavity", {"U": [0.03, 0.0, 0.0], "regions": ["plan_xy_l"]}),
           "sides": Op("neumann", {"U": [0.0, 0.0, 0.0], "regions": ["plan_xz_0", "plan_xz_l"]}),
           "inlet": Op("neumann", {"U": [0.01, 0.0, 0.0], "regions": ["plan_yz_0"]})}
    return Case(name="-".join(faces), cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=(False,) * 3, tau=0.9, nuth=0.4 / 3,
                collision=collision, obstacles=[("ball", k, (c, r)) for k, (c, r) in enumerate(balls)],
                pre_stream_bcs=[Op("pre_bounce_back")] + ([Op("wall_bounce_back")] if balls else []),
                post_stream_bcs=[Op("post_bounce_back")], boundary_conditions=[ops[f] for f in faces])


CASES = [case((48, 13, 11), ("lid",), []), case((45, 12, 10), ("inlet", "lid"), [((40.0, 3.0, 2.0), 5.0)]),
         case((48, 14, 12), ("sides", "inlet"), [((2.0, 7.0, 6.0), 4.0), ((30.0, 0.0, 11.0), 3.0)]),
         case((132, 9, 8), ("sides", "lid", "inlet"), [((60.0, 4.0, 4.0), 2.5)])]


def run(c, precision, variant, steps, wait=False):
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(c, precision) as lat:
        lat.tune(variant)
        for n in [1] * steps if wait else [steps]:
            lat.step(n)
            if wait:
                lat.sync()
        return lat.populations(), lat.flags() != -2


@pytest.mark.parametrize("precision,variants", [("f16", (4, 5, 8, 9)), ("f32", (4, 1)), ("f64", (4, 1))])
@pytest.mark.parametrize("c", CASES, ids=lambda c: f"{c.name}-{c.cell_dims[0]}")
def test_fixup_equals_inline(c, precision, variants):
    ref, fluid = run(c, precision, variants[0], 14)
    for v in variants[1:]:
        f, _ = run(c, precision, v, 14)
        if precision == "f64":  # the same expressions in another kernel: the tier's bound
            assert (np.abs(f - ref)[:, fluid] <= 1e-12 * np.abs(ref)[:, fluid]).all()
        else:
            assert np.array_equal(f[:, fluid], ref[:, fluid]), v


@pytest.mark.parametrize("precision,variant", [("f16", 9), ("f32", 1), ("f64", 4)])
def test_queued_steps_equal_steps_waited_for(precision, variant):
    for c in CASES:
        a, fluid = run(c, precision, variant, 1000)
        b, _ = run(c, precision, variant, 1000, wait=True)
        assert np.array_equal(a[:, fluid], b[:, fluid])

"""post_bounce_back in every place of the operator lists, against the oracle.

While no neumann / lid operator has run on a node, the pulled values are those post_bounce_back
restores, and the step applies only the z faces' cavity increments for it (and leaves the other
faces out of the face pass).  After one it restores the saved values as the reference does.  The
strict FP64 tier equals the oracle in every population; the 16-bit kernels that read the faces in
different ways (pair kernel, row / span pipelines) equal each other."""
import numpy as np
import pytest

from hippolbm_b200.deck import Case, Op

pytestmark = pytest.mark.gpu

BB, LID = Op("post_bounce_back"), Op("lid_driven_cavity", {"U": [0.03, 0.01, 0.0], "regions": ["plan_xy_l", "plan_xz_0"]})
NEU = Op("neumann", {"U": [0.01, 0.0, 0.0], "regions": ["plan_yz_0", "plan_xy_0"]})
MOVING = [Op("cavity_z_0", {"U": [0.02, 0.0, 0.0]}), Op("cavity_z_l", {"U": [0.0, 0.05, 0.0]}),
          Op("cavity_z_l", {"U": [0.01, 0.0, 0.0]})]
ORDERS = {  # (cavity operators, post_stream_bcs, boundary_conditions)
    "plain": ([], [BB], []),
    "twice": (MOVING, [BB, BB], [BB]),
    "moving_then_planes": (MOVING, [BB, LID], [NEU]),
    "after_planes": (MOVING, [LID, BB], [NEU, BB]),
    "between_planes": (MOVING, [BB, NEU, BB], [LID]),
    "outlet_first": ([], [Op("zero_gradient", {"regions": ["plan_yz_l"]}), BB], [NEU]),
}


def case(order, nodes, collision="bgk"):
    cavity, post, bcs = ORDERS[order]
    d = tuple(n - 1 for n in nodes)
    return Case(name=order, cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=(False, order == "twice", False), tau=0.8,
                nuth=0.1, collision=collision, pre_stream_bcs=[Op("pre_bounce_back")] + cavity, post_stream_bcs=post,
                boundary_conditions=bcs, steps=9)


# the outlet pass runs before the step whatever its place in the lists, so a post_bounce_back listed
# after it does not undo it, as it does in the oracle: that order is compared between kernels only
@pytest.mark.parametrize("order", sorted(set(ORDERS) - {"outlet_first"}))
def test_strict_fp64_equals_oracle(order, oracle_mod):
    from hippolbm_b200.lattice import Lattice

    c = case(order, (13, 9, 11))
    o = oracle_mod.run_case(c)
    f_ref = o.real(o.f()).copy()
    for variant in (4, 1, 6):
        with Lattice.from_case(c, "f64_strict") as lat:
            lat.tune(variant).step(c.steps)
            assert np.array_equal(lat.populations(), f_ref), (order, variant)


@pytest.mark.parametrize("order", sorted(ORDERS))
@pytest.mark.parametrize("nodes", [(48, 10, 12), (21, 14, 9), (5, 6, 7)])
def test_16bit_kernels_agree(order, nodes):
    from hippolbm_b200.lattice import Lattice

    c = case(order, nodes)
    out = []
    for variant in (4, 8, 9):
        with Lattice.from_case(c, "f16") as lat:
            lat.tune(variant).step(c.steps)
            out.append(lat.populations())
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])

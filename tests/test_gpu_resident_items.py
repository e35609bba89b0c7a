"""The resident kernel on 16-bit lattices of more nodes than the GPU has resident threads: face nodes and node
pairs as work items, against the one-launch-a-step kernel bit for bit with stochastic rounding.  Odd
planes (pairs across rows and planes), odd rows on even planes, axes of two and three nodes, periodic
and closed axes, operators on some faces, walls that touch a face, a body force, and the plans
whose every node takes the one-node path (start_iteration boxes, walls without bounce-back).
Lattices of at most that many nodes take the other branch (test_gpu_resident.py)."""
import numpy as np
import pytest
import torch

from hippolbm_b200.deck import Case, Op, lid_cavity_case, poiseuille_case
from hippolbm_b200.serve import solve_case

pytestmark = pytest.mark.gpu

BB = [Op("pre_bounce_back"), Op("cavity_z_l", {"U": [0.03, 0.0, 0.0]})]
AXES = [(False,) * 3, (True, True, False), (False, False, True), (True,) * 3, (False, True, False)]


def box(nodes, periodic, **kw):
    d = tuple(n - 1 for n in nodes)
    kw.setdefault("pre_stream_bcs", BB)
    return Case(name="box", cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=periodic, tau=0.7, nuth=0.2 / 3,
                post_stream_bcs=[Op("post_bounce_back")], **kw)


def cases(kind):
    if kind == "special":
        rng, ball = np.random.default_rng(5), [("ball", 0, ((2.0, 7.0, 6.0), 5.0)), ("ball", 1, ((30.0, 25.0, 39.0), 6.0))]
        walls = [Op("pre_bounce_back"), Op("wall_bounce_back")]
        inlet = [Op("neumann", {"U": [0.01, 0.0, 0.0], "regions": ["plan_yz_0"]})]
        return [lid_cavity_case((91, 87, 37), 0.8, 0.05, 0), poiseuille_case((91, 87, 37), 0.8, 1e-5, 0),
                solve_case("sphere", (61, 57, 59), 0.9, rng), solve_case("channel", (61, 57, 59), 0.9, rng),
                box((61, 51, 41), (False, True, False), obstacles=ball, pre_stream_bcs=walls, boundary_conditions=inlet),
                box((62, 51, 40), (True, False, False), obstacles=ball, pre_stream_bcs=walls),
                box((61, 51, 41), (False, True, False),
                    start_iteration=[Op("set_distribution", {"value": 1.01, "bounds": [[3.0, 4.0, 5.0], [9.0, 9.0, 9.0]]})]),
                box((61, 51, 41), (False, True, False), obstacles=ball)]
    # a lattice without boundary operators is stepped launch by launch from 24 MB on
    return [box(kind, axes, double_couette={"U": [0.03, 0.02, 0.0], "dimension": "Z"}) for axes in AXES if not (all(axes) and np.prod(kind) * 76 > 24 << 20)]


@pytest.mark.parametrize("precision", ["f16", "bf16"])
@pytest.mark.parametrize("kind", [(91, 87, 37), (90, 86, 41), (91, 86, 40), (2, 300, 301), (301, 2, 300),
                                  (300, 301, 2), (3, 301, 233), (64, 64, 64), (88, 87, 86), "special"], ids=str)
def test_items_equal_step_kernel(kind, precision):
    from hippolbm_b200.lattice import Lattice

    threads = torch.cuda.get_device_properties(0).multi_processor_count * 512
    for c in cases(kind):
        with Lattice.from_case(c, precision) as lat, Lattice.from_case(c, precision) as ref:
            assert lat.ncell > threads
            ref.tune(4).step(17)
            for n in (1, 1, 9, 6):
                lat.step(n)
            assert lat.info()["launches"] < ref.info()["launches"]  # many steps a launch
            fluid = ref.flags() != -2
            f, g = lat.populations()[:, fluid], ref.populations()[:, fluid]
            assert np.isfinite(g).all() and np.array_equal(f, g), (c.name, c.nodes, c.periodic)

"""The resident kernel (many steps of an L2-sized lattice in one cooperative launch) against the step
kernels that run one launch per step, and against the oracle.

The lattices cover rows shorter than a warp, odd rows and planes (node pairs across rows), two
nodes along an axis (no node off the faces), every axis periodic or bounced, boundary operators,
wall obstacles and a body force; the step counts cover one step, both buffer parities and two
launches (more steps than one launch takes).  The 16-bit tiers run BGK on them: with MRT the
node-pair and the one-node form may differ by one FP32 ulp in rare values."""
import numpy as np
import pytest

from hippolbm_b200.deck import Case, Op, lid_cavity_case, poiseuille_case
from hippolbm_b200.serve import solve_case

pytestmark = pytest.mark.gpu


def box(name, nodes, periodic, collision, **kw):
    d = tuple(n - 1 for n in nodes)
    return Case(name=name, cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=periodic, tau=0.75, nuth=0.25 / 3,
                collision=collision, **kw)


def cases(collision):
    rng = np.random.default_rng(3)
    bb = dict(pre_stream_bcs=[Op("pre_bounce_back"), Op("cavity_z_l", {"U": [0.05, 0.0, 0.0]})],
              post_stream_bcs=[Op("post_bounce_back")])
    out = [box("periodic", (37, 23, 19), (True, True, True), collision,
               obstacles=[("ball", 0, ((18.0, 11.0, 9.0), 4.0))], pre_stream_bcs=[Op("wall_bounce_back")]),
           box("couette", (45, 31, 26), (True, True, False), collision, **bb),
           box("rows5", (5, 10, 8), (True, False, False), collision, **bb),
           box("thin", (9, 2, 11), (False, True, False), collision, **bb),
           box("plate", (2, 14, 2), (False, False, True), collision, pre_stream_bcs=[Op("pre_bounce_back")],
               post_stream_bcs=[Op("post_bounce_back")]),
           lid_cavity_case((33, 18, 27), 0.8, 0.06, 0, collision),
           poiseuille_case((24, 11, 17), 0.9, 1e-5, 0, collision)]
    if collision == "bgk":
        out += [solve_case("channel", (35, 22, 19), 0.9, rng), solve_case("sphere", (41, 24, 29), 0.9, rng)]
    return out


def run(case, precision, steps, variant=None, rounding="stochastic"):
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(case, precision) as lat:
        lat.rounding(rounding)
        if variant is not None:
            lat.tune(variant)
        for n in steps:
            lat.step(n)
        return lat.populations(), lat.flags(), lat.info()["launches"]


@pytest.mark.parametrize("precision,collision", [("f16", "bgk"), ("bf16", "bgk"), ("f32", "bgk"), ("f32", "mrt"),
                                                 ("f64", "bgk"), ("f64", "mrt")])
def test_resident_equals_step_kernels(precision, collision):
    for c in cases(collision):
        f, flags, launches = run(c, precision, (1, 1, 12, 7))
        ref, _, many = run(c, precision, (21,), variant=4)
        assert launches < many, c.name  # one launch per call, not one per step
        keep = flags != -2  # wall nodes' populations are scratch
        assert np.isfinite(f).all()
        if precision == "f64":
            # the same expressions in another kernel: FMA contraction may differ, the bound is the tier's
            d = np.abs(f - ref)[:, keep]
            assert (d <= 1e-12 * np.abs(ref)[:, keep]).all(), (c.name, d.max())
        else:
            assert np.array_equal(f[:, keep], ref[:, keep]), c.name


@pytest.mark.parametrize("collision", ["bgk", "mrt"])
def test_resident_strict_fp64_equals_oracle(collision, oracle_mod):
    for c in cases(collision):
        f, flags, _ = run(c, "f64_strict", (25,))
        o = oracle_mod.run_case(c, 25)
        keep = flags != -2
        assert np.array_equal(f[:, keep], o.real(o.f())[:, keep]), c.name


def test_more_steps_than_one_launch_takes():
    c = lid_cavity_case((12, 9, 10), 0.9, 0.05, 0)
    f, _, _ = run(c, "f16", (2200,), rounding="nearest")
    ref, _, _ = run(c, "f16", (2200,), variant=4, rounding="nearest")
    assert np.array_equal(f, ref)

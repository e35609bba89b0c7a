"""FP64 lattices round alike in every kernel: the resident kernel that steps a small lattice alone, the step
kernels and the batch launches give the same bits, so a batch member equals its lattice stepped alone.
Random populations, walls and a body force."""
import numpy as np
import pytest

from hippolbm_b200.deck import Case, Op

pytestmark = pytest.mark.gpu

NODES = (64, 40, 28)  # 71,680 nodes: alone they step in the resident kernel
W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def case(collision, force, walls):
    d = tuple(n - 1 for n in NODES)
    return Case(name="random", cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=(True, False, True), tau=0.83, nuth=0.11,
                collision=collision, Fext=(1e-3, 2e-3, -5e-4) if force else (0.0, 0.0, 0.0),
                obstacles=[("ball", 0, ((25.0, 16.0, 14.0), 5.0))] if walls else [],
                pre_stream_bcs=[Op("pre_bounce_back")] + ([Op("wall_bounce_back")] if walls else []),
                post_stream_bcs=[Op("post_bounce_back")],
                boundary_conditions=[Op("neumann", {"U": [0.01, 0.02, -0.01], "regions": ["plan_xz_0"]}),
                                     Op("lid_driven_cavity", {"U": [0.03, 0.0, 0.01], "regions": ["plan_xz_l"]})])


@pytest.mark.parametrize("collision", ["bgk", "mrt"])
@pytest.mark.parametrize("force", [False, True], ids=["", "force"])
@pytest.mark.parametrize("walls", [False, True], ids=["", "walls"])
def test_fp64_kernels_agree(collision, force, walls):
    from hippolbm_b200.batch import Batch
    from hippolbm_b200.lattice import Lattice

    f0 = W[:, None, None, None] * (1 + 0.1 * np.random.default_rng(7).standard_normal((19,) + NODES[::-1]))
    out = {}
    for how in ("alone", 0, 1, 4, 6, "batch 8", "batch 6", "batch 10"):
        with Lattice.from_case(case(collision, force, walls), "f64") as lat:
            lat.put_populations(f0)
            if isinstance(how, int):
                lat.tune(how)
            if str(how).startswith("batch"):
                batch = Batch("f64").tune(int(how.split()[1]))
                batch.add(lat)
                batch.step(4)
            else:
                lat.step(4)
            out[how] = lat.populations()[:, lat.flags() != -2]
    assert np.isfinite(out["alone"]).all()
    for how, f in out.items():
        assert np.array_equal(f, out["alone"]), how

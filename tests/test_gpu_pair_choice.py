"""The 16-bit kernel a lattice starts with (pair kernel where face nodes are no operator's and rows are not
whole chunks, else a pipeline) gives the stored bits of every other one, with periodic and closed faces,
odd and even z-planes, and with a body force: BGK by node pairs, MRT by the one-node kernel."""
import numpy as np
import pytest

from hippolbm_b200.deck import Case, Op, poiseuille_case

pytestmark = pytest.mark.gpu


def box(nodes, periodic, collision="bgk"):
    d = tuple(n - 1 for n in nodes)
    return Case(name=f"{nodes}{periodic}{collision}", cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=periodic, tau=0.7,
                nuth=0.2 / 3, collision=collision, double_couette={"U": [0.03, 0.02, 0.0], "dimension": "Z"},
                pre_stream_bcs=[Op("pre_bounce_back")], post_stream_bcs=[Op("post_bounce_back")])


CASES = [box((103, 91, 90), (True, True, False)), box((102, 91, 90), (True, False, False)),
         box((102, 91, 90), (True, True, True), "mrt"), box((100, 90, 95), (False, False, False)),
         poiseuille_case((102, 91, 90), 0.8, 1e-5, 0), poiseuille_case((96, 91, 98), 0.8, 1e-5, 0),
         poiseuille_case((103, 91, 90), 0.8, 1e-5, 0), poiseuille_case((46, 31, 30), 0.8, 1e-5, 0, "mrt"),
         poiseuille_case((21, 10, 12), 0.8, 1e-5, 0)]


@pytest.mark.parametrize("precision", ["f16", "bf16"])
@pytest.mark.parametrize("c", CASES, ids=lambda c: c.name)
def test_default_equals_every_variant(c, precision):
    from hippolbm_b200.lattice import Lattice

    out = []
    for variant in (None, 4, 8, 9):
        with Lattice.from_case(c, precision) as lat:
            if variant is not None:
                lat.tune(variant)
            lat.step(11)
            out.append(lat.populations())
    assert np.isfinite(out[0]).all()
    for f in out[1:]:
        assert np.array_equal(f, out[0])

"""The row pipeline with 15 consumer warps (rows that fill its tile a tenth better than the tile of 12
warps: nx = 160, 320, 640) equals the pair kernel bit for bit, and so do row lengths around the rule and
plane heights that leave a last tile of fewer rows; the vectorised FP32 kernel on rows that leave part
of a block idle equals the one-node kernel."""
import numpy as np
import pytest

from hippolbm_b200.deck import Case, Op

pytestmark = pytest.mark.gpu


def couette(nodes, collision):
    d = tuple(n - 1 for n in nodes)
    return Case(name=f"c{nodes}", cell_dims=d, bmin=(0, 0, 0), bmax=d, periodic=(True, True, False), tau=0.7,
                nuth=0.2 / 3, collision=collision, pre_stream_bcs=[Op("pre_bounce_back"), Op("cavity_z_l", {"U": [0.05, 0.0, 0.0]})],
                post_stream_bcs=[Op("post_bounce_back")], double_couette={"U": [0.03, 0.02, 0.0], "dimension": "Z"})


def run(c, precision, variant):
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(c, precision) as lat:
        lat.tune(variant).step(9)
        return lat.populations()


@pytest.mark.parametrize("nodes", [(320, 6, 5), (320, 13, 4), (640, 7, 4), (160, 12, 6), (304, 9, 4), (336, 6, 4)])
@pytest.mark.parametrize("collision", ["bgk", "mrt"])
def test_wide_rows_equal_pairs(nodes, collision):
    c = couette(nodes, collision)
    for precision in ("f16", "bf16"):
        assert np.array_equal(run(c, precision, 9), run(c, precision, 4))


@pytest.mark.parametrize("nodes", [(128, 5, 4), (320, 9, 4), (260, 7, 5), (388, 3, 4), (512, 4, 3)])
def test_vector_rows_equal_one_node(nodes):
    c = couette(nodes, "mrt")
    assert np.array_equal(run(c, "f32", 1), run(c, "f32", 4))

"""The row pipeline at the row lengths around the ends of each range whose tiles 15 consumer warps fill a tenth
better than 12 (272, 320, 528 to 640, 784 to 960), planes lower than a tile and last tiles of fewer
rows, against the pair kernel bit for bit."""
import numpy as np
import pytest

import test_gpu_rows_wide as wide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [(256, 8, 3), (272, 9, 3), (288, 7, 3), (320, 3, 3), (512, 4, 3), (528, 7, 3), (640, 5, 3),
                                   (656, 4, 3), (768, 5, 3), (784, 5, 3), (960, 4, 3), (976, 3, 3), (960, 2, 2)], ids=str)
@pytest.mark.parametrize("collision", ["bgk", "mrt"])
def test_rows_equal_pairs(nodes, collision):
    c = wide.couette(nodes, collision)
    for precision in ("f16", "bf16"):
        assert np.array_equal(wide.run(c, precision, 9), wide.run(c, precision, 4))

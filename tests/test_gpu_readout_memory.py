"""Reading the populations of a large 16-bit lattice decodes into the plane that writing them used: a program that
has written them needs no more device memory to read them back."""
import numpy as np
import pytest
import torch

from hippolbm_b200 import capi
from hippolbm_b200.deck import couette_case

pytestmark = pytest.mark.gpu


def test_read_after_write_needs_no_more_memory():
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(couette_case(204, 0.8, 0.05, 0), "f16") as lat:
        f = lat.populations()
        lat.put_populations(f)
        capi.check(lat.L.hlbm_trim_memory(0))
        free = torch.cuda.mem_get_info(0)[0]
        g = lat.populations()
        assert free - torch.cuda.mem_get_info(0)[0] < lat.ncell * 8 // 2
        assert np.array_equal(f, g)

"""The barrier waits of many-step launches are bounded: with one poll allowed a 16-bit lattice's launch gives up, the
next read-out fails with HLBM_ECUDA and the context steps on; the bound that callers set leaves the other
tiers' small lattices as they are (their step kernels wait for nothing)."""
import numpy as np
import pytest

from hippolbm_b200 import capi
from hippolbm_b200.deck import couette_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f16", "f32", "f64"])
def test_wait_limit(precision):
    from hippolbm_b200.lattice import Lattice

    case = couette_case(31, tau=0.8, u_wall=0.05, steps=40)
    with Lattice.from_case(case, precision) as ref:
        ref.step(20)
        f0 = ref.populations()
        ref.put_populations(f0)
        ref.step(20)
        f1 = ref.populations()
    with Lattice.from_case(case, precision) as lat:
        capi.check(lat.L.hlbm_set_wait_limit(lat.h, 1))
        lat.step(20)
        if precision == "f16":
            with pytest.raises(capi.HlbmError) as e:
                lat.populations()
            assert e.value.code == -3 and "timed out" in str(e.value)  # HLBM_ECUDA
            capi.check(lat.L.hlbm_set_wait_limit(lat.h, 0))
            lat.put_populations(f0)
            lat.step(20)
            assert np.array_equal(lat.populations(), f1)
        else:
            assert np.array_equal(lat.populations(), f0)

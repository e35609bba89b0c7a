"""Read-outs of rho, u and the populations into pageable arrays that go through the pinned double buffer (several chunks, a last
one that is no whole number of shares) equal those into pinned memory, which are copied straight, before and
after the buffer is given back; threads that read different lattices at once get theirs."""
import ctypes as C
import threading

import numpy as np
import pytest

from hippolbm_b200 import capi
from hippolbm_b200.deck import lid_cavity_case

pytestmark = pytest.mark.gpu


def pinned(lat):
    import torch

    out = torch.empty(23 * lat.ncell, dtype=torch.float64, pin_memory=True)
    at = [C.cast(out.data_ptr() + 8 * k * lat.ncell, C.POINTER(C.c_double)) for k in (0, 1, 4)]
    capi.check(lat.L.hlbm_macro_variables(lat.h, *at[:2]))
    capi.check(lat.L.hlbm_get_populations(lat.h, at[2]))
    return out.numpy()


def pageable(lat):
    rho, u = lat.macro()
    return np.concatenate([rho.ravel(), u.ravel(), lat.populations().ravel()])


@pytest.mark.parametrize("precision", ["f64", "f32", "f16"])
@pytest.mark.parametrize("nodes", [(9, 8, 7), (67, 83, 101), (151, 139, 53)])
def test_pageable_equals_pinned(precision, nodes):
    from hippolbm_b200.lattice import Lattice

    with Lattice.from_case(lid_cavity_case(nodes, 0.8, 0.05, 0), precision) as lat:
        lat.step(5)
        want = pinned(lat)
        assert np.array_equal(pageable(lat), want)
        capi.check(lat.L.hlbm_trim_memory(0))
        assert np.array_equal(pageable(lat), want)


def test_threads_read_their_own_lattices():
    from hippolbm_b200.lattice import Lattice

    lats = [Lattice.from_case(lid_cavity_case((90 + k, 80, 70), 0.8, 0.02 + 0.02 * k, 0), "f16") for k in range(4)]
    want = []
    for lat in lats:
        lat.step(4)
        want.append(pinned(lat).copy())
    got = [None] * 4

    def read(k):
        got[k] = pageable(lats[k])

    threads = [threading.Thread(target=read, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, lat in enumerate(lats):
        assert np.array_equal(got[k], want[k])
        lat.close()

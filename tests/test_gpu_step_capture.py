"""Steps captured in a caller's CUDA graph on a lattice's stream replay as the steps launched directly: a small
lattice (many steps a launch outside a capture) and one with a fix-up launch after each step."""
import numpy as np
import pytest
import torch

from hippolbm_b200.deck import lid_cavity_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nodes", [(31, 20, 17), (96, 90, 84)], ids=str)
def test_captured_steps(nodes, precision):
    from hippolbm_b200.lattice import Lattice

    case = lid_cavity_case(nodes, 0.7, 0.05, 0)
    with Lattice.from_case(case, precision) as lat, Lattice.from_case(case, precision) as direct:
        lat.step(3)
        lat.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(lat.stream_handle())):
            graph.capture_begin(capture_error_mode="thread_local")
            lat.step(2)
            graph.capture_end()
            for _ in range(4):
                graph.replay()
        lat.sync()
        direct.step(3 + 2 * 4)
        assert np.array_equal(lat.populations(), direct.populations())

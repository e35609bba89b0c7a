"""A caller's capture of steps on a lattice whose plan is new: the first steps of a lattice, steps after the
flags changed, and an older graph replayed after them.  Replays, and the steps launched directly
afterwards (many a launch on the small lattice), equal the steps of a lattice that was never captured."""
import numpy as np
import pytest
import torch

from hippolbm_b200.deck import sphere_channel_case

pytestmark = pytest.mark.gpu


def capture(lat, steps):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(lat.stream_handle())):
        graph.capture_begin(capture_error_mode="thread_local")
        lat.step(steps)
        graph.capture_end()
    return graph


def replay(lat, graph, times):
    with torch.cuda.stream(torch.cuda.ExternalStream(lat.stream_handle())):
        for _ in range(times):
            graph.replay()
    lat.sync()


@pytest.mark.parametrize("precision", ["f64", "f32", "f16"])
@pytest.mark.parametrize("nodes", [(48, 21, 23), (132, 40, 31)], ids=str)
@pytest.mark.parametrize("collision", ["bgk", "mrt"])
def test_capture_of_a_new_plan(nodes, precision, collision):
    from hippolbm_b200.lattice import Lattice

    case = sphere_channel_case(nodes, (14.0, 10.0, 11.0), 4.0, 0.7, 0.02, 0, collision)
    with Lattice.from_case(case, precision) as lat, Lattice.from_case(case, precision) as direct:
        lat.rounding("nearest"), direct.rounding("nearest")
        if precision == "f64":  # one kernel on both sides: FP64 bits are the kernel's
            lat.tune(4), direct.tune(4)
        first = capture(lat, 2)  # collides the initial state
        replay(lat, first, 1)
        two = capture(lat, 2)
        replay(lat, two, 3)
        lat.step(5)
        direct.step(13)
        assert np.array_equal(lat.populations(), direct.populations())

        # flags change (every wall node gets fluid populations with them), steps are captured with the new
        # plan, the flags change again and the same graph replays: it follows the flags
        f = lat.populations()
        flags = lat.flags()
        f[:, flags == -2] = f[:, :1, 0, 0]

        def change(shift, axis):
            for k in (lat, direct):
                k.put_flags(np.roll(flags, shift, axis=axis))
                k.put_populations(f)
                k.step(1)

        change(3, 2)
        graph = capture(lat, 2)
        replay(lat, graph, 2)
        lat.step(4)
        direct.step(8)
        fluid = lat.flags() != -2
        assert np.array_equal(lat.populations()[:, fluid], direct.populations()[:, fluid])
        change(2, 1)
        lat.step(1)
        replay(lat, graph, 3)
        direct.step(7)
        fluid = lat.flags() != -2
        assert np.array_equal(lat.populations()[:, fluid], direct.populations()[:, fluid])
        del first, two, graph

"""Steps captured on the handle's stream and replayed between direct steps: the
same run as direct steps alone, bit for bit (a captured step runs the same
kernels, and every launch follows what is on the stream)."""
import numpy as np
import pytest

from tests.test_gpu_replaced_lists import ALPHA, BETA, outputs, same, sphere, unit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
@pytest.mark.parametrize("storage,box", [("fp32", False), ("fp16", False), ("fp16", True)])
@pytest.mark.parametrize("overlap", [None, "always"])
def test_replayed_and_direct_steps(gpu, streaming, storage, box, overlap):
    import torch

    tb = gpu

    def start():
        cu = unit(tb, streaming, storage, overlap)
        if box:
            cu.set_residual_box(30, 50, 30, 50, 30, 50)
        cu.initialise(1.0)
        cu.set_markers(sphere(tb, (40, 42, 44)))
        cu.forcing_resident(ALPHA, BETA)
        for _ in range(4):
            cu.step(ALPHA, BETA)
        return cu

    cu = start()
    stream = torch.cuda.ExternalStream(cu.stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        for _ in range(2):
            cu.step(ALPHA, BETA)
    for _ in range(6):
        if overlap is not None:
            cu.join()
        with torch.cuda.stream(stream):
            graph.replay()
        for _ in range(2):
            cu.step(ALPHA, BETA)
    cu.synchronize()
    plain = start()
    plain.set_overlap(False)
    for _ in range(24):
        plain.step(ALPHA, BETA)
    same(outputs(cu), outputs(plain))
    del graph


def test_a_captured_load_after_another_attach(gpu):
    """The impeller load inside a captured step, first thing after the impeller was
    attached again: the loads of the same steps queued directly."""
    import torch

    tb = gpu
    e, steps = 40, 4
    rt = tb.RushtonTurbine(e, e, e, tip_speed=0.1, startup_steps=0)
    d = rt.increment(1)

    def start():
        cu = tb.ComputeUnit(x=e, y=e, z=e, nu=1e-3, cs0=0.1, useLES=1)
        for _ in range(2):
            cu.attach_rushton(rt, d, 0.3, d)
        cu.initialise(1.0)
        cu.forcing_resident(ALPHA, BETA)
        cu.step(ALPHA, BETA)
        return cu

    cu = start()
    out = torch.zeros(5, dtype=torch.float64, pin_memory=True)
    stream = torch.cuda.ExternalStream(cu.stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        for _ in range(2):
            cu.step(ALPHA, BETA)
        cu.impeller_load_async(out.data_ptr())
    plain = start()
    for _ in range(steps):
        with torch.cuda.stream(stream):
            graph.replay()
        cu.synchronize()
        for _ in range(2):
            plain.step(ALPHA, BETA)
        np.testing.assert_array_equal(out.numpy(), plain.impeller_load())
    cu.close()
    plain.close()
    del graph

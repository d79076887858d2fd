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

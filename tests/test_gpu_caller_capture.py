"""Calls inside the caller's own stream capture: an eager frame, and the adjoint, whose second stream
has to join the capture. Replays against the same calls made directly."""
import numpy as np
import pytest

import trayracer_gb300 as tr

pytestmark = pytest.mark.gpu

W, H = 96, 64


@pytest.fixture
def setup():
    import torch

    scene = tr.cornell_box(width=W, height=H)
    r = tr.DeviceRenderer(0)
    r.UpdateScene(scene)
    r.SetCamera(scene.camera)
    r.Resize((W, H))
    r.SetSettings(tr.KernelSettings(multiSample=2, maxDepth=8, seed=3, rrStart=3))
    stream = torch.cuda.Stream()
    r.RenderFrame(stream=stream.cuda_stream)  # buffers are allocated before the capture
    torch.cuda.synchronize()
    yield torch, r, stream, scene.materials.shape[0]
    r.close()


def test_eager_frame(setup):
    torch, r, stream, _ = setup
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        r.RenderFrame(stream=stream.cuda_stream)
    images = []
    for replay in (True, False):
        r.Reset()
        for _ in range(2):
            graph.replay() if replay else r.RenderFrame()
        torch.cuda.synchronize()
        images.append(r.ColorBuffer().copy())
    assert (images[0] == images[1]).all() and images[0].max() > 0.0


def test_adjoint(setup):
    torch, r, stream, materials = setup
    pixels = torch.rand((H, W, 4), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    grads = torch.zeros((materials, 9), device="cuda")

    def adjoint():
        r.AdjointFrame(pixels.data_ptr(), 0.5, grads.data_ptr(), stream=stream.cuda_stream)

    adjoint()
    torch.cuda.synchronize()
    r.Reset()
    r.RenderFrame()  # the first frame's samples: those that the captured replay differentiates
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        adjoint()
    got = []
    for call in (graph.replay, adjoint, graph.replay):
        grads.zero_()
        torch.cuda.synchronize()
        call()
        torch.cuda.synchronize()
        got.append(grads.cpu().numpy().astype(np.float64))
    # sums of at most 2 * 96 * 64 * 8 terms of one material in any order: their rounding moves a sum by
    # less than 2^-24 * sqrt(1e5) of the largest gradient, on average
    assert np.abs(got[0]).max() > 0.0
    for g in got[::2]:
        assert np.abs(g - got[1]).max() <= 1e-4 * np.abs(got[1]).max()

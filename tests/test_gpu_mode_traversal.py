"""Closest hits of the other render modes, a thread a ray in small images and by lane refill in large
ones: the hit records of the primary rays against the host's run of the traversal, bit for bit."""
import numpy as np
import pytest

import trayracer_gb300 as tr

from test_gpu_traversal_counts import host_trace

pytestmark = pytest.mark.gpu

MISS = 0xFFFFFFFF


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("name", ["heightfield", "instanced"])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 1), (33, 1), (127, 1), (43, 3), (61, 37), (1024, 608), (1024, 609)])
def test_primary_hits(name, w, h, quant):
    # 4096 rays for each of 152 SMs: 1024 x 608 is the largest image of a thread a ray
    scene = tr.heightfield(n=33, seed=1) if name == "heightfield" else tr.instanced_cornell()
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetTuning(bvh_nodes=2 if quant else 1)
        r.SetCamera(scene.camera)
        r.Resize((w, h))
        st = tr.KernelSettings(maxDepth=1, seed=4)
        r.RenderFrame(st, tr.RenderModes.ShadingNormal)
        assert r.Statistics()["device_error"] == 0
        n, buf = w * h, r.Buffers()
        state = r.read_device(buf["path_state"][0], np.float32, 12 * n).reshape(3, n, 4)
        got = r.read_device(buf["hits"], np.uint32, 4 * n).reshape(n, 4)
    want, _ = host_trace(scene, np.ascontiguousarray(state[0]), np.ascontiguousarray(state[1]), st.rayEpsilon, 0, quant)
    hit = want[:, 2] != MISS
    assert hit.any() or n == 1
    assert (got[hit] == want[hit]).all() and (got[~hit, 2] == MISS).all()

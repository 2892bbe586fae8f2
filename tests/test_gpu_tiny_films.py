"""Films of one pixel, part of a warp, a warp and a ray: every pixel against the CPU oracle and the
numbers of rays exactly, over several seeds (nothing here may be off, unlike in a large image, where
a last-bit difference may flip some path's decision)."""
import numpy as np
import pytest

import trayracer_gb300 as tr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("name", ["cornell", "heightfield", "instanced"])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 1), (33, 1)])
def test_every_pixel_and_every_ray(name, w, h, layout):
    from oracle import Oracle

    scene = {"cornell": lambda: tr.cornell_box(width=w, height=h),
             "heightfield": lambda: tr.heightfield(n=33, width=w, height=h),
             "instanced": lambda: tr.instanced_cornell(width=w, height=h)}[name]()
    oracle = Oracle(scene)
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetTuning(bvh_nodes=layout)
        r.SetCamera(scene.camera)
        r.Resize((w, h))
        for seed in range(6):
            st = tr.KernelSettings(maxDepth=4, rrStart=1 << 30, seed=seed)
            acc, _, counts = oracle.render(scene.camera, st, w, h)
            ref = (acc[:, :3] / acc[:, 3:4]).reshape(h, w, 3)
            for graph in (False, True):
                r.SetSettings(st)
                r.Reset()
                r.RenderFrame(use_graph=graph)
                img, s = r.ColorBuffer()[..., :3], r.Statistics()
                assert s["device_error"] == 0
                assert (sum(s["extend_rays"]), sum(s["shadow_rays"])) == counts, (seed, graph)
                assert (np.abs(img - ref) <= 1e-4 * np.maximum(1.0, np.abs(ref))).all(), (seed, graph)

"""Persistent traversal kernels at small and ragged queue lengths, in both node layouts: every
path's pixel against the CPU oracle (single rays, part of a warp, a warp and a ray, ragged films;
scenes whose rays list few and many leaf triangles)."""
import numpy as np
import pytest

import trayracer_gb300 as tr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("name,w,h,ms", [("cornell", 1, 1, 1), ("cornell", 31, 1, 1), ("cornell", 33, 1, 1),
                                         ("cornell", 17, 13, 3), ("heightfield", 1, 1, 2), ("heightfield", 37, 29, 2),
                                         ("instanced", 33, 7, 2)])
def test_frames_match_the_oracle(name, w, h, ms, layout):
    from oracle import Oracle

    scene = {"cornell": lambda: tr.cornell_box(width=w, height=h, max_depth=4),
             "heightfield": lambda: tr.heightfield(n=33, width=w, height=h, max_depth=4),
             "instanced": lambda: tr.instanced_cornell(width=w, height=h, max_depth=4)}[name]()
    st = tr.settings_for(scene, multi_sample=ms)
    acc, _, counts = Oracle(scene).render(scene.camera, st, w, h, frames=2)
    ref = (acc[:, :3] / acc[:, 3:4]).reshape(h, w, 3)
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetTuning(bvh_nodes=layout)
        r.SetCamera(scene.camera)
        r.Resize((w, h))
        r.SetSettings(st)
        for graph in (False, True):
            r.Reset()
            r.RenderFrame(use_graph=graph)
            r.RenderFrame(use_graph=graph)
            img, stats = r.ColorBuffer(), r.Statistics()
            assert stats["device_error"] == 0
            close = (np.abs(img[..., :3] - ref) <= 1e-4 * np.maximum(1.0, np.abs(ref))).all(axis=-1)
            # a last-bit difference may flip a sampling decision of a path: one pixel in a hundred
            assert (~close).sum() <= max(1, 0.01 * close.size), (close.mean(), graph)

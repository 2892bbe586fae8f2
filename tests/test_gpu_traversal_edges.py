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


@pytest.mark.parametrize("name,w,h,ms,depth,rr,ref", [
    ("cornell", 3, 1, 1, 5, 1 << 30, False),      # taken at bounce 3 with fewer paths than a warp
    ("cornell", 64, 48, 1, 16, 1, False),
    ("lambert", 61, 37, 2, 16, 1, True),          # the reference's sampling
    ("disney", 256, 256, 2, 9, 1 << 30, False),   # too many at bounce 3, still too many at 6
    ("cornell", 300, 200, 3, 12, 2, False),       # too many at bounce 3, taken at 6
    ("sky", 160, 90, 2, 8, 3, False),             # paths that leave
    ("textured", 50, 41, 1, 8, 2, False),
    ("instanced", 50, 41, 1, 8, 2, False),
])
def test_frames_equal_their_stages(name, w, h, ms, depth, rr, ref):
    """A frame hands its remaining paths to one launch where a late bounce holds few (from bounce
    3 or 6 of frames of 5 bounces and more): the ray counts of the stage entries, which launch
    every bounce, and their images to the rounding of separately compiled shading code."""
    scene = {"cornell": lambda: tr.cornell_box(width=w, height=h),
             "lambert": lambda: tr.cornell_box(width=w, height=h, wall_closure=tr.TR_CLOSURE_LAMBERT),
             "disney": lambda: tr.cornell_box(width=w, height=h, wall_closure=tr.TR_CLOSURE_DISNEY),
             "sky": lambda: tr.outdoor_heightfield(n=64, width=w, height=h),
             "textured": lambda: tr.textured_cornell(width=w, height=h),
             "instanced": lambda: tr.instanced_cornell(width=w, height=h)}[name]()
    st = tr.KernelSettings(multiSample=ms, maxDepth=depth, rrStart=rr, seed=9,
                           flags=tr.TR_FLAG_REFERENCE_SAMPLING if ref else 0)
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetCamera(scene.camera)
        r.Resize((w, h))
        if name == "sky":
            r.SetSky(tr.SkySettings(sunDir=(0.2, 0.6, 0.4)))
        r.SetSettings(st)
        got = []
        for how in ("stages", "eager", "graph"):
            r.Reset()
            for _ in range(3):
                if how != "stages":
                    r.RenderFrame(use_graph=how == "graph")
                    continue
                r.BeginFrame()
                r.Generate()
                for b in range(depth):
                    r.Extend(b)
                    r.Shade(b)
                    r.Connect(b)
                r.Finalize()
            s = r.Statistics()
            got.append((r.ColorBuffer().copy(), s["extend_rays"], s["shadow_rays"], s["hit_rays"], s["device_error"]))
    for g in got[1:]:
        assert got[0][1:] == g[1:] and g[4] == 0
        # 3 frames of a few products each differ by at most some ulps of the 10.0 radiance limit
        assert np.abs(got[0][0] - g[0]).max() <= 1e-5


@pytest.mark.parametrize("ref,mode", [(False, tr.RenderModes.PathTracing), (True, tr.RenderModes.PathTracing),
                                      (False, tr.RenderModes.AmbientOcclusion)])
def test_stage_times_of_an_eager_frame(ref, mode):
    """Stage times are differences of the launches' start times: none negative, together within
    the frame's time between its events (5 us for the timers' steps)."""
    scene = tr.cornell_box(width=128, height=96)
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetCamera(scene.camera)
        r.Resize((128, 96))
        st = tr.KernelSettings(multiSample=2, maxDepth=16, rrStart=1,
                               flags=tr.TR_FLAG_REFERENCE_SAMPLING if ref else 0)
        for _ in range(3):
            r.RenderFrame(st, mode)
        s = r.Statistics()
        stages = [s[f"{k}_time_ms"] for k in ("generate", "extend", "shade", "connect", "finalize")]
        assert min(stages) >= 0.0 and stages[1] > 0.0 and stages[4] > 0.0
        assert sum(stages) <= s["render_time_ms"] + 0.005
        if mode == tr.RenderModes.PathTracing:
            assert stages[2] > 0.0 and stages[3] > 0.0
            assert sum(stages) >= 0.5 * s["render_time_ms"]

"""Which captured frames hand their remaining paths to one launch, and from which bounce: the word
that the launch leaves, against the ray counts of the stage entries, which launch every bounce."""
import numpy as np
import pytest

import trayracer_gb300 as tr

pytestmark = pytest.mark.gpu

TAKEN = 3 * 17 + 16  # counter word: the bounce from which the launch took the paths
FEW, FEW_STEADY = 32768, 4096
OFF = 1 << 30


def cornell(w, h):
    return tr.cornell_box(width=w, height=h)


def white(w, h):
    """Walls that reflect everything: roulette ends no path."""
    scene = tr.cornell_box(width=w, height=h, wall_closure=tr.TR_CLOSURE_LAMBERT)
    dark = scene.materials["emissive"].max(axis=-1) == 0
    scene.materials["diffuse"][dark] = 1.0
    return scene


def outdoor(w, h):
    return tr.outdoor_heightfield(n=64, width=w, height=h)


@pytest.mark.parametrize("make,w,h,ms,depth,rr,sky,asked,taken", [
    (cornell, 64, 64, 1, 6, OFF, False, 3, 3),      # 4096 paths: all of them, no condition
    (cornell, 3, 1, 1, 16, OFF, False, 3, 3),
    (white, 13, 7, 2, 16, OFF, False, 3, 3),
    (cornell, 64, 64, 1, 5, OFF, False, 0, 0),      # too few bounces to follow
    (cornell, 241, 17, 1, 16, OFF, False, 0, 0),    # 4097 paths, nothing makes them fade
    (cornell, 180, 180, 1, 16, OFF, False, 0, 0),
    (cornell, 256, 256, 1, 7, 1, False, 3, 3),      # roulette from 1, 2, 3
    (cornell, 150, 100, 1, 16, 2, False, 3, 3),
    (cornell, 300, 200, 1, 8, 3, False, 4, 4),
    (cornell, 300, 200, 1, 7, 3, False, 0, 0),
    (cornell, 512, 512, 1, 16, 1, False, 5, 5),     # more paths: two bounces later
    (cornell, 1400, 1000, 2, 9, 1, False, 5, 0),    # still too many
    (white, 200, 150, 1, 8, 1, False, 3, 0),        # few, but nearly all of the last bounce's
    (outdoor, 160, 90, 1, 8, OFF, True, 3, 3),
    (outdoor, 160, 90, 1, 5, OFF, True, 3, 3),
    (white, 200, 150, 1, 8, OFF, True, 3, 0),
])
def test_who_takes_the_last_paths(make, w, h, ms, depth, rr, sky, asked, taken):
    scene = make(w, h)
    st = tr.KernelSettings(multiSample=ms, maxDepth=depth, rrStart=rr, seed=9)
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetCamera(scene.camera)
        r.Resize((w, h))
        if sky:
            r.SetSky(tr.SkySettings(sunDir=(0.2, 0.6, 0.4)))
        r.SetSettings(st)
        got = []
        for graph in (False, True):
            r.Reset()
            for _ in range(2):
                if graph:
                    r.RenderFrame(use_graph=True)
                    continue
                r.BeginFrame()
                r.Generate()
                for b in range(depth):
                    r.Extend(b)
                    r.Shade(b)
                    r.Connect(b)
                r.Finalize()
            s = r.Statistics()
            assert s["device_error"] == 0
            word = int(r.read_device(r.Buffers()["counters"], np.uint32, TAKEN + 1)[TAKEN])
            got.append((r.ColorBuffer().copy(), s["extend_rays"], s["shadow_rays"], s["hit_rays"], word))
        rays = got[0][1]
        assert got[0][4] == 0 and got[1][4] == taken, rays
        assert got[0][1:4] == got[1][1:4]
        if taken:
            assert 0 < rays[asked] <= FEW
        else:  # the same launches: the same bits
            assert (got[0][0] == got[1][0]).all()
        if asked and not taken:  # declined: too many, or more than two thirds of the bounce before
            steady = 3 * rays[asked] > 2 * rays[asked - 1]
            assert rays[asked] > (FEW_STEADY if steady else FEW), rays


def test_counting_and_other_modes_launch_every_bounce():
    scene = cornell(40, 30)
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetCamera(scene.camera)
        r.Resize((40, 30))
        for flags, mode in ((tr._abi.TR_FLAG_COUNT_TRAVERSAL, tr.RenderModes.PathTracing), (0, tr.RenderModes.ShadingNormal)):
            r.RenderFrame(tr.KernelSettings(maxDepth=12, rrStart=1, flags=flags), mode, use_graph=True)
            assert r.Statistics()["device_error"] == 0
            assert int(r.read_device(r.Buffers()["counters"], np.uint32, TAKEN + 1)[TAKEN]) == 0

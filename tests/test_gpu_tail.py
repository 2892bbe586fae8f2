"""Which captured frames hand their remaining paths to one launch, and from which bounce: the word
that the launch leaves, against the ray counts of the stage entries, which launch every bounce."""
import dataclasses

import numpy as np
import pytest

import trayracer_gb300 as tr
from trayracer_gb300.scenes import random_soup

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


def terrain(w, h):
    """833 nodes: many."""
    return tr.heightfield(n=65, width=w, height=h)


def small_terrain(w, h):
    """34 nodes: not many."""
    return tr.heightfield(n=9, width=w, height=h)


def room(w, h):
    """The closed box around 1000 small triangles: many nodes."""
    box, soup = cornell(w, h), random_soup(1000, seed=5)
    join = lambda a, b: None if a is None else np.concatenate([a, b]).astype(a.dtype)  # noqa: E731
    n = soup.positions.shape[0]
    return dataclasses.replace(
        box, positions=join(box.positions, soup.positions * np.float32(0.3)),
        normals=join(box.normals, np.tile(np.float32([0, 1, 0]), (n, 1))),
        texcoords=join(box.texcoords, np.zeros((n, 2), np.float32)),
        indices=join(box.indices, soup.indices + box.positions.shape[0]),
        material_indices=join(box.material_indices, np.zeros(soup.indices.shape[0], np.uint32)))


def spheres(w, h):
    """Many nodes, and paths that hardly end."""
    return tr.displaced_spheres(count=40, n_emissive=2, width=w, height=h, extent=40.0 * (40 / 4096.0) ** (1.0 / 3.0))


@pytest.mark.parametrize("make,w,h,ms,depth,rr,sky,asked,taken", [
    (cornell, 64, 64, 1, 6, OFF, False, (3,), 3),       # 4096 paths: all of them, no condition
    (cornell, 3, 1, 1, 16, OFF, False, (3,), 3),
    (white, 13, 7, 2, 16, OFF, False, (3,), 3),
    (cornell, 64, 64, 1, 5, OFF, False, (), 0),         # too few bounces to follow
    (cornell, 241, 17, 1, 16, OFF, False, (), 0),       # 4097 paths, nothing makes them fade
    (cornell, 180, 180, 1, 16, OFF, False, (), 0),
    (cornell, 256, 256, 1, 7, 1, False, (3,), 3),       # roulette from 1, 2, 3
    (cornell, 150, 100, 1, 16, 2, False, (3,), 3),
    (cornell, 300, 200, 1, 8, 3, False, (4,), 4),
    (cornell, 300, 200, 1, 7, 3, False, (), 0),
    (cornell, 512, 512, 1, 16, 1, False, (5,), 5),      # more paths: two bounces later
    (cornell, 1400, 1000, 2, 9, 1, False, (5,), 0),     # still too many
    (white, 200, 150, 1, 8, 1, False, (3,), 0),         # few, but nearly all of the last bounce's
    (outdoor, 160, 90, 1, 8, OFF, True, (3,), 3),
    (outdoor, 160, 90, 1, 5, OFF, True, (3,), 3),
    (white, 200, 150, 1, 8, OFF, True, (3,), 0),
    (terrain, 300, 200, 1, 5, OFF, False, (3,), 3),     # many nodes: without a sky or roulette too
    (small_terrain, 300, 200, 1, 16, OFF, False, (), 0),
    (terrain, 240, 200, 1, 6, 3, False, (3,), 3),       # 48 000 paths
    (terrain, 300, 200, 1, 6, 3, False, (3, 4), 3),     # more: a second chance
    (room, 400, 300, 1, 8, 3, False, (3, 4), 4),
    (room, 150, 150, 1, 8, 3, False, (3,), 3),
    (spheres, 700, 500, 1, 8, 3, False, (3, 6), 6),
    (spheres, 300, 300, 1, 8, OFF, False, (3,), 3),     # nearly all of the last bounce's, but not too many
    (spheres, 1200, 1000, 1, 8, OFF, False, (3, 6), 0),
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
        many_nodes = r.SceneInfo()["bvh_node_count"] >= 64
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
    if not taken:  # the same launches: the same bits
        assert (got[0][0] == got[1][0]).all()
    assert not taken or taken in asked
    for b in asked[:asked.index(taken) + 1] if taken else asked:
        steady = 3 * rays[b] > 2 * rays[b - 1]
        few = FEW_STEADY if steady and not many_nodes else FEW
        assert 0 < rays[b] and (rays[b] <= few) == (b == taken), rays
    if make is spheres and rr == OFF and taken:
        assert steady and rays[taken] > FEW_STEADY, rays


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

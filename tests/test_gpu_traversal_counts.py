"""The traversal kernels on given rays (written into the queues that the stage entries read)
against the host's run of the same traversal: hits bit for bit, and the nodes and triangles that
TR_FLAG_COUNT_TRAVERSAL sums up."""
import ctypes as C

import numpy as np
import pytest

import trayracer_gb300 as tr
from trayracer_gb300 import _abi
from trayracer_gb300.renderer import SceneDescHolder
from trayracer_gb300.scenes import random_soup

from test_box_test import CLOSE_CALLS

pytestmark = pytest.mark.gpu

BOUNCES = 17  # counters per bounce: extend and shadow queue lengths, two cursors, hit queue length
N = 6000      # rays: more than a warp's refill takes, not a multiple of a warp


def host_trace(scene, O, D, tmin, any_hit, quant):
    h = SceneDescHolder(scene)
    hits = np.zeros((O.shape[0], 4), np.uint32)
    counts = np.zeros((O.shape[0], 2), np.uint32)
    st = _abi.load_library().tr_trace_host(C.byref(h.desc), O.ctypes.data, D.ctypes.data, O.shape[0], tmin,
                                           any_hit | (2 if quant else 0), hits.ctypes.data, counts.ctypes.data)
    assert st == 0
    return hits, counts


def the_scene(name):
    if name == "heightfield":
        return tr.heightfield(n=33, seed=1)
    if name == "instanced":
        return tr.instanced_cornell()
    scene = random_soup(3000, seed=5)
    if name == "triangle":
        scene = random_soup(1, seed=2)
        scene.positions[:] = np.array([[-1, 0, -1], [1, 0, -1], [0, 0, 1]], np.float32)
    return scene


def the_rays(name, scene, seed):
    rng = np.random.default_rng(seed)
    O = np.zeros((N, 4), np.float32)
    D = np.zeros((N, 4), np.float32)
    O[:, :3] = rng.uniform(-1.0, 1.0, (N, 3)) * (0.8 if name == "instanced" else 1.0)
    if name == "heightfield":
        O[:, :3] = scene.camera.position
    d = rng.normal(size=(N, 3))
    if name == "heightfield":
        d[:, 1] = -np.abs(d[:, 1])
    d[rng.random(N) < 0.1, 1] = 0.0  # along a coordinate plane
    D[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    D[:, 3] = rng.uniform(0.5, 20.0, N) * (4.0 if name == "heightfield" else 1.0)
    if name == "heightfield":
        close = np.array([c[1] for c in CLOSE_CALLS], np.uint32).view(np.float32)
        D[:500, :3] = close[np.arange(500) % len(close)]
    if name == "triangle":  # from the triangle itself, up and down
        O[:, :3] = 0.0
        D[:, :3] = 0.0
        D[::2, 1], D[1::2, 1] = 1.0, -1.0
    return O, D


def renderer(scene, quant, eps, step_limit=0):
    r = tr.DeviceRenderer(0)
    r.UpdateScene(scene)
    r.SetTuning(bvh_nodes=2 if quant else 1)
    r.SetCamera(scene.camera)
    r.Resize((N, 1))
    r.SetSettings(tr.KernelSettings(maxDepth=2, rayEpsilon=eps, flags=_abi.TR_FLAG_COUNT_TRAVERSAL,
                                    traversalStepLimit=step_limit))
    r.BeginFrame()
    r.Synchronize()
    return r, r.Buffers()


CASES = [("heightfield", 1e-3), ("soup", 1e-3), ("instanced", 1e-3), ("triangle", 0.0)]


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("name,eps", CASES)
def test_closest_hits_and_their_counts(name, eps, quant):
    scene = the_scene(name)
    O, D = the_rays(name, scene, 3)
    want, counts = host_trace(scene, O, D, eps, 0, quant)
    r, buf = renderer(scene, quant, eps)
    state = np.zeros((3, N, 4), np.float32)
    state[0], state[1] = O, D
    state[0][:, 3] = (np.arange(N, dtype=np.uint32) << 4).view(np.float32)
    r.write_device(buf["path_state"][0], state)
    r.write_device(buf["counters"] + 4 * 1, np.array([N], np.uint32))  # bounce 1's extend queue
    r.Extend(1)
    s = r.Statistics()
    n_hit = s["hit_rays"][1]
    path = r.read_device(buf["path_state"][1], np.uint32, n_hit * 4).reshape(n_hit, 4)[:, 3] >> 4
    hits = r.read_device(buf["hits"], np.uint32, n_hit * 4).reshape(n_hit, 4)
    r.close()
    got = np.tile(np.array([0, 0xFFFFFFFF, 0xFFFFFFFF, 0], np.uint32), (N, 1))
    got[path] = hits
    hit = want[:, 2] != 0xFFFFFFFF
    assert s["device_error"] == 0 and n_hit == hit.sum() > 0.05 * N
    assert (got[hit] == want[hit]).all() and (got[~hit, 2] == 0xFFFFFFFF).all()
    assert (s["traversal_extend_nodes"], s["traversal_extend_tris"]) == tuple(counts.sum(0, dtype=int))


def connect(r, buf, O, D, eps):
    """Runs bounce 1's connect launch over the given rays (D.w: how far each may be occluded);
    returns whether each was, and the statistics."""
    n = O.shape[0]
    shadow = np.zeros((3, N, 4), np.float32)
    shadow[0, :n], shadow[1, :n] = O, D
    shadow[0, :n, 3] = np.arange(n, dtype=np.uint32).view(np.float32)
    shadow[1, :n, 3] = D[:, 3] + np.float32(2.0) * np.float32(eps)
    shadow[2, :n, 0] = 1.0
    r.write_device(buf["shadow"], shadow)
    r.write_device(buf["radiance"], np.zeros((N, 4), np.float32))
    r.write_device(buf["counters"] + 4 * (BOUNCES + 1), np.array([n], np.uint32))  # bounce 1's shadow queue
    r.Connect(1)
    return r.read_device(buf["radiance"], np.float32, 4 * N).reshape(N, 4)[:n, 0] == 0.0, r.Statistics()


def shadow_rays(name, scene, eps, seed):
    O, D = the_rays(name, scene, seed)
    # the distance that the kernel is left with after it took 2 eps off again
    D[:, 3] = (D[:, 3] + np.float32(2.0) * np.float32(eps)) - np.float32(2.0) * np.float32(eps)
    return O, D


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("name,eps", CASES)
def test_shadow_rays_and_their_counts(name, eps, quant):
    """What is visited and tested up to a ray's first hit, although a warp tests the triangles of
    its rays together."""
    scene = the_scene(name)
    O, D = shadow_rays(name, scene, eps, 4)
    want, counts = host_trace(scene, O, D, eps, 1, quant)
    r, buf = renderer(scene, quant, eps)
    occluded, s = connect(r, buf, O, D, eps)
    r.close()
    assert s["device_error"] == 0 and 0.05 * N < occluded.sum()
    assert (occluded == (want[:, 2] != 0xFFFFFFFF)).all()
    assert (s["traversal_connect_nodes"], s["traversal_connect_tris"]) == tuple(counts.sum(0, dtype=int))


@pytest.mark.parametrize("name", ["heightfield", "soup"])
def test_a_hit_within_the_step_limit_is_no_error(name):
    """Occluded rays at the step limit that each reaches its hit with, and one step below it."""
    scene = the_scene(name)
    O, D = shadow_rays(name, scene, 1e-3, 6)
    want, counts = host_trace(scene, O, D, 1e-3, 1, False)
    hit = want[:, 2] != 0xFFFFFFFF
    steps = counts[hit, 0]
    limit = int(np.median(steps))
    for ok, chosen in ((True, steps <= limit), (False, steps == limit + 1)):
        o, d = np.ascontiguousarray(O[hit][chosen]), np.ascontiguousarray(D[hit][chosen])
        assert o.shape[0] > 100
        r, buf = renderer(scene, False, 1e-3, limit)
        occluded, s = connect(r, buf, o, d, 1e-3)
        r.close()
        assert s["device_error"] == (0 if ok else 1)
        assert occluded.all() if ok else not occluded.all()

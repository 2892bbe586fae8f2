"""The two BVH node layouts at the edges of what the quantized one takes: every ray octant and
axis-parallel rays, geometry far from the origin and very small, and scenes beyond its exponents
(which keep fp32 child boxes) - host traversal, closest and any hit, both layouts hit for hit."""
import ctypes as C

import numpy as np
import pytest

import trayracer_gb300 as tr
from trayracer_gb300 import _abi
from trayracer_gb300.renderer import SceneDescHolder
from trayracer_gb300.scenes import placement, random_soup


def _trace(scene, O, D, any_hit, quant, tmin=0.0):
    h = SceneDescHolder(scene)
    hits = np.zeros((O.shape[0], 4), np.uint32)
    counts = np.zeros((O.shape[0], 2), np.uint32)
    st = _abi.load_library().tr_trace_host(C.byref(h.desc), O.ctypes.data, D.ctypes.data, O.shape[0], tmin,
                                           int(any_hit) | (2 if quant else 0), hits.ctypes.data, counts.ctypes.data)
    assert st == 0
    return hits, counts


def _rays(scene, n, scale, offset, seed):
    rng = np.random.default_rng(seed)
    O = np.zeros((n, 4), np.float32)
    D = np.zeros((n, 4), np.float32)
    O[:, :3] = rng.uniform(-1.2, 1.2, (n, 3)) * scale + offset
    d = rng.normal(size=(n, 3))
    d *= np.where(np.arange(n)[:, None] >> np.arange(3) & 1, 1.0, -1.0) * np.sign(d)  # octant n & 7
    axis = rng.random(n) < 0.2
    d[axis, rng.integers(0, 3, axis.sum())] = 0.0  # parallel to a coordinate plane
    D[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    D[:, 3] = 8.0 * scale
    return O, D


@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1.0, 1000.0), (1e-5, 0.0), (1e6, 0.0), (3e7, 0.0), (1e12, 0.0)])
def test_layouts_hit_the_same(scale, offset):
    scene = random_soup(3000, seed=5)
    scene.positions = (scene.positions * np.float32(scale) + np.float32(offset)).astype(np.float32)
    O, D = _rays(scene, 6000, scale, offset, 11)
    for any_hit in (False, True):
        wide, cw = _trace(scene, O, D, any_hit, False)
        quant, cq = _trace(scene, O, D, any_hit, True)
        assert (wide[:, 2] != 0xFFFFFFFF).mean() > 0.3
        if any_hit:  # any hit: another triangle may end the ray first
            assert ((wide[:, 2] != 0xFFFFFFFF) == (quant[:, 2] != 0xFFFFFFFF)).all()
        else:
            assert (wide == quant).all()
        if scale >= 3e7:  # past 2^24: fp32 nodes serve both
            assert (cw == cq).all()
        else:
            assert (cw != cq).any()


@pytest.mark.parametrize("scale,falls_back", [(1e-3, False), (1e-5, False), (1e-7, True)])
def test_layouts_hit_the_same_inside_small_instances(scale, falls_back):
    """An instance of scale s magnifies ray directions by 1 / s in its space."""
    scene = tr.instanced_cornell()
    scene.instances = [(m, x * np.float32(scale)) for m, x in scene.instances]
    O, D = _rays(scene, 4000, 0.8 * scale, 0.0, 3)
    wide, cw = _trace(scene, O, D, False, False)
    quant, cq = _trace(scene, O, D, False, True)
    assert (wide[:, 2] != 0xFFFFFFFF).mean() > 0.3
    assert (wide == quant).all(axis=1).mean() >= 0.999  # coplanar faces of touching instances tie
    assert (cw == cq).all() == falls_back


def test_one_triangle_and_flat_scenes():
    scene = random_soup(1, seed=2)
    O, D = _rays(scene, 2000, 1.0, 0.0, 4)
    assert (_trace(scene, O, D, False, False)[0] == _trace(scene, O, D, False, True)[0]).all()
    flat = random_soup(500, seed=3)
    flat.positions[:, 1] = np.float32(0.25)  # all boxes without extent along y
    O, D = _rays(flat, 2000, 1.0, 0.0, 5)
    wide, quant = _trace(flat, O, D, True, False)[0], _trace(flat, O, D, True, True)[0]
    assert ((wide[:, 2] != 0xFFFFFFFF) == (quant[:, 2] != 0xFFFFFFFF)).all()

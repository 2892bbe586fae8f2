"""The box test's decision where its two distances meet: tn <= 1.0000004 tf with a rounded product
and no sign of zero. Host traversal, both node layouts."""
import ctypes as C

import numpy as np
import pytest

import trayracer_gb300 as tr
from trayracer_gb300 import _abi
from trayracer_gb300.renderer import SceneDescHolder
from trayracer_gb300.scenes import random_soup

# Camera rays of heightfield(n=33, seed=1) (direction as float bits) for which a product fused with
# the difference decides otherwise at some node: (layout, direction, nodes, triangles tested, primitive).
CLOSE_CALLS = [
    (0, (3190206878, 3192778105, 1064781946), 4, 0, 0xFFFFFFFF),
    (0, (1034095069, 3198996392, 1064312112), 8, 5, 1574),
    (0, (3199137219, 3200537246, 1062971202), 8, 4, 970),
    (2, (1053980202, 3201249144, 1062280866), 8, 4, 953),
    (2, (3204698120, 3206166870, 1058808099), 4, 4, 11),
    (2, (3191608589, 3201145042, 1063628970), 7, 2, 980),
    (2, (3199137219, 3200537246, 1062971202), 8, 4, 970),
]


def _trace(scene, O, D, tmin, flags):
    h = SceneDescHolder(scene)
    hits = np.zeros((O.shape[0], 4), np.uint32)
    counts = np.zeros((O.shape[0], 2), np.uint32)
    st = _abi.load_library().tr_trace_host(C.byref(h.desc), O.ctypes.data, D.ctypes.data, O.shape[0], tmin, flags,
                                           hits.ctypes.data, counts.ctypes.data)
    assert st == 0
    return hits, counts


@pytest.mark.parametrize("any_hit", [0, 1])
@pytest.mark.parametrize("layout", [0, 2])
def test_hits_at_distance_zero(layout, any_hit):
    """Rays of both directions that start on a triangle (and on the planes of its flat box)."""
    scene = random_soup(1, seed=2)
    for axis in range(3):
        scene.positions[:] = np.roll(np.array([[-1, 0, -1], [1, 0, -1], [0, 0, 1]], np.float32), axis - 1, axis=1)
        O = np.zeros((2, 4), np.float32)
        D = np.zeros((2, 4), np.float32)
        D[:, axis] = (1.0, -1.0)
        D[:, 3] = 5.0
        hits, _ = _trace(scene, O, D, 0.0, any_hit | layout)
        assert (hits[:, 2] == 0).all() and (hits[:, 3].view(np.float32) == 0.0).all(), axis


@pytest.mark.parametrize("layout,direction,nodes,tris,prim", CLOSE_CALLS)
def test_product_is_rounded_before_the_comparison(layout, direction, nodes, tris, prim):
    scene = tr.heightfield(n=33, seed=1)
    O = np.zeros((1, 4), np.float32)
    O[0, :3] = scene.camera.position
    D = np.zeros((1, 4), np.float32)
    D[0, :3] = np.array(direction, np.uint32).view(np.float32)
    hits, counts = _trace(scene, O, D, 1e-3, layout)
    assert tuple(counts[0]) == (nodes, tris) and hits[0, 2] == prim

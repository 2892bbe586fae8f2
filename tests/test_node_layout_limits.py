"""Where the quantized node layout hands over to fp32 child boxes: scenes too small for its scaled
distances. Host traversal: the layout asked for finds the same hits, hit for hit, at every scale."""
import numpy as np
import pytest

from test_box_test import _trace
from trayracer_gb300.scenes import random_soup


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    O = np.zeros((n, 4), np.float32)
    D = np.zeros((n, 4), np.float32)
    O[:, :3] = rng.uniform(-1.2, 1.2, (n, 3))
    d = rng.normal(size=(n, 3))
    D[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    D[:, 3] = 8.0
    return O, D


@pytest.mark.parametrize("exponent,falls_back", [(0, False), (-20, False), (-31, False), (-40, True), (-50, True)])
def test_small_scenes(exponent, falls_back):
    """The scene and its rays scaled by a power of two."""
    scene = random_soup(3000, seed=5)
    O, D = _rays(20000, 7)
    scale = np.float32(2.0) ** exponent
    scene.positions = scene.positions * scale
    O[:, :3] *= scale
    want, wide = _trace(scene, O, D, 0.0, 0)
    got, counts = _trace(scene, O, D, 0.0, 2)
    assert (want[:, 2] != 0xFFFFFFFF).mean() > 0.3
    assert (got == want).all()
    assert (counts == wide).all() == falls_back

"""The ends of what the quantized node layout's scaled distances take: scenes too small for them (fp32
child boxes serve), directions far from unit length. Host traversal, hit for hit."""
import numpy as np
import pytest

import trayracer_gb300 as tr

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


@pytest.mark.parametrize("any_hit", [0, 1])
@pytest.mark.parametrize("exponent", [-20, 2, 20, 27, 40])
@pytest.mark.parametrize("name", ["soup", "instanced"])
def test_long_and_short_directions(name, exponent, any_hit):
    """Directions scaled by a power of two: the same hits and visits, distances scaled the other way.
    The instances magnify directions by 2^18."""
    scene = random_soup(3000, seed=5)
    O, D = _rays(5000, 9)
    if name == "instanced":
        scene = tr.instanced_cornell()
        scene.instances = [(m, x * np.float32(2.0**-18)) for m, x in scene.instances]
        O[:, :3] *= np.float32(0.7 * 2.0**-18)
    want, counts = _trace(scene, O, D, 0.0, any_hit | 2)
    scale = np.float32(2.0) ** exponent
    D[:, :3] *= scale
    D[:, 3] /= scale
    got, counts2 = _trace(scene, O, D, 0.0, any_hit | 2)
    hit = want[:, 2] != 0xFFFFFFFF
    assert hit.mean() > 0.3
    assert (got[:, :3] == want[:, :3]).all() and (counts == counts2).all()
    assert (got[hit, 3].view(np.float32) * scale == want[hit, 3].view(np.float32)).all()

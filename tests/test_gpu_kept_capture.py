"""Captured frames and sample graphs around tr_update_materials, which keeps them while the lights'
energies stay and drops them when one changes: a replay shows the new materials either way, bit for
bit the image of a renderer that was given them from the start."""
import dataclasses

import numpy as np
import pytest

import trayracer_gb300 as tr

pytestmark = pytest.mark.gpu

W, H = 80, 60


def two_lights():
    """The Cornell box with a second light material: the light's two triangles one each."""
    s = tr.cornell_box(width=W, height=H)
    lit = int(np.argmax(s.materials["emissive"].max(axis=-1)))
    mats = np.concatenate([s.materials, s.materials[lit:lit + 1]])
    mats["emissive"][lit] = (15, 10, 5)
    mats["emissive"][-1] = (3, 5, 7)
    ix = s.material_indices.copy()
    ix[np.where(ix == lit)[0][1]] = len(mats) - 1
    return dataclasses.replace(s, materials=mats, material_indices=ix), lit


def surfaces(s, lit):
    m = s.materials.copy()
    dark = m["emissive"].max(axis=-1) == 0
    m["diffuse"][dark] = np.float32(0.9) * m["diffuse"][dark][:, ::-1]
    m["roughness"][dark] = np.float32(0.6)
    m["closure"][np.where(dark)[0][:3]] = tr.TR_CLOSURE_DISNEY
    return m


def brighter(s, lit):
    m = surfaces(s, lit)
    m["emissive"] = m["emissive"] * np.float32(1.5)
    return m


def swapped(s, lit):
    """The two lights' radiances (of equal areas) exchanged: the energies' sum stays."""
    m = surfaces(s, lit)
    m["emissive"][[lit, -1]] = s.materials["emissive"][[-1, lit]]
    return m


def textured():
    return tr.textured_cornell(width=W, height=H), None


def render(r, how, st):
    r.Reset()
    if how == "samples":
        r.RenderSamples(4 * st.multiSample)
    else:
        for _ in range(2):
            r.RenderFrame(st, use_graph=True)
    assert r.Statistics()["device_error"] == 0
    return r.ColorBuffer().copy()


def renderer(scene, st):
    r = tr.DeviceRenderer(0)
    r.UpdateScene(scene)
    r.SetCamera(scene.camera)
    r.Resize((W, H))
    r.SetSettings(st)
    return r


@pytest.mark.parametrize("how,depth", [("frames", 4), ("frames", 8), ("samples", 5)])  # depth 8: with a tail launch
@pytest.mark.parametrize("make,change", [(two_lights, surfaces), (two_lights, brighter), (two_lights, swapped),
                                         (textured, surfaces)])
def test_replay_shows_the_new_materials(make, change, how, depth):
    scene, lit = make()
    st = tr.KernelSettings(multiSample=2, maxDepth=depth, rrStart=2, seed=5)
    mats = change(scene, lit)
    with renderer(scene, st) as r:
        before = render(r, how, st)
        r.UpdateMaterials(mats)
        after = render(r, how, st)
        r.UpdateMaterials(scene.materials)
        back = render(r, how, st)
    with renderer(dataclasses.replace(scene, materials=mats), st) as r:
        fresh = render(r, how, st)
    assert (after == fresh).all() and (back == before).all()
    assert (after != before).any(axis=-1).mean() > 0.3

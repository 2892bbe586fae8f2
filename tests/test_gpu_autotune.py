"""What tr_autotune times, from a tuning that is none of its candidates: every candidate once."""
import pytest

import trayracer_gb300 as tr

pytestmark = pytest.mark.gpu


def test_every_candidate_is_timed():
    scene = tr.cornell_box(width=64, height=48)
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetCamera(scene.camera)
        r.Resize((64, 48))
        r.SetSettings(tr.KernelSettings(maxDepth=4))
        r.SetTuning(refill_below=5, shade_waves=3)
        # the tuning it starts from; 64-thread traversal and shade blocks; 9 refill thresholds; 1/2 and
        # 3/4 of the extend and of the connect grid; 1, 2, 4 and 8 shade waves; the hit sort
        assert r.Autotune(skip_bvh=True)["trials"] == 1 + 2 + 9 + 4 + 4 + 1

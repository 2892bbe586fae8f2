"""Stage times of an eager frame that are asked for after the frame's buffers were laid out anew."""
import pytest

import trayracer_gb300 as tr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [tr.RenderModes.PathTracing, tr.RenderModes.AmbientOcclusion])
def test_stage_times_outlive_a_resize(mode):
    scene = tr.cornell_box(width=128, height=96)
    names = [f"{k}_time_ms" for k in ("generate", "extend", "shade", "connect", "finalize", "render")]
    with tr.DeviceRenderer(0) as r:
        r.UpdateScene(scene)
        r.SetCamera(scene.camera)
        r.Resize((128, 96))
        r.RenderFrame(tr.KernelSettings(maxDepth=8), mode)
        before = [r.Statistics()[k] for k in names]
        assert before[1] > 0.0 and before[4] > 0.0
        r.Resize((200, 120))
        assert r.Buffers()["capacity"] == 200 * 120
        assert [r.Statistics()[k] for k in names] == before

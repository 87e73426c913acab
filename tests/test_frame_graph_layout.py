"""Frames whose cameras change shape while the path count stays: the captured
frame graph carries the denoiser's batch shapes and pixel offsets, so a frame
after the change must equal a fresh renderer's, with and without a scene
preparation in between that leaves every address and count in place."""
import numpy as np
import pytest

from helpers import pinhole, rig_of
from ray_tracing_gb300 import denoiser, scenes

pytestmark = pytest.mark.gpu

# (width, height) of each camera and samples per pixel, before and after: the same number of paths
LAYOUTS = {
    "turned": (((96, 64),), 1, ((64, 96),), 1),
    "swapped": (((96, 64), (48, 32)), 1, ((48, 32), (96, 64)), 1),
    "merged": (((64, 48), (64, 48)), 1, ((64, 96),), 1),
    "fewer pixels": (((96, 64),), 1, ((48, 32),), 4),
}


def _rig(sizes):
    base = scenes.default_rig("random_spheres", len(sizes))
    cams = []
    for i, (w, h) in enumerate(sizes):
        cam = pinhole(w, h, 80.0)
        cam.rotation[:] = base.cameras[i].rotation[:]
        cam.translation[:] = base.cameras[i].translation[:]
        cams.append(cam)
    return rig_of(*cams)


def _frame(r, rig, spp):
    prof = scenes.profile("balanced", samples_per_pixel=spp, max_bounces=2, enable_denoise=1, enable_restir_di=0)
    r.reset_sequence(7)
    r.render_frame(rig, prof, rig.active_count)
    return [r.download(c).beauty_rgba.copy() for c in range(rig.active_count)]


@pytest.mark.parametrize("change", ["none", "update", "refit"])
@pytest.mark.parametrize("layout", list(LAYOUTS))
def test_denoised_frame_after_a_layout_change(layout, change):
    from ray_tracing_gb300.renderer import Renderer
    sizes0, spp0, sizes1, spp1 = LAYOUTS[layout]
    flat = denoiser.load_weights()
    sc = scenes.HostScene("random_spheres", detail=64)
    with Renderer() as r, Renderer() as fresh:
        r.prepare_scene(sc.view)
        r.set_denoiser(flat)
        for _ in range(2):
            _frame(r, _rig(sizes0), spp0)
        if change == "update":
            sc.view.textures[0].color[0] *= 0.5
        elif change == "refit":
            sc.view.spheres[1].center[1] += 0.25
        r.prepare_scene(sc.view)
        got = _frame(r, _rig(sizes1), spp1)
        fresh.prepare_scene(sc.view)
        fresh.set_denoiser(flat)
        want = _frame(fresh, _rig(sizes1), spp1)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)

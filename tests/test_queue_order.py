"""The wavefront queues at sizes around a warp, a block and the primary rays'
8 x 4-pixel tiles: every path is traced once, whatever order the queues hold it
in, so each path's hit codes and radiance are the oracle's. Tolerance as
test_gpu_parity (identical paths 1e-4 relative; these legacy-material paths
agree bit for bit there)."""
import pytest

from helpers import compare_paths, pinhole, render_both, rig_of
from ray_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,restir", [
    (1, 1, 1, 0), (7, 3, 1, 0), (8, 4, 1, 1), (9, 5, 1, 1), (33, 6, 3, 0), (16, 17, 2, 1), (130, 41, 1, 1),
])
def test_every_path_once_at_odd_sizes(w, h, spp, restir):
    base = scenes.default_rig("random_spheres", 2)
    cams = []
    for i, (cw, ch) in enumerate(((w, h), (max(1, w - 1), h + 2))):
        cam = pinhole(cw, ch, 80.0)
        cam.rotation[:] = base.cameras[i].rotation[:]
        cam.translation[:] = base.cameras[i].translation[:]
        cams.append(cam)
    prof = scenes.profile("balanced", samples_per_pixel=spp, max_bounces=3, enable_denoise=0, enable_restir_di=restir)
    sc, gpu, orc = render_both("random_spheres", rig_of(*cams), prof, frames=2, detail=64)
    for c in range(2):
        gc, gr = gpu.path_records(c, spp, 3)
        oc, orad = orc.path_records(c, spp, 3)
        diverged, max_err, bad = compare_paths(gc, gr, oc, orad, rel=1e-4)
        assert diverged <= 2e-3 and bad == 0, (c, diverged, max_err)
    assert gpu.last_views.primary_rays == sum(c.width * c.height * spp for c in cams)

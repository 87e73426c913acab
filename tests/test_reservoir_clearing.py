"""Frames without ReSTIR leave the reservoir records clear, so the clearing of
a frame's records is left out after them: sequences that turn ReSTIR on and off,
change the resolution and the samples a pixel keep the oracle's paths, and the
records of a frame without ReSTIR hold no reservoir. Tolerance as test_gpu_parity."""
import pytest

from helpers import compare_paths, pinhole, rig_of
from ray_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu

# (ReSTIR, width, height, samples per pixel) of each frame
SEQUENCES = [
    [(1, 40, 24, 1), (0, 40, 24, 1), (1, 40, 24, 1), (1, 40, 24, 1)],
    [(1, 40, 24, 1), (1, 40, 24, 1), (0, 40, 24, 1), (0, 40, 24, 1), (0, 40, 24, 1), (1, 40, 24, 1), (0, 40, 24, 1),
     (1, 40, 24, 1)],
    [(0, 24, 16, 1), (0, 24, 16, 1), (0, 40, 24, 1), (1, 40, 24, 1), (0, 24, 16, 1), (1, 24, 16, 1), (0, 40, 24, 1),
     (1, 40, 24, 1)],
    [(1, 24, 16, 2), (0, 24, 16, 2), (0, 24, 16, 1), (1, 24, 16, 2), (0, 24, 16, 1), (1, 24, 16, 1)],
]


@pytest.mark.parametrize("sequence", SEQUENCES)
def test_restir_switched_between_frames(sequence):
    from oracle.binding import OracleRenderer
    from ray_tracing_gb300.renderer import Renderer
    base = scenes.default_rig("random_spheres", 1).cameras[0]
    sc = scenes.HostScene("random_spheres", detail=64)
    with Renderer(debug_path_records=True) as gpu:
        gpu.prepare_scene(sc.view)
        orc = OracleRenderer(sc.view)
        orc.set_path_records(True)
        for restir, w, h, spp in sequence:
            cam = pinhole(w, h, 80.0)
            cam.rotation[:] = base.rotation[:]
            cam.translation[:] = base.translation[:]
            prof = scenes.profile("balanced", samples_per_pixel=spp, max_bounces=2, enable_denoise=0,
                                  enable_restir_di=restir, restir_initial_candidates=8, restir_min_analytic_lights=8)
            for r in (gpu, orc):
                r.render_frame(rig_of(cam), prof, 1)
            diverged, max_err, bad = compare_paths(*gpu.path_records(0, spp, 2), *orc.path_records(0, spp, 2), rel=1e-4)
            assert diverged <= 2e-3 and bad == 0, (diverged, max_err)
            assert bool(gpu.reservoirs(0)["valid"].any()) == bool(restir)

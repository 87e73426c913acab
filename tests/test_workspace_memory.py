"""Preparation workspaces stay with the handle between scenes of a size and are
given back when a much smaller scene is prepared."""
import numpy as np
import pytest

from helpers import scaled_rig
from ray_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_workspaces_of_a_large_scene_are_given_back():
    torch = pytest.importorskip("torch")
    from ray_tracing_gb300.renderer import Renderer

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    large, small = scenes.HostScene("triangle_terrain", detail=2000000), scenes.HostScene("cornell_box")
    n = large.view.triangle_count
    rig = scaled_rig(scenes.default_rig("cornell_box", 1), 0.25)
    prof = scenes.profile("balanced", samples_per_pixel=1, max_bounces=3, enable_denoise=0, enable_restir_di=0)
    with Renderer() as r, Renderer() as fresh:
        r.prepare_scene(large.view)
        held = free()
        r.prepare_scene(large.view)
        assert free() == held
        r.prepare_scene(small.view)
        # unsorted records and triangle attributes 64 bytes each, the build's scratch about 100; all past the size that stays
        assert free() - held >= 200 * n
        fresh.prepare_scene(small.view)
        for x in (r, fresh):
            x.render_frame(rig, prof, 1)
        assert np.array_equal(r.download(0).beauty_rgba, fresh.download(0).beauty_rgba)

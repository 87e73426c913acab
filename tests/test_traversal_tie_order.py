"""Primitives hit at the same distance: the one traversed first stays, and
sibling nodes are visited by their entry distance however little it differs.
Two coplanar quads cross a camera's one ray at the same t; a second quad beside
each sets its node's box some units in the last place further forward."""
import numpy as np
import pytest

from helpers import pinhole, rig_of
from ray_tracing_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

Z = np.float32(0.75)
ULP = np.float32(2.0 ** -24)


def _scene(left, right):
    tex = (abi.Texture * 1)()
    tex[0].color[:] = (0.5, 0.5, 0.5)
    mat = (abi.Material * 1)()
    mat[0].openpbr_index = -1
    # (origin, edge u, edge v): 0 / 2 cross the ray, 1 / 3 lie beside it and carry the shift, 4 / 5 are far away
    rows = [((-6, -1, Z), 8), ((-6, 1.5, Z - left * ULP), 8), ((-2, -1, Z), 8), ((-2, 1.5, Z - right * ULP), 8),
            ((-6, 99, 10), 8), ((-2, 99, 10), 8)]
    quads = (abi.Quad * len(rows))()
    for q, (origin, width) in zip(quads, rows):
        q.origin[:] = [float(v) for v in origin]
        q.edge_u[:] = (float(width), 0.0, 0.0)
        q.edge_v[:] = (0.0, 2.0, 0.0)
    s = abi.Scene()
    s.textures, s.texture_count = tex, 1
    s.materials, s.material_count = mat, 1
    s.quads, s.quad_count = quads, len(rows)
    return s, (tex, mat, quads)


def test_equal_hits_follow_the_nodes_entry_distance():
    from ray_tracing_gb300.renderer import Renderer
    cam = pinhole(1, 1, 60.0)
    cam.rotation[:] = (1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0)
    cam.translation[:] = (0.0, 0.0, 0.0)
    prof = scenes.profile("balanced", samples_per_pixel=1, max_bounces=1, enable_denoise=0, enable_restir_di=0)
    with Renderer(debug_path_records=True) as r:
        for left in range(6):
            for right in range(6):
                scene, keep = _scene(left, right)
                r.prepare_scene(scene)
                _, order, _ = r.lbvh()
                wide, boxes = r.bvh4()
                inner = [k for k in range(4) if wide[0, k] >= 0]
                assert len(inner) == 2
                near = sorted(inner, key=lambda k: boxes[0, 0, 2, k])[0]  # stable: equal entries keep their order
                leaves = [int(order[~c]) for c in wide[wide[0, near]] if np.iinfo(np.int32).min < c < 0]
                want = [q for q in leaves if q in (0, 2)]
                assert len(want) == 1
                r.render_frame(rig_of(cam), prof, 1)
                codes, _ = r.path_records(0, 1, 1)
                assert int(codes[0, 0]) & 0x0fffffff == want[0], (left, right, boxes[0, 0, 2])

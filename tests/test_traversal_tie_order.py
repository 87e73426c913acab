"""Primitives hit at the same distance: the one traversed first stays, and
sibling nodes are visited by their entry distance however little it differs.
Two coplanar quads cross a camera's one ray at the same t; a second quad beside
each sets its node's box some units in the last place further forward."""
import itertools

import numpy as np
import pytest

from helpers import pinhole, rig_of
from ray_tracing_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

Z = np.float32(0.75)
ULP = np.float32(2.0 ** -24)


def _quads(rows):
    """A scene of (origin, width) quads two high."""
    tex = (abi.Texture * 1)()
    tex[0].color[:] = (0.5, 0.5, 0.5)
    mat = (abi.Material * 1)()
    mat[0].openpbr_index = -1
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


def _scene(left, right):
    # 0 / 2 cross the ray, 1 / 3 lie beside it and carry the shift, 4 / 5 are far away
    return _quads([((-6, -1, Z), 8), ((-6, 1.5, Z - left * ULP), 8), ((-2, -1, Z), 8), ((-2, 1.5, Z - right * ULP), 8),
                   ((-6, 99, 10), 8), ((-2, 99, 10), 8)])


def _four(shifts, crossing):
    """Four pairs side by side, 2 k (crossing the ray, or not) and 2 k + 1 (the
    shift, never), and two quads far off that put the pairs' nodes into one
    node of the wide hierarchy."""
    rows = []
    for k, c in enumerate((-3, -1, 1, 3)):
        half = 5 if crossing >> k & 1 else 0.1
        rows += [((c - half, -1, Z), 2 * half), ((c - 0.1, -1, Z - shifts[k] * ULP), 0.2)]
    return _quads(rows + [((300, -1, Z), 1), ((1000, -1, 1000), 1)])


def _camera():
    cam = pinhole(1, 1, 60.0)
    cam.rotation[:] = (1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0)
    cam.translation[:] = (0.0, 0.0, 0.0)
    return cam


def _hit(r):
    prof = scenes.profile("balanced", samples_per_pixel=1, max_bounces=1, enable_denoise=0, enable_restir_di=0)
    r.render_frame(rig_of(_camera()), prof, 1)
    codes, _ = r.path_records(0, 1, 1)
    return int(codes[0, 0]) & 0x0fffffff


def _leaves(wide, order, node):
    return [int(order[~c]) for c in wide[node] if np.iinfo(np.int32).min < c < 0]


def test_equal_hits_follow_the_nodes_entry_distance():
    from ray_tracing_gb300.renderer import Renderer
    with Renderer(debug_path_records=True) as r:
        for left, right in itertools.product(range(6), range(6)):
            scene, keep = _scene(left, right)
            r.prepare_scene(scene)
            _, order, _ = r.lbvh()
            wide, boxes = r.bvh4()
            inner = [k for k in range(4) if wide[0, k] >= 0]
            assert len(inner) == 2
            near = sorted(inner, key=lambda k: boxes[0, 0, 2, k])[0]  # stable: equal entries keep their order
            want = [q for q in _leaves(wide, order, wide[0, near]) if q in (0, 2)]
            assert len(want) == 1 and _hit(r) == want[0], (left, right, boxes[0, 0, 2])


def test_four_children_in_every_order():
    from ray_tracing_gb300.renderer import Renderer
    with Renderer(debug_path_records=True) as r:
        for shifts in itertools.product(range(3), repeat=4):
            for crossing in range(1, 16):
                scene, keep = _four(shifts, crossing)
                r.prepare_scene(scene)
                _, order, _ = r.lbvh()
                wide, boxes = r.bvh4()
                node = [n for n in range(len(wide)) if (wide[n] >= 0).sum() == 4]
                assert len(node) == 1
                children = sorted(range(4), key=lambda k: boxes[node[0], 0, 2, k])
                visited = [q for k in children for q in _leaves(wide, order, wide[node[0], k])]
                want = [q for q in visited if q % 2 == 0 and crossing >> (q // 2) & 1]
                assert _hit(r) == want[0], (shifts, crossing, boxes[node[0], 0, 2])

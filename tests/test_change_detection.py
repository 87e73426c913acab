"""Scene changes that rtgb_prepare_scene has to see: signs flipped in several
words at once, which cancel in a hash whose high bit never reaches the others."""
import ctypes as C

import numpy as np
import pytest

from ray_tracing_gb300 import scenes

pytestmark = pytest.mark.gpu

REUSE, UPDATE, REFIT = 0, 1, 2


def _words(array, count):
    """An array of ABI structs as its 32-bit words."""
    bytes_ = C.sizeof(array._type_) * count
    return np.frombuffer((C.c_uint32 * (bytes_ // 4)).from_address(C.addressof(array.contents)), np.uint32)


@pytest.mark.parametrize("words", [
    (1, 11),           # center.y of spheres 0 and 2: the high halves of two 64-bit words
    (1, 17, 16),       # a high half, then both halves eight words on
    (3, 13, 23, 33),   # radii
    (21, 121),
])
def test_negated_sphere_words_are_a_change(words):
    from ray_tracing_gb300.renderer import Renderer
    sc = scenes.HostScene("random_spheres", detail=64)
    with Renderer() as r:
        r.prepare_scene(sc.view)
        w = _words(sc.view.spheres, sc.view.sphere_count)
        for k in words:
            w[k] ^= 0x80000000
        r.prepare_scene(sc.view)
        assert r.acceleration_info().update_kind == REFIT
        r.prepare_scene(sc.view)
        assert r.acceleration_info().update_kind == REUSE


@pytest.mark.parametrize("detail", [2000, 80000])  # one thread; four
def test_negated_triangle_corners_are_a_change(detail):
    from ray_tracing_gb300.renderer import Renderer
    sc = scenes.HostScene("triangle_terrain", detail=detail)
    n = sc.view.triangle_count
    with Renderer() as r:
        r.prepare_scene(sc.view)
        w = _words(sc.view.triangles, n)
        for first, second in ((1, 7), (27 * 2 + 1, 27 * (n - 2) + 1), (27 * (n - 2) + 1, 27 * (n - 2) + 7)):
            w[first] ^= 0x80000000
            w[second] ^= 0x80000000
            r.prepare_scene(sc.view)
            assert r.acceleration_info().update_kind == REFIT, (first, second)


def test_negated_colours_are_an_update():
    from ray_tracing_gb300.renderer import Renderer
    sc = scenes.HostScene("random_spheres", detail=64)
    with Renderer() as r:
        r.prepare_scene(sc.view)
        w = _words(sc.view.textures, sc.view.texture_count)
        w[[11, 37]] ^= 0x80000000  # color[1] of textures 0 and 2
        r.prepare_scene(sc.view)
        assert r.acceleration_info().update_kind == UPDATE

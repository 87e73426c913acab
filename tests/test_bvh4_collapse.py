"""The device collapse of the binary hierarchy into the wide BVH against a
sequential restatement (breadth-first, an internal child replaced by its own two
children), word for word, at primitive counts around the collapse's 2048-node
tiles and the smallest hierarchies."""
import ctypes as C

import numpy as np
import pytest

from ray_tracing_gb300 import abi

pytestmark = pytest.mark.gpu


def _spheres(n, seed):
    rng = np.random.default_rng(seed)
    tex = (abi.Texture * 1)()
    tex[0].color[:] = (0.5, 0.5, 0.5)
    mat = (abi.Material * 1)()
    mat[0].openpbr_index = -1
    spheres = (abi.Sphere * n)()
    pos = rng.uniform(-4, 4, (n, 3))
    pos[: n // 3] = pos[0]  # equal Morton codes: the hierarchy splits them by index
    for i in range(n):
        spheres[i].center[:] = pos[i].tolist()
        spheres[i].radius = 0.01
    s = abi.Scene()
    s.textures, s.texture_count = tex, 1
    s.materials, s.material_count = mat, 1
    s.spheres, s.sphere_count = spheres, n
    return s, (tex, mat, spheres)


def _collapse(children):
    source, out = [0], []
    for p in source:
        slots = []
        for c in children[p]:
            slots += [int(g) for g in children[c]] if c >= 0 else [int(c)]
        row = []
        for g in slots:
            if g >= 0:
                source.append(g)
                g = len(source) - 1
            row.append(g)
        out.append(row + [np.iinfo(np.int32).min] * (4 - len(row)))
    return np.array(out, np.int32)


@pytest.mark.parametrize("n", [2, 3, 4, 5, 33, 2048, 2049, 2050, 4097, 9000])
def test_collapse_matches_sequential(n):
    from ray_tracing_gb300.renderer import Renderer
    scene, keep = _spheres(n, n)
    with Renderer() as r:
        r.prepare_scene(scene)
        _, _, children = r.lbvh()
        wide, _ = r.bvh4()
        want = _collapse(children)
        assert r.acceleration_info().wide_node_count == len(want)
        assert np.array_equal(wide, want)

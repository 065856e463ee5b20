"""The 8-wide persistent kernels, whose warps pool their triangle tests: a path's
result must not depend on the rays that share its warp. Paths traced together,
at counts around a warp and a block and where a warp's tests fill several
rounds, against the same paths traced a few at a time. Needs a B200."""
import dataclasses

import numpy as np
import pytest

import gyunity_b200 as g
from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu


def _crowd(count, seed=3):
    """A Cornell box with `count` large random triangles through one another."""
    sd = scenes.cornell_box(res=64, spp=1, spheres=True)
    rng = np.random.default_rng(seed)
    c = rng.uniform(-0.4, 0.4, (count, 1, 3))
    v = (c + rng.normal(scale=0.3, size=(count, 3, 3))).reshape(-1, 3).clip(-0.95, 0.95).astype(np.float32)
    fn = np.cross(v[1::3] - v[0::3], v[2::3] - v[0::3])
    fn /= np.linalg.norm(fn, axis=1, keepdims=True)
    nv = sd.vertices.shape[0]
    idx = (nv + np.arange(3 * count, dtype=np.uint32)).reshape(-1, 3)
    return dataclasses.replace(
        sd, vertices=np.concatenate([sd.vertices, v]),
        normals=np.concatenate([sd.normals, np.repeat(fn, 3, 0).astype(np.float32)]),
        indices=np.concatenate([sd.indices, idx]),
        tri_material=np.concatenate([sd.tri_material, np.zeros(count, np.uint32)]),
        tri_emission=np.concatenate([sd.tri_emission, np.full(count, -1, np.int32)]))


@pytest.mark.parametrize("triangles", [1, 24, 700])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 4096])
def test_paths_do_not_depend_on_their_warp(triangles, n):
    ctx = g.Context(0, capacity=2048, bvh_width=8)
    sc = g.Scene(_crowd(triangles), ctx)
    k = np.arange(n)
    xys = np.stack([(k * 7) % 64, (k * 5 // 3) % 64, k // 64 % 4], 1).astype(np.uint32)
    prm = scenes.RenderParams(4, 8, 3)
    together = sc.trace_paths(xys, params=prm, decisions=True)
    few = [sc.trace_paths(xys[i:i + 1 + i % 19], params=prm, decisions=True) for i in range(0, n, 19 if n > 400 else 1)]
    first = np.concatenate([np.arange(i, min(n, i + 1 + i % 19)) for i in range(0, n, 19 if n > 400 else 1)])
    sc.close()
    ctx.close()
    for whole, parts in zip(together, zip(*few)):
        assert np.array_equal(whole[first], np.concatenate(parts))

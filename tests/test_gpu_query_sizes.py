"""Ray queries around and beyond the number of rays that one pass of
gyt_intersect takes (2^20): the same answers as in small calls, and as before
in a small call that follows. Needs a B200."""
import numpy as np
import pytest

import gyunity_b200 as g
from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu

PASS = 1 << 20


@pytest.fixture(scope="module", params=[2, 8])
def scene(request):
    ctx = g.Context(0, capacity=1024, bvh_width=request.param)
    sc = g.Scene(scenes.mixed_materials_box(level=2), ctx)
    yield sc
    sc.close()
    ctx.close()


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("n", [PASS - 1, PASS, PASS + 1, 2 * PASS + 37])
def test_large_queries_equal_small_ones(scene, n, any_hit):
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    tmax = np.where(rng.uniform(size=n) < 0.3, rng.uniform(0.05, 1.5, n), np.inf)
    rays = np.concatenate([rng.uniform(-0.95, 0.95, (n, 3)), d, tmax[:, None]], 1).astype(np.float32)
    step = 300_000
    parts = [scene.intersect(rays[i:i + step], any_hit=any_hit) for i in range(0, n, step)]
    whole = scene.intersect(rays, any_hit=any_hit)
    after = scene.intersect(rays[-1000:], any_hit=any_hit)
    for w, a, p in zip(whole, after, zip(*parts)):
        p = np.concatenate(p)
        assert w.shape == (n,)
        assert np.array_equal(w, p)
        assert np.array_equal(a, p[-1000:])

"""Device memory that calls leave reserved on their context: as much as the
next call of the kind needs, up to a bound, and no more per path slot of the
adjoint pass than its state takes. Needs a B200."""
import dataclasses

import numpy as np
import pytest
import torch

import gyunity_b200 as g
from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu

BLOCK = 2 << 20        # cudaMalloc takes device memory in blocks of 2 MB
KEPT = 128 << 20       # what a context keeps of each film buffer (include/gyt.h)


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def ctx2():
    """A fresh context, every kernel these tests use loaded by another one."""
    torch.cuda.init()
    warm = g.Context(0, capacity=1024)
    c = g.Context(0, capacity=1024)
    yield warm, c
    c.close()
    warm.close()


def _rays(n):
    rng = np.random.default_rng(1)
    d = rng.normal(size=(n, 3))
    return np.concatenate([rng.uniform(-0.9, 0.9, (n, 3)), d, np.full((n, 1), np.inf)], 1).astype(np.float32)


def test_ray_queries_reserve_what_they_need(ctx2):
    warm, c = ctx2
    sd = scenes.cornell_box(res=16, spp=1)
    g.Scene(sd, warm).intersect(_rays(1))
    sc = g.Scene(sd, c)
    before = _free()
    sc.intersect(_rays(1))
    assert before - _free() <= BLOCK
    sc.intersect(_rays(100_000))
    assert before - _free() <= 100_000 * 44 + BLOCK
    sc.intersect(_rays((1 << 20) + 7))
    held = before - _free()
    assert held <= (1 << 20) * 44 + BLOCK
    sc.intersect(_rays(5))
    assert before - _free() == held
    sc.close()


def test_adjoint_state_per_path_slot():
    torch.cuda.init()
    cap = 1 << 22
    c = g.Context(0, capacity=cap)
    p = scenes.inverse_params(groups=4, seed=1)
    sd = scenes.inverse_box(p, level=3, res=32, spp=2, max_depth=4, rr_depth=4)
    sc = g.Scene(sd, c)
    k = np.arange(200)
    xys = np.stack([k % 32, k // 32, k % 2], 1).astype(np.uint32)
    L = sc.trace_paths(xys)[0]
    warm = g.Context(0, capacity=1024)  # loads the adjoint pass's kernels
    warm.diff_backward_paths(g.Scene(sd, warm), xys, np.ones((200, 3)), L)
    before = _free()
    c.diff_backward_paths(sc, xys, np.ones((200, 3)), L)
    # per slot two copies of the replay state (adjoint weight, primal radiance,
    # pending continuation: 16 + 16 + 8) and the payload of two rays (16 each)
    assert before - _free() <= cap * (2 * 40 + 32) + 8 * BLOCK
    warm.close()
    sc.close()
    c.close()


@pytest.mark.parametrize("call", ["light", "volume", "quantize"])
def test_large_films_are_given_back(ctx2, call):
    warm, c = ctx2

    def run(ctx, res):
        if call == "quantize":
            film = torch.ones(res * res * 4, dtype=torch.float64, device="cuda")
            ctx.film_quantize(film.data_ptr(), res, res)
            del film
            torch.cuda.empty_cache()
            return
        sd = scenes.cornell_box(res=16, spp=1) if call == "light" else scenes.cornell_fog(res=16, spp=1, max_depth=1)
        cam = dataclasses.replace(sd.camera, res_x=res, res_y=res)
        sc = g.Scene(sd, ctx)
        film = g.Film(res, res)
        camera = g.PinHoleCamera(film, cam.pos, cam.look_at, cam.up, cam.fovy, cam.film_distance)
        integrator = g.LightTracing(1, 1) if call == "light" else g.VolPathTracing(1, 1)
        g.Renderer(sc, camera, integrator).Render()
        sc.close()

    run(warm, 16)
    run(c, 16)  # pools
    before = _free()
    run(c, 8000 if call == "quantize" else 3400)
    # the colour sums and the staging buffer (quantize: the latter), each at most the bound
    bound = KEPT if call == "quantize" else 2 * KEPT
    assert before - _free() <= bound
    run(c, 700)
    assert before - _free() <= bound

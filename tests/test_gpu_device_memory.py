"""Device memory that calls leave reserved on their context: as much as the
next call of the kind needs, up to a bound. Needs a B200."""
import numpy as np
import pytest
import torch

import gyunity_b200 as g
from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu

BLOCK = 2 << 20        # cudaMalloc takes device memory in blocks of 2 MB


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

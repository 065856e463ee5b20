"""The shade kernels compiled with and without the environment light: a batch
takes the one its instances need and gives every instance the film of its own
render, with environment lights in none, some or all of them. Needs a B200."""
import dataclasses

import numpy as np
import pytest
import torch

import gyunity_b200 as g
from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampler", ["sobol", "halton"])
@pytest.mark.parametrize("kinds", ["a", "e", "ae", "ea", "aea"])
def test_batch_films_with_and_without_environment(kinds, sampler):
    ctx = g.Context(0, capacity=4096, bvh_width=8)
    descs = [scenes.cornell_box(res=33, spp=3) if k == "a" else scenes.env_knot_small() for k in kinds]
    held = [g.Scene(d, ctx) for d in descs]
    cams = [dataclasses.replace(d.camera, res_x=33 + i, res_y=21) for i, d in enumerate(descs)]
    prms = [scenes.RenderParams(3, 6, 3, sampler) for _ in descs]
    size = [c.res_x * c.res_y * 4 for c in cams]
    single = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in size]
    batch = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in size]
    for s, c, p, f in zip(held, cams, prms, single):
        ctx.render_device(s, c, p, f.data_ptr())
    ctx.render_batch_device(held, cams, prms, [f.data_ptr() for f in batch])
    for a, b in zip(single, batch):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        # the same paths, FP64 sums of at most 12 samples a pixel in another order
        assert np.abs(a - b).max() <= 12 * 2.3e-16 * np.abs(a).max()
        assert a.max() > 0
    for s in held:
        s.close()
    ctx.close()

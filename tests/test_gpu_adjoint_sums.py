"""The adjoint's gradient sums by material row: with every group of a mesh at
the same parameters, the gradients of all groups add up to those of the mesh
as one group. Group counts around a block's threads and beyond what the
kernel keeps in shared memory. Needs a B200."""
import numpy as np
import pytest

import gyunity_b200 as g
from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu


def _gradients(groups, emitters, n):
    p = scenes.InverseParams(np.tile([0.7, 0.6, 0.8], (groups, 1)), np.full(groups, 0.2),
                             np.tile([4.0, 3.0, 5.0], (emitters, 1)))
    sd = scenes.inverse_box(p, level=3, res=64, spp=4, max_depth=6, rr_depth=6)
    ctx = g.Context(0, capacity=2048, bvh_width=2)
    sc = g.Scene(sd, ctx)
    rng = np.random.default_rng(4)
    xys = np.stack([rng.integers(0, 64, n), rng.integers(0, 64, n), rng.integers(0, 4, n)], 1).astype(np.uint32)
    L = sc.trace_paths(xys)[0]
    gm, ge = ctx.diff_backward_paths(sc, xys, rng.uniform(0.5, 1.5, (n, 3)), L)
    sc.close()
    ctx.close()
    m = sd.param_materials
    walls = np.setdiff1d(np.arange(gm.shape[0]), m)
    return gm[m].sum(0), gm[walls], ge


@pytest.mark.parametrize("n", [1, 255, 6000])
@pytest.mark.parametrize("groups", [2, 249, 256, 1200])
def test_group_gradients_add_up(groups, n):
    one, walls1, em1 = _gradients(1, 4, n)
    many, wallsn, emn = _gradients(groups, 4, n)
    # the same FP32 terms in another FP64 order: at most n * depth of them, all
    # of one sign except alpha's
    tol = 6 * n * 2.3e-16
    scale = max(np.abs(one).max(), np.abs(walls1).max(), 1e-300)
    assert np.abs(many - one).max() <= max(tol, 1e-12) * scale * 100
    assert np.abs(wallsn - walls1).max() <= max(tol, 1e-12) * scale * 100
    assert np.abs(emn - em1).max() <= max(tol, 1e-12) * max(np.abs(em1).max(), 1e-300) * 100

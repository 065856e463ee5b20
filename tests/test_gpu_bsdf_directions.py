"""The direction that the MIS half of direct lighting samples on its own is that
of the whole BSDF sample, bit for bit, for every lobe kind; a sample of nonzero
pdf is never called void. Needs a B200."""
import numpy as np
import pytest

from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu

KINDS = [scenes.MAT_DIFFUSE, scenes.MAT_MIRROR, scenes.MAT_GLASS, scenes.MAT_CONDUCTOR, scenes.MAT_DIELECTRIC]


@pytest.mark.parametrize("kind", KINDS)
def test_direction_alone_equals_the_sample(ctx, kind):
    rng = np.random.default_rng(kind)
    n = 400_000
    wo = rng.normal(size=(n, 3))
    wo[::5, 2] *= 1e-3   # grazing, from either side
    wo[::17, 2] = 0.0    # in the surface
    wo[::19] = 0.0, 0.0, 1.0  # along the normal
    wo /= np.linalg.norm(wo, axis=1, keepdims=True)
    u = rng.uniform(size=(n, 3)).astype(np.float32)
    u[::23, 0], u[::29, 1], u[::31, 2] = 0.5, 0.5, 0.0
    u[::37, 1], u[::41, 0] = np.float32(1) - np.float32(2.0 ** -24), 0.0
    p = np.zeros((n, 16), np.float32)
    p[:, 0:6] = rng.uniform(0, 1, (n, 6))
    p[:, 6] = np.exp(rng.uniform(np.log(1e-3), 0, n))
    p[:, 7] = np.where(rng.uniform(size=n) < 0.5, p[:, 6], np.exp(rng.uniform(np.log(1e-3), 0, n)))
    p[:, 8] = rng.uniform(0.5, 2.5, n)      # eta: total internal reflection from either side
    p[:, 9:15] = rng.uniform(0.1, 4.0, (n, 6))
    p[:, 15] = 1.0
    wi, pdf, alone, ok = ctx.bsdf_directions(np.full(n, kind), p, wo, u)
    valid = pdf != 0
    print("kind %d: pdf not 0 %.3f, not void %.3f" % (kind, valid.mean(), ok.mean()))
    assert valid.mean() > 0.4
    assert ok[valid].all()
    assert np.array_equal(wi[valid].view(np.uint32), alone[valid].view(np.uint32))

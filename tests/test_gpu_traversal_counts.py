"""The profile's triangle tests (counting mode) over the 8-wide BVH: a shadow ray
counts the tests up to the one that finds it occluded, whatever its warp tests
beside it. Needs a B200."""
import numpy as np
import pytest
import torch

import gyunity_b200 as g
from gyunity_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("screens", [1, 12, 40])
def test_occluded_shadow_rays_count_to_their_first_hit(screens):
    """A floor seen from below a stack of screens, a light above them: every
    shadow ray meets every screen, so it tests at most the floor's and the
    light's two triangles each and one screen."""
    def quad(y, r):
        return np.array([[-r, y, -r], [r, y, -r], [r, y, r], [-r, y, r]], np.float32)

    screen = np.array([[-60, 0, -40], [60, 0, -40], [0, 0, 80]], np.float32)
    v = np.concatenate([quad(-1.0, 1.0), quad(3.0, 0.2)] +
                       [screen + np.float32([0, 1.0 + k / 64, 0]) for k in range(screens)])
    up, down = [(0, 2, 1), (0, 3, 2)], [(4, 5, 6), (4, 6, 7)]  # the floor, the light
    idx = np.array(up + down + [(8 + 3 * k, 9 + 3 * k, 10 + 3 * k) for k in range(screens)], np.uint32)
    p = np.zeros((1, 16), np.float32)
    p[0, :3] = 0.5
    sd = scenes.SceneDesc(
        vertices=v, indices=idx, tri_material=np.zeros(4 + screens, np.uint32),
        tri_emission=np.array([-1, -1, 0, 0] + [-1] * screens, np.int32),
        mat_type=np.array([scenes.MAT_DIFFUSE], np.uint32), mat_params=p, emission=np.array([[5, 5, 5]], np.float32),
        camera=scenes.Camera(pos=(0.0, 0.5, 0.01), look_at=(0.0, -1.0, 0.0), res_x=64, res_y=64),
        params=scenes.RenderParams(1, 1, 3))
    ctx = g.Context(0, capacity=8192, bvh_width=8)
    sc = g.Scene(sd, ctx)
    film = torch.zeros(64 * 64 * 4, dtype=torch.float64, device="cuda")
    ctx.set_profile(2)
    ctx.render_device(sc, sd.camera, sd.params, film.data_ptr())
    prof = ctx.read_profile()
    rays, tests = prof["rays"]["shadow"], prof["tri_tests"]["shadow"]
    print("%d screens: %d shadow rays, %.2f tests each" % (screens, rays, tests / max(rays, 1)))
    assert rays > 1000
    assert rays <= tests <= 5 * rays
    sc.close()
    ctx.close()

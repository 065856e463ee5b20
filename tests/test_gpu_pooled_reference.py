"""The pooled triangle tests of the 8-wide kernels on a crowd of triangles,
where a warp's tests fill several rounds: all paths in one call against the same
paths in groups of 1 to 33, against the binary BVH's kernels, whose lanes test
their own triangles, and against the oracle's FP64 replay. Needs a B200."""
import numpy as np
import pytest

import gyunity_b200 as g
from gyunity_b200 import scenes
from oracle.port import oracle as orc
from test_gpu_pooled_trace import _crowd

pytestmark = pytest.mark.gpu

N = 4096
PRM = scenes.RenderParams(4, 8, 3)


@pytest.fixture(scope="module")
def crowd():
    sd = _crowd(700)
    k = np.arange(N)
    xys = np.stack([(k * 7) % 64, (k * 5 // 3) % 64, k // 64 % 4], 1).astype(np.uint32)
    ctx = g.Context(0, capacity=2048, bvh_width=8)
    sc = g.Scene(sd, ctx)
    yield sd, sc, xys, sc.trace_paths(xys, params=PRM, decisions=True)
    sc.close()
    ctx.close()


def test_paths_equal_those_of_small_groups(crowd):
    _, sc, xys, whole = crowd
    sizes = [1 + i % 33 for i in range(N)]
    ends = np.cumsum(sizes)
    ends = ends[ends < N].tolist() + [N]
    parts = [sc.trace_paths(xys[a:b], params=PRM, decisions=True) for a, b in zip([0] + ends[:-1], ends)]
    for w, p in zip(whole, zip(*parts)):
        assert np.array_equal(w, np.concatenate(p))


def test_paths_equal_the_binary_kernels(crowd):
    sd, _, xys, whole = crowd
    ctx = g.Context(0, capacity=2048, bvh_width=2)
    sc = g.Scene(sd, ctx)
    other = sc.trace_paths(xys, params=PRM, decisions=True)
    sc.close()
    ctx.close()
    same = np.all([(a == b).reshape(N, -1).all(1) for a, b in zip(whole, other)], axis=0)
    print("paths equal in every output: %.4f" % same.mean())
    # not where a ray meets the shared edge of two triangles exactly, as some do
    # on the walls' diagonals (about 0.4% of these)
    assert same.mean() > 0.99


def test_paths_match_the_fp64_replay(crowd):
    sd, _, xys, (L, cur, rr, occ, mis) = crowd
    Lo, co = orc.OracleScene(sd).paths(xys[:, 0], xys[:, 1], xys[:, 2], params=PRM, precision=64, force_rr=rr,
                                       force_occ=occ, force_mis=mis)
    rel = np.abs(L - Lo).max(1) / np.maximum(np.abs(Lo).max(1), 1e-3)
    print("within 1e-4 of the replay: %.4f, same dimensions: %.4f" % ((rel < 1e-4).mean(), (cur == co).mean()))
    assert (rel < 1e-4).mean() > 0.97

"""GPU: the 4-wide traversal of the binary layout against the counted traversal of its binary nodes (same BVH, same leaf
tests; the closest hit does not depend on the traversal, so every record is equal bit for bit)."""
import numpy as np
import pytest
import torch

from diplodocus_b200 import accel as A
from diplodocus_b200 import scenes as S
from gpu_util import build

pytestmark = pytest.mark.gpu

EMC = A.AccelerationStructureType.kPlocEmc


def check(bvh, rays, **kw):
    rd = torch.from_numpy(np.ascontiguousarray(rays, np.float32)).cuda()
    got = bvh.Intersect(A.Stats(), rd, **kw)
    want = bvh.Intersect(A.Stats(), rd, count=True, **kw)
    any_kw = {k: v for k, v in kw.items() if k != "coherent_order"}
    occ = bvh.IntersectAny(A.Stats(), rd, **any_kw)
    torch.cuda.synchronize()
    bvh.check_errors()
    assert torch.equal(got.raw, want.raw)
    assert torch.equal(occ, want.prim >= 0)
    return want


# one ray, a warp's edges, several rays per warp, the last batch the resident lanes hold (148 SMs x 36 warps x 32) and
# the first that refills lanes, and the sorted order
@pytest.mark.parametrize("n", [1, 31, 33, 5000, 170_496, 170_497, 400_001, (1 << 20) + 5])
@pytest.mark.parametrize("leaf_test", ["ref_mt", "watertight"])
def test_batch_sizes(n, leaf_test):
    bvh = build(S.soup(20_000, seed=7), EMC, split_budget=20)
    h = check(bvh, S.random_rays(n, seed=n), leaf_test=leaf_test, coherent_order=n > (1 << 20))
    if n > 1000:
        assert 0 < int((h.prim >= 0).sum()) < n


# leaves of 1..7 triangles (opened into the node's free slots), trees of a few triangles, roots that are leaves
@pytest.mark.parametrize("leaf", [2, 3, 5, 8])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 9, 33, 3001])
def test_leaf_sizes_and_small_trees(leaf, count):
    tris = S.soup(count, seed=count, mu=-1.5)
    bvh = build(tris, max_triangles_per_leaf=leaf, split_budget=40)
    check(bvh, S.random_rays(3000, seed=leaf), backface_culling=leaf == 3)


@pytest.mark.parametrize("scale,shift", [(1e-6, 0.0), (1e6, 0.0), (1e-3, 1e3), (1.0, -1e5)])
def test_scales_and_offsets(scale, shift):
    """Node frames of very small and large extents, and of extents near the rounding of their coordinates."""
    tris = S.uv_sphere(64, 32, 1.0, displacement=0.1, seed=3) * np.float32(scale) + np.float32(shift)
    rays = S.sphere_inward_rays(20_000, 9)
    rays[:, 0:3] = rays[:, 0:3] * np.float32(scale) + np.float32(shift)
    h = check(build(tris, EMC), rays, leaf_test="watertight")
    assert int((h.prim >= 0).sum()) > 1000


def test_unusual_rays():
    tris = S.soup(2000, seed=5, mu=-2.0)
    rays = S.random_rays(4096, seed=6)
    inf = np.float32(np.inf)
    rays[0:512, 4] = 0.0                        # axis-parallel
    rays[512:640, 4:6] = 0.0
    rays[640:700, 4:7] = 0.0                    # no direction
    rays[700:800, 3] = -0.25                    # hits behind the origin
    rays[800:900, 7] = 0.0                      # empty interval
    rays[900:1000, 7] = inf
    rays[1000:1010, 0] = np.nan
    rays[1010:1020, 5] = np.nan
    rays[1020:1030, 7] = np.nan
    rays[1030:1040, 3] = np.nan
    rays[1040:1050, 1] = inf
    rays[1050:1060, 6] = -inf
    rays[1060:1100, 4:7] *= np.float32(1e-12)   # long parameters
    rays[1100:1140, 4:7] *= np.float32(1e12)
    rays[1140:1142].view(np.uint32)[:, 7] = 0xFFFFFFFF
    for lt in ("ref_mt", "watertight"):
        check(build(tris), rays, leaf_test=lt)


def test_non_finite_triangles():
    tris = S.soup(3000, seed=8, mu=-2.0)
    tris[::7, 1, 2] = np.nan
    tris[1::11, 0, 0] = np.inf
    tris[64:128] = np.nan
    check(build(tris, max_triangles_per_leaf=8), S.random_rays(5000, seed=8))


@pytest.mark.parametrize("count,least", [(20, 1), (60, 41), (180, 105)])
def test_deep_trees(count, least):
    """Nested triangles whose sizes are a geometric progression: each one's nearest neighbour is the next smaller, so the
    global clustering makes a chain, deep enough for each size of the traversal stack."""
    s = (1.25 ** -np.arange(count)[::-1]).astype(np.float32)[:, None]
    tris = np.stack([s * np.float32([0, 0, 0]), s * np.float32([1, 0, 0.25]), s * np.float32([0.25, 1, 1])], axis=1)
    bvh = build(tris, clustering="ploc")
    assert bvh.info().depth >= least, bvh.info().depth
    rays = S.random_rays(4096, seed=1)
    rays[:, 0:3] *= 1.25 ** -(np.arange(4096, dtype=np.float32)[:, None] % count)
    h = check(bvh, rays, leaf_test="watertight")
    assert int((h.prim >= 0).sum()) > 100

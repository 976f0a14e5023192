"""GPU: the uncounted traversals of the 8-wide and the oriented-box layouts against the counted ones of the same nodes (the
closest hit does not depend on the traversal, so every record is equal bit for bit)."""
import numpy as np
import pytest
import torch

from diplodocus_b200 import accel as A
from diplodocus_b200 import scenes as S
from gpu_util import build

pytestmark = pytest.mark.gpu

T = A.AccelerationStructureType
LAYOUTS = {
    "wide": dict(layout="wide8_q8"),
    "sobb6": dict(type_=T.kPlocSobb, kdop_size=6),
    "sobb32": dict(type_=T.kPlocEmcSobb, kdop_size=32),
}


def make(name, tris, **kw):
    kw = {**LAYOUTS[name], **kw}
    return build(tris, kw.pop("type_", T.kPlocEmc), **kw)


def check(bvh, rays, coherent_order=False, **kw):
    rd = torch.from_numpy(np.ascontiguousarray(rays, np.float32)).cuda()
    got = bvh.Intersect(A.Stats(), rd, coherent_order=coherent_order, **kw)
    want = bvh.Intersect(A.Stats(), rd, count=True, coherent_order=coherent_order, **kw)
    occ = bvh.IntersectAny(A.Stats(), rd, **kw)
    torch.cuda.synchronize()
    bvh.check_errors()
    assert torch.equal(got.raw, want.raw)
    assert torch.equal(occ, want.prim >= 0)
    return want


@pytest.mark.parametrize("n", [1, 31, 33, 5000, 170_497, (1 << 20) + 5])
@pytest.mark.parametrize("leaf_test", ["ref_mt", "watertight"])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_batch_sizes(name, n, leaf_test):
    h = check(make(name, S.soup(20_000, seed=7), split_budget=20), S.random_rays(n, seed=n),
              coherent_order=n > (1 << 20), leaf_test=leaf_test)
    if n > 1000:
        assert 0 < int((h.prim >= 0).sum()) < n


@pytest.mark.parametrize("leaf", [2, 4, 5])  # the 8-wide layout takes at most 5
@pytest.mark.parametrize("count", [1, 2, 5, 9, 33, 3001])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_leaf_sizes_and_small_trees(name, leaf, count):
    bvh = make(name, S.soup(count, seed=count, mu=-1.5), max_triangles_per_leaf=leaf, split_budget=40)
    check(bvh, S.random_rays(3000, seed=leaf), backface_culling=leaf == 5)


@pytest.mark.parametrize("scale,shift", [(1e-6, 0.0), (1e6, 0.0), (1e-3, 1e3), (1.0, -1e5)])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_scales_and_offsets(name, scale, shift):
    tris = S.uv_sphere(64, 32, 1.0, displacement=0.1, seed=3) * np.float32(scale) + np.float32(shift)
    rays = S.sphere_inward_rays(20_000, 9)
    rays[:, 0:3] = rays[:, 0:3] * np.float32(scale) + np.float32(shift)
    h = check(make(name, tris), rays, leaf_test="watertight")
    assert int((h.prim >= 0).sum()) > 1000


@pytest.mark.parametrize("name", list(LAYOUTS))
def test_unusual_rays(name):
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
    bvh = make(name, S.soup(2000, seed=5, mu=-2.0))
    for lt in ("ref_mt", "watertight"):
        check(bvh, rays, leaf_test=lt)


@pytest.mark.parametrize("count,least", [(60, 41), (180, 105)])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_deep_trees(name, count, least):
    """Nested triangles whose sizes are a geometric progression: chains that pass the stack entries in shared memory."""
    s = (1.25 ** -np.arange(count)[::-1]).astype(np.float32)[:, None]
    tris = np.stack([s * np.float32([0, 0, 0]), s * np.float32([1, 0, 0.25]), s * np.float32([0.25, 1, 1])], axis=1)
    bvh = make(name, tris, clustering="ploc", type_=T.kPloc if name == "wide" else T.kPlocSobb)
    assert name == "wide" or bvh.info().depth >= least, bvh.info().depth
    rays = S.random_rays(4096, seed=1)
    rays[:, 0:3] *= 1.25 ** -(np.arange(4096, dtype=np.float32)[:, None] % count)
    h = check(bvh, rays, leaf_test="watertight")
    assert int((h.prim >= 0).sum()) > 100


# Closest hits of the binary layout change from pooled to held leaves above 2^19 rays.
@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1])
@pytest.mark.parametrize("leaf", [2, 8])
def test_binary_layout_around_the_pool_limit(n, leaf):
    bvh = build(S.soup(5000, seed=4), T.kPlocEmc, max_triangles_per_leaf=leaf)
    rays = S.random_rays(n, seed=5)
    rays[: n // 4, 3] = -np.inf
    rays[n // 4: n // 2, 3] = -0.5
    h = check(bvh, rays)
    assert 0 < int((h.prim >= 0).sum()) < n


@pytest.mark.parametrize("name", list(LAYOUTS))
def test_unbounded_intervals(name):
    rays = S.random_rays(5000, seed=5)
    rays[:2500, 3] = -np.inf
    rays[1250:, 7] = np.inf
    for lt in ("ref_mt", "watertight"):
        check(make(name, S.soup(5000, seed=4)), rays, leaf_test=lt)

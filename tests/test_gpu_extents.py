"""GPU: scenes and rays near the ends of FP32's range. Every layout's traversal against the brute force over all triangles
and against the counted traversal: quantised nodes and slab distances that overflow may cost visits, never a hit."""
import numpy as np
import pytest
import torch

from diplodocus_b200 import accel as A
from diplodocus_b200 import scenes as S
from gpu_util import build

pytestmark = pytest.mark.gpu

T = A.AccelerationStructureType
LAYOUTS = {
    "binary": dict(),
    "wide": dict(layout="wide8_q8"),
    "sobb": dict(kind=T.kPlocSobb, kdop_size=14),
}
LEAF_TESTS = ("ref_mt", "watertight")


def check(bvh, rays, leaf_test, many=False):
    """`many`: once more with the rays repeated past 2^19, where the binary layout changes its loop."""
    rd = torch.from_numpy(np.ascontiguousarray(rays, np.float32)).cuda()
    want = bvh.Intersect(A.Stats(), rd, leaf_test=leaf_test, count=True)
    got = bvh.Intersect(A.Stats(), rd, leaf_test=leaf_test)
    occ = bvh.IntersectAny(A.Stats(), rd, leaf_test=leaf_test)
    torch.cuda.synchronize()
    bvh.check_errors()
    assert torch.equal(got.raw, want.raw)
    assert torch.equal(occ, want.prim >= 0)
    if many:
        times = (1 << 19) // len(rd) + 1
        got = bvh.Intersect(A.Stats(), rd.repeat(times, 1), leaf_test=leaf_test)
        assert torch.equal(got.raw, want.raw.repeat(times, 1))
    return want


@pytest.mark.parametrize("at", [-1e36, -1e37, -1e38, -3.4e38, 1e36, 3.4e38])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_one_far_vertex(orc, name, axis, at):
    tris = S.uv_sphere(32, 16, 1.0, displacement=0.1, seed=3)
    tris[100, 1, axis] = at
    bvh = build(tris, **LAYOUTS[name])
    rays = S.sphere_inward_rays(3000, 9)
    for k, leaf_test in enumerate(LEAF_TESTS):
        h = check(bvh, rays, leaf_test, many=True)
        truth = orc.brute(tris, rays, leaf_test=k)
        assert int((truth.prim >= 0).sum()) > 100
        np.testing.assert_array_equal(h.prim.cpu().numpy(), truth.prim)


def scattered(count, extent, size, away, seed):
    """Triangles of about `size` anywhere within +-extent, and for each a ray parallel to an axis towards its centroid from
    `away` (towards the positive and the negative end in turn)."""
    g = np.random.default_rng(seed)
    centre = g.uniform(-extent, extent, (count, 1, 3)).astype(np.float32)
    tris = (centre + g.uniform(-size, size, (count, 3, 3)).astype(np.float32)).astype(np.float32)
    c = tris.astype(np.float64).mean(axis=1)
    d = np.zeros((count, 3))
    d[np.arange(count), np.arange(count) % 3] = np.where(np.arange(count) % 2, 1.0, -1.0)
    return tris, S.pack_rays((c - away * d).astype(np.float32), d.astype(np.float32))


@pytest.mark.parametrize("extent,size", [(1e8, 1e4), (3e16, 1e11), (1e18, 1e12)])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_axis_parallel_rays_in_large_scenes(orc, name, extent, size):
    """A ray without a component on an axis has slab distances that overflow in scenes larger than 1e18 steps."""
    tris, rays = scattered(3000, extent, size, 10.0 * size, seed=11)
    bvh = build(tris, **LAYOUTS[name])
    for k, leaf_test in enumerate(LEAF_TESTS):
        h = check(bvh, rays, leaf_test)
        truth = orc.brute(tris, rays, leaf_test=k)
        assert int((truth.prim >= 0).sum()) > 500
        np.testing.assert_array_equal(h.prim.cpu().numpy(), truth.prim)


@pytest.mark.parametrize("name", ["wide", "sobb"])  # the binary layout's reciprocal flushes such directions to zero
def test_long_directions(orc, name):
    """Directions whose reciprocals are subnormal (watertight: products in the other test overflow)."""
    tris, rays = scattered(3000, 1e3, 0.3, 1e3, seed=12)
    rays[:, 4:7] *= np.float32(1.5e38)
    rays[:, 3] = 1e-42
    h = check(build(tris, **LAYOUTS[name]), rays, "watertight")
    truth = orc.brute(tris, rays, leaf_test=1)
    assert int((truth.prim >= 0).sum()) > 500
    np.testing.assert_array_equal(h.prim.cpu().numpy(), truth.prim)


@pytest.mark.parametrize("length", [1e30, 1e33, 1e36])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_short_parameters(orc, name, length):
    """Directions so long that a node's steps are subnormal as distances along the ray, towards the corners of small
    triangles (ref_mt: products of the other test underflow)."""
    tris, _ = scattered(3000, 1e-3, 1e-5, 0.0, seed=13)
    g = np.random.default_rng(14)
    d = g.standard_normal((len(tris), 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    corner = 0.98 * tris[:, 0].astype(np.float64) + 0.02 * tris.astype(np.float64).mean(axis=1)
    rays = S.pack_rays((corner - 0.05 * d).astype(np.float32), (d * length).astype(np.float32), tmin=0.0)
    h = check(build(tris, **LAYOUTS[name]), rays, "ref_mt", many=True)
    truth = orc.brute(tris, rays, leaf_test=0)
    assert int((truth.prim >= 0).sum()) > 1000
    np.testing.assert_array_equal(h.prim.cpu().numpy(), truth.prim)


@pytest.mark.parametrize("split", [10, 40])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_pre_splitting_of_huge_triangles(orc, name, split):
    """Triangles whose area overflows saturate the weights of pre-splitting: more pieces than the budget, and a build."""
    tris = S.uv_sphere(32, 16, 1.0, displacement=0.1, seed=3)
    for k in range(20):
        tris[19 * k, k % 3, :2] = 1e22, -1e22
    assert orc.presplit(tris, split)[0].sum() > len(tris) * (100 + split) // 100
    bvh = build(tris, split_budget=split, **LAYOUTS[name])
    rays = S.sphere_inward_rays(3000, 9)
    h = check(bvh, rays, "watertight", many=True)
    truth = orc.brute(tris, rays, leaf_test=1)
    assert int((truth.prim >= 0).sum()) > 100
    np.testing.assert_array_equal(h.prim.cpu().numpy(), truth.prim)

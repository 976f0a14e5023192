"""GPU: the ends of a ray's interval are exclusive, tmin < t < tmax, in every traversal: rays are traced again with tmax
(or tmin) set to the distance they found, and the records compared with those of the counted traversal and of any-hit."""
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


def scene(count):
    """A soup whose primitive 0 is a large triangle in front of it, so that many rays find primitive 0."""
    tris = S.soup(count, seed=count, mu=-2.0)
    tris[0] = np.float32([[0.4, -1.0, -1.0], [0.5, 2.0, 0.4], [0.6, 0.3, 2.0]])
    return tris


def check(bvh, rays, leaf_test):
    got = bvh.Intersect(A.Stats(), rays, leaf_test=leaf_test)
    want = bvh.Intersect(A.Stats(), rays, leaf_test=leaf_test, count=True)
    occ = bvh.IntersectAny(A.Stats(), rays, leaf_test=leaf_test)
    torch.cuda.synchronize()
    bvh.check_errors()
    assert torch.equal(got.raw, want.raw)
    assert torch.equal(occ, want.prim >= 0)
    return want


# a root that is a leaf, a small tree, a tree; both sides of 2^19 rays, where the binary layout changes its loop
@pytest.mark.parametrize("count", [1, 3, 2000])
@pytest.mark.parametrize("n", [4096, (1 << 19) + 1])
@pytest.mark.parametrize("leaf_test", ["ref_mt", "watertight"])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_interval_ends_are_exclusive(name, leaf_test, n, count):
    bvh = build(scene(count), **LAYOUTS[name])
    rays = torch.from_numpy(S.random_rays(n, seed=count)).cuda()
    first = check(bvh, rays, leaf_test)
    hit = first.prim >= 0
    assert int((first.prim == 0).sum()) > 0
    far = rays.clone()
    far[hit, 7] = first.t[hit]
    again = check(bvh, far, leaf_test)
    assert not bool((again.prim >= 0).any())  # nothing lies nearer than the closest hit
    near = rays.clone()
    near[hit, 3] = first.t[hit]
    again = check(bvh, near, leaf_test)
    assert bool((again.t[hit] > first.t[hit]).all())

"""GPU: trees whose every level leaves siblings with inner nodes of their own on the stack, so that it runs past the entries
in shared memory: the uncounted traversals against the counted one."""
import numpy as np
import pytest
import torch

from diplodocus_b200 import accel as A
from diplodocus_b200 import scenes as S
from gpu_util import build

pytestmark = pytest.mark.gpu

T = A.AccelerationStructureType
GROUP = 4
LAYOUTS = {
    "binary": dict(),
    "wide": dict(layout="wide8_q8"),
    "sobb": dict(kind=T.kPlocSobb, kdop_size=6),
}


def comb(levels, ratio, smallest):
    """Groups of GROUP triangles on a diagonal, each `ratio` times as large and as far out as the one before. A group's
    triangles merge first, then every group with all the smaller ones: a spine with a subtree at every node."""
    g = np.random.default_rng(levels)
    s = smallest * ratio ** np.arange(levels, dtype=np.float64)
    return (s[:, None, None, None] * (1.0 + g.uniform(-0.05, 0.05, (levels, GROUP, 3, 3)))).reshape(-1, 3, 3).astype(np.float32)


def spine(bvh):
    """Nodes of the longest path, and how many of their other children are inner nodes with inner children."""
    _, ch, _ = bvh.download_topology()
    n = len(ch) + 1
    count, height = np.ones(n + len(ch), np.int64), np.zeros(n + len(ch), np.int64)
    for k in range(len(ch)):  # the global clustering makes children before their parents
        count[n + k], height[n + k] = count[ch[k]].sum(), 1 + height[ch[k]].max()
    node, nodes, pending = n + len(ch) - 1, 0, 0
    while node >= n:
        a, b = sorted(ch[node - n], key=lambda c: height[c])
        nodes, pending, node = nodes + 1, pending + int(count[a] >= GROUP), b
    return nodes, pending


# a ray from the small end outwards enters the spine's boxes at once and the groups' after it: all of them are pending when
# the smallest group is reached, 3 entries per two levels of the 4-wide nodes, one group per 7 levels of the 8-wide ones
@pytest.mark.parametrize("levels,ratio,smallest", [(30, 2.1, 1e-8), (45, 2.1, 1e-9), (120, 2.0, 1e-17)])
@pytest.mark.parametrize("leaf_test", ["ref_mt", "watertight"])
@pytest.mark.parametrize("name", list(LAYOUTS))
def test_combs(name, leaf_test, levels, ratio, smallest):
    tris = comb(levels, ratio, smallest)
    bvh = build(tris, clustering="ploc", max_triangles_per_leaf=2, **LAYOUTS[name])
    nodes, pending = spine(bvh)
    assert nodes >= levels and pending >= levels - 2, (nodes, pending)
    g = np.random.default_rng(1)
    # no hits below 1e-9: products of the watertight test turn subnormal there and t has no valid digits
    rays = S.pack_rays(np.zeros((4096, 3)), 1.0 + g.uniform(-0.05, 0.05, (4096, 3)), tmin=1e-9)
    rd = torch.from_numpy(rays).cuda()
    want = bvh.Intersect(A.Stats(), rd, leaf_test=leaf_test, count=True)
    got = bvh.Intersect(A.Stats(), rd, leaf_test=leaf_test)
    occ = bvh.IntersectAny(A.Stats(), rd, leaf_test=leaf_test)
    many = bvh.Intersect(A.Stats(), rd.repeat(129, 1), leaf_test=leaf_test)  # past 2^19 rays
    torch.cuda.synchronize()
    bvh.check_errors()
    assert int((want.prim >= 0).sum()) > 100
    assert torch.equal(got.raw, want.raw)
    assert torch.equal(occ, want.prim >= 0)
    assert torch.equal(many.raw, want.raw.repeat(129, 1))

"""GPU: the hierarchical clustering's block-local part at the borders of its blocks (64 leaves below 2^17 leaves, 512
from there on): topology bit-exact against the sequential restatement, and batches whose meshes end at such borders."""
import numpy as np
import pytest
import torch

import oracle as O
from diplodocus_b200 import accel as A
from diplodocus_b200 import scenes as S
from gpu_util import build

pytestmark = pytest.mark.gpu

EMC = A.AccelerationStructureType.kPlocEmc


def check_topology(orc, tris, kind=A.AccelerationStructureType.kPloc, radius=16):
    bvh = build(tris, kind, nn_search_radius=radius)
    perm, ch, bx = bvh.download_topology()
    codes = orc.emc60(tris) if kind is EMC else orc.morton30(tris)
    exp_perm = O.sort_perm(codes)
    np.testing.assert_array_equal(perm, exp_perm)
    ech, ebx, it = orc.hploc(tris, exp_perm, np.asarray(codes)[exp_perm], radius=radius)
    np.testing.assert_array_equal(ch, ech)
    np.testing.assert_array_equal(bx.view(np.uint32), ebx.view(np.uint32))
    assert bvh.info().ploc_iterations == it


@pytest.mark.parametrize("n", [63, 64, 65, 128, 8193, (1 << 17) - 1, 1 << 17, (1 << 17) + 1, 257 * 512 + 511])
def test_block_borders(orc, n):
    check_topology(orc, S.soup(n, seed=n), EMC if n % 2 else A.AccelerationStructureType.kPloc)


@pytest.mark.parametrize("radius", [1, 15, 17, 32])
def test_large_blocks_radius(orc, radius):
    check_topology(orc, S.soup(140_001, seed=radius), radius=radius)


def test_large_blocks_equal_codes(orc):
    """Runs of equal codes longer than a block: the radix tree over the positions, and ties of the distances."""
    check_topology(orc, np.concatenate([np.repeat(S.soup(3, seed=1), 40_000, axis=0), S.soup(30_000, seed=2)]))


def test_batch_of_meshes_ending_at_block_borders():
    sizes = [512, 1, 511, 2, 1022, 513, 65, 63, 100_000, 31, 40_000]
    meshes = [torch.from_numpy(S.soup(n, seed=n)) for n in sizes]
    assert sum(sizes) > 1 << 17
    for b, m in zip(A.build_batched(A.AccelerationStructureConfig(), meshes), meshes):
        ref = build(m.numpy())
        rays = torch.from_numpy(S.random_rays(2000, seed=len(m))).cuda()
        assert torch.equal(b.Intersect(A.Stats(), rays).raw, ref.Intersect(A.Stats(), rays).raw)
        assert b.sah_cost() == pytest.approx(ref.sah_cost(), rel=1e-9)

"""GPU: what a handle holds is what it reports, and builds that fit under a limit of device memory still do."""
import numpy as np
import pytest
import torch

from diplodocus_b200 import accel as A
from diplodocus_b200 import scenes as S

pytestmark = pytest.mark.gpu

T = A.AccelerationStructureType


def make(tris, kind=T.kPloc, **kw):
    bvh, stats = A.GpuPlocBvh(), A.Stats()
    bvh.Build(A.AccelerationStructureConfig(kind, **kw), stats, tris)
    return bvh, stats


@pytest.mark.parametrize("name,kw,quads", [("binary", {}, True), ("wide", dict(layout="wide8_q8"), False),
                                           ("sobb", dict(kind=T.kPlocSobb), False)])
def test_reported_memory_counts_the_nodes_that_traces_walk(name, kw, quads):
    bvh, stats = make(torch.from_numpy(S.soup(5000, seed=2)), **kw)
    info = bvh.info()
    assert info.quad_nodes == (info.num_inner_nodes if quads else 0)
    assert len(bvh.download_layout()[0]) == info.node_bytes
    assert stats.accel_stats.memory_consumption == info.node_bytes + 64 * info.quad_nodes + info.triangle_bytes

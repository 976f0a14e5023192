"""GPU: what a handle holds is what it reports, and builds that fit under a limit of device memory still do."""
import gc

import numpy as np
import pytest
import torch

from diplodocus_b200 import _lib as L
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


# Device memory in bytes that a build of the 20,000-triangle soup needs without the 4-wide nodes, without rounding and with
# scratch by the count of references (smallest limits that such builds passed under).
NEEDS = {
    "hploc": (7035382, {}),
    "hploc_emc": (7295835, dict(kind=T.kPlocEmc)),
    "ploc": (6795417, dict(clustering="ploc")),
    "ploc_emc": (7055870, dict(kind=T.kPlocEmc, clustering="ploc")),
    "sobb": (13675192, dict(kind=T.kPlocSobb)),
    "sobb_ploc": (13695682, dict(kind=T.kPlocEmcSobb, clustering="ploc")),
    "wide": (10815926, dict(kind=T.kPlocEmc, layout="wide8_q8")),
    "wide_ploc": (10315323, dict(layout="wide8_q8", clustering="ploc")),
    "split40": (9453114, dict(kind=T.kPlocEmc, split_budget=40)),
    "split10_ploc": (7496666, dict(split_budget=10, clustering="ploc")),
    "split40_wide": (13891899, dict(kind=T.kPlocEmc, split_budget=40, layout="wide8_q8")),
    "split40_sobb": (17595839, dict(kind=T.kPlocSobb, split_budget=40)),
}


@pytest.fixture
def limits():
    L.set_limits()
    yield L.set_limits
    L.set_limits()


# A build that has to do without something answers every trace as one that has it: batch sizes on both sides of the resident
# lanes and of 2^20 (the sorted order), both leaf tests, closest and any hits.
@pytest.mark.parametrize("name", list(NEEDS))
def test_builds_fit_where_memory_is_short(limits, name):
    need, kw = NEEDS[name]
    tris = torch.from_numpy(S.soup(20_000, seed=9)).cuda()
    whole, _ = make(tris, **kw)
    whole_quads = whole.info().quad_nodes
    gc.collect()
    torch.cuda.synchronize()
    limits(device_memory_bytes=L.get_limits()[1] + need)
    short, _ = make(tris, **kw)
    limits()
    assert (whole_quads > 0) == (kw.get("layout") is None and kw.get("kind") in (None, T.kPloc, T.kPlocEmc))
    assert short.info().quad_nodes == 0
    rays = torch.from_numpy(S.random_rays((1 << 20) + 5, seed=9)).cuda()
    for n in (1, 33, 5000, 300_001, len(rays)):
        for leaf_test in ("ref_mt", "watertight"):
            r = rays[:n].contiguous()
            want = whole.Intersect(A.Stats(), r, leaf_test=leaf_test)
            got = short.Intersect(A.Stats(), r, leaf_test=leaf_test, coherent_order=True)
            assert torch.equal(got.raw, want.raw)
            assert torch.equal(short.IntersectAny(A.Stats(), r, leaf_test=leaf_test), want.prim >= 0)
    short.check_errors()


@pytest.mark.parametrize("count,least", [(1, 0), (2, 1), (60, 41), (180, 105)])
def test_binary_nodes_without_the_4_wide_ones(limits, count, least):
    """Small trees, and chains deep enough for each size of the stack."""
    s = (1.25 ** -np.arange(count)[::-1]).astype(np.float32)[:, None]
    tris = np.stack([s * np.float32([0, 0, 0]), s * np.float32([1, 0, 0.25]), s * np.float32([0.25, 1, 1])], axis=1)
    tris = torch.from_numpy(tris).cuda()
    whole, _ = make(tris, clustering="ploc")
    assert whole.info().depth >= least
    gc.collect()
    torch.cuda.synchronize()
    base = L.get_limits()[1]
    lo, hi = 0, 1 << 20  # the smallest limit a build passes under
    while hi - lo > 16:
        limits(device_memory_bytes=base + (lo + hi) // 2)
        try:
            make(tris, clustering="ploc")[0].close()
            hi = (lo + hi) // 2
        except L.DiplError as e:
            assert e.status == 3
            lo = (lo + hi) // 2
        torch.cuda.synchronize()
    limits(device_memory_bytes=base + hi)
    short, _ = make(tris, clustering="ploc")
    limits()
    assert short.info().quad_nodes == 0
    rays = S.random_rays(200_000, seed=1)
    rays[:, 0:3] *= 1.25 ** -(np.arange(200_000, dtype=np.float32)[:, None] % count)
    for n in (4096, 200_000):
        for leaf_test in ("ref_mt", "watertight"):
            r = torch.from_numpy(rays[:n]).cuda()
            want = whole.Intersect(A.Stats(), r, leaf_test=leaf_test, count=True)
            assert int((want.prim >= 0).sum()) > 10
            assert torch.equal(short.Intersect(A.Stats(), r, leaf_test=leaf_test).raw, want.raw)
            assert torch.equal(short.IntersectAny(A.Stats(), r, leaf_test=leaf_test), want.prim >= 0)
    short.check_errors()


def test_a_captured_plan_without_the_4_wide_nodes(limits):
    """A plan made where memory is short replays, and its handles are traced through the binary nodes."""
    need, kw = NEEDS["hploc_emc"]
    tris = torch.from_numpy(S.soup(20_000, seed=9)).cuda()
    moved = tris * 0.5 + 0.25
    whole, _ = make(moved, **kw)
    gc.collect()
    torch.cuda.synchronize()
    limits(device_memory_bytes=L.get_limits()[1] + need)
    plan = A.BuildPlan(A.AccelerationStructureConfig(kw["kind"]), [tris])
    limits()
    for mine, new in zip(plan.verts[0], A.soa_vertices(moved)):
        mine.copy_(new)
    plan.launch()
    (short,) = plan.bvhs()
    assert short.info().quad_nodes == 0 and whole.info().quad_nodes > 0
    rays = torch.from_numpy(S.random_rays(50_000, seed=9)).cuda()
    want = whole.Intersect(A.Stats(), rays)
    assert torch.equal(short.Intersect(A.Stats(), rays).raw, want.raw)
    assert torch.equal(short.IntersectAny(A.Stats(), rays), want.prim >= 0)
    short.check_errors()

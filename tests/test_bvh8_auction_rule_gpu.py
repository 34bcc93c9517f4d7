"""Auctions on both sides of the line between eight lanes and one lane per item
(2,000,000 primitives, of a plain build, of a batch, or of a mesh group of
one): canonically the nodes that the stage entry point makes of the same BVH2."""
import numpy as np
import pytest

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S
from tests.test_bvh8_groups_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2_000_000, 2_000_001])
def test_plain(gpu, orc, n):
    check(scenes.uniform_soup(n, seed=2), 30, True, orc)


@pytest.mark.parametrize("total,groups", [(2_000_000, 1), (2_000_001, 1), (4_000_000, 2), (4_000_003, 2)])
def test_batch(gpu, orc, total, groups):
    counts = [50_000, 1, 0, 9, 300, 2, 70_000]
    half = total // groups
    counts += [half - sum(counts)] + [total - half] * (groups - 1)
    prims = scenes.uniform_soup(total, seed=groups)
    batch = nxb.Batch(counts, config=nxb.BuildConfig(prioritize_speed=True, auction=True))
    t = batch.tuning()
    t.fusion_groups = groups
    batch.set_tuning(t)
    meshes = batch.build(S.dev(prims))
    for m, n in enumerate(counts):
        if n < 2:
            continue
        b2 = batch.mesh_bvh2_host(m, meshes)
        want, want_prim, count, _ = S.stage_bvh8(S.dev(b2.view(np.uint8)), n, 1)
        b8, prim = batch.mesh_bvh8_host(m)
        assert len(b8) == count and meshes[m].bvh8_leaf_count == n
        assert orc.compare_bvh8(b8, prim, want, want_prim, n) == 0

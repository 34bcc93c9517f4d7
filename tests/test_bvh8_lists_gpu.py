"""The collapse that reads what every BVH2 node would hold as a BVH8 node from
lists made before (greedy builds of up to 800,000 primitives, and batches of
that many in one group): against the one-lane form, which the stage entry
point runs on the same BVH2, at the edge of the rule, around the widths of a
list and of a CTA, and in a batch cut into groups, which takes no lists."""
import numpy as np
import pytest

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 8, 9, 10, 127, 128, 129, 130, 65_553, 800_000, 800_001])
def test_sizes(gpu, orc, n):
    prims = scenes.uniform_soup(n, seed=n)
    out = nxb.Builder().build(S.dev(prims), nxb.BuildConfig(prioritize_speed=True))
    b8 = S.host(out.nodes.reshape(-1)).view(nxb.BVH8_NODE_DTYPE)
    prim = S.host(out.prim_idx).view(np.uint32)
    want, want_prim, count, leaves = S.stage_bvh8(out.bvh2.nodes.view(-1), n, 0)
    assert out.node_count == count and leaves == n
    assert orc.compare_bvh8(b8, prim, want, want_prim, n) == 0


@pytest.mark.parametrize("groups", [1, 3])
def test_batch(gpu, orc, groups):
    counts = [4000, 1, 0, 2, 128, 129, 9000, 8, 0, 70_000, 3]
    batch = nxb.Batch(counts)
    t = batch.tuning()
    t.fusion_groups = groups
    batch.set_tuning(t)
    meshes = batch.build(S.dev(scenes.batch_meshes(counts, seed=4)))
    for m, n in enumerate(counts):
        if n < 2:
            continue
        want, want_prim, count, _ = S.stage_bvh8(S.dev(batch.mesh_bvh2_host(m, meshes).view(np.uint8)), n, 0)
        b8, prim = batch.mesh_bvh8_host(m)
        assert len(b8) == count
        assert orc.compare_bvh8(b8, prim, want, want_prim, n) == 0

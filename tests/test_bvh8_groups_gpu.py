"""The collapse with eight lanes per item (whole-pipeline builds up to 600,000
primitives, and every auction) against the one-lane form, which the stage
entry point runs on the same BVH2: canonically the same nodes, byte for byte
but the base indices, with the greedy and the auction assignment."""
import numpy as np
import pytest

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu


def check(prims, bits, auction, orc):
    n = prims.shape[0]
    out = nxb.Builder().build(S.dev(prims.astype(np.float32)), nxb.BuildConfig(prioritize_speed=bits == 30, auction=auction))
    b8 = S.host(out.nodes.reshape(-1)).view(nxb.BVH8_NODE_DTYPE)
    prim = S.host(out.prim_idx).view(np.uint32)
    want, want_prim, count, leaves = S.stage_bvh8(out.bvh2.nodes.view(-1), n, 1 if auction else 0)
    assert out.node_count == count and leaves == n
    assert orc.compare_bvh8(b8, prim, want, want_prim, n) == 0


@pytest.mark.parametrize("auction", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 33, 255, 257, 4097, 40_001])
def test_sizes(gpu, orc, n, auction):
    check(scenes.clustered(n, seed=n), 63, auction, orc)


@pytest.mark.parametrize("auction", [False, True])
def test_degenerate_boxes(gpu, orc, auction):
    """Equal, flat and mirrored primitives: costs that tie, with both signs of zero."""
    p = scenes.uniform_soup(3000, seed=3).reshape(-1, 3, 3)
    p[:700] = p[0]
    p[700:1500, :, 2] = -0.0
    p[1500:2000, :, :2] = 0.0
    p[2000:] -= p[2000:].mean()
    check(p.reshape(-1, 9), 30, auction, orc)


@pytest.mark.parametrize("n", [600_000, 600_001])
def test_both_sides_of_the_rule(gpu, orc, n):
    check(scenes.uniform_soup(n, seed=1), 30, False, orc)


@pytest.mark.parametrize("auction", [False, True])
def test_batch(gpu, orc, auction):
    counts = [0, 1, 2, 9, 300, 5000, 0, 64, 20_000]
    prims = scenes.batch_meshes(counts, seed=6)
    batch = nxb.Batch(counts, config=nxb.BuildConfig(prioritize_speed=True, auction=auction))
    meshes = batch.build(S.dev(prims))
    for m, n in enumerate(counts):
        if n < 2:
            continue
        b2 = batch.mesh_bvh2_host(m, meshes)
        want, want_prim, count, _ = S.stage_bvh8(S.dev(b2.view(np.uint8)), n, 1 if auction else 0)
        b8, prim = batch.mesh_bvh8_host(m)
        assert len(b8) == count
        assert orc.compare_bvh8(b8, prim, want, want_prim, n) == 0

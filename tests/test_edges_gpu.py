"""Paths and edges that the sizes of other tests pass by: batches sorted as a
whole (mesh << 32 | code) with every digit width, the smallest H-PLOC tiles and
where they start to grow, and the collapse with eight lanes per item and no
lists, which only mesh groups of up to 600,000 primitives take."""
import ctypes

import numpy as np
import pytest
import torch

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S
from tests.test_batch_gpu import check_against_plain, make_batch
from tests.test_hploc_tiles_gpu import check as check_hploc

pytestmark = pytest.mark.gpu

RNG = np.random.default_rng(17)
# (mesh bits, counts): a mesh above what a cluster sorts, and so many small ones that mesh-by-mesh passes don't pay
WHOLE = {7: [65_537] + [5] * 80, 10: [int(x) for x in RNG.integers(0, 300, 511)] + [65_537] + [int(x) for x in RNG.integers(0, 300, 512)]}


@pytest.mark.parametrize("groups", [1, 3])
@pytest.mark.parametrize("digits", [4, 5, 6, 7, 8])
@pytest.mark.parametrize("mesh_bits", sorted(WHOLE))
def test_batch_sorted_as_a_whole(gpu, orc, mesh_bits, digits, groups):
    counts = WHOLE[mesh_bits]
    prims = make_batch(counts, seed=mesh_bits)
    batch = nxb.Batch(counts)
    t = batch.tuning()
    t.sort_digit_bits, t.fusion_groups = digits, groups
    batch.set_tuning(t)
    info = nxb.CLaunchInfo()
    nxb.check(gpu.nxb_query_batch_launches(batch._handle, ctypes.byref(info)), "launches")
    assert (info.sort_key_bytes, info.sort_passes) == (8, -(-(30 + mesh_bits) // digits))  # 4 to 10 passes, odd and even
    d = S.dev(prims)
    for _ in range(2):  # capture, then replay
        meshes = batch.build(d)
    big = int(np.argmax(counts))
    only = sorted({0, 1, len(counts) - 1, big, *([big - 1] if big else []), *range(2, len(counts), 97)})
    check_against_plain(batch, meshes, prims, counts, orc, only=only)


def tile_edges():
    """The smallest tile has 20 leaves; tiles grow once there is one per resident warp (28 on every SM)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 152
    grow = 20 * 28 * sms
    return [19, 20, 21, 39, 40, 41, grow - 1, grow, grow + 1, grow + 28 * sms + 1]


@pytest.mark.parametrize("radius", [4, 8, 16])
@pytest.mark.parametrize("n", tile_edges())
def test_tile_sizes(gpu, orc, n, radius):
    check_hploc(n, 63 if n % 2 else 30, "random", "soup", radius, orc, n)


def check_group_collapse(prims, counts, groups, orc):
    batch = nxb.Batch(counts)
    t = batch.tuning()
    t.fusion_groups = groups
    batch.set_tuning(t)
    meshes = batch.build(S.dev(prims))
    for m, n in enumerate(counts):
        if n < 2:
            continue
        want, want_prim, count, _ = S.stage_bvh8(S.dev(batch.mesh_bvh2_host(m, meshes).view(np.uint8)), n, 0)
        b8, prim = batch.mesh_bvh8_host(m)
        assert len(b8) == count and meshes[m].bvh8_leaf_count == n
        assert orc.compare_bvh8(b8, prim, want, want_prim, n) == 0


@pytest.mark.parametrize("first,second", [(599_999, 600_000), (600_000, 600_001), (600_001, 600_001)])
def test_groups_at_the_line(gpu, orc, first, second):
    small = [7, 1, 0, 300, 40_000]
    counts = small + [first - sum(small), second]
    check_group_collapse(scenes.uniform_soup(first + second, seed=3), counts, 2, orc)


def test_groups_with_degenerate_boxes(gpu, orc):
    p = scenes.uniform_soup(6000, seed=3).reshape(-1, 3, 3)
    p[:700] = p[0]
    p[700:1500, :, 2] = -0.0
    p[1500:2000, :, :2] = 0.0
    p[2000:] -= p[2000:].mean()
    check_group_collapse(p.reshape(-1, 9), [700, 800, 500, 1000, 3000], 3, orc)

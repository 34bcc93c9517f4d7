"""Batches cut into mesh groups of which the last holds empty meshes only: such
a group has a collapse queue (the empty meshes' items) but nothing to climb.
Each must build like the plain builds of its meshes, and be tunable (autotune
tries groups of its own accord)."""
import pytest

import nexusbvh_gb300 as nxb
from tests import stages as S
from tests.test_batch_gpu import check_against_plain, make_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,groups", [([1000, 0, 0], 2), ([300, 500, 4000, 0], 2), ([300, 500, 4000, 0], 4),
                                           ([300, 500, 4000, 0], 8)])
def test_last_group_without_primitives(gpu, orc, counts, groups):
    prims = make_batch(counts, seed=21)
    d = S.dev(prims)
    batch = nxb.Batch(counts)
    t = batch.tuning()
    t.fusion_groups = groups
    batch.set_tuning(t)
    for _ in range(2):  # capture, then replay
        meshes = batch.build(d)
        check_against_plain(batch, meshes, prims, counts, orc)


@pytest.mark.parametrize("counts", [[1000, 0, 0], [300, 500, 4000, 0]])
def test_autotune(gpu, orc, counts):
    prims = make_batch(counts, seed=22)
    d = S.dev(prims)
    batch = nxb.Batch(counts)
    chosen = batch.autotune(d, repeats=1)
    assert chosen.build_ms > 0
    check_against_plain(batch, batch.build(d), prims, counts, orc)

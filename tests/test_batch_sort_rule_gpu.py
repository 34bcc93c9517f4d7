"""Batches on both sides of the line between the cluster sort and the passes over
all meshes: sizes around the cluster's CTAs (4,096 keys each) and keys per
thread, many small meshes beside one large one, and hundreds of mixed sizes.
Every mesh's trees are those of its plain build."""
import numpy as np
import pytest
import torch

import nexusbvh_gb300 as nxb
from tests import stages as S
from tests.test_batch_gpu import check_against_plain, make_batch

pytestmark = pytest.mark.gpu


def few(counts, how_many=12):
    """Some meshes to compare: the first and last, the largest, and others."""
    big = int(np.argmax(counts))
    near = [m for m in (big - 1, big + 1) if 0 <= m < len(counts)]
    rng = np.random.default_rng(len(counts))
    return sorted({0, len(counts) - 1, big, *near, *(int(x) for x in rng.integers(0, len(counts), how_many))})


def sparse(largest, others, size):
    c = [size] * others
    c.insert(others // 2, largest)
    return c


SPARSE = [(1024, 2300), (1024, 2600), (1025, 1500), (2049, 590), (4096, 590), (4096, 640), (4097, 230), (4097, 260),
          (8193, 120), (8193, 150), (60_000, 8), (60_000, 12), (60_000, 300), (65_536, 400)]


@pytest.mark.parametrize("largest,others", SPARSE)
def test_small_meshes_beside_a_large_one(gpu, orc, largest, others):
    counts = sparse(largest, others, 5)
    prims = make_batch(counts, seed=largest)
    batch = nxb.Batch(counts)
    meshes = batch.build(S.dev(prims))
    check_against_plain(batch, meshes, prims, counts, orc, only=few(counts))


@pytest.mark.parametrize("how_many,largest", [(400, 5000), (300, 60_000), (1300, 1024), (900, 4096)])
def test_mixed_sizes(gpu, orc, how_many, largest):
    rng = np.random.default_rng(largest)
    counts = [int(x) for x in np.exp(rng.uniform(0.0, np.log(largest), how_many))]
    counts[7], counts[11] = 0, largest
    prims = make_batch(counts, seed=3)
    batch = nxb.Batch(counts)
    meshes = batch.build(S.dev(prims))
    check_against_plain(batch, meshes, prims, counts, orc, only=few(counts))


def test_a_large_mesh_does_not_cost_every_other_mesh_its_cluster(gpu):
    """20,000 meshes of 3 primitives, alone and with one of 60,000 among them: a
    60,000-primitive plain build takes less than such a batch, so the two
    differ by a small factor, not by the hundred and more that a 15-CTA
    cluster per mesh takes."""

    def ms(counts):
        prims = S.dev(make_batch(counts, seed=1))
        batch = nxb.Batch(counts)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            batch.build_async(prims)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert ms(sparse(60_000, 20_000, 3)) < 10 * ms([3] * 20_000)

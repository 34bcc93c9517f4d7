"""The pipeline's one-launch sort (up to 65,536 keys of a mesh, in a cluster
of up to 16 CTAs): whole builds against the stage chain, whose sort takes the
onesweep passes, at the sizes where the keys per thread and the cluster
change, on keys that are spread, all equal, few, and already in order.  The
BVH2 depends on every key's place, so equal trees, byte for byte, mean equal
sorts."""
import numpy as np
import pytest

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu


def prims_of(n, kind):
    p = scenes.uniform_soup(n, seed=n)
    if kind == "equal":
        p[:] = p[0]
    elif kind == "few":  # long runs of equal keys, shuffled
        p = p[np.random.default_rng(n).integers(0, max(1, min(n, 37)), n)]
    elif kind == "ordered":
        p = p[np.argsort(p[:, 0])]
    return np.ascontiguousarray(p)


def check(n, bits, kind):
    prims = prims_of(n, kind)
    d_nodes, d_scene = S.stage_bounds(prims)
    d_keys = S.stage_morton(d_nodes, d_scene, n, bits)
    d_sk, d_perm = S.stage_sort(d_keys, n, bits)
    want = S.host(S.stage_hploc(d_sk, d_perm, d_nodes, n, bits))
    got = S.host(S.build_async(prims, bits).bvh2.nodes.view(-1))
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [2, 511, 513, 1023, 1024, 1025, 2049, 16_383, 16_384, 16_385, 30_000, 32_768, 32_769,
                               61_441, 65_535, 65_536, 65_537])
def test_sizes(gpu, n, bits):
    check(n, bits, "spread")


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("kind", ["equal", "few", "ordered"])
def test_key_patterns(gpu, kind, bits):
    for n in (700, 5000, 40_001):
        check(n, bits, kind)


@pytest.mark.parametrize("largest", [1024, 1025, 4096, 4097, 65_536])
def test_batches(gpu, largest):
    counts = [3, 0, largest, 1, 700, min(largest, 2049)]
    prims = scenes.batch_meshes(counts, seed=2)
    batch = nxb.Batch(counts)
    meshes = batch.build(S.dev(prims))
    off = np.concatenate([[0], np.cumsum(counts)])
    for m, n in enumerate(counts):
        if n:
            out = S.build_async(np.ascontiguousarray(prims[off[m]:off[m + 1]]), 30)
            assert batch.mesh_bvh2_host(m, meshes).tobytes() == S.nodes2(out.bvh2.nodes.view(-1)).tobytes()

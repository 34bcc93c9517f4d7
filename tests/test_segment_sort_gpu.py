"""The segmented sort of batches with meshes of more than 65,536 primitives
(four 7-bit passes within each mesh, in tiles of 4,096 keys): every mesh's
BVH2 against a build of that mesh alone, byte for byte, with mesh sizes at
the edges of the tiles, empty meshes, and keys that are spread, all equal or
few."""
import numpy as np
import pytest

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu

COUNTS = {
    "one mesh": [65_537],
    "tile edges": [0, 4095, 1, 4096, 4097, 0, 0, 65_537, 8192, 2, 131_072],
    "edge of the rule": [65_537] + [5] * 41,  # 42 meshes of 1,536 on average
    "past the rule": [65_537] + [5] * 42,     # the passes over mesh and code
    "large": [700_001, 3, 300_000, 0],
}


@pytest.mark.parametrize("kind", ["spread", "equal", "few"])
@pytest.mark.parametrize("case", list(COUNTS))
def test_meshes(gpu, case, kind):
    counts = COUNTS[case]
    prims = scenes.batch_meshes(counts, seed=len(case))
    off = np.concatenate([[0], np.cumsum(counts)])
    for a, b in zip(off[:-1], off[1:]):
        if b > a and kind == "equal":
            prims[a:b] = prims[a]
        elif b > a and kind == "few":
            prims[a:b] = prims[a:b][np.random.default_rng(b).integers(0, min(b - a, 37), b - a)]
    batch = nxb.Batch(counts)
    for _ in range(2):
        meshes = batch.build(S.dev(prims))
    for m, n in enumerate(counts):
        if n:
            out = S.build_async(np.ascontiguousarray(prims[off[m]:off[m + 1]]), 30)
            assert batch.mesh_bvh2_host(m, meshes).tobytes() == S.nodes2(out.bvh2.nodes.view(-1)).tobytes()


@pytest.mark.parametrize("kind", ["spread", "equal", "few"])
@pytest.mark.parametrize("n", [65_537, 69_632, 69_633, 131_071, 1_000_001])
def test_plain_30_bit_builds(gpu, n, kind):
    """The same passes with the whole build as one segment, against the stage
    chain, whose sort takes the onesweep passes over bits [2, 32)."""
    prims = scenes.uniform_soup(n, seed=n)
    if kind == "equal":
        prims[:] = prims[0]
    elif kind == "few":
        prims = prims[np.random.default_rng(n).integers(0, 37, n)]
    prims = np.ascontiguousarray(prims)
    d_nodes, d_scene = S.stage_bounds(prims)
    d_sk, d_perm = S.stage_sort(S.stage_morton(d_nodes, d_scene, n, 30), n, 30)
    want = S.host(S.stage_hploc(d_sk, d_perm, d_nodes, n, 30))
    assert S.host(S.build_async(prims, 30).bvh2.nodes.view(-1)).tobytes() == want.tobytes()

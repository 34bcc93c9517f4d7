"""The H-PLOC stage against the oracle where its tiles can go wrong: sizes
around the smallest tile (32 leaves), around the point where tiles start to
grow with the build (one tile per resident warp) and where they stop (144
leaves), key patterns that leave all, few or no subtrees inside a tile, and
leaf boxes whose areas are infinite, NaN or equal.  Every tree is compared
canonically, boxes bit for bit."""
import numpy as np
import pytest

import nexusbvh_gb300 as nxb
from tests import stages as S

pytestmark = pytest.mark.gpu


def leaves_of(n, rng, kind="soup"):
    lo = rng.random((n, 3)).astype(np.float32)
    hi = (lo + rng.random((n, 3)) * 0.01).astype(np.float32)
    if kind == "equal":
        lo[:], hi[:] = 0.25, 0.5
    elif kind == "nested":  # many ties: one box holds every other
        lo[::7], hi[::7] = 0.0, 2.0
    elif kind == "overflow":  # every area is +inf
        lo, hi = lo * np.float32(1e30) - np.float32(5e29), hi * np.float32(1e30) + np.float32(1e30)
    elif kind == "mixed":  # finite, infinite, NaN and negative areas side by side
        hi[::3] = np.float32(1e30)
        hi[1::5, 0] = np.inf
        lo[1::10, 0] = np.inf
        lo[2::11], hi[2::11] = hi[2::11].copy(), lo[2::11].copy()
    nodes = np.zeros(2 * n - 1, dtype=nxb.BVH2_NODE_DTYPE)
    nodes["bmin"][:n], nodes["bmax"][:n] = lo, hi
    nodes["left"][:n], nodes["right"][:n] = nxb.INVALID_IDX, np.arange(n, dtype=np.uint32)
    return nodes


def keys_of(n, rng, bits, kind):
    top = (1 << bits) - 1
    if kind == "random":
        k = rng.integers(0, top, n, dtype=np.uint64)
    elif kind == "equal":
        k = np.full(n, 12345, dtype=np.uint64)
    elif kind == "runs":  # long runs of equal keys
        k = rng.integers(0, top, max(1, n // 40), dtype=np.uint64)[rng.integers(0, max(1, n // 40), n)]
    else:  # "chains": ranges that grow one leaf at a time, to the right and to the left
        e = rng.integers(0, bits - 16, n)
        k = (rng.integers(0, 1 << 12, n).astype(np.uint64) << np.uint64(bits - 13)) + (np.uint64(1) << e.astype(np.uint64))
    k = np.sort(k)
    return k.astype(np.uint32) if bits == 30 else k


def check(n, bits, key_kind, leaf_kind, radius, orc, seed):
    rng = np.random.default_rng(seed)
    nodes = leaves_of(n, rng, leaf_kind)
    keys = keys_of(n, rng, bits, key_kind)
    perm = rng.permutation(n).astype(np.uint32)
    got = S.nodes2(S.stage_hploc(S.dev(keys.view(np.int32 if bits == 30 else np.int64)), S.dev(perm.view(np.int32)),
                                 S.dev(nodes.view(np.uint8)), n, bits, radius))
    want, root, err = orc.hploc(keys, perm, nodes[:n], radius)
    assert err == 0
    assert orc.compare_bvh2(got, 2 * n - 2, want, root, n) == 0


@pytest.mark.parametrize("n", [2, 16, 17, 31, 32, 33, 63, 64, 65, 1023, 136_191, 136_193, 200_001, 612_865])
def test_tile_sizes(gpu, orc, n):
    check(n, 63 if n % 2 else 30, "random", "soup", 8, orc, n)


@pytest.mark.parametrize("key_kind", ["equal", "runs", "chains"])
@pytest.mark.parametrize("radius", [4, 8, 16])
def test_key_patterns(gpu, orc, key_kind, radius):
    for n, bits in ((5000, 63), (150_001, 30)):
        check(n, bits, key_kind, "soup", radius, orc, radius + n)


@pytest.mark.parametrize("leaf_kind", ["equal", "nested", "overflow", "mixed"])
@pytest.mark.parametrize("radius", [4, 8, 16])
def test_boxes_without_a_finite_neighbour(gpu, orc, leaf_kind, radius):
    check(3001, 63, "random", leaf_kind, radius, orc, radius)


def test_batch_tiles_over_many_meshes(gpu, orc):
    """Tiles of 144 leaves over meshes of 1 to 300 primitives: most hold
    several whole meshes and the ends of two more."""
    rng = np.random.default_rng(9)
    counts = rng.integers(0, 301, 4400)
    from nexusbvh_gb300 import scenes
    total = int(counts.sum())
    assert total > 612_864
    prims = np.ascontiguousarray(scenes.uniform_soup(total, seed=4))
    batch = nxb.Batch(counts)
    meshes = batch.build(S.dev(prims))
    off = np.concatenate([[0], np.cumsum(counts)])
    for m in range(0, len(counts), 97):
        n = int(counts[m])
        if n < 1:
            continue
        out = S.build_async(prims[off[m]:off[m + 1]], 30)
        assert batch.mesh_bvh2_host(m, meshes).tobytes() == S.nodes2(out.bvh2.nodes.view(-1))[:2 * n - 1].tobytes()

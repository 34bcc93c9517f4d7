"""Stages that are set up while the one before still runs (plain builds of up
to 1,000,000 primitives): builds of different inputs queued one after another
in one workspace, and captured in a graph, give the trees of builds that run
alone."""
import ctypes

import pytest
import torch

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu


def tree(bvh2, bvh8, prim_idx, result, n):
    r = nxb.CResult.from_buffer_copy(result.cpu().numpy().tobytes())
    assert r.error_word == 0 and r.bvh8_leaf_count == n
    return bvh2.cpu().numpy()[:(2 * n - 1) * 32].tobytes(), r.bvh8_node_count


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("sizes", [(1021, 2, 700), (70_000, 65_536, 1), (1_000_000, 900, 1_000_001)])
def test_queued_builds(gpu, sizes, captured):
    cfg = nxb.BuildConfig(prioritize_speed=True)
    b = nxb.Builder()
    most = max(sizes)
    ws = torch.empty(b.sizes(most, cfg).workspace_bytes, dtype=torch.uint8, device="cuda")
    outs = []
    for k, n in enumerate(sizes):
        sz = b.sizes(n, cfg)
        outs.append((S.dev(scenes.uniform_soup(n, seed=k)), n,
                     torch.empty(sz.bvh2_node_count * 32, dtype=torch.uint8, device="cuda"),
                     torch.empty(sz.bvh8_node_capacity * 80, dtype=torch.uint8, device="cuda"),
                     torch.empty(n, dtype=torch.int32, device="cuda"),
                     torch.empty(ctypes.sizeof(nxb.CResult), dtype=torch.uint8, device="cuda")))

    def queue():
        for prims, n, b2, b8, pi, res in outs:
            b.enqueue(prims, n, cfg, ws, b2, b8, pi, res)

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        queue()
        if captured:
            stream.synchronize()
            for o in outs:
                o[2].zero_()
            stream.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                queue()
            g.replay()
    stream.synchronize()
    for prims, n, b2, b8, pi, res in outs:
        alone = nxb.Builder().build(prims, cfg)
        assert tree(b2, b8, pi, res, n) == (S.host(alone.bvh2.nodes.reshape(-1)).tobytes(), alone.node_count)

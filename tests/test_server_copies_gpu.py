"""The server's gather of device inputs and scatter of results, beside the
copies of host inputs: requests of one primitive up, inputs that start on odd
words, triangles and boxes, in the batches that form behind a large build."""
import numpy as np
import pytest

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [9, 6])
def test_inputs(gpu, orc, width):
    counts = [1, 2, 3, 255, 257, 1023, 1025, 4097, 30_001, 1]
    soup = scenes.uniform_soup(sum(counts), seed=width)
    flat = S.dev(soup if width == 9 else scenes.to_boxes(soup)).reshape(-1)
    srv = nxb.Server(streams=1)
    cfg = nxb.BuildConfig(prioritize_speed=True)
    tickets = [srv.submit(scenes.clustered(1_000_000, seed=3), cfg)]
    inputs, at = [], 0
    for k, n in enumerate(counts):
        p = flat[at:at + n * width].view(n, width)  # starts on any word
        at += n * width
        inputs.append(p)
        tickets.append(srv.submit(p.cpu().numpy() if k % 4 == 3 else p, cfg))
    batched = 0
    for t, p in zip(tickets, [None] + inputs):
        r = srv.wait(t)
        if p is not None:
            out = nxb.Builder().build(p.clone(), cfg)
            b8, prim = nxb.Server.bvh8_host(r)
            want = S.host(out.nodes.reshape(-1)).view(nxb.BVH8_NODE_DTYPE)
            assert len(b8) == out.node_count
            assert orc.compare_bvh8(b8, prim, want, S.host(out.prim_idx).view(np.uint32), p.shape[0]) == 0
            batched += r.batched_with > 1
        srv.release(t)
    assert batched >= 2
    srv.close()

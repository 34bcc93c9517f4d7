"""The launch counts that reports are made from: those of a plain build against
the kernel nodes of its capture, and those of a batch's ways of sorting."""
import ctypes

import pytest
import torch

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu


def captured_kernels(enqueue):
    """Kernel nodes of what enqueue(stream) launches."""
    rt = ctypes.CDLL("libcudart.so.%s" % torch.version.cuda.split(".")[0])
    stream = torch.cuda.Stream()
    s, graph, count, kind = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t(), ctypes.c_int()
    assert rt.cudaStreamBeginCapture(s, 2) == 0  # relaxed
    try:
        enqueue(stream)
    finally:
        assert rt.cudaStreamEndCapture(s, ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(count)) == 0
    kernels = 0
    for node in nodes:
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kernels += kind.value == 0
    assert rt.cudaGraphDestroy(graph) == 0
    return kernels


@pytest.mark.parametrize("wide", [True, False])
@pytest.mark.parametrize("auction", [False, True])
@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [1, 1000, 65_536, 65_537, 800_000, 800_001])
def test_plain(gpu, n, bits, auction, wide):
    config = nxb.BuildConfig(prioritize_speed=bits == 30, auction=auction)
    b = nxb.Builder()
    z = b.sizes(n, config)
    prims = S.dev(scenes.uniform_soup(n, seed=1))
    ws = b.workspace(z.workspace_bytes)
    bvh2 = torch.empty((z.bvh2_node_count, 32), dtype=torch.uint8, device="cuda")
    bvh8 = torch.empty((z.bvh8_node_capacity, 80), dtype=torch.uint8, device="cuda") if wide else None
    idx = torch.empty(n, dtype=torch.int32, device="cuda") if wide else None
    result = torch.empty(64, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    info, c = nxb.CLaunchInfo(), config.to_c()
    nxb.check(gpu.nxb_query_build_launches(n, ctypes.byref(c), int(wide), ctypes.byref(info)), "launches")
    got = captured_kernels(lambda s: b.enqueue(prims, n, config, ws, bvh2, bvh8, idx, result, s))
    assert info.kernels == got


@pytest.mark.parametrize("counts,groups,want", [
    ([900, 0, 4000, 33], 1, (8, 4, 4)),         # begin, bounds, Morton, clusters, H-PLOC, lists, collapse, finalize
    ([900, 0, 4000, 33], 2, (9, 4, 4)),         # no lists, but H-PLOC and a collapse per group
    ([1000, 0, 0], 2, (8, 4, 4)),               # nothing to climb in the second
    ([500_000, 300_001], 1, (11, 4, 4)),        # a list of tiles and four passes; too large for lists
    ([65_537] + [5] * 80, 1, (12, 5, 8)),       # 37 bits in digits of 8
])
def test_batch(gpu, counts, groups, want):
    batch = nxb.Batch(counts)
    t = batch.tuning()
    t.fusion_groups = groups
    batch.set_tuning(t)
    info = nxb.CLaunchInfo()
    nxb.check(gpu.nxb_query_batch_launches(batch._handle, ctypes.byref(info)), "launches")
    assert (info.kernels, info.sort_passes, info.sort_key_bytes) == want

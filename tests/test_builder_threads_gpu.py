"""One Builder shared by two threads: each build returns its own result, also
when the other thread's build finishes between this one's wait and its read."""
import threading

import pytest
import torch

import nexusbvh_gb300 as nxb
from nexusbvh_gb300 import scenes
from tests import stages as S

pytestmark = pytest.mark.gpu


class _Stream:
    """A stream whose synchronize also waits for the other thread's."""

    def __init__(self, stream, meet):
        self._stream, self._meet = stream, meet

    def __getattr__(self, name):
        return getattr(self._stream, name)

    def synchronize(self):
        self._stream.synchronize()
        self._meet.wait(60)


def test_each_thread_reads_its_own_result(gpu, monkeypatch):
    prims = [S.dev(scenes.uniform_soup(n, seed=n)) for n in (3000, 5000)]
    builder = nxb.Builder()
    config = nxb.BuildConfig(prioritize_speed=True)
    builder.workspace(max(builder.sizes(p.shape[0], config).workspace_bytes for p in prims))
    want = [builder.build(p, config) for p in prims]
    meet = threading.Barrier(2)
    real = torch.cuda.current_stream
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: _Stream(real(*a), meet))
    got = [None, None]

    def work(k):
        got[k] = builder.build(prims[k], config)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    for w, g in zip(want, got):
        assert g is not None
        assert (g.node_count, g.bounds) == (w.node_count, w.bounds)
        assert torch.equal(g.bvh2.nodes, w.bvh2.nodes)

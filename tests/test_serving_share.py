"""Which launches of the server may take the GPU's idle lanes (host logic, no
GPU): none while another batch is in flight, be it a whole main trace, a
window of one or the pseudo-lines; and whole batches of large requests leave
block slots to small ones."""
import contextlib
import types

import pytest
import torch

from fastqsl_gb300 import serving


class Stream:
    def wait_event(self, ev):
        pass


class Event:
    def record(self, stream):
        pass

    def query(self):
        return False


class Batch:
    """Stands for PlaneQBatch: keeps the launches asked of it."""
    log = []
    caps = []

    def __init__(self, jobs, device, tile, stream, blocks_per_sm):
        Batch.caps.append(blocks_per_sm)
        self.main_lines = sum(j["n0"] * j["n1"] * j["nplanes"] for j in jobs)

    def run_main(self, stream=None, lo=0, hi=-1, share=False):
        Batch.log.append(("main", lo, hi, share))

    def run_post(self, stream=None, share=False):
        Batch.log.append(("post", share))
        return []


@pytest.fixture
def server(monkeypatch):
    cuda = types.SimpleNamespace(Stream=lambda device=None, priority=0: Stream(), Event=Event,
                                 stream=lambda s: contextlib.nullcontext())
    empty = lambda n, dtype=None, pin_memory=False: torch.empty(n, dtype=dtype)  # noqa: E731
    monkeypatch.setattr(serving, "torch", types.SimpleNamespace(cuda=cuda, device=torch.device, empty=empty,
                                                                float64=torch.float64))
    monkeypatch.setattr(serving, "api", types.SimpleNamespace(PlaneQBatch=Batch))
    Batch.log, Batch.caps = [], []
    return serving.QServer({"f": object()}, classes=((600, 1, 4), (float("inf"), 1, 2)), chunk_lines=1024,
                           max_chunks=8, chunks_when_interactive=8)


def _request(rid, n):
    return serving.QRequest(rid=rid, field="f", n0=n, n1=n)


def test_alone_a_batch_may_take_every_lane(server):
    server.submit(_request(0, 50))
    server.step()
    assert Batch.log == [("main", 0, 1024, False), ("main", 1024, 2048, False), ("main", 2048, 2500, False),
                         ("post", False)]


def test_beside_another_batch_no_launch_takes_spare_lanes(server):
    server.submit(_request(0, 20))
    server.step()
    assert Batch.log == [("main", 0, -1, False), ("post", False)]
    Batch.log.clear()
    server.submit(_request(1, 50))
    server.step()
    assert Batch.log == [("main", 0, 1024, True), ("main", 1024, 2048, True), ("main", 2048, 2500, True),
                         ("post", True)]


def test_large_whole_batches_leave_block_slots(server):
    from fastqsl_gb300 import api
    server.chunk_lines = 0
    server.submit(_request(0, 20))
    server.submit(_request(1, 50))
    server.step()
    small, large = Batch.caps
    assert small == 0 and 0 < large < api.BATCH_BLOCKS_PER_SM

"""The one-launch form of a compiled matvec is built on first use: a replay on another stream
waits for the tables and the barrier that the building stream uploads."""

import pytest
import torch

from tenet import _exec, _lib
from tenet.program import heff2_program

pytestmark = pytest.mark.gpu


def test_fused_replay_waits_for_the_stream_that_built_it(monkeypatch):
    import bench

    *operands, aa = bench.build_workload()
    prog = heff2_program(*operands, aa.structure, defer=False)
    want, got = (torch.full_like(prog.y_slot, float("nan")) for _ in range(2))
    prog.run(aa.arena, want)
    torch.cuda.synchronize()
    built, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(built):
        torch.cuda._sleep(200_000_000)  # (about 0.1 s: the uploads queue behind it)
        assert prog.fused is not None
    assert not built.query()
    monkeypatch.setattr(_exec, "FUSE", True)
    with torch.cuda.stream(other):
        prog.run(aa.arena, got)
        done = torch.cuda.Event()
        done.record()
    done.synchronize()
    assert built.query()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and int(prog.barrier[0]) == 0 and _lib.device_error(0) == 0


def test_a_capture_that_comes_first_takes_the_launches(monkeypatch):
    import bench

    *operands, aa = bench.build_workload()
    prog = heff2_program(*operands, aa.structure, defer=False)
    want, got = (torch.full_like(prog.y_slot, float("nan")) for _ in range(2))
    prog.run(aa.arena, want)
    torch.cuda.synchronize()
    monkeypatch.setattr(_exec, "FUSE", True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        prog.run(aa.arena, got)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    got.fill_(float("nan"))
    prog.run(aa.arena, got)
    torch.cuda.synchronize()
    assert torch.equal(got, want) and len(prog.fused) == 1


def test_another_threads_recording_keeps_its_form():
    import threading

    seen = []
    with _exec.standard_gathers():
        th = threading.Thread(target=lambda: seen.append(_exec.standard()))
        th.start()
        th.join()
        assert _exec.standard() and seen == [False]
    assert not _exec.standard()

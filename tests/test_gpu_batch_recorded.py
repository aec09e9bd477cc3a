"""``batch.BatchedHeff2`` from its recorded launches: the same bits as launch by launch, on any
input and output buffers, on another stream, under a launch log and inside a CUDA graph."""
import pytest
import torch

from tenet import _exec, batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, precision, defer, recorded", [
    (1, "f64", False, True), (3, "f64", False, True), (3, "f64", True, True),
    (3, "tf32", False, False), (40, "f64", False, True), (40, "f64", False, False)])
def test_recorded_launches_give_the_same_bits(n, precision, defer, recorded, monkeypatch):
    import bench

    if n == 40:  # either side of the size rule
        monkeypatch.setattr(batch, "RECORD_MAX_TILES", 1 << 30 if recorded else 1)

    members = [bench.build_workload(seed=10 * k) for k in range(min(n, 3))]
    fl, w1, w2, fr, aa = (batch.TensorBatch.stack([members[k % 3][i] for k in range(n)])
                          for i in range(5))
    w1, w2 = (batch.TensorBatch.broadcast(members[0][i], n) for i in (1, 2))
    prog = batch.BatchedHeff2(fl, w1, w2, fr, aa.structure, precision=precision, defer=defer,
                              tc_min_flops=1 if precision != "f64" else None)
    assert (prog._seq is not None) == recorded
    want = torch.full((n, prog.out_size), float("nan"), dtype=torch.float64, device="cuda")
    prog._launch(aa.arena.reshape(-1), want.reshape(-1))
    got = torch.full_like(want, float("nan"))
    prog.run(aa.arena, got)
    assert torch.equal(got, want) and not torch.isnan(got).any()

    side = torch.cuda.Stream()
    again = torch.empty_like(want)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # other buffers, another stream
        prog.run(aa.arena.clone(), again)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(again, want)
    with _exec.LaunchLog() as log:
        prog.run(aa.arena, again.zero_())
    assert torch.equal(again, want) and log.count > 1

    x, y = aa.arena.clone(), torch.empty_like(want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        prog.run(x, y)
    x.neg_()
    g.replay()
    assert torch.equal(y, -want)

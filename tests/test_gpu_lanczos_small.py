"""The one-launch Lanczos solve of a small problem (``tnb_lanczos_small.cu``) against the same
call launch by launch: the Krylov vectors, the recurrence's words and the residual, bit for bit,
at the smallest and largest vectors it takes, past the size rule, for a single step and through
breakdowns of the recurrence.  A row outside its buffers sets the error word and is left out."""
import numpy as np
import pytest
import torch

from tenet import _exec, _lib, network
from tenet.program import heff2_program
from tenet.structure import IN, OUT, Leg, TensorStructure, layout
from tenet.symmetry import SU2
from tenet.tensor import SymmetricTensor

pytestmark = pytest.mark.gpu


def chain(bond):
    """The two-site matvec of an SU(2) chain with these multiplets on its bonds."""
    from tenet import GradedSpace

    def space(d):
        return GradedSpace.new(SU2, {SU2.sector(j): k for j, k in d.items()})

    B, M, P = space(bond), space({0: 2, 2: 1}), space({1: 1})
    fl = TensorStructure((Leg(B, IN), Leg(M, OUT, True), Leg(B, OUT)))
    w = TensorStructure((Leg(M, IN, True), Leg(P, OUT), Leg(P, IN), Leg(M, OUT, True)))
    fr = TensorStructure((Leg(B, OUT), Leg(M, IN, True), Leg(B, IN)))
    aa = TensorStructure((Leg(B, OUT), Leg(P, OUT), Leg(P, OUT), Leg(B, IN)))
    g = torch.Generator(device="cuda").manual_seed(3)

    def draw(s):
        return SymmetricTensor(s, arena=torch.randn(layout(s).size, dtype=torch.float64,
                                                    device="cuda", generator=g))

    return heff2_program(draw(fl), draw(w), draw(w), draw(fr), aa), draw(aa).arena


def solve(prog, seq, x, ncv, tol):
    dl = network.DeviceLanczos(prog, ncv, tol)
    old, prog.seq = prog.seq, seq
    try:
        dl.launch(x)
        torch.cuda.synchronize()
    finally:
        prog.seq = old
    return [t.cpu().numpy() for t in (dl.V, dl.state, dl.scal[:1], dl.W)]


@pytest.mark.parametrize("bond", [
    {0: 1}, {0: 1, 2: 1}, {0: 2, 2: 2, 4: 1}, {1: 3, 3: 4, 5: 1}, {0: 4, 2: 6, 4: 3, 6: 1},
    {0: 6, 2: 9, 4: 4, 6: 1}, {0: 7, 2: 11, 4: 5, 6: 1}, {0: 8, 2: 12, 4: 5, 6: 1}])
@pytest.mark.parametrize("ncv, tol", [(1, 1e-13), (12, 1e-13), (12, 1e6)])
def test_one_launch_gives_the_same_bits(bond, ncv, tol):
    prog, x = chain(bond)
    one = torch.ones(1, dtype=torch.float64, device="cuda")
    sink = torch.empty(1, dtype=torch.float64, device="cuda")
    table = _exec.make_gemm([(1, 1, 1, 0, 1, 0, 1, 0, 1)], _exec.TILE_32)
    launched = _exec.Seq()  # the same stages behind more than a small solve takes
    with launched:
        for _ in range(13):
            table.run(one, one, sink)
        prog._run_tables(prog.x_slot, prog.y_slot)
    sink.zero_()
    got = solve(prog, prog.seq, x, ncv, tol)
    assert float(sink[0]) == 0.0
    want = solve(prog, launched, x, ncv, tol)
    assert float(sink[0]) == 1.0
    for a, b in zip(got, want):
        assert np.isfinite(a).all() and np.array_equal(a, b)
    assert _lib.device_error(0) == 0


def test_a_row_outside_its_buffers_is_refused():
    x = torch.arange(1.0, 5.0, dtype=torch.float64, device="cuda")
    slots = [torch.zeros(4, dtype=torch.float64, device="cuda") for _ in range(2)]
    a = torch.eye(4, dtype=torch.float64, device="cuda").reshape(-1).contiguous()
    run_start = torch.tensor([0, 4], dtype=torch.int64, device="cuda")
    run_w = torch.ones(1, dtype=torch.float64, device="cuda")
    for row, good in (((1, 4, 4, 0, 4, 0, 4, 0, 4), True), ((1, 4, 4, 0, 4, 4, 4, 0, 4), False),
                      ((1, 4, 4, 0, 4, 0, 4, 1, 4), False), ((1, 4, 5, 0, 5, 0, 4, 0, 4), False)):
        table = _exec.make_gemm([row], _exec.TILE_32)
        seq = _exec.Seq()
        with seq:
            table.run(slots[0], a, slots[1])
        ncv = 3
        V = torch.full((ncv + 1, 4), float("nan"), dtype=torch.float64, device="cuda")
        w, state, scal = (torch.zeros(k, dtype=torch.float64, device="cuda")
                          for k in (4, 3 * ncv + 2, 2))
        work = torch.zeros(int(_lib.load().tnb_dot_work_bytes(4)), dtype=torch.uint8, device="cuda")
        P = _exec.ptr
        _lib.call("tnb_lanczos_solve", seq.handle, P(slots[0]), P(slots[1]), 4, ncv, 1e-12, 0,
                  P(x), P(V), 4, P(w), P(state), P(scal), None, None, P(run_start), P(run_w), 1,
                  P(work), None, _exec.stream_ptr())
        torch.cuda.synchronize()
        assert (_lib.device_error(0) == 0) == good
        if good:  # the identity: one vector, alpha = 1, then a breakdown
            assert np.allclose(V[0].cpu().numpy(), x.cpu().numpy() / np.sqrt(30.0), rtol=1e-15)
            assert abs(float(state[0]) - 1.0) < 1e-14 and float(state[3 * ncv]) == 1.0
            assert not V[1:].any()
    assert _lib.device_error(0) == 0

"""Which solves ``tnb_lanczos_solve`` runs as one launch of one CTA: by the multiply-adds, the
elements and the number of a matvec's products together.  The one launch leaves the recorded buffers
between the stages as they were, the launches write them; both give the same bits."""

import numpy as np
import pytest
import torch

from tenet import _exec, _lib

pytestmark = pytest.mark.gpu
P = _exec.ptr


def _solve(stages, m, k, ncv=4):
    f64 = dict(dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(m * k)
    bufs = [torch.zeros(m * k, **f64) for _ in range(stages + 1)]
    mats = [torch.randn(k * k, generator=g, **f64) for _ in range(stages)]
    tables = [_exec.make_gemm([(m, k, k, 0, k, 0, k, 0, k)], _exec.TILE_32, split_k=False)
              for _ in range(stages)]
    seq = _exec.Seq()
    with seq:
        for t, b, x, y in zip(tables, mats, bufs, bufs[1:]):
            t.run(x, b, y)
    n = m * k
    V = torch.zeros((ncv + 1, n), **f64)
    w, state, scal = (torch.zeros(s, **f64) for s in (n, 3 * ncv + 2, 2))
    x = torch.randn(n, generator=g, **f64)
    start, weight = torch.tensor([0, n], device="cuda"), torch.ones(1, **f64)
    work = torch.zeros(int(_lib.load().tnb_dot_work_bytes(n)), dtype=torch.uint8, device="cuda")
    _lib.call("tnb_lanczos_solve", seq.handle, P(bufs[0]), P(bufs[-1]), n, ncv, 1e-30, 0, P(x),
              P(V), n, P(w), P(state), P(scal), None, None, P(start), P(weight), 1, P(work), None,
              _exec.stream_ptr())
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0 and torch.isfinite(V).all()
    one_launch = not any(b.any() for b in bufs[1:-1])
    return one_launch, [t.cpu().numpy() for t in (V, state)]


@pytest.mark.parametrize("stages, m, k, one", [
    (2, 16, 64, True), (2, 64, 32, True), (2, 65, 32, False),
    (2, 40, 48, False), (3, 64, 32, False), (3, 16, 64, False), (6, 30, 32, True),
    (6, 100, 16, True)])
def test_the_work_of_all_products_counts(stages, m, k, one):
    got, (v, state) = _solve(stages, m, k)
    assert got == one
    # one vector more than the recurrence needs, against NumPy: alpha_0 = v_0 . H v_0
    x = v[0].reshape(m, k)
    g = torch.Generator(device="cuda").manual_seed(m * k)
    y = x
    for _ in range(stages):
        y = y @ torch.randn(k * k, generator=g, dtype=torch.float64,
                            device="cuda").cpu().numpy().reshape(k, k)
    scale = np.abs(x * y).sum()
    assert abs(state[0] - (x * y).sum()) <= 1e-13 * scale * (stages * k) ** 0.5


def _gather(n, kind):
    """A gather of ``n`` elements, as a user may record one: backwards through the source, or
    the sum of two terms over a matrix read from its last row up (``n`` = 6 rows)."""
    row = np.zeros(_exec.SEG_W, np.int64)
    if kind == "backwards":
        row[:5] = 0, n, 1, 0, 1
        row[8], row[16], row[32] = n, 1, -1
        return _exec.make_gather(([row], [n - 1], [2.0], [0]))
    c = n // 6
    row[:5] = 0, n, 2, 0, 2
    row[8:10], row[16:18], row[24:26], row[32:34] = (6, c), (c, 1), (-1, 0), (0, 1)
    return _exec.make_gather(([row], [5 * c, 5 * c], [2.0, -0.5], [c, c]))


@pytest.mark.parametrize("kind", ["backwards", "rows up"])
def test_sources_read_backwards(kind, n=48, ncv=5):
    f64 = dict(dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(2)
    x_slot, mid, y_slot = (torch.zeros(n, **f64) for _ in range(3))
    mat, x = torch.randn(n * n, generator=g, **f64), torch.randn(n, generator=g, **f64)
    gather, gemm = _gather(n, kind), _exec.make_gemm([(1, n, n, 0, n, 0, n, 0, n)], _exec.TILE_32,
                                                     split_k=False)
    assert gather.takes_items(True)
    one, sink = torch.ones(1, **f64), torch.zeros(1, **f64)
    extra = _exec.make_gemm([(1, 1, 1, 0, 1, 0, 1, 0, 1)], _exec.TILE_32)
    start, weight = torch.tensor([0, n], device="cuda"), torch.ones(1, **f64)
    work = torch.zeros(int(_lib.load().tnb_dot_work_bytes(n)), dtype=torch.uint8, device="cuda")
    out = []
    for more in (0, 13):  # one launch, and behind more stages than it takes
        seq = _exec.Seq()
        with seq:
            for _ in range(more):
                extra.run(one, one, sink)
            gather.run(x_slot, mid)
            gemm.run(mid, mat, y_slot)
        V = torch.zeros((ncv + 1, n), **f64)
        w, state, scal = (torch.zeros(s, **f64) for s in (n, 3 * ncv + 2, 2))
        _lib.call("tnb_lanczos_solve", seq.handle, P(x_slot), P(y_slot), n, ncv, 1e-30, 0, P(x),
                  P(V), n, P(w), P(state), P(scal), None, None, P(start), P(weight), 1, P(work),
                  None, _exec.stream_ptr())
        torch.cuda.synchronize()
        assert _lib.device_error(0) == 0 and bool(mid.any()) == bool(more)
        out.append((V.cpu().numpy(), state.cpu().numpy()))
    assert all(np.array_equal(a, b) for a, b in zip(*out)) and out[0][0].any()


@pytest.mark.parametrize("n, runs", [(8193, 0), (100000, 1500), (100000, 3)])
def test_long_solves_of_any_runs(n, runs, ncv=3):
    """No runs (every sum is zero), more than the cluster step takes at this length, few."""
    f64 = dict(dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n + runs)
    x_slot, y_slot = (torch.zeros(n, **f64) for _ in range(2))
    row = np.zeros(_exec.SEG_W, np.int64)
    row[:5] = 0, n, 1, 0, 1
    row[8], row[16], row[32] = n, 1, -1
    gather = _exec.make_gather(([row], [n - 1], [1.5], [0]))  # 1.5 x backwards
    seq = _exec.Seq()
    with seq:
        gather.run(x_slot, y_slot)
    cuts = np.linspace(0, n, runs + 1).astype(np.int64)
    wts = np.arange(1.0, runs + 1.0) % 5 + 1
    start = torch.tensor(cuts, device="cuda")
    weight = torch.tensor(np.append(wts, 1.0), device="cuda")
    x = torch.randn(n, generator=g, **f64)
    V = torch.zeros((ncv + 1, n), **f64)
    w, state, scal = (torch.zeros(s, **f64) for s in (n, 3 * ncv + 2, 2))
    work = torch.zeros(int(_lib.load().tnb_dot_work_bytes(n)), dtype=torch.uint8, device="cuda")
    _lib.call("tnb_lanczos_solve", seq.handle, P(x_slot), P(y_slot), n, ncv, 1e-30, 0, P(x), P(V),
              n, P(w), P(state), P(scal), None, None, P(start), P(weight), runs, P(work),
              None, _exec.stream_ptr())
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0
    if not runs:
        assert float(scal[0]) == 0.0
        return
    q, xh = np.repeat(wts, np.diff(cuts)), x.cpu().numpy()
    v = xh / np.sqrt(np.sum(q * xh * xh))
    a = np.sum(q * v * 1.5 * v[::-1])
    assert abs(float(state[0]) - a) <= 1e-12 * np.sum(q * np.abs(v * v[::-1]))
    r = 1.5 * v[::-1] - a * v
    assert abs(float(state[2 * ncv]) - np.sum(q * r * r)) <= 1e-11 * np.sum(q * r * r)

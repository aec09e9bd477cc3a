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

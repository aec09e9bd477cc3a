"""NaN and infinity through the blockwise SVD's two kernels: every element of the factors is
written, and the same by both (a column whose norm is NaN stays as it is)."""

import numpy as np
import pytest
import torch

from tenet import _exec, _lib

pytestmark = pytest.mark.gpu
P = _exec.ptr
NAN, INF = float("nan"), float("inf")
UNWRITTEN = -1234.5  # (no element of an input)


def _factors(entry, a):
    m, n = a.shape
    k = min(m, n)
    f64 = dict(dtype=torch.float64, device="cuda")
    A = torch.tensor(a.ravel(), device="cuda")
    U, S, V = (torch.full((x,), UNWRITTEN, **f64) for x in (m * k, k, k * n))
    R = torch.tensor([(m, n, 0, 0, 0, 0, -1, 0)], dtype=torch.int64, device="cuda")
    info = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    args = (P(R), 1, P(A), A.numel(), P(U), U.numel(), P(S), S.numel(), P(V), V.numel())
    if entry == "tnb_block_svd":
        smem = max(m, n) * k + k * k + 2 * k
        _lib.call(entry, *args, None, 0, P(info), smem, _exec.stream_ptr())
    else:
        _lib.call(entry, *args, P(info), max(m, n), k, _exec.stream_ptr())
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0 and int(info[0]) == 0
    return [x.cpu().numpy() for x in (U, S, V)]


# (NaN norms have no order among several columns)
@pytest.mark.parametrize("shape, value", [
    *(((m, n), x) for m, n in ((1, 1), (5, 1), (1, 5), (40, 1), (1, 130)) for x in (NAN, INF)),
    ((6, 3), INF), ((3, 6), -INF)])
def test_both_kernels_write_the_same_factors(shape, value):
    a = np.arange(1.0, 1.0 + shape[0] * shape[1]).reshape(shape)
    a[shape[0] // 2, shape[1] // 2] = value
    got, want = (_factors(e, a) for e in ("tnb_block_svd_cluster", "tnb_block_svd"))
    for x, y in zip(got, want):
        assert np.array_equal(x, y, equal_nan=True)
        assert not (x == UNWRITTEN).any()

"""Every form and every build of the wide kernel (a few rows, a long N) at the edges of its
rows, contracted lengths and columns: tables of 78 to 1,560 tiles reach the build of few
tiles, of many, and the one between.  Operands are small integers, a few of them infinite, in
buffers of NaN, so results are compared for equality; C starts at either parity of eight
bytes, with even and odd leading dimensions."""

import numpy as np
import pytest
import torch

from tenet import _exec, _lib
from test_gpu_gemm_tiles import _products

pytestmark = pytest.mark.gpu

SHAPES = [(m, n) for m in (1, 4, 5, 8, 9, 16) for n in (1, 7, 8, 9, 127, 128, 129, 256, 257, 600)]


@pytest.mark.parametrize("K", [0, 1, 4, 5, 8, 9, 12, 13, 16])
@pytest.mark.parametrize("copies, tiles", [(1, 78), (8, 624), (11, 858), (20, 1560)])
def test_wide_builds(K, copies, tiles):
    rng = np.random.default_rng(K)
    prods, a, b, want, n_c = _products(rng, [(m, n, K) for m, n in SHAPES])
    infinite = rng.choice(np.flatnonzero(np.isfinite(b)), 5 if K else 0)
    b[infinite] = np.inf
    values = []
    with np.errstate(invalid="ignore"):
        for M, N, _, ao, lda, bo, ldb, co, ldc in prods:
            A = np.lib.stride_tricks.as_strided(a[ao:], (M, K), (8 * lda, 8))
            B = np.lib.stride_tricks.as_strided(b[bo:], (K, N), (8 * ldb, 8))
            values.append((A[:, :, None] * B[None]).sum(1) if K else np.zeros((M, N)))
    g = _exec.make_gemm([(*p[:7], p[7] + i * n_c, p[8]) for i in range(copies) for p in prods],
                        _exec.TILE_WIDE)
    assert g.tiles == tiles
    da, db = torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda")
    for shift in (0, 1):
        c = torch.full((shift + copies * n_c,), 9.0, dtype=torch.float64, device="cuda")
        g.run(da, db, c[shift:])
        torch.cuda.synchronize()
        assert _lib.device_error(0) == 0
        got = c[shift:].cpu().numpy().reshape(copies, n_c)
        rest = np.ones(n_c, bool)
        for (M, N, _, _, _, _, _, co, ldc), v in zip(prods, values):
            at = co + ldc * np.arange(M)[:, None] + np.arange(N)
            assert np.array_equal(got[:, at], np.broadcast_to(v, (copies, M, N)), equal_nan=True)
            rest[at] = False
        assert (got[:, rest] == 9.0).all()  # nothing outside the products' rows is written

"""The FP64 grouped GEMM kinds at the edges of their tiles, K slabs and splits.

Operands are small integers, so every product and sum is exact and results are compared
for equality; the operands sit in buffers of NaN at odd offsets with padded leading
dimensions, so a read outside a product's own block shows."""

import numpy as np
import pytest
import torch

from tenet import _exec, _lib

pytestmark = pytest.mark.gpu


def _products(rng, shapes):
    """Products ``(M, N, K, ...)`` over NaN-padded buffers, and their values."""
    prods, a_parts, b_parts, want, at = [], [], [], [], [3, 5, 1]
    for M, N, K in shapes:
        lda, ldb, ldc = K + 3, N + 1, N + 2
        A = np.full((M, lda), np.nan)
        B = np.full((max(K, 1), ldb), np.nan)
        A[:, :K] = rng.integers(-4, 5, (M, K))
        B[:K, :N] = rng.integers(-4, 5, (K, N))
        prods.append((M, N, K, at[0], lda, at[1], ldb, at[2], ldc))
        want.append((at[2], ldc, A[:, :K] @ B[:K, :N] if K else np.zeros((M, N))))
        a_parts.append(A.ravel()), b_parts.append(B.ravel())
        at = [at[0] + A.size, at[1] + B.size, at[2] + M * ldc]
    a = np.concatenate([np.full(3, np.nan), *a_parts])
    b = np.concatenate([np.full(5, np.nan), *b_parts])
    return prods, a, b, want, at[2]


def _check(prods, a, b, want, n_c, kind, split):
    g = _exec.make_gemm(prods, kind, split_k=split)
    da, db = torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda")
    old = _exec.DIRECT_MIN_TILES
    for least in (10 ** 9, 0):  # the tile map, then one row per tile
        _exec.DIRECT_MIN_TILES = least
        try:
            for _ in range(2):  # twice: the split counters are left ready for the next run
                c = torch.full((n_c + 4,), 9.0, dtype=torch.float64, device="cuda")
                g.run(da, db, c)
        finally:
            _exec.DIRECT_MIN_TILES = old
        torch.cuda.synchronize()
        assert _lib.device_error(0) == 0
        got, rest = c.cpu().numpy(), np.ones(n_c + 4, bool)
        for off, ldc, w in want:
            for i in range(w.shape[0]):
                lo = off + i * ldc
                assert np.array_equal(got[lo:lo + w.shape[1]], w[i])
                rest[lo:lo + w.shape[1]] = False
        assert (got[rest] == 9.0).all()  # nothing outside the products' rows is written


MN = [(1, 1), (8, 16), (16, 8), (31, 33), (32, 32), (33, 31), (63, 65), (64, 64), (65, 130)]


@pytest.mark.parametrize("kind", [_exec.TILE_64, _exec.TILE_32])
@pytest.mark.parametrize("K", [0, 1, 4, 7, 8, 9, 15, 16, 17, 24, 25, 33, 50])
def test_tiles(kind, K):
    rng = np.random.default_rng(K)
    _check(*_products(rng, [(m, n, K) for m, n in MN]), kind, False)


@pytest.mark.parametrize("kind", [_exec.TILE_64, _exec.TILE_32])
@pytest.mark.parametrize("K", [65, 127, 128, 129, 700])
def test_split_tiles(kind, K):
    rng = np.random.default_rng(K)
    _check(*_products(rng, [(5, 70, K), (64, 33, K), (33, 64, 30)]), kind, True)


@pytest.mark.parametrize("K", [0, 1, 3, 4, 5, 16])
def test_wide(K):
    rng = np.random.default_rng(K)
    shapes = [(m, n, K) for m in (1, 4, 16) for n in (1, 127, 128, 129, 255, 256, 257, 600)]
    _check(*_products(rng, shapes), _exec.TILE_WIDE, False)


@pytest.mark.parametrize("precision", ["tf32", "3xbf16"])
@pytest.mark.parametrize("rows", [1, 2, 31, 32, 33, 1025])
def test_packed_slabs_of_many_rows(precision, rows):
    """Tensor-core tables of every size class of the pack kernel's search for a slab's row:
    integers of up to 3 bits are exact in either form."""
    rng = np.random.default_rng(rows)
    shapes = [(int(m), int(n), int(k)) for m, n, k in
              zip(rng.integers(1, 140, rows), rng.integers(1, 140, rows),
                  rng.choice([0, 1, 31, 32, 33, 70], rows))]
    prods, a, b, want, n_c = _products(rng, shapes)
    _check(prods, a, b, want, n_c, _exec.TC_KINDS[precision], False)

"""The warp form of the blockwise LQ (``tnb_block_lq_warp``) at the edges of its
elements-per-lane classes and of a warp's column count: L and Q against NumPy's LAPACK QR
of each transpose element by element (the reference's gauge), and rank-deficient sectors.

Tolerances as for ``tnb_block_lq``: 1e-12 of the block's scale for the factors (a
Householder QR's backward error at a few hundred rows, magnified by the inverse of the
smallest pivot of a normal random block), 1e-13 for the product and Q's rows."""

import numpy as np
import pytest
import torch

from tenet import SymmetricTensor, _exec, _lib, linalg
from tenet.structure import IN, OUT, GradedSpace, Leg
from tenet.symmetry import U1

pytestmark = pytest.mark.gpu
P = _exec.ptr


def _lq_warp(mats):
    rows, parts, bo, lo, qo = [], [], 0, 0, 0
    for b in mats:
        mb, nb = b.shape
        k = min(mb, nb)
        rows.append((mb, nb, bo, lo, qo, -1, 0, 0))
        parts.append(b.ravel())
        bo, lo, qo = bo + b.size, lo + mb * k, qo + k * nb
    B = torch.tensor(np.concatenate(parts), device="cuda")
    L, Q = (torch.full((max(1, x),), np.nan, dtype=torch.float64, device="cuda")
            for x in (lo, qo))
    R = torch.tensor(rows, dtype=torch.int64, device="cuda")
    smem = max(b.size + 3 * min(b.shape) for b in mats)
    _lib.call("tnb_block_lq_warp", P(R), len(rows), P(B), B.numel(), P(L), L.numel(), P(Q),
              Q.numel(), max(b.shape[1] for b in mats), smem, _exec.stream_ptr())
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0
    L, Q = L.cpu().numpy(), Q.cpu().numpy()
    out = []
    for (mb, nb, _, l, q, _, _, _) in rows:
        k = min(mb, nb)
        out.append((L[l:l + mb * k].reshape(mb, k), Q[q:q + k * nb].reshape(k, nb)))
    return out


@pytest.mark.parametrize("shapes", [
    [(1, 1), (1, 6), (6, 1), (2, 2), (3, 7), (31, 32), (32, 31), (32, 32), (70, 5)],
    [(33, 33), (31, 64), (64, 33), (65, 60)],
    [(77, 128), (32, 65), (100, 40), (128, 127), (16, 128), (17, 100)],
    [(129, 60), (200, 100)],
    [(77, 206), (65, 256), (80, 129), (15, 200)],
    [(77, 206), (110, 256), (256, 110)],
    [(40, 257), (56, 512), (1, 512)],
])
def test_lq_warp_shapes(shapes):
    rng = np.random.default_rng(21)
    mats = [rng.standard_normal(sh) for sh in shapes]
    for b, (lf, qf) in zip(mats, _lq_warp(mats)):
        q, r = np.linalg.qr(b.T)
        scale = max(np.abs(b).max(), 1e-300)
        assert np.abs(lf - r.T).max() <= 1e-12 * scale * max(b.shape) ** 0.5, b.shape
        assert np.abs(qf - q.T).max() <= 1e-12, b.shape
        assert np.abs(lf @ qf - b).max() <= 1e-13 * scale * max(b.shape) ** 0.5
        assert np.all(np.triu(lf, 1) == 0.0)


def test_lq_warp_one_row_sectors_bit_exact():
    rng = np.random.default_rng(7)
    mats = [rng.standard_normal((1, 2)) * 10.0 ** rng.uniform(-3, 6) for _ in range(200)]
    for b, (lf, qf) in zip(mats, _lq_warp(mats)):
        q, r = np.linalg.qr(b.T)
        assert np.array_equal(lf, r.T) and np.array_equal(qf, q.T), b


def test_lq_warp_rank_deficient():
    rng = np.random.default_rng(6)
    zero_rows = rng.standard_normal((9, 12))
    zero_rows[[2, 7], :] = 0.0
    zero_cols = rng.standard_normal((40, 35))
    zero_cols[:, [0, 3]] = 0.0
    rank_one = np.outer(rng.standard_normal(10), rng.standard_normal(70))
    mats = [zero_rows, zero_cols, rank_one, np.zeros((4, 3)), np.zeros((3, 40))]
    for b, (lf, qf) in zip(mats, _lq_warp(mats)):
        k = min(b.shape)
        assert np.abs(qf @ qf.T - np.eye(k)).max() <= 1e-13
        assert np.abs(lf @ qf - b).max() <= 1e-13 * max(np.abs(b).max(), 1.0)


def test_lq_mixes_both_kernels():
    """A tensor with sectors on either side of the warp kernel's limits: W of 120 x 300
    doubles beyond shared memory, a 2 x 600 one of more than 512 columns, and small ones."""
    rows = GradedSpace.new(U1, {U1.sector(0): 120, U1.sector(1): 2, U1.sector(2): 30})
    cols = GradedSpace.new(U1, {U1.sector(0): 300, U1.sector(1): 600, U1.sector(2): 7})
    t = SymmetricTensor.random((Leg(rows, OUT), Leg(cols, IN)), seed=3)
    left, q = linalg.lq(t)
    for b, lf, qf in zip(t.blocks, left.blocks, q.blocks):
        w, r = np.linalg.qr(b.cpu().numpy().T)
        assert np.abs(lf.cpu().numpy() - r.T).max() <= 1e-11
        assert np.abs(qf.cpu().numpy() - w.T).max() <= 1e-11
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0

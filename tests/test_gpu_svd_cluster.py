"""The cluster form of the blockwise SVD (``tnb_block_svd_cluster``) at the edges of its
elements-per-lane classes, cluster sizes and pair counts: singular values, isometry and
reconstruction against NumPy as for ``tnb_block_svd``, and that kernel's bits (the two run
the same rotations in the same arithmetic)."""

import numpy as np
import pytest
import torch

from test_gpu_svd import _check, _svd_batch
from tenet import _exec, _lib, linalg
from tenet.symmetry import SU2

pytestmark = pytest.mark.gpu
P = _exec.ptr


def _cluster_batch(mats):
    rows, parts, ao, uo, so, vo = [], [], 0, 0, 0, 0
    for a in mats:
        m, n = a.shape
        k = min(m, n)
        rows.append((m, n, ao, uo, so, vo, -1, 0))
        parts.append(a.ravel())
        ao, uo, so, vo = ao + a.size, uo + m * k, so + k, vo + k * n
    f64 = dict(dtype=torch.float64, device="cuda")
    A = torch.tensor(np.concatenate(parts), device="cuda")
    U, S, V = (torch.full((max(1, x),), np.nan, **f64) for x in (uo, so, vo))
    R = torch.tensor(rows, dtype=torch.int64, device="cuda")
    info = torch.full((len(rows),), 7, dtype=torch.int32, device="cuda")
    r = max(max(a.shape) for a in mats)
    c = max(min(a.shape) for a in mats)
    assert _lib.load().tnb_block_svd_cluster_ok(r, c) == 1
    _lib.call("tnb_block_svd_cluster", P(R), len(rows), P(A), A.numel(), P(U), U.numel(), P(S),
              S.numel(), P(V), V.numel(), P(info), r, c, _exec.stream_ptr())
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0
    assert (info == 0).all(), info
    U, S, V = U.cpu().numpy(), S.cpu().numpy(), V.cpu().numpy()
    out = []
    for (m, n, _, u, s, v, _, _) in rows:
        k = min(m, n)
        out.append((U[u:u + m * k].reshape(m, k), S[s:s + k], V[v:v + k * n].reshape(k, n)))
    return out


def _matrix(rng, m, n):
    k = min(m, n)
    x = np.linalg.qr(rng.standard_normal((m, k)))[0]
    y = np.linalg.qr(rng.standard_normal((n, k)))[0]
    return x * 10.0 ** -(2.0 * np.arange(k) / max(k, 2)) @ y.T


@pytest.mark.parametrize("shapes", [
    [(1, 1), (1, 5), (5, 1), (2, 2), (3, 2), (2, 3), (3, 3)],
    [(8, 8), (9, 9), (10, 7), (7, 10), (32, 31), (33, 16), (17, 32)],
    [(32, 32), (33, 33), (64, 40), (40, 65), (65, 64), (63, 64), (2, 60)],
    [(128, 128), (127, 129), (129, 66), (1, 128), (90, 127)],
    [(256, 130), (257, 129), (60, 300)],
    [(512, 256)],
])
def test_cluster_svd_shapes(shapes):
    rng = np.random.default_rng(11)
    mats = [_matrix(rng, *sh) for sh in shapes]
    for a, got, ref in zip(mats, _cluster_batch(mats), _svd_batch(mats)):
        _check(a, *got)
        for x, y in zip(got, ref):
            assert np.array_equal(x, y)


def test_cluster_svd_zero_columns_and_graded_spectra():
    rng = np.random.default_rng(12)
    zero_cols = rng.standard_normal((12, 8))
    zero_cols[:, [1, 5]] = 0.0
    zero_rows = rng.standard_normal((70, 99))
    zero_rows[[0, 3], :] = 0.0
    rank_one = np.outer(rng.standard_normal(10), rng.standard_normal(7))
    one_entry = np.zeros((37, 20))
    one_entry[4, 3] = 2.0
    mats = [zero_cols, zero_rows, rank_one, np.zeros((4, 3)), np.zeros((3, 4)), one_entry]
    for a, got in zip(mats, _cluster_batch(mats)):
        _check(a, *got)


def test_cluster_svd_refuses_what_it_cannot_hold():
    lib = _lib.load()
    assert lib.tnb_block_svd_cluster_ok(513, 4) == 0
    assert lib.tnb_block_svd_cluster_ok(300, 257) == 0
    assert lib.tnb_block_svd_cluster_ok(4, 8) == 0
    assert lib.tnb_block_svd_cluster(None, 1, None, 0, None, 0, None, 0, None, 0, None, 600, 10,
                                     None) == 1


@pytest.mark.parametrize("total", [1, 31, 1023, 1024, 1025, 2500])
@pytest.mark.parametrize("mode,cutoff", [("rsum2", 1e-6), ("sum1", 1e-2), ("rel", 1e-3),
                                         ("rsum2", None)])
def test_decision_staged_and_streamed(total, mode, cutoff):
    """Spectra on both sides of the staged decision's limit (1024 values) against the host
    rule: kept counts, order and sums (sums to 1e-12: a few thousand roundings)."""
    rng = np.random.default_rng(total)
    labels = [0, 2, 4, 6, 8][:min(5, total)]
    cuts = np.sort(rng.choice(np.arange(1, total), size=len(labels) - 1, replace=False)) \
        if len(labels) > 1 else np.zeros(0, int)
    sizes = np.diff(np.concatenate([[0], cuts, [total]]))
    spectra = [np.sort(10.0 ** -rng.integers(0, 400, n).astype(float) ** 0.25)[::-1]
               for n in sizes]
    spectrum = sorted(((float(x), c, i) for c, sp in zip(labels, spectra)
                       for i, x in enumerate(sp)), key=lambda e: (-e[0], e[1], e[2]))
    offs = np.concatenate([[0], np.cumsum(sizes)])
    i64 = dict(dtype=torch.int64, device="cuda")
    s = torch.tensor(np.concatenate(spectra), device="cuda")
    sec = torch.tensor([(n, offs[k], c, 0) for k, (c, n) in enumerate(zip(labels, sizes))], **i64)
    qd = torch.tensor([c + 1.0 for c in labels], dtype=torch.float64, device="cuda")
    for max_bond in (None, 1, total, 3 * total) if cutoff is not None else (1, total):
        keep = torch.full((len(labels),), 9, **i64)
        ss = torch.zeros(total, dtype=torch.float64, device="cuda")
        sc = torch.zeros(total, dtype=torch.int32, device="cuda")
        st = torch.zeros(8, dtype=torch.float64, device="cuda")
        for budget in ("dense", "reduced"):
            try:
                want = linalg.decide(spectrum, SU2, max_bond, cutoff, mode, budget=budget)
            except ValueError:  # nothing kept
                want = None
            _lib.call("tnb_truncate_decide", P(sec), P(qd), len(labels), P(s), total,
                      -1.0 if cutoff is None else cutoff, linalg._MODES[mode],
                      -1.0 if max_bond is None else float(max_bond), int(budget == "reduced"),
                      P(keep), P(ss), P(sc), P(st), _exec.stream_ptr())
            torch.cuda.synchronize()
            stats = st.cpu().numpy()
            got = {c: int(k) for c, k in zip(labels, keep.cpu().numpy()) if k}
            assert got == ({} if want is None else want.keep)
            order = [(float(x), labels[k]) for x, k in zip(ss.cpu().numpy(), sc.cpu().numpy())]
            assert order == [(x, c) for x, c, _ in spectrum]
            if want is not None:
                assert stats[0] == want.reduced_dim and stats[1] == want.dense_dim
                assert stats[2] == pytest.approx(want.discarded_weight, rel=1e-12, abs=1e-300)
                assert stats[3] == pytest.approx(sum(SU2._qdim(c) * x * x for x, c, _ in spectrum),
                                                 rel=1e-12)

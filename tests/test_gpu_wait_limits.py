"""Kernels whose bounded waits run out say so in what the caller reads.  The limit is an
argument: with 0 every wait counts as given up, so none is long and nothing hangs."""

import numpy as np
import pytest
import torch

from tenet import SymmetricTensor, _exec, _lib, linalg
from tenet.structure import IN, OUT, GradedSpace, Leg
from tenet.symmetry import U1

pytestmark = pytest.mark.gpu
P = _exec.ptr
TIMEOUT = 4  # TNB_ETIMEOUT


def _svd(mats, limit):
    rows, parts, ao, uo, so, vo = [], [], 0, 0, 0, 0
    for a in mats:
        (m, n), k = a.shape, min(a.shape)
        rows.append((m, n, ao, uo, so, vo, -1, 0))
        parts.append(a.ravel())
        ao, uo, so, vo = ao + a.size, uo + m * k, so + k, vo + k * n
    A = torch.tensor(np.concatenate(parts), device="cuda")
    U, S, V = (torch.zeros(x, dtype=torch.float64, device="cuda") for x in (uo, so, vo))
    R = torch.tensor(rows, dtype=torch.int64, device="cuda")
    info = torch.full((len(rows),), 7, dtype=torch.int32, device="cuda")
    args = (P(R), len(rows), P(A), A.numel(), P(U), U.numel(), P(S), S.numel(), P(V), V.numel(),
            P(info), max(max(a.shape) for a in mats), max(min(a.shape) for a in mats))
    if limit is None:
        _lib.call("tnb_block_svd_cluster", *args, _exec.stream_ptr())
    else:
        _lib.call("tnb_block_svd_cluster_bounded", *args, limit, _exec.stream_ptr())
    torch.cuda.synchronize()
    return info.cpu().tolist(), S.cpu().numpy()


# one CTA, the hand-over after a sweep without rotations, 2, 4 and 16 CTAs, several sectors
@pytest.mark.parametrize("shapes", [[(3, 3)], [(2, 2)], [(9, 12)], [(33, 20)], [(128, 128)],
                                    [(60, 40), (1, 1), (2, 5), (40, 60)]])
def test_svd_reports_a_wait_that_gave_up(shapes):
    rng = np.random.default_rng(4)
    mats = [rng.standard_normal(s) if s != (2, 2) else np.diag([2.0, 1.0]) for s in shapes]
    info, _ = _svd(mats, 0)
    assert info == [0 if min(s) == 1 else -TIMEOUT for s in shapes]  # (one column waits for none)
    assert _lib.device_error(0) == TIMEOUT
    info, got = _svd(mats, None)  # and the device is as before
    assert info == [0] * len(shapes) and _lib.device_error(0) == 0
    want = np.concatenate([np.linalg.svd(a, compute_uv=False) for a in mats])
    assert np.abs(got - want).max() <= 1e-13 * want.max() * max(max(s) for s in shapes)


def test_svd_truncated_raises(monkeypatch):
    legs = (Leg(GradedSpace.new(U1, {U1.sector(q): 6 + q for q in range(3)}), OUT),
            Leg(GradedSpace.new(U1, {U1.sector(q): 9 - q for q in range(3)}), IN))
    t = SymmetricTensor.random(legs, seed=1)
    call = _lib.call

    def run_out(name, *args):
        if name == "tnb_block_svd_cluster":
            return call("tnb_block_svd_cluster_bounded", *args[:-1], 0, args[-1])
        return call(name, *args)

    with monkeypatch.context() as m:
        m.setattr(_lib, "call", run_out)
        with pytest.raises(RuntimeError, match="did not converge"):
            linalg.svd_truncated(t, max_bond=5)
    assert _lib.device_error(0) != 0
    linalg.svd_truncated(t, max_bond=5)
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0


@pytest.mark.parametrize("shapes", [[(2, 2)], [(3, 7), (1, 4), (40, 5)], [(77, 197)], [(6, 1)]])
def test_lq_fills_a_sector_whose_wait_gave_up_with_nan(shapes):
    rng = np.random.default_rng(5)
    mats = [rng.standard_normal(s) for s in shapes]
    rows, bo, lo, qo = [], 0, 0, 0
    for mb, nb in shapes:
        k = min(mb, nb)
        rows.append((mb, nb, bo, lo, qo, -1, 0, 0))
        bo, lo, qo = bo + mb * nb, lo + mb * k, qo + k * nb
    B = torch.tensor(np.concatenate([a.ravel() for a in mats]), device="cuda")
    L, Q = (torch.zeros(x, dtype=torch.float64, device="cuda") for x in (lo, qo))
    R = torch.tensor(rows, dtype=torch.int64, device="cuda")
    args = (P(R), len(rows), P(B), B.numel(), P(L), L.numel(), P(Q), Q.numel(),
            max(nb for _, nb in shapes), max(mb * nb + 3 * min(mb, nb) for mb, nb in shapes))
    for limit in (0, None):
        if limit is None:
            _lib.call("tnb_block_lq_warp", *args, _exec.stream_ptr())
        else:
            _lib.call("tnb_block_lq_warp_bounded", *args, limit, _exec.stream_ptr())
        torch.cuda.synchronize()
        assert _lib.device_error(0) == (0 if limit is None else TIMEOUT)
        for (mb, nb, b, l, q, *_), a in zip(rows, mats):
            k = min(mb, nb)
            lf, qf = L[l:l + mb * k].cpu().numpy(), Q[q:q + k * nb].cpu().numpy()
            if limit is None or mb == 1:  # (one row waits for no reflector)
                got = lf.reshape(mb, k) @ qf.reshape(k, nb)
                assert np.abs(got - a).max() <= 1e-13 * np.abs(a).max() * max(mb, nb) ** 0.5
            else:
                assert np.isnan(lf).all() and np.isnan(qf).all()

"""One Lanczos step on a thread-block cluster (``tnb_lanczos_step_cluster``) against the same
recurrence in NumPy, at vector lengths around the cluster's chunks, with several weighted
runs, through a stop and past it.

Tolerance: each sum has at most n terms summed pairwise per thread, so its relative error is
far below 1e-13 for positive terms; the update and the division round as NumPy's."""

import numpy as np
import pytest
import torch

from tenet import _exec, _lib

pytestmark = pytest.mark.gpu
P = _exec.ptr


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4097, 8191, 8193, 65537, 131071, 131072])
@pytest.mark.parametrize("runs", [1, 3, 40])
def test_cluster_step(n, runs):
    lib = _lib.load()
    assert n <= lib.tnb_lanczos_step_cluster_max_n()
    rng = np.random.default_rng(n + runs)
    cuts = np.unique(np.concatenate([[0], rng.integers(0, n, runs - 1), [n]]))
    wts = rng.integers(1, 6, len(cuts) - 1).astype(float)
    q = np.repeat(wts, np.diff(cuts))
    ncv, tol = 4, 1e-13
    host = {k: rng.standard_normal(n) for k in ("w", "v", "vprev")}
    dev = {k: torch.tensor(x, device="cuda") for k, x in host.items()}
    rs = torch.tensor(cuts, dtype=torch.int64, device="cuda")
    rw = torch.tensor(wts, device="cuda")
    for j, case in ((0, "go"), (2, "go"), (ncv - 1, "last"), (1, "breakdown"), (1, "stopped")):
        state = torch.zeros(3 * ncv + 2, dtype=torch.float64, device="cuda")
        if j:
            state[ncv + j - 1] = 0.75
        state[3 * ncv + 1] = 1.0 if case == "stopped" else 0.0
        out = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
        w = dev["w"]
        if case == "breakdown":  # w - a v - b vprev vanishes
            w = dev["v"] * 2.0 + dev["vprev"] * 0.75
        _lib.call("tnb_lanczos_step_cluster", n, P(w), P(dev["v"]), P(dev["vprev"]), P(out),
                  P(state), j, ncv, 1e9 if case == "breakdown" else tol, P(rs), P(rw), len(wts),
                  _exec.stream_ptr())
        torch.cuda.synchronize()
        st, got = state.cpu().numpy(), out.cpu().numpy()
        if case == "stopped":
            assert (got == 0.0).all() and st[3 * ncv] == 0.0
            continue
        wh = w.cpu().numpy()
        a = float(np.sum(q * host["v"] * wh))
        scale = float(np.sum(q * np.abs(host["v"] * wh)))
        assert abs(st[j] - a) <= 1e-13 * scale
        x = wh - host["v"] * st[j] - (host["vprev"] * 0.75 if j else 0.0)
        nrm2 = float(np.sum(q * x * x))
        assert abs(st[2 * ncv + j] - nrm2) <= 1e-12 * max(nrm2, 1e-300)
        if case == "go":
            beta = st[ncv + j]
            assert beta == np.sqrt(st[2 * ncv + j]) and st[3 * ncv] == j + 2
            assert st[3 * ncv + 1] == 0.0
            assert np.abs(got - x / beta).max() <= 1e-14 * np.abs(got).max()
        else:
            assert (got == 0.0).all() and st[3 * ncv] == j + 1 and st[3 * ncv + 1] == 1.0


def test_cluster_step_refuses_long_vectors():
    lib = _lib.load()
    x = torch.zeros(4, dtype=torch.float64, device="cuda")
    assert lib.tnb_lanczos_step_cluster(
        lib.tnb_lanczos_step_cluster_max_n() + 1, P(x), P(x), None, P(x), P(x), 0, 1, 0.0, P(x),
        P(x), 1, None) == 1

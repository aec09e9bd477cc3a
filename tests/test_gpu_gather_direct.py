"""Gathers from per-chunk rows (``tnb_block_gather_direct``): what tables run whose offsets
within a segment need more than 32 bits, in both of its builds, against the table's semantics
and the chunk-map gather.  The data are small integers, so equality is exact."""

import numpy as np
import pytest
import torch

import _emulate
from tenet import _exec, _lib
from test_gather_items import SEGMENTS, _table

pytestmark = pytest.mark.gpu
P = _exec.ptr


def _wide(segments):
    """A table of these segments and one whose leading dimension (no row stride uses it) is
    2^31, which warp items cannot hold."""
    t, n_src, n_dst = _table(np.random.default_rng(3), [*segments, ((5, 9), 1), ((40,), 1)],
                             two_buffers=True)
    t.seg[-1, 24:32] = 0
    t.seg[-1, 32] = 1
    t.tld[t.seg[-1, 3]] = 1 << 31
    return t, n_src, n_dst


@pytest.mark.parametrize("name, copies, many", [
    ("rank1", 1, False), ("rank2", 1, False), ("rank34", 1, False), ("terms", 1, False),
    ("rank2", 200, True), ("terms", 200, True), ("rank34", 300, True)])
def test_tables_past_32_bits(monkeypatch, name, copies, many):
    t, n_src, n_dst = _wide(SEGMENTS[name] * copies)
    assert t.item_rows() is None and t.direct_ok
    assert (t.chunks > 2 * 3 * _exec.N_SM) == many
    rng = np.random.default_rng(4)
    srcs = [rng.integers(-5, 6, x).astype(float) for x in n_src]
    want = [np.full(x, np.nan) for x in n_dst]
    _emulate.gather(t, srcs[0], want[0], srcs[1], want[1])
    ds = [torch.tensor(x, device="cuda") for x in srcs]
    got, plain = ([torch.full((x,), float("nan"), dtype=torch.float64, device="cuda")
                   for x in n_dst] for _ in range(2))
    names, call = [], _lib.call
    monkeypatch.setattr(_lib, "call", lambda n, *a: (names.append(n), call(n, *a))[1])
    t.run(ds[0], got[0], ds[1], got[1])
    monkeypatch.setattr(_exec, "DIRECT_GATHER", False)
    t.run(ds[0], plain[0], ds[1], plain[1])
    torch.cuda.synchronize()
    assert [n for n in names if "gather" in n] == ["tnb_block_gather_direct", "tnb_block_gather"]
    assert _lib.device_error(0) == 0
    for w, g, p in zip(want, got, plain):
        assert np.array_equal(w, g.cpu().numpy(), equal_nan=True)
        assert np.array_equal(w, p.cpu().numpy(), equal_nan=True)

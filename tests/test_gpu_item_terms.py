"""Gathers of several terms from warp items: terms past the inline ones and past the 32 that a
warp decodes together, ragged items, and rows of 32 words whose segments have several terms (as
a caller of the library may build them).  Integer data: equality is exact."""

import numpy as np
import pytest
import torch

import _emulate
from tenet import _exec, _lib
from test_gather_items import _table

pytestmark = pytest.mark.gpu
P = _exec.ptr

DIMS = [(7,), (33,), (65, 2), (9, 40), (5, 6, 7), (3, 4, 5, 6), (257,)]


def _run(terms, copies, width=None, cap=None):
    rng = np.random.default_rng(sum(terms))
    t, n_src, n_dst = _table(rng, [(d, k) for k in terms for d in DIMS] * copies, signed=True)
    src = rng.integers(-3, 4, n_src[0]).astype(float)
    want = np.full(n_dst[0], np.nan)
    _emulate.gather(t, src, want)
    ds = torch.tensor(src, device="cuda")
    dd = torch.full((n_dst[0],), float("nan"), dtype=torch.float64, device="cuda")
    if width is None:
        assert t.takes_items(False) and t.item_rows()[0] == 64
        t.run(ds, dd)
    else:
        lib, seg = _lib.load(), np.ascontiguousarray(t.seg)
        args = (t.n_seg, seg.ctypes.data, t.tsrc.ctypes.data, t.tcf.ctypes.data, t.tld.ctypes.data,
                t.n_term, cap, width)
        n = lib.tnb_plan_gather_items(*args, None, 0)
        rows = np.empty((n, width), np.int32)
        assert lib.tnb_plan_gather_items(*args, rows.ctypes.data, n) == n
        up = [torch.tensor(x, device="cuda") for x in (rows, t.tsrc, t.tcf, t.tld)]
        _lib.call("tnb_block_gather_items", P(up[0]), width, n, *(P(x) for x in up[1:]), t.n_term,
                  P(ds), ds.numel(), P(dd), dd.numel(), None, 0, None, 0, _exec.stream_ptr())
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0
    assert np.array_equal(want, dd.cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("terms", [[2], [0, 3, 7, 8], [5, 9, 10, 11], [31, 32, 33], [64, 65, 100]])
def test_terms(terms):
    _run(terms, 1)


@pytest.mark.parametrize("copies", [12, 120])  # the builds of more warps
def test_many_items(copies):
    _run([1, 4, 9], copies)


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("cap, copies", [(32, 1), (64, 1), (96, 1), (256, 1), (64, 12), (32, 30)])
def test_rows_of_either_width(width, cap, copies):
    _run([0, 1, 2, 8, 40], copies, width, cap)


def test_long_tables_of_many_terms_keep_to_the_chunk_forms():
    t, _, _ = _table(np.random.default_rng(1), [((1000,), 12)] * 1000)
    few, _, _ = _table(np.random.default_rng(1), [((1000,), 9)] * 1000)
    short, _, _ = _table(np.random.default_rng(1), [((1000,), 12)] * 100)
    assert not t.takes_items(False) and not t.takes_items(True)
    assert few.takes_items(False) and short.takes_items(False)
    assert _exec.item_size(10 ** 9, 9) == 256 and _exec.item_size(1000, 9) == 32
    assert _exec.item_size(1000, 3) == 64 and _exec.item_size(100000) == 256

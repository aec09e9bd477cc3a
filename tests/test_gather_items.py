"""The warp-item form of the block gather (``tnb_plan_gather_items``,
``tnb_block_gather_items``): its rows on the CPU and its kernel on the GPU against the plain
table's semantics (``_emulate.gather``), at the edges of items, ranks and term counts.

Bit-equality is expected: each destination element is one chain of fused multiply-adds over
its terms from zero; the test data are small integers, so rounding cannot enter."""

import numpy as np
import pytest

import _emulate
from tenet import _exec, _lib

P = _exec.ptr


def _table(rng, segments, two_buffers=False, signed=False):
    """A gather table with one segment per ``(dims, terms)``: destination dims in C order, the
    source a random permutation of them, as a packed matrix (row strides for the leading
    source dims, column strides for the rest)."""
    rows, tsrc, tcf, tld = [], [], [], []
    d_at, s_at = [0, 0], [0, 0]
    for k, (dims, terms) in enumerate(segments):
        buf = k % 2 if two_buffers else 0
        size, rank = int(np.prod(dims)), len(dims)
        perm = rng.permutation(rank)
        src_stride, acc = np.zeros(rank, np.int64), 1
        split = rng.integers(0, rank + 1)  # source dims before `split` are matrix rows
        rstr, cstr = np.zeros(rank, np.int64), np.zeros(rank, np.int64)
        cols = int(np.prod([dims[p] for p in perm[split:]])) if split < rank else 1
        ld = cols + int(rng.integers(0, 3))
        acc = 1
        for p in perm[split:][::-1]:
            cstr[p], acc = acc, acc * dims[p]
        acc = 1
        for p in perm[:split][::-1]:
            rstr[p], acc = acc, acc * dims[p]
        row = np.zeros(_exec.SEG_W, np.int64)
        row[:6] = d_at[buf], size, rank, len(tsrc), len(tsrc) + terms, buf
        row[8:8 + rank] = dims
        row[16:16 + rank] = np.concatenate([np.cumprod(dims[::-1])[::-1][1:], [1]])
        row[24:24 + rank], row[32:32 + rank] = rstr, cstr
        if signed and rank > 1:  # a reversed destination dim: negative stride from its end
            row[0] += row[16] * (dims[0] - 1)
            row[16] = -row[16]
        for _ in range(terms):
            tsrc.append(s_at[buf] + int(rng.integers(0, 4)))
            tcf.append(float(rng.integers(-3, 4)) or 2.0)
            tld.append(ld)
        d_at[buf] += size
        s_at[buf] += acc * ld + 8
        rows.append(row)
    seg = _exec._chunked(np.array(rows))
    return _exec.GatherTable(seg, tsrc, tcf, tld), [max(1, x) for x in s_at], \
        [max(1, x) for x in d_at]


SEGMENTS = {
    "rank1": [((n,), 1) for n in (2, 31, 32, 33, 255, 256, 257, 511, 513, 1000)],
    "rank2": [((a, b), 1) for a, b in ((2, 3), (24, 25), (16, 16), (2, 300), (300, 2), (129, 7))],
    "rank34": [((3, 5, 7), 1), ((2, 2, 2, 2), 1), ((9, 2, 31), 1), ((4, 8, 3, 11), 1)],
    "terms": [((6, 7), t) for t in (0, 1, 2, 3, 6, 7, 8, 9, 20)] + [((3, 90), 5), ((2, 3, 50), 0)],
}


def _run_items(width, n, rows, table, srcs, dsts):
    """The kernel's semantics from the item rows alone."""
    u = rows.view(np.uint32)
    def i64(r, at):
        return int(np.frombuffer(r[at:at + 2].tobytes(), np.int64)[0])
    for k in range(n):
        r, ru = rows[k], u[k]
        rank, buf = int(r[10]) & 255, (int(r[10]) >> 8) & 1
        q = np.arange(int(r[8]), int(r[8]) + int(r[9]))
        assert 0 < len(q) <= _exec.item_size(1 << 40)
        J, rem = [None] * rank, q.astype(object)
        for d in range(rank - 1, 0, -1):
            mul, shr = int(ru[15 + d]), (int(r[10]) >> (11 + 5 * d)) & 31
            quo = np.array([((x * mul) >> 32) >> shr for x in rem], dtype=object)
            J[d], rem = (rem - quo * int(r[12 + d])).astype(np.int64), quo
        J[0] = rem.astype(np.int64)
        to = i64(r, 0) + sum(j * int(r[20 + d]) for d, j in enumerate(J))
        R = sum(j * int(r[24 + d]) for d, j in enumerate(J))
        C = sum(j * int(r[28 + d]) for d, j in enumerate(J))
        acc = np.zeros(len(q))
        t0, t1 = int(r[6]), int(r[7])
        for i in range(t1 - t0):
            if i == 0:
                ts, cf, ld = i64(r, 2), np.frombuffer(r[4:6].tobytes(), np.float64)[0], int(r[11])
            elif width == 64 and i <= 6:
                at = 32 + 5 * (i - 1)
                ts, cf, ld = (i64(r, at), np.frombuffer(r[at + 2:at + 4].tobytes(), np.float64)[0],
                              int(r[at + 4]))
            else:
                ts, cf, ld = (int(table.tsrc[t0 + i]), float(table.tcf[t0 + i]),
                              int(table.tld[t0 + i]))
            acc = acc + cf * srcs[buf][ts + ld * R + C]
        dsts[buf][to] = acc


@pytest.mark.parametrize("name", list(SEGMENTS))
@pytest.mark.parametrize("signed", [False, True])
def test_item_rows_reproduce_the_table(name, signed):
    rng = np.random.default_rng(5)
    t, n_src, n_dst = _table(rng, SEGMENTS[name], two_buffers=True, signed=signed)
    width, n, rows = t.item_rows()
    assert width == (64 if name == "terms" else 32) and rows.shape == (n, width)
    srcs = [rng.integers(-5, 6, x).astype(float) for x in n_src]
    want = [np.full(x, np.nan) for x in n_dst]
    got = [np.full(x, np.nan) for x in n_dst]
    _emulate.gather(t, srcs[0], want[0], srcs[1], want[1])
    _run_items(width, n, rows, t, srcs, got)
    for w, g in zip(want, got):
        assert np.array_equal(w, g, equal_nan=True)


def test_item_rows_refuse_what_does_not_fit():
    rng = np.random.default_rng(6)
    t, _, _ = _table(rng, [((2, 3, 2, 3, 2), 1)])
    assert t.item_rows() is None  # rank 5
    for col, value in ((16, 1 << 31), (24, 1 << 31), (32, 1 << 40)):
        t, _, _ = _table(rng, [((4, 5), 1)])
        t.seg[0, col] = value
        assert t.item_rows() is None
    t, _, _ = _table(rng, [((4, 5), 1)])
    t.seg[0, 24], t.tld[0] = 3, 1 << 30  # ld x row stride past 32 bits
    assert t.item_rows() is None
    lib = _lib.load()
    a = (t.n_seg, t.seg.ctypes.data, t.tsrc.ctypes.data, t.tcf.ctypes.data, t.tld.ctypes.data)
    assert lib.tnb_plan_gather_items(*a, t.n_term, 48, 32, None, 0) == -2
    assert lib.tnb_plan_gather_items(*a, t.n_term, 256, 40, None, 0) == -2
    assert lib.tnb_plan_gather_items(*a, 0, 256, 32, None, 0) == -2  # terms past the end


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(SEGMENTS))
@pytest.mark.parametrize("copies", [1, 60, 600])  # the three kernels
def test_item_kernel(name, copies):
    import torch

    rng = np.random.default_rng(7)
    t, n_src, n_dst = _table(rng, SEGMENTS[name] * copies, two_buffers=True)
    srcs = [rng.integers(-5, 6, x).astype(float) for x in n_src]
    want = [np.full(x, np.nan) for x in n_dst]
    _emulate.gather(t, srcs[0], want[0], srcs[1], want[1])
    ds = [torch.tensor(x, device="cuda") for x in srcs]
    dd = [torch.full((x,), float("nan"), dtype=torch.float64, device="cuda") for x in n_dst]
    assert t.takes_items(False)
    t.run(ds[0], dd[0], ds[1], dd[1])
    seq = _exec.Seq()  # and recorded, with the buffers substituted at replay
    d2 = [torch.full_like(x, float("nan")) for x in dd]
    with seq:
        t.run(ds[0], dd[0], ds[1], dd[1])
    seq.run({dd[0].data_ptr(): d2[0].data_ptr(), dd[1].data_ptr(): d2[1].data_ptr()})
    torch.cuda.synchronize()
    assert _lib.device_error(0) == 0
    for w, g, h in zip(want, dd, d2):
        assert np.array_equal(w, g.cpu().numpy(), equal_nan=True)
        assert np.array_equal(w, h.cpu().numpy(), equal_nan=True)


@pytest.mark.gpu
def test_item_kernel_skips_and_reports_out_of_range_segments():
    """Buffers shorter than the table reaches: the kernel's own checks raise the bounds error
    and leave the destination of the offending segment untouched."""
    import torch

    rng = np.random.default_rng(8)
    t, n_src, n_dst = _table(rng, [((24, 25), 1), ((6, 7), 3)])
    src = torch.ones(n_src[0], dtype=torch.float64, device="cuda")
    dst = torch.full((n_dst[0],), 7.0, dtype=torch.float64, device="cuda")
    width, n, _ = t.item_rows()
    rows, tsrc, tcf, tld = t.item_arrays()
    for ns, nd in ((100, n_dst[0]), (n_src[0], 599)):
        dst.fill_(7.0)
        _lib.call("tnb_block_gather_items", P(rows), width, n, P(tsrc), P(tcf), P(tld), t.n_term,
                  P(src), ns, P(dst), nd, None, 0, None, 0, _exec.stream_ptr())
        torch.cuda.synchronize()
        assert _lib.device_error(0) != 0
        assert (dst[:600] == 7.0).all()
    assert _lib.device_error(0) == 0


@pytest.mark.gpu
def test_a_second_upload_of_a_table_is_the_one_read():
    """Two threads that meet at a table's first run may both upload it; a run reads the upload
    the table holds, never the addresses of one that went away."""
    import torch

    rng = np.random.default_rng(9)
    t, n_src, n_dst = _table(rng, [((24, 25), 1), ((6, 7), 3)])
    src = torch.randn(n_src[0], dtype=torch.float64, device="cuda")
    want, got = (torch.zeros(n_dst[0], dtype=torch.float64, device="cuda") for _ in range(2))
    t.run(src, want)
    first = t._idev
    t._idev = None
    t.run(src, got)
    assert t._idev is not first and t._head[0] is t._idev
    assert torch.equal(got, want)

"""A table's device copy is made once, whoever meets at its first use: addresses launched or
recorded by one thread must not go away because another made a second copy."""

import threading
import time

import numpy as np
import pytest

from tenet import _exec


class _SlowUpload:
    """Stands for ``_exec.Uploaded``: takes long enough for a second thread to arrive."""

    made = 0

    def __init__(self, arrays):
        self.arrays = tuple(_exec._DevArray(64 * (i + 1), x.size) for i, x in enumerate(arrays))
        time.sleep(0.02)
        type(self).made += 1

    def ready(self):
        return self.arrays


def _gather():
    seg = np.zeros((1, _exec.SEG_W), np.int64)
    seg[0, :5] = 0, 12, 1, 0, 1
    seg[0, 8] = 12
    seg[0, 16] = seg[0, 32] = 1
    return _exec.make_gather((seg, [0], [1.0], [0]))


def _gemm(kind):
    return _exec.make_gemm([(8, 8, 16, 0, 16, 0, 8, 0, 8)], kind)


def _run(table, monkeypatch):
    """``table.run`` up to the library call, as many tiles as the direct forms want."""
    table.tiles = _exec.DIRECT_MIN_TILES
    monkeypatch.setattr(type(table), "work", lambda self: None)
    x = _exec._DevArray(4096, 1024)
    return lambda: table.run(x, x, x)


@pytest.mark.parametrize("use", ["chunk_map", "chunk_rows", "items", "gemm", "gather_a", "rows",
                                 "slabs", "together"])
def test_two_threads_make_one_upload(monkeypatch, use):
    monkeypatch.setattr(_exec, "Uploaded", _SlowUpload)
    monkeypatch.setattr(_exec, "stream_ptr", lambda: 0)
    monkeypatch.setattr(_exec._lib, "call", lambda *a: None)
    _SlowUpload.made = 0
    if use in ("chunk_map", "chunk_rows", "items"):
        t = _gather()
        call = {"chunk_map": t.device_arrays, "chunk_rows": t.direct_arrays,
                "items": t.item_arrays}[use]
    elif use == "together":
        t = _gather()
        call = lambda: (_exec.upload_together([t]), t.item_arrays())  # noqa: E731
    elif use == "gather_a":
        t = _exec.GatherAGemm((np.zeros(129, np.int32), np.zeros(0, np.int32), np.zeros(0)),
                              [(8, 8, 16, 0, 16, 0, 8, 0, 8)], 128)
        call = t.device_tables
    elif use == "gemm":
        call = _gemm(_exec.TILE_32).device_tables
    else:
        call = _run(_gemm(_exec.TILE_32 if use == "rows" else _exec.TILE_TC_3XBF16), monkeypatch)
    threads = [threading.Thread(target=call) for _ in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert _SlowUpload.made == 1


@pytest.mark.parametrize("kind", [_exec.TILE_32, _exec.TILE_64, _exec.TILE_SKINNY,
                                  _exec.TILE_TC_3XBF16])
@pytest.mark.parametrize("many", [False, True])
def test_a_launch_uploads_the_form_it_reads(monkeypatch, kind, many):
    monkeypatch.setattr(_exec, "Uploaded", _SlowUpload)
    monkeypatch.setattr(_exec, "stream_ptr", lambda: 0)
    monkeypatch.setattr(_exec._lib, "call", lambda *a: None)
    t = _gemm(kind)
    run = _run(t, monkeypatch)
    t.tiles = _exec.DIRECT_MIN_TILES - (not many)
    _SlowUpload.made = 0
    _exec.upload_together([t])
    run()
    run()
    assert _SlowUpload.made == 1 and _exec.upload_together([t]) is None
    _exec.upload_together([t], recorded=True)  # a recording reads the tile map whatever the size
    assert _SlowUpload.made == 1 + many and t._dev is not None


def test_uploads_never_share_staging_bytes(monkeypatch):
    """Two threads upload through a ring that wraps at every second upload: the bytes of one are
    not written over before its copy has been queued."""
    class Buffer:
        def __init__(self, n):
            self.data = np.zeros(n, np.uint8)

        def pin_memory(self):
            return self

        def numpy(self):
            return self.data

        def __getitem__(self, part):
            return self.data[part]

        def copy_(self, staged, non_blocking):
            time.sleep(0.002)  # (a thread that wraps the ring meanwhile would overwrite it)
            self.data[:] = staged

        def data_ptr(self):
            return 64

    class Event:
        def record(self):
            pass

        def synchronize(self):
            pass

    monkeypatch.setattr(_exec.torch, "empty", lambda n, **k: Buffer(n))
    monkeypatch.setattr(_exec.torch.cuda, "Event", Event)
    monkeypatch.setattr(_exec.torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(_exec, "device", lambda: None)
    monkeypatch.setattr(_exec, "stream_ptr", lambda: 0)
    monkeypatch.setattr(_exec, "_STAGING", _exec._Staging(4096))
    bad = []

    def upload(value):
        for k in range(20):
            x, y = np.full(100, value + k), np.full(3, value - k, np.int32)
            got = _exec.Uploaded((x, y))
            if not (np.array_equal(got.buf.data[:800].view(np.int64), x)
                    and np.array_equal(got.buf.data[800:812].view(np.int32), y)):
                bad.append((value, k))

    threads = [threading.Thread(target=upload, args=(1000 * t,)) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad

"""Results of GPU encodes read back by the host: an encode that was lost (a wait
on the device ran out, here because its limit is 0) is an error and its column
decodes to nothing; deferred encodes finish in any order, on any stream, from
any thread."""
import threading

import numpy as np
import pytest
import torch

from fastlanesgpu_b200 import LAYOUT_TRANSPOSED, FlsError, _lib, datagen, ops
from fastlanesgpu_b200 import column as column_module
from fastlanesgpu_b200.column import (DeviceEncodedColumn, PendingEncode, encode_column_gpu, encode_column_learned_gpu)

MAX_POLLS = 1 << 22


def test_lost_encode_is_an_error():
    info = torch.zeros(4, dtype=torch.int64)
    p = PendingEncode(torch.zeros(8), torch.zeros(4), info, torch.zeros(1), 1024, LAYOUT_TRANSPOSED, False, defer=False)
    with pytest.raises(FlsError) as e:
        p.finish()
    assert e.value.status == 6


def _values(n, seed=0):
    return torch.from_numpy(datagen.for_bitpack_mixed(n, seed=seed).astype(np.int32)).cuda()


def _params(seed=0):
    return torch.randn(_lib.MLP_N_PARAMS, generator=torch.Generator().manual_seed(seed)).cuda()


class _ShortWaits:
    """The library, with the encoder's waits ended after the given tries."""

    def __init__(self, scan_polls, tile_polls):
        self._polls = scan_polls, tile_polls

    def __getattr__(self, name):
        return getattr(_lib.lib(), name)

    def fls_encode_column_gpu(self, v, n, schemes, scheme, layout, round4, out, cap, meta, info, ws, ws_bytes, stream):
        return _lib.lib().fls_selftest_encode_waits(v, n, scheme, None, out, cap, meta, info, ws, ws_bytes, 444,
                                                    *self._polls, stream)

    def fls_encode_learned_gpu(self, v, n, params, threshold, kappa, layout, out, cap, meta, info, schemes, ws,
                               ws_bytes, stream):
        return _lib.lib().fls_selftest_encode_waits(v, n, 0, params, out, cap, meta, info, ws, ws_bytes, 444,
                                                    *self._polls, stream)


def _expect_timeout():
    with pytest.raises(FlsError) as e:
        ops.check_device_error()
    assert e.value.status == 6


@pytest.mark.gpu
@pytest.mark.parametrize("polls", [(0, MAX_POLLS), (MAX_POLLS, 0), (0, 0)], ids=["scan", "tile", "both"])
@pytest.mark.parametrize("n_vec", [1, 9, 8 * 500 + 3])
@pytest.mark.parametrize("learned", [False, True])
def test_lost_encode(cuda, monkeypatch, polls, n_vec, learned):
    n = n_vec * 1024 - 1
    v = _values(n)
    ops.check_device_error()
    # the call: totals of 0, words untouched, metadata that no decoder takes
    cap = int(_lib.lib().fls_encode_bound_words(n)) + 4
    words = torch.zeros(cap, dtype=torch.int32, device="cuda")
    meta = torch.zeros(n_vec * 4, dtype=torch.int32, device="cuda")  # taken for constant vectors otherwise
    meta.view(torch.uint8)[12::16] = 3
    info = torch.full((4,), 5, dtype=torch.int64, device="cuda")
    ws = torch.empty(int(_lib.lib().fls_encode_learned_workspace_bytes(n)), dtype=torch.uint8, device="cuda")
    params = _params()
    stream = torch.cuda.current_stream().cuda_stream
    assert _lib.lib().fls_selftest_encode_waits(v.data_ptr(), n, 0, params.data_ptr() if learned else None,
                                                words.data_ptr(), cap, meta.data_ptr(), info.data_ptr(), ws.data_ptr(),
                                                ws.numel(), 444, *polls, stream) == 0
    assert info.tolist()[:3] == [0, 0, 0]
    _expect_timeout()
    schemes = meta.view(torch.uint8)[12::16]
    assert int((schemes == 3).sum()) == 0 and int((schemes == 5).sum()) > 0
    col = DeviceEncodedColumn(words, meta, n, LAYOUT_TRANSPOSED, cap, 1344, 31)
    out = torch.full((n_vec * 1024,), -7, dtype=torch.int32, device="cuda")
    ops.unpack_global(col, 1, out=out)
    with pytest.raises(FlsError) as e:
        ops.check_device_error()
    assert e.value.status == 5
    assert bool((out.view(n_vec, 1024)[schemes == 5] == -7).all())
    # the Python face
    monkeypatch.setattr(column_module, "lib", lambda: _ShortWaits(*polls))
    pending = encode_column_learned_gpu(v, params, defer=True) if learned else None
    for call in ((pending.finish, lambda: encode_column_learned_gpu(v, params)) if learned
                 else (lambda: encode_column_gpu(v, 0),)):
        with pytest.raises(FlsError) as e:
            call()
        assert e.value.status == 6
    _expect_timeout()
    # and afterwards
    monkeypatch.undo()
    assert torch.equal(ops.unpack_global(encode_column_gpu(v, 0), 1)[:n], v)
    ops.check_device_error()


def _check(result, want):
    (col, schemes, fallback), (wcol, wschemes, wfallback) = result, want
    assert (col.payload_words, col.desc.max_vec_words, col.desc.scheme_mask, fallback) == \
        (wcol.payload_words, wcol.desc.max_vec_words, wcol.desc.scheme_mask, wfallback)
    assert torch.equal(col.data[:col.payload_words], wcol.data[:wcol.payload_words])
    assert torch.equal(col.meta, wcol.meta) and torch.equal(schemes, wschemes)


SIZES = (1, 1024, 5000, 300_000, 77_777, 2_000_001)


@pytest.mark.gpu
@pytest.mark.parametrize("compact", [True, False])
@pytest.mark.parametrize("finish_on", ["same", "other"])
def test_deferred_encodes_in_any_order(cuda, compact, finish_on):
    """Several pending at once, on several streams, finished last to first,
    under the encode's stream or another one."""
    params = _params(1)
    vals = [_values(n, seed=n) for n in SIZES]
    want = [encode_column_learned_gpu(v, params, compact=compact) for v in vals]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(3)]
    pending = []
    for i, v in enumerate(vals):
        with torch.cuda.stream(streams[i % 3]):
            pending.append(encode_column_learned_gpu(v, params, compact=compact, defer=True))
    got = []
    for i in reversed(range(len(vals))):
        with torch.cuda.stream(streams[(i + (finish_on == "other")) % 3]):
            got.insert(0, pending[i].finish())
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        _check(g, w)
    ops.check_device_error()


@pytest.mark.gpu
@pytest.mark.parametrize("compact", [True, False])
def test_finished_column_outlives_its_encode(cuda, compact):
    """finish() under a busy stream: what the encode allocated is not handed out
    again while that stream still has to read it."""
    params, v = _params(2), _values(300_000, seed=9)
    want = encode_column_learned_gpu(v, params, compact=True)
    pending = encode_column_learned_gpu(v, params, compact=compact, defer=True)
    sizes = [pending.out.numel(), pending.meta.numel()]
    busy = torch.cuda.Stream()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(40_000_000)  # some 20 ms
        col, schemes, fallback = pending.finish()
        result = DeviceEncodedColumn(col.data.clone(), col.meta.clone(), col.n_values, col.layout, col.payload_words,
                                     col.desc.max_vec_words, col.desc.scheme_mask), schemes.clone(), fallback
    del pending, col, schemes
    junk = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for n in sizes for _ in range(4)]
    busy.synchronize()
    _check(result, want)
    del junk


@pytest.mark.gpu
def test_deferred_encodes_finished_by_threads(cuda):
    params = _params(3)
    vals = [_values(n, seed=n) for n in SIZES]
    want = [encode_column_learned_gpu(v, params) for v in vals]
    pending = [encode_column_learned_gpu(v, params, defer=True) for v in vals]
    got, failed = [None] * len(vals), []

    def work(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(t, len(vals), 2):
                    got[i] = pending[i].finish()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not failed and not any(t.is_alive() for t in threads)
    for g, w in zip(got, want):
        _check(g, w)
    ops.check_device_error()

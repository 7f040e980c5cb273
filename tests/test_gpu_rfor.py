"""GPU decode of the tile-based run-length format (RFOR): decode to HBM
restores the input and decode fused with a sum gives its exact uint64 sum, for
ragged tails, 32-bit fields and the reference benchmark's pattern; a tile
whose block was damaged is skipped and reported through the error word while
the other tiles decode."""
import numpy as np
import pytest

from fastlanesgpu_b200 import FlsError, datagen, ops
from fastlanesgpu_b200.column import RforColumn

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


def _cases():
    g = np.random.default_rng(15)
    yield "geometric-runs", datagen.geometric_runs(300 * 512 + 77, seed=13)
    yield "alternating", np.tile(np.repeat(np.array([200, 300], np.int32), 8), 4096)
    yield "short-runs", g.integers(0, 3, 64 * 512).astype(np.int32)
    yield "all-distinct", g.integers(-2**31, 2**31 - 1, 40 * 512 + 3).astype(np.int32)
    yield "constant", np.full(5000, -3, np.int32)
    yield "one-value", np.array([42], np.int32)
    yield "sorted-keys", datagen.sorted_geometric(200 * 512, p=0.3, seed=14)


CASES = list(_cases())


@pytest.mark.parametrize("name,vals", CASES, ids=[c[0] for c in CASES])
def test_rfor_decode_and_sum(cuda, name, vals):
    d = RforColumn.encode(vals).to_device()
    out = ops.rfor_decode(d).cpu().numpy()
    ops.check_device_error()
    assert np.array_equal(out, vals), name
    s = int(ops.rfor_decode_sum(d).cpu()[0]) & M64
    ops.check_device_error()
    assert s == int(vals.view(np.uint32).astype(np.uint64).sum()) & M64, name


def test_damaged_block_is_flagged_and_skipped(cuda):
    vals = datagen.geometric_runs(20 * 512, seed=16)
    col = RforColumn.encode(vals)
    bad = 7
    col.values[col.val_offsets[bad] + 2] = 600  # run count above the tile's 512 values
    d = col.to_device()
    import torch
    out = torch.full((vals.size,), -1, dtype=torch.int32, device=cuda)
    ops.rfor_decode(d, out=out)
    with pytest.raises(FlsError) as e:
        ops.check_device_error()
    assert "bad-vector-metadata" in str(e.value)
    got = out.cpu().numpy()
    keep = np.ones(vals.size, bool)
    keep[bad * 512:(bad + 1) * 512] = False
    assert np.array_equal(got[keep], vals[keep]) and (got[~keep] == -1).all()


def _ref_gpu():
    import ctypes
    import os
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "_ref",
                        "libref_rfor_gpu.so")
    if not os.path.exists(path):
        pytest.skip("libref_rfor_gpu.so not built (make -C oracle dropin needs the reference sources)")
    return ctypes.CDLL(path)


@pytest.mark.parametrize("name", ["geometric-runs", "alternating", "short-runs", "constant", "sorted-keys"])
def test_reference_gpu_decoder_reads_the_same_streams(cuda, name):
    """The reference's own GPU decoder (LoadRBinPack) decodes the library's
    streams to the input, as the library's decoder does.  (Tiles whose value
    block exceeds 512 words -- 512 runs of 32-bit values -- are outside what
    the reference loader copies, rlebinpack_kernel.cuh:52-61, and are not used
    here.)"""
    import ctypes

    import torch
    L = _ref_gpu()
    vals = dict(CASES)[name]
    col = RforColumn.encode(vals)
    d = col.to_device()
    out = torch.zeros(vals.size, dtype=torch.int32, device=cuda)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert L.ref_rfor_decode_gpu(p(d.values), p(d.val_offsets), p(d.run_lengths), p(d.rl_offsets),
                                 ctypes.c_uint32(vals.size), p(out)) == 0
    assert np.array_equal(out.cpu().numpy(), vals), name
    assert np.array_equal(ops.rfor_decode(d).cpu().numpy(), vals)


def test_decode_time_against_reference_gpu_decoder(cuda):
    """Both decoders on 2^26 values of geometric runs (mean 16) of values in
    [0, 2^16): each result equals the input, and the CUDA-event time of each
    (20 launches after 5, on the default stream) is printed."""
    import ctypes

    import torch
    L = _ref_gpu()
    n = 1 << 26
    vals = datagen.geometric_runs(n, mean_run=16.0, value_bits=16, seed=2804)
    d = RforColumn.encode(vals).to_device()
    out = torch.empty(n, dtype=torch.int32, device=cuda)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731

    def ref():
        assert L.ref_rfor_decode_gpu_launch(p(d.values), p(d.val_offsets), p(d.run_lengths), p(d.rl_offsets),
                                            ctypes.c_uint32(n), p(out)) == 0

    def ours():
        ops.rfor_decode(d, out=out)
    ms = {}
    for name, f in (("reference LoadRBinPack", ref), ("fls_rfor_decode_u32", ours)):
        out.fill_(-1)
        for _ in range(5):
            f()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(20):
            f()
        e1.record()
        torch.cuda.synchronize()
        ms[name] = e0.elapsed_time(e1) / 20
        ops.check_device_error()
        assert torch.equal(out.cpu(), torch.from_numpy(vals)), name
    print("\nRFOR decode of 2^26 values to HBM, ms per launch:",
          ", ".join(f"{k} {v:.4f}" for k, v in ms.items()))


@pytest.mark.parametrize("n", [1, 511, 512, 513, 512 * 40 + 3])
@pytest.mark.parametrize("mean_run", [1.0, 1.02, 8.0, 600.0])
def test_rfor_rows_and_alignment(cuda, n, mean_run):
    """From one run per value (16 groups of 32 runs) to one run per tile, into
    16-byte aligned outputs and into ones that are not."""
    import torch
    vals = datagen.geometric_runs(n, mean_run=mean_run, value_bits=30, seed=n).astype(np.int32)
    col = RforColumn.encode(vals).to_device()
    for shift in (0, 1, 3):
        buf = torch.full((n + shift + 4,), -1, dtype=torch.int32, device="cuda")
        ops.rfor_decode(col, out=buf[shift:shift + n])
        got = buf.cpu().numpy()
        assert np.array_equal(got[shift:shift + n], vals)
        assert np.all(got[:shift] == -1) and np.all(got[shift + n:] == -1)
    assert int(ops.rfor_decode_sum(col).cpu()[0]) == int(vals.view(np.uint32).astype(np.uint64).sum())
    ops.check_device_error()


def _block(x, bw):
    """A block of a stream: minimum 0, bw in every byte, count, fields LSB first."""
    bits = "".join(format(int(v), f"0{bw}b")[::-1] for v in x)
    bits += "0" * (-len(bits) % 32)
    return [0, bw * 0x01010101, len(x)] + [int(bits[i:i + 32][::-1], 2) for i in range(0, len(bits), 32)]


EMPTY_RUNS = {
    "first": [0, 512], "second": [2, 0, 510], "middle": [100, 0, 200, 0, 0, 212], "last": [300, 212, 0],
    "most": [0] * 31 + [1] + [0] * 200 + [256, 0, 255] + [0] * 277, "group-edge": [8] * 31 + [0, 0] + [8] * 33,
    "each-other": [2, 0] * 256, "trailing-group": [16] * 32 + [0] * 40,
}


@pytest.mark.parametrize("shift", [0, 1])
def test_empty_runs_cover_no_row(cuda, shift):
    """Runs of length 0, which no encoder here writes but the format holds:
    before, between, after and instead of others, on both sides of a group of
    32 runs; decode and sum expand the runs that are there."""
    import torch
    vs, rs, vo, ro, want = [512, 4, 0, 0], [512, 4, 0, 0], [], [], []
    for i, (name, lens) in enumerate(EMPTY_RUNS.items()):
        assert sum(lens) == 512 and len(lens) <= 512, name
        vals = np.arange(1, len(lens) + 1) * 3 + 1000 * i
        vo.append(len(vs))
        ro.append(len(rs))
        vs += _block(vals, 17)
        rs += _block(lens, 10)
        want.append(np.repeat(vals, lens))
    want = np.concatenate(want).astype(np.int32)
    u32 = lambda x: np.array(x, np.uint64).astype(np.uint32)  # noqa: E731
    for n in (want.size, want.size - 300):
        d = RforColumn(u32(vs), u32(rs), u32(vo + [len(vs)]), u32(ro + [len(rs)]), n).to_device()
        buf = torch.full((n + shift,), -1, dtype=torch.int32, device="cuda")
        ops.rfor_decode(d, out=buf[shift:])
        assert np.array_equal(buf[shift:].cpu().numpy(), want[:n])
        assert int(ops.rfor_decode_sum(d).cpu()[0]) == int(want[:n].astype(np.int64).sum())
    ops.check_device_error()


def test_tiles_of_every_run_count(cuda):
    """Tiles of 1..512 runs cut at random, so that both sides of every group of
    32 runs and of the count that changes the kernel's path are met, with the
    last tile whole and partial."""
    g = np.random.default_rng(64)
    tiles = []
    for count in g.permutation(np.arange(1, 513)):
        cuts = np.sort(g.permutation(511)[:count - 1]) + 1
        lens = np.diff(np.concatenate([[0], cuts, [512]]))
        tiles.append(np.repeat(g.integers(0, 1 << 20, count) * 2 + np.arange(count) % 2, lens))
    vals = np.concatenate(tiles).astype(np.int32)
    for n in (vals.size, vals.size - 1, vals.size - 300):
        d = RforColumn.encode(vals[:n]).to_device()
        assert np.array_equal(ops.rfor_decode(d).cpu().numpy(), vals[:n])
        assert int(ops.rfor_decode_sum(d).cpu()[0]) == int(vals[:n].astype(np.int64).sum())
    ops.check_device_error()

"""GPU encoder (fls_encode_column_gpu) against the host encoder: identical
payload words and metadata for every scheme, layout, tail length, per-vector
scheme arrays and round-to-4 widths; the encoded column decodes back to the
input."""
import numpy as np
import pytest

from fastlanesgpu_b200 import LAYOUT_NORMAL, LAYOUT_TRANSPOSED, ORDER_ORIGINAL, EncodedColumn, FlsError, datagen, ops
from fastlanesgpu_b200.column import encode_column_gpu

pytestmark = pytest.mark.gpu


def _families(n, seed):
    g = np.random.default_rng(seed)
    return {
        "uniform": datagen.uniform_bits(n, int(g.integers(1, 33)), seed=seed),
        "negative": g.integers(-2**31, 2**31, n, dtype=np.int64).astype(np.int32),
        "zipf": datagen.zipf_values(n, s=1.1, domain=1 << 20, seed=seed),
        "sorted": datagen.sorted_geometric(n, p=0.3, seed=seed),
        "runs": datagen.geometric_runs(n, mean_run=16.0, value_bits=16, seed=seed),
        "few_distinct": g.integers(-3, 4, n).astype(np.int32),
        "constant": np.full(n, -77, np.int32),
    }


def _compare(vals, schemes, layout, round4=False):
    import torch
    host = EncodedColumn.encode(vals, schemes, layout=layout, round4=round4)
    sch = schemes if isinstance(schemes, int) else torch.from_numpy(np.ascontiguousarray(schemes, np.uint8)).cuda()
    dcol = encode_column_gpu(torch.from_numpy(vals).cuda(), sch, layout=layout, round4=round4)
    gpu = dcol.to_host()
    ops.check_device_error()
    assert gpu.payload_words == host.payload_words
    assert np.array_equal(gpu.words[:host.payload_words], host.words[:host.payload_words])
    assert np.array_equal(gpu.meta, host.meta)
    assert gpu.max_vec_words == host.max_vec_words and gpu.scheme_mask == host.scheme_mask
    order = ORDER_ORIGINAL if layout == LAYOUT_TRANSPOSED else 0
    assert np.array_equal(ops.unpack_global(dcol, order=order).cpu().numpy()[:vals.size], vals)


@pytest.mark.parametrize("n", [1, 1000, 1025, 20 * 1024 + 5])
@pytest.mark.parametrize("scheme", [0, 1, 2, 3, 4])
def test_gpu_encoder_every_scheme(cuda, n, scheme):
    for name, vals in _families(n, 1000 + n + scheme).items():
        _compare(vals, scheme, LAYOUT_TRANSPOSED)
        if scheme in (0, 3, 4):  # bit-packed codes exist in both row orders
            _compare(vals, scheme, LAYOUT_NORMAL)


@pytest.mark.parametrize("seed", range(4))
def test_gpu_encoder_per_vector_schemes(cuda, seed):
    g = np.random.default_rng(seed)
    parts = list(_families(4096, seed).values())
    vals = np.concatenate([parts[i] for i in g.integers(0, len(parts), 24)] + [parts[0][:333]])
    nv = (vals.size + 1023) // 1024
    _compare(vals, g.integers(0, 5, nv).astype(np.uint8), LAYOUT_TRANSPOSED)
    _, best = ops.encode_exhaustive(vals)
    _compare(vals, best, LAYOUT_TRANSPOSED)


def test_gpu_encoder_round4(cuda):
    vals = datagen.uniform_bits(9 * 1024 + 9, 13, seed=5)
    _compare(vals, 0, LAYOUT_NORMAL, round4=True)
    _compare(vals, 0, LAYOUT_TRANSPOSED, round4=True)


def test_gpu_encoder_bad_scheme_is_flagged(cuda):
    """An out-of-range per-vector scheme is encoded as FOR and reported in the
    device error word (no fault)."""
    import torch
    vals = datagen.uniform_bits(3 * 1024, 9, seed=6)
    sch = torch.tensor([0, 7, 0], dtype=torch.uint8, device="cuda")
    dcol = encode_column_gpu(torch.from_numpy(vals).cuda(), sch, layout=LAYOUT_TRANSPOSED)
    with pytest.raises(FlsError):
        ops.check_device_error()
    host = EncodedColumn.encode(vals, 0, layout=LAYOUT_TRANSPOSED)
    got = dcol.to_host()
    assert np.array_equal(got.words[:host.payload_words], host.words[:host.payload_words])


def test_container_columns_decode_on_gpu(cuda, tmp_path):
    """Columns written to an encoded-column container and read back (host
    encoder through a file; GPU encoder through bytes) decode to the original
    values on the GPU."""
    import torch
    from fastlanesgpu_b200.column import encode_column_gpu
    from fastlanesgpu_b200.selector import training_corpus
    vals = training_corpus(300, seed=21)[: 300 * 1024 - 17]
    _, best = ops.encode_exhaustive(vals)
    col = EncodedColumn.encode(vals, best, layout=LAYOUT_TRANSPOSED)
    p = tmp_path / "col.flsc"
    col.save(str(p))
    back = EncodedColumn.load(str(p))
    out = ops.unpack_global(back.to_device(), ORDER_ORIGINAL).cpu().numpy()[: vals.size]
    assert np.array_equal(out, vals)
    g = encode_column_gpu(torch.from_numpy(vals).cuda(), torch.from_numpy(best).cuda()).to_host()
    g2 = EncodedColumn.from_bytes(g.to_bytes())
    want = int(vals.view(np.uint32).astype(np.uint64).sum())
    assert int(ops.query_aggregate(g2.to_device()).cpu()[0]) & 0xFFFFFFFFFFFFFFFF == want
    ops.check_device_error()


@pytest.mark.parametrize("bits", [0, 1, 9, 21, 22, 23, 31, 32])
@pytest.mark.parametrize("n_distinct", [1, 2, 255, 1023, 1024])
def test_gpu_encoder_dictionary_ranges(cuda, bits, n_distinct):
    """Dictionaries around the widest range whose sort keys carry the value's
    index (22 bits), from one distinct value to all 1024, in both layouts."""
    g = np.random.default_rng(bits * 1024 + n_distinct)
    lo, n = -(1 << 31) if bits == 32 else -12345, min(n_distinct, 1 << bits)
    pool = lo + np.unique(np.concatenate([[0, (1 << bits) - 1], g.integers(0, 1 << bits, 4 * n, dtype=np.int64)]))
    pool = np.concatenate([[pool[0], pool[-1]], g.permutation(pool[1:-1])])[:n]
    vals = np.concatenate([g.permutation(np.resize(pool, 1024)) for _ in range(9)] + [pool[:1]]).astype(np.int32)
    for layout in (LAYOUT_NORMAL, LAYOUT_TRANSPOSED):
        _compare(vals, 4, layout)


@pytest.mark.parametrize("n_vec", [7, 8, 9, 8 * 32 + 1, 8 * 128, 8 * 256, 8 * 257 + 3, 8 * 1500 + 5])
def test_gpu_encoder_offsets_over_many_tiles(cuda, n_vec):
    """Offsets, total, largest vector and scheme mask around the tiles of 8
    vectors, the scan's groups of 32 and rounds of 256 tiles, and past the
    resident CTAs."""
    g = np.random.default_rng(n_vec)
    vals = (g.integers(0, 1 << 31, (n_vec, 1024)) >> g.integers(0, 31, (n_vec, 1))).astype(np.int32).reshape(-1)[:-11]
    schemes = np.where(g.integers(0, 50, n_vec) == 0, g.integers(0, 5, n_vec), 0).astype(np.uint8)
    _compare(vals, schemes, LAYOUT_TRANSPOSED)


def _encode_waits(values, scheme=0, params=None, ctas=1, scan_polls=1 << 22, tile_polls=1 << 22):
    """The encoder with few CTAs and short waits: (words, metadata, info)."""
    import torch
    from fastlanesgpu_b200._lib import check, lib
    n = values.numel()
    cap = int(lib().fls_encode_bound_words(n)) + 4
    out = torch.full((cap,), -1, dtype=torch.int32, device="cuda")
    meta = torch.full(((n + 1023) // 1024 * 4,), -1, dtype=torch.int32, device="cuda")
    info = torch.full((4,), 99, dtype=torch.int64, device="cuda")
    ws = torch.empty(int(lib().fls_encode_learned_workspace_bytes(n)), dtype=torch.uint8, device="cuda")
    check(lib().fls_selftest_encode_waits(values.data_ptr(), n, scheme, params.data_ptr() if params is not None else None,
                                          out.data_ptr(), cap, meta.data_ptr(), info.data_ptr(), ws.data_ptr(),
                                          ws.numel(), ctas, scan_polls, tile_polls,
                                          torch.cuda.current_stream().cuda_stream), "fls_selftest_encode_waits")
    return out, meta, info.tolist()


@pytest.mark.parametrize("ctas", [1, 2, 3])
@pytest.mark.parametrize("n_vec", [1, 8, 9, 8 * 33 + 5, 8 * 300])
def test_encoder_by_few_ctas(cuda, ctas, n_vec):
    """However few CTAs of the encoder are on the GPU, one included, the column
    is encoded whole and as by many, without a timeout."""
    import torch
    from fastlanesgpu_b200 import _lib
    from fastlanesgpu_b200.column import encode_column_learned_gpu
    n = n_vec * 1024 - 7
    for scheme, name in enumerate(("uniform", "sorted", "runs", "constant", "zipf")):
        v = torch.from_numpy(_families(n, n_vec)[name]).cuda()
        want = encode_column_gpu(v, scheme)
        out, meta, info = _encode_waits(v, scheme, ctas=ctas)
        assert info[:3] == [want.payload_words, want.desc.max_vec_words, want.desc.scheme_mask]
        assert torch.equal(out[:info[0]], want.data[:info[0]]) and torch.equal(meta, want.meta)
    params = torch.randn(_lib.MLP_N_PARAMS, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n_vec))
    want, _, fallbacks = encode_column_learned_gpu(v, params, threshold=0.9, kappa=0.0)
    out, meta, info = _encode_waits(v, params=params, ctas=ctas)
    assert info == [want.payload_words, want.desc.max_vec_words, want.desc.scheme_mask, fallbacks]
    assert torch.equal(out[:info[0]], want.data[:info[0]]) and torch.equal(meta, want.meta)
    ops.check_device_error()

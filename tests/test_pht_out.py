"""build_pht into a table that the caller passes: refused, before anything is
enqueued, where the table's slots would not lie in it; otherwise zeroed whole
and filled, whatever its size and type."""
import pytest
import torch

from fastlanesgpu_b200 import ops


@pytest.mark.parametrize("payload", [False, True])
@pytest.mark.parametrize("make", [
    lambda size: torch.empty(size - 1, dtype=torch.int32),
    lambda size: torch.empty(0, dtype=torch.int32),
    lambda size: torch.empty(2 * size - 1, dtype=torch.int16),
    lambda size: torch.empty(2 * size, dtype=torch.int32)[::2],
    lambda size: torch.empty(size, 2, dtype=torch.int32).t(),
], ids=["short", "empty", "short-int16", "strided", "transposed"])
def test_table_that_does_not_hold_the_slots_is_refused(make, payload):
    keys = torch.arange(4, dtype=torch.int32)
    size = 200 if payload else 100
    with pytest.raises(ValueError):
        ops.build_pht(keys, 100, vals=keys if payload else None, out=make(size))


@pytest.mark.gpu
@pytest.mark.parametrize("payload", [False, True])
@pytest.mark.parametrize("extra,dtype", [(0, torch.int32), (1, torch.int32), (777, torch.int32), (0, torch.int64),
                                         (0, torch.float32)])
def test_table_given(cuda, payload, extra, dtype):
    g = torch.Generator(device="cuda")
    g.manual_seed(extra)
    n = 5003
    keys = torch.randperm(n, device="cuda", generator=g).int()[:4000]
    vals, filt = keys * 3 + 1, keys % 4
    size = 2 * n if payload else n
    want = ops.build_pht(keys, n, vals=vals if payload else None, filt=filt, filter_eq=2)
    store = torch.full((size + extra + 64,), 7, device="cuda").to(dtype)
    out = store[:size + extra]
    got = ops.build_pht(keys, n, vals=vals if payload else None, filt=filt, filter_eq=2, out=out)
    assert got.data_ptr() == out.data_ptr()
    words = out.view(torch.int32)
    assert torch.equal(words[:size], want) and int(words[size:].abs().sum()) == 0
    assert torch.equal(store[size + extra:], torch.full((64,), 7, device="cuda").to(dtype))
    ops.check_device_error()

"""bench.py where the reference's compiled code is absent: its reference arm says
so in one line, and the product's arm checks its result against the oracle's
restatement on columns that numpy unpacks."""
import argparse
import types

import numpy as np
import pytest
import torch

import bench
from fastlanesgpu_b200 import EncodedColumn, datagen


@pytest.fixture
def no_reference(monkeypatch, oracle):
    import oracle as orc

    def absent():
        raise FileNotFoundError("libflsref.so not built")

    monkeypatch.setattr(orc, "Reference", absent)


def test_unpack_every_width():
    g = np.random.default_rng(3)
    for bw in range(33):
        v = (g.integers(0, 1 << 32, 3 * 1024 + 5, dtype=np.uint64) & np.uint64((1 << bw) - 1)).astype(np.uint32)
        col = EncodedColumn.uniform(v.view(np.int32), bw=bw)
        assert np.array_equal(bench.unpack_column(np.ascontiguousarray(col.words).view(np.uint32), bw, v.size),
                              v.view(np.int32)), bw


@pytest.mark.parametrize("workload", ["q11", "q21", "q41", "decode"])
def test_reference_arm_says_why(no_reference, workload):
    a = argparse.Namespace(workload=workload, decode_scheme="for", decode_width=32, decode_bw=8, rows=1024)
    d = bench.run_reference(a, None)
    assert set(d) == {"impl", "unavailable"} and d["impl"] == "reference" and "\n" not in d["unavailable"]


def test_result_check_by_the_oracle(no_reference, oracle):
    n = 5 * 1024 + 77
    t = datagen.lineorder_q11(n, seed=8)
    names = ("date", "discount", "quantity", "price")
    f = datagen.Q11_FILTER
    want = oracle.filter_agg(*(t[k] for k in names), *f["date"], *f["discount"], f["quantity"][1] + 1)
    ctx = {"workload": "q11", "tabs": None, "res": torch.tensor([want]),
           "hcols": [EncodedColumn.uniform(t[k], bw=datagen.Q11_BITS[k]) for k in names]}
    a = types.SimpleNamespace(rows=n, decode_bw=8)
    cb = bench.cpu_baseline(a, ctx, 0.1)
    assert cb["unavailable"] and cb["result_equal"] is True
    ctx["res"] = torch.tensor([want + 1])
    assert bench.cpu_baseline(a, ctx, 0.1)["result_equal"] is False

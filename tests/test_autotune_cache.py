"""The autotuner's cache (no GPU): entries written for an earlier meaning of the
knobs are not used, entries of this version are."""
import json
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from bcl_b200 import autotune


def operands(kind):
    a = SimpleNamespace(dtype=np.dtype(np.float32), tm=512, tn=512, gm=4, gn=4, m=2048, n=2048, nnz=lambda: 30000)
    b = SimpleNamespace(torch_dtype=torch.float32, tn=128, gn=1, n=128) if kind == "spmm" else a
    return a, b


def unversioned(a, b, kind):
    if kind == "spmm":
        return "spmm|torch.float32|t512x512x128|g4x4x1|m11|n7|nnz15"
    return f"{kind}|<f4|t512x512x512|g4x4x4|a15|b15"


@pytest.mark.parametrize("kind", ["spgemm", "spmm", "learned"])
def test_entries_of_other_kernels_are_not_used(tmp_path, monkeypatch, kind):
    monkeypatch.setenv("BCLX_CACHE", str(tmp_path))
    a, b = operands(kind)
    with open(autotune.cache_path(), "w") as f:
        json.dump({unversioned(a, b, kind): {"params": {"grab": 1, "blocks_per_sm": 4, "long_seg": 32}}}, f)
    assert autotune.signature(a, b, kind).endswith(unversioned(a, b, kind))
    assert autotune.lookup(a, b, kind) is None


@pytest.mark.parametrize("kind", ["spgemm", "spmm", "learned"])
def test_entries_of_this_version_are(tmp_path, monkeypatch, kind):
    monkeypatch.setenv("BCLX_CACHE", str(tmp_path))
    a, b = operands(kind)
    autotune._store({autotune.signature(a, b, kind): {"params": {"grab": 2}}})
    assert autotune.lookup(a, b, kind) == {"grab": 2}

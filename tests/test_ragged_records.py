"""Descriptor arrays built for a whole batch at once hold what the per-instance records do (CPU)."""
import numpy as np
import pytest
import torch

from blast_gb300 import desc
from blast_gb300.ragged import Packed, _workspace_offsets


@pytest.mark.parametrize("rows,cols", [([], []), ([1], [1]), ([0, 3, 0, 2], [0, 3, 5, 1]), ([5, 4, 7], [5, 4, 7])])
@pytest.mark.parametrize("dtype", [torch.float64, torch.int32])
def test_records_match_record(rows, cols, dtype):
    p = Packed(rows, cols, "cpu", dtype=dtype)
    want = np.zeros(len(rows), dtype=desc.MAT_DTYPE)
    for i in range(len(rows)):
        want[i] = p.record(i)
    assert np.array_equal(p.records(), want)
    assert [int(x) for x in p.ptrs()] == [p.ptr(i) for i in range(len(rows))]


@pytest.mark.parametrize("n", [[], [4], [3, 9, 3, 1, 9]])
def test_workspace_offsets(n):
    n = np.array(n, dtype=np.int64)
    order = np.argsort(-n, kind="stable")
    off, total = _workspace_offsets(lambda k: 16 * k, n, order)
    at = 0
    for i in order:
        assert off[i] == at
        at += 16 * int(n[i])
    assert total == at

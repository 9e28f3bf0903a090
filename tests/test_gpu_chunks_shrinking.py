"""Chunks of three frames, the first one split and the end shrinking (1, 2, 3, 2, 1: test_host_code.py pins the budgets that
give them), through one and two chunk slots: the same rows as one chunk."""
import pytest

import test_gpu_chunks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget_mb,slots", [("40", "1"), ("76", "2")])
def test_shrinking_chunks_match_one_chunk(lib, orc, tmp_path, monkeypatch, budget_mb, slots):
    test_gpu_chunks.test_many_chunks_match_one_chunk(lib, orc, tmp_path, monkeypatch, budget_mb, slots)

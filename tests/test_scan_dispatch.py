"""Which steps run the scans of recurrent layers as matrix products over chunks: by sizes alone, so without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from atoma_infer_b200.csrc.ops import CudaOps


LONG = [([127], False), ([128], True), ([2048], True), ([256 * 128], True), ([256 * 128 + 1], False)]


def check(lengths, chunked, tokens):
    ctx = SimpleNamespace(T=sum(lengths), S=len(lengths), max_tokens_per_entry=max(lengths))
    chunks = CudaOps._matrix_scan_chunks(CudaOps, ctx, tokens)
    assert bool(chunks) == chunked
    if chunked:
        assert chunks >= sum(-(-n // CudaOps.MATRIX_SCAN_CHUNK) for n in lengths)


@pytest.mark.parametrize("lengths,chunked", LONG + [
    ([128] + [1] * 16, True), ([128] + [1] * 17, True), ([128] + [1] * 18, False), ([128] + [1] * 60, False), ([128] + [1] * 250, False),
    ([512] + [1] * 60, True), ([300] + [1] * 60, False), ([1988] + [1] * 60, True), ([200] + [20] * 60, True), ([128] + [7] * 500, False),
])
def test_state_space_prompts_beside_many_single_tokens_go_in_order(lengths, chunked):
    check(lengths, chunked, CudaOps.MATRIX_SCAN_TOKENS)


@pytest.mark.parametrize("lengths,chunked", LONG + [([128] + [1] * 60, True), ([128] + [1] * 126, True), ([128] + [1] * 127, False), ([300] + [1] * 250, True)])
def test_matrix_memory_prompts_beside_many_single_tokens_go_in_order(lengths, chunked):
    check(lengths, chunked, CudaOps.MATRIX_SCAN_TOKENS_OTHER)


@pytest.mark.parametrize("singles", [126, 127, 250])
def test_prompts_with_a_decay_per_row_beside_many_single_tokens_go_in_order(singles):
    lengths = [128] + [1] * singles
    ctx = SimpleNamespace(T=sum(lengths), S=len(lengths))
    ops = SimpleNamespace(matrix_scan=True, MATRIX_SCAN_TOKENS_OTHER=2, ROW_SCAN_CHUNK=64, ROW_SCAN_SCRATCH=1 << 20, launches=0)
    lib = SimpleNamespace(gla_row_scan_head_floats=lambda *args: 64, gla_scan_scratch_floats=lambda *args: 0)
    rows = CudaOps._row_scan(ops, lib, "gla", (), torch.empty(0, dtype=torch.bfloat16), ctx, torch.empty(1), 4, 64, 64, 64, 2)
    assert (rows is None) == (singles > 126)

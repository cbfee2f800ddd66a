"""Which steps run the state-space and matrix-memory scans as matrix products over chunks: by sizes alone, so without a GPU."""
from types import SimpleNamespace

import pytest

from atoma_infer_b200.csrc.ops import CudaOps


@pytest.mark.parametrize("lengths,chunked", [
    ([127], False), ([128], True), ([2048], True), ([256 * 128], True), ([256 * 128 + 1], False),
    ([128] + [1] * 16, True), ([128] + [1] * 17, True), ([128] + [1] * 18, False), ([128] + [1] * 60, False), ([128] + [1] * 250, False),
    ([512] + [1] * 60, True), ([300] + [1] * 60, False), ([1988] + [1] * 60, True), ([200] + [20] * 60, True), ([128] + [7] * 500, False),
])
def test_prompts_beside_many_single_tokens_go_in_order(lengths, chunked):
    ctx = SimpleNamespace(T=sum(lengths), S=len(lengths), max_tokens_per_entry=max(lengths))
    chunks = CudaOps._matrix_scan_chunks(CudaOps, ctx)
    assert bool(chunks) == chunked
    if chunked:
        assert chunks >= sum(-(-n // CudaOps.MATRIX_SCAN_CHUNK) for n in lengths)

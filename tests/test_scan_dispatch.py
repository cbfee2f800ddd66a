"""Which steps run the scans of recurrent layers as matrix products over chunks, and other rules by sizes alone: without a GPU."""
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


@pytest.mark.parametrize("dtype,N,P,blocks", [("bfloat16", 128, 64, 14), ("bfloat16", 96, 64, 14), ("bfloat16", 64, 64, 6), ("bfloat16", 16, 64, 3),
                                              ("bfloat16", 32, 128, 14), ("bfloat16", 16, 128, 3), ("bfloat16", 256, 32, 2),
                                              ("float32", 128, 64, 3), ("float32", 64, 128, 14), ("float32", 31, 128, 3), ("float32", 16, 32, 2)])
def test_decode_steps_of_the_state_space_mixer_in_two_launches(dtype, N, P, blocks):
    """Up to so many heads of all requests a multiprocessor; beyond, the call is refused before anything is launched."""
    sms, heads = 148, 4
    taken = []
    ops = SimpleNamespace(num_sms=sms, _token_step_blocks=CudaOps._token_step_blocks, _rows=lambda t, what: (None, 0), launches=0,
                          _mixers=lambda: SimpleNamespace(ssm_token_step_takes=lambda *args: taken.append(args) or 0))
    for S, takes in ((1, True), (blocks * sms // heads, True), (blocks * sms // heads + 1, False)):
        taken.clear()
        state = torch.empty(1, heads, N, P).expand(S, heads, N, P)
        u = torch.empty(S, 8, dtype=getattr(torch, dtype))
        ctx = SimpleNamespace(decode_only=True, T=S, S=S)
        CudaOps.ssm_token_step(ops, u, u, u, torch.empty(4, 8), None, None, None, None, None, state, None, 1, 1, 1e-5, ctx, u)
        assert bool(taken) == takes


@pytest.mark.parametrize("dtype,longest,one_pass", [("bfloat16", 15, False), ("bfloat16", 16, True), ("bfloat16", 127, True),
                                                    ("float32", 16, False), ("float32", 127, False), ("float32", 128, True), ("float32", 2048, True)])
def test_selective_scans_of_float32_go_in_order_below_the_chunks_of_time(dtype, longest, one_pass):
    """The one pass sums a token's states in another order, and it is chosen by the whole step: where chunks of time are not, a float32
    request must not see what else the step brings."""
    ops = SimpleNamespace(selective_prompt=None, num_sms=148, SCAN_CHUNK_FROM=CudaOps.SCAN_CHUNK_FROM)
    ctx = SimpleNamespace(T=longest, S=1, max_tokens_per_entry=longest)
    assert CudaOps._selective_in_order(ops, ctx, 4096, 16, getattr(torch, dtype)) == one_pass


@pytest.mark.parametrize("nstate,inner,lengths,one_pass", [
    (16, 2048, [2048], True), (8, 2048, [2048], False), (8, 4096, [2048], True), (16, 1024, [3000], False), (8, 1024, [1000], True),
    (16, 4096, [128] + [1] * 20, True), (8, 4096, [1000] + [1] * 40, True), (16, 4096, [16] * 8, False), (8, 4096, [64] * 8, False),
    (16, 6144, [16] * 2, False), (8, 4096, [20] * 3, False), (8, 6144, [67, 75, 46], True), (16, 4096, [16], True)])
def test_selective_scans_in_one_pass_where_that_was_measured_to_be_shorter(nstate, inner, lengths, one_pass):
    ops = SimpleNamespace(selective_prompt=None, num_sms=148, SCAN_CHUNK_FROM=CudaOps.SCAN_CHUNK_FROM)
    ctx = SimpleNamespace(T=sum(lengths), S=len(lengths), max_tokens_per_entry=max(lengths))
    assert CudaOps._selective_in_order(ops, ctx, inner, nstate, torch.bfloat16) == one_pass


@pytest.mark.parametrize("N,K,takes", [(1024, 1024, True), (1023, 1024, False), (512, 2048, True), (4096, 1020, False), (1024, 1026, False),
                                       (18944, 1024, True), (18945, 1024, False), (32768, 2048, True), (32769, 2048, False), (32768, 2044, False)])
def test_float32_products_on_the_tensor_cores_by_the_weight_alone(N, K, takes):
    w, ops = torch.empty(N, K, device="meta"), SimpleNamespace(tc_f32=True, num_sms=148)
    for M in (1, 17, 4096):
        x, y = torch.empty(M, K, device="meta"), torch.empty(M, N, device="meta")
        assert CudaOps._f32_on_tcgen05(ops, x, w, y) == takes

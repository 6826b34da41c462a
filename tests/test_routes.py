"""Which kernel a call goes to, on the CPU with the kernels replaced by recorders: a kernel that does not take a size says so
before it is launched, and the one that takes every size gets the call."""
from types import SimpleNamespace

import pytest
import torch

from supersonic_b200.csrc import ops
from supersonic_b200.csrc.fast_sets import FastKernels
from supersonic_b200.csrc.kernel_sets import PlainKernels


@pytest.fixture
def calls(monkeypatch):
    seen = []
    for name in ("latent_attention_mma", "latent_attention_tc", "attention_plain", "attention_f32_prompt"):
        monkeypatch.setattr(ops, name, lambda *a, _n=name, **k: seen.append(_n))
    monkeypatch.setattr(ops, "sm_count", lambda *a: 148)
    return seen


def batch_of(n_seqs, max_new, n_tokens=None, max_total=4000, kv_pages=32):
    none = torch.empty(0, dtype=torch.int32)
    return SimpleNamespace(n_seqs=n_seqs, max_new=max_new, is_decode=max_new == 1, n_tokens=n_tokens or n_seqs * max_new,
                           max_total=max_total, kv_pages=kv_pages, cu_new=none, seq_start=none, seq_slot=none,
                           slot_of_token=none, pos=none)


def test_latent_attention_of_more_row_tiles_than_a_grid_counts(calls):
    """tcgen05 tiles are 128 (token, head) rows, and a grid's y side counts to 65,535 of them: 128 heads over 65,536 tokens
    are one too many and go to the kernel that counts them along x."""
    heads, rank, rot = 128, 32, 16
    bf16 = lambda *shape: torch.empty(shape, dtype=torch.bfloat16)  # noqa: E731
    q, cache, out = bf16(1, heads * (rank + rot)), bf16(1, 1, 64, rank + rot), bf16(1, heads * rank)
    for max_new in (64, 65535, 65536):
        FastKernels().latent_attention(q, cache, batch_of(1, max_new), None, out, heads, rank, rot, 6, None, 1.0, None)
    assert calls == ["latent_attention_tc", "latent_attention_tc", "latent_attention_mma"]
    assert ops.latent_attention_tc_ok(q, cache, out, heads, rank + rot, rank, 6, 65535)
    assert not ops.latent_attention_tc_ok(q, cache, out, heads, rank + rot, rank, 6, 65536)


@pytest.mark.parametrize("heads,rank,rot,batch,tc", [
    (16, 512, 64, batch_of(1, 7, kv_pages=32), False), (16, 512, 64, batch_of(1, 8, kv_pages=2), True),
    (16, 512, 64, batch_of(1, 64, kv_pages=1), False), (16, 512, 64, batch_of(8, 64, kv_pages=1), True),
    (8, 256, 32, batch_of(1, 64, kv_pages=2), False), (8, 256, 32, batch_of(1, 16, kv_pages=4), True),
    (8, 256, 32, batch_of(8, 64, kv_pages=1), False), (8, 256, 32, batch_of(8, 128, kv_pages=2), True),
    (8, 256, 32, batch_of(700, 1, kv_pages=32), False)])
def test_latent_attention_goes_to_tcgen05_where_pages_or_rows_pay_for_its_start(calls, heads, rank, rot, batch, tc):
    bf16 = lambda *shape: torch.empty(shape, dtype=torch.bfloat16)  # noqa: E731
    q, cache, out = bf16(1, heads * (rank + rot)), bf16(1, 1, 64, rank + rot), bf16(1, heads * rank)
    for kernels in (FastKernels(), FastKernels(deterministic=True)):
        kernels._buffer = lambda *a, **k: None
        kernels.latent_attention(q, cache, batch, None, out, heads, rank, rot, 6, None, 1.0, None)
    assert calls == ["latent_attention_tc" if tc else "latent_attention_mma", "latent_attention_mma"]


def test_float32_prompts_of_more_sequences_than_a_grid_counts(calls):
    """Tiles of 64 (token, head) rows have a sequence each along the grid's z side, which counts to 65,535."""
    q, out = torch.empty(8, 128), torch.empty(8, 128)
    cache = torch.empty(1, 1, 64, 64)
    for n_seqs in (64, 65535, 65536):
        PlainKernels().attention(q, cache, cache, batch_of(n_seqs, 16), None, out, 2, 1, 64, 6, None, 1.0)
    assert calls == ["attention_f32_prompt", "attention_f32_prompt", "attention_plain"]


@pytest.mark.parametrize("head_dim,batch,shared", [
    (64, batch_of(1, 35), False), (64, batch_of(1, 36), True), (128, batch_of(1, 31), False), (128, batch_of(1, 32), True),
    (64, batch_of(1, 32, max_total=128), False), (64, batch_of(4, 16, max_total=128), True),
    (128, batch_of(64, 8, n_tokens=71), False),                      # one short prompt among 63 single tokens
    (64, batch_of(3, 500, n_tokens=890), True), (128, batch_of(16, 2048, n_tokens=18000), True)])
def test_float32_prompts_share_the_fetch_of_a_key_where_their_rows_fill_the_blocks(calls, head_dim, batch, shared):
    q, out = torch.empty(8, 32 * head_dim), torch.empty(8, 32 * head_dim)
    cache = torch.empty(1, 8, 64, head_dim)
    PlainKernels().attention(q, cache, cache, batch, None, out, 32, 8, head_dim, 6, None, 1.0)
    assert calls == ["attention_f32_prompt" if shared else "attention_plain"]


@pytest.mark.parametrize("n_seqs,n_kv,most,usual,blocks", [
    (1, 4, 15, None, 8), (3, 4, 15, None, 8), (4, 4, 15, None, 4), (9, 4, 15, None, 4), (10, 4, 15, None, 2), (18, 4, 15, None, 2), (19, 4, 15, None, 1),
    (1, 4, 7, None, 4), (10, 4, 7, None, 1), (1, 4, 3, None, 1), (8, 2, 5, 3, 4), (13, 2, 5, 3, 1), (2, 4, 9, 5, 8), (8, 4, 9, 5, 4)])
def test_blocks_that_share_a_decode_steps_pages(calls, n_seqs, n_kv, most, usual, blocks):
    assert FastKernels()._shares(batch_of(n_seqs, 1), n_kv, most, usual) == blocks
    assert FastKernels()._shares(batch_of(2, 1), 8, 31, small=True) == 8 and FastKernels()._shares(batch_of(2, 1), 8, 31) == 4
    assert FastKernels(deterministic=True)._shares(batch_of(n_seqs, 1), n_kv, most, usual) == 1
    assert FastKernels()._shares(batch_of(n_seqs, 2), n_kv, most, usual) == 1

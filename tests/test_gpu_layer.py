"""Attention.forward (the reference-facing layer) on the GPU against the oracle's
restatement of the same control flow."""
import pytest
import torch

from conftest import assert_close_to_oracle, ticking
from nano_vllm_b200 import _lib, attention as A, context as C, workloads as W
from oracle import paged_attention_ref as R

pytestmark = pytest.mark.gpu


def test_prefill_then_decode_through_the_layer(cuda):
    hq, hkv, d = 16, 8, 128
    case = W.make_prefill_case(31, 8, 100, 700, hq, hkv, d)
    dev = case.to(cuda)
    layer = A.Attention(hq, d, case.scale, hkv)
    assert layer.k_cache.numel() == 0
    layer.k_cache, layer.v_cache = dev.k_cache, dev.v_cache
    C.set_context(True, dev.cu_seqlens_q, dev.cu_seqlens_k, case.max_seqlen_q, case.max_seqlen_k,
                  dev.slot_mapping, None, dev.block_tables)
    n = case.q.shape[0]
    o = layer(dev.q.view(n, -1), dev.k.view(n, -1), dev.v.view(n, -1))
    C.set_context(True, case.cu_seqlens_q, case.cu_seqlens_k, case.max_seqlen_q, case.max_seqlen_k,
                  case.slot_mapping, None, case.block_tables)
    ref = R.attention_forward_ref(case.q, case.k, case.v, case.k_cache, case.v_cache, C.get_context(), case.scale)
    assert o.shape == (n, hq * d)
    assert_close_to_oracle(o.view(n, hq, d), ref, "layer prefill")

    # one decode step on top of the prefilled cache
    B = case.cu_seqlens_k.numel() - 1
    lens = (case.cu_seqlens_k[1:] - case.cu_seqlens_k[:-1]) + 1
    g = torch.Generator().manual_seed(32)
    q1 = torch.randn(B, hq, d, generator=g).bfloat16()
    k1 = torch.randn(B, hkv, d, generator=g).bfloat16()
    v1 = torch.randn(B, hkv, d, generator=g).bfloat16()
    bt = case.block_tables
    slots = torch.zeros(B, dtype=torch.int32)
    for b in range(B):
        pos = int(lens[b]) - 1
        if pos % 256 == 0:  # needs a fresh block: take a spare one
            free = (set(range(case.k_cache.shape[0])) - set(bt[bt >= 0].tolist())).pop()
            if pos // 256 >= bt.shape[1]:
                bt = torch.cat([bt, torch.full((B, 1), -1, dtype=torch.int32)], dim=1)
            bt[b, pos // 256] = free
        slots[b] = int(bt[b, pos // 256]) * 256 + pos % 256
    C.set_context(False, slot_mapping=slots.to(cuda), context_lens=lens.to(torch.int32).to(cuda),
                  block_tables=bt.to(cuda))
    o1 = layer(q1.to(cuda).view(B, -1), k1.to(cuda).view(B, -1), v1.to(cuda).view(B, -1))
    C.set_context(False, slot_mapping=slots, context_lens=lens.to(torch.int32), block_tables=bt)
    ref1 = R.attention_forward_ref(q1, k1, v1, case.k_cache, case.v_cache, C.get_context(), case.scale)
    C.reset_context()
    assert_close_to_oracle(o1.view(B, hq, d), ref1, "layer decode")
    assert torch.equal(dev.k_cache.cpu().view(torch.int16), case.k_cache.view(torch.int16))


def test_other_threads_run_while_launches_wait_for_the_queue(cuda):
    """More calls than the device's queue takes while it is busy: the last ones wait, the interpreter does not."""
    case = W.make_decode_case(33, 2, 1, 1, 16, 8, 128, context_lens=[300, 17])
    dev = case.to(cuda)
    layer = A.Attention(16, 128, case.scale, 8)
    layer.k_cache, layer.v_cache = dev.k_cache, dev.v_cache
    qkv = [t.view(2, -1) for t in (dev.q, dev.k_new, dev.v_new)]
    C.set_context(False, slot_mapping=dev.slot_mapping, context_lens=dev.context_lens, block_tables=dev.block_tables)
    first = layer(*qkv)
    torch.cuda.synchronize()

    def many():
        torch.cuda._sleep(1_000_000_000)  # half a second
        for _ in range(4000):
            last = layer(*qkv)
        return last

    seconds, ticks = ticking(many)
    torch.cuda.synchronize()
    last = layer(*qkv)
    C.reset_context()
    assert seconds > 0.2, "the queue took every launch"
    assert ticks > 40 * seconds, f"another thread ran {ticks} times in {seconds:.2f} s"
    assert torch.equal(first, last)


def test_shapes_without_kv_heads_are_refused(cuda):
    """No key heads, or a cache of none: an error from every entry point, as from any other shape the
    kernels do not take."""
    bf = dict(dtype=torch.bfloat16, device=cuda)
    i32 = dict(dtype=torch.int32, device=cuda)
    q, none = torch.zeros(2, 4, 128, **bf), torch.zeros(2, 0, 128, **bf)
    cache, empty = torch.zeros(3, 256, 1, 128, **bf), torch.zeros(3, 256, 0, 128, **bf)
    slots, lens, table = torch.zeros(2, **i32), torch.ones(2, **i32), torch.zeros(2, 1, **i32)
    flat = torch.zeros(1, **bf).expand(3, 256, 1, 128)  # a plane whose tokens lie zero elements apart
    with pytest.raises(RuntimeError):
        A.store_kvcache(none, none, flat, flat, slots)
    with pytest.raises(RuntimeError):
        A.decode_paged(q, empty, empty, lens, table, 0.1)
    with pytest.raises(RuntimeError):
        A.decode_step(q, none, none, empty, empty, slots, lens, table, 0.1)
    with pytest.raises(RuntimeError):
        A.qk_norm_rope_store(torch.zeros(2, 512, **bf), torch.zeros(2, dtype=torch.int64, device=cuda), None, None,
                             torch.zeros(8, 128, device=cuda), 1e-6, slots, cache, cache, 4, 0, 128)
    layer = A.Attention(4, 128, 0.1, 0)
    layer.k_cache = layer.v_cache = flat
    for prefill in (False, True):
        C.set_context(prefill, cu_seqlens_q=slots, cu_seqlens_k=slots, max_seqlen_q=1, max_seqlen_k=1, slot_mapping=slots,
                      context_lens=lens, block_tables=None if prefill else table)
        with pytest.raises((RuntimeError, AssertionError)):
            layer(q.view(2, -1), none.view(2, 0), none.view(2, 0))
    C.reset_context()
    torch.cuda.synchronize()
    assert _lib.read_status() == 0

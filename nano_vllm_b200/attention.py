"""Attention layer of nano-vllm on the B200 kernels: the host side of the C ABI.

Same surface as nanovllm/layers/attention.py:32-79 — ``store_kvcache(key, value, k_cache,
v_cache, slot_mapping)`` and ``Attention(num_heads, head_dim, scale, num_kv_heads)`` with the
``k_cache`` / ``v_cache`` attributes that the model runner binds
(nanovllm/engine/model_runner.py:145-149) and ``forward(q, k, v)`` driven by the per-step
context — but every device operation goes through libnvllm_b200.so.  Tensors must live on a
CUDA device and be bf16; anything else raises (there is no CPU or eager fallback).
"""
from __future__ import annotations

from typing import Callable

import torch
from torch import nn

from . import _lib
from . import context as _own_context

BLOCK_SIZE = 256

_get_context: Callable[[], object] = _own_context.get_context


def use_context_getter(getter: Callable[[], object]) -> None:
    """Makes ``Attention.forward`` read its metadata from another module's ``get_context``
    (nano-vllm's ``nanovllm.utils.context.get_context`` when running inside that engine)."""
    global _get_context
    _get_context = getter


def _stream(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


def _require_cuda_bf16(name: str, t: torch.Tensor) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{name} must be a CUDA tensor (nano_vllm_b200 has no CPU path)")
    if t.dtype != torch.bfloat16:
        raise RuntimeError(f"{name} must be bfloat16, got {t.dtype}")


def _require_i32(name: str, t: torch.Tensor) -> None:
    if not t.is_cuda or t.dtype != torch.int32 or (t.dim() > 0 and t.stride(-1) != 1):
        raise RuntimeError(f"{name} must be a CUDA int32 tensor with unit inner stride")


# ---- native host path ---------------------------------------------------------------------
# Checks, output allocation, decode scratch and the C-ABI calls live in the extension module
# (csrc/host.cpp); the functions below give its positional entry points their Python signatures.
_host = None


def _native(t: torch.Tensor):
    """The extension module; the first call loads it, after the one check that needs no library."""
    global _host
    if _host is None:
        if not t.is_cuda:
            raise RuntimeError("tensors must be CUDA tensors (nano_vllm_b200 has no CPU path)")
        _host = _lib.host()
    return _host


# ---- functional entry points ------------------------------------------------------------

def store_kvcache(key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                  slot_mapping: torch.Tensor) -> None:
    """k_cache.view(-1, Hkv*D)[slot_mapping[i]] = key[i] (same for value); bit-exact copy.

    Same argument contract and asserts as nanovllm/layers/attention.py:32-39.
    """
    (_host or _native(key)).store_kvcache(key, value, k_cache, v_cache, slot_mapping)


def decode_paged(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, context_lens: torch.Tensor,
                 block_tables: torch.Tensor, scale: float, out: torch.Tensor | None = None) -> torch.Tensor:
    """One query token per sequence against the paged cache; q/out are ``[B, Hq, D]``.

    Stands where ``flash_attn_with_kvcache(q.unsqueeze(1), k_cache, v_cache,
    cache_seqlens=context_lens, block_table=block_tables, softmax_scale=scale, causal=True)``
    stands in nanovllm/layers/attention.py:74-77.
    """
    return (_host or _native(q)).decode_paged(q, k_cache, v_cache, context_lens, block_tables, scale, out)


def decode_step(q: torch.Tensor, key: torch.Tensor, value: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                slot_mapping: torch.Tensor, context_lens: torch.Tensor, block_tables: torch.Tensor, scale: float,
                out: torch.Tensor | None = None) -> torch.Tensor:
    """``store_kvcache(key, value, k_cache, v_cache, slot_mapping)`` followed by ``decode_paged`` as
    ONE launch: what nanovllm/layers/attention.py:65-66 and :74-77 do for a decode batch.  The
    thread block that streams a sequence's newest position takes that row from ``key`` /
    ``value`` and writes it to the cache on the way.  ``slot_mapping[b]`` must be the slot of
    position ``context_lens[b] - 1`` (what the model runner passes) or negative (nothing stored);
    rows with ``context_lens[b] == 0`` store nothing.  q/out ``[B, Hq, D]``, key/value ``[B, Hkv, D]``.
    """
    return (_host or _native(q)).decode_step(q, key, value, k_cache, v_cache, slot_mapping, context_lens, block_tables,
                                             scale, out)


def decode_paged_static(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, context_lens: torch.Tensor,
                        block_tables: torch.Tensor, scale: float, out: torch.Tensor) -> torch.Tensor:
    """``decode_paged`` for hosts that may not allocate device memory while serving (all free
    HBM already belongs to the KV cache, or an allocation's implicit synchronisation is not
    acceptable): the arrival counters and partials go to a 32 MiB array inside the library instead
    of a torch-allocated workspace, and ``out`` must be supplied, so this call allocates nothing.
    Raises ``NvllmError`` (NVLLM_E_WORKSPACE) for geometries whose scratch exceeds the array.
    Calls on one device share that array: keep them ordered on the GPU.  Make the first call
    on a device outside CUDA graph capture.  No counterpart in nano-vllm."""
    B, Hq, D = q.shape
    Hkv = k_cache.shape[-2]
    _require_cuda_bf16("q", q)
    _require_cuda_bf16("k_cache", k_cache)
    _require_cuda_bf16("v_cache", v_cache)
    _require_cuda_bf16("out", out)
    _require_i32("context_lens", context_lens)
    _require_i32("block_tables", block_tables)
    assert q.stride(-1) == 1 and q.stride(1) == D and out.stride(-1) == 1 and out.stride(1) == D
    assert k_cache.is_contiguous() and v_cache.is_contiguous()
    assert block_tables.dim() == 2 and block_tables.shape[0] == B and context_lens.numel() == B
    num_blocks = k_cache.numel() // (BLOCK_SIZE * Hkv * D)
    with torch.cuda.device(q.device):
        _lib.check(_lib.load().nvllm_decode_paged_static(
            q.data_ptr(), q.stride(0), k_cache.data_ptr(), v_cache.data_ptr(),
            context_lens.data_ptr(), block_tables.data_ptr(), block_tables.stride(0), block_tables.shape[1],
            out.data_ptr(), out.stride(0), B, Hq, Hkv, D, float(scale), num_blocks, _stream(q)))
    return out


def prefill_varlen(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens_q: torch.Tensor,
                   cu_seqlens_k: torch.Tensor, max_seqlen_q: int, max_seqlen_k: int, scale: float,
                   block_tables: torch.Tensor | None = None, out: torch.Tensor | None = None) -> torch.Tensor:
    """Varlen causal GQA attention over packed K/V rows, or over the paged cache when
    ``block_tables`` is given (then ``k``/``v`` are the cache planes).  q/out: ``[N, Hq, D]``.

    Stands where ``flash_attn_varlen_func(..., causal=True, block_table=block_tables)`` stands
    in nanovllm/layers/attention.py:70-73.
    """
    return (_host or _native(q)).prefill_varlen(q, k, v, cu_seqlens_q, cu_seqlens_k, int(max_seqlen_q), int(max_seqlen_k),
                                                scale, block_tables, out)


def qk_norm_rope_store(qkv: torch.Tensor, positions: torch.Tensor, q_weight: torch.Tensor | None,
                       k_weight: torch.Tensor | None, cos_sin_cache: torch.Tensor, eps: float,
                       slot_mapping: torch.Tensor | None, k_cache: torch.Tensor, v_cache: torch.Tensor,
                       num_q_heads: int, num_kv_heads: int, head_dim: int) -> None:
    """In place on the fused ``qkv`` activation ``[N, (Hq + 2*Hkv) * D]``: per-head RMSNorm of
    q and k (when weights are given), rotary embedding of q and k, and the scatter of the new
    K/V rows into the cache (when ``slot_mapping`` is given and the cache exists).

    One launch for what nanovllm/models/qwen3.py:89-107 does with ``q_norm``, ``k_norm``,
    ``rotary_emb`` and, inside the attention layer, ``store_kvcache``.
    """
    (_host or _native(qkv)).qk_norm_rope_store(qkv, positions, q_weight, k_weight, cos_sin_cache, eps, slot_mapping, k_cache,
                                               v_cache, num_q_heads, num_kv_heads, head_dim)


def sample_tokens(logits: torch.Tensor, temperatures: torch.Tensor, noise: torch.Tensor | None = None,
                  seed: int = 0, step: int = 0, out: torch.Tensor | None = None) -> torch.Tensor:
    """One token per row of ``logits`` ``[B, V]`` (bf16 or fp32): argmax where the row's temperature
    is 0, else a draw from ``softmax(logits / T)``.  One launch for what
    nanovllm/layers/sampler.py:10-26 does in eight.  ``noise`` ``[B, V]`` fp32, when given, is the
    Exponential(1) draw to use (the reference's ``torch.empty_like(probs).exponential_(1)``);
    otherwise the kernel generates its own from ``(seed, step)``.  Returns int64 ``[B]``.
    """
    return (_host or _native(logits)).sample_tokens(logits, temperatures, noise, seed, step, out)


def sample_candidates(logits: torch.Tensor, temperatures: torch.Tensor, vocab_offset: int, noise: torch.Tensor | None = None,
                      seed: int = 0, step: int = 0, out: torch.Tensor | None = None) -> torch.Tensor:
    """``sample_tokens`` for one rank's slice ``[B, V / ranks]`` of the vocabulary, starting at global
    index ``vocab_offset``: returns int64 ``[B]`` candidates whose element-wise maximum over the ranks
    (``dist.reduce(..., op=MAX)``) decodes, with ``sample_unpack``, to the token ``sample_tokens``
    picks from the concatenated logits.  Replaces the gather + cat of
    nanovllm/layers/embed_head.py:78-87 by 8 bytes per row."""
    return (_host or _native(logits)).sample_candidates(logits, temperatures, noise, seed, step, out, int(vocab_offset))


def sample_unpack(candidates: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """Token ids int64 ``[B]`` of (merged) candidates from ``sample_candidates``."""
    assert candidates.is_cuda and candidates.dtype == torch.int64 and candidates.is_contiguous()
    B = candidates.numel()
    if out is None:
        out = torch.empty(B, dtype=torch.int64, device=candidates.device)
    with torch.cuda.device(candidates.device):
        _lib.check(_lib.load().nvllm_sample_unpack(candidates.data_ptr(), out.data_ptr(), B, _stream(candidates)))
    return out


# ---- the layer --------------------------------------------------------------------------

class Attention(nn.Module):
    """Drop-in for nanovllm/layers/attention.py:42-79 (same constructor, attributes, forward)."""

    def __init__(self, num_heads, head_dim, scale, num_kv_heads):
        super().__init__()
        self.num_heads = num_heads
        self.head_dim = head_dim
        self.scale = scale
        self.num_kv_heads = num_kv_heads
        self.k_cache = self.v_cache = torch.tensor([])

    def forward(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, kv_stored: bool = False):
        """``kv_stored=True``: the caller has already written this step's K/V rows into the cache
        (the fused pre-attention step does); the reference signature is ``forward(q, k, v)``."""
        return (_host or _native(q)).attention_forward(self, _get_context(), q, k, v, kv_stored)

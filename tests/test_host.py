"""Host-side logic that needs no GPU: the layer's contract, the workload generators and the
oracle's own consistency."""
import ctypes

import pytest
import torch

from nano_vllm_b200 import attention as A, context as C, workloads as W
from oracle import paged_attention_ref as R


def test_layer_surface_matches_the_reference_module():
    layer = A.Attention(16, 128, 128 ** -0.5, 8)
    assert (layer.num_heads, layer.head_dim, layer.num_kv_heads) == (16, 128, 8)
    assert layer.k_cache.numel() == 0 and layer.v_cache.numel() == 0  # what allocate_kv_cache looks for
    assert hasattr(layer, "k_cache") and hasattr(layer, "v_cache")
    C.set_context(False, slot_mapping=torch.zeros(1, dtype=torch.int32))
    assert C.get_context().is_prefill is False and C.get_context().block_tables is None
    C.reset_context()
    assert C.get_context().slot_mapping is None


def test_there_is_no_cpu_fallback():
    q = torch.zeros(2, 16, 128, dtype=torch.bfloat16)
    kc = torch.zeros(1, 256, 8, 128, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="CUDA"):
        A.store_kvcache(q[:, :8], q[:, :8], kc, kc, torch.zeros(2, dtype=torch.int32))
    with pytest.raises(RuntimeError, match="CUDA"):
        A.decode_paged(q, kc, kc, torch.ones(2, dtype=torch.int32), torch.zeros(2, 1, dtype=torch.int32), 0.1)
    with pytest.raises(RuntimeError, match="CUDA"):
        cu = torch.tensor([0, 2], dtype=torch.int32)
        A.prefill_varlen(q, q[:, :8], q[:, :8], cu, cu, 2, 2, 0.1)


def test_decode_workload_metadata_is_what_the_runner_would_build():
    case = W.cfg1_decode()
    B = case.q.shape[0]
    assert case.block_tables.dtype == torch.int32 and case.context_lens.dtype == torch.int32
    used = case.block_tables[case.block_tables >= 0]
    assert used.unique().numel() == used.numel(), "physical blocks are not shared between sequences"
    for b in range(B):
        n = int(case.context_lens[b])
        nblk = (n + 255) // 256
        assert (case.block_tables[b, :nblk] >= 0).all() and (case.block_tables[b, nblk:] == -1).all()
        # slot of the token being decoded: last block, last position (model_runner.py:225-229)
        assert int(case.slot_mapping[b]) == int(case.block_tables[b, nblk - 1]) * 256 + (n - 1) % 256
    assert 100 <= int(case.context_lens.min()) and int(case.context_lens.max()) <= 1024


def test_prefill_workload_prefix_sharing_structure():
    case = W.cfg2_prefill()
    lq = (case.cu_seqlens_q[1:] - case.cu_seqlens_q[:-1]).tolist()
    lk = (case.cu_seqlens_k[1:] - case.cu_seqlens_k[:-1]).tolist()
    assert len(lq) == 64 and case.block_tables is not None
    sharers = [i for i in range(64) if lk[i] != lq[i]]
    assert sharers == list(range(3, 64, 4))
    for i in sharers:
        cached = lk[i] - lq[i]
        assert cached % 256 == 0 and 256 <= cached <= 768 and lq[i] >= 1
        nshared = cached // 256
        assert torch.equal(case.block_tables[i, :nshared], case.block_tables[i - 1, :nshared])
    assert case.slot_mapping.numel() == sum(lq) == case.q.shape[0]
    assert case.slot_mapping.unique().numel() == case.slot_mapping.numel()
    assert case.max_seqlen_q == max(lq) and case.max_seqlen_k == max(lk)


def test_oracle_decode_equals_plain_softmax():
    case = W.make_decode_case(51, 3, 1, 1, 4, 2, 64, context_lens=[5, 300, 257])
    out = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    for b in range(3):
        n = int(case.context_lens[b])
        k = R.gather_paged(case.k_cache, case.block_tables[b], n).float()
        v = R.gather_paged(case.v_cache, case.block_tables[b], n).float()
        for h in range(4):
            s = (k[:, h // 2] @ case.q[b, h].float()) * case.scale
            ref = torch.softmax(s, 0) @ v[:, h // 2]
            assert torch.allclose(out[b, h], ref, atol=1e-5, rtol=1e-4)


def test_oracle_prefix_prefill_equals_suffix_of_full_prefill():
    """A sequence with a cached prefix must get the rows a full prefill would give it."""
    case = W.make_prefill_case(52, 2, 1, 1, 4, 2, 64, lengths=[700, 700], shared_blocks=[0, 2])
    R.store_kvcache_ref(case.k, case.v, case.k_cache, case.v_cache, case.slot_mapping)
    out = R.prefill_ref(case.q, case.k_cache, case.v_cache, case.cu_seqlens_q, case.cu_seqlens_k, case.scale,
                        case.block_tables)
    # sequence 1 recomputed from scratch: its K/V = 512 shared rows of sequence 0 + its own 188
    k_full = torch.cat([case.k[:512], case.k[700:]])
    v_full = torch.cat([case.v[:512], case.v[700:]])
    q_full = torch.cat([torch.zeros(512, 4, 64, dtype=torch.bfloat16), case.q[700:]])
    cu = torch.tensor([0, 700], dtype=torch.int32)
    full = R.prefill_ref(q_full, k_full, v_full, cu, cu, case.scale)
    assert torch.allclose(out[700:], full[512:], atol=1e-6)


def test_algorithmic_work_formulas():
    assert W.decode_bytes([256, 1], 16, 8, 128) == 257 * 8 * 128 * 4 + 2 * 2 * 16 * 128 * 2 + 4 * (2 + 2)
    assert W.store_bytes(10, 1024) == 10 * 1024 * 8 + 40
    assert W.prefill_flops([3], [3], 1, 1) == 4 * 6
    assert W.prefill_flops([2], [258], 2, 64) == 4 * 2 * 64 * (2 * 256 + 3)


def test_when_the_peer_memory_all_reduce_is_preferred():
    """Decode-sized tensors go to the peer kernel, prefill-sized ones to the library collective."""
    from nano_vllm_b200.allreduce import prefer_peer_kernel as prefer
    mb = 8 << 20
    assert prefer(256 * 1024 * 2, 2, mb) and prefer(256 * 4096 * 2, 2, mb) and prefer(4 << 20, 2, mb)
    assert not prefer(16384 * 1024 * 2, 2, mb)            # a 16k-token prefill batch: 32 MiB
    assert prefer(256 * 1024 * 2, 4, mb) and prefer(256 * 1024 * 2, 8, mb)
    assert prefer(256 * 4096 * 2, 4, mb) and prefer(256 * 4096 * 2, 8, mb)
    assert not prefer(0, 2, mb)


def test_all_reduce_protocol_choice_is_host_arithmetic(lib):
    """Cells for small tensors, two shots for larger ones at more than two ranks, one shot at two
    ranks and for tensors with a ragged tail; a forced protocol that does not apply falls back."""
    from nano_vllm_b200.allreduce import protocol_for
    mb = 8 << 20
    assert protocol_for(32 << 10, 2, mb) == "cells" and protocol_for(2 << 20, 2, mb) == "cells"
    assert protocol_for(4 << 20, 2, mb) == "one-shot"
    assert protocol_for(32 << 10, 8, mb) == "cells" and protocol_for(128 << 10, 8, mb) == "cells"
    assert protocol_for(512 << 10, 4, mb) == "cells" and protocol_for(1 << 20, 4, mb) == "cells-two-shot"
    assert protocol_for(512 << 10, 8, mb) == "cells" and protocol_for(1 << 20, 8, mb) == "cells-two-shot"
    assert protocol_for(2 << 20, 4, mb) == "cells-two-shot" and protocol_for(2 << 20, 8, mb) == "cells-two-shot"
    assert protocol_for(2 << 20, 8, mb, forced=3) == "two-shot" and protocol_for(6 << 20, 4, mb) == "two-shot"
    assert protocol_for((2 << 20) + 6, 8, mb) == "cells-two-shot"    # a ragged tail is fine for cells
    assert protocol_for(2 << 20, 8, mb, forced=2) == "one-shot"
    assert protocol_for(2 << 20, 2, mb, forced=3) == "cells"           # two shots need more than two ranks
    assert protocol_for(2 << 20, 8, mb, forced=1) == "cells-two-shot"  # cells to every peer do not fit: 2 x 2 MiB x 8 > 8 MiB


@pytest.mark.parametrize("sms", [148, 132, 20])
def test_sampler_takes_no_larger_cluster_than_the_device_grants(lib, sms):
    """Sixteen blocks to a row for the fewest rows where that is possible, else eight; the same plan
    for larger batches and rows too short for it."""
    for batch in (1, 2, 9, 10, 32, 64, 256, 512):
        for vocab in (7, 2047, 4096, 16384, 32768, 151936):
            wide, portable = lib.nvllm_sample_plan(batch, vocab, sms, 16), lib.nvllm_sample_plan(batch, vocab, sms, 8)
            assert portable in (1, 2, 4, 8) and wide == (16 if batch * 16 <= sms and vocab >= 16 * 2048 else portable)
    assert lib.nvllm_sample_plan(1, 151936, sms, 8) == 8 and lib.nvllm_sample_plan(1, 0, sms, 8) == -3


@pytest.mark.parametrize("sms", [148, 132, 20])
@pytest.mark.parametrize("device", ["full", "gaps", "no sixteen", "silent"])
def test_sampler_lays_launches_out_for_what_the_device_holds(lib, sms, device):
    """One wave of clusters that the device holds at a time, or blocks of 256 threads in powers of two: more than two
    rows to a multiprocessor, and devices that do not say what they hold."""
    threads_of, per_sm = (768, 512, 512, 384, 256, 256), (1, 2, 2, 2, 4, 4)
    counts = [[0] * 17 for _ in threads_of]
    for f in range(6):
        for c in range(2, 17):
            counts[f][c] = sms * per_sm[f] // c * (device != "silent") * (c <= 8 or device != "no sixteen")
            if device == "gaps":
                counts[f][c] = max(0, counts[f][c] - c) * (c not in (3, 6))
    table = (ctypes.c_int32 * (6 * 17))(*[n for row in counts for n in row])
    blocks, threads = ctypes.c_int32(), ctypes.c_int32()
    seen = set()
    for batch in (*range(1, 64), 74, 100, 148, 180, 222, 2 * sms, 2 * sms + 1, 512):
        for fp32 in (0, 1):
            for vocab in (7, 1000, 2047, 4096, 18992, 32768, 50257, 151936):
                assert lib.nvllm_sample_layout(batch, vocab, 0, fp32, sms, table, ctypes.byref(blocks), ctypes.byref(threads)) == 0
                c, n = blocks.value, threads.value
                assert 256 <= n <= 768 and n % 32 == 0
                waves = 1
                while waves < 8 and batch * waves < 3 * sms and vocab >= 2 * waves * 2048:
                    waves *= 2
                held = [counts[f][c] if c > 1 else sms * per_sm[f] for f in range(6) if n == threads_of[f] or (f == 0 and 256 <= n <= 768)]
                assert (c, n) == (waves, 256) or (batch <= 2 * sms and max(held) >= batch), f"{batch} rows of {vocab}: {c} x {n}"
                if device == "silent" or batch > 2 * sms:
                    assert (c, n) == (waves, 256)
                seen.add((c, n))
    assert (16 in {c for c, _ in seen}) == (device == "full" and sms > 16)
    args = (0, 0, sms, table, ctypes.byref(blocks), ctypes.byref(threads))
    assert lib.nvllm_sample_layout(1, 0, *args) == -3 and lib.nvllm_sample_layout(-1, 5, *args) == -3
    assert lib.nvllm_sample_layout(1, 5, 0, 0, sms, table, None, ctypes.byref(threads)) == -1


@pytest.mark.parametrize("batch,tiles", [(2, 10), (2, 3), (6, 30), (7, 7), (9, 5), (20, 21), (3, 296), (5, 37)])
def test_every_item_is_drawn_once_whatever_block_draws_when(lib, batch, tiles):
    """The order of a launch with an item to a block: a permutation of the list, so that blocks that draw again (for a
    tile without a visible key) before others have drawn at all leave nothing out."""
    groups = 296 // tiles
    total = tiles * groups
    items = [lib.nvllm_prefill_item(n, tiles, batch, groups) for n in range(total)]
    assert sorted(items) == list(range(total))
    assert [i % groups for i in items] == [n % groups for n in range(total)]  # head groups fastest, as in the list
    stride = -(-tiles // batch)
    assert [i // groups for i in items[:(tiles // stride) * groups:groups]] == list(range(0, tiles // stride * stride, stride))
    assert lib.nvllm_prefill_item(total, tiles, batch, groups) == -3 and lib.nvllm_prefill_item(0, tiles, 0, groups) == -3


def test_fused_projection_tile_choice_is_host_arithmetic(lib):
    """Tile width of the projection fused with its all-reduce: the narrowest of 32 / 64 / 128 columns
    that leaves one tile per thread block (128 blocks), 0 for shapes the kernel refuses."""
    mb = 8 << 20
    assert lib.nvllm_ar_gemm_tile(16, 4096, 512, 8, mb) == 32
    assert lib.nvllm_ar_gemm_tile(256, 4096, 1536, 8, mb) == 64
    assert lib.nvllm_ar_gemm_tile(512, 4096, 512, 8, mb) == 128
    assert lib.nvllm_ar_gemm_tile(256, 1024, 1024, 2, mb) == 32
    assert lib.nvllm_ar_gemm_tile(1024, 4096, 512, 8, mb) == 0   # cell areas too small
    assert lib.nvllm_ar_gemm_tile(256, 4096, 512, 8, 1 << 20) == 0
    assert lib.nvllm_ar_gemm_tile(8, 4096, 100, 2, mb) == 0      # k not a multiple of 8
    assert lib.nvllm_ar_gemm_tile(8, 48, 64, 2, mb) == 0         # n not a multiple of 32
    assert lib.nvllm_ar_gemm_tile(8, 4096, 512, 9, mb) == 0      # more ranks than the areas have regions for


def test_oracle_row_parallel_projection_rounds_every_rank_once():
    """The oracle's partials are bf16 (what each rank's GEMM returns), not fp32: the sum of rounded
    partials differs from the rounded product over the whole k."""
    g = torch.Generator().manual_seed(3)
    xs = [torch.randn(4, 64, generator=g).to(torch.bfloat16) for _ in range(4)]
    ws = [torch.randn(32, 64, generator=g).to(torch.bfloat16) for _ in range(4)]
    got = R.row_parallel_linear_ref(xs, ws)
    partials = [(x.float() @ w.float().t()).to(torch.bfloat16) for x, w in zip(xs, ws)]
    assert torch.equal(got, R.allreduce_ref(partials))
    whole = (torch.cat(xs, 1).float() @ torch.cat(ws, 1).float().t()).to(torch.bfloat16)
    assert got.shape == whole.shape and not torch.equal(got, whole)
    assert float((got.float() - whole.float()).abs().max()) <= 4 * 2.0 ** -8 * float(whole.float().abs().max())


@pytest.mark.parametrize("status", range(8))
def test_reading_an_expired_wait_zeroes_the_decode_scratch(monkeypatch, status):
    """Marks that such a launch leaves would be taken for a later one's partials; other bits leave the scratch alone."""
    import ctypes

    from nano_vllm_b200 import _lib
    cleared = []

    class Library:
        @staticmethod
        def nvllm_read_status(out):
            ctypes.cast(out, ctypes.POINTER(ctypes.c_int32))[0] = status
            return 0

    class Host:
        @staticmethod
        def clear_workspaces():
            cleared.append(True)

    monkeypatch.setattr(_lib, "_lib", Library)
    monkeypatch.setattr(_lib, "_host", Host)
    assert _lib.read_status() == status
    assert len(cleared) == (status >= 4)
    monkeypatch.setattr(_lib, "_host", None)  # no call has been made: there is nothing to clear
    assert _lib.read_status() == status


def _prefill_plan(lib, lens, hq, hkv, d, rows=0, sms=148, max_k=None):
    out = [ctypes.c_int32() for _ in range(3)]
    args = (sum(lens), sum(lens), len(lens), max(lens), max_k or max(lens), hq, hkv, d, rows, sms)
    rc = lib.nvllm_prefill_plan(*args, *(ctypes.byref(x) for x in out))
    return rc if rc else tuple(x.value for x in out)


def test_prefill_layout_is_host_arithmetic(lib):
    never, none, spare, tiles = 1 << 30, 0, 1, 2
    # head_dim 64: prompts of the same number of query tiles, more than two items to a multiprocessor; a spare warp stores rows while there are few
    assert _prefill_plan(lib, [512] * 7, 14, 2, 64) == (3, 0, none)
    assert _prefill_plan(lib, [512] * 7, 14, 2, 64, rows=1) == (3, 0, spare)
    assert _prefill_plan(lib, [512] * 7, 14, 2, 64, rows=2) == (3, 0, tiles)
    assert _prefill_plan(lib, [512] * 16, 14, 2, 64, rows=1) == (3, 0, tiles)
    assert _prefill_plan(lib, [512] * 5, 14, 2, 64) == (2, never, none)                 # 285 items
    assert _prefill_plan(lib, [512] * 7, 14, 2, 64, sms=300) == (2, never, none)
    assert _prefill_plan(lib, [255] * 60, 14, 2, 64) == (2, never, none)                # less than four key tiles
    assert _prefill_plan(lib, [256] * 60, 14, 2, 64) == (3, 0, none)
    assert _prefill_plan(lib, [896] * 60, 16, 16, 64) == (2, never, none)               # seven query tiles to a prompt
    assert _prefill_plan(lib, [897] * 60, 16, 16, 64) == (3, 0, none)
    # 29 tiles of 18 tokens, 8 in the last: lengths spread evenly over 505-512 have it, over 500-512 not
    assert _prefill_plan(lib, [512, 505, 512, 505] * 3, 14, 2, 64) == (3, 0, none)
    assert _prefill_plan(lib, [512, 500, 512, 500] * 3, 14, 2, 64) == (2, never, none)
    # through the table one prompt may take all that is missing
    assert _prefill_plan(lib, [512] * 11 + [505], 14, 2, 64, rows=3) == (3, 0, none)
    assert _prefill_plan(lib, [512] * 11 + [504], 14, 2, 64, rows=3) == (2, never, none)
    assert _prefill_plan(lib, [2048] * 4 + [1792], 16, 16, 64, rows=2) == (2, never, tiles)
    # other prompts: eight times the longest item's key tiles to a multiprocessor, cached ones among them, or four times and
    # twelve prompts of different lengths; in the list's order
    mixed = [1024, 300, 700, 400]
    assert _prefill_plan(lib, mixed * 8, 14, 2, 64) == (3, never, none)
    assert _prefill_plan(lib, mixed * 8, 14, 2, 64, rows=2) == (3, never, tiles)
    assert _prefill_plan(lib, mixed * 6, 14, 2, 64) == (2, never, none)                 # 3.9 times
    assert _prefill_plan(lib, mixed * 8, 14, 2, 64, max_k=2048) == (2, never, none)
    assert _prefill_plan(lib, mixed * 16, 14, 14, 64) == (2, never, none)               # one head to a tile
    assert _prefill_plan(lib, [1022, 1001] * 8, 14, 2, 64) == (2, never, none)          # 6.4 times, of about one length
    assert _prefill_plan(lib, [4096, 3000] * 3, 14, 2, 64) == (2, never, none)          # 6 times, six prompts
    assert _prefill_plan(lib, [16384], 14, 2, 64) == (2, never, none) and _prefill_plan(lib, [32768], 14, 2, 64) == (3, never, none)
    # head_dim 128: two blocks
    for lens in ([512] * 40, mixed, [4096] * 4):
        assert _prefill_plan(lib, lens, 16, 8, 128)[0] == 2
    assert _prefill_plan(lib, [300] * 6, 16, 8, 128) == (2, 148, none)
    assert _prefill_plan(lib, [512], 14, 2, 96) == -3 and _prefill_plan(lib, [512], 14, 3, 64) == -3
    assert _prefill_plan(lib, [512], 14, 2, 64, rows=4) == -3 and _prefill_plan(lib, [512], 14, 2, 64, sms=0) == -3

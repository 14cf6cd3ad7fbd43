"""Paged GQA decode on the GPU, through the C ABI, against the fp32 CPU oracle."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from conftest import assert_close_to_oracle
from nano_vllm_b200 import _lib, attention as A, context as C, workloads as W
from oracle import paged_attention_ref as R

pytestmark = pytest.mark.gpu


def _check(cuda, case, what, store_first=True):
    dev = case.to(cuda)
    if store_first:
        A.store_kvcache(dev.k_new, dev.v_new, dev.k_cache, dev.v_cache, dev.slot_mapping)
        R.store_kvcache_ref(case.k_new, case.v_new, case.k_cache, case.v_cache, case.slot_mapping)
    out = A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale)
    torch.cuda.synchronize()
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(out, ref, what)
    assert _lib.read_status() == 0
    return out


def test_cfg1(cuda):
    """8 sequences, contexts in [100,1024], 16 query / 8 KV heads, head_dim 128 (the CPU-runnable
    decode configuration)."""
    _check(cuda, W.cfg1_decode(), "cfg1")


@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (32, 8, 128), (14, 2, 64), (4, 1, 128), (7, 1, 64), (8, 1, 128), (2, 2, 64),
                                      (40, 8, 128), (12, 2, 128), (6, 2, 64)])
def test_geometries(cuda, hq, hkv, d):
    case = W.make_decode_case(11, 6, 1, 1500, hq, hkv, d,
                              context_lens=[1, 255, 256, 257, 1024, 1500])
    _check(cuda, case, f"hq{hq} hkv{hkv} d{d}")


@pytest.mark.parametrize("width", [1, 4, 16, 64])
def test_table_width(cuda, width):
    """The table width is static under CUDA graphs and only bounds the lengths; results must not
    depend on it."""
    lens = [min(200, width * 256), min(width * 256, 3000), 17, width * 256]
    case = W.make_decode_case(12, 4, 1, 1, 16, 8, 128, context_lens=lens, table_width=width)
    _check(cuda, case, f"width{width}")


def test_long_context_split_and_combine(cuda):
    """Qwen2-0.5B geometry, 32768-token contexts in 128 scattered blocks (config 5 shape,
    small batch so the oracle finishes in seconds)."""
    case = W.make_decode_case(13, 3, 1, 1, 14, 2, 64, context_lens=[32768, 20000, 32767])
    _check(cuda, case, "long")


def test_long_context_one_kv_head_per_rank(cuda):
    """The tensor-parallel (2 ranks) shard of the long-context configuration: 7 query heads on 1 KV
    head, head_dim 64, 32768-token contexts."""
    case = W.make_decode_case(23, 3, 1, 1, 7, 1, 64, context_lens=[32768, 32768, 32768])
    _check(cuda, case, "long tp2 shard")


def test_qwen3_8b_geometry_at_8192_tokens(cuda):
    """32 query / 8 KV heads, head_dim 128, contexts up to the 8192 tokens of the decode benchmark."""
    case = W.make_decode_case(24, 5, 1, 1, 32, 8, 128, context_lens=[8192, 2048, 8191, 5000, 4097], table_width=32)
    _check(cuda, case, "8b geometry 8192")


def test_many_short_sequences_share_a_thread_block(cuda):
    """More sequences than threads in a block and far more than thread blocks per KV head: every
    block walks several sequences, a few of them empty, most cut by no range boundary."""
    g = torch.Generator().manual_seed(25)
    lens = torch.randint(0, 200, (300,), generator=g).tolist()
    lens[0] = 0
    lens[-1] = 0
    case = W.make_decode_case(25, 300, 1, 1, 16, 8, 128, context_lens=lens, table_width=4)
    case.slot_mapping.clamp_(min=0)
    dev = case.to(cuda)
    out = A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale)
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(out, ref, "many short")
    assert _lib.read_status() == 0


def test_one_sequence_spread_over_every_thread_block(cuda):
    """A single long sequence among empty ones: every range holds a piece of it, and the block that
    delivers the last partial merges them all."""
    case = W.make_decode_case(26, 4, 1, 1, 4, 1, 128, context_lens=[0, 30000, 0, 0], table_width=128)
    case.slot_mapping.clamp_(min=0)
    dev = case.to(cuda)
    for _ in range(2):  # the second call finds the counters as the first one left them
        out = A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale)
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(out, ref, "one long")


@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (32, 8, 128), (14, 2, 64), (4, 1, 128)])
def test_decode_step_equals_store_then_decode(cuda, hq, hkv, d):
    """The one-launch step (store of the new token + decode) must leave the cache exactly as
    store_kvcache does (nanovllm/layers/attention.py:65-66) and give the output of the two
    separate calls; both are compared with the oracle as well."""
    case = W.make_decode_case(27, 9, 1, 1, hq, hkv, d, context_lens=[1, 64, 65, 256, 257, 1000, 1024, 3000, 16],
                              table_width=12)
    sep, fus = case.to(cuda), case.to(cuda)
    A.store_kvcache(sep.k_new, sep.v_new, sep.k_cache, sep.v_cache, sep.slot_mapping)
    expected = A.decode_paged(sep.q, sep.k_cache, sep.v_cache, sep.context_lens, sep.block_tables, case.scale)
    got = A.decode_step(fus.q, fus.k_new, fus.v_new, fus.k_cache, fus.v_cache, fus.slot_mapping, fus.context_lens,
                        fus.block_tables, case.scale)
    torch.cuda.synchronize()
    assert torch.equal(fus.k_cache, sep.k_cache) and torch.equal(fus.v_cache, sep.v_cache)
    assert torch.equal(got, expected)
    R.store_kvcache_ref(case.k_new, case.v_new, case.k_cache, case.v_cache, case.slot_mapping)
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(got, ref, "decode step")
    assert _lib.read_status() == 0


def test_decode_step_slot_rules(cuda):
    """slot < 0: nothing stored, the cached row is used.  A slot that is not the position of the
    newest token: flagged, nothing stored.  Empty rows: nothing stored."""
    case = W.make_decode_case(28, 4, 1, 1, 16, 8, 128, context_lens=[300, 300, 0, 300], table_width=4)
    case.slot_mapping[0] = -1
    case.slot_mapping[1] += 1
    case.slot_mapping[2] = 0
    dev = case.to(cuda)
    k_before, v_before = dev.k_cache.clone(), dev.v_cache.clone()
    _lib.read_status()
    out = A.decode_step(dev.q, dev.k_new, dev.v_new, dev.k_cache, dev.v_cache, dev.slot_mapping, dev.context_lens,
                        dev.block_tables, case.scale)
    torch.cuda.synchronize()
    assert _lib.read_status() == 1  # NVLLM_STATUS_BAD_SLOT, from row 1 only
    s3 = int(case.slot_mapping[3])
    flat_k, flat_kb = dev.k_cache.view(-1, 8, 128), k_before.view(-1, 8, 128)
    assert torch.equal(flat_k[s3], dev.k_new[3]) and torch.equal(dev.v_cache.view(-1, 8, 128)[s3], dev.v_new[3])
    flat_kb[s3] = flat_k[s3]
    v_before.view(-1, 8, 128)[s3] = dev.v_cache.view(-1, 8, 128)[s3]
    assert torch.equal(dev.k_cache, k_before) and torch.equal(dev.v_cache, v_before)  # nothing else was written
    host_k, host_v = dev.k_cache.cpu(), dev.v_cache.cpu()
    ref = R.decode_ref(case.q, host_k, host_v, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(out, ref, "slot rules")


def test_zero_context_rows_and_graph_padding(cuda):
    """Padding rows under graph replay have context_len 0, slot 0 and table row 0
    (nanovllm/engine/model_runner.py:271-280): output rows must be zero, no fault."""
    case = W.make_decode_case(14, 5, 1, 1, 16, 8, 128, context_lens=[300, 0, 0, 513, 0], table_width=16)
    case.block_tables[case.context_lens == 0] = 0
    dev = case.to(cuda)
    out = A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale)
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(out, ref, "padding")
    assert out[1].abs().max() == 0 and out[4].abs().max() == 0


def test_stale_cache_beyond_context_cannot_leak(cuda):
    """Positions past the context hold NaN/Inf garbage; the output must stay finite."""
    case = W.make_decode_case(15, 3, 1, 1, 16, 8, 128, context_lens=[100, 257, 511])
    for b, n in enumerate(case.context_lens.tolist()):
        blk = int(case.block_tables[b, (n - 1) // 256])
        case.k_cache[blk, n % 256 or 256:] = float("nan")
        case.v_cache[blk, n % 256 or 256:] = float("inf")
    _check(cuda, case, "stale", store_first=False)


def test_bad_block_id_is_flagged_not_dereferenced(cuda):
    case = W.make_decode_case(16, 2, 1, 1, 16, 8, 128, context_lens=[300, 300])
    case.block_tables[1, 1] = 10 ** 6
    dev = case.to(cuda)
    _lib.read_status()
    out = A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale)
    torch.cuda.synchronize()
    assert _lib.read_status() & 2
    assert torch.isfinite(out.float()).all()


def test_strided_q_and_cuda_graph_replay(cuda):
    """q is a view of the fused qkv activation; the launch is captured once with zeroed
    metadata and replayed with real metadata (nanovllm/engine/model_runner.py:296-336)."""
    hq, hkv, d, B, width = 16, 8, 128, 8, 16
    case = W.make_decode_case(17, B, 100, 3000, hq, hkv, d, table_width=width)
    dev = case.to(cuda)
    qkv = torch.zeros(B, (hq + 2 * hkv) * d, dtype=torch.bfloat16, device=cuda)
    q_view = qkv[:, :hq * d].view(B, hq, d)
    ctx = torch.zeros(B, dtype=torch.int32, device=cuda)
    bt = torch.zeros(B, width, dtype=torch.int32, device=cuda)
    out = torch.zeros(B, hq, d, dtype=torch.bfloat16, device=cuda)
    A.decode_paged(q_view, dev.k_cache, dev.v_cache, ctx, bt, case.scale, out=out)  # warm-up (allocates scratch)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        A.decode_paged(q_view, dev.k_cache, dev.v_cache, ctx, bt, case.scale, out=out)
    q_view.copy_(dev.q)
    ctx.copy_(dev.context_lens)
    bt.copy_(dev.block_tables)
    graph.replay()
    torch.cuda.synchronize()
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(out, ref, "graph replay")
    # replay again with other lengths: the ranges, the pieces and the arrival counters all change
    shorter = (case.context_lens // 3).clamp(min=1)
    ctx.copy_(shorter.to(cuda))
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, shorter, case.block_tables, case.scale)
    assert_close_to_oracle(out, ref, "graph replay, shorter contexts")


@pytest.mark.parametrize("hq,hkv,d", [(1, 1, 128), (3, 1, 128), (16, 2, 128), (1, 1, 64), (5, 1, 64), (8, 1, 64), (28, 4, 64)])
@pytest.mark.parametrize("lens", [[32000], [20000, 1, 0, 9001], [129, 65, 64, 63], [20000, 3000] + [0, 70] * 16])
def test_sequences_cut_into_many_parts(cuda, hq, hkv, d, lens):
    """Merges of two to a hundred and more partials, with lane groups to spare (parts split between
    them), as many as heads, and fewer; also through the layer, which is one launch for the first three
    and reads its lengths under the store for the last."""
    case = W.make_decode_case(29, len(lens), 1, 1, hq, hkv, d, context_lens=lens)
    _check(cuda, case, f"hq{hq} hkv{hkv} d{d} {lens}")
    dev = case.to(cuda)
    layer = A.Attention(hq, d, dev.scale, hkv)
    layer.k_cache, layer.v_cache = dev.k_cache, dev.v_cache
    C.set_context(False, slot_mapping=dev.slot_mapping, context_lens=dev.context_lens, block_tables=dev.block_tables)
    got = layer(dev.q.view(len(lens), -1), dev.k_new.view(len(lens), -1), dev.v_new.view(len(lens), -1))
    C.reset_context()
    assert torch.equal(got.view_as(dev.q), A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, dev.scale))


@pytest.mark.parametrize("batch", [12, 13, 14, 32, 53, 54, 55])
@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (8, 8, 128), (32, 8, 64)])
def test_cut_sequences_around_the_sizes_of_marked_cells(cuda, batch, hq, hkv, d):
    """Partials as marked cells and plain ones in turn in one workspace: nothing that one launch leaves is taken for a
    partial of the next.  Many parts beside sequences of a few units and empty ones."""
    lens = ([5000, 64, 0, 65, 129, 700, 1] * 8)[:batch]
    case = W.make_decode_case(29, batch, 1, 1, hq, hkv, d, context_lens=lens)
    few = W.make_decode_case(30, 2, 1, 1, hq, hkv, d, context_lens=[4000, 300]).to(cuda)
    outs = [_check(cuda, case, f"batch {batch}", store_first=False)]
    dev = case.to(cuda)
    for _ in range(3):
        A.decode_paged(few.q, few.k_cache, few.v_cache, few.context_lens, few.block_tables, few.scale)
        outs.append(A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale))
        outs.append(A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale))
    torch.cuda.synchronize()
    assert all(torch.equal(o, outs[0]) for o in outs[1:])
    assert _lib.read_status() == 0


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e-38])
def test_no_partial_of_another_launch_is_taken_for_a_marked_cell(cuda, value):
    """Plain partials that are NaN, infinite or next to zero, over the whole area that the marked cells of the next launch
    lie in."""
    case = W.make_decode_case(44, 32, 1, 1, 16, 8, 128, context_lens=([700, 64, 0, 129, 1000, 300] * 6)[:32])
    want = _check(cuda, case, "marked", store_first=False)
    dev = case.to(cuda)
    few = W.make_decode_case(45, 11, 1, 1, 16, 8, 128, context_lens=[3000] * 11).to(cuda)  # 37 ranges, 47 partials
    few.v_cache.fill_(value)
    for _ in range(3):
        A.decode_paged(few.q, few.k_cache, few.v_cache, few.context_lens, few.block_tables, few.scale)
        got = A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        few.k_cache.fill_(value)
    assert _lib.read_status() == 0


@pytest.mark.parametrize("batch", [1, 2, 31, 32, 33])
@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (14, 2, 64)])
def test_layer_equals_store_then_decode_wherever_the_slots_lie(cuda, batch, hq, hkv, d):
    """One launch for few sequences, a store in front for more than 32: rows stored at their position, elsewhere
    in the same sequence, in another sequence's context, at a padding row's slot 0, twice to one slot, and nowhere."""
    g = torch.Generator().manual_seed(batch)
    lens = torch.randint(1, 1500, (batch,), generator=g)
    case = W.make_decode_case(37, batch, 1, 1, hq, hkv, d, context_lens=lens.tolist())
    slots = case.slot_mapping.clone()
    ctx = case.context_lens.clone()
    first = case.block_tables[:, 0].long() * 256
    slots[0] = first[0] + int(lens[0]) // 2 % 256  # in the middle of its own context
    if batch > 2:
        slots[1] = first[2]  # the first row of its neighbour
        ctx[3], slots[3] = 0, 0  # graph padding
        slots[4] = -1
        slots[5] = slots[6]
        case.k_new[5], case.v_new[5] = case.k_new[6], case.v_new[6]
        slots[batch - 1] = first[batch - 2] + 1
    dev = case.to(cuda)
    slots, ctx = slots.to(cuda), ctx.to(cuda)
    k2, v2 = dev.k_cache.clone(), dev.v_cache.clone()
    layer = A.Attention(hq, d, dev.scale, hkv)
    layer.k_cache, layer.v_cache = dev.k_cache, dev.v_cache
    for _ in range(2):
        C.set_context(False, slot_mapping=slots, context_lens=ctx, block_tables=dev.block_tables)
        got = layer(dev.q.view(batch, -1), dev.k_new.view(batch, -1), dev.v_new.view(batch, -1))
        C.reset_context()
        A.store_kvcache(dev.k_new, dev.v_new, k2, v2, slots)
        want = A.decode_paged(dev.q, k2, v2, ctx, dev.block_tables, dev.scale)
        assert torch.equal(got.view_as(want), want)
        assert torch.equal(dev.k_cache, k2) and torch.equal(dev.v_cache, v2)
        dev.k_new, dev.v_new = dev.k_new.flip(-1).contiguous(), dev.v_new.flip(-1).contiguous()
        slots = torch.where(slots >= 0, (slots // 256) * 256 + (slots + 77) % 256, slots)  # other rows of those blocks
    assert _lib.read_status() == 0
    slots[0] = dev.k_cache.shape[0] * 256
    C.set_context(False, slot_mapping=slots, context_lens=ctx, block_tables=dev.block_tables)
    layer(dev.q.view(batch, -1), dev.k_new.view(batch, -1), dev.v_new.view(batch, -1))
    C.reset_context()
    torch.cuda.synchronize()
    assert _lib.read_status() == 1  # NVLLM_STATUS_BAD_SLOT


@pytest.mark.parametrize("batch", [1, 31, 128, 129])
def test_lengths_written_by_the_kernel_just_before(cuda, batch):
    """The lengths are the rows of a cache that the launch in front stores to: the decode, which may
    start on the lengths of the time before, must use the new ones, longer, shorter or none, and
    report nothing about table entries that only the old ones reach."""
    g = torch.Generator().manual_seed(batch)
    longest = torch.randint(1, 3000, (batch,), generator=g)
    case = W.make_decode_case(31, batch, 1, 1, 16, 8, 128, context_lens=longest.tolist())
    dev = case.to(cuda)
    plane = torch.zeros(2, 256, 1, 256, dtype=torch.bfloat16, device=cuda)  # rows of 128 int32
    lens = plane[1].view(-1).view(torch.int32)[:batch]
    slots = torch.arange(511, -1, -1, dtype=torch.int32, device=cuda)  # the rows that hold the lengths last
    scratch = torch.zeros_like(plane)
    steps = []
    for i in range(6):
        now = [longest, longest // 2, torch.zeros_like(longest), longest * (torch.arange(batch) % 2), longest // 9, longest][i]
        table = case.block_tables.clone()
        for b in range(batch):
            table[b, (int(now[b]) + 255) // 256:] = -1
        rows = torch.zeros(512, 128, dtype=torch.int32)
        flat = torch.zeros(256 * 128, dtype=torch.int32)
        flat[:batch] = now.int()
        rows[:256] = flat.view(256, 128).flip(0)
        key = rows.to(cuda).view(torch.bfloat16).view(512, 1, 256)
        steps.append((now.int(), table.to(cuda), key))
    outs = []
    torch.cuda.synchronize()
    for now, table, key in steps:
        A.store_kvcache(key, key, plane, scratch, slots)
        outs.append(A.decode_paged(dev.q, dev.k_cache, dev.v_cache, lens, table, case.scale))
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    for (now, table, _), out in zip(steps, outs):
        ref = R.decode_ref(case.q, case.k_cache, case.v_cache, now, case.block_tables, case.scale)
        assert_close_to_oracle(out, ref, f"batch {batch}, lengths to {int(now.max())}")


@pytest.mark.parametrize("hq,hkv,d,lens", [(16, 8, 128, list(range(100, 1024, 60))), (32, 32, 128, [3500] * 6), (14, 2, 64, [1, 0, 5000, 127, 129]),
                                           (8, 8, 128, [64, 0, 65] * 42)])
def test_tables_written_by_the_kernel_just_before(cuda, hq, hkv, d, lens):
    """The block table is in the rows of a cache that the launch in front stores to: the decode, which may list its tiles
    by the entries of the time before, must use the new ones.  In a thread block: a few units, more than a warp lists
    (3500 tokens and 32 KV heads), sequences without a token, several sequences."""
    case = W.make_decode_case(37, len(lens), 1, 1, hq, hkv, d, context_lens=lens)
    dev = case.to(cuda)
    g = torch.Generator().manual_seed(5)
    width = case.block_tables.shape[1]
    plane = torch.zeros(2, 256, 1, 256, dtype=torch.bfloat16, device=cuda)  # rows of 128 int32
    table = plane[1].view(-1).view(torch.int32)[:len(lens) * width].view(len(lens), width)
    slots = torch.arange(511, -1, -1, dtype=torch.int32, device=cuda)  # the rows that hold the table last
    scratch = torch.zeros_like(plane)
    steps = []
    for i in range(4):
        perm = torch.cat([torch.randperm(case.k_cache.shape[0], generator=g).int(), torch.tensor([-1], dtype=torch.int32)])
        now = perm[case.block_tables.long()]  # -1 stays -1
        flat = torch.zeros(256 * 128, dtype=torch.int32)
        flat[:now.numel()] = now.flatten()
        rows = torch.cat([flat.view(256, 128).flip(0), torch.zeros(256, 128, dtype=torch.int32)])
        steps.append((now, rows.to(cuda).view(torch.bfloat16).view(512, 1, 256)))
    outs = []
    torch.cuda.synchronize()
    for _, key in steps:
        A.store_kvcache(key, key, plane, scratch, slots)
        outs.append(A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, table, case.scale))
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    for (now, _), out in zip(steps, outs):
        ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, now, case.scale)
        assert_close_to_oracle(out, ref, f"{hq}/{hkv} heads of {d}, {len(lens)} sequences")


@pytest.mark.parametrize("hq,hkv,d,batch", [(16, 8, 128, 1), (16, 8, 128, 16), (8, 2, 128, 128), (14, 2, 64, 20), (2, 1, 64, 129)])
def test_step_whose_inputs_the_kernel_just_before_writes(cuda, hq, hkv, d, batch):
    """Lengths, table and slots are in the rows of a cache that the launch in front stores to: a step that has listed
    its tiles by what was there before must store and read by what is there now, and report nothing."""
    g = torch.Generator().manual_seed(batch)
    case = W.make_decode_case(41, batch, 1, 1, hq, hkv, d, context_lens=torch.randint(200, 1500, (batch,), generator=g).tolist())
    dev = case.to(cuda)
    width = case.block_tables.shape[1]
    plane = torch.zeros(2, 256, 1, 256, dtype=torch.bfloat16, device=cuda)  # rows of 128 int32
    words = plane[1].view(-1).view(torch.int32)
    lens, slots, table = words[:batch], words[batch:2 * batch], words[2 * batch:(2 + width) * batch].view(batch, width)
    backwards = torch.arange(511, -1, -1, dtype=torch.int32, device=cuda)  # the rows that hold the words last
    scratch = torch.zeros_like(plane)
    steps = []
    for _ in range(4):
        perm = torch.cat([torch.randperm(case.k_cache.shape[0], generator=g).int(), torch.tensor([-1], dtype=torch.int32)])
        now = (case.context_lens * torch.rand(batch, generator=g)).int() + 1
        t = perm[case.block_tables.long()]
        s = t[torch.arange(batch), ((now - 1) // 256).long()] * 256 + (now - 1) % 256
        flat = torch.zeros(256 * 128, dtype=torch.int32)
        flat[:(2 + width) * batch] = torch.cat([now, s, t.flatten()])
        rows = torch.cat([flat.view(256, 128).flip(0), torch.zeros(256, 128, dtype=torch.int32)])
        steps.append((now, s, t, rows.to(cuda).view(torch.bfloat16).view(512, 1, 256)))
    outs = []
    torch.cuda.synchronize()
    for *_, key in steps:
        A.store_kvcache(key, key, plane, scratch, backwards)
        outs.append(A.decode_step(dev.q, dev.k_new, dev.v_new, dev.k_cache, dev.v_cache, slots, lens, table, case.scale))
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    for (now, s, t, _), out in zip(steps, outs):
        R.store_kvcache_ref(case.k_new, case.v_new, case.k_cache, case.v_cache, s)
        assert_close_to_oracle(out, R.decode_ref(case.q, case.k_cache, case.v_cache, now, t, case.scale), f"batch {batch}")
    assert torch.equal(dev.k_cache.cpu().view(torch.int16), case.k_cache.view(torch.int16))


def _units_to_a_range(cuda, lens, hq, hkv, d):
    """Ranges that a KV head's units are cut into, and the units."""
    unit, blocks = _lib.decode_plan(len(lens), 32, hq, hkv, d)
    return blocks // hkv, sum(-(-n // unit) for n in lens)


@pytest.mark.parametrize("hq,hkv,d,lens", [(32, 32, 128, [3500] * 6), (32, 32, 128, [2100, 5, 4000, 70, 3333, 1, 6000, 4321, 0]), (64, 64, 64, [3000] * 7)])
def test_step_with_more_units_in_a_range_than_a_warp_lists(cuda, hq, hkv, d, lens):
    """Over 32 units to a thread block, of a batch small enough to be listed ahead: new tokens on both sides of the 32nd."""
    ranges, units = _units_to_a_range(cuda, lens, hq, hkv, d)
    assert units > 32 * ranges or torch.cuda.get_device_properties(cuda).multi_processor_count != 148
    case = W.make_decode_case(61, len(lens), 1, 1, hq, hkv, d, context_lens=lens)
    sep, fus = case.to(cuda), case.to(cuda)
    A.store_kvcache(sep.k_new, sep.v_new, sep.k_cache, sep.v_cache, sep.slot_mapping)
    expected = A.decode_paged(sep.q, sep.k_cache, sep.v_cache, sep.context_lens, sep.block_tables, case.scale)
    for _ in range(2):
        got = A.decode_step(fus.q, fus.k_new, fus.v_new, fus.k_cache, fus.v_cache, fus.slot_mapping, fus.context_lens, fus.block_tables,
                            case.scale)
    torch.cuda.synchronize()
    assert torch.equal(fus.k_cache, sep.k_cache) and torch.equal(fus.v_cache, sep.v_cache)
    assert torch.equal(got, expected)
    R.store_kvcache_ref(case.k_new, case.v_new, case.k_cache, case.v_cache, case.slot_mapping)
    assert_close_to_oracle(got, R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale), f"{lens}")
    assert _lib.read_status() == 0


@pytest.mark.parametrize("entries", [[(0, 8)], [(1, 13)], [(0, 8), (1, 13)]])
def test_step_whose_only_change_lies_beyond_the_list(cuda, entries):
    """Six sequences of 3500 tokens, 32 KV heads: ranges of 37 units, the first 32 of them listed.  The launch in front
    changes only table entries of units past the 32nd of a range (and the slot of the new token in the second one's)."""
    hq, hkv, d, lens = 32, 32, 128, [3500] * 6
    ranges, units = _units_to_a_range(cuda, lens, hq, hkv, d)
    if torch.cuda.get_device_properties(cuda).multi_processor_count == 148:
        assert (ranges, units) == (9, 330)
        for b, i in entries:  # 55 units a sequence, four to a block; the first six ranges have 37
            spots = [b * 55 + u for u in range(4 * i, min(4 * i + 4, 55))]
            assert all(s < 6 * 37 and s % 37 >= 32 for s in spots)
    case = W.make_decode_case(67, 6, 1, 1, hq, hkv, d, context_lens=lens)
    dev = case.to(cuda)
    width, used = case.block_tables.shape[1], set(case.block_tables.flatten().tolist())
    spare = [x for x in range(case.k_cache.shape[0]) if x not in used]
    plane = torch.zeros(2, 256, 1, 256, dtype=torch.bfloat16, device=cuda)  # rows of 128 int32
    words = plane[1].view(-1).view(torch.int32)
    slots, table = words[:6], words[6:6 + 6 * width].view(6, width)
    backwards = torch.arange(511, -1, -1, dtype=torch.int32, device=cuda)  # the rows that hold the words last
    scratch = torch.zeros_like(plane)
    steps = []
    for i in range(4):
        t = case.block_tables.clone()
        for k, (b, e) in enumerate(entries):
            t[b, e] = spare[2 * k + i % 2] if i else t[b, e]
        s = t[:, 13] * 256 + 3499 % 256
        flat = torch.zeros(256 * 128, dtype=torch.int32)
        flat[:6 + 6 * width] = torch.cat([s, t.flatten()])
        rows = torch.cat([flat.view(256, 128).flip(0), torch.zeros(256, 128, dtype=torch.int32)])
        steps.append((s, t, rows.to(cuda).view(torch.bfloat16).view(512, 1, 256)))
    outs = []
    torch.cuda.synchronize()
    for *_, key in steps:
        A.store_kvcache(key, key, plane, scratch, backwards)
        outs.append(A.decode_step(dev.q, dev.k_new, dev.v_new, dev.k_cache, dev.v_cache, slots, dev.context_lens, table, case.scale))
    torch.cuda.synchronize()
    assert _lib.read_status() == 0
    for (s, t, _), out in zip(steps, outs):
        R.store_kvcache_ref(case.k_new, case.v_new, case.k_cache, case.v_cache, s)
        assert_close_to_oracle(out, R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, t, case.scale), f"{entries}")
    assert torch.equal(dev.k_cache.cpu().view(torch.int16), case.k_cache.view(torch.int16))


@pytest.mark.parametrize("batch", [33, 129])
def test_a_batch_of_empty_sequences_completes_after_its_store(cuda, batch):
    """The layer call of more than 32 sequences that are all empty has no tile to stream.  The launch
    behind it takes its completion for that of the store as well, here one of 48 MB whose last rows
    are read: they must be there."""
    hq, hkv, d = 16, 8, 128
    case = W.make_decode_case(43, 4, 1, 1, hq, hkv, d, context_lens=[1, 255, 256, 257])
    dev = case.to(cuda)
    n_new = 12000
    slots = torch.full((n_new,), -1, dtype=torch.int32, device=cuda)  # the last rows are tokens of the batch read afterwards
    slots[-4:] = dev.slot_mapping
    kv = torch.randn(2, n_new, hkv, d, generator=torch.Generator().manual_seed(batch)).bfloat16().to(cuda)
    spare = torch.arange(256, dtype=torch.int32, device=cuda) + 256 * dev.k_cache.shape[0]
    slots[:-4] = spare.repeat(n_new // 256 + 1)[:n_new - 4]
    kv[:, :-4] = 0  # rows that go to the same slot are the same
    pad = torch.zeros(1, 256, hkv, d, dtype=torch.bfloat16, device=cuda)
    layer = A.Attention(hq, d, dev.scale, hkv)
    layer.k_cache, layer.v_cache = torch.cat([dev.k_cache, pad]), torch.cat([dev.v_cache, pad])
    zeros = torch.zeros(batch, dtype=torch.int32, device=cuda)
    q, table = torch.randn(batch, hq * d, device=cuda).bfloat16(), torch.zeros(batch, 16, dtype=torch.int32, device=cuda)
    for _ in range(3):
        torch.cuda.synchronize()
        C.set_context(False, slot_mapping=slots, context_lens=zeros, block_tables=table)
        empty = layer(q, kv[0].view(n_new, -1), kv[1].view(n_new, -1))
        C.reset_context()
        got = A.decode_paged(dev.q, layer.k_cache, layer.v_cache, dev.context_lens, dev.block_tables, dev.scale)
        torch.cuda.synchronize()
        assert not empty.any()
        R.store_kvcache_ref(kv[0, -4:].cpu(), kv[1, -4:].cpu(), case.k_cache, case.v_cache, case.slot_mapping)
        ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
        assert_close_to_oracle(got, ref, f"behind {batch} empty sequences")
        kv[:, -4:] = -kv[:, -4:]
    assert _lib.read_status() == 0


@pytest.mark.parametrize("tp", [2, 4, 8])
def test_head_sharded_ranks_reassemble_the_unsharded_result(cuda, tp):
    """Tensor parallelism: rank r holds query heads [r*Hq/tp, ...) and KV heads [r*Hkv/tp, ...) of
    every cache row (nanovllm/engine/model_runner.py:117, nanovllm/layers/linear.py:141-163) and
    sees identical metadata.  All shards run here on one GPU, one after the other; their outputs
    side by side must match the oracle (and the unsharded kernel's output within rounding: the
    number of ranges, hence where a sequence is cut, depends on the KV heads per rank)."""
    hq, hkv, d = 32, 8, 128
    case = W.make_decode_case(18, 6, 1, 1, hq, hkv, d, context_lens=[700, 1, 2049, 256, 3000, 513], table_width=12)
    dev = case.to(cuda)
    full = A.decode_paged(dev.q, dev.k_cache, dev.v_cache, dev.context_lens, dev.block_tables, case.scale)
    parts = []
    for r in range(tp):
        qs = dev.q[:, r * hq // tp:(r + 1) * hq // tp].contiguous()
        ks = dev.k_cache[:, :, r * hkv // tp:(r + 1) * hkv // tp].contiguous()
        vs = dev.v_cache[:, :, r * hkv // tp:(r + 1) * hkv // tp].contiguous()
        parts.append(A.decode_paged(qs, ks, vs, dev.context_lens, dev.block_tables, case.scale))
    torch.cuda.synchronize()
    ref = R.decode_ref(case.q, case.k_cache, case.v_cache, case.context_lens, case.block_tables, case.scale)
    assert_close_to_oracle(torch.cat(parts, dim=1), ref, f"tp{tp}")
    assert (torch.cat(parts, dim=1).float() - full.float()).abs().max().item() <= 2e-2


SMALL_THEN_CAPTURE = """
import sys
import torch
from nano_vllm_b200 import _lib, attention as A, context as C, workloads as W
dev = torch.device("cuda:0")


def decode(batch, one_launch):
    c = W.make_decode_case(50 + batch, batch, 1, 1, 16, 8, 128, context_lens=([700, 64, 1000, 129] * 8)[:batch], device=dev).to(dev)
    if one_launch is None:
        return lambda: A.decode_paged(c.q, c.k_cache, c.v_cache, c.context_lens, c.block_tables, c.scale)
    if one_launch:
        return lambda: A.decode_step(c.q, c.k_new, c.v_new, c.k_cache, c.v_cache, c.slot_mapping, c.context_lens, c.block_tables, c.scale)
    layer = A.Attention(16, 128, c.scale, 8)
    layer.k_cache, layer.v_cache = c.k_cache, c.v_cache

    def run():
        C.set_context(False, slot_mapping=c.slot_mapping, context_lens=c.context_lens, block_tables=c.block_tables)
        return layer(c.q.view(batch, -1), c.k_new.view(batch, -1), c.v_new.view(batch, -1))
    return run


def prefill(batch):
    c = W.make_prefill_case(60 + batch, batch, 1, 1, 16, 8, 128, lengths=([700, 300, 1000, 600] * 8)[:batch], device=dev).to(dev)
    layer = A.Attention(16, 128, c.scale, 8)
    layer.k_cache, layer.v_cache = c.k_cache, c.v_cache

    def run():
        C.set_context(True, c.cu_seqlens_q, c.cu_seqlens_k, c.max_seqlen_q, c.max_seqlen_k, c.slot_mapping, None, c.block_tables)
        return layer(c.q.view(c.q.shape[0], -1), c.k.view(c.q.shape[0], -1), c.v.view(c.q.shape[0], -1))
    return run


kind = sys.argv[1]
small, large = {"plain": (decode(2, None), decode(16, None)), "step": (decode(2, True), decode(16, True)),
                "layer": (decode(2, False), decode(32, False)), "prefill": (prefill(2), prefill(16))}[kind]
small()
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    got = large()
for _ in range(2):
    graph.replay()
torch.cuda.synchronize()
replayed = got.clone()
assert torch.equal(large(), replayed) and replayed.abs().max() > 0
assert _lib.read_status() == 0
print("captured")
"""


@pytest.mark.parametrize("kind", ["plain", "step", "layer", "prefill"])
def test_a_larger_batch_may_be_captured_after_a_small_one_has_run(cuda, kind):
    """The first call of a head_dim sets up whatever kernel a later one of it takes, so that this one may be the first inside
    a capture: a process of its own, as every kernel has run here already."""
    root = Path(__file__).resolve().parents[1]
    done = subprocess.run([sys.executable, "-c", SMALL_THEN_CAPTURE, kind], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "captured" in done.stdout, done.stderr[-2000:]

"""Varlen causal GQA prefill on the GPU, through the C ABI, against the fp32 CPU oracle."""
import ctypes
import random

import pytest
import torch

from conftest import assert_close_to_oracle
from nano_vllm_b200 import _lib, attention as A, context as C, workloads as W
from oracle import paged_attention_ref as R

pytestmark = pytest.mark.gpu


def _check(cuda, case, what):
    dev = case.to(cuda)
    if case.k_cache.numel():
        A.store_kvcache(dev.k, dev.v, dev.k_cache, dev.v_cache, dev.slot_mapping)
        R.store_kvcache_ref(case.k, case.v, case.k_cache, case.v_cache, case.slot_mapping)
    if case.block_tables is not None:
        out = A.prefill_varlen(dev.q, dev.k_cache, dev.v_cache, dev.cu_seqlens_q, dev.cu_seqlens_k,
                               case.max_seqlen_q, case.max_seqlen_k, case.scale, block_tables=dev.block_tables)
        ref = R.prefill_ref(case.q, case.k_cache, case.v_cache, case.cu_seqlens_q, case.cu_seqlens_k, case.scale,
                            case.block_tables)
    else:
        out = A.prefill_varlen(dev.q, dev.k, dev.v, dev.cu_seqlens_q, dev.cu_seqlens_k,
                               case.max_seqlen_q, case.max_seqlen_k, case.scale)
        ref = R.prefill_ref(case.q, case.k, case.v, case.cu_seqlens_q, case.cu_seqlens_k, case.scale)
    torch.cuda.synchronize()
    assert_close_to_oracle(out, ref, what)
    if case.k_cache.numel():
        assert torch.equal(dev.k_cache.cpu().view(torch.int16), case.k_cache.view(torch.int16))
        assert torch.equal(dev.v_cache.cpu().view(torch.int16), case.v_cache.view(torch.int16))
    assert _lib.read_status() == 0


def test_cfg2(cuda):
    """The prefill configuration at full size: 64 prompts in [100,1024], every 4th shares 1-3 cached blocks."""
    case = W.cfg2_prefill()
    assert case.block_tables is not None and int(case.cu_seqlens_k[-1]) > int(case.cu_seqlens_q[-1])
    _check(cuda, case, "cfg2")


@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (32, 8, 128), (14, 2, 64), (4, 1, 128), (2, 2, 64),
                                      (8, 1, 128), (12, 2, 64), (16, 2, 64), (10, 2, 128), (6, 2, 128), (14, 2, 128)])
def test_packed_lengths(cuda, hq, hkv, d):
    case = W.make_prefill_case(21, 8, 1, 1, hq, hkv, d, share_every=0,
                               lengths=[1, 100, 127, 128, 129, 256, 257, 1024])
    assert case.block_tables is None
    _check(cuda, case, f"packed hq{hq} hkv{hkv} d{d}")


@pytest.mark.parametrize("d", [64, 128])
def test_prefix_cached_blocks(cuda, d):
    """Lk - Lq in {0, 256, 768}; a fully cached prompt leaves Lq == 0."""
    case = W.make_prefill_case(22, 6, 1, 1, 8, 2, d, lengths=[1024, 1024, 300, 257, 512, 512],
                               shared_blocks=[0, 3, 0, 1, 0, 2])
    lq = (case.cu_seqlens_q[1:] - case.cu_seqlens_q[:-1]).tolist()
    assert lq == [1024, 256, 300, 1, 512, 0]
    _check(cuda, case, f"prefix d{d}")


def test_warmup_shape_without_cache(cuda):
    """Engine warm-up: 4096-token sequences before the cache exists
    (nanovllm/engine/model_runner.py:96-108)."""
    case = W.make_prefill_case(23, 2, 1, 1, 16, 8, 128, lengths=[4096, 4096], with_cache=False)
    _check(cuda, case, "warmup")


def test_strided_v_view(cuda):
    hq, hkv, d, n = 16, 8, 128, 700
    g = torch.Generator().manual_seed(24)
    qkv = torch.randn(n, (hq + 2 * hkv) * d, generator=g).bfloat16()
    cu = torch.tensor([0, 300, 700], dtype=torch.int32)
    q, k, v = (t.view(n, -1, d) for t in qkv.split([hq * d, hkv * d, hkv * d], dim=-1))
    qd, kd, vd = (t.view(n, -1, d) for t in qkv.to(cuda).split([hq * d, hkv * d, hkv * d], dim=-1))
    out = A.prefill_varlen(qd, kd, vd, cu.to(cuda), cu.to(cuda), 400, 400, d ** -0.5)
    ref = R.prefill_ref(q, k, v, cu, cu, d ** -0.5)
    assert_close_to_oracle(out, ref, "strided")


@pytest.mark.parametrize("d", [64, 128])
def test_stale_cache_rows_past_the_sequence_cannot_leak(cuda, d):
    """A partly filled last block holds NaN/Inf past the sequence end; outputs stay finite."""
    case = W.make_prefill_case(25, 3, 1, 1, 8, 2, d, lengths=[300, 700, 513], shared_blocks=[0, 1, 2])
    assert case.block_tables is not None
    case.k_cache[:] = float("nan")
    case.v_cache[:] = float("inf")
    _check(cuda, case, f"stale d{d}")


@pytest.mark.parametrize("impl,d", [("mma", 64), ("mma", 128), ("tcp", 64), ("tcp", 128)])
def test_every_prefill_kernel_on_the_same_case(cuda, monkeypatch, impl, d):
    """NVLLM_PREFILL_IMPL=mma selects the warp-level cross-check kernel instead of the persistent
    tcgen05 kernel (tcp, the default); both must agree with the oracle on packed and on
    prefix-cached inputs."""
    monkeypatch.setenv("NVLLM_PREFILL_IMPL", impl)
    case = W.make_prefill_case(26, 7, 1, 1, 8, 2, d, lengths=[1, 130, 1024, 1024, 513, 700, 64],
                               shared_blocks=[0, 0, 0, 3, 0, 2, 0])
    _check(cuda, case, f"{impl} d{d} prefix")
    case = W.make_prefill_case(27, 5, 1, 1, 8, 8, d, share_every=0, lengths=[257, 2, 900, 128, 64])
    _check(cuda, case, f"{impl} d{d} packed")


@pytest.mark.parametrize("impl", ["", "mma"])
@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (14, 2, 64), (3, 3, 64)])
@pytest.mark.parametrize("lengths", [[1], [63, 1, 130], [3000, 2500]])
def test_layer_stores_packed_rows_as_the_store_does(cuda, monkeypatch, impl, hq, hkv, d, lengths):
    """The prefill's own copy of the rows into the cache: fewer rows than lanes, several trips, K and V of
    different strides, rows without a slot, a slot past the cache."""
    monkeypatch.setenv("NVLLM_PREFILL_IMPL", impl)
    dev = W.make_prefill_case(41, len(lengths), 1, 1, hq, hkv, d, lengths=lengths, share_every=0).to(cuda)
    n = dev.q.shape[0]
    qkv = torch.cat([dev.q.view(n, -1), dev.k.view(n, -1), dev.v.view(n, -1)], dim=1)
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
    v = v.contiguous()
    slots = dev.slot_mapping.clone()
    slots[n // 3::7] = -1
    layer = A.Attention(hq, d, dev.scale, hkv)
    layer.k_cache, layer.v_cache = dev.k_cache.clone(), dev.v_cache.clone()
    k2, v2 = dev.k_cache.clone(), dev.v_cache.clone()
    for status in (0, 1):
        C.set_context(True, dev.cu_seqlens_q, dev.cu_seqlens_k, dev.max_seqlen_q, dev.max_seqlen_k, slots, None, None)
        got = layer(q, k, v)
        C.reset_context()
        A.store_kvcache(dev.k, dev.v, k2, v2, torch.where(slots < k2.shape[0] * 256, slots, -1))
        want = A.prefill_varlen(dev.q, dev.k, dev.v, dev.cu_seqlens_q, dev.cu_seqlens_k, dev.max_seqlen_q, dev.max_seqlen_k, dev.scale)
        torch.cuda.synchronize()
        assert torch.equal(got.view_as(want), want)
        assert torch.equal(layer.k_cache, k2) and torch.equal(layer.v_cache, v2)
        assert _lib.read_status() == status
        slots[n - 1] = k2.shape[0] * 256  # NVLLM_STATUS_BAD_SLOT the second time


@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (32, 8, 128), (14, 2, 64), (3, 3, 64)])
def test_layer_stores_every_packed_row_from_the_key_tiles(cuda, hq, hkv, d):
    """More items than blocks: rows are stored from the key tiles.  Sequences with more keys than queries, fewer, or
    no query at all, rows in front of the first sequence and behind the last, ends around a tile's, scattered slots."""
    lq = [1, 0, 63, 64, 65, 700, 0, 127, 129, 30, 1000, 300, 1, 40] * 3
    lk = [1, 70, 63, 64, 200, 700, 1, 128, 100, 300, 1000, 310, 129, 40] * 3
    front, behind = 3, 70
    gen = torch.Generator(device=cuda).manual_seed(5)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device=cuda).bfloat16()
    n_q, n_k = sum(lq), front + sum(lk) + behind
    q, k, v = rand(n_q, hq * d), rand(n_k, hkv * d), rand(n_k, 2 * hkv * d)[:, : hkv * d]
    cu_q = torch.tensor([0] + lq, device=cuda).cumsum(0).int()
    cu_k = (torch.tensor([0] + lk, device=cuda).cumsum(0) + front).int()
    blocks = n_k // 256 + 3
    slots = torch.randperm(blocks * 256, generator=gen, device=cuda)[:n_k].int()
    slots[::11] = -1
    layer = A.Attention(hq, d, d ** -0.5, hkv)
    layer.k_cache, layer.v_cache = rand(blocks, 256, hkv, d), rand(blocks, 256, hkv, d)
    k2, v2 = layer.k_cache.clone(), layer.v_cache.clone()
    A.store_kvcache(k.view(n_k, hkv, d), v.unflatten(1, (hkv, d)), k2, v2, slots)
    want = A.prefill_varlen(q.view(n_q, hq, d), k.view(n_k, hkv, d), v.unflatten(1, (hkv, d)), cu_q, cu_k, max(lq), max(lk), d ** -0.5)
    C.set_context(True, cu_q, cu_k, max(lq), max(lk), slots, None, None)
    for _ in range(2):
        got = layer(q, k, v)
    C.reset_context()
    torch.cuda.synchronize()
    assert torch.equal(got.view_as(want), want)
    assert torch.equal(layer.k_cache, k2) and torch.equal(layer.v_cache, v2)
    assert _lib.read_status() == 0


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (32, 8, 128), (14, 2, 64), (4, 4, 64)])
def test_layer_through_the_table_reads_and_stores_new_rows_as_store_then_prefill_does(cuda, hq, hkv, d, odd):
    """Cached blocks that were there before, that another sequence fills in the same step, and that end ragged; with
    ``odd`` also rows without a slot, slots that are not the table's, cached tokens that end inside a block or a
    tile, one block in two tables as new, more queries than keys, rows behind the last sequence."""
    lq = [1, 63, 64, 65, 255, 256, 257, 700, 1000, 2000, 130, 40, 512, 900, 300, 777] * 2
    cached = [0, 256, 512, 0, 1024, 0, 256, 0, 512, 0, 256, 0, 0, 256, 0, 0] * 2
    if odd:
        cached[1], cached[4], cached[20], cached[11], cached[17] = 100, 64, 500, -20, 320
    lk = [a + c for a, c in zip(lq, cached)]
    behind = 30 if odd else 0
    gen = torch.Generator(device=cuda).manual_seed(9)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device=cuda).bfloat16()
    width = max(lk) // 256 + 3
    counts = [(n + 255) // 256 for n in lk]
    blocks = sum(counts) + 5
    ids = torch.randperm(blocks, generator=gen, device=cuda).cpu().tolist()
    tables, at = [], 0
    for n in counts:
        tables.append(ids[at:at + n] + [-1] * (width - n))
        at += n
    tables[6][0] = tables[5][0]     # full new blocks of another sequence
    tables[8][:2] = tables[7][:2]
    tables[13][0] = tables[3][0]    # a block that its sequence fills only in part
    slots = []
    for a, c, row in zip(lq, cached, tables):
        slots += [row[p // 256] * 256 + p % 256 if p >= 0 else -1 for p in range(c, c + a)]
    slots = torch.tensor(slots, dtype=torch.int32)
    if odd:
        starts = torch.tensor([0] + lq).cumsum(0)
        slots[starts[7] + 100] = -1
        slots[starts[9] + 70: starts[9] + 75] = -1
        spare = ids[-1] * 256
        slots[starts[12]: starts[12] + 64] = torch.arange(spare, spare + 64, dtype=torch.int32)
        tables[15][1] = tables[14][1]  # both fill it: only one of them gives it slots
        slots[starts[15] + 256: starts[15] + 512] = -1
        slots = torch.cat([slots, torch.arange(spare + 100, spare + 100 + behind, dtype=torch.int32)])
    slots = slots.to(cuda)
    n_q, n_k = sum(lq), sum(lq) + behind
    q, k, v = rand(n_q, hq * d), rand(n_k, hkv * d), rand(n_k, 2 * hkv * d)[:, : hkv * d]
    cu = lambda x: torch.tensor([0] + x, device=cuda).cumsum(0).int()
    bt = torch.tensor(tables, dtype=torch.int32, device=cuda)
    layer = A.Attention(hq, d, d ** -0.5, hkv)
    layer.k_cache, layer.v_cache = rand(blocks, 256, hkv, d), rand(blocks, 256, hkv, d)
    for again in range(2):
        k2, v2 = layer.k_cache.clone(), layer.v_cache.clone()
        A.store_kvcache(k.view(n_k, hkv, d), v.unflatten(1, (hkv, d)), k2, v2, slots)
        want = A.prefill_varlen(q.view(n_q, hq, d), k2, v2, cu(lq), cu(lk), max(lq), max(lk), d ** -0.5, bt)
        C.set_context(True, cu(lq), cu(lk), max(lq), max(lk), slots, None, bt)
        got = layer(q, k, v)
        C.reset_context()
        torch.cuda.synchronize()
        assert torch.equal(layer.k_cache, k2) and torch.equal(layer.v_cache, v2)
        assert torch.equal(got.view_as(want), want)
        assert _lib.read_status() == 0
        k, v, bt = -k, -v, bt.clone()


@pytest.mark.parametrize("front", [1, 255, 256, 700])
@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (14, 2, 64)])
def test_layer_through_the_table_stores_rows_in_front_of_the_first_sequence(cuda, hq, hkv, d, front):
    """More items than blocks and cu_seqlens_q[0] > 0: the rows in front belong to no sequence and are stored like those
    behind the last."""
    lq, cached, behind = [700, 300, 64, 1000, 513] * 4, [0, 256, 512, 0, 256] * 4, 3
    lk = [a + c for a, c in zip(lq, cached)]
    gen = torch.Generator(device=cuda).manual_seed(front)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device=cuda).bfloat16()
    counts = [(n + 255) // 256 for n in lk]
    blocks = sum(counts) + 8
    ids = torch.randperm(blocks, generator=gen, device=cuda).cpu().tolist()
    tables, slots, at = [], [], 0
    for a, c, n in zip(lq, cached, counts):
        tables.append(ids[at:at + n] + [-1] * (max(counts) - n))
        slots += [tables[-1][p // 256] * 256 + p % 256 for p in range(c, c + a)]
        at += n
    spare = [b * 256 + i for b in ids[at:] for i in range(256)]
    slots = torch.tensor(spare[:front] + slots + spare[front:front + behind], dtype=torch.int32, device=cuda)
    slots[1 + front // 2] = -1
    n = front + sum(lq) + behind
    q, k, v = rand(n, hq * d), rand(n, hkv * d), rand(n, hkv * d)
    cu_q = (torch.tensor([0] + lq, device=cuda).cumsum(0) + front).int()
    cu_k = torch.tensor([0] + lk, device=cuda).cumsum(0).int()
    bt = torch.tensor(tables, dtype=torch.int32, device=cuda)
    layer = A.Attention(hq, d, d ** -0.5, hkv)
    layer.k_cache, layer.v_cache = rand(blocks, 256, hkv, d), rand(blocks, 256, hkv, d)
    k2, v2 = layer.k_cache.clone(), layer.v_cache.clone()
    A.store_kvcache(k.view(n, hkv, d), v.view(n, hkv, d), k2, v2, slots)
    want = A.prefill_varlen(q.view(n, hq, d), k2, v2, cu_q, cu_k, max(lq), max(lk), d ** -0.5, bt)
    C.set_context(True, cu_q, cu_k, max(lq), max(lk), slots, None, bt)
    got = layer(q, k, v)
    C.reset_context()
    torch.cuda.synchronize()
    assert torch.equal(layer.k_cache, k2) and torch.equal(layer.v_cache, v2)
    assert torch.equal(got.view_as(want)[front:n - behind], want[front:n - behind])
    assert _lib.read_status() == 0


@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (4, 2, 128)])
@pytest.mark.parametrize("batch,width", [(16, 1024), (33, 9), (129, 127), (300, 54), (300, 55)])
def test_layer_through_wide_tables_finds_blocks_that_others_fill(cuda, hq, hkv, d, batch, width):
    """Every third sequence has blocks of the one before it cached, up to ten of them and behind others of its own; tables
    near and past the largest that are routed, and more sequences than one trip of the search takes."""
    r = random.Random(batch)
    lq = [r.choice([1, 64, 257, 300, 513, 700]) for _ in range(batch)]
    lq[1], lq[7], lq[batch - 2] = 2300, 2560, 1024
    cached, tables, fresh = [], [], 0
    for i in range(batch):
        own = list(range(fresh, fresh + (i % 4 == 2)))  # a block that was there before
        fresh += len(own)
        if i % 3 == 2:
            own += tables[i - 1][cached[i - 1] // 256:][:min(lq[i - 1] // 256, width - 5)]
        if len(own) + 4 > width or len(own) * 256 + lq[i] > width * 256:
            own, lq[i] = own[:1], min(lq[i], 700)
        cached.append(len(own) * 256)
        n = (lq[i] + 255) // 256
        tables.append(own + list(range(fresh, fresh + n)))
        fresh += n
    lk = [a + c for a, c in zip(lq, cached)]
    gen = torch.Generator(device=cuda).manual_seed(batch)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device=cuda).bfloat16()
    perm = torch.randperm(fresh + 2, generator=gen, device=cuda).cpu()
    tables = [[int(perm[x]) for x in row] for row in tables]
    slots = [row[p // 256] * 256 + p % 256 for a, c, row in zip(lq, cached, tables) for p in range(c, c + a)]
    slots = torch.tensor(slots, dtype=torch.int32, device=cuda)
    bt = torch.tensor([row + [-1] * (width - len(row)) for row in tables], dtype=torch.int32, device=cuda)
    n = sum(lq)
    q, k, v = rand(n, hq * d), rand(n, hkv * d), rand(n, hkv * d)
    cu = lambda x: torch.tensor([0] + x, device=cuda).cumsum(0).int()
    layer = A.Attention(hq, d, d ** -0.5, hkv)
    layer.k_cache, layer.v_cache = rand(fresh + 2, 256, hkv, d), rand(fresh + 2, 256, hkv, d)
    k2, v2 = layer.k_cache.clone(), layer.v_cache.clone()
    A.store_kvcache(k.view(n, hkv, d), v.view(n, hkv, d), k2, v2, slots)
    want = A.prefill_varlen(q.view(n, hq, d), k2, v2, cu(lq), cu(lk), max(lq), max(lk), d ** -0.5, bt)
    C.set_context(True, cu(lq), cu(lk), max(lq), max(lk), slots, None, bt)
    got = layer(q, k, v)
    C.reset_context()
    torch.cuda.synchronize()
    assert torch.equal(layer.k_cache, k2) and torch.equal(layer.v_cache, v2)
    assert torch.equal(got.view_as(want), want)
    assert _lib.read_status() == 0


@pytest.mark.parametrize("hq,hkv,d", [(16, 8, 128), (14, 2, 64), (2, 2, 64)])
@pytest.mark.parametrize("lengths", [[300] * 6, [1, 700], [129, 1, 64, 65, 257, 3, 2, 128], [64] * 18, [63] * 19])
def test_every_item_of_a_launch_with_an_item_to_a_block(cuda, hq, hkv, d, lengths):
    """The items of several short prompts go out in another order than the list's: none twice, none left out."""
    case = W.make_prefill_case(47, len(lengths), 1, 1, hq, hkv, d, lengths=lengths, share_every=0)
    _check(cuda, case, f"{lengths} hq{hq} d{d}")


@pytest.mark.parametrize("hq,hkv", [(14, 2), (7, 1), (4, 4)])
@pytest.mark.parametrize("lengths,share", [([130] * 40, 0), ([257] * 40, 4), ([500] * 20 + [510] * 19, 0), ([511] * 40, 4), ([128] * 45, 0)])
def test_several_items_a_block_of_prompts_of_one_length(cuda, hq, hkv, lengths, share):
    """head_dim 64, more items than blocks: all prompts' long tiles go first, packed and through the table."""
    case = W.make_prefill_case(53, len(lengths), 1, 1, hq, hkv, 64, lengths=lengths, share_every=share)
    _check(cuda, case, f"{len(lengths)} of {lengths[0]} hq{hq}")


@pytest.mark.parametrize("hq,hkv,batch", [(14, 2, 70), (7, 1, 140), (4, 4, 180)])
@pytest.mark.parametrize("table", [False, True])
def test_rows_are_stored_with_three_blocks_to_an_sm(cuda, hq, hkv, batch, table):
    """head_dim 64, enough items for three blocks an SM: packed rows are stored by one warp of each.  Ends around a tile's,
    sequences without a query, rows in front and behind, scattered slots; through the table with blocks that others fill."""
    d, r = 64, random.Random(batch)
    lens = [r.choice([320, 319, 320, 257, 256, 255, 193, 320] + [0] * (not table)) for _ in range(batch)]
    gen = torch.Generator(device=cuda).manual_seed(batch)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device=cuda).bfloat16()
    layer = A.Attention(hq, d, d ** -0.5, hkv)
    if table:
        c = W.make_prefill_case(59, batch, 1, 1, hq, hkv, d, device=cuda, lengths=lens, shared_blocks=[(i % 4 == 3) * min(1, min(lens[i - 1], lens[i] - 1) // 256) for i in range(batch)]).to(cuda)
        q, k, v, cu_q, cu_k, slots, bt = c.q, c.k, c.v, c.cu_seqlens_q, c.cu_seqlens_k, c.slot_mapping, c.block_tables
        layer.k_cache, layer.v_cache = c.k_cache, c.v_cache
        max_q, max_k = c.max_seqlen_q, c.max_seqlen_k
    else:
        front, behind = 3, 70
        n, n_k = sum(lens), front + sum(lens) + behind
        q, k, v = rand(n, hq, d), rand(n_k, hkv, d), rand(n_k, hkv, d)
        cu_q = torch.tensor([0] + lens, device=cuda).cumsum(0).int()
        cu_k, bt, max_q, max_k = cu_q + front, None, max(lens), max(lens)
        slots = torch.randperm((n_k // 256 + 3) * 256, generator=gen, device=cuda)[:n_k].int()
        slots[::11] = -1
        layer.k_cache, layer.v_cache = rand(n_k // 256 + 3, 256, hkv, d), rand(n_k // 256 + 3, 256, hkv, d)
    k2, v2 = layer.k_cache.clone(), layer.v_cache.clone()
    A.store_kvcache(k, v, k2, v2, slots)
    want = A.prefill_varlen(q, k2 if table else k, v2 if table else v, cu_q, cu_k, max_q, max_k, d ** -0.5, bt)
    C.set_context(True, cu_q, cu_k, max_q, max_k, slots, None, bt)
    for _ in range(3):
        got = layer(q.flatten(1), k.flatten(1), v.flatten(1))
    C.reset_context()
    torch.cuda.synchronize()
    assert torch.equal(layer.k_cache, k2) and torch.equal(layer.v_cache, v2)
    assert torch.equal(got.view_as(want), want)
    assert _lib.read_status() == 0


# ---- head_dim 64 with three blocks to an SM ------------------------------------------------------

FORM_64 = [(14, 2), (7, 1), (16, 4)]
NONE, SPARE, TILES = range(3)


def _takes(cuda, lib, max_q, max_k, total_q, batch, hq, hkv, even, store, total_k=0, table=False):
    """That a launch of head_dim 64 has three blocks to an SM, deals its items out long tiles first where the prompts have the
    same number of them, and stores rows as named."""
    out = [ctypes.c_int32() for _ in range(3)]
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    assert lib.nvllm_prefill_plan(total_q, total_k, batch, max_q, max_k, hq, hkv, 64, 3 if table else 1 if store else 0, sms, *(ctypes.byref(x) for x in out)) == 0
    assert [x.value for x in out] == [3, 0 if even else 1 << 30, store] or sms != 148


@pytest.mark.parametrize("hq,hkv,lens,shared,even", [(*heads, *x) for heads in FORM_64 for x in [
    ([257] * 60, 0, True), ([320] * 40, 0, True), ([511, 512, 512, 510] * 6, 0, True), ([1024] * 15, 0, True), ([576] + [832] * 23, 1, True),
    ([257] + [513] * 59, 1, True), ([700, 320, 1023, 300] * 32, 0, False), ([700, 964, 1023, 556] * 32, 1, False)]] + [
    (4, 4, [1024] * 15, 0, True), (4, 4, [1024] + [1280] * 14, 1, True)])
def test_three_blocks_to_an_sm(cuda, lib, hq, hkv, lens, shared, even):
    """Prompts of the same number of query tiles, whose long tiles go first, and others; packed and through the table, where
    all but the first begin with a cached block."""
    case = W.make_prefill_case(71, len(lens), 1, 1, hq, hkv, 64, lengths=lens, shared_blocks=[shared * (i > 0) for i in range(len(lens))])
    _takes(cuda, lib, case.max_seqlen_q, case.max_seqlen_k, case.q.shape[0], len(lens), hq, hkv, even, NONE, table=bool(shared))
    _check(cuda, case, f"{len(lens)} of {lens[0]} hq{hq}")


@pytest.mark.parametrize("d_heads,batch", [((14, 2), 7), ((7, 1), 14), ((8, 1), 12), ((16, 2), 6)])
@pytest.mark.parametrize("low", [510, 512])
def test_three_blocks_to_an_sm_whose_spare_warps_store_rows(cuda, lib, d_heads, batch, low):
    """Few rows for many items: copied by a warp that no item has to do with.  Rows without a slot, in front of the first
    sequence and behind the last, scattered slots; cache and output against the reference."""
    (hq, hkv), d, r = d_heads, 64, random.Random(low)
    lens = [r.randint(low, 512) for _ in range(batch - 1)] + [512]
    front, behind = 3, 70
    n, n_k = sum(lens), front + sum(lens) + behind
    _takes(cuda, lib, 512, 512, n, batch, hq, hkv, True, SPARE, total_k=n_k)
    gen = torch.Generator().manual_seed(batch)
    rand = lambda *shape: torch.randn(*shape, generator=gen).bfloat16()
    q, k, v = rand(n, hq, d), rand(n_k, hkv, d), rand(n_k, hkv, d)
    cu_q = torch.tensor([0] + lens).cumsum(0).int()
    cu_k = cu_q + front
    blocks = n_k // 256 + 3
    slots = torch.randperm(blocks * 256, generator=gen)[:n_k].int()
    slots[::11] = -1
    k_cache, v_cache = rand(blocks, 256, hkv, d), rand(blocks, 256, hkv, d)
    layer = A.Attention(hq, d, d ** -0.5, hkv)
    layer.k_cache, layer.v_cache = k_cache.to(cuda), v_cache.to(cuda)
    C.set_context(True, cu_q.to(cuda), cu_k.to(cuda), 512, 512, slots.to(cuda), None, None)
    for _ in range(3):
        got = layer(q.to(cuda).flatten(1), k.to(cuda).flatten(1), v.to(cuda).flatten(1))
    C.reset_context()
    torch.cuda.synchronize()
    R.store_kvcache_ref(k, v, k_cache, v_cache, slots)
    assert torch.equal(layer.k_cache.cpu().view(torch.int16), k_cache.view(torch.int16))
    assert torch.equal(layer.v_cache.cpu().view(torch.int16), v_cache.view(torch.int16))
    assert_close_to_oracle(got.view(n, hq, d), R.prefill_ref(q, k, v, cu_q, cu_k, d ** -0.5), f"{lens} hq{hq}")
    assert _lib.read_status() == 0


@pytest.mark.parametrize("hq,hkv,batch", [(14, 2, 70), (7, 1, 140), (16, 4, 70)])
@pytest.mark.parametrize("table", [False, True])
def test_three_blocks_to_an_sm_store_rows_from_the_key_tiles(cuda, lib, hq, hkv, batch, table):
    """Rows stored by one warp of each block: ends around a tile's, sequences of one token and of none, rows in front and behind,
    scattered slots; through the table with blocks that others fill.  Cache and output against the reference."""
    d, r = 64, random.Random(batch + table)
    lens = [r.choice([512, 511, 449, 448, 447, 321, 1 if not table else 300, 512] + [0] * (not table)) for _ in range(batch - 1)] + [512]
    if table:
        shared = [(i % 4 == 3) * min(1, min(lens[i - 1], lens[i] - 1) // 256) for i in range(batch)]
        c = W.make_prefill_case(89, batch, 1, 1, hq, hkv, d, lengths=lens, shared_blocks=shared)
        q, k, v, cu_q, cu_k, slots, bt, k_cache, v_cache = c.q, c.k, c.v, c.cu_seqlens_q, c.cu_seqlens_k, c.slot_mapping, c.block_tables, c.k_cache, c.v_cache
        max_q, max_k, n, n_k = c.max_seqlen_q, c.max_seqlen_k, q.shape[0], k.shape[0]
    else:
        front, behind, bt = 3, 70, None
        n, n_k, max_q, max_k = sum(lens), front + sum(lens) + behind, 512, 512
        gen = torch.Generator().manual_seed(batch)
        rand = lambda *shape: torch.randn(*shape, generator=gen).bfloat16()
        q, k, v = rand(n, hq, d), rand(n_k, hkv, d), rand(n_k, hkv, d)
        cu_q = torch.tensor([0] + lens).cumsum(0).int()
        cu_k = cu_q + front
        blocks = n_k // 256 + 3
        slots = torch.randperm(blocks * 256, generator=gen)[:n_k].int()
        slots[::11] = -1
        k_cache, v_cache = rand(blocks, 256, hkv, d), rand(blocks, 256, hkv, d)
    out = [ctypes.c_int32() for _ in range(3)]
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    assert lib.nvllm_prefill_plan(n, n_k, batch, max_q, max_k, hq, hkv, d, 2 if table else 1, sms, *(ctypes.byref(x) for x in out)) == 0
    assert [x.value for x in out] == [3, 1 << 30, TILES] or sms != 148
    layer = A.Attention(hq, d, d ** -0.5, hkv)
    layer.k_cache, layer.v_cache = k_cache.to(cuda), v_cache.to(cuda)
    C.set_context(True, cu_q.to(cuda), cu_k.to(cuda), max_q, max_k, slots.to(cuda), None, bt.to(cuda) if table else None)
    for _ in range(2):
        got = layer(q.to(cuda).flatten(1), k.to(cuda).flatten(1), v.to(cuda).flatten(1))
    C.reset_context()
    torch.cuda.synchronize()
    R.store_kvcache_ref(k, v, k_cache, v_cache, slots)
    assert torch.equal(layer.k_cache.cpu().view(torch.int16), k_cache.view(torch.int16))
    assert torch.equal(layer.v_cache.cpu().view(torch.int16), v_cache.view(torch.int16))
    ref = R.prefill_ref(q, k_cache, v_cache, cu_q, cu_k, d ** -0.5, bt) if table else R.prefill_ref(q, k, v, cu_q, cu_k, d ** -0.5)
    assert_close_to_oracle(got.view(n, hq, d), ref, f"{batch} sequences hq{hq}")
    assert _lib.read_status() == 0


@pytest.mark.parametrize("hq,hkv", FORM_64)
@pytest.mark.parametrize("table", [False, True])
def test_three_blocks_to_an_sm_see_nothing_behind_a_sequence(cuda, lib, hq, hkv, table):
    """NaN and infinities behind the sequences: in the rest of their last blocks, and in the rows behind the last packed one."""
    lens = [300] + [556 if table else 300] * 47
    case = W.make_prefill_case(73, 48, 1, 1, hq, hkv, 64, lengths=lens, shared_blocks=[int(table and i > 0) for i in range(48)])
    _takes(cuda, lib, 300, max(lens), 300 * 48, 48, hq, hkv, True, NONE, table=table)
    if table:
        case.k_cache[:], case.v_cache[:] = float("nan"), float("inf")
        return _check(cuda, case, "stale rows of the cache")
    k = torch.cat([case.k, torch.full_like(case.k[:64], float("nan"))])
    v = torch.cat([case.v, torch.full_like(case.v[:64], float("inf"))])
    out = A.prefill_varlen(case.q.to(cuda), k.to(cuda), v.to(cuda), case.cu_seqlens_q.to(cuda), case.cu_seqlens_k.to(cuda), 300, 300, case.scale)
    ref = R.prefill_ref(case.q, case.k, case.v, case.cu_seqlens_q, case.cu_seqlens_k, case.scale)
    assert_close_to_oracle(out, ref, "rows behind the last")
    assert _lib.read_status() == 0


@pytest.mark.parametrize("hq,hkv", FORM_64)
@pytest.mark.parametrize("lq", [[320] * 60, [320, 200, 319, 250] * 40])
def test_three_blocks_to_an_sm_with_tiles_without_a_visible_key(cuda, lib, hq, hkv, lq):
    """More queries than keys in every other sequence: blocks write zeros and draw again, in both orders of the items."""
    lk = [n if i % 2 == 0 else (50, 128, 1)[i // 2 % 3] for i, n in enumerate(lq)]
    _takes(cuda, lib, 320, 320, sum(lq), len(lq), hq, hkv, len(set(lq)) == 1, NONE)
    gen = torch.Generator().manual_seed(len(lq))
    rand = lambda *shape: torch.randn(*shape, generator=gen).bfloat16()
    q, k, v = rand(sum(lq), hq, 64), rand(sum(lk), hkv, 64), rand(sum(lk), hkv, 64)
    cu = lambda x: torch.tensor([0] + x).cumsum(0).int()
    args = [t.to(cuda) for t in (q, k, v, cu(lq), cu(lk))]
    ref = R.prefill_ref(q, k, v, cu(lq), cu(lk), 0.125)
    for _ in range(3):
        out = torch.full((sum(lq), hq, 64), float("nan"), dtype=torch.bfloat16, device=cuda)
        A.prefill_varlen(*args, 320, 320, 0.125, out=out)
        assert_close_to_oracle(out, ref, f"hq{hq}")
    assert _lib.read_status() == 0


@pytest.mark.parametrize("hq,hkv", FORM_64)
def test_three_blocks_to_an_sm_from_slices_in_graphs_and_on_two_streams(cuda, lib, hq, hkv):
    """q, k and v as slices of one activation, v of another width; layers captured with their stores and replayed at the same
    time on two streams, one of them beside launches of two blocks to an SM."""
    d, lens, short = 64, [384] * 36, [100] * 30
    _takes(cuda, lib, 384, 384, sum(lens), len(lens), hq, hkv, True, TILES, total_k=sum(lens))
    gen = torch.Generator(device=cuda).manual_seed(83)
    rand = lambda *shape: torch.randn(*shape, generator=gen, device=cuda).bfloat16()
    runs = []
    for seqs in ([lens], [lens, short]):
        parts = []
        for ls in seqs:
            n = sum(ls)
            qkv = rand(n, (hq + 2 * hkv) * d)
            q, k, _ = qkv.split([hq * d, hkv * d, hkv * d], dim=1)
            v = rand(n, 2 * hkv * d)[:, hkv * d:]
            blocks = n // 256 + 3
            layer = A.Attention(hq, d, d ** -0.5, hkv)
            layer.k_cache, layer.v_cache = rand(blocks, 256, hkv, d), rand(blocks, 256, hkv, d)
            slots = torch.randperm(blocks * 256, generator=gen, device=cuda)[:n].int()
            parts.append((layer, q, k, v, torch.tensor([0] + ls, device=cuda).cumsum(0).int(), max(ls), slots))
        runs.append(parts)

    def go(parts):
        outs = []
        for layer, q, k, v, cu, longest, slots in parts:
            C.set_context(True, cu, cu, longest, longest, slots, None, None)
            outs.append(layer(q, k, v))
        C.reset_context()
        return outs

    q, k, v, cu = (x.cpu() for x in runs[0][0][1:5])
    ref = R.prefill_ref(q.unflatten(1, (hq, d)), k.unflatten(1, (hkv, d)), v.unflatten(1, (hkv, d)), cu, cu, d ** -0.5)
    assert_close_to_oracle(go(runs[0])[0].view(-1, hq, d), ref, "slices")
    want = [go(parts) for parts in runs]
    planes = [[(p[0].k_cache.clone(), p[0].v_cache.clone()) for p in parts] for parts in runs]
    torch.cuda.synchronize()
    streams, graphs, outs = [torch.cuda.Stream() for _ in runs], [], []
    for parts in runs:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            outs.append(go(parts))
    for _ in range(5):
        for parts in runs:
            for p in parts:
                p[0].k_cache.zero_(), p[0].v_cache.zero_()
        for got in outs:
            for o in got:
                o.fill_(float("nan"))
        torch.cuda.synchronize()
        for stream, graph in zip(streams, graphs):
            with torch.cuda.stream(stream):
                graph.replay()
        torch.cuda.synchronize()
        for parts, got, exp, kept in zip(runs, outs, want, planes):
            for p, o, e, (kc, vc) in zip(parts, got, exp, kept):
                stored = p[6].long()
                assert torch.equal(o, e)
                assert torch.equal(p[0].k_cache.flatten(0, 1)[stored], kc.flatten(0, 1)[stored])
                assert torch.equal(p[0].v_cache.flatten(0, 1)[stored], vc.flatten(0, 1)[stored])
    assert _lib.read_status() == 0


@pytest.mark.parametrize("repeat", range(4))
def test_items_without_a_visible_key_where_blocks_start_late(cuda, repeat):
    """An item to a block, some of them tiles in front of all keys (more queries than keys), for which a block draws again:
    a launch on another stream keeps all SMs but one, so that its blocks draw twice before others have drawn at all."""
    hq, hkv, d = 16, 8, 128
    lq, lk = [300] * 5, [300, 50, 300, 50, 300][repeat % 2:] + [300] * (repeat % 2)
    gen = torch.Generator().manual_seed(48 + repeat)
    rand = lambda *shape: torch.randn(*shape, generator=gen).bfloat16()
    q, k, v = rand(sum(lq), hq, d), rand(sum(lk), hkv, d), rand(sum(lk), hkv, d)
    cu = lambda x: torch.tensor([0] + x).cumsum(0).int()
    other = torch.cuda.Stream()
    rows = (128 * (torch.cuda.get_device_properties(cuda).multi_processor_count - 1), 65536, 65536)  # all blocks but two
    longer = [torch.randn(n, 2, d, device=cuda).bfloat16() for n in rows]
    ends = [torch.tensor([0, n], dtype=torch.int32, device=cuda) for n in rows[:2]]
    args = [t.to(cuda) for t in (q, k, v, cu(lq), cu(lk))]
    out = torch.full((sum(lq), hq, d), float("nan"), dtype=torch.bfloat16, device=cuda)
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        A.prefill_varlen(*longer, *ends, *rows[:2], d ** -0.5)
    A.prefill_varlen(*args, max(lq), max(lk), d ** -0.5, out=out)
    torch.cuda.synchronize()
    assert_close_to_oracle(out, R.prefill_ref(q, k, v, cu(lq), cu(lk), d ** -0.5), f"{lk}")
    assert _lib.read_status() == 0


def test_many_sequences_through_the_persistent_kernel(cuda):
    """More work items than resident blocks, and more sequences than one warp scans at once."""
    case = W.make_prefill_case(28, 150, 1, 300, 4, 2, 128, share_every=0)
    _check(cuda, case, "150 sequences")


@pytest.mark.parametrize("cap", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("d", [64, 128])
def test_head_packing_of_the_persistent_kernel(cuda, monkeypatch, cap, d):
    """The persistent kernel packs up to 8 query heads of one KV head into the 128 rows of a tile
    (16 to 128 tokens per tile; the number of heads is the largest divisor of the group size
    within the cap, so 3, 5, 6 or 7 heads leave a few rows unused); NVLLM_PREFILL_PACK caps the
    number.  Every packing must agree with the oracle on ragged packed input and on
    prefix-cached input."""
    monkeypatch.setenv("NVLLM_PREFILL_IMPL", "tcp")
    monkeypatch.setenv("NVLLM_PREFILL_PACK", str(cap))
    case = W.make_prefill_case(28, 9, 1, 1, 16, 2, d, share_every=0,
                               lengths=[1, 15, 16, 17, 33, 130, 511, 1024, 700])
    _check(cuda, case, f"packed cap{cap} d{d}")
    case = W.make_prefill_case(29, 5, 1, 1, 16, 2, d, lengths=[1024, 1024, 300, 257, 600],
                               shared_blocks=[0, 3, 0, 1, 0])
    _check(cuda, case, f"paged cap{cap} d{d}")

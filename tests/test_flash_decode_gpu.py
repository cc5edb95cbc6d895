"""Flash decode on one GPU against a plain fp32 paged-attention statement; parameter grid follows
the reference's test_decode_attn.py:126-293 (kv_lens incl. 1, heads (16,16),(32,8),(64,8),(6,1),
D in {128,256}, atol 1e-2) and its sequence-parallel check (test_sp_decode_attn.py, atol 0.05)."""
import math

import pytest
import torch

from triton_distributed_b200.ops import flash_decode as FD
from triton_distributed_b200.runtime import LocalWorld, check_status

pytestmark = pytest.mark.gpu


def _make_cache(B, kv_lens, Hkv, D, page, dtype, dev, shuffle=True):
    max_blocks = max(1, (max(kv_lens) + page - 1) // page)
    nblocks = B * max_blocks + 3
    k = torch.randn(nblocks, page, Hkv, D, device=dev).to(dtype)
    v = torch.randn(nblocks, page, Hkv, D, device=dev).to(dtype)
    perm = torch.randperm(nblocks, device=dev) if shuffle else torch.arange(nblocks, device=dev)
    table = perm[: B * max_blocks].view(B, max_blocks).to(torch.int32)
    return k, v, table


@pytest.mark.parametrize("Hq,Hkv", [(16, 16), (32, 8), (64, 8), (6, 1), (96, 12)])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("kv_lens", [[1], [17, 300], [4096, 1, 1023, 2048]])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_decode_matches_reference(cuda_device, Hq, Hkv, D, kv_lens, dtype):
    torch.manual_seed(Hq * D + len(kv_lens))
    B, page = len(kv_lens), 16
    q = torch.randn(B, Hq, D, device=cuda_device).to(dtype)
    k, v, table = _make_cache(B, kv_lens, Hkv, D, page, dtype, cuda_device)
    lens = torch.tensor(kv_lens, dtype=torch.int32, device=cuda_device)
    scale = 1.0 / math.sqrt(D)
    out = FD.gqa_fwd_batch_decode(q, k, v, None, None, lens, table, scale)
    check_status()
    ref = FD.ref_paged_attn(q, k, v, lens, table, scale)
    torch.testing.assert_close(out.float(), ref, atol=1e-2, rtol=1e-2)


@pytest.mark.parametrize("G", [1, 7, 8, 9, 16])                       # columns of one MMA tile and of two
@pytest.mark.parametrize("D,page", [(64, 1), (64, 64), (128, 3), (128, 48), (256, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_decode_tiles_and_pages(cuda_device, G, D, page, dtype):
    """Lengths at the edges of a 16-token block, of a page and of the copies' ring; 40 sequences (some empty, some equal) are
    more than one wave of CTAs. The bound is the rounding of the probabilities and of the result, 2^-8 (bf16, half a unit
    of 8 significant bits) or 2^-11 (fp16, 11 bits) of sum p |v| and of the result; a soft cap's tanh is the hardware's approximation, 2^-11 of itself, so that a score is off by
    up to cap x 2^-11 and a probability by as much of itself, twice (its own score, the sum's)."""
    torch.manual_seed(G * D + page)
    Hkv, splits = 6, 3
    kv_lens = [0, 1, 15, 16, 17, 47, 48, 49, 63, 64, 65, 255, 256, 257, 1000] + [(37 * i) % 700 for i in range(23)] + [512, 512]
    B = len(kv_lens)
    q = torch.randn(B, G * Hkv, D, device=cuda_device).to(dtype)
    k, v, table = _make_cache(B, kv_lens, Hkv, D, page, dtype, cuda_device)
    lens = torch.tensor(kv_lens, dtype=torch.int32, device=cuda_device)
    scale = 1.5 / math.sqrt(D)
    for cap in (0.0, 20.0):
        out = FD.gqa_fwd_batch_decode(q, k, v, None, None, lens, table, scale, cap, kv_split=splits).float()
        check_status()
        ref = FD.ref_paged_attn(q, k, v, lens, table, scale, cap)
        spread = FD.ref_paged_attn(q, k, v.abs(), lens, table, scale, cap)
        u = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
        bound = u * (spread + ref.abs()) + (1e-3 + 2 * cap * 2.0 ** -11) * spread + 1e-6
        assert ((out - ref).abs() <= bound).all(), (cap, float(((out - ref).abs() - bound).max()))
        assert (out[0] == 0).all()


@pytest.mark.parametrize("splits", [1, 3, 8, 16, 32])   # up to 8: one cluster per (batch, kv head), merged through shared memory
@pytest.mark.parametrize("soft_cap", [0.0, 30.0])
def test_intra_rank_partials_and_merge(cuda_device, splits, soft_cap):
    torch.manual_seed(splits)
    B, Hq, Hkv, D, page = 3, 32, 8, 128, 64
    kv_lens = [777, 0, 5000]
    q = torch.randn(B, Hq, D, device=cuda_device).to(torch.bfloat16)
    k, v, table = _make_cache(B, kv_lens, Hkv, D, page, torch.bfloat16, cuda_device)
    lens = torch.tensor(kv_lens, dtype=torch.int32, device=cuda_device)
    scale = 0.09
    part = FD.gqa_fwd_batch_decode_intra_rank(q, k, v, None, None, lens, table, scale, soft_cap, kv_split=splits)
    check_status()
    ro, rl = FD.ref_paged_attn(q, k, v, lens, table, scale, soft_cap, return_lse=True)
    torch.testing.assert_close(part[..., :D], ro, atol=1e-2, rtol=1e-2)
    torch.testing.assert_close(part[[0, 2], :, D], rl[[0, 2]], atol=2e-3, rtol=2e-3)
    assert torch.isinf(part[1, :, D]).all()
    # two "ranks" merged by the standalone combine kernel
    parts = torch.stack([part, part])
    merged = FD.inter_rank_combine(parts, torch.bfloat16)
    torch.testing.assert_close(merged.float(), ro, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("world,B", [(2, 1), (4, 3), (8, 8)])
def test_sequence_parallel_decode_emulated(cuda_device, world, B):
    """Every emulated rank computes and sends first; then every rank redoes its step and gathers."""
    torch.manual_seed(world * 10 + B)
    Hq, Hkv, D, page = 32, 8, 128, 16
    lw = LocalWorld(world, cuda_device)
    ctxs = [FD.create_sp_decode_context(r, world, B, Hq, D, heap=lw.heap(r), device=cuda_device) for r in range(world)]
    q = torch.randn(B, Hq, D, device=cuda_device).to(torch.bfloat16)
    for it in range(3):
        glens = torch.randint(0, 600, (world, B), dtype=torch.int32, device=cuda_device)
        glens[0, 0] = 5  # at least one key somewhere
        if it == 1:
            glens[1 % world] = 0  # a rank with no keys at all
        shards = [_make_cache(B, [max(1, int(x)) for x in glens[r]], Hkv, D, page, torch.bfloat16, cuda_device) for r in range(world)]
        for r in range(world):
            FD.sp_gqa_fwd_batch_decode(ctxs[r], q, shards[r][0], shards[r][1], glens, shards[r][2], phase=1)
        outs = [FD.sp_gqa_fwd_batch_decode(ctxs[r], q, shards[r][0], shards[r][1], glens, shards[r][2], phase=2) for r in range(world)]
        check_status()
        parts = []
        for r in range(world):
            o, l = FD.ref_paged_attn(q, shards[r][0], shards[r][1], glens[r], shards[r][2], 1.0 / math.sqrt(D), return_lse=True)
            parts.append(torch.cat([o, l.unsqueeze(-1)], -1))
        ref = FD.ref_lse_merge(torch.stack(parts))
        for r in range(world):
            torch.testing.assert_close(outs[r].float(), ref, atol=5e-2, rtol=5e-2)


@pytest.mark.parametrize("world,B", [(2, 2), (4, 3)])
@pytest.mark.parametrize("graph", [False, True], ids=["eager", "cuda_graph"])
def test_sequence_parallel_decode_with_device_call_number(cuda_device, world, B, graph):
    """The call number lives in device memory and the kernel advances it, so the launches of a step (all
    emulated ranks send, then all redo and gather) can be captured once and replayed: every replay uses the
    next number and the other buffer parity."""
    torch.manual_seed(world * 7 + B)
    Hq, Hkv, D, page = 32, 8, 128, 16
    lw = LocalWorld(world, cuda_device)
    ctxs = [FD.create_sp_decode_context(r, world, B, Hq, D, heap=lw.heap(r), device=cuda_device, device_epoch=True)
            for r in range(world)]
    q = torch.randn(B, Hq, D, device=cuda_device).to(torch.bfloat16)
    glens = torch.randint(1, 600, (world, B), dtype=torch.int32, device=cuda_device)
    shards = [_make_cache(B, [600] * B, Hkv, D, page, torch.bfloat16, cuda_device) for r in range(world)]
    outs = [torch.empty_like(q) for _ in range(world)]

    def step():
        for r in range(world):
            FD.sp_gqa_fwd_batch_decode(ctxs[r], q, shards[r][0], shards[r][1], glens, shards[r][2], phase=1)
        for r in range(world):
            FD.sp_gqa_fwd_batch_decode(ctxs[r], q, shards[r][0], shards[r][1], glens, shards[r][2], phase=2, out=outs[r])

    g = None
    if graph:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()                       # warm-up (advances every rank's call number by one)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            step()
    for it in range(4):
        q.copy_(torch.randn(B, Hq, D, device=cuda_device).to(torch.bfloat16))
        glens.copy_(torch.randint(1, 600, (world, B), dtype=torch.int32, device=cuda_device))
        if it == 2:
            glens[1 % world] = 0         # a rank without keys
            glens[0, :] = 9
        if g is not None:
            g.replay()
        else:
            step()
        torch.cuda.synchronize()
        check_status()
        parts = []
        for r in range(world):
            o, l = FD.ref_paged_attn(q, shards[r][0], shards[r][1], glens[r], shards[r][2], 1.0 / math.sqrt(D), return_lse=True)
            parts.append(torch.cat([o, l.unsqueeze(-1)], -1))
        ref = FD.ref_lse_merge(torch.stack(parts))
        for r in range(world):
            torch.testing.assert_close(outs[r].float(), ref, atol=5e-2, rtol=5e-2)
    done = 4 + (1 if graph else 0)
    for r in range(world):
        assert int(ctxs[r].epoch_dev[0]) == done and int(ctxs[r].epoch_dev[1]) == 0


@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 7, 8, 9, 12])
@pytest.mark.parametrize("Hq,Hkv,D", [(32, 8, 128), (16, 16, 64), (16, 1, 256), (64, 4, 128)])
def test_splits_meet_in_the_ring_or_in_global_memory(cuda_device, splits, Hq, Hkv, D):
    """Partials of up to eight splits land in the ring of the cluster's first CTA while that is still merging its warps;
    with 16 heads per kv head and eight splits they no longer fit and go through global memory. Ragged, empty and
    one-key sequences."""
    torch.manual_seed(splits + D)
    lens = [3000, 0, 1, 17, 1024]
    B, page, per = len(lens), 16, -(-3000 // 16)
    k = torch.randn(B * per, page, Hkv, D, device=cuda_device).to(torch.bfloat16)
    v = torch.randn(B * per, page, Hkv, D, device=cuda_device).to(torch.bfloat16)
    q = torch.randn(B, Hq, D, device=cuda_device).to(torch.bfloat16)
    table = torch.randperm(B * per, device=cuda_device).to(torch.int32).view(B, per)
    kv = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    ref = FD.ref_paged_attn(q, k, v, kv, table, D ** -0.5)
    for _ in range(3):
        out = FD.gqa_fwd_batch_decode(q, k, v, None, None, kv, table, D ** -0.5, kv_split=splits)
        check_status()
        torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("splits", [2, 10])          # one cluster per (batch, kv head); through global memory
@pytest.mark.parametrize("blocks_over", [0, 1])      # 2560 keys per CTA and just above: with and without the early launch
def test_a_decode_reads_the_result_of_the_one_before(cuda_device, B, splits, blocks_over):
    """Calls in a row whose queries are the outputs of the call before, not synchronised in between."""
    torch.manual_seed(B + splits)
    Hq, Hkv, D, page = 32, 8, 128, 16
    per = splits * (2560 // page + blocks_over)
    lens = [per * page, 37][:B]
    k = torch.randn(B * per, page, Hkv, D, device=cuda_device).to(torch.bfloat16)
    v = torch.randn(B * per, page, Hkv, D, device=cuda_device).to(torch.bfloat16)
    table = torch.randperm(B * per, device=cuda_device).to(torch.int32).view(B, per)
    kv = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    qs = [4 * torch.randn(B, Hq, D, device=cuda_device).to(torch.bfloat16)]
    for _ in range(5):
        qs.append(FD.gqa_fwd_batch_decode(qs[-1], k, v, None, None, kv, table, D ** -0.5, kv_split=splits))
    check_status()
    for q, out in zip(qs, qs[1:]):
        torch.testing.assert_close(out.float(), FD.ref_paged_attn(q, k, v, kv, table, D ** -0.5), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("explicit", [False, True])   # torch's current stream; a stream handed over
def test_two_streams_do_not_share_their_scratch(cuda_device, explicit):
    """16 splits meet in global memory: launches of the same shape on two streams at once, with different queries and caches,
    each give what they give alone."""
    torch.manual_seed(9)
    Hq, Hkv, D, page, per = 32, 8, 128, 16, 256
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    jobs = []
    for _ in streams:
        q = torch.randn(1, Hq, D, device=cuda_device).to(torch.bfloat16)
        k, v, table = _make_cache(1, [per * page], Hkv, D, page, torch.bfloat16, cuda_device)
        kv = torch.tensor([per * page - 5], dtype=torch.int32, device=cuda_device)
        ref = FD.gqa_fwd_batch_decode(q, k, v, None, None, kv, table, D ** -0.5, kv_split=16)
        torch.testing.assert_close(ref.float(), FD.ref_paged_attn(q, k, v, kv, table, D ** -0.5), atol=1e-2, rtol=1e-2)
        jobs.append((q, k, v, kv, table, ref))
    torch.cuda.synchronize()
    outs = [[torch.empty_like(jobs[0][0]) for _ in range(100)] for _ in streams]
    torch.cuda.synchronize()
    for n in range(100):
        for i, s in enumerate(streams):
            q, k, v, kv, table, _ = jobs[i]
            if explicit:
                FD._launch(q, k, v, kv, table, D ** -0.5, 0.0, outs[i][n], 0, 16, stream=s)
            else:
                with torch.cuda.stream(s):
                    FD.gqa_fwd_batch_decode(q, k, v, None, None, kv, table, D ** -0.5, kv_split=16, output_combine=outs[i][n])
    torch.cuda.synchronize()
    check_status()
    for i in range(2):
        assert all(torch.equal(o, jobs[i][5]) for o in outs[i])
    assert len({k[1] for k in FD._Workspace.cache if k[1] in (streams[0].cuda_stream, streams[1].cuda_stream)}) == 2


def test_batch_splits_fill_the_last_wave_and_even_out_lengths():
    assert FD._batch_splits(32 * 8, 8192, 128, 148, 1) == 2        # ragged batches gain, full ones lose next to nothing
    assert FD._batch_splits(8 * 8, 32768, 128, 148, 4) == 4        # one wave of 256 CTAs is hard to beat
    assert FD._batch_splits(48 * 8, 4096, 128, 148, 1) == 2        # 384 CTAs are 1.3 waves, 768 are 2.6
    assert FD._batch_splits(64 * 8, 512, 128, 148, 1) == 1         # short sequences: the fixed cost decides
    assert FD._batch_splits(16 * 8, 1024, 128, 148, 2) == 2
    assert FD._batch_splits(32 * 8, 131072, 128, 148, 1) == 6
    assert FD._batch_splits(32 * 8, 131072, 128, 148, 1, True) == 2   # more table than cache: one round of CTAs more at most
    assert FD._batch_splits(64 * 16, 131072, 128, 148, 1, True) == 1


def test_a_table_wider_than_the_cache_does_not_ask_for_more_splits(cuda_device, monkeypatch):
    """The same sequences and cache behind tables of any width: never more splits than the cache could fill."""
    asked = []
    rule = FD._batch_splits
    monkeypatch.setattr(FD, "_batch_splits", lambda *a: asked.append(a) or rule(*a))
    torch.manual_seed(0)
    B, Hq, Hkv, D, page = 32, 32, 8, 128, 16
    lens = torch.randint(1, 200, (B,), dtype=torch.int32, device=cuda_device)
    q = torch.randn(B, Hq, D, device=cuda_device).to(torch.bfloat16)
    k, v, table = _make_cache(B, [256] * B, Hkv, D, page, torch.bfloat16, cuda_device)
    ref = FD.ref_paged_attn(q, k, v, lens, table, D ** -0.5)
    for width in (16, 512, 8192):
        padded = torch.zeros(B, width, dtype=torch.int32, device=cuda_device)
        padded[:, :16] = table
        out = FD.gqa_fwd_batch_decode(q, k, v, None, None, lens, padded, D ** -0.5)
        check_status()
        torch.testing.assert_close(out.float(), ref, atol=1e-2, rtol=1e-2)
    held = k.shape[0] * page
    assert [a[1] for a in asked] == [256, 2 * held // B, 2 * held // B] and [a[5] for a in asked] == [False, True, True]


@pytest.mark.parametrize("kind", ["dispatch", "own rows", "combine", "ag_gemm", "gemm_rs", "decode"])
def test_a_launch_behind_a_waiting_one_leaves_the_machine_free(cuda_device, monkeypatch, kind):
    """A kernel that waits for a flag of another launch (here one that nothing sets, until its limit) does not let the next
    launch of its stream in early: that one, here a decode that takes every SM's shared memory, would keep out the work of
    other streams that the flag may depend on. The product on the other stream waits for nothing and must finish meanwhile."""
    import time
    from triton_distributed_b200.ops import gemm as G, moe_ep as EP
    from triton_distributed_b200.runtime import global_status
    monkeypatch.setenv("TDIST_WAIT_TIMEOUT_MS", "600")
    torch.manual_seed(1)
    lw, keep = LocalWorld(2, cuda_device), []
    bf = lambda *shape: torch.randn(*shape, device=cuda_device).to(torch.bfloat16)  # noqa: E731
    x, w = bf(256, 256), bf(512, 256)
    if kind in ("dispatch", "combine", "own rows"):
        ids = torch.zeros(4, 1, dtype=torch.int32, device=cuda_device)
        ranks = 1 if kind == "own rows" else 2
        heap = LocalWorld(1, cuda_device).heap(0) if ranks == 1 else lw.heap(0)
        ctx = EP.create_ep_context(4, 256, 1, 2, 0, ranks, compact=False, heap=heap)
        if ranks == 2:
            keep.append(EP.create_ep_context(4, 256, 1, 2, 1, 2, compact=False, heap=lw.heap(1)))
        ctx.topk_ids, ctx.ntok = ids, 4
        if kind == "combine":
            EP.ep_dispatch(ctx, x[:4], ids, None, phase=3)
            wait = lambda: EP.ep_combine(ctx, weighted=False)  # noqa: E731
        elif kind == "dispatch":
            wait = lambda: EP.ep_dispatch(ctx, x[:4], ids, None)  # noqa: E731
        else:
            ctx.call_count += 1
            wait = lambda: EP.ep_dispatch(ctx, x[:4], ids, None, phase=4)  # noqa: E731
    elif kind == "decode":
        ctxs = [FD.create_sp_decode_context(r, 2, 1, 32, 128, heap=lw.heap(r), device=cuda_device) for r in range(2)]
        shard = _make_cache(1, [64], 8, 128, 16, torch.bfloat16, cuda_device)
        q1, glens = bf(1, 32, 128), torch.full((2, 1), 64, dtype=torch.int32, device=cuda_device)
        wait = lambda: FD.sp_gqa_fwd_batch_decode(ctxs[0], q1, shard[0], shard[1], glens, shard[2])  # noqa: E731
    else:
        if kind == "ag_gemm":
            ctxs = [G.create_ag_gemm_intra_node_context(x, w, r, 2, max_M=512, heap=lw.heap(r)) for r in range(2)]
            wait = lambda: G.ag_gemm_intra_node(x, w, ctxs[0])  # noqa: E731
        else:
            ctxs = [G.create_gemm_rs_context(256, 512, r, 2, heap=lw.heap(r)) for r in range(2)]
            wait = lambda: G.gemm_rs(x, w, ctxs[0])  # noqa: E731
        ctxs[0].num_sms = 16
    # a decode whose 37 x 8 CTAs take two places on each of 148 SMs
    kv = torch.full((37,), 32, dtype=torch.int32, device=cuda_device)
    cache = _make_cache(37, [32] * 37, 8, 128, 16, torch.bfloat16, cuda_device)
    q = bf(37, 32, 128)
    fill = lambda: FD.gqa_fwd_batch_decode(q, cache[0], cache[1], None, None, kv, cache[2], 128 ** -0.5, kv_split=1)  # noqa: E731
    other, done, waited = torch.cuda.Stream(), torch.cuda.Event(), torch.cuda.Event()
    want = fill()
    G.gemm_persistent(x, w, num_sms=148)
    torch.cuda.synchronize()
    wait()
    got = fill()
    waited.record()
    time.sleep(0.05)
    with torch.cuda.stream(other):
        c = G.gemm_persistent(x, w, num_sms=148)
        done.record()
    until = time.monotonic() + 0.25
    while not done.query() and time.monotonic() < until:
        time.sleep(0.005)
    free, waiting = done.query(), not waited.query()
    torch.cuda.synchronize()
    rec = global_status().record
    assert (rec.abort_flag, rec.code) == (1, 1) and waiting
    with pytest.raises(Exception, match="timed out"):
        check_status()
    assert free
    torch.testing.assert_close(c.float(), x.float() @ w.float().t(), atol=1e-1, rtol=2e-2)
    assert torch.equal(got, want)


def _exact_attn(q, k, v, lens, table, scale):
    """Output, sum of p |v|, log-sum-exp, in float64."""
    B, Hq, D = q.shape
    Hkv, page = k.shape[2], k.shape[1]
    o, spread = (torch.zeros(B, Hq, D, dtype=torch.float64, device=q.device) for _ in range(2))
    lse = torch.full((B, Hq), float("-inf"), dtype=torch.float64, device=q.device)
    for b, n in enumerate(lens.tolist()):
        if n:
            pages = table[b, : -(-n // page)].long()
            kk, vv = (c[pages].reshape(-1, Hkv, D)[:n].double() for c in (k, v))
            s = torch.einsum("hgd,nhd->hgn", q[b].double().view(Hkv, -1, D), kk) * scale
            p = torch.softmax(s, -1)
            o[b], spread[b] = (torch.einsum("hgn,nhd->hgd", p, x).reshape(Hq, D) for x in (vv, vv.abs()))
            lse[b] = torch.logsumexp(s, -1).reshape(Hq)
    return o, spread, lse


@pytest.mark.parametrize("B,splits,Hq,Hkv,D,most", [
    (127, 2, 24, 2, 128, 700), (128, 2, 24, 2, 128, 700), (129, 2, 24, 2, 128, 700),   # the largest batch ordered by length, and beyond
    (128, 1, 8, 4, 64, 600), (50, 2, 8, 2, 256, 300),
    (24, 10, 8, 2, 128, 2700),                                                         # merged through global memory
    (128, 12, 8, 2, 64, 700)])                                                         # not ordered: too short for so many rounds
def test_ragged_batches_of_more_than_one_round(cuda_device, B, splits, Hq, Hkv, D, most):
    """Sequences of any length, equal and empty ones among them, in a grid of more CTAs than run at once: results, partials with
    their log-sum-exp, and a captured launch that is replayed with other lengths, with short ones only, and with equal ones. fp16
    rounds a probability and the result to 2^-11
    of themselves (small probabilities to 2^-25); scores, exponentials and sums in fp32 add less than 2^-14."""
    torch.manual_seed(B + splits + D)
    page = 16
    k, v, table = _make_cache(B, [most] * B, Hkv, D, page, torch.float16, cuda_device)
    q = torch.randn(B, Hq, D, device=cuda_device).half()
    scale = D ** -0.5
    lens = torch.randint(0, most + 1, (B,), device=cuda_device).to(torch.int32)
    lens[3], lens[5], lens[6:9], lens[B - 1] = 0, most, most // 2, 1

    def check():
        o, spread, lse = _exact_attn(q, k, v, lens, table, scale)
        small = most * 2.0 ** -25 * v.float().abs().max().double()
        out = FD.gqa_fwd_batch_decode(q, k, v, None, None, lens, table, scale, kv_split=splits)
        part = FD.gqa_fwd_batch_decode_intra_rank(q, k, v, None, None, lens, table, scale, 0.0, kv_split=splits).double()
        check_status()
        assert ((out.double() - o).abs() <= (2.0 ** -11 + 2.0 ** -14) * spread + 2.0 ** -11 * o.abs() + small).all()
        assert ((part[..., :D] - o).abs() <= (2.0 ** -11 + 2.0 ** -14) * spread + small).all()
        live = lens > 0
        assert ((part[live][..., D] - lse[live]).abs() <= 2.0 ** -14).all() and (part[~live][..., D] == float("-inf")).all()
        return out

    check()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        FD.gqa_fwd_batch_decode(q, k, v, None, None, lens, table, scale, kv_split=splits)
    torch.cuda.current_stream().wait_stream(side)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        replayed = FD.gqa_fwd_batch_decode(q, k, v, None, None, lens, table, scale, kv_split=splits)
    for other in (lens[torch.randperm(B, device=cuda_device)], lens[torch.randperm(B, device=cuda_device)], lens // 4, torch.full_like(lens, most)):
        lens.copy_(other)
        g.replay()
        assert torch.equal(replayed, check())

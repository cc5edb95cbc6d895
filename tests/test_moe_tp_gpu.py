"""Tensor-parallel MoE ops on one GPU (ranks emulated send-half / receive-half). Oracle: masked
per-expert fp32 matmuls, as in the reference's test_ag_moe.py:24-39 and test_moe_reduce_rs.py."""
import pytest
import torch

from triton_distributed_b200.ops import moe_tp as MT
from triton_distributed_b200.ops import moe_utils as MU
from triton_distributed_b200.runtime import LocalWorld, check_status

pytestmark = pytest.mark.gpu


def _expert_matmul(rows, ids, b_ekn):
    out = torch.zeros(rows.shape[0], b_ekn.shape[2], device=rows.device)
    for e in range(b_ekn.shape[0]):
        m = ids == e
        if m.any():
            out[m] = rows[m].float() @ b_ekn[e].float()
    return out


@pytest.mark.parametrize("T,E,K,N,topk", [(256, 8, 256, 512, 2), (1000, 32, 520, 264, 4), (64, 60, 128, 1024, 6)])
def test_group_gemm_blocks_pick_their_expert(cuda_device, T, E, K, N, topk):
    torch.manual_seed(T + E)
    x = torch.randn(T, K, device=cuda_device).to(torch.bfloat16)
    b = (torch.randn(E, K, N, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    ids = torch.randint(0, E, (T, topk), dtype=torch.int32, device=cuda_device)
    sorted_ids, expert_ids, _, _, post_pad = MU.sort_topk_ids_align_block_size(ids, E, 1, T, 128)
    n = int(post_pad)
    a_sorted, pos_of = MT.gather_rows(x, sorted_ids[:n].contiguous(), topk, T * topk, want_inverse=True)
    c = MT.group_gemm(a_sorted, b.transpose(1, 2).contiguous(), expert_ids, (post_pad // 128).to(torch.int32))
    check_status()
    got = c[pos_of.long()].float()
    ref = _expert_matmul(x[torch.arange(T * topk, device=cuda_device) // topk], ids.reshape(-1), b)
    torch.testing.assert_close(got, ref, atol=3e-2, rtol=3e-2)
    red = MT.topk_reduce(c, pos_of, torch.ones(T, topk, device=cuda_device), T, topk)
    torch.testing.assert_close(red.float(), ref.view(T, topk, N).sum(1), atol=6e-2, rtol=3e-2)


@pytest.mark.parametrize("world,tpr,E,K,N,topk", [(1, 256, 8, 256, 256, 2), (4, 128, 16, 512, 264, 2), (8, 64, 32, 256, 512, 4)])
@pytest.mark.parametrize("mode", ["fused", "cp_async", "staged"])
def test_ag_group_gemm(cuda_device, monkeypatch, world, tpr, E, K, N, topk, mode):
    """`fused`: the all-gather only sends; one grouped-GEMM launch stages the rows block by block as the source
    rank's segment arrives, feeds the MMAs by TMA from this rank's own blocks on, and stores every row at its
    (token, k) position. `cp_async`: the producer warps gather by index. `staged`: four separate launches."""
    monkeypatch.setattr(MT, "AG_GROUP_GEMM_MODE", mode)
    torch.manual_seed(world * 7 + tpr)
    lw = LocalWorld(world, cuda_device)
    M = world * tpr
    shards = [torch.randn(tpr, K, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
    bs = [(torch.randn(E, K, N, device=cuda_device) * K ** -0.5).to(torch.bfloat16) for _ in range(world)]
    ids = torch.randint(0, E, (M, topk), dtype=torch.int32, device=cuda_device)
    ctxs = [MT.create_ag_group_gemm_intra_node_context(None, shards[r], bs[r], ids, E, max_M=M, rank=r, num_ranks=world,
                                                       heap=lw.heap(r)) for r in range(world)]
    for it in range(2):   # two calls: both gather buffers
        if it == 1:
            shards = [torch.randn(tpr, K, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
        if world > 1:
            for r in range(world):
                MT.ag_group_gemm_intra_node(shards[r], bs[r], ctxs[r], phase=1)
        outs = [MT.ag_group_gemm_intra_node(shards[r], bs[r], ctxs[r], phase=2 if world > 1 else 3) for r in range(world)]
        check_status()
        full = torch.cat(shards)
        rows = full[torch.arange(M * topk, device=cuda_device) // topk]
        for r in range(world):
            ref = _expert_matmul(rows, ids.reshape(-1), bs[r])
            torch.testing.assert_close(outs[r].float(), ref, atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("world,M,E,Kl,N,topk", [(1, 256, 8, 256, 256, 2), (2, 512, 16, 128, 512, 2), (4, 256, 32, 256, 1024, 4)])
@pytest.mark.parametrize("fused", [True, False], ids=["fused_topk_rs", "staged"])
def test_moe_reduce_rs(cuda_device, monkeypatch, world, M, E, Kl, N, topk, fused):
    """`fused`: the rows are sorted by expert inside the grouped-GEMM launch and the top-k weighted reduce happens
    inside the reduce-scatter kernel (the [M, N] partial is never written); staged: row-gather kernel, grouped GEMM,
    top-k reduce kernel, plain reduce-scatter."""
    monkeypatch.setattr(MT, "FUSED_TOPK_RS", fused)
    monkeypatch.setattr(MT, "AG_GROUP_GEMM_MODE", "fused" if fused else "staged")
    torch.manual_seed(world * 11 + M)
    lw = LocalWorld(world, cuda_device)
    ids = torch.randint(0, E, (M, topk), dtype=torch.int32, device=cuda_device)
    w = torch.rand(M, topk, device=cuda_device)
    a = [torch.randn(M * topk, Kl, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
    b = [(torch.randn(E, Kl, N, device=cuda_device) * (Kl * world) ** -0.5).to(torch.bfloat16) for _ in range(world)]
    ctxs = [MT.create_moe_rs_context(None, r, world, world, M, N, E, topk, torch.bfloat16, torch.bfloat16, cuda_device,
                                     full_topk_ids=ids, full_topk_weight=w, heap=lw.heap(r)) for r in range(world)]
    for it in range(2):   # two calls: both staging parities
        if it == 1:
            a = [torch.randn(M * topk, Kl, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
        for r in range(world):
            MT.moe_reduce_rs(r, world, world, a[r], b[r], ctxs[r], phase=1)
        outs = [MT.moe_reduce_rs(r, world, world, a[r], b[r], ctxs[r], phase=2) for r in range(world)]
        check_status()
        total = sum((_expert_matmul(a[r], ids.reshape(-1), b[r]).view(M, topk, N) * w.view(M, topk, 1)).sum(1) for r in range(world))
        mpr = M // world
        for r in range(world):
            torch.testing.assert_close(outs[r].float(), total[r * mpr:(r + 1) * mpr], atol=6e-2, rtol=3e-2)


@pytest.mark.parametrize("T,E,K,N,topk", [(300, 8, 264, 520, 2), (128, 4, 64, 256, 1), (777, 16, 1024, 384, 3)])
def test_group_gemm_gathers_rows_in_kernel(cuda_device, T, E, K, N, topk):
    """The cp.async row-gathering producer against the staged path (row gather kernel + TMA-fed grouped GEMM):
    same sorted layout, ragged K (not a multiple of the 64-wide K block), padding rows."""
    torch.manual_seed(T + K)
    x = torch.randn(T, K, device=cuda_device).to(torch.bfloat16)
    b = (torch.randn(E, N, K, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    ids = torch.randint(0, E, (T, topk), dtype=torch.int32, device=cuda_device)
    sorted_ids, expert_ids, _, _, post_pad = MU.sort_topk_ids_align_block_size(ids, E, 1, T, 128)
    n = int(post_pad)
    sid = sorted_ids[:n].contiguous()
    nb = (post_pad // 128).to(torch.int32)
    a_sorted, _ = MT.gather_rows(x, sid, topk, T * topk)
    want = MT.group_gemm(a_sorted, b, expert_ids, nb)
    row_index = torch.div(sid, topk, rounding_mode="floor").to(torch.int32)
    got = MT.group_gemm_gather(x, row_index, b, expert_ids, nb)
    check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("K", [8, 40, 256, 264, 504, 1024, 1032, 2048, 2056])
def test_staged_gather_copies_rows_of_every_length(cuda_device, K):
    """Rows of one 16-byte vector up to several steps of the copy; T and E leave blocks to the prologue and to the epilogue
    warps (more blocks than the first wave has), with padding rows in every expert's last block."""
    torch.manual_seed(K)
    T, E, N, topk = 2900, 7, 2048, 2
    x = torch.randn(T, K, device=cuda_device).to(torch.bfloat16)
    b = (torch.randn(E, N, K, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    ids = torch.randint(0, E, (T, topk), dtype=torch.int32, device=cuda_device)
    sorted_ids, expert_ids, _, _, post_pad = MU.sort_topk_ids_align_block_size(ids, E, 1, T, 128)
    sid = sorted_ids[:int(post_pad)].contiguous()
    nb = (post_pad // 128).to(torch.int32)
    a_sorted, _ = MT.gather_rows(x, sid, topk, T * topk)
    want = MT.group_gemm(a_sorted, b, expert_ids, nb)
    row_index = torch.div(sid, topk, rounding_mode="floor").to(torch.int32)
    staging = torch.full((sid.numel(), K), float("nan"), dtype=x.dtype, device=cuda_device)
    flags = MT.staging_flags(sid.numel(), cuda_device)
    live = sid < T * topk
    for epoch in (1, 2):
        got = MT.group_gemm_gather(x, row_index, b, expert_ids, nb, staging=staging, block_ready=flags, epoch=epoch)
        check_status()
        assert torch.equal(got[live], want[live])


@pytest.mark.parametrize("T,E,K,N,topk,rot", [(300, 8, 264, 520, 2, 0), (1500, 16, 512, 776, 3, 7), (128, 4, 64, 256, 1, 1)])
def test_group_gemm_staged_gather_rotation_and_scatter(cuda_device, T, E, K, N, topk, rot):
    """In-launch row staging (all-thread prologue + epilogue warps) + TMA-fed MMAs + scattering epilogue in one launch against the four-launch path, over several
    calls with fresh data (the per-block flags carry the call number), starting the schedule at block `rot`."""
    torch.manual_seed(T + K)
    b = (torch.randn(E, N, K, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    ids = torch.randint(0, E, (T, topk), dtype=torch.int32, device=cuda_device)
    sorted_ids, expert_ids, _, _, post_pad = MU.sort_topk_ids_align_block_size(ids, E, 1, T, 128)
    n = int(post_pad)
    sid = sorted_ids[:n].contiguous()
    nb = (post_pad // 128).to(torch.int32)
    row_index = torch.div(sid, topk, rounding_mode="floor").to(torch.int32)
    staging = torch.full((n, K), float("nan"), device=cuda_device, dtype=torch.bfloat16)
    ready = MT.staging_flags(n, cuda_device)
    rot_t = torch.tensor([min(rot, n // 128 - 1)], dtype=torch.int32, device=cuda_device)
    for call in range(1, 4):
        x = torch.randn(T, K, device=cuda_device).to(torch.bfloat16)
        a_sorted, pos_of = MT.gather_rows(x, sid, topk, T * topk, want_inverse=True)
        want_sorted = MT.group_gemm(a_sorted, b, expert_ids, nb)
        want, _ = MT.gather_rows(want_sorted, pos_of, 1, n)
        got_sorted = MT.group_gemm_gather(x, row_index, b, expert_ids, nb, staging=staging, block_ready=ready, epoch=2 * call - 1,
                                          block_rot=rot_t)
        staging.fill_(float("nan"))    # the second launch must stage the rows again, not reuse what is there
        got = MT.group_gemm_gather(x, row_index, b, expert_ids, nb, staging=staging, block_ready=ready, epoch=2 * call,
                                   block_rot=rot_t, c_scatter=sid, c_rows=T * topk)
        check_status()
        live = sid < T * topk
        assert torch.equal(got_sorted[live], want_sorted[live])
        assert torch.equal(got, want)
        assert int(ready[n // 128:].abs().sum()) == 0      # the kernel leaves its counters at zero for the next launch


@pytest.mark.parametrize("world,tpr,E,K,N,topk", [(1, 2000, 4, 264, 520, 2), (1, 3000, 3, 4104, 776, 2), (1, 300, 8, 256, 512, 2),
                                                  (4, 700, 2, 512, 264, 2), (1, 90, 2, 64, 8, 1)])
def test_grouped_gemm_on_block_pairs(cuda_device, monkeypatch, world, tpr, E, K, N, topk):
    """Two blocks of an expert per CTA pair, odd blocks alone (forced where they are many), ragged last blocks, K and N
    off the tile edges; up-projection with staged rows, rotation and scatter, then down-projection with staged rows and top-k reduce.
    Tolerance as above: 16-bit results and the 16-bit intermediate of the reduce."""
    monkeypatch.setattr(MT, "PAIR_MAX_OVERHEAD", 2.0)
    torch.manual_seed(tpr + E)
    lw = LocalWorld(world, cuda_device)
    M = world * tpr
    shards = [torch.randn(tpr, K, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
    bs = [(torch.randn(E, K, N, device=cuda_device) * K ** -0.5).to(torch.bfloat16) for _ in range(world)]
    ids = torch.stack([torch.randperm(E, device=cuda_device)[:topk] for _ in range(M)]).to(torch.int32)
    ctxs = [MT.create_ag_group_gemm_intra_node_context(None, shards[r], bs[r], ids, E, max_M=M, rank=r, num_ranks=world,
                                                       heap=lw.heap(r)) for r in range(world)]
    assert all(c.pairs is not None for c in ctxs)
    for r in range(world if world > 1 else 0):
        MT.ag_group_gemm_intra_node(shards[r], bs[r], ctxs[r], phase=1)
    rows = torch.cat(shards)[torch.arange(M * topk, device=cuda_device) // topk]
    for r in range(world):
        for _ in range(2 if world == 1 else 1):
            out = MT.ag_group_gemm_intra_node(shards[r], bs[r], ctxs[r], phase=2 if world > 1 else 3)
            check_status()
            torch.testing.assert_close(out.float(), _expert_matmul(rows, ids.reshape(-1), bs[r]), atol=3e-2, rtol=3e-2)
    if world == 1:
        w = torch.rand(M, topk, device=cuda_device)
        down = MT.create_moe_rs_context(None, 0, 1, 1, M, N, E, topk, torch.bfloat16, torch.bfloat16, cuda_device, full_topk_ids=ids,
                                        full_topk_weight=w, heap=lw.heap(0))
        assert down.pairs is not None
        y = MT.moe_reduce_rs(0, 1, 1, rows, bs[0], down)
        check_status()
        ref = (_expert_matmul(rows, ids.reshape(-1), bs[0]).view(M, topk, N) * w.unsqueeze(-1)).sum(1)
        torch.testing.assert_close(y.float(), ref, atol=6e-2, rtol=3e-2)


def test_pair_blocks_keeps_experts_and_ranks_apart():
    experts = torch.tensor([0, 0, 0, 1, 1, 1, 1, 2, 2, 0, 0, 3, 3], dtype=torch.int32)
    ranks = torch.tensor([0] * 9 + [1] * 4, dtype=torch.int32)
    pairs = MT.pair_blocks(experts, ranks, 13, 9)
    assert pairs.block.tolist() == [0, 5, 6, 10, 14, 18, 22] and pairs.rot.tolist() == [5]
    assert MT.pair_blocks(torch.arange(6, dtype=torch.int32), torch.zeros(6, dtype=torch.int32), 6) is None
    assert MT.pair_blocks(experts, ranks, 0) is None


@pytest.mark.parametrize("blocks,E,K,N", [(3, 2, 264, 520), (9, 4, 1024, 256)])
def test_grouped_gemm_applies_silu_to_the_fp32_sums(cuda_device, blocks, E, K, N):
    torch.manual_seed(blocks)
    a = torch.randn(blocks * 128, K, device=cuda_device).mul_(4).to(torch.bfloat16)
    b = (torch.randn(E, N, K, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    experts = torch.randint(0, E, (blocks,), dtype=torch.int32, device=cuda_device)
    out = MT.group_gemm(a, b, experts, activation="silu")
    check_status()
    for i in range(blocks):
        blk = slice(128 * i, 128 * i + 128)
        ref = torch.nn.functional.silu(a[blk].double() @ b[int(experts[i])].double().t())
        torch.testing.assert_close(out[blk].double(), ref, atol=1e-4, rtol=2.0 ** -8)


@pytest.mark.parametrize("blocks,most,E,K,N", [(4, 2, 4, 264, 520), (8, 3, 4, 1024, 2048), (40, 0, 8, 512, 136), (60, 30, 60, 256, 1024)])
def test_grouped_gemm_tile_width_follows_the_live_blocks(cuda_device, blocks, most, E, K, N):
    """64 to 256 columns per tile by the number of blocks the host knows of; the count on the device may be lower, and
    blocks past it stay untouched."""
    torch.manual_seed(blocks + N)
    a = torch.randn(blocks * 128, K, device=cuda_device).to(torch.bfloat16)
    b = (torch.randn(E, N, K, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    experts = torch.randint(0, E, (blocks,), dtype=torch.int32, device=cuda_device)
    live = max(1, (most or blocks) - 1)
    out = torch.full((blocks * 128, N), 7.0, dtype=torch.bfloat16, device=cuda_device)
    MT.group_gemm(a, b, experts, torch.tensor([live], dtype=torch.int32, device=cuda_device), out=out, max_blocks=most)
    check_status()
    for i in range(live):
        blk = slice(128 * i, 128 * i + 128)
        torch.testing.assert_close(out[blk].float(), a[blk].float() @ b[int(experts[i])].float().t(), atol=2.0 ** -8 / 4, rtol=2.0 ** -8)
    assert (out[128 * live:] == 7.0).all()


@pytest.mark.parametrize("blocks,E,K,N,width", [(91, 16, 512, 384, 128), (75, 8, 1032, 392, 192), (170, 8, 1032, 392, 256), (300, 4, 64, 72, 128)])
def test_grouped_gemm_tile_width_beyond_one_round(cuda_device, blocks, E, K, N, width):
    """Narrower tiles where whole ones leave the last round or the last tile of a row mostly empty, for both layouts of B."""
    from triton_distributed_b200 import _lib
    torch.manual_seed(blocks + N)
    a = torch.randn(blocks * 128, K, device=cuda_device).to(torch.bfloat16)
    b = (torch.randn(E, K, N, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    t = b.transpose(1, 2).contiguous()
    experts = torch.sort(torch.randint(0, E, (blocks,), dtype=torch.int32, device=cuda_device)).values.to(torch.int32)
    g = MT._grouped_args(a, t, False)
    g.m_per_rank, g.expert_ids = blocks * 128, experts.data_ptr()
    assert _lib.lib().tdist_gemm_tile_width(g) == width
    out, nm, act = MT.group_gemm(a, t, experts), MT.group_gemm(a, b, experts, kn=True), MT.group_gemm(a, t, experts, activation="relu")
    check_status()
    ref = torch.bmm(a.view(blocks, 128, K).double(), b[experts.long()].double()).view(-1, N)
    torch.testing.assert_close(out.double(), ref, atol=2e-5, rtol=2.0 ** -8)
    assert torch.equal(nm, out) and torch.equal(act, out.relu())


@pytest.mark.parametrize("blocks,E,K,N", [(1, 1, 8, 8), (3, 2, 72, 136), (5, 3, 264, 520), (20, 4, 1000, 264), (9, 4, 4104, 1032)])
def test_grouped_gemm_on_n_major_weights_gives_the_same_bits(cuda_device, blocks, E, K, N):
    """[E, K, N] read in place against its transposed copy: the same products summed in the same order, for tiles of 64 to 256
    columns, remainders in K and N, rows in place, gathered by the producers, staged, and staged on block pairs."""
    torch.manual_seed(blocks + N)
    rows = blocks * 128
    a = torch.randn(rows, K, device=cuda_device).to(torch.bfloat16)
    b = (torch.randn(E, K, N, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    t = b.transpose(1, 2).contiguous()
    experts = torch.sort(torch.randint(0, E, (blocks,), dtype=torch.int32, device=cuda_device)).values.to(torch.int32)
    for most in (0, 1):
        want = MT.group_gemm(a, t, experts, max_blocks=most)
        assert torch.equal(MT.group_gemm(a, b, experts, max_blocks=most, kn=True), want)
    for i in range(blocks):
        blk = slice(128 * i, 128 * i + 128)
        torch.testing.assert_close(want[blk].double(), a[blk].double() @ b[int(experts[i])].double(), atol=2e-5, rtol=2.0 ** -8)
    index = torch.randperm(rows, device=cuda_device).to(torch.int32)
    gathered = MT.group_gemm_gather(a, index, t, experts)
    assert torch.equal(MT.group_gemm_gather(a, index, b, experts, kn=True), gathered)
    count = torch.tensor([blocks], dtype=torch.int32, device=cuda_device)
    pairs = MT.pair_blocks(experts, torch.zeros_like(experts), blocks)
    for p in (None, pairs):
        staging, ready = torch.empty_like(a), MT.staging_flags(rows, cuda_device)
        for epoch in (1, 2):
            got = MT.group_gemm_gather(a, index, b, experts, count, staging=staging, block_ready=ready, epoch=epoch, pairs=p, kn=True)
            check_status()
            torch.testing.assert_close(got.float(), gathered.float(), atol=1e-5, rtol=2.0 ** -8)
    with pytest.raises(ValueError):
        MT.group_gemm(a, b, experts, activation="silu", kn=True)
    wider = torch.cat([b, b], dim=2)
    assert torch.equal(MT.group_gemm(a, wider[:, :, :N], experts, kn=True), MT.group_gemm(a, t, experts))
    assert torch.equal(MT.group_gemm(a, t.transpose(1, 2), experts, kn=True), MT.group_gemm(a, t, experts))
    with pytest.raises(ValueError):
        MT.group_gemm(a, torch.stack([b, b], dim=3)[..., 0], experts, kn=True)


@pytest.mark.parametrize("mode", ["fused", "cp_async", "staged"])
def test_contexts_use_the_weights_of_the_call(cuda_device, monkeypatch, mode):
    """Other weights on the same context, weights changed in place (through .data as well, which no version counter sees), and
    weights of every layout: each call multiplies by what it is given."""
    monkeypatch.setattr(MT, "AG_GROUP_GEMM_MODE", mode)
    torch.manual_seed(2)
    M, E, K, N, topk = 300, 4, 264, 136, 2
    x = torch.randn(M, K, device=cuda_device).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, device=cuda_device)[:topk] for _ in range(M)]).to(torch.int32)
    w = torch.rand(M, topk, device=cuda_device)
    make = lambda: (torch.randn(E, K, N, device=cuda_device) * K ** -0.5).to(torch.bfloat16)  # noqa: E731
    b = make()
    heap = LocalWorld(1, cuda_device).heap(0)
    up = MT.create_ag_group_gemm_intra_node_context(None, x, b, ids, E, max_M=M, rank=0, num_ranks=1, heap=heap)
    down = MT.create_moe_rs_context(None, 0, 1, 1, M, N, E, topk, torch.bfloat16, torch.bfloat16, cuda_device, full_topk_ids=ids,
                                    full_topk_weight=w, heap=heap)
    rows = x[torch.arange(M * topk, device=cuda_device) // topk]

    def check(weights):
        ref = _expert_matmul(rows, ids.reshape(-1), weights)
        torch.testing.assert_close(MT.ag_group_gemm_intra_node(x, weights, up).float(), ref, atol=3e-2, rtol=3e-2)
        out = MT.moe_reduce_rs(0, 1, 1, rows, weights, down)
        check_status()
        torch.testing.assert_close(out.float(), (ref.view(M, topk, N) * w.unsqueeze(-1)).sum(1), atol=6e-2, rtol=3e-2)

    check(b)
    check(make())
    b.neg_()
    check(b)
    b.data.copy_(make())
    check(b)
    check(make().transpose(1, 2).contiguous().transpose(1, 2))             # K contiguous
    check(torch.cat([make(), make()], dim=2)[:, :, N:])                    # a shard of wider weights
    check(torch.cat([make(), make()], dim=1)[:, :K])
    check(torch.cat([make(), make()], dim=2).transpose(1, 2).contiguous()[:, :N].transpose(1, 2))
    check(make()[:1].expand(E, K, N))                                      # one expert's weights for all: copied
    check(torch.stack([make(), make()], dim=3)[..., 0])                    # neither N nor K contiguous: copied
    room = torch.empty(E * K * N + 1, dtype=torch.bfloat16, device=cuda_device)
    room[1:].copy_(b.flatten())
    check(room[1:].view(E, K, N))                                          # not 16-byte aligned


@pytest.mark.parametrize("mode", ["fused", "cp_async"])
@pytest.mark.parametrize("tpr,E,K,N", [(90, 4, 264, 136), (700, 2, 2048, 520)])   # single blocks, block pairs; K within and beyond the stages
def test_abandoned_all_gather_leaves_the_grouped_gemm_usable(cuda_device, monkeypatch, mode, tpr, E, K, N):
    """A peer whose rows never come: the launch gives up, drains in step and reports a flag; the next call on the same context,
    with the rows there, is right."""
    from triton_distributed_b200.runtime import global_status
    monkeypatch.setattr(MT, "AG_GROUP_GEMM_MODE", mode)
    monkeypatch.setenv("TDIST_WAIT_TIMEOUT_MS", "50")
    torch.manual_seed(tpr)
    world, topk = 2, 2
    lw = LocalWorld(world, cuda_device)
    M = world * tpr
    shards = [torch.randn(tpr, K, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
    b = (torch.randn(E, K, N, device=cuda_device) * K ** -0.5).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, device=cuda_device)[:topk] for _ in range(M)]).to(torch.int32)
    ctxs = [MT.create_ag_group_gemm_intra_node_context(None, shards[r], b, ids, E, max_M=M, rank=r, num_ranks=world, heap=lw.heap(r))
            for r in range(world)]
    rows = torch.cat(shards)[torch.arange(M * topk, device=cuda_device) // topk]
    for call in range(2):
        MT.ag_group_gemm_intra_node(shards[0], b, ctxs[0])
        torch.cuda.synchronize()
        rec = global_status().record
        assert (rec.abort_flag, rec.code) == (1, 1)
        with pytest.raises(Exception, match="timed out"):
            check_status()
        MT.ag_group_gemm_intra_node(shards[1], b, ctxs[1], phase=1)    # the peer's send of the call that was given up
        for r in range(world):
            MT.ag_group_gemm_intra_node(shards[r], b, ctxs[r], phase=1)
        out = MT.ag_group_gemm_intra_node(shards[0], b, ctxs[0], phase=2)
        check_status()
        torch.testing.assert_close(out.float(), _expert_matmul(rows, ids.reshape(-1), b), atol=3e-2, rtol=3e-2)

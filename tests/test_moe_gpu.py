"""MoE routing kernels and the low-latency all-to-all on one GPU (ranks emulated: all send halves,
then all receive halves). Oracles: torch softmax/topk/sort, the torch restatement of the aligned
sort, and a direct gather of the rows each rank should receive (the reference checks the same
against NCCL all_to_all_single, test_all_to_all.py:184-241)."""
import pytest
import torch

from triton_distributed_b200.ops import all_to_all as A
from triton_distributed_b200.ops import moe_tp as MT
from triton_distributed_b200.ops import moe_utils as MU
from triton_distributed_b200.runtime import LocalWorld, check_status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,K", [(128, 256, 8), (7, 64, 2), (1000, 32, 4), (33, 1024, 8)])
def test_topk_softmax(cuda_device, T, E, K):
    torch.manual_seed(T + E)
    logits = torch.randn(T, E, device=cuda_device)
    ids, w = MU.topk_softmax(logits, K)
    ref_ids, ref_w = MU.topk_softmax(logits.cpu(), K)
    assert torch.equal(ids.cpu(), ref_ids)
    torch.testing.assert_close(w.cpu(), ref_w, atol=1e-6, rtol=1e-4)
    _, wn = MU.topk_softmax(logits, K, renormalize=True)
    torch.testing.assert_close(wn.sum(-1).cpu(), torch.ones(T), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("T,E,K", [(128, 256, 8), (5, 16, 2), (4096, 64, 6), (600, 300, 3)])
def test_route_is_a_stable_expert_sort(cuda_device, T, E, K):
    torch.manual_seed(T)
    ids = torch.randint(0, E, (T, K), dtype=torch.int32, device=cuda_device)
    r = MU.route(ids, E)
    ref = MU.route(ids.cpu(), E)
    for got, want in zip(r, ref):
        assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("E", [1, 7, 1024, 1025, 2048])   # 1024 | 1025: 32 and 16 warps
@pytest.mark.parametrize("T,K", [(1, 1), (33, 1), (1024, 1), (1025, 1), (513, 8), (4099, 5)])
def test_route_runs_of_every_length(cuda_device, T, E, K):
    """Pairs that end inside a warp's run, runs that are empty, and dropped pairs (id -1 or E) anywhere among them."""
    from triton_distributed_b200._lib import TdistError
    torch.manual_seed(T + E)
    ids = torch.randint(0, E, (T, K), dtype=torch.int32, device=cuda_device)
    for dropped in (False, True):
        if dropped:
            ids.view(-1)[torch.randperm(T * K, device=cuda_device)[: 1 + T * K // 9]] = -1
            ids[0, 0] = E
        r, ref = MU.route(ids, E), MU.route(ids.cpu(), E)
        if dropped:
            with pytest.raises(TdistError, match="bad argument"):
                check_status()
        else:
            check_status()
        live = int(ref.splits.sum())
        for got, want in zip(r, ref):
            n = live if want is ref.sorted_token else want.numel()
            assert torch.equal(got.cpu()[:n], want[:n])


@pytest.mark.parametrize("ranks,tpr,E,K,bs", [(8, 128, 32, 2, 128), (4, 1000, 8, 4, 64), (2, 17, 256, 8, 16), (1, 300, 60, 5, 128)])
def test_align_block_size_matches_oracle(cuda_device, ranks, tpr, E, K, bs):
    torch.manual_seed(ranks * tpr)
    ids = torch.randint(0, E, (ranks * tpr, K), dtype=torch.int32, device=cuda_device)
    got = MU.sort_topk_ids_align_block_size(ids, E, ranks, tpr, bs)
    want = MU.full_moe_align_block_size(ids, bs, E, ranks, tpr)
    total = int(want[4].item())
    assert int(got[4].item()) == total
    assert torch.equal(got[0], want[0])  # sorted ids incl. padding up to capacity
    nb = total // bs
    assert torch.equal(got[1][:nb], want[1][:nb]) and torch.equal(got[2][:nb], want[2][:nb])
    assert torch.equal(got[3], want[3])


def _emulated(world, fn_send, fn_recv):
    for r in range(world):
        fn_send(r)
    outs = [fn_recv(r) for r in range(world)]
    check_status()
    return outs


@pytest.mark.parametrize("world,T,E,K,H,with_scale", [(2, 16, 8, 2, 256, True), (4, 128, 32, 4, 1024, False), (8, 128, 256, 8, 7168, True)])
def test_fast_all_to_all_rows_land_in_source_slots(cuda_device, world, T, E, K, H, with_scale):
    torch.manual_seed(world + T)
    lw = LocalWorld(world, cuda_device)
    epr = E // world
    max_m = T * K
    ctxs = [A.create_all_to_all_context(max_m, H, r, E, world, epr, heap=lw.heap(r), device=cuda_device) for r in range(world)]
    for it in range(3):
        sends, cums, scales = [], [], []
        for r in range(world):
            ids = torch.randint(0, E, (T, K), dtype=torch.int32, device=cuda_device)
            rt = MU.route(ids, E)
            x = torch.randn(T, H, device=cuda_device).to(torch.bfloat16)
            sends.append(x[rt.sorted_token.long()].contiguous())
            cums.append(rt.cumsum)
            scales.append(torch.rand(T * K, device=cuda_device) if with_scale else None)
        _emulated(world, lambda r: A.fast_all_to_all(ctxs[r], sends[r], cums[r], scales[r], phase=1), lambda r: None)
        outs = [A.fast_all_to_all(ctxs[r], sends[r], cums[r], scales[r], phase=2) for r in range(world)]
        check_status()
        for d in range(world):
            splits, recv, rscale = outs[d]
            for s in range(world):
                lo, hi = int(cums[s][d * epr]), int(cums[s][(d + 1) * epr])
                assert torch.equal(recv[s * max_m: s * max_m + hi - lo], sends[s][lo:hi]), (it, d, s)
                want = cums[s][d * epr + 1:(d + 1) * epr + 1] - cums[s][d * epr:(d + 1) * epr]
                assert torch.equal(splits[s * epr:(s + 1) * epr], want)
                if with_scale:
                    assert torch.equal(rscale[s * max_m: s * max_m + hi - lo, 0], scales[s][lo:hi])
            data, _ = A.all_to_all_post_process(ctxs[d], splits, recv, rscale)
            assert data.shape[0] == int(splits.sum())


@pytest.mark.parametrize("world,T,E,K,H", [(2, 8, 4, 2, 256), (8, 128, 256, 8, 7168), (4, 100, 64, 6, 2048)])
def test_fused_dispatch_combine_roundtrip(cuda_device, world, T, E, K, H):
    """Identity experts: out[t] = sum_k w[t,k] * dequant(quant(x[t]))."""
    torch.manual_seed(world * 3 + T)
    lw = LocalWorld(world, cuda_device)
    ctxs = [A.create_moe_dispatch_context(T, H, K, E, r, world, heap=lw.heap(r), device=cuda_device) for r in range(world)]
    for it in range(2):
        xs = [torch.randn(T, H, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
        routed = [MU.topk_softmax(torch.randn(T, E, device=cuda_device), K) for _ in range(world)]
        for r in range(world):
            A.moe_dispatch(ctxs[r], xs[r], routed[r][0], routed[r][1], phase=1)
        recvs = [A.moe_dispatch(ctxs[r], xs[r], routed[r][0], routed[r][1], phase=2) for r in range(world)]
        check_status()
        for r in range(world):   # per-source splits as the receiver sees them
            want = torch.stack([torch.bincount(routed[s][0].reshape(-1).long(), minlength=E)[r * (E // world):(r + 1) * (E // world)]
                                for s in range(world)])
            assert torch.equal(recvs[r][2].long(), want)
        # quantisation matches the torch statement on what rank 0 received from rank 1 (or itself)
        d, s = 0, world - 1
        rx, rs, splits = recvs[d]
        n = int(splits[s].sum())
        rt = MU.route(routed[s][0], E)
        rows = rt.sorted_token.long()[int(rt.cumsum[0]): int(rt.cumsum[E // world])]
        q_ref, s_ref = A.quant_fp8_reference(xs[s][rows])
        mm = T * K
        torch.testing.assert_close(rs[s * mm: s * mm + n], s_ref, rtol=1e-6, atol=0)
        assert (rx[s * mm: s * mm + n].view(torch.uint8).int() - q_ref.view(torch.uint8).int()).abs().max() <= 1
        # identity experts
        # identity experts: odd iterations write straight into the symmetric output buffer, even ones pass a tensor
        if it & 1:
            ys = [A.dequant_fp8(recvs[r][0], recvs[r][1], out=A.moe_expert_out_buffer(ctxs[r])) for r in range(world)]
        else:
            ys = [A.dequant_fp8(recvs[r][0], recvs[r][1]) for r in range(world)]
        outs = [None] * world
        for r in range(world):
            A.moe_combine(ctxs[r], ys[r], recvs[r][2], phase=1)
        for r in range(world):
            outs[r] = A.moe_combine(ctxs[r], ys[r], recvs[r][2], phase=2)
        check_status()
        for r in range(world):
            q, sc = A.quant_fp8_reference(xs[r])
            deq = (q.float().view(T, H // 128, 128) * sc.unsqueeze(-1)).view(T, H).to(torch.bfloat16).float()
            ref = deq * routed[r][1].sum(-1, keepdim=True)
            torch.testing.assert_close(outs[r].float(), ref, atol=2e-2, rtol=2e-2)


def test_route_rejects_out_of_range_expert_ids(cuda_device):
    """An id of -1 (a dropped pair) or E must not index shared memory: the pair is left out, its slot is -1, and the
    status block carries a bad-argument record that check_status() raises."""
    from triton_distributed_b200._lib import TdistError
    T, E, K = 64, 16, 2
    torch.manual_seed(5)
    ids = torch.randint(0, E, (T, K), dtype=torch.int32, device=cuda_device)
    ids[3, 1] = -1
    ids[40, 0] = E
    r = MU.route(ids, E)
    with pytest.raises(TdistError, match="bad argument"):
        check_status()
    ref = MU.route(ids.cpu(), E)
    assert int(r.splits.sum()) == T * K - 2
    assert torch.equal(r.splits.cpu(), ref.splits) and torch.equal(r.cumsum.cpu(), ref.cumsum)
    assert torch.equal(r.slot_of.cpu(), ref.slot_of)
    assert int(r.slot_of[3 * K + 1]) == -1 and int(r.slot_of[40 * K]) == -1
    live = T * K - 2
    assert torch.equal(r.sorted_token[:live].cpu(), ref.sorted_token[:live])
    # the aligned sort drops the same pairs: no sorted entry names them
    got = MU.sort_topk_ids_align_block_size(ids, E, 1, T, 16)
    with pytest.raises(TdistError, match="bad argument"):
        check_status()
    named = got[0][got[0] < T * K]
    assert named.numel() == live and (3 * K + 1) not in named.tolist() and (40 * K) not in named.tolist()
    # a clean call afterwards reports nothing
    MU.route(torch.randint(0, E, (T, K), dtype=torch.int32, device=cuda_device), E)
    check_status()


def test_fast_all_to_all_reports_a_destination_overflow(cuda_device):
    """More than max_m rows for one destination: max_m rows are sent, the published splits say so, and the status
    block records the bad argument instead of rows spilling into the next source's slot."""
    from triton_distributed_b200._lib import TdistError
    world, E, H, max_m = 2, 4, 256, 8
    lw = LocalWorld(world, cuda_device)
    epr = E // world
    ctxs = [A.create_all_to_all_context(max_m, H, r, E, world, epr, heap=lw.heap(r), device=cuda_device) for r in range(world)]
    # rank 0 sends 12 rows to rank 1's experts (2 and 3): 7 + 5 > max_m
    cums = torch.tensor([0, 1, 2, 9, 14], dtype=torch.int32, device=cuda_device)
    send = torch.randn(14, H, device=cuda_device).to(torch.bfloat16)
    A.fast_all_to_all(ctxs[0], send, cums, None, phase=1)
    with pytest.raises(TdistError, match="bad argument"):
        check_status()
    empty = torch.zeros(E + 1, dtype=torch.int32, device=cuda_device)   # rank 1 sends nothing
    A.fast_all_to_all(ctxs[1], send[:1], empty, None, phase=1)
    splits, recv, _ = A.fast_all_to_all(ctxs[1], send[:1], empty, None, phase=2)
    check_status()
    assert splits[:epr].tolist() == [7, 1]          # clamped to the 8 rows that were sent
    assert torch.equal(recv[:max_m], send[2:2 + max_m])


@pytest.mark.parametrize("world,T,E,K,H,align", [(2, 33, 8, 2, 256, 1), (4, 64, 32, 4, 512, 128), (8, 128, 256, 8, 1024, 128), (1, 50, 4, 3, 128, 16)])
def test_ep_dispatch_compact_layout_and_pull_combine(cuda_device, world, T, E, K, H, align):
    """Compact (expert-major) receive layout with block-aligned groups: every rank's rows sit where the gathered
    counts say, the block -> expert table covers them, and the pull combine returns K x the input (identity
    experts, plain sum). The (token, k) pairs of rank 1 include a dropped pair (id -1)."""
    from triton_distributed_b200._lib import TdistError
    from triton_distributed_b200.ops import moe_ep as EP
    torch.manual_seed(world * 11 + T)
    lw = LocalWorld(world, cuda_device)
    ctxs = [EP.create_ep_context(T, H, K, E, r, world, quant=False, compact=True, align=align, heap=lw.heap(r), device=cuda_device)
            for r in range(world)]
    epr = E // world
    for it in range(3):
        xs = [torch.randn(T, H, device=cuda_device).to(torch.bfloat16) for _ in range(world)]
        ids = [torch.randint(0, E, (T, K), dtype=torch.int32, device=cuda_device) for _ in range(world)]
        dropped = world > 1 and it == 1
        if dropped:
            ids[1][5, 0] = -1
        for phase in (1, 2):
            for r in range(world):
                EP.ep_dispatch(ctxs[r], xs[r], ids[r], None, phase=phase)
        recv = [EP.ep_dispatch(ctxs[r], xs[r], ids[r], None, phase=4) for r in range(world)]
        if dropped:
            with pytest.raises(TdistError, match="bad argument"):
                check_status()
        else:
            check_status()
        for d in range(world):
            rows, _, splits, num_recv = recv[d]
            off, total = 0, 0
            for le in range(epr):
                e = d * epr + le
                group = torch.cat([xs[s][(ids[s].reshape(-1) == e).nonzero().flatten() // K] for s in range(world)])
                n = group.shape[0]
                assert torch.equal(rows[off: off + n], group), (it, d, le)
                nb = (n + align - 1) // align
                assert (ctxs[d].block_expert[off // align: off // align + nb] == le).all()
                off += nb * align
                total += n
            assert int(num_recv) == total and int(ctxs[d].num_blocks) == off // align
        for r in range(world):
            EP.expert_out_buffer(ctxs[r]).copy_(recv[r][0])     # identity experts, written in place
            EP.ep_combine(ctxs[r], None, weighted=False, phase=1)
        outs = [EP.ep_combine(ctxs[r], None, weighted=False, phase=2) for r in range(world)]
        check_status()
        for r in range(world):
            live = (ids[r] >= 0).sum(-1, keepdim=True).float()
            torch.testing.assert_close(outs[r].float(), xs[r].float() * live, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("E", [1, 8, 31, 32, 33, 60, 64, 100, 256, 300, 1024])
def test_topk_softmax_over_every_register_width(cuda_device, E):
    torch.manual_seed(E)
    logits = torch.randn(37, E, device=cuda_device)
    logits[3] = 0.0                               # ties: the lower expert ids
    logits[4, 1:] = torch.finfo(torch.float32).min
    k = min(E, 8)
    for renorm in (False, True):
        ids, w = MU.topk_softmax(logits, k, renormalize=renorm)
        ids_c, w_c = MU.topk_softmax(logits.cpu(), k, renormalize=renorm)
        rows = [i for i in range(37) if i != 4]   # row 4: equal (zero) probabilities in any order after the first
        assert torch.equal(ids.cpu()[rows], ids_c[rows]) and ids[4, 0] == 0
        torch.testing.assert_close(w.cpu(), w_c, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("T,hidden,E,k", [(1, 32, 8, 1), (3, 512, 8, 2), (16, 544, 16, 4), (17, 2048, 32, 8), (128, 7168, 32, 8),
                                          (33, 1024, 60, 5), (50, 4096, 64, 8), (40, 512, 130, 6), (9, 64, 1024, 8)])
def test_gate_topk_is_no_further_from_float64_than_the_fp32_product(cuda_device, T, hidden, E, k):
    torch.manual_seed(T + hidden + E)
    x = torch.randn(T, hidden, device=cuda_device).bfloat16()
    gate = (torch.randn(E, hidden, device=cuda_device) * hidden ** -0.5).bfloat16()
    logits = torch.empty(T, E, device=cuda_device)
    ids, w = MU.gate_topk(x, gate, k, renormalize=True, logits=logits)
    exact = x.double() @ gate.double().t()
    before = (x.float() @ gate.float().t()).double()
    assert (logits.double() - exact).norm() <= max((before - exact).norm().item(), 1e-7 * exact.norm().item())
    ids_t, w_t = MU.topk_softmax(logits, k, renormalize=True)
    assert torch.equal(ids, ids_t)
    torch.testing.assert_close(w, w_t, rtol=1e-6, atol=0)


@pytest.mark.parametrize("T,hidden,E,k", [(1, 1024, 3, 2), (1, 8192, 1024, 8), (15, 2080, 16, 4), (300, 1536, 8, 2), (600, 4096, 64, 6), (1184, 1024, 60, 4)])
def test_gate_topk_parts_of_the_hidden_dimension(cuda_device, T, hidden, E, k):
    """One to eight parts, and the token counts from which on there are fewer. The products of bf16 are exact; a sum passes at most
    hidden / 512 additions in a warp, 16 over the warps, 8 over the parts and two inside an MMA, each off by at most 2^-23 of the
    sum of the magnitudes."""
    torch.manual_seed(T + hidden + E)
    x = torch.randn(T, hidden, device=cuda_device).bfloat16()
    gate = (torch.randn(E, hidden, device=cuda_device) * hidden ** -0.5).bfloat16()
    logits = torch.empty(T, E, device=cuda_device)
    ids, w = MU.gate_topk(x, gate, k, logits=logits)
    exact = x.double() @ gate.double().t()
    spread = x.double().abs() @ gate.double().abs().t()
    assert ((logits.double() - exact).abs() <= (hidden / 512 + 26) * 2.0 ** -23 * spread).all()
    ids_t, w_t = MU.topk_softmax(logits, k)
    assert torch.equal(ids, ids_t)
    torch.testing.assert_close(w, w_t, rtol=1e-6, atol=0)


@pytest.mark.parametrize("hidden,E,k", [(64, 3, 1), (544, 8, 2), (992, 40, 4), (1024, 16, 4), (2080, 60, 6), (4096, 8, 2), (7168, 64, 8),
                                        (8192, 64, 8), (7168, 130, 8), (12288, 64, 8), (2048, 520, 6), (512, 1024, 32), (2048, 24, 3),
                                        (4096, 16, 2), (8192, 32, 8), (12288, 32, 4)])
def test_gate_topk_of_a_token_is_the_same_in_any_batch(cuda_device, hidden, E, k):
    """Every form of the launch, at both sides of the token counts and sizes from which on there is another: bit by bit the
    logits, experts and weights of the largest batch."""
    torch.manual_seed(hidden + E)
    x = torch.randn(1200, hidden, device=cuda_device).bfloat16()
    gate = (torch.randn(E, hidden, device=cuda_device) * hidden ** -0.5).bfloat16()
    want = torch.empty(1200, E, device=cuda_device)
    ids, w = MU.gate_topk(x, gate, k, renormalize=True, logits=want)
    exact, spread = x.double() @ gate.double().t(), x.double().abs() @ gate.double().abs().t()
    # additions of a chain, of the chains, and inside an MMA, each off by at most 2^-23 of the sum of the magnitudes
    assert ((want.double() - exact).abs() <= (hidden / 512 + 18) * 2.0 ** -23 * spread).all()
    for T in (1, 17, 240, 241, 528, 529, 1184, 1185):
        logits = torch.empty(T, E, device=cuda_device)
        ids_t, w_t = MU.gate_topk(x[:T], gate, k, renormalize=True, logits=logits)
        assert torch.equal(logits, want[:T]), T
        assert torch.equal(ids_t, ids[:T]) and torch.equal(w_t, w[:T]), T


@pytest.mark.parametrize("T,hidden,E,k", [(1, 256, 64, 1), (37, 1032, 64, 33), (5, 256, 64, 64), (513, 128, 64, 1), (1024, 256, 8, 8), (700, 4096, 16, 5), (1100, 4096, 16, 8)])
@pytest.mark.parametrize("compact", [False, True])
def test_dispatch_rows_of_every_pair(cuda_device, T, hidden, E, k, compact):
    """Runs of pairs shorter and longer than the ids a lane loads at a time, a ragged last segment, more items than warps, and routing
    both in place and by a launch of its own (1100 x 8 pairs, recorded by all CTAs): every pair's row is its token's, bit by
    bit; dropped pairs (id -1) have none."""
    from triton_distributed_b200._lib import TdistError
    from triton_distributed_b200.ops import moe_ep as EP
    torch.manual_seed(T + k)
    x = torch.randn(T, hidden, device=cuda_device).bfloat16()
    ids = torch.randint(0, E, (T, k), dtype=torch.int32, device=cuda_device)
    ctx = EP.create_ep_context(T, hidden, k, E, 0, 1, quant=False, compact=compact, heap=LocalWorld(1, cuda_device).heap(0), device=cuda_device)
    for dropped in (False, True):
        if dropped:
            ids[T // 2, k - 1] = -1
        rows, _, _, num = EP.ep_dispatch(ctx, x, ids)
        if dropped:
            with pytest.raises(TdistError, match="bad argument"):
                check_status()
        else:
            check_status()
        at = ctx.pair_row[: T * k].long()
        live = ids.reshape(-1) >= 0
        assert (at[~live] == -1).all() and int(num) == int(live.sum()) == at[live].unique().numel()
        assert torch.equal(rows[at[live]], x.repeat_interleave(k, 0)[live])


@pytest.mark.parametrize("form", ["bf16", "strided", "misaligned", "short", "cpu"])
def test_gate_topk_writes_logits_of_any_form_or_refuses_them(cuda_device, form):
    """Only a dense fp32 [T, E] buffer may be handed to the kernel as a pointer; the others are copied into, converted and
    strided as they are, or refused, and nothing around them is written."""
    torch.manual_seed(5)
    T, hidden, E, k = 9, 64, 16, 2
    x = torch.randn(T, hidden, device=cuda_device).bfloat16()
    gate = torch.randn(E, hidden, device=cuda_device).bfloat16()
    want = x.double() @ gate.double().t()
    room = torch.full((4 * T * E,), 7.0, dtype=torch.bfloat16 if form == "bf16" else torch.float32, device="cpu" if form == "cpu" else cuda_device)
    if form == "strided":
        logits = room.view(2 * T, 2 * E)[:T, ::2]
    elif form == "misaligned":
        logits = room[1: 1 + T * E].view(T, E)
    elif form == "short":
        logits = room[: (T - 1) * E].view(T - 1, E)
        with pytest.raises(RuntimeError):
            MU.gate_topk(x, gate, k, logits=logits)
        assert (room == 7.0).all()
        return
    else:
        logits = room[: T * E].view(T, E)
    ids, _ = MU.gate_topk(x, gate, k, logits=logits)
    # fp32 sums of 64 products, then the buffer's rounding
    torch.testing.assert_close(logits.double().cpu(), want.cpu(), rtol=2.0 ** -8 if form == "bf16" else 1e-5, atol=1e-5)
    assert torch.equal(ids.long(), want.topk(k, -1).indices)
    logits.fill_(7.0)
    assert (room == 7.0).all()


@pytest.mark.parametrize("T,k,hidden", [(1, 1, 8), (3, 2, 0), (5, 2, 1024), (64, 3, 1032), (7, 8, 7168), (300, 2, 4096), (2, 1, 1016)])
def test_topk_reduce_over_ragged_rows_and_rejected_pairs(cuda_device, T, k, hidden):
    torch.manual_seed(T + hidden)
    y = torch.randn(T * k + 3, hidden, device=cuda_device).bfloat16()
    pos = torch.randperm(T * k + 3, device=cuda_device)[:T * k].to(torch.int32)
    w = torch.rand(T, k, device=cuda_device)
    if T > 2:
        pos[k] = -1                               # a pair that routing rejected contributes nothing
    rows = torch.where((pos >= 0).unsqueeze(1), y[pos.long().clamp(min=0)].float(), torch.zeros((), device=cuda_device)).view(T, k, hidden)
    for weights in (w, None):
        ref = (rows * (weights.unsqueeze(-1) if weights is not None else 1.0)).sum(1)
        out = MT.topk_reduce(y, pos, weights, T, k)
        torch.testing.assert_close(out.float(), ref, rtol=2.0 ** -8, atol=1e-5)


@pytest.mark.parametrize("T,topk,E", [(1, 1, 1), (31, 1, 8), (64, 8, 32), (513, 1, 16), (171, 3, 60), (1024, 8, 256), (300, 2, 1024)])
@pytest.mark.parametrize("align", [1, 128])
def test_dispatch_sorts_the_pairs_stably(cuda_device, T, topk, E, align):
    """Rows land in stable expert order for pair counts around the 32 and 512 pairs the sort steps by, and up to the most
    it routes in place; some pairs are rejected (id -1 and E)."""
    from triton_distributed_b200.ops import moe_ep as EP
    from triton_distributed_b200.runtime import global_status
    torch.manual_seed(T + E)
    x = torch.randn(T, 256, device=cuda_device).to(torch.bfloat16)
    ids = torch.randint(0, E, (T, topk), dtype=torch.int32, device=cuda_device)
    ctx = EP.create_ep_context(T, 256, topk, E, 0, 1, quant=False, compact=True, align=align, heap=LocalWorld(1, cuda_device).heap(0))
    for bad in (False, True):
        if bad and T > 30:
            ids[3, 0], ids[T - 1, topk - 1] = -1, E
        recv, _, splits, num = EP.ep_dispatch(ctx, x, ids, None)
        torch.cuda.synchronize()
        if bad and T > 30:
            with pytest.raises(Exception, match="bad argument"):
                global_status().check()
        else:
            check_status()
        flat = ids.reshape(-1).long()
        counts = torch.bincount(flat[(flat >= 0) & (flat < E)], minlength=E)
        assert torch.equal(splits.view(-1).long(), counts) and int(num) == int(counts.sum())
        padded = (counts + align - 1) // align * align
        start = torch.cumsum(padded, 0) - padded
        for e in range(E):
            tokens = torch.nonzero(flat == e).flatten() // topk
            assert torch.equal(recv[start[e]: start[e] + tokens.numel()], x[tokens])
        blocks = int(padded.sum()) // align
        assert int(ctx.num_blocks) == blocks
        want = torch.repeat_interleave(torch.arange(E, device=cuda_device), padded // align)
        assert torch.equal(ctx.block_expert[:blocks].long(), want)


@pytest.mark.parametrize("compact", [False, True])
def test_halves_launched_apart_meet_at_the_own_flag(cuda_device, monkeypatch, compact):
    """One rank. The wait half must not return before the send half has raised this rank's flag: with nothing sent it gives
    up after its limit and names the rank; after the send half (synchronised: the two never run at once) it finds flag,
    counts and rows, from another stream."""
    from triton_distributed_b200.ops import moe_ep as EP
    from triton_distributed_b200.runtime import global_status
    monkeypatch.setenv("TDIST_WAIT_TIMEOUT_MS", "50")
    torch.manual_seed(3)
    T, hidden, E, k = 33, 256, 8, 2
    x = torch.randn(T, hidden, device=cuda_device).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, device=cuda_device)[:k] for _ in range(T)]).to(torch.int32)
    ctx = EP.create_ep_context(T, hidden, k, E, 0, 1, quant=False, compact=compact, heap=LocalWorld(1, cuda_device).heap(0))

    ctx.topk_ids, ctx.ntok = ids, T

    def gives_up(launch):
        launch()
        torch.cuda.synchronize()
        rec = global_status().record
        assert (rec.abort_flag, rec.code, rec.peer) == (1, 1, 0)
        with pytest.raises(Exception, match="timed out"):
            check_status()

    send, wait = torch.cuda.Stream(), torch.cuda.Stream()
    for call in (1, 2):
        # as a wait half sees it that reaches the GPU before the send half of its call
        ctx.call_count += 1
        gives_up(lambda: EP.ep_dispatch(ctx, x, ids, None, phase=4))
        if compact:
            gives_up(lambda: EP.ep_dispatch(ctx, x, ids, None, phase=6))   # the counts' flag
        ctx.call_count -= 1
        torch.cuda.synchronize()
        EP.ep_dispatch(ctx, x, ids, None, phase=3, stream=send)
        send.synchronize()
        assert int(ctx.sig.local[0]) == ctx.call_count == call
        rows, _, splits, num = EP.ep_dispatch(ctx, x, ids, None, phase=4, stream=wait)
        wait.synchronize()
        check_status()
        order = torch.sort(ids.reshape(-1).long(), stable=True).indices
        assert torch.equal(rows[: T * k], x[order // k]) and int(num) == T * k
        assert torch.equal(splits.view(-1).long(), torch.bincount(ids.reshape(-1).long(), minlength=E))
        ctx.combine_count += 1
        gives_up(lambda: EP.ep_combine(ctx, weighted=False, phase=2))
        ctx.combine_count -= 1
        out = torch.zeros(T, hidden, dtype=torch.bfloat16, device=cuda_device)
        EP.ep_combine(ctx, rows, weighted=False, phase=1)
        torch.cuda.synchronize()
        assert int(ctx.comb_sig.local[0]) == ctx.combine_count
        EP.ep_combine(ctx, weighted=False, out=out, phase=2, stream=wait)
        wait.synchronize()
        check_status()
        torch.testing.assert_close(out.float(), k * x.float(), rtol=2.0 ** -8, atol=0)
    # whole calls in between leave the flags behind; halves after them still meet at theirs
    EP.ep_dispatch(ctx, x, ids, None)
    EP.ep_dispatch(ctx, x, ids, None, phase=3)
    EP.ep_dispatch(ctx, x, ids, None, phase=4)
    check_status()
    assert int(ctx.sig.local[0]) == ctx.call_count

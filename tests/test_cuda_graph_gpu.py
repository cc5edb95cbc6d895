"""Single-GPU ops inside a CUDA graph: a decode step (attention + a tcgen05 GEMM on its output + top-k routing)
is captured once and replayed with new contents in the same buffers. The launchers take the stream from
torch, allocate nothing during capture once warmed up, and read lengths and routing on the device, so the
graph stays valid when the data changes. (Ops whose flags carry a host-side call number - the fused
collectives - are not captured: every launch needs a new number.)"""
import math

import pytest
import torch

from triton_distributed_b200.ops import flash_decode as FD
from triton_distributed_b200.ops import gemm as G
from triton_distributed_b200.ops import moe_utils as MU
from triton_distributed_b200.runtime import check_status

pytestmark = pytest.mark.gpu


def test_decode_step_replays_from_a_cuda_graph(cuda_device):
    torch.manual_seed(0)
    dev = cuda_device
    B, Hq, Hkv, D, page, max_len = 4, 32, 8, 128, 16, 2048
    blocks = B * (max_len // page)
    k = torch.randn(blocks, page, Hkv, D, device=dev).to(torch.bfloat16)
    v = torch.randn(blocks, page, Hkv, D, device=dev).to(torch.bfloat16)
    table = torch.randperm(blocks, device=dev).view(B, max_len // page).to(torch.int32)
    q = torch.randn(B, Hq, D, device=dev).to(torch.bfloat16)
    lens = torch.tensor([5, 700, 2048, 1], dtype=torch.int32, device=dev)
    w_o = (torch.randn(512, Hq * D, device=dev) * (Hq * D) ** -0.5).to(torch.bfloat16)
    w_gate = (torch.randn(64, 512, device=dev) * 512 ** -0.5).to(torch.bfloat16)
    attn = torch.empty_like(q)
    proj = torch.empty(B, 512, device=dev, dtype=torch.bfloat16)
    logits = torch.empty(B, 64, device=dev, dtype=torch.bfloat16)
    scale = 1.0 / math.sqrt(D)

    def step():
        FD.gqa_fwd_batch_decode(q, k, v, None, None, lens, table, scale, output_combine=attn)
        G.gemm_persistent(attn.view(B, Hq * D), w_o, out=proj)
        G.gemm_persistent(proj, w_gate, out=logits)
        return MU.topk_softmax(logits.float(), 4, True)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):          # warm-up: workspaces, function attributes, tensor-map cache
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ids_g, w_g = step()
    for trial in range(3):
        q.copy_(torch.randn(B, Hq, D, device=dev).to(torch.bfloat16))
        lens.copy_(torch.randint(1, max_len + 1, (B,), device=dev, dtype=torch.int32))
        graph.replay()
        torch.cuda.synchronize()
        check_status()
        got_attn, got_ids, got_w = attn.clone(), ids_g.clone(), w_g.clone()
        ref = FD.ref_paged_attn(q, k, v, lens, table, scale)
        torch.testing.assert_close(got_attn.float(), ref, atol=1e-2, rtol=1e-2)
        ids_e, w_e = step()           # the same ops launched eagerly on the same inputs
        torch.cuda.synchronize()
        assert torch.equal(got_ids, ids_e)
        torch.testing.assert_close(got_w, w_e, atol=0, rtol=0)


@pytest.mark.parametrize("captured", [False, True], ids=["eager", "cuda_graph"])
def test_early_launches_on_two_streams_meet_at_their_events(cuda_device, captured):
    """Early-launched kernels before a fork, on both branches and behind the join, each reading what the one before it, or the
    other branch, has just written: few-row and large tiles, activation, routing, decode."""
    torch.manual_seed(1)
    dev = cuda_device
    bf = lambda *shape, scale=1.0: (torch.randn(*shape, device=dev) * scale).to(torch.bfloat16)  # noqa: E731
    M, H = 64, 1024
    w = [bf(H, H, scale=H ** -0.5) for _ in range(4)]
    gate = bf(16, H, scale=H ** -0.5)
    ctx = G.create_ag_gemm_intra_node_context(w[0], w[0], 0, 1, max_M=4 * M)
    x = bf(4 * M, H)
    buf = [torch.empty_like(x) for _ in range(4)]
    attn = torch.empty(8, 32, 128, dtype=torch.bfloat16, device=dev)
    k, v = bf(64, 16, 8, 128), bf(64, 16, 8, 128)
    table = torch.randperm(64, device=dev).to(torch.int32).view(8, 8)
    lens = torch.randint(1, 129, (8,), dtype=torch.int32, device=dev)
    q_from = torch.empty(32, H, dtype=torch.bfloat16, device=dev)
    other = torch.cuda.Stream()

    def step(concurrent=True):
        stream = torch.cuda.current_stream()
        G.ag_gemm_intra_node(x, w[0], ctx, out=buf[0], activation="gelu")         # large tiles, activation in place
        side = other if concurrent else stream
        side.wait_stream(stream)
        with torch.cuda.stream(side):
            G.gemm_persistent(buf[0][:32], w[1], out=q_from)                      # few rows
            FD.gqa_fwd_batch_decode(q_from.view(8, 32, 128), k, v, None, None, lens, table, 128 ** -0.5, output_combine=attn)
        G.gemm_persistent(buf[0][:M], w[2], out=buf[2][:M])
        ids, weights = MU.gate_topk(buf[2][:M], gate, 4, renormalize=True)
        stream.wait_stream(side)
        G.gemm_persistent(attn.view(32, H), w[3], out=buf[3][:32])                # behind the join: reads the other branch
        G.gemm_persistent(buf[3][:32], w[0], out=buf[1][:32])
        return ids, weights

    step()
    torch.cuda.synchronize()
    graph = None
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ids, weights = step()
    for _ in range(5):
        x.copy_(bf(4 * M, H))
        if graph is not None:
            graph.replay()
        else:
            ids, weights = step()
        torch.cuda.synchronize()
        check_status()
        got = [ids.clone(), weights.clone(), buf[0].clone(), buf[1][:32].clone(), attn.clone()]
        torch.testing.assert_close(buf[0].float(), torch.nn.functional.gelu(x.float() @ w[0].float().t(), approximate="tanh"), atol=3e-2, rtol=2e-2)
        one = step(concurrent=False)
        torch.cuda.synchronize()
        for have, need in zip(got, [*one, buf[0], buf[1][:32], attn]):
            assert torch.equal(have, need)

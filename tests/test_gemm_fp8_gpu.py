"""Block-scaled fp8 GEMM on one GPU: plain numerics, and the fused AG kernel of one emulated rank at a
time against peer buffers prepared by the host (LocalWorld).

Oracle: fp32 torch matmul of the dequantised operands (values = fp8 * scale), i.e. the same op
restated without tensor cores. The kernel accumulates each 128-wide K block in fp32 on the tensor
core and folds it in with an fp32 FMA, so the only rounding besides summation order is the final
bf16 store.
"""
import pytest
import torch

from triton_distributed_b200.ops import gemm_fp8 as F
from triton_distributed_b200.runtime import LocalWorld, check_status

pytestmark = pytest.mark.gpu



def _operands(M, N, K, dev, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    # per-block magnitudes spread over several octaves so that a wrong or misplaced scale is visible
    x = torch.randn(M, K, generator=g) * torch.exp2(torch.randint(-3, 4, (M, K // 128), generator=g).float()).repeat_interleave(128, 1)
    w = torch.randn(N, K, generator=g) * K ** -0.5
    wblk = torch.exp2(torch.randint(-2, 3, ((N + 127) // 128, K // 128), generator=g).float())
    w = w * wblk.repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    a, sa = F.quantize_fp8_rowwise(x.to(dev))
    b, sb = F.quantize_fp8_blockwise(w.to(dev))
    return a, sa, b, sb


def test_quantisers_round_trip(cuda_device):
    a, sa, b, sb = _operands(200, 264, 384, cuda_device, 1)
    assert a.dtype == F.FP8 and sa.shape == (200, 3) and sb.shape == (3, 3)
    x = F.dequantize_fp8(a, sa, 1)
    a2, sa2 = F.quantize_fp8_rowwise(x)
    torch.testing.assert_close(F.dequantize_fp8(a2, sa2, 1), x, rtol=0.07, atol=1e-6)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,K", [(1, 128), (3, 384), (63, 128), (65, 128), (1000, 7168)])
def test_rowwise_quantiser_gives_the_bytes_of_its_torch_statement(cuda_device, M, K, dtype):
    g = torch.Generator(device="cpu").manual_seed(M + K)
    x = torch.randn(M, K, generator=g) * torch.exp2(torch.randint(-14, 15, (M, K // 128), generator=g).float()).repeat_interleave(128, 1)
    x = x.to(dtype).to(cuda_device)
    x[0, :128] = 0
    if K > 128 and M > 2:   # an infinity, a NaN, the largest and the smallest values of the type
        x[1, 5], x[1, 6], x[2, 7] = float("inf"), 1.0, float("nan")
        x[2, 128:256] = torch.finfo(dtype).max
        x[2, 256:384] = torch.finfo(dtype).smallest_normal
    (q, s), (qt, st) = F.quantize_fp8_rowwise(x), F._quantize_rowwise_torch(x)
    assert torch.equal(q.view(torch.uint8), qt.view(torch.uint8))
    torch.testing.assert_close(s, st, rtol=0, atol=0, equal_nan=True)


def _quantised_values(x):
    q, s = F.quantize_fp8_rowwise(x)
    return q.float(), s


@pytest.mark.parametrize("how", ["jit.trace", "compile", "vmap", "jvp", "grad", "functionalize", "dispatch mode", "saved tensor hooks"])
def test_rowwise_quantiser_is_torch_operations_to_whoever_traces_it(cuda_device, how):
    """The one-pass kernel stands in for torch operations only where nothing has to see them; every tracer and transform gets
    the values of the statement in torch operations, on inputs other than the ones it was traced with too."""
    g = torch.Generator(device="cpu").manual_seed(7)
    x, other = (torch.randn(6, 256, generator=g).to(cuda_device) for _ in range(2))
    want_q, want_s = F._quantize_rowwise_torch(other)
    want = (want_q.float(), want_s)
    if how == "jit.trace":
        got = torch.jit.trace(_quantised_values, (x,), check_trace=False)(other)
    elif how == "compile":
        got = torch.compile(_quantised_values, backend="eager", fullgraph=True)(other)
    elif how == "vmap":
        got = tuple(t.flatten(0, 1) for t in torch.vmap(_quantised_values)(other.view(2, 3, 256)))
    elif how == "jvp":
        # the scale is the largest magnitude / 448, so along x itself its derivative is the scale
        primal, tangent = torch.func.jvp(lambda v: F.quantize_fp8_rowwise(v)[1], (other,), (other,))
        torch.testing.assert_close(tangent, primal, rtol=1e-6, atol=0)
        got = (want[0], primal)
    elif how == "grad":
        leaf = other.clone().requires_grad_()
        F.quantize_fp8_rowwise(leaf)[1].sum().backward()
        top = other.view(6, 2, 128).abs() == other.view(6, 2, 128).abs().amax(-1, keepdim=True)
        torch.testing.assert_close(leaf.grad.view(6, 2, 128), top * other.view(6, 2, 128).sign() / 448.0, rtol=1e-6, atol=0)
        return
    elif how == "functionalize":
        got = torch.func.functionalize(_quantised_values)(other)
    elif how == "dispatch mode":
        from torch.utils._python_dispatch import TorchDispatchMode
        seen = []

        class Log(TorchDispatchMode):
            def __torch_dispatch__(self, func, types, args=(), kwargs=None):
                seen.append(str(func))
                return func(*args, **(kwargs or {}))

        with Log():
            got = _quantised_values(other)
        assert any("amax" in f for f in seen)
    else:
        packed = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t, lambda t: t):
            q, s = F.quantize_fp8_rowwise(other.clone().requires_grad_())
        assert packed
        got = (q.float(), s)
    for have, need in zip(got, want):
        torch.testing.assert_close(have, need, rtol=0, atol=0)


def test_rowwise_quantiser_takes_the_kernel_for_plain_tensors(cuda_device):
    from triton_distributed_b200.utils.misc import plain_cuda
    x = torch.randn(4, 128, device=cuda_device)
    assert plain_cuda(x) and plain_cuda(torch.nn.Parameter(x, requires_grad=False))
    with torch.no_grad():
        assert plain_cuda(torch.nn.Parameter(x))
    assert not plain_cuda(torch.nn.Parameter(x)) and not plain_cuda(x.t()) and not plain_cuda(x.flatten()[1:]) and not plain_cuda(x.cpu())


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (256, 512, 512), (300, 264, 384), (1000, 1000, 896), (4096, 768, 2048)])
def test_plain_fp8_gemm_matches_fp32_reference(cuda_device, M, N, K):
    a, sa, b, sb = _operands(M, N, K, cuda_device, M + N + K)
    c = F.gemm_fp8_blockscaled(a, sa, b, sb)
    check_status()
    ref = F.dequantize_fp8(a, sa, 1) @ F.dequantize_fp8(b, sb, 128).t()
    assert torch.isfinite(c).all()
    torch.testing.assert_close(c.float(), ref, atol=2e-2 * ref.abs().max().item() / 4, rtol=1e-2)


def test_fp8_gemm_is_deterministic_across_calls(cuda_device):
    a, sa, b, sb = _operands(512, 512, 1024, cuda_device, 7)
    c1 = F.gemm_fp8_blockscaled(a, sa, b, sb)
    c2 = F.gemm_fp8_blockscaled(a, sa, b, sb, num_sms=37)
    check_status()
    assert torch.equal(c1, c2)


@pytest.mark.parametrize("world,mpr,N,K", [(1, 200, 256, 256), (2, 128, 256, 128), (4, 250, 520, 384), (8, 96, 256, 512)])
def test_ag_fp8_gemm_single_rank_kernels_against_prepared_peers(cuda_device, world, mpr, N, K):
    """Each emulated rank's fused kernel runs alone: rows and scales of lower ranks were really pushed
    by their kernels, those of higher ranks are written by the host together with their flags."""
    lw = LocalWorld(world, cuda_device)
    ops = [_operands(mpr, N, K, cuda_device, 100 * world + r) for r in range(world)]
    ctxs = [F.create_ag_gemm_fp8_context(world * mpr + 64, K, r, world, device=cuda_device, heap=lw.heap(r)) for r in range(world)]
    full = torch.cat([F.dequantize_fp8(o[0], o[1], 1) for o in ops])
    mt, kb = (mpr + 127) // 128, K // 128
    for r in range(world):
        ctx = ctxs[r]
        a, sa, b, sb = ops[r]
        if world > 1:
            half = (ctx.epoch + 1) & 1
            ws = ctx.workspace.local[half][: world * mpr * K].view(world, mpr, K)
            sws = ctx.scale_ws.local[half][: world * mpr * kb].view(world, mpr, kb)
            flags = ctx.flags.local[half][: world * mt].view(world, mt)
            for s in range(r + 1, world):
                ws[s].copy_(ops[s][0].view(torch.uint8))
                sws[s].copy_(ops[s][1])
                flags[s].fill_(ctx.epoch + 1)
            ws[r].fill_(0x7F)          # e4m3 NaN: the own slot is never read from the workspace
            sws[r].fill_(float("nan"))
        c = F.ag_gemm_fp8(a, sa, b, sb, ctx)
        check_status()
        ref = full @ F.dequantize_fp8(b, sb, 128).t()
        assert torch.isfinite(c).all()
        torch.testing.assert_close(c.float(), ref, atol=2e-2 * ref.abs().max().item() / 4, rtol=1e-2)
    for r in range(world):
        if world == 1:
            break
        ws = ctxs[r].workspace.local[1][: world * mpr * K].view(world, mpr, K)
        sws = ctxs[r].scale_ws.local[1][: world * mpr * kb].view(world, mpr, kb)
        for s in range(world):
            if s != r:
                assert torch.equal(ws[s], ops[s][0].view(torch.uint8)), f"rank {r} rows of {s}"
                assert torch.equal(sws[s], ops[s][1]), f"rank {r} scales of {s}"


@pytest.mark.parametrize("N,K", [(8, 128), (264, 384), (1000, 896), (4096, 8192), (520, 16384)])
def test_few_row_fp8_gemm_matches_fp32_reference(cuda_device, N, K):
    """The automatic choice at few rows: one or two groups of folding warps, token and weight-row remainders, one to eight
    CTAs per cluster. Tolerance: half an ulp of bf16 and fp32 sums (1e-5 of the terms' spread)."""
    b = sb = None
    for M in (1, 5, 16, 17, 31, 63, 64, 65, 100, 127, 128, 129, 200, 256):
        a, sa, bn, sbn = _operands(M, N, K, cuda_device, M)
        if b is None:
            b, sb = bn, sbn
        guard = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=cuda_device)
        c = F.gemm_fp8_blockscaled(a, sa, b, sb, out=guard[:M])
        check_status()
        ref = F.dequantize_fp8(a, sa, 1).double() @ F.dequantize_fp8(b, sb, 128).double().t()
        torch.testing.assert_close(c.double(), ref, rtol=2.0 ** -8, atol=1e-5 * ref.abs().max().item())
        assert (guard[M] == 7.0).all()
        again = F.gemm_fp8_blockscaled(a, sa, b, sb, num_sms=148)   # the large tiles
        torch.testing.assert_close(again.double(), ref, rtol=2.0 ** -8, atol=1e-5 * ref.abs().max().item())


@pytest.mark.parametrize("M,N,K", [(128, 512, 256), (300, 1000, 4096)])
def test_fp8_pipeline_stays_whole_when_a_flag_wait_is_abandoned(cuda_device, monkeypatch, M, N, K):
    """As for the bf16 product: the kernel runs to its end in step and reports the flag and its peer."""
    monkeypatch.setenv("TDIST_WAIT_TIMEOUT_MS", "50")
    from triton_distributed_b200.runtime import global_status
    a, sa, b, sb = _operands(M, N, K, cuda_device, M)
    ref = F.dequantize_fp8(a, sa, 1).float() @ F.dequantize_fp8(b, sb, 128).float().t()
    lw = LocalWorld(2, cuda_device)
    ctxs = [F.create_ag_gemm_fp8_context(2 * M, K, r, 2, heap=lw.heap(r)) for r in range(2)]
    for _ in range(3):
        out = F.ag_gemm_fp8(a, sa, b, sb, ctxs[0])
        torch.cuda.synchronize()
        rec = global_status().record
        assert (rec.abort_flag, rec.code, rec.peer) == (1, 1, 1)
        torch.testing.assert_close(out[:M].float(), ref, atol=3e-2, rtol=2e-2)
        with pytest.raises(Exception, match="timed out"):
            check_status()

"""tcgen05 GEMM family on one GPU: plain GEMM numerics, and the fused AG / RS kernels of one
emulated rank at a time against peer buffers prepared by the host (LocalWorld).

Oracle: plain PyTorch fp32 matmul of the same operands. Mirrors the reference's
test_ag_gemm_intra_node.py / test_gemm_rs.py checks (non-tile-aligned M, stale workspace poisoning)
without needing several GPUs.
"""
import pytest
import torch

from triton_distributed_b200 import _lib
from triton_distributed_b200.ops import gemm as G
from triton_distributed_b200.runtime import LocalWorld, check_status, global_status

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1, 2], ids=["cta1", "cta_pair", "cta_pair_wide"])
def tiling(request, monkeypatch):
    """Run a test under every tiling of the kernel (one CTA per 128x256 tile, CTA pair per 256x256 tile, CTA pair
    per 256x512 tile)."""
    monkeypatch.setattr(G, "CTA_PAIR", request.param)
    return request.param


def _rand(shape, dtype, dev, scale=1.0):
    return (torch.randn(shape, device=dev, dtype=torch.float32) * scale).to(dtype)


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 512), (300, 264, 136), (1000, 1000, 992), (4096, 768, 2048),
                                   (520, 1288, 200), (8192, 1536, 1024), (2304, 5128, 320)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_plain_gemm_matches_fp32_reference(cuda_device, tiling, M, N, K, dtype):
    torch.manual_seed(M + N + K)
    a = _rand((M, K), dtype, cuda_device)
    b = _rand((N, K), dtype, cuda_device, K ** -0.5)
    c = G.gemm_persistent(a, b)
    check_status()
    ref = a.float() @ b.float().t()
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert torch.isfinite(c).all()
    torch.testing.assert_close(c.float(), ref, atol=tol, rtol=tol)


@pytest.mark.parametrize("world,mpr,N,K", [(2, 128, 256, 128), (4, 250, 520, 264), (8, 96, 256, 512), (4, 999, 768, 1024),
                                           (2, 520, 1288, 192), (4, 384, 1224, 128), (2, 130, 2048 + 64, 256)])
def test_ag_gemm_single_rank_kernels_against_prepared_peers(cuda_device, tiling, world, mpr, N, K):
    """Each emulated rank's fused kernel runs alone: blocks of lower ranks were really pushed by
    their kernels, blocks of higher ranks are written by the host together with their flags."""
    torch.manual_seed(world * 1000 + mpr)
    dtype = torch.bfloat16
    lw = LocalWorld(world, cuda_device)
    A = [_rand((mpr, K), dtype, cuda_device) for _ in range(world)]
    B = [_rand((N, K), dtype, cuda_device, K ** -0.5) for _ in range(world)]
    ctxs = [G.create_ag_gemm_intra_node_context(A[r], B[r], r, world, max_M=world * mpr + 64, heap=lw.heap(r))
            for r in range(world)]
    full = torch.cat(A).float()
    mt = (mpr + 127) // 128
    for r in range(world):
        ctx = ctxs[r]
        half = (ctx.epoch + 1) & 1
        ws = ctx.workspace.local[half][: world * mpr * K].view(world, mpr, K)
        flags = ctx.flags.local[half][: world * mt].view(world, mt)
        # poison what no kernel has written yet, then stand in for the ranks that have not run
        for s in range(r + 1, world):
            ws[s].copy_(A[s])
            flags[s].fill_(ctx.epoch + 1)
        ws[r].fill_(float("nan"))  # own slot is never read from the workspace
        c = G.ag_gemm_intra_node(A[r], B[r], ctx)
        check_status()
        ref = full @ B[r].float().t()
        torch.testing.assert_close(c.float(), ref, atol=2e-2, rtol=2e-2)
    # every rank's shard was pushed to every other rank, with its flags
    for r in range(world):
        ws = ctxs[r].workspace.local[1][: world * mpr * K].view(world, mpr, K)
        flags = ctxs[r].flags.local[1][: world * mt].view(world, mt)
        for s in range(world):
            if s == r:
                continue
            assert torch.equal(ws[s], A[s]), f"rank {r} workspace slot {s}"
            assert (flags[s] == 1).all()


@pytest.mark.parametrize("world,mpr,N,K", [(2, 128, 256, 128), (4, 250, 520, 264), (8, 96, 512, 256), (4, 512, 1024, 512),
                                           (2, 520, 1288, 192), (4, 300, 1224, 128), (2, 130, 2048 + 64, 256)])
def test_gemm_rs_single_rank_kernels_against_prepared_peers(cuda_device, tiling, world, mpr, N, K):
    torch.manual_seed(world * 77 + mpr)
    dtype = torch.bfloat16
    lw = LocalWorld(world, cuda_device)
    M = world * mpr
    A = [_rand((M, K), dtype, cuda_device) for _ in range(world)]
    B = [_rand((N, K), dtype, cuda_device, (K * world) ** -0.5) for _ in range(world)]
    partial = [(A[s].float() @ B[s].float().t()) for s in range(world)]
    total = sum(partial)
    ctxs = [G.create_gemm_rs_context(M + 8, N, r, world, heap=lw.heap(r), device=cuda_device) for r in range(world)]
    tiles = ((mpr + 127) // 128) * ((N + 255) // 256)
    for r in range(world):
        ctx = ctxs[r]
        half = (ctx.epoch + 1) & 1
        stage = ctx.staging.local[half][: world * mpr * N].view(world, mpr, N)
        flags = ctx.flags.local[half][: tiles * world].view(tiles, world)
        for s in range(r + 1, world):
            stage[s].copy_(partial[s][r * mpr:(r + 1) * mpr].to(dtype))
            flags[:, s].fill_(ctx.epoch + 1)
        out = G.gemm_rs(A[r], B[r], ctx)
        check_status()
        ref = total[r * mpr:(r + 1) * mpr]
        torch.testing.assert_close(out.float(), ref, atol=3e-2, rtol=3e-2)


def test_abandoned_wait_reports_timeout_and_leaves_the_context_usable(cuda_device, monkeypatch):
    """A flag that nothing sets: the kernel must give up after its limit, report which flag it was
    waiting for, and return, and the next launch must work."""
    monkeypatch.setenv("TDIST_WAIT_TIMEOUT_MS", "50")
    dtype = torch.bfloat16
    lw = LocalWorld(2, cuda_device)
    a = _rand((128, 128), dtype, cuda_device)
    b = _rand((256, 128), dtype, cuda_device)
    ctx = G.create_ag_gemm_intra_node_context(a, b, 0, 2, max_M=256, heap=lw.heap(0))
    G.create_ag_gemm_intra_node_context(a, b, 1, 2, max_M=256, heap=lw.heap(1))
    G.ag_gemm_intra_node(a, b, ctx)
    torch.cuda.synchronize()
    st = global_status()
    assert st.aborted()
    rec = st.record
    assert rec.code == 1 and rec.peer == 1 and rec.expected == 1
    with pytest.raises(_lib.TdistTimeoutError):
        check_status()
    # the context is still usable
    c = G.gemm_persistent(a, b)
    check_status()
    torch.testing.assert_close(c.float(), a.float() @ b.float().t(), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("kind", ["ag", "rs"])
@pytest.mark.parametrize("tiling", [0, 1, 2])
@pytest.mark.parametrize("mpr,N,K", [(128, 512, 128), (300, 1032, 4104)])
def test_pipeline_stays_whole_when_a_flag_wait_is_abandoned(cuda_device, monkeypatch, kind, tiling, mpr, N, K):
    """K within and well beyond the stages of the pipeline: after the flag wait gives up the copies, MMAs and epilogue run to
    the end in step, the report names the flag and its peer and not a barrier behind it, and a product launched before anybody has
    read the report is right."""
    monkeypatch.setenv("TDIST_WAIT_TIMEOUT_MS", "50")
    torch.manual_seed(tiling)
    dtype, world = torch.bfloat16, 2
    lw = LocalWorld(world, cuda_device)
    b = _rand((N, K), dtype, cuda_device, K ** -0.5)
    for _ in range(3):
        if kind == "ag":
            a = _rand((mpr, K), dtype, cuda_device)
            ctxs = [G.create_ag_gemm_intra_node_context(a, b, r, world, max_M=world * mpr, heap=lw.heap(r)) for r in range(world)]
            ctxs[0].cta_pair = tiling
            out = G.ag_gemm_intra_node(a, b, ctxs[0])
            own = a
        else:
            a = _rand((world * mpr, K), dtype, cuda_device)
            ctxs = [G.create_gemm_rs_context(world * mpr, N, r, world, heap=lw.heap(r)) for r in range(world)]
            ctxs[0].cta_pair = tiling
            G.gemm_rs(a, b, ctxs[0])
            own = a[:mpr]
        after = G.gemm_persistent(own, b, num_sms=148)
        torch.cuda.synchronize()
        rec = global_status().record
        assert (rec.abort_flag, rec.code, rec.peer) == (1, 1, 1)
        ref = own.float() @ b.float().t()
        if kind == "ag":   # this rank's own rows do not depend on the missing ones
            torch.testing.assert_close(out[:mpr].float(), ref, atol=2e-2, rtol=2e-2)
        torch.testing.assert_close(after.float(), ref, atol=2e-2, rtol=2e-2)
        with pytest.raises(_lib.TdistTimeoutError):
            check_status()


def test_consumer_blocks_until_the_host_sets_the_flags(cuda_device):
    """The fused AG-GEMM of one emulated rank is launched while the peer's rows are in the workspace but their flags
    are not set; the host sets them a moment later with stream write-values (no kernel involved). The kernel must
    wait, then finish with the right result (the reference's test_distributed_wait.py `correctness` case)."""
    import time

    from triton_distributed_b200.ops import collectives as CO

    torch.manual_seed(5)
    dtype = torch.bfloat16
    world, mpr, N, K = 2, 256, 512, 256
    lw = LocalWorld(world, cuda_device)
    A = [_rand((mpr, K), dtype, cuda_device) for _ in range(world)]
    B = _rand((N, K), dtype, cuda_device, K ** -0.5)
    ctxs = [G.create_ag_gemm_intra_node_context(A[r], B, r, world, max_M=world * mpr, heap=lw.heap(r)) for r in range(world)]
    ctx = ctxs[0]
    half = (ctx.epoch + 1) & 1
    mt = (mpr + 127) // 128
    ws = ctx.workspace.local[half][: world * mpr * K].view(world, mpr, K)
    flags = ctx.flags.local[half][: world * mt].view(world, mt)
    ws[1].copy_(A[1])
    assert int(flags[1].abs().sum()) == 0          # nothing has announced rank 1's blocks
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    t0 = time.time()
    c = G.ag_gemm_intra_node(A[0], B, ctx)         # asynchronous: the kernel now spins on rank 1's flags
    time.sleep(0.3)
    for b in range(mt):
        CO.set_signal(flags[1, b:b + 1].data_ptr(), ctx.epoch, stream=side)
    torch.cuda.synchronize()
    took = time.time() - t0
    check_status()
    assert took >= 0.3                               # it really waited for the host
    ref = torch.cat(A).float() @ B.float().t()
    torch.testing.assert_close(c.float(), ref, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("N,K", [(264, 128), (320, 192), (456, 64), (1288, 128)])
def test_partial_column_tiles_over_many_fresh_inputs(cuda_device, tiling, N, K):
    """Column counts whose last 256-column tile holds 8, 64, 200 and 8 (after two and a half wide tiles) columns,
    row counts that are no multiple of 128 or 256, 20 iterations with fresh data: a stale or misplaced partial
    tile shows up as a wrong element in some iteration."""
    dtype = torch.bfloat16
    gen = torch.Generator(device=cuda_device).manual_seed(N * 7 + K)
    for it in range(20):
        M = int(torch.randint(1, 700, (1,), generator=gen, device=cuda_device))
        a = torch.randn(M, K, device=cuda_device, generator=gen).to(dtype)
        b = (torch.randn(N, K, device=cuda_device, generator=gen) * K ** -0.5).to(dtype)
        c = torch.full((M, N), float("nan"), device=cuda_device, dtype=dtype)
        G.gemm_persistent(a, b, out=c)
        check_status()
        torch.testing.assert_close(c.float(), a.float() @ b.float().t(), atol=2e-2, rtol=2e-2, msg=lambda m: f"iteration {it}, M={M}: {m}")


@pytest.mark.parametrize("world", [2, 4])
def test_gemm_rs_random_m_sweep(cuda_device, tiling, world):
    """Seeded sweep over random M (any multiple of the world size up to the context's limit), one context reused
    across the calls as in serving (the reference's test_gemm_rs.py:209-231 draws M the same way)."""
    dtype = torch.bfloat16
    N, K, max_mpr = 776, 192, 300
    gen = torch.Generator(device=cuda_device).manual_seed(world)
    lw = LocalWorld(world, cuda_device)
    ctxs = [G.create_gemm_rs_context(world * max_mpr, N, r, world, heap=lw.heap(r), device=cuda_device) for r in range(world)]
    for it in range(12):
        mpr = int(torch.randint(1, max_mpr + 1, (1,), generator=gen, device=cuda_device))
        M = world * mpr
        A = [torch.randn(M, K, device=cuda_device, generator=gen).to(dtype) for _ in range(world)]
        B = [(torch.randn(N, K, device=cuda_device, generator=gen) * (K * world) ** -0.5).to(dtype) for _ in range(world)]
        partial = [(A[s].float() @ B[s].float().t()) for s in range(world)]
        total = sum(partial)
        tiles = ((mpr + 127) // 128) * ((N + 255) // 256)
        for r in range(world):
            ctx = ctxs[r]
            half = (ctx.epoch + 1) & 1
            stage = ctx.staging.local[half][: world * mpr * N].view(world, mpr, N)
            flags = ctx.flags.local[half][: tiles * world].view(tiles, world)
            for s in range(r + 1, world):
                stage[s].copy_(partial[s][r * mpr:(r + 1) * mpr].to(dtype))
                flags[:, s].fill_(ctx.epoch + 1)
            out = G.gemm_rs(A[r], B[r], ctx)
            check_status()
            torch.testing.assert_close(out.float(), total[r * mpr:(r + 1) * mpr], atol=3e-2, rtol=3e-2,
                                       msg=lambda m: f"iteration {it}, mpr={mpr}, rank {r}: {m}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 72), (256, 4096), (1288, 8192 + 8), (6144, 1536), (20480, 256)])
def test_few_row_gemm_matches_fp32_reference(cuda_device, N, K, dtype):
    """The automatic choice at few rows: every token-tile width (1 row to 4 x 128 with remainders), N and K off the tile
    edges, one to eight CTAs per cluster. Tolerance: the 16-bit rounding of the result (half an ulp) and fp32 sums of K
    products of unit-variance terms, whose order changes nothing above 1e-5."""
    import ctypes as C
    torch.manual_seed(N + K)
    b = _rand((N, K), dtype, cuda_device, K ** -0.5)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    few = 0
    for M in (1, 2, 15, 16, 17, 31, 48, 64, 65, 100, 127, 128, 129, 255, 257, 385, 500, 512):
        a = _rand((M, K), dtype, cuda_device)
        guard = torch.full((M + 1, N), 7.0, dtype=dtype, device=cuda_device)
        c = G.gemm_persistent(a, b, out=guard[:M])
        check_status()
        torch.testing.assert_close(c.float(), a.float() @ b.float().t(), atol=eps / 16, rtol=eps)
        assert (guard[M] == 7.0).all()   # nothing written past the last row
        g = G._base_args(a, b, 1, 0, _lib.GEMM_PLAIN)
        g.c, g.m_per_rank = c.data_ptr(), M
        out = (C.c_int * 4)()
        assert _lib.lib().tdist_gemm_plan(C.byref(g), out) == 0
        few += out[0] == 1 and out[3] % (-(-N // 128)) == 0
    assert few >= 8 or K < 1024   # the few-row kernel did run (with so short a K the large tiles are as good)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("activation", ["gelu", "silu", "relu"])
@pytest.mark.parametrize("M,N,K", [(5, 264, 136), (100, 520, 4096), (300, 264, 136), (128, 1288, 8192)])
def test_epilogue_activation_matches_fp32_reference(cuda_device, M, N, K, activation, dtype):
    """Few-row and one-CTA kernels, and the pass of its own above 128 rows (two roundings there). Pre-activations reach +-40, far into both tails. Tolerance: the 16-bit
    rounding of the result, and for gelu / silu fp32 sums whose error (1e-5 of their spread) the activation passes on."""
    torch.manual_seed(M + N)
    a, b = _rand((M, K), dtype, cuda_device, 8.0), _rand((N, K), dtype, cuda_device, K ** -0.5)
    ctx = G.create_ag_gemm_intra_node_context(a, b, 0, 1, max_M=M)
    h = a.double() @ b.double().t()
    ref = {"gelu": lambda v: torch.nn.functional.gelu(v, approximate="tanh"), "silu": torch.nn.functional.silu,
           "relu": torch.nn.functional.relu}[activation](h)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for pair in (-1, 0, 1):
        ctx.cta_pair = pair
        out = G.ag_gemm_intra_node(a, b, ctx, activation=activation)
        check_status()
        torch.testing.assert_close(out.double(), ref, atol=2e-4 if M <= 128 and pair <= 0 else 40 * eps, rtol=2 * eps)


def test_activation_of_a_nan_is_a_nan(cuda_device):
    a = torch.ones(4, 64, dtype=torch.bfloat16, device=cuda_device)
    a[1, 3] = float("nan")
    b = torch.ones(8, 64, dtype=torch.bfloat16, device=cuda_device)
    ctx = G.create_ag_gemm_intra_node_context(a, b, 0, 1, max_M=4)
    for activation in ("gelu", "silu", "relu"):
        out = G.ag_gemm_intra_node(a, b, ctx, activation=activation)
        assert out[1].isnan().all() and not out[[0, 2, 3]].isnan().any()


def _tile_width(M, N, K):
    g = _lib.GemmArgs()
    g.mode, g.world, g.rank, g.m_per_rank, g.n, g.k, g.cta_pair, g.c = _lib.GEMM_PLAIN, 1, 0, M, N, K, -1, 16
    return _lib.lib().tdist_gemm_tile_width(g)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1000, 5504, 4096), (999, 5496, 4104), (520, 2048, 512), (600, 2056, 520), (512, 6144, 12288), (777, 1928, 5000)])
def test_automatic_tile_width_matches_fp32_reference(cuda_device, M, N, K, dtype):
    """Narrow and wide pair tiles of fewer than 256 columns, with remainders in M, N and K. Tolerance: half an ulp of
    the 16-bit result, and K / 16 accumulation steps on partial sums below 3, each off by less than 2^-23 of them."""
    torch.manual_seed(M + N)
    a, b = _rand((M, K), dtype, cuda_device), _rand((N, K), dtype, cuda_device, K ** -0.5)
    guard = torch.full((M + 1, N), 7.0, dtype=dtype, device=cuda_device)
    c = G.gemm_persistent(a, b, out=guard[:M])
    check_status()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    torch.testing.assert_close(c.double(), a.double() @ b.double().t(), atol=eps / 16 + 3 * K / 16 * 2.0 ** -23, rtol=eps)
    assert (guard[M] == 7.0).all()


def test_narrower_tiles_only_where_a_round_is_nearly_empty(cuda_device):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("calibrated for 148 SMs")
    assert _tile_width(8192, 49152, 12288) == 256       # many rounds
    assert _tile_width(1000, 5504, 4096) == 192         # 44 wide tiles of 2 x 256 on 74 pairs, or 60 of 2 x 192
    assert _tile_width(16, 6144, 12288) == 0            # few rows


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N", [(129, 8), (200, 1032), (1000, 4104)])
@pytest.mark.parametrize("activation", ["gelu", "silu", "relu"])
def test_activation_in_place_behind_the_large_tiles(cuda_device, M, N, activation, dtype):
    """Above 128 rows the result is rounded, then activated in place: the values of torch's pass over the same result up
    to an ulp, into `out` as well, and nothing past it."""
    torch.manual_seed(M + N)
    K = 264
    a, b = _rand((M, K), dtype, cuda_device, 8.0), _rand((N, K), dtype, cuda_device, K ** -0.5)
    ctx = G.create_ag_gemm_intra_node_context(a, b, 0, 1, max_M=M)
    ref = G.apply_activation(G.ag_gemm_intra_node(a, b, ctx), activation)
    guard = torch.full((M + 1, N), 7.0, dtype=dtype, device=cuda_device)
    out = G.ag_gemm_intra_node(a, b, ctx, out=guard[:M], activation=activation)
    check_status()
    assert out.data_ptr() == guard.data_ptr() and (guard[M] == 7.0).all()
    eps = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    torch.testing.assert_close(out.float(), ref.float(), atol=1e-6, rtol=eps)


@pytest.mark.parametrize("M", [64, 256])
def test_an_unknown_activation_launches_nothing(cuda_device, M):
    a, b = _rand((M, 64), torch.bfloat16, cuda_device), _rand((8, 64), torch.bfloat16, cuda_device)
    ctx = G.create_ag_gemm_intra_node_context(a, b, 0, 1, max_M=M)
    out = torch.full((M, 8), 7.0, dtype=torch.bfloat16, device=cuda_device)
    with pytest.raises(ValueError, match="unknown activation"):
        G.ag_gemm_intra_node(a, b, ctx, out=out, activation="typo")
    torch.cuda.synchronize()
    assert ctx.epoch == 0 and (out == 7.0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("activation", ["gelu", "silu", "relu"])
def test_activation_of_every_16_bit_value(cuda_device, activation, dtype):
    """The in-place kernel over all 65536 values against float64, tails included. Allowed: the rounding of the result (half a
    quantum where it is subnormal), (5 + 3.2 |z|) 2^-23 of it for z, __expf and the fast division, and 1.1e-36 where the divisor
    leaves that division's range."""
    bits = torch.arange(65536, dtype=torch.int32, device=cuda_device).to(torch.int16)
    v = bits.view(dtype)
    h = v.clone()
    lib = _lib.lib()
    _lib.check(lib.tdist_activate(h.data_ptr(), h.numel(), G._DTYPES[dtype], _lib.ACTIVATIONS[activation], torch.cuda.current_stream().cuda_stream), "tdist_activate")
    torch.cuda.synchronize()
    x = v.double()
    z = {"gelu": 1.5957691216057308 * x * (1 + 0.044715 * x * x), "silu": x, "relu": torch.zeros_like(x)}[activation]
    ref = x.clamp_min(0) if activation == "relu" else x / (1 + torch.exp(-z))
    ok = torch.isfinite(x)
    rounding, half_quantum = (2.0 ** -8, 2.0 ** -134) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -25)
    allowed = ref.abs() * (rounding + (5 + 3.2 * z.abs().clamp_max(200)) * 2.0 ** -23) * (1 + rounding) + half_quantum
    allowed = allowed + (1.1e-36 if activation != "relu" else 0.0)
    err = (h.double() - ref).abs()
    worst = (err / allowed)[ok].max().item()
    assert worst <= 1.0, (worst, v[ok][(err / allowed)[ok].argmax()].item())
    edge = lambda t: h[(v == t).nonzero().flatten()]  # noqa: E731
    assert h[torch.isnan(v)].isnan().all() and (edge(float("inf")) == float("inf")).all()
    assert (edge(-float("inf")) == 0).all() if activation == "relu" else edge(-float("inf")).isnan().all()   # as torch

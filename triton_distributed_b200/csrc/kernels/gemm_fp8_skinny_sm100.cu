// Few-row block-scaled fp8 GEMM for sm_100a: the product of gemm_fp8_sm100.cu for a decode step's or a short prompt's
// worth of tokens.
//
//   C[m, n] = sum over 128-wide K blocks kb of  SA[m, kb] * SB[n / 128, kb] * (A_kb[m, :] . B_kb[n, :])
//
// Bound by reading B (the weights) once from HBM, and cut up as gemm_skinny_sm100.cu does it: 128 weight rows are the M
// operand of tcgen05.mma (kind::f8f6f4), up to 128 tokens its N operand, and the K ranges of a tile form a cluster whose
// CTAs add their fp32 partial sums through shared memory. (128 x 256 tiles over all of K: m16 n4096 k8192 as 16 CTAs
// 37.3 us, 12.3 us here; m64 39.6 and 17.1 us; m16 n16384 k4096 22.8 and 17.0 us.) 128 weight rows are one row of scale blocks, so SB is one number per K block and
// CTA, and SA one per token.
//
// Every K block goes to a fresh TMEM accumulator and is folded into fp32 registers with its scale, one thread per weight
// row, 64 tokens per thread at most. The accumulators are at most 128 columns wide here, so TMEM holds four of them (two
// above 64 tokens) and the hand-over between the MMA issuer and the folding warps stays ahead of the loads.
//
// Warps: 0 = TMA producer, 1 = MMA issuer and TMEM owner, 2..5 = folding and exchange of tokens 0..63, 6..9 = of tokens
// 64..127 (launched only where there are any).
#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>

#include "../device/ptx.cuh"
#include "../device/signal.cuh"
#include "../include/tdist.h"
#include "../runtime/host_common.h"
#include "gemm_skinny.h"

namespace tdist {
namespace fp8_skinny {

constexpr int ROWS = 128;            // weight rows per CTA (UMMA M)
constexpr int MAX_TOK = 128;         // tokens per CTA (UMMA N)
constexpr int TOK = 64;              // tokens a thread accumulates
constexpr int BK = 128, UMMA_K = 32; // bytes = elements
constexpr int W_BYTES = ROWS * BK;
constexpr int MAX_STAGES = 6, MAX_SPLIT = 8, MAX_BUFS = 4;
constexpr int MAX_THREADS = 64 + 2 * 128;
constexpr int STAGE_AREA = 104 * 1024;
constexpr int SCALE_BYTES = 8 * TOK * 4;   // every folding warp's scales of the K block it is at
constexpr int SMEM_BYTES = STAGE_AREA + SCALE_BYTES + 1024 + 256;
static_assert((MAX_TOK + MAX_SPLIT) * ROWS * 4 <= STAGE_AREA, "the partial sums reuse the stages");

constexpr int kKernelGemmFp8 = 7;

struct Params {
    CUtensorMap tm_w;   // {K, N}, box {128, 128}
    CUtensorMap tm_x;   // {K, M}, box {128, tok}
    const float* sa;    // [M, kb_total]
    const float* sb;    // [ceil(N / 128), kb_total]
    void* out;          // [M, N] bf16
    int m, n, kb_total, tok, m_tiles, split, stages, bufs, buf_cols, tmem_cols;
    WaitCtx wctx;
};

__global__ void __launch_bounds__(MAX_THREADS, 1) gemm_fp8_skinny_kernel(const __grid_constant__ Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* scales = reinterpret_cast<float*>(smem + STAGE_AREA);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGE_AREA + SCALE_BYTES);   // full, empty [S each]; accumulator full, empty
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 2 * MAX_BUFS);
    const int warp = static_cast<int>(threadIdx.x) >> 5;
    const int lane = static_cast<int>(threadIdx.x) & 31;
    const int fold_warps = static_cast<int>(blockDim.x) / 32 - 2;
    const uint32_t bars_u32 = smem_u32(bars);
    auto bar_full = [&](uint32_t s) { return bars_u32 + 8u * s; };
    auto bar_empty = [&](uint32_t s) { return bars_u32 + 8u * (MAX_STAGES + s); };
    auto bar_tfull = [&](uint32_t b) { return bars_u32 + 8u * (2 * MAX_STAGES + b); };
    auto bar_tempty = [&](uint32_t b) { return bars_u32 + 8u * (2 * MAX_STAGES + MAX_BUFS + b); };

    const int tile = static_cast<int>(blockIdx.x) / p.split;
    const int part = static_cast<int>(blockIdx.x) - tile * p.split;   // = rank in the cluster
    const int m0 = (tile % p.m_tiles) * p.tok;
    const int n0 = (tile / p.m_tiles) * ROWS;
    const int kb0 = static_cast<int>(static_cast<long long>(p.kb_total) * part / p.split);
    const int kb1 = static_cast<int>(static_cast<long long>(p.kb_total) * (part + 1) / p.split);
    const uint32_t stage_bytes = W_BYTES + static_cast<uint32_t>(p.tok) * BK;
    const uint32_t stages = static_cast<uint32_t>(p.stages), bufs = static_cast<uint32_t>(p.bufs);

    if (threadIdx.x == 0) {
        prefetch_tensormap(&p.tm_w);
        prefetch_tensormap(&p.tm_x);
        for (uint32_t s = 0; s < stages; ++s) {
            mbar_init(bar_full(s), 1);
            mbar_init(bar_empty(s), 1);
        }
        for (uint32_t b = 0; b < bufs; ++b) {
            mbar_init(bar_tfull(b), 1);
            mbar_init(bar_tempty(b), static_cast<uint32_t>(fold_warps));
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc<1>(smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
        tmem_relinquish<1>();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    pdl_wait_and_release();

    unsigned long long acc[TOK / 2];   // folding warps: this thread's weight row x 64 tokens, as pairs of fp32
#pragma unroll
    for (int i = 0; i < TOK / 2; ++i) acc[i] = 0ull;
    const int group = (warp - 2) >> 2;                       // folding warps: which 64 tokens
    const int q = warp & 3;                                  // TMEM lane quadrant this warp may read
    const int cols = min(TOK, p.tok - group * TOK);          // a multiple of 16

    if (warp == 0) {
        if (lane == 0) {
            uint32_t s = 0, phase = 1;
            for (int kb = kb0; kb < kb1; ++kb) {
                mbar_wait(bar_empty(s), phase, p.wctx, 2);
                const uint32_t dst = smem_u32(smem) + s * stage_bytes;
                mbar_expect_tx(bar_full(s), stage_bytes);
                tma_load_2d(dst, &p.tm_w, bar_full(s), kb * BK, n0);
                tma_load_2d(dst + W_BYTES, &p.tm_x, bar_full(s), kb * BK, m0);
                if (++s == stages) {
                    s = 0;
                    phase ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc(0u, 0u, ROWS, static_cast<uint32_t>(p.tok));   // e4m3 x e4m3 -> f32
            uint32_t s = 0, phase = 0, b = 0, bphase = 1;
            for (int kb = kb0; kb < kb1; ++kb) {
                mbar_wait(bar_tempty(b), bphase, p.wctx, 3);
                mbar_wait(bar_full(s), phase, p.wctx, 4);
                tc_fence_after();
                const uint32_t src = smem_u32(smem) + s * stage_bytes;
                const uint64_t wdesc = umma_desc_k_sw128(src);
                const uint64_t xdesc = umma_desc_k_sw128(src + W_BYTES);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k)
                    umma_fp8<1>(tmem_base + b * static_cast<uint32_t>(p.buf_cols), wdesc + 2 * k, xdesc + 2 * k, idesc, k != 0 ? 1u : 0u);
                umma_commit(bar_empty(s));
                umma_commit(bar_tfull(b));
                if (++s == stages) {
                    s = 0;
                    phase ^= 1u;
                }
                if (++b == bufs) {
                    b = 0;
                    bphase ^= 1u;
                }
            }
        }
        __syncwarp();
    } else {
        // ---- folding: acc += (K block's sums) * (SA of the token x SB)
        float* my_scales = scales + (warp - 2) * TOK;
        const float* sb_row = p.sb + static_cast<size_t>(n0 / ROWS) * p.kb_total;
        // lane t keeps the scales of tokens t and t + 32 of its group; rows past the end repeat the last one, unused
        const float* sa0 = p.sa + static_cast<size_t>(min(m0 + group * TOK + lane, p.m - 1)) * p.kb_total;
        const float* sa1 = p.sa + static_cast<size_t>(min(m0 + group * TOK + 32 + lane, p.m - 1)) * p.kb_total;
        float next0 = sa0[kb0] * sb_row[kb0], next1 = sa1[kb0] * sb_row[kb0];
        uint32_t b = 0, bphase = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            my_scales[lane] = next0;
            my_scales[lane + 32] = next1;
            if (kb + 1 < kb1) {
                next0 = sa0[kb + 1] * sb_row[kb + 1];
                next1 = sa1[kb + 1] * sb_row[kb + 1];
            }
            __syncwarp();
            mbar_wait(bar_tfull(b), bphase, p.wctx, 5);
            tc_fence_after();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + b * static_cast<uint32_t>(p.buf_cols) + group * TOK;
#pragma unroll
            for (int c = 0; c < TOK; c += 16) {
                if (c >= cols) break;
                uint32_t r[16];
                tmem_ld_32x16(taddr + c, r);
                tmem_ld_wait();
                if (c + 16 >= cols) {
                    // all of the accumulator is in registers: hand it back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_tempty(b));
                }
                const ulonglong2* sc = reinterpret_cast<const ulonglong2*>(my_scales + c);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const ulonglong2 s2 = sc[i];   // the same address in every lane
                    unsigned long long v;
                    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(r[4 * i]), "r"(r[4 * i + 1]));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[c / 2 + 2 * i]) : "l"(v), "l"(s2.x));
                    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(r[4 * i + 2]), "r"(r[4 * i + 3]));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[c / 2 + 2 * i + 1]) : "l"(v), "l"(s2.y));
                }
            }
            __syncwarp();   // every lane has read the scales
            if (++b == bufs) {
                b = 0;
                bphase ^= 1u;
            }
        }
    }

    // ---- exchange, as in gemm_skinny_sm100.cu: [source part][token of the share][weight row] fp32 in every CTA. The folding
    // warps have seen every accumulator of this CTA, so its MMAs and loads are complete and the stages may be overwritten.
    cluster_arrive();
    cluster_wait();
    const int live = min(p.tok, p.m - m0);
    const int per = (p.tok + p.split - 1) / p.split;
    float* sums = reinterpret_cast<float*>(smem);
    if (warp >= 2) {
        const uint32_t mine = smem_u32(sums) + static_cast<uint32_t>((part * per * ROWS + q * 32 + lane) * 4);
        int owner = (group * TOK) / per, j = group * TOK - owner * per;
        uint32_t dst = mapa_u32(mine, static_cast<uint32_t>(min(owner, p.split - 1)));
#pragma unroll
        for (int c = 0; c < TOK; ++c) {
            if (c < cols) {
                const unsigned long long a2 = acc[c / 2];
                st_shared_cluster_f32(dst + static_cast<uint32_t>(j) * (ROWS * 4), __uint_as_float(static_cast<uint32_t>(c & 1 ? a2 >> 32 : a2)));
                if (++j == per) {
                    j = 0;
                    ++owner;
                    dst = mapa_u32(mine, static_cast<uint32_t>(min(owner, p.split - 1)));
                }
            }
        }
    }
    tc_fence_before();
    cluster_arrive();
    cluster_wait();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<1>(tmem_base, static_cast<uint32_t>(p.tmem_cols));
    }
    const int t0 = part * per;
    const int items = min(per, live - t0) * (ROWS / 4);   // 4 columns of a token each; this CTA's share may be empty
    for (int i = static_cast<int>(threadIdx.x); i < items; i += static_cast<int>(blockDim.x)) {
        const int t = i / (ROWS / 4), c = (i % (ROWS / 4)) * 4;
        if (n0 + c >= p.n) continue;   // N is a multiple of 8: all four columns or none
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int s = 0; s < p.split; ++s) {
            const float4 u = *reinterpret_cast<const float4*>(sums + (s * per + t) * ROWS + c);
            v.x += u.x;
            v.y += u.y;
            v.z += u.z;
            v.w += u.w;
        }
        *reinterpret_cast<uint2*>(static_cast<char*>(p.out) + (static_cast<size_t>(m0 + t0 + t) * p.n + n0 + c) * 2) =
            make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
    }
}

}  // namespace fp8_skinny
}  // namespace tdist

using namespace tdist;
using tdist_host::fail;

namespace tdist_host {

bool fp8_skinny_plan(int m, int n, int k, double other_s, SkinnyPlan* plan) {
    using namespace tdist::fp8_skinny;
    if (m > MAX_TOK) return false;   // a second tile of tokens costs more than the large tiles' padding (m200 n6144 k4096: 32 us, 22 us there)
    const int m_tiles = 1;
    const int tok = (m + 15) / 16 * 16;
    const int n_tiles = (n + ROWS - 1) / ROWS;
    const int kbs = k / BK;
    const int tiles = n_tiles * m_tiles;
    // The model of gemm_skinny_sm100.cu, with a CTA's rate as measured here; above 64 tokens it has its SM to itself
    // (registers) and moves less.
    const int sms = sm_count();
    const int fit = tok <= TOK ? 2 : 1;
    const double stage = W_BYTES + tok * BK;
    const double hbm_s = (static_cast<double>(n) * k + static_cast<double>(m) * (k + 2.0 * n)) / 6.4e12;
    double best = 1e30;
    int best_split = 1;
    for (int split = 1; split <= MAX_SPLIT; ++split) {
        if (split > 1 && kbs < 3 * split) break;
        // clusters that do not divide a GPC leave some of its SMs unused
        const int slots = split <= 2 ? fit * sms : fit * sms * 9 / 10;
        const int ctas = tiles * split;
        const int rounds = (ctas + slots - 1) / slots;
        const double sm_s = rounds * ((kbs + split - 1) / split) * stage / (tok <= TOK ? 60e9 : 40e9);
        const double loads = std::pow(std::pow(sm_s * 1e6, 6) + std::pow(hbm_s * 1e6, 6), 1.0 / 6) * 1e-6;
        const double fixed = 5.3e-6 + tok * (15e-9 + 16e-9 / split + (ctas > sms ? 20e-9 : 0.0)) + 0.05e-6 * split;
        const double t = loads + fixed * (1 + 0.5 * (rounds - 1));
        if (t < best) {
            best = t;
            best_split = split;
        }
    }
    if (best >= other_s) return false;
    plan->tok = tok;
    plan->m_tiles = m_tiles;
    plan->n_tiles = n_tiles;
    plan->split = best_split;
    plan->stages = STAGE_AREA / (W_BYTES + tok * BK);
    if (plan->stages > MAX_STAGES) plan->stages = MAX_STAGES;
    plan->grid = tiles * best_split;
    return true;
}

int fp8_skinny_run(const TdistGemmFp8Args* a, const SkinnyPlan& plan) {
    using namespace tdist::fp8_skinny;
    Params p;
    memset(&p, 0, sizeof(p));
    const uint64_t K = a->k, N = a->n, M = a->m_per_rank;
    const uint64_t strides[1] = {K};
    int rc;
    {
        const uint64_t dims[2] = {K, N};
        const uint32_t box[2] = {BK, ROWS};
        if ((rc = encode_tmap(&p.tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 2, a->b, dims, strides, box, Swizzle::B128))) return rc;
    }
    {
        const uint64_t dims[2] = {K, M};
        const uint32_t box[2] = {BK, static_cast<uint32_t>(plan.tok)};
        if ((rc = encode_tmap(&p.tm_x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 2, a->a, dims, strides, box, Swizzle::B128))) return rc;
    }
    p.sa = static_cast<const float*>(a->sa);
    p.sb = static_cast<const float*>(a->sb);
    p.out = a->c;
    p.m = a->m_per_rank;
    p.n = a->n;
    p.kb_total = a->k / BK;
    p.tok = plan.tok;
    p.m_tiles = plan.m_tiles;
    p.split = plan.split;
    p.stages = plan.stages;
    p.buf_cols = plan.tok <= 32 ? 32 : (plan.tok <= 64 ? 64 : 128);
    p.bufs = plan.tok <= 64 ? 4 : 2;
    p.tmem_cols = p.bufs * p.buf_cols;   // 128 or 256: two CTAs fit an SM
    p.wctx.status = static_cast<Status*>(a->status);
    p.wctx.timeout_ns = a->timeout_ns;
    p.wctx.kernel_id = kKernelGemmFp8;
    p.wctx.rank = a->rank;
    {
        static bool done[64] = {};
        static std::mutex lock;
        std::lock_guard<std::mutex> guard(lock);
        int dev = 0;
        TDIST_CUDA_OK(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64) return fail(TDIST_EINVAL, "fp8 gemm: device ordinal out of range");
        if (!done[dev]) {
            TDIST_CUDA_OK(cudaFuncSetAttribute(gemm_fp8_skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
            done[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(plan.grid));
    cfg.blockDim = dim3(plan.tok <= TOK ? 192 : MAX_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = static_cast<cudaStream_t>(a->stream);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(plan.split);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1] = pdl_attribute();
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    TDIST_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_fp8_skinny_kernel, p));
    return 0;
}

}  // namespace tdist_host

// Few-row GEMM for sm_100a: C[M,N] = A[M,K] * B[N,K]^T where M is a decode step's or a short prompt's worth of tokens.
//
// Bound by reading B (the weights) once from HBM, so the work is cut by rows of B and not by rows of A: the weights are
// the M = 128 operand of tcgen05.mma and up to 128 tokens are its N operand. A CTA owns 128 weight rows x `tok` tokens
// (tok = tokens rounded up to 16) over a range of K; the ranges of one tile (`split` of them) form a thread-block
// cluster. 128 x tok leaves 16 KB + 128 tok bytes per 64-wide K block, small enough for two CTAs of 3..6 stages per SM:
// 130-200 KB in flight per SM, and the prologue and epilogue of one CTA run under the loads of the other.
//
// Why the clusters: N / 128 tiles fill the machine only from N ~ 19000 on; below that the rest of the parallelism has to
// come from K. The split partials meet in shared memory: CTA r of a cluster sums the r-th share of the tokens, every
// CTA stores its fp32 accumulators of that share into CTA r's shared memory (st.shared::cluster; the stages are free by
// then), and CTA r adds them in the order of K and writes bf16 / fp16 once. No workspace, no counters, no atomics, so
// calls on any number of streams are independent and the result does not depend on timing.
//
// Measured, weights from HBM every time, before (128 x 256 tiles over all of K) and here: m16 n6144 k12288 77.9 us (1.9 TB/s)
// and 27.3 us (5.5 TB/s); m16 n1024 k8192 52 and 9 us; m128 n4096 k4096 30 and 15 us; m16 n49152 k4096 79 and 69 us.
//
// Warps (192 threads): 0 = TMA producer, 1 = MMA issuer and TMEM owner, 2..5 = epilogue. One tile per CTA.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>

#include "../device/act.cuh"
#include "../device/ptx.cuh"
#include "../device/signal.cuh"
#include "../include/tdist.h"
#include "../runtime/host_common.h"
#include "gemm_skinny.h"

namespace tdist {
namespace skinny {

constexpr int ROWS = 128;      // weight rows per CTA (UMMA M)
constexpr int MAX_TOK = 128;   // tokens per CTA (UMMA N)
constexpr int BK = 64, UMMA_K = 16;
constexpr int W_BYTES = ROWS * BK * 2;
constexpr int MAX_STAGES = 6, MAX_SPLIT = 8;
constexpr int THREADS = 192;
constexpr int STAGE_AREA = 108 * 1024;   // with alignment and barriers below half of an SM's 227 KB: two CTAs per SM
constexpr int SMEM_BYTES = STAGE_AREA + 1024 + 256;
// the partials of one cluster share: split x ceil(tok / split) tokens x 128 rows of fp32
static_assert((MAX_TOK + MAX_SPLIT) * ROWS * 4 <= STAGE_AREA, "the partial sums reuse the stages");

constexpr int kKernelSkinny = 1;   // reported as the GEMM family

struct Params {
    CUtensorMap tm_w;   // {K, N}, box {64, 128}
    CUtensorMap tm_x;   // {K, M}, box {64, tok}
    void* out;          // [M, N] bf16 / fp16
    int m, n, k_blocks, tok, m_tiles, split, stages, is_f16, act, tmem_cols;
    WaitCtx wctx;
};

__global__ void __launch_bounds__(THREADS, 2) gemm_skinny_kernel(const __grid_constant__ Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGE_AREA);   // [0,S) full, [S,2S) empty, [2S] accumulator done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 1);
    const int warp = static_cast<int>(threadIdx.x) >> 5;
    const int lane = static_cast<int>(threadIdx.x) & 31;
    const uint32_t bars_u32 = smem_u32(bars);
    auto bar_full = [&](uint32_t s) { return bars_u32 + 8u * s; };
    auto bar_empty = [&](uint32_t s) { return bars_u32 + 8u * (MAX_STAGES + s); };
    const uint32_t bar_done = bars_u32 + 8u * (2 * MAX_STAGES);

    const int tile = static_cast<int>(blockIdx.x) / p.split;
    const int part = static_cast<int>(blockIdx.x) - tile * p.split;   // = rank in the cluster
    const int m0 = (tile % p.m_tiles) * p.tok;    // the token tiles of one weight tile run side by side: it is read from HBM once
    const int n0 = (tile / p.m_tiles) * ROWS;
    const int kb0 = static_cast<int>(static_cast<long long>(p.k_blocks) * part / p.split);
    const int kb1 = static_cast<int>(static_cast<long long>(p.k_blocks) * (part + 1) / p.split);
    const uint32_t stage_bytes = W_BYTES + static_cast<uint32_t>(p.tok) * (BK * 2);
    const uint32_t stages = static_cast<uint32_t>(p.stages);

    if (threadIdx.x == 0) {
        prefetch_tensormap(&p.tm_w);
        prefetch_tensormap(&p.tm_x);
        for (uint32_t s = 0; s < stages; ++s) {
            mbar_init(bar_full(s), 1);
            mbar_init(bar_empty(s), 1);
        }
        mbar_init(bar_done, 1);
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
            const uint32_t idesc = umma_idesc(p.is_f16 ? 0u : 1u, p.is_f16 ? 0u : 1u, ROWS, static_cast<uint32_t>(p.tok));
            uint32_t s = 0, phase = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                mbar_wait(bar_full(s), phase, p.wctx, 4);
                tc_fence_after();
                const uint32_t src = smem_u32(smem) + s * stage_bytes;
                const uint64_t wdesc = umma_desc_k_sw128(src);
                const uint64_t xdesc = umma_desc_k_sw128(src + W_BYTES);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) umma_bf16<1>(tmem_base, wdesc + 2 * k, xdesc + 2 * k, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
                umma_commit(bar_empty(s));
                if (++s == stages) {
                    s = 0;
                    phase ^= 1u;
                }
            }
            umma_commit(bar_done);
        }
        __syncwarp();
    } else {
        mbar_wait(bar_done, 0, p.wctx, 5);
        tc_fence_after();
    }

    // ---- exchange: [source part][token of the share][weight row] fp32 in every CTA's shared memory
    cluster_arrive();   // this CTA's MMAs (and with them its loads) are complete: its stages may be overwritten
    cluster_wait();
    const int live = min(p.tok, p.m - m0);
    const int per = (p.tok + p.split - 1) / p.split;
    float* sums = reinterpret_cast<float*>(smem);
    if (warp >= 2) {
        const int q = warp & 3;   // TMEM lane quadrant this warp may read
        const uint32_t mine = smem_u32(sums) + static_cast<uint32_t>((part * per * ROWS + q * 32 + lane) * 4);
        int owner = 0, j = 0;
        uint32_t dst = mapa_u32(mine, 0);
        for (int c = 0; c < live; c += 16) {
            uint32_t r[16];
            tmem_ld_32x16(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(c), r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                st_shared_cluster_f32(dst + static_cast<uint32_t>(j) * (ROWS * 4), __uint_as_float(r[i]));
                if (++j == per) {
                    j = 0;
                    owner = min(owner + 1, p.split - 1);
                    dst = mapa_u32(mine, static_cast<uint32_t>(owner));
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
    constexpr int UNROLL = 4;   // items per thread and step: their loads of one source part are in flight together
    for (int i0 = static_cast<int>(threadIdx.x); i0 < items; i0 += UNROLL * THREADS) {
        float4 acc[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s = 0; s < p.split; ++s) {
            const float4* src = reinterpret_cast<const float4*>(sums + s * per * ROWS);
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                if (i0 + u * THREADS >= items) continue;
                const float4 v = src[i0 + u * THREADS];
                acc[u].x += v.x;
                acc[u].y += v.y;
                acc[u].z += v.z;
                acc[u].w += v.w;
            }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int i = i0 + u * THREADS;
            const int t = i / (ROWS / 4), c = (i % (ROWS / 4)) * 4;
            if (i >= items || n0 + c >= p.n) continue;   // N is a multiple of 8: all four columns or none
            float4 v = acc[u];
            if (p.act != TDIST_ACT_NONE) {
                v.x = activate(v.x, p.act);
                v.y = activate(v.y, p.act);
                v.z = activate(v.z, p.act);
                v.w = activate(v.w, p.act);
            }
            const uint2 w = p.is_f16 ? make_uint2(pack_f16x2(v.x, v.y), pack_f16x2(v.z, v.w)) : make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
            *reinterpret_cast<uint2*>(static_cast<char*>(p.out) + (static_cast<size_t>(m0 + t0 + t) * p.n + n0 + c) * 2) = w;
        }
    }
}

}  // namespace skinny
}  // namespace tdist

using namespace tdist;
using tdist_host::fail;

namespace {

// CTAs of the kernel that are resident at once when they come in clusters of `split` (a cluster needs its SMs in one GPC,
// so sizes that do not divide a GPC leave some unused). The occupancy query counts one CTA per SM here whatever the
// carveout; two do run (clusters of four, n6144 k12288: 192 CTAs finish sooner than 144 in clusters of three). Cached per device.
int skinny_slots(int split) {
    using namespace tdist::skinny;
    static int cache[64][MAX_SPLIT + 1] = {};
    static std::mutex lock;
    std::lock_guard<std::mutex> guard(lock);
    int dev = 0;
    const int nominal = 2 * tdist_host::sm_count() / split * split;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return nominal;   // planning on a host without a GPU
    }
    int& slot = cache[dev][split];
    if (slot > 0) return slot;
    int clusters = 0;
    const void* fn = reinterpret_cast<const void*>(&gemm_skinny_kernel);
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(nominal));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(split);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters > 0)
        slot = clusters * split <= tdist_host::sm_count() ? 2 * clusters * split : clusters * split;
    else
        slot = nominal;
    cudaGetLastError();
    return slot;
}

}  // namespace

namespace tdist_host {

bool skinny_plan(int m, int n, int k, double other_s, SkinnyPlan* plan) {
    using namespace tdist::skinny;
    if (m > 4 * MAX_TOK) return false;   // every further 128 tokens read the weights once more out of L2
    const int m_tiles = (m + MAX_TOK - 1) / MAX_TOK;
    const int tok = ((m + m_tiles - 1) / m_tiles + 15) / 16 * 16;
    const int n_tiles = (n + ROWS - 1) / ROWS;
    const int k_blocks = (k + BK - 1) / BK;
    const int tiles = n_tiles * m_tiles;
    // Model of a run, fitted to sweeps over M 1..512, N 256..49152, K 1024..16384 and every split: a CTA moves 70 GB/s
    // whatever its tile (twice the stages on a CTA that has its SM to itself changed nothing), HBM delivers 6.4 TB/s and
    // the two bend into one another; launch, first loads and the exchange of the partial sums cost 5.3 us and 15-50 ns per
    // token of the tile, the most where two CTAs share an SM; half of that again for every further round. Chosen splits are within 8 % of the best one measured
    // (m16 n14336 k4096: 2, 24 us; 3, which needs a second wave, 29 us; 1, 27 us).
    const double stage = W_BYTES + tok * BK * 2;
    const double hbm_s = 2.0 * (static_cast<double>(n) * k + static_cast<double>(m) * (k + n)) / 6.4e12;
    const int sms = tdist_host::sm_count();
    double best = 1e30;
    int best_split = 1;
    for (int split = 1; split <= MAX_SPLIT; ++split) {
        if (split > 1 && k_blocks < 3 * split) break;   // a part shorter than the pipeline only adds partial sums
        const int slots = skinny_slots(split);
        const int ctas = tiles * split;
        const int blocks = (k_blocks + split - 1) / split;
        const int rounds = (ctas + slots - 1) / slots;
        const double sm_s = rounds * blocks * stage / 70e9;
        const double loads = std::pow(std::pow(sm_s * 1e6, 6) + std::pow(hbm_s * 1e6, 6), 1.0 / 6) * 1e-6;
        const double fixed = 5.3e-6 + tok * (15e-9 + 16e-9 / split + (ctas > sms ? 20e-9 : 0.0)) + 0.05e-6 * split;
        const double t = loads + fixed * (1 + 0.5 * (rounds - 1));
        if (t < best) {
            best = t;
            best_split = split;
        }
    }
    // above 256 rows the two are close (m384 n49152 k4096: 165 us here, 152 us on the large tiles) and the model is not that sharp
    if (best >= (m > 2 * MAX_TOK ? 0.9 : 1.0) * other_s) return false;
    plan->tok = tok;
    plan->m_tiles = m_tiles;
    plan->n_tiles = n_tiles;
    plan->split = best_split;
    plan->stages = STAGE_AREA / (W_BYTES + tok * BK * 2);
    if (plan->stages > MAX_STAGES) plan->stages = MAX_STAGES;
    plan->grid = tiles * best_split;
    return true;
}

int skinny_run(const TdistGemmArgs* a, const SkinnyPlan& plan) {
    using namespace tdist::skinny;
    Params p;
    memset(&p, 0, sizeof(p));
    const CUtensorMapDataType dt = a->dtype == TDIST_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const uint64_t K = a->k, N = a->n, M = a->m_per_rank;
    const uint64_t strides[1] = {K * 2};
    int rc;
    {
        const uint64_t dims[2] = {K, N};
        const uint32_t box[2] = {BK, ROWS};
        if ((rc = encode_tmap(&p.tm_w, dt, 2, 2, a->b, dims, strides, box, Swizzle::B128))) return rc;
    }
    {
        const uint64_t dims[2] = {K, M};
        const uint32_t box[2] = {BK, static_cast<uint32_t>(plan.tok)};
        if ((rc = encode_tmap(&p.tm_x, dt, 2, 2, a->a, dims, strides, box, Swizzle::B128))) return rc;
    }
    p.out = a->c;
    p.m = a->m_per_rank;
    p.n = a->n;
    p.k_blocks = (a->k + BK - 1) / BK;
    p.tok = plan.tok;
    p.m_tiles = plan.m_tiles;
    p.split = plan.split;
    p.stages = plan.stages;
    p.is_f16 = a->dtype == TDIST_F16;
    p.act = a->act;
    p.tmem_cols = plan.tok <= 32 ? 32 : (plan.tok <= 64 ? 64 : 128);
    p.wctx.status = static_cast<Status*>(a->status);
    p.wctx.timeout_ns = a->timeout_ns;
    p.wctx.kernel_id = kKernelSkinny;
    p.wctx.rank = a->rank;
    skinny_slots(plan.split);   // opts in to the shared memory on this device
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(static_cast<unsigned>(plan.grid));
    cfg.blockDim = dim3(THREADS);
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
    TDIST_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_skinny_kernel, p));
    return 0;
}

}  // namespace tdist_host

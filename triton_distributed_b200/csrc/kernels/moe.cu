// MoE routing kernels: softmax + top-k selection, expert-sorted permutation of (token, k) pairs,
// and the block-aligned, rank-major sort that the MoE group-GEMMs consume.
//
// Reference counterparts: `select_experts` (torch softmax/topk; kernels/nvidia/moe_reduce_rs.py:180-197),
// `kernel_bincount` + torch argsort/cumsum (kernels/nvidia/ep_a2a.py:309-321, test_all_to_all.py
// `calc_gather_index`), and the hand-written `moe_ag_scatter_align_block_size_kernel`
// (csrc/lib/moe_utils.cu:60-192) with its Python oracle `full_moe_align_block_size`
// (kernels/nvidia/moe_reduce_rs.py:87-177). The sorts here are stable (ascending pair index inside
// an expert), so results are reproducible and comparable element by element with the oracle.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "../device/moe_sort.cuh"
#include "../device/ptx.cuh"
#include "../device/signal.cuh"
#include "../include/tdist.h"
#include "../runtime/host_common.h"

namespace tdist {

// ---------------------------------------------------------------------------- routing for EP
// ids[n] (n = tokens * topk, token-major) -> splits[E], cumsum[E+1], sorted_token[n] (token of the
// pair at each sorted position), slot_of[n] (sorted position of each pair). One CTA; a chain of latencies, so few steps: every
// warp counts a contiguous run of the pairs by itself (position inside the run's group = count so far + equal ids in lower
// lanes, kept in slot_of meanwhile), prefix sums over the warps and over the experts follow, then every pair's position is
// known. Steps past the end of a run are left out: a match of 32 different values takes longest of all (1024 pairs of 64 experts 7.8 us with
// them, 4.5 without). (Histogram, then 512 pairs at a time with the CTA meeting four times for each: the
// whole expert-parallel block of 1194 tokens, top 8 of 16, 280 us, 267 here; 1831 tokens, top 7 of 16, 323 and 314.)
constexpr int kRouteAhead = 4;   // loads of a lane in flight
__global__ void __launch_bounds__(1024) moe_route_kernel(const int* ids, int n, int topk, int E, int* splits,
                                                         int* cumsum, int* sorted_token, int* slot_of, WaitCtx w) {
    extern __shared__ int sm[];
    const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    const int threads = static_cast<int>(blockDim.x), warps = threads >> 5;
    int* first = sm;        // sorted position of an expert's first pair
    int* hist = sm + E;
    int* cnt = sm + 2 * E;  // [warps][E]
    for (int j = tid; j < warps * E; j += threads) cnt[j] = 0;
    pdl_wait_and_release();
    __syncthreads();
    const int run = (n + threads - 1) / threads * 32;   // pairs of a warp
    const int begin = warp * run, end = min(n, begin + run);
    int* mine = cnt + warp * E;
    for (int i0 = begin; i0 < end; i0 += 32 * kRouteAhead) {
        int es[kRouteAhead];
#pragma unroll
        for (int u = 0; u < kRouteAhead; ++u) es[u] = i0 + u * 32 + lane < end ? ids[i0 + u * 32 + lane] : -1;
#pragma unroll
        for (int u = 0; u < kRouteAhead; ++u) {
            if (i0 + u * 32 >= end) break;
            const int i = i0 + u * 32 + lane, e = es[u];
            const bool valid = i < end && expert_in_range(e, E);
            if (i < end && !valid) report_bad_expert(w, i, e, E, 1);
            const unsigned same = __match_any_sync(0xffffffffu, valid ? e : E + lane);   // idle lanes and rejected ids match nobody
            const int before = valid ? mine[e] : 0;
            __syncwarp();
            if (valid && (same & lanemask_lt()) == 0) mine[e] = before + __popc(same);
            __syncwarp();
            if (i < end) slot_of[i] = valid ? before + __popc(same & lanemask_lt()) : -1;   // -1: a pair whose expert id was rejected
        }
    }
    __syncthreads();
    for (int e = tid; e < E; e += threads) {
        int total = 0;
        for (int k = 0; k < warps; ++k) {
            const int c = cnt[k * E + e];
            cnt[k * E + e] = total;
            total += c;
        }
        hist[e] = total;
        splits[e] = total;
    }
    __syncthreads();
    if (warp == 0) {
        // exclusive scan of the histogram by one warp: a contiguous chunk of experts per lane
        const int per = (E + 31) / 32;
        const int e0 = min(E, lane * per), e1 = min(E, e0 + per);
        int local = 0;
        for (int e = e0; e < e1; ++e) local += hist[e];
        int incl = local;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        int acc = incl - local;
        for (int e = e0; e < e1; ++e) {
            first[e] = acc;
            cumsum[e] = acc;
            acc += hist[e];
        }
        if (lane == 31) cumsum[E] = incl;
    }
    __syncthreads();
    // the same lanes as above: they read back their own stores
    for (int i0 = begin; i0 < end; i0 += 32 * kRouteAhead) {
        int es[kRouteAhead], in_run[kRouteAhead];
#pragma unroll
        for (int u = 0; u < kRouteAhead; ++u) {
            const int i = i0 + u * 32 + lane;
            es[u] = i < end ? ids[i] : 0;
            in_run[u] = i < end ? slot_of[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < kRouteAhead; ++u) {
            if (in_run[u] < 0) continue;
            const int i = i0 + u * 32 + lane;
            const int pos = first[es[u]] + mine[es[u]] + in_run[u];
            slot_of[i] = pos;
            sorted_token[pos] = i / topk;
        }
    }
}

// ---------------------------------------------------------------------------- block-aligned sort
// One CTA per source rank. See the header comment for the layout.
__global__ void __launch_bounds__(kMoeThreads) moe_align_kernel(const int* ids, int numel_per_rank, int E, int num_ranks,
                                                                int block_size, int* sorted_ids, int sorted_cap,
                                                                int* expert_ids, int* block_barrier_ids,
                                                                int* rank_block_num, int* num_tokens_post_pad,
                                                                WaitCtx w) {
    extern __shared__ int sm[];
    int* hist = sm;
    int* running = sm + E;
    int* cnt = sm + 2 * E;
    __shared__ int base_s, total_s;
    const int r = static_cast<int>(blockIdx.x);
    const int pad_value = numel_per_rank * num_ranks;
    if (threadIdx.x == 0) base_s = 0;
    // padded sizes of the earlier ranks give this rank's base offset
    for (int q = 0; q <= r; ++q) {
        histogram(ids + static_cast<size_t>(q) * numel_per_rank, numel_per_rank, E, hist, w);
        if (threadIdx.x == 0) {
            int acc = 0;
            for (int e = 0; e < E; ++e) {
                if (q == r) running[e] = acc;
                acc += (hist[e] + block_size - 1) / block_size * block_size;
            }
            if (q < r) base_s += acc;
            else total_s = acc;
        }
        __syncthreads();
    }
    const int base = base_s, total = total_s;
    if (threadIdx.x == 0) {
        rank_block_num[r] = total / block_size;
        if (r == num_ranks - 1) *num_tokens_post_pad = base + total;
    }
    // block -> expert / source-rank tables and padding of this rank's region (and of the tail)
    for (int e = threadIdx.x; e < E; e += kMoeThreads) {
        const int b0 = running[e] / block_size;
        const int nb = (hist[e] + block_size - 1) / block_size;
        for (int b = 0; b < nb; ++b) {
            expert_ids[base / block_size + b0 + b] = e;
            block_barrier_ids[base / block_size + b0 + b] = r;
        }
    }
    const int fill_end = (r == num_ranks - 1) ? sorted_cap : base + total;
    for (int i = base + threadIdx.x; i < fill_end; i += kMoeThreads) sorted_ids[i] = pad_value;
    __syncthreads();
    const int* my = ids + static_cast<size_t>(r) * numel_per_rank;
    stable_positions(my, numel_per_rank, E, running, cnt, w, [&](int i, int pos) {
        if (pos >= 0) sorted_ids[base + pos] = i + r * numel_per_rank;
    });
}

// ---------------------------------------------------------------------------- softmax + top-k
// One warp per token; E <= 1024, J = ceil(E / 32) logits per lane rounded up to a power of two: the selection walks them
// topk times, so 32 per lane whatever E is costs more than the loads (128 tokens, 8 of 256: 6.2 us with 32 per lane, 4.1 us with 8).
// weights = softmax probabilities of the selected experts, optionally renormalised to sum to one. Ties go to the lower
// expert index.
template <int J>
__device__ __forceinline__ void topk_softmax_row(const float* row, int E, int topk, int renorm, int lane, int* ids, float* w) {
    float v[J];
    float mx = -CUDART_INF_F;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int e = j * 32 + lane;
        v[j] = e < E ? row[e] : -CUDART_INF_F;
        mx = fmaxf(mx, v[j]);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j) sum += (j * 32 + lane < E) ? __expf(v[j] - mx) : 0.f;
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    float picked_sum = 0.f;
    float my_w = 0.f;
    int my_id = 0;
    for (int k = 0; k < topk; ++k) {
        float best = -CUDART_INF_F;
        int best_e = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int e = j * 32 + lane;
            if (v[j] > best) {
                best = v[j];
                best_e = e;
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
            if (ob > best || (ob == best && oe < best_e)) {
                best = ob;
                best_e = oe;
            }
        }
        const float prob = __expf(best - mx) / sum;
        picked_sum += prob;
        if (lane == k) {
            my_w = prob;
            my_id = best_e;
        }
        if ((best_e & 31) == lane) {
#pragma unroll
            for (int j = 0; j < J; ++j)
                if (j == (best_e >> 5)) v[j] = -CUDART_INF_F;
        }
    }
    if (lane < topk) {
        ids[lane] = my_id;
        w[lane] = renorm ? my_w / picked_sum : my_w;
    }
}
__device__ __forceinline__ void topk_softmax_any(const float* row, int E, int topk, int renorm, int lane, int* ids, float* w) {
    if (E <= 32) topk_softmax_row<1>(row, E, topk, renorm, lane, ids, w);
    else if (E <= 64) topk_softmax_row<2>(row, E, topk, renorm, lane, ids, w);
    else if (E <= 128) topk_softmax_row<4>(row, E, topk, renorm, lane, ids, w);
    else if (E <= 256) topk_softmax_row<8>(row, E, topk, renorm, lane, ids, w);
    else topk_softmax_row<32>(row, E, topk, renorm, lane, ids, w);
}
__global__ void moe_topk_softmax_kernel(const float* logits, int ntok, int E, int topk, int renorm, int* ids, float* w) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    pdl_wait_and_release();
    if (warp >= ntok) return;
    const size_t at = static_cast<size_t>(warp) * topk;
    topk_softmax_any(logits + static_cast<size_t>(warp) * E, E, topk, renorm, static_cast<int>(threadIdx.x) & 31, ids + at, w + at);
}

// ---------------------------------------------------------------------------- gate: logits, softmax and top-k in one launch
// logits[t, e] = x[t, :] . gate[e, :] (bf16 in, fp32 sums), then the selection above. A decode step has few tokens and
// few experts, so the product is short of parallelism, not of arithmetic: 16 tokens are a tile, and its hidden dimension, 32 values
// at a time, is dealt over 16 chains of sums (what a cuBLAS SGEMM of the fp32 copies does serially; 128 x
// 7168 x 32 experts: 53 us as two copies, SGEMM, reduction and selection, 12 us on one CTA per tile). mma.sync m16n8k16: the
// products of bf16 values are exact in fp32, the tensor core sums 32 of them at a time (its accumulator truncates, so longer
// chains there would lose bits against an fp32 FMA loop), the rest is added in fp32: a chain's steps in order, then the 16 chains
// in order. A tcgen05 tile (M 128) would leave all but 16 rows of this split idle. Any order of k will do as long as x and gate
// agree, so a thread takes 8 consecutive values of its row per step: one 16-byte load feeds two MMAs.
//
// That order of the sums is the same in all forms below, which the number of tokens chooses between: a token's logits, and with
// them the choice between near ties, do not depend on how many others are in the call. The forms, us per call at 16 tokens x 4096,
// 8 experts / 128 x 7168, 32 / 300 x 7168, 64 / 1200 x 6720, 64:
//   a CTA per tile, a chain per warp                                        4.0 / 10.2 / 15.5 / 15.3
//   a cluster of up to eight CTAs per tile, which share the experts           - /  7.6 /  9.0 / 21.6
//   a cluster of eight (or four) CTAs per tile, which share the chains      2.9 /  5.4 / 14.3 / 36
// (Up to eight parts of the hidden dimension, each a sum of its own, took 2.9 / 5.7 / 9.5 / 15.3: there the order of the sums followed the
// number of parts, and that the number of tokens. Eight such sums whatever the number of CTAs: 29 us for the last of these.)
constexpr int kGateTok = 16, kGateThreads = 512, kGateWarps = kGateThreads / 32;

constexpr int kGateMaxParts = 8;

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Rows past the end repeat the last one; their results are not used.
__device__ __forceinline__ const __nv_bfloat16* gate_row(const __nv_bfloat16* m, int row, int rows, int hidden, int tig) {
    return m + static_cast<size_t>(min(row, rows - 1)) * hidden + tig * 8;
}

// NT: groups of 8 experts per pass over the tokens' rows; SPLIT: a cluster of `split` CTAs per tile, which share the experts
template <int NT, bool SPLIT>
__global__ void __launch_bounds__(kGateThreads, 1) moe_gate_topk_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gate, int ntok, int hidden, int E,
                                                                        int topk, int renorm, int split, int* ids, float* w, float* logits) {
    const int parts = SPLIT ? split : 1;
    extern __shared__ float gate_sm[];
    constexpr int COLS = NT * 8;
    // steps whose loads are in flight: a split tile's CTA has an SM to itself and few steps (more of them cost 4096 tokens x 7168, 8
    // experts 12.6 us on one CTA per tile, 11.5 so)
    constexpr int AHEAD = SPLIT ? (NT == 8 ? 1 : (NT == 4 ? 2 : 8 / NT)) : 1, UNROLL = SPLIT || NT == 8 ? 1 : 2;
    float* part = gate_sm;                                   // [warps][16 tokens][COLS]
    float* row_s = gate_sm + kGateWarps * kGateTok * COLS;   // [16 / parts tokens][E]: the tokens this CTA selects for
    const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tig = lane & 3;                 // row / column group of the MMA fragments
    const int part_id = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
    const int t0 = static_cast<int>(blockIdx.x) / parts * kGateTok;
    const int own = kGateTok / parts;   // tokens a CTA selects for
    const int steps = hidden / 32;
    if (SPLIT) cluster_arrive();    // its counterpart stands before the first store into another CTA
    pdl_wait_and_release();
    const __nv_bfloat16* xa = gate_row(x, t0 + g, ntok, hidden, tig);
    const __nv_bfloat16* xb = gate_row(x, t0 + g + 8, ntok, hidden, tig);
    bool apart = SPLIT;   // the other CTAs of the cluster may not run yet
    for (int e0 = part_id * COLS; e0 < E; e0 += parts * COLS) {
        const __nv_bfloat16* ge[NT];
        float acc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            ge[n] = gate_row(gate, e0 + n * 8 + g, E, hidden, tig);
            acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
        }
#pragma unroll(UNROLL)
        for (int s0 = warp; s0 < steps; s0 += AHEAD * kGateWarps) {
            uint4 a[AHEAD], c[AHEAD], b[AHEAD][NT];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int s = s0 + u * kGateWarps;
                if (s >= steps) break;
                a[u] = ld_v4(xa + s * 32);
                c[u] = ld_v4(xb + s * 32);
#pragma unroll
                for (int n = 0; n < NT; ++n) b[u][n] = ld_v4(ge[n] + s * 32);
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                if (s0 + u * kGateWarps >= steps) break;
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    float d[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_bf16_16816(d, a[u].x, c[u].x, a[u].y, c[u].y, b[u][n].x, b[u][n].y);
                    mma_bf16_16816(d, a[u].z, c[u].z, a[u].w, c[u].w, b[u][n].z, b[u][n].w);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[n][i] += d[i];
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float* p = part + (warp * kGateTok + g) * COLS + n * 8 + tig * 2;
            *reinterpret_cast<float2*>(p) = make_float2(acc[n][0], acc[n][1]);
            *reinterpret_cast<float2*>(p + 8 * COLS) = make_float2(acc[n][2], acc[n][3]);
        }
        __syncthreads();
        if (apart) cluster_wait();
        apart = false;
        for (int i = tid; i < kGateTok * COLS; i += kGateThreads) {
            const int t = i / COLS, e = e0 + i % COLS;
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < kGateWarps; ++k) sum += part[k * kGateTok * COLS + i];
            if (e >= E) continue;
            if (SPLIT) {
                st_shared_cluster_f32(mapa_u32(smem_u32(row_s + (t % own) * E + e), static_cast<uint32_t>(t / own)), sum);
            } else {
                row_s[t * E + e] = sum;
            }
            if (logits != nullptr && t0 + t < ntok) logits[static_cast<size_t>(t0 + t) * E + e] = sum;
        }
        __syncthreads();
    }
    if (SPLIT) {
        if (apart) cluster_wait();   // no experts were left for this CTA
        cluster_arrive();
        cluster_wait();
    }
    const int t = t0 + part_id * own + warp;   // a warp per token: kGateWarps == kGateTok
    static_assert(kGateWarps == kGateTok, "a warp per token");
    if (warp < own && t < ntok) topk_softmax_any(row_s + warp * E, E, topk, renorm, lane, ids + static_cast<size_t>(t) * topk, w + static_cast<size_t>(t) * topk);
}

// A cluster of PARTS CTAs per tile, 16 / PARTS chains each, for at most 8 NT experts. The products of a chain's steps, which PARTS
// warps take in turn, meet in shared memory and are added there in order; the chain's sum goes to the CTA that selects for the
// token, which adds the 16 chains. Every row is read once per tile.
constexpr int kGateChains = kGateWarps;
// floats between the rows of a step's products: those that a warp stores at once spread over the banks
__host__ __device__ constexpr int gate_pitch(int nt) { return nt * 8 + 8; }
static int gate_chains_smem(int hidden, int nt, int E, int parts) {
    const int most = (hidden / 32 + kGateChains - 1) / kGateChains;   // steps of a chain
    return (kGateChains / parts * most * kGateTok * gate_pitch(nt) + kGateChains * (kGateTok / parts) * E) * static_cast<int>(sizeof(float));
}

template <int NT, int PARTS>
__global__ void __launch_bounds__(kGateThreads, 1) moe_gate_topk_chains_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gate, int ntok, int hidden, int E,
                                                                               int topk, int renorm, int* ids, float* w, float* logits) {
    extern __shared__ float gate_sm[];
    constexpr int COLS = NT * 8, PITCH = gate_pitch(NT), STEP = kGateTok * PITCH;
    constexpr int AHEAD = NT == 8 ? 1 : 2;
    constexpr int OWN_CHAINS = kGateChains / PARTS, OWN_TOK = kGateTok / PARTS;
    const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int part_id = static_cast<int>(cluster_ctarank());
    const int t0 = static_cast<int>(blockIdx.x) / PARTS * kGateTok;
    const int steps = hidden / 32, most = (steps + kGateChains - 1) / kGateChains;
    float* prod = gate_sm;                                     // [own chains][most][16 tokens][PITCH]
    float* chain_s = gate_sm + OWN_CHAINS * most * STEP;   // [16 chains][own tokens][E]
    cluster_arrive();    // its counterpart stands before the first store into another CTA
    pdl_wait_and_release();
    const __nv_bfloat16* xa = gate_row(x, t0 + g, ntok, hidden, tig);
    const __nv_bfloat16* xb = gate_row(x, t0 + g + 8, ntok, hidden, tig);
    const __nv_bfloat16* ge[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) ge[n] = gate_row(gate, n * 8 + g, E, hidden, tig);
    const int mine = warp % OWN_CHAINS;                    // this warp's chain, among the CTA's and among all
    const int chain = part_id * OWN_CHAINS + mine;
#pragma unroll 1
    for (int j0 = warp / OWN_CHAINS; chain + j0 * kGateChains < steps; j0 += AHEAD * PARTS) {
        uint4 a[AHEAD], c[AHEAD], b[AHEAD][NT];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int s = chain + (j0 + u * PARTS) * kGateChains;
            if (s >= steps) break;
            a[u] = ld_v4(xa + s * 32);
            c[u] = ld_v4(xb + s * 32);
#pragma unroll
            for (int n = 0; n < NT; ++n) b[u][n] = ld_v4(ge[n] + s * 32);
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int j = j0 + u * PARTS;
            if (chain + j * kGateChains >= steps) break;
            float* p = prod + (mine * most + j) * STEP + g * PITCH + tig * 2;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                mma_bf16_16816(d, a[u].x, c[u].x, a[u].y, c[u].y, b[u][n].x, b[u][n].y);
                mma_bf16_16816(d, a[u].z, c[u].z, a[u].w, c[u].w, b[u][n].z, b[u][n].w);
                *reinterpret_cast<float2*>(p + n * 8) = make_float2(d[0], d[1]);
                *reinterpret_cast<float2*>(p + 8 * PITCH + n * 8) = make_float2(d[2], d[3]);
            }
        }
    }
    __syncthreads();
    cluster_wait();   // every CTA of the cluster runs
    for (int i = tid; i < OWN_CHAINS * kGateTok * COLS; i += kGateThreads) {
        const int k = i / (kGateTok * COLS), t = i / COLS % kGateTok, e = i % COLS, at = part_id * OWN_CHAINS + k;
        if (e >= E) continue;
        float sum = 0.f;
        const float* p = prod + k * most * STEP + t * PITCH + e;
#pragma unroll 4
        for (int s = at; s < steps; s += kGateChains, p += STEP) sum += *p;
        st_shared_cluster_f32(mapa_u32(smem_u32(chain_s + (at * OWN_TOK + t % OWN_TOK) * E + e), static_cast<uint32_t>(t / OWN_TOK)), sum);
    }
    cluster_arrive();
    cluster_wait();
    for (int i = tid; i < OWN_TOK * E; i += kGateThreads) {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < kGateChains; ++k) sum += chain_s[k * OWN_TOK * E + i];
        chain_s[i] = sum;   // chain 0's own slot: this thread's alone
        const int t = t0 + part_id * OWN_TOK + i / E;
        if (logits != nullptr && t < ntok) logits[static_cast<size_t>(t) * E + i % E] = sum;
    }
    __syncthreads();
    const int t = t0 + part_id * OWN_TOK + warp;
    if (warp < OWN_TOK && t < ntok) topk_softmax_any(chain_s + warp * E, E, topk, renorm, lane, ids + static_cast<size_t>(t) * topk, w + static_cast<size_t>(t) * topk);
}

// ---------------------------------------------------------------------------- row gather / top-k reduce
// dst[p] = src[index[p] / div] for index[p] < limit, zeros otherwise (padding rows of the aligned
// sort); optionally records the inverse map pos_of[index[p]] = p. One warp per row, 16-byte vectors.
__global__ void gather_rows_kernel(const uint4* src, const int* index, int rows_out, int div, int limit, int vec_per_row,
                                   uint4* dst, int* pos_of) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int p = warp; p < rows_out; p += nwarps) {
        const int id = index[p];
        const bool live = id >= 0 && id < limit;
        if (live && pos_of != nullptr && lane == 0) pos_of[id] = p;
        const uint4* s = src + static_cast<size_t>(live ? id / div : 0) * vec_per_row;
        uint4* d = dst + static_cast<size_t>(p) * vec_per_row;
        for (int c = lane; c < vec_per_row; c += 32) d[c] = live ? s[c] : make_uint4(0, 0, 0, 0);
    }
}

// out[t] = sum_k w[t*topk+k] * y[pos_of[t*topk+k]] in fp32 (bf16 in/out), bound by reading y. A warp takes a token's 128
// vectors of 16 bytes at a time (a row shorter than that still goes to one warp): four loads per lane and row are in
// flight, twice that with two rows (8192 tokens x 4096, top 2: 53 us with one load per lane and row, 30 us).
constexpr int kReduceVecs = 4;
__global__ void __launch_bounds__(256) topk_reduce_kernel(const uint4* y, const int* pos_of, const float* w, int ntok, int topk, int vec_per_row,
                                                          uint4* out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int segs = (vec_per_row + 32 * kReduceVecs - 1) / (32 * kReduceVecs);
    pdl_wait_and_release();
    for (long long item = warp; item < static_cast<long long>(ntok) * segs; item += nwarps) {
        const int t = static_cast<int>(item / segs);
        const int c0 = static_cast<int>(item - static_cast<long long>(t) * segs) * 32 * kReduceVecs + lane;
        float acc[kReduceVecs][8];
#pragma unroll
        for (int u = 0; u < kReduceVecs; ++u)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[u][i] = 0.f;
#pragma unroll 2
        for (int k = 0; k < topk; ++k) {
            const int pos = pos_of[static_cast<size_t>(t) * topk + k];
            // a pair that routing rejected contributes nothing
            const float wk = pos < 0 ? 0.f : (w ? w[static_cast<size_t>(t) * topk + k] : 1.f);
            uint4 q[kReduceVecs];
#pragma unroll
            for (int u = 0; u < kReduceVecs; ++u)
                q[u] = pos >= 0 && c0 + u * 32 < vec_per_row ? ld_v4(y + static_cast<size_t>(pos) * vec_per_row + c0 + u * 32) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int u = 0; u < kReduceVecs; ++u) {
                const uint32_t v[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[u][2 * i] += wk * __uint_as_float(v[i] << 16);
                    acc[u][2 * i + 1] += wk * __uint_as_float(v[i] & 0xffff0000u);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kReduceVecs; ++u) {
            if (c0 + u * 32 >= vec_per_row) continue;
            uint4 o;
            uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t r;
                asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(acc[u][2 * i + 1]), "f"(acc[u][2 * i]));
                ow[i] = r;
            }
            out[static_cast<size_t>(t) * vec_per_row + c0 + u * 32] = o;
        }
    }
}

}  // namespace tdist

using namespace tdist;
using tdist_host::fail;

static int moe_smem_bytes(int E) { return (2 * E + kMoeWarps * E) * static_cast<int>(sizeof(int)); }

template <typename K>
static int ensure_smem(K kernel, int bytes) {
    if (bytes > 48 * 1024) TDIST_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    return 0;
}

static WaitCtx moe_wctx(void* status) {
    WaitCtx w;
    w.status = static_cast<Status*>(status);
    w.timeout_ns = 0;
    w.kernel_id = kKernelMoe;
    w.rank = 0;
    return w;
}

extern "C" int tdist_moe_route(const void* ids, int n, int topk, int num_experts, void* splits, void* cumsum,
                               void* sorted_token, void* slot_of, void* status, void* stream) {
    if (num_experts < 1 || num_experts > 2048) return fail(TDIST_ELIMIT, "moe_route: at most 2048 experts");
    if (topk < 1 || n < 0) return fail(TDIST_EINVAL, "moe_route: bad sizes");
    const int threads = num_experts <= 1024 ? 1024 : 512;   // a row of counts per warp has to fit
    const int smem = (2 + threads / 32) * num_experts * static_cast<int>(sizeof(int));
    int rc = ensure_smem(moe_route_kernel, smem);
    if (rc) return rc;
    TDIST_CUDA_OK(tdist_host::launch_pdl(moe_route_kernel, dim3(1), threads, smem, static_cast<cudaStream_t>(stream),
                                         static_cast<const int*>(ids), n, topk, num_experts, static_cast<int*>(splits), static_cast<int*>(cumsum),
                                         static_cast<int*>(sorted_token), static_cast<int*>(slot_of), moe_wctx(status)));
    return 0;
}

extern "C" int tdist_moe_align_block_size(const void* ids, int numel_per_rank, int num_experts, int num_ranks,
                                          int block_size, void* sorted_ids, int sorted_cap, void* expert_ids,
                                          void* block_barrier_ids, void* rank_block_num, void* num_tokens_post_pad,
                                          void* status, void* stream) {
    if (num_experts < 1 || num_experts > 2048) return fail(TDIST_ELIMIT, "moe_align: at most 2048 experts");
    if (block_size < 1 || num_ranks < 1) return fail(TDIST_EINVAL, "moe_align: bad sizes");
    const int smem = moe_smem_bytes(num_experts);
    int rc = ensure_smem(moe_align_kernel, smem);
    if (rc) return rc;
    moe_align_kernel<<<num_ranks, kMoeThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const int*>(ids), numel_per_rank, num_experts, num_ranks, block_size, static_cast<int*>(sorted_ids),
        sorted_cap, static_cast<int*>(expert_ids), static_cast<int*>(block_barrier_ids), static_cast<int*>(rank_block_num),
        static_cast<int*>(num_tokens_post_pad), moe_wctx(status));
    TDIST_CUDA_OK(cudaGetLastError());
    return 0;
}

extern "C" int tdist_moe_topk_softmax(const void* logits, int ntok, int num_experts, int topk, int renormalize,
                                      void* ids, void* weights, void* stream) {
    if (num_experts < 1 || num_experts > 1024) return fail(TDIST_ELIMIT, "moe_topk_softmax: at most 1024 experts");
    if (topk < 1 || topk > 32 || topk > num_experts) return fail(TDIST_EINVAL, "moe_topk_softmax: topk must be in [1, min(32, experts)]");
    if (ntok <= 0) return 0;
    const int warps_per_block = 8;
    const int blocks = (ntok + warps_per_block - 1) / warps_per_block;
    TDIST_CUDA_OK(tdist_host::launch_pdl(moe_topk_softmax_kernel, dim3(blocks), warps_per_block * 32, 0, static_cast<cudaStream_t>(stream),
                                         static_cast<const float*>(logits), ntok, num_experts, topk, renormalize,
                                         static_cast<int*>(ids), static_cast<float*>(weights)));
    return 0;
}

extern "C" int tdist_moe_gate_topk(const void* x, const void* gate, int ntok, int hidden, int num_experts, int topk, int renormalize,
                                   void* ids, void* weights, void* logits, void* stream) {
    if (num_experts < 1 || num_experts > 1024) return fail(TDIST_ELIMIT, "moe_gate_topk: at most 1024 experts");
    if (topk < 1 || topk > 32 || topk > num_experts) return fail(TDIST_EINVAL, "moe_gate_topk: topk must be in [1, min(32, experts)]");
    if (hidden < 32 || hidden % 32) return fail(TDIST_EINVAL, "moe_gate_topk: hidden must be a multiple of 32");
    if (reinterpret_cast<uintptr_t>(x) % 16 || reinterpret_cast<uintptr_t>(gate) % 16) return fail(TDIST_EINVAL, "moe_gate_topk: x and gate must be 16-byte aligned");
    if (ntok <= 0) return 0;
    // A cluster's SMs lie in one GPC: clusters of 2, 4 and 8 CTAs fill 100, 90 and 82 % of the machine (64 experts x 7168, experts shared
    // by 2 / 4 / 8 CTAs: 240 tokens 11.2 / 8.9 / 8.4 us, 300 tokens 11.3 / 9.0 / 15.6, 592 tokens 11.4 / 17.0 / 23.6). Chains are shared
    // out by eight CTAs of a tile where all run at once, the experts take one pass (64 tokens x 7168, 256 experts: 52 us, 11.4 by
    // experts), a chain has four steps or more (4 tokens x 1024, 64 experts: 4.7 us, 4.1 by experts; 100 x 2048, 32 experts 3.1 and
    // 3.8) and the products of the steps fit; by four CTAs up to 32 experts, where the experts have few CTAs to go to (cold, 300 tokens x
    // 4096: 8 experts 4.3 us, 6.3 on one CTA; 32 experts 5.5, 5.7 by experts; 64 experts 8.4 and 7.1). The experts are shared out
    // elsewhere, while each CTA gets some.
    const int tiles = (ntok + kGateTok - 1) / kGateTok, groups = (num_experts + 7) / 8;
    const int fit[4] = {100, 100, 90, 82};
    const auto runs_at_once = [&](int i) { return (100LL * tiles << i) <= static_cast<long long>(fit[i]) * tdist_host::sm_count(); };
    const auto width = [](int n) { return n <= 1 ? 1 : (n <= 2 ? 2 : (n <= 4 ? 4 : 8)); };
    static_assert(1 << 3 == kGateMaxParts, "the largest cluster");
    const auto chains_on = [&](int i) {
        return runs_at_once(i) && groups <= (i == 3 ? 8 : 4) && hidden >= 4 * kGateChains * 32 &&
               gate_chains_smem(hidden, width(groups), num_experts, 1 << i) <= 200 * 1024;
    };
    const bool chains = chains_on(3) || chains_on(2);
    int parts = chains ? (chains_on(3) ? 8 : 4) : 1;
    for (int i = 1; i <= 3 && parts < groups && !chains && runs_at_once(i); ++i) parts *= 2;
    const int nt = width(chains ? groups : (groups + parts - 1) / parts);
    const int smem = chains ? gate_chains_smem(hidden, nt, num_experts, parts)
                            : (kGateWarps * kGateTok * nt * 8 + kGateTok / parts * num_experts) * static_cast<int>(sizeof(float));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * parts));
    cfg.blockDim = dim3(kGateThreads);
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[2];
    attr[0] = tdist_host::pdl_attribute();
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(parts);
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = parts > 1 ? 2 : 1;
    const auto* xp = static_cast<const __nv_bfloat16*>(x);
    const auto* gp = static_cast<const __nv_bfloat16*>(gate);
    int* idp = static_cast<int*>(ids);
    float *wp = static_cast<float*>(weights), *lp = static_cast<float*>(logits);
#define TDIST_GATE_CASE(NT)                                                                                                              \
    {                                                                                                                                    \
        if (chains) {                                                                                                                    \
            const auto kernel = parts == 8 ? moe_gate_topk_chains_kernel<NT, 8> : moe_gate_topk_chains_kernel<NT, 4>;                    \
            if (int rc = ensure_smem(kernel, smem)) return rc;                                                                           \
            TDIST_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, xp, gp, ntok, hidden, num_experts, topk, renormalize, idp, wp, lp));          \
        } else {                                                                                                                         \
            const auto kernel = parts > 1 ? moe_gate_topk_kernel<NT, true> : moe_gate_topk_kernel<NT, false>;                            \
            if (int rc = ensure_smem(kernel, smem)) return rc;                                                                           \
            TDIST_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, xp, gp, ntok, hidden, num_experts, topk, renormalize, parts, idp, wp, lp));   \
        }                                                                                                                                \
    }
    if (nt == 1) TDIST_GATE_CASE(1)
    else if (nt == 2) TDIST_GATE_CASE(2)
    else if (nt == 4) TDIST_GATE_CASE(4)
    else TDIST_GATE_CASE(8)
#undef TDIST_GATE_CASE
    return 0;
}

extern "C" int tdist_gather_rows(const void* src, const void* index, int rows_out, int div, int limit, int row_bytes,
                                 void* dst, void* pos_of, void* stream) {
    if (row_bytes % 16 || div < 1) return fail(TDIST_EINVAL, "gather_rows: rows must be multiples of 16 bytes");
    if (rows_out <= 0) return 0;
    const int blocks = (rows_out + 7) / 8 < 1184 ? (rows_out + 7) / 8 : 1184;
    gather_rows_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(src), static_cast<const int*>(index), rows_out, div, limit, row_bytes / 16,
        static_cast<uint4*>(dst), static_cast<int*>(pos_of));
    TDIST_CUDA_OK(cudaGetLastError());
    return 0;
}

extern "C" int tdist_topk_reduce(const void* y, const void* pos_of, const void* weights, int ntok, int topk, int row_bytes,
                                 void* out, void* stream) {
    if (row_bytes % 16 || topk < 1) return fail(TDIST_EINVAL, "topk_reduce: rows must be multiples of 16 bytes");
    if (ntok <= 0 || row_bytes <= 0) return 0;
    const long long items = static_cast<long long>(ntok) * ((row_bytes / 16 + 32 * kReduceVecs - 1) / (32 * kReduceVecs));
    const int blocks = static_cast<int>((items + 7) / 8 < 1184 ? (items + 7) / 8 : 1184);
    TDIST_CUDA_OK(tdist_host::launch_pdl(topk_reduce_kernel, dim3(blocks), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(y),
                                         static_cast<const int*>(pos_of), static_cast<const float*>(weights), ntok, topk, row_bytes / 16,
                                         static_cast<uint4*>(out)));
    return 0;
}

// Logprobs of emitted tokens: for every row of RAW logits, log_softmax at the emitted token and the n_top most likely
// alternatives -- what engine/runtime/scheduler.py:714-722 computes with log_softmax + gather + topk (three full-vocabulary
// passes and a [r, V] temporary) -- in ONE pass over the row.
//
// Two 512-thread CTAs per SM walk over rows (persistent): every row costs the same, so the SM's rows split evenly, and
// while one CTA is in its short block-wide steps (the sample's bound, the selection of the alternatives) the other one
// streams.  Warp w owns a contiguous region of the row; lanes read 128-bit groups, four in flight per thread.  Each thread keeps an online (maximum, sum of exp) pair; the first batch
// of every warp (a tenth of the row at 151,936 logits) bounds the n_top-th largest logit from below, and the pass lists
// what reaches the bound (a few hundred logits), from which the exact top n_top are taken by rank, in descending order
// (equal logits: lower token first).  Up to 111 rows are shared by the CTAs of a cluster, whose first one merges the slices' maxima,
// sums and alternatives.  256 rows of 151,936 fp32 logits: 50.8 -> 47.7 us, 74 rows 35 -> 26 us.  A row whose lists overflow (long runs of equal logits) takes n_top extra passes.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <mutex>

#include "common.cuh"
#include "../../include/colinfer_b200.h"

namespace lpk {

constexpr int NT = 512, NW = NT / 32;
constexpr int CTAS_PER_SM = 2;
constexpr int BINS = 512;            // bins of the sample histogram and of the candidate selection
constexpr float SAMPLE_SCALE = 32.0f;
constexpr int WLIST = 128;           // list entries per warp
constexpr int FCAP = 128;            // candidates of the one-warp selection
constexpr int MAX_TOP = 32;          // n_top <= MAX_TOP
#define LP_FLT_MAX 3.402823466e38f
#define LP_POS_INF (__int_as_float(0x7f800000))

struct Cand { uint32_t idx; float l; };

struct Sc {
    float wm[32], ws[32];            // per-warp (maximum, sum)
    float wf[32];
    int wcount[32];
    int overflow;
    uint32_t fc_idx[FCAP]; float fc_l[FCAP];
    float sel_l; int sel_i;          // slow path: the previous pick
    float cm[8], cs[8];              // a cluster's first CTA: every CTA's (maximum, sum),
    uint32_t ct_idx[8 * MAX_TOP]; float ct_l[8 * MAX_TOP];   // and its slice's top n_top, in order
};

struct Row {
    const float* p32; const __nv_bfloat16* p16; int V; bool vec, vec16;
    __device__ __forceinline__ float4 load4(int i) const {
        if (vec) return i < V ? __ldcg(reinterpret_cast<const float4*>(p32 + i)) : make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
        if (vec16) {
            if (i >= V) return make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
            const uint2 u = __ldcg(reinterpret_cast<const uint2*>(p16 + i));        // four bf16: a float's upper halves
            return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u),
                               __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xFFFF0000u));
        }
        float e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int t = i + j;
            e[j] = t < V ? (p16 ? __bfloat162float(p16[t]) : __ldg(p32 + t)) : CI_NEG_INF;
        }
        return make_float4(e[0], e[1], e[2], e[3]);
    }
    __device__ __forceinline__ float at(int t) const { return p16 ? __bfloat162float(p16[t]) : __ldg(p32 + t); }
};

// (m, s) <- (m, s) + (m2, s2): sums of exp relative to their maxima
__device__ __forceinline__ void lse_merge(float& m, float& s, float m2, float s2) {
    const float M = fmaxf(m, m2);
    if (M == CI_NEG_INF) { s = 0.0f; return; }                      // both empty
    s = s * __expf(m - M) + s2 * __expf(m2 - M);                    // exp(-inf) = 0 for an empty side
    m = M;
}

// value descending, then token ascending
__device__ __forceinline__ bool before(float l1, uint32_t i1, float l2, uint32_t i2) { return l1 > l2 || (l1 == l2 && i1 < i2); }

__device__ __forceinline__ int warp_count_bin(const uint32_t* hist, uint32_t kk, int lane, uint32_t& run_out) {
    constexpr int PERB = BINS / 32;
    uint32_t h[PERB]; uint32_t s = 0;
#pragma unroll
    for (int t = 0; t < PERB; t += 4) {
        const uint4 x = *reinterpret_cast<const uint4*>(hist + lane * PERB + t);
        h[t] = x.x; h[t + 1] = x.y; h[t + 2] = x.z; h[t + 3] = x.w;
        s += x.x + x.y + x.z + x.w;
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += x; }
    const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
    if (all < kk) { run_out = all; return -1; }
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= kk);
    const int hl = __ffs(hit) - 1;
    uint32_t run = incl - s; int b = lane * PERB;
#pragma unroll
    for (int t = 0; t < PERB; ++t) { if (run + h[t] >= kk) { b = lane * PERB + t; run += h[t]; break; } run += h[t]; }
    run_out = __shfl_sync(0xffffffffu, run, hl);
    return __shfl_sync(0xffffffffu, b, hl);
}

struct Args {
    const void* logits; int dtype; int vec;
    const int64_t* toks; int n_top;
    float* chosen; int64_t* top_ids; float* top_lp;
    int rows, V;
};

// LOADER: 1 = fp32 rows that take 128-bit loads, 2 = bf16 rows that take 64-bit loads of four logits, 0 = the general
// loader (unaligned rows, vocabularies that are not a multiple of 4).
// CL: a cluster shares a row, a slice each; every CTA takes its slice's log-sum-exp and top n_top, the first one merges them.
template <int LOADER, bool CL>
__global__ void __launch_bounds__(NT, CTAS_PER_SM) k_logprobs(const __grid_constant__ Args a) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int V = a.V, n_top = a.n_top;
    __shared__ __align__(16) uint32_t hist[BINS];
    __shared__ Cand ownlist[NW * WLIST];
    __shared__ Sc sc;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = CL ? (int)cluster.num_blocks() : 1, crank = CL ? (int)cluster.block_rank() : 0;
    if (CL) cluster.barrier_arrive();                               // (waited for before the first write into a peer)
    bool running = false;
    // the row's groups of 128 logits, dealt evenly: a warp has a run of consecutive ones
    const int groups = (V + 127) / 128, part = crank * NW + warp;
    const int r_lo = min((int)((long long)groups * part / (C * NW)) * 128, V), r_hi = min((int)((long long)groups * (part + 1) / (C * NW)) * 128, V);
    Cand* mylist = ownlist + warp * WLIST;
    if (tid >= NW && tid < 32) {                                    // neutral entries for the warps this CTA does not have
        sc.wm[tid] = CI_NEG_INF; sc.ws[tid] = 0.0f; sc.wf[tid] = CI_NEG_INF; sc.wcount[tid] = -1;
    }

    for (int row = blockIdx.x / C; row < a.rows; row += gridDim.x / C) {
        __syncthreads();
        Row rw;
        rw.V = V; rw.vec = LOADER == 1; rw.vec16 = LOADER == 2;
        rw.p32 = a.dtype == COLINFER_F32 ? reinterpret_cast<const float*>(a.logits) + (size_t)row * V : nullptr;
        rw.p16 = a.dtype == COLINFER_BF16 ? reinterpret_cast<const __nv_bfloat16*>(a.logits) + (size_t)row * V : nullptr;

        // ------------------------------------------------------------------------------------ the sample's bound
        float tw = LP_POS_INF;                                      // n_top == 0: nothing to list
        if (n_top > 0) {
            float gm[4], sm = CI_NEG_INF;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = r_lo + k * 128 + lane * 4;
                const float4 v = i < r_hi ? rw.load4(i) : make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
                gm[k] = fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w));
                sm = fmaxf(sm, gm[k]);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) sm = fmaxf(sm, __shfl_xor_sync(0xffffffffu, sm, o));
            if (lane == 0) sc.wf[warp] = sm;
            for (int i = tid; i < BINS; i += NT) hist[i] = 0u;
            __syncthreads();
            // the bins hang from the smallest finite warp maximum plus 4: a dominant token in the sample (far above
            // everything else) must not stretch them beyond the bulk
            float lref = sc.wf[lane];
            float lbulk = lref > CI_NEG_INF ? lref : LP_POS_INF;
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                lref = fmaxf(lref, __shfl_xor_sync(0xffffffffu, lref, o));
                lbulk = fminf(lbulk, __shfl_xor_sync(0xffffffffu, lbulk, o));
            }
            const float top = fminf(lbulk + 4.0f, lref);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (gm[k] > CI_NEG_INF && top < LP_POS_INF)
                    atomicAdd(&hist[max(0, min(BINS - 1, __float2int_rz((top - gm[k]) * SAMPLE_SCALE)))], 1u);
            __syncthreads();
            uint32_t have;
            const int bk = warp_count_bin(hist, (uint32_t)n_top, lane, have);
            tw = (bk >= 0 && bk < BINS - 1) ? top - ((float)(bk + 1) + 0.01f) / SAMPLE_SCALE - fabsf(top) * 1e-6f : -LP_FLT_MAX;
            __syncthreads();                                        // every warp has read the sample's bins
        }

        // ------------------------------------------------------------------------------------ the pass
        float m = CI_NEG_INF, s = 0.0f;
        int wn = 0;
        // (the next batch is under way while this one is worked on: with one batch in flight a warp's nineteen round trips to
        // HBM are most of the row's time)
        float4 nv[4];
        auto fetch = [&](int i0) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = i0 + k * 128 + lane * 4;
                nv[k] = i < r_hi ? rw.load4(i) : make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
            }
        };
        fetch(r_lo);
#pragma unroll 1
        for (int i0 = r_lo; i0 < r_hi; i0 += 512) {
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = nv[k];
            fetch(i0 + 512);
            float bm = CI_NEG_INF;
#pragma unroll
            for (int k = 0; k < 4; ++k) bm = fmaxf(bm, fmaxf(fmaxf(v[k].x, v[k].y), fmaxf(v[k].z, v[k].w)));
            if (bm > m) { s = m > CI_NEG_INF ? s * __expf(m - bm) : 0.0f; m = bm; }
            if (m > CI_NEG_INF) {
                float add = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    add += (__expf(v[k].x - m) + __expf(v[k].y - m)) + (__expf(v[k].z - m) + __expf(v[k].w - m));
                s += add;
            }
            unsigned mk[4], anym = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                mk[k] = (v[k].x >= tw ? 1u : 0u) | (v[k].y >= tw ? 2u : 0u) | (v[k].z >= tw ? 4u : 0u) | (v[k].w >= tw ? 8u : 0u);
                anym |= mk[k];
            }
            if (__ballot_sync(0xffffffffu, anym != 0u)) {
                // per-lane counts of the four groups, one byte each; one packed scan gives every group's offsets
                const unsigned cnt = __popc(mk[0]) | (__popc(mk[1]) << 8) | (__popc(mk[2]) << 16) | (__popc(mk[3]) << 24);
                unsigned incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const unsigned t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
                const unsigned tot = __shfl_sync(0xffffffffu, incl, 31), excl = incl - cnt;
                int base = wn;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (mk[k]) {
                        int at = base + (int)((excl >> (8 * k)) & 0xFFu);
                        const float e4[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (mk[k] & (1u << j)) {
                                if (at < WLIST) { mylist[at].idx = (uint32_t)(i0 + k * 128 + lane * 4 + j); mylist[at].l = e4[j]; }
                                ++at;
                            }
                        }
                    }
                    base += (int)((tot >> (8 * k)) & 0xFFu);
                }
                wn = base;
            }
        }

        // ------------------------------------------------------------------------------------ log-sum-exp of the row
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
            lse_merge(m, s, m2, s2);
        }
        if (lane == 0) { sc.wm[warp] = m; sc.ws[warp] = s; }
        for (int i = tid; i < BINS; i += NT) hist[i] = 0u;
        if (lane == 0) sc.wcount[warp] = wn;
        const int over = __syncthreads_or(wn > WLIST);
        float M = sc.wm[lane], S = sc.ws[lane];
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float m2 = __shfl_xor_sync(0xffffffffu, M, o), s2 = __shfl_xor_sync(0xffffffffu, S, o);
            lse_merge(M, S, m2, s2);
        }
        // (of a slice with nothing in it 0: only the merged value counts)
        const float lse = CL ? 0.0f : M + logf(S);                              // -inf + log(0) = NaN for a row without finite logits
        auto put = [&](int rank, uint32_t idx, float l) {           // the slice's alternative of that rank
            if (CL) { Sc* first = cluster.map_shared_rank(&sc, 0); first->ct_idx[crank * MAX_TOP + rank] = idx; first->ct_l[crank * MAX_TOP + rank] = l; }
            else { a.top_ids[(size_t)row * n_top + rank] = idx == 0xFFFFFFFFu ? -1ll : (long long)idx; a.top_lp[(size_t)row * n_top + rank] = l - lse; }
        };
        if (CL) {
            if (!running) { cluster.barrier_wait(); running = true; }
            if (tid == 0) { Sc* first = cluster.map_shared_rank(&sc, 0); first->cm[crank] = M; first->cs[crank] = S; }
        } else if (tid == 0 && a.chosen) {
            const long long t = a.toks ? a.toks[row] : -1;
            a.chosen[row] = (t >= 0 && t < V) ? rw.at((int)t) - lse : __int_as_float(0x7fc00000);
        }
        if (!CL && n_top <= 0) continue;

        // ------------------------------------------------------------------------------------ the top n_top
        bool done = n_top <= 0;
        const bool usable = !done && !over && tw > -LP_FLT_MAX && tw <= M;
        const int listed = __reduce_add_sync(0xffffffffu, lane < NW ? sc.wcount[lane] : 0);
        if (usable && listed >= n_top && listed <= FCAP) {
            // few enough to be ranked as they are: every one against all others, four threads each
            const int off = __reduce_add_sync(0xffffffffu, lane < warp ? sc.wcount[lane] : 0);
            for (int j = lane; j < wn; j += 32) { sc.fc_idx[off + j] = mylist[j].idx; sc.fc_l[off + j] = mylist[j].l; }
            __syncthreads();
            const int c = tid / 4;
            int rank = 0;
            if (c < listed) {
                const float lc = sc.fc_l[c]; const uint32_t ic = sc.fc_idx[c];
                for (int o = tid & 3; o < listed; o += 4) rank += before(sc.fc_l[o], sc.fc_idx[o], lc, ic) ? 1 : 0;
            }
            rank += __shfl_xor_sync(0xffffffffu, rank, 1);
            rank += __shfl_xor_sync(0xffffffffu, rank, 2);
            if (c < listed && (tid & 3) == 0 && rank < n_top) put(rank, sc.fc_idx[c], sc.fc_l[c]);
            done = true;
        } else if (usable) {
            __syncthreads();                                        // (the counts have been read)
            const float scale = M > tw ? (float)(BINS - 2) / (M - tw) : 0.0f;
            auto bin_of = [&](float l) { return min(BINS - 1, __float2int_rz((M - l) * scale)); };
            for (int j = lane; j < wn; j += 32) atomicAdd(&hist[bin_of(mylist[j].l)], 1u);
            __syncthreads();
            uint32_t nc;
            const int bstar = warp_count_bin(hist, (uint32_t)n_top, lane, nc);
            if (bstar >= 0 && (int)nc <= FCAP) {
                int cnt = 0;
                for (int j0 = 0; j0 < wn; j0 += 32) {
                    const int j = j0 + lane;
                    cnt += __popc(__ballot_sync(0xffffffffu, j < wn && bin_of(mylist[j].l) <= bstar));
                }
                if (lane == 0) sc.wcount[warp] = cnt;
                __syncthreads();
                int off = 0;
                for (int w2 = 0; w2 < warp; ++w2) off += sc.wcount[w2];
                const unsigned lt = (1u << lane) - 1u;
                for (int j0 = 0; j0 < wn; j0 += 32) {
                    const int j = j0 + lane;
                    const bool is = j < wn && bin_of(mylist[j].l) <= bstar;
                    const unsigned bal = __ballot_sync(0xffffffffu, is);
                    if (is) { const int at = off + __popc(bal & lt); if (at < FCAP) { sc.fc_idx[at] = mylist[j].idx; sc.fc_l[at] = mylist[j].l; } }
                    off += __popc(bal);
                }
                __syncthreads();
                {
                    // rank of every candidate among the candidates (value descending, then token ascending): a few threads
                    // per candidate compare it with a share of the others each; a candidate of rank < n_top is that alternative
                    constexpr int TPC = NT / FCAP;                  // threads per candidate
                    static_assert(TPC == 4 || TPC == 8, "four or eight threads per candidate");
                    const int c = tid / TPC, part = tid % TPC;
                    int rank = 0;
                    if (c < (int)nc) {
                        const float lc = sc.fc_l[c]; const uint32_t ic = sc.fc_idx[c];
#pragma unroll
                        for (int t = 0; t < FCAP / TPC; ++t) {
                            const int o = part * (FCAP / TPC) + t;
                            if (o < (int)nc && before(sc.fc_l[o], sc.fc_idx[o], lc, ic)) ++rank;
                        }
                    }
                    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
                    rank += __shfl_xor_sync(0xffffffffu, rank, 2);
                    if (TPC == 8) rank += __shfl_xor_sync(0xffffffffu, rank, 4);
                    if (part == 0 && c < (int)nc && rank < n_top) {
                        put(rank, sc.fc_idx[c], sc.fc_l[c]);
                    }
                }
                done = true;
            }
        }
        if (!done) {
            // lists overflowed (long runs of equal logits) or the bound did not hold: n_top passes, each taking the
            // best logit after the previous pick in (value descending, token ascending) order
            if (tid == 0) { sc.sel_l = LP_POS_INF; sc.sel_i = -1; }
            __syncthreads();
            for (int r = 0; r < n_top; ++r) {
                const float pl = sc.sel_l; const uint32_t pi = (uint32_t)sc.sel_i;
                const bool first = sc.sel_i == -1, none = sc.sel_i == -2;   // none: the slice has no further logits
                float bl = CI_NEG_INF; uint32_t bi = 0xFFFFFFFFu;
                for (int i0 = r_lo; i0 < r_hi; i0 += 128) {
                    const int i = i0 + lane * 4;
                    const float4 v = rw.load4(i);
                    const float e4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t id = (uint32_t)(i + j);
                        if (i + j < V && !none && (first || before(pl, pi, e4[j], id)) && (bi == 0xFFFFFFFFu || before(e4[j], id, bl, bi))) { bl = e4[j]; bi = id; }
                    }
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    const float ol = __shfl_xor_sync(0xffffffffu, bl, o);
                    const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (oi != 0xFFFFFFFFu && (bi == 0xFFFFFFFFu || before(ol, oi, bl, bi))) { bl = ol; bi = oi; }
                }
                __syncthreads();
                if (lane == 0) { sc.wf[warp] = bl; sc.wcount[warp] = (int)bi; }
                __syncthreads();
                if (warp == 0) {
                    float cl = sc.wf[lane]; uint32_t ci = (uint32_t)sc.wcount[lane];
#pragma unroll
                    for (int o = 16; o; o >>= 1) {
                        const float ol = __shfl_xor_sync(0xffffffffu, cl, o);
                        const uint32_t oi = __shfl_xor_sync(0xffffffffu, ci, o);
                        if (oi != 0xFFFFFFFFu && (ci == 0xFFFFFFFFu || before(ol, oi, cl, ci))) { cl = ol; ci = oi; }
                    }
                    if (lane == 0) {
                        sc.sel_l = cl; sc.sel_i = ci == 0xFFFFFFFFu ? -2 : (int)ci;
                        put(r, ci, cl);
                    }
                }
                __syncthreads();
            }
        }
        if (CL) {
            // ------------------------------------------------------------------------------------ the first CTA merges
            cluster.sync();
            if (crank == 0) {
                M = sc.cm[0]; S = sc.cs[0];
                for (int q = 1; q < C; ++q) lse_merge(M, S, sc.cm[q], sc.cs[q]);
                const float all = M + logf(S);
                if (tid == 0 && a.chosen) {
                    const long long t = a.toks ? a.toks[row] : -1;
                    a.chosen[row] = (t >= 0 && t < V) ? rw.at((int)t) - all : __int_as_float(0x7fc00000);
                }
                // two threads per candidate count those before it
                const int e = tid >> 1, q = e / MAX_TOP, j = e % MAX_TOP;
                int rank = 0;
                const bool is = q < C && j < n_top;
                if (is) {
                    const float l = sc.ct_l[e]; const uint32_t x = sc.ct_idx[e];
                    for (int o = tid & 1; o < C * n_top; o += 2) {
                        const int f = (o / n_top) * MAX_TOP + o % n_top;
                        if (f != e && (before(sc.ct_l[f], sc.ct_idx[f], l, x) || (f < e && sc.ct_l[f] == l && sc.ct_idx[f] == x))) ++rank;
                    }
                }
                rank += __shfl_xor_sync(0xffffffffu, rank, 1);
                if (is && !(tid & 1) && rank < n_top) {
                    const uint32_t x = sc.ct_idx[e];
                    a.top_ids[(size_t)row * n_top + rank] = x == 0xFFFFFFFFu ? -1ll : (long long)x;
                    a.top_lp[(size_t)row * n_top + rank] = sc.ct_l[e] - all;
                }
            }
            cluster.sync();
        }
    }
    if (CL && !running) cluster.barrier_wait();
}

}  // namespace lpk

// Replaces Scheduler._logprobs (engine/runtime/scheduler.py:714-722).
extern "C" int colinfer_logprobs(const void* logits, int dtype, const int64_t* toks, int n_top, float* chosen,
                                 int64_t* top_ids, float* top_lp, int rows, int V, void* stream) {
    if (rows == 0) return (int)cudaSuccess;
    if (logits == nullptr || rows < 0 || V < 1 || n_top < 0 || n_top > lpk::MAX_TOP || n_top > V ||
        (dtype != COLINFER_F32 && dtype != COLINFER_BF16) || (n_top > 0 && (top_ids == nullptr || top_lp == nullptr)))
        return (int)cudaErrorInvalidValue;
    static int sm_count[64] = {};
    static std::mutex guard;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lock(guard);
        if (sm_count[dev] == 0) {
            int n = 0;
            e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return (int)e;
            sm_count[dev] = n > 0 ? n : 1;
        }
    }
    lpk::Args a;
    a.logits = logits; a.dtype = dtype;
    a.vec = (dtype == COLINFER_F32 && (V % 4) == 0 && (((uintptr_t)logits) & 15) == 0) ? 1 : 0;
    a.toks = toks; a.n_top = n_top; a.chosen = chosen; a.top_ids = top_ids; a.top_lp = top_lp;
    a.rows = rows; a.V = V;
    const int slots = sm_count[dev] * lpk::CTAS_PER_SM;
    const bool vec16 = dtype == COLINFER_BF16 && (V % 4) == 0 && (((uintptr_t)logits) & 7) == 0;
    const int loader = a.vec ? 1 : vec16 ? 2 : 0;
    // Fewer rows than half the CTAs the device holds (three quarters of them, as clusters): a cluster of 8, 4 or 2 shares a row, as far as its slices have a batch for
    // every warp or so (one row of 151,936 logits took 29 us in one CTA).
    int C = 8;
    while (C > 1 && ((long long)rows * C > slots * 3 / 4 || V < 4096 * C)) C /= 2;
    if (C > 1) {
        const void* const kernels[3] = {(const void*)lpk::k_logprobs<0, true>, (const void*)lpk::k_logprobs<1, true>, (const void*)lpk::k_logprobs<2, true>};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(rows * C), 1, 1);
        cfg.blockDim = dim3(lpk::NT, 1, 1);
        cfg.stream = (cudaStream_t)stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)C;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        void* args[] = {&a};
        return (int)cudaLaunchKernelExC(&cfg, kernels[loader], args);
    }
    const int grid = rows < slots ? rows : slots;
    if (loader == 1) lpk::k_logprobs<1, false><<<grid, lpk::NT, 0, (cudaStream_t)stream>>>(a);
    else if (loader == 2) lpk::k_logprobs<2, false><<<grid, lpk::NT, 0, (cudaStream_t)stream>>>(a);
    else lpk::k_logprobs<0, false><<<grid, lpk::NT, 0, (cudaStream_t)stream>>>(a);
    return (int)cudaGetLastError();
}

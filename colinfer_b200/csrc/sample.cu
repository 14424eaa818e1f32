// sample.cu -- the fused logits -> token kernel (sm_100a).
//
// One thread-block cluster per row.  Each CTA of the cluster copies its slice of the row from HBM into its own shared
// memory exactly once (1-D bulk copies completed on mbarriers when the row is 16-byte aligned fp32, plain loads
// otherwise) and the whole row stays resident in the cluster's distributed shared memory.  Everything after that --
// penalties, grammar mask, row maximum / argmax, the min-p / top-k / top-p threshold selects and the inverse-CDF draw --
// works on shared memory, so HBM is read once per row whatever the sampling parameters are.
//
// Selection is exact.  The kept set is always {logit >= threshold}.  Masses are exp(z - max) rounded to integers in
// units of 2^-30 and summed as integers, so every sum, every cumulative-mass crossing and the CDF crossing are
// independent of thread, CTA and cluster geometry and of the other rows in the launch (the reference's row-invariance
// property).  How the threshold is found depends on the row's parameters:
//   top_k <= 100   each CTA bounds its slice's k-th largest logit from below with a histogram of its threads' maxima,
//                  collects the few logits above that bound in token order, and the cluster's first CTA finishes
//                  top-k, top-p and the draw exactly on the gathered list (two cluster barriers in all);
//   larger top_k   a fine count histogram over the distance from the row maximum (4096 buckets, reduced across the
//                  cluster) gives the bucket of the k-th largest logit; the logits down to it are gathered as above;
//   top_p alone    the same histogram with per-bucket mass estimates gives the bucket of the top-p pivot approximately;
//                  one pass sums the exact mass above a narrow band around it and gathers the band, the pivot is found
//                  exactly on the list, and the draw walks the row once more only inside one warp's region;
//   neither        one mass pass and the draw.
// If a list would overflow, or the estimated band misses the true pivot, an exact select over the order-preserving 32-bit keys
// runs instead: a pass over the resident slices per 1,024-fold narrowing (slower, same result).
//
// What bounds it is latency: one row's chain of block-wide steps, and code that every step executes for the first time, not bytes
// (one row, top_k 50: of the warps' stall cycles 43 % are waits at barriers, 23 % instruction fetches).  So: one CTA of 512 threads per SM (with 256 the passes over a slice took
// twice as long, at 1,024 there are too few registers), searches repeated by every warp instead of published by one, sums pushed to the peers before a
// barrier instead of fetched after it, masses two logits per instruction, 64-bit shared-memory additions as 32-bit ones with a
// carry.  One fp32 row of 151,936 logits on a B200, device time: top_k 100 23.1 -> 16.5 us, top-p alone 33.5 -> 26 us, no filter
// 14.5 -> 12 us; four rows with a grammar mask 21.5 -> 13.8 us.
//
// What the reference does in ~25 torch / FlashInfer launches per slot (engine/spec/accept.py:23-52 after
// engine/runtime/sampler.py:50-56) is one launch here.
#include <mutex>

#include "common.cuh"
#include "host_util.h"
#include "sample_host.h"
#include "../../include/colinfer_b200.h"

#define CI_THREADS 512
#define CI_WARPS (CI_THREADS / 32)
#define CI_CHUNK 4096            // elements per bulk copy
#define CI_MAX_CHUNKS 16
#define CI_NB1 4096              // fine buckets over the distance from the row maximum
#define CI_TOP 2.0f              // logits up to CI_TOP * temperature below the maximum correct a row's estimated mass
#define CI_RANGE 25.0f           // the buckets cover distances up to CI_RANGE * temperature
#define CI_FASTK 100             // largest top_k handled by the per-slice candidate lists
#define CI_FAST_BINS 512         // bins of the thread-maxima histogram and of the exact finish
#define CI_TGROUPS 4              // maxima each thread keeps (interleaved groups of its elements) for the top-k bound
#define CI_FIN_MAX 1024          // candidates of one row at the CTA that finishes it (8 x CI_PCAP)
#define CI_FAST_SCALE 32.0f      // its bins per unit logit (covers 16 units below the slice maximum)
#define CI_PCAP 128              // candidates one CTA may push to the CTA that finishes the row
#define CI_FIN_KEEP 128          // candidates that may be left after top-k
#define CI_FIN_CAND 64           // candidates of one bin examined pairwise
#define CI_RETRY 8               // rows a CTA may set aside for the generic path before the fast path is switched off
#define CI_WLIST 24              // list entries per warp of a cluster of eight (in smaller ones as many more as there are fewer warps: SampleArgs::list_cap)
#define CI_GLIST 1365            // gathered list entries (16 KB)
#define CI_SEL_BINS 256          // coarse bins of the exact selection on a gathered list
#define CI_FB_NB 1024             // buckets per level of the fallback select
#define CI_MAX_CAND 128          // tied / neighbouring candidates examined one by one in the final list step
#define CI_PEN_TABLE 2048        // distinct history ids per slice with an O(1) count
#define CI_WAIT_CYCLES 400000000LL
#define CI_FLT_MAX 3.402823466e38f
#define CI_POS_INF (__int_as_float(0x7f800000))

struct SampleArgs {
    const void* logits; int dtype; int use_bulk;
    const int32_t* mask; int mask_rows; int W;
    colinfer_sampler_params p;
    const void* pos; int pos_i64; const float* u;
    int64_t* out; colinfer_row_stats* stats; int32_t* status;
    int B, R, V; int slice_elems; int list_cap; int flags;
    colinfer_second_rows second;
    long long* prof; int prof_slots;   // optional per-CTA phase timestamps (profiling hook)
};
// Profiling hook: thread 0 adds the cycles since its previous marker to the slot's total (summed over the CTA's rows).
#define CI_PROF(slot) do { if (a.prof && tid == 0) { const long long t_ = clock64(); sc->prof[slot] += t_ - prof_last; prof_last = t_; } } while (0)

#define CI_PROF_END() do { if (a.prof && tid == 0 && (int)blockIdx.x < a.prof_slots) { \
    unsigned long long gt; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(gt)); \
    a.prof[(size_t)blockIdx.x * 16 + 13] = (long long)gt; a.prof[(size_t)blockIdx.x * 16 + 12] = clock64() - prof_t0; \
    for (int i = 0; i < 12; ++i) a.prof[(size_t)blockIdx.x * 16 + i] = sc->prof[i]; } } while (0)

struct ListEntry { uint32_t idx; float l; uint32_t q; };   // gathered list: token, logit, mass
struct Cand { uint32_t idx; float l; };                      // a warp's list / pushed candidates: token, logit

// A row whose candidates have been pushed to this CTA and that waits for its exact finish.
struct Pending { int row; float L; int aidx; int status; int kk; float tc, topp, lmp, u; int count[8]; };

// What every CTA writes into each peer's shared memory before the first cluster barrier.
struct Hello { float lmax; int lidx; int flags; int pad; };   // flags: 1 = a bounded wait gave up, 4 = slow history path, 8 = stop using the fast path; pad: candidates pushed

// Values one CTA publishes in its own shared memory for its peers to read after a later barrier.
struct Xch {
    u64 fb_segtot;                 // the same for the fallback radix select
    u64 cta_mass;                  // kept mass of the slice under the final threshold
    unsigned short wcount[CI_WARPS];   // entries in each warp's list
    int list_overflow;
};

struct Scratch {
    Hello hello[2][8];             // written by the peers, one set per row parity
    u64 warp_tot[CI_WARPS];
    u64 warp_aux[CI_WARPS];
    float warp_f[CI_WARPS]; int warp_i[CI_WARPS];
    uint32_t warp_u[CI_WARPS], warp_v[CI_WARPS];
    unsigned short pcount[8 * CI_WARPS]; unsigned short poff[8 * CI_WARPS + 1];
    int found_idx; u64 found_before;
    int ncand; float sel_value; int sel_ok;
    int fail;
    int hist_slow;
    u64 wsum[CI_WARPS], woff[CI_WARPS], wtotal;   // block scan
    int found_tid; u64 found_excl;
    float cand_l[CI_FIN_CAND]; float res_f;
    Pending pend;
    int n_retry_common, n_retry_mine, any_retry, want_fast_off;   // any_retry: a CTA of the cluster has set a row aside
    int retry_common[CI_RETRY], retry_mine[CI_RETRY], retry_all[CI_RETRY * 9];
    long long prof[12];            // profiling hook: cycles per phase, summed over the CTA's rows
    u64 seg_off[8];                // ... and what the estimates are off by on the largest logits
    u64 seg_cnt[8], seg_est[8];    // totals of every CTA's reduced bucket segment, written by the peers: counts, estimated mass
    u64 all_in[8], above_in[8];    // band pass: kept mass of every CTA's slice, and of its part above the band, written by the peers
    int bcast_i[2];                // written by the cluster's first CTA, per row parity
    u64 mass_in[2][8];             // kept mass of every CTA's slice, written by the peers, per row parity
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ int warp_id() { return threadIdx.x >> 5; }

// Maximum over a warp; NaN counts as less than everything else.
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Block-wide: index of the first entry (ascending) at which the running sum of get(0..n-1) reaches `target`
// (1 <= target <= total), and the sum before it.  All threads call; all threads get the result.
template <class F>
__device__ void block_find(F get, int n, u64 target, Scratch* s, int& idx, u64& before) {
    const int ipt = (n + CI_THREADS - 1) / CI_THREADS;
    const int lo = threadIdx.x * ipt;
    u64 local = 0;
    for (int i = lo; i < lo + ipt && i < n; ++i) local += get(i);
    const u64 incl = warp_incl_scan_u64(local, lane_id());
    if (threadIdx.x == 0) { s->found_idx = n - 1; s->found_before = 0; }
    if (lane_id() == 31) s->warp_tot[warp_id()] = incl;
    __syncthreads();
    u64 off = 0;
    for (int w = 0; w < warp_id(); ++w) off += s->warp_tot[w];
    u64 excl = off + incl - local;
    if (excl < target && target <= excl + local) {
        for (int i = lo; i < lo + ipt && i < n; ++i) {
            const u64 v = get(i);
            if (excl + v >= target) { s->found_idx = i; s->found_before = excl; break; }
            excl += v;
        }
    }
    __syncthreads();
    idx = s->found_idx;
    before = s->found_before;
    __syncthreads();
}

__device__ u64 block_sum_u64(u64 v, Scratch* s) {
    v = warp_sum_u64(v);
    if (lane_id() == 0) s->warp_tot[warp_id()] = v;
    __syncthreads();
    u64 t = 0;
    for (int w = 0; w < CI_WARPS; ++w) t += s->warp_tot[w];
    __syncthreads();
    return t;
}


// Estimated mass (units of 2^-30) of one element in distance bucket b: exp(-(b + 0.5) * CI_RANGE / CI_NB1).
__device__ __forceinline__ u64 bucket_mass_est(int b) {
    return (u64)__float2uint_rn(exp2f(-((float)b + 0.5f) * (CI_RANGE * CI_LOG2E / (float)CI_NB1)) * CI_MASS_SCALE);
}

__device__ __forceinline__ u64 ceil_target(float frac, u64 total) {
    const double t = ceil((double)frac * (double)total);
    u64 q = t <= 1.0 ? 1ull : (u64)t;
    return q > total ? total : q;
}

// The row's uniform in (0, 1]: explicit, or Philox keyed by (seed, position + row of the slot), or 1 when no draw is asked.
__device__ __forceinline__ float row_uniform(const SampleArgs& a, int row, int b, int r) {
    if (row >= a.second.rows1) return 1.0f;
    if (a.u != nullptr) return a.u[row];
    if (a.pos != nullptr && a.p.seed != nullptr) {
        const long long p0 = a.pos_i64 ? reinterpret_cast<const long long*>(a.pos)[b]
                                       : (long long)reinterpret_cast<const int*>(a.pos)[b];
        return u32_to_uniform(philox_word(philox_key(a.p.seed[b]), (u64)p0 + (u64)r));
    }
    return 1.0f;
}

// Bin of 32 * PER bins (ascending index) in which the running sum reaches `target` (1 <= target), and the sum before it;
// bin = 32 * PER when the total falls short.  Every warp searches for itself: cheaper than publishing one warp's result.
template <int PER, class T, class S>
__device__ __forceinline__ void warp_find(const T* bins, S target, int& bin, S& before) {
    const int lane = lane_id();
    S loc[PER], sum = 0;
    constexpr int STEP = 16 / sizeof(T);
#pragma unroll
    for (int t = 0; t < PER; t += STEP) {
        const uint4 x = *reinterpret_cast<const uint4*>(bins + lane * PER + t);
        if constexpr (sizeof(T) == 4) { loc[t] = x.x; loc[t + 1] = x.y; loc[t + 2] = x.z; loc[t + 3] = x.w; }
        else { loc[t] = ((u64)x.y << 32) | x.x; loc[t + 1] = ((u64)x.w << 32) | x.z; }
    }
#pragma unroll
    for (int t = 0; t < PER; ++t) sum += loc[t];
    S incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const S x = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += x; }
    const unsigned reached = __ballot_sync(0xffffffffu, incl >= target);
    if (!reached) { bin = 32 * PER; before = 0; return; }
    const int src = __ffs(reached) - 1;
    S run = incl - sum, run_at = run;
    int at = PER - 1;
    bool found = false;
#pragma unroll
    for (int t = 0; t < PER; ++t) { if (!found && run + loc[t] >= target) { found = true; at = t; run_at = run; } run += loc[t]; }
    bin = src * PER + __shfl_sync(0xffffffffu, at, src);
    before = __shfl_sync(0xffffffffu, run_at, src);
}

// Block-wide, one value per thread: the first thread at which the running sum reaches `target` (1 <= target <= total), and the
// sum before it.  Two block barriers.
__device__ __forceinline__ void thread_find(u64 v, u64 target, Scratch* s, int& idx, u64& before) {
    const int lane = lane_id(), warp = warp_id();
    const u64 incl = warp_incl_scan_u64(v, lane);
    if (lane == 31) s->wsum[warp] = incl;
    if (threadIdx.x == 0) { s->found_idx = CI_THREADS - 1; s->found_before = 0; }
    __syncthreads();
    const u64 excl = warp_sum_u64(lane < warp ? s->wsum[lane] : 0ull) + incl - v;
    if (excl < target && target <= excl + v) { s->found_idx = threadIdx.x; s->found_before = excl; }
    __syncthreads();
    idx = s->found_idx; before = s->found_before;
}

// Exact weighted selection on a gathered list: the value v among the entries with wt > 0 such that
// W(l > v) < target <= W(l >= v).  Coarse bins over the entries' key range (a shift, so monotone), then the entries of the
// pivot bin pairwise (by every warp).  Returns false when the pivot bin holds more than CI_MAX_CAND entries.  All threads of
// the CTA call; 1 <= target <= total weight.
template <class W>
__device__ __noinline__ bool list_select(const ListEntry* gl, int n, W wt, u64 target, u64* bins, uint32_t* cand, Scratch* sc, float& value) {
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    uint32_t kmin = 0xFFFFFFFFu, kmax = 0u;
    for (int i = tid; i < n; i += CI_THREADS) {
        if (wt(i) > 0) { const uint32_t k = f2key(gl[i].l); kmin = min(kmin, k); kmax = max(kmax, k); }
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin); kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) { sc->warp_u[warp] = kmin; sc->warp_v[warp] = kmax; }
    for (int i = tid; i < CI_SEL_BINS; i += CI_THREADS) bins[i] = 0;
    if (tid == 0) sc->ncand = 0;
    __syncthreads();
    kmin = __reduce_min_sync(0xffffffffu, sc->warp_u[lane % CI_WARPS]); kmax = __reduce_max_sync(0xffffffffu, sc->warp_v[lane % CI_WARPS]);
    const int sh = max(0, 32 - __clz(kmax - kmin) - 8);                  // the bins cover [0, kmax - kmin] >> sh
    for (int i = tid; i < n; i += CI_THREADS) {
        const u64 w = wt(i);
        if (w > 0) add64(&bins[(kmax - f2key(gl[i].l)) >> sh], w);
    }
    __syncthreads();
    int b_star; u64 before;
    warp_find<CI_SEL_BINS / 32>(bins, target, b_star, before);
    for (int i = tid; i < n; i += CI_THREADS) {
        if (wt(i) > 0 && (int)((kmax - f2key(gl[i].l)) >> sh) == b_star) {
            const int slot = atomicAdd(&sc->ncand, 1);
            if (slot < CI_MAX_CAND) cand[slot] = (uint32_t)i;
        }
    }
    __syncthreads();
    const int nc = sc->ncand;
    bool ok = false;
    if (nc <= CI_MAX_CAND) {
        for (int c0 = 0; c0 < nc && !ok; c0 += 32) {
            const float mine = c0 + lane < nc ? gl[cand[c0 + lane]].l : CI_NEG_INF;
            u64 gt = before, ge = before;
            for (int j = 0; j < nc; ++j) {                               // only the pivot bin's entries matter
                const int e = (int)cand[j];
                const float o = gl[e].l; const u64 w = wt(e);
                gt += o > mine ? w : 0ull; ge += o >= mine ? w : 0ull;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, c0 + lane < nc && gt < target && target <= ge);
            if (hit) { ok = true; value = __shfl_sync(0xffffffffu, mine, __ffs(hit) - 1); }
        }
    }
    __syncthreads();
    return ok;
}

// Exact select among the keys [klo, khi] of the row, across the cluster: a pass over the slices per 1,024-fold narrowing of the
// bracket.  by_mass: where the descending cumulative mass reaches `target` (0: top_p of the bracket's mass); else the target-th
// largest.  coarse: every logit is a bf16, of which any 2^16 neighbouring keys hold one.  Returns false when the bracket falls
// short of the target (a top-k that removes nothing); else pivot holds the pivot logit.  Every CTA of the cluster calls it with
// identical arguments and takes identical decisions.
struct RadixCtx {
    const float* rowbuf; int n_pad; u64* fb_hist; u64* fb_seg; Xch* xch; Scratch* sc; int rank, CS;
};
__device__ __noinline__ bool radix_select(cg::cluster_group& cluster, const RadixCtx& c, const MassFn& mass, uint32_t klo, uint32_t khi,
                                          bool coarse, bool by_mass, u64 target, float topp, float& pivot) {
    const int tid = threadIdx.x;
    for (int lvl = 0; lvl < 5; ++lvl) {
        const uint32_t span = khi - klo;
        if (lvl && span < (coarse ? 65536u : 1u)) {
            uint32_t k = khi;
            if (coarse) k = khi >= 0x80000000u && (khi & 0xFFFF0000u) >= klo ? khi & 0xFFFF0000u : ((khi + 1u) & 0xFFFF0000u) - 1u;
            pivot = key2f(k);
            return true;
        }
        const int sh = max(coarse ? 16 : 0, 22 - __clz(span));            // at most CI_FB_NB bins
        __syncthreads();
        for (int i = tid; i < CI_FB_NB; i += CI_THREADS) c.fb_hist[i] = 0;
        __syncthreads();
        const float4* row4 = reinterpret_cast<const float4*>(c.rowbuf);
        for (int i = tid; i * 4 < c.n_pad; i += CI_THREADS) {
            const float4 v = row4[i];
            const float e4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t key = f2key(e4[j]);
                if (key >= klo && key <= khi) add64(&c.fb_hist[(khi - key) >> sh], by_mass ? (u64)mass(e4[j]) : 1ull);
            }
        }
        __syncthreads();
        cluster.sync();                                                    // local histograms complete
        const int G = CI_FB_NB / c.CS;
        u64 part = 0;
        for (int g = tid; g < G; g += CI_THREADS) {
            u64 sum = 0;
            for (int q = 0; q < c.CS; ++q) sum += cluster.map_shared_rank(c.fb_hist, q)[c.rank * G + g];
            c.fb_seg[g] = sum;
            part += sum;
        }
        const u64 tot = block_sum_u64(part, c.sc);
        if (tid == 0) c.xch->fb_segtot = tot;
        __syncthreads();
        cluster.sync();                                                    // reduced segments published
        u64 grand = 0, segtots[8];
        for (int q = 0; q < c.CS; ++q) { segtots[q] = cluster.map_shared_rank(c.xch, q)->fb_segtot; grand += segtots[q]; }
        if (lvl == 0 && target == 0) target = ceil_target(topp, grand);
        if (grand == 0 || target > grand || (!by_mass && lvl == 0 && target >= grand)) { cluster.sync(); return false; }
        int s_star = c.CS - 1; u64 before_seg = 0, run = 0;
        for (int q = 0; q < c.CS; ++q) {
            if (run + segtots[q] >= target) { s_star = q; before_seg = run; break; }
            run += segtots[q];
        }
        const u64* pseg = cluster.map_shared_rank(c.fb_seg, s_star);
        int g_star; u64 before;
        block_find([&](int i) { return pseg[i]; }, G, target - before_seg, c.sc, g_star, before);
        target -= before_seg + before;
        khi -= (uint32_t)(s_star * G + g_star) << sh;
        klo = max(klo, khi - ((1u << sh) - 1u));
        cluster.sync();                                                    // (the segments have been read)
    }
    return false;
}

// Gathers the per-warp lists of every CTA of the cluster into glist, in token order (CTA rank, warp, position).
// Returns the number of entries, or -1 when a list overflowed or the total exceeds the capacity.  The entries' masses
// are computed here (the warps' lists hold token and logit only).  All threads call.
__device__ int gather_lists(cg::cluster_group& cluster, int CS, Xch* xch, Cand* ownlist, ListEntry* glist, Scratch* sc,
                            const MassFn& mass, int list_cap) {
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    const int np = CS * CI_WARPS;                                          // (CTA, warp) pairs, at most 128
    int overflow = 0;
    if (tid < CS) overflow = cluster.map_shared_rank(xch, tid)->list_overflow;
    if (tid < np) sc->pcount[tid] = cluster.map_shared_rank(xch, tid / CI_WARPS)->wcount[tid % CI_WARPS];
    overflow = __syncthreads_or(overflow);
    if (warp == 0) {                                                       // exclusive prefix of up to 128 counts
        int c4[4], s = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) { c4[j] = lane * 4 + j < np ? sc->pcount[lane * 4 + j] : 0; s += c4[j]; }
        int incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
        int run = incl - s;
#pragma unroll
        for (int j = 0; j < 4; ++j) { if (lane * 4 + j < np) sc->poff[lane * 4 + j] = (unsigned short)run; run += c4[j]; }
        if (lane == 31) sc->poff[np] = (unsigned short)min(incl, 65535);
    }
    __syncthreads();
    const int n = sc->poff[np];
    if (overflow || n > CI_GLIST) return -1;
    for (int e = tid; e < n; e += CI_THREADS) {
        int lo = 0, hi = np - 1;                                           // last pair p with poff[p] <= e
        while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (sc->poff[mid] <= e) lo = mid; else hi = mid - 1; }
        const Cand c = *(cluster.map_shared_rank(ownlist, lo / CI_WARPS) + (lo % CI_WARPS) * list_cap + (e - sc->poff[lo]));
        ListEntry en;
        en.idx = c.idx; en.l = c.l; en.q = mass(c.l);
        glist[e] = en;
    }
    __syncthreads();
    return n;
}

// Top-k, top-p and the draw on a gathered list that is known to hold every logit >= tl of the row (tl below the
// top-k pivot).  Returns false when the result cannot be trusted from the list alone (the caller falls back).
// On success: token, lcut (final threshold) and total (kept mass).  All threads of the CTA call.
__device__ bool finish_on_list(const ListEntry* glist, int n, float tl, float lcut_in, float tc, int kk, bool need_topp,
                               float topp, float u, u64* bins, uint32_t* cand, Scratch* sc,
                               long long& token, float& lcut, u64& total) {
    const int tid = threadIdx.x;
    float cut = lcut_in;
    u64 cnt = 0;
    for (int i = tid; i < n; i += CI_THREADS) cnt += glist[i].l >= cut ? 1 : 0;
    const u64 survivors = block_sum_u64(cnt, sc);
    if (survivors == 0) return false;
    if ((u64)kk <= survivors) {                                            // else fewer than k survive min-p: top-k removes nothing
        float lk_val;
        if (!list_select(glist, n, [&](int i) { return (u64)(glist[i].l >= cut ? 1 : 0); }, (u64)kk, bins, cand, sc, lk_val))
            return false;
        cut = fmaxf(cut, lower_logit_for(scale_logit(lk_val, tc), tc, lk_val));
        if (cut < tl) return false;                                        // a tie partner could lie outside the list
    }
    if (need_topp) {
        u64 part = 0;
        for (int i = tid; i < n; i += CI_THREADS) if (glist[i].l >= cut) part += glist[i].q;
        const u64 s1 = block_sum_u64(part, sc);
        if (s1 == 0) return false;
        float lp_val;
        const float c0 = cut;
        if (!list_select(glist, n, [&](int i) { return (u64)(glist[i].l >= c0 ? glist[i].q : 0u); }, ceil_target(topp, s1), bins,
                         cand, sc, lp_val))
            return false;
        cut = fmaxf(cut, lower_logit_for(scale_logit(lp_val, tc), tc, lp_val));
        if (cut < tl) return false;
    }
    u64 part = 0;
    for (int i = tid; i < n; i += CI_THREADS) if (glist[i].l >= cut) part += glist[i].q;
    total = block_sum_u64(part, sc);
    if (total == 0) return false;
    int at; u64 before;
    block_find([&](int i) { return (u64)(glist[i].l >= cut ? glist[i].q : 0u); }, n, ceil_target(u, total), sc, at, before);
    token = (long long)glist[at].idx;
    lcut = cut;
    return true;
}

// Appends the components of one float4 group selected by the 4-bit mask mk to the warp's list, in token order
// (lane, then component).  Positions come from four ballots, no scan.  wn is the warp's running count (uniform over
// the warp); entries beyond list_cap are dropped and counted.
__device__ __forceinline__ void warp_append(Cand* mylist, int list_cap, int& wn, unsigned mk, const float* e4, uint32_t idx0, int lane) {
    const unsigned any = __ballot_sync(0xffffffffu, mk != 0u);
    if (!any) return;
    const unsigned lt = (1u << lane) - 1u;
    int at, add;
    if (!__ballot_sync(0xffffffffu, (mk & (mk - 1u)) != 0u)) {              // no lane has two
        at = wn + __popc(any & lt); add = __popc(any);
    } else {
        const unsigned b0 = __ballot_sync(0xffffffffu, mk & 1u), b1 = __ballot_sync(0xffffffffu, mk & 2u);
        const unsigned b2 = __ballot_sync(0xffffffffu, mk & 4u), b3 = __ballot_sync(0xffffffffu, mk & 8u);
        at = wn + __popc(b0 & lt) + __popc(b1 & lt) + __popc(b2 & lt) + __popc(b3 & lt);
        add = __popc(b0) + __popc(b1) + __popc(b2) + __popc(b3);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (mk & (1u << j)) {
            if (at < list_cap) { mylist[at].idx = idx0 + j; mylist[at].l = e4[j]; }
            ++at;
        }
    }
    wn += add;
}

// Collects, in token order, the logits >= tl of one warp's region [r_lo, r_hi) of the slice into the warp's list.
// Four float4 groups per lane and step are loaded together (their latencies overlap); appends are rare.
__device__ __forceinline__ void collect_region(const float* rowbuf, int r_lo, int r_hi, float tl, Cand* mylist, int list_cap, int& wn,
                                               uint32_t slice_lo, int lane) {
    for (int i0 = r_lo; i0 < r_hi; i0 += 512) {
        float4 v[4];
        unsigned mk[4], anym = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + k * 128 + lane * 4;
            v[k] = i < r_hi ? *reinterpret_cast<const float4*>(rowbuf + i) : make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
            mk[k] = (v[k].x >= tl ? 1u : 0u) | (v[k].y >= tl ? 2u : 0u) | (v[k].z >= tl ? 4u : 0u) | (v[k].w >= tl ? 8u : 0u);
            anym |= mk[k];
        }
        if (__ballot_sync(0xffffffffu, anym != 0u)) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float e4[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
                warp_append(mylist, list_cap, wn, mk[k], e4, slice_lo + (uint32_t)(i0 + k * 128 + lane * 4), lane);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ lean block primitives
// Exclusive prefix of one value per thread over the CTA (thread order), and the total.  Two __syncthreads.
__device__ __forceinline__ u64 block_excl_scan(u64 v, Scratch* sc, u64& total) {
    const int lane = lane_id(), warp = warp_id();
    const u64 incl = warp_incl_scan_u64(v, lane);
    if (lane == 31) sc->wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const u64 w = lane < CI_WARPS ? sc->wsum[lane] : 0ull;
        const u64 wi = warp_incl_scan_u64(w, lane);
        if (lane < CI_WARPS) sc->woff[lane] = wi - w;
        if (lane == CI_WARPS - 1) sc->wtotal = wi;
        if (lane == 0) sc->found_tid = -1;
    }
    __syncthreads();
    total = sc->wtotal;
    return sc->woff[warp] + incl - v;
}

// Exact finish of a row from the candidates its CTAs pushed into this CTA's shared memory: min-p, top-k, top-p and
// the draw, all inside this CTA (no cluster traffic).  The candidates contain the row's top k logits (and possibly
// more), in token order: CTA by CTA, each CTA's in token order; a thread holds two of them.  Writes the row's outputs and
// returns true, or returns false when the row has to take the generic path.  `work` is scratch.  All threads of the CTA call.
// Latency is all there is to it: five block barriers, the searches repeated by every warp instead of published, the draw
// by one warp.
__device__ __noinline__ bool finish_pending(const SampleArgs& a, const Pending& pd, const Cand* plist, int CS, unsigned char* work, Scratch* sc) {
    static_assert(CI_FIN_MAX == 2 * CI_THREADS && CI_WARPS == 16 && CI_FAST_BINS == 512 && CI_FIN_KEEP * 4 == CI_THREADS, "two candidates a thread");
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    uint32_t* bins = reinterpret_cast<uint32_t*>(work);
    float* kl = reinterpret_cast<float*>(work + CI_FAST_BINS * 4);
    uint32_t* kq = reinterpret_cast<uint32_t*>(kl + CI_FIN_KEEP), *ki = kq + CI_FIN_KEEP;
    const float tc = pd.tc, L = pd.L, topp = pd.topp;
    const int kk = pd.kk;
    const float m = scale_logit(L, tc);
    MassFn mass;
    mass.init(tc, m);
    const float thr = __fadd_rn(m, pd.lmp);
    float cut = lower_logit_for(thr, tc, __fmul_rn(thr, tc));
    cut = fmaxf(cut, L - 22.0f * tc - fabsf(L) * 1e-6f);           // the mass horizon (see the generic path)
    int pre[9];
    pre[0] = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) pre[q + 1] = pre[q] + (q < CS ? pd.count[q] : 0);
    const int n = pre[8];
    if (n > CI_FIN_MAX || n <= 0) return false;
    // ---- this thread's candidates; how many survive min-p, and their range of keys
    Cand c[2]; bool in[2]; uint32_t key[2];
    uint32_t kmin = 0xFFFFFFFFu, kmax = 0u;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int e = 2 * tid + j;
        int q = 0;
#pragma unroll
        for (int t = 1; t < 8; ++t) q += (pre[t] <= e) ? 1 : 0;
        c[j].l = CI_NEG_INF; c[j].idx = 0;
        if (e < n) c[j] = plist[q * CI_PCAP + (e - pre[q])];
        in[j] = c[j].l >= cut && c[j].l > CI_NEG_INF;
        key[j] = f2key(c[j].l);
        if (in[j]) { kmin = min(kmin, key[j]); kmax = max(kmax, key[j]); }
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin); kmax = __reduce_max_sync(0xffffffffu, kmax);
    const int wcnt = __popc(__ballot_sync(0xffffffffu, in[0])) + __popc(__ballot_sync(0xffffffffu, in[1]));
    if (lane == 0) { sc->warp_u[warp] = kmin; sc->warp_v[warp] = kmax; sc->warp_i[warp] = wcnt; }
    bins[tid] = 0u;
    if (tid == 0) { sc->ncand = 0; sc->sel_ok = 0; }
    __syncthreads();
    kmin = __reduce_min_sync(0xffffffffu, sc->warp_u[lane & 15]); kmax = __reduce_max_sync(0xffffffffu, sc->warp_v[lane & 15]);
    const int survivors = __reduce_add_sync(0xffffffffu, lane < 16 ? sc->warp_i[lane] : 0);
    if (survivors == 0) return false;
    // ---- top-k: the kk-th largest of them
    if (kk <= survivors) {                                    // else fewer than k survive min-p: top-k removes nothing
        const int sh = max(0, 32 - __clz(kmax - kmin) - 9);   // the bins cover [0, kmax - kmin] >> sh, at most 512
#pragma unroll
        for (int j = 0; j < 2; ++j) if (in[j]) atomicAdd(&bins[(kmax - key[j]) >> sh], 1u);
        __syncthreads();
        int b_star, before;
        warp_find<CI_FAST_BINS / 32>(bins, kk, b_star, before);
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (in[j] && (int)((kmax - key[j]) >> sh) == b_star) {
                const int slot = atomicAdd(&sc->ncand, 1);
                if (slot < CI_FIN_CAND) sc->cand_l[slot] = c[j].l;
            }
        __syncthreads();
        const int nc = sc->ncand, want = kk - before;
        if (nc > CI_FIN_CAND) return false;
        float lk = CI_NEG_INF;
        for (int b0 = 0; b0 < nc; b0 += 32) {                 // (every warp, pairwise)
            const float mine = b0 + lane < nc ? sc->cand_l[b0 + lane] : CI_NEG_INF;
            int gt = 0, ge = 0;
            for (int i = 0; i < nc; ++i) { const float o = sc->cand_l[i]; gt += o > mine ? 1 : 0; ge += o >= mine ? 1 : 0; }
            const unsigned hit = __ballot_sync(0xffffffffu, b0 + lane < nc && gt < want && want <= ge);
            if (hit) { lk = __shfl_sync(0xffffffffu, mine, __ffs(hit) - 1); break; }
        }
        cut = fmaxf(cut, lower_logit_for(scale_logit(lk, tc), tc, lk));
    }
    // ---- what is left, in token order, with its masses
    const bool k0 = in[0] && c[0].l >= cut, k1 = in[1] && c[1].l >= cut;
    const unsigned lt = (1u << lane) - 1u, m0 = __ballot_sync(0xffffffffu, k0), m1 = __ballot_sync(0xffffffffu, k1);
    if (lane == 0) sc->pcount[warp] = (unsigned short)(__popc(m0) + __popc(m1));
    __syncthreads();
    const int others = lane < 16 ? sc->pcount[lane] : 0;
    const int nk = __reduce_add_sync(0xffffffffu, others);
    if (nk == 0 || nk > CI_FIN_KEEP) return false;
    {
        int at = __reduce_add_sync(0xffffffffu, lane < warp ? others : 0) + __popc(m0 & lt) + __popc(m1 & lt);
        if (k0) { kl[at] = c[0].l; kq[at] = mass(c[0].l); ki[at] = c[0].idx; ++at; }
        if (k1) { kl[at] = c[1].l; kq[at] = mass(c[1].l); ki[at] = c[1].idx; }
    }
    __syncthreads();
    // ---- top-p: the logit where the descending running mass reaches its share, four threads an entry
    u64 s1 = 0;
#pragma unroll
    for (int t = 0; t < CI_FIN_KEEP / 32; ++t) s1 += t * 32 + lane < nk ? kq[t * 32 + lane] : 0u;
    s1 = warp_sum_u64(s1);
    if (s1 == 0) return false;
    u64 total = s1;
    if (topp < 1.0f) {
        const u64 target = ceil_target(topp, s1);
        const int e = tid >> 2;
        const float mine = e < nk ? kl[e] : CI_NEG_INF;
        u64 gt = 0, ge = 0;
        for (int i = tid & 3; i < nk; i += 4) {
            const float o = kl[i]; const u64 q = kq[i];
            gt += o > mine ? q : 0ull; ge += o >= mine ? q : 0ull;
        }
        gt += __shfl_xor_sync(0xffffffffu, gt, 1); ge += __shfl_xor_sync(0xffffffffu, ge, 1);
        gt += __shfl_xor_sync(0xffffffffu, gt, 2); ge += __shfl_xor_sync(0xffffffffu, ge, 2);
        if (e < nk && gt < target && target <= ge) { sc->res_f = mine; sc->sel_ok = 1; }
        __syncthreads();
        if (!sc->sel_ok) return false;
        const float lp = sc->res_f;
        cut = fmaxf(cut, lower_logit_for(scale_logit(lp, tc), tc, lp));
    }
    // ---- the draw: first candidate (token order) whose running kept mass reaches u * total
    if (warp == 0) {
        u64 q[4], mine = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) { const int e = 4 * lane + j; q[j] = e < nk && kl[e] >= cut ? kq[e] : 0u; mine += q[j]; }
        const u64 incl = warp_incl_scan_u64(mine, lane);
        total = __shfl_sync(0xffffffffu, incl, 31);
        const u64 target = ceil_target(pd.u, total);
        u64 run = incl - mine;
        if (run < target && target <= incl) {
            int j = 0;
            for (; j < 3; ++j) { run += q[j]; if (run >= target) break; }
            const int row = pd.row;
            if (draws(a, row)) a.out[row] = (long long)ki[4 * lane + j];
            if (a.status) a.status[row] = pd.status;
            if (a.stats) {
                colinfer_row_stats st;
                st.lmax = L; st.lcut = cut; st.tc = tc; st.status = pd.status; st.argmax = pd.aidx; st.mass_q = total;
                a.stats[row] = st;
            }
        }
        __syncwarp();                                         // (the caller takes the row off)
    }
    return true;
}

// EIGHT: clusters of eight, whose lists have CI_WLIST entries a warp (a size known only at launch cost them 2 %).
template <bool EIGHT>
__global__ void __launch_bounds__(CI_THREADS, 1) k_sample(const __grid_constant__ SampleArgs a) {
    cg::cluster_group cluster = cg::this_cluster();
    // Every CTA announces that it runs; the matching wait comes just before the first write into a peer's shared memory.
    cluster.barrier_arrive();
    const int CS = (int)cluster.num_blocks();
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    const int V = a.V;

    const int slice_cap = a.slice_elems;                      // multiple of 128
    const int slice_lo = rank * slice_cap;
    const int slice_len = max(0, min(slice_cap, V - slice_lo));
    const int n_pad = (slice_len + 127) & ~127;               // processed elements (tail holds -inf)
    const int nchunks = (slice_len + CI_CHUNK - 1) / CI_CHUNK;

    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* rowbuf = reinterpret_cast<float*>(smem_raw);
    unsigned char* hreg = smem_raw + (size_t)slice_cap * 4;                 // 24 KB work area
    uint32_t* hist1 = reinterpret_cast<uint32_t*>(hreg);                      // [CI_NB1] fine counts
    uint32_t* segcnt = reinterpret_cast<uint32_t*>(hreg + CI_NB1 * 4);        // [<= 2048] reduced segment
    ListEntry* glist = reinterpret_cast<ListEntry*>(hreg);                    // gathered list, over hist1
    u64* bins = reinterpret_cast<u64*>(hreg + CI_NB1 * 4);                    // [512] selection bins, over segcnt
    uint32_t* cand = reinterpret_cast<uint32_t*>(hreg + CI_NB1 * 4 + CI_SEL_BINS * 8);
    u64* fb_hist = reinterpret_cast<u64*>(hreg);                              // fallback radix, over hist1
    u64* fb_seg = fb_hist + CI_FB_NB;
    Cand* plist = reinterpret_cast<Cand*>(hreg + 24 * 1024);                  // [8][CI_PCAP] candidates pushed by the cluster
    u64* mbar = reinterpret_cast<u64*>(plist + 8 * CI_PCAP);
    Xch* xch = reinterpret_cast<Xch*>(mbar + CI_MAX_CHUNKS);
    Scratch* sc = reinterpret_cast<Scratch*>(xch + 1);
    Cand* ownlist = reinterpret_cast<Cand*>(sc + 1);                          // [CI_WARPS][list_cap] this CTA's lists: last, so that the others lie at fixed offsets
    // penalty tables alias the work area (used before the first histogram)
    uint32_t* pen_bits = reinterpret_cast<uint32_t*>(hreg);
    const int nw = slice_cap >> 5;
    uint32_t* pen_prefix = pen_bits + nw;
    uint32_t* pen_cnt = pen_prefix + nw;

    // The mbarriers of the bulk copies are set up once; each row completes one phase of each.
    if (tid == 0 && a.use_bulk) {
        for (int c = 0; c < nchunks; ++c) mbar_init(&mbar[c], 1);
        fence_mbar_init();
    }
    const int n_clusters = (int)gridDim.x / CS;
    const long long n_rows = a.second.rows;
    long long prof_last = clock64();
    const long long prof_t0 = prof_last;
    if (a.prof && tid == 0) for (int i = 0; i < 12; ++i) sc->prof[i] = 0;

    // Starts the bulk copies of one row's slice (thread 0 only; every thread must be done reading the buffer).
    auto issue_row = [&](const long long rw, bool first) {
        if (!first) fence_proxy_async();                       // earlier reads of the buffer precede these writes
        const float* src = reinterpret_cast<const float*>(logits_of(a, (int)rw)) + (size_t)rw * V + slice_lo;
        if (a.flags & COLINFER_TEST_DROP_COPY) return;        // test flag: nothing is armed, nothing is in flight; the waits run out
        for (int c = 0; c < nchunks; ++c) {
            const int len = min(CI_CHUNK, slice_len - c * CI_CHUNK);
            mbar_expect_tx(&mbar[c], (uint32_t)len * 4u);
            bulk_g2s(rowbuf + c * CI_CHUNK, src + c * CI_CHUNK, (uint32_t)len * 4u, &mbar[c]);
        }
    };
    bool prefetched = false;          // the next row's copies are already in flight
    bool fast_enabled = true;         // small top-k rows may take the deferred path (identical in every CTA)
    int fast_seq = 0;                 // deferred rows so far: row j is finished by CTA j % CS
    int n_set_aside = 0;              // rows set aside for the generic path by every CTA alike
    if (tid == 0) { sc->pend.row = -1; sc->n_retry_common = 0; sc->n_retry_mine = 0; sc->any_retry = 0; sc->want_fast_off = 0; }

    // Every CTA that holds a deferred row finishes it; then the cluster meets so that candidates may be pushed again.
    auto flush = [&]() {
        __syncthreads();
        if (sc->pend.row >= 0) {
            const bool ok = finish_pending(a, sc->pend, plist, CS, hreg, sc);
            if (tid == 0) {
                if (!ok) {
                    for (int q = 0; q < CS; ++q) *cluster.map_shared_rank(&sc->any_retry, q) = 1;
                    if (sc->n_retry_mine < CI_RETRY) sc->retry_mine[sc->n_retry_mine++] = sc->pend.row;
                    if (sc->n_retry_mine >= CI_RETRY - 1) sc->want_fast_off = 1;
                }
                sc->pend.row = -1;
            }
        }
        cluster.sync();
    };

    // One row of the batch.  `it` counts this cluster's rows: its parity selects the mbarrier phase and the exchange slots.
    auto process_row = [&](const int row, const int it, const bool allow_fast, const long long next_row) {
    const int par = it & 1;
    int r;
    const int b = slot_of(a, row, r);
    // ---------------------------------------------------------------------------------------- start the HBM read
    // One thread issues every bulk copy of the slice at once, before anything else (unless the previous row already
    // started this row's copies because it no longer needed the buffer).
    if (tid == 0) {
        sc->fail = 0; sc->hist_slow = 0; xch->list_overflow = 0;
        if (a.use_bulk && !prefetched) issue_row(row, it == 0);
    }
    prefetched = false;
    CI_PROF(0);

    // ---------------------------------------------------------------------------------------- parameters of the slot
    const float T = a.p.temperature[b];
    const bool sampled = (T > 0.0f) || (a.flags & COLINFER_FORCE_DISTRIBUTION);
    const float tc = fmaxf(T, 1e-6f);
    const float rp = a.p.repetition_penalty ? a.p.repetition_penalty[b] : 1.0f;
    const float pp = a.p.presence_penalty ? a.p.presence_penalty[b] : 0.0f;
    const float fp = a.p.frequency_penalty ? a.p.frequency_penalty[b] : 0.0f;
    const int32_t* hist = a.p.history ? a.p.history + (size_t)b * a.p.hist_stride : nullptr;
    int hlen = hist ? (a.p.hist_len ? a.p.hist_len[b] : a.p.hist_stride) : 0;
    hlen = max(0, min(hlen, a.p.hist_stride));
    const bool has_pen = hlen > 0 && !(rp == 1.0f && pp == 0.0f && fp == 0.0f);
    const int32_t* mrow = a.mask ? a.mask + ((size_t)b * a.mask_rows + r) * a.W : nullptr;
    const int kk = a.p.top_k[b];
    const float topp = a.p.top_p[b];
    const float log_min_p = a.p.log_min_p[b];
    const float u = row_uniform(a, row, b, r);
    const bool fastk = allow_fast && fast_enabled && sampled && kk >= 1 && kk <= CI_FASTK && kk < V &&
                       !(a.flags & COLINFER_FORCE_DISTRIBUTION);         // identical in every CTA of the cluster

    // tail of the slice buffer: -inf (never selected, zero mass); disjoint from the bulk-copy destinations
    for (int i = slice_len + tid; i < n_pad; i += CI_THREADS) rowbuf[i] = CI_NEG_INF;
    __syncthreads();                                           // mbarriers initialised, tail filled

    // ---------------------------------------------------------------------------------------- penalty tables
    // bitmap of the slice's tokens that occur in the history, their ranks, and the occurrence count per rank
    if (has_pen) {
        // this thread's share of the history, loaded once (8 ids per thread cover 2,048 ids; longer histories loop)
        constexpr int HREG = 8;
        int hv[HREG];
#pragma unroll
        for (int j = 0; j < HREG; ++j) { const int i = tid + j * CI_THREADS; hv[j] = i < hlen ? __ldg(hist + i) - slice_lo : -1; }
        for (int i = tid; i < nw; i += CI_THREADS) pen_bits[i] = 0u;
        for (int i = tid; i < CI_PEN_TABLE; i += CI_THREADS) pen_cnt[i] = 0u;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < HREG; ++j) if (hv[j] >= 0 && hv[j] < slice_len) atomicOr(&pen_bits[hv[j] >> 5], 1u << (hv[j] & 31));
        for (int i = tid + HREG * CI_THREADS; i < hlen; i += CI_THREADS) {
            const int v = __ldg(hist + i) - slice_lo;
            if (v >= 0 && v < slice_len) atomicOr(&pen_bits[v >> 5], 1u << (v & 31));
        }
        __syncthreads();
        if (fp != 0.0f) {
            // ranks of the set bits (exclusive prefix of popcounts over the bitmap words), then the count per rank
            const int ipt = (nw + CI_THREADS - 1) / CI_THREADS;
            const int lo = tid * ipt;
            u64 local = 0;
            for (int i = lo; i < lo + ipt && i < nw; ++i) local += __popc(pen_bits[i]);
            u64 total_bits;
            uint32_t run = (uint32_t)block_excl_scan(local, sc, total_bits);
            for (int i = lo; i < lo + ipt && i < nw; ++i) { pen_prefix[i] = run; run += __popc(pen_bits[i]); }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < HREG; ++j) {
                const int v = hv[j];
                if (v >= 0 && v < slice_len) {
                    const uint32_t rk = pen_prefix[v >> 5] + __popc(pen_bits[v >> 5] & ((1u << (v & 31)) - 1u));
                    if (rk < CI_PEN_TABLE) atomicAdd(&pen_cnt[rk], 1u);
                }
            }
            for (int i = tid + HREG * CI_THREADS; i < hlen; i += CI_THREADS) {
                const int v = __ldg(hist + i) - slice_lo;
                if (v >= 0 && v < slice_len) {
                    const uint32_t rk = pen_prefix[v >> 5] + __popc(pen_bits[v >> 5] & ((1u << (v & 31)) - 1u));
                    if (rk < CI_PEN_TABLE) atomicAdd(&pen_cnt[rk], 1u);
                }
            }
            __syncthreads();
        }
    }

    CI_PROF(1);
    // ---------------------------------------------------------------------------------------- pass A: land, penalise, mask, maximum
    float lmax = CI_NEG_INF;
    int lidx = 0x7fffffff;
    int lpos = -1;                                              // float4 group of the slice that holds this thread's maximum
    float tg[CI_TGROUPS];                                       // maxima of this thread's interleaved element groups
#pragma unroll
    for (int j = 0; j < CI_TGROUPS; ++j) tg[j] = CI_NEG_INF;
    // the mask words of this thread's first groups, on their way while the slice lands
    constexpr int MPRE = 3;
    uint32_t mw[MPRE][CI_TGROUPS];
    if (mrow != nullptr) {
#pragma unroll
        for (int o = 0; o < MPRE; ++o)
#pragma unroll
            for (int k = 0; k < CI_TGROUPS; ++k) {
                const int g = slice_lo + (tid + (o * CI_TGROUPS + k) * CI_THREADS) * 4;
                mw[o][k] = g < min(slice_lo + n_pad, V) ? (uint32_t)__ldg(mrow + (g >> 5)) : 0xFFFFFFFFu;
            }
    }
    // (1) the slice lands: wait for the bulk copies, or load it with plain loads (unaligned fp32 rows, bf16)
    if (a.use_bulk) {
        const bool drop = (a.flags & COLINFER_TEST_DROP_COPY) != 0;
        if (drop) for (int i = tid; i < slice_len; i += CI_THREADS) rowbuf[i] = 0.0f;   // (the test reads a defined buffer)
        for (int c = 0; c < nchunks; ++c)
            if (!mbar_wait_bounded(&mbar[c], (uint32_t)par, drop ? 20000LL : CI_WAIT_CYCLES)) sc->fail = 1;
    } else {
        const size_t g0 = (size_t)row * V + slice_lo;
        if (a.dtype == COLINFER_BF16) {
            const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(logits_of(a, row)) + g0;
            if ((((uintptr_t)src) & 15) == 0) {
                const uint4* s4 = reinterpret_cast<const uint4*>(src);
                for (int i = tid; i * 8 < slice_len; i += CI_THREADS) {
                    if (i * 8 + 8 <= slice_len) {
                        const uint4 q = __ldg(s4 + i);
                        const uint32_t ww[4] = {q.x, q.y, q.z, q.w};
                        float* d = rowbuf + i * 8;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            d[2 * j] = __uint_as_float(ww[j] << 16);
                            d[2 * j + 1] = __uint_as_float(ww[j] & 0xFFFF0000u);
                        }
                    } else {
                        for (int j = i * 8; j < slice_len; ++j) rowbuf[j] = __bfloat162float(src[j]);
                    }
                }
            } else {
                for (int i = tid; i < slice_len; i += CI_THREADS) rowbuf[i] = __bfloat162float(src[i]);
            }
        } else {
            const float* src = reinterpret_cast<const float*>(logits_of(a, row)) + g0;
            for (int i = tid; i < slice_len; i += CI_THREADS) rowbuf[i] = __ldg(src + i);
        }
        __syncthreads();
    }
    CI_PROF(5);
    // (2) penalties: one bitmap word (32 tokens) per thread and step
    if (has_pen) {
        const int wn = n_pad >> 5;
        for (int wi = tid; wi < wn; wi += CI_THREADS) {
            const uint32_t word = pen_bits[wi];
            uint32_t rest = word;
            while (rest) {
                const int bit = __ffs(rest) - 1;
                rest &= rest - 1;
                const int v = (wi << 5) + bit;
                int cnt = 1;
                if (fp != 0.0f) {
                    const uint32_t rk = pen_prefix[wi] + __popc(word & ((1u << bit) - 1u));
                    if (rk < CI_PEN_TABLE) cnt = (int)pen_cnt[rk];
                    else {
                        cnt = 0; sc->hist_slow = 1;
                        for (int i = 0; i < hlen; ++i) cnt += (hist[i] == v + slice_lo);
                    }
                }
                rowbuf[v] = apply_penalty(rowbuf[v], cnt, rp, pp, fp);
            }
        }
        __syncthreads();
    }
    // (3) mask and maximum: four float4 groups per thread and step, loaded together so that their latencies overlap
    {
        float4* row4 = reinterpret_cast<float4*>(rowbuf);
        const int n4 = n_pad >> 2;
        auto step = [&](int i0, auto word) {
            float4 v[CI_TGROUPS];
#pragma unroll
            for (int k = 0; k < CI_TGROUPS; ++k) {
                const int i = i0 + k * CI_THREADS;
                v[k] = i < n4 ? row4[i] : make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
            }
            if (mrow != nullptr) {
#pragma unroll
                for (int k = 0; k < CI_TGROUPS; ++k) {
                    const int i = i0 + k * CI_THREADS;
                    const int g = slice_lo + i * 4;             // global token index of v[k].x
                    if (i < n4 && g < V) {
                        const uint32_t bits = (word(k, g) >> (g & 31)) & 0xFu;
                        if (bits != 0xFu) {
                            if (!(bits & 1u)) v[k].x = CI_NEG_INF;
                            if (!(bits & 2u)) v[k].y = CI_NEG_INF;
                            if (!(bits & 4u)) v[k].z = CI_NEG_INF;
                            if (!(bits & 8u)) v[k].w = CI_NEG_INF;
                            row4[i] = v[k];
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < CI_TGROUPS; ++k) {
                const float m4 = fmaxf(fmaxf(v[k].x, v[k].y), fmaxf(v[k].z, v[k].w));
                tg[k] = fmaxf(tg[k], m4);
                const bool up = m4 > lmax;                      // strict: the first (lowest) position of the maximum stays
                lmax = up ? m4 : lmax;
                lpos = up ? i0 + k * CI_THREADS : lpos;
            }
        };
#pragma unroll
        for (int o = 0; o < MPRE; ++o) {
            const int i0 = tid + o * CI_TGROUPS * CI_THREADS;
            if (i0 < n4) step(i0, [&](int k, int) { return mw[o][k]; });
        }
        for (int i0 = tid + MPRE * CI_TGROUPS * CI_THREADS; i0 < n4; i0 += CI_TGROUPS * CI_THREADS)
            step(i0, [&](int, int g) { return (uint32_t)__ldg(mrow + (g >> 5)); });
    }
    CI_PROF(2);
    if (lpos >= 0) {
        const float4 v = reinterpret_cast<const float4*>(rowbuf)[lpos];
        lidx = slice_lo + lpos * 4 + (v.x == lmax ? 0 : v.y == lmax ? 1 : v.z == lmax ? 2 : 3);
    }
    // block reduce (largest value, lowest index among equals)
    {
        const float wm = warp_max(lmax);
        lidx = __reduce_min_sync(0xffffffffu, lmax == wm ? lidx : 0x7fffffff);
        if (lane == 0) { sc->warp_f[warp] = wm; sc->warp_i[warp] = lidx; }
    }
    if (fastk) for (int i = tid; i < CI_FAST_BINS; i += CI_THREADS) hist1[i] = 0u;   // (the penalty tables are done with)
    __syncthreads();
    {
        const float om = sc->warp_f[lane % CI_WARPS]; const int oi = sc->warp_i[lane % CI_WARPS];
        lmax = warp_max(om);                                    // the slice maximum, in every thread
        lidx = __reduce_min_sync(0xffffffffu, om == lmax ? oi : 0x7fffffff);
    }

    // warp w owns the contiguous region [r_lo, r_hi) of the slice; lanes interleave float4 groups, so the token
    // order inside a region is (step, lane, component).
    const int reg = ((n_pad / 128 + CI_WARPS - 1) / CI_WARPS) * 128;
    const int r_lo = min(warp * reg, n_pad), r_hi = min(r_lo + reg, n_pad);
    const int list_cap = EIGHT ? CI_WLIST : a.list_cap;
    Cand* mylist = ownlist + warp * list_cap;

    // ---------------------------------------------------------------------------------------- small top-k: candidates of the slice
    // The k-th largest of the threads' group maxima (CI_TGROUPS disjoint groups per thread) bounds the slice's k-th largest logit from below, and every logit of the
    // row's top k is among its own slice's top k: the logits >= that bound, over all slices, contain the row's top k.
    float tl_fast = CI_NEG_INF;
    int my_count = 0;
    if (it == 0) cluster.barrier_wait();                        // every CTA of the cluster runs: peers' memory may be written
    if (fastk) {
#pragma unroll
        for (int j = 0; j < CI_TGROUPS; ++j)
            if (tg[j] > CI_NEG_INF) atomicAdd(&hist1[min(CI_FAST_BINS - 1, __float2int_rz((lmax - tg[j]) * CI_FAST_SCALE))], 1u);
        __syncthreads();
        int bk, before;
        warp_find<CI_FAST_BINS / 32>(hist1, kk, bk, before);    // (512 without k maxima)
        if (bk < CI_FAST_BINS - 1)
            tl_fast = lmax - ((float)(bk + 1) + 0.01f) / CI_FAST_SCALE - fabsf(lmax) * 1e-6f;
        else tl_fast = -CI_FLT_MAX;                             // fewer than k threads saw a finite logit: take them all
        CI_PROF(10);
        int wn = 0;
        collect_region(rowbuf, r_lo, r_hi, tl_fast, mylist, list_cap, wn, (uint32_t)slice_lo, lane);
        CI_PROF(11);
        if (lane == 0) sc->warp_i[warp] = wn;
        __syncthreads();                                        // every thread is done with the row buffer
        int woff = 0;
        bool over = false;
#pragma unroll
        for (int w = 0; w < CI_WARPS; ++w) {
            const int c = sc->warp_i[w];
            if (w < warp) woff += c;
            my_count += c;
            over |= c > list_cap;
        }
        if (over || my_count > CI_PCAP) my_count = 0xFFFF;      // overflow marker: the row takes the generic path later
        else {
            // push this CTA's candidates, in token order, to the CTA that will finish the row
            Cand* dst = cluster.map_shared_rank(plist, fast_seq % CS) + rank * CI_PCAP + woff;
            for (int j = lane; j < wn; j += 32) dst[j] = mylist[j];
        }
        // the row buffer is free: start the next row's copies now
        if (a.use_bulk && next_row >= 0) {
            if (tid == 0) issue_row(next_row, false);
            prefetched = true;
        }
    } else if (!sampled && a.use_bulk && next_row >= 0) {
        // greedy row: only the maximum is needed from here on
        if (tid == 0) issue_row(next_row, false);
        prefetched = true;
    }

    // ---------------------------------------------------------------------------------------- first exchange
    CI_PROF(3);
    if (tid < CS) {
        Hello h;
        h.lmax = lmax; h.lidx = lidx;
        h.flags = (sc->fail ? 1 : 0) | (sc->hist_slow ? 4 : 0) | (sc->want_fast_off ? 8 : 0);
        h.pad = my_count;
        cluster.map_shared_rank(sc, tid)->hello[par][rank] = h;
    }
    cluster.sync();                                                                    // (1) slice maxima (and list sizes) exchanged
    CI_PROF(4);
    float L = CI_NEG_INF; int aidx = 0x7fffffff; int hflags = 0; int fast_total = 0; bool fast_overflow = false;
    for (int q = 0; q < CS; ++q) {
        const Hello h = sc->hello[par][q];
        if (h.lmax > L || (h.lmax == L && h.lidx < aidx)) { L = h.lmax; aidx = h.lidx; }
        hflags |= h.flags;
        fast_total += h.pad;
        if (h.pad >= 0xFFFF) fast_overflow = true;
    }
    if (aidx == 0x7fffffff) aidx = 0;
    if (hflags & 8) fast_enabled = false;                       // a CTA ran out of room for set-aside rows

    int status = ((hflags & 1) ? COLINFER_ROW_TIMEOUT : 0) | ((hflags & 4) ? COLINFER_ROW_HIST_SLOW : 0);
    const bool finite_max = (L > CI_NEG_INF) && (L < CI_POS_INF);
    if (sampled && !finite_max) status |= COLINFER_ROW_DEGENERATE;
    const bool do_dist = sampled && finite_max && !(hflags & 1);   // identical in every CTA of the cluster

    float lcut = CI_NEG_INF;
    u64 total_mass = 0;
    long long token = aidx;

    if (!do_dist) {
        // greedy, degenerate or failed row: the argmax.  Nobody reads a peer's memory after the barrier: leave at once.
        if (rank == 0 && tid == 0) {
            if (draws(a, row)) a.out[row] = token;
            if (a.status) a.status[row] = status;
            if (a.stats) {
                colinfer_row_stats st;
                st.lmax = L; st.lcut = lcut; st.tc = tc; st.status = status; st.argmax = aidx; st.mass_q = 0;
                a.stats[row] = st;
            }
        }
        return;
    }

    // ---------------------------------------------------------------------------------------- small top-k: defer the exact finish
    if (fastk) {
        // The candidates of every CTA sit in the shared memory of CTA fast_seq % CS, which finishes the row later, on its
        // own, while the cluster moves on.  A row whose lists overflowed is set aside for the generic path instead.
        const bool deferred = !fast_overflow && fast_total >= 1;
        if (deferred) {
            if (rank == fast_seq % CS && tid == 0) {
                Pending pd;
                pd.row = row; pd.L = L; pd.aidx = aidx; pd.status = status;
                pd.kk = kk; pd.tc = tc; pd.topp = topp; pd.lmp = log_min_p; pd.u = u;
                for (int q = 0; q < 8; ++q) pd.count[q] = q < CS ? sc->hello[par][q].pad : 0;
                sc->pend = pd;
            }
            ++fast_seq;
            if (fast_seq % CS == 0) flush();                    // every CTA holds a row now
        } else {
            if (tid == 0) { sc->any_retry = 1; if (sc->n_retry_common < CI_RETRY) sc->retry_common[sc->n_retry_common++] = row; }
            if (++n_set_aside >= CI_RETRY) fast_enabled = false;
        }
        return;
    }

    const float m = scale_logit(L, tc);
    MassFn mass;
    mass.init(tc, m);
    // ---------------------------------------------------------------------------------------- min-p threshold
    const float thr = __fadd_rn(m, log_min_p);
    lcut = lower_logit_for(thr, tc, __fmul_rn(thr, tc));
    // Mass horizon: a logit more than 22 temperatures below the maximum has integer mass 0 (2^30 exp(-22) < 1/2); it can
    // never be drawn and adds nothing to any sum, so every selection works above it.
    lcut = fmaxf(lcut, L - 22.0f * tc - fabsf(L) * 1e-6f);
    bool need_topk = kk > 0 && kk < V;
    const bool need_topp = topp < 1.0f;

    // (generic path from here on: the whole cluster works on the row until its token is out)
    const bool coarse = a.dtype == COLINFER_BF16 && !has_pen;   // every logit is a bf16
    enum { PATH_PURE = 0, PATH_LIST = 1, PATH_BAND = 2, PATH_FALLBACK = 3 };
    int path = PATH_PURE;
    float t_hi = CI_NEG_INF, t_lo = CI_POS_INF;                 // band thresholds (PATH_BAND), list threshold (PATH_LIST: t_lo)

    if (need_topk || need_topp) {
        // ------------------------------------------------------------------------------------ fine count histogram
        const float SC = (float)CI_NB1 / (CI_RANGE * tc);
        const float lk = fmaxf(lcut, -CI_FLT_MAX);             // excludes -inf (masked / padding) as well
        for (int i = tid; i < CI_NB1; i += CI_THREADS) hist1[i] = 0u;
        if (tid == 0) xch->list_overflow = 0;
        const bool exact_top = need_topp && !need_topk;
        float* toplist = reinterpret_cast<float*>(ownlist);
        const float t_top = fmaxf(L - CI_TOP * tc, lk);
        if (tid == 0) sc->ncand = 0;
        __syncthreads();
        {
            const float4* row4 = reinterpret_cast<const float4*>(rowbuf);
            const int n4 = n_pad >> 2;
            for (int i0 = tid; i0 < n4; i0 += 4 * CI_THREADS) {
                float e[16];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = i0 + k * CI_THREADS;
                    const float4 v = i < n4 ? row4[i] : make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
                    e[4 * k] = v.x; e[4 * k + 1] = v.y; e[4 * k + 2] = v.z; e[4 * k + 3] = v.w;
                }
                int bkt[16];
#pragma unroll
                for (int j = 0; j < 16; ++j)                  // (the integer part, by an addition rounded towards zero: conversions have a quarter of its rate)
                    bkt[j] = min(CI_NB1 - 1, __float_as_int(__fadd_rz((L - e[j]) * SC, 8388608.0f)) - 0x4B000000);
#pragma unroll
                for (int j = 0; j < 16; ++j) if (e[j] >= lk) atomicAdd(&hist1[bkt[j]], 1u);
                // The largest logits are noted: what their buckets' estimates are off by is worked out below.  (They make up most
                // of a peaked row's mass, and a band that misses the pivot costs two more passes and a select.)
                if (exact_top) {
                    float top = e[0];
#pragma unroll
                    for (int j = 1; j < 16; ++j) top = fmaxf(top, e[j]);
                    if (top >= t_top) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (e[j] >= t_top) { const int at = atomicAdd(&sc->ncand, 1); if (at < CI_THREADS) toplist[at] = e[j]; }
                    }
                }
            }
        }
        __syncthreads();
        CI_PROF(10);
        cluster.sync();                                                                // (A) local histograms complete
        CI_PROF(11);
        // each CTA reduces its segment of the buckets over the cluster, and sends the segment's totals to its peers
        const int G = CI_NB1 / CS;
        uint32_t* myseg = (CS == 1) ? hist1 : segcnt;
        u64 pc = 0, pe = 0;
        for (int g = tid; g < G; g += CI_THREADS) {
            uint32_t sum = 0;
            if (CS == 1) sum = hist1[g];
            else {
                uint32_t x[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) x[q] = q < CS ? cluster.map_shared_rank(hist1, q)[rank * G + g] : 0u;
#pragma unroll
                for (int q = 0; q < 8; ++q) sum += x[q];
                segcnt[g] = sum;
            }
            pc += sum;
            pe += (u64)sum * bucket_mass_est(rank * G + g);
        }
        pc = warp_sum_u64(pc); pe = warp_sum_u64(pe);
        if (lane == 0) { sc->warp_tot[warp] = pc; sc->warp_aux[warp] = pe; }
        if (exact_top) {
            long long off = 0;
            if (tid < sc->ncand) {
                const float x = toplist[tid];
                off = (long long)mass(x) - (long long)bucket_mass_est(min(CI_NB1 - 1, __float_as_int(__fadd_rz((L - x) * SC, 8388608.0f)) - 0x4B000000));
            }
            const u64 o = warp_sum_u64((u64)off);
            if (lane == 0) sc->wsum[warp] = o;
        }
        __syncthreads();
        if (warp == 0) {
            pc = warp_sum_u64(lane < CI_WARPS ? sc->warp_tot[lane] : 0ull); pe = warp_sum_u64(lane < CI_WARPS ? sc->warp_aux[lane] : 0ull);
            const u64 po = exact_top ? warp_sum_u64(lane < CI_WARPS ? sc->wsum[lane] : 0ull) : 0ull;
            if (lane < CS) { Scratch* ps = cluster.map_shared_rank(sc, lane); ps->seg_cnt[rank] = pc; ps->seg_est[rank] = pe; ps->seg_off[rank] = po; }
        }
        cluster.sync();                                                                // (B) reduced segments published
        u64 segc[8], sege[8], survivors = 0, est_total = 0;
        long long off_total = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            segc[q] = q < CS ? sc->seg_cnt[q] : 0ull; sege[q] = q < CS ? sc->seg_est[q] : 0ull;
            survivors += segc[q]; est_total += sege[q];
            off_total += q < CS ? (long long)sc->seg_off[q] : 0ll;
        }
        if (need_topk && (u64)kk >= survivors) need_topk = false;   // fewer survivors than k: top-k removes nothing
        if (need_topk) {
            // bucket of the k-th largest logit, exactly
            int s_star = CS - 1; u64 before_seg = 0, run = 0;
#pragma unroll
            for (int q = 7; q >= 0; --q) if (q < CS) {          // (from the last one down: the first that reaches it stays)
                run = 0;
#pragma unroll
                for (int t = 0; t < 8; ++t) if (t < q) run += segc[t];
                if (run + segc[q] >= (u64)kk) { s_star = q; before_seg = run; }
            }
            const uint32_t* pseg = cluster.map_shared_rank(myseg, s_star);
            int g_star; u64 before;
            if (G <= CI_THREADS) thread_find(tid < G ? (u64)pseg[tid] : 0ull, (u64)kk - before_seg, sc, g_star, before);
            else block_find([&](int i) { return (u64)pseg[i]; }, G, (u64)kk - before_seg, sc, g_star, before);
            const int bk = s_star * G + g_star;
            const u64 n_upto = before_seg + before + pseg[g_star];
            if (bk >= CI_NB1 - 3 || n_upto > CI_GLIST - 64) path = PATH_FALLBACK;
            else {
                path = PATH_LIST;
                // every element of buckets <= bk + 1 satisfies l >= t_lo (a slightly wider set is harmless)
                t_lo = L - ((float)(bk + 2) + 0.01f) / SC - fabsf(L) * 1e-6f;
            }
        } else if (need_topp) {
            // bucket where the descending cumulative estimated mass reaches top_p of the estimated total
            if (est_total == 0) path = PATH_FALLBACK;
            else {
                const long long t_off = (long long)est_total + off_total > 0 ? (long long)ceil_target(topp, (u64)((long long)est_total + off_total)) - off_total : 1;
                const u64 target = t_off < 1 ? 1ull : min((u64)t_off, est_total);
                int s_star = CS - 1; u64 before_seg = 0, run = 0;
#pragma unroll
                for (int q = 7; q >= 0; --q) if (q < CS) {
                    run = 0;
#pragma unroll
                    for (int t = 0; t < 8; ++t) if (t < q) run += sege[t];
                    if (run + sege[q] >= target) { s_star = q; before_seg = run; }
                }
                const uint32_t* pseg = cluster.map_shared_rank(myseg, s_star);
                int g_star; u64 before;
                if (G <= CI_THREADS) thread_find(tid < G ? (u64)pseg[tid] * bucket_mass_est(s_star * G + tid) : 0ull, target - before_seg, sc, g_star, before);
                else block_find([&](int i) { return (u64)pseg[i] * bucket_mass_est(s_star * G + i); }, G, target - before_seg, sc, g_star, before);
                int bp = s_star * G + g_star;
                const int up = a.dtype == COLINFER_BF16 ? 3 : 1, dn = a.dtype == COLINFER_BF16 ? 4 : 2;
                const int s8 = (a.flags & COLINFER_TEST_MISS_BAND) ? (row & 1 ? 8 : -8) : 0;   // test hook: a band eight buckets off
                bp = max(0, min(bp + s8, CI_NB1 - 1));
                if (bp + dn + 2 >= CI_NB1) path = PATH_FALLBACK;
                else {
                    path = PATH_BAND;
                    t_hi = bp - up <= 0 ? CI_POS_INF : L - (float)(bp - up) / SC;
                    t_lo = L - (float)(bp + dn + 1) / SC;
                }
            }
        }
    }
    CI_PROF(5);

    // ---------------------------------------------------------------------------------------- large top-k (then top-p) on a gathered list
    bool done = false;
    if (path == PATH_LIST) {
        const float tl = fmaxf(fmaxf(t_lo, lcut), -CI_FLT_MAX);
        int wn = 0;
        collect_region(rowbuf, r_lo, r_hi, tl, mylist, list_cap, wn, (uint32_t)slice_lo, lane);
        if (lane == 0) {
            xch->wcount[warp] = (unsigned short)min(wn, list_cap);
            if (wn > list_cap) xch->list_overflow = 1;
        }
        __syncthreads();
        CI_PROF(6);
        cluster.sync();                                                                // (L) lists published
        // every CTA gathers the lists and finishes alike (identical inputs, identical decisions)
        const int n = gather_lists(cluster, CS, xch, ownlist, glist, sc, mass, list_cap);
        if (n > 0 && finish_on_list(glist, n, tl, lcut, tc, kk, need_topp, topp, u, bins, cand, sc, token, lcut, total_mass)) done = true;
        else path = PATH_FALLBACK;
    }

    // ---------------------------------------------------------------------------------------- fallback: exact radix select over the 32-bit keys
    if (path == PATH_FALLBACK) {
        // (a CTA reaches this point only after every peer finished reading its reduced segment and its lists: those
        // reads precede the peers' next cluster barrier, and the first write below follows this CTA's next barrier)
        const RadixCtx rc = {rowbuf, n_pad, fb_hist, fb_seg, xch, sc, rank, CS};
        float lpiv;
        status |= COLINFER_ROW_SELECT_SLOW;
        if (kk > 0 && kk < V && radix_select(cluster, rc, mass, f2key(fmaxf(lcut, -CI_FLT_MAX)), f2key(L), coarse, false, (u64)kk, topp, lpiv))
            lcut = fmaxf(lcut, lower_logit_for(scale_logit(lpiv, tc), tc, lpiv));
        if (need_topp && radix_select(cluster, rc, mass, f2key(fmaxf(lcut, -CI_FLT_MAX)), f2key(L), coarse, true, 0, topp, lpiv))
            lcut = fmaxf(lcut, lower_logit_for(scale_logit(lpiv, tc), tc, lpiv));
        path = PATH_PURE;
        t_hi = CI_NEG_INF; t_lo = CI_POS_INF;
    }

    // ---------------------------------------------------------------------------------------- mass pass and inverse CDF over the row
    if (!done) {
        const bool band = path == PATH_BAND;
        const float lk = fmaxf(lcut, -CI_FLT_MAX);
        u64 acc_all = 0, acc_above = 0;
        int wn = 0;
        Mass2 mass2;
        mass2.init(mass);
        const float t_low = fmaxf(t_lo, lk);
#pragma unroll 1
        for (int i0 = r_lo; i0 < r_hi; i0 += 512) {
            float e[16];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = i0 + k * 128 + lane * 4;
                const float4 v = i < r_hi ? *reinterpret_cast<const float4*>(rowbuf + i) : make_float4(CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF);
                e[4 * k] = v.x; e[4 * k + 1] = v.y; e[4 * k + 2] = v.z; e[4 * k + 3] = v.w;
            }
            unsigned mk = 0;                                    // the band's logits among the sixteen
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                uint32_t q0, q1;
                mass2.whole(e[j], e[j + 1], lk, q0, q1);
                acc_all += q0 + q1;                             // (at most 2^31)
                if (band) {
                    const bool a0 = e[j] > t_hi, a1 = e[j + 1] > t_hi;
                    acc_above += (a0 ? q0 : 0u) + (a1 ? q1 : 0u);
                    if (!a0 && e[j] >= t_low) mk |= 1u << j;
                    if (!a1 && e[j + 1] >= t_low) mk |= 2u << j;
                }
            }
            // the band's logits are appended in no particular order: only their values and masses are looked at
            for (unsigned any = __ballot_sync(0xffffffffu, mk != 0u); any; any = __ballot_sync(0xffffffffu, mk != 0u)) {
                const int at = wn + __popc(any & ((1u << lane) - 1u));
                if (mk && at < list_cap) {
                    const int t = __ffs(mk) - 1, i = i0 + (t >> 2) * 128 + lane * 4 + (t & 3);
                    mylist[at].idx = (uint32_t)(slice_lo + i); mylist[at].l = rowbuf[i];
                }
                mk &= mk - 1;
                wn += __popc(any);
            }
        }
        u64 wkeep = warp_sum_u64(band ? acc_above : acc_all);   // kept mass of the region known so far
        if (band) {
            const u64 wall = warp_sum_u64(acc_all);
            if (lane == 0) {
                sc->warp_tot[warp] = wkeep; sc->warp_aux[warp] = wall;
                xch->wcount[warp] = (unsigned short)min(wn, list_cap);
                if (wn > list_cap) xch->list_overflow = 1;
            }
            __syncthreads();
            if (warp == 0) {
                const u64 ta = warp_sum_u64(lane < CI_WARPS ? sc->warp_aux[lane] : 0ull), tb = warp_sum_u64(lane < CI_WARPS ? sc->warp_tot[lane] : 0ull);
                if (lane < CS) { Scratch* ps = cluster.map_shared_rank(sc, lane); ps->all_in[rank] = ta; ps->above_in[rank] = tb; }
            }
            CI_PROF(11);
            cluster.sync();                                                            // (L) band lists and sums published
            u64 s1 = 0, s_above = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) if (q < CS) { s1 += sc->all_in[q]; s_above += sc->above_in[q]; }
            const int n = gather_lists(cluster, CS, xch, ownlist, glist, sc, mass, list_cap);
            bool ok = n >= 0 && s1 > 0;
            float cut2 = lcut;
            if (ok) {
                u64 part = 0;
                for (int i = tid; i < n; i += CI_THREADS) part += glist[i].q;
                const u64 s_band = block_sum_u64(part, sc);
                const u64 target = ceil_target(topp, s1);
                ok = s_above < target && target <= s_above + s_band;           // the pivot lies inside the band
                if (ok) {
                    float lp_val;
                    ok = list_select(glist, n, [&](int i) { return (u64)glist[i].q; }, target - s_above, bins, cand, sc, lp_val);
                    if (ok) {
                        cut2 = fmaxf(lcut, lower_logit_for(scale_logit(lp_val, tc), tc, lp_val));
                        if (cut2 < t_lo) ok = false;                           // a tie partner could lie below the band
                    }
                }
            }
            if (ok) {
                lcut = cut2;
                // add the kept band entries of this warp's own list to its region's kept mass
                u64 add = 0;
                const int mine = min(wn, list_cap);
                for (int j = lane; j < mine; j += 32) if (mylist[j].l >= lcut) add += mass(mylist[j].l);
                wkeep += warp_sum_u64(add);
            } else {
                // The estimated band missed the pivot (or a list overflowed): every CTA takes the exact radix select
                // by mass, then recomputes its regions' kept mass.  Rare; same result, more time.
                const RadixCtx rc = {rowbuf, n_pad, fb_hist, fb_seg, xch, sc, rank, CS};
                float lpiv;
                uint32_t klo = f2key(fmaxf(lcut, -CI_FLT_MAX)), khi = f2key(L);
                u64 want = 0;
                status |= COLINFER_ROW_SELECT_SLOW;
                if (s1 > 0) {                                                  // on which side of the band's upper edge it lies is known
                    want = ceil_target(topp, s1);
                    if (want <= s_above) klo = f2key(t_hi) + 1u;
                    else { khi = min(khi, f2key(t_hi)); want -= s_above; }
                }
                if (radix_select(cluster, rc, mass, klo, khi, coarse, true, want, topp, lpiv))
                    lcut = fmaxf(lcut, lower_logit_for(scale_logit(lpiv, tc), tc, lpiv));
                const float lk3 = fmaxf(lcut, -CI_FLT_MAX);
                u64 acc = 0;
                for (int i0 = r_lo; i0 < r_hi; i0 += 128) {
                    const float4 v = *reinterpret_cast<const float4*>(rowbuf + i0 + lane * 4);
                    acc += (u64)(v.x >= lk3 ? mass(v.x) : 0u) + (v.y >= lk3 ? mass(v.y) : 0u);
                    acc += (u64)(v.z >= lk3 ? mass(v.z) : 0u) + (v.w >= lk3 ? mass(v.w) : 0u);
                }
                wkeep = warp_sum_u64(acc);
            }
        }
        __syncthreads();
        if (lane == 0) sc->warp_tot[warp] = wkeep;
        __syncthreads();
        u64 my_mass = 0;
        for (int w = 0; w < CI_WARPS; ++w) my_mass += sc->warp_tot[w];
        if (tid < CS) cluster.map_shared_rank(sc, tid)->mass_in[par][rank] = my_mass;
        CI_PROF(6);
        cluster.sync();                                                                // (C) slice masses exchanged
        CI_PROF(7);
        u64 my_off = 0;
        for (int q = 0; q < CS; ++q) {
            const u64 cm = sc->mass_in[par][q];
            if (q < rank) my_off += cm;
            total_mass += cm;
        }
        const u64 target = ceil_target(u, total_mass);
        token = -1;
        if (total_mass > 0 && my_off < target && target <= my_off + my_mass) {
            // the crossing lies in this CTA: find the warp region, then the element
            u64 woff = my_off;
            for (int w = 0; w < warp; ++w) woff += sc->warp_tot[w];
            if (woff < target && target <= woff + wkeep) {
                const float lkf = fmaxf(lcut, -CI_FLT_MAX);
                u64 run = woff;
                for (int i0 = r_lo; i0 < r_hi; i0 += 128) {
                    const int i = i0 + lane * 4;
                    const float4 v = *reinterpret_cast<const float4*>(rowbuf + i);
                    u64 q4[4];
                    q4[0] = v.x >= lkf ? mass(v.x) : 0u; q4[1] = v.y >= lkf ? mass(v.y) : 0u;
                    q4[2] = v.z >= lkf ? mass(v.z) : 0u; q4[3] = v.w >= lkf ? mass(v.w) : 0u;
                    const u64 s4 = q4[0] + q4[1] + q4[2] + q4[3];
                    const u64 incl = warp_incl_scan_u64(s4, lane);
                    const u64 grp = __shfl_sync(0xffffffffu, incl, 31);
                    if (run + grp >= target) {
                        const unsigned hit = __ballot_sync(0xffffffffu, run + incl >= target);
                        const int first = __ffs(hit) - 1;
                        if (lane == first) {
                            u64 c = run + incl - s4;
                            int j = 0;
                            for (; j < 3; ++j) { c += q4[j]; if (c >= target) break; }
                            if (draws(a, row)) a.out[row] = (long long)(slice_lo + i + j);
                        }
                        break;
                    }
                    run += grp;
                }
            }
        }
        if (total_mass == 0) { status |= COLINFER_ROW_DEGENERATE; token = aidx; }
    }

    if (rank == 0 && tid == 0) {
        if (token >= 0 && draws(a, row)) a.out[row] = token;           // list-path or degenerate rows (else the crossing lane stored it)
        if (a.status) a.status[row] = status;
        if (a.stats) {
            colinfer_row_stats st;
            st.lmax = L; st.lcut = lcut; st.tc = tc; st.status = status; st.argmax = aidx; st.mass_q = total_mass;
            a.stats[row] = st;
        }
    }
    CI_PROF(8);
    // After the mass exchange nobody reads a peer's memory; after a list path peers may still be gathering: wait for them.
    if (done) cluster.sync();
    CI_PROF(9);
    };  // process_row

    if (a.prof && tid == 0 && (int)blockIdx.x < a.prof_slots) {
        unsigned long long gt; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(gt));
        unsigned smid; asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        a.prof[(size_t)blockIdx.x * 16 + 15] = (long long)gt; a.prof[(size_t)blockIdx.x * 16 + 14] = smid;
    }
    int it = 0;
    for (long long row = blockIdx.x / CS; row < n_rows; row += n_clusters, ++it) {
        if (it) __syncthreads();                               // every thread is done with the previous row's buffers
        const long long nxt = row + n_clusters < n_rows ? row + n_clusters : -1;
        process_row((int)row, it, true, nxt);
    }
    // Deferred rows still waiting; then the rows that were set aside take the generic path.
    if (it == 0) cluster.barrier_wait();                       // (a cluster without rows still completes the opening barrier)
    // (A cluster that has deferred no row and set none aside is done: nobody reads a peer's memory any more.)
    if (fast_seq == 0 && n_set_aside == 0) { CI_PROF_END(); return; }
    flush();
    if (sc->any_retry) {
        int n_all = 0;
        if (tid == 0) {
            for (int i = 0; i < sc->n_retry_common; ++i) sc->retry_all[n_all++] = sc->retry_common[i];
            for (int q = 0; q < CS; ++q) {
                const Scratch* ps = cluster.map_shared_rank(sc, q);
                const int nq = ps->n_retry_mine;
                for (int i = 0; i < nq && i < CI_RETRY; ++i) sc->retry_all[n_all++] = ps->retry_mine[i];
            }
            sc->bcast_i[0] = n_all;
        }
        cluster.sync();                                        // every CTA has read the peers' lists
        n_all = sc->bcast_i[0];
        for (int i = 0; i < n_all; ++i, ++it) {
            __syncthreads();
            process_row(sc->retry_all[i], it, false, -1);
        }
    }
    CI_PROF_END();
}

// ------------------------------------------------------------------------------------------------ host side
int colinfer_launch_stream(const void*, int, const int32_t*, int, int, const colinfer_sampler_params*, const void*, int, const float*,
                           int64_t*, colinfer_row_stats*, int32_t*, int, int, int, int, cudaStream_t);

#ifdef COLINFER_PROFILE
static long long* g_prof = nullptr;                        // profiling builds only: cycles per phase of later launches
static int g_prof_slots = 0;
#endif
static const int kFixedSmem = 24 * 1024 + (CI_WARPS * CI_WLIST + 8 * CI_PCAP) * (int)sizeof(Cand) + CI_MAX_CHUNKS * 8 +
                              (int)sizeof(Xch) + (int)sizeof(Scratch) + 64;

static const int kMaxSmem = 226 * 1024;                    // of any geometry
static const void* sample_kernel(int cluster) { return cluster == 8 ? (const void*)k_sample<true> : (const void*)k_sample<false>; }
static cudaError_t sample_opt_in(int cluster) {
    static SmemOptIn opt_in[2];
    return opt_in[cluster == 8](sample_kernel(cluster), kMaxSmem);
}

// List entries per warp: what clusters of eight hold in 128 warps, spread over fewer, as far as the slice leaves room.  With 24 a
// warp whatever the cluster, rows with a top_k of a thousand overflowed a list in clusters of four and went through the radix
// select: 24 fp32 rows of 151,936 logits 99 us, 43 us with these.
static int list_cap(int cluster, int slice) {
    const int want = CI_WLIST * 8 / cluster, room = CI_WLIST + (kMaxSmem - slice * 4 - kFixedSmem) / (CI_WARPS * (int)sizeof(Cand));
    return want < room ? want : room;
}

// forced: 0 = the smallest cluster that holds the row; 1, 2, 4, 8 = that cluster size
static int pick_geometry(int V, int dtype, const void* logits, int forced, colinfer_geometry* g) {
    if (V <= 0) return 1;
    const int cap2 = (113 * 1024 - kFixedSmem) / 4;           // slice elements that allow two CTAs per SM
    const int cap1 = (kMaxSmem - kFixedSmem) / 4;           // one CTA per SM
    const int max_slice = CI_CHUNK * CI_MAX_CHUNKS;
    int cs = 0, slice = 0;
    auto slice_for = [&](int c) { return (((V + c - 1) / c) + 127) & ~127; };
    if (forced > 0) {
        cs = forced; slice = slice_for(cs);
        if (slice > cap1 || slice > max_slice) return 1;
    } else {
        for (int c = 1; c <= 8 && !cs; c *= 2) if (slice_for(c) <= cap2 && slice_for(c) <= max_slice) { cs = c; slice = slice_for(c); }
        for (int c = 1; c <= 8 && !cs; c *= 2) if (slice_for(c) <= cap1 && slice_for(c) <= max_slice) { cs = c; slice = slice_for(c); }
        if (!cs) return 1;
    }
    g->cluster = cs;
    g->slice_elems = slice;
    g->smem_bytes = slice * 4 + kFixedSmem + CI_WARPS * (list_cap(cs, slice) - CI_WLIST) * (int)sizeof(Cand);
    g->bulk_copy = (dtype == COLINFER_F32 && (V % 4) == 0 && (((uintptr_t)logits) & 15) == 0) ? 1 : 0;
    return 0;
}

extern "C" int colinfer_sample_geometry(int V, int dtype, const void* logits, int cluster, colinfer_geometry* out) {
    if (cluster != 0 && cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8) return (int)cudaErrorInvalidValue;
    return pick_geometry(V, dtype, logits, cluster, out) ? (int)cudaErrorInvalidValue : 0;
}

#ifdef COLINFER_PROFILE
void colinfer_profile_buffer(long long** buf, int* slots) { *buf = g_prof; *slots = g_prof_slots; }
// (profiling builds) the first `ctas` CTAs of later launches add their cycles per phase into dev[ctas * 16]
extern "C" int colinfer_set_profile_buffer(void* dev, int ctas) {
    g_prof = reinterpret_cast<long long*>(dev);
    g_prof_slots = dev ? ctas : 0;
    return 0;
}
#else
void colinfer_profile_buffer(long long** buf, int* slots) { *buf = nullptr; *slots = 0; }
#endif

static void fill_launch(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, const colinfer_geometry& g, long long clusters, cudaStream_t st) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)(clusters * g.cluster), 1, 1);
    cfg.blockDim = dim3(CI_THREADS, 1, 1);
    cfg.dynamicSmemBytes = (size_t)g.smem_bytes;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)g.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

// Clusters of this geometry that the current device holds at once (remembered per device and geometry): the kernel is
// persistent, each cluster walks over rows, so the grid never exceeds this.
static int active_clusters(const colinfer_geometry& g) {
    static Remembered known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    return known(((uint64_t)dev << 32) | ((uint64_t)g.cluster << 24) | (uint64_t)g.smem_bytes, [&]() {
        if (sample_opt_in(g.cluster) != cudaSuccess) return -2;
        cudaLaunchConfig_t cfg; cudaLaunchAttribute attr[1];
        fill_launch(cfg, attr, g, 1024, nullptr);
        int n = 0;
        return cudaOccupancyMaxActiveClusters(&n, sample_kernel(g.cluster), &cfg) == cudaSuccess && n > 0 ? n : -3;
    });
}

extern "C" int colinfer_sample_copy_range(const void* logits, int dtype, int rows, int V, int row, int64_t* begin, int64_t* end) {
    if (rows < 1 || V < 1 || row < 0 || row >= rows || !begin || !end || (dtype != COLINFER_F32 && dtype != COLINFER_BF16)) return (int)cudaErrorInvalidValue;
    const u64 bytes = (u64)V * (dtype == COLINFER_F32 ? 4 : 2), start = (u64)(uintptr_t)logits, addr = start + (u64)row * bytes, base = addr & ~15ull;
    const uint32_t span = row_span(addr, bytes, (u64)row, (u64)(rows - 1 - row));
    *begin = (int64_t)(base + (span & 1u ? 16 : 0) - start);
    *end = (int64_t)(base + ((span & ~15u) - (uint32_t)base) - start);
    if (*end <= *begin) *begin = *end = (int64_t)(addr - start);
    return 0;
}

extern "C" int colinfer_max_active_clusters(int V, int dtype) {
    colinfer_geometry g;
    if (pick_geometry(V, dtype, nullptr, 0, &g)) return -1;
    return active_clusters(g);
}

// ---- the chunk kernel (sample_rows.cu: a CTA per row, sample_few.cu: a cluster per row)
namespace {
constexpr int kChunkMaxV = 524288, kChunkMaxSmem = 226 * 1024;
// More rows than SMs: two CTAs of 384 threads per SM, one of which reads while the other one is in its block-wide steps.  One of
// 768 where two do not fit (penalty tables of vocabularies beyond some 330,000), and for long rows with histories (one_per_sm).
// One CTA per SM over two, histories of 2,048, geometric mean of the times of mixed, top_p, top_k 1000, half greedy and top_k 50 rows:
//   rows                160/180   210    240    296    360    512    700   1,024
//   bf16  200,000         0.99                  1.04   0.99   1.14   1.11   1.14
//         216,064         0.96   1.03   1.08   0.99   1.03   1.12   1.04   1.10
//         262,144         0.95   1.01   1.05   0.94   0.99   1.09   1.07   1.09
//         280,000         0.91   0.94   1.01   0.96   0.93   1.01   1.02
//         300,000         0.91                 0.96   0.94   1.01   1.01
//   fp32  200,000         1.02                 1.07   1.09   1.19   1.16   1.21
//         216,064         1.01   1.05   1.12   1.07   1.05   1.17   1.14   1.19
//         262,144         1.00   1.05   1.11   1.05   1.00   1.15   1.10   1.14
//         280,000         0.94   1.01   1.05   0.99
//         300,000         0.97                 0.99   0.96   1.06   1.04
// The host does not see the filters, which differ: 262,144 bf16 logits, 160 rows, mixed 120 and 162 us, half greedy 77 and 110, top_p 228
// and 198, top_k 1000 141 and 111.  Where the mean is even the mixed rows decide (280,000, 512 bf16 rows: 276 and 364).
// Without histories two are the faster everywhere but for up to two rows per SM half greedy (200,000 to 262,144, either type: 0.80 to
// 0.95), and mixed at 160 (0.85 to 0.91): over the five 1.07 to 1.26.
constexpr int kTwoPerSm = 113 * 1024, kRowV = 216000, kLongRowV = 280000;
bool one_per_sm(int V, int dtype, bool pen, long long rows, int sms) {
    if (!pen || V <= kRowV) return false;
    const bool bf16 = dtype == COLINFER_BF16;
    return V >= kLongRowV ? bf16 || rows <= 2 * sms : rows <= (bf16 ? 2 * sms : sms * 5 / 4);
}

// The sets of instantiations: a CTA of 384 threads per row, two per SM (ROWS); a CTA of 768 threads per row (ROW); a cluster of
// CTAs per row (FEW).
enum { ROWS = 0, FEW = 1, ROW = 2 };
int chunk_index(int set, int dtype, bool mask) { return 4 * set + (dtype == COLINFER_F32 ? 0 : 2) + (mask ? 1 : 0); }
const void* chunk_kernel(int ki) { return ki >= 8 ? colinfer_row_kernel(ki - 8) : ki >= 4 ? colinfer_few_kernel(ki - 4) : colinfer_rows_kernel(ki); }
int chunk_smem(int set, int V, bool pen) { return set == FEW ? colinfer_few_smem(V, pen) : set == ROW ? colinfer_row_smem(V, pen) : colinfer_rows_smem(V, pen); }

// The device's number of SMs, and once per device and kernel the opt-in to large shared memory.
int chunk_device(int ki, int* dev_out, int* sms_out) {
    static bool opted[kMaxDevices][12] = {};
    static int sms[kMaxDevices] = {};
    static std::mutex guard;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return (int)cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(guard);
    if (!opted[dev][ki]) {
        e = cudaFuncSetAttribute(chunk_kernel(ki), cudaFuncAttributeMaxDynamicSharedMemorySize, kChunkMaxSmem);
        if (e == cudaSuccess && !sms[dev]) e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        opted[dev][ki] = true;
    }
    *dev_out = dev; *sms_out = sms[dev];
    return 0;
}

void chunk_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int set, int cluster, long long groups, int smem, cudaStream_t st) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)(groups * cluster), 1, 1);
    cfg.blockDim = dim3((unsigned)(set == FEW ? colinfer_few_threads() : set == ROW ? colinfer_row_threads() : colinfer_rows_threads()), 1, 1);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = set == FEW ? 1 : 0;
}

// Clusters of `cluster` CTAs that the device holds at once (remembered).
int chunk_clusters(int dev, int ki, int cluster, int smem) {
    static Remembered known;
    return known(((uint64_t)dev << 40) | ((uint64_t)ki << 32) | ((uint64_t)cluster << 24) | (uint64_t)smem, [&]() {
        cudaLaunchConfig_t cfg; cudaLaunchAttribute attr[1];
        chunk_config(cfg, attr, FEW, cluster, 1024, smem, nullptr);
        int n = 0;
        return cudaOccupancyMaxActiveClusters(&n, chunk_kernel(ki), &cfg) == cudaSuccess ? n : -1;
    });
}

// Launches the chunk kernel where it is the faster one; returns -1 where it is not (nothing launched), else a CUDA error code.
int launch_chunk(const void* logits, int dtype, const int32_t* mask, int mask_rows, int W, const colinfer_sampler_params* params, const void* pos,
                 int pos_is_i64, const float* u, int64_t* out_ids, colinfer_row_stats* stats, int32_t* status, int B, int R, int V, int flags,
                 const colinfer_second_rows& second, cudaStream_t stream) {
    const long long rows = second.rows;
    if (V > kChunkMaxV || rows > 0x7ffffffeLL) return -1;
    const bool pen = params->history != nullptr;
    int set = ROWS, C = 1, dev = 0, sms = 0;
    {
        const int rc = chunk_device(chunk_index(ROWS, dtype, mask != nullptr), &dev, &sms);
        if (rc) return rc;
    }
    if (rows <= sms) {
        // At most a row per SM, more than the cluster-resident kernel holds at once: a cluster of two or four CTAs per row, where
        // they all run at once.  From 75 rows on there is one CTA per row either way, and the streaming kernel's 1,024 threads get
        // a row through sooner.  60 fp32 rows of 151,936 logits, streaming kernel (half of the SMs idle) and here: mixed filters 61
        // and 52 us, top-p 59 and 52, top_k 50 34 and 24, top_k 1000 67 and 65, no filter 27 and 28, greedy 11 and 16; bf16 mixed 97
        // and 57, top-p 73 and 54, no filter 27 and 27.  The host does not see the filters.
        const int ki = chunk_index(FEW, dtype, mask != nullptr), smem = colinfer_few_smem(V, pen);
        if (smem > kChunkMaxSmem) return -1;
        const int rc = chunk_device(ki, &dev, &sms);
        if (rc) return rc;
        for (C = 4; C >= 2; C /= 2) {
            if (V >= 16384 * C && rows <= chunk_clusters(dev, ki, C, smem)) { set = FEW; break; }
        }
        if (set != FEW) return -1;
        // More rows than SMs.  149 and 200 fp32 rows of 151,936, streaming kernel and here: mixed 67, 68 and 69, 73 us; top-p 122, 124
        // and 94, 99; top_k 50 60, 74 and 35, 37; top_k 1000 123, 127 and 56, 61; half greedy 46, 48 and 45, 50; greedy 29, 30 and
        // 24, 28 (a wide row alone on an SM has a third of the threads here).  400 rows: mixed 120 and 103, top-p 187 and 158, no filter
        // 99 and 103; 592: 168 and 135, 245 and 195, 133 and 130.
    } else if (one_per_sm(V, dtype, pen, rows, sms) || colinfer_rows_smem(V, pen) > kTwoPerSm) set = ROW;
    const int smem = chunk_smem(set, V, pen), ki = chunk_index(set, dtype, mask != nullptr);
    if (smem > kChunkMaxSmem) return -1;
    {
        const int rc = chunk_device(ki, &dev, &sms);
        if (rc) return rc;
    }
    colinfer_sample_args a;
    a.logits = logits;
    a.mask = mask; a.mask_rows = mask_rows; a.W = W;
    a.p = *params;
    a.pos = pos; a.pos_i64 = pos_is_i64; a.u = u;
    a.out = out_ids; a.stats = stats; a.status = status;
    a.B = B; a.R = R; a.V = V; a.flags = flags; a.cluster = C; a.second = second;
    cudaLaunchConfig_t cfg; cudaLaunchAttribute attr[1];
    chunk_config(cfg, attr, set, C, rows, smem, stream);
    void* args[] = {&a};
    return (int)cudaLaunchKernelExC(&cfg, chunk_kernel(ki), args);
}
}  // namespace

static const int kMinSlice = 4096;                         // logits per CTA of a cluster at least

// Both sets of rows (colinfer_second_rows), or -1 where only separate launches take them (nothing is launched then).
static int sample_rows(const void* logits, const void* logits2, int dtype, const int32_t* mask, int mask_rows, int W,
                       const colinfer_sampler_params* params, const void* pos, int pos_is_i64, const float* u,
                       int64_t* out_ids, colinfer_row_stats* stats, int32_t* status,
                       int B, int R, int R2, int V, int flags, void* stream) {
    if (B < 0 || R < 0 || V <= 0) return (int)cudaErrorInvalidValue;
    if ((long long)B * R == 0) return 0;
    if (!logits || !params || (!out_ids && !stats)) return (int)cudaErrorInvalidValue;
    if (dtype != COLINFER_F32 && dtype != COLINFER_BF16) return (int)cudaErrorInvalidValue;
    if (!params->temperature || !params->top_k || !params->top_p || !params->log_min_p) return (int)cudaErrorInvalidValue;
    if (out_ids && u == nullptr && (pos == nullptr || params->seed == nullptr)) return (int)cudaErrorInvalidValue;
    if (mask && (W < (V + 31) / 32 || mask_rows < R)) return (int)cudaErrorInvalidValue;
    if ((long long)B * R > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
    const long long rows = (long long)B * R + (long long)B * R2;
    if (rows > 0x7fffffffLL) return -1;
    colinfer_second_rows second;
    second.R = R2 > 0 ? R2 : 1; second.rows1 = R2 > 0 ? B * R : 0x7fffffff; second.rows = (int)rows;
    second.logits = R2 > 0 ? reinterpret_cast<const void*>((uintptr_t)logits2 - (uintptr_t)second.rows1 * V * (dtype == COLINFER_F32 ? 4 : 2)) : nullptr;
    // Which kernel: the caller's choice (bits COLINFER_KERNEL_* of flags), else automatic.  Few rows -- at most as many
    // as the device holds clusters at once -- are a latency problem: each row gets a cluster of eight, four or two CTAs of the
    // cluster-resident kernel.  More go to the chunk kernel, or, about a row per SM, to the streaming kernel (launch_chunk).  The
    // cluster-resident kernel also runs when a row's tables do not fit the others.
    const int choice = (flags >> 8) & 7;                   // 0 auto, 1 streaming, 2 .. 5: clusters of 1, 2, 4, 8
    if (choice > 5) return (int)cudaErrorInvalidValue;
    int forced = choice >= 2 ? (1 << (choice - 2)) : 0;
    if (choice <= 1) {
        bool use_stream = true;
        if (choice == 0) {
            // the widest cluster of which the device holds as many as there are rows, and whose CTAs have a few thousand logits
            // each (17 fp32 rows of 151,936 logits with mixed filters: clusters of four 36 us, of eight, in two turns, 46 us)
            for (int c = 8; c >= 1 && use_stream; c /= 2) {
                colinfer_geometry g0;
                if ((c > 1 ? V < kMinSlice * c : V >= 4 * kMinSlice) || pick_geometry(V, dtype, logits, c, &g0)) continue;
                const int res0 = active_clusters(g0);
                if (res0 > 0 && rows <= res0) { use_stream = false; forced = c; }
            }
        }
        if (use_stream && choice == 0) {
            const int rc = launch_chunk(logits, dtype, mask, mask_rows, W, params, pos, pos_is_i64, u, out_ids, stats, status,
                                        B, R, V, flags, second, (cudaStream_t)stream);
            if (rc >= 0) return rc;
        }
        if (use_stream && R2 > 0) return -1;
        if (use_stream) {
            const int rc = colinfer_launch_stream(logits, dtype, mask, mask_rows, W, params, pos, pos_is_i64, u, out_ids, stats, status,
                                                  B, R, V, flags, (cudaStream_t)stream);
            if (rc != (int)cudaErrorInvalidValue) return rc;
        }
    }
    colinfer_geometry g;
    if (pick_geometry(V, dtype, logits, forced, &g)) return (int)cudaErrorInvalidValue;
    const int resident = active_clusters(g);
    if (resident <= 0) return (int)cudaErrorInvalidConfiguration;
    const long long clusters = rows < resident ? rows : resident;

    SampleArgs a;
    a.logits = logits; a.dtype = dtype; a.use_bulk = g.bulk_copy && (R2 == 0 || ((uintptr_t)logits2 & 15) == 0);
    a.mask = mask; a.mask_rows = mask_rows; a.W = W;
    a.p = *params;
    a.pos = pos; a.pos_i64 = pos_is_i64; a.u = u;
    a.out = out_ids; a.stats = stats; a.status = status;
    a.B = B; a.R = R; a.V = V; a.slice_elems = g.slice_elems; a.list_cap = list_cap(g.cluster, g.slice_elems); a.flags = flags; a.second = second;
    colinfer_profile_buffer(&a.prof, &a.prof_slots);

    cudaError_t e = sample_opt_in(g.cluster);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg; cudaLaunchAttribute attr[1];
    fill_launch(cfg, attr, g, clusters, (cudaStream_t)stream);
    void* args[] = {&a};
    return (int)cudaLaunchKernelExC(&cfg, sample_kernel(g.cluster), args);
}

extern "C" int colinfer_sample(const void* logits, int dtype, const int32_t* mask, int mask_rows, int W,
                               const colinfer_sampler_params* params, const void* pos, int pos_is_i64, const float* u,
                               int64_t* out_ids, colinfer_row_stats* stats, int32_t* status,
                               int B, int R, int V, int flags, void* stream) {
    return sample_rows(logits, nullptr, dtype, mask, mask_rows, W, params, pos, pos_is_i64, u, out_ids, stats, status, B, R, 0, V, flags, stream);
}

int colinfer_sample_two(const void* logits, const void* logits2, int dtype, const int32_t* mask, int mask_rows, int W,
                        const colinfer_sampler_params* params, const void* pos, int pos_is_i64, const float* u, int64_t* out_ids,
                        colinfer_row_stats* stats, int32_t* status, int B, int R, int R2, int V, int flags, void* stream) {
    const int rc = sample_rows(logits, logits2, dtype, mask, mask_rows, W, params, pos, pos_is_i64, u, out_ids, stats, status, B, R, R2, V, flags, stream);
    if (rc >= 0) return rc;
    const int e = sample_rows(logits, nullptr, dtype, mask, mask_rows, W, params, pos, pos_is_i64, u, out_ids, stats, status, B, R, 0, V, flags, stream);
    if (e) return e;
    return sample_rows(logits2, nullptr, dtype, mask, mask_rows, W, params, nullptr, 0, nullptr, nullptr, stats + (size_t)B * R, nullptr, B, R2, 0, V, flags, stream);
}

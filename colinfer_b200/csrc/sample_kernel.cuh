// sample_kernel.cuh -- the fused logits -> token kernel (sm_100a).
//
// A row of logits is cut into chunks of 512 and read by the 16 warps of a CTA, chunk c by warp c mod 16; with few rows
// in a launch the CTAs of a thread-block cluster (2, 4 or 8) share a row, chunk c going to warp c mod 16 C of the cluster.
// Every warp pulls its own chunks into a private two-stage ring in shared memory with bulk copies (TMA, one mbarrier per
// stage, every wait bounded), so that loads are in flight while the warps compute, meet at barriers or finish a row, and
// the first chunks of the row's next pass, or of the CTA's next row, are on their way before the current pass ends.
// Two CTAs of 512 threads per SM: one streams while the other one is in its short block-wide steps.
//
// Rows start at any alignment: chunks are counted from the 16-byte boundary at or below the row's first logit ("position"
// p = token + a), what lies outside the row reads as -inf.  History penalties are applied to a chunk in shared memory before
// the pass reads it, the grammar mask to the registers it is read into; all passes then see effective logits.
//
//   greedy        one pass: maximum and its lowest index
//   top_k <= 100  one pass.  The first chunk of every warp (the CTA's sample) bounds the k-th largest logit from below; the
//                 pass lists what reaches the bound, the row is finished on the list
//   top_p, large top_k   pass 1 also counts a 4096-bucket histogram laid out from the sample's maximum; it gives the bucket
//                 of the k-th largest (the logits down to it are listed in a second pass and selected exactly), or, by
//                 estimated masses, of the top-p pivot: pass 2 sums the exact masses, per chunk those above a narrow band
//                 around the estimate, and lists the band, in which the pivot is found exactly
//   neither       pass 2 sums the masses per chunk
// The draw: the chunk in which the running kept mass reaches its target, then one warp inside that chunk.  Rows whose
// listed logits hold all of their mass (peaked rows, an active min-p) are finished from the list after one pass.
// Masses are exp(z - max) in integer units of 2^-30 and all sums are integer: results depend neither on the batch nor on
// the order of arrival nor on how many CTAs share a row.  Where a list overflows, a bound does not hold or the estimated
// band misses the pivot, an exact select over the 32-bit keys runs (slower, same result).
#pragma once
#include "common.cuh"
#include "../../include/colinfer_b200.h"

namespace smp {

constexpr int NT = 512, NW = NT / 32;
constexpr int CTAS_PER_SM = 2;
constexpr int CHUNK = 512;           // logits per chunk: 16 per lane
constexpr int RING = 4096;           // bytes of ring per warp: fp32 two stages of 2 KB; bf16 two of 1 KB and one chunk in fp32
constexpr int NB1 = 4096;            // histogram buckets
constexpr int HOFF = 1024;           // of these, above the sample's maximum
constexpr float RANGE = 25.0f;       // they span RANGE temperatures
constexpr int FASTK = 100;           // largest top_k finished from the sample's bound
constexpr int BINS = 512;            // bins of the sample and of the selections on lists
constexpr int BINS_PAD = BINS + BINS / 16;   // one spare word per sixteen: a lane reading its sixteen bins hits a bank of its own
constexpr float FAST_SCALE = 32.0f;  // sample bins per unit logit (16 units)
constexpr int KCAP = 208;            // list entries per warp: rows without a histogram,
constexpr int KCAP_CL = 144;         // the same in a CTA of a cluster (behind the pushed candidates),
constexpr int WCAP = 80;             // rows with a histogram
constexpr int GCAP = 128;            // list entries per warp gathered from all CTAs of a cluster
constexpr int FCAP = 128;            // candidates of the one-warp finish
constexpr int FIN_CAND = 64;         // entries of one bin compared pairwise
constexpr int FB_NB = 256;           // radix buckets per level of the fallback select
constexpr int PEN_TABLE = 2048;      // distinct history ids with an O(1) count
constexpr int LIST_MAX = 1400;       // logits a list selection may hold
constexpr int BAL_ROWS = 16384;      // launches up to this many rows deal their rows to the CTAs by cost class
constexpr int BAL_MINE = BAL_ROWS / 128 + 8;
constexpr int MAX_V = 524288;
constexpr long long WAIT_CYCLES = 400000000LL;
#define SM_FLT_MAX 3.402823466e38f
#define SM_POS_INF (__int_as_float(0x7f800000))
#define SM_LOW (-1e30f)              // stands in for logits without mass in the mass pass: finite through every step

struct Args {
    const void* logits;
    const int32_t* mask; int mask_rows; int W;
    colinfer_sampler_params p;
    const void* pos; int pos_i64; const float* u;
    int64_t* out; colinfer_row_stats* stats; int32_t* status;
    int B, R, V; int flags;
    int cluster;                       // CTAs per row
    int smem_bins, smem_csum, smem_bars, smem_sc, smem_pen;   // offsets of the shared-memory parts behind the ring and the lists
};

template <bool B> struct BoolTag { static constexpr bool value = B; };
struct Cand { uint32_t idx; float l; };

// A row's parameters, fetched asynchronously while the CTA works on the row before.
struct RowP {
    float T; int kk; float topp, lmp; long long seed; float rp, pp, fp; int hlen; long long pos; float u; int pad;
};

struct Sc {
    RowP rp[2];
    // published to the CTAs of the cluster (or to the CTA's own warps): the sample's maxima; the row's maximum and argmax per
    // warp; the CTA's list bound and flags; the warps' list lengths; mass sums
    float swf[NW];
    float wf[NW]; int wi[NW];
    float tw; int flags;               // 1 list overflow or no bound, 2 a wait ran out, 4 histogram not counted
    int wn[NW];
    u64 g_all[NW], g_keep[NW];
    u64 t_cnt, t_est;                  // totals of the CTA's share of the histogram
    int npush; float push_lo;          // candidates pushed to the leader, the value down to which they are complete
    int ok; float fin_cut; u64 fin_total; int fin_token;
    int fb[3]; u64 fe[3];              // finds of fine_decide
    // CTA-local
    u64 wsum[NW], woff[NW], wtotal, wsum2[NW], woff2[NW], wtotal2;
    int found; u64 found_excl;
    int ncand; float res_f; int sel_ok; uint32_t cand_kmin, cand_kmax;
    float cand_l[FIN_CAND]; u64 cand_w[FIN_CAND];
    uint32_t fo_idx[FCAP]; float fo_l[FCAP];
    int nsel; int aidx; int hist_slow; int x_chunk; u64 x_before;
    int my_rows[BAL_MINE]; int my_count;
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ int warp_id() { return threadIdx.x >> 5; }
__host__ __device__ __forceinline__ int padbin(int i) { return i + (i >> 4); }
__device__ __forceinline__ float fmax3(float a, float b, float c) { float d; asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c)); return d; }
__device__ __forceinline__ float max16(const float (&v)[16]) {
    const float a = fmax3(v[0], v[1], v[2]), b = fmax3(v[3], v[4], v[5]), c = fmax3(v[6], v[7], v[8]);
    const float d = fmax3(v[9], v[10], v[11]), e = fmax3(v[12], v[13], v[14]);
    return fmax3(fmax3(a, b, c), fmax3(d, e, v[15]), CI_NEG_INF);
}

// ------------------------------------------------------------------------------------------------ the CTAs that share a row
template <bool CL> struct Grp {
    int C, rank;
    __device__ __forceinline__ void sync() const {
        if constexpr (CL) {
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
    }
    template <class T> __device__ __forceinline__ T* at(T* p, int r) const {
        if constexpr (CL) {
            u64 out;
            asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<u64>(p)), "r"(r));
            return reinterpret_cast<T*>(out);
        } else {
            return p;
        }
    }
};

// Exclusive prefix of one value per thread (thread order) and the total.  Two __syncthreads.
__device__ __forceinline__ u64 block_excl_scan(u64 v, Sc* sc, u64& total) {
    const int lane = lane_id(), warp = warp_id();
    const u64 incl = warp_incl_scan_u64(v, lane);
    if (lane == 31) sc->wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const u64 w = lane < NW ? sc->wsum[lane] : 0ull;
        const u64 wi = warp_incl_scan_u64(w, lane);
        if (lane < NW) sc->woff[lane] = wi - w;
        if (lane == NW - 1) sc->wtotal = wi;
        if (lane == 0) sc->found = -1;
    }
    __syncthreads();
    total = sc->wtotal;
    return sc->woff[warp] + incl - v;
}

// Where the running sum of get(0..nbins-1) first reaches target: bin (-1 if never, or target 0), sum before it, total.
// Three __syncthreads.  All threads call.
template <class F>
__device__ void bins_find(F get, int nbins, u64 target, Sc* sc, int& bin, u64& before, u64& total) {
    const int per = (nbins + NT - 1) / NT;
    const int lo = min((int)threadIdx.x * per, nbins), hi = min(lo + per, nbins);
    u64 s = 0;
    for (int i = lo; i < hi; ++i) s += (u64)get(i);
    const u64 excl = block_excl_scan(s, sc, total);
    if (excl < target && target <= excl + s) {
        u64 run = excl;
        for (int i = lo; i < hi; ++i) {
            const u64 b = (u64)get(i);
            if (run + b >= target) { sc->found = i; sc->found_excl = run; break; }
            run += b;
        }
    }
    __syncthreads();
    bin = sc->found;
    before = sc->found_excl;
}

__device__ __forceinline__ u64 ceil_target(float frac, u64 total) {
    const double t = ceil((double)frac * (double)total);
    u64 q = t <= 1.0 ? 1ull : (u64)t;
    return q > total ? total : q;
}

// Bucket of a logit: floor((href - x) * scale) + hoff clamped to [0, NB1), as a rounding float add (no conversion
// instruction).  A logit exactly on an edge may land in either neighbour; every user keeps a whole bucket of margin.
__device__ __forceinline__ int fine_bucket(float x, float href, float scale, float hoff_minus_half) {
    const float t = fminf(fmaxf(fmaf(href - x, scale, hoff_minus_half), 0.0f), (float)(NB1 - 1));
    return __float_as_int(t + 8388608.0f) - 0x4B000000;
}

// Bin of a BINS-bin count histogram in which the running count reaches kk, or -1; computed by the calling warp alone.
// run_out: count down to and including that bin (all of them for -1).
__device__ __forceinline__ int warp_count_bin(const uint32_t* hist, uint32_t kk, int lane, uint32_t& run_out) {
    constexpr int PERB = BINS / 32;
    static_assert(PERB == 16, "padbin() pads after every sixteenth bin");
    uint32_t s = 0;
#pragma unroll
    for (int t = 0; t < PERB; ++t) s += hist[lane * (PERB + 1) + t];
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += x; }
    const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
    if (all < kk) { run_out = all; return -1; }
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= kk);
    const int hl = __ffs(hit) - 1;
    // the crossing lane's sixteen bins, one per lane
    const uint32_t h = lane < PERB ? hist[hl * (PERB + 1) + lane] : 0u;
    uint32_t in2 = h;
#pragma unroll
    for (int o = 1; o < PERB; o <<= 1) { const uint32_t x = __shfl_up_sync(0xffffffffu, in2, o); if (lane >= o) in2 += x; }
    in2 += __shfl_sync(0xffffffffu, incl - s, hl);
    const unsigned h2 = __ballot_sync(0xffffffffu, in2 >= kk);
    const int bl = __ffs(h2) - 1;
    run_out = __shfl_sync(0xffffffffu, in2, bl);
    return hl * PERB + bl;
}

// Sorts 128 ordered keys held four per lane (element lane * 4 + t) into descending order across the warp: a bitonic
// network of 28 compare-exchange stages, the wide ones by shuffle.
__device__ __forceinline__ void warp_sort_desc4(uint32_t (&a)[4], int lane) {
#pragma unroll
    for (int k = 2; k <= 128; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            uint32_t b[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int i = lane * 4 + t;
                const uint32_t o = j >= 4 ? __shfl_xor_sync(0xffffffffu, a[t], j >> 2) : a[t ^ (j & 3)];
                const bool take_max = ((i & j) == 0) == ((i & k) == 0);
                b[t] = take_max ? max(a[t], o) : min(a[t], o);
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) a[t] = b[t];
        }
    }
}

// ------------------------------------------------------------------------------------------------ packed fp32 pairs
__device__ __forceinline__ u64 pk2(float a, float b) { u64 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void up2(u64 p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p)); }
__device__ __forceinline__ u64 mul2(u64 a, u64 b) { u64 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ u64 add2(u64 a, u64 b) { u64 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) { u64 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }

// The masses of MassFn for pairs of logits, each as two integers: mass = (hi - HI0) * 2^15 + (lo - LO0).  The arithmetic is
// MassFn's, operation by operation, two logits per instruction; rounding the exponential to a multiple of 2^-30 takes
// two rounding additions instead of a conversion, which would double the load of the exponentials' pipe.
struct Mass2 {
    static constexpr uint32_t HI0 = 0x43C00000u, LO0 = 0x4B400000u;    // the bits of 384 = 1.5 * 2^8 and of 1.5 * 2^23
    u64 rinv, ntc, nm;
    __device__ __forceinline__ void init(const MassFn& f) { rinv = pk2(f.rinv, f.rinv); ntc = pk2(-f.tc, -f.tc); nm = pk2(-f.m, -f.m); }
    __device__ __forceinline__ void operator()(float l0, float l1, uint32_t& hi0, uint32_t& hi1, uint32_t& lo0, uint32_t& lo1) const {
        const u64 l = pk2(l0, l1);
        const u64 q0 = mul2(l, rinv);
        const u64 z = fma2(fma2(q0, ntc, l), rinv, q0);
        float y0, y1, e0, e1, a, b;
        up2(mul2(add2(z, nm), pk2(CI_LOG2E, CI_LOG2E)), y0, y1);
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(y0));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(y1));
        const u64 e = pk2(e0, e1);
        const u64 t1 = add2(e, pk2(384.0f, 384.0f));                   // e rounded to a multiple of 2^-15
        const u64 h = add2(t1, pk2(-384.0f, -384.0f));
        const u64 r = fma2(h, pk2(-1.0f, -1.0f), e);                   // the rest, exactly
        const u64 t2 = fma2(r, pk2(CI_MASS_SCALE, CI_MASS_SCALE), pk2(12582912.0f, 12582912.0f));   // in units of 2^-30, to the nearest integer
        up2(t1, a, b); hi0 = __float_as_uint(a); hi1 = __float_as_uint(b);
        up2(t2, a, b); lo0 = __float_as_uint(a); lo1 = __float_as_uint(b);
    }
};

// ------------------------------------------------------------------------------------------------ the row as its warps read it
// L2 policies: rows that are read twice ask to be kept on their first pass; everything else asks to go first.
__device__ __forceinline__ u64 l2_keep() { u64 p; asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p)); return p; }
__device__ __forceinline__ u64 l2_stream() { u64 p; asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p)); return p; }

// A warp's ring: two stages, filled in the order of the passes.  `np` is the next chunk to ask for, `rem` how many are
// left in this pass, nnp / nrem the same for the pass that follows.
struct Ring {
    uint32_t buf, bar;                 // shared-memory addresses of the stages and of their barriers
    const char* np; const char* nnp;
    int next_key;                      // the row the next pass reads (its index + 1; 0: unknown)
    uint32_t end, nend;                // low words of the rows' end addresses (16-byte aligned)
    int rem, nrem;
    int cons, iss;                     // chunks consumed and asked for
    bool keep, nkeep;
    bool dead, drop;
};

template <int ELT>
struct Reader {
    static constexpr int CHB = CHUNK * ELT;
    Ring g;
    int stride;                        // bytes between a warp's chunks
    int lane;

    __device__ __forceinline__ void issue_one(const char* p, uint32_t end, bool keep) {
        if (lane == 0) {
            const uint32_t left = end - (uint32_t)reinterpret_cast<u64>(p);
            const uint32_t bytes = left < (uint32_t)CHB ? left : (uint32_t)CHB;
            const uint32_t s = (uint32_t)g.iss & 1u;
            const u64 pol = keep ? l2_keep() : l2_stream();
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(g.bar + 8 * s), "r"(bytes) : "memory");
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                         ::"r"(g.buf + s * CHB), "l"(p), "r"(bytes), "r"(g.bar + 8 * s), "l"(pol) : "memory");
        }
    }
    // Asks for chunks until both stages are under way.
    __device__ __forceinline__ void fill() {
        while (g.iss - g.cons < 2) {
            if (g.rem > 0) {
                if (!g.drop && !g.dead) issue_one(g.np, g.end, g.keep);
                g.np += stride; --g.rem;
            } else if (g.nrem > 0) {
                if (!g.drop && !g.dead) issue_one(g.nnp, g.nend, g.nkeep);
                g.nnp += stride; --g.nrem;
            } else break;
            ++g.iss;
        }
    }
    // The stage of the next chunk; waits for its bytes.
    __device__ __forceinline__ void wait() {
        if (g.dead) return;
        const uint32_t bar = g.bar + 8 * ((uint32_t)g.cons & 1u), par = ((uint32_t)g.cons >> 1) & 1u;
        auto test = [&]() {
            uint32_t ok;
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok) : "r"(bar), "r"(par), "r"(20000u) : "memory");
            return ok != 0;
        };
        if (!test()) {
            const long long t0 = clock64();
            bool late = false;
            while (!test()) if (clock64() - t0 > WAIT_CYCLES) { late = true; break; }
            g.dead = __any_sync(0xffffffffu, late);
        }
    }
    // Gives the stage back.  `wrote`: the warp changed it with ordinary stores.
    __device__ __forceinline__ void release(bool wrote) {
        if (wrote) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        ++g.cons;
        fill();
    }
    // Begins a pass over row `key`: n chunks from `first`, the row's last byte before `end`.  Chunks that were asked for
    // ahead are used when they belong to this pass.
    __device__ __forceinline__ void begin(int key, const char* first, u64 end, int n, bool keep) {
        if (g.next_key == key) {
            g.np = g.nnp; g.rem = g.nrem;
        } else {
            while (g.iss != g.cons) { wait(); ++g.cons; }            // something else was on its way: let it land
            g.np = first; g.rem = n;
        }
        g.end = (uint32_t)end; g.keep = keep;
        g.next_key = 0; g.nrem = 0;
        fill();
    }
    __device__ __forceinline__ void then(int key, const char* first, u64 end, int n, bool keep) {
        g.next_key = key; g.nnp = first; g.nend = (uint32_t)end; g.nrem = n; g.nkeep = keep;
    }
    __device__ __forceinline__ uint32_t stage() const { return g.buf + ((uint32_t)g.cons & 1u) * CHB; }
};

__device__ __forceinline__ float lds32(uint32_t a) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory"); return v; }
__device__ __forceinline__ void sts32(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts16(uint32_t a, unsigned short v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(v) : "memory"); }
__device__ __forceinline__ float4 lds128(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts128(uint32_t a, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// Position in the chunk of a lane's e-th logit (e = 0 .. 15).
template <int ELT> __device__ __forceinline__ int pos_of(int e, int lane) {
    return ELT == 4 ? (e >> 2) * 128 + lane * 4 + (e & 3) : (e >> 3) * 256 + lane * 8 + (e & 7);
}

// The penalties of a row: its history's tokens among the CTA's chunks, in ascending order, with their counts.
struct Pen {
    bool on;
    const uint32_t* pre;               // [chunks + 1] first entry of every chunk
    const unsigned short* pos;         // [PEN_TABLE] position in its chunk
    const unsigned short* cnt;         // [PEN_TABLE]
    int cap;                           // entries in the tables; tokens beyond are counted by scanning the history
    const int32_t* hist; int hlen; float rp, pp, fp;
};

// Replaces the penalised logits of chunk c (fp32, at shared address `at`) by their penalised values.  A warp calls.
static __device__ __noinline__ void pen_patch_slow(const Pen& pen, uint32_t at, int c, int a, int V, int lane, int* hist_slow) {
    // tokens without a table entry: every first occurrence in the history whose rank lies beyond the tables
    *hist_slow = 1;
    const int t_lo = max(c * CHUNK - a, 0), t_hi = min(c * CHUNK - a + CHUNK, V);
    for (int i = lane; i < pen.hlen; i += 32) {
        const int v = __ldg(pen.hist + i);
        if (v < t_lo || v >= t_hi) continue;
        int count = 0; bool first = true;
        for (int j = 0; j < pen.hlen; ++j) {
            if (__ldg(pen.hist + j) == v) { if (j < i) { first = false; break; } ++count; }
        }
        if (!first) continue;
        const int pos = v + a - c * CHUNK;
        bool tabled = false;
        for (uint32_t r = pen.pre[c]; r < pen.pre[c + 1] && (int)r < pen.cap; ++r) tabled |= (int)pen.pos[r] == pos;
        if (tabled) continue;
        const float x = lds32(at + 4 * pos);
        if (x > CI_NEG_INF) sts32(at + 4 * pos, apply_penalty(x, count, pen.rp, pen.pp, pen.fp));
    }
}
__device__ __forceinline__ void pen_patch(const Pen& pen, uint32_t at, int c, int a, int V, int lane, int* hist_slow) {
    const uint32_t r0 = pen.pre[c], r1 = pen.pre[c + 1];
    const uint32_t rt = min(r1, (uint32_t)pen.cap);
    for (uint32_t r = r0 + lane; r < rt; r += 32) {
        const uint32_t q = at + 4 * (uint32_t)pen.pos[r];
        const float x = lds32(q);
        if (x > CI_NEG_INF) sts32(q, apply_penalty(x, (int)pen.cnt[r], pen.rp, pen.pp, pen.fp));
    }
    if (r1 > rt) pen_patch_slow(pen, at, c, a, V, lane, hist_slow);
}

// What the passes need to know of a row.
struct RowV {
    int V, a, Nc;                      // logits, position of the first one, chunks
    const int32_t* mrow; int W;        // grammar mask (NULL: none)
    Pen pen;
};

// The mask word of one lane for chunk c: words (512 c - a) / 32 + lane, lanes 0 .. 16.
__device__ __forceinline__ uint32_t mask_word(const RowV& rw, int c, int lane) {
    const int w = ((c * CHUNK - rw.a) >> 5) + lane;
    return (lane <= 16 && w >= 0 && w < rw.W) ? (uint32_t)__ldg(rw.mrow + w) : 0u;
}

// The chunk at the reader's current stage as 16 effective logits per lane.  fresh: the stage has just arrived (its edges and,
// for fp32, its penalties are still to be applied).  mw: the lane's mask word.  wrote: the stage was changed.
template <int ELT>
__device__ __forceinline__ void read_chunk(const RowV& rw, uint32_t st, uint32_t conv, int c, bool fresh, uint32_t mw, float (&v)[16], int lane,
                                           bool& wrote, int* hist_slow) {
    wrote = false;
    if (fresh) {
        if ((c == 0 && rw.a > 0) || c == rw.Nc - 1) {
            const int lo = c == 0 ? rw.a : 0, hi = rw.V + rw.a - c * CHUNK;
            for (int p = lane; p < CHUNK; p += 32)
                if (p < lo || p >= hi) { if (ELT == 4) sts32(st + 4 * p, CI_NEG_INF); else sts16(st + 2 * p, 0xFF80u); }
            wrote = true;
            __syncwarp();
        }
        if (ELT == 4 && rw.pen.on && rw.pen.pre[c] != rw.pen.pre[c + 1]) {
            pen_patch(rw.pen, st, c, rw.a, rw.V, lane, hist_slow);
            wrote = true;
            __syncwarp();
        }
    }
    if (ELT == 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 x = lds128(st + k * 512 + lane * 16);
            v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float4 x = lds128(st + k * 512 + lane * 16);           // eight bf16: upper halves of floats
            const uint32_t u[4] = {__float_as_uint(x.x), __float_as_uint(x.y), __float_as_uint(x.z), __float_as_uint(x.w)};
#pragma unroll
            for (int j = 0; j < 4; ++j) { v[8 * k + 2 * j] = __uint_as_float(u[j] << 16); v[8 * k + 2 * j + 1] = __uint_as_float(u[j] & 0xFFFF0000u); }
        }
        if (rw.pen.on && rw.pen.pre[c] != rw.pen.pre[c + 1]) {           // penalised values are fp32: through an fp32 copy of the chunk
#pragma unroll
            for (int k = 0; k < 4; ++k)
                sts128(conv + ((k >> 1) * 256 + lane * 8 + (k & 1) * 4) * 4, make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]));
            __syncwarp();
            pen_patch(rw.pen, conv, c, rw.a, rw.V, lane, hist_slow);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 x = lds128(conv + ((k >> 1) * 256 + lane * 8 + (k & 1) * 4) * 4);
                v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
            }
            __syncwarp();
        }
    }
    if (rw.mrow != nullptr) {
        constexpr int GE = ELT == 4 ? 4 : 8;                             // consecutive logits per lane
        const int sh = (-rw.a) & 31;                                     // bit of position 0 in the lanes' words
#pragma unroll
        for (int k = 0; k < 16 / GE; ++k) {
            const int bit = sh + k * (32 * GE) + lane * GE;
            const uint32_t lo = __shfl_sync(0xffffffffu, mw, bit >> 5);
            uint32_t bits = lo >> (bit & 31);
            if (sh % GE) {                                               // groups straddle words (an unaligned row)
                const uint32_t hi = __shfl_sync(0xffffffffu, mw, (bit >> 5) + 1);
                bits = __funnelshift_r(lo, hi, bit & 31);
            }
#pragma unroll
            for (int j = 0; j < GE; ++j) if (!(bits & (1u << j))) v[k * GE + j] = CI_NEG_INF;
        }
    }
}

// A lane's logit e of the current chunk, as the pass saw it (penalties; not the mask, which only removes).
template <int ELT>
__device__ __forceinline__ float peek(const RowV& rw, uint32_t st, uint32_t conv, int c, int pos) {
    if (ELT == 4) return lds32(st + 4 * pos);
    if (rw.pen.on && rw.pen.pre[c] != rw.pen.pre[c + 1]) return lds32(conv + 4 * pos);
    unsigned short h;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(st + 2 * pos) : "memory");
    return __uint_as_float((uint32_t)h << 16);
}

// Appends the logits of the chunk selected by the lanes' masks mk to the warp's list (no particular order).
template <int ELT>
__device__ __forceinline__ void list_append(const RowV& rw, Cand* list, int cap, int* wn, unsigned mk, uint32_t st, uint32_t conv, int c, int lane) {
    if (mk) {
        int at = atomicAdd(wn, __popc(mk));
        do {
            const int e = __ffs(mk) - 1;
            mk &= mk - 1;
            const int pos = pos_of<ELT>(e, lane);
            if (at < cap) { list[at].idx = (uint32_t)(c * CHUNK - rw.a + pos); list[at].l = peek<ELT>(rw, st, conv, c, pos); }
            ++at;
        } while (mk);
    }
}

// A warp's share of a set of listed logits: entries start, start + step, ... below n.
struct View { const Cand* p; int start, n, step; };

// Selects the logits of the warps' views that can belong to the top kk: BINS linear bins over [max(bound, cut), L] give the
// bin of the kk-th largest, everything down to it goes to `dst` (at most FCAP, no particular order).  Returns how many, or
// -1 when the views cannot decide.  Every logit >= bound of the row (CTA's share) is in the views.  complete: nothing that
// could tie with the kk-th lies outside dst; all_cut: dst holds everything >= cut.  bins zeroed by the caller before its last
// barrier.  Two __syncthreads.
__device__ __forceinline__ int select_top(const View& w, float bound, bool bound_is_cut, float cut, float L, int kk, uint32_t* bins, Cand* dst, Sc* sc,
                                          float& lo_out, float& scale_out, int& bstar_out, bool& complete, bool& all_cut, bool may_be_empty) {
    const int lane = lane_id();
    const float lo = fmaxf(bound, cut);
    const float scale = L > lo ? (float)(BINS - 2) / (L - lo) : 0.0f;
    auto bin_of = [&](float l) { return max(0, min(BINS - 1, __float2int_rz((L - l) * scale))); };
    for (int j = w.start; j < w.n; j += w.step) { const float l = w.p[j].l; if (l >= lo) atomicAdd(&bins[padbin(bin_of(l))], 1u); }
    if (threadIdx.x == 0) sc->nsel = 0;
    __syncthreads();
    uint32_t run_b;
    int bstar = warp_count_bin(bins, (uint32_t)kk, lane, run_b);     // every warp scans the bins itself
    lo_out = lo; scale_out = scale;
    all_cut = false;
    int n = (int)run_b;
    if (!(lo <= L)) { n = may_be_empty ? 0 : -1; bstar = BINS - 1; complete = all_cut = true; }
    else if (bstar < 0) {
        // fewer than kk listed logits reach lo: if lo is the cut, fewer than kk logits survive it and top-k removes nothing
        if (!(lo > bound || bound_is_cut) || (run_b == 0 && !may_be_empty)) n = -1;
        bstar = BINS - 1;
        complete = all_cut = true;
    } else {
        complete = true;                                             // every logit >= lo is listed, every listed one down to bstar taken
    }
    bstar_out = bstar;
    if (n > FCAP) n = -1;
    if (n > 0) {
        for (int j = w.start; j < w.n; j += w.step) {
            const Cand c = w.p[j];
            if (c.l >= lo && bin_of(c.l) <= bstar) { const int at = atomicAdd(&sc->nsel, 1); if (at < FCAP) dst[at] = c; }
        }
    }
    __syncthreads();
    return n;
}

// Top-k, top-p and the draw on nc <= FCAP candidates (sc->fo_*, token order), by warp 0.  Writes sc->ok / fin_*.
static __device__ __noinline__ void finish_warp(int nc, float lo, float scale, int bstar, bool complete, float L, float lcut_in, float tc, const MassFn mass,
                                                int kk, float topp, float u, Sc* sc) {
    const int lane = lane_id();
    auto bin_of = [&](float l) { return max(0, min(BINS - 1, __float2int_rz((L - l) * scale))); };
    constexpr int PERC = FCAP / 32;
    float l[PERC]; uint32_t q[PERC];
    static_assert(PERC == 4, "the warp sort holds four keys per lane");
    uint32_t sk[PERC];
    int surv = 0;
#pragma unroll
    for (int t = 0; t < PERC; ++t) {
        const int e = lane * PERC + t;
        l[t] = e < nc ? sc->fo_l[e] : CI_NEG_INF;
        sk[t] = e < nc ? f2key(l[t]) : 0u;
        surv += (e < nc && l[t] >= lcut_in) ? 1 : 0;
    }
    surv = (int)__reduce_add_sync(0xffffffffu, (unsigned)surv);
    // the candidates' keys in descending order (absent entries, key 0, come last): the kk-th largest is read off, the
    // top-p pivot is where the running mass of the sorted candidates reaches its target
    warp_sort_desc4(sk, lane);
    auto sorted_at = [&](int pos) {                                  // key at sorted position pos (warp-uniform pos)
        const int t = pos & 3;
        const uint32_t mine = t == 0 ? sk[0] : t == 1 ? sk[1] : t == 2 ? sk[2] : sk[3];
        return __shfl_sync(0xffffffffu, mine, pos >> 2);
    };
    float cut = lcut_in;
    bool ok = surv > 0;
    if (ok && kk <= surv) {                                          // else fewer than k survive min-p: top-k removes nothing
        const float lk = key2f(sorted_at(kk - 1));
        const float ck = lower_logit_for(scale_logit(lk, tc), tc, lk);
        ok = complete && ck >= lo && bin_of(ck) <= bstar;            // else a tie partner could lie outside the candidates
        cut = fmaxf(cut, ck);
    } else {
        ok = ok && complete;                                         // every logit >= the min-p cut is a candidate
    }
#pragma unroll
    for (int t = 0; t < PERC; ++t) q[t] = l[t] >= cut ? mass(l[t]) : 0u;
    if (ok && topp < 1.0f) {
        u64 sq[PERC], s = 0;
#pragma unroll
        for (int t = 0; t < PERC; ++t) {
            const float sl = sk[t] ? key2f(sk[t]) : CI_NEG_INF;
            sq[t] = sl >= cut ? (u64)mass(sl) : 0ull;
            s += sq[t];
        }
        const u64 incl = warp_incl_scan_u64(s, lane);
        const u64 s1 = __shfl_sync(0xffffffffu, incl, 31);
        ok = s1 > 0;
        const u64 target = ceil_target(topp, s1);
        const unsigned hit = __ballot_sync(0xffffffffu, incl >= target);
        int pos = 0;
        if (hit) {
            const int hl = __ffs(hit) - 1;
            u64 run = incl - s; int tt = 0;
#pragma unroll
            for (int t = 0; t < PERC; ++t) { run += sq[t]; if (run >= target) { tt = t; break; } }
            pos = hl * PERC + __shfl_sync(0xffffffffu, tt, hl);
        }
        const float lp = key2f(sorted_at(pos));
        if (ok) cut = fmaxf(cut, lower_logit_for(scale_logit(lp, tc), tc, lp));
#pragma unroll
        for (int t = 0; t < PERC; ++t) q[t] = l[t] >= cut ? q[t] : 0u;
    }
    u64 s = 0;
#pragma unroll
    for (int t = 0; t < PERC; ++t) s += q[t];
    const u64 incl = warp_incl_scan_u64(s, lane);
    const u64 tot = __shfl_sync(0xffffffffu, incl, 31);
    ok = ok && tot > 0;
    const u64 target = ceil_target(u, tot);
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= target);
    if (lane == 0) sc->ok = 0;
    __syncwarp();
    if (ok && lane == __ffs(hit) - 1) {
        u64 run = incl - s; int e = lane * PERC;
#pragma unroll
        for (int t = 0; t < PERC; ++t) { run += q[t]; if (run >= target) { e = lane * PERC + t; break; } }
        sc->fin_token = (int)sc->fo_idx[e]; sc->fin_cut = cut; sc->fin_total = tot; sc->ok = 1;
    }
}

// Candidates in token order: every candidate's rank among the indices, four threads per candidate.  src: nc <= FCAP entries.
__device__ __forceinline__ void order_candidates(const Cand* src, int nc, Sc* sc) {
    const int i = threadIdx.x >> 2, part = threadIdx.x & 3;          // NT / 4 = FCAP candidates
    const Cand me = i < nc ? src[i] : Cand{0xFFFFFFFFu, 0.0f};
    int r = 0;
    for (int j = part; j < nc; j += 4) r += src[j].idx < me.idx ? 1 : 0;
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    if (part == 0 && i < nc) { sc->fo_idx[r] = me.idx; sc->fo_l[r] = me.l; }
}

// Exact weighted selection among the listed logits of the warps' views: the value v with W(l > v) < target <= W(l >= v).
// BINS linear bins over (base - l) * scale, then the pivot bin's entries pairwise.  False when the pivot leaves the binned
// range or its bin is too crowded.  total: the weight of all entries.  All threads call with the same arguments.
template <class W>
__device__ bool list_select(const View& w, W wt, float base, float scale, u64 target, u64* bins, Sc* sc, float& value, u64& total) {
    const int tid = threadIdx.x;
    for (int i = tid; i < BINS; i += NT) bins[i] = 0;
    if (tid == 0) { sc->ncand = 0; sc->sel_ok = 0; sc->cand_kmin = 0xFFFFFFFFu; sc->cand_kmax = 0u; }
    __syncthreads();
    auto bin_of = [&](float l) { return max(0, min(BINS - 1, __float2int_rz((base - l) * scale))); };
    for (int i = w.start; i < w.n; i += w.step) {
        const float l = w.p[i].l;
        const u64 q = wt(l);
        if (q) atomicAdd(&bins[bin_of(l)], q);
    }
    __syncthreads();
    int b_star; u64 before;
    bins_find([&](int i) { return bins[i]; }, BINS, target, sc, b_star, before, total);
    if (b_star < 0 || b_star >= BINS - 1) return false;
    for (int i = w.start; i < w.n; i += w.step) {
        const float l = w.p[i].l;
        const u64 q = wt(l);
        if (q && bin_of(l) == b_star) {
            const int slot = atomicAdd(&sc->ncand, 1);
            if (slot < FIN_CAND) { sc->cand_l[slot] = l; sc->cand_w[slot] = q; }
            else { const uint32_t k = f2key(l); atomicMin(&sc->cand_kmin, k); atomicMax(&sc->cand_kmax, k); }
        }
    }
    __syncthreads();
    const int nc = sc->ncand;
    if (nc > FIN_CAND) {
        // A crowded pivot bin.  When all of its entries are one value (bf16 logits: a hundred tokens share every value)
        // that value is the pivot: the weight above the bin is below the target, with the bin it reaches it.
        uint32_t kmin = sc->cand_kmin, kmax = sc->cand_kmax;
        for (int i = 0; i < FIN_CAND; ++i) { const uint32_t k = f2key(sc->cand_l[i]); kmin = min(kmin, k); kmax = max(kmax, k); }
        if (kmin != kmax) return false;
        value = key2f(kmin);
        return true;
    }
    if (tid < nc) {
        const float mine = sc->cand_l[tid];
        u64 gt = 0, eq = 0;
        for (int i = 0; i < nc; ++i) {
            const float o = sc->cand_l[i];
            if (o > mine) gt += sc->cand_w[i]; else if (o == mine) eq += sc->cand_w[i];
        }
        if (before + gt < target && target <= before + gt + eq) { sc->res_f = mine; sc->sel_ok = 1; }
    }
    __syncthreads();
    value = sc->res_f;
    return sc->sel_ok != 0;
}

// One pass over the histogram, summed over the CTAs of the cluster, for everything the path decision needs: the bucket of the
// kk-th largest count, the bucket where the running count reaches cap, and the bucket where the running estimated mass
// reaches topp of its total.  CTA r sums the buckets [r, r + 1) * NB1 / C.  Buckets beyond `last` count nothing.
struct FineDecision { int b_k; u64 n_upto; u64 total_cnt; int b_cap; int b_p; u64 est_total; };
template <bool CL, class W>
__device__ FineDecision fine_decide(const Grp<CL>& g, uint32_t* hist, W west, int last, u64 kk_target, u64 cap_target, float topp, bool want_p, Sc* sc) {
    constexpr int PER = NB1 / NT;
    const int lane = lane_id(), warp = warp_id();
    const int per = CL ? PER / g.C : PER;
    const int lo = (CL ? g.rank * (NB1 / g.C) : 0) + (int)threadIdx.x * per;
    uint32_t c[PER];
#pragma unroll
    for (int t = 0; t < PER; ++t) c[t] = 0;
    if constexpr (CL) {
        for (int r = 0; r < g.C; ++r) {
            const uint32_t* h = g.at(hist, r);
#pragma unroll
            for (int t = 0; t < PER; ++t) if (t < per) c[t] += h[lo + t];
        }
    } else {
#pragma unroll
        for (int t = 0; t < PER; t += 4) {
            const uint4 x = *reinterpret_cast<const uint4*>(hist + lo + t);
            c[t] = x.x; c[t + 1] = x.y; c[t + 2] = x.z; c[t + 3] = x.w;
        }
    }
    u64 sc_c = 0, sc_e = 0;
#pragma unroll
    for (int t = 0; t < PER; ++t) {
        if (lo + t <= last && c[t]) { sc_c += c[t]; if (want_p) sc_e += (u64)c[t] * west(lo + t); } else c[t] = 0;
    }
    const u64 in_c = warp_incl_scan_u64(sc_c, lane), in_e = warp_incl_scan_u64(sc_e, lane);
    if (lane == 31) { sc->wsum[warp] = in_c; sc->wsum2[warp] = in_e; }
    __syncthreads();
    if (warp == 0) {
        const u64 w1 = lane < NW ? sc->wsum[lane] : 0ull, w2 = lane < NW ? sc->wsum2[lane] : 0ull;
        const u64 i1 = warp_incl_scan_u64(w1, lane), i2 = warp_incl_scan_u64(w2, lane);
        if (lane < NW) { sc->woff[lane] = i1 - w1; sc->woff2[lane] = i2 - w2; }
        if (lane == NW - 1) { sc->t_cnt = i1; sc->t_est = i2; }
        if (lane < 3) { sc->fb[lane] = -1; sc->fe[lane] = 0; }
    }
    g.sync();
    FineDecision o;
    u64 off_c = 0, off_e = 0;
    o.total_cnt = 0; o.est_total = 0;
    for (int r = 0; r < (CL ? g.C : 1); ++r) {
        const Sc* ps = g.at(sc, r);
        const u64 tc = ps->t_cnt, te = ps->t_est;
        if (r < g.rank) { off_c += tc; off_e += te; }
        o.total_cnt += tc; o.est_total += te;
    }
    const u64 ex_c = off_c + sc->woff[warp] + in_c - sc_c, ex_e = off_e + sc->woff2[warp] + in_e - sc_e;
    const u64 t_p = (want_p && o.est_total > 0) ? ceil_target(topp, o.est_total) : 0ull;
    auto tell = [&](int k, int b, u64 v) { for (int r = 0; r < (CL ? g.C : 1); ++r) { Sc* ps = g.at(sc, r); ps->fb[k] = b; ps->fe[k] = v; } };
    if (kk_target && ex_c < kk_target && kk_target <= ex_c + sc_c) {
        u64 run = ex_c;
#pragma unroll
        for (int t = 0; t < PER; ++t) { run += c[t]; if (run >= kk_target) { tell(0, lo + t, run); break; } }
    }
    if (cap_target && ex_c < cap_target && cap_target <= ex_c + sc_c) {
        u64 run = ex_c;
#pragma unroll
        for (int t = 0; t < PER; ++t) { run += c[t]; if (run >= cap_target) { tell(1, lo + t, 0); break; } }
    }
    if (t_p && ex_e < t_p && t_p <= ex_e + sc_e) {
        u64 run = ex_e;
#pragma unroll
        for (int t = 0; t < PER; ++t) { run += c[t] ? (u64)c[t] * west(lo + t) : 0ull; if (run >= t_p) { tell(2, lo + t, 0); break; } }
    }
    g.sync();
    o.b_k = sc->fb[0]; o.n_upto = sc->fe[0]; o.b_cap = sc->fb[1]; o.b_p = sc->fb[2];
    return o;
}

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Fetches a row's parameters into `rp` (asynchronously; cp.async.wait_all before use).  One warp, a lane per parameter.
__device__ __forceinline__ void fetch_params(const Args& a, long long row, RowP* rp, int lane) {
    const int b = (int)(row / a.R);
    auto get = [&](float* dst, const float* src, float dflt) { if (src) cp_async4(dst, src + b); else *dst = dflt; };
    switch (lane) {
        case 0: cp_async4(&rp->T, a.p.temperature + b); break;
        case 1: cp_async4(&rp->kk, a.p.top_k + b); break;
        case 2: cp_async4(&rp->topp, a.p.top_p + b); break;
        case 3: cp_async4(&rp->lmp, a.p.log_min_p + b); break;
        case 4: get(&rp->rp, a.p.repetition_penalty, 1.0f); break;
        case 5: get(&rp->pp, a.p.presence_penalty, 0.0f); break;
        case 6: get(&rp->fp, a.p.frequency_penalty, 0.0f); break;
        case 7: if (a.p.history && a.p.hist_len) cp_async4(&rp->hlen, a.p.hist_len + b); else rp->hlen = a.p.history ? a.p.hist_stride : 0; break;
        case 8: if (a.u == nullptr && a.p.seed) cp_async8(&rp->seed, a.p.seed + b); break;
        case 9:
            if (a.u == nullptr && a.pos) {
                if (a.pos_i64) cp_async8(&rp->pos, reinterpret_cast<const long long*>(a.pos) + b);
                else cp_async4(&rp->pos, reinterpret_cast<const int*>(a.pos) + b);
            }
            break;
        case 10: if (a.u) cp_async4(&rp->u, a.u + row); break;
        default: break;
    }
}
__device__ __forceinline__ float row_uniform(const Args& a, const RowP* rp, int r) {
    if (a.u != nullptr) return rp->u;
    if (a.pos != nullptr && a.p.seed != nullptr) {
        const long long p0 = a.pos_i64 ? rp->pos : (long long)*reinterpret_cast<const int*>(&rp->pos);
        return u32_to_uniform(philox_word(philox_key(rp->seed), (u64)p0 + (u64)r));
    }
    return 1.0f;
}

// CL: the launch uses clusters (a.cluster > 1 CTAs per row); ELT: bytes per logit (4 fp32, 2 bf16).
template <bool CL, int ELT>
__global__ void __launch_bounds__(NT, CTAS_PER_SM) k_sample(const __grid_constant__ Args a) {
    constexpr int CHB = CHUNK * ELT;
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    const int V = a.V;
    Grp<CL> g;
    g.C = CL ? a.cluster : 1;
    g.rank = CL ? (int)(blockIdx.x % a.cluster) : 0;
    const int GW = NW * g.C, gw = g.rank * NW + warp;            // warps of the group, this warp among them

    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* U = smem + NW * RING;
    Cand* klist = reinterpret_cast<Cand*>(U);                    // [NW][KCAP]: rows without a histogram, one CTA per row
    uint32_t* hist = reinterpret_cast<uint32_t*>(U);             // [NB1], else
    Cand* wlist = reinterpret_cast<Cand*>(U + NB1 * 4);          // [NW][WCAP]
    Cand* gath = reinterpret_cast<Cand*>(U);                     // [NW][GCAP] lists of all CTAs, over the histogram
    Cand* push = reinterpret_cast<Cand*>(U);                     // [8][FCAP] candidates of all CTAs, over the histogram
    uint32_t* bitmap = reinterpret_cast<uint32_t*>(U);           // history bitmap while the tables are built (may reach into bins, csum)
    uint32_t* sbins = reinterpret_cast<uint32_t*>(smem + a.smem_bins);   // [BINS_PAD] sample
    uint32_t* fbins = sbins + BINS_PAD;                          // [BINS_PAD] selection
    Cand* fc = reinterpret_cast<Cand*>(sbins);                   // [FCAP] candidates, over the sample's bins
    u64* bins = reinterpret_cast<u64*>(sbins);                   // [BINS] weighted selections, radix levels
    float* xbuf = reinterpret_cast<float*>(sbins);               // [CHUNK] the chunk the draw falls into
    u64* csum = reinterpret_cast<u64*>(smem + a.smem_csum);      // [chunks] kept mass per chunk (the CTA's own)
    Sc* sc = reinterpret_cast<Sc*>(smem + a.smem_sc);
    unsigned short* pcnt = reinterpret_cast<unsigned short*>(smem + a.smem_pen);   // [PEN_TABLE] (launches with histories)
    unsigned short* ppos = pcnt + PEN_TABLE;                     // [PEN_TABLE]
    uint32_t* cpre = reinterpret_cast<uint32_t*>(ppos + PEN_TABLE);    // [chunks + 1]

    Reader<ELT> rd;
    rd.lane = lane;
    rd.stride = GW * CHB;
    rd.g.buf = smem_u32(smem + warp * RING);
    rd.g.bar = smem_u32(smem + a.smem_bars) + 16 * warp;
    rd.g.rem = rd.g.nrem = 0; rd.g.cons = rd.g.iss = 0;
    rd.g.np = rd.g.nnp = nullptr; rd.g.next_key = 0; rd.g.end = rd.g.nend = 0;
    rd.g.keep = rd.g.nkeep = false;
    rd.g.dead = false; rd.g.drop = (a.flags & COLINFER_TEST_DROP_COPY) != 0;
    const uint32_t conv = rd.g.buf + 2 * CHB;                    // bf16: an fp32 copy of one chunk
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(rd.g.bar) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(rd.g.bar + 8) : "memory");
        fence_mbar_init();
    }
    __syncwarp();

    // ---------------------------------------------------------------------------------------- which rows are this group's
    const long long n_rows = (long long)a.B * a.R;
    const long long grp = CL ? blockIdx.x / a.cluster : blockIdx.x, n_grp = CL ? gridDim.x / a.cluster : gridDim.x;
    long long my_n = n_rows > grp ? (n_rows - grp + n_grp - 1) / n_grp : 0;
    // Rows differ in cost (a wide row takes two or three passes, any other one): every CTA orders them by cost class with one
    // scan -- the same order in all CTAs -- and takes every gridDim-th entry.
    const bool dealt = !CL && n_rows > n_grp && n_rows <= BAL_ROWS && gridDim.x >= 128;
    if (dealt) {
        auto row_class = [&](int row) {
            const int b = row / a.R;
            const float T = a.p.temperature[b];
            const int k = a.p.top_k[b];
            if (!((T > 0.0f) || (a.flags & COLINFER_FORCE_DISTRIBUTION))) return 2;
            return (k > 0 && k <= FASTK && k < V) ? 1 : 0;
        };
        const int per = ((int)n_rows + NT - 1) / NT;             // consecutive rows per thread
        const int lo = min(tid * per, (int)n_rows), hi = min(lo + per, (int)n_rows);
        u64 packed = 0;
        for (int row = lo; row < hi; ++row) packed += 1ull << (21 * row_class(row));
        if (tid == 0) sc->my_count = 0;
        u64 tot;
        u64 ex = block_excl_scan(packed, sc, tot);
        const int G = (int)gridDim.x;
        const long long n0 = (long long)(tot & 0x1FFFFFull), n1 = (long long)((tot >> 21) & 0x1FFFFFull);
        // Wide rows go round the CTAs first; where that round ends some CTAs hold one fewer: those get two small-top-k rows each
        // before the rest of that class (and then the greedy rows) continue round the CTAs from there.
        const int r0 = (int)(n0 % G), n_short = r0 ? G - r0 : 0;
        const long long extra = min(2ll * n_short, n1);
        for (int row = lo; row < hi; ++row) {
            const int j = row_class(row);
            const long long q = (long long)((ex >> (21 * j)) & 0x1FFFFFull);     // position inside the class
            ex += 1ull << (21 * j);
            int cta;
            if (j == 0) cta = (int)(q % G);
            else if (j == 1) cta = q < extra ? r0 + (int)(q % n_short) : (int)((r0 + q - extra) % G);
            else cta = (int)((r0 + n1 - extra + q) % G);
            if (cta == (int)blockIdx.x) sc->my_rows[atomicAdd(&sc->my_count, 1)] = row;   // any order
        }
        __syncthreads();
        my_n = sc->my_count;
    }
    auto row_at = [&](long long it) { return dealt ? (long long)sc->my_rows[it] : grp + it * n_grp; };
    auto row_base = [&](long long row, int& al, u64& end) {
        const u64 addr = reinterpret_cast<u64>(a.logits) + (u64)row * (u64)V * ELT;
        al = (int)((addr & 15) / ELT);
        end = (addr + (u64)V * ELT + 15) & ~15ull;
        return reinterpret_cast<const char*>(addr & ~15ull);
    };
    auto chunks_of = [&](int al) { return (V + al + CHUNK - 1) / CHUNK; };
    auto mine_of = [&](int nc) { return gw < nc ? (nc - gw + GW - 1) / GW : 0; };

    if (warp == 0 && my_n > 0) { fetch_params(a, row_at(0), &sc->rp[0], lane); asm volatile("cp.async.commit_group;" ::: "memory"); }

    for (long long it = 0; it < my_n; ++it) {
        const long long row = row_at(it);
        const int b = (int)(row / a.R), r = (int)(row % a.R);
        RowV rw;
        u64 row_end;
        const char* base = row_base(row, rw.a, row_end);
        rw.V = V; rw.Nc = chunks_of(rw.a); rw.W = a.W;
        rw.mrow = a.mask ? a.mask + ((size_t)b * a.mask_rows + r) * a.W : nullptr;
        const int nch = mine_of(rw.Nc);
        const char* first = base + (size_t)gw * CHB;
        const int key = (int)row + 1;
        rd.begin(key, first, row_end, nch, true);
        RowP* rp = &sc->rp[it & 1];
        if (warp == 0) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
            if (lane == 0) { rp->u = row_uniform(a, rp, r); sc->hist_slow = 0; sc->flags = 0; }
        }
        if (tid < NW) { sc->wn[tid] = 0; sc->swf[tid] = CI_NEG_INF; }
        __syncthreads();                                         // parameters are here, the previous row's shared memory is free
        const float T = rp->T;
        const bool sampled = (T > 0.0f) || (a.flags & COLINFER_FORCE_DISTRIBUTION);
        const float tc = fmaxf(T, 1e-6f);
        const int kk = rp->kk;
        const float topp = rp->topp;
        const bool fastk = sampled && kk > 0 && kk <= FASTK && kk < V;
        bool need_topk = kk > 0 && kk < V;
        const bool need_topp = topp < 1.0f;
        const bool wide = sampled && !fastk && (need_topk || need_topp);
        const bool lists = fastk || wide;
        Cand* mylist = !fastk ? wlist + warp * WCAP : CL ? push + 8 * FCAP + warp * KCAP_CL : klist + warp * KCAP;
        const int lcap = !fastk ? WCAP : CL ? KCAP_CL : KCAP;

        // ------------------------------------------------------------------------------------ penalty tables
        {
            const int hlen = max(0, min(rp->hlen, a.p.hist_stride));
            Pen& pen = rw.pen;
            pen.hist = a.p.history ? a.p.history + (size_t)b * a.p.hist_stride : nullptr;
            pen.hlen = hlen;
            pen.rp = rp->rp; pen.pp = rp->pp; pen.fp = rp->fp;
            pen.on = pen.hist != nullptr && hlen > 0 && !(pen.rp == 1.0f && pen.pp == 0.0f && pen.fp == 0.0f);
            pen.pre = cpre; pen.pos = ppos; pen.cnt = pcnt;
            pen.cap = hlen <= 65535 ? PEN_TABLE : 0;             // (the counts are 16 bits)
            if (pen.on) {
                // A bitmap of the history's tokens among the CTA's chunks (position order), popcounts per chunk, their prefix: a
                // token's rank is its table entry.  The first four ids per thread stay in registers.
                constexpr int HP = 4;
                int ht[HP];
#pragma unroll
                for (int j = 0; j < HP; ++j) { const int i = tid + j * NT; ht[j] = i < hlen ? __ldg(pen.hist + i) : -1; }
                for (int i = tid; i < rw.Nc * 4; i += NT) reinterpret_cast<uint4*>(bitmap)[i] = make_uint4(0, 0, 0, 0);
                for (int i = tid; i < PEN_TABLE / 8; i += NT) reinterpret_cast<uint4*>(pcnt)[i] = make_uint4(0, 0, 0, 0);
                auto mine = [&](int v, int& p) {
                    if (v < 0 || v >= V) return false;
                    p = v + rw.a;
                    return !CL || ((p >> 13) % g.C) == g.rank;   // chunk / 16 mod C
                };
                __syncthreads();
                auto mark = [&](int v) { int p; if (mine(v, p)) atomicOr(&bitmap[p >> 5], 1u << (p & 31)); };
#pragma unroll
                for (int j = 0; j < HP; ++j) mark(ht[j]);
                for (int i = tid + HP * NT; i < hlen; i += NT) mark(__ldg(pen.hist + i));
                __syncthreads();
                const int per = (rw.Nc + NT - 1) / NT;
                const int lo = min(tid * per, rw.Nc), hi = min(lo + per, rw.Nc);
                auto chunk_pop = [&](int c) {
                    uint32_t s = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) { const uint4 x = reinterpret_cast<const uint4*>(bitmap)[c * 4 + k]; s += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w); }
                    return s;
                };
                u64 local = 0, total_bits;
                for (int c = lo; c < hi; ++c) local += chunk_pop(c);
                uint32_t run = (uint32_t)block_excl_scan(local, sc, total_bits);
                for (int c = lo; c < hi; ++c) { cpre[c] = run; run += chunk_pop(c); }
                if (tid == 0) cpre[rw.Nc] = (uint32_t)total_bits;
                __syncthreads();
                auto enter = [&](int v) {
                    int p;
                    if (!mine(v, p)) return;
                    const int c = p >> 9, w = p >> 5;
                    uint32_t rk = cpre[c] + __popc(bitmap[w] & ((1u << (p & 31)) - 1u));
                    for (int i = c * 16; i < w; ++i) rk += __popc(bitmap[i]);
                    if ((int)rk < pen.cap) {
                        ppos[rk] = (unsigned short)(p & (CHUNK - 1));
                        atomicAdd(reinterpret_cast<uint32_t*>(pcnt) + (rk >> 1), (rk & 1) ? 65536u : 1u);
                    }
                };
#pragma unroll
                for (int j = 0; j < HP; ++j) enter(ht[j]);
                for (int i = tid + HP * NT; i < hlen; i += NT) enter(__ldg(pen.hist + i));
                __syncthreads();
            }
        }

        // ------------------------------------------------------------------------------------ what the passes ask for next
        const long long nrow = it + 1 < my_n && !CL ? row_at(it + 1) : -1;
        if (warp == 0 && it + 1 < my_n) { fetch_params(a, row_at(it + 1), &sc->rp[(it + 1) & 1], lane); asm volatile("cp.async.commit_group;" ::: "memory"); }
        auto then_next_row = [&]() {
            if (nrow >= 0) {
                int al; u64 e2;
                const char* nb = row_base(nrow, al, e2);
                rd.then((int)nrow + 1, nb + (size_t)gw * CHB, e2, mine_of(chunks_of(al)), true);
            }
        };
        auto then_this_row = [&]() { rd.then(key, first, row_end, nch, false); };

        // ------------------------------------------------------------------------------------ the sample: list bound, histogram layout
        float tw = -SM_FLT_MAX;                                  // the CTA's list bound
        float lref = CI_NEG_INF;                                 // the sample's maximum (the group's): buckets hang from it
        bool count_hist = false;
        bool fresh0 = true;                                      // the first chunk has not been read yet
        const float SCW = (float)NB1 / (RANGE * tc);
        if (lists) {
            for (int i = tid; i < 2 * BINS_PAD; i += NT) sbins[i] = 0u;
            if (wide) for (int i = tid; i < NB1 / 4; i += NT) reinterpret_cast<uint4*>(hist)[i] = make_uint4(0, 0, 0, 0);
            float gm[4] = {CI_NEG_INF, CI_NEG_INF, CI_NEG_INF, CI_NEG_INF};
            if (nch > 0) {
                float v[16];
                bool wrote;
                const uint32_t mw = rw.mrow ? mask_word(rw, gw, lane) : 0u;
                rd.wait();
                read_chunk<ELT>(rw, rd.stage(), conv, gw, true, mw, v, lane, wrote, &sc->hist_slow);
                fresh0 = false;
#pragma unroll
                for (int k = 0; k < 4; ++k) gm[k] = fmaxf(fmaxf(v[4 * k], v[4 * k + 1]), fmaxf(v[4 * k + 2], v[4 * k + 3]));
                float sm = fmaxf(fmaxf(gm[0], gm[1]), fmaxf(gm[2], gm[3]));
#pragma unroll
                for (int o = 16; o; o >>= 1) sm = fmaxf(sm, __shfl_xor_sync(0xffffffffu, sm, o));
                if (lane == 0) sc->swf[warp] = sm;
            }
            if (CL && wide) g.sync(); else __syncthreads();
            // the bins of the bound hang from the smallest finite warp maximum plus 4: a few dominant tokens in the sample
            // must not stretch them beyond the bulk
            float hi = CI_NEG_INF, lo = SM_POS_INF;
            for (int i = lane; i < ((CL && wide) ? GW : NW); i += 32) {
                const float x = (CL && wide) ? g.at(sc, i >> 4)->swf[i & 15] : sc->swf[i];
                hi = fmaxf(hi, x);
                if (x > CI_NEG_INF) lo = fminf(lo, x);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
                lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            }
            lref = hi;
            const float top = fminf(lo + 4.0f, hi);              // +inf when no warp saw a finite logit
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (gm[k] > CI_NEG_INF && top < SM_POS_INF)
                    atomicAdd(&sbins[padbin(max(0, min(BINS - 1, __float2int_rz((top - gm[k]) * FAST_SCALE))))], 1u);
            __syncthreads();
            uint32_t have;
            const int bk = warp_count_bin(sbins, (uint32_t)(fastk ? kk : 8), lane, have);
            if (bk >= 0 && bk < BINS - 1) tw = top - ((float)(bk + 1) + 0.01f) / FAST_SCALE - fabsf(top) * 1e-6f;
            if (wide && lref > CI_NEG_INF && lref < SM_POS_INF) {
                // no histogram where the list is sure to hold all the mass: the bound lies below the min-p cut, or the mass
                // horizon, of the sample's maximum already (the row's can only be larger)
                const float sure = fmaxf(lref + rp->lmp * tc, lref - 22.0f * tc) - fabsf(lref) * 1e-5f - 1e-5f * tc;
                count_hist = !(tw > -SM_FLT_MAX && tw < sure);
            }
        }

        // ------------------------------------------------------------------------------------ pass 1
        float lmax = CI_NEG_INF;
        int lidx = 0x7fffffff;
        // One pass of the warp over its chunks: f(v, chunk, stage) on every chunk.
        auto pass = [&](auto f) {
            uint32_t mw = (rw.mrow && nch > 0) ? mask_word(rw, gw, lane) : 0u;
            for (int i = 0, c = gw; i < nch; ++i, c += GW) {
                const uint32_t mcur = mw;
                if (rw.mrow && i + 1 < nch) mw = mask_word(rw, c + GW, lane);
                float v[16];
                bool wrote;
                const bool fresh = i > 0 || fresh0;
                if (fresh) rd.wait();
                const uint32_t st = rd.stage();
                read_chunk<ELT>(rw, st, conv, c, fresh, mcur, v, lane, wrote, &sc->hist_slow);
                f(v, c, st);
                rd.release(wrote || !fresh);
            }
            fresh0 = true;
        };
        auto pass_max = [&]() {
            lmax = CI_NEG_INF; lidx = 0x7fffffff;
            pass([&](const float (&v)[16], int c, uint32_t) {
                const float m = max16(v);
                if (m > lmax) {                                  // strict: the first (lowest) position of the maximum stays
                    lmax = m;
                    int e = 15;
#pragma unroll
                    for (int j = 14; j >= 0; --j) e = v[j] == m ? j : e;
                    lidx = c * CHUNK - rw.a + pos_of<ELT>(e, lane);
                }
            });
        };
        auto pass_list = [&](auto hist_tag, float t) {
            constexpr bool HIST = decltype(hist_tag)::value;
            pass([&](const float (&v)[16], int c, uint32_t st) {
                const float m = max16(v);
                lmax = fmaxf(lmax, m);
                if (HIST) {
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if (v[e] > CI_NEG_INF) atomicAdd(&hist[fine_bucket(v[e], lref, SCW, (float)HOFF - 0.5f)], 1u);
                }
                if (__ballot_sync(0xffffffffu, m >= t)) {
                    unsigned mk = 0;
#pragma unroll
                    for (int e = 0; e < 16; ++e) mk |= v[e] >= t ? 1u << e : 0u;
                    list_append<ELT>(rw, mylist, lcap, &sc->wn[warp], mk, st, conv, c, lane);
                }
            });
        };
        const bool one_pass = !sampled || fastk || (wide && !count_hist && tw > -SM_FLT_MAX);
        rd.g.keep = !one_pass;
        if (one_pass) then_next_row(); else then_this_row();
        if (!lists) pass_max();
        else if (count_hist) pass_list(BoolTag<true>{}, tw > -SM_FLT_MAX ? tw : SM_POS_INF);
        else pass_list(BoolTag<false>{}, tw > -SM_FLT_MAX ? tw : SM_POS_INF);

        // ------------------------------------------------------------------------------------ the row's maximum
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float om = __shfl_xor_sync(0xffffffffu, lmax, o);
            const int oi = __shfl_xor_sync(0xffffffffu, lidx, o);
            if (om > lmax || (om == lmax && oi < lidx)) { lmax = om; lidx = oi; }
        }
        if (lane == 0) { sc->wf[warp] = lmax; sc->wi[warp] = lidx; }
        if (lists) {
            const int bad = (sc->wn[warp] > lcap || !(tw > -SM_FLT_MAX)) ? 1 : 0;
            const int f = bad | (wide && !count_hist ? 4 : 0);
            if (lane == 0 && f) atomicOr(&sc->flags, f);
        }
        if (lane == 0 && rd.g.dead) atomicOr(&sc->flags, 2);
        if (tid == 0) sc->tw = tw;
        g.sync();
        float L = CI_NEG_INF, lo_all = -SM_FLT_MAX;
        int aidx = 0x7fffffff, fl = 0;
        for (int i = lane; i < GW; i += 32) {
            const Sc* ps = g.at(sc, i >> 4);
            const float om = ps->wf[i & 15]; const int oi = ps->wi[i & 15];
            if (om > L || (om == L && oi < aidx)) { L = om; aidx = oi; }
            lo_all = fmaxf(lo_all, ps->tw);
            fl |= ps->flags;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float om = __shfl_xor_sync(0xffffffffu, L, o);
            const int oi = __shfl_xor_sync(0xffffffffu, aidx, o);
            if (om > L || (om == L && oi < aidx)) { L = om; aidx = oi; }
            lo_all = fmaxf(lo_all, __shfl_xor_sync(0xffffffffu, lo_all, o));
            fl |= __shfl_xor_sync(0xffffffffu, fl, o);
        }
        const bool lists_ok = lists && !(fl & 1);
        bool hist_ready = count_hist && !(fl & 4) && (L - lref) * SCW < (float)(HOFF - 2);   // the maximum lies inside the buckets

        int status = 0;
        const bool finite_max = (L > CI_NEG_INF) && (L < SM_POS_INF);
        if (sampled && !finite_max) status |= COLINFER_ROW_DEGENERATE;
        float lcut = CI_NEG_INF;
        u64 total_mass = 0;
        long long token = -1;
        bool leader_wrote = false;                               // the draw's warp has stored the token itself

        // The lowest index of the maximum, for rows whose pass only listed: from the lists, else from one more pass.
        auto find_argmax = [&](bool from_lists) {
            if (from_lists) {
                uint32_t best = 0x7fffffffu;
                for (int j = lane; j < min(sc->wn[warp], lcap); j += 32) if (mylist[j].l == L) best = min(best, mylist[j].idx);
                lidx = (int)__reduce_min_sync(0xffffffffu, best);
            } else {
                rd.begin(key, first, row_end, nch, false);
                pass_max();
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    const float om = __shfl_xor_sync(0xffffffffu, lmax, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, lidx, o);
                    if (om > lmax || (om == lmax && oi < lidx)) { lmax = om; lidx = oi; }
                }
                if (lmax != L) lidx = 0x7fffffff;
            }
            if (lane == 0) sc->wi[warp] = lidx;
            g.sync();
            int x = 0x7fffffff;
            for (int i = lane; i < GW; i += 32) x = min(x, g.at(sc, i >> 4)->wi[i & 15]);
            aidx = (int)__reduce_min_sync(0xffffffffu, (unsigned)x);
        };
        if (lists && (a.stats || !finite_max)) find_argmax(lists_ok && finite_max);
        if (aidx == 0x7fffffff) aidx = 0;
        if (!sampled || !finite_max) token = aidx;

        if (sampled && finite_max) {
            const float m = scale_logit(L, tc);
            MassFn mass;
            mass.init(tc, m);
            const float thr = __fadd_rn(m, rp->lmp);
            lcut = lower_logit_for(thr, tc, __fmul_rn(thr, tc));
            const bool minp = lcut > L - 22.0f * tc - fabsf(L) * 1e-6f;
            // Logits more than 22 temperatures below the maximum have integer mass 0 (2^30 exp(-22) < 1/2): they can never
            // be drawn and add nothing to any sum, so every selection works above that horizon.  (A top-k whose k-th
            // largest lies below it removes nothing that could be drawn.)
            lcut = fmaxf(lcut, L - 22.0f * tc - fabsf(L) * 1e-6f);
            const float u = rp->u;
            bool done = false;

            // -------------------------------------------------------------------------------- finish from the lists
            // Small top-k rows; and any other row whose bound lies below the cut: every logit that carries mass is listed
            // (top-k, if any, then removes nothing beyond the list).
            if (lists_ok && (fastk || lo_all < lcut)) {
                const int kq = need_topk ? kk : 0x7fffffff;
                View w{mylist, lane, min(sc->wn[warp], lcap), 32};
                float lo, scale; int bstar; bool complete, all_cut;
                bool ok;
                int n = select_top(w, tw, false, lcut, L, kq, fbins, CL ? push + g.rank * FCAP : fc, sc, lo, scale, bstar, complete, all_cut, CL);
                const Cand* src = fc;
                if constexpr (CL) {
                    // every CTA selects its own top k, its candidates go to the first one, which selects among them
                    float plo = SM_POS_INF;
                    const Cand* own = push + g.rank * FCAP;
                    if (n > 0 && g.rank != 0) for (int i = tid; i < n; i += NT) g.at(push, 0)[g.rank * FCAP + i] = own[i];
                    if (all_cut) plo = lo;
                    else for (int i = lane; i < n; i += 32) plo = fminf(plo, own[i].l);
#pragma unroll
                    for (int o = 16; o; o >>= 1) plo = fminf(plo, __shfl_xor_sync(0xffffffffu, plo, o));
                    if (tid == 0) { sc->npush = all_cut || n < 0 || complete ? n : -1; sc->push_lo = plo; sc->ok = 0; }
                    if (tid < BINS_PAD) fbins[tid] = 0u;
                    if (NT < BINS_PAD && tid < BINS_PAD - NT) fbins[NT + tid] = 0u;
                    g.sync();
                    if (g.rank == 0) {
                        float bound = CI_NEG_INF; bool every = true; bool good = true;
                        for (int q = 0; q < g.C; ++q) {
                            const Sc* ps = g.at(sc, q);
                            good = good && ps->npush >= 0;
                            bound = fmaxf(bound, ps->push_lo);
                            every = every && ps->push_lo <= lcut;
                        }
                        if (good) {
                            const int wpr = NW / g.C, q = warp / wpr, sub = warp % wpr;
                            View w2{push + q * FCAP, sub * 32 + lane, g.at(sc, q)->npush, 32 * wpr};
                            n = select_top(w2, bound, every, lcut, L, kq, fbins, fc, sc, lo, scale, bstar, complete, all_cut, false);
                        } else n = -1;
                    }
                    ok = g.rank == 0 && n > 0;
                } else ok = n > 0;
                if (ok) {
                    order_candidates(src, n, sc);
                    __syncthreads();
                    if (warp == 0) finish_warp(n, lo, scale, bstar, complete, L, lcut, tc, mass, kq, topp, u, sc);
                } else if (tid == 0) sc->ok = 0;
                g.sync();
                const Sc* ps = g.at(sc, 0);
                done = ps->ok != 0;
                if (done) { token = ps->fin_token; lcut = ps->fin_cut; total_mass = ps->fin_total; }
                else hist_ready = hist_ready && !CL;             // (the candidates were pushed over the histogram)
                if (!done && fastk) hist_ready = false;
                // (what follows writes sc->ok / push again only after another barrier)
            }

            if (!done) {
                enum { PATH_PURE = 0, PATH_LIST = 1, PATH_BAND = 2, PATH_FALLBACK = 3 };
                int path = PATH_PURE;
                float t_hi = CI_NEG_INF, t_lo = SM_POS_INF;
                int band_top = 0, band_bot = 0;                  // buckets the band covers (from, to)
                // Bucket b holds the logits in (edge(b + 1), edge(b)].
                auto zero_hist = [&]() { for (int i = tid; i < NB1 / 4; i += NT) reinterpret_cast<uint4*>(hist)[i] = make_uint4(0, 0, 0, 0); };
                float href = lref; int hoff = HOFF;
                if (need_topk || need_topp) {
                    if (!hist_ready) {
                        // ------------------------------------------------------------------------ the histogram, from the row's maximum
                        href = L; hoff = 0;
                        if (CL) g.sync(); else __syncthreads();  // nobody reads the lists or candidates over it any more
                        zero_hist();
                        __syncthreads();
                        rd.begin(key, first, row_end, nch, true);
                        then_this_row();
                        pass([&](const float (&v)[16], int, uint32_t) {
#pragma unroll
                            for (int e = 0; e < 16; ++e) if (v[e] > CI_NEG_INF) atomicAdd(&hist[fine_bucket(v[e], href, SCW, -0.5f)], 1u);
                        });
                        g.sync();
                    }
                    auto bucket1 = [&](float x) { return fine_bucket(x, href, SCW, (float)hoff - 0.5f); };
                    auto edge = [&](int bb) { return href - (float)(bb - hoff) / SCW; };
                    // the histogram counts every finite logit; buckets wholly below the cut are left out
                    const int b_cut = bucket1(lcut);
                    const float dL = (L - href) / tc;
                    auto mass_est = [&](int i) {
                        return (u64)__float2uint_rn(exp2f(fminf(0.0f, -(((float)(i - hoff) + 0.5f) * (RANGE / (float)NB1) + dL) * CI_LOG2E)) * CI_MASS_SCALE);
                    };
                    // 700: how far down the lists reach in a small nucleus (~ 44 per warp)
                    const FineDecision fd = fine_decide<CL>(g, hist, mass_est, b_cut, need_topk ? (u64)kk : 0ull, 700ull, topp, need_topp, sc);
                    if (need_topk && (u64)kk >= fd.total_cnt) need_topk = false;   // at most k reach the cut's bucket: top-k removes nothing
                    if (need_topk) {
                        // (bucket 0 of a histogram laid out from the sample may hold logits from far above it)
                        if (fd.b_k < (hist_ready ? 1 : 0) || fd.b_k >= NB1 - 3 || fd.n_upto > (u64)LIST_MAX) path = PATH_FALLBACK;
                        else { path = PATH_LIST; t_lo = edge(fd.b_k + 2) - 0.01f / SCW - fabsf(href) * 1e-6f; }
                    } else if (need_topp) {
                        const int bp = fd.b_p, bcap = fd.b_cap;
                        const int up = ELT == 2 ? 3 : 1, dn = ELT == 2 ? 4 : 2;
                        if (fd.est_total == 0 || bp < (hist_ready ? 1 : 0)) path = PATH_FALLBACK;
                        else if (bcap < 0 || bcap > bp + dn + 1) {
                            // small nucleus: list everything down to well below the estimated pivot; nothing is "above"
                            path = PATH_BAND;
                            t_hi = SM_POS_INF;
                            t_lo = bcap < 0 ? -SM_FLT_MAX : edge(bcap);
                            band_top = 0; band_bot = bcap < 0 ? NB1 - 1 : bcap;
                        } else if (bp + dn + 2 >= NB1) path = PATH_FALLBACK;
                        else {
                            path = PATH_BAND;
                            t_hi = bp - up <= 0 ? SM_POS_INF : edge(bp - up);
                            t_lo = edge(bp + dn + 1);
                            band_top = max(0, bp - up); band_bot = bp + dn;
                            if (a.flags & COLINFER_TEST_MISS_BAND) {     // test hook: a band eight buckets off (above or below by row parity)
                                const int s8 = (row & 1) ? 8 : -8;
                                if (bp - up + s8 > 0 && bp + dn + s8 + 2 < NB1) {
                                    t_hi = edge(bp - up + s8); t_lo = edge(bp + dn + 1 + s8);
                                    band_top = bp - up + s8; band_bot = bp + dn + s8;
                                }
                            }
                        }
                    }
                }
                const float lk = fmaxf(lcut, -SM_FLT_MAX);
                if (CL) g.sync(); else __syncthreads();          // (the finds are read, the lists are free)
                auto zero_csum = [&]() { for (int c = tid; c < rw.Nc; c += NT) csum[c] = 0; };
                // adds the listed logits that survive `cut` to their chunks' kept masses (the CTA's own lists)
                auto keep_listed = [&](const Cand* list, int n, float cut) {
                    for (int j = lane; j < n; j += 32) {
                        const Cand c = list[j];
                        if (c.l >= cut) { const uint32_t q = mass(c.l); if (q) atomicAdd(&csum[(c.idx + rw.a) / CHUNK], (u64)q); }
                    }
                };
                // the warps' view of the listed logits of all CTAs (n < 0: a list overflowed)
                auto view_all = [&](Cand* list, int cap, bool& over) {
                    View w{list, lane, 0, 32};
                    over = false;
                    if constexpr (CL) {
                        int n = 0;
                        for (int q = 0; q < g.C; ++q) {
                            const int c = g.at(sc, q)->wn[warp];
                            const Cand* src = g.at(list, q);
                            if (c > cap) over = true;
                            for (int j = lane; j < min(c, cap); j += 32) if (n + j < GCAP) gath[warp * GCAP + n + j] = src[j];
                            n += min(c, cap);
                        }
                        if (n > GCAP) over = true;
                        w.p = gath + warp * GCAP; w.n = min(n, GCAP);
                        __syncwarp();
                    } else {
                        w.n = min(sc->wn[warp], cap);
                        over = sc->wn[warp] > cap;
                    }
                    over = __syncthreads_or(over) != 0;
                    return w;
                };

                // ---------------------------------------------------------------------------- large top-k (then top-p) on a list
                if (path == PATH_LIST) {
                    const float tl = fmaxf(fmaxf(t_lo, lcut), -SM_FLT_MAX);
                    mylist = CL ? wlist + warp * WCAP : klist + warp * KCAP;
                    const int cap = CL ? WCAP : KCAP;
                    if (lane == 0) sc->wn[warp] = 0;
                    __syncwarp();
                    zero_csum();
                    rd.begin(key, first, row_end, nch, false);
                    then_next_row();
                    pass([&](const float (&v)[16], int c, uint32_t st) {
                        if (__ballot_sync(0xffffffffu, max16(v) >= tl)) {
                            unsigned mk = 0;
#pragma unroll
                            for (int e = 0; e < 16; ++e) mk |= v[e] >= tl ? 1u << e : 0u;
                            list_append<ELT>(rw, mylist, cap, &sc->wn[warp], mk, st, conv, c, lane);
                        }
                    });
                    g.sync();
                    bool over;
                    View w = view_all(mylist, cap, over);
                    float cut = fmaxf(lcut, -SM_FLT_MAX);
                    bool ok = !over;
                    const float scale = (float)(BINS - 2) / fmaxf(L - tl, 1e-30f);
                    if (ok) {
                        u64 cnt = 0, surv;
                        for (int j = w.start; j < w.n; j += w.step) cnt += w.p[j].l >= cut ? 1 : 0;
                        block_excl_scan(cnt, sc, surv);
                        ok = surv > 0;
                        if (ok && (u64)kk <= surv) {             // else fewer than k survive min-p: top-k removes nothing
                            float lkk; u64 tot;
                            const float c0 = cut;
                            ok = list_select(w, [&](float l) { return (u64)(l >= c0 ? 1 : 0); }, L, scale, (u64)kk, bins, sc, lkk, tot);
                            if (ok) { cut = fmaxf(cut, lower_logit_for(scale_logit(lkk, tc), tc, lkk)); ok = cut >= tl; }   // else a tie partner could lie outside the list
                        }
                    }
                    if (ok && need_topp) {
                        const float c0 = cut;
                        u64 part = 0, s1;
                        for (int j = w.start; j < w.n; j += w.step) part += w.p[j].l >= c0 ? (u64)mass(w.p[j].l) : 0ull;
                        block_excl_scan(part, sc, s1);
                        ok = s1 > 0;
                        if (ok) {
                            float lp; u64 tot;
                            ok = list_select(w, [&](float l) { return l >= c0 ? (u64)mass(l) : 0ull; }, L, scale, ceil_target(topp, s1), bins, sc, lp, tot);
                            if (ok) { cut = fmaxf(cut, lower_logit_for(scale_logit(lp, tc), tc, lp)); ok = cut >= tl; }
                        }
                    }
                    if (ok) { lcut = cut; keep_listed(mylist, min(sc->wn[warp], cap), cut); }
                    else path = PATH_FALLBACK;
                }

                // ---------------------------------------------------------------------------- exact radix select over the keys
                // Four 8-bit levels, one pass each.  by_mass: the top-p pivot; else the kk-th largest.  False when the filter
                // removes nothing.
                auto radix_select = [&](bool by_mass, float& pivot) {
                    const float lkr = fmaxf(lcut, -SM_FLT_MAX);
                    uint32_t prefix = 0;
                    u64 target = by_mass ? 0 : (u64)kk;
                    for (int lvl = 0; lvl < 4; ++lvl) {
                        const int shift = 24 - 8 * lvl;
                        g.sync();
                        for (int i = tid; i < FB_NB; i += NT) bins[i] = 0;
                        __syncthreads();
                        rd.begin(key, first, row_end, nch, false);
                        pass([&](const float (&v)[16], int, uint32_t) {
                            for (int e = 0; e < 16; ++e) {
                                float l = v[0];
#pragma unroll
                                for (int j = 1; j < 16; ++j) l = e == j ? v[j] : l;
                                int bin = -1;
                                if (l >= lkr) {
                                    const uint32_t key = f2key(l);
                                    if (lvl == 0 || (key >> (shift + 8)) == prefix) bin = FB_NB - 1 - (int)((key >> shift) & 0xFFu);
                                }
                                // lanes of one bin add once (most keys of a level share a few bins: plain atomics would serialise)
                                const unsigned peers = __match_any_sync(0xffffffffu, bin);
                                const uint32_t w = bin < 0 ? 0u : (by_mass ? mass(l) : 1u);
                                const uint32_t lo = __reduce_add_sync(peers, w & 0xFFFFu), hi = __reduce_add_sync(peers, w >> 16);
                                if (bin >= 0 && lane == __ffs(peers) - 1) atomicAdd(&bins[bin], ((u64)hi << 16) + lo);
                            }
                        });
                        g.sync();
                        auto level = [&](int i) { u64 s = 0; for (int q = 0; q < (CL ? g.C : 1); ++q) s += g.at(bins, q)[i]; return s; };
                        int b_star; u64 before, grand;
                        if (lvl == 0) {
                            bins_find(level, FB_NB, 0, sc, b_star, before, grand);
                            if (by_mass) target = ceil_target(topp, grand);
                            else if (target >= grand) return false;
                            if (grand == 0) return false;
                            __syncthreads();
                        }
                        bins_find(level, FB_NB, target, sc, b_star, before, grand);
                        if (b_star < 0) return false;
                        target -= before;
                        prefix = (prefix << 8) | (uint32_t)(FB_NB - 1 - b_star);
                    }
                    pivot = key2f(prefix);
                    return true;
                };
                if (path == PATH_FALLBACK) {
                    status |= COLINFER_ROW_SELECT_SLOW;
                    float lpiv;
                    if (kk > 0 && kk < V && radix_select(false, lpiv)) lcut = fmaxf(lcut, lower_logit_for(scale_logit(lpiv, tc), tc, lpiv));
                    if (need_topp && radix_select(true, lpiv)) lcut = fmaxf(lcut, lower_logit_for(scale_logit(lpiv, tc), tc, lpiv));
                    path = PATH_PURE;
                }

                // ---------------------------------------------------------------------------- mass pass: kept mass per chunk
                // What bounds it: ~ 14 issue slots and one exponential per logit.
                if (path != PATH_LIST) {
                    mylist = wlist + warp * WCAP;
                    Mass2 m2;
                    m2.init(mass);
                    for (int attempt = 0; attempt < 3; ++attempt) {
                        const float lk3 = fmaxf(lcut, -SM_FLT_MAX);
                        const bool band = path == PATH_BAND;
                        uint32_t all_hi = 0, all_lo = 0;
                        u64 keep = 0;                            // lane 0: the warp's kept mass
                        const float tl = fmaxf(t_lo, lk3);
                        if (lane == 0) sc->wn[warp] = 0;
                        __syncwarp();
                        auto mass_pass = [&](auto band_tag, auto minp_tag) {
                            constexpr bool BAND = decltype(band_tag)::value;
                            constexpr bool MINP = decltype(minp_tag)::value;
                            pass([&](const float (&v)[16], int c, uint32_t st) {
                                uint32_t hi = 0, lo = 0, ahi = 0, alo = 0;
                                unsigned mk = 0;
#pragma unroll
                                for (int e = 0; e < 16; e += 2) {
                                    uint32_t h0, h1, l0, l1;
                                    // logits without mass: below the cut, or -inf
                                    const float x0 = MINP ? (v[e] >= lk3 ? v[e] : SM_LOW) : fmaxf(v[e], SM_LOW);
                                    const float x1 = MINP ? (v[e + 1] >= lk3 ? v[e + 1] : SM_LOW) : fmaxf(v[e + 1], SM_LOW);
                                    m2(x0, x1, h0, h1, l0, l1);
                                    hi += h0 + h1; lo += l0 + l1;
                                    if (BAND) {
                                        if (x0 > t_hi) { ahi += h0 - Mass2::HI0; alo += l0 - Mass2::LO0; }
                                        else if (x0 >= tl) mk |= 1u << e;
                                        if (x1 > t_hi) { ahi += h1 - Mass2::HI0; alo += l1 - Mass2::LO0; }
                                        else if (x1 >= tl) mk |= 2u << e;
                                    }
                                }
                                hi -= 16 * Mass2::HI0; lo -= 16 * Mass2::LO0;
                                if (BAND) { all_hi += hi; all_lo += lo; hi = ahi; lo = alo; }
                                const uint32_t chi = __reduce_add_sync(0xffffffffu, hi);
                                const int clo = (int)__reduce_add_sync(0xffffffffu, lo);
                                if (lane == 0) { const u64 q = ((u64)chi << 15) + (u64)(long long)clo; csum[c] = q; keep += q; }
                                if (BAND) list_append<ELT>(rw, mylist, WCAP, &sc->wn[warp], mk, st, conv, c, lane);
                            });
                        };
                        rd.begin(key, first, row_end, nch, false);
                        then_next_row();
                        const bool mp = minp || path == PATH_PURE;   // after the fallback the cut is a pivot
                        if (band) { if (mp) mass_pass(BoolTag<true>{}, BoolTag<true>{}); else mass_pass(BoolTag<true>{}, BoolTag<false>{}); }
                        else { if (mp) mass_pass(BoolTag<false>{}, BoolTag<true>{}); else mass_pass(BoolTag<false>{}, BoolTag<false>{}); }
                        if (!band) break;
                        const u64 wall = ((u64)__reduce_add_sync(0xffffffffu, all_hi) << 15) + (u64)(long long)(int)__reduce_add_sync(0xffffffffu, all_lo);
                        if (lane == 0) { sc->g_all[warp] = wall; sc->g_keep[warp] = keep; }
                        g.sync();
                        u64 s1 = 0, s_above = 0;
                        for (int i = lane; i < GW; i += 32) { const Sc* ps = g.at(sc, i >> 4); s1 += ps->g_all[i & 15]; s_above += ps->g_keep[i & 15]; }
                        s1 = warp_sum_u64(s1); s_above = warp_sum_u64(s_above);
                        bool over;
                        View w = view_all(mylist, WCAP, over);
                        const u64 target = ceil_target(topp, s1);
                        bool ok = !over && s1 > 0 && s_above < target;
                        if (ok) {
                            const float bs = t_hi < SM_POS_INF ? t_hi : L;
                            // (a small nucleus lists everything above the cut: the bins span [cut, base], not [-max, base])
                            const float scale = (float)(BINS - 2) / fmaxf(bs - fmaxf(t_lo, lk3), 1e-30f);
                            float lp; u64 s_band;
                            ok = list_select(w, [&](float l) { return (u64)mass(l); }, bs, scale, target - s_above, bins, sc, lp, s_band);
                            if (ok) {
                                const float cut2 = fmaxf(lcut, lower_logit_for(scale_logit(lp, tc), tc, lp));
                                if (cut2 < t_lo) ok = false;     // a tie partner could lie below the band
                                else { lcut = cut2; keep_listed(mylist, min(sc->wn[warp], WCAP), lcut); }
                            }
                        }
                        if (ok) break;
                        status |= COLINFER_ROW_SELECT_SLOW;
                        bool found_band = false;
                        if (attempt == 0 && !over && s1 > 0) {
                            // The estimated band missed the pivot.  Exact masses of the BINS buckets next to the band, on the side
                            // the pivot lies, give its bucket; the mass pass then runs again around it.
                            const int w0 = target <= s_above ? max(0, band_top - BINS + 1) : max(0, band_bot);
                            g.sync();
                            for (int i = tid; i < BINS; i += NT) bins[i] = 0;
                            __syncthreads();
                            u64 hi = 0;
                            rd.begin(key, first, row_end, nch, false);
                            pass([&](const float (&v)[16], int, uint32_t) {
#pragma unroll
                                for (int e = 0; e < 16; ++e) {
                                    if (v[e] >= lk3) {
                                        const int bb = fine_bucket(v[e], href, SCW, (float)hoff - 0.5f);
                                        if (bb < w0) hi += (u64)mass(v[e]);
                                        else if (bb < w0 + BINS) atomicAdd(&bins[bb - w0], (u64)mass(v[e]));
                                    }
                                }
                            });
                            hi = warp_sum_u64(hi);
                            if (lane == 0) sc->g_all[warp] = hi;
                            g.sync();
                            u64 s_hi = 0;
                            for (int i = lane; i < GW; i += 32) s_hi += g.at(sc, i >> 4)->g_all[i & 15];
                            s_hi = warp_sum_u64(s_hi);
                            int bw = -1; u64 bef, tw2;
                            auto win = [&](int i) { u64 s = 0; for (int q = 0; q < (CL ? g.C : 1); ++q) s += g.at(bins, q)[i]; return s; };
                            if (target > s_hi) bins_find(win, BINS, target - s_hi, sc, bw, bef, tw2);
                            g.sync();
                            if (bw >= 0) {
                                const int bstar = w0 + bw;
                                t_hi = bstar - 1 <= 0 ? SM_POS_INF : href - (float)(bstar - 1 - hoff) / SCW;
                                t_lo = href - (float)(bstar + 2 - hoff) / SCW;
                                found_band = true;
                            }
                        }
                        if (!found_band) {
                            // a list overflowed, or the pivot lies far from the estimate: exact radix select by mass
                            float lpiv;
                            if (radix_select(true, lpiv)) lcut = fmaxf(lcut, lower_logit_for(scale_logit(lpiv, tc), tc, lpiv));
                            path = PATH_PURE;
                        }
                        g.sync();
                    }
                }

                // ---------------------------------------------------------------------------- the draw: chunk, then logit
                g.sync();                                        // the chunks' kept masses are complete
                {
                    const int per = (rw.Nc + NT - 1) / NT;
                    const int c_lo = min(tid * per, rw.Nc), c_hi = min(c_lo + per, rw.Nc);
                    auto kept = [&](int c) { return g.at(csum, CL ? (c >> 4) % g.C : 0)[c]; };
                    u64 s = 0;
                    for (int c = c_lo; c < c_hi; ++c) s += kept(c);
                    const u64 excl = block_excl_scan(s, sc, total_mass);
                    const u64 target = ceil_target(u, total_mass);
                    if (total_mass > 0 && excl < target && target <= excl + s) {
                        u64 run = excl;
                        for (int c = c_lo; c < c_hi; ++c) {
                            const u64 q = kept(c);
                            if (run + q >= target) { sc->x_chunk = c; sc->x_before = run; break; }
                            run += q;
                        }
                    }
                    __syncthreads();
                    if (total_mass == 0) { status |= COLINFER_ROW_DEGENERATE; if (lists && !a.stats) find_argmax(false); token = aidx; }
                    else {
                        leader_wrote = true;
                        const int c = sc->x_chunk;
                        if (warp == 0 && (!CL || ((c >> 4) % g.C) == g.rank)) {
                            // the chunk in fp32, penalties applied (its CTA has the tables), then masked
                            const uint32_t xb = smem_u32(xbuf);
                            for (int p = lane; p < CHUNK; p += 32) {
                                const int t = c * CHUNK + p - rw.a;
                                float x = CI_NEG_INF;
                                if (t >= 0 && t < V)
                                    x = ELT == 4 ? __ldcg(reinterpret_cast<const float*>(base) + c * CHUNK + p)
                                                 : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[c * CHUNK + p]);
                                xbuf[p] = x;
                            }
                            __syncwarp();
                            if (rw.pen.on) pen_patch(rw.pen, xb, c, rw.a, V, lane, &sc->hist_slow);
                            __syncwarp();
                            const float lkf = fmaxf(lcut, -SM_FLT_MAX);
                            u64 q16 = 0; uint32_t q[16];
#pragma unroll
                            for (int e = 0; e < 16; ++e) {       // sixteen consecutive logits per lane
                                const int p = lane * 16 + e, t = c * CHUNK + p - rw.a;
                                float x = xbuf[p];
                                if (rw.mrow && t >= 0 && t < V && !((__ldg(rw.mrow + (t >> 5)) >> (t & 31)) & 1)) x = CI_NEG_INF;
                                q[e] = x >= lkf ? mass(x) : 0u;
                                q16 += q[e];
                            }
                            const u64 before = sc->x_before;
                            const u64 incl = before + warp_incl_scan_u64(q16, lane);
                            const unsigned hit = __ballot_sync(0xffffffffu, incl >= target);
                            if (hit && lane == __ffs(hit) - 1) {
                                u64 cum = incl - q16; int e = 15;
#pragma unroll
                                for (int j = 0; j < 16; ++j) { cum += q[j]; if (cum >= target) { e = j; break; } }
                                if (a.out) a.out[row] = (long long)(c * CHUNK + lane * 16 + e - rw.a);
                            }
                        }
                    }
                }
            }
        }
        if (lane == 0 && rd.g.dead) atomicOr(&sc->flags, 2);
        if (CL) g.sync(); else __syncthreads();
        if (tid == 0 && g.rank == 0) {
            for (int q = 0; q < g.C; ++q) {
                const Sc* ps = g.at(sc, q);
                if (ps->hist_slow) status |= COLINFER_ROW_HIST_SLOW;
                if (ps->flags & 2) status |= COLINFER_ROW_TIMEOUT;
            }
            if (!leader_wrote && a.out) a.out[row] = token;
            if (a.status) a.status[row] = status;
            if (a.stats) {
                colinfer_row_stats st;
                st.lmax = L; st.lcut = lcut; st.tc = tc; st.status = status; st.argmax = aidx; st.mass_q = total_mass;
                a.stats[row] = st;
            }
        }
        if (CL) g.sync();                                        // nobody reads this CTA's shared memory any more
    }
    while (rd.g.iss != rd.g.cons) { rd.wait(); ++rd.g.cons; }    // nothing is on its way when the CTA ends
}

}  // namespace smp

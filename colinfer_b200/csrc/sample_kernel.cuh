// sample_kernel.cuh -- the fused logits -> token kernel (sm_100a).
//
// A row of logits is cut into chunks of 512 and read by the NW warps of a CTA, chunk c by warp c mod NW; with few rows
// in a launch the CTAs of a thread-block cluster share a row, chunk c going to warp c mod NW * C of the cluster.
// Every warp pulls its own chunks into a private ring of NST stages in shared memory with bulk copies (TMA, one mbarrier per
// stage, every wait bounded), so that loads are in flight while the warps compute, meet at barriers or finish a row, and
// the first chunks of the row's next pass, or of the CTA's next row, are on their way before the current pass ends.
// sample_rows.cu, sample_row.cu and sample_few.cu say how many threads and CTAs per SM, and why.
//
// Rows start at any alignment: chunks are counted from the 16-byte boundary at or below the row's first logit ("position"
// p = token + a), what lies outside the row reads as -inf.  Nothing outside the buffer is read (row_span).  History penalties are
// applied to a chunk in shared memory before the pass reads it, the grammar mask to the registers it is read into; all passes then
// see effective logits.
//
//   greedy        one pass: maximum and its lowest index
//   top_k <= 100  one pass.  The first two chunks of every warp (the CTA's sample) bound the k-th largest logit from below;
//                 the pass lists what reaches the bound, the row is finished on the list
//   larger top_k  one pass as well where the sample says that the lists can hold the k largest; they are selected from there
//                 exactly.  Else a full histogram gives the bucket of the k-th largest, and a second pass lists what reaches it
//   top_p         pass 1 also sums the row's mass (approximately) and counts a histogram, laid out from the sample's maximum: of
//                 a quarter of the logits with a CTA per row, where the rows of an SM share its time, of all of them in a cluster.
//                 They say where the top-p pivot lies: pass 2 sums the exact masses, per chunk those above a band around the
//                 estimate, and lists the band, in which the pivot is found exactly
//   neither       pass 2 sums the masses per chunk
// The draw: the chunk in which the running kept mass reaches its target, then one warp inside that chunk.  Rows whose
// listed logits hold all of their mass (peaked rows, an active min-p) are finished from the list after one pass.
// Masses are exp(z - max) in integer units of 2^-30 and all sums are integer: results depend neither on the batch nor on
// the order of arrival nor on how many CTAs share a row.  Where a list overflows, a bound does not hold or the estimated
// band misses the pivot, an exact select over the 32-bit keys runs (slower, same result).
//
// What bounds it.  A pass over a row that is in HBM: bytes (592 greedy rows of 151,936 fp32 logits 64 us, of which 53 at the copy
// rate).  A wide row: the second pass's instructions, and the chains of block-wide steps between the passes, three tenths of
// its time, during which the SM's other row has the pipes to itself.  Hence masses two logits per instruction with rounding additions
// instead of conversions, a histogram of a sample, one warp that decides and one that draws while searches are repeated by every warp
// instead of published behind barriers.  A thread has 80 registers: with 64 (512 threads) the passes kept what a row needs in local
// memory, which beside 226 KB of shared memory is L2, and two rows on an SM were slower than one after the other.
// The version with 512 threads, a full histogram and two passes for every top_k above 100, and now, one B200, 151,936 fp32 logits, us:
// 592 rows greedy 69 -> 64, without a filter 138 -> 127, top_p 202 -> 194, top_k 50 82 -> 78, top_k 1000 190 -> 120; 360 bf16 rows with
// mixed filters 123 -> 99, top_p 207 -> 154.
#pragma once
#include <stddef.h>

#include "common.cuh"
#include "sample_host.h"

namespace SMP_NAME {

#ifdef COLINFER_PROFILE
// Profiling builds only: cycles per phase, summed over rows and CTAs (thread 0's clock).
__device__ unsigned long long g_prof[16];
#define SM_PROF(slot) do { if (tid == 0) { const long long t_ = clock64(); atomicAdd(&g_prof[slot], (unsigned long long)(t_ - prof_last)); prof_last = clock64(); } } while (0)
#else
#define SM_PROF(slot) do { } while (0)
#endif

constexpr int NT = SMP_THREADS, NW = NT / 32;
constexpr int NUM_SM = 148;          // (a B200's; says from how many rows on their order matters, and which CTAs start later)
constexpr int CTAS_PER_SM = SMP_CTAS;
constexpr int NST = SMP_STAGES;      // stages of a warp's ring
constexpr int CHUNK = 512;           // logits per chunk: 16 per lane
constexpr int RING = NST * 2048;     // bytes of ring per warp: a stage is 2 KB of fp32, or 1 KB of bf16 (and an fp32 copy of one chunk behind them)
constexpr int NB1 = 1024;            // histogram buckets
constexpr int HOFF = 256;            // of these, above the sample's maximum (what lies above them counts in the first)
constexpr float RANGE = 29.0f;       // they span RANGE temperatures: three quarters of that reach from the sample's maximum to the mass horizon
                                     // (what falls short of it is missing from the estimates: at 25, a row of T = 0.53 and top_p = 0.996 missed its band)
constexpr int FASTK = 100;           // largest top_k finished from the sample's bound
constexpr int BINS = 256;            // bins of the sample and of the selections on lists
constexpr float FAST_SCALE = 16.0f;  // sample bins per unit logit (16 units)
constexpr int BINS_BYTES = 4096;     // two sets of counts (or one of weights, a chunk in fp32, the candidates)
constexpr int U_BYTES = SMP_LISTS;   // lists, or histogram and lists
constexpr int FCAP = 128;            // candidates of the one-warp finish
constexpr int OFF_LISTS = NB1 * 4;   // lists behind a histogram
constexpr int KCAP = U_BYTES / 8 / NW;                       // list entries per warp: rows without a histogram,
constexpr int WCAP = (U_BYTES - NB1 * 4) / 8 / NW;           // rows with one;
// in a CTA of a cluster half of that, the other half being for what the CTAs of a cluster send each other:
constexpr int GCAP = WCAP / 2;                               // entries per warp gathered from all CTAs,
constexpr int OFF_GATHER = OFF_LISTS + GCAP * NW * 8;        // or the candidates sent to the first one, in equal shares
constexpr int PUSH = 2048;
constexpr int WCAP_CL = GCAP, KCAP_CL = OFF_GATHER / 8 / NW;
static_assert(PUSH <= GCAP * NW || SMP_CTAS == 2 || SMP_THREADS > 512, "candidates over the gathered entries");
// A band is to hold this many logits on either side of the estimated pivot: a third of what the lists hold.
constexpr int BAND_SIDE = 7 * KCAP * NW / 20 < 1200 ? 7 * KCAP * NW / 20 : 1200;
constexpr int FIN_CAND = 128;        // entries of one bin compared pairwise
constexpr int FB_NB = 256;           // radix buckets per level of the fallback select
constexpr int PEN_TABLE = 2048;      // distinct history ids with an O(1) count
constexpr int LIST_MAX = 2200;       // logits a list selection may hold
constexpr int BAL_ROWS = 16384;      // launches up to this many rows deal their rows to the CTAs by cost class
constexpr long long WAIT_CYCLES = 400000000LL;
#define SM_FLT_MAX 3.402823466e38f
#define SM_POS_INF (__int_as_float(0x7f800000))
#define SM_LOW (-1e30f)              // stands in for logits without mass in the mass pass: finite through every step

using Args = colinfer_sample_args;

template <bool B> struct BoolTag { static constexpr bool value = B; };
struct Cand { uint32_t idx; float l; };

// A row at hand.  What the phases of a row hand on lives here, not in registers: at 80 registers per thread what stays alive
// across a pass is spilled, and with 226 KB of an SM's 256 in shared memory a spill is a round trip to L2.
struct RowS {
    const char* base; uint32_t end;    // the 16-byte boundary at or below its first logit; what of it is copied (row_span)
    int row, key;                      // its index, and that plus 1
    int a, Nc;                         // position of the first logit, chunks
    const int32_t* mrow;               // grammar mask (NULL: none)
    int pen_on, pen_cap;               // penalties; entries in the tables (tokens beyond are counted by scanning the history)
    const int32_t* hist; int hlen; float rp, pp, fp;
    int cls;                           // ROW_* below
    float tc, topp, lmp, u; int kk;
    float scw;                         // histogram buckets per unit logit
    float lref; int count_hist, hist_full;   // the sample's maximum (the group's); pass 1 counts the histogram, of all logits
    float L; int aidx, status;         // the row's maximum, the lowest token that has it
    int hist_ready;
    float lcut, horizon; int minp;     // smallest kept logit; the mass horizon; the cut lies above it
    MassFn mass;
    float href; int hoff;              // histogram: bucket b holds the logits in (href - (b + 1 - hoff) / scw, href - (b - hoff) / scw]
    int path; float t_hi, t_lo; int band_top, band_bot;   // how a wide row is cut; its band, in logits and in buckets
    int drawn; long long token; u64 total;                // the draw's warp stores the token itself
    int listed;                        // the lists of pass 1 hold everything that can be kept
    int hist_slow;                     // the history has more tokens than the tables
};
enum { ROW_SAMPLED = 1, ROW_FASTK = 2, ROW_WIDE = 4 };
enum { PATH_PURE = 0, PATH_LIST = 1, PATH_BAND = 2, PATH_FALLBACK = 3 };

// A warp's ring between passes: chunks consumed, chunks under way, and of which row (index + 1; 0: none) they are; whether the warp
// asks for chunks, whether a wait of its own ran out (it then waits for nothing any more).
struct WarpRing { int cons, out, key, asks, lost; };

// Where the row after the one at hand lies (key 0: none).
struct NextRow { const char* base; uint32_t end; int key, Nc; };

struct Sc {
    RowS rows[2];                      // the row at hand and the one after it, by the parity of the row's number in the CTA
    NextRow next[2];
    WarpRing ring[NW];
    int V, W, GW, rank;                // logits per row; mask words per row; warps that share a row; this CTA among them
    int dead;                          // a wait ran out
    __align__(16) uint4 clc; u64 clc_bar;   // the answer of the hardware's work queue, its barrier
    int cls_tot[3]; unsigned short cls_pre[3][NT];   // rows per cost class: all, before each thread's
    int pen_off;                       // offset of the penalty tables in shared memory
    // published to the CTAs of the cluster (or to the CTA's own warps): the sample's maxima; the row's maximum and argmax per
    // warp; the CTA's list bound and flags; the warps' list lengths; mass sums
    float swf[NW];
    float wf[NW]; int wi[NW];
    int in_klist;                      // the lists of the row at hand take the histogram's place
    float4 pub;                        // the CTA's maximum, its lowest token, tw and flags
    float tw; int flags;               // 1 list overflow or no bound, 2 a wait ran out, 4 histogram not counted, 8 mass out of range, 16 lists behind a histogram
    int wn[NW];
    u64 g_all[NW];
    float est[NW];                     // the warps' shares of the row's mass relative to the sample's maximum
    u64 sum_all, sum_keep;             // masses of the CTA's chunks
    int nsel, npush;                   // candidates selected, candidates sent to the group's first CTA
    int ok; float fin_cut; u64 fin_total; int fin_token;
    // CTA-local
    u64 wsum[NW], woff[NW], wtotal;
    int found; u64 found_excl;
    int ncand; uint32_t cand_kmin, cand_kmax;
    float cand_l[FIN_CAND]; uint32_t cand_w[FIN_CAND];
};

// Candidates: as selected (over the sample's bins); by descending logit and by ascending token, with masses (over those of the
// selection too, once every warp has read them).
struct Fin {
    uint32_t fc_idx[FCAP]; float fc_l[FCAP];
    float sv_l[FCAP]; uint32_t sv_q[FCAP];
    uint32_t so_idx[FCAP]; float so_l[FCAP]; uint32_t so_q[FCAP];
    int ties[FCAP];
};
static_assert(sizeof(Fin) <= BINS_BYTES && 2 * FCAP * 4 <= BINS * 4, "candidates over the bins");

// Shared memory: rings, scratch, lists (or histogram and lists), bins, barriers, chunk sums, penalty tables (launches with
// histories).  The history bitmap, a bit per position, lies over lists, bins and chunk sums while the tables are built.
constexpr int OFF_SC = NW * RING;
constexpr int OFF_BARS = (OFF_SC + (int)sizeof(Sc) + 15) & ~15;
constexpr int OFF_U = (OFF_BARS + NW * 8 * NST + 127) & ~127;
constexpr int OFF_BINS = OFF_U + U_BYTES;
constexpr int OFF_CSUM = OFF_BINS + BINS_BYTES;
static_assert(NB1 == 1024, "decide_row: 32 buckets per lane");
static_assert(BINS_BYTES >= 2 * BINS * 4 && BINS_BYTES >= BINS * 8 && BINS_BYTES >= FB_NB * 8 && BINS_BYTES >= CHUNK * 4, "what lies over the bins");
__host__ __device__ inline int max_chunks(int V) { return (V + 7 + CHUNK - 1) / CHUNK; }   // a row may start seven logits into its first chunk
__host__ __device__ inline int pen_offset(int V, bool pen) {
    const int nc = max_chunks(V);
    const int over = pen ? nc * 64 - U_BYTES - BINS_BYTES : 0;      // what of the bitmap reaches into the chunk sums
    return (OFF_CSUM + (nc * 8 > over ? nc * 8 : over) + 15) & ~15;
}
__host__ __device__ inline int smem_bytes(int V, bool pen) { return pen_offset(V, pen) + (pen ? 4 * PEN_TABLE + (max_chunks(V) + 1) * 4 : 0); }

extern __shared__ __align__(128) unsigned char smem[];
__device__ __forceinline__ Sc* scratch() { return reinterpret_cast<Sc*>(smem + OFF_SC); }
__device__ __forceinline__ Fin* fin_area() { return reinterpret_cast<Fin*>(smem + OFF_BINS); }

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ int warp_id() { return threadIdx.x >> 5; }
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

// Bin of a BINS-bin count histogram in which the running count reaches kk, or -1; computed by the calling warp alone, eight
// bins per lane.  run_out: count down to and including that bin (all of them for -1).
static __device__ __noinline__ int warp_count_bin(const uint32_t* hist, uint32_t kk, uint32_t& run_out) {
    static_assert(BINS == 256, "eight bins per lane");
    const int lane = lane_id();
    const uint4 a = reinterpret_cast<const uint4*>(hist)[2 * lane], b = reinterpret_cast<const uint4*>(hist)[2 * lane + 1];
    const uint32_t p1 = a.x + a.y, p3 = p1 + a.z + a.w, p5 = p3 + b.x + b.y, s = p5 + b.z + b.w;
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += x; }
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= kk);
    if (!hit) { run_out = __shfl_sync(0xffffffffu, incl, 31); return -1; }
    const uint32_t e = incl - s, need = kk - min(kk, e);             // (of the crossing lane: how far into its bins)
    int t; uint32_t r;
    if (need <= p3) { if (need <= p1) { t = need <= a.x ? 0 : 1; r = t ? p1 : a.x; } else { t = need <= p1 + a.z ? 2 : 3; r = t == 2 ? p1 + a.z : p3; } }
    else { if (need <= p5) { t = need <= p3 + b.x ? 4 : 5; r = t == 4 ? p3 + b.x : p5; } else { t = need <= p5 + b.z ? 6 : 7; r = t == 6 ? p5 + b.z : s; } }
    const int hl = __ffs(hit) - 1;
    run_out = __shfl_sync(0xffffffffu, e + r, hl);
    return __shfl_sync(0xffffffffu, 8 * lane + t, hl);
}

// ------------------------------------------------------------------------------------------------ the row as its warps read it
// L2 policies: rows that are read twice ask to be kept on their first pass; everything else asks to go first.
__device__ __forceinline__ u64 l2_policy(bool keep) {
    u64 p;
    if (keep) asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    else asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
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

// Position in the chunk of a lane's e-th logit (e = 0 .. 15): groups of four, a group of every lane side by side.
__device__ __forceinline__ int pos_of(int e, int lane) { return (e >> 2) * 128 + lane * 4 + (e & 3); }

// The penalties of a row: its history's tokens among the CTA's chunks, in ascending order, with their counts.
struct PenTab {
    uint32_t* ent;                     // [PEN_TABLE] position in its chunk (low half), occurrences (high half)
    uint32_t* pre;                     // [chunks + 1] first entry of every chunk
};
__device__ __forceinline__ PenTab pen_tab(const Sc* sc) {
    PenTab t;
    t.ent = reinterpret_cast<uint32_t*>(smem + sc->pen_off);
    t.pre = t.ent + PEN_TABLE;
    return t;
}
// The entries of one chunk, and a lane's first one, fetched a chunk ahead.
struct PenPeek { uint32_t r0, r1, ent; };
// A row's penalties, and how many entries its tables hold.
struct PenVals { float rp, pp, fp; int cap; };
__device__ __forceinline__ PenVals pen_vals(const RowS& rw) { return PenVals{rw.rp, rw.pp, rw.fp, rw.pen_cap}; }
__device__ __forceinline__ PenPeek pen_peek(const PenTab& t, int cap, int c, int lane) {
    PenPeek k;
    k.r0 = t.pre[c]; k.r1 = t.pre[c + 1];
    k.ent = k.r0 + lane < min(k.r1, (uint32_t)cap) ? t.ent[k.r0 + lane] : 0u;
    return k;
}

// Entries beyond the warp's first 32, and tokens without a table entry (every first occurrence in the history that the tables
// do not hold).
static __device__ __noinline__ void pen_patch_more(RowS& rw, uint32_t at, int c, uint32_t r0, uint32_t r1) {
    const Sc* sc = scratch();
    const PenTab t = pen_tab(sc);
    const int lane = lane_id();
    const uint32_t rt = min(r1, (uint32_t)rw.pen_cap);
    for (uint32_t r = r0 + 32 + lane; r < rt; r += 32) {
        const uint32_t q = at + 4 * (t.ent[r] & 0xFFFFu);
        const float x = lds32(q);
        if (x > CI_NEG_INF) sts32(q, apply_penalty(x, (int)(t.ent[r] >> 16), rw.rp, rw.pp, rw.fp));
    }
    if (r1 <= rt) return;
    rw.hist_slow = 1;
    const int t_lo = max(c * CHUNK - rw.a, 0), t_hi = min(c * CHUNK - rw.a + CHUNK, sc->V);
    for (int i = lane; i < rw.hlen; i += 32) {
        const int v = __ldg(rw.hist + i);
        if (v < t_lo || v >= t_hi) continue;
        int count = 0; bool first = true;
        for (int j = 0; j < rw.hlen; ++j) {
            if (__ldg(rw.hist + j) == v) { if (j < i) { first = false; break; } ++count; }
        }
        if (!first) continue;
        const uint32_t pos = (uint32_t)(v + rw.a - c * CHUNK);
        bool tabled = false;
        for (uint32_t r = r0; r < rt; ++r) tabled |= (t.ent[r] & 0xFFFFu) == pos;
        if (tabled) continue;
        const float x = lds32(at + 4 * pos);
        if (x > CI_NEG_INF) sts32(at + 4 * pos, apply_penalty(x, count, rw.rp, rw.pp, rw.fp));
    }
}
// Replaces the penalised logits of chunk c (fp32, at shared address `at`) by their penalised values.  A warp calls.
__device__ __forceinline__ void pen_patch(RowS& rw, uint32_t at, int c, const PenPeek& k, const PenVals& v) {
    if (k.ent) {                                                         // (an entry counts at least one occurrence)
        const uint32_t q = at + 4 * (k.ent & 0xFFFFu);
        const float x = lds32(q);
        if (x > CI_NEG_INF) sts32(q, apply_penalty(x, (int)(k.ent >> 16), v.rp, v.pp, v.fp));
    }
    if (k.r1 - k.r0 > 32 || k.r1 > (uint32_t)v.cap) pen_patch_more(rw, at, c, k.r0, k.r1);
    __syncwarp();
}

// Completes the first or last chunk of a row at stage `st`: what lies outside the row reads as -inf, and the units of 16 bytes
// that no copy may fetch whole (row_span) come by ordinary loads.
template <int ELT>
static __device__ __noinline__ void mend_edges(const RowS& rw, uint32_t st, int c) {
    constexpr int UNIT = 16 / ELT;
    const int lane = lane_id(), lo = c == 0 ? rw.a : 0, hi = scratch()->V + rw.a - c * CHUNK;
    auto put = [&](int p) {
        if (ELT == 4) sts32(st + 4 * p, __ldcg(reinterpret_cast<const float*>(rw.base) + c * CHUNK + p));
        else sts16(st + 2 * p, __ldcg(reinterpret_cast<const unsigned short*>(rw.base) + c * CHUNK + p));
    };
    auto none = [&](int p) { if (ELT == 4) sts32(st + 4 * p, CI_NEG_INF); else sts16(st + 2 * p, 0xFF80u); };
    if (lane < lo) none(lane);
    for (int p = hi + lane; p < CHUNK; p += 32) none(p);
    if (c == 0 && (rw.end & 1u) && lane >= lo && lane < min(UNIT, hi)) put(lane);
    const int p = (int)((rw.end & ~15u) - (uint32_t)reinterpret_cast<u64>(rw.base)) / ELT - c * CHUNK + lane;   // from where the copies end
    if (lane < UNIT && p >= lo && p < min(hi, CHUNK)) put(p);
    __syncwarp();
}

__device__ __forceinline__ bool ring_test(uint32_t bar, uint32_t par, uint32_t ns) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(par), "r"(ns) : "memory");
    return ok != 0;
}
// Waits on where a first test failed, with a limit; the warp calls, and learns whether it may still ask for chunks.  Every warp waits
// for its own copies.  Where one does not come the row is lost, but the CTA goes on to its end, when another one gets its shared
// memory: the warp asks for no more, and what else it has under way, the stages from that one on in turn, is let land first (with a
// limit of its own; what was never asked for does not come either).
template <int N>
static __device__ __noinline__ bool ring_wait(uint32_t bar, uint32_t par) {
    WarpRing& r = scratch()->ring[warp_id()];
    if (*(volatile int*)&r.lost) return false;
    auto wait = [&](uint32_t b, uint32_t p, long long t0) {
        while (!__all_sync(0xffffffffu, ring_test(b, p, 20000u)))
            if (__any_sync(0xffffffffu, clock64() - t0 > WAIT_CYCLES)) return false;
        return true;
    };
    if (wait(bar, par, clock64())) return r.asks != 0;
    const bool asked = r.asks != 0;
    __syncwarp();
    if (lane_id() == 0) { r.asks = 0; r.lost = 1; scratch()->dead = 1; }
    if (asked) {
        const uint32_t first = smem_u32(smem) + OFF_BARS + warp_id() * (8 * N), s = (bar - first) / 8;
        const long long t0 = clock64();
        for (uint32_t j = 0; j < N; ++j) wait(first + 8 * ((s + j) % N), s + j >= N ? par ^ 1u : par, t0);
    }
    __syncwarp();
    return false;
}

// A warp's ring.  While a pass runs its state lives in registers, between passes in Sc.
template <int ELT>
struct Pipe {
    static constexpr int CHB = CHUNK * ELT;
    uint32_t buf, bar;                 // shared-memory addresses of the stages and of their barriers
    int cons, out;                     // chunks consumed, chunks under way
    bool asks;                         // the lane asks for chunks (no more once a wait ran out)

    __device__ __forceinline__ Pipe() {
        const int warp = warp_id();
        buf = smem_u32(smem) + warp * RING;
        bar = smem_u32(smem) + OFF_BARS + warp * (8 * NST);
        const WarpRing& r = scratch()->ring[warp];
        cons = r.cons; out = r.out; asks = r.asks != 0;
    }
    __device__ __forceinline__ uint32_t conv() const { return buf + NST * CHB; }          // bf16: an fp32 copy of one chunk
    __device__ __forceinline__ uint32_t stage(int j = 0) const { return buf + ((uint32_t)(cons + j) % NST) * CHB; }
    // Copies `bytes` to `dst`, counted on `bar`.  The warp calls, one lane acts (unless a wait of its own ran out).  None: the last
    // chunk of the buffer's last row may hold less than a unit of 16 bytes, which comes by ordinary loads (mend_edges).
    __device__ __forceinline__ void copy(uint32_t dst, const char* p, uint32_t bytes, uint32_t bar, u64 pol) const {
        asm volatile("{\n\t.reg .pred e, a;\n\tsetp.ne.u32 a, %5, 0;\n\telect.sync _|e, 0xffffffff;\n\tand.pred e, e, a;\n\t"
                     "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %2;\n\tsetp.ne.and.u32 e, %2, 0, e;\n\t"
                     "@e cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n\t}"
                     ::"r"(dst), "l"(p), "r"(bytes), "r"(bar), "l"(pol), "r"((uint32_t)asks) : "memory");
    }
    // skip: bytes at the start of the stage that are left out
    __device__ __forceinline__ void issue(const char* p, uint32_t bytes, u64 pol, uint32_t skip = 0) {
        const uint32_t s = (uint32_t)(cons + out) % NST;
        copy(buf + s * CHB + skip, p, bytes, bar + 8 * s, pol);
        ++out;
    }
    // The bytes of the chunk j places from the next one to consume are there.
    __device__ __forceinline__ void wait(int j = 0) { wait_at(bar + 8 * ((uint32_t)(cons + j) % NST), ((uint32_t)(cons + j) / NST) & 1u); }
    __device__ __forceinline__ void wait_at(uint32_t b, uint32_t par) {
        if (!__all_sync(0xffffffffu, ring_test(b, par, 20000u))) asks = ring_wait<NST>(b, par);
    }
    // Between passes: what was asked for ahead stays when it belongs to row `key`, else it is let land and dropped.
    __device__ __forceinline__ void expect(int key) {
        Sc* sc = scratch();
        if (out > 0 && sc->ring[warp_id()].key != key)
            while (out > 0) { wait(); ++cons; --out; }
    }
    __device__ __forceinline__ void save(int key) {
        __syncwarp();
        if (lane_id() == 0) { WarpRing& r = scratch()->ring[warp_id()]; r.cons = cons; r.out = out; r.key = key; }
        __syncwarp();
    }
};

// Bytes of the chunk at p that are copied of a row whose copies end at `end` (RowS; low words, as all of it: rows are short).
template <int ELT>
__device__ __forceinline__ uint32_t chunk_bytes(const char* p, uint32_t end) {
    const uint32_t left = (end & ~15u) - (uint32_t)reinterpret_cast<u64>(p);
    return left < (uint32_t)(CHUNK * ELT) ? left : (uint32_t)(CHUNK * ELT);
}
// Asks for the first chunks of row `key`, as far as they are not under way.  Every pass starts and ends with it: out of line where
// a thread has 80 registers and what it needs would be spilled (592 fp32 rows of 151,936 top_p 202 us inline, 194 us so, 200 without a
// filter 65 and 63), inline in the kernels of clusters (21 rows of 217,408, top_k 50: 25 us out of line, 24 us so).
template <int ELT>
__device__ __forceinline__ void ring_start_here(int key, const char* base, uint32_t end, int Nc, int gw, int GW, bool keep) {
    Pipe<ELT> p;
    p.expect(key);
    for (int c = gw + p.out * GW; p.out < NST && c < Nc; c += GW) {
        const char* q = base + (size_t)c * Pipe<ELT>::CHB;
        const uint32_t skip = c == 0 && (end & 1u) ? 16u : 0u, bytes = chunk_bytes<ELT>(q, end);
        p.issue(q + skip, bytes > skip ? bytes - skip : 0u, l2_policy(keep), skip);
    }
    p.save(key);
}
template <int ELT>
static __device__ __noinline__ void ring_start_call(int key, const char* base, uint32_t end, int Nc, int gw, int GW, bool keep) {
    ring_start_here<ELT>(key, base, end, Nc, gw, GW, keep);
}
template <bool CL, int ELT>
__device__ __forceinline__ void ring_start(int key, const char* base, uint32_t end, int Nc, int gw, int GW, bool keep) {
    if constexpr (CL) ring_start_here<ELT>(key, base, end, Nc, gw, GW, keep);
    else ring_start_call<ELT>(key, base, end, Nc, gw, GW, keep);
}

// The mask word of one lane for chunk c: words (512 c - a) / 32 + lane, lanes 0 .. 16.
__device__ __forceinline__ uint32_t mask_word(const int32_t* mrow, int W, int a, int c, int lane) {
    const int w = ((c * CHUNK - a) >> 5) + lane;
    return (lane <= 16 && w >= 0 && w < W) ? (uint32_t)__ldg(mrow + w) : 0u;
}

// A chunk as a pass reads it: group k (0 .. 3) of the lane's effective logits.
template <int ELT, bool MASK>
struct Chunk {
    uint32_t at;                       // the lane's first group: in the stage, or (bf16 chunks with penalties) in the fp32 copy
    bool wide;                         // fp32 values
    uint32_t mw; int sh;               // the lane's mask word, the bit of position 0
    int c;

    __device__ __forceinline__ float4 stored(int k) const {
        if (ELT == 4 || wide) return lds128(at + k * 512);
        uint32_t x, y;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(at + k * 256) : "memory");
        return make_float4(__uint_as_float(x << 16), __uint_as_float(x & 0xFFFF0000u), __uint_as_float(y << 16), __uint_as_float(y & 0xFFFF0000u));
    }
    // the mask bits of group k (bit 0 .. 3)
    __device__ __forceinline__ uint32_t bits4(int k) const {
        const int bit = sh + k * 128 + lane_id() * 4;
        const uint32_t w = __shfl_sync(0xffffffffu, mw, bit >> 5);
        if (sh & 3) return __funnelshift_r(w, __shfl_sync(0xffffffffu, mw, (bit >> 5) + 1), bit & 31);   // groups straddle words (an unaligned row)
        return w >> (bit & 31);
    }
    __device__ __forceinline__ float4 group(int k, float none) const {
        float4 v = stored(k);
        if (MASK) {
            const uint32_t bits = bits4(k);
            if (!(bits & 1u)) v.x = none;
            if (!(bits & 2u)) v.y = none;
            if (!(bits & 4u)) v.z = none;
            if (!(bits & 8u)) v.w = none;
        }
        return v;
    }
    // the lane's largest logit; bf16 chunks two at a time, masked ones as NaN, which a maximum passes over
    __device__ __forceinline__ float max16() const {
        float m = CI_NEG_INF;
        if (ELT == 2 && !wide) {
            uint32_t r = 0xFF80FF80u;                                    // two bf16 of -inf
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t x, y;
                asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(at + k * 256) : "memory");
                if (MASK) {
                    // the group's four bits spread to the top bits of four bytes (i to 7 + 8 i), those replicated to halves
                    const uint32_t top = (~bits4(k) & 0xFu) * 0x10204080u;
                    uint32_t h;
                    asm("prmt.b32 %0, %1, 0, 0x9988;" : "=r"(h) : "r"(top)); x |= h;
                    asm("prmt.b32 %0, %1, 0, 0xBBAA;" : "=r"(h) : "r"(top)); y |= h;
                }
                asm("max.bf16x2 %0, %0, %1;" : "+r"(r) : "r"(x));
                asm("max.bf16x2 %0, %0, %1;" : "+r"(r) : "r"(y));
            }
            return fmaxf(__uint_as_float(r << 16), __uint_as_float(r & 0xFFFF0000u));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) { const float4 v = group(k, CI_NEG_INF); m = fmax3(fmax3(v.x, v.y, v.z), v.w, m); }
        return m;
    }
    // logit e of the lane as stored (penalties; not the mask, which only removes)
    __device__ __forceinline__ float one(int e) const {
        if (ELT == 4 || wide) return lds32(at + (e >> 2) * 512 + (e & 3) * 4);
        unsigned short h;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(at + (e >> 2) * 256 + (e & 3) * 2) : "memory");
        return __uint_as_float((uint32_t)h << 16);
    }
};

// The chunk at stage `st`, its edges mended; the penalties of a row with them: fp32 chunks in place, once (fresh), bf16 ones
// through an fp32 copy at `conv`.
template <int ELT, bool MASK>
__device__ __forceinline__ Chunk<ELT, MASK> open_chunk(const RowS& rw, uint32_t st, int c, uint32_t mw) {
    Chunk<ELT, MASK> k;
    k.c = c; k.mw = mw; k.sh = MASK ? (-rw.a) & 31 : 0; k.wide = ELT == 4;
    k.at = st + lane_id() * 4 * ELT;
    return k;
}
template <int ELT, bool MASK>
__device__ __forceinline__ void penalise(RowS& rw, Chunk<ELT, MASK>& k, uint32_t st, uint32_t conv, bool fresh, const PenPeek& pk, const PenVals& v) {
    if (ELT == 4) { if (fresh) pen_patch(rw, st, k.c, pk, v); }
    else {
        const int lane = lane_id();
#pragma unroll
        for (int j = 0; j < 4; ++j) sts128(conv + lane * 16 + j * 512, k.stored(j));
        __syncwarp();
        pen_patch(rw, conv, k.c, pk, v);
        k.at = conv + lane * 16; k.wide = true;
    }
}

// What the ring asks for when a pass has asked for all of its own chunks.
enum { THEN_NOTHING = 0, THEN_AGAIN = 1, THEN_NEXT_ROW = 2 };

// One pass of the calling warp over its chunks of the row at hand: f(chunk) on every one.  keep: the row's L2 policy; seen: how
// many of its first chunks have been read before (and lie in the ring as they were left).
// A chunk is refilled where it lay: as long as there is more to ask for the ring is full, so the chunk asked for next belongs in the
// stage just read.  The state of the ring is three registers, edges are one comparison, the copy is issued by an elected lane (known
// to be one, its operands need no loop over lanes).
template <bool CL, int ELT, bool MASK, class F>
__device__ __forceinline__ void run_pass(RowS& rw, const NextRow& nx, bool keep, int seen, int then, F f) {
    constexpr int CHB = CHUNK * ELT;
    Sc* sc = scratch();
    const int GW = CL ? sc->GW : NW;
    const int gw = (CL ? sc->rank * NW : 0) + warp_id();
    const int Nc = rw.Nc;
    const bool pen_on = rw.pen_on != 0;
    ring_start<CL, ELT>(rw.key, rw.base, rw.end, Nc, gw, GW, keep);
    Pipe<ELT> p;
    const u64 pol = l2_policy(keep);
    const int n = gw < Nc ? (Nc - 1 - gw) / GW + 1 : 0;                  // chunks of the warp
    const char* next = rw.base + (size_t)(gw + NST * GW) * CHB;          // the next chunk to ask for, and how many there are
    int ask = max(n - NST, 0);
    const int last = (Nc - 1) % GW == gw ? (int)chunk_bytes<ELT>(rw.base + (size_t)(Nc - 1) * CHB, rw.end) : CHB;   // bytes of the warp's last chunk
    int edge = gw == 0 && rw.a ? 0 : Nc - 1;                             // the next chunk whose edges want mending
    uint32_t mw[MASK ? 3 : 1];                                           // mask words of this chunk and the next two
    if (MASK) {
#pragma unroll
        for (int j = 0; j < 3; ++j) mw[MASK ? j : 0] = gw + j * GW < Nc ? mask_word(rw.mrow, sc->W, rw.a, gw + j * GW, lane_id()) : 0u;
    }
    PenPeek pk = {0, 0, 0};
    if (pen_on && gw < Nc) pk = pen_peek(pen_tab(sc), rw.pen_cap, gw, lane_id());
    uint32_t s = (uint32_t)p.cons % NST, par = ((uint32_t)p.cons / NST) & 1u;
    int c = gw;
    auto loop = [&](auto pen) {
        constexpr bool PEN = decltype(pen)::value;
        const PenTab pt = pen_tab(sc);
        const PenVals pv = PEN ? pen_vals(rw) : PenVals{};
        uint32_t after0 = 0, after1 = 0;                                     // of the chunk after the next one
        if (PEN && n > 1) { after0 = pt.pre[c + GW]; after1 = pt.pre[c + GW + 1]; }
#pragma unroll 1
        for (int left = n; left; --left) {
            const uint32_t st = p.buf + s * CHB, bar = p.bar + 8 * s;
            const bool fresh = seen <= 0;
            bool wrote = !fresh;                                             // the stage was changed by ordinary stores
            if (fresh) {
                p.wait_at(bar, par);
                if (c == edge) { mend_edges<ELT>(rw, st, c); wrote = true; }
            }
            if (c == edge) edge = Nc - 1;
            --seen;
            auto k = open_chunk<ELT, MASK>(rw, st, c, mw[0]);
            if (PEN) {
                const PenPeek cur = pk;
                pk.r0 = after0; pk.r1 = after1;                          // (loads of which nothing waits in this turn)
                pk.ent = left > 1 && after0 + lane_id() < min(after1, (uint32_t)pv.cap) ? pt.ent[after0 + lane_id()] : 0u;
                if (left > 2) { after0 = pt.pre[c + 2 * GW]; after1 = pt.pre[c + 2 * GW + 1]; }
                if (cur.r0 != cur.r1) { penalise(rw, k, st, p.conv(), fresh, cur, pv); wrote = true; }
            }
            f(k);
            if (MASK) {
                mw[0] = mw[MASK ? 1 : 0]; mw[MASK ? 1 : 0] = mw[MASK ? 2 : 0];
                if (c + 3 * GW < Nc) mw[MASK ? 2 : 0] = mask_word(rw.mrow, sc->W, rw.a, c + 3 * GW, lane_id());
            }
            // gives the stage back (what the warp changed in it with ordinary stores comes before the next copy) and asks for more
            if (wrote) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (ask) {
                p.copy(st, next, --ask ? CHB : last, bar, pol);
                next += (size_t)GW * CHB;
            }
            c += GW;
            if (++s == NST) { s = 0; par ^= 1u; }
        }
    };
    if (pen_on) loop(BoolTag<true>{}); else loop(BoolTag<false>{});
    p.cons += n; p.out = 0;
    p.save(rw.key);
    // the first chunks of what comes next
    const int nkey = *(volatile const int*)&nx.key;
    __threadfence_block();
    if (then == THEN_AGAIN) ring_start<CL, ELT>(rw.key, rw.base, rw.end, Nc, gw, GW, false);
    else if (then == THEN_NEXT_ROW && nkey) ring_start<CL, ELT>(nkey, nx.base, nx.end, nx.Nc, gw, GW, true);
}

// Appends the logits of the chunk selected by the lanes' masks mk to the warp's list (no particular order).
template <class C>
__device__ __forceinline__ void list_append(int a, Cand* list, int cap, unsigned mk, const C& k) {
    if (mk) {
        Sc* sc = scratch();
        int at = atomicAdd(&sc->wn[warp_id()], __popc(mk));
        const int t0 = k.c * CHUNK - a;
        do {
            const int e = __ffs(mk) - 1;
            mk &= mk - 1;
            if (at < cap) { list[at].idx = (uint32_t)(t0 + pos_of(e, lane_id())); list[at].l = k.one(e); }
            ++at;
        } while (mk);
    }
}
// The same for the logits >= t (looked for again: few lanes have any).
template <class C>
__device__ __forceinline__ void list_above(int a, Cand* list, int cap, float t, bool any, const C& k) {
    if (__any_sync(0xffffffffu, any)) {
        unsigned mk = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = k.group(j, CI_NEG_INF);
            mk |= ((v.x >= t ? 1u : 0u) | (v.y >= t ? 2u : 0u) | (v.z >= t ? 4u : 0u) | (v.w >= t ? 8u : 0u)) << (4 * j);
        }
        list_append(a, list, cap, mk, k);
    }
}
__device__ __forceinline__ float max4(float4 v, float m) { return fmax3(fmax3(v.x, v.y, v.z), v.w, m); }

// The passes.
struct Top { float l; int idx; };

// Maximum of the warp's chunks and the lowest token that has it (the same in all lanes).
__device__ __forceinline__ float warp_max(float x) {
    float m;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(x));
    return m;
}
template <bool CL, int ELT, bool MASK>
__device__ __forceinline__ Top pass_max(RowS& rw, const NextRow& nx, bool keep, int then) {
    float wmax = CI_NEG_INF;
    int widx = 0x7fffffff;
    run_pass<CL, ELT, MASK>(rw, nx, keep, 0, then, [&](const auto& k) {
        const float m = k.max16(), top = warp_max(m);
        if (top > wmax) {                                                // strict: the first (lowest) position of the maximum stays
            wmax = top;
            unsigned p = 0x7fffffff;
#pragma unroll 1
            for (int j = 3; j >= 0; --j) {
                const float4 v = k.group(j, CI_NEG_INF);
                const int e = v.x == top ? 0 : v.y == top ? 1 : v.z == top ? 2 : v.w == top ? 3 : 4;
                if (e < 4) p = min(p, (unsigned)(4 * j + e));
            }
            widx = (int)__reduce_min_sync(0xffffffffu, p == 0x7fffffffu ? p : (unsigned)(k.c * CHUNK - rw.a + pos_of(p, lane_id())));
        }
    });
    return Top{wmax, widx};
}

// Lists the logits >= t of the warp's chunks; returns the lane's maximum.
template <bool CL, int ELT, bool MASK>
__device__ __forceinline__ float pass_list(RowS& rw, const NextRow& nx, bool keep, int seen, int then, float t, Cand* list, int cap) {
    float lmax = CI_NEG_INF;
    run_pass<CL, ELT, MASK>(rw, nx, keep, seen, then, [&](const auto& k) {
        const float m = k.max16();
        lmax = fmaxf(lmax, m);
        list_above(rw.a, list, cap, t, m >= t, k);
    });
    return lmax;
}

// Histogram bucket of a logit: floor((href - x) * scale) + hoff clamped to [0, NB1).  The clamp is a saturating
// multiply-add, the conversion a rounding addition (neither the ALU nor the conversion pipe is asked).  A logit exactly on an
// edge may land in either neighbour; every user keeps a whole bucket of margin.
struct Buckets {
    float href, s, c;                  // saturate((href - x) * s + c) in units of NB1 - 1 buckets
    __device__ __forceinline__ Buckets(float h, float scale, int hoff) : href(h), s(scale / (float)(NB1 - 1)), c(((float)hoff - 0.5f) / (float)(NB1 - 1)) {}
    __device__ __forceinline__ float sat(float d) const { float r; asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(d), "f"(s), "f"(c)); return r; }
    __device__ __forceinline__ int operator()(float x) const {
        return __float_as_int(fmaf(sat(href - x), (float)(NB1 - 1), 8388608.0f)) - 0x4B000000;
    }
};

// The same with a count of the buckets of the logits >= from (what lies below, and -inf, cannot be kept).  FULL: of all of them.
// Else of a quarter of those that are not listed, one group of every lane and chunk, each counting four (the listed ones are added
// when the pass is over), and with the mass of all logits relative to href (fp32, in `mass`): with that known, the quarter only has
// to say how much mass lies below a logit, to which the largest logits, whose share a sample would miss, do not belong.  What is
// left to the sample moves the estimated top-p pivot by about 200 places of 30,000 (standard deviation; N(0, 2^2), T = 0.5 - 1.2), a
// fifth of what the band around it reaches to either side.
// Counting all of a row takes 10 instructions per logit and a shared-memory addition per logit, the mass 2.
constexpr uint32_t SAMPLED = 4;
template <bool CL, int ELT, bool MASK, bool FULL, bool SUM>
__device__ __forceinline__ float pass_hist(RowS& rw, const NextRow& nx, bool keep, int seen, int then, float t, Cand* list, int cap, float href, float scale, int hoff, float from, float tc, float& mass) {
    float lmax = CI_NEG_INF;
    const float yc = CI_LOG2E / tc;
    const u64 yk = pk2(yc, yc), y0 = pk2(-href * yc, -href * yc);
    u64 sum = 0;
    const Buckets bk(href, scale, hoff);
    const uint32_t h0 = smem_u32(smem) + OFF_U - (0x4B000000u << 2);
    const u64 hr = pk2(href, href), k4 = pk2((float)(NB1 - 1), (float)(NB1 - 1)), mg = pk2(8388608.0f, 8388608.0f), neg = pk2(-1.0f, -1.0f);
    run_pass<CL, ELT, MASK>(rw, nx, keep, seen, then, [&](const auto& k) {
        auto count = [&](float x, float b) {
            const uint32_t at = h0 + (__float_as_uint(b) << 2);
            if (FULL) asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %1, %2;\n\t@p red.shared.add.u32 [%0], 1;\n\t}" ::"r"(at), "f"(x), "f"(from) : "memory");
            else asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %1, %2;\n\tsetp.lt.and.f32 p, %1, %3, p;\n\t@p red.shared.add.u32 [%0], %4;\n\t}" ::"r"(at), "f"(x), "f"(from), "f"(t), "n"(SAMPLED) : "memory");
        };
        auto count4 = [&](const float4 v) {
            float d0, d1, d2, d3, b0, b1, b2, b3;
            up2(fma2(pk2(v.x, v.y), neg, hr), d0, d1);
            up2(fma2(pk2(v.z, v.w), neg, hr), d2, d3);
            up2(fma2(pk2(bk.sat(d0), bk.sat(d1)), k4, mg), b0, b1);
            up2(fma2(pk2(bk.sat(d2), bk.sat(d3)), k4, mg), b2, b3);
            count(v.x, b0); count(v.y, b1); count(v.z, b2); count(v.w, b3);
        };
        float m = CI_NEG_INF;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = k.group(j, CI_NEG_INF);
            m = max4(v, m);
            if (FULL) count4(v);
            if (SUM) {
                float a0, a1, a2, a3;
                up2(fma2(pk2(v.x, v.y), yk, y0), a0, a1);
                up2(fma2(pk2(v.z, v.w), yk, y0), a2, a3);
                asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a0)); asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a1));
                asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a2)); asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a3));
                sum = add2(sum, add2(pk2(a0, a1), pk2(a2, a3)));
            }
        }
        if (!FULL) count4(k.group(k.c & 3, CI_NEG_INF));
        lmax = fmaxf(lmax, m);
        list_above(rw.a, list, cap, t, m >= t, k);
    });
    float s0, s1;
    up2(sum, s0, s1);
    mass = s0 + s1;
    return lmax;
}

// The mass pass: per chunk the mass of the logits >= lk (BAND: of those above t_hi) into csum, and, BAND, the logits of
// [tl, t_hi] into the warp's list and the mass of all logits >= lk.  MINP: lk may lie above the mass horizon.
// The masses come in two parts (Mass2): multiples of 2^-15, and the rest at 12582912, whose bits are summed as integers.  What bounds
// it is issue and the pipes about alike: two logits take 10 packed instructions of two cycles, two exponentials of eight, and, BAND,
// 12 compares, selects and additions.
struct Masses { u64 all, keep; };
// Above t_hi: the two parts of a mass to their sums; from tl on: the logit's bit to the mask.  Five instructions without a branch.
__device__ __forceinline__ void band_add(float x, float t_hi, float tl, float hi, uint32_t lo, uint32_t bit, float& sh, uint32_t& sl, uint32_t& mk) {
    asm("{\n\t.reg .pred p, q;\n\tsetp.gt.f32 p, %3, %4;\n\tsetp.ge.and.f32 q, %3, %5, !p;\n\t"
        "@p add.f32 %0, %0, %6;\n\t@p add.u32 %1, %1, %7;\n\t@q or.b32 %2, %2, %8;\n\t}"
        : "+f"(sh), "+r"(sl), "+r"(mk) : "f"(x), "f"(t_hi), "f"(tl), "f"(hi), "r"(lo), "r"(bit));
}
template <bool CL, int ELT, bool MASK, bool BAND, bool MINP>
__device__ __forceinline__ Masses pass_mass(RowS& rw, const NextRow& nx, int then, MassFn mass, float lk, float t_hi, float tl, Cand* list, u64* csum) {
    Mass2 m2;
    m2.init(mass);
    u64 keep = 0;
    int all_h = 0, all_l = 0;
    run_pass<CL, ELT, MASK>(rw, nx, false, 0, then, [&](const auto& k) {
        bool mend = MINP;
        u64 sh;                                                          // sums of the chunk: exact (multiples of 2^-15 up to 16, integers up to 2^18)
        uint32_t sl, al;
        float ah, s0, s1;
        unsigned mk;
        while (true) {
            sh = 0; sl = al = 0; ah = 0.0f; mk = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float4 v = k.group(j, SM_LOW);
                if (mend) {                                              // logits without mass
                    v.x = v.x >= lk ? v.x : SM_LOW; v.y = v.y >= lk ? v.y : SM_LOW;
                    v.z = v.z >= lk ? v.z : SM_LOW; v.w = v.w >= lk ? v.w : SM_LOW;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float x0 = h ? v.z : v.x, x1 = h ? v.w : v.y;
                    u64 hi, w;
                    m2.parts(x0, x1, hi, w);
                    const uint32_t w0 = (uint32_t)w, w1 = (uint32_t)(w >> 32);
                    sh = add2(sh, hi);
                    sl += w0 + w1;
                    if (BAND) {
                        float h0, h1;
                        up2(hi, h0, h1);
                        band_add(x0, t_hi, tl, h0, w0, 1u << (4 * j + 2 * h), ah, al, mk);
                        band_add(x1, t_hi, tl, h1, w1, 2u << (4 * j + 2 * h), ah, al, mk);
                    }
                }
            }
            up2(sh, s0, s1);
            if (MINP || mend || !__any_sync(0xffffffffu, !(s0 + s1 < 1e9f))) break;
            mend = true;                                                 // a logit of -inf: once more
        }
        // (12582912's bits are a multiple of 2^22: below that stands the sum of the rests)
        static_assert((0x4B400000u & 0x3FFFFFu) == 0, "the bits of 12582912");
        const int ch = __float2int_rn((s0 + s1) * 32768.0f), cl = (int)(sl << 10) >> 10;
        if (BAND) { all_h += ch; all_l += cl; }
        const uint32_t wh = __reduce_add_sync(0xffffffffu, (unsigned)(BAND ? __float2int_rn(ah * 32768.0f) : ch));
        const int wl = (int)__reduce_add_sync(0xffffffffu, (unsigned)(BAND ? (int)(al << 10) >> 10 : cl));
        const u64 q = ((u64)wh << 15) + (u64)(long long)wl;
        if (lane_id() == 0) csum[k.c] = q;
        keep += q;
        if (BAND) list_append(rw.a, list, CL ? WCAP_CL : KCAP, mk, k);
    });
    Masses r;
    r.keep = keep;
    r.all = BAND ? ((u64)__reduce_add_sync(0xffffffffu, (unsigned)all_h) << 15) + (u64)(long long)(int)__reduce_add_sync(0xffffffffu, (unsigned)all_l) : keep;
    return r;
}

// One level of the exact radix select over the order-preserving keys of the logits >= lk: the bins of the keys that begin with
// `prefix`, by count or by mass.
template <bool CL, int ELT, bool MASK>
static __device__ __noinline__ void pass_radix(RowS& rw, const NextRow& nx, MassFn mass, float lk, int lvl, uint32_t prefix, bool by_mass, u64* bins) {
    const int lane = lane_id(), shift = 24 - 8 * lvl;
    run_pass<CL, ELT, MASK>(rw, nx, false, 0, THEN_NOTHING, [&](const auto& k) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            const float4 v = k.group(j, CI_NEG_INF);
#pragma unroll 1
            for (int e = 0; e < 4; ++e) {
                const float l = e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w;
                int bin = -1;
                if (l >= lk) {
                    const uint32_t f = f2key(l);
                    if (lvl == 0 || (f >> (shift + 8)) == prefix) bin = FB_NB - 1 - (int)((f >> shift) & 0xFFu);
                }
                // lanes of one bin add once (most keys of a level share a few bins: plain atomics would serialise)
                const unsigned peers = __match_any_sync(0xffffffffu, bin);
                const uint32_t w = bin < 0 ? 0u : (by_mass ? mass(l) : 1u);
                const uint32_t lo = __reduce_add_sync(peers, w & 0xFFFFu), hi = __reduce_add_sync(peers, w >> 16);
                if (bin >= 0 && lane == __ffs(peers) - 1) add64(&bins[bin], ((u64)hi << 16) + lo);
            }
        }
    });
}

// Exact masses of the buckets [w0, w0 + BINS), and the warp's mass above them.
template <bool CL, int ELT, bool MASK>
static __device__ __noinline__ u64 pass_window(RowS& rw, const NextRow& nx, MassFn mass, float lk, float href, float scale, int hoff, int w0, u64* bins) {
    u64 hi = 0;
    const Buckets bk(href, scale, hoff);
    run_pass<CL, ELT, MASK>(rw, nx, false, 0, THEN_NOTHING, [&](const auto& k) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            const float4 v = k.group(j, CI_NEG_INF);
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (x[e] >= lk) {
                    const int bb = bk(x[e]);
                    if (bb < w0) hi += (u64)mass(x[e]);
                    else if (bb < w0 + BINS) add64(&bins[bb - w0], (u64)mass(x[e]));
                }
            }
        }
    });
    return warp_sum_u64(hi);
}

// Exact masses of the keys [klo, khi], 2^sh of them a bin, from the largest down.
template <bool CL, int ELT, bool MASK>
static __device__ __noinline__ void pass_bracket(RowS& rw, const NextRow& nx, MassFn mass, uint32_t klo, uint32_t khi, int sh, u64* bins) {
    run_pass<CL, ELT, MASK>(rw, nx, false, 0, THEN_NOTHING, [&](const auto& k) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            const float4 v = k.group(j, CI_NEG_INF);
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t f = f2key(x[e]);
                if (f >= klo && f <= khi) add64(&bins[(khi - f) >> sh], (u64)mass(x[e]));
            }
        }
    });
}

// The rarer uses of the passes, as functions of their own.
// The lowest token of the warp's chunks whose logit is L.
template <bool CL, int ELT, bool MASK>
static __device__ __noinline__ int argmax_pass(RowS& rw, const NextRow& nx, float L) {
    const Top m = pass_max<CL, ELT, MASK>(rw, nx, false, THEN_NOTHING);
    return m.l == L ? m.idx : 0x7fffffff;
}
// The histogram counted from the row's maximum.
template <bool CL, int ELT, bool MASK>
static __device__ __noinline__ void recount_pass(RowS& rw, const NextRow& nx) {
    float est;
    pass_hist<CL, ELT, MASK, true, true>(rw, nx, true, 0, THEN_AGAIN, SM_POS_INF, nullptr, 0, rw.L, rw.scw, 0, rw.lcut, rw.tc, est);
#pragma unroll
    for (int o = 16; o; o >>= 1) est += __shfl_xor_sync(0xffffffffu, est, o);
    if (lane_id() == 0) scratch()->est[warp_id()] = est;
}
// The logits a large top-k can keep.
template <bool CL, int ELT, bool MASK>
static __device__ __noinline__ void relist_pass(RowS& rw, const NextRow& nx, Cand* list, int cap) {
    pass_list<CL, ELT, MASK>(rw, nx, false, 0, THEN_NEXT_ROW, fmaxf(fmaxf(rw.t_lo, rw.lcut), -SM_FLT_MAX), list, cap);
}

// A warp's share of a set of listed logits: entries start, start + step, ... below n.
struct View { const Cand* p; int start, n, step; };

// Selects the listed logits that can belong to the top kk: BINS linear bins over [max(bound, cut), L] give the bin of the
// kk-th largest, everything down to it goes to the CTA's candidates (at most FCAP, no particular order).  Returns how many,
// or -1 when the lists cannot decide.  Every logit >= bound of the row is in the lists.  bins and nsel are zeroed before the caller's last barrier.
// Two __syncthreads.
__device__ __forceinline__ int select_top(const View& w, float bound, float cut, float L, int kk, uint32_t* bins, Sc* sc, float& scale, int& bstar) {
    const int lane = lane_id();
    const float lo = fmaxf(bound, cut);
    scale = L > lo ? (float)(BINS - 2) / (L - lo) : 0.0f;
    auto bin_of = [&](float l) { return max(0, min(BINS - 1, __float2int_rz((L - l) * scale))); };
    for (int j = w.start; j < w.n; j += w.step) { const float l = w.p[j].l; if (l >= lo) atomicAdd(&bins[(bin_of(l))], 1u); }
    __syncthreads();
    uint32_t run_b;
    bstar = warp_count_bin(bins, (uint32_t)kk, run_b);         // every warp scans the bins itself
    int n = (int)run_b;
    if (bstar < 0) {
        // fewer than kk listed logits reach lo: if lo is the cut, fewer than kk logits survive it and top-k removes nothing
        if (!(lo > bound)) n = -1;
        bstar = BINS - 1;
    }
    if (n > FCAP || !(lo <= L)) n = -1;
    if (n > 0) {
        for (int j = w.start; j < w.n; j += w.step) {
            const Cand c = w.p[j];
            if (c.l >= lo && bin_of(c.l) <= bstar) { const int at = atomicAdd(&sc->nsel, 1); if (at < FCAP) { fin_area()->fc_idx[at] = c.idx; fin_area()->fc_l[at] = c.l; } }
        }
    }
    __syncthreads();
    return n;
}

// Candidates in order: every one's rank by descending logit (equal logits: as selected) and by token, a few threads per
// candidate, and its mass.
static __device__ __noinline__ void order_candidates(int nc, const MassFn mass) {
    Sc* sc = scratch();
    constexpr int TPC = NT >= 1024 ? 8 : NT >= 512 ? 4 : 2;          // threads per candidate
    static_assert(TPC * FCAP <= NT, "a few threads per candidate");
    const int i = threadIdx.x / TPC, part = threadIdx.x % TPC;         // (none of i >= FCAP)
    if (threadIdx.x < FCAP) {
        const int t = threadIdx.x;
        if (t >= nc) { fin_area()->fc_idx[t] = 0xFFFFFFu; fin_area()->fc_l[t] = CI_NEG_INF; fin_area()->sv_l[t] = CI_NEG_INF; fin_area()->sv_q[t] = 0; fin_area()->so_l[t] = CI_NEG_INF; fin_area()->so_q[t] = 0; }
        fin_area()->ties[t] = 0;
    }
    __syncthreads();
    // (tokens: their difference saturated to 1; equal logits share a rank and are told apart by arrival)
    const float my_l = i < FCAP ? fin_area()->fc_l[i] : CI_NEG_INF, my_i = i < FCAP ? (float)fin_area()->fc_idx[i] : 0.0f;
    int rv = 0; float rif = 0.0f;
    auto sat = [](float d) { float r; asm("add.rn.sat.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(d)); return r; };
    for (int j = part * 4; j < nc; j += 4 * TPC) {
        const float4 l = *reinterpret_cast<const float4*>(&fin_area()->fc_l[j]);
        const uint4 d = *reinterpret_cast<const uint4*>(&fin_area()->fc_idx[j]);
        rv += (l.x > my_l) + (l.y > my_l) + (l.z > my_l) + (l.w > my_l);
        rif += sat(my_i - (float)d.x) + sat(my_i - (float)d.y); rif += sat(my_i - (float)d.z) + sat(my_i - (float)d.w);
    }
#pragma unroll
    for (int o = 1; o < TPC; o <<= 1) { rv += __shfl_xor_sync(0xffffffffu, rv, o); rif += __shfl_xor_sync(0xffffffffu, rif, o); }
    const int ri = (int)rif;
    const uint32_t q = my_l > CI_NEG_INF ? mass(my_l) : 0u;
    if (i < nc) {
        if (part == 0) { rv += atomicAdd(&fin_area()->ties[rv], 1); fin_area()->sv_l[rv] = my_l; fin_area()->sv_q[rv] = q; }
        else if (part == 1) { fin_area()->so_idx[ri] = fin_area()->fc_idx[i]; fin_area()->so_l[ri] = my_l; fin_area()->so_q[ri] = q; }
    }
    __syncthreads();
}

// Top-k, top-p and the draw on the ordered candidates (every logit of the row >= lo in the bins down to bstar), by one
// warp.  Writes ok, fin_*.
static __device__ __noinline__ void finish_warp(float lo, float L, float scale, int bstar, float lcut_in, float tc, int kk, float topp, float u) {
    Sc* sc = scratch();
    const int lane = lane_id();
    constexpr int PERC = FCAP / 32;
    static_assert(PERC == 4, "128-bit loads");
    const float4 l4 = *reinterpret_cast<const float4*>(&fin_area()->sv_l[lane * 4]);
    const uint4 q4 = *reinterpret_cast<const uint4*>(&fin_area()->sv_q[lane * 4]);
    const float l[4] = {l4.x, l4.y, l4.z, l4.w}; const uint32_t q[4] = {q4.x, q4.y, q4.z, q4.w};
    int surv = 0;
#pragma unroll
    for (int t = 0; t < PERC; ++t) surv += l[t] >= lcut_in && l[t] > CI_NEG_INF ? 1 : 0;
    surv = (int)__reduce_add_sync(0xffffffffu, (unsigned)surv);
    float cut = lcut_in;
    bool ok = surv > 0;
    if (ok && kk <= surv) {                                          // else fewer than k survive min-p: top-k removes nothing
        const float lk = fin_area()->sv_l[kk - 1];
        const float ck = lower_logit_for(scale_logit(lk, tc), tc, lk);
        ok = ck >= lo && __float2int_rz((L - ck) * scale) <= bstar;  // else a tie partner could lie outside the candidates
        cut = fmaxf(cut, ck);
    }
    if (ok && topp < 1.0f) {
        u64 s = 0;
#pragma unroll
        for (int t = 0; t < PERC; ++t) s += l[t] >= cut ? (u64)q[t] : 0ull;
        const u64 incl = warp_incl_scan_u64(s, lane);
        const u64 s1 = __shfl_sync(0xffffffffu, incl, 31);
        ok = s1 > 0;
        const u64 target = ceil_target(topp, s1);
        const unsigned hit = __ballot_sync(0xffffffffu, incl >= target);
        const int hl = hit ? __ffs(hit) - 1 : 0;
        u64 run = incl - s; int tt = 0;
#pragma unroll
        for (int t = PERC - 1; t >= 0; --t) {                        // the first t whose running mass reaches the target
            u64 r = run;
#pragma unroll
            for (int k = 0; k <= t; ++k) r += l[k] >= cut ? (u64)q[k] : 0ull;
            if (r >= target) tt = t;
        }
        const float lp = fin_area()->sv_l[hl * PERC + __shfl_sync(0xffffffffu, tt, hl)];
        if (ok) cut = fmaxf(cut, lower_logit_for(scale_logit(lp, tc), tc, lp));
    }
    const float4 ol4 = *reinterpret_cast<const float4*>(&fin_area()->so_l[lane * 4]);
    const uint4 oq4 = *reinterpret_cast<const uint4*>(&fin_area()->so_q[lane * 4]);
    const uint32_t o[4] = {ol4.x >= cut ? oq4.x : 0u, ol4.y >= cut ? oq4.y : 0u, ol4.z >= cut ? oq4.z : 0u, ol4.w >= cut ? oq4.w : 0u};
    const u64 s = ((u64)o[0] + o[1]) + ((u64)o[2] + o[3]);
    const u64 incl = warp_incl_scan_u64(s, lane);
    const u64 tot = __shfl_sync(0xffffffffu, incl, 31);
    ok = ok && tot > 0;
    const u64 target = ceil_target(u, tot);
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= target);
    if (lane == 0) sc->ok = 0;
    __syncwarp();
    if (ok && lane == __ffs(hit) - 1) {
        u64 run = incl - s; int e = PERC - 1;
        for (int t = 0; t < PERC - 1; ++t) { run += o[t]; if (run >= target) { e = t; break; } }
        sc->fin_token = (int)fin_area()->so_idx[lane * PERC + e]; sc->fin_cut = cut; sc->fin_total = tot; sc->ok = 1;
    }
}

// Exact weighted selection among the listed logits >= c0 of the warps' views, each weighing 1 or its mass: the value v with
// W(l > v) < target <= W(l >= v).  BINS linear bins over (base - l) * scale, then the pivot bin's entries pairwise; every warp does
// the searches itself, so that they cost no barriers.  False when the pivot leaves the binned range or its bin is too crowded.
// total: the weight of all entries.  All threads call with the same arguments; a barrier lies between two calls.
static __device__ __noinline__ bool list_select(const View w, bool by_mass, const MassFn mass, float c0, float base, float scale, u64 target, float& value, u64& total) {
    Sc* sc = scratch();
    const int tid = threadIdx.x, lane = lane_id();
    uint32_t* lo = reinterpret_cast<uint32_t*>(smem + OFF_BINS);         // a bin's weight: low and high 16 bits of the entries' summed apart
    uint32_t* hi = lo + BINS;
    // (again, within a bin of several values and more entries than are compared pairwise: a penalised logit beside many equal ones)
    float top = SM_POS_INF;
#pragma unroll 1
    for (int level = 0; level < 3; ++level) {
    for (int i = tid; i < 2 * BINS; i += NT) lo[i] = 0;
    if (tid == 0) { sc->ncand = 0; sc->cand_kmin = 0xFFFFFFFFu; sc->cand_kmax = 0u; }
    __syncthreads();
    auto bin_of = [&](float l) { return max(0, min(BINS - 1, __float2int_rz((base - l) * scale))); };
    auto weight = [&](float l) { return l >= c0 && l <= top ? by_mass ? mass(l) : 1u : 0u; };
#pragma unroll 2
    for (int i = w.start; i < w.n; i += w.step) {
        const float l = w.p[i].l;
        const uint32_t q = weight(l);
        if (q) { const int b = bin_of(l); atomicAdd(&lo[b], q & 0xFFFFu); if (q >> 16) atomicAdd(&hi[b], q >> 16); }
    }
    __syncthreads();
    static_assert(BINS == 256, "eight bins per lane");
    u64 s = 0;
    {
        const uint4 a = reinterpret_cast<const uint4*>(lo)[2 * lane], b = reinterpret_cast<const uint4*>(lo)[2 * lane + 1];
        const uint4 c = reinterpret_cast<const uint4*>(hi)[2 * lane], d = reinterpret_cast<const uint4*>(hi)[2 * lane + 1];
        s = ((u64)a.x + a.y) + ((u64)a.z + a.w) + ((u64)b.x + b.y) + ((u64)b.z + b.w) + ((((u64)c.x + c.y) + ((u64)c.z + c.w) + ((u64)d.x + d.y) + ((u64)d.z + d.w)) << 16);
    }
    const u64 incl = warp_incl_scan_u64(s, lane);
    if (level == 0) total = __shfl_sync(0xffffffffu, incl, 31);
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= target);
    if (!hit || target == 0) return false;
    const int hl = __ffs(hit) - 1, bl = 8 * hl + (lane & 7);
    const u64 one = ((u64)hi[bl] << 16) + lo[bl];                        // (lanes 0 .. 7: the bins of that lane)
    u64 run = one;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) { const u64 t = __shfl_up_sync(0xffffffffu, run, o); if ((lane & 7) >= o) run += t; }
    run += __shfl_sync(0xffffffffu, incl - s, hl);
    const int first = __ffs(__ballot_sync(0xffffffffu, run >= target)) - 1;
    const int b_star = 8 * hl + first;
    const u64 before = __shfl_sync(0xffffffffu, run - one, first);
    if (b_star >= BINS - 1) return false;
    for (int i = w.start; i < w.n; i += w.step) {
        const float l = w.p[i].l;
        if (bin_of(l) != b_star) continue;
        const uint32_t q = weight(l);
        if (!q) continue;
        const int slot = atomicAdd(&sc->ncand, 1);
        if (slot < FIN_CAND) { sc->cand_l[slot] = l; sc->cand_w[slot] = q; }
        else { const uint32_t k = f2key(l); atomicMin(&sc->cand_kmin, k); atomicMax(&sc->cand_kmax, k); }
    }
    __syncthreads();
    const int nc = sc->ncand;
    if (nc > FIN_CAND) {
        // A crowded pivot bin.  When all of its entries are one value (bf16 logits: a hundred tokens share every value)
        // that value is the pivot: the weight above the bin is below the target, with the bin it reaches it.
        uint32_t kmin = sc->cand_kmin, kmax = sc->cand_kmax;
        for (int i = 0; i < FIN_CAND; ++i) { const uint32_t k = f2key(sc->cand_l[i]); kmin = min(kmin, k); kmax = max(kmax, k); }
        value = key2f(kmin);
        if (kmin == kmax) return true;
        c0 = value; top = base = key2f(kmax);
        scale = (float)(BINS - 2) / (top - c0);
        target -= before;
        __syncthreads();                                             // (the candidates have been read)
        continue;
    }
    float mine = 0.0f;
    bool found = false;
#pragma unroll 1
    for (int j = lane; j < nc && !found; j += 32) {
        mine = sc->cand_l[j];
        u64 gt = 0, eq = 0;
        for (int i = 0; i < nc; ++i) {
            const float o = sc->cand_l[i];
            if (o > mine) gt += sc->cand_w[i]; else if (o == mine) eq += sc->cand_w[i];
        }
        found = before + gt < target && target <= before + gt + eq;
    }
    __syncwarp();
    const unsigned who = __ballot_sync(0xffffffffu, found);
    if (!who) return false;
    value = __shfl_sync(0xffffffffu, mine, __ffs(who) - 1);
    return true;
    }
    return false;
}

// The mass of what the group's warps have listed, beyond what their lists hold too, where that is one value.
template <bool CL>
static __device__ __noinline__ u64 listed_mass(const Grp<CL> g, const RowS& rw, float value) {
    Sc* sc = scratch();
    uint32_t n = 0;
    for (int i = lane_id(); i < NW * (CL ? g.C : 1); i += 32) n += (uint32_t)g.at(sc, i / NW)->wn[i % NW];
    return (u64)__reduce_add_sync(0xffffffffu, n) * (u64)rw.mass(value);
}

// How a wide row is cut, from its histogram (summed over the CTAs of the cluster): by one warp of every CTA.  A lane holds 32
// buckets; a rank or a share of the estimated mass is found by a scan over the lanes and one over the buckets of the lane it
// falls into.  The estimated mass of a logit of bucket b is 2^min(0, e0 - b * e1) (of the last bucket, which holds everything
// beyond, 0; of the cut's bucket the part above the cut): float sums, they only say where to look.
// The bucket that holds the rank-th largest logit (-1: there are fewer), and how many there are before it and with it.  inc, cnt: of
// the lane's buckets and those before, and of the lane's alone.
struct Ranked { int b; uint32_t before, with; };
static __device__ __noinline__ Ranked ranked(const uint32_t* hist, int last, uint32_t inc, uint32_t cnt, uint32_t rank) {
    const int lane = lane_id();
    const unsigned hit = __ballot_sync(0xffffffffu, inc >= rank);
    const int hl = hit ? __ffs(hit) - 1 : 31, b = hl * 32 + lane;
    const uint32_t n = b > last ? 0u : hist[b];
    uint32_t i = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t x = __shfl_up_sync(0xffffffffu, i, o); if (lane >= o) i += x; }
    i += __shfl_sync(0xffffffffu, inc - cnt, hl);
    const unsigned in = __ballot_sync(0xffffffffu, i >= rank);
    const int t = in ? __ffs(in) - 1 : 31;
    return Ranked{hit ? hl * 32 + t : -1, __shfl_sync(0xffffffffu, i - n, t), __shfl_sync(0xffffffffu, i, t)};
}
// The middle between the first bf16 >= x (below: the last one <= x) and the next one above: in a row of bf16 logits the edge of a set
// of values.
__device__ __forceinline__ float above_bf16(float x, bool below) {
    int s = __float_as_int(x);
    s = s < 0 ? (int)(0x80000000u - (uint32_t)s) : s;                    // in the order of the floats
    s = ((s + (below ? 0 : 0xFFFF)) & ~0xFFFF) + 0x8000;
    return s >= 0x7F800000 ? SM_POS_INF : __int_as_float(s < 0 ? (int)(0x80000000u - (uint32_t)s) : s);
}
template <bool CL>
static __device__ __noinline__ void decide_row(const Grp<CL> g, RowS& rw, int elt, bool miss) {
    Sc* sc = scratch();
    const uint32_t* hist = reinterpret_cast<const uint32_t*>(smem + (CL ? OFF_BINS : OFF_U));
    const int lane = lane_id(), C = CL ? g.C : 1;
    const bool ready = rw.hist_ready != 0, full = !ready || rw.hist_full;
    const float href = ready ? rw.lref : rw.L, lcut = rw.lcut, scw = rw.scw, width = RANGE / (float)NB1 * rw.tc;
    const int hoff = ready ? HOFF : 0;
    const int last = Buckets(href, scw, hoff)(lcut);                     // buckets wholly below the cut are left out
    // bucket b's centre lies (b - hoff + 1/2) * RANGE / NB1 + dL temperatures below the row's maximum
    const float e1 = RANGE / (float)NB1 * CI_LOG2E;
    const float e0 = ((float)hoff - 0.5f) * e1 - (rw.L - href) * __frcp_rn(rw.tc) * CI_LOG2E;
    const float last_part = fminf(fmaxf((href - (float)(last - hoff) * width - lcut) * scw, 0.0f), 1.0f);
    auto edge = [&](int b) { return href - (float)(b - hoff) * width; };
    auto weight = [&](int b) {
        float e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(fminf(0.0f, fmaf(-(float)b, e1, e0))));
        return b == NB1 - 1 ? 0.0f : e;
    };
    auto at = [&](int b) { return b > last ? 0u : hist[b]; };
    // the lane's buckets
    uint32_t cnt = 0; float est = 0.0f, cut_off = 0.0f;                  // (cut_off: what lies below the cut)
#pragma unroll 2
    for (int j = 0; j < 8; ++j) {
        const int b = lane * 32 + 4 * ((j + lane) & 7);                  // (the lanes start at different banks)
        const uint4 x = *reinterpret_cast<const uint4*>(hist + b);
        const uint32_t n[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float w = (float)n[i] * weight(b + i);
            if (b + i <= last) { cnt += n[i]; est += b + i == last ? w * last_part : w; }
            if (b + i >= last) cut_off += b + i == last ? w * (1.0f - last_part) : w;
        }
    }
    uint32_t inc_c = cnt; float inc_e = est;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, inc_c, o); const float y = __shfl_up_sync(0xffffffffu, inc_e, o);
        if (lane >= o) { inc_c += x; inc_e += y; }
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc_c, 31);
    const float mass = __shfl_sync(0xffffffffu, inc_e, 31);
    // the row's mass relative to its maximum, without what lies below the cut
    float all = 0.0f;
    for (int i = lane; i < NW * C; i += 32) all += g.at(sc, i / NW)->est[i % NW];
#pragma unroll
    for (int o = 16; o; o >>= 1) { all += __shfl_xor_sync(0xffffffffu, all, o); cut_off += __shfl_xor_sync(0xffffffffu, cut_off, o); }
    {
        float e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"((href - rw.L) * __frcp_rn(rw.tc) * CI_LOG2E));
        all = all * e - cut_off;
    }
    if (!CL && ready && rw.hist_full) all = mass;                        // (counted in full by a pass that does not sum)
    auto find_rank = [&](uint32_t rank, uint32_t& before, uint32_t& with) {
        const Ranked r = ranked(hist, last, inc_c, cnt, rank);
        before = r.before; with = r.with;
        return r.b;
    };
    int path = PATH_PURE;
    float t_hi = CI_NEG_INF, t_lo = SM_POS_INF;
    int band_top = 0, band_bot = 0;
    uint32_t before, with;
    if (rw.kk > 0 && rw.kk < sc->V && (uint32_t)rw.kk < total) {         // (else at most k reach the cut's bucket: top-k removes nothing)
        const int b = find_rank((uint32_t)rw.kk, before, with);
        // (bucket 0 of a histogram laid out from the sample may hold logits from far above it)
        if (b < (ready ? 1 : 0) || b >= NB1 - 3 || with > (uint32_t)LIST_MAX) path = PATH_FALLBACK;
        else { path = PATH_LIST; t_lo = edge(b + 2) - 0.01f * width - fabsf(href) * 1e-6f; }
    } else if (rw.topp < 1.0f) {
        const float target = mass - (1.0f - rw.topp) * all;
        const unsigned hit = __ballot_sync(0xffffffffu, inc_e >= target);
        int bp = -1;
        float part = 0.5f;                                               // of the pivot's bucket, what lies above it
        if (mass > 0.0f) {
            const int hl = hit ? __ffs(hit) - 1 : 31;
            const float w = (float)at(hl * 32 + lane) * weight(hl * 32 + lane) * (hl * 32 + lane == last ? last_part : 1.0f);
            float i = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const float x = __shfl_up_sync(0xffffffffu, i, o); if (lane >= o) i += x; }
            i += __shfl_sync(0xffffffffu, inc_e - est, hl);
            const unsigned in = __ballot_sync(0xffffffffu, i >= target);
            bp = hl * 32 + (in ? __ffs(in) - 1 : 31);
            bp = min(bp, last);
            part = __saturatef(__fdividef(target - __shfl_sync(0xffffffffu, i - w, bp & 31), fmaxf(__shfl_sync(0xffffffffu, w, bp & 31), 1e-30f)));
        }
        if (bp < 0) path = PATH_FALLBACK;
        else {
            // how many lie before the pivot's bucket and with it (at least one logit's rank apart)
            uint32_t n = hist[(bp & ~31) + lane];
            if ((bp & ~31) + lane > last) n = 0;
            uint32_t i = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const uint32_t x = __shfl_up_sync(0xffffffffu, i, o); if (lane >= o) i += x; }
            i += __shfl_sync(0xffffffffu, inc_c - cnt, bp >> 5);
            const uint32_t n0 = __shfl_sync(0xffffffffu, i - n, bp & 31), n1 = __shfl_sync(0xffffffffu, i, bp & 31);
            // The band: so many logits on either side of the estimated pivot, within buckets by interpolation.  After a full count a
            // hundred (bf16: four hundred, one value's logits are many), after a sample more, the more the further down.
            uint32_t x0 = 0, x1 = 0;
            const uint32_t rank = n0 + (uint32_t)(part * (float)(n1 - n0)), near = elt == 2 ? 400u : 100u;
            uint32_t side = full ? near : min(min((uint32_t)BAND_SIDE, 300u + (uint32_t)sc->V / 256), near + rank / 4);
            // bf16 logits there: from one to the next, in buckets.  (Four to a bucket and more: as good as evenly spread over it.)
            const float x = href - ((float)(bp - hoff) + part) * width;
            const float step = __int_as_float(max((__float_as_int(x) & 0x7F800000) - (7 << 23), 0)) * scw;
            const bool coarse = elt == 2 && step > 0.25f;
            // (either end moves out by up to a value's logits, and by a part of them more where the pivot's bucket holds fewer values than
            // others: that the lists hold them all it gives way, by half at most.)  512 rows of 262,144 logits N(0, 2^2), T = 0.8,
            // top_p 0.95: 13 of them overflowed a list where half a value was made room for, 282 -> 350 us; now as before.
            if (coarse) {
                const uint32_t room = CL ? 7 * GCAP * NW / 20 : BAND_SIDE, value = (uint32_t)((float)(n1 - n0) * fminf(1.5f * step, 1.25f));
                side = min(side, max(room - min(value, room), side / 2));
            }
            auto logit_at = [&](uint32_t r, int& bb) {                   // about the r-th largest
                bb = find_rank(r, x0, x1);
                return href - ((float)(bb - hoff) + __fdividef((float)(r - x0), fmaxf((float)(x1 - x0), 1.0f))) * width;
            };
            band_top = 0; t_hi = SM_POS_INF;
            if (rank > side) t_hi = logit_at(rank - side, band_top);
            t_lo = rank + side > total ? -SM_FLT_MAX : logit_at(rank + side, band_bot);
            if (!(t_lo > -SM_FLT_MAX)) band_bot = NB1 - 1;
            if (coarse) {
                // A bucket may hold a single value, of thousands of logits, which lies anywhere in it: the band ends between values,
                // and reaches to the ends of its buckets where the next value lies beyond them.  300 rows of N(16, 1), 151,936
                // logits: 245 -> 160 us at 150 rows in the launch, 551 -> 345 at 592 (191 of 300 bands missed the pivot, now none).
                const float eps = 0.01f * width + fabsf(href) * 1e-6f;
                if (t_hi < SM_POS_INF) t_hi = fminf(above_bf16(t_hi, false), above_bf16(edge(band_top) + eps, true));
                if (t_lo > -SM_FLT_MAX) t_lo = -fminf(above_bf16(-t_lo, false), above_bf16(-(edge(band_bot + 1) - eps), true));
            }
            const int cap = find_rank(500u, x0, x1);
            if (cap < 0 || cap > band_bot) {
                band_top = 0; band_bot = cap < 0 ? NB1 - 1 : cap - 1;
                t_hi = SM_POS_INF; t_lo = cap < 0 ? -SM_FLT_MAX : edge(cap);
            }
            path = PATH_BAND;
            if (band_bot >= NB1 - 2) { t_lo = -SM_FLT_MAX; band_bot = NB1 - 1; }
            band_top = max(band_top, 0);
            if (!(t_lo < t_hi)) t_lo = t_hi - width;
            if (miss && band_top > 0) {                                  // test hook: a band off by its own width and eight buckets (above or below by row parity)
                const int by = band_bot - band_top + 8, s8 = (rw.row & 1) ? by : -by;
                if (band_top + s8 > 0 && band_bot + s8 + 2 < NB1) {
                    band_top += s8; band_bot += s8;
                    t_hi = edge(band_top); t_lo = edge(band_bot + 1);
                }
            }
        }
    }
    if (lane == 0) { rw.path = path; rw.t_hi = t_hi; rw.t_lo = t_lo; rw.band_top = band_top; rw.band_bot = band_bot; rw.href = href; rw.hoff = hoff; }
}

// A row's parameters, one 32-bit word per lane: temperature, top_k, top_p, log_min_p, seed (low), the three penalties, seed (high),
// hist_len, position (low, high), explicit uniform.
__device__ __forceinline__ uint32_t load_params(const Args& a, int row, int lane) {
    int r;
    const int b = slot_of(a, row, r);
    const uint32_t* src = nullptr;
    size_t at = b;
    if (lane < 10) {
        src = reinterpret_cast<const uint32_t*>(reinterpret_cast<const void* const*>(&a.p)[lane == 8 ? 4 : lane]);
        if (lane == 4 || lane == 8) at = 2 * (size_t)b + (lane == 8);
    } else if (lane < 12) {
        if (a.u == nullptr && (a.pos_i64 || lane == 10)) src = reinterpret_cast<const uint32_t*>(a.pos);
        if (a.pos_i64) at = 2 * (size_t)b + (lane - 10);
    } else if (lane == 12) {
        if (row < a.second.rows1) src = reinterpret_cast<const uint32_t*>(a.u);
        at = row;
    }
    return src ? __ldg(src + at) : lane == 5 || lane == 12 ? 0x3F800000u : lane == 9 ? (uint32_t)a.p.hist_stride : 0u;
}
static_assert(offsetof(colinfer_sampler_params, hist_len) == 9 * sizeof(void*) && offsetof(colinfer_sampler_params, seed) == 4 * sizeof(void*) &&
              offsetof(colinfer_sampler_params, frequency_penalty) == 7 * sizeof(void*), "load_params indexes the pointers");

// Where a row lies.
template <int ELT>
__device__ __forceinline__ const char* place_row(const Args& a, int row, int& al, uint32_t& end, int& nc) {
    const u64 bytes = (u64)a.V * ELT, addr = reinterpret_cast<u64>(logits_of(a, row)) + (u64)row * bytes;
    const bool two = row >= a.second.rows1;
    al = (int)((addr & 15) / ELT);
    end = row_span(addr, bytes, two ? row - a.second.rows1 : row, (two ? a.second.rows : min(a.second.rows1, a.second.rows)) - 1 - row);
    nc = (a.V + al + CHUNK - 1) / CHUNK;
    return reinterpret_cast<const char*>(addr & ~15ull);
}
// Fills in a row from its parameters (load_params' words).  One warp.
template <int ELT>
static __device__ __noinline__ void derive_row(const Args& a, RowS& rw, int row, uint32_t words) {
    auto word = [&](int l) { return __shfl_sync(0xffffffffu, words, l); };
    auto num = [&](int l) { return __uint_as_float(word(l)); };
    int r;
    const int b = slot_of(a, row, r);
    const float T = num(0), topp = num(2), rp = num(5), pp = num(6), fp = num(7);
    const int kk = (int)word(1);
    float u = num(12);
    if (a.u == nullptr) {
        const u64 seed = ((u64)word(8) << 32) | word(4);
        long long pos = (int)word(10);
        if (a.pos_i64) pos = (long long)(((u64)word(11) << 32) | word(10));
        u = a.pos != nullptr && a.p.seed != nullptr ? u32_to_uniform(philox_word(philox_key((int64_t)seed), (u64)pos + (u64)r)) : 1.0f;
    }
    const float lmp = num(3);
    const int hlen = a.p.history ? max(0, min((int)word(9), a.p.hist_stride)) : 0;
    if (lane_id() == 0) {
        rw.base = place_row<ELT>(a, row, rw.a, rw.end, rw.Nc);
        rw.row = row; rw.key = row + 1;
        rw.mrow = a.mask ? a.mask + ((size_t)b * a.mask_rows + r) * a.W : nullptr;
        rw.hist = a.p.history ? a.p.history + (size_t)b * a.p.hist_stride : nullptr;
        rw.hlen = hlen; rw.rp = rp; rw.pp = pp; rw.fp = fp;
        rw.pen_on = hlen > 0 && !(rp == 1.0f && pp == 0.0f && fp == 0.0f);
        rw.pen_cap = hlen <= 65535 ? PEN_TABLE : 0;              // (the counts are 16 bits)
        const bool sampled = (T > 0.0f) || (a.flags & COLINFER_FORCE_DISTRIBUTION);
        const bool fastk = sampled && kk > 0 && kk <= FASTK && kk < a.V;
        const bool wide = sampled && !fastk && ((kk > 0 && kk < a.V) || topp < 1.0f);
        rw.cls = (sampled ? ROW_SAMPLED : 0) | (fastk ? ROW_FASTK : 0) | (wide ? ROW_WIDE : 0);
        rw.tc = fmaxf(T, 1e-6f); rw.kk = kk; rw.topp = topp; rw.lmp = lmp;
        rw.scw = (float)NB1 / (RANGE * rw.tc);
        rw.u = u;
        rw.hist_slow = 0;
    }
}

// The hardware's queue of the grid's CTAs that have not started: a running CTA asks for the index of one of them, which then
// never starts (cluster launch control).  One thread; the answer lands in sc->clc.
__device__ __forceinline__ void queue_ask(Sc* sc) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // (the last answer has been read)
    mbar_expect_tx(&sc->clc_bar, 16);
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                 ::"r"(smem_u32(&sc->clc)), "r"(smem_u32(&sc->clc_bar)) : "memory");
}
// The index, -1 when none was left (or the answer does not come).
__device__ __forceinline__ int queue_answer(Sc* sc, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_test(&sc->clc_bar, parity)) if (clock64() - t0 > WAIT_CYCLES) { sc->dead = 1; return -1; }
    uint32_t ok, x;
    asm volatile("{\n\t.reg .b128 h;\n\t.reg .pred p;\n\tld.shared.b128 h, [%2];\n\t"
                 "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\tselp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
                 "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
                 : "=r"(ok), "=r"(x) : "r"(smem_u32(&sc->clc)) : "memory");
    return ok ? (int)x : -1;
}

// CL: the launch uses clusters (a.cluster > 1 CTAs per row); ELT: bytes per logit (4 fp32, 2 bf16); MASK: it has a grammar mask.
template <bool CL, int ELT, bool MASK>
__global__ void __launch_bounds__(NT, CTAS_PER_SM) k_sample(const __grid_constant__ Args a) {
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    const int V = a.V;
    Grp<CL> g;
    g.C = CL ? a.cluster : 1;
    g.rank = CL ? (int)(blockIdx.x % a.cluster) : 0;
    const int GW = NW * g.C, gw = g.rank * NW + warp;            // warps of the group, this warp among them

    Sc* sc = scratch();
    Cand* klist = reinterpret_cast<Cand*>(smem + OFF_U);         // [NW][KCAPC]: rows without a histogram,
    uint32_t* hist = reinterpret_cast<uint32_t*>(smem + OFF_U);  // or [NB1],
    Cand* wlist = reinterpret_cast<Cand*>(smem + OFF_U + OFF_LISTS);     // [NW][WCAPC]
    Cand* push = reinterpret_cast<Cand*>(smem + OFF_U + OFF_GATHER);     // [C][PUSH / C] candidates of all CTAs,
    Cand* gath = push;                                           // or [NW][GCAP] lists of all CTAs
    constexpr int WCAPC = CL ? WCAP_CL : WCAP, KCAPC = CL ? KCAP_CL : KCAP;
    uint32_t* bitmap = reinterpret_cast<uint32_t*>(smem + OFF_U);        // history bitmap while the tables are built (may reach over bins and csum)
    uint32_t* sbins = reinterpret_cast<uint32_t*>(smem + OFF_BINS);      // [BINS] sample
    uint32_t* fbins = sbins + BINS;                          // [BINS] selection
    u64* bins = reinterpret_cast<u64*>(sbins);                   // [BINS] weighted selections, radix levels
    float* xbuf = reinterpret_cast<float*>(sbins);               // [CHUNK] the chunk the draw falls into
    u64* csum = reinterpret_cast<u64*>(smem + OFF_CSUM);         // [chunks] kept mass per chunk (the CTA's own)

    constexpr int PW = NW - 1;                                   // the warp that looks after the row that comes next
    uint32_t next_words = 0;                                     // (its parameters, a word per lane)
    if (CL && warp == PW) next_words = load_params(a, blockIdx.x / a.cluster, lane);   // (before the logits keep the memory busy)
    if (tid == 0) {
        sc->V = V; sc->W = a.W; sc->GW = GW; sc->rank = g.rank;
        sc->dead = 0;
        sc->pen_off = pen_offset(V, a.p.history != nullptr);
        sc->flags = 0; sc->nsel = sc->npush = 0; sc->sum_all = sc->sum_keep = 0;
    }
    if (lane == 0) {
        const uint32_t bar = smem_u32(smem) + OFF_BARS + warp * (8 * NST);
        sc->ring[warp] = WarpRing{0, 0, 0, !((a.flags & COLINFER_TEST_DROP_COPY) && !(warp & 1)), 0};   // (test flag: every other warp asks for nothing)
        sc->wn[warp] = 0; sc->swf[warp] = CI_NEG_INF;
        for (int j = 0; j < NST; ++j) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * j) : "memory");
        fence_mbar_init();
    }
    __syncthreads();

    // ---------------------------------------------------------------------------------------- which rows are this group's
    const int n_rows = a.second.rows;
    const int grp = CL ? blockIdx.x / a.cluster : blockIdx.x, n_grp = CL ? gridDim.x / a.cluster : gridDim.x;
    // Without clusters the grid has a CTA per row, of which as many start as fit; a CTA that is through with its row takes the
    // next one off the hardware's queue.  Rows differ in cost (a wide row takes two or three passes, any other one): the CTAs'
    // indices are positions in an order of the rows by cost class, dearest first, which every CTA works out for itself.
    // With at most two rows per SM they all start at once, CTA j + NUM_SM beside CTA j: the dearest rows get an SM of their own,
    // of the others the dearest goes with the cheapest.
    const bool dealt = !CL && n_rows > NUM_SM && n_rows <= BAL_ROWS;
    auto row_class = [&](int row) {
        int r;
        const int b = slot_of(a, row, r);
        const float T = a.p.temperature[b];
        const int k = a.p.top_k[b];
        if (!((T > 0.0f) || (a.flags & COLINFER_FORCE_DISTRIBUTION))) return 2;
        return (k > 0 && k <= FASTK && k < V) ? 1 : 0;
    };
    const int per_thread = (n_rows + NT - 1) / NT;               // consecutive rows per thread
    if (dealt) {
        u64 packed = 0, tot;
#pragma unroll 4
        for (int j = 0; j < per_thread; ++j) { const int row = tid * per_thread + j; if (row < n_rows) packed += 1ull << (21 * row_class(row)); }
        const u64 ex = block_excl_scan(packed, sc, tot);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            sc->cls_pre[j][tid] = (unsigned short)((ex >> (21 * j)) & 0x1FFFFFull);
            if (tid == 0) sc->cls_tot[j] = (int)((tot >> (21 * j)) & 0x1FFFFFull);
        }
        __syncthreads();
    }
    // The row at a position of that order.  One warp.
    auto row_of = [&](int pos) {
        if (!dealt) return pos;
        if (CTAS_PER_SM == 2 && n_rows <= 2 * NUM_SM) {
            const int pairs = n_rows - NUM_SM;
            pos = pos >= NUM_SM ? n_rows - 1 - (pos - NUM_SM) : pos < pairs ? NUM_SM - pairs + pos : pos - pairs;
        }
        int j = 0;
        while (j < 2 && pos >= sc->cls_tot[j]) { pos -= sc->cls_tot[j]; ++j; }
        int t = 0;                                               // the last thread with at most pos rows of class j before its own
#pragma unroll
        for (int step = 512; step; step >>= 1) if (t + step < NT && sc->cls_pre[j][t + step] <= pos) t += step;
        int left = pos - sc->cls_pre[j][t], row = 0;
        for (int j0 = 0; j0 < per_thread; j0 += 32) {
            const int k = t * per_thread + j0 + lane;
            const unsigned is = __ballot_sync(0xffffffffu, j0 + lane < per_thread && k < n_rows && row_class(k) == j);
            const int c = __popc(is);
            if (left < c) {
                unsigned m = is;
                for (int q = 0; q < left; ++q) m &= m - 1;
                row = t * per_thread + j0 + __ffs(m) - 1;
                break;
            }
            left -= c;
        }
        return row;
    };
    // The last warp looks after the row that comes next: takes it off the queue early in the first pass of the row at hand, notes
    // where it lies, fetches its parameters, and derives the rest before the row at hand ends.
    int next_row = -1;                                           // (the last warp's)
    auto find_next = [&](int it) {                               // number it + 1
        if (CL) { const int row = grp + (it + 1) * n_grp; next_row = row < n_rows ? row : -1; }
        else {
            int pos = -1;
            if (lane == 0) pos = queue_answer(sc, it & 1);
            pos = __shfl_sync(0xffffffffu, pos, 0);
            next_row = pos >= 0 ? row_of(pos) : -1;
        }
        if (next_row >= 0) {
            next_words = load_params(a, next_row, lane);
            if (a.p.history) {                                   // the history's lines into L2
                int r;
                const char* h = reinterpret_cast<const char*>(a.p.history + (size_t)slot_of(a, next_row, r) * a.p.hist_stride);
                for (int i = lane * 128; i < min(a.p.hist_stride, 4096) * 4; i += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(h + i));
            }
            if (lane == 0) {
                NextRow& nx = sc->next[it & 1];
                int al;
                nx.base = place_row<ELT>(a, next_row, al, nx.end, nx.Nc);
                __threadfence_block();
                *(volatile int*)&nx.key = next_row + 1;
            }
        }
        __syncwarp();
    };
    auto derive = [&](int it) { if (next_row >= 0) derive_row<ELT>(a, sc->rows[it & 1], next_row, next_words); };
#ifdef COLINFER_PROFILE
    long long prof_last = clock64();
#endif
    if (warp == PW) {
        next_row = row_of(grp);
        if (!CL) next_words = load_params(a, next_row, lane);
        if (lane == 0) {
            RowS& rw = sc->rows[0];
            rw.base = place_row<ELT>(a, next_row, rw.a, rw.end, rw.Nc);
            sc->next[0].key = sc->next[1].key = 0;
            sc->rows[0].key = next_row + 1;
            mbar_init(&sc->clc_bar, 1);
            fence_mbar_init();
        }
    }
    __syncthreads();
    // Equal rows beside each other on an SM get through together and take the next ones together: where the last turn has rows for
    // half of the CTAs they would go to every other SM in pairs.  So in such launches the second CTA of an SM starts a little later;
    // with rows of several passes by what the first pass takes alone (16 bytes a cycle).  432 top-p rows 187 -> 160 us, 360 without a
    // filter 113 -> 93, 1,024 mixed ones 212 -> 194, 1,024 greedy ones 109 -> 103.  (Mixed rows with penalties,
    // whose passes take longer than their bytes, do not stay in step: 1,024 of them 259 us with the short delay, 263 with the long one.
    // Rows that are not dealt have not been counted: the short delay.)
    if (!CL && CTAS_PER_SM == 2 && n_rows > 2 * NUM_SM && (n_rows - 1) % (2 * NUM_SM) < NUM_SM && (int)blockIdx.x >= NUM_SM && (int)blockIdx.x < 2 * NUM_SM) {
        const bool wide = dealt && (int)blockIdx.x < sc->cls_tot[0] && (a.p.history == nullptr || 2 * sc->cls_tot[0] > n_rows);
        const long long t0 = clock64(), d = (long long)V * ELT / (wide ? 16 : 48);
        while (clock64() - t0 < d) __nanosleep(200);
    }
    ring_start<CL, ELT>(sc->rows[0].key, sc->rows[0].base, sc->rows[0].end, sc->rows[0].Nc, gw, GW, true);   // the logits travel while the parameters do
    if (warp == PW) derive(0);
    __syncthreads();

    for (int it = 0; ; ++it) {
        RowS& rw = sc->rows[it & 1];
        const NextRow& nx = sc->next[it & 1];
        ring_start<CL, ELT>(rw.key, rw.base, rw.end, rw.Nc, gw, GW, true);
        bool asked = false, found = false, derived = false;      // (the last warp's)
        // (A row of several passes asks when its first one is through: the CTAs that ask before it have less left to do.)
        auto ask = [&]() { if (!CL && warp == PW && !asked) { if (lane == 0) queue_ask(sc); asked = true; } };
        auto look_ahead = [&]() { if (warp == PW && !found) { ask(); __syncwarp(); find_next(it); found = true; } };
        auto derive_next = [&]() { if (warp == PW && !derived) { look_ahead(); derive(it + 1); derived = true; if (lane == 0) sc->next[(it + 1) & 1].key = 0; } };
        SM_PROF(0);

        // ------------------------------------------------------------------------------------ penalty tables
        if (rw.pen_on) {
            // A bitmap of the history's tokens among the CTA's chunks (position order), popcounts per chunk, their prefix: a
            // token's rank is its table entry.  The first PEN_TABLE ids stay in registers.
            const PenTab pt = pen_tab(sc);
            const int hlen = rw.hlen, Nc = rw.Nc, al = rw.a;
            const int32_t* h = rw.hist;
            constexpr int HP = (PEN_TABLE + NT - 1) / NT;
            int ht[HP];
#pragma unroll
            for (int j = 0; j < HP; ++j) { const int i = tid + j * NT; ht[j] = i < hlen ? __ldg(h + i) : -1; }
            for (int i = tid; i < Nc * 4; i += NT) reinterpret_cast<uint4*>(bitmap)[i] = make_uint4(0, 0, 0, 0);
            for (int i = tid; i < PEN_TABLE / 4; i += NT) reinterpret_cast<uint4*>(pt.ent)[i] = make_uint4(0, 0, 0, 0);
            auto mine = [&](int v, int& p) {
                if (v < 0 || v >= V) return false;
                p = v + al;
                return !CL || ((p / (CHUNK * NW)) % g.C) == g.rank;
            };
            __syncthreads();
            auto mark = [&](int v) { int p; if (mine(v, p)) atomicOr(&bitmap[p >> 5], 1u << (p & 31)); };
#pragma unroll
            for (int j = 0; j < HP; ++j) mark(ht[j]);
            for (int i = tid + HP * NT; i < hlen; i += NT) mark(__ldg(h + i));
            __syncthreads();
            const int per = (Nc + NT - 1) / NT;
            const int lo = min(tid * per, Nc), hi = min(lo + per, Nc);
            auto chunk_pop = [&](int c) {
                uint32_t s = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) { const uint4 x = reinterpret_cast<const uint4*>(bitmap)[c * 4 + k]; s += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w); }
                return s;
            };
            // (where there is room behind the bitmap: every word's rank in its chunk)
            unsigned short* wpre = reinterpret_cast<unsigned short*>(smem + OFF_U) + Nc * 32;
            const bool ranked = Nc * 96 <= sc->pen_off - OFF_U;
            u64 local = 0, total_bits;
            for (int c = lo; c < hi; ++c) local += chunk_pop(c);
            uint32_t run = (uint32_t)block_excl_scan(local, sc, total_bits);
            for (int c = lo; c < hi; ++c) {
                pt.pre[c] = run;
                uint32_t in = 0;
#pragma unroll 1
                for (int k = 0; k < 4; ++k) {
                    const uint4 x = reinterpret_cast<const uint4*>(bitmap)[c * 4 + k];
                    const uint32_t n1 = in + __popc(x.x), n2 = n1 + __popc(x.y), n3 = n2 + __popc(x.z);
                    if (ranked) reinterpret_cast<uint2*>(wpre)[c * 4 + k] = make_uint2(in | (n1 << 16), n2 | (n3 << 16));
                    in = n3 + __popc(x.w);
                }
                run += in;
            }
            if (tid == 0) pt.pre[Nc] = (uint32_t)total_bits;
            __syncthreads();
            const int cap = rw.pen_cap;
            auto enter = [&](int v) {
                int p;
                if (!mine(v, p)) return;
                const int c = p >> 9;
                uint32_t rk = pt.pre[c] + __popc(bitmap[p >> 5] & ((1u << (p & 31)) - 1u));
                if (ranked) rk += wpre[p >> 5];
                else for (int i = c * 16; i < (p >> 5); ++i) rk += __popc(bitmap[i]);
                if ((int)rk < cap) { atomicOr(&pt.ent[rk], (uint32_t)(p & (CHUNK - 1))); atomicAdd(&pt.ent[rk], 65536u); }
            };
#pragma unroll
            for (int j = 0; j < HP; ++j) enter(ht[j]);
            for (int i = tid + HP * NT; i < hlen; i += NT) enter(__ldg(h + i));
            __syncthreads();
        }
        SM_PROF(1);

        // ------------------------------------------------------------------------------------ pass 1
        {
            const int cls = rw.cls;
            const bool fastk = (cls & ROW_FASTK) != 0, wide = (cls & ROW_WIDE) != 0, lists = fastk || wide;
            Cand* list = wlist + warp * WCAPC;
            int lcap = WCAPC;
            float tw = -SM_FLT_MAX;                              // the CTA's list bound
            float lref = CI_NEG_INF;                             // the sample's maximum (the group's): buckets hang from it
            float from = -SM_FLT_MAX;                            // nothing below can be kept
            bool count_hist = false;
            int seen = 0;                                        // first chunks of the warp that have been read
            bool in_klist = fastk;
            if (lists) {
                // The sample, the first two chunks of every warp: list bound, histogram layout.
                for (int i = tid; i < 2 * BINS; i += NT) sbins[i] = 0u;
                if (wide) for (int i = tid; i < NB1 / 4; i += NT) reinterpret_cast<uint4*>(hist)[i] = make_uint4(0, 0, 0, 0);
                float gm[8], sm = CI_NEG_INF;
#pragma unroll
                for (int j = 0; j < 8; ++j) gm[j] = CI_NEG_INF;
                {
                    Pipe<ELT> p;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int c = gw + j * GW;
                        if (c >= rw.Nc) continue;
                        const uint32_t mw = MASK ? mask_word(rw.mrow, a.W, rw.a, c, lane) : 0u;
                        PenPeek pk = {0, 0, 0};
                        if (rw.pen_on) pk = pen_peek(pen_tab(sc), rw.pen_cap, c, lane);
                        p.wait(j);
                        if ((c == 0 && rw.a) || c == rw.Nc - 1) mend_edges<ELT>(rw, p.stage(j), c);
                        auto k = open_chunk<ELT, MASK>(rw, p.stage(j), c, mw);
                        if (pk.r0 != pk.r1) penalise(rw, k, p.stage(j), p.conv(), true, pk, pen_vals(rw));
                        ++seen;
#pragma unroll
                        for (int e = 0; e < 4; ++e) { gm[4 * j + e] = max4(k.group(e, CI_NEG_INF), CI_NEG_INF); sm = fmaxf(sm, gm[4 * j + e]); }
                        __syncwarp();
                    }
                }
                sm = warp_max(sm);
                if (lane == 0) sc->swf[warp] = sm;
                if (CL && wide) g.sync(); else __syncthreads();
                // the bins of the bound hang from the smallest finite warp maximum plus 4: a few dominant tokens in the sample
                // must not stretch them beyond the bulk
                float hi = CI_NEG_INF, lo = SM_POS_INF;
                for (int i = lane; i < ((CL && wide) ? GW : NW); i += 32) {
                    const float x = (CL && wide) ? g.at(sc, i / NW)->swf[i % NW] : sc->swf[i];
                    hi = fmaxf(hi, x);
                    if (x > CI_NEG_INF) lo = fminf(lo, x);
                }
                hi = warp_max(hi); lo = -warp_max(-lo);
                lref = hi;
                const float top = fminf(lo + 4.0f, hi);          // +inf when no warp saw a finite logit
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (gm[k] > CI_NEG_INF && top < SM_POS_INF)
                        atomicAdd(&sbins[(max(0, min(BINS - 1, __float2int_rz((top - gm[k]) * FAST_SCALE))))], 1u);
                __syncthreads();
                auto bound = [&](int k) {                        // what at least k logits of the CTA's share reach (-FLT_MAX: unknown)
                    uint32_t have;
                    const int bk = warp_count_bin(sbins, (uint32_t)k, have);
                    return bk >= 0 && bk < BINS - 1 ? top - ((float)(bk + 1) + 0.01f) / FAST_SCALE - fabsf(top) * 1e-6f : -SM_FLT_MAX;
                };
                tw = bound(fastk ? rw.kk : 8);
                if (wide && lref > CI_NEG_INF && lref < SM_POS_INF) {
                    // A wide row does without a histogram where a list is sure to hold all the mass: what can be kept lies above the
                    // min-p cut, or the mass horizon, of the sample's maximum (the row's can only be larger), and the sample says
                    // that this is at most half of what the lists hold.
                    const float tc = rw.tc;
                    const float sure = fmaxf(lref + rw.lmp * tc, lref - 22.0f * tc) - fabsf(lref) * 1e-5f - 1e-5f * tc;
                    const int share = (rw.Nc + g.C - 1) / g.C;   // chunks of the CTA
                    const float t2 = bound(max(1, KCAPC * NW * NW / share));
                    count_hist = !(t2 > -SM_FLT_MAX && t2 < sure);
                    from = lref - 22.0f * tc - fabsf(lref) * 1e-5f - 1e-5f * tc;
                    if (!count_hist) { tw = sure; in_klist = true; }
                    else if (rw.kk > 0 && rw.kk < V) {
                        // So does a row with a top-k, where the sample says how far down the k-th largest lies: four standard
                        // deviations below that, and so many logits as fill 65 % of the lists, or a warp's may not hold its share
                        // (180 of 277 logits with two CTAs per SM; the share's standard deviation, the bound's included, is 20).  592 fp32
                        // rows, one pass and two: 151,936 logits, top_k up to 1,500, 136 and 203 us; 262,144, up to 1,200, 163 and 272.
                        const float f = (float)min(2 * NW, share) / (float)share, want = (float)rw.kk / (float)g.C * f;
                        const int r = (int)(want + 4.0f * sqrtf(want)) + 8;
                        const float t3 = bound(r);
                        if ((float)r < 0.65f * f * (float)(KCAPC * NW) && t3 > -SM_FLT_MAX) { count_hist = false; tw = fmaxf(t3, sure); in_klist = true; }
                    }
                }
                if (in_klist) { list = klist + warp * KCAPC; lcap = KCAPC; }
                if (tid == 0) sc->in_klist = in_klist;
                if (tid == 0) { rw.lref = lref; rw.count_hist = count_hist; rw.hist_full = CL || (rw.kk > 0 && rw.kk < V); }
            }
            SM_PROF(2);
            if (tid == 0) sc->tw = tw;
            const bool one_pass = !(cls & ROW_SAMPLED) || in_klist;
            if (one_pass) look_ahead();
            const int then = one_pass ? THEN_NEXT_ROW : THEN_AGAIN;
            const float t = tw > -SM_FLT_MAX ? tw : SM_POS_INF;  // no bound: nothing is listed
            const int bad = (lists && !(tw > -SM_FLT_MAX) ? 1 : 0) | (wide && !count_hist ? 4 : 0) | (lists && !in_klist ? 16 : 0);
            Top top1{CI_NEG_INF, 0x7fffffff};
            float est = 0.0f;                                    // the lane's share of the row's mass relative to lref
            if (!lists) top1 = pass_max<CL, ELT, MASK>(rw, nx, !one_pass, then);
            else if (count_hist && (CL || (rw.kk > 0 && rw.kk < V))) top1.l = pass_hist<CL, ELT, MASK, true, CL>(rw, nx, true, seen, then, t, list, lcap, lref, rw.scw, HOFF, from, rw.tc, est);
            else if (!CL && count_hist) top1.l = pass_hist<CL, ELT, MASK, CL, true>(rw, nx, true, seen, then, t, list, lcap, lref, rw.scw, HOFF, from, rw.tc, est);
            else top1.l = pass_list<CL, ELT, MASK>(rw, nx, !one_pass, seen, then, t, list, lcap);
            SM_PROF(3);
            ask();
            if (lists) top1.l = warp_max(top1.l);
            if (count_hist) {
#pragma unroll
                for (int o = 16; o; o >>= 1) est += __shfl_xor_sync(0xffffffffu, est, o);
            }
            if (lane == 0) {
                sc->est[warp] = est;
                sc->wf[warp] = top1.l; sc->wi[warp] = top1.idx;
                const int f = bad | (lists && sc->wn[warp] > lcap ? 1 : 0) | (est < 1e30f ? 0 : 8);
                if (f) atomicOr(&sc->flags, f);
            }
        }
        __syncthreads();
        if constexpr (CL) {
            // one record per CTA for the others to read
            if (warp == 0) {
                float l = lane < NW ? sc->wf[lane] : CI_NEG_INF;
                int i = lane < NW ? sc->wi[lane] : 0x7fffffff;
                const float m = warp_max(l);
                i = (int)__reduce_min_sync(0xffffffffu, l == m ? (unsigned)i : 0x7fffffffu);
                if (lane == 0) sc->pub = make_float4(m, __int_as_float(i), sc->tw, __int_as_float(sc->flags));
            }
            g.sync();
        }

        // ------------------------------------------------------------------------------------ the row's maximum and cut
        bool done = true;                                        // the row needs no further pass
        {
            const int cls = rw.cls;
            const bool sampled = (cls & ROW_SAMPLED) != 0, fastk = (cls & ROW_FASTK) != 0, lists = (cls & (ROW_FASTK | ROW_WIDE)) != 0;
            const bool in_klist = sc->in_klist != 0;
            Cand* list = !in_klist ? wlist + warp * WCAPC : klist + warp * KCAPC;
            const int lcap = !in_klist ? WCAPC : KCAPC;
            float L = CI_NEG_INF, lo_all = -SM_FLT_MAX;
            int aidx = 0x7fffffff, fl = 0;
            {
                float4 e = make_float4(CI_NEG_INF, __int_as_float(0x7fffffff), -SM_FLT_MAX, 0.0f);
                if (CL) { if (lane < g.C) e = g.at(sc, lane)->pub; }
                else if (lane < NW) e = make_float4(sc->wf[lane], __int_as_float(sc->wi[lane]), sc->tw, __int_as_float(sc->flags));
                L = warp_max(e.x);
                aidx = (int)__reduce_min_sync(0xffffffffu, e.x == L ? (unsigned)__float_as_int(e.y) : 0x7fffffffu);
                lo_all = warp_max(e.z);
                fl = (int)__reduce_or_sync(0xffffffffu, (unsigned)__float_as_int(e.w));
            }
            const bool lists_ok = lists && !(fl & 1), all_klist = lists && !(fl & 16);   // (of all CTAs)
            const bool finite_max = (L > CI_NEG_INF) && (L < SM_POS_INF);
            if (lists && (a.stats || !finite_max)) {
                // the lowest index of the maximum, for rows whose pass only listed: from the lists, else from one more pass
                int x;
                if (lists_ok && finite_max) {
                    uint32_t best = 0x7fffffffu;
                    for (int j = lane; j < min(sc->wn[warp], lcap); j += 32) if (list[j].l == L) best = min(best, list[j].idx);
                    x = (int)__reduce_min_sync(0xffffffffu, best);
                } else {
                    x = argmax_pass<CL, ELT, MASK>(rw, nx, L);
                }
                if (lane == 0) sc->wi[warp] = x;
                g.sync();
                x = 0x7fffffff;
                for (int i = lane; i < GW; i += 32) x = min(x, g.at(sc, i / NW)->wi[i % NW]);
                aidx = (int)__reduce_min_sync(0xffffffffu, (unsigned)x);
            }
            if (aidx == 0x7fffffff) aidx = 0;
            const float tc = rw.tc;
            float lcut = CI_NEG_INF, horizon = CI_NEG_INF;
            MassFn mass;
            mass.tc = tc; mass.rinv = 0.0f; mass.m = 0.0f;
            const bool go = sampled && finite_max;
            if (go) {
                const float m = scale_logit(L, tc);
                mass.init(tc, m);
                if (rw.lmp > CI_NEG_INF) {
                    const float thr = __fadd_rn(m, rw.lmp);
                    lcut = lower_logit_for(thr, tc, __fmul_rn(thr, tc));
                }
                // Logits more than 22 temperatures below the maximum have integer mass 0 (2^30 exp(-22) < 1/2): they can never
                // be drawn and add nothing to any sum, so every selection works above that horizon.  (A top-k whose k-th
                // largest lies below it removes nothing that could be drawn.)
                horizon = L - 22.0f * tc - fabsf(L) * 1e-6f;
            }
            if (tid == 0) {
                rw.L = L; rw.aidx = aidx; rw.status = sampled && !finite_max ? COLINFER_ROW_DEGENERATE : 0;
                rw.hist_ready = rw.count_hist && !(fl & 12) && !fastk && (rw.hist_full ? (L - rw.lref) * rw.scw < (float)(HOFF - 2) : !(fl & 1));   // the maximum lies inside the buckets; what was not sampled is listed
                rw.minp = lcut > horizon;
                rw.lcut = fmaxf(lcut, horizon); rw.horizon = horizon; rw.mass = mass;
                rw.drawn = 0; rw.token = aidx; rw.total = 0; rw.listed = 0;
            }
            lcut = fmaxf(lcut, horizon);
            SM_PROF(4);
            if (go) {
                done = false;
                // ---------------------------------------------------------------------------- finish from the lists
                // Small top-k rows; and any other row whose bound lies below the cut: every logit that carries mass is listed
                // (top-k, if any, then removes nothing beyond the list).
                if (lists_ok && (fastk || lo_all < lcut)) {
                    const int kq = rw.kk > 0 && rw.kk < V ? rw.kk : 0x7fffffff;
                    const View w{list, lane, min(sc->wn[warp], lcap), 32};
                    float scale; int bstar, n = -1;
                    const float lo = fmaxf(lo_all, lcut);
                    if constexpr (CL) {
                        // what reaches the highest of the CTAs' bounds (at least kk logits of the CTA it comes from do) goes to the
                        // first CTA, which selects
                        const int pcap = PUSH / g.C;
                        Cand* to = g.at(push, 0) + g.rank * pcap;
                        for (int j = w.start; j < w.n; j += 32) {
                            const Cand c = w.p[j];
                            if (c.l >= lo) { const int at = atomicAdd(&sc->npush, 1); if (at < pcap) to[at] = c; }
                        }
                        g.sync();
                        if (g.rank == 0) {
                            bool good = true;
                            for (int q = 0; q < g.C; ++q) good = good && g.at(sc, q)->npush <= pcap;
                            const int wpr = NW / g.C, q = warp / wpr, mine = g.at(sc, q)->npush;
                            const View w2{push + q * pcap, (warp % wpr) * 32 + lane, mine, 32 * wpr};
                            if (good) n = select_top(w2, lo_all, lcut, L, kq, fbins, sc, scale, bstar);
                        }
                    } else {
                        n = select_top(w, lo_all, lcut, L, kq, fbins, sc, scale, bstar);
                    }
                    if (g.rank == 0) {
                        if (n > 0) {
                            order_candidates(n, mass);
                            if (warp == 0) finish_warp(lo, L, scale, bstar, lcut, tc, kq, rw.topp, rw.u);
                        } else if (tid == 0) sc->ok = 0;
                    }
                    derive_next();
                    g.sync();
                    const Sc* ps = g.at(sc, 0);
                    done = ps->ok != 0;
                    if (tid == 0) {
                        if (done) { rw.token = ps->fin_token; rw.lcut = ps->fin_cut; rw.total = ps->fin_total; }
                        // lists that hold all the mass, too long for the one-warp finish: selected on as they are
                        if (!done && !fastk && all_klist) {
                            int n = 0;
                            if (CL) for (int q = 0; q < g.C; ++q) n += g.at(sc, q)->npush;
                            if (n <= GCAP * NW * 3 / 4) { rw.path = PATH_LIST; rw.listed = 1; rw.t_lo = lo_all; }
                        }
                    }
                } else if (lists_ok && all_klist) {
                    // a top-k's list reaches down to its bound: it does if it has k logits
                    int n = 0;
                    for (int j = lane; j < min(sc->wn[warp], lcap); j += 32) n += list[j].l >= lo_all ? 1 : 0;
                    n = (int)__reduce_add_sync(0xffffffffu, (unsigned)n);
                    if (lane == 0 && n) atomicAdd(&sc->npush, n);
                    g.sync();
                    n = 0;
                    for (int q = 0; q < (CL ? g.C : 1); ++q) n += g.at(sc, q)->npush;
                    if (tid == 0 && n >= rw.kk && (!CL || n <= GCAP * NW * 3 / 4)) { rw.path = PATH_LIST; rw.listed = 1; rw.t_lo = lo_all; }
                }
            }
        }
        SM_PROF(5);

        if (!done) {
            // -------------------------------------------------------------------------------- how the row is cut
            __syncthreads();                                     // (the first thread's notes on the row)
            auto need_topk = [&]() { return rw.kk > 0 && rw.kk < V; };
            if (rw.listed) {
            } else if (need_topk() || rw.topp < 1.0f) {
                if (!rw.hist_ready) {
                    // the histogram, from the row's maximum
                    if (CL) g.sync(); else __syncthreads();      // nobody reads the lists over it any more
                    for (int i = tid; i < NB1 / 4; i += NT) reinterpret_cast<uint4*>(hist)[i] = make_uint4(0, 0, 0, 0);
                    __syncthreads();
                    recount_pass<CL, ELT, MASK>(rw, nx);
                    g.sync();
                }
                // a histogram that was sampled left the listed logits out
                if (rw.hist_ready && !rw.hist_full) {
                    const Cand* list = wlist + warp * WCAPC;
                    const Buckets bucket(rw.lref, rw.scw, HOFF);
                    for (int j = lane; j < min(sc->wn[warp], WCAPC); j += 32) atomicAdd(&hist[bucket(list[j].l)], 1u);
                }
                g.sync();
                if constexpr (CL) {                              // the histograms of all CTAs
                    for (int b = 2 * tid; b < NB1; b += 2 * NT) {
                        uint2 n = make_uint2(0, 0);
                        for (int r = 0; r < g.C; ++r) { const uint2 x = *reinterpret_cast<const uint2*>(g.at(hist, r) + b); n.x += x.x; n.y += x.y; }
                        *reinterpret_cast<uint2*>(sbins + b) = n;
                    }
                    __syncthreads();
                }
                if (warp == 0) decide_row<CL>(g, rw, ELT, (a.flags & COLINFER_TEST_MISS_BAND) != 0);
            } else if (tid == 0) { rw.path = PATH_PURE; rw.t_hi = CI_NEG_INF; rw.t_lo = SM_POS_INF; }
            if (CL) g.sync(); else __syncthreads();              // (the path is known, the finds are read, the lists are free)
            SM_PROF(6);

            // adds the listed logits that survive `cut` to their chunks' kept masses (the warp's own list)
            auto keep_listed = [&](const Cand* list, int cap, float cut, const MassFn& mass) {
                for (int j = lane; j < min(sc->wn[warp], cap); j += 32) {
                    const Cand c = list[j];
                    if (c.l >= cut) { const uint32_t q = mass(c.l); if (q) add64(&csum[(c.idx + rw.a) / CHUNK], (u64)q); }
                }
            };
            // the warps' view of the listed logits of all CTAs, in a cluster those >= floor; over: a list overflowed
            auto view_all = [&](Cand* list, int cap, float floor, bool& over) {
                View w{list, lane, 0, 32};
                over = false;
                if constexpr (CL) {
                    int n = 0;
                    for (int q = 0; q < g.C; ++q) {
                        const int c = g.at(sc, q)->wn[warp];
                        const Cand* src = g.at(list, q);
                        if (c > cap) over = true;
                        for (int j = lane; j - lane < min(c, cap); j += 32) {
                            const Cand x = src[min(j, cap - 1)];
                            const bool is = j < min(c, cap) && x.l >= floor;
                            const unsigned who = __ballot_sync(0xffffffffu, is);
                            const int at = n + __popc(who & ((1u << lane) - 1u));
                            if (is && at < GCAP) gath[warp * GCAP + at] = x;
                            n += __popc(who);
                        }
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
            // Exact radix select over the keys, four 8-bit levels, one pass each, above lcut.  by_mass: the top-p pivot; else
            // the kk-th largest.  False when the filter removes nothing.
            auto radix_select = [&](bool by_mass, float& pivot) {
                uint32_t prefix = 0;
                u64 target = by_mass ? 0 : (u64)rw.kk;
                for (int lvl = 0; lvl < 4; ++lvl) {
                    g.sync();
                    for (int i = tid; i < FB_NB; i += NT) bins[i] = 0;
                    __syncthreads();
                    pass_radix<CL, ELT, MASK>(rw, nx, rw.mass, fmaxf(rw.lcut, -SM_FLT_MAX), lvl, prefix, by_mass, bins);
                    g.sync();
                    auto level = [&](int i) { u64 s = 0; for (int q = 0; q < (CL ? g.C : 1); ++q) s += g.at(bins, q)[i]; return s; };
                    int b_star; u64 before, grand;
                    if (lvl == 0) {
                        bins_find(level, FB_NB, 0, sc, b_star, before, grand);
                        if (by_mass) target = ceil_target(rw.topp, grand);
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
            // The pivot by mass among the logits of [lo, hi], `above` being the mass beyond them: a pass per 256-fold narrowing of
            // the bracket.  A band of bf16 logits, which may hold thousands of equal ones, has at most 256 values: one pass.
            // False when the pivot lies elsewhere.  A band of a single value takes no pass at all: the lists have counted its logits
            // beyond what they hold, and so many masses of the value either reach the target or do not.
            auto bracket_select = [&](float lo, float hi, u64 target, u64 above, float& pivot) {
                uint32_t klo = f2key(lo), khi = f2key(hi);
                const bool coarse = ELT == 2 && !rw.pen_on;      // every logit is a bf16: one value among any 2^16 neighbouring keys
                for (int step = 0; step < 5; ++step) {
                    const uint32_t span = khi - klo;
                    if (span < (coarse ? 65536u : 1u)) {
                        uint32_t k = khi;
                        if (coarse) k = khi >= 0x80000000u && (khi & 0xFFFF0000u) >= klo ? khi & 0xFFFF0000u : ((khi + 1u) & 0xFFFF0000u) - 1u;
                        pivot = key2f(k);
                        if (step) return true;
                        return target - above <= listed_mass(g, rw, pivot);
                    }
                    const int sh = max(coarse ? 16 : 0, 24 - __clz(span));       // at most BINS bins
                    g.sync();
                    for (int i = tid; i < BINS; i += NT) bins[i] = 0;
                    __syncthreads();
                    pass_bracket<CL, ELT, MASK>(rw, nx, rw.mass, klo, khi, sh, bins);
                    g.sync();
                    int b; u64 before, tot;
                    bins_find([&](int i) { u64 t = 0; for (int q = 0; q < (CL ? g.C : 1); ++q) t += g.at(bins, q)[i]; return t; }, BINS, target - above, sc, b, before, tot);
                    __syncthreads();
                    if (b < 0) return false;
                    above += before;
                    khi -= (uint32_t)b << sh;
                    klo = max(klo, khi - ((1u << sh) - 1u));
                }
                return false;
            };
            // raises the cut to a pivot (ties at the pivot are kept)
            auto raise_cut = [&](float pivot) {
                const float cut = fmaxf(rw.lcut, lower_logit_for(scale_logit(pivot, rw.tc), rw.tc, pivot));
                __syncthreads();
                if (tid == 0) rw.lcut = cut;
                __syncthreads();
            };

            // -------------------------------------------------------------------------------- large top-k (then top-p) on a list
            if (rw.path == PATH_LIST) {
                Cand* list = CL && !rw.listed ? wlist + warp * WCAPC : klist + warp * KCAPC;
                const int cap = CL && !rw.listed ? WCAPC : KCAPC;
                for (int c = tid; c < rw.Nc; c += NT) csum[c] = 0;
                if (!rw.listed) {
                    if (lane == 0) sc->wn[warp] = 0;
                    __syncwarp();
                    relist_pass<CL, ELT, MASK>(rw, nx, list, cap);
                }
                g.sync();
                const MassFn mass = rw.mass;
                const float tc = rw.tc, tl = fmaxf(fmaxf(rw.t_lo, rw.lcut), -SM_FLT_MAX);
                bool over;
                const View w = view_all(list, cap, tl, over);
                float cut = fmaxf(rw.lcut, -SM_FLT_MAX);
                bool ok = !over;
                const float L = rw.L, scale = (float)(BINS - 2) / fmaxf(L - tl, 1e-30f);
                if (ok) {
                    u64 cnt = 0, surv;
                    for (int j = w.start; j < w.n; j += w.step) cnt += w.p[j].l >= cut ? 1 : 0;
                    block_excl_scan(cnt, sc, surv);
                    ok = surv > 0;
                    if (ok && need_topk() && (u64)rw.kk <= surv) {   // else fewer than k survive min-p: top-k removes nothing
                        float lkk; u64 tot;
                        const float c0 = cut;
                        ok = list_select(w, false, mass, c0, L, scale, (u64)rw.kk, lkk, tot);
                        if (ok) { cut = fmaxf(cut, lower_logit_for(scale_logit(lkk, tc), tc, lkk)); ok = cut >= tl; }   // else a tie partner could lie outside the list
                    }
                }
                if (ok && rw.topp < 1.0f) {
                    const float c0 = cut;
                    u64 part = 0, s1;
                    for (int j = w.start; j < w.n; j += w.step) part += w.p[j].l >= c0 ? (u64)mass(w.p[j].l) : 0ull;
                    block_excl_scan(part, sc, s1);
                    ok = s1 > 0;
                    if (ok) {
                        float lp; u64 tot;
                        ok = list_select(w, true, mass, c0, L, scale, ceil_target(rw.topp, s1), lp, tot);
                        if (ok) { cut = fmaxf(cut, lower_logit_for(scale_logit(lp, tc), tc, lp)); ok = cut >= tl; }
                    }
                }
                if (ok) keep_listed(list, cap, cut, mass);
                __syncthreads();
                if (tid == 0) { if (ok) rw.lcut = cut; else rw.path = PATH_FALLBACK; }
                __syncthreads();
            }
            if (rw.path == PATH_FALLBACK) {
                float lpiv;
                if (need_topk() && radix_select(false, lpiv)) raise_cut(lpiv);
                if (rw.topp < 1.0f && radix_select(true, lpiv)) raise_cut(lpiv);
                __syncthreads();
                if (tid == 0) { rw.path = PATH_PURE; rw.status |= COLINFER_ROW_SELECT_SLOW; }
                __syncthreads();
            }
            SM_PROF(7);

            // -------------------------------------------------------------------------------- mass pass: kept mass per chunk
            look_ahead();
            for (int attempt = 0; rw.path != PATH_LIST && attempt < 3; ++attempt) {
                // (with one CTA per row the band's list takes the histogram's place: the path is decided)
                Cand* blist = CL ? wlist + warp * WCAPC : klist + warp * KCAP;
                constexpr int bcap = CL ? WCAPC : KCAP;
                if (lane == 0) sc->wn[warp] = 0;
                if (attempt) {                                   // (they start a row at zero)
                    if (tid == 0) sc->sum_all = sc->sum_keep = 0;
                    __syncthreads();
                }
                __syncwarp();
                {
                    const float lk3 = fmaxf(rw.lcut, -SM_FLT_MAX), tl = fmaxf(rw.t_lo, lk3), t_hi = rw.t_hi;
                    const MassFn mass = rw.mass;
                    const bool mp = rw.minp || lk3 > rw.horizon; // (after the fallback the cut is a pivot)
                    Masses ms;
                    if (rw.path == PATH_BAND) {
                        if (!mp) ms = pass_mass<CL, ELT, MASK, true, false>(rw, nx, THEN_NEXT_ROW, mass, lk3, t_hi, tl, blist, csum);
                        else ms = pass_mass<CL, ELT, MASK, true, true>(rw, nx, THEN_NEXT_ROW, mass, lk3, t_hi, tl, blist, csum);
                        if (lane == 0) { add64(&sc->sum_all, ms.all); add64(&sc->sum_keep, ms.keep); }
                    } else if (!mp) pass_mass<CL, ELT, MASK, false, false>(rw, nx, THEN_NEXT_ROW, mass, lk3, t_hi, tl, blist, csum);
                    else pass_mass<CL, ELT, MASK, false, true>(rw, nx, THEN_NEXT_ROW, mass, lk3, t_hi, tl, blist, csum);
                }
                SM_PROF(8);
                if (rw.path != PATH_BAND) break;
                g.sync();
                u64 s1 = 0, s_above = 0;
                for (int q = 0; q < (CL ? g.C : 1); ++q) { const Sc* ps = g.at(sc, q); s1 += ps->sum_all; s_above += ps->sum_keep; }
                bool over;
                const View w = view_all(blist, bcap, -SM_FLT_MAX, over);
                const u64 target = ceil_target(rw.topp, s1);
                bool ok = !over && s1 > 0 && s_above < target;
                u64 s_band = 0;
                if (ok) {
                    const float t_hi = rw.t_hi, t_lo = rw.t_lo, lcut = rw.lcut;
                    const MassFn mass = rw.mass;
                    const float bs = t_hi < SM_POS_INF ? t_hi : rw.L;
                    // (a small nucleus lists everything above the cut: the bins span [cut, base], not [-max, base])
                    const float scale = (float)(BINS - 2) / fmaxf(bs - fmaxf(t_lo, lcut), 1e-30f);
                    float lp;
                    ok = list_select(w, true, mass, -SM_FLT_MAX, bs, scale, target - s_above, lp, s_band);
                    if (ok) {
                        const float cut2 = fmaxf(lcut, lower_logit_for(scale_logit(lp, mass.tc), mass.tc, lp));
                        if (cut2 < t_lo) ok = false;             // a tie partner could lie below the band
                        else {
                            keep_listed(blist, bcap, cut2, mass);
                            __syncthreads();
                            if (tid == 0) rw.lcut = cut2;
                        }
                    }
                }
                if (ok) break;
                bool found_band = false;
                float lpiv;
                if (s1 > 0 && s_above < target && (over || target <= s_above + s_band) && bracket_select(fmaxf(rw.t_lo, fmaxf(rw.lcut, -SM_FLT_MAX)), fminf(rw.t_hi, rw.L), target, s_above, lpiv)) {
                    // the band holds the pivot, but more logits than the lists
                    raise_cut(lpiv);
                    if (tid == 0) rw.path = PATH_PURE;
                    found_band = true;
                } else if (attempt == 0 && s1 > 0) {
                    // The estimated band missed the pivot.  Exact masses of the BINS buckets next to the band, on the side
                    // the pivot lies, give its bucket; the mass pass then runs again around it.
                    const int w0 = target <= s_above ? max(0, rw.band_top - BINS + 1) : max(0, rw.band_bot);
                    g.sync();
                    for (int i = tid; i < BINS; i += NT) bins[i] = 0;
                    __syncthreads();
                    const u64 hi = pass_window<CL, ELT, MASK>(rw, nx, rw.mass, fmaxf(rw.lcut, -SM_FLT_MAX), rw.href, rw.scw, rw.hoff, w0, bins);
                    if (lane == 0) sc->g_all[warp] = hi;
                    g.sync();
                    u64 s_hi = 0;
                    for (int i = lane; i < GW; i += 32) s_hi += g.at(sc, i / NW)->g_all[i % NW];
                    s_hi = warp_sum_u64(s_hi);
                    int bw = -1; u64 bef, tot;
                    auto win = [&](int i) { u64 s = 0; for (int q = 0; q < (CL ? g.C : 1); ++q) s += g.at(bins, q)[i]; return s; };
                    if (target > s_hi) bins_find(win, BINS, target - s_hi, sc, bw, bef, tot);
                    g.sync();
                    if (bw >= 0) {
                        const int bst = w0 + bw;
                        if (tid == 0) {
                            rw.t_hi = bst - 1 <= 0 ? SM_POS_INF : rw.href - (float)(bst - 1 - rw.hoff) / rw.scw;
                            rw.t_lo = rw.href - (float)(bst + 2 - rw.hoff) / rw.scw;
                        }
                        found_band = true;
                    }
                }
                if (!found_band) {
                    // the pivot lies far from the estimate: exact radix select by mass
                    if (radix_select(true, lpiv)) raise_cut(lpiv);
                    __syncthreads();
                    if (tid == 0) rw.path = PATH_PURE;
                }
                if (tid == 0) rw.status |= COLINFER_ROW_SELECT_SLOW;
                g.sync();
            }
            SM_PROF(9);

            // -------------------------------------------------------------------------------- the draw: chunk, then logit
            g.sync();                                            // the chunks' kept masses are complete
            {
                // the chunk in which the running kept mass reaches its target: a stretch of chunks per warp, a run of them per lane; the
                // warp whose stretch it is goes on
                const int Nc = rw.Nc, stretch = (Nc + NW - 1) / NW, run = (stretch + 31) / 32;
                const int c_lo = min(min(warp * stretch + lane * run, (warp + 1) * stretch), Nc), c_hi = min(min(c_lo + run, (warp + 1) * stretch), Nc);
                auto kept = [&](int c) { return g.at(csum, CL ? (c / NW) % g.C : 0)[c]; };
                u64 s = 0;
                for (int c = c_lo; c < c_hi; ++c) s += kept(c);
                u64 before = warp_incl_scan_u64(s, lane);
                if (lane == 31) sc->wsum[warp] = before;
                __syncthreads();
                const u64 ws = lane < NW ? sc->wsum[lane] : 0ull, upto = warp_incl_scan_u64(ws, lane), total = __shfl_sync(0xffffffffu, upto, 31);
                const u64 target = ceil_target(rw.u, total);
                const int it_is = __ffs(__ballot_sync(0xffffffffu, upto >= target)) - 1;
                if (tid == 0) { rw.total = total; if (total > 0) rw.drawn = 1; else rw.status |= COLINFER_ROW_DEGENERATE; }
                if (total > 0 && warp == it_is) {
                    before += __shfl_sync(0xffffffffu, upto - ws, warp);
                    const int hl = __ffs(__ballot_sync(0xffffffffu, before >= target)) - 1;
                    before -= s;
                    int c = c_lo;
                    if (lane == hl) {
                        for (; c < c_hi - 1; ++c) { const u64 q = kept(c); if (before + q >= target) break; before += q; }
                    }
                    before = __shfl_sync(0xffffffffu, before, hl);
                    c = __shfl_sync(0xffffffffu, c, hl);
                    if (!CL || ((c / NW) % g.C) == g.rank) {
                        // the chunk in fp32, penalties applied (its CTA has the tables), then masked
                        const char* base = rw.base;
                        const int al = rw.a;
                        float x[CHUNK / 32];                     // (loaded all at once)
#pragma unroll
                        for (int j = 0; j < CHUNK / 32; ++j) {
                            const int p = j * 32 + lane, t = c * CHUNK + p - al;
                            x[j] = CI_NEG_INF;
                            if (t >= 0 && t < V)
                                x[j] = ELT == 4 ? __ldcg(reinterpret_cast<const float*>(base) + c * CHUNK + p)
                                                : __uint_as_float((uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(base) + c * CHUNK + p) << 16);
                        }
#pragma unroll
                        for (int j = 0; j < CHUNK / 32; ++j) xbuf[j * 32 + lane] = x[j];
                        __syncwarp();
                        if (rw.pen_on) { const PenPeek pk = pen_peek(pen_tab(sc), rw.pen_cap, c, lane); if (pk.r0 != pk.r1) pen_patch(rw, smem_u32(xbuf), c, pk, pen_vals(rw)); }
                        const float lkf = fmaxf(rw.lcut, -SM_FLT_MAX);
                        const MassFn mass = rw.mass;
                        u64 q16 = 0; uint32_t q[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) {           // sixteen consecutive logits per lane
                            const int p = lane * 16 + e, t = c * CHUNK + p - al;
                            float x = xbuf[p];
                            if (MASK && t >= 0 && t < V && !((__ldg(rw.mrow + (t >> 5)) >> (t & 31)) & 1)) x = CI_NEG_INF;
                            q[e] = x >= lkf ? mass(x) : 0u;
                            q16 += q[e];
                        }
                        const u64 incl = before + warp_incl_scan_u64(q16, lane);
                        const unsigned hit = __ballot_sync(0xffffffffu, incl >= target);
                        if (hit && lane == __ffs(hit) - 1) {
                            u64 cum = incl; int e = 0;
#pragma unroll
                            for (int j = 15; j >= 0; --j) { if (cum >= target) e = j; cum -= q[j]; }   // the first whose running mass reaches the target
                            if (draws(a, rw.row)) a.out[rw.row] = (long long)(c * CHUNK + lane * 16 + e - al);
                        }
                    }
                }
                derive_next();
            }
        }
        SM_PROF(10);
        derive_next();
        // (nobody reads these of this row any more)
        if (tid < NW) { sc->wn[tid] = 0; sc->swf[tid] = CI_NEG_INF; }
        if (tid == 0) { sc->flags = 0; sc->nsel = sc->npush = 0; sc->sum_all = sc->sum_keep = 0; }
        if (CL) g.sync(); else __syncthreads();
        if (!done && rw.total == 0 && (rw.cls & ROW_WIDE) && !a.stats) {         // (a row without any kept mass emits its argmax)
            const int x = argmax_pass<CL, ELT, MASK>(rw, nx, rw.L);
            if (lane == 0) sc->wi[warp] = x;
            g.sync();
            int y = 0x7fffffff;
            for (int i = lane; i < GW; i += 32) y = min(y, g.at(sc, i / NW)->wi[i % NW]);
            y = (int)__reduce_min_sync(0xffffffffu, (unsigned)y);
            if (tid == 0) rw.token = y == 0x7fffffff ? 0 : y;
        }
        if (tid == 0 && g.rank == 0) {
            int status = rw.status;
            for (int q = 0; q < g.C; ++q) {
                if (g.at(&rw, q)->hist_slow) status |= COLINFER_ROW_HIST_SLOW;
                if (g.at(sc, q)->dead) status |= COLINFER_ROW_TIMEOUT;
            }
            if (!rw.drawn && draws(a, rw.row)) a.out[rw.row] = rw.token;
            if (a.status) a.status[rw.row] = status;
            if (a.stats) {
                colinfer_row_stats st;
                st.lmax = rw.L; st.lcut = rw.lcut; st.tc = rw.tc; st.status = status; st.argmax = rw.aidx; st.mass_q = rw.total;
                a.stats[rw.row] = st;
            }
        }
        if (CL) g.sync();                                        // nobody reads this CTA's shared memory any more
        if (nx.key == 0) break;
    }
    Pipe<ELT> p;
    p.expect(-1);                                                // nothing is on its way when the CTA ends
}

}  // namespace SMP_NAME

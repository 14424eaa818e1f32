// sample_host.h -- what the host side of the fused kernel and its three sets of instantiations know of each other.
#pragma once
#include "../../include/colinfer_b200.h"

// A second set of rows that one launch takes after the first: rows rows1 .. rows - 1 are R rows of every slot, read from
// `logits` (moved back by rows1 rows, so that the launch's row number finds them).  They have their statistics written, behind
// the first set's, but draw no token.
struct colinfer_second_rows {
    const void* logits; int R; int rows1; int rows;
};
#ifdef __CUDACC__
// What the chunk kernel's bulk copies fetch of a row of `bytes` bytes at `addr`: whole units of 16 bytes, of which the first and
// the last may hold bytes of the neighbouring rows (`before` and `after` of which the buffer has).  Where a unit would reach
// beyond the buffer the copies begin a unit later (bit 0 of the result) or end a unit earlier (the result's other bits: the low
// word of the address at which they end); the kernel reads the logits left out by ordinary loads.
__host__ __device__ inline uint32_t row_span(unsigned long long addr, unsigned long long bytes, unsigned long long before, unsigned long long after) {
    const unsigned long long end = addr + bytes, up = (end + 15) & ~15ull;
    return (uint32_t)(up - end > after * bytes ? up - 16 : up) | ((addr & 15) > before * bytes ? 1u : 0u);
}

template <class A> __device__ __forceinline__ int slot_of(const A& a, int row, int& r) {
    const bool two = row >= a.second.rows1;
    const int i = two ? row - a.second.rows1 : row, R = two ? a.second.R : a.R;
    const int b = R == 1 ? i : i / R;
    r = i - b * R;
    return b;
}
template <class A> __device__ __forceinline__ const void* logits_of(const A& a, int row) { return row >= a.second.rows1 ? a.second.logits : a.logits; }
template <class A> __device__ __forceinline__ bool draws(const A& a, int row) { return a.out != nullptr && row < a.second.rows1; }
#endif

struct colinfer_sample_args {
    const void* logits;
    const int32_t* mask; int mask_rows; int W;
    colinfer_sampler_params p;
    const void* pos; int pos_i64; const float* u;
    int64_t* out; colinfer_row_stats* stats; int32_t* status;
    int B, R, V; int flags;
    int cluster;                       // CTAs per row
    colinfer_second_rows second;
};

// index: 2 for bf16, plus 1 with a grammar mask
const void* colinfer_rows_kernel(int index);   // a CTA per row (sample_rows.cu)
int colinfer_rows_smem(int V, bool pen);
int colinfer_rows_threads();
const void* colinfer_row_kernel(int index);    // a CTA of twice the threads per row (sample_row.cu)
int colinfer_row_smem(int V, bool pen);
int colinfer_row_threads();
const void* colinfer_few_kernel(int index);    // a cluster of CTAs per row (sample_few.cu)
int colinfer_few_smem(int V, bool pen);
int colinfer_few_threads();

// colinfer_sample() on a slot's R rows and, in the same launch where there is one, statistics of R2 further rows of every slot.
int colinfer_sample_two(const void* logits, const void* logits2, int dtype, const int32_t* mask, int mask_rows, int W,
                        const colinfer_sampler_params* params, const void* pos, int pos_is_i64, const float* u, int64_t* out_ids,
                        colinfer_row_stats* stats, int32_t* status, int B, int R, int R2, int V, int flags, void* stream);

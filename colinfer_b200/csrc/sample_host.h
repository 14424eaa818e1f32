// sample_host.h -- what the host side of the fused kernel and its two sets of instantiations know of each other.
#pragma once
#include "../../include/colinfer_b200.h"

struct colinfer_sample_args {
    const void* logits;
    const int32_t* mask; int mask_rows; int W;
    colinfer_sampler_params p;
    const void* pos; int pos_i64; const float* u;
    int64_t* out; colinfer_row_stats* stats; int32_t* status;
    int B, R, V; int flags;
    int cluster;                       // CTAs per row
};

// index: 2 for bf16, plus 1 with a grammar mask
const void* colinfer_rows_kernel(int index);   // a CTA per row (sample_rows.cu)
int colinfer_rows_smem(int V, bool pen);
int colinfer_rows_threads();
const void* colinfer_few_kernel(int index);    // a cluster of CTAs per row (sample_few.cu)
int colinfer_few_smem(int V, bool pen);
int colinfer_few_threads();

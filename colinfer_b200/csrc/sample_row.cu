// sample_row.cu -- the fused kernel with one CTA of 768 threads per row and SM, for launches of more rows than SMs whose rows
// want more shared memory than half an SM has, and for long rows with histories (one_per_sm in sample.cu).
#define SMP_NAME smp_row
#define SMP_THREADS 768
#define SMP_CTAS 1
#define SMP_STAGES 2
#define SMP_LISTS 53248
#include "sample_kernel.cuh"

const void* colinfer_row_kernel(int index) {
    static const void* const k[4] = {(const void*)SMP_NAME::k_sample<false, 4, false>, (const void*)SMP_NAME::k_sample<false, 4, true>,
                                     (const void*)SMP_NAME::k_sample<false, 2, false>, (const void*)SMP_NAME::k_sample<false, 2, true>};
    return k[index];
}
int colinfer_row_smem(int V, bool pen) { return SMP_NAME::smem_bytes(V, pen); }
int colinfer_row_threads() { return SMP_NAME::NT; }

// sample_few.cu -- the fused kernel with a cluster of two or four CTAs per row, for launches of fewer rows than SMs: one CTA of 512
// threads per SM with four chunks under way per warp.  64 rows of 151,936 fp32 logits with mixed filters and histories 74 -> 61 us
// (with a CTA per row half of the SMs had none).
#define SMP_NAME smp_few
#define SMP_THREADS 512
#define SMP_CTAS 1
#define SMP_STAGES 4
#define SMP_LISTS 65536
#include "sample_kernel.cuh"

const void* colinfer_few_kernel(int index) {
    static const void* const k[4] = {(const void*)SMP_NAME::k_sample<true, 4, false>, (const void*)SMP_NAME::k_sample<true, 4, true>,
                                     (const void*)SMP_NAME::k_sample<true, 2, false>, (const void*)SMP_NAME::k_sample<true, 2, true>};
    return k[index];
}
int colinfer_few_smem(int V, bool pen) { return SMP_NAME::smem_bytes(V, pen); }
int colinfer_few_threads() { return SMP_NAME::NT; }

#ifdef COLINFER_PROFILE
extern "C" int colinfer_profile_read_few(unsigned long long* out16) {
    cudaDeviceSynchronize();
    int e = (int)cudaMemcpyFromSymbol(out16, SMP_NAME::g_prof, 128);
    unsigned long long z[16] = {};
    if (!e) e = (int)cudaMemcpyToSymbol(SMP_NAME::g_prof, z, 128);
    return e;
}
#endif

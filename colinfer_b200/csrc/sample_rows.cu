// sample_rows.cu -- the fused kernel with one CTA per row, for launches of more rows than SMs: two CTAs of 384 threads per SM, so
// that one of them reads while the other one is in its block-wide steps.  384 and not 512 threads: 80 registers each instead of 64,
// and 32 KB less of rings, which goes to the L1 (592 rows of 151,936 fp32 logits, greedy 78 -> 64 us, top_k 50 92 -> 78, top_p 208 -> 194).
// Two chunks under way per warp: with three a launch is no faster (98,304 bytes per SM are enough to keep HBM busy).
#define SMP_NAME smp_rows
#define SMP_THREADS 384
#define SMP_CTAS 2
#define SMP_STAGES 2
#define SMP_LISTS 26624
#include "sample_kernel.cuh"

const void* colinfer_rows_kernel(int index) {
    static const void* const k[4] = {(const void*)SMP_NAME::k_sample<false, 4, false>, (const void*)SMP_NAME::k_sample<false, 4, true>,
                                     (const void*)SMP_NAME::k_sample<false, 2, false>, (const void*)SMP_NAME::k_sample<false, 2, true>};
    return k[index];
}
int colinfer_rows_smem(int V, bool pen) { return SMP_NAME::smem_bytes(V, pen); }
int colinfer_rows_threads() { return SMP_NAME::NT; }

#ifdef COLINFER_PROFILE
extern "C" int colinfer_profile_read_rows(unsigned long long* out16) {
    cudaDeviceSynchronize();
    int e = (int)cudaMemcpyFromSymbol(out16, SMP_NAME::g_prof, 128);
    unsigned long long z[16] = {};
    if (!e) e = (int)cudaMemcpyToSymbol(SMP_NAME::g_prof, z, 128);
    return e;
}
#endif

// mass_probe.cu -- the arithmetic of the kept masses (csrc/common.cuh) over whole ranges of operands, for test_masses.py.
#include "../colinfer_b200/csrc/common.cuh"

// All 2^23 significands at 2^exp0 and 2^(exp0 + 1), sign by parity, divided by tc[blockIdx.y]: bad[0] counts quotients that are not
// __fdiv_rn's, bad[1] those more than one unit off.
__global__ void k_quotients(const float* tcs, int exp0, u64* bad) {
    const float tc = tcs[blockIdx.y], r = __frcp_rn(tc);
    u64 n = 0, far = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 24; i += gridDim.x * blockDim.x) {
        const float l = __uint_as_float(((uint32_t)(exp0 + 127) << 23) + i) * (i & 1u ? -1.0f : 1.0f);
        float a, b;
        up2(quotient2(pk2(l, l), pk2(-tc, -tc), pk2(r, r)), a, b);
        const float q = quotient(l, tc, r), want = __fdiv_rn(l, tc);
        const int d = max(abs(__float_as_int(q) - __float_as_int(want)), max(abs(__float_as_int(a) - __float_as_int(want)), abs(__float_as_int(b) - __float_as_int(want))));
        n += d != 0; far += d > 1;
    }
    if (n) atomicAdd(bad + 2 * blockIdx.y, n);
    if (far) atomicAdd(bad + 2 * blockIdx.y + 1, far);
}

// Masses of 2^20 logits between lmax - 24 tc and lmax: bad[blockIdx.y] counts pairs whose masses differ from MassFn's in either form.
__global__ void k_masses(const float* tcs, const float* lmax, u64* bad) {
    const float tc = tcs[blockIdx.y], L = lmax[blockIdx.y];
    MassFn f;
    f.init(tc, scale_logit(L, tc));
    Mass2 g;
    g.init(f);
    u64 n = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 1 << 20; i += gridDim.x * blockDim.x) {
        const float l0 = L - 24.0f * tc * ((float)i / 1048576.0f), l1 = L - 24.0f * tc * ((float)(1048576 - i) / 1048576.0f);
        uint32_t a, b;
        g.whole(l0, l1, -1e30f, a, b);
        u64 hi, w;
        g.parts(l0, l1, hi, w);
        float h0, h1, o0, o1;
        up2(hi, h0, h1); up2(add2(w, pk2(-12582912.0f, -12582912.0f)), o0, o1);
        const uint32_t c = (uint32_t)((double)h0 * 1073741824.0 + (double)o0), d = (uint32_t)((double)h1 * 1073741824.0 + (double)o1);
        n += a != f(l0) || b != f(l1) || c != f(l0) || d != f(l1);
    }
    if (n) atomicAdd(bad + blockIdx.y, n);
}

extern "C" int probe_quotients(const float* tcs, int n, int exp0, unsigned long long* bad) {
    k_quotients<<<dim3(64, n), 256>>>(tcs, exp0, bad);
    return (int)cudaDeviceSynchronize();
}
extern "C" int probe_masses(const float* tcs, const float* lmax, int n, unsigned long long* bad) {
    k_masses<<<dim3(16, n), 256>>>(tcs, lmax, bad);
    return (int)cudaDeviceSynchronize();
}

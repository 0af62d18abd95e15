// pll_check.cu -- the pilot PLL's step by itself, for its tests.
//
// Built into its own library (libgpudemod_check.so) so the product library's
// ABI stays the path's; only the tests load it.
#include <cuda_runtime.h>

#include "pll_step.cuh"

namespace {

using namespace gpud;

struct Loop {
    double alpha, beta, lpa, fmin, fmax, freq;
};

// One loop per CTA over its n pilot samples from phase 0, the frequency and
// zero I/Q; phase[t]: the loop's phase above the ramp after step t.
// `rounded`: the plain form of the step in the same types, its angle from the
// float64 phase at every step and atan2f.
__global__ void k_loop(const float *pilot, int n, Loop c, int rounded, double *phase) {
    if (threadIdx.x) return;
    const float *p = pilot + (size_t)blockIdx.x * n;
    double *out = phase + (size_t)blockIdx.x * n;
    PllK k;
    k.alpha = c.alpha;
    k.beta = c.beta;
    k.lpa = (float)c.lpa;
    k.dfmin = c.fmin - c.freq;
    k.dfmax = c.fmax - c.freq;
    k.q0 = 0;
    k.qf = (uint64_t)(c.freq / (2.0 * GPUD_PI) * 18446744073709551616.0);
    uint64_t q = 0;
    if (rounded) {
        double dphi = 0.0, df = 0.0;
        float I = 0.f, Q = 0.f;
        for (int t = 0; t < n; ++t, q += k.qf) {
            const float h = (float)(int32_t)(q >> 32) * 4.656612873077393e-10f + (float)(dphi * (1.0 / GPUD_PI));
            float sn, cs;
            __sincosf(h * 3.14159265358979f, &sn, &cs);
            I = fmaf(k.lpa, fmaf(p[t], cs, -I), I);
            Q = fmaf(k.lpa, fmaf(p[t], -sn, -Q), Q);
            const double e = (double)atan2f(Q, I);
            df = fmin(fmax(df + k.beta * e, k.dfmin), k.dfmax);
            dphi += df + k.alpha * e;
            out[t] = dphi;
        }
        return;
    }
    PllRun s = pll_begin(0.0, 0.0, 0.f, 0.f);
    for (int t = 0; t < n; ++t, q += k.qf) {
        if (t % kPllSeg == 0) s = pll_begin(s.dphi(), s.df, s.I, s.Q);
        PllEval o;
        pll_step<false>(q, s, p[t], k, o);
        out[t] = s.dphi();
    }
}

__global__ void k_atan2(const float *y, const float *x, int n, int plain, float *out) {
    const int i = blockIdx.x * blockDim.x + (int)threadIdx.x;
    if (i < n) out[i] = plain ? atan2f(y[i], x[i]) : pll_atan2(y[i], x[i], pll_scale(fmaxf(fabsf(y[i]), fabsf(x[i]))));
}

}  // namespace

extern "C" {

// Device pointers; returns 0 or a cudaError_t, after the kernel is done.
__attribute__((visibility("default"))) int gpud_check_pll_loop(const float *pilot, int n, int loops, double alpha,
                                                               double beta, double lpa, double fmin, double fmax,
                                                               double freq, int rounded, double *phase) {
    if (!pilot || !phase || n <= 0 || loops <= 0) return -1;
    k_loop<<<loops, 32>>>(pilot, n, Loop{alpha, beta, lpa, fmin, fmax, freq}, rounded, phase);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

__attribute__((visibility("default"))) int gpud_check_pll_atan2(const float *y, const float *x, int n, int plain,
                                                                float *out) {
    if (!y || !x || !out || n <= 0) return -1;
    k_atan2<<<(n + 255) / 256, 256>>>(y, x, n, plain, out);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

}  // extern "C"

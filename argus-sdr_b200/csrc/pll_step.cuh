// pll_step.cuh -- one step of the stereo pilot PLL, shared by the runner's
// kernels and the check library (pll_check.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#ifndef GPUD_PI
#define GPUD_PI 3.14159265358979323846
#endif

namespace gpud {

constexpr int kPllSeg = 16;  // steps per segment of the parallel solver, after which turns are taken out anew

struct PllK {
    double alpha, beta;
    float lpa;
    double dfmin, dfmax;  // frequency clamp as deviations from the block-start frequency
    uint64_t q0, qf;      // block-start phase and frequency in Q0.64 turns
};

// One loop step (recorder/streamer.go:1588-1613) in deviation form: the phase
// is phase0 + t*freq0 + dphi, the frequency freq0 + df (dphi, df float64); the
// ramp phase0 + t*freq0 is exact in Q0.64 turns, so the sin/cos argument needs
// no float64 range reduction.  The I/Q lowpass states are float32.  The serial
// loop and the Newton solver both use this step, so they iterate the same map.
//
// A trajectory is one chain of dependent operations, so a step costs its
// latency.  The angle of a step is the float64 phase of one step earlier, ramp
// included, rounded once, plus the last advance in float32 (the float64 phase
// advances beside it): the conversions of the float64 state are off the chain,
// which runs from the error to the next angle through two float32 multiply-adds.
// Cycles a step, and the rms error of a locked loop's phase against float64 over
// 200 to 312.5 kS/s (64 loops each; tests/test_gpu_pll_step.py):
//   angle from the float64 phase, atan2f        373   2.7e-8 to 3.1e-8 rad
//   angle summed in float32 over 16 steps       222   3.7e-8 to 4.8e-8
//   this                                        233   2.5e-8 to 2.8e-8
struct PllRun {
    double red, turns;  // phase above the ramp: what is left of it, and the whole turns taken out
    double prev, df;    // red one step earlier; frequency
    float I, Q;
    float adv;          // the last step's advance, red - prev
    __device__ __forceinline__ double dphi() const { return fma(turns, 2.0 * GPUD_PI, red); }
};

struct PllEval {
    float e;
    float ja, jb, jc, jd;   // phase row: d/dphase, d/dfreq, d/dI, d/dQ
    float ka, kb, kc, kd;   // freq row
    float iphi, qphi;       // I/Q rows' d/dphase (diagonals are 1 - lpa)
};

// The phase deviation of an unlocked loop grows to hundreds of radians: whole
// turns are taken out in float64 at the start of a segment, else the rounding of
// the angle (4e-6 rad at 50 rad) keeps the parallel solver above its tolerance.
__device__ __forceinline__ PllRun pll_begin(double dphi, double df, float I, float Q) {
    const double turns = rint(dphi * (1.0 / (2.0 * GPUD_PI)));
    const double red = fma(turns, -2.0 * GPUD_PI, dphi);
    return PllRun{red, turns, red, df, I, Q, 0.f};
}

__device__ __forceinline__ float pll_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// atan2 in float32 (within 1.8 ulp; atan2f: 2.0; tests/test_gpu_pll_step.py): the quotient t of the smaller
// by the larger magnitude from an approximate reciprocal and one residual
// correction, then t + t u P(u), u = t^2, P fitted to atan on [0, 1] by
// reweighted least squares (relative error 1.7e-8) and evaluated as short
// chains; octant and signs enter as a factor of t and an offset, both ready
// before the quotient is.  `scale` keeps the reciprocal's argument normal: 2^64
// as I and Q die out (and the offset above zero), 2^-64 above 2^60, so that all of
// float32's range is covered, as by atan2f.  It may come from any bound on the two.
__device__ __forceinline__ float pll_scale(float bound) { return bound > 1.1529215e18f ? 5.4210109e-20f : 1.8446744e19f; }

__device__ __forceinline__ float pll_atan2(float y, float x, float scale) {
    const float ax = fabsf(x), ay = fabsf(y);
    const float hi = fmaf(fmaxf(ax, ay), scale, 1e-30f), lo = fminf(ax, ay) * scale;
    const bool swap = ay > ax, neg = x < 0.f;
    // angle of (ax, ay): r or pi/2 - r; of (x, ay): that or pi minus it
    const float sg = copysignf(1.f, y), st = swap != neg ? -sg : sg;
    const float oh = swap ? 1.57079637f : neg ? 3.14159274f : 0.f;
    const float ol = swap ? -4.371139e-8f : neg ? -8.742278e-8f : 0.f;
    const float sh = sg * oh, sl = sg * ol;
    const float rc = pll_rcp(hi);
    float t = lo * rc;
    t = fmaf(fmaf(-hi, t, lo), rc, t);
    const float u = t * t, u2 = u * u, u4 = u2 * u2;
    const float p01 = fmaf(u, 0.19993773f, -0.33333153f), p23 = fmaf(u, 0.10666005f, -0.14211056f);
    const float p45 = fmaf(u, 0.04321186f, -0.07552214f), p67 = fmaf(u, 0.00292069f, -0.01636793f);
    const float pp = fmaf(u4, fmaf(u2, p67, p45), fmaf(u2, p23, p01));
    const float ts = t * st;
    return (fmaf(ts * u, pp, ts) + sl) + sh;
}

// q: the ramp phase phase0 + t*freq0 of step t in Q0.64 turns (callers carry
// it by adding k.qf per step: the same integer as k.q0 + t*k.qf); radians.
__device__ __forceinline__ float pll_ramp(uint64_t q) { return (float)(int32_t)(q >> 32) * 1.46291808e-9f; }

// The same in half-turns, of which float64 holds every bit: the top 32 bits go
// into the low word of 2^52 + 2^31 + n, so nothing is converted.
__device__ __forceinline__ double pll_ramp_half(uint64_t q) {
    const double m = __hiloint2double(0x43300000, (int)((uint32_t)(q >> 32) ^ 0x80000000u));
    return (m - 4503601774854144.0) * (1.0 / 2147483648.0);
}

template <bool kJac>
__device__ __forceinline__ void pll_step(uint64_t q, PllRun &s, float p, const PllK &k, PllEval &o) {
    float sn, cs;
    const float h = (float)fma(s.prev, 1.0 / GPUD_PI, pll_ramp_half(q));
    __sincosf(fmaf(h, 3.14159265358979f, s.adv), &sn, &cs);  // |angle| <= 2 pi and a step
    const float I1 = fmaf(k.lpa, fmaf(p, cs, -s.I), s.I);
    const float Q1 = fmaf(k.lpa, fmaf(p, -sn, -s.Q), s.Q);
    const float e = pll_atan2(Q1, I1, pll_scale(fmaxf(fmaxf(fabsf(s.I), fabsf(s.Q)), fabsf(p))));  // known before I1, Q1
    o.e = e;
    const float df1 = fminf(fmaxf(fmaf((float)k.beta, e, (float)s.df), (float)k.dfmin), (float)k.dfmax);
    s.adv = fmaf((float)k.alpha, e, df1);
    const double ed = (double)e;
    double d = fma(k.beta, ed, s.df);
    const bool clamped = d < k.dfmin || d > k.dfmax;
    d = d < k.dfmin ? k.dfmin : (d > k.dfmax ? k.dfmax : d);
    s.prev = s.red;
    s.red = fma(k.alpha, ed, s.red) + d;
    s.df = d;
    s.I = I1;
    s.Q = Q1;
    if (kJac) {
        // the Jacobian sets the convergence rate only, not the fixed point:
        // an approximate reciprocal is enough
        const float r2 = fmaf(I1, I1, Q1 * Q1);
        const float inv = r2 > 0.f ? __fdividef(1.f, r2) : 0.f;
        const float gI = -Q1 * inv, gQ = I1 * inv;
        const float dIphi = -k.lpa * p * sn;  // d/dphase of lpa*p*cos(phase)
        const float dQphi = -k.lpa * p * cs;  // d/dphase of -lpa*p*sin(phase)
        const float ePhi = fmaf(gI, dIphi, gQ * dQphi);
        const float om = 1.f - k.lpa;
        const float eI = gI * om, eQ = gQ * om;
        const float g = clamped ? 0.f : (float)k.beta, h = clamped ? 0.f : 1.f;
        const float ga = g + (float)k.alpha;
        o.ka = g * ePhi;
        o.kb = h;
        o.kc = g * eI;
        o.kd = g * eQ;
        o.ja = 1.f + ga * ePhi;
        o.jb = h;
        o.jc = ga * eI;
        o.jd = ga * eQ;
        o.iphi = dIphi;
        o.qphi = dQphi;
    }
}

// Twice the loop phase in half-turns, float32 (lr = bpf * 2 sin(pi h)); q is
// the ramp phase of the same step in Q0.64 turns.  (The whole turns taken out of
// the state are four half-turns each here: they drop out.)
__device__ __forceinline__ float pll_twice(uint64_t q, const PllRun &s) {
    const uint64_t q2 = 2 * q;
    return (float)(int32_t)(q2 >> 32) * 4.656612873077393e-10f + (float)(s.red * (2.0 / GPUD_PI));
}

}  // namespace gpud

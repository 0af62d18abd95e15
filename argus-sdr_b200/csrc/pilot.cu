// pilot.cu -- long-window stereo pilot detector on the device.
//
// classifier.StereoPilotPresent / estimateWFMPilot (internal/classifier/
// pll.go:75-131, 170-196): float64 FM discriminator of an FM-multiplex
// baseband, magnitude of its spectrum at 201 frequencies 19 kHz +- 1 kHz in
// 10 Hz steps (the reference runs one Goertzel recurrence per frequency), a
// stereo pilot when the largest magnitude exceeds `threshold` times the median
// (4.0 in the reference, SDRD_PILOT_RATIO overrides it there).
//
// Every analysis frequency f is a multiple of 10 Hz, so exp(-j 2 pi f i / fs)
// repeats with period P = fs / gcd(fs, 10) in i.  The discriminator output is
// folded modulo P once (y[m] = sum of d[m + pP]) and the 201 bins are direct
// float64 DFT sums of y over [0, P): the Goertzel magnitudes without the
// Goertzel recurrence's error growth.
//
// y is real, so a window of at least one period folds once more: with
// s[m] = y[m] + y[P-m] and d[m] = y[m] - y[P-m] the real part of a bin is the
// sum of s cos and its imaginary part the sum of d sin over m <= P/2.
//
// The bins of all stations of one rate are a matrix product, (201 x 2) x P/2
// twiddles times P/2 x stations samples, and float64 multiply-adds are its bound
// (40 stations at 312.5 kS/s: 0.25 G, 14 us at the chip's rate; 61 us measured,
// the staging and barriers of 8-term chunks and the prologue the rest).  k_pilot_bins
// gives every CTA a contiguous share of m for all bins and up to 40 stations:
// a thread keeps 7 bins x (cos, sin) x SPT stations in registers and reads 7
// twiddles and SPT samples from shared memory for 14 SPT multiply-adds.  The
// CTA copies its operands 16 (8 with many stations) m's ahead with asynchronous copies, the twiddles
// from a table of the P-th roots of unity (rotating 16 from one sincospi instead
// was as fast but doubled the error, 6e-15 -> 1e-14); periods beyond the table
// take a sincospi per term.  (One CTA per station and bin, each thread walking
// its own run of y: 1045 us.)  k_pilot_decide adds the CTAs' shares in
// order and takes the max / median decision.  The shares of one full pass are
// kept at a time; a call with more stations decides as it goes.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <numeric>
#include <tuple>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/gpudemod.h"
#include "gpud_internal.cuh"

extern "C" void gpud_count_launch(int n);

namespace {

constexpr int kBins = 201;
constexpr int kPilotThreads = 256;
constexpr int64_t kMaxTable = 1 << 20;  // roots-of-unity table entries (16 MiB)
constexpr int kBinsPT = 7;        // bins per thread: 4 warps x 8 lanes x 7 >= 201
constexpr int kStGroups = 8;      // station groups of a CTA: 2 warp rows x 4 lane groups
constexpr int kMaxSpt = 5;        // stations per thread
constexpr int kMaxSt = kStGroups * kMaxSpt;  // stations per pass
// The longer a chain of sums, the more of the station's programme, far above a
// bin, is rounded into it, so a thread's sums are taken into second ones every
// kChain terms.  With one chain per CTA the error was 1.04 (312.5 kS/s x 156250
// samples) and 1.7 times (320 kS/s x 30000) that of 256 chains per bin; now it is
// 0.5 times in both.  Up to three stations per thread the second sums are in
// registers, above in shared memory, with smaller chunks to make room; the order
// of sums is the same, so a station's result does not depend on how many others
// there are.
constexpr int kChain = 32;
__host__ __device__ constexpr bool second_in_registers(int spt) { return spt <= 3; }
__host__ __device__ constexpr int chunk_of(int spt) { return second_in_registers(spt) ? 16 : 8; }  // m's staged at a time
constexpr int kShareMin = 32;  // fewest terms of a CTA's share

struct PilotJob {
    const float2 *iq;  // first sample of the analysed window
    int32_t nd;        // discriminator samples (window length - 1)
    int32_t period;    // P = fs / gcd(fs, 10)
    int32_t folded;    // terms of a bin: P/2 + 1 pairs (s, d) of a whole period, else the nd samples
    int32_t paired;
    int32_t nshare;    // CTAs of its pass
    int32_t column;    // its column in the pass
    int32_t ncol;      // columns of the pass
    int32_t fstep;     // 10 / gcd(fs, 10)
    int32_t span;      // terms of its pass: the longest folded of its stations
    int64_t part_off;  // its pass's partial sums
    int64_t y_off;     // offset of this job's folded vector
};

// Stations of one rate whose bins one launch computes: jobs first..first+count-1.
struct PilotPass {
    int first, count, period, folded, paired, fstep, spt;
    int64_t part_off;  // double2 offset of its partial sums [share][column][bin]
    int nshare;
    bool each;         // few terms: k_pilot_bins_each
};

// fmDemod (pll.go:170-183): float64 products of the float32 samples, atan2.
__device__ __forceinline__ double pilot_disc(const float2 *iq, int i) {
    const float2 p = iq[i], c = iq[i + 1];
    const double num = (double)p.x * (double)c.y - (double)p.y * (double)c.x;
    const double den = (double)p.x * (double)c.x + (double)p.y * (double)c.y;
    return atan2(num, den);
}

__device__ __forceinline__ double pilot_folded(const PilotJob &jb, int m) {
    double acc = 0.0;
    for (int i = m; i < jb.nd; i += jb.period) acc += pilot_disc(jb.iq, i);
    return acc;
}

__global__ void __launch_bounds__(kPilotThreads)
k_pilot_fold(const PilotJob *__restrict__ jobs, double *__restrict__ y) {
    const PilotJob jb = jobs[blockIdx.y];
    for (int m = blockIdx.x * kPilotThreads + threadIdx.x; m < jb.folded; m += gridDim.x * kPilotThreads) {
        const double a = pilot_folded(jb, m);
        if (!jb.paired) {
            y[jb.y_off + m] = a;
        } else {
            const int o = jb.period - m;
            const double b = m > 0 && o != m ? pilot_folded(jb, o) : 0.0;
            reinterpret_cast<double2 *>(y + jb.y_off)[m] = make_double2(a + b, a - b);
        }
    }
}

// Shared memory of a CTA, both halves of a double buffer: twiddles | samples.
template <int CH>
struct PilotStage {
    double2 w[2][CH][32 * kBinsPT];
    double2 y[2][CH][kMaxSt];  // (s, d); the first alone where not paired
};

template <int SPT>
constexpr int pilot_smem() {
    return (int)sizeof(PilotStage<chunk_of(SPT)>) +
           (second_in_registers(SPT) ? 0 : kBinsPT * SPT * kPilotThreads * (int)sizeof(double2));
}
static_assert(pilot_smem<kMaxSpt>() <= 227 * 1024, "shared memory of a CTA");

// tab[a] = exp(j 2 pi a / P), a < P
__global__ void k_pilot_table(int P, double2 *__restrict__ tab) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < P; a += gridDim.x * blockDim.x) {
        double s, c;
        sincospi(2.0 * (double)a / (double)P, &s, &c);
        tab[a] = make_double2(c, s);
    }
}

// Asynchronous copy of 8 or 16 bytes global -> shared, zeros where !ok.
template <int BYTES>
__device__ __forceinline__ void copy_async(void *dst, const void *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(gpud::smem_u32(dst)), "l"(src), "n"(BYTES),
                 "r"(ok ? BYTES : 0)
                 : "memory");
}

__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Partial DFT sums of a pass: CTA b takes m in its share of [0, folded), and
// writes re + j im of every (bin, station) to part[b][station][bin].  While the
// warps multiply one chunk the copies of the next are under way: one barrier a
// chunk.
template <int SPT, bool PAIRED>
__global__ void __launch_bounds__(kPilotThreads)
k_pilot_bins(const PilotJob *__restrict__ jobs, int count, int P, int folded, int fstep, const double *__restrict__ y,
             const double2 *__restrict__ tab, double2 *__restrict__ part) {
    constexpr int NS = kStGroups * SPT, kChunk = chunk_of(SPT);
    constexpr int NL = (kChunk * NS + kPilotThreads - 1) / kPilotThreads;  // samples a thread fetches
    extern __shared__ __align__(16) unsigned char psm[];
    PilotStage<kChunk> &sm = *reinterpret_cast<PilotStage<kChunk> *>(psm);
    const int t = (int)threadIdx.x, lane = t & 31, warp = t >> 5;
    // a warp takes 8 bins x 4 station groups at a time: both operands are
    // broadcast to the lanes that share them
    const int bin0 = (warp & 3) * (8 * kBinsPT) + (lane & 7), grp = (warp >> 2) * 4 + (lane >> 3);
    const int m0 = (int)((int64_t)folded * blockIdx.x / gridDim.x);
    const int m1 = (int)((int64_t)folded * (blockIdx.x + 1) / gridDim.x);
    // the chain under way, and the sums of the chains before it
    constexpr bool kRegs = second_in_registers(SPT);
    double re[kBinsPT][SPT], im[kBinsPT][SPT];
    double2 own[kRegs ? kBinsPT : 1][SPT];
    double2 *far = reinterpret_cast<double2 *>(psm + sizeof(PilotStage<kChunk>)) + t;
    auto second = [&](int b, int s) -> double2 & {
        if constexpr (kRegs) return own[b][s];
        else return far[(b * SPT + s) * kPilotThreads];
    };
#pragma unroll
    for (int b = 0; b < kBinsPT; ++b)
#pragma unroll
        for (int s = 0; s < SPT; ++s) {
            re[b][s] = im[b][s] = 0.0;
            second(b, s) = make_double2(0.0, 0.0);
        }
    auto chain_end = [&]() {
#pragma unroll
        for (int b = 0; b < kBinsPT; ++b)
#pragma unroll
            for (int s = 0; s < SPT; ++s) {
                double2 v = second(b, s);
                v.x += re[b][s];
                v.y += im[b][s];
                second(b, s) = v;
                re[b][s] = im[b][s] = 0.0;
            }
    };
    // thread t's twiddles: bin t; f / gcd(fs, 10) = (1800 + bin) * fstep
    const int64_t fq = ((int64_t)(1800 + t) * fstep) % P;
    // its samples of a chunk: consecutive threads on consecutive samples of a station
    const double *src[NL];
    int end[NL];
#pragma unroll
    for (int u = 0; u < NL; ++u) {
        const int st = (t + u * kPilotThreads) / kChunk;
        src[u] = st < count ? y + jobs[st].y_off : y;
        end[u] = st < count ? min(m1, jobs[st].folded) : 0;
    }
    auto stage = [&](int buf, int mc) {
#pragma unroll
        for (int u = 0; u < NL; ++u) {
            const int i = t + u * kPilotThreads, m = mc + i % kChunk;
            if (i >= kChunk * NS) continue;
            const int k = min(m, m1 - 1);
            if (PAIRED)
                copy_async<16>(&sm.y[buf][i % kChunk][i / kChunk], src[u] + 2 * (int64_t)k, m < end[u]);
            else
                copy_async<8>(&sm.y[buf][i % kChunk][i / kChunk], src[u] + k, m < end[u]);
        }
        if (t < kBins) {
            int64_t a = (fq * (int64_t)mc) % P;
#pragma unroll 4
            for (int i = 0; i < kChunk; ++i) {
                if (tab) {
                    copy_async<16>(&sm.w[buf][i][t], tab + a, true);
                } else {
                    double s, c;
                    sincospi(2.0 * (double)a / (double)P, &s, &c);
                    sm.w[buf][i][t] = make_double2(c, s);
                }
                a += fq;
                if (a >= P) a -= P;
            }
        }
    };
    if (m0 < m1) stage(0, m0);
    copies_wait();
    __syncthreads();
    int buf = 0;
    for (int mc = m0; mc < m1; mc += kChunk, buf ^= 1) {
        if (mc != m0 && (mc - m0) % kChain == 0) chain_end();
        if (mc + kChunk < m1) stage(buf ^ 1, mc + kChunk);
        for (int i = 0; i < kChunk; ++i) {  // samples past the share are zero
            double2 v[SPT];
#pragma unroll
            for (int s = 0; s < SPT; ++s) {
                v[s] = sm.y[buf][i][grp * SPT + s];
                if (!PAIRED) v[s].y = v[s].x;
            }
#pragma unroll
            for (int b = 0; b < kBinsPT; ++b) {
                const double2 w = sm.w[buf][i][bin0 + 8 * b];
#pragma unroll
                for (int s = 0; s < SPT; ++s) {
                    re[b][s] = fma(v[s].x, w.x, re[b][s]);
                    im[b][s] = fma(v[s].y, w.y, im[b][s]);
                }
            }
        }
        copies_wait();
        __syncthreads();
    }
    chain_end();
    double2 *out = part + (int64_t)blockIdx.x * kBins * count;
#pragma unroll
    for (int b = 0; b < kBinsPT; ++b) {
        const int bin = bin0 + 8 * b;
#pragma unroll
        for (int s = 0; s < SPT; ++s) {
            const int st = grp * SPT + s;
            if (bin < kBins && st < count) out[st * kBins + bin] = second(b, s);
        }
    }
}

// The sums of a few stations: one CTA per (share, station), a thread per bin, any
// rates together; twiddles from the table for the rate that it holds, else computed.
// The shares, the chains and so the bits are those of k_pilot_bins, which takes 14 us
// and about 2.4 for every 16 terms of a share whatever it is given (its 100 KB and
// more of shared memory, one chunk ahead), and a launch and a table a rate; here a
// thousand station-terms cost 0.6 us, more than there from the third station on.
// Calls at 312.5 kS/s, this and that: one station of 23000 samples 68 and 89 us, two
// 82 and 91, three 97 and 95, five of 4000 75 and 65, eight of 1000 64 and 69.
constexpr int kEachStations = 2;
constexpr int kEachTerms = 12288;  // station-terms that more of them may have

__global__ void __launch_bounds__(kPilotThreads)
k_pilot_bins_each(const PilotJob *__restrict__ jobs, const double *__restrict__ y, const double2 *__restrict__ tab,
                  int tab_period, double2 *__restrict__ part) {
    const PilotJob jb = jobs[blockIdx.y];
    const int share = blockIdx.x, bin = (int)threadIdx.x, P = jb.period;
    if (share >= jb.nshare || bin >= kBins) return;
    const int64_t fq = ((int64_t)(1800 + bin) * jb.fstep) % P;
    const int m0 = (int)((int64_t)jb.span * share / jb.nshare);
    const int m1 = min(jb.folded, (int)((int64_t)jb.span * (share + 1) / jb.nshare));
    const double *ym = y + jb.y_off;
    double2 all = make_double2(0.0, 0.0);
    const unsigned up = (unsigned)P, uf = (unsigned)fq;  // both below 2^31
    unsigned a = (unsigned)((fq * (int64_t)m0) % P);
    for (int mc = m0; mc < m1; mc += kChain) {
        const int me = min(m1, mc + kChain);
        double2 v = make_double2(0.0, 0.0);
        auto term = [&](int m, const double2 w) {
            v.x = fma(ym[jb.paired ? 2 * m : m], w.x, v.x);
            v.y = fma(ym[jb.paired ? 2 * m + 1 : m], w.y, v.y);
        };
        auto next = [&]() {
            const unsigned at = a;
            a += uf;
            if (a >= up) a -= up;
            return at;
        };
        int m = mc;
        if (P == tab_period) {
            for (; m + 8 <= me; m += 8) {  // eight gathers in flight
                double2 w[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) w[u] = __ldg(tab + next());
#pragma unroll
                for (int u = 0; u < 8; ++u) term(m + u, w[u]);
            }
            for (; m < me; ++m) term(m, __ldg(tab + next()));
        } else {
#pragma unroll 4
            for (; m < me; ++m) {
                double s, c;
                sincospi(2.0 * (double)next() / (double)P, &s, &c);
                term(m, make_double2(c, s));
            }
        }
        all.x += v.x;
        all.y += v.y;
    }
    part[jb.part_off + ((int64_t)share * jb.ncol + jb.column) * kBins + bin] = all;
}

// max (first occurrence, as the reference's strict '>' scan from 0) and the
// median (element 100 of the sorted 201) of each job's magnitudes
// s += v with the rounding error kept in e (Knuth's two-sum): the shares of a
// bin far below the station's programme are large and cancel.
__device__ __forceinline__ void add_exact(double &s, double &e, double v) {
    const double t = s + v, z = t - s;
    e += (s - (t - z)) + (v - z);
    s = t;
}

constexpr int kDecideParts = 4;  // thread groups that add a bin's shares and rank it

__global__ void __launch_bounds__(kDecideParts * kPilotThreads)
k_pilot_decide(const PilotJob *__restrict__ jobs, const double2 *__restrict__ part, double threshold,
               gpud_pilot_result *__restrict__ out) {
    __shared__ double2 s_p[kDecideParts][kBins];
    __shared__ double s_m[kBins], s_med;
    __shared__ unsigned long long s_best;
    __shared__ int s_rank[kBins], s_bin;
    const PilotJob jb = jobs[blockIdx.x];
    const int i = threadIdx.x % kPilotThreads, q = threadIdx.x / kPilotThreads;
    if (threadIdx.x == 0) {
        s_best = 0ull;
        s_bin = kBins;
    }
    if (i < kBins) {
        const double2 *p = part + jb.part_off + (int64_t)jb.column * kBins + i;
        double re = 0.0, im = 0.0, er = 0.0, ei = 0.0;
        for (int k0 = q; k0 < jb.nshare; k0 += 8 * kDecideParts) {  // eight loads in flight
            double2 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int k = k0 + u * kDecideParts;
                v[u] = k < jb.nshare ? p[(int64_t)k * kBins * jb.ncol] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (k0 + u * kDecideParts >= jb.nshare) break;
                add_exact(re, er, v[u].x);
                add_exact(im, ei, v[u].y);
            }
        }
        s_p[q][i] = make_double2(re + er, im + ei);
    }
    __syncthreads();
    if (q == 0 && i < kBins) {
        double re = 0.0, im = 0.0, er = 0.0, ei = 0.0;
        for (int k = 0; k < kDecideParts; ++k) {
            add_exact(re, er, s_p[k][i].x);
            add_exact(im, ei, s_p[k][i].y);
        }
        re += er;
        im += ei;
        s_m[i] = sqrt(re * re + im * im);
        s_rank[i] = 0;
    }
    __syncthreads();
    if (i < kBins) {
        const double mi = s_m[i];
        int rank = 0;
        for (int j = q; j < kBins; j += kDecideParts) rank += (s_m[j] < mi) || (s_m[j] == mi && j < i);
        atomicAdd(&s_rank[i], rank);
        // magnitudes are not negative: they order as their bits
        if (q == 0 && mi > 0.0) atomicMax(&s_best, (unsigned long long)__double_as_longlong(mi));
    }
    __syncthreads();
    if (q == 0 && i < kBins) {
        if (s_rank[i] == kBins / 2) s_med = s_m[i];
        if (s_m[i] > 0.0 && (unsigned long long)__double_as_longlong(s_m[i]) == s_best) atomicMin(&s_bin, i);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double best = __longlong_as_double((long long)s_best), med = s_med;
        gpud_pilot_result r{};
        r.best_bin = s_bin == kBins ? 100 : s_bin;
        r.best_hz = 18000.0 + 10.0 * (double)r.best_bin;
        r.median = med;
        r.ratio = med > 0 ? best / med : 0.0;
        r.present = (med > 0 && r.ratio > threshold) ? 1 : 0;
        out[blockIdx.x] = r;
    }
}

template <int SPT, bool PAIRED>
cudaError_t launch_pilot_bins_as(const PilotPass &ps, cudaStream_t s, const PilotJob *jobs, const double *y,
                                 const double2 *tab, double2 *part) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = gpud::smem_optin_once(optin, (const void *)k_pilot_bins<SPT, PAIRED>, pilot_smem<SPT>());
    if (e != cudaSuccess) return e;
    k_pilot_bins<SPT, PAIRED><<<ps.nshare, kPilotThreads, pilot_smem<SPT>(), s>>>(
        jobs + ps.first, ps.count, ps.period, ps.folded, ps.fstep, y, tab, part + ps.part_off);
    return cudaGetLastError();
}

cudaError_t launch_pilot_bins(const PilotPass &ps, cudaStream_t s, const PilotJob *jobs, const double *y,
                              const double2 *tab, double2 *part) {
    switch (2 * ps.spt + ps.paired) {
#define GPUD_CASE(N)                                                              \
    case 2 * N: return launch_pilot_bins_as<N, false>(ps, s, jobs, y, tab, part); \
    case 2 * N + 1: return launch_pilot_bins_as<N, true>(ps, s, jobs, y, tab, part);
        GPUD_CASE(1) GPUD_CASE(2) GPUD_CASE(3) GPUD_CASE(4) GPUD_CASE(5)
#undef GPUD_CASE
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

struct gpud_pilot {
    int max_jobs = 0, max_samples = 0, num_sms = 148;
    double *d_y = nullptr;
    double2 *d_part = nullptr;  // partial sums [share][column][bin] of the passes between two decisions
    int64_t part_cap = 0;       // its entries: one full pass (passes of one call take turns in it)
    double2 *d_tab = nullptr;   // roots of unity of the last pass's period
    int tab_period = 0;
    PilotJob *d_jobs = nullptr;
    gpud_pilot_result *d_res = nullptr;
    std::vector<PilotJob> jobs;
    std::vector<int> fstep;        // per device job
    std::vector<PilotPass> passes;
    std::vector<int> job_of;  // job index -> index into the device list (-1: no decision possible)
};

extern "C" {

// Folded values of a job: P/2 + 1 pairs with P below the window length, or the
// window's samples; an even number, so that the pairs are aligned.
static int64_t pilot_row(int max_samples) { return ((int64_t)max_samples + 3) & ~(int64_t)1; }

// Shares of a pass: CTAs that split its terms.
static int pilot_shares(const gpud_pilot *p, int folded) {
    return std::max(1, std::min(p->num_sms, folded / kShareMin));
}

GPUD_API int GPUD_CALL gpud_pilot_create(int max_jobs, int max_samples, gpud_pilot **out) {
    if (!out || max_jobs <= 0 || max_samples <= 1) return GPUD_E_ARG;
    auto *p = new gpud_pilot();
    p->max_jobs = max_jobs;
    p->max_samples = max_samples;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0)
        p->num_sms = sms;
    // a pass has at most kMaxSt columns and no more terms than a window has samples
    p->part_cap = (int64_t)std::min(max_jobs, kMaxSt) * kBins * pilot_shares(p, max_samples);
    bool ok = cudaMalloc((void **)&p->d_y, sizeof(double) * (size_t)max_jobs * (size_t)pilot_row(max_samples)) == cudaSuccess &&
              cudaMalloc((void **)&p->d_part, sizeof(double2) * (size_t)p->part_cap) == cudaSuccess &&
              cudaMalloc((void **)&p->d_tab, sizeof(double2) * (size_t)kMaxTable) == cudaSuccess &&
              cudaMalloc((void **)&p->d_jobs, sizeof(PilotJob) * (size_t)max_jobs) == cudaSuccess &&
              cudaMalloc((void **)&p->d_res, sizeof(gpud_pilot_result) * (size_t)max_jobs) == cudaSuccess;
    if (!ok) {
        gpud_pilot_destroy(p);
        return GPUD_E_CUDA;
    }
    *out = p;
    return 0;
}

GPUD_API int GPUD_CALL gpud_pilot_destroy(gpud_pilot *p) {
    if (!p) return 0;
    cudaFree(p->d_y);
    cudaFree(p->d_part);
    cudaFree(p->d_tab);
    cudaFree(p->d_jobs);
    cudaFree(p->d_res);
    delete p;
    return 0;
}

GPUD_API int GPUD_CALL gpud_pilot_run(gpud_pilot *p, const gpud_pilot_job *jobs, int count, double threshold,
                                      gpud_stream_handle stream, gpud_pilot_result *results) {
    if (!p || count < 0 || count > p->max_jobs || (count > 0 && (!jobs || !results))) return GPUD_E_ARG;
    if (threshold <= 0) threshold = 4.0;
    cudaStream_t s = (cudaStream_t)stream;
    p->jobs.clear();
    p->fstep.clear();
    p->job_of.assign((size_t)count, -1);
    for (int j = 0; j < count; ++j) {
        const gpud_pilot_job &q = jobs[j];
        results[j] = gpud_pilot_result{};
        results[j].best_hz = 19000.0;
        results[j].best_bin = 100;
        int n = q.n, start = 0;
        if (!q.iq || n < 0) return GPUD_E_ARG;
        if (q.window) {  // StereoPilotPresent: the last sample_rate/2 samples
            const int mx = q.sample_rate / 2;
            if (mx > 0 && n > mx) {
                start = n - mx;
                n = mx;
            }
        }
        if (n > p->max_samples) return GPUD_E_ARG;
        if (q.sample_rate < 40000 || n < 2) continue;  // the reference returns unlocked
        PilotJob jb{};
        const int g = std::gcd(q.sample_rate, 10);
        jb.iq = reinterpret_cast<const float2 *>(q.iq) + start;
        jb.nd = n - 1;
        jb.period = q.sample_rate / g;
        jb.paired = jb.nd >= jb.period ? 1 : 0;
        jb.folded = jb.paired ? jb.period / 2 + 1 : jb.nd;
        jb.fstep = 10 / g;
        jb.y_off = (int64_t)p->jobs.size() * pilot_row(p->max_samples);
        p->job_of[(size_t)j] = (int)p->jobs.size();
        p->jobs.push_back(jb);
        p->fstep.push_back(10 / g);
    }
    const int nj = (int)p->jobs.size();
    if (nj == 0) return 0;
    // passes: the jobs of one rate (period, step, paired or not), at most kMaxSt
    // of them at a time, side by side on the device
    std::vector<int> order((size_t)nj);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        const PilotJob &x = p->jobs[(size_t)a], &z = p->jobs[(size_t)b];
        return std::make_tuple(x.period, p->fstep[(size_t)a], x.paired) <
               std::make_tuple(z.period, p->fstep[(size_t)b], z.paired);
    });
    std::vector<PilotJob> sorted((size_t)nj);
    std::vector<int> at((size_t)nj);
    for (int k = 0; k < nj; ++k) {
        sorted[(size_t)k] = p->jobs[(size_t)order[(size_t)k]];
        at[(size_t)order[(size_t)k]] = k;
    }
    // Partial sums stand side by side while they fit the workspace; a pass that
    // finds no room starts a new round, after the decisions on the one before.
    p->passes.clear();
    int64_t part = 0;
    for (int k = 0; k < nj;) {
        PilotPass ps{};
        ps.first = k;
        ps.period = sorted[(size_t)k].period;
        ps.fstep = p->fstep[(size_t)order[(size_t)k]];
        ps.paired = sorted[(size_t)k].paired;
        while (k < nj && ps.count < kMaxSt && sorted[(size_t)k].period == ps.period &&
               sorted[(size_t)k].paired == ps.paired &&
               p->fstep[(size_t)order[(size_t)k]] == ps.fstep) {
            ps.folded = std::max(ps.folded, sorted[(size_t)k].folded);
            ++ps.count;
            ++k;
        }
        ps.spt = (ps.count + kStGroups - 1) / kStGroups;
        ps.each = ps.count <= kEachStations || (int64_t)ps.count * ps.folded <= kEachTerms;
        ps.nshare = pilot_shares(p, ps.folded);
        const int64_t need = (int64_t)ps.nshare * kBins * ps.count;
        if (part + need > p->part_cap) part = 0;
        ps.part_off = part;
        for (int c = 0; c < ps.count; ++c) {
            PilotJob &jb = sorted[(size_t)(ps.first + c)];
            jb.nshare = ps.nshare;
            jb.span = ps.folded;
            jb.column = c;
            jb.ncol = ps.count;
            jb.part_off = part;
        }
        part += need;
        p->passes.push_back(ps);
    }
    if (cudaMemcpyAsync(p->d_jobs, sorted.data(), sizeof(PilotJob) * (size_t)nj, cudaMemcpyHostToDevice, s) !=
        cudaSuccess)
        return GPUD_E_CUDA;
    int maxf = 0;
    for (auto &jb : sorted) maxf = std::max(maxf, jb.folded);
    dim3 gf((unsigned)std::min(1024, (maxf + kPilotThreads - 1) / kPilotThreads), (unsigned)nj);
    k_pilot_fold<<<gf, kPilotThreads, 0, s>>>(p->d_jobs, p->d_y);
    int decided = 0, launches = 1;  // jobs decided; kernels
    for (size_t k = 0; k < p->passes.size(); ++k) {
        PilotPass ps = p->passes[k];
        bool table = ps.period <= kMaxTable, have = ps.period == p->tab_period;
        if (ps.each)  // with the next rates of a station or two, or of short windows
            for (; k + 1 < p->passes.size() && p->passes[k + 1].each && p->passes[k + 1].part_off != 0; ++k) {
                ps.count += p->passes[k + 1].count;
                ps.nshare = std::max(ps.nshare, p->passes[k + 1].nshare);
                have = have || p->passes[k + 1].period == p->tab_period;
            }
        if (table && !have) {  // the pass before has read the old one (stream order)
            k_pilot_table<<<std::min(1024, (ps.period + 255) / 256), 256, 0, s>>>(ps.period, p->d_tab);
            launches++;
            p->tab_period = ps.period;
        }
        if (ps.each)
            k_pilot_bins_each<<<dim3((unsigned)ps.nshare, (unsigned)ps.count), kPilotThreads, 0, s>>>(
                p->d_jobs + ps.first, p->d_y, p->d_tab, p->tab_period, p->d_part);
        else if (launch_pilot_bins(ps, s, p->d_jobs, p->d_y, table ? p->d_tab : nullptr, p->d_part) !=
                 cudaSuccess)
            return GPUD_E_CUDA;
        launches++;
        if (k + 1 < p->passes.size() && p->passes[k + 1].part_off != 0) continue;
        const int end = ps.first + ps.count;
        k_pilot_decide<<<end - decided, kDecideParts * kPilotThreads, 0, s>>>(p->d_jobs + decided, p->d_part, threshold,
                                                                              p->d_res + decided);
        launches++;
        decided = end;
    }
    if (cudaGetLastError() != cudaSuccess) return GPUD_E_CUDA;
    gpud_count_launch(launches);
    std::vector<gpud_pilot_result> tmp((size_t)nj);
    if (cudaMemcpyAsync(tmp.data(), p->d_res, sizeof(gpud_pilot_result) * (size_t)nj, cudaMemcpyDeviceToHost, s) !=
            cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return GPUD_E_CUDA;
    for (int j = 0; j < count; ++j)
        if (p->job_of[(size_t)j] >= 0) results[j] = tmp[(size_t)at[(size_t)p->job_of[(size_t)j]]];
    return 0;
}

}  // extern "C"

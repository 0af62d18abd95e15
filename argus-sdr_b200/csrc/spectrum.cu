// spectrum.cu -- surveillance spectrum on the device (internal/fft/fft.go:
// 19-55 Spectrum, welch.go:15-66 WelchPSD; cmd/sdrd/pipeline_runtime.go:
// 294-341 calls them, or cuFFT, per frame).
//
// The reference transforms in complex128 (gonum) on the CPU, or in complex64
// through cuFFT.  Here one CTA transforms one segment entirely in shared
// memory in float64: the windowed samples are loaded in bit-reversed order,
// then log2(N) radix-2 butterfly stages, three at a time on eight values in
// registers (one barrier instead of three), with twiddles exp(-j 2 pi k / m)
// from a table of sincospi of exact rational arguments, made with the plan.
// (A sincospi per butterfly and a barrier per stage: 35 us for 16 segments of
// 4096, now 14; what is left is the float64 window, magnitude and the latency of
// four passes on one CTA per segment.)  Welch segments write |X|^2 / N^2 per
// bin; a second kernel adds them in segment order (deterministic) and writes
// the fftshifted dB spectrum.  Power-of-two sizes up to 8192 (128 KB of
// float64 pairs in shared memory).
#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/gpudemod.h"
#include "gpud_internal.cuh"

extern "C" void gpud_count_launch(int n);

namespace {

constexpr int kSpecThreads = 512;
constexpr int kMaxFft = 8192;

__device__ __forceinline__ unsigned bitrev(unsigned x, int bits) { return __brev(x) >> (32 - bits); }

// tab[j] = exp(-j 2 pi j / kMaxFft), j < kMaxFft / 2: the twiddle k of a stage
// of span m is entry k * (kMaxFft / m).
__global__ void k_spectrum_twiddles(double2 *__restrict__ tab) {
    const int j = blockIdx.x * blockDim.x + (int)threadIdx.x;
    if (j >= kMaxFft / 2) return;
    double sn, cs;
    sincospi(-2.0 * (double)j / (double)kMaxFft, &sn, &cs);
    tab[j] = make_double2(cs, sn);
}

// Value i sits at i + i/8: values a power of two apart fall in different banks.
__host__ __device__ constexpr int slot(int i) { return i + (i >> 3); }

__device__ __forceinline__ void butterfly(double2 &a, double2 &c, const double2 w) {
    const double tr = c.x * w.x - c.y * w.y, ti = c.x * w.y + c.y * w.x;
    c = make_double2(a.x - tr, a.y - ti);
    a = make_double2(a.x + tr, a.y + ti);
}

// Stages s+1 .. s+K (spans 2^(s+1) .. 2^(s+K)) of the transform in sx: a thread
// holds the 2^K values 2^s apart that those stages combine among themselves.
template <int K>
__device__ __forceinline__ void fft_stages(double2 *sx, int N, int s, const double2 *__restrict__ tab) {
    constexpr int R = 1 << K;
    const int half = 1 << s;  // distance of the first of the stages
    for (int b = threadIdx.x; b < N / R; b += kSpecThreads) {
        const int k0 = b & (half - 1), i0 = ((b >> s) << (s + K)) + k0;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = sx[slot(i0 + r * half)];
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int step = kMaxFft >> (s + q + 1);  // table step of span 2^(s+q+1)
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (!(r & (1 << q))) butterfly(v[r], v[r | (1 << q)], __ldg(tab + (k0 + (r & ((1 << q) - 1)) * half) * step));
        }
#pragma unroll
        for (int r = 0; r < R; ++r) sx[slot(i0 + r * half)] = v[r];
    }
    __syncthreads();
}

// One segment: x[start + i] * w[i] (Hann when hann != 0), i < N, into |X_k|.
// pow_out[k] = |X_k|^2 / N^2 (welch) or |X_k| / N (single).
__global__ void __launch_bounds__(kSpecThreads)
k_spectrum_seg(const float2 *__restrict__ iq, int N, int log2n, int step, int hann, int welch,
               const double2 *__restrict__ tab, double *__restrict__ pow_out) {
    extern __shared__ double2 sx[];
    const int seg = blockIdx.x;
    const int64_t start = (int64_t)seg * step;
    for (int i = threadIdx.x; i < N; i += kSpecThreads) {
        const float2 v = iq[start + i];
        double w = 1.0;
        // fftutil.Hann: 0.5 (1 - cos(2 pi i / (n-1)))
        if (hann && N > 1) w = 0.5 * (1.0 - cospi(2.0 * (double)i / (double)(N - 1)));
        sx[slot((int)bitrev((unsigned)i, log2n))] = make_double2((double)v.x * w, (double)v.y * w);
    }
    __syncthreads();
    int s = 0;
    for (; s + 3 <= log2n; s += 3) fft_stages<3>(sx, N, s, tab);
    if (log2n - s == 2) fft_stages<2>(sx, N, s, tab);
    if (log2n - s == 1) fft_stages<1>(sx, N, s, tab);
    const double invN = 1.0 / (double)N;
    for (int k = threadIdx.x; k < N; k += kSpecThreads) {
        const double mag = hypot(sx[slot(k)].x, sx[slot(k)].y) * invN;
        pow_out[(int64_t)seg * N + k] = welch ? mag * mag : mag;
    }
}

// dB and fftshift: Welch 10 log10(mean power + 1e-24) (welch.go:57-63),
// single 20 log10(|X|/N + 1e-12) (fft.go:42-50); output bin i is bin
// (i + N/2) mod N.
__global__ void __launch_bounds__(256)
k_spectrum_db(const double *__restrict__ pw, int N, int segs, int welch, double *__restrict__ out) {
    const int i = blockIdx.x * 256 + (int)threadIdx.x;
    if (i >= N) return;
    const int idx = (i + N / 2) % N;
    if (welch) {
        double acc = 0.0;
        for (int s = 0; s < segs; ++s) acc += pw[(int64_t)s * N + idx];
        out[i] = 10.0 * log10(acc / (double)segs + 1e-24);
    } else {
        out[i] = 20.0 * log10(pw[idx] + 1e-12);
    }
}

int ilog2_exact(int n) {
    if (n <= 0 || (n & (n - 1))) return -1;
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
}

}  // namespace

struct gpud_spectrum {
    int max_fft = 0, max_segments = 0;
    double *d_pow = nullptr;  // max_segments x max_fft
    double *d_db = nullptr;   // max_fft
    double2 *d_tab = nullptr; // twiddles
};

extern "C" {

GPUD_API int GPUD_CALL gpud_spectrum_destroy(gpud_spectrum *s) {
    if (!s) return 0;
    cudaFree(s->d_pow);
    cudaFree(s->d_db);
    cudaFree(s->d_tab);
    delete s;
    return 0;
}

GPUD_API int GPUD_CALL gpud_spectrum_create(int max_fft, int max_segments, gpud_spectrum **out) {
    if (!out || ilog2_exact(max_fft) < 0 || max_fft > kMaxFft || max_segments <= 0) return GPUD_E_ARG;
    auto *s = new gpud_spectrum();
    s->max_fft = max_fft;
    s->max_segments = max_segments;
    if (cudaMalloc((void **)&s->d_pow, sizeof(double) * (size_t)max_fft * (size_t)max_segments) != cudaSuccess ||
        cudaMalloc((void **)&s->d_db, sizeof(double) * (size_t)max_fft) != cudaSuccess ||
        cudaMalloc((void **)&s->d_tab, sizeof(double2) * (size_t)(kMaxFft / 2)) != cudaSuccess) {
        gpud_spectrum_destroy(s);
        return GPUD_E_CUDA;
    }
    const cudaError_t e = gpud::launch_alone(k_spectrum_twiddles, dim3(kMaxFft / 2 / 256), 256, 0, nullptr, s->d_tab);
    gpud_count_launch(1);
    if (e != cudaSuccess || cudaStreamSynchronize(0) != cudaSuccess) {
        gpud_spectrum_destroy(s);
        return GPUD_E_CUDA;
    }
    *out = s;
    return 0;
}

static int spectrum_launch(gpud_spectrum *s, const gpud_float2 *iq, int N, int segs, int step, int hann, int welch,
                           cudaStream_t st, double *out_db) {
    const int l2 = ilog2_exact(N);
    // the shared-memory opt-in is per device: made on the launching device
    static std::atomic<uint64_t> optin{0};
    if (gpud::smem_optin_once(optin, (const void *)k_spectrum_seg, slot(kMaxFft) * 16) != cudaSuccess) return GPUD_E_CUDA;
    k_spectrum_seg<<<segs, kSpecThreads, slot(N) * 16, st>>>(reinterpret_cast<const float2 *>(iq), N, l2, step, hann, welch,
                                                       s->d_tab, s->d_pow);
    k_spectrum_db<<<(N + 255) / 256, 256, 0, st>>>(s->d_pow, N, segs, welch, s->d_db);
    if (cudaGetLastError() != cudaSuccess) return GPUD_E_CUDA;
    gpud_count_launch(2);
    if (cudaMemcpyAsync(out_db, s->d_db, sizeof(double) * (size_t)N, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return GPUD_E_CUDA;
    return 0;
}

GPUD_API int GPUD_CALL gpud_spectrum_single(gpud_spectrum *s, const gpud_float2 *iq, int n, int hann,
                                            gpud_stream_handle stream, double *out_db) {
    if (!s || !iq || !out_db || ilog2_exact(n) < 0 || n > s->max_fft) return GPUD_E_ARG;
    return spectrum_launch(s, iq, n, 1, 0, hann, 0, (cudaStream_t)stream, out_db);
}

GPUD_API int GPUD_CALL gpud_spectrum_welch(gpud_spectrum *s, const gpud_float2 *iq, int64_t n, int seg_size,
                                           double overlap, int hann, gpud_stream_handle stream, double *out_db,
                                           int *n_out) {
    if (!s || !iq || !out_db || !n_out || n < 0 || seg_size <= 0) return GPUD_E_ARG;
    *n_out = 0;
    if (overlap < 0) overlap = 0;
    if (overlap > 0.95) overlap = 0.95;
    int step = (int)((double)seg_size * (1 - overlap));
    if (step < 1) step = 1;
    const int64_t segs = n >= seg_size ? (n - seg_size) / step + 1 : 0;
    if (segs == 0) {
        // fewer samples than one segment: Spectrum of the whole vector, no window (welch.go:52-55)
        if (ilog2_exact((int)n) < 0 || n > s->max_fft) return GPUD_E_ARG;
        *n_out = (int)n;
        return spectrum_launch(s, iq, (int)n, 1, 0, 0, 0, (cudaStream_t)stream, out_db);
    }
    if (ilog2_exact(seg_size) < 0 || seg_size > s->max_fft || segs > s->max_segments) return GPUD_E_ARG;
    *n_out = seg_size;
    return spectrum_launch(s, iq, seg_size, (int)segs, step, hann, 1, (cudaStream_t)stream, out_db);
}

}  // extern "C"

// runner_kernels.cu -- sm_100a kernels of the batched / serving runner.
//
// One IQ block flows through, in stream order:
//   k_extract_dense<L> / k_extract_wide   NCO + polyphase FIR + decimation
//   k_demod, k_am                         FM discriminator (with bridge), SSB/CW, AM
//   k_wfm_fir                             stereo FIR bank: L+R, L-R band, pilot band
//   k_pll                                 19 kHz pilot PLL, L-R product, lock decision
//   k_wfm_out                             L-R 15 kHz LPF and L/R matrix, or mono fallback
//   k_rds                                 57 kHz RDS baseband (exact FreqShift phase)
//   k_post                                per-slot state carry (histories, phases)
// Every kernel takes a work list of (slot-block index, tile) pairs so channels
// with uneven taps / decimation run in the same launch.
#include <climits>
#include <cooperative_groups.h>
#include <cstdint>
#include <cuda_runtime.h>

#include "gpud_internal.cuh"
#include "pll_step.cuh"

#ifndef GPUD_DENSE_STAGE_U
#define GPUD_DENSE_STAGE_U 4
#endif
#ifndef GPUD_COLUMN_STAGE_U
#define GPUD_COLUMN_STAGE_U 4
#endif

namespace gpud {

// ===========================================================================
// Extraction: NCO shift -> FIR -> decimate  (streaming_host_core.go:5-64)
// ===========================================================================
//
// Output j of a block takes the input sample n_j = (D - pc - 1) + j*D as its
// newest sample (exports.cu:583) and y_j = sum_{k<T} h[k] * s(n_j - k), where
// s(i) = x[i] * exp(j*phi_i) for i >= 0 and the carried shifted history for
// i < 0 (zero before the stream start).
//
// Dense form (L = ceil(T/D) >= 2): the rotated samples of a tile are staged in
// shared memory transposed into the D polyphase components,
//     Z[p][m] = s(s0 + m*D - p),   p < D,
// so that y_j = sum_p sum_u h[p + u*D] * Z[p][j - u].  Warp w owns the phases
// p = w, w+8, ...; each lane owns R = 8 consecutive outputs and keeps a
// register window of R + L - 1 samples per phase (R*L FMAs per R+L-1 shared
// loads).  A row stride padded by one slot every 8 keeps the lane-strided
// window loads free of bank conflicts.  The 8 warps' partial sums are reduced
// through shared memory at the end.
constexpr int kDenseR = 8;
constexpr int kDenseOT = 32 * kDenseR;  // outputs per tile
constexpr int kDenseThreads = 256;

// Row stride in float2: one pad slot per 8 (lane-strided window reads stay
// conflict-free) and odd (the staging stores, which walk down a column with
// consecutive threads on consecutive phases, spread over all banks).
__host__ __device__ inline int dense_row_stride(int L) {
    int M = kDenseOT + L - 1;
    return (M + (M >> 3) + 1) | 1;
}

// Rotation table entries: one per 256-sample staging round.
__host__ __device__ inline int dense_rounds(int P, int L) { return (P * (kDenseOT + L - 1) + kDenseThreads - 1) / kDenseThreads; }

// Shared memory: Z (reused for the cross-warp reduction) | taps | rotation
// table.
__host__ __device__ inline int dense_zbytes(int P, int L) {
    int z = (P * dense_row_stride(L) * 8 + 15) & ~15;
    int red = 8 * (kDenseOT + kDenseOT / 8) * 16;  // float64 reduction of precise channels
    return z > red ? z : red;
}

__host__ __device__ inline int dense_smem_bytes(int P, int L) {
    return dense_zbytes(P, L) + ((P * L + 3) & ~3) * 4 + dense_rounds(P, L) * 8 + 16;
}

// Rotation of tile sample i' = t + 256k: exp(j phi(ibase + t)) * exp(j 256 k inc).
struct RotPair {
    float2 a;
    const float2 *tab;
    __device__ __forceinline__ float2 operator()(int k) const { return cmulf(a, tab[k]); }
};

__device__ __forceinline__ void dense_stage(float2 *Z, int Mp, int D, int total, int nk, int ibase, int n,
                                            const float2 *__restrict__ x, const float2 *__restrict__ hist, int H,
                                            const RotPair &rp) {
    const int t = (int)threadIdx.x;
    int mr = t / D, q = t - (t / D) * D;
    const int dm = kDenseThreads / D, dq = kDenseThreads - dm * D;
    const int nfull = total / kDenseThreads;  // rounds in which every thread has a sample
    const bool interior = ibase >= 0 && ibase + total <= n;
    constexpr int U = GPUD_DENSE_STAGE_U;  // staged loads in flight per thread
    int k = 0;
    if (interior && 32 % D == 0) {
        // D divides 32: the thread's phase row never changes (256 is a
        // multiple of D) and its column advances by dm = 256/D, a multiple of
        // 8, so the padded column c + c/8 advances by the constant 9*dm/8.
        const float2 *xp = x + ibase + t;
        float2 *zp = Z + (D - 1 - q) * Mp + mr + (mr >> 3);
        const int dz = dm + (dm >> 3);
        for (; k + U <= nfull; k += U) {
            float2 xv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = __ldg(xp + (k + u) * kDenseThreads);
#pragma unroll
            for (int u = 0; u < U; ++u) zp[(k + u) * dz] = cmulf(xv[u], rp(k + u));
        }
        mr += k * dm;  // hand the position to the remaining rounds
    } else if (interior) {
        const float2 *xp = x + ibase + t;
        for (; k + U <= nfull; k += U) {
            float2 xv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = __ldg(xp + (k + u) * kDenseThreads);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float2 rot = rp(k + u);
                Z[(D - 1 - q) * Mp + mr + (mr >> 3)] = cmulf(xv[u], rot);
                q += dq;
                mr += dm;
                if (q >= D) {
                    q -= D;
                    ++mr;
                }
            }
        }
    }
    // remaining rounds, and every round of tiles at the block edges
    for (; k < nk; ++k) {
        const int ip = t + k * kDenseThreads;
        if (ip < total) {
            const int i = ibase + ip;
            float2 v;
            if (i >= 0) {
                v = i < n ? cmulf(__ldg(x + i), rp(k)) : make_float2(0.f, 0.f);
            } else {
                const int hi = H + i;
                v = hi >= 0 ? hist[hi] : make_float2(0.f, 0.f);
            }
            Z[(D - 1 - q) * Mp + mr + (mr >> 3)] = v;
        }
        q += dq;
        mr += dm;
        if (q >= D) {
            q -= D;
            ++mr;
        }
    }
}

int dense_smem_bytes_host(int P, int L) { return dense_smem_bytes(P, L); }
int dense_tile() { return kDenseOT; }

// One phase row, L <= 16 taps: lane's R outputs from a window of R+L-1.
template <int L>
__device__ __forceinline__ void group_row(const float2 *zrow, const float *hrow, int lane, float2 *acc) {
    constexpr int R = kDenseR;
    float2 win[R + L - 1];
#pragma unroll
    for (int tt = 0; tt < R + L - 1; ++tt) {
        const int c = lane * R + tt;
        win[tt] = zrow[c + (c >> 3)];
    }
    float h[L];
#pragma unroll
    for (int u = 0; u < L; ++u) h[u] = hrow[u];
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int u = 0; u < L; ++u) acc[r] = ffma2(make_float2(h[u], h[u]), win[r + L - 1 - u], acc[r]);
    }
}

// One phase row, long arm (Le a multiple of 8 > 16): chunks of 8 taps with a
// window of R+7 samples that slides 8 columns per chunk (8 new loads).
__device__ __forceinline__ void group_row_long(const float2 *zrow, const float *hrow, int Le, int lane, float2 *acc) {
    constexpr int R = kDenseR;
    constexpr int W = R + 7;
    float2 win[W];
    int base = lane * R + Le - 8;  // chunk c: columns base - 8c + t
#pragma unroll
    for (int t = 0; t < W; ++t) {
        const int c = base + t;
        win[t] = zrow[c + (c >> 3)];
    }
    const int nc = Le >> 3;
    for (int ch = 0; ch < nc; ++ch) {
        const float4 h0 = *reinterpret_cast<const float4 *>(hrow + 8 * ch);
        const float4 h1 = *reinterpret_cast<const float4 *>(hrow + 8 * ch + 4);
        const float h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int v = 0; v < 8; ++v) acc[r] = ffma2(make_float2(h[v], h[v]), win[r + 7 - v], acc[r]);
        }
        if (ch + 1 < nc) {
#pragma unroll
            for (int t = W - 1; t >= 8; --t) win[t] = win[t - 8];
            base -= 8;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int c = base + t;
                win[t] = zrow[c + (c >> 3)];
            }
        }
    }
}

// Sum of a tile: the rows pp = warp, warp+8, ... < rows accumulate into each
// lane's R outputs, then the 8 warps' partial sums are reduced through shared
// memory (Z reused) and out(o, sum) receives tile output o.  With PREC each
// row is summed in float32 on its own and the rows are added in float64
// (channels whose demodulator magnifies white output error: the float32
// rounding then no longer grows with the running sum of the whole tile).
constexpr int kRedStride = kDenseOT + kDenseOT / 8;
constexpr int kRedBytes = 8 * kRedStride * 16;

template <bool PREC, class Row, class Out>
__device__ __forceinline__ void tile_sum(int rows, const Row &row, float2 *Z, const Out &out) {
    constexpr int R = kDenseR;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (!PREC) {
        float2 acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
        for (int pp = warp; pp < rows; pp += 8) row(pp, lane, acc);
        __syncthreads();
        float2 *red = Z + warp * kRedStride;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int o = lane * R + r;
            red[o + (o >> 3)] = acc[r];
        }
        __syncthreads();
        for (int o = threadIdx.x; o < kDenseOT; o += kDenseThreads) {
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int wv = 0; wv < 8; ++wv) {
                const float2 v = Z[wv * kRedStride + o + (o >> 3)];
                sum.x += v.x;
                sum.y += v.y;
            }
            out(o, sum);
        }
    } else {
        double dr[R], di[R];
#pragma unroll
        for (int r = 0; r < R; ++r) dr[r] = di[r] = 0.0;
        for (int pp = warp; pp < rows; pp += 8) {
            float2 acc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
            row(pp, lane, acc);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                dr[r] += (double)acc[r].x;
                di[r] += (double)acc[r].y;
            }
        }
        __syncthreads();
        double2 *Z64 = reinterpret_cast<double2 *>(Z);
        double2 *red = Z64 + warp * kRedStride;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int o = lane * R + r;
            red[o + (o >> 3)] = make_double2(dr[r], di[r]);
        }
        __syncthreads();
        for (int o = threadIdx.x; o < kDenseOT; o += kDenseThreads) {
            double2 sum = make_double2(0.0, 0.0);
#pragma unroll
            for (int wv = 0; wv < 8; ++wv) {
                const double2 v = Z64[wv * kRedStride + o + (o >> 3)];
                sum.x += v.x;
                sum.y += v.y;
            }
            out(o, sum);
        }
    }
}

// One 256-output tile of the dense form (work item w), arm length L.
template <int L>
__device__ __forceinline__ void dense_tile(const int2 w, const SlotBlock &sb, const ChanParams &cp,
                                           const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
                                           const float2 *__restrict__ hist_arena,
                                           const float *__restrict__ taps_arena, float2 *__restrict__ ext,
                                           float4 *smem4) {
    const int j0 = w.y * kDenseOT;
    const int D = cp.decim;
    const int P = cp.nphase;
    const int M = kDenseOT + L - 1;
    const int Mp = dense_row_stride(L);
    float2 *Z = reinterpret_cast<float2 *>(smem4);
    float *tsm = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + dense_zbytes(P, L));
    void *wtab = tsm + ((P * L + 3) & ~3);

    const int s0 = D - sb.pc - 1;
    const int m_base = j0 - (L - 1);
    const uint64_t u0 = st[sb.slot].nco_q;
    const uint64_t inc = cp.inc_q;
    const float2 *hist = hist_arena + cp.hist_off + sb.hist_sel * cp.hcap;
    const int H = sb.hist_len;
    // Staging.  Tile sample i' = 0..M*D-1 is block sample i = ibase + i' and
    // lands in Z[p][m] with m = i'/D, p = D-1 - i'%D.  Thread t takes
    // i' = t + 256*k: consecutive threads hit consecutive phases (odd row
    // stride: no bank conflicts), and (m, p) advance by a constant step with
    // one carry.  The rotation of sample i' is exp(j*phi(ibase + t)) *
    // exp(j*256*k*inc), both exact from the Q0.64 phase (the second from a
    // per-tile table).
    const int total = P * M;  // P == D in the dense form
    const int ibase = s0 + m_base * D - (D - 1);
    const int nk = dense_rounds(P, L);
    const float *tg = taps_arena + cp.taps_off;
    for (int i = threadIdx.x; i < P * L; i += kDenseThreads) tsm[i] = tg[i];
    const int t = (int)threadIdx.x;
    {
        float2 *w32 = reinterpret_cast<float2 *>(wtab);
        for (int k = threadIdx.x; k < nk; k += kDenseThreads)
            w32[k] = q64_phasor((uint64_t)k * (uint64_t)kDenseThreads * inc);
        const RotPair rp{q64_phasor(u0 + (uint64_t)(int64_t)(ibase + t) * inc), w32};
        __syncthreads();
        dense_stage(Z, Mp, D, total, nk, ibase, n, x, hist, H, rp);
    }
    __syncthreads();

    auto row = [&](int p, int lane, float2 *acc) { group_row<L>(Z + p * Mp, tsm + p * L, lane, acc); };
    float2 *dst = ext + sb.ext_off + j0;
    const int nv = sb.n_out - j0;
    if (cp.precise_sum)
        tile_sum<true>(P, row, Z, [&](int o, double2 v) {
            if (o < nv) dst[o] = make_float2((float)v.x, (float)v.y);
        });
    else
        tile_sum<false>(P, row, Z, [&](int o, float2 v) {
            if (o < nv) dst[o] = v;
        });
}

template <int L>
__global__ void __launch_bounds__(kDenseThreads, 2)
k_extract_dense(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
                const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
                const float2 *__restrict__ hist_arena, const float *__restrict__ taps_arena,
                float2 *__restrict__ ext) {
    dependency_wait();
    extern __shared__ float4 smem4[];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    if (w.y * kDenseOT >= sb.n_out) return;
    dense_tile<L>(w, sb, prm[sb.slot], st, x, n, hist_arena, taps_arena, ext, smem4);
}

// Several dense classes in one launch (each too small to fill the GPU alone):
// every CTA takes its tile's arm length from the channel.
__global__ void __launch_bounds__(kDenseThreads, 2)
k_extract_dense_any(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt,
                    const ChanParams *__restrict__ prm, const ChanState *__restrict__ st,
                    const float2 *__restrict__ x, int n, const float2 *__restrict__ hist_arena,
                    const float *__restrict__ taps_arena, float2 *__restrict__ ext) {
    dependency_wait();
    extern __shared__ float4 smem4[];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    if (w.y * kDenseOT >= sb.n_out) return;
    const ChanParams &cp = prm[sb.slot];
    switch (cp.plen) {  // uniform per CTA
#define GPUD_ANY(LL) \
    case LL: dense_tile<LL>(w, sb, cp, st, x, n, hist_arena, taps_arena, ext, smem4); break;
        GPUD_ANY(2) GPUD_ANY(3) GPUD_ANY(4) GPUD_ANY(5) GPUD_ANY(6) GPUD_ANY(7) GPUD_ANY(8) GPUD_ANY(9)
        GPUD_ANY(10) GPUD_ANY(11) GPUD_ANY(12) GPUD_ANY(13) GPUD_ANY(14) GPUD_ANY(15) GPUD_ANY(16)
#undef GPUD_ANY
    default: break;
    }
}

// ---------------------------------------------------------------------------
// Dense form, persistent pipelined variant (k_extract_dense_pipe<L, NG>).
//
// One CTA per SM walks a contiguous run of the class's tiles (consecutive
// tiles of a channel stay together).  Warp 16 is the producer: it loads the
// next tile's descriptors ahead of time and, as soon as the previous tile has
// been staged, brings the next tile's polyphase taps and (for tiles inside
// the block) its raw input span into shared memory with bulk copies whose
// completion is counted on an mbarrier.  The 16 consumer warps form NG groups
// that take the tiles in turn, each with its own Z: a group rotates and
// transposes its tile from the raw span into Z (tiles that reach into the
// history or past the block end stage from global memory as k_extract_dense
// does), releases the raw span, then runs the FIR rows and the cross-warp
// reduction while the other group stages the next tile.  The global-load
// latency of the one-tile-per-CTA kernel (descriptor chain, then staging
// loads) thereby overlaps arithmetic.  Every mbarrier wait is bounded: a wait
// that gives up stores a code in the runner's fault word and the CTA returns
// (the host reports GPUD_E_DEVICE_STATUS).
//
// Barrier use: full[g] completes once per tile of group g (the producer's
// arrival plus the bulk-copy bytes), `empty` once per staged tile (tiles are
// staged strictly in order, each after the previous one's release), named
// barrier 1 + g synchronises group g.
// ---------------------------------------------------------------------------
constexpr int kPipeCW = 16;                     // consumer warps
constexpr int kPipeThreads = 32 * kPipeCW + 32;  // + the producer warp
constexpr int kPipeMaxRounds = 64;              // staging rounds per tile (two table entries per producer lane)

struct PipeDesc {
    const float2 *hist;
    uint64_t u0, inc;
    int j0, n_out, ext_off, ibase, total, nk, D, P, H, precise, tma, off;
};
static_assert(32 + sizeof(PipeDesc) <= 128, "the descriptor sits between the mbarriers and the rotation table");

struct PipeLayout {
    int o_w, o_taps, tstride, o_z, zstride, o_r, bytes;
};

// Shared memory of a launch whose channels have at most pmax phases, ng
// consumer groups: mbarriers (full[2], empty) | descriptor | rotation table |
// taps x4 | Z (and reduction) per group | raw span.
__host__ __device__ inline PipeLayout pipe_layout(int pmax, int L, int ng) {
    PipeLayout lo;
    lo.o_w = 128;
    lo.o_taps = lo.o_w + kPipeMaxRounds * 8;
    lo.tstride = (pmax * L + 3) & ~3;  // floats; bulk-copy sizes are multiples of 16 bytes
    lo.o_z = lo.o_taps + 4 * lo.tstride * 4;
    const int z = pmax * dense_row_stride(L) * 8;
    const int red = (kPipeCW / ng) * kRedStride * 16;
    lo.zstride = ((z > red ? z : red) + 15) & ~15;
    lo.o_r = lo.o_z + ng * lo.zstride;
    lo.bytes = lo.o_r + (((pmax * (kDenseOT + L - 1) + 2) * 8 + 15) & ~15);
    return lo;
}

__device__ __forceinline__ void named_sync(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Named barrier that also ORs a predicate over the participating threads.
__device__ __forceinline__ bool named_sync_or(int id, int count, bool pred) {
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)pred), "r"(id), "r"(count)
        : "memory");
    return r != 0;
}

// Rows, cross-warp reduction (Z reused) and output of one tile for a consumer
// group of GW warps synchronised on named barrier `bar`.
template <bool PREC, int GW, class Row, class Out>
__device__ __forceinline__ void pipe_tile_sum(int rows, int gw, int lane, int gt, int bar, const Row &row, float2 *Z,
                                              const Out &out) {
    constexpr int R = kDenseR;
    constexpr int GNT = 32 * GW;
    if constexpr (!PREC) {
        float2 acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
        for (int pp = gw; pp < rows; pp += GW) row(pp, lane, acc);
        named_sync(bar, GNT);
        float2 *red = Z + gw * kRedStride;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int o = lane * R + r;
            red[o + (o >> 3)] = acc[r];
        }
        named_sync(bar, GNT);
        for (int o = gt; o < kDenseOT; o += GNT) {
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int wv = 0; wv < GW; ++wv) {
                const float2 v = Z[wv * kRedStride + o + (o >> 3)];
                sum.x += v.x;
                sum.y += v.y;
            }
            out(o, sum);
        }
    } else {
        double dr[R], di[R];
#pragma unroll
        for (int r = 0; r < R; ++r) dr[r] = di[r] = 0.0;
        for (int pp = gw; pp < rows; pp += GW) {
            float2 acc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
            row(pp, lane, acc);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                dr[r] += (double)acc[r].x;
                di[r] += (double)acc[r].y;
            }
        }
        named_sync(bar, GNT);
        double2 *Z64 = reinterpret_cast<double2 *>(Z);
        double2 *red = Z64 + gw * kRedStride;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int o = lane * R + r;
            red[o + (o >> 3)] = make_double2(dr[r], di[r]);
        }
        named_sync(bar, GNT);
        for (int o = gt; o < kDenseOT; o += GNT) {
            double2 sum = make_double2(0.0, 0.0);
#pragma unroll
            for (int wv = 0; wv < GW; ++wv) {
                const double2 v = Z64[wv * kRedStride + o + (o >> 3)];
                sum.x += v.x;
                sum.y += v.y;
            }
            out(o, sum);
        }
    }
}

template <int L, int NG>
__global__ void __launch_bounds__(kPipeThreads, 1)
k_extract_dense_pipe(const int2 *__restrict__ work, int ntiles, int pmax, const SlotBlock *__restrict__ sbt,
                     const ChanParams *__restrict__ prm, const ChanState *__restrict__ st,
                     const float2 *__restrict__ x, int n, const float2 *__restrict__ hist_arena,
                     const float *__restrict__ taps_arena, float2 *__restrict__ ext, unsigned *fault) {
    dependency_wait();
    constexpr int GW = kPipeCW / NG;  // warps per consumer group
    constexpr int GNT = 32 * GW;      // threads per consumer group
    extern __shared__ __align__(128) unsigned char psm[];
    const PipeLayout lo = pipe_layout(pmax, L, NG);
    uint64_t *full = reinterpret_cast<uint64_t *>(psm);  // full[0], full[1]
    uint64_t *empty = full + 2;
    PipeDesc *dsc = reinterpret_cast<PipeDesc *>(psm + 32);
    float2 *wt = reinterpret_cast<float2 *>(psm + lo.o_w);
    float *tsm = reinterpret_cast<float *>(psm + lo.o_taps);
    float2 *Rw = reinterpret_cast<float2 *>(psm + lo.o_r);
    const int b0 = (int)((long long)ntiles * blockIdx.x / gridDim.x);
    const int b1 = (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);
    const int nt = b1 - b0;
    if (threadIdx.x == 0) {
        mbar_init(full, 1);
        mbar_init(full + 1, 1);
        mbar_init(empty, 1);
        mbar_init_fence();
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int M = kDenseOT + L - 1;
    const int Mp = dense_row_stride(L);

    if (warp == kPipeCW) {
        // ---- producer ----
        for (int it = 0; it < nt; ++it) {
            const int2 w = work[b0 + it];
            const SlotBlock &sb = sbt[w.x];
            const ChanParams &cp = prm[sb.slot];
            PipeDesc d;
            d.D = cp.decim;
            d.P = cp.nphase;
            d.j0 = w.y * kDenseOT;
            d.n_out = sb.n_out;
            d.ext_off = sb.ext_off;
            d.u0 = st[sb.slot].nco_q;
            d.inc = cp.inc_q;
            d.ibase = (d.D - sb.pc - 1) + (d.j0 - (L - 1)) * d.D - (d.D - 1);
            d.total = d.P * M;
            d.nk = (d.total + GNT - 1) / GNT;
            d.hist = hist_arena + cp.hist_off + sb.hist_sel * cp.hcap;
            d.H = sb.hist_len;
            d.precise = cp.precise_sum;
            const int a0 = d.ibase & ~1;
            const int cnt = (d.ibase - a0 + d.total + 1) & ~1;
            d.tma = d.ibase >= 0 && (long long)a0 + cnt <= (long long)n;
            d.off = d.tma ? d.ibase - a0 : 0;
            // rotation of staging round k: exp(j k GNT inc), exact from the Q0.64 phase
            const float2 w0 = q64_phasor((uint64_t)lane * (uint64_t)GNT * d.inc);
            const float2 w1 = q64_phasor((uint64_t)(lane + 32) * (uint64_t)GNT * d.inc);
            const float *tsrc = taps_arena + cp.taps_off;
            // the previous tile has been staged: the raw span, the table and
            // the descriptor are free; taps buffer it & 3 was last read by
            // tile it - 4, finished before tile it - 2 of its group was staged
            if (it > 0 && !mbar_wait_bounded(empty, (unsigned)(it - 1) & 1u)) {
                if (lane == 0) device_fault(fault, 1u);
                return;
            }
            if (lane < d.nk) wt[lane] = w0;
            if (lane + 32 < d.nk) wt[lane + 32] = w1;
            if (lane == 0) *dsc = d;
            __syncwarp();
            if (lane == 0) {
                uint64_t *fb = full + (NG == 2 ? (it & 1) : 0);
                const unsigned tb = (unsigned)(((d.P * L + 3) & ~3) * 4);
                const unsigned rb = d.tma ? (unsigned)cnt * 8u : 0u;
                mbar_arrive_expect_tx(fb, tb + rb);
                bulk_to_smem(tsm + (it & 3) * lo.tstride, tsrc, tb, fb);
                if (d.tma) bulk_to_smem(Rw, x + a0, rb, fb);
            }
        }
        return;
    }

    // ---- consumers: group g takes tiles g, g + NG, ... ----
    const int g = warp / GW, gw = warp - g * GW;
    const int gt = (int)threadIdx.x - g * GNT;
    float2 *Z = reinterpret_cast<float2 *>(psm + lo.o_z + g * lo.zstride);
    uint64_t *fb = full + g;
    for (int it = g, kl = 0; it < nt; it += NG, ++kl) {
        const bool ok = mbar_wait_bounded(fb, (unsigned)kl & 1u);
        // the group has read its previous tile's reduction; all agree whether
        // to go on
        if (named_sync_or(1 + g, GNT, !ok)) {
            if (gt == 0) device_fault(fault, 2u);
            return;
        }
        const PipeDesc d = *dsc;
        const int D = d.D;
        const float2 a = q64_phasor(d.u0 + (uint64_t)(int64_t)(d.ibase + gt) * d.inc);
        int mr = gt / D, q = gt - (gt / D) * D;
        const int dm = GNT / D, dq = GNT - dm * D;
        if (d.tma) {
            const float2 *sp = Rw + d.off + gt;
            const int nfull = d.total / GNT;
            int k = 0;
            if ((GNT / 8) % D == 0) {
                // the thread's phase row is fixed and its padded column
                // advances by the constant dm + dm/8 (dm a multiple of 8)
                float2 *zp = Z + (D - 1 - q) * Mp + mr + (mr >> 3);
                const int dz = dm + (dm >> 3);
                for (; k + 4 <= nfull; k += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) zp[(k + u) * dz] = cmulf(sp[(k + u) * GNT], cmulf(a, wt[k + u]));
                }
                for (; k < nfull; ++k) zp[k * dz] = cmulf(sp[k * GNT], cmulf(a, wt[k]));
                mr += k * dm;
            }
            for (; k < d.nk; ++k) {
                if (gt + k * GNT < d.total)
                    Z[(D - 1 - q) * Mp + mr + (mr >> 3)] = cmulf(sp[k * GNT], cmulf(a, wt[k]));
                q += dq;
                mr += dm;
                if (q >= D) {
                    q -= D;
                    ++mr;
                }
            }
        } else {
            // tile at a block edge: history before sample 0, zeros past n;
            // four loads in flight per thread
            constexpr int U = 4;
            for (int k0 = 0; k0 < d.nk; k0 += U) {
                float2 v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int ip = gt + (k0 + u) * GNT, i = d.ibase + ip;
                    v[u] = make_float2(0.f, 0.f);
                    if (k0 + u < d.nk && ip < d.total) {
                        if (i >= 0) {
                            if (i < n) v[u] = __ldg(x + i);
                        } else if (d.H + i >= 0) {
                            v[u] = d.hist[d.H + i];
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int k = k0 + u, ip = gt + k * GNT;
                    if (k < d.nk && ip < d.total) {
                        // block samples are rotated here; history samples were stored rotated
                        const float2 z = d.ibase + ip >= 0 ? cmulf(v[u], cmulf(a, wt[k])) : v[u];
                        Z[(D - 1 - q) * Mp + mr + (mr >> 3)] = z;
                    }
                    q += dq;
                    mr += dm;
                    if (q >= D) {
                        q -= D;
                        ++mr;
                    }
                }
            }
        }
        named_sync(1 + g, GNT);
        if (gt == 0) mbar_arrive(empty);  // the raw span, the table and the descriptor may be refilled

        const float *hb = tsm + (it & 3) * lo.tstride;
        auto row = [&](int p, int ln, float2 *acc) { group_row<L>(Z + p * Mp, hb + p * L, ln, acc); };
        float2 *dst = ext + d.ext_off + d.j0;
        const int nv = d.n_out - d.j0;
        if (d.precise)
            pipe_tile_sum<true, GW>(d.P, gw, lane, gt, 1 + g, row, Z, [&](int o, double2 v) {
                if (o < nv) dst[o] = make_float2((float)v.x, (float)v.y);
            });
        else
            pipe_tile_sum<false, GW>(d.P, gw, lane, gt, 1 + g, row, Z, [&](int o, float2 v) {
                if (o < nv) dst[o] = v;
            });
    }
}

// Wide form (short polyphase arms, or tiles too large for shared memory): one
// warp per kWideOPW outputs, lanes stride the taps, warp-shuffle reduction.
// The NCO rotation is folded into the taps: for a sample of this block,
//     h[k] * x[n-k] * exp(j phi(n-k)) = exp(j phi(n)) * (h[k] exp(-j k inc)) * x[n-k],
// so each CTA builds the modulated taps hc[k] = h[k] exp(-j k inc) once (exact
// Q0.64 phases) and each output takes one rotation exp(j phi(n)) at the end;
// history samples (already shifted) take the real taps directly.
constexpr int kWideOPW = 4;                  // outputs per warp
constexpr int kWideOT = 8 * kWideOPW;        // outputs per 256-thread tile

int wide_smem_bytes_host(int T) { return T * 12; }

__global__ void __launch_bounds__(256)
k_extract_wide(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
               const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
               const float2 *__restrict__ hist_arena, const float *__restrict__ taps_arena,
               float2 *__restrict__ ext) {
    dependency_wait();
    extern __shared__ float4 smemw4[];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const int j0 = w.y * kWideOT;
    // a banked channel: only the outputs before its bank's first one
    const int n_end = sb.wide_end > 0 ? min(sb.wide_end, sb.n_out) : sb.n_out;
    if (j0 >= n_end) return;
    const ChanParams &cp = prm[sb.slot];
    const int T = cp.ntaps, D = cp.decim;
    const uint64_t u0 = st[sb.slot].nco_q;
    const uint64_t inc = cp.inc_q;
    float2 *hc = reinterpret_cast<float2 *>(smemw4);
    float *hr = reinterpret_cast<float *>(hc + T);
    for (int k = threadIdx.x; k < T; k += 256) {
        const float h = taps_arena[cp.dtaps_off + k];
        const float2 ph = q64_phasor((uint64_t)0 - (uint64_t)k * inc);
        hr[k] = h;
        hc[k] = make_float2(h * ph.x, h * ph.y);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s0 = D - sb.pc - 1;
    const float2 *hist = hist_arena + cp.hist_off + sb.hist_sel * cp.hcap;
    const int H = sb.hist_len;
    const int jw = j0 + warp * kWideOPW;
    if (jw >= n_end) return;
    const int no = min(kWideOPW, n_end - jw);
    float ar[kWideOPW], ai[kWideOPW], br[kWideOPW], bi[kWideOPW];
#pragma unroll
    for (int o = 0; o < kWideOPW; ++o) ar[o] = ai[o] = br[o] = bi[o] = 0.f;
    const int nj0 = s0 + jw * D;
    for (int k = lane; k < T; k += 32) {
        const float2 c = hc[k];
#pragma unroll
        for (int o = 0; o < kWideOPW; ++o) {
            if (o >= no) break;
            const int i = nj0 + o * D - k;
            if (i >= 0) {
                const float2 v = __ldg(x + i);
                ar[o] = fmaf(c.x, v.x, fmaf(-c.y, v.y, ar[o]));
                ai[o] = fmaf(c.x, v.y, fmaf(c.y, v.x, ai[o]));
            } else if (H + i >= 0) {
                const float2 v = hist[H + i];
                const float h = hr[k];
                br[o] = fmaf(h, v.x, br[o]);
                bi[o] = fmaf(h, v.y, bi[o]);
            }
        }
    }
#pragma unroll
    for (int o = 0; o < kWideOPW; ++o) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            ar[o] += __shfl_xor_sync(0xffffffffu, ar[o], off);
            ai[o] += __shfl_xor_sync(0xffffffffu, ai[o], off);
            br[o] += __shfl_xor_sync(0xffffffffu, br[o], off);
            bi[o] += __shfl_xor_sync(0xffffffffu, bi[o], off);
        }
    }
    if (lane < no) {
        // lane o writes output o (register arrays indexed by a compile-time loop)
#pragma unroll
        for (int o = 0; o < kWideOPW; ++o) {
            if (o == lane) {
                const int nj = nj0 + o * D;
                const float2 rot = q64_phasor(u0 + (uint64_t)(int64_t)nj * inc);
                const float2 y = cmulf(make_float2(ar[o], ai[o]), rot);
                ext[sb.ext_off + jw + o] = make_float2(y.x + br[o], y.y + bi[o]);
            }
        }
    }
}

// ===========================================================================
// Phase-grouped polyphase form: channels whose D phases of a 256-output tile
// do not fit in shared memory (large D), channels with one tap per phase
// (T <= D), and long arms (L > 16).  Arms of up to 16 taps run on
// k_extract_rot (below), whose warps work alone; here, for longer arms,
// the CTA stages the rotated samples of phases p_lo .. p_lo+Pc-1 only,
//     Z[pp][m] = s(s0 + (m_base + m)*D - (p_lo + pp)),
// -- for each column m a contiguous run of Pc samples -- and computes the
// group's share of the 256 outputs with the same warp/lane layout as the dense
// form.  One CTA takes all groups of its tile in turn, restaging shared memory
// per group, and each thread adds its output's group shares in group order in
// a register (deterministic: the grouping depends on the channel only), so no
// partial sums leave the SM.
// The rotation of sample cb(m) + r is A[m] * B[r], A[m] = exp(j phi(cb(m))),
// B[r] = exp(j r inc), both exact from the Q0.64 phase.
// ===========================================================================
// Arm length as k_extract_group runs it (whole chunks of 8 taps).  Shorter arms
// run elsewhere, but their groups are sized by the same rule.
__host__ __device__ inline int group_Le(int L) { return L > kRotMaxL ? (L + 7) & ~7 : L; }

__host__ __device__ inline int group_smem_bytes(int Pc, int L) {
    const int Le = group_Le(L);
    const int M = kDenseOT + Le - 1;
    int z = (Pc * dense_row_stride(Le) * 8 + 15) & ~15;  // the taps after Z are read as float4
    const int red = 8 * (kDenseOT + kDenseOT / 8) * 16;
    if (z < red) z = red;
    return z + ((Pc * Le + 3) & ~3) * 4 + (M + Pc) * 8 + 16;
}

int group_smem_bytes_host(int Pc, int L) { return group_smem_bytes(Pc, L); }

struct GroupTile {
    int j0, g, p_lo, Pc, Le, M, Mp;
};

// Sample x(cb0 + m*D + r) of column m lands in Z[Pc-1-r][m].  Warp w takes
// the columns m = w, w+8, ...; its lanes walk the column's contiguous run
// (coalesced loads; the stores go down one column of Z, odd row stride: no
// bank conflicts), four columns in flight.  fetch(i) returns the tile's
// value of block sample i.
template <class Fetch>
__device__ __forceinline__ void stage_columns(int Pc, int M, int Mp, int D, int cb0, float2 *Z, const Fetch &fetch) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int U = GPUD_COLUMN_STAGE_U;  // columns in flight per lane
    for (int m0 = warp; m0 < M; m0 += 8 * U) {
        for (int r = lane; r < Pc; r += 32) {
            float2 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int m = m0 + 8 * u;
                v[u] = m < M ? fetch(cb0 + m * D + r, m, r) : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int m = m0 + 8 * u;
                if (m < M) Z[(Pc - 1 - r) * Mp + m + (m >> 3)] = v[u];
            }
        }
    }
}

__device__ __forceinline__ void group_stage_samples(const GroupTile &gt, int D, int cb0, int n, int H,
                                                    const float2 *__restrict__ x, const float2 *__restrict__ hist,
                                                    float2 *Z, const float2 *A, const float2 *B) {
    const bool interior = cb0 >= 0 && cb0 + (gt.M - 1) * D + gt.Pc <= n;
    if (interior) {
        stage_columns(gt.Pc, gt.M, gt.Mp, D, cb0, Z, [&](int i, int m, int r) {
            return cmulf(__ldg(x + i), cmulf(A[m], B[r]));
        });
    } else {
        stage_columns(gt.Pc, gt.M, gt.Mp, D, cb0, Z, [&](int i, int m, int r) {
            if (i >= n) return make_float2(0.f, 0.f);
            if (i >= 0) return cmulf(__ldg(x + i), cmulf(A[m], B[r]));
            const int hi = H + i;  // carried history: shifted already
            return hi >= 0 ? hist[hi] : make_float2(0.f, 0.f);
        });
    }
}

// Stage Z (row stride Mp, column c stored at c + c/8), the taps of the
// group's phases (padded with zeros to Le per phase) and the rotation tables
// (tabs: M + Pc float2 entries).
__device__ __forceinline__ void group_stage(const GroupTile &gt, const SlotBlock &sb, const ChanParams &cp,
                                            uint64_t u0, const float2 *__restrict__ x, int n,
                                            const float2 *__restrict__ hist, const float *__restrict__ tg,
                                            float2 *Z, float *tsm, void *tabs) {
    const int D = cp.decim, L = cp.plen;
    const uint64_t inc = cp.inc_q;
    const int s0 = D - sb.pc - 1;
    const int m_base = gt.j0 - (gt.Le - 1);
    const int Pc = gt.Pc;
    // cb(m): first sample of column m's run
    const int cb0 = s0 + m_base * D - gt.p_lo - Pc + 1;
    for (int i = threadIdx.x; i < Pc * gt.Le; i += kDenseThreads) {
        const int pp = i / gt.Le, u = i - pp * gt.Le;
        tsm[i] = u < L ? tg[(gt.p_lo + pp) * L + u] : 0.f;
    }
    {
        float2 *A = reinterpret_cast<float2 *>(tabs), *B = A + gt.M;
        for (int m = threadIdx.x; m < gt.M; m += kDenseThreads)
            A[m] = q64_phasor(u0 + (uint64_t)(int64_t)(cb0 + m * D) * inc);
        for (int r = threadIdx.x; r < Pc; r += kDenseThreads) B[r] = q64_phasor((uint64_t)r * inc);
        __syncthreads();
        group_stage_samples(gt, D, cb0, n, sb.hist_len, x, hist, Z, A, B);
    }
    __syncthreads();
}

static_assert(kDenseOT == kDenseThreads, "the phase-group kernels keep one output per thread");

__global__ void __launch_bounds__(kDenseThreads, 2)
k_extract_group(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
                const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
                const float2 *__restrict__ hist_arena, const float *__restrict__ taps_arena,
                float2 *__restrict__ ext) {
    dependency_wait();
    extern __shared__ float4 smemg4[];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const ChanParams &cp = prm[sb.slot];
    GroupTile gt;
    gt.j0 = w.y * kDenseOT;
    if (gt.j0 >= sb.n_out) return;
    const int L = cp.plen;
    gt.Le = group_Le(L);
    gt.M = kDenseOT + gt.Le - 1;
    gt.Mp = dense_row_stride(gt.Le);
    int zb = (sb.pg * gt.Mp * 8 + 15) & ~15;
    const int red_b = kRedBytes;
    if (zb < red_b) zb = red_b;
    float2 *Z = reinterpret_cast<float2 *>(smemg4);
    float *tsm = reinterpret_cast<float *>(reinterpret_cast<char *>(smemg4) + zb);
    void *tabs = tsm + ((sb.pg * gt.Le + 3) & ~3);
    const float2 *hist = hist_arena + cp.hist_off + sb.hist_sel * cp.hcap;
    const uint64_t u0 = st[sb.slot].nco_q;

    auto row = [&](int pp, int lane, float2 *acc) {
        const float2 *zrow = Z + pp * gt.Mp;
        const float *hrow = tsm + pp * gt.Le;
        group_row_long(zrow, hrow, gt.Le, lane, acc);
    };
    const int nv = sb.n_out - gt.j0;
    const int o = (int)threadIdx.x;  // this thread's output of the tile
    double2 acc64 = make_double2(0.0, 0.0);
    float2 acc = make_float2(0.f, 0.f);
    for (int g = 0; g < sb.ng; ++g) {
        gt.g = g;
        gt.p_lo = g * sb.pg;
        gt.Pc = min(sb.pg, cp.nphase - gt.p_lo);
        if (g) __syncthreads();  // the last group's reduction has read Z
        group_stage(gt, sb, cp, u0, x, n, hist, taps_arena + cp.taps_off, Z, tsm, tabs);
        if (cp.precise_sum) {
            tile_sum<true>(gt.Pc, row, Z, [&](int, double2 v) {
                acc64.x += v.x;
                acc64.y += v.y;
            });
        } else {
            tile_sum<false>(gt.Pc, row, Z, [&](int, float2 v) {
                acc.x += v.x;
                acc.y += v.y;
            });
        }
    }
    if (o < nv)
        ext[sb.ext_off + gt.j0 + o] = cp.precise_sum ? make_float2((float)acc64.x, (float)acc64.y) : acc;
}

// Short arms (L <= 4) in phase groups with the NCO folded into the taps: with
// few taps per staged sample, rotating every sample costs more than the
// multiply-adds it feeds.  The tile stages raw samples (history samples, kept
// shifted, are turned back by exp(-j phi(i))), each CTA builds the modulated
// taps hc[p + uD] = h[p + uD] exp(-j (p + uD) inc) of its phases, and every
// output takes one rotation exp(j phi(n_j)) at the end:
//     y_j = exp(j phi(n_j)) * sum_k hc[k] x(n_j - k).
//
// A warp works on 32 of its tile's outputs by itself: lane w + 8g runs chain w
// (the phases pp = w, w+8, ... of a group) of the outputs 8g .. 8g+7, with the
// R + L - 1 samples of a phase in a register window, and the eight chains of an
// output are added in order at the end of each group.  Raw samples need no work
// on their way, so the window of a warp's outputs comes into its own piece of
// shared memory by asynchronous copies, kModKC phases at a time, each column a
// contiguous run: 16 bytes per copy where all columns start at one parity (D
// even), else 8.  Eight columns are followed by a pad of 64 bytes, so the window
// loads of two output groups fall on the two halves of the banks.  Nothing waits
// for another warp but the taps, which are built once per work item.
// Bound by the instructions of four warps a scheduler (two CTAs per SM by shared
// memory): issue slots 51 % busy, multiply-adds 38 % of the instructions, staging
// addresses and window loads the rest, waits for fixed latencies the largest
// stall (profiles/extraction_headroom_512.md).  1344 such channels of
// 64..768 taps among 2048: 1954 us with a tile's samples staged by the whole CTA
// through registers, 1288 now.  Chunks of 16 with the next one in flight: 1643
// (per-chunk work weighs more than the latency that 16 warps hide); rows of a
// chunk unrolled by four: 1435, by two: 1344 (instruction cache).
constexpr int kModKC = 32;                 // phases per staged chunk
constexpr int kModPitch = kModKC + 2;      // column stride (float2): even, room for a copy that starts one early
constexpr int kModR = 8;                   // outputs per lane
constexpr int kModBuf = 34 * kModPitch + (34 >> 3) * 8 + kModPitch;  // 32 + L - 1 <= 35 columns
constexpr int kModWarps = kDenseThreads / 32;
constexpr int kModRed = 33;                // row stride of the chains' sums
static_assert(kModBuf % 2 == 0 && kModBuf >= 2 * kModWarps * kModRed, "16-byte copies; float64 sums of eight chains");
constexpr int kModTileBits = 24, kModTileMask = (1 << kModTileBits) - 1;  // work item: (entry, first tile | tiles)
constexpr int kModTaps = 2048;             // modulated taps held at a time: all of them for most channels

// Dynamic shared memory that sizes a channel's phase groups (they order its
// sums, so this is kept as it was when a group was staged whole).
int mod_smem_bytes_host(int Pc, int L) {
    int z = (Pc * dense_row_stride(L) * 8 + 15) & ~15;
    if (z < kRedBytes) z = kRedBytes;
    return z + Pc * L * 8 + 16;
}

int mod_item(int tile, int tiles) { return tile | tiles << kModTileBits; }

// What a launch needs: two chunks per warp and the modulated taps of as many
// groups as kModTaps holds (at least one group's).
int mod_launch_bytes_host(int P, int Pc, int L) {
    return kModWarps * kModBuf * 8 + std::max(Pc * L, std::min(P * L, kModTaps)) * 8;
}

template <int BYTES>
__device__ __forceinline__ void copy_async(float2 *dst, const float2 *src) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// A warp's 32 outputs of a tile: column m (of 32 + L - 1), phase p is sample
// a0 + m*D - p.  Columns m0 .. m1-1 lie inside the block, with a sample to spare
// on each side.
struct WarpPart {
    int jw, nv, a0, m0, m1, cols;
};

__device__ __forceinline__ WarpPart warp_part(int tile, int warp, int L, int D, int P, int s0, int n_out, int n) {
    WarpPart t;
    t.jw = tile * kDenseOT + 32 * warp;
    t.nv = min(32, n_out - t.jw);
    t.cols = t.nv + L - 1;
    t.a0 = s0 + (t.jw - (L - 1)) * D;
    t.m0 = t.a0 >= P ? 0 : min(t.cols, (P - t.a0 + D - 1) / D);
    t.m1 = t.a0 + (t.cols - 1) * D + 1 < n ? t.cols : max(t.m0, t.cols - 1);
    return t;
}

// Stage phases p0 .. p0+np-1 (np <= KC) of a part's columns: phase p in position
// KC-1-(p-p0) + par of its column, par (returned) such that pairs of positions are
// aligned pairs of samples.  edge(i) is the value of sample i outside the block.
template <int L, int KC, class Edge>
__device__ __forceinline__ int stage_part(const WarpPart &t, float2 *z, int p0, int np, int D,
                                          const float2 *__restrict__ x, int n, const Edge &edge) {
    constexpr int pitch = KC + 2, per = 64 / KC, C = 32 + L - 1;  // columns per warp-wide 16-byte copy; all
    const int lane = threadIdx.x & 31;
    const bool wide = (D & 1) == 0;
    const int ab = t.a0 - p0 - (KC - 1);
    const int par = wide ? (ab + (int)(reinterpret_cast<uintptr_t>(x) >> 3)) & 1 : 0;
    if (wide) {
        const int fc = lane / (KC / 2), fq = 2 * (lane % (KC / 2));
        const int64_t step = per * (int64_t)D;
        if (fq + 1 >= KC - np + par) {
            const float2 *src = x + ((int64_t)(ab - par + fq) + (int64_t)fc * D);
            float2 *dst = z + fc * pitch + fq;
            constexpr int full = C / per, rest = C % per;
            if (t.m0 == 0 && t.m1 == C) {
#pragma unroll
                for (int i = 0; i < full; ++i, src += step)
                    copy_async<16>(dst + per * i * pitch + (per * i >> 3) * 8, src);
                if (fc < rest) copy_async<16>(dst + per * full * pitch + (per * full >> 3) * 8, src);
            } else {
                for (int m = fc; m < t.m1; m += per, src += step)
                    if (m >= t.m0) copy_async<16>(z + m * pitch + (m >> 3) * 8 + fq, src);
            }
        }
        if (par)
            for (int m = t.m0 + lane; m < t.m1; m += 32)
                copy_async<16>(z + m * pitch + (m >> 3) * 8 + KC, x + ((int64_t)(ab - 1 + KC) + (int64_t)m * D));
    }
    // by 8 bytes: odd D, and the columns at the block's ends
    const int q = lane % KC, c = lane / KC;
    if (q >= KC - np) {
        if (!wide) {
            const float2 *src = x + ((int64_t)(ab + q) + (int64_t)(t.m0 + c) * D);
#pragma unroll 4
            for (int m = t.m0 + c; m < t.m1; m += 32 / KC, src += 32 / KC * D)
                copy_async<8>(z + m * pitch + (m >> 3) * 8 + q, src);
        }
        auto end = [&](int m) {
            const int i = ab + q + m * D;
            float2 *dst = z + m * pitch + (m >> 3) * 8 + q + par;
            if (i >= 0 && i < n) copy_async<8>(dst, x + i);
            else *dst = edge(i);
        };
        for (int m = c; m < t.m0; m += 32 / KC) end(m);
        for (int m = t.m1 + c; m < t.cols; m += 32 / KC) end(m);
    }
    return par;
}

// Sum of the eight chains of this lane's output, in order; lane chain + 8 og holds
// the outputs 8 og .. 8 og + 7 of its chain.  red: the consumed chunk.
template <class V>
__device__ __forceinline__ V chain_sum(V *red, const V (&part)[kModR], int chain, int og, int lane) {
#pragma unroll
    for (int r = 0; r < kModR; ++r) red[chain * kModRed + og * kModR + r] = part[r];
    __syncwarp();
    V v;
    v.x = v.y = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const V e = red[k * kModRed + lane];
        v.x += e.x;
        v.y += e.y;
    }
    __syncwarp();
    return v;
}

template <int L, bool PREC>
__device__ __forceinline__ void mod_tile(const int2 w, const SlotBlock &sb, const ChanParams &cp,
                                         const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
                                         const float2 *__restrict__ hist_arena, const float *__restrict__ taps_arena,
                                         float2 *__restrict__ ext, float2 *smem) {
    constexpr int R = kModR;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chain = lane & 7, og = lane >> 3;
    const int D = cp.decim, P = cp.nphase, pg = sb.pg, ng = sb.ng;
    const uint64_t u0 = st[sb.slot].nco_q;
    const uint64_t inc = cp.inc_q;
    const float *tg = taps_arena + cp.taps_off;
    const float2 *hist = hist_arena + cp.hist_off + sb.hist_sel * cp.hcap;
    const int H = sb.hist_len;
    const int s0 = D - sb.pc - 1;
    float2 *z = smem + warp * kModBuf;
    float2 *hc = smem + kModWarps * kModBuf;
    const int gb = max(1, kModTaps / (pg * L));  // groups whose taps are held at a time

    auto edge = [&](int i) {  // a carried sample is shifted already: undo its rotation
        return i < 0 && H + i >= 0 ? cmulf(hist[H + i], q64_phasor((uint64_t)0 - (u0 + (uint64_t)(int64_t)i * inc)))
                                   : make_float2(0.f, 0.f);
    };

    const int tile0 = w.y & kModTileMask, tiles = w.y >> kModTileBits;
    for (int tile = tile0; tile < tile0 + tiles; ++tile) {
        const WarpPart t = warp_part(tile, warp, L, D, P, s0, sb.n_out, n);
        const int jw = t.jw, nv = t.nv;
        const bool live = nv > 0;
        // this lane's output and its rotation exp(j phi(n_j)), taken by every group's share
        const float2 ph = q64_phasor(u0 + (uint64_t)(int64_t)(s0 + (jw + lane) * D) * inc);
        double2 acc64 = make_double2(0.0, 0.0);
        float2 acc32 = make_float2(0.f, 0.f);

        for (int g = 0, gt = 0; g < ng; ++g) {
            const int p_lo = g * pg, Pc = min(pg, P - p_lo);
            if (g == gt) {
                gt += gb;
                if (tile == tile0 || gb < ng) {
                    if (g || tile != tile0) __syncthreads();  // every warp is done with the last groups' taps
                    for (int i = threadIdx.x, e = (min(P, gt * pg) - p_lo) * L; i < e; i += kDenseThreads) {
                        const int p = p_lo + i / L, u = i % L;
                        const float h = tg[p * L + u];
                        const float2 rot = q64_phasor((uint64_t)0 - (uint64_t)(p + u * D) * inc);
                        hc[i] = make_float2(h * rot.x, h * rot.y);
                    }
                    __syncthreads();
                }
            }
            if (live) {
                const float2 *h2 = hc + (p_lo - (gt - gb) * pg) * L;
                float2 acc[R];
                double2 d[PREC ? R : 1];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    acc[r] = make_float2(0.f, 0.f);
                    if constexpr (PREC) d[r] = make_double2(0.0, 0.0);
                }
                for (int c0 = 0; c0 < Pc; c0 += kModKC) {
                    const int np = min(kModKC, Pc - c0);
                    const int par = stage_part<L, kModKC>(t, z, p_lo + c0, np, D, x, n, edge);
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    __syncwarp();
                    const float2 *zc = z + og * (8 * kModPitch + 8) + (kModKC - 1) + par;
#pragma unroll 1
                    for (int s = 0; s < kModKC / 8; ++s) {
                        const int pl = 8 * s + chain;
                        if (pl < np) {
                            float2 win[R + L - 1], h[L];
#pragma unroll
                            for (int t = 0; t < R + L - 1; ++t) win[t] = zc[t * kModPitch + (t >> 3) * 8 - pl];
#pragma unroll
                            for (int u = 0; u < L; ++u) h[u] = h2[(c0 + pl) * L + u];
                            if constexpr (PREC) {
#pragma unroll
                                for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
                            }
#pragma unroll
                            for (int r = 0; r < R; ++r) {
#pragma unroll
                                for (int u = 0; u < L; ++u) {
                                    const float2 v = win[r + L - 1 - u];
                                    acc[r].x = fmaf(h[u].x, v.x, fmaf(-h[u].y, v.y, acc[r].x));
                                    acc[r].y = fmaf(h[u].x, v.y, fmaf(h[u].y, v.x, acc[r].y));
                                }
                            }
                            if constexpr (PREC) {
#pragma unroll
                                for (int r = 0; r < R; ++r) {
                                    d[r].x += (double)acc[r].x;
                                    d[r].y += (double)acc[r].y;
                                }
                            }
                        }
                    }
                    __syncwarp();
                }
                if constexpr (PREC) {
                    const double2 v = chain_sum(reinterpret_cast<double2 *>(z), d, chain, og, lane);
                    acc64.x += v.x * (double)ph.x - v.y * (double)ph.y;
                    acc64.y += v.x * (double)ph.y + v.y * (double)ph.x;
                } else {
                    const float2 y = cmulf(chain_sum(z, acc, chain, og, lane), ph);
                    acc32.x += y.x;
                    acc32.y += y.y;
                }
            }
        }
        if (lane < nv) ext[sb.ext_off + jw + lane] = PREC ? make_float2((float)acc64.x, (float)acc64.y) : acc32;
    }
}

__global__ void __launch_bounds__(kDenseThreads, 2)
k_extract_mod(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
              const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
              const float2 *__restrict__ hist_arena, const float *__restrict__ taps_arena,
              float2 *__restrict__ ext) {
    dependency_wait();
    extern __shared__ float4 smemm4[];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    if ((w.y & kModTileMask) * kDenseOT >= sb.n_out) return;
    const ChanParams &cp = prm[sb.slot];
    float2 *smem = reinterpret_cast<float2 *>(smemm4);
#define GPUD_MOD(LL)                                                                                      \
    if (cp.precise_sum) mod_tile<LL, true>(w, sb, cp, st, x, n, hist_arena, taps_arena, ext, smem);       \
    else mod_tile<LL, false>(w, sb, cp, st, x, n, hist_arena, taps_arena, ext, smem);                     \
    break;
    switch (cp.plen) {  // uniform per CTA
    case 1: GPUD_MOD(1)
    case 2: GPUD_MOD(2)
    case 3: GPUD_MOD(3)
    default: GPUD_MOD(4)
    }
#undef GPUD_MOD
}

// Phase groups of arms up to 16 taps with the warp layout of the modulated form:
// the copied samples are rotated in place (sample r of column m by A[m] B[r],
// the phase group's two exact phasors), then each lane runs its chain of rows.
// Chunks hold 32 phases, 16 for arms above 8 taps (whose windows have more
// columns), so two CTAs fit on an SM.  Arms above 16 taps stay with the whole CTA
// on one tile: a warp's 32 + L - 1 columns would be staged for 32 outputs.
// 480 phase-grouped channels among 2048 (300 with arms of 5..11 taps): 2057 us
// with every tile staged by its whole CTA through registers, 679 + 1182 us (the
// long arms) now.
__host__ __device__ constexpr int rot_kc(int L) { return L > 8 ? 16 : 32; }
__host__ __device__ constexpr int rot_buf(int L) {  // float2 entries of a warp's chunk
    return (32 + L - 1) * (rot_kc(L) + 2) + ((32 + L - 2) >> 3) * 8;
}
constexpr int kRotCols = 32 + kRotMaxL;  // column phasors of a warp
constexpr int kRotTaps = 1024;           // taps held at a time
static_assert(rot_buf(9) >= 2 * 8 * kModRed && rot_buf(1) >= 2 * 8 * kModRed, "float64 sums of eight chains");

int rot_launch_bytes_host(int P, int pg, int L) {
    return (kModWarps * (rot_buf(L) + kRotCols) + pg) * 8 + std::max(pg * L, std::min(P * L, kRotTaps)) * 4;
}

int rot_dense_bytes_host(int P, int L) {
    return (kModWarps * rot_buf(L) + kDenseThreads + dense_rounds(P, L)) * 8 + P * L * 4;
}

// DENSE: one group of all D phases with the dense form's rotation, sample i' of
// the tile by T1[i' % 256] T2[i' / 256].
// For many tiles whose classes need too much shared memory for the pipelined
// kernel: k_extract_dense_any then fits one CTA on an SM (224 channels among 2048:
// 1077 us there, 903 here with one tile per item, 840 with several).
template <int L, bool PREC, bool DENSE>
__device__ __forceinline__ void rot_tile(const int2 w, const SlotBlock &sb, const ChanParams &cp,
                                         const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
                                         const float2 *__restrict__ hist_arena, const float *__restrict__ taps_arena,
                                         float2 *__restrict__ ext, float2 *smem) {
    constexpr int R = kModR, KC = rot_kc(L), pitch = KC + 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chain = lane & 7, og = lane >> 3;
    const int D = cp.decim, P = cp.nphase, pg = DENSE ? P : sb.pg, ng = DENSE ? 1 : sb.ng;
    const uint64_t u0 = st[sb.slot].nco_q;
    const uint64_t inc = cp.inc_q;
    const float *tg = taps_arena + cp.taps_off;
    const float2 *hist = hist_arena + cp.hist_off + sb.hist_sel * cp.hcap;
    const int H = sb.hist_len;
    const int s0 = D - sb.pc - 1;
    float2 *z = smem + warp * rot_buf(L);
    // column and row phasors; DENSE: T1 and T2
    const int nk = DENSE ? dense_rounds(P, L) : pg;
    float2 *A = smem + kModWarps * rot_buf(L) + (DENSE ? 0 : warp * kRotCols);
    float2 *B = smem + kModWarps * (rot_buf(L) + (DENSE ? 0 : kRotCols)) + (DENSE ? kDenseThreads : 0);
    float *hs = reinterpret_cast<float *>(B + nk);
    const int gb = max(1, kRotTaps / (pg * L));  // groups whose taps are held at a time
    auto edge = [&](int i) { return i < 0 && H + i >= 0 ? hist[H + i] : make_float2(0.f, 0.f); };  // shifted already

    for (int r = threadIdx.x; r < nk; r += kDenseThreads)
        B[r] = q64_phasor((uint64_t)r * (uint64_t)(DENSE ? kDenseThreads : 1) * inc);
    const int tile0 = w.y & kModTileMask, tiles = w.y >> kModTileBits;
    for (int tile = tile0; tile < tile0 + tiles; ++tile) {
        const WarpPart t = warp_part(tile, warp, L, D, P, s0, sb.n_out, n);
        const bool live = t.nv > 0;
        double2 acc64 = make_double2(0.0, 0.0);
        float2 acc32 = make_float2(0.f, 0.f);
        if constexpr (DENSE) {
            const int ibase = s0 + (tile * kDenseOT - (L - 1)) * D - (D - 1);
            if (tile != tile0) __syncthreads();  // every warp is done with the last tile's T1
            A[threadIdx.x] = q64_phasor(u0 + (uint64_t)(int64_t)(ibase + (int)threadIdx.x) * inc);
            if (tile != tile0) __syncthreads();  // (the first tile's: with the taps)
        }
        for (int g = 0, gt = 0; g < ng; ++g) {
            const int p_lo = g * pg, Pc = min(pg, P - p_lo);
            if (g == gt) {
                gt += gb;
                if (tile == tile0 || (!DENSE && gb < ng)) {
                    if (g || tile != tile0) __syncthreads();  // every warp is done with the last groups' taps
                    for (int i = threadIdx.x, e = (min(P, gt * pg) - p_lo) * L; i < e; i += kDenseThreads)
                        hs[i] = tg[p_lo * L + i];
                    __syncthreads();
                }
            }
            if (live) {
                const float *h2 = hs + (p_lo - (gt - gb) * pg) * L;
                if constexpr (!DENSE)
                    for (int m = lane; m < t.cols; m += 32)
                        A[m] = q64_phasor(u0 + (uint64_t)(int64_t)(t.a0 - (p_lo + Pc - 1) + m * D) * inc);
                float2 acc[R];
                double2 d[PREC ? R : 1];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    acc[r] = make_float2(0.f, 0.f);
                    if constexpr (PREC) d[r] = make_double2(0.0, 0.0);
                }
                for (int c0 = 0; c0 < Pc; c0 += KC) {
                    const int np = min(KC, Pc - c0);
                    const int par = stage_part<L, KC>(t, z, p_lo + c0, np, D, x, n, edge);
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    __syncwarp();
                    {
                        // the rotation: this lane's position of every (32/KC)-th column
                        constexpr int S = 32 / KC, U = 4;
                        const int q = lane % KC, c = lane / KC;
                        if (q >= KC - np) {
                            const int r = Pc - 1 - (c0 + KC - 1 - q);  // of the column's samples, oldest first
                            const float2 b = B[DENSE ? 0 : r];
                            auto rotate = [&](float2 v, int m) {
                                if constexpr (DENSE) {
                                    const int i = (32 * warp + m) * D + r;
                                    return cmulf(v, cmulf(A[i & (kDenseThreads - 1)], B[i / kDenseThreads]));
                                } else {
                                    return cmulf(v, cmulf(A[m], b));
                                }
                            };
                            float2 *zq = z + q + par;
                            int m = c;
                            for (; m < t.m0; m += S) {  // carried samples stay
                                float2 &v = zq[m * pitch + (m >> 3) * 8];
                                if (t.a0 - (p_lo + c0 + KC - 1) + q + m * D >= 0) v = rotate(v, m);
                            }
                            for (; m < t.cols; m += S * U) {
                                float2 v[U];
#pragma unroll
                                for (int u = 0; u < U; ++u) {
                                    const int mu = m + S * u;
                                    if (mu < t.cols) v[u] = rotate(zq[mu * pitch + (mu >> 3) * 8], mu);
                                }
#pragma unroll
                                for (int u = 0; u < U; ++u) {
                                    const int mu = m + S * u;
                                    if (mu < t.cols) zq[mu * pitch + (mu >> 3) * 8] = v[u];
                                }
                            }
                        }
                        __syncwarp();
                    }
                    const float2 *zc = z + og * (8 * pitch + 8) + (KC - 1) + par;
#pragma unroll 1
                    for (int k = 0; k < KC / 8; ++k) {
                        const int pl = 8 * k + chain;
                        if (pl < np) {
                            float2 win[R + L - 1];
                            float h[L];
#pragma unroll
                            for (int i = 0; i < R + L - 1; ++i) win[i] = zc[i * pitch + (i >> 3) * 8 - pl];
#pragma unroll
                            for (int u = 0; u < L; ++u) h[u] = h2[(c0 + pl) * L + u];
                            if constexpr (PREC) {
#pragma unroll
                                for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
                            }
#pragma unroll
                            for (int r = 0; r < R; ++r) {
#pragma unroll
                                for (int u = 0; u < L; ++u)
                                    acc[r] = ffma2(make_float2(h[u], h[u]), win[r + L - 1 - u], acc[r]);
                            }
                            if constexpr (PREC) {
#pragma unroll
                                for (int r = 0; r < R; ++r) {
                                    d[r].x += (double)acc[r].x;
                                    d[r].y += (double)acc[r].y;
                                }
                            }
                        }
                    }
                    __syncwarp();
                }
                if constexpr (PREC) {
                    const double2 v = chain_sum(reinterpret_cast<double2 *>(z), d, chain, og, lane);
                    acc64 = DENSE ? v : make_double2(acc64.x + v.x, acc64.y + v.y);
                } else {
                    const float2 v = chain_sum(z, acc, chain, og, lane);
                    acc32 = DENSE ? v : make_float2(acc32.x + v.x, acc32.y + v.y);
                }
            }
        }
        if (lane < t.nv) ext[sb.ext_off + t.jw + lane] = PREC ? make_float2((float)acc64.x, (float)acc64.y) : acc32;
    }
}

template <bool DENSE>
__global__ void __launch_bounds__(kDenseThreads, 2)
k_extract_rot(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
              const ChanState *__restrict__ st, const float2 *__restrict__ x, int n,
              const float2 *__restrict__ hist_arena, const float *__restrict__ taps_arena,
              float2 *__restrict__ ext) {
    dependency_wait();
    extern __shared__ float4 smemr4[];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    if ((w.y & kModTileMask) * kDenseOT >= sb.n_out) return;
    const ChanParams &cp = prm[sb.slot];
    float2 *smem = reinterpret_cast<float2 *>(smemr4);
    switch (cp.plen) {  // uniform per CTA
#define GPUD_ROT(LL)                                                                                          \
    case LL:                                                                                                  \
        if (cp.precise_sum) rot_tile<LL, true, DENSE>(w, sb, cp, st, x, n, hist_arena, taps_arena, ext, smem);       \
        else rot_tile<LL, false, DENSE>(w, sb, cp, st, x, n, hist_arena, taps_arena, ext, smem);                     \
        break;
        GPUD_ROT(1) GPUD_ROT(2) GPUD_ROT(3) GPUD_ROT(4) GPUD_ROT(5) GPUD_ROT(6) GPUD_ROT(7) GPUD_ROT(8)
        GPUD_ROT(9) GPUD_ROT(10) GPUD_ROT(11) GPUD_ROT(12) GPUD_ROT(13) GPUD_ROT(14) GPUD_ROT(15) GPUD_ROT(16)
#undef GPUD_ROT
    default: break;
    }
}

// ===========================================================================
// Pre-demod decimation (recorder/streamer.go:1098-1146 with
// dsp/decimating_fir.go:56-95): 101-tap float64 low-pass, one output each
// time the decimator's phase counter is 0 -- stream samples d1_phase + j*d1
// of this block -- over the newest 101 extraction outputs (earlier blocks'
// from the carried 100-sample history), float64 accumulate in the
// reference's order, complex64 output.
// ===========================================================================
constexpr int kDecOT = 256;

__global__ void __launch_bounds__(kDecOT)
k_decim2(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
         const double *__restrict__ d1taps, const float2 *__restrict__ d1hist, float2 *__restrict__ ext) {
    dependency_wait();
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const int j = w.y * kDecOT + (int)threadIdx.x;
    if (j >= sb.n_dem) return;
    const ChanParams &cp = prm[sb.slot];
    const double *h = d1taps + (int64_t)sb.slot * kD1Taps;
    const float2 *hist = d1hist + (int64_t)sb.slot * kWfmHist;  // oldest first
    const float2 *x = ext + sb.ext_off;
    const int i = sb.d1_phase + j * cp.d1;
    double ar = 0.0, ai = 0.0;
    for (int k = 0; k < kD1Taps; ++k) {
        const int q = i - k;
        const float2 v = q >= 0 ? x[q] : hist[kWfmHist + q];
        ar = __dadd_rn(ar, __dmul_rn((double)v.x, h[k]));
        ai = __dadd_rn(ai, __dmul_rn((double)v.y, h[k]));
    }
    ext[sb.dem_off + j] = make_float2((float)ar, (float)ai);
}

// ===========================================================================
// Demodulators (internal/demod/*.go; bridge per recorder/streamer.go:1287-1302)
// ===========================================================================
constexpr int kDemodOT = 1024;

__global__ void __launch_bounds__(256)
k_demod(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
        const ChanState *__restrict__ st, const float2 *__restrict__ ext, float *__restrict__ comp,
        float *__restrict__ audio) {
    dependency_wait();
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const ChanParams &cp = prm[sb.slot];
    const int q0 = w.y * kDemodOT;
    const float2 *iq = ext + sb.dem_off;
    const int mode = cp.mode;
    if (mode == 1 || mode == 2 || mode == 3) {  // NFM / WFM / WFM_STEREO: fmDiscrimInto (fm.go:179-196)
        const float2 last = st[sb.slot].last_iq;
        float *dst = (mode == 1) ? (audio + sb.audio_off) : (comp + sb.comp_off);
        for (int q = q0 + threadIdx.x; q < q0 + kDemodOT && q < sb.n_disc; q += blockDim.x) {
            float2 p, c;
            if (sb.bridge) {
                p = q == 0 ? last : iq[q - 1];
                c = iq[q];
            } else {
                p = iq[q];
                c = iq[q + 1];
            }
            double num = (double)p.x * (double)c.y - (double)p.y * (double)c.x;
            double den = (double)p.x * (double)c.x + (double)p.y * (double)c.y;
            dst[q] = (float)atan2(num, den);
        }
    } else if (mode == 5 || mode == 6 || mode == 7) {  // ssb.go:19-39, cw.go:11-26
        float *dst = audio + sb.audio_off;
        for (int q = q0 + threadIdx.x; q < q0 + kDemodOT && q < sb.n_dem; q += blockDim.x) {
            double ph = (double)(q + 1) * cp.ssb_inc;
            double s, c;
            sincos(ph, &s, &c);
            float2 v = iq[q];
            dst[q] = (mode == 7) ? (float)((double)v.x * c) : (float)((double)v.x * c - (double)v.y * s);
        }
    }
}

// AM.Demod (am.go:11-27): envelope minus the per-call mean.  One CTA per slot.
__global__ void __launch_bounds__(256)
k_am(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const float2 *__restrict__ ext,
     float *__restrict__ audio) {
    dependency_wait();
    __shared__ double red[256];
    const SlotBlock sb = sbt[work[blockIdx.x].x];
    const float2 *iq = ext + sb.dem_off;
    double acc = 0.0;
    for (int q = threadIdx.x; q < sb.n_dem; q += 256) acc += hypot((double)iq[q].x, (double)iq[q].y);
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    const float mean = (float)(red[0] / (double)sb.n_dem);
    float *dst = audio + sb.audio_off;
    for (int q = threadIdx.x; q < sb.n_dem; q += 256) {
        float mag = (float)hypot((double)iq[q].x, (double)iq[q].y);
        dst[q] = mag - mean;
    }
}

// ===========================================================================
// WFM multiplex (recorder/streamer.go:1525-1644)
// ===========================================================================
//
// Rate-class tables: the stereo filters as float taps padded to 104
//   x = LPF 15 kHz (L+R and L-R lowpass), y = LPF 53 kHz - LPF 23 kHz (L-R
//   band), z = LPF 21 kHz - LPF 17 kHz (pilot band); the band-pass pairs are
//   differenced in float64 before rounding, one filter each instead of two;
// and the RDS lowpass (7.5 kHz, fm.go:155) in float64.
constexpr int kWfmTapsPad = 104;
struct WfmTaps {
    float4 t[kWfmTapsPad];
    double rds[kWfmTaps];
};
static_assert(sizeof(WfmTaps) == kWfmTapsBytes, "the rates' stride of the host");

// Composite-rate work arrays (all float, same offsets comp_off):
//   work + 0*W comp (discriminator output), 1*W lpr, 2*W bpf, 3*W pilot, 4*W lr
constexpr int kFirOT = 1024;   // composite samples per tile
constexpr int kAudioDlStride = kWfmHist + 4;  // 100 samples + valid count
constexpr int kFirThreads = 128;  // 8 outputs each

__host__ __device__ constexpr int padi(int e) { return e + (e >> 3); }

// Loads composite samples [q0-104, q0+kFirOT) into shared memory; indices
// below 0 come from the 100-sample delay line `dl` (oldest first, newest at
// 99) with `valid` trailing entries, zero before that.
__device__ __forceinline__ void stage_window(float *win, const float *__restrict__ src, int q0, int nvalid,
                                             const float *__restrict__ dl, int valid) {
    for (int i = threadIdx.x; i < kFirOT + kWfmTapsPad; i += blockDim.x) {
        int q = q0 - kWfmTapsPad + i;
        float v = 0.f;
        if (q >= 0) {
            if (q < nvalid) v = src[q];
        } else if (q >= -valid) {
            v = dl[kWfmHist + q];
        }
        win[padi(i)] = v;
    }
}

__global__ void __launch_bounds__(kFirThreads)
k_wfm_fir(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
          const WfmTaps *__restrict__ taps, float *__restrict__ wk, int W, const float *__restrict__ comp_dl) {
    dependency_wait();
    __shared__ float win[padi(kFirOT + kWfmTapsPad) + 8];
    __shared__ float4 tp[kWfmTapsPad];
    __shared__ float s_out[3 * (kFirOT + kFirOT / 32)];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const ChanParams &cp = prm[sb.slot];
    const int q0 = w.y * kFirOT;
    if (q0 >= sb.n_disc) return;
    const WfmTaps &tb = taps[cp.rds_tab];
    for (int i = threadIdx.x; i < kWfmTapsPad; i += kFirThreads) tp[i] = tb.t[i];
    const float *comp = wk + sb.comp_off;
    stage_window(win, comp, q0, sb.n_disc, comp_dl + cp.wfm_idx * kWfmHist, sb.comp_hist_len);
    __syncthreads();
    const int t = threadIdx.x;
    // window index of composite sample q0 + 8t + r - k is 8t + r - k + 104
    const int base = 8 * t + kWfmTapsPad;
    float2 ab[8];  // outputs of the first two filters
    float c[8], ring[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        ab[r] = make_float2(0.f, 0.f);
        c[r] = 0.f;
    }
#pragma unroll
    for (int j = 1; j < 8; ++j) ring[j] = win[padi(base + j)];
    for (int kb = 0; kb < kWfmTapsPad; kb += 8) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const int k = kb + kk;
            ring[(8 - kk) & 7] = win[padi(base - k)];
            const float4 h = tp[k];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float v = ring[(r - kk + 8) & 7];
                ab[r] = ffma2(make_float2(h.x, h.y), make_float2(v, v), ab[r]);
                c[r] = fmaf(h.z, v, c[r]);
            }
        }
    }
    // outputs through shared memory (index i + i/32: conflict-free both
    // ways), then coalesced stores of the three arrays
    constexpr int kS = kFirOT + kFirOT / 32;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = 8 * t + r, j = i + (i >> 5);
        s_out[j] = ab[r].x;
        s_out[kS + j] = ab[r].y;
        s_out[2 * kS + j] = c[r];
    }
    __syncthreads();
    float *lpr = wk + 1 * W + sb.comp_off, *bpf = wk + 2 * W + sb.comp_off, *pil = wk + 3 * W + sb.comp_off;
    const int nq = min(kFirOT, sb.n_disc - q0);
    for (int i = t; i < nq; i += kFirThreads) {
        const int j = i + (i >> 5);
        lpr[q0 + i] = s_out[j];
        bpf[q0 + i] = s_out[kS + j];
        pil[q0 + i] = s_out[2 * kS + j];
    }
}

__device__ __forceinline__ PllK pll_consts(const ChanParams &cp, const ChanState &s) {
    PllK k;
    k.alpha = cp.pll_alpha;
    k.beta = cp.pll_beta;
    k.lpa = (float)cp.pll_lpa;
    k.dfmin = cp.pll_fmin - s.pll_freq;
    k.dfmax = cp.pll_fmax - s.pll_freq;
    k.q0 = rad_to_q64(s.pll_phase);
    k.qf = rad_to_q64(s.pll_freq);
    return k;
}

// Loop phase after t steps, wrapped to [0, 2pi) (the serial loop's range).
__device__ __forceinline__ double pll_phase_at(const PllK &k, int t, double dphi) {
    const uint64_t q = k.q0 + (uint64_t)t * k.qf;
    double ph = (double)q * (2.0 * GPUD_PI / 18446744073709551616.0) + dphi;
    ph -= (2.0 * GPUD_PI) * floor(ph * (1.0 / (2.0 * GPUD_PI)));
    return ph;
}

// End of one stereoDecodeStateful call: store the loop state, update errAvg
// (EMA per call), the coherence / frequency / errAvg lock test and the
// hysteresis counters (streamer.go:1614-1635, 1363-1380).
__device__ void pll_finish(ChanState &s, const ChanParams &cp, int n, double ph, double fr, double I, double Q,
                           double es, double pp) {
    const double twopi = 2.0 * GPUD_PI;
    s.pll_phase = ph;
    s.pll_freq = fr;
    s.pll_i = I;
    s.pll_q = Q;
    const double block_err = es / (double)n;
    if (cp.flags & kChBatchStereo) {
        // wfmStereoDecodeBatch (wfm_batch_stereo.go:137-142): one call, no
        // hysteresis; locked by the pilot-band share of the composite's power
        const double ratio = s.comp_power > 0.0 ? pp / s.comp_power : 0.0;
        const double fhz = fr * (double)cp.out_rate / twopi;
        const int locked = ratio > 0.003 && fabs(fhz - 19000.0) < 250.0 && block_err < 0.35;
        s.locked = locked;
        s.enabled = locked;
        s.coherence = (float)ratio;
        s.pilot_hz = (float)fhz;
        s.last_err_avg = (float)block_err;
        return;
    }
    const double ea = 0.9 * s.err_avg + 0.1 * block_err;
    s.err_avg = ea;
    double coherence = 0.0;
    if (pp > 1e-12) coherence = (I * I + Q * Q) * (double)n / pp;
    const double fhz = fr * (double)cp.out_rate / twopi;
    const int locked = coherence > 0.15 && fabs(fhz - 19000.0) < 250.0 && ea < 0.35;
    s.locked = locked;
    s.coherence = (float)coherence;
    s.pilot_hz = (float)fhz;
    s.last_err_avg = (float)ea;
    if (locked) {
        s.on_count += 1;
        s.off_count = 0;
        if (s.on_count >= 4) s.enabled = 1;
    } else {
        s.on_count = 0;
        s.off_count += 1;
        if (s.off_count >= 10) s.enabled = 0;
    }
}

// Pilot PLL, serial per channel (recorder/streamer.go:1560-1619).  Phase,
// frequency and the I/Q lowpass states are float64 (the frequency integrator
// moves by ~1e-10 rad/sample, below float32 resolution); the loop's sin/cos and
// atan2 are float32.  One CTA per channel: lane 0 of warp 0 runs the recurrence
// from shared memory; warp 1 prefetches the next chunk of the pilot band and
// finishes the previous chunk off the critical path (lr = bpf * float32(2 sin
// 2phase), pilot power).  Per-call lock decision and hysteresis at the end
// (streamer.go:1363-1380, 1615-1635).
constexpr int kPllChunk = 2048;

__global__ void __launch_bounds__(64)
k_pll(const int *__restrict__ list, int count, const SlotBlock *__restrict__ sbt,
      const ChanParams *__restrict__ prm, ChanState *__restrict__ st, float *__restrict__ wk, int W) {
    dependency_wait();
    __shared__ float s_pil[2][kPllChunk];
    __shared__ float s_th[2][kPllChunk];
    __shared__ double s_red[32];
    const int idx = blockIdx.x;
    if (idx >= count) return;
    const SlotBlock sb = sbt[list[idx]];
    const int n = sb.n_disc;
    if (n <= 0) return;
    const ChanParams &cp = prm[sb.slot];
    ChanState &s = st[sb.slot];
    const float *pil = wk + 3 * W + sb.comp_off;
    const float *bpf = wk + 2 * W + sb.comp_off;
    float *lr = wk + 4 * W + sb.comp_off;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nc = (n + kPllChunk - 1) / kPllChunk;
    double pp = 0.0;  // pilot power, accumulated by warp 1
    // prologue: chunk 0 into buffer 0
    if (warp == 1) {
        for (int q = lane; q < min(n, kPllChunk); q += 32) s_pil[0][q] = pil[q];
    }
    __syncthreads();
    const PllK k = pll_consts(cp, s);
    PllRun x = pll_begin(0.0, 0.0, (float)s.pll_i, (float)s.pll_q);
    double es = 0.0;
    for (int c = 0; c <= nc; ++c) {
        if (warp == 0) {
            if (lane == 0 && c < nc) {
                const float *sp = s_pil[c & 1];
                float *th = s_th[c & 1];
                const int base = c * kPllChunk;
                const int len = min(kPllChunk, n - base);
                uint64_t qr = k.q0 + (uint64_t)base * k.qf;
                for (int q = 0; q < len; ++q) {
                    PllEval o;
                    if (q % kPllSeg == 0) x = pll_begin(x.dphi(), x.df, x.I, x.Q);
                    pll_step<false>(qr, x, sp[q], k, o);
                    qr += k.qf;
                    es += fabs((double)o.e);
                    th[q] = pll_twice(qr, x);
                }
            }
        } else {
            // finish chunk c-1, then prefetch chunk c+1 into the buffer it frees
            if (c >= 1) {
                const int base = (c - 1) * kPllChunk;
                const int len = min(kPllChunk, n - base);
                const float *th = s_th[(c - 1) & 1];
                const float *sp = s_pil[(c - 1) & 1];
                for (int q = lane; q < len; q += 32) {
                    const double p = (double)sp[q];
                    pp += p * p;
                    lr[base + q] = bpf[base + q] * (2.0f * sinpif(th[q]));
                }
            }
            __syncwarp();
            if (c + 1 < nc) {
                const int base = (c + 1) * kPllChunk;
                const int len = min(kPllChunk, n - base);
                float *dst = s_pil[(c + 1) & 1];
                for (int q = lane; q < len; q += 32) dst[q] = pil[base + q];
            }
        }
        __syncthreads();
    }
    if (warp == 1) {
        for (int off = 16; off > 0; off >>= 1) pp += __shfl_xor_sync(0xffffffffu, pp, off);
        if (lane == 0) s_red[0] = pp;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    pll_finish(s, cp, n, pll_phase_at(k, n, x.dphi()), s.pll_freq + x.df, (double)x.I, (double)x.Q, es, s_red[0]);
    s.pll_path = 2;
}


// ===========================================================================
// Pilot PLL, parallel in time: a coarse model of the loop, then
// multiple-shooting Newton on the loop itself.
// ===========================================================================
// The block's loop trajectory x_t = (phase, freq, I, Q), t = 0..n, obeys
// x_{t+1} = F(x_t, p_t) with the serial kernel's exact step F.  The block is
// cut into one segment of S = 16 consecutive steps per thread; the unknowns
// are the segment start states s_g.  Each iteration every thread integrates
// its segment with F from s_g (the exact nonlinear loop, no linearisation
// inside the segment), giving the end state E_g(s_g), and Newton's update of
// the start states,
//     d_{g+1} = M_g d_g + (E_g(s_g) - s_{g+1}),   d_0 = 0,   s_g <- s_g + d_g,
// is a linear recurrence over segments, solved by an associative scan over
// affine maps (4x4 matrix + vector, float32; states and residuals float64 /
// float32 as in F): warp shuffles, then shared memory across warps, then
// distributed shared memory across the cluster's CTAs.  The fixed point is the
// serial trajectory whatever M_g is and wherever the iteration starts: both
// set the number of iterations only.
//
// Where it starts: the loop is slow (50 Hz bandwidth, 200 Hz I/Q lowpass)
// against a segment, so a segment's effect on the state is known to ~1e-4 rad
// from four sums over its pilot samples (CoarseSeg), taken once.  The start
// states come from Newton on that coarse map -- no sweep over samples, one
// scan each -- and then iterations with F, at first with the coarse map's
// Jacobian for M_g: two for a locked loop.  Loops that turn against the
// free-running ramp (acquisition, requests on noise) go on with F's own segment
// Jacobians.
//
// Measured (kernel alone; before: Newton with F's Jacobians from the
// free-running ramp and scans by shuffles): 40 channels x 32768 steps 78 -> 53
// us (3-5 -> 2 iterations), one channel of 7680 steps 48 -> 31 us, 154 channels
// of 8192 steps of which half on noise 360-495 -> 122 us (up to 64 iterations
// and a serial rest -> 11).  What bounds it: the latency of 16 dependent steps
// (~250 cycles each) and of a scan (~4500 cycles) per iteration.
//
// A block not converged after max_iters iterations keeps its consistent
// prefix (a segment whose start is exact is exact after one more iteration)
// and one warp runs the serial loop from its last segment on.  Blocks longer than one
// segment per thread of the largest cluster (32768 steps) are solved chunk by
// chunk, each from the end state of the one before.
#ifndef GPUD_PLL_CLUSTER
#define GPUD_PLL_CLUSTER 8  // CTAs per channel at most
#endif
constexpr int kNewtonThreads = 256;
constexpr int kNewtonMaxCluster = GPUD_PLL_CLUSTER;
constexpr int kPllChunkSteps = kNewtonMaxCluster * kNewtonThreads * kPllSeg;  // steps solved at once
#ifndef GPUD_PLL_COARSE
#define GPUD_PLL_COARSE 2  // Newton iterations on the coarse map of a locked loop
#endif
#ifndef GPUD_PLL_COARSE_FREE
#define GPUD_PLL_COARSE_FREE 8  // ... and of one that was not
#endif
#ifndef GPUD_PLL_QUASI
#define GPUD_PLL_QUASI 8  // iterations on the loop that take the coarse map's Jacobian
#endif
constexpr int kPllCoarse = GPUD_PLL_COARSE, kPllCoarseFree = GPUD_PLL_COARSE_FREE, kPllQuasi = GPUD_PLL_QUASI;
static_assert(kPllCoarse > 0 && kPllCoarseFree > 0, "sh.next starts in the coarse iterations");
constexpr int kPllOnce = 3;       // iterations within which a locked loop converges
constexpr int kPllJacSweeps = 2;  // then: sweeps that evaluate F's segment Jacobians before chord steps may start

// CTAs per cluster that give every channel of a launch (at most max_n steps)
// one thread per segment of a chunk.
int pll_cluster_for(int max_n) {
    const int steps = max_n < kPllChunkSteps ? max_n : kPllChunkSteps;
    const int seg = (steps + kPllSeg - 1) / kPllSeg;
    const int c = (seg + kNewtonThreads - 1) / kNewtonThreads;
    int p = 1;
    while (p < c) p *= 2;
    return p < 1 ? 1 : (p > kNewtonMaxCluster ? kNewtonMaxCluster : p);
}
// Convergence: the last correction of every segment start is below what the
// outputs resolve (the float32 sin/cos/atan2 and lowpass states leave a floor
// near 1e-10 rad and 1e-9 in I/Q).
constexpr float kTolPhase = 1e-8f, kTolFreq = 1e-12f, kTolIQ = 1e-7f;
constexpr float kTolAngle = 2.4e-7f;  // half an ulp of an angle of up to 2 pi in float32
constexpr int kNW = kNewtonThreads / 32;

// M <- J M, with J's sparsity (phase/freq rows dense, I/Q rows phase + diagonal).
__device__ __forceinline__ void mat_push(float (&m)[16], const PllEval &o, float om) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float p0 = m[j], f0 = m[4 + j], i0 = m[8 + j], q0 = m[12 + j];
        m[j] = fmaf(o.ja, p0, fmaf(o.jb, f0, fmaf(o.jc, i0, o.jd * q0)));
        m[4 + j] = fmaf(o.ka, p0, fmaf(o.kb, f0, fmaf(o.kc, i0, o.kd * q0)));
        m[8 + j] = fmaf(o.iphi, p0, om * i0);
        m[12 + j] = fmaf(o.qphi, p0, om * q0);
    }
}

// Segment start state, deviation form (see pll_step).
struct SegState {
    double dphi, df;
    float I, Q;
};

// What the coarse map knows of a segment of m steps with the loop phase held
// at the free-running ramp theta_i plus a constant: with r = 1 - lpa,
//     C + jS   = sum_i r^(m-1-i) p_i exp(j theta_i)
//     C2 + jS2 = sum over the steps of the same sum up to that step,
// so that I and Q after the segment and their means over it are linear in the
// state and in the sine and cosine of the constant.
struct CoarseSeg {
    float4 c;      // C, S, C2, S2
    float rm, r1;  // r^m, (r + ... + r^m) / m
    float m;
};

// atan2 to 1e-5 rad (the odd polynomial of Abramowitz and Stegun 4.4.49 on
// the smaller over the larger): the coarse map only sets where Newton starts.
__device__ __forceinline__ float coarse_atan2(float y, float x) {
    const float ax = fabsf(x), ay = fabsf(y);
    const float hi = fmaxf(ax, ay), lo = fminf(ax, ay);
    const float t = hi > 0.f ? __fdividef(lo, hi) : 0.f;
    const float u = t * t;
    float r = fmaf(u, fmaf(u, fmaf(u, fmaf(u, 0.0208351f, -0.0851330f), 0.1801410f), -0.3302995f), 0.9998660f) * t;
    r = ay > ax ? 1.57079633f - r : r;
    r = x < 0.f ? 3.14159265f - r : r;
    return copysignf(r, y);
}

// The coarse map of one segment from start state x: the map's matrix in a
// (row-major) and, in float32, the mismatch of the segment's end with the next
// start nx (the float64 differences are taken first).
__device__ __forceinline__ float4 coarse_step(const CoarseSeg &c, const PllK &k, const SegState &x, const SegState &nx,
                                              float (&a)[16]) {
    const float alpha = (float)k.alpha, beta = (float)k.beta, half = 0.5f * (c.m - 1.f);
    const float df = (float)x.df;
    // the phase at the middle of the segment
    float sn, cs;
    __sincosf(fmaf(half, fmaf(alpha, coarse_atan2(x.Q, x.I), df), (float)x.dphi), &sn, &cs);
    const float ri = c.rm * x.I, rq = c.rm * x.Q;
    const float dI = k.lpa * fmaf(cs, c.c.x, -sn * c.c.y), dQ = -k.lpa * fmaf(sn, c.c.x, cs * c.c.y);
    const float lm = k.lpa * pll_rcp(c.m);
    const float mi = lm * fmaf(cs, c.c.z, -sn * c.c.w), mq = -lm * fmaf(sn, c.c.z, cs * c.c.w);
    const float Im = fmaf(c.r1, x.I, mi), Qm = fmaf(c.r1, x.Q, mq);
    const float e = coarse_atan2(Qm, Im);
    const float ka = c.m * alpha, kf = c.m * beta, kp = fmaf(0.5f * (c.m + 1.f), kf, ka);
    const float f1 = fmaf(kf, e, df);
    const bool clamped = f1 < (float)k.dfmin || f1 > (float)k.dfmax;
    const float fc = fminf(fmaxf(f1, (float)k.dfmin), (float)k.dfmax);
    const float r2 = fmaf(Im, Im, Qm * Qm);
    const float inv = r2 > 0.f ? pll_rcp(r2) : 0.f;
    const float gI = -Qm * inv, gQ = Im * inv;
    const float ePhi = fmaf(gI, mq, -gQ * mi), eI = gI * c.r1, eQ = gQ * c.r1;
    const float pF = clamped ? 0.f : 1.f, kfe = clamped ? 0.f : kf, kpe = clamped ? ka : kp;
    a[0] = fmaf(kpe, ePhi, 1.f);
    a[1] = fmaf(kpe * half, ePhi, pF * c.m);
    a[2] = kpe * eI;
    a[3] = kpe * eQ;
    a[4] = kfe * ePhi;
    a[5] = fmaf(kfe * half, ePhi, pF);
    a[6] = kfe * eI;
    a[7] = kfe * eQ;
    a[8] = dQ;
    a[9] = half * dQ;
    a[10] = c.rm;
    a[11] = 0.f;
    a[12] = -dI;
    a[13] = half * -dI;
    a[14] = 0.f;
    a[15] = c.rm;
    return make_float4((float)(x.dphi - nx.dphi) + fmaf(c.m, clamped ? fc : df, kpe * e),
                       (float)(x.df - nx.df) + (fc - df), ri + dI - nx.I, rq + dQ - nx.Q);
}

// An affine map of the state, column by column: four matrix columns (the
// images of phase, freq, I and Q), then the vector.
struct AffCols {
    float4 c[5];
};

// Columns of a (without its vector) times v, plus w.
__device__ __forceinline__ float4 aff_mul(const AffCols &a, const float4 &v, const float4 &w) {
    const float4 c0 = a.c[0], c1 = a.c[1], c2 = a.c[2], c3 = a.c[3];
    float4 r;
    r.x = fmaf(c0.x, v.x, fmaf(c1.x, v.y, fmaf(c2.x, v.z, fmaf(c3.x, v.w, w.x))));
    r.y = fmaf(c0.y, v.x, fmaf(c1.y, v.y, fmaf(c2.y, v.z, fmaf(c3.y, v.w, w.y))));
    r.z = fmaf(c0.z, v.x, fmaf(c1.z, v.y, fmaf(c2.z, v.z, fmaf(c3.z, v.w, w.z))));
    r.w = fmaf(c0.w, v.x, fmaf(c1.w, v.y, fmaf(c2.w, v.z, fmaf(c3.w, v.w, w.w))));
    return r;
}

__device__ __forceinline__ float4 aff_apply(const AffCols &a, const float4 &v) { return aff_mul(a, v, a.c[4]); }

// Column `col` of the composition of N maps, the first applied first (the next
// map is loaded while one is applied).
template <int N>
__device__ __forceinline__ float4 aff_chain(const AffCols *a, int col) {
    float4 v = a[0].c[col];
    AffCols m = a[1];
#pragma unroll
    for (int i = 1; i < N; ++i) {
        const AffCols cur = m;
        if (i + 1 < N) m = a[i + 1];
        v = aff_mul(cur, v, col == 4 ? cur.c[4] : make_float4(0.f, 0.f, 0.f, 0.f));
    }
    return v;
}

constexpr int kPllRun = 8;  // segments per run of the scan

struct PllShared {
    AffCols aff[kNewtonThreads];       // the segments' maps (their matrices kept for chord steps)
    AffCols run[kNewtonThreads / kPllRun];  // compositions: runs of 8 segments,
    AffCols warp[kNW];                      // warps,
    AffCols cta[2][kNewtonMaxCluster];      // and CTAs of the cluster (double-buffered across scans)
    float4 coarse[kNewtonThreads];     // CoarseSeg::c of every segment
    float4 dmax[2][kNewtonMaxCluster * kNW];  // every warp's largest corrections (double-buffered)
    SegState first[kNW];               // each warp's first segment start
    SegState next;                     // the next CTA's first segment start
    SegState end;                      // the chunk's end state
    float seg[kPllSeg][kNewtonThreads + 1];  // staged pilot band, then twice the loop phase
    double sum[kNewtonMaxCluster * kNW][2];  // every warp's sums over the block (in CTA 0)
    int badw[kNW];
    int cbad;
};

// d at each segment start from the segments' affine maps in sh.aff (each
// written by its thread): the recurrence over the whole cluster.  The maps are
// composed upwards column by column -- a lane carries one of the five columns
// through a run of 8 segments, then through the warp's 4 runs, the CTA's 8
// warps -- so a composition is 16 multiply-adds in a lane and nothing is
// shuffled; downwards only the vector d is applied.  pb alternates from scan
// to scan; one cluster barrier.  (With whole maps per lane and shuffles, 5 + 3
// + 3 rounds of 20 shuffles and 84 multiply-adds, a scan took 7000 cycles;
// this one ~2500.)
template <class Cluster>
__device__ __forceinline__ float4 pll_scan(Cluster &cl, PllShared &sh, int pb, int crank, int csize) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rn = lane >> 3, col = lane & 7;
    const AffCols *seg = sh.aff + warp * 32;
    AffCols *run = sh.run + warp * (32 / kPllRun);
    __syncwarp();
    if (col < 5) run[rn].c[col] = aff_chain<kPllRun>(seg + rn * kPllRun, col);
    __syncwarp();
    if (lane < 5) sh.warp[warp].c[lane] = aff_chain<32 / kPllRun>(run, lane);
    __syncthreads();
    if (csize > 1) {
        if (warp == 0 && lane < 5) {
            const float4 v = aff_chain<kNW>(sh.warp, lane);
            for (int r = crank + 1; r < csize; ++r) cl.map_shared_rank(&sh.cta[pb][crank], r)->c[lane] = v;
        }
        cl.sync();  // the CTAs before this one have written their maps here
    }
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int r = 0; r < crank; ++r) d = aff_apply(sh.cta[pb][r], d);
#pragma unroll 2
    for (int w = 0; w < warp; ++w) d = aff_apply(sh.warp[w], d);
#pragma unroll
    for (int r = 0; r < 32 / kPllRun - 1; ++r) {
        const float4 v = aff_apply(run[r], d);
        if (r < rn) d = v;
    }
    // inside a run d moves from lane to lane, each applying its own map
    const AffCols own = seg[lane];
#pragma unroll
    for (int i = 1; i < kPllRun; ++i) {
        const float4 v = aff_apply(own, d);
        const float4 u = make_float4(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1),
                                     __shfl_up_sync(0xffffffffu, v.z, 1), __shfl_up_sync(0xffffffffu, v.w, 1));
        if (col == i) d = u;
    }
    __syncwarp();  // the segments' maps have been read
    return d;
}

// The next segment's start state: the next lane's, the next warp's first, or
// (the CTA's last thread) the next CTA's first.
__device__ __forceinline__ SegState pll_next_start(const SegState &x0, const PllShared &sh) {
    SegState nx{__shfl_down_sync(0xffffffffu, x0.dphi, 1), __shfl_down_sync(0xffffffffu, x0.df, 1),
                __shfl_down_sync(0xffffffffu, x0.I, 1), __shfl_down_sync(0xffffffffu, x0.Q, 1)};
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 31) nx = warp < kNW - 1 ? sh.first[warp + 1] : sh.next;
    return nx;
}

// A segment's map for the scan: its matrix (row-major a) and the mismatch of
// its end state x with the next segment's start nx.
__device__ __forceinline__ void pll_put_matrix(AffCols &m, const float (&a)[16]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) m.c[c] = make_float4(a[c], a[4 + c], a[8 + c], a[12 + c]);
}

__device__ __forceinline__ void pll_put_identity(AffCols &m) {
#pragma unroll
    for (int c = 0; c < 5; ++c) m.c[c] = make_float4(c == 0, c == 1, c == 2, c == 3);
}

__device__ __forceinline__ float pll_max(float a, float b) {
    return __uint_as_float(max(__float_as_uint(a), __float_as_uint(b)));
}

__device__ __forceinline__ float4 pll_warp_max(const float4 &v) {
    return make_float4(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v.x))),
                       __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v.y))),
                       __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v.z))),
                       __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v.w))));
}

__device__ __forceinline__ void pll_put_gap(AffCols &m, const SegState &x, const SegState &nx, bool has_next) {
    m.c[4] = has_next ? make_float4((float)(x.dphi - nx.dphi), (float)(x.df - nx.df), x.I - nx.I, x.Q - nx.Q)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
}

// x += d, the frequency kept within `reach` of f0: a step changes it by at most
// pi beta, so a start t steps on cannot be further off.  (An iterate that
// overshoots on noise would run into the frequency clamp, where the map forgets
// its start, and only the consistent prefix would grow, a segment an iteration.)
// A correction that overflowed or is not a number moves nothing: in a start it
// would stay for good (the residuals of a NaN start are NaN), while a finite guess
// gets its exact value once the segments before it have theirs.
__device__ __forceinline__ void pll_move(SegState &x, const float4 &d, double f0, double reach) {
    if (!(fabsf(d.x) + fabsf(d.y) + fabsf(d.z) + fabsf(d.w) < 1e38f)) return;
    x.dphi += (double)d.x;
    x.df = fmin(fmax(x.df + (double)d.y, f0 - reach), f0 + reach);
    x.I += d.z;
    x.Q += d.w;
}

// One channel-block per cluster of `gridDim.x / count` CTAs.  Each CTA stages
// its span of the chunk's pilot band in shared memory, transposed (step i of
// thread j's segment at [i][j], conflict-free), so every sweep reads it from
// there; the output sweep writes twice the loop phase back into the same cells
// and the CTA then writes the L-R products with coalesced stores.
__global__ void __launch_bounds__(kNewtonThreads, 3)
k_pll_newton(const int *__restrict__ list, int count, const SlotBlock *__restrict__ sbt,
             const ChanParams *__restrict__ prm, ChanState *__restrict__ st, float *__restrict__ wk, int W,
             int max_iters) {
    dependency_wait();
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ PllShared sh;
    const int csize = (int)cl.num_blocks();
    const int crank = (int)cl.block_rank();
    const int idx = blockIdx.x / csize;
    if (idx >= count) return;  // uniform per cluster
    const SlotBlock sb = sbt[list[idx]];
    const int n = sb.n_disc;
    if (n <= 0) return;  // uniform per cluster
    // Another CTA's shared memory may be touched once that CTA is known to run:
    // every CTA of the cluster arrives here and waits before the first scan, so
    // the staging and the coarse sums hide the barrier.
    cl.barrier_arrive();
    const ChanParams &cp = prm[sb.slot];
    ChanState &s = st[sb.slot];
    const float *pil = wk + 3 * W + sb.comp_off;
    const float *bpf = wk + 2 * W + sb.comp_off;
    float *lr = wk + 4 * W + sb.comp_off;
    const PllK k = pll_consts(cp, s);
    const float om = 1.f - k.lpa;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tid = (int)threadIdx.x;
    const int g = crank * kNewtonThreads + tid;
    // The segmentation depends on the channel's own block length only, so a
    // channel's trajectory (and every rounding in it) is the same whatever
    // other channels share the launch; the cluster supplies at least one
    // thread per segment.
    SegState start{0.0, 0.0, (float)s.pll_i, (float)s.pll_q};  // the chunk's start state
    bool all_converged = true;
    bool locked = s.locked != 0;  // the loop of the last block, then whether the last chunk's converged at once
    int iters = 0, pb = 0;
    double es = 0.0, pp = 0.0;  // this thread's sums over the block
    for (int c0 = 0; c0 < n; c0 += kPllChunkSteps) {
        const int nc = min(n - c0, kPllChunkSteps);
        const int t0 = c0 + min(nc, g * kPllSeg), t1 = min(c0 + nc, t0 + kPllSeg);
        const bool has_next = t1 < c0 + nc;  // the next thread's segment is not empty
        const int nseg = (nc + kPllSeg - 1) / kPllSeg;
        const int cbase = c0 + min(nc, crank * kNewtonThreads * kPllSeg);
        const int cend = min(c0 + nc, cbase + kNewtonThreads * kPllSeg);
        {
            float v[kPllSeg];
#pragma unroll
            for (int i = 0; i < kPllSeg; ++i) {
                const int t = cbase + tid + i * kNewtonThreads;
                v[i] = t < cend ? __ldg(pil + t) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < kPllSeg; ++i) {
                const int r = tid + i * kNewtonThreads;
                sh.seg[r % kPllSeg][r / kPllSeg] = v[i];
            }
        }
        __syncthreads();
        // ---- the segment's coarse sums ------------------------------------
        CoarseSeg co{make_float4(0.f, 0.f, 0.f, 0.f), 1.f, 0.f, (float)(t1 - t0)};
        {
            uint64_t qr = k.q0 + (uint64_t)t0 * k.qf;
            float C = 0.f, S = 0.f, C2 = 0.f, S2 = 0.f;
#pragma unroll 4
            for (int t = t0; t < t1; ++t) {
                float sn, cs;
                __sincosf(pll_ramp(qr), &sn, &cs);
                qr += k.qf;
                const float p = sh.seg[t - t0][tid];
                C = fmaf(om, C, p * cs);
                S = fmaf(om, S, p * sn);
                C2 += C;
                S2 += S;
                co.rm *= om;
                co.r1 += co.rm;
            }
            if (t0 < t1) co.r1 = __fdividef(co.r1, co.m);
            sh.coarse[tid] = make_float4(C, S, C2, S2);
        }
        // ---- Newton on the coarse map, from the free-running guess ----------
        // The next CTA's first start moves by this CTA's maps applied to its
        // first correction (its own thread adds the same up to float32
        // rounding), so an iteration takes one cluster barrier.
        SegState x0{start.dphi + (double)(t0 - c0) * start.df, start.df, start.I, start.Q};
        const double pi_beta = GPUD_PI * k.beta, reach = (double)(t0 - c0) * pi_beta;
        if (tid == kNewtonThreads - 1)
            sh.next = SegState{start.dphi + (double)(t1 - c0) * start.df, start.df, start.I, start.Q};
        // A loop that a non-finite sample has gone through stays not a number, here
        // as in the serial loop: there is nothing to solve.
        const bool dead = !(isfinite(start.dphi) && isfinite(start.df) && isfinite(start.I) && isfinite(start.Q) &&
                            isfinite(s.pll_phase) && isfinite(s.pll_freq));
        const int ncoarse = dead ? 0 : locked ? kPllCoarse : kPllCoarseFree;
        if (c0 == 0) cl.barrier_wait();  // the arrive above
        for (int it = 0; it < ncoarse; ++it) {
            if (lane == 0) sh.first[warp] = x0;
            __syncthreads();
            const SegState nx = pll_next_start(x0, sh);
            float a[16];
            co.c = sh.coarse[tid];
            const float4 gap = coarse_step(co, k, x0, nx, a);
            if (t0 < t1) {
                pll_put_matrix(sh.aff[tid], a);
                sh.aff[tid].c[4] = has_next ? gap : make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
                pll_put_identity(sh.aff[tid]);
            }
            const float4 d = pll_scan(cl, sh, pb, crank, csize);
            pb ^= 1;
            if (t0 < t1) pll_move(x0, d, start.df, reach);
            if (tid == kNewtonThreads - 1 && it + 1 < ncoarse) {
                SegState y = sh.next;
                pll_move(y, aff_apply(sh.aff[tid], d), start.df, reach + kPllSeg * pi_beta);
                sh.next = y;
            }
        }
        if (g == 0) x0 = start;  // exact
        __syncthreads();         // the coarse iterations have read sh.first
        if (lane == 0) sh.first[warp] = x0;
        if (tid == 0 && crank > 0) *cl.map_shared_rank(&sh.next, crank - 1) = x0;
        cl.sync();
        // ---- Newton on the loop -------------------------------------------
        bool converged = dead, bad = true;
        bool quasi = true;      // the coarse map's Jacobian (uniform in the cluster)
        int sweeps = 0;         // of F with its own Jacobian
        float prev_m0 = 1e30f;  // last iteration's largest phase correction (uniform in the cluster)
        int it = 0;
        for (; it < max_iters && !converged; ++it) {
            const SegState nx = pll_next_start(x0, sh);
            // Close to the solution (the last corrections below 1e-2 rad) the
            // segment Jacobians barely move: they are kept from the last full
            // evaluation (chord steps), which converge as fast as Newton there.
            const bool jac = !quasi && (sweeps < kPllJacSweeps || prev_m0 > 1e-2f);
            if (t0 < t1) {
                PllRun x = pll_begin(x0.dphi, x0.df, x0.I, x0.Q);
                PllEval o;
                uint64_t qr = k.q0 + (uint64_t)t0 * k.qf;
                if (jac) {
                    float a[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) a[i] = i % 5 == 0 ? 1.f : 0.f;
                    for (int t = t0; t < t1; ++t) {
                        pll_step<true>(qr, x, sh.seg[t - t0][tid], k, o);
                        qr += k.qf;
                        mat_push(a, o, om);
                    }
                    pll_put_matrix(sh.aff[tid], a);
                } else {
                    float p = sh.seg[0][tid];
#pragma unroll 2
                    for (int t = t0; t < t1; ++t) {
                        const float pn = sh.seg[min(t - t0 + 1, kPllSeg - 1)][tid];  // one step ahead
                        pll_step<false>(qr, x, p, k, o);
                        qr += k.qf;
                        p = pn;
                    }
                    if (quasi) {
                        float a[16];
                        co.c = sh.coarse[tid];
                        coarse_step(co, k, x0, nx, a);
                        pll_put_matrix(sh.aff[tid], a);
                    }
                }
                pll_put_gap(sh.aff[tid], SegState{x.dphi(), x.df, x.I, x.Q}, nx, has_next);
            } else {
                pll_put_identity(sh.aff[tid]);
            }
            if (jac) ++sweeps;
            const float4 d = pll_scan(cl, sh, pb, crank, csize);
            // ---- update the start state ------------------------------------
            float4 mx = make_float4(0.f, 0.f, 0.f, 0.f);
            bad = false;
            if (t0 < t1) {
                mx = make_float4(fabsf(d.x), fabsf(d.y), fabsf(d.z), fabsf(d.w));
                bad = !(mx.x <= kTolPhase && mx.y <= kTolFreq && mx.z <= kTolIQ && mx.w <= kTolIQ);
                pll_move(x0, d, start.df, reach);
            }
            if (lane == 0) sh.first[warp] = x0;
            if (tid == 0 && crank > 0) *cl.map_shared_rank(&sh.next, crank - 1) = x0;
            // ---- convergence, agreed by every CTA of the cluster -----------
            // (magnitudes compare as their bits, a NaN above all numbers)
            mx = pll_warp_max(mx);
            if (lane < csize) cl.map_shared_rank(&sh.dmax[pb][0], lane)[crank * kNW + warp] = mx;
            cl.sync();  // also publishes the start states for the next iteration's reads
            mx = lane < csize * kNW ? sh.dmax[pb][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane + 32 < csize * kNW) {
                const float4 v = sh.dmax[pb][lane + 32];
                mx = make_float4(pll_max(mx.x, v.x), pll_max(mx.y, v.y), pll_max(mx.z, v.z), pll_max(mx.w, v.w));
            }
            mx = pll_warp_max(mx);
            pb ^= 1;
            converged = mx.x <= kTolPhase && mx.y <= kTolFreq && mx.z <= kTolIQ && mx.w <= kTolIQ;
            // Accepted one iteration early when the next correction is predicted
            // below the tolerance: corrections shrinking at least linearly at rate
            // m0 / prev_m0 leave a next one of m0^2 / prev_m0 (Newton's quadratic
            // rate leaves less), with the other components already near their floor.
            if (!converged && it >= 1 && mx.x <= 1e-5f && mx.x * mx.x <= kTolPhase * prev_m0 && mx.y <= 1e-10f &&
                mx.z <= 1e-6f && mx.w <= 1e-6f)
                converged = true;
            // Or when the corrections no longer shrink and are below the rounding of
            // a step's angle: unlocked loops, where I and Q pass near zero, stay
            // there (2e-8 to 2e-7 rad) and would take every iteration allowed.  What
            // is left is no more than the step's own distance to float64 on noise
            // (1.1e-7 to 1.4e-7 rad rms, 1e-6 at most; 2e-6 to 7e-6 rms where the
            // turns of the phase deviation stayed in the angle).
            if (!converged && mx.x <= kTolAngle && mx.x > 0.25f * prev_m0 && mx.y <= 1e-10f && mx.z <= 1e-6f &&
                mx.w <= 1e-6f)
                converged = true;
            if (it + 1 >= kPllQuasi) quasi = false;
            prev_m0 = mx.x;
        }
        iters = max(iters, it);
        // ---- not converged: the longest consistent prefix is kept ----------
        // Segments before the first one whose start still moved by more than the
        // tolerance form a consistent trajectory from the chunk start; one warp
        // continues the serial loop from the start of the last of them to the chunk
        // end.
        int gstar = INT_MAX;
        if (!converged) {
            int v = bad ? g : INT_MAX;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, off));
            if (lane == 0) sh.badw[warp] = v;
            __syncthreads();
            if (tid == 0) {
                int c = INT_MAX;
                for (int w2 = 0; w2 < kNW; ++w2) c = min(c, sh.badw[w2]);
                sh.cbad = c;
            }
            cl.sync();
            for (int r = 0; r < csize; ++r) gstar = min(gstar, *cl.map_shared_rank(&sh.cbad, r));
            gstar = gstar == INT_MAX ? 0 : max(gstar - 1, 0);  // INT_MAX: none moved past the tolerance in the last iteration
        }
        // ---- outputs: each converged segment again from its start ----------
        PllRun x = pll_begin(x0.dphi, x0.df, x0.I, x0.Q);
        if (t0 < t1) {
            for (int t = t0; t < t1; ++t) {
                const double pt = (double)sh.seg[t - t0][tid];
                pp += pt * pt;
            }
            if (g < gstar) {
                uint64_t qr = k.q0 + (uint64_t)t0 * k.qf;
                float p = sh.seg[0][tid];
#pragma unroll 2
                for (int t = t0; t < t1; ++t) {
                    const float pn = sh.seg[min(t - t0 + 1, kPllSeg - 1)][tid];  // one step ahead
                    PllEval o;
                    pll_step<false>(qr, x, p, k, o);
                    qr += k.qf;
                    es += fabs((double)o.e);
                    sh.seg[t - t0][tid] = pll_twice(qr, x);  // this thread's own cell, already read
                    p = pn;
                }
            }
        }
        // the L-R products of this CTA's output segments, coalesced, eight
        // loads in flight per thread
        __syncthreads();
        const int cout = gstar == INT_MAX ? cend : min(cend, c0 + gstar * kPllSeg);
#pragma unroll
        for (int h = 0; h < kPllSeg; h += 8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int t = cbase + tid + (h + i) * kNewtonThreads;
                v[i] = t < cout ? __ldg(bpf + t) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = tid + (h + i) * kNewtonThreads, t = cbase + r;
                if (t < cout) lr[t] = v[i] * (2.0f * sinpif(sh.seg[r % kPllSeg][r / kPllSeg]));
            }
        }
        // the owner of the chunk's end: the thread holding the last segment, or
        // the warp of the thread at the first inconsistent segment start
        const int owner = converged ? nseg - 1 : gstar;
        if (!converged && (g >> 5) == (owner >> 5)) {
            // Serial loop from the exact start of segment gstar to the chunk
            // end, by the owner's whole warp: the lanes load the pilot band and
            // the L-R band of the next 32 steps (coalesced, one chunk ahead), all
            // of them evaluate the same recurrence (uniform values, so the loop
            // never waits on a load), and lane i keeps step i's L-R product for
            // one coalesced store per 32 steps.
            const int ol = owner & 31;
            PllRun xs = pll_begin(__shfl_sync(0xffffffffu, x.dphi(), ol), __shfl_sync(0xffffffffu, x.df, ol),
                                  __shfl_sync(0xffffffffu, x.I, ol), __shfl_sync(0xffffffffu, x.Q, ol));
            const int ts = __shfl_sync(0xffffffffu, t0, ol), te = c0 + nc;
            double es_w = __shfl_sync(0xffffffffu, es, ol);
            uint64_t qr = k.q0 + (uint64_t)ts * k.qf;
            float pcur = ts + lane < te ? __ldg(pil + ts + lane) : 0.f;
            float bcur = ts + lane < te ? __ldg(bpf + ts + lane) : 0.f;
            for (int s0 = ts; s0 < te; s0 += 32) {
                const int sn = s0 + 32;
                const float pnext = sn + lane < te ? __ldg(pil + sn + lane) : 0.f;
                const float bnext = sn + lane < te ? __ldg(bpf + sn + lane) : 0.f;
                const int cnt = min(32, te - s0);  // uniform in the warp
                float mine = 0.f;
#pragma unroll 4
                for (int i = 0; i < cnt; ++i) {
                    const float pt = __shfl_sync(0xffffffffu, pcur, i);
                    PllEval o;
                    if (i % kPllSeg == 0) xs = pll_begin(xs.dphi(), xs.df, xs.I, xs.Q);
                    pll_step<false>(qr, xs, pt, k, o);
                    qr += k.qf;
                    es_w += fabs((double)o.e);
                    const float th = pll_twice(qr, xs);
                    if (lane == i) mine = th;
                }
                if (lane < cnt) lr[s0 + lane] = bcur * (2.0f * sinpif(mine));
                pcur = pnext;
                bcur = bnext;
            }
            if (lane == ol) {
                x = xs;
                es = es_w;
            }
        }
        if (g == owner)
            for (int r = 0; r < csize; ++r) *cl.map_shared_rank(&sh.end, r) = SegState{x.dphi(), x.df, x.I, x.Q};
        all_converged = all_converged && converged;
        locked = converged && it <= kPllOnce;
        if (c0 + kPllChunkSteps < n) {
            cl.sync();  // the end state is everywhere
            start = sh.end;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        es += __shfl_xor_sync(0xffffffffu, es, off);
        pp += __shfl_xor_sync(0xffffffffu, pp, off);
    }
    if (lane == 0) {
        double *q = cl.map_shared_rank(&sh.sum[0][0], 0) + 2 * (crank * kNW + warp);
        q[0] = es;
        q[1] = pp;
    }
    cl.sync();  // CTA 0 has the end state and every warp's sums; no shared memory of another CTA is touched after this
    if (g != 0) return;
    double es_all = 0.0, pp_all = 0.0;
    for (int r = 0; r < csize; ++r) {
        double a = 0, b = 0;
        for (int w2 = 0; w2 < kNW; ++w2) {
            a += sh.sum[r * kNW + w2][0];
            b += sh.sum[r * kNW + w2][1];
        }
        es_all += a;
        pp_all += b;
    }
    const SegState xe = sh.end;
    pll_finish(s, cp, n, pll_phase_at(k, n, xe.dphi), s.pll_freq + xe.df, (double)xe.I, (double)xe.Q, es_all, pp_all);
    s.pll_path = all_converged ? 1 : 2;
    s.pll_iters = iters;
}

// Sum of the block's composite squared for batch-stereo channels (the
// denominator of their lock test), one CTA per channel, fixed reduction order.
__global__ void __launch_bounds__(256)
k_comp_power(const int *__restrict__ list, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
             ChanState *__restrict__ st, const float *__restrict__ wk) {
    dependency_wait();
    __shared__ double red[256];
    const SlotBlock sb = sbt[list[blockIdx.x]];
    const ChanParams &cp = prm[sb.slot];
    if (!(cp.flags & kChBatchStereo)) return;
    const float *m = wk + sb.comp_off;
    double acc = 0.0;
    for (int q = threadIdx.x; q < sb.n_disc; q += 256) acc += (double)m[q] * (double)m[q];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) st[sb.slot].comp_power = red[0];
}

// WFMStereo.Demod's L-R product with a free-running carrier (demod/fm.go:
// 106-112): lr[q] = bpf[q] * float32(2 cos x_{q+1}), x_k = fl(x_{k-1} + inc),
// inc = 2 pi 38000 / rate, the reference's sequential float64 phase evaluated
// exactly from its binade table.
__global__ void __launch_bounds__(256)
k_free_stereo(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
              const BinadeTable *__restrict__ tabs38, float *__restrict__ wk, int W) {
    dependency_wait();
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const ChanParams &cp = prm[sb.slot];
    const BinadeTable &tab = tabs38[cp.rds_tab];
    const float *bpf = wk + 2 * W + sb.comp_off;
    float *lr = wk + 4 * W + sb.comp_off;
    const int q0 = w.y * 1024;
    for (int q = q0 + threadIdx.x; q < q0 + 1024 && q < sb.n_disc; q += 256)
        lr[q] = bpf[q] * (float)(2.0 * cos(binade_value(tab, (int64_t)q + 1)));
}

// L-R lowpass and L/R matrix when stereo is enabled; otherwise the 15 kHz mono
// fallback filter (its own delay line, advanced only on fallback blocks) duplicated
// to both channels.  WFM (mono) mode always takes the mono filter, one channel.
__global__ void __launch_bounds__(kFirThreads)
k_wfm_out(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
          const ChanState *__restrict__ st, const WfmTaps *__restrict__ taps, const float *__restrict__ wk, int W,
          const float *__restrict__ lr_dl, const float *__restrict__ audio_dl, float *__restrict__ audio) {
    dependency_wait();
    __shared__ float win[padi(kFirOT + kWfmTapsPad) + 8];
    __shared__ float tp[kWfmTapsPad];
    __shared__ float s_out[kFirOT + kFirOT / 32];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const ChanParams &cp = prm[sb.slot];
    const int q0 = w.y * kFirOT;
    if (q0 >= sb.n_disc) return;
    const bool stereo = (cp.mode == 3) && (st[sb.slot].enabled || (cp.flags & kChFreeStereo));
    if (cp.mode == 3 && !stereo && (cp.flags & kChBatchStereo)) {
        // batch decoder not locked: the discriminator output itself on both
        // channels (wfm_batch_stereo.go:43-49)
        const float *m = wk + sb.comp_off;
        float *dst = audio + sb.audio_off;
        for (int q = q0 + threadIdx.x; q < q0 + kFirOT && q < sb.n_disc; q += kFirThreads)
            dst[2 * q] = dst[2 * q + 1] = m[q];
        return;
    }
    const WfmTaps &tb = taps[cp.rds_tab];
    for (int i = threadIdx.x; i < kWfmTapsPad; i += kFirThreads) tp[i] = tb.t[i].x;
    if (stereo) {
        stage_window(win, wk + 4 * W + sb.comp_off, q0, sb.n_disc, lr_dl + cp.wfm_idx * kWfmHist,
                     sb.comp_hist_len);
    } else {
        // The fallback filter's delay line holds composite samples of earlier
        // fallback blocks only; its valid count sits after the 100 samples.
        const float *adl = audio_dl + cp.wfm_idx * kAudioDlStride;
        stage_window(win, wk + sb.comp_off, q0, sb.n_disc, adl, __float_as_int(adl[kWfmHist]));
    }
    __syncthreads();
    const int t = threadIdx.x;
    const int base = 8 * t + kWfmTapsPad;
    float a[8], ring[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) a[r] = 0.f;
#pragma unroll
    for (int j = 1; j < 8; ++j) ring[j] = win[padi(base + j)];
    for (int kb = 0; kb < kWfmTapsPad; kb += 8) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const int k = kb + kk;
            ring[(8 - kk) & 7] = win[padi(base - k)];
            const float h = tp[k];
#pragma unroll
            for (int r = 0; r < 8; ++r) a[r] = fmaf(h, ring[(r - kk + 8) & 7], a[r]);
        }
    }
    // the tile's filter outputs through shared memory (index i + i/32: the
    // stores of a register row and the reads of consecutive outputs are both
    // conflict-free), then coalesced reads of L+R and stores of (L, R) pairs
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = 8 * t + r;
        s_out[i + (i >> 5)] = a[r];
    }
    __syncthreads();
    float *dst = audio + sb.audio_off;
    const int nq = min(kFirOT, sb.n_disc - q0);
    if (cp.mode == 2) {
        for (int i = t; i < nq; i += kFirThreads) dst[q0 + i] = s_out[i + (i >> 5)];
    } else if (stereo) {
        const float *lpr = wk + 1 * W + sb.comp_off;
        float2 *d2 = reinterpret_cast<float2 *>(dst);
        for (int i = t; i < nq; i += kFirThreads) {
            const float v = s_out[i + (i >> 5)], l = lpr[q0 + i];
            d2[q0 + i] = make_float2(0.5f * (l + v), 0.5f * (l - v));
        }
    } else {
        float2 *d2 = reinterpret_cast<float2 *>(dst);
        for (int i = t; i < nq; i += kFirThreads) {
            const float v = s_out[i + (i >> 5)];
            d2[q0 + i] = make_float2(v, v);
        }
    }
}

// RDS baseband (fm.go:143-163 / 234-271) over the continuous discriminator
// stream: cplx[g] = disc[g] * exp(j x_{g+1}) with x the exact sequential
// float64 FreqShift phase, a 101-tap lowpass accumulated in float64 in the
// reference's order (separate multiply and add, as Go's amd64 code does), and
// every Dr-th stream sample kept.
constexpr int kRdsOT = 128;     // RDS outputs per CTA (one per thread)
constexpr int kRdsThreads = 128;

// Index of the binade entry covering stream index k.
__device__ __forceinline__ int binade_find(const BinadeTable &t, int64_t k) {
    int lo = 0, hi = t.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (t.e[mid].k_start <= k) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// RDS baseband (demod/fm.go:143-163, 234-271): the composite shifted by the
// reference's float64 FreqShift phase (exact values from the binade table),
// 101-tap float64 low-pass evaluated at the kept outputs only.  Staging: each
// thread takes a contiguous run of composite samples, evaluates sin/cos of
// the exact phase once at the run start (and at any binade start inside it)
// and advances by the exact in-binade step with a float64 rotation
// (relative error < 1e-14 over a run, far below the float32 the shifted
// samples are stored in).
__global__ void __launch_bounds__(kRdsThreads)
k_rds(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
      const ChanState *__restrict__ st, const WfmTaps *__restrict__ taps, const BinadeTable *__restrict__ tabs,
      const float *__restrict__ wk, const float2 *__restrict__ rds_dl, float2 *__restrict__ rds_out) {
    dependency_wait();
    extern __shared__ float2 cpl[];
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const int r0 = w.y * kRdsOT;
    if (r0 >= sb.n_rds) return;
    const ChanParams &cp = prm[sb.slot];
    const int dr = cp.rds_dr;
    const int r1 = min(r0 + kRdsOT, sb.n_rds);
    const int qlo = sb.rds_first + r0 * dr - (kWfmTaps - 1);
    const int qhi = sb.rds_first + (r1 - 1) * dr;
    const int span = qhi - qlo + 1;
    const ChanState &s = st[sb.slot];
    const int64_t c0 = s.rds_count;
    const BinadeTable &tab = tabs[cp.rds_tab];
    const float *comp = wk + sb.comp_off;
    const float2 *dl = rds_dl + cp.wfm_idx * kWfmHist;
    const int per = (span + kRdsThreads - 1) / kRdsThreads;
    const int i0 = min(span, (int)threadIdx.x * per), i1 = min(span, i0 + per);
    int ent = -1;
    int64_t next_k = 0;
    double cs = 0.0, sn = 0.0, wc = 1.0, ws = 0.0;
    for (int i = i0; i < i1; ++i) {
        const int q = qlo + i;
        float2 v = make_float2(0.f, 0.f);
        if (q >= 0) {
            const int64_t k = c0 + q + 1;  // phase index: incremented before use (freqshift.go:13-15)
            if (ent < 0 || k >= next_k) {
                ent = binade_find(tab, k);
                const BinadeEntry &be = tab.e[ent];
                next_k = ent + 1 < tab.count ? tab.e[ent + 1].k_start : INT64_MAX;
                sincos(be.x_start + (double)(k - be.k_start) * be.q, &sn, &cs);
                sincos(be.q, &ws, &wc);
            } else {
                const double c1 = cs * wc - sn * ws;
                sn = sn * wc + cs * ws;
                cs = c1;
            }
            const double b = (double)comp[q];
            v = make_float2((float)(b * cs), (float)(b * sn));
        } else if (q >= -s.rds_hist_len) {
            v = dl[kWfmHist + q];
        }
        cpl[i + (i >> 4)] = v;
    }
    __syncthreads();
    // outputs dr samples apart read through one pad slot every 16: the lanes'
    // addresses fall in distinct banks
    const WfmTaps &tb = taps[cp.rds_tab];
    for (int r = r0 + threadIdx.x; r < r1; r += kRdsThreads) {
        const int qr = sb.rds_first + r * dr;
        const int li = qr - qlo;
        double ar = 0.0, ai = 0.0;
        for (int k = 0; k < kWfmTaps; ++k) {
            const int c = li - k;
            const float2 v = cpl[c + (c >> 4)];
            ar = __dadd_rn(ar, __dmul_rn((double)v.x, tb.rds[k]));
            ai = __dadd_rn(ai, __dmul_rn((double)v.y, tb.rds[k]));
        }
        rds_out[sb.rds_off + r] = make_float2((float)ar, (float)ai);
    }
}

// ===========================================================================
// Per-slot state carry, one CTA per slot, after every other kernel.
// ===========================================================================
__device__ void shift_delay_line(float *dl, const float *__restrict__ src, int n) {
    // dl: 100 floats oldest-first; append src[0..n) and keep the last 100.
    __shared__ float tmp[kWfmHist];
    for (int i = threadIdx.x; i < kWfmHist; i += blockDim.x) {
        int g = n + i - kWfmHist;  // index into (dl ++ src) shifted so dl occupies [-100, 0)
        tmp[i] = g >= 0 ? src[g] : dl[kWfmHist + g];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kWfmHist; i += blockDim.x) dl[i] = tmp[i];
    __syncthreads();
}

// Front half: everything the next block's extraction, demod, stereo FIR bank
// and RDS read (extraction history and NCO phase, discriminator bridge,
// composite delay line, RDS stream history).  Runs right after those stages,
// so the next block's front half can overlap this block's PLL.
__global__ void __launch_bounds__(128)
k_post_front(const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm, ChanState *__restrict__ st,
             const float2 *__restrict__ ext, const float *__restrict__ wk, float *__restrict__ comp_dl,
             float2 *__restrict__ rds_dl, const BinadeTable *__restrict__ tabs, float2 *__restrict__ d1hist,
             DevResult *__restrict__ res) {
    dependency_wait();
    const SlotBlock sb = sbt[blockIdx.x];
    const ChanParams &cp = prm[sb.slot];
    ChanState &s = st[sb.slot];
    if (cp.d1 > 1 && sb.n_out > 0) {
        // pre-demod decimator history: the last 100 extraction outputs
        __shared__ float2 dtmp[kWfmHist];
        float2 *dh = d1hist + (int64_t)sb.slot * kWfmHist;
        for (int i = threadIdx.x; i < kWfmHist; i += blockDim.x) {
            const int g = sb.n_out + i - kWfmHist;
            dtmp[i] = g >= 0 ? ext[sb.ext_off + g] : dh[kWfmHist + g];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < kWfmHist; i += blockDim.x) dh[i] = dtmp[i];
        __syncthreads();
    }
    if (cp.wfm_idx >= 0 && sb.n_disc > 0) {
        const float *comp = wk + sb.comp_off;
        // RDS shifted history: the last 100 values of cplx over the stream
        if (cp.flags & 2) {
            __shared__ float2 rtmp[kWfmHist];
            const BinadeTable &tab = tabs[cp.rds_tab];
            float2 *dl = rds_dl + cp.wfm_idx * kWfmHist;
            const int64_t c0 = s.rds_count;
            for (int i = threadIdx.x; i < kWfmHist; i += blockDim.x) {
                int q = sb.n_disc + i - kWfmHist;
                float2 v = make_float2(0.f, 0.f);
                if (q >= 0) {
                    double ph = binade_value(tab, c0 + q + 1);
                    double sn, cs;
                    sincos(ph, &sn, &cs);
                    double b = (double)comp[q];
                    v = make_float2((float)(b * cs), (float)(b * sn));
                } else {
                    v = dl[kWfmHist + q];
                }
                rtmp[i] = v;
            }
            __syncthreads();
            for (int i = threadIdx.x; i < kWfmHist; i += blockDim.x) dl[i] = rtmp[i];
            __syncthreads();
        }
        shift_delay_line(comp_dl + cp.wfm_idx * kWfmHist, comp, sb.n_disc);
    }
    if (threadIdx.x == 0) {
        if (sb.n_dem > 0) {
            s.last_iq = ext[sb.dem_off + sb.n_dem - 1];
            s.has_last = 1;
        }
        if (cp.wfm_idx >= 0 && sb.n_disc > 0) {
            s.rds_count += sb.n_disc;
            s.rds_hist_len = (int)min((int64_t)kWfmHist, s.rds_count);
        }
    }
}

// Extraction state of a block, carried as soon as the block's extraction
// kernels are done (the next block's extraction waits only for this): the
// last min(T-1, H+n) samples of (history ++ shifted block) into the other
// history buffer, and the NCO phase advanced by the block.
__global__ void __launch_bounds__(128)
k_post_extract(const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm, ChanState *__restrict__ st,
               const float2 *__restrict__ x, int n, float2 *__restrict__ hist_arena, DevResult *__restrict__ res) {
    dependency_wait();
    const SlotBlock sb = sbt[blockIdx.x];
    const ChanParams &cp = prm[sb.slot];
    ChanState &s = st[sb.slot];
    const uint64_t u0 = s.nco_q;
    const int keep = cp.ntaps - 1;
    const int H = sb.hist_len;
    const int newH = min(keep, H + n);
    const float2 *hold = hist_arena + cp.hist_off + sb.hist_sel * cp.hcap;
    float2 *hnew = hist_arena + cp.hist_off + (1 - sb.hist_sel) * cp.hcap;
    for (int q = threadIdx.x; q < newH; q += blockDim.x) {
        int g = H + n - newH + q;
        hnew[q] = g < H ? hold[g] : cmulf(__ldg(x + (g - H)), q64_phasor(u0 + (uint64_t)(g - H) * cp.inc_q));
    }
    __syncthreads();  // every thread has read the block-start phase
    if (threadIdx.x == 0) {
        s.nco_q = u0 + (uint64_t)n * cp.inc_q;
        res[sb.res_idx].nco_phase = q64_to_rad(s.nco_q);
    }
}

// Back half: the L-R and mono-fallback delay lines and the block's lock
// flags, margins and PLL solver info, after the PLL and the stereo output.
__global__ void __launch_bounds__(128)
k_post_back(const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm, ChanState *__restrict__ st,
            const float *__restrict__ wk, int W, float *__restrict__ lr_dl, float *__restrict__ audio_dl,
            DevResult *__restrict__ res) {
    dependency_wait();
    const SlotBlock sb = sbt[blockIdx.x];
    const ChanParams &cp = prm[sb.slot];
    ChanState &s = st[sb.slot];
    if (cp.wfm_idx >= 0 && sb.n_disc > 0) {
        const float *comp = wk + sb.comp_off;
        const bool fallback = (cp.mode == 2) || !s.enabled;
        if (fallback) {
            float *adl = audio_dl + cp.wfm_idx * kAudioDlStride;
            int valid = __float_as_int(adl[kWfmHist]);
            shift_delay_line(adl, comp, sb.n_disc);
            if (threadIdx.x == 0) adl[kWfmHist] = __int_as_float(min(kWfmHist, valid + sb.n_disc));
            __syncthreads();
        }
        if (cp.mode == 3) shift_delay_line(lr_dl + cp.wfm_idx * kWfmHist, wk + 4 * W + sb.comp_off, sb.n_disc);
    }
    if (threadIdx.x == 0) {
        DevResult &o = res[sb.res_idx];
        o.flags = (cp.mode == 3 && sb.n_disc > 0) ? ((s.locked ? 1 : 0) | (s.enabled ? 2 : 0))
                                                  : (s.enabled ? 2 : 0);
        o.coherence = s.coherence;
        o.pilot_hz = s.pilot_hz;
        o.err_avg = s.last_err_avg;
        o.status = (cp.mode == 3 && sb.n_disc > 0) ? s.pll_path : 0;
        o.pll_iters = s.pll_iters;
    }
}

// ===========================================================================
// 48 kHz audio back end (recorder/streamer.go:1408-1470, 569-575)
// ===========================================================================
// Resampling: output o of the block sits at the resampler's phase position
// t0 + o*M: it is produced after consuming c = floor((t0+o*M)/L) inputs, at
// arm (t0+o*M) - c*L, over the last K consumed samples (earlier blocks'
// samples from the carried delay line) -- the closed form of
// Resampler.Process (dsp/resample.go:105-153); the host mirrors the phase
// counter, including that method's exits, so every output is independent and
// k_audio48_rs computes one per thread over the whole grid.  The float64 dot
// products keep the reference's separate multiply and add.
// k_audio48_out, one CTA per channel: de-emphasis y = a*y + (1-a)*x (float64),
// a first-order recurrence -- each thread takes a contiguous run of outputs,
// the runs' affine maps are scanned across the CTA and each run is replayed
// from its start -- then the WFM gain 0.35 and s16le: int16(clip(s * 32767)),
// truncating; it also carries the delay lines and the de-emphasis state.
constexpr int kAudThreads = 256;
constexpr int kAudOT = 256;       // resampled frames per CTA where each thread takes one
constexpr int kAudWin = 2600;     // most staged input frames of a tile
constexpr int kAudBank = 4096;    // most staged bank coefficients (doubles)
constexpr int kAudLive = 160;     // fewest busy threads of a tile with several outputs per thread

// Tile of one resampler ratio: outputs o, o+L, o+2L, o+3L stand at one phase, so
// a thread takes r = 4 of them and reads each of its arm's coefficients once,
// unless the tile's input window then leaves too few threads busy (M/L above
// about 3: 40 stereo channels at 312.5 kHz 14.0 us with r = 1, 16.4 with 2,
// 24.5 with 4 and 96 threads).  r = 0: arms or window too large for shared
// memory (one output per thread from global memory).
struct AudTile {
    int r, ot, smem;
};
__host__ __device__ inline int aud_window(int ot, int L, int M, int K) {
    return (int)((int64_t)(ot - 1) * M / L) + K + 2;
}
__host__ __device__ inline AudTile aud_tile(int L, int M, int K, int C) {
    if (L == M || (int64_t)L * K > kAudBank) return {0, kAudOT, 0};
    for (int r = 4; r >= 1; r -= 3) {
        // one output per thread: whole warps; four: whole blocks of 4L
        const int unit = r > 1 ? r * L : 32;
        // most outputs whose window fits, without a search: every thread of a CTA
        // works this out (a search down from 1024 in steps of 4 L took 240 kS/s, L = 1,
        // from 3.7 to 20.7 us)
        const int fit = ((kAudWin - K - 1) * L - 1) / M + 1;
        const int ot = (fit < kAudThreads * r ? fit : kAudThreads * r) / unit * unit;
        if (ot < kAudLive * r) continue;
        return {r, ot, ((L * K + 1) & ~1) * 8 + C * aud_window(ot, L, M, K) * 4};
    }
    return {0, kAudOT, 0};
}

// R outputs of a staged tile, C channels: the products and sums of one output
// in its arm's order.
template <int R, int C>
__device__ __forceinline__ void aud_dot(const double *arm, const float *x, int M, int K, double (&acc)[R][C]) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < C; ++c) acc[r][c] = 0.0;
#pragma unroll 11
    for (int k = 0; k < K; ++k) {
        const double h = arm[k];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float *p = x + (r * M - k) * C;
            if constexpr (C == 2) {
                const float2 v = *reinterpret_cast<const float2 *>(p);
                acc[r][0] = __dadd_rn(acc[r][0], __dmul_rn((double)v.x, h));
                acc[r][1] = __dadd_rn(acc[r][1], __dmul_rn((double)v.y, h));
            } else {
                acc[r][0] = __dadd_rn(acc[r][0], __dmul_rn((double)*p, h));
            }
        }
    }
}

template <int R, int C>
__device__ __forceinline__ void aud_outputs(const SlotBlock &sb, int oa, int ob, int ot, const double *s_bank,
                                            const float *s_in, int ph0, int L, int M, int K,
                                            float *__restrict__ rs_out) {
    // thread i: phase slot i % L of block i / L, outputs oa + (i/L)*R*L + i%L + r*L
    const int i = (int)threadIdx.x, o0 = oa + (R > 1 ? (i / L) * (R * L) + i % L : i);
    if (i * R >= ot || o0 >= ob) return;
    const unsigned t = (unsigned)ph0 + (unsigned)(o0 - oa) * (unsigned)M, cc = t / (unsigned)L;
    double acc[R][C];
    aud_dot<R, C>(s_bank + (int)(t - cc * (unsigned)L) * K, s_in + ((int)cc + K - 1) * C, M, K, acc);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int o = o0 + r * L;
        if (o >= ob) break;
        float *dst = rs_out + sb.pcm_off + o * C;
        dst[0] = (float)acc[r][0];
        if constexpr (C == 2) dst[1] = (float)acc[r][1];
    }
}

// Bound by its latencies (the channel's tables, then the arms and the window into
// shared memory, then the chains of 33 sums): four outputs per thread stage the
// arms a quarter as often, load a coefficient once for four products, keep four
// chains in flight and fit 120 narrow channels in about one wave of CTAs.
// Measured, one output per thread before and now: 120 mono channels 20.9 ->
// 12.8 us, 512 channels of all modes 26.0 -> 19.6, 40 stereo ones (r = 1) 14.0 ->
// 13.6 (the two last with 8 bytes reserved for a float of the window: 20.5, 14.0).
// (A window staged in float64 spares 33 conversions per output but strides of M/L
// doubles conflict in the banks: 40 stereo channels 21.7 us.)
__global__ void __launch_bounds__(kAudThreads)
k_audio48_rs(const int2 *__restrict__ work, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
             const RsBank *__restrict__ banks, const AudState *__restrict__ aud, const float *__restrict__ audio,
             float *__restrict__ rs_out) {
    dependency_wait();
    extern __shared__ __align__(16) double s_aud[];  // arms (L*K, rounded to even) | window (win x C)
    const int2 w = work[blockIdx.x];
    const SlotBlock sb = sbt[w.x];
    const ChanParams &cp = prm[sb.slot];
    const AudState &as = aud[sb.slot];
    const RsBank bk = banks[cp.rs_bank];
    const int C = cp.aud_ch, L = bk.L, M = bk.M, K = bk.K;
    const AudTile at = aud_tile(L, M, K, C);
    const int oa = w.y * at.ot, ob = min(sb.rs_nout, oa + at.ot);  // this CTA's outputs
    if (oa >= ob) return;
    const float *in = audio + sb.audio_off;
    if (L == M) {
        for (int o = oa + (int)threadIdx.x; o < ob; o += kAudThreads)
            for (int c = 0; c < C; ++c) rs_out[sb.pcm_off + o * C + c] = in[o * C + c];
        return;
    }
    if (at.r) {
        // inputs consumed before the tile's first output, and its phase
        const int64_t Ta = (int64_t)sb.rs_t0 + (int64_t)oa * M, ca = Ta / L;
        const int ph0 = (int)(Ta - ca * L);
        const int win = (int)(((int64_t)ph0 + (int64_t)(ob - 1 - oa) * M) / L) + K;  // from input ca - K on
        float *s_in = reinterpret_cast<float *>(s_aud + ((L * K + 1) & ~1));
        constexpr int U = 8;  // loads in flight per thread
        const int nb = L * K;
        for (int i0 = threadIdx.x; i0 < nb; i0 += U * kAudThreads) {
            double v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * kAudThreads;
                v[u] = i < nb ? bk.arm[i] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * kAudThreads;
                if (i < nb) s_aud[i] = v[u];
            }
        }
        const int64_t g0 = (ca - K) * C;  // element e of the window is in[g0 + e], or carried
        for (int i0 = threadIdx.x; i0 < win * C; i0 += U * kAudThreads) {
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * kAudThreads;
                const int64_t g = g0 + i;
                v[u] = 0.f;
                if (i < win * C) v[u] = g >= 0 ? in[g] : C == 2 ? as.dl[i & 1][-1 - (g >> 1)] : as.dl[0][-1 - g];
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * kAudThreads;
                if (i < win * C) s_in[i] = v[u];
            }
        }
        __syncthreads();
#define GPUD_AUD(R)                                                                                  \
    if (C == 2) aud_outputs<R, 2>(sb, oa, ob, at.ot, s_aud, s_in, ph0, L, M, K, rs_out);             \
    else aud_outputs<R, 1>(sb, oa, ob, at.ot, s_aud, s_in, ph0, L, M, K, rs_out);
        if (at.r == 4) {
            GPUD_AUD(4)
        } else {
            GPUD_AUD(1)
        }
#undef GPUD_AUD
        return;
    }
    for (int o = oa + (int)threadIdx.x; o < ob; o += kAudThreads) {
        const int64_t T = (int64_t)sb.rs_t0 + (int64_t)o * M;
        const int64_t cc = T / L;  // T >= 0
        const int ph = (int)(T - cc * L);
        double acc0 = 0.0, acc1 = 0.0;
        const double *arm = bk.arm + ph * K;
        for (int k = 0; k < K; ++k) {
            const int64_t i = cc - 1 - k;
            const double h = arm[k];
            const float v0 = i >= 0 ? in[i * C] : as.dl[0][-1 - i];
            acc0 = __dadd_rn(acc0, __dmul_rn((double)v0, h));
            if (C == 2) {
                const float v1 = i >= 0 ? in[i * 2 + 1] : as.dl[1][-1 - i];
                acc1 = __dadd_rn(acc1, __dmul_rn((double)v1, h));
            }
        }
        float *dst = rs_out + sb.pcm_off + o * C;
        dst[0] = (float)acc0;
        if (C == 2) dst[1] = (float)acc1;
    }
}

constexpr int kAudOutThreads = 1024;  // one CTA per channel: short serial runs
constexpr int kAudOutStage = 16384;   // resampled samples of a channel staged in shared memory (64 KB)

__global__ void __launch_bounds__(kAudOutThreads)
k_audio48_out(const int *__restrict__ list, const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
              const RsBank *__restrict__ banks, AudState *__restrict__ aud, const float *__restrict__ audio,
              const float *__restrict__ rs_out, int16_t *__restrict__ pcm) {
    dependency_wait();
    constexpr int kWarps = kAudOutThreads / 32;
    __shared__ double s_wa[kWarps], s_wb[2][kWarps];  // warp totals, then exclusive warp prefixes
    extern __shared__ float s_rs[];  // the channel's resampled block (when it fits), then its output samples
    const SlotBlock sb = sbt[list[blockIdx.x]];
    const ChanParams &cp = prm[sb.slot];
    AudState &as = aud[sb.slot];
    const int C = cp.aud_ch;
    const int n = sb.rs_frames, nout = sb.rs_nout;
    if (n <= 0) return;
    const RsBank &bk = banks[cp.rs_bank];
    // each thread takes a run of consecutive frames: the block is staged with
    // coalesced loads and the PCM written back coalesced
    const bool staged = nout * C <= kAudOutStage;
    if (staged) {
        const float *src = rs_out + sb.pcm_off;
        for (int i = threadIdx.x; i < nout * C; i += kAudOutThreads) s_rs[i] = src[i];
        __syncthreads();
    }
    const float *r = staged ? s_rs : rs_out + sb.pcm_off;
    const int per = (nout + kAudOutThreads - 1) / kAudOutThreads;
    const int o0 = min(nout, (int)threadIdx.x * per), o1 = min(nout, o0 + per);
    const bool wfm = cp.mode == 2 || cp.mode == 3;
    const double a = cp.deemph_a;
    const bool de = wfm && a > 0.0;
    double y0 = as.y[0], y1 = as.y[1];
    if (de) {
        // this run's map y_end = A*y_start + B, per channel
        double A = 1.0, B0 = 0.0, B1 = 0.0;
        for (int o = o0; o < o1; ++o) {
            A = __dmul_rn(A, a);
            B0 = __dadd_rn(__dmul_rn(a, B0), __dmul_rn(1.0 - a, (double)r[o * C]));
            if (C == 2) B1 = __dadd_rn(__dmul_rn(a, B1), __dmul_rn(1.0 - a, (double)r[o * 2 + 1]));
        }
        // inclusive scan of the maps across the warp (a later run applied
        // after an earlier one), then across the warps' totals
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double pa = __shfl_up_sync(0xffffffffu, A, d);
            const double pb0 = __shfl_up_sync(0xffffffffu, B0, d);
            const double pb1 = __shfl_up_sync(0xffffffffu, B1, d);
            if (lane >= d) {
                B0 = A * pb0 + B0;
                B1 = A * pb1 + B1;
                A = A * pa;
            }
        }
        if (lane == 31) {
            s_wa[warp] = A;
            s_wb[0][warp] = B0;
            s_wb[1][warp] = B1;
        }
        __syncthreads();
        if (warp == 0) {
            double wa = lane < kWarps ? s_wa[lane] : 1.0;
            double wb0 = lane < kWarps ? s_wb[0][lane] : 0.0, wb1 = lane < kWarps ? s_wb[1][lane] : 0.0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const double pa = __shfl_up_sync(0xffffffffu, wa, d);
                const double pb0 = __shfl_up_sync(0xffffffffu, wb0, d);
                const double pb1 = __shfl_up_sync(0xffffffffu, wb1, d);
                if (lane >= d) {
                    wb0 = wa * pb0 + wb0;
                    wb1 = wa * pb1 + wb1;
                    wa = wa * pa;
                }
            }
            // exclusive: the warps before this one
            const double ea = __shfl_up_sync(0xffffffffu, wa, 1);
            const double eb0 = __shfl_up_sync(0xffffffffu, wb0, 1);
            const double eb1 = __shfl_up_sync(0xffffffffu, wb1, 1);
            if (lane < kWarps) {
                s_wa[lane] = lane ? ea : 1.0;
                s_wb[0][lane] = lane ? eb0 : 0.0;
                s_wb[1][lane] = lane ? eb1 : 0.0;
            }
        }
        __syncthreads();
        // this run's start: the warps before it, then the lanes before it
        const double la = __shfl_up_sync(0xffffffffu, A, 1);
        const double lb0 = __shfl_up_sync(0xffffffffu, B0, 1);
        const double lb1 = __shfl_up_sync(0xffffffffu, B1, 1);
        const double ws0 = s_wa[warp] * as.y[0] + s_wb[0][warp];
        const double ws1 = s_wa[warp] * as.y[1] + s_wb[1][warp];
        y0 = lane ? la * ws0 + lb0 : ws0;
        y1 = lane ? la * ws1 + lb1 : ws1;
    }
    for (int o = o0; o < o1; ++o) {
        for (int c = 0; c < C; ++c) {
            float s = r[o * C + c];
            if (de) {
                double &y = c == 0 ? y0 : y1;
                y = __dadd_rn(__dmul_rn(a, y), __dmul_rn(1.0 - a, (double)s));
                s = (float)y;
            }
            if (wfm) s = s * 0.35f;
            if (staged) {
                s_rs[o * C + c] = s;  // this thread's own cell, already read
            } else if (cp.flags & kChPcmF32) {
                reinterpret_cast<float *>(pcm + sb.pcm_off)[o * C + c] = s;
            } else {
                float v = s * 32767.0f;
                v = fminf(fmaxf(v, -32768.0f), 32767.0f);
                pcm[sb.pcm_off + o * C + c] = (int16_t)v;
            }
        }
    }
    if (staged) {
        __syncthreads();
        if (cp.flags & kChPcmF32) {
            float *dst = reinterpret_cast<float *>(pcm + sb.pcm_off);
            for (int i = threadIdx.x; i < nout * C; i += kAudOutThreads) dst[i] = s_rs[i];
        } else {
            for (int i = threadIdx.x; i < nout * C; i += kAudOutThreads) {
                float v = s_rs[i] * 32767.0f;
                v = fminf(fmaxf(v, -32768.0f), 32767.0f);
                pcm[sb.pcm_off + i] = (int16_t)v;
            }
        }
    }
    __syncthreads();  // every read of the old state is done
    // carried state: the last K consumed samples, newest first; the last y
    const int c = threadIdx.x / kRsTaps, k = threadIdx.x % kRsTaps;
    const bool mine = bk.L != bk.M && threadIdx.x < 2 * kRsTaps && c < C;
    float v = 0.f;
    if (mine) {
        const int i = n - 1 - k;
        v = i >= 0 ? audio[sb.audio_off + i * C + c] : as.dl[c][-1 - i];
    }
    __syncthreads();  // the shifted entries are read before any is overwritten
    if (mine) as.dl[c][k] = v;
    if (de && nout > 0 && o1 == nout && o0 < o1) {
        as.y[0] = y0;
        as.y[1] = y1;
    }
}

// ===========================================================================
// launch helpers (host)
// ===========================================================================
template <int L>
static cudaError_t launch_dense_L(int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                                  const ChanParams *prm, const ChanState *st, const float2 *x, int n,
                                  const float2 *hist, const float *taps, float2 *ext) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_dense<L>, 220 * 1024);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_extract_dense<L>, dim3((unsigned)grid), kDenseThreads, (size_t)smem, sm, work, sbt,
                            prm, st, x, n, hist, taps, ext);
}

cudaError_t launch_extract_dense_any(int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                                     const ChanParams *prm, const ChanState *st, const float2 *x, int n,
                                     const float2 *hist, const float *taps, float2 *ext) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_dense_any, 220 * 1024);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_extract_dense_any, dim3((unsigned)grid), kDenseThreads, (size_t)smem, sm, work, sbt,
                            prm, st, x, n, hist, taps, ext);
}

cudaError_t launch_extract_dense(int L, int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                                 const ChanParams *prm, const ChanState *st, const float2 *x, int n,
                                 const float2 *hist, const float *taps, float2 *ext) {
    switch (L) {
#define GPUD_CASE(LL) \
    case LL: return launch_dense_L<LL>(grid, smem, sm, work, sbt, prm, st, x, n, hist, taps, ext);
        GPUD_CASE(2) GPUD_CASE(3) GPUD_CASE(4) GPUD_CASE(5) GPUD_CASE(6) GPUD_CASE(7) GPUD_CASE(8)
        GPUD_CASE(9) GPUD_CASE(10) GPUD_CASE(11) GPUD_CASE(12) GPUD_CASE(13) GPUD_CASE(14)
        GPUD_CASE(15) GPUD_CASE(16)
#undef GPUD_CASE
    default: return cudaErrorInvalidValue;
    }
}

template <int L, int NG>
static cudaError_t launch_dense_pipe_LG(int ntiles, int grid, int pmax, cudaStream_t sm, const int2 *work,
                                        const SlotBlock *sbt, const ChanParams *prm, const ChanState *st,
                                        const float2 *x, int n, const float2 *hist, const float *taps, float2 *ext,
                                        unsigned *fault) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_dense_pipe<L, NG>, 220 * 1024);
    if (e != cudaSuccess) return e;
    const int smem = pipe_layout(pmax, L, NG).bytes;
    return launch_dependent(k_extract_dense_pipe<L, NG>, dim3((unsigned)grid), kPipeThreads, (size_t)smem, sm,
                            work, ntiles, pmax, sbt, prm, st, x, n, hist, taps, ext, fault);
}

// Consumer groups of the pipelined dense form for a class whose channels have
// at most P phases (two when both groups' Z fit beside the raw span), or 0
// when it does not fit in cap bytes or needs more rotation-table rounds than
// the producer warp fills.
int dense_pipe_groups_host(int P, int L, int cap) {
    const int total = P * (kDenseOT + L - 1);
    if (total <= kPipeMaxRounds * 32 * (kPipeCW / 2) && pipe_layout(P, L, 2).bytes <= cap) return 2;
    if (total <= kPipeMaxRounds * 32 * kPipeCW && pipe_layout(P, L, 1).bytes <= cap) return 1;
    return 0;
}

cudaError_t launch_extract_dense_pipe(int L, int ng, int ntiles, int grid, int pmax, cudaStream_t sm,
                                      const int2 *work, const SlotBlock *sbt, const ChanParams *prm,
                                      const ChanState *st, const float2 *x, int n, const float2 *hist,
                                      const float *taps, float2 *ext, unsigned *fault) {
    if (((uintptr_t)x & 15) != 0 || (ng != 1 && ng != 2)) return cudaErrorInvalidValue;
    switch (L * 4 + ng) {
#define GPUD_CASE(LL)                                                                                              \
    case LL * 4 + 1:                                                                                               \
        return launch_dense_pipe_LG<LL, 1>(ntiles, grid, pmax, sm, work, sbt, prm, st, x, n, hist, taps, ext,     \
                                           fault);                                                                 \
    case LL * 4 + 2:                                                                                               \
        return launch_dense_pipe_LG<LL, 2>(ntiles, grid, pmax, sm, work, sbt, prm, st, x, n, hist, taps, ext,     \
                                           fault);
        GPUD_CASE(2) GPUD_CASE(3) GPUD_CASE(4) GPUD_CASE(5) GPUD_CASE(6) GPUD_CASE(7) GPUD_CASE(8)
        GPUD_CASE(9) GPUD_CASE(10) GPUD_CASE(11) GPUD_CASE(12) GPUD_CASE(13) GPUD_CASE(14)
        GPUD_CASE(15) GPUD_CASE(16)
#undef GPUD_CASE
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_extract_wide(int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                                const ChanParams *prm, const ChanState *st, const float2 *x, int n,
                                const float2 *hist, const float *taps, float2 *ext) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_wide, 64 * 1024);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_extract_wide, dim3((unsigned)grid), 256, (size_t)smem, sm, work, sbt, prm, st, x, n,
                            hist, taps, ext);
}

cudaError_t launch_extract_group(int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                                 const ChanParams *prm, const ChanState *st, const float2 *x, int n,
                                 const float2 *hist, const float *taps, float2 *ext) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_group, 220 * 1024);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_extract_group, dim3((unsigned)grid), kDenseThreads, (size_t)smem, sm, work, sbt, prm,
                            st, x, n, hist, taps, ext);
}

template <bool DENSE>
static cudaError_t launch_rot(int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                              const ChanParams *prm, const ChanState *st, const float2 *x, int n,
                              const float2 *hist, const float *taps, float2 *ext) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_rot<DENSE>, 220 * 1024);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_extract_rot<DENSE>, dim3((unsigned)grid), kDenseThreads, (size_t)smem, sm, work, sbt,
                            prm, st, x, n, hist, taps, ext);
}

cudaError_t launch_extract_rot(bool dense, int grid, int smem, cudaStream_t sm, const int2 *work,
                               const SlotBlock *sbt, const ChanParams *prm, const ChanState *st, const float2 *x,
                               int n, const float2 *hist, const float *taps, float2 *ext) {
    return dense ? launch_rot<true>(grid, smem, sm, work, sbt, prm, st, x, n, hist, taps, ext)
                 : launch_rot<false>(grid, smem, sm, work, sbt, prm, st, x, n, hist, taps, ext);
}

cudaError_t launch_extract_mod(int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                               const ChanParams *prm, const ChanState *st, const float2 *x, int n,
                               const float2 *hist, const float *taps, float2 *ext) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_mod, 220 * 1024);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_extract_mod, dim3((unsigned)grid), kDenseThreads, (size_t)smem, sm, work, sbt, prm,
                            st, x, n, hist, taps, ext);
}

cudaError_t launch_comp_power(int count, cudaStream_t sm, const int *list, const SlotBlock *sbt,
                              const ChanParams *prm, ChanState *st, const float *wk) {
    return launch_dependent(k_comp_power, dim3((unsigned)count), 256, 0, sm, list, sbt, prm, st, wk);
}

cudaError_t launch_free_stereo(int grid, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                               const ChanParams *prm, const BinadeTable *tabs38, float *wk, int W) {
    return launch_dependent(k_free_stereo, dim3((unsigned)grid), 256, 0, sm, work, sbt, prm, tabs38, wk, W);
}

// Second decimation of the one-shot segment demod (recorder/cpu_audio.go:
// 35-72): ApplyFIRReal with the 63-tap anti-alias filter per audio channel
// (float64 taps and sum, separate multiply and add) at frames i*d2.
__global__ void __launch_bounds__(256)
k_seg_aa(const float *__restrict__ in, int C, const double *__restrict__ taps, int nt, int d2, int of,
         float *__restrict__ out) {
    const int idx = blockIdx.x * blockDim.x + (int)threadIdx.x;
    if (idx >= of * C) return;
    const int i = idx / C, c = idx - i * C;
    const int64_t src = (int64_t)i * d2;
    double acc = 0.0;
    for (int k = 0; k < nt; ++k) {
        const int64_t j = src - k;
        if (j < 0) break;
        acc = __dadd_rn(acc, __dmul_rn((double)in[j * C + c], taps[k]));
    }
    out[idx] = (float)acc;
}

cudaError_t launch_seg_aa(cudaStream_t sm, const float *in, int C, const double *taps, int nt, int d2, int of,
                          float *out) {
    const int total = of * C;
    if (total > 0) k_seg_aa<<<(total + 255) / 256, 256, 0, sm>>>(in, C, taps, nt, d2, of, out);
    return cudaGetLastError();
}

cudaError_t launch_demod(int grid, cudaStream_t sm, const int2 *work, const SlotBlock *sbt, const ChanParams *prm,
                         const ChanState *st, const float2 *ext, float *comp, float *audio) {
    return launch_dependent(k_demod, dim3((unsigned)grid), 256, 0, sm, work, sbt, prm, st, ext, comp,
                            audio);
}

cudaError_t launch_am(int grid, cudaStream_t sm, const int2 *work, const SlotBlock *sbt, const float2 *ext,
                      float *audio) {
    return launch_dependent(k_am, dim3((unsigned)grid), 256, 0, sm, work, sbt, ext, audio);
}

cudaError_t launch_wfm_fir(int grid, cudaStream_t sm, const int2 *work, const SlotBlock *sbt, const ChanParams *prm,
                           const WfmTaps *taps, float *wk, int W, const float *comp_dl) {
    return launch_dependent(k_wfm_fir, dim3((unsigned)grid), kFirThreads, 0, sm, work, sbt, prm, taps, wk,
                            W, comp_dl);
}

cudaError_t launch_pll(int count, cudaStream_t sm, const int *list, const SlotBlock *sbt, const ChanParams *prm,
                       ChanState *st, float *wk, int W) {
    return launch_dependent(k_pll, dim3((unsigned)count), 64, 0, sm, list, count, sbt, prm, st, wk, W);
}

cudaError_t launch_pll_newton(int count, int cluster, cudaStream_t sm, const int *list, const SlotBlock *sbt,
                              const ChanParams *prm, ChanState *st, float *wk, int W, int max_iters) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(count * cluster), 1, 1);
    cfg.blockDim = dim3(kNewtonThreads, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = sm;
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return launch_status(cudaLaunchKernelEx(&cfg, k_pll_newton, list, count, sbt, prm, st, wk, W, max_iters));
}

int pll_newton_threads() { return kNewtonThreads; }

cudaError_t launch_wfm_out(int grid, cudaStream_t sm, const int2 *work, const SlotBlock *sbt, const ChanParams *prm,
                           const ChanState *st, const WfmTaps *taps, const float *wk, int W, const float *lr_dl,
                           const float *audio_dl, float *audio) {
    return launch_dependent(k_wfm_out, dim3((unsigned)grid), kFirThreads, 0, sm, work, sbt, prm, st, taps,
                            wk, W, lr_dl, audio_dl, audio);
}

cudaError_t launch_rds(int grid, int smem, cudaStream_t sm, const int2 *work, const SlotBlock *sbt,
                       const ChanParams *prm, const ChanState *st, const WfmTaps *taps, const BinadeTable *tabs,
                       const float *wk, const float2 *rds_dl, float2 *rds_out) {
    return launch_dependent(k_rds, dim3((unsigned)grid), kRdsThreads, (size_t)smem, sm, work, sbt, prm, st, taps,
                            tabs, wk, rds_dl, rds_out);
}

cudaError_t launch_decim2(int grid, cudaStream_t sm, const int2 *work, const SlotBlock *sbt, const ChanParams *prm,
                          const double *d1taps, const float2 *d1hist, float2 *ext) {
    return launch_dependent(k_decim2, dim3((unsigned)grid), kDecOT, 0, sm, work, sbt, prm, d1taps, d1hist,
                            ext);
}

int decim2_tile() { return kDecOT; }

cudaError_t launch_post_front(int grid, cudaStream_t sm, const SlotBlock *sbt, const ChanParams *prm, ChanState *st,
                              const float2 *ext, const float *wk, float *comp_dl, float2 *rds_dl,
                              const BinadeTable *tabs, float2 *d1hist, DevResult *res) {
    return launch_dependent(k_post_front, dim3((unsigned)grid), 128, 0, sm, sbt, prm, st, ext, wk, comp_dl,
                            rds_dl, tabs, d1hist, res);
}

cudaError_t launch_audio48(int grid_rs, int rs_smem, int count, cudaStream_t sm, const int2 *work, const int *list,
                           const SlotBlock *sbt, const ChanParams *prm, const RsBank *banks, AudState *aud,
                           const float *audio, float *rs_buf, int16_t *pcm) {
    static std::atomic<uint64_t> optin{0};  // more than 48 KiB of dynamic shared memory needs the opt-in
    cudaError_t e = smem_optin_once(optin, (const void *)k_audio48_rs, kAudBank * 8 + 2 * kAudWin * 4);
    if (e != cudaSuccess) return e;
    if (grid_rs > 0)
        e = launch_dependent(k_audio48_rs, dim3((unsigned)grid_rs), kAudThreads, (size_t)rs_smem, sm, work, sbt, prm, banks,
                             aud, audio, rs_buf);
    if (e != cudaSuccess) return e;
    static std::atomic<uint64_t> optin_out{0};
    e = smem_optin_once(optin_out, (const void *)k_audio48_out, kAudOutStage * 4);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_audio48_out, dim3((unsigned)count), kAudOutThreads, kAudOutStage * 4, sm,
                            list, sbt, prm, banks, aud, audio, rs_buf, pcm);
}

void audio48_tile(int L, int M, int C, int *outputs, int *smem) {
    const AudTile t = aud_tile(L, M, kRsTaps, C);
    *outputs = t.ot;
    *smem = t.smem;
}

// Arms of a resampler bank (NewResampler, dsp/resample.go:45-93, 256-295):
// windowed sinc fc = 0.90/max(L, M), Kaiser beta 6 by the reference's Bessel
// series, gain L; arm[p*K + t] = prototype tap p + t*L.  One thread per tap: a
// rate that shares no factor with 48 kHz has up to 48000 arms of 33 taps, which
// took the host longer than the rest of an event's demod together.
__device__ __forceinline__ double rs_bessel0(double x) {
    double sum = 1.0, term = 1.0;
    for (int k = 1; k < 30; k++) {
        const double q = __ddiv_rn(x, 2.0 * (double)k);
        term = __dmul_rn(term, __dmul_rn(q, q));
        sum = __dadd_rn(sum, term);
        if (term < __dmul_rn(1e-12, sum)) break;
    }
    return sum;
}

__global__ void __launch_bounds__(256) k_rs_bank(int L, int M, int K, double *__restrict__ arm) {
    const int i = blockIdx.x * blockDim.x + (int)threadIdx.x;
    if (i >= L * K) return;
    const int plen = (L * 32) | 1, p = i / K, n = p + (i - p * K) * L;
    double v = 0.0;
    if (n < plen) {
        const double fc = 0.90 / (double)max(L, M), mid = (double)(plen - 1) / 2.0, x = (double)n - mid;
        const double sn = fabs(x) < 1e-12 ? 2 * GPUD_PI * fc : sin(2 * GPUD_PI * fc * x) / x;
        const double xx = x / mid;
        v = sn * (rs_bessel0(6.0 * sqrt(__dsub_rn(1.0, __dmul_rn(xx, xx)))) / rs_bessel0(6.0)) * (double)L;
    }
    arm[i] = v;
}

cudaError_t launch_rs_bank(cudaStream_t sm, int L, int M, int K, double *arm) {
    return launch_alone(k_rs_bank, dim3((unsigned)((L * K + 255) / 256)), 256, 0, sm, L, M, K, arm);
}

cudaError_t launch_post_extract(int grid, cudaStream_t sm, const SlotBlock *sbt, const ChanParams *prm, ChanState *st,
                                const float2 *x, int n, float2 *hist, DevResult *res) {
    return launch_dependent(k_post_extract, dim3((unsigned)grid), 128, 0, sm, sbt, prm, st, x, n, hist,
                            res);
}

cudaError_t launch_post_back(int grid, cudaStream_t sm, const SlotBlock *sbt, const ChanParams *prm, ChanState *st,
                             const float *wk, int W, float *lr_dl, float *audio_dl, DevResult *res) {
    return launch_dependent(k_post_back, dim3((unsigned)grid), 128, 0, sm, sbt, prm, st, wk, W, lr_dl,
                            audio_dl, res);
}

int rds_smem_bytes(int dr) {
    const int span = kRdsOT * dr + kWfmTaps + 8;
    return (span + span / 16 + 1) * 8;
}
int rds_tile() { return kRdsOT; }

}  // namespace gpud

// bank_extract.cu -- extraction of short-arm channel banks.
//
// Channels that share the decimation D, the tap count T (T <= 4D: at most four
// taps per polyphase arm) and the phase count before the block take their
// outputs on the same input grid n_j = (D - pc - 1) + j*D.  With the NCO moved
// from the samples onto the taps (the modulated-taps identity of the
// reference's NCO-then-FIR chain, streaming_host_core.go:5-64):
//
//     y_c(j) = exp(j phi_c(n_j)) * sum_{k<T} g_c[k] x(n_j - k),   g_c[k] = h_c[k] exp(-j k inc_c),
//
// every channel of the bank filters the same unrotated block x.  One work item
// is up to 32 outputs x 32 channels: the outputs' input windows and the
// channels' modulated taps come into shared memory 64 taps at a time by
// asynchronous copies, one chunk ahead of the arithmetic (staged through
// registers between barriers, 128 taps at a time, the loads' latency stood open
// in every item); a lane accumulates up to 4 outputs of one channel in registers
// across all tap chunks, then rotates by exp(j phi_c(n_j)) from the exact Q0.64
// phase and stores.  Window samples are broadcasts and the taps one 16-byte load
// per lane for two taps: shared-memory loads bound it.  Measured, register
// staging before and this kernel now: the mixed batch's four banks (120
// channels) 58.5 -> 43.5 us, 512 serving channels 55.9 -> 35.6 us, the banked
// part of 2048 mixed channels 79 -> 36.5 us.
//
// The block is read once per bank and tile instead of once per channel, and no
// partial sums leave the SM.  Outputs whose window reaches into the carried
// history (before the bank's first tile) stay on the warp-per-output kernel.
#include <algorithm>

#include "gpud_internal.cuh"

namespace gpud {

constexpr int kBankThreads = 256;
constexpr int kBankLanes = 32;                 // channels per work item (one per lane)
constexpr int kBankR = 4;                      // most outputs per lane
constexpr int kBankJ = (kBankThreads / 32) * kBankR;  // most outputs per work item
constexpr int kBankKC = 64;                    // taps per staged chunk

struct BankStage {
    float4 g[kBankKC / 2][kBankLanes];  // (g_c[k], g_c[k+1])
    float2 x[kBankJ][kBankKC];          // window of output o, oldest sample first
};
constexpr int kBankSmem = 2 * (int)sizeof(BankStage);

int bank_lanes() { return kBankLanes; }
int bank_warps() { return kBankThreads / 32; }

int64_t bank_pack_entries(int T, int cpad) { return (int64_t)((T + 1) & ~1) * cpad; }

// Modulated taps of every bank in pairs, g[b.g_off + ((k/2)*cpad + c)*2 + k%2]
// (float2), zero for padding columns and the pair of an odd last tap; the same
// products as the other modulated forms.
__global__ void __launch_bounds__(256)
k_bank_pack(const BankGroup *__restrict__ groups, const int *__restrict__ members, const SlotBlock *__restrict__ sbt,
            const ChanParams *__restrict__ prm, const float *__restrict__ taps_arena, float2 *__restrict__ gtab) {
    dependency_wait();
    const BankGroup b = groups[blockIdx.y];
    const int total = ((b.T + 1) & ~1) * b.cpad;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int q = (i >> 1) / b.cpad, c = (i >> 1) - q * b.cpad, k = 2 * q + (i & 1);
        float2 v = make_float2(0.f, 0.f);
        if (c < b.nmem && k < b.T) {
            const ChanParams &cp = prm[sbt[members[b.mem_off + c]].slot];
            const float h = taps_arena[cp.dtaps_off + k];
            const float2 ph = q64_phasor((uint64_t)0 - (uint64_t)k * cp.inc_q);
            v = make_float2(h * ph.x, h * ph.y);
        }
        gtab[b.g_off + i] = v;
    }
}

// Asynchronous copy of BYTES global -> shared, zeros where !ok.
template <int BYTES>
__device__ __forceinline__ void bank_copy(void *dst, const void *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES),
                 "r"(ok ? BYTES : 0)
                 : "memory");
}

// One work item: G lane groups of 32 / G channels, R outputs per lane, 8 G R
// outputs.  A chunk of at most 16 or 8 channels (the rest of a bank's 32s) takes
// two or four groups, so that its lanes work on more outputs instead of idling:
// every output's sum is the same chain whichever lane has it.
template <int R, int G>
__device__ __forceinline__ void bank_item(const BankGroup &b, int tile, int chunk, BankStage *st2,
                                          const int *__restrict__ members, const SlotBlock *__restrict__ sbt,
                                          const ChanParams *__restrict__ prm, const ChanState *__restrict__ st,
                                          const float2 *__restrict__ x, const float2 *__restrict__ gtab,
                                          float2 *__restrict__ ext) {
    constexpr int J = (kBankThreads / 32) * G * R, CL = kBankLanes / G;
    const int j0 = b.jt0 + tile * J;
    if (j0 >= b.n_out) return;
    const int D = b.D, T = b.T, s0 = D - b.pc - 1, c0 = chunk * kBankLanes;
    const int tid = (int)threadIdx.x, cl = tid % CL, o0 = tid / CL * R;  // lane's channel, first output
    const float4 *g4 = reinterpret_cast<const float4 *>(gtab + b.g_off) + c0;
    // windows: sample u of output o's chunk is n_o - kc - (63 - u) (inside the
    // block: the bank starts at the first output whose window is)
    auto stage = [&](BankStage &sm, int kc) {
        const int kn = min(kBankKC, T - kc);
#pragma unroll
        for (int i = 0; i < (kBankKC / 2) * CL / kBankThreads; ++i) {
            const int e = tid + i * kBankThreads, q = e / CL, c = e % CL;
            const bool ok = 2 * q < kn;
            bank_copy<16>(&sm.g[q][c], g4 + (ok ? (int64_t)((kc >> 1) + q) * b.cpad + c : 0), ok);
        }
#pragma unroll
        for (int i = 0; i < J * kBankKC / kBankThreads; ++i) {
            const int e = tid + i * kBankThreads, o = e / kBankKC, u = e % kBankKC, j = j0 + o;
            const bool ok = kBankKC - 1 - u < kn && j < b.n_out;
            bank_copy<8>(&sm.x[o][u], x + (ok ? s0 + j * D - kc - (kBankKC - 1 - u) : 0), ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float ar[R], ai[R];
#pragma unroll
    for (int r = 0; r < R; ++r) ar[r] = ai[r] = 0.f;
    stage(st2[0], 0);
    for (int kc = 0, h = 0; kc < T; kc += kBankKC, h ^= 1) {
        if (kc + kBankKC < T) {
            stage(st2[h ^ 1], kc + kBankKC);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const BankStage &sm = st2[h];
        const int nq = (min(kBankKC, T - kc) + 1) >> 1;
#pragma unroll 4
        for (int q = 0; q < nq; ++q) {
            const float4 g = sm.g[q][cl];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                // one address per group: (x(n-k-1), x(n-k)) for the taps k = kc + 2q and k + 1
                const float4 v = *reinterpret_cast<const float4 *>(&sm.x[o0 + r][kBankKC - 2 - 2 * q]);
                ar[r] = fmaf(g.x, v.z, ar[r]);
                ar[r] = fmaf(-g.y, v.w, ar[r]);
                ar[r] = fmaf(g.z, v.x, ar[r]);
                ar[r] = fmaf(-g.w, v.y, ar[r]);
                ai[r] = fmaf(g.x, v.w, ai[r]);
                ai[r] = fmaf(g.y, v.z, ai[r]);
                ai[r] = fmaf(g.z, v.y, ai[r]);
                ai[r] = fmaf(g.w, v.x, ai[r]);
            }
        }
        __syncthreads();  // the chunk is rewritten by the one after next
    }
    const int c = c0 + cl;
    if (c >= b.nmem) return;
    const SlotBlock &sb = sbt[members[b.mem_off + c]];
    const uint64_t u0 = st[sb.slot].nco_q, inc = prm[sb.slot].inc_q;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int j = j0 + o0 + r;
        if (j < b.n_out) {
            const float2 rot = q64_phasor(u0 + (uint64_t)(int64_t)(s0 + j * D) * inc);
            ext[sb.ext_off + j] = cmulf(make_float2(ar[r], ai[r]), rot);
        }
    }
}

// Work item (bank, tile * chunks + chunk): outputs jt0 + 8r*tile .. of
// channels 32*chunk .. +31, r outputs per lane of a full chunk.
__global__ void __launch_bounds__(kBankThreads, 3)
k_extract_bank(const int2 *__restrict__ work, const BankGroup *__restrict__ groups, const int *__restrict__ members,
               const SlotBlock *__restrict__ sbt, const ChanParams *__restrict__ prm,
               const ChanState *__restrict__ st, const float2 *__restrict__ x, const float2 *__restrict__ gtab,
               float2 *__restrict__ ext) {
    dependency_wait();
    extern __shared__ float4 bsm[];
    BankStage *st2 = reinterpret_cast<BankStage *>(bsm);
    const int2 w = work[blockIdx.x];
    const BankGroup b = groups[w.x];
    const int nch = b.cpad / kBankLanes, tile = w.y / nch, chunk = w.y - tile * nch;
    const int m = b.nmem - chunk * kBankLanes;  // channels of this chunk
#define GPUD_BANK(R, G) bank_item<R, G>(b, tile, chunk, st2, members, sbt, prm, st, x, gtab, ext)
    if (b.r == 4) {  // uniform per CTA
        if (m <= 8) GPUD_BANK(1, 4);
        else if (m <= 16) GPUD_BANK(2, 2);
        else GPUD_BANK(4, 1);
    } else if (b.r == 2) {
        if (m <= 16) GPUD_BANK(1, 2);
        else GPUD_BANK(2, 1);
    } else {
        GPUD_BANK(1, 1);
    }
#undef GPUD_BANK
}

cudaError_t launch_bank_pack(int ngroups, int max_total, cudaStream_t sm, const BankGroup *groups,
                             const int *members, const SlotBlock *sbt, const ChanParams *prm, const float *taps,
                             float2 *gtab) {
    const int gx = std::min(64, (max_total + 255) / 256);
    return launch_dependent(k_bank_pack, dim3(gx > 0 ? gx : 1, ngroups), 256, 0, sm, groups, members, sbt, prm, taps,
                            gtab);
}

cudaError_t launch_extract_bank(int grid, cudaStream_t sm, const int2 *work, const BankGroup *groups,
                                const int *members, const SlotBlock *sbt, const ChanParams *prm, const ChanState *st,
                                const float2 *x, const float2 *gtab, float2 *ext) {
    static std::atomic<uint64_t> optin{0};
    cudaError_t e = smem_optin_once(optin, (const void *)k_extract_bank, kBankSmem);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_extract_bank, dim3((unsigned)grid), kBankThreads, kBankSmem, sm, work,
                            groups, members, sbt, prm, st, x, gtab, ext);
}

}  // namespace gpud

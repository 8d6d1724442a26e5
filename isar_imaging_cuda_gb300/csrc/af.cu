// Doppler tracking and fast minimum-entropy autofocus on the M x 512 cut.
// Reference: phase_adjustment.cu:4-41 (dopplerTracking), :167-332
// (fastEntropy), common.cu:341-391 (maxCols/sumCols), :436-462 (sumRows).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "fft.cuh"
#include "isar_kernels.h"
#include "launch.cuh"
#include "nn.h"

namespace isar {

constexpr int C = kRangeCut;

// The cluster engines' entropy of the selected bins (stop criterion, choice
// of start, trace) sums p log2 p with the hardware base-2 logarithm
// (__log2f, ~2^-22 relative error, a few instructions instead of ~20 for
// logf) and converts once: H = ln S1 - ln 2 * S2 / S1.
constexpr float kLn2 = 0.693147180559945309f;

// The stop criterion compares the entropy every kStopEvery iterations: stop
// at iteration it (a multiple of kStopEvery, it > 0, before its update) once
// |E(it) - E(it - kStopEvery)| <= kStopEvery * tol * |E(it)|, i.e. once the
// entropy changes by at most tol * |E| per iteration on average.  Iterations
// in between skip the entropy terms and its cluster reduction.
constexpr int kStopEvery = 4;

// Column max of |cut| over rows [0, min(M,256)) per CTA of R rows, and the
// Doppler sums s[m] = sum_c conj(x[m,c]) x[m+1,c] (one warp per row).
__global__ void __launch_bounds__(256)
k_fe_stats(const float2* __restrict__ cut, int M, int rows_max, int R, float* __restrict__ cmax_part,
           float2* __restrict__ dsum)
{
    pdl_begin();
    const int r0 = blockIdx.x * R;
    const int tid = threadIdx.x;
    if (cmax_part != nullptr && r0 < rows_max) {
        const int r1 = min(r0 + R, rows_max);
        for (int c = tid; c < C; c += blockDim.x) {
            float mx = 0.0f;   // of |x|^2: the root is monotonic, and without it the loads overlap
#pragma unroll 8
            for (int r = r0; r < r1; ++r) {
                const float2 v = cut[(size_t)r * C + c];
                mx = fmaxf(mx, v.x * v.x + v.y * v.y);
            }
            cmax_part[(size_t)blockIdx.x * C + c] = sqrtf(mx);
        }
    }
    const int w = tid >> 5, lane = tid & 31;
    for (int m = r0 + w; m < min(r0 + R, M - 1); m += blockDim.x >> 5) {
        float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int c = lane; c < C; c += 32) {
            const float2 a = cut[(size_t)m * C + c];
            const float2 b = cut[(size_t)(m + 1) * C + c];
            const float2 p = cmulc(a, b);
            s.x += p.x;
            s.y += p.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if (lane == 0) dsum[m] = s;
    }
}

// Same Doppler sums on the U gathered bins: s[m] = sum_u conj(g[m,u]) g[m+1,u].
__global__ void __launch_bounds__(256)
k_af_doppler(const float2* __restrict__ cut, const int* __restrict__ bins, const int* __restrict__ fdec,
             int M, float2* __restrict__ dsum)
{
    pdl_begin();
    const int U = fdec[1];
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int m = w;
    if (m >= M - 1) return;
    float2 s = make_float2(0.0f, 0.0f);
    for (int u = lane; u < U; u += 32) {
        const int b = bins[u];
        const float2 p = cmulc(cut[(size_t)m * C + b], cut[(size_t)(m + 1) * C + b]);
        s.x += p.x;
        s.y += p.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    if (lane == 0) dsum[m] = s;
}

// Doppler phase: psi = arg(s), Phi = inclusive scan, phase[0] = 0,
// phase[m+1] = exp(-j*Phi[m]) (phase_adjustment.cu:17-31); M threads per CTA,
// warp b of CTA b writes the phases of its 32 pulses.  Every CTA scans all of psi:
// in 64-bit fixed point (units of 2^-50 rad, exact for the float angles down
// to 2^-27 rad), which is faster than adding doubles and as exact.  The
// double sine and cosine are what the kernel is bound by (FP64 issues ~2 per
// clock and SM): spread over M / 32 CTAs, one warp each (one CTA took
// 25000 clocks at 1024 pulses, 8900 of them in a scan of doubles).
// CTA 0 also counts the targets (phase_adjustment.cu:180-194) when nparts > 0:
// colmax, mean with an int accumulator (Q3), threshold 1.48*mean.
// fdec: [0] tgt_num, [1] U.
__global__ void __launch_bounds__(1024)
k_fe_phase(const float* __restrict__ cmax_part, int nparts, const float2* __restrict__ dsum, int M,
           float2* __restrict__ phase, int* __restrict__ fdec)
{
    __shared__ long long s_tot[32];
    __shared__ unsigned s_nan[32];
    __shared__ int s_cnt[32];
    __shared__ int s_sum[32];
    pdl_begin();
    const int tid = threadIdx.x;
    const int lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    // inclusive scan of arg(s); a NaN reaches every later phase
    long long v = 0;
    bool bad = false;
    if (tid < M - 1) {
        const float2 s = dsum[tid];
        const float psi = atan2f(s.y, s.x);
        bad = isnan(psi);
        v = bad ? 0 : __float2ll_rn(psi * 1125899906842624.0f);   // 2^50, exact
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    const unsigned nans = __ballot_sync(0xffffffffu, bad);
    if (lane == 31) {
        s_tot[w] = v;
        s_nan[w] = nans;
    }
    __syncthreads();
    if (w == (int)blockIdx.x) {   // this CTA's 32 pulses
        unsigned any = nans & ((2u << lane) - 1u);
        for (int i = 0; i < w; ++i) {
            v += s_tot[i];
            any |= s_nan[i];
        }
        if (tid < M - 1) {
            double sn, cs;
            sincos(any ? CUDART_NAN : (double)v * 8.8817841970012523234e-16, &sn, &cs);   // 2^-50
            phase[tid + 1] = make_float2((float)cs, (float)-sn);
        }
        if (tid == 0) phase[0] = make_float2(0.0f, 0.0f);
    }
    if (nparts == 0 || blockIdx.x != 0) return;
    float mx[C / 128];   // M >= 128 threads: up to four columns each
    int isum = 0;
#pragma unroll
    for (int q = 0; q < C / 128; ++q) {
        const int c = tid + q * (int)blockDim.x;
        mx[q] = 0.0f;
        if (c < C) {
#pragma unroll 8
            for (int p = 0; p < nparts; ++p) mx[q] = fmaxf(mx[q], cmax_part[(size_t)p * C + c]);
            isum += (int)mx[q];
        }
    }
    // the int accumulator wraps, as the reference's does
    isum = (int)__reduce_add_sync(0xffffffffu, (unsigned)isum);
    if (lane == 0) s_sum[w] = isum;
    __syncthreads();
    isum = (int)__reduce_add_sync(0xffffffffu, lane < nw ? (unsigned)s_sum[lane] : 0u);
    const float mean_val = (float)isum / (float)C;
    const float thr = 1.48f * mean_val;
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < C / 128; ++q) cnt += (tid + q * (int)blockDim.x < C && mx[q] > thr) ? 1 : 0;
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) s_cnt[w] = cnt;
    __syncthreads();
    if (tid == 0) {
        int t = 0;
        for (int i = 0; i < nw; ++i) t += s_cnt[i];
        // U = nextPow2(tgt_num / 2) (common.cu:521-529)
        int n = t / 2, u = 1;
        while (n >> 1) {
            u <<= 1;
            n >>= 1;
        }
        fdec[0] = t;
        fdec[1] = u << 1;
    }
}

// team reduction (sum) of a double over the T threads of a team.
template <int T>
__device__ __forceinline__ double team_sum(double v, int lt, double* red /* per-team, >= T/32 */)
{
    if constexpr (T >= 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        constexpr int W = T / 32;
        if constexpr (W > 1) {
            if ((lt & 31) == 0) red[lt >> 5] = v;
            __syncthreads();
            double t = 0.0;
#pragma unroll
            for (int i = 0; i < W; ++i) t += red[i];
            __syncthreads();
            return t;
        }
        return v;
    } else {
#pragma unroll
        for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, T);
        return v;
    }
}

// Per column: FFT over pulses of phase[m]*cut[m,c], energy E = sum |X|^2 and
// entropy H = -sum p ln p, p = |X|^2/E (phase_adjustment.cu:215-246).
// CB columns per CTA, one team of M/16 threads per column.
template <int M, int CB>
__global__ void __launch_bounds__(CB * M / 16)
k_fe_colfft(const float2* __restrict__ cut, const float2* __restrict__ phase, double* __restrict__ E,
            double* __restrict__ H, const float2* __restrict__ tw)
{
    using F = FFTShape<M>;
    extern __shared__ float4 dyn_smem[];
    float2* smb = reinterpret_cast<float2*>(dyn_smem);
    __shared__ double red[CB][(F::T + 31) / 32];
    const int tid = threadIdx.x;
    const int team = tid / F::T, lt = tid % F::T;
    const int c0 = blockIdx.x * CB;
    float2* twt = smb + CB * F::SMEM;
    TwShared<M>::fill(twt, tw, tid, blockDim.x);
    pdl_begin();
    for (int i = tid; i < M * CB; i += blockDim.x) {
        const int m = i / CB, cc = i % CB;
        smb[cc * F::SMEM + fpad(m)] = cmul(phase[m], cut[(size_t)m * C + c0 + cc]);
    }
    __syncthreads();
    float2* sm = smb + team * F::SMEM;
    float p[16];
    team_fft<M, false>([&](int i) { return sm[fpad(i)]; },
                       [&](int, float2 v, int slot) { p[slot] = v.x * v.x + v.y * v.y; }, sm, lt,
                       TwShared<M>{twt});
    // per-thread partials in float (16 terms), team sums in double
    float ep = 0.0f;
#pragma unroll
    for (int q = 0; q < 16; ++q) ep += p[q];
    const double e = team_sum<F::T>((double)ep, lt, red[team]);
    const float ef = (float)e;
    float hp = 0.0f;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const float x = p[q] / ef;
        hp += -(x * logf(x));
    }
    const double h = team_sum<F::T>((double)hp, lt, red[team]);
    if (lt == 0) {
        E[c0 + team] = e;
        H[c0 + team] = h;
    }
}

// One element per thread of a 512-thread CTA, sorted ascending by (key, tie):
// thread i ends with the i-th element.  Strides below 32 are exchanged by warp
// shuffles, larger ones through shared memory (10 of the 45 stages).  Keys are
// unsigned integers (double_order): compares of doubles run on the FP64 pipe,
// which issues ~2 per clock and SM.
struct SelKey {
    unsigned long long key;
    int tie;   // distinct
    int val;   // payload
};
__device__ __forceinline__ SelKey shfl_xor_key(const SelKey& v, int j)
{
    SelKey w;
    w.key = __shfl_xor_sync(0xffffffffu, v.key, j);
    w.tie = __shfl_xor_sync(0xffffffffu, v.tie, j);
    w.val = __shfl_xor_sync(0xffffffffu, v.val, j);
    return w;
}
// Unsigned order of a double (ascending).
__device__ __forceinline__ unsigned long long double_order(double d)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(d + 0.0);   // -0 orders as 0
    return b ^ ((b >> 63) ? ~0ull : 1ull << 63);
}
__device__ __forceinline__ void sort512(SelKey& v, SelKey* sm)
{
    const int i = threadIdx.x;
#pragma unroll 1
    for (int k = 2; k <= C; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            SelKey w;
            if (j >= 32) {
                sm[i] = v;
                __syncthreads();
                w = sm[i ^ j];
                __syncthreads();
            } else {
                w = shfl_xor_key(v, j);
            }
            const bool up = (i & k) == 0;      // this region ascends
            const bool lower = (i & j) == 0;   // i is the lower index of its pair
            const bool v_first = v.key < w.key || (v.key == w.key && v.tie < w.tie);
            if (!((lower == up) ? v_first : !v_first)) v = w;
        }
}

// Bin selection (phase_adjustment.cu:248-264), one CTA of 512 threads, one
// column per thread: stable sort by energy (descending), keep tgt_num, stable
// sort by entropy (ascending), keep U (indices beyond tgt_num are 0, as
// device_vector::resize pads), sort the kept indices.  NaN keys sort last.
// The stable sorts are strict orders with the position as tie-break; the kept
// indices are put in order by a prefix count of their columns' flags.
// Latency of one CTA: ~19500 clocks, bound by the shuffles of its 90 stages (33 us
// with double keys and a third sort).
__global__ void __launch_bounds__(C)
k_fe_select(const double* __restrict__ E, const double* __restrict__ H, int* __restrict__ fdec,
            int* __restrict__ bins)
{
    __shared__ SelKey sm[C];
    __shared__ int s_flag[C];
    __shared__ int s_cnt[C / 32];
    pdl_begin();
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int tgt = fdec[0], U = fdec[1];
    SelKey v;
    const double h_own = H[tid];
    {
        const double e = E[tid];
        v.key = ~double_order(isnan(e) ? -CUDART_INF : e);   // descending
        v.tie = tid;
        v.val = tid;
    }
    sort512(v, sm);
    // second key: entropy of the first tgt entries; the rest are sentinels
    __syncthreads();
    double* s_h = reinterpret_cast<double*>(sm);
    s_h[tid] = h_own;
    s_flag[tid] = 0;
    __syncthreads();
    {
        double h = (tid < tgt) ? s_h[v.val] : CUDART_INF;
        if (isnan(h)) h = CUDART_INF;
        v.key = double_order(h);
        v.tie = (tid < tgt) ? tid : (C + tid);
    }
    __syncthreads();
    sort512(v, sm);
    // the first U of the tgt kept entries; U > tgt pads with index 0 in front
    const int kept = min(U, tgt), pad = U - kept;
    if (tid < kept) s_flag[v.val] = 1;
    __syncthreads();
    const unsigned b = __ballot_sync(0xffffffffu, s_flag[tid] != 0);
    if (lane == 0) s_cnt[w] = __popc(b);
    __syncthreads();
    int before = 0;
    for (int i = 0; i < w; ++i) before += s_cnt[i];
    if (s_flag[tid]) bins[pad + before + __popc(b & ((1u << lane) - 1u))] = tid;
    if (tid < pad) bins[tid] = 0;
}

// Grid-wide barrier for cooperative launches (all CTAs co-resident): arrive
// on a monotonic counter and wait, with at most `limit` polls (kSpinLimit,
// about a second), until it reaches `target`.  A timeout sets *err and makes
// every later barrier fail fast, so that all CTAs leave the kernel.  Returns
// false on failure.
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned target, int* err, unsigned long long limit)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(count, 1u);
        int ok = 1;
        unsigned long long spins = 0;
        for (;;) {
            if (*(volatile unsigned*)count >= target) break;
            if (*(volatile int*)err) {
                ok = 0;
                break;
            }
            if (++spins > limit) {
                atomicExch(err, 1);
                ok = 0;
                break;
            }
            __nanosleep(40);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// All minimum-entropy iterations (phase_adjustment.cu:302-322) in one
// cooperative launch of G CTAs.  CTA b owns up to 4 of the U selected bins
// (one team of M/16 threads per bin), keeps them in shared memory, and per
// iteration computes t = phase .* g, T = FFT(t), T .* |T|, h = IFFT(T)/M,
// q = conj(g) .* h and writes its partial row sums to P[m][b].  After a grid
// barrier CTA b sums the rows m = b, b+G, ... over all partials and writes
// phase[m] = sigma / |sigma|; a second barrier publishes the new phase.
// phase: in the Doppler-tracking start, out the final phase.  Frames with
// fewer than min_u bins are left alone.
template <int M>
__global__ void __launch_bounds__(4 * (M / 16))
k_af_persist(const float2* __restrict__ cut, const int* __restrict__ bins, const int* __restrict__ fdec,
             float2* phase, float2* P, unsigned* bar, int* err, int iters, const float2* __restrict__ tw,
             BarrierTest bt, int min_u)
{
    if (fdec[1] < min_u) return;   // the whole grid, before any barrier
    using F = FFTShape<M>;
    constexpr int TEAMS = 4;
    extern __shared__ float4 dyn_smem[];
    float2* gs = reinterpret_cast<float2*>(dyn_smem);   // [TEAMS][M]
    float2* smb = gs + TEAMS * M;                        // [TEAMS][SMEM]
    float2* ph = smb + TEAMS * F::SMEM;                  // [M]
    float2* twt = ph + M;                                // twiddle table
    TwShared<M>::fill(twt, tw, threadIdx.x, blockDim.x);
    const TwShared<M> tws{twt};
    const int G = gridDim.x;
    const int U = fdec[1];
    const int cpc = (U + G - 1) / G;
    const int nact = (U + cpc - 1) / cpc;                 // CTAs that own bins
    const int tid = threadIdx.x;
    const int team = tid / F::T, lt = tid % F::T;
    const int u = blockIdx.x * cpc + team;
    const bool valid = team < cpc && u < U;
    float2* g = gs + team * M;
    float2* sm = smb + team * F::SMEM;
    {
        const int b = valid ? bins[u] : 0;
        for (int m = lt; m < M; m += F::T) g[m] = valid ? cut[(size_t)m * C + b] : make_float2(0.0f, 0.0f);
    }
    const float invM = 1.0f / (float)M;
    const int lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
#pragma unroll 1
    for (int it = 0; it < iters; ++it) {
        for (int m = tid; m < M; m += blockDim.x) ph[m] = __ldcg(&phase[m]);
        __syncthreads();
        if (blockIdx.x < nact) {
            team_fft<M, false>([&](int i) { return cmul(ph[i], g[i]); },
                               [&](int i, float2 v, int) { sm[fpad(i)] = cscale(v, sqrtf(v.x * v.x + v.y * v.y)); },
                               sm, lt, tws, valid);
            team_fft<M, true>([&](int i) { return sm[fpad(i)]; },
                              [&](int i, float2 v, int) { sm[fpad(i)] = cmulc(g[i], cscale(v, invM)); }, sm, lt,
                              tws, valid);
            __syncthreads();
            const int nt = min(cpc, U - (int)blockIdx.x * cpc);   // bins of this CTA
            for (int m = tid; m < M; m += blockDim.x) {
                float2 s = make_float2(0.0f, 0.0f);
                for (int t = 0; t < nt; ++t) {
                    const float2 q = smb[t * F::SMEM + fpad(m)];
                    s.x += q.x;
                    s.y += q.y;
                }
                __stcg(&P[(size_t)m * G + blockIdx.x], s);
            }
        }
        if (!grid_barrier(bar, (unsigned)(2 * it + 1) * G + bt.extra, err, bt.limit)) return;
        for (int m = blockIdx.x + warp * G; m < M; m += nwarp * G) {
            float2 s = make_float2(0.0f, 0.0f);
            for (int b = lane; b < nact; b += 32) {
                const float2 q = __ldcg(&P[(size_t)m * G + b]);
                s.x += q.x;
                s.y += q.y;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
                s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            }
            if (lane == 0) {
                const float a = sqrtf(s.x * s.x + s.y * s.y);
                __stcg(&phase[m], make_float2(s.x / a, s.y / a));
            }
        }
        if (!grid_barrier(bar, (unsigned)(2 * it + 2) * G + bt.extra, err, bt.limit)) return;
    }
}

// ---------------------------------------------------------------------------
// Cluster-resident autofocus: the same iteration as k_af_persist, with all
// state of one frame held in the shared memory of one thread-block cluster
// and every transform inside one warp.
//
// CTA r of a cluster of CL owns bins [r*bpc, r*bpc + nb), bpc = ceil(U/CL).
// L lanes own one bin (a warp; half a warp at 128 pulses): element
// m = l + L i lives in lane l, register i (i < P, M = P L).  The forward
// transform runs as
//   DFT_P over i -> k1, twiddle W_M^(l k1), exchange through the warp's tile:
//   lane (k1, q) gets l = q + Q b (Q = L / P), DFT_P over b -> c, twiddle
//   W_L^(q c), DFT_Q over q between neighbouring lanes by shuffles (AfCross),
// and the inverse is its mirror image from that order back to pulse order, so
// T |T| (order independent) sits between them with no reordering.  Shared
// memory bandwidth is what the transforms of 8 or more bins per CTA run
// into, so there is one exchange through it per transform, and the twiddles
// of the short transforms stay in registers.  At 1024 pulses Q = 1 and both
// transforms share one copy of the code (conj-forward-conj), which keeps the
// kernel within the instruction cache.
//
// Per iteration: each CTA sums conj(g) .* IFFT(T |T|) / M over its bins and
// sends slice q of the sums to CTA q; CTA r adds the CL partials of its rows
// in a fixed tree, normalises and sends the new phase to every CTA.  Both
// messages are asynchronous stores into distributed shared memory that
// count their bytes on the receiver's mbarrier: one one-way latency each,
// where a cluster barrier also waits for the answer.  A receiver's buffer is
// free again when its answer has come back, so one copy of each suffices.
// The entropy of the selected bins, E = ln S1 - ln 2 * S2/S1 with
// S1 = sum |T|^2, S2 = sum |T|^2 log2 |T|^2, comes out of the same epilogue
// and drives the optional stop criterion (iterations that need it take a
// cluster barrier more).
//
// Bound by latency: at 4 bins per CTA and 256 pulses an iteration is ~1700
// clocks of transforms, 500 of the two reductions and 500 for each message.
// Per iteration at U = 64 / 128 (team transforms with block barriers, gathers
// by remote loads and two cluster barriers before -> now): 128 pulses
// 5.4 / 6.2 -> 1.9 / 2.9 us (4 CTAs), 256 pulses 6.2 / 6.4 -> 1.9 / 3.0
// (8 CTAs), 512 pulses 8.1 / 8.8 -> 2.8 / 3.6 (16 CTAs), 1024 pulses
// 6.1 / 7.5 -> 4.2 / 5.9 (16 CTAs).  Two warps per bin (16 elements per lane,
// two tile exchanges) measured slower at 512 and 1024 pulses.
// ---------------------------------------------------------------------------
template <int M>
struct AFC {
    static constexpr int P = M >= 1024 ? 32 : M == 512 ? 16 : 8;   // elements per lane
    static constexpr int L = M / P;                                // lanes per bin
    static constexpr int Q = L / P;
    static constexpr int BW = 32 / L;                              // bins per warp
    static constexpr int WARPS = 8;
    static constexpr int THREADS = WARPS * 32;
    static constexpr int BINS = WARPS * BW;                        // bins per round
    static constexpr int CTAS = M >= 1024 ? 1 : 2;                 // per SM (registers)
    static constexpr int S1 = L + Q;   // tile row stride: both directions free of bank conflicts
    static constexpr int TILE = P * S1;                            // per bin; also its M partial sums
    static constexpr int NSLOT = 2;                                // cached rounds
    static constexpr int BUF = M + 64;                             // [CL][M / CL + pad]
    static constexpr size_t SMEM_F2 =
        (size_t)M + BUF + (size_t)BINS * TILE + (size_t)NSLOT * BINS * M + (size_t)M + (size_t)P * Q;
    static constexpr size_t SMEM = SMEM_F2 * sizeof(float2) + 64 * sizeof(double);
    static_assert(TILE >= M && TILE % 2 == 0 && BUF % 2 == 0, "the tile also holds the bin's partial sums");
    static_assert(P * L == M && P * Q == L && Q <= 4, "exchange pattern");
    static_assert(SMEM <= 227 * 1024, "shared memory");
};

struct AFFrame {
    const float2* cut;     // [M][512]
    const int* bins;       // [U]
    const int* fdec;       // [1] = U
    float2* phase;         // [M] in: Doppler-tracking start phase, out: final phase
    int* stat;             // [0] iterations applied (both legs), [1] entropy bits of the
                           // selected bins at the last evaluated phase, [2] learned leg
                           // kept (set by the image judge), [3], [4] those entropy bits
                           // of the plain and the learned leg, [5], [6] their
                           // iterations; may be null
    float2* alt;           // [M] learned start phase in, the learned leg's final phase
                           // out (warm start), or null
    float2* gcol;          // [U][M] scratch: contiguous copy of the bin columns
    unsigned* err;         // set when a message between the CTAs does not arrive
    int max_u;             // the kernel leaves frames with more bins alone
    unsigned polls;        // limit of a message wait
    unsigned extra;        // bytes expected beyond those sent (test hook)
};

// The DFT over q (q = lane mod Q) of the elements c = 0..P-1 that Q
// neighbouring lanes hold, as radix-2 steps: in a step lanes l and l ^ B keep
// one half of the elements each, so every lane ends with P outputs.  The
// lane with the bit set gets differences with the opposite sign; T |T| is
// odd in T and the mirrored inverse undoes the sign, so it is not corrected.
// step: v[2e], v[2e+1] -> v[2e] = kept + received, v[2e+1] = kept - received.
template <int P, int B>
__device__ __forceinline__ void cross_step(float2* v, bool hi)
{
#pragma unroll
    for (int e = 0; e < P / 2; ++e) {
        const float2 send = hi ? v[2 * e] : v[2 * e + 1], keep = hi ? v[2 * e + 1] : v[2 * e];
        float2 got;
        got.x = __shfl_xor_sync(0xffffffffu, send.x, B);
        got.y = __shfl_xor_sync(0xffffffffu, send.y, B);
        v[2 * e] = cadd(keep, got);
        v[2 * e + 1] = csub(keep, got);
    }
}
// The mirror image: kept = v[2e] + v[2e+1], the difference goes back.
template <int P, int B>
__device__ __forceinline__ void cross_step_back(float2* v, bool hi)
{
#pragma unroll
    for (int e = 0; e < P / 2; ++e) {
        const float2 keep = cadd(v[2 * e], v[2 * e + 1]), send = csub(v[2 * e], v[2 * e + 1]);
        float2 got;
        got.x = __shfl_xor_sync(0xffffffffu, send.x, B);
        got.y = __shfl_xor_sync(0xffffffffu, send.y, B);
        v[2 * e] = hi ? got : keep;
        v[2 * e + 1] = hi ? keep : got;
    }
}
template <int P, int Q>
struct AfCross {
    __device__ __forceinline__ static void forward(float2* v, int q)
    {
        if constexpr (Q == 2) {
            cross_step<P, 1>(v, q & 1);
        } else {
            cross_step<P, 2>(v, q & 2);   // d0 = 0 in even registers, 1 in odd ones
            float2 t[P];
#pragma unroll
            for (int e = 0; e < P / 2; ++e) {   // W_4^(q0 d0), then pair equal d0
                const float2 x = v[2 * e + 1];
                t[e] = v[2 * e];
                t[P / 2 + e] = (q & 1) ? make_float2(x.y, -x.x) : x;
            }
            cross_step<P, 1>(t, q & 1);
#pragma unroll
            for (int e = 0; e < P; ++e) v[e] = t[e];
        }
    }
    __device__ __forceinline__ static void inverse(float2* v, int q)
    {
        if constexpr (Q == 2) {
            cross_step_back<P, 1>(v, q & 1);
        } else {
            cross_step_back<P, 1>(v, q & 1);
            float2 t[P];
#pragma unroll
            for (int e = 0; e < P / 2; ++e) {
                const float2 x = v[P / 2 + e];
                t[2 * e] = v[e];
                t[2 * e + 1] = (q & 1) ? make_float2(-x.y, x.x) : x;
            }
            cross_step_back<P, 2>(t, q & 2);
#pragma unroll
            for (int e = 0; e < P; ++e) v[e] = t[e];
        }
    }
};

// One mbarrier per message direction, one arrival (the receiver's own
// expect_tx) and the message's bytes per phase.  Waits are bounded (leg()
// below says how a CTA goes on after one has run out); kMsgDrainLimit polls
// are the limit of its last wait for messages still in flight.
constexpr unsigned kMsgWaitLimit = 1u << 20;
constexpr unsigned kMsgDrainLimit = 1u << 12;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, int rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void msg_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void msg_expect(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void msg_send(uint32_t dst, uint32_t bar, float2 a)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "f"(a.x), "f"(a.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void msg_send2(uint32_t dst, uint32_t bar, float2 a, float2 b)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool msg_wait(uint64_t* bar, uint32_t parity, unsigned polls)
{
    for (unsigned i = 0; i < polls; ++i) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n"
                     " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done)
                     : "r"(smem_u32(bar)), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

// T -> T |T|; an exact zero stays zero.  |T| is |T|^2 times the hardware's
// reciprocal root.  Error of the whole stage against 64 bits over 60 seeds at
// 128 / 256 / 512 pulses, 60 iterations: 2.47 / 3.21 / 4.88e-7, with sqrtf 2.35 /
// 3.09 / 4.96e-7 at up to 6 % more time (the team kernels with sqrtf before:
// 2.62 / 3.73 / 5.41e-7).
__device__ __forceinline__ float2 times_abs(float2 v, bool ent, float& s1, float& s2)
{
    const float p = v.x * v.x + v.y * v.y;
    if (ent) {
        s1 += p;
        if (p > 0.0f) s2 += p * __log2f(p);
    }
    const float a = p > 0.0f ? p * rsqrtf(p) : 0.0f;
    return make_float2(v.x * a, v.y * a);
}

// s / |s| with one reciprocal square root and a Newton step (as exact as the
// square root and two divisions it stands for, a third of their latency).
// As s / sqrtf(|s|^2): 0 / 0 is NaN, an overflowing |s|^2 gives 0.
__device__ __forceinline__ float2 unit(float2 s)
{
    const float p = s.x * s.x + s.y * s.y;
    float y = rsqrtf(p);
    if (p > 0.0f && p < CUDART_INF_F) y = fmaf(y, fmaf(-0.5f * y * p, y, 0.5f), y);   // y first: p / 2 may round
    return make_float2(s.x * y, s.y * y);
}

// With a learned start (AFFrame::alt) the engine runs two legs: the
// autofocus from the learned start until the stop criterion (`tol`), then the
// plain autofocus, the reference's algorithm (Doppler-tracking start, `iters`
// updates, no stop criterion).  Both final phases are returned (alt, phase);
// the judge downstream images both and keeps the lower final image entropy,
// so a frame on which the learned start ends worse reverts to the plain
// result.  (The entropy of the selected bins cannot judge: it ignores a
// linear phase, a Doppler shift of the image, which MTRC does not.)
//
// A CTA keeps NSLOT rounds of its bins in shared memory; when it has more,
// the others are read from gcol, a contiguous copy of the gathered columns
// ([U][M], written by the loading lanes themselves on entry), and successive
// sweeps alternate direction so that the NSLOT rounds left in shared memory
// by one sweep are the first of the next.
template <int M, int CL>
__global__ void __launch_bounds__(AFC<M>::THREADS, AFC<M>::CTAS)
k_af_cluster(AFFrame f, int iters, float tol, const float2* __restrict__ tw)
{
    namespace cg = cooperative_groups;
    using A = AFC<M>;
    constexpr int P = A::P, L = A::L, Q = A::Q;
    cg::cluster_group cl = cg::this_cluster();
    const int r = (int)cl.block_rank();
    extern __shared__ float4 dyn_smem[];
    __shared__ __align__(8) uint64_t bar_part, bar_ph;          // partial sums, phase slices arrived
    float2* ph = reinterpret_cast<float2*>(dyn_smem);          // [M]
    float2* buf = ph + M;                                       // [CL][bs] partial sums of this CTA's rows
    float2* tiles = buf + A::BUF;                               // [BINS][TILE]
    float2* cache = tiles + A::BINS * A::TILE;                  // [NSLOT][BINS][M]
    float2* T1 = cache + (size_t)A::NSLOT * A::BINS * M;        // [P][L] W_M^(l k)
    float2* T2 = T1 + M;                                        // [P][Q] W_L^(q c)
    double* red = reinterpret_cast<double*>(T2 + P * Q);        // [64]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int slot = tid / L, l = tid & (L - 1);                // bin within a round, lane within the bin
    const int k1 = l / Q, q = l & (Q - 1);
    if (tid == 0) {
        msg_init(&bar_part);
        msg_init(&bar_ph);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < M; i += A::THREADS) T1[i] = tw[(i / L) * (i & (L - 1)) * (kTwN / M)];
    for (int i = tid; i < P * Q; i += A::THREADS) T2[i] = tw[(i / Q) * (i & (Q - 1)) * (kTwN / L)];
    float2* ta = tiles + slot * A::TILE;
    pdl_begin();
    const int U = f.fdec[1];
    if (U > f.max_u) return;   // the whole cluster, before any message
    const int bpc = (U + CL - 1) / CL;
    const int b0 = r * bpc;
    const int nb = max(0, min(bpc, U - b0));
    const int nrd = (nb + A::BINS - 1) / A::BINS;
    const int nact = min(A::BINS, nb);                          // bins with partial sums
    const bool reload = nrd > A::NSLOT;
    float2* gw = f.gcol + (size_t)(b0 + slot) * M;              // its column of round 0

    for (int m = tid; m < M; m += A::THREADS) ph[m] = f.phase[m];
    for (int j = 0; j < nrd; ++j) {
        const int t = j * A::BINS + slot;
        if (j >= A::NSLOT && !reload) continue;
        float2* g = cache + ((size_t)(j % A::NSLOT) * A::BINS + slot) * M;
        if (t >= nb) {   // a half-empty warp computes on zeros
            if (A::BW == 2 && j < A::NSLOT)
                for (int i = 0; i < P; ++i) g[l + L * i] = make_float2(0.0f, 0.0f);
            continue;
        }
        const int b = f.bins[b0 + t];
        float2* gg = gw + (size_t)j * A::BINS * M;
#pragma unroll 4
        for (int i = 0; i < P; ++i) {
            const int m = l + L * i;
            const float2 x = f.cut[(size_t)m * C + b];
            if (j < A::NSLOT) g[m] = x;
            if (reload) gg[m] = x;
        }
    }
    cl.sync();   // every CTA of the cluster runs and has its mbarriers: messages may be sent

    const float invM = 1.0f / (float)M;
    constexpr int rows = M / CL;
    // threads per row of the cluster reduction, and the row stride of buf that
    // keeps their reads in different banks
    constexpr int tpr = CL < A::THREADS / rows ? CL : A::THREADS / rows;
    constexpr int bs = rows + 16 / tpr + ((16 / tpr) & 1);
    static_assert(CL * bs <= A::BUF && rows * tpr <= A::THREADS && (rows * tpr) % 32 == 0, "cluster reduction");
    // twiddles of the short transforms in registers
    constexpr bool kRegTw = P <= 8;
    float2 w1[kRegTw ? P : 1], w2[kRegTw ? P : 1];
    if constexpr (kRegTw) {
#pragma unroll
        for (int k = 0; k < P; ++k) {
            w1[k] = T1[k * L + l];
            w2[k] = T2[k * Q + q];
        }
    }
    auto t1 = [&](int k) {
        if constexpr (kRegTw) return w1[k];
        else return T1[k * L + l];
    };
    auto t2 = [&](int c) {
        if constexpr (kRegTw) return w2[c];
        else return T2[c * Q + q];
    };
    int nsweep = 0;
    uint32_t par = 0;   // phase parity of both mbarriers: bit 0 bar_part, bit 1 bar_ph
    unsigned polls = f.polls;   // 0 once one of this thread's waits has run out
    auto await = [&](uint64_t* bar, uint32_t bit) {
        const uint32_t parity = (par & bit) ? 1u : 0u;
        par ^= bit;
        if (__builtin_expect(!msg_wait(bar, parity, polls), 0)) {
            polls = 0;
            par ^= bit;
            atomicOr(f.err, 1u);
        }
    };

    // One sweep over this CTA's bins with the phase in ph: entropy sums
    // (s1, s2, only when `ent`) and the partial row sums of the update, sent
    // to the CTAs that own the rows (by threads whose waits have not run out).
    auto sweep = [&](bool ent, float& s1, float& s2) {
        float2 pacc[P];
#pragma unroll
        for (int i = 0; i < P; ++i) pacc[i] = make_float2(0.0f, 0.0f);
        const bool back = (nsweep++ & 1) != 0;
#pragma unroll 1
        for (int jj = 0; jj < nrd; ++jj) {
            const int j = back ? nrd - 1 - jj : jj;
            if (j * A::BINS + warp * A::BW >= nb) continue;   // warp-uniform; no block barrier inside
            float2* g = cache + ((size_t)(j % A::NSLOT) * A::BINS + slot) * M;
            __syncwarp();   // the slot and the tile of the previous round are read
            if (jj >= A::NSLOT) {   // only when reload: read the copy in gcol
                const bool valid = A::BW == 1 || j * A::BINS + slot < nb;
                const float4* src = reinterpret_cast<const float4*>(gw + (size_t)j * A::BINS * M);
                float4* dst = reinterpret_cast<float4*>(g);
#pragma unroll 4
                for (int i = l; i < M / 2; i += L) dst[i] = valid ? src[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            __syncwarp();
            float2 v[P];
#pragma unroll
            for (int i = 0; i < P; ++i) v[i] = cmul(ph[l + L * i], g[l + L * i]);
            if constexpr (Q == 1) {
                // pass 0: T = FFT(phase * g); pass 1: conj(IFFT(T |T|)) * M as
                // the forward FFT of conj(T |T|)
#pragma unroll 1
                for (int pass = 0; pass < 2; ++pass) {
                    // two DFT steps sharing one copy of the code
#pragma unroll 1
                    for (int step = 0;; ++step) {
                        dft32_reg(v);
                        if (step == 1) break;
#pragma unroll
                        for (int k = 1; k < P; ++k) v[k] = cmul(v[k], T1[k * L + l]);
#pragma unroll
                        for (int k = 0; k < P; ++k) ta[l * A::S1 + k] = v[k];
                        __syncwarp();
#pragma unroll
                        for (int n = 0; n < P; ++n) v[n] = ta[n * A::S1 + l];
                        __syncwarp();
                    }
                    if (pass == 0) {
#pragma unroll
                        for (int i = 0; i < P; ++i) v[i] = conjf2(times_abs(v[i], ent, s1, s2));
                    } else {
                        // conj(g) conj(v) = conj(g v): the conjugate is applied once per sweep
#pragma unroll
                        for (int i = 0; i < P; ++i) {
                            const float2 x = g[l + L * i];
                            pacc[i].x = fmaf(x.x, v[i].x, fmaf(-x.y, v[i].y, pacc[i].x));
                            pacc[i].y = fmaf(x.x, v[i].y, fmaf(x.y, v[i].x, pacc[i].y));
                        }
                    }
                }
            } else {
                dft_reg<P, false>(v);
#pragma unroll
                for (int k = 1; k < P; ++k) v[k] = cmul(v[k], t1(k));
#pragma unroll
                for (int k = 0; k < P; ++k) ta[k * A::S1 + l] = v[k];
                __syncwarp();
#pragma unroll
                for (int b = 0; b < P; ++b) v[b] = ta[k1 * A::S1 + q + Q * b];
                dft_reg<P, false>(v);
#pragma unroll
                for (int c = 1; c < P; ++c) v[c] = cmul(v[c], t2(c));
                AfCross<P, Q>::forward(v, q);
#pragma unroll
                for (int i = 0; i < P; ++i) v[i] = times_abs(v[i], ent, s1, s2);
                AfCross<P, Q>::inverse(v, q);
#pragma unroll
                for (int c = 1; c < P; ++c) v[c] = cmulc(t2(c), v[c]);
                dft_reg<P, true>(v);
                __syncwarp();   // every lane has read the tile
#pragma unroll
                for (int b = 0; b < P; ++b) ta[k1 * A::S1 + q + Q * b] = v[b];
                __syncwarp();
#pragma unroll
                for (int k = 0; k < P; ++k) v[k] = ta[k * A::S1 + l];
#pragma unroll
                for (int k = 1; k < P; ++k) v[k] = cmulc(t1(k), v[k]);
                dft_reg<P, true>(v);
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    const float2 x = g[l + L * i];   // conj(x) v
                    pacc[i].x = fmaf(x.x, v[i].x, fmaf(x.y, v[i].y, pacc[i].x));
                    pacc[i].y = fmaf(x.x, v[i].y, fmaf(-x.y, v[i].x, pacc[i].y));
                }
            }
        }
        // the bins' sums to the rows' owners, two rows per message
        __syncwarp();   // the tile is read
        if (slot < nact) {
            const float sy = Q == 1 ? -invM : invM;
#pragma unroll
            for (int i = 0; i < P; ++i) ta[l + L * i] = make_float2(pacc[i].x * invM, pacc[i].y * sy);
        }
        __syncthreads();
        if (polls == 0) return;
        for (int m = 2 * tid; m < M; m += 2 * A::THREADS) {
            float2 a = make_float2(0.0f, 0.0f), b = a;
#pragma unroll
            for (int x = 0; x < A::BINS; ++x)
                if (x < nact) {
                    const float4 t = *reinterpret_cast<const float4*>(&tiles[x * A::TILE + m]);
                    a = cadd(a, make_float2(t.x, t.y));
                    b = cadd(b, make_float2(t.z, t.w));
                }
            const int to = m / rows;
            msg_send2(cluster_addr(smem_u32(&buf[r * bs + (m & (rows - 1))]), to), cluster_addr(smem_u32(&bar_part), to),
                      a, b);
        }
    };

    // Entropy of the selected bins, in two halves around a cluster barrier:
    // this CTA's sums (s1 = sum p, s2 = sum p log2 p) into one of two slots,
    // red[32..33] and red[34..35] in turn, then after the barrier warp 0 adds
    // the CL CTAs' sums (one remote read per lane, a fixed-order tree: every CTA
    // gets the same value) and returns ln S1 - ln 2 * S2 / S1 in lane 0 of warp 0.
    // A CTA writes a slot again after the next barrier, which no CTA passes
    // before all have read it.
    int eslot = 32;
    auto entropy_part = [&](float s1, float s2) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        if (lane == 0) {
            red[warp] = s1;
            red[16 + warp] = s2;
        }
        __syncthreads();
        if (tid == 0) {
            double a1 = 0.0, a2 = 0.0;
            for (int w = 0; w < A::WARPS; ++w) {
                a1 += red[w];
                a2 += red[16 + w];
            }
            red[eslot] = a1;
            red[eslot + 1] = a2;
        }
    };
    auto entropy_total = [&]() {   // warp 0, after the cluster barrier
        double S1 = 0.0, S2 = 0.0;
        if (lane < CL) {
            const double* rr = cl.map_shared_rank(red, lane);
            S1 = rr[eslot];
            S2 = rr[eslot + 1];
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            S1 += __shfl_xor_sync(0xffffffffu, S1, o);
            S2 += __shfl_xor_sync(0xffffffffu, S2, o);
        }
        return logf((float)S1) - kLn2 * (float)S2 / (float)S1;
    };

    // One autofocus run from the phase in ph: up to `iters` updates, fewer
    // when the stop criterion ends it.  Returns, in warp 0, the entropy at the
    // last evaluated phase.
    //
    // A thread whose wait has run out waits no more, sends no message and, thread
    // 0, expects none: a phase that has not completed gets no second arrival,
    // and at most one phase's bytes come unexpected.  The peers then miss its
    // messages and run out in the same way; whoever does not can only be one whose
    // messages are all there.  All threads go on through the sweeps and their
    // barriers and meet at every cluster barrier, whose number depends only on
    // the iteration count and on the entropies, the same in all CTAs.
    auto leg = [&](float ltol, int& used) -> float {
        float e_prev = 0.0f, e_last = 0.0f;   // meaningful in warp 0
        used = iters;
#pragma unroll 1
        for (int it = 0; it < iters; ++it) {
            // the entropy is needed by the stop criterion or for the last trace
            const bool check = ltol > 0.0f && it % kStopEvery == 0;
            const bool need_e = check || it == iters - 1;
            float s1 = 0.0f, s2 = 0.0f;
            sweep(need_e, s1, s2);
            bool stop = false;
            if (need_e) {
                entropy_part(s1, s2);
                cl.sync();   // the slots of every CTA are complete
                if (warp == 0) {
                    const float E = entropy_total();
                    if (check) {
                        stop = it > 0 && fabsf(E - e_prev) <= (float)kStopEvery * ltol * fabsf(E);
                        e_prev = E;
                    }
                    e_last = E;
                    if (lane == 0) red[40] = stop ? 1.0 : 0.0;
                }
                __syncthreads();
                stop = red[40] != 0.0;
                eslot ^= 2;
            }
            if (tid == 0 && polls > 0) msg_expect(&bar_part, M * sizeof(float2) + f.extra);
            await(&bar_part, 1u);
            if (stop) {
                cl.sync();   // every CTA has these messages: the next leg may send
                used = it;
                break;
            }
            // tpr neighbouring threads add a row's CL partial sums (fixed
            // tree) and send its new phase to CL / tpr CTAs each
            if (tid < rows * tpr) {
                const int part = tid & (tpr - 1), ml = tid / tpr;
                float2 s = buf[part * bs + ml];
#pragma unroll
                for (int x = tpr; x < CL; x += tpr) s = cadd(s, buf[(part + x) * bs + ml]);
#pragma unroll
                for (int o = tpr >> 1; o > 0; o >>= 1) {
                    float2 t;
                    t.x = __shfl_xor_sync(0xffffffffu, s.x, o);
                    t.y = __shfl_xor_sync(0xffffffffu, s.y, o);
                    s = cadd(s, t);
                }
                s = unit(s);
                if (polls > 0) {
#pragma unroll
                    for (int x = 0; x < CL; x += tpr)
                        msg_send(cluster_addr(smem_u32(&ph[r * rows + ml]), part + x),
                                 cluster_addr(smem_u32(&bar_ph), part + x), s);
                }
            }
            if (tid == 0 && polls > 0) msg_expect(&bar_ph, M * sizeof(float2));
            await(&bar_ph, 2u);
        }
        return e_last;
    };
    // No CTA leaves while another may still send to it.  One that has received
    // all it waited for is done once the others send no more (the barrier); one
    // that gave up waits again, with a limit, for messages still in flight.
    auto leave = [&]() {
        cl.sync();
        if (polls == 0) {
            msg_wait(&bar_part, par & 1u, kMsgDrainLimit);
            msg_wait(&bar_ph, par >> 1, kMsgDrainLimit);
        }
    };

    if (!f.alt) {
        int used;
        const float e = leg(tol, used);
        for (int m = r * rows + tid; m < (r + 1) * rows; m += A::THREADS) f.phase[m] = ph[m];
        if (r == 0 && tid == 0 && f.stat) {
            f.stat[0] = used;
            f.stat[1] = __float_as_int(e);
        }
        leave();
        return;
    }
    // the learned leg, then the plain leg (one copy of the code)
    int used[2];
    float e[2];
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        float2* p = k == 0 ? f.alt : f.phase;
        __syncthreads();
        for (int m = tid; m < M; m += A::THREADS) ph[m] = p[m];
        __syncthreads();
        int u;
        const float x = leg(k == 0 ? tol : 0.0f, u);
        if (k == 0) {
            used[0] = u;
            e[0] = x;
        } else {
            used[1] = u;
            e[1] = x;
        }
        for (int m = r * rows + tid; m < (r + 1) * rows; m += A::THREADS) p[m] = ph[m];
    }
    if (r == 0 && tid == 0 && f.stat) {
        f.stat[0] = used[0] + used[1];
        f.stat[1] = __float_as_int(e[1]);
        f.stat[2] = 0;
        f.stat[3] = __float_as_int(e[1]);
        f.stat[4] = __float_as_int(e[0]);
        f.stat[5] = used[1];
        f.stat[6] = used[0];
    }
    leave();
}

// cut[m][c] *= phase[m]  (phase_adjustment.cu:324)
__global__ void k_af_apply(float2* __restrict__ cut, const float2* __restrict__ phase, int M)
{
    pdl_begin();
    const int m = blockIdx.x;
    const float2 p = phase[m];
    for (int c = threadIdx.x; c < C; c += blockDim.x) cut[(size_t)m * C + c] = cmul(p, cut[(size_t)m * C + c]);
}

// Both legs of a warm-started frame in one pass: cut2 = diag(phase_l) cut
// (the learned leg), then cut = diag(phase) cut in place (the plain leg).
__global__ void k_af_apply2(float2* __restrict__ cut, const float2* __restrict__ phase,
                            const float2* __restrict__ phase_l, float2* __restrict__ cut2, int M)
{
    const int m = blockIdx.x;
    const float2 p = phase[m], pl = phase_l[m];
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        const float2 x = cut[(size_t)m * C + c];
        cut2[(size_t)m * C + c] = cmul(pl, x);
        cut[(size_t)m * C + c] = cmul(p, x);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <int M>
static constexpr int af_cb() { return M >= 512 ? 8 : (M >= 256 ? 16 : 32); }

using AfKernel = void (*)(AFFrame, int, float, const float2*);
template <int M>
static AfKernel af_kernel(int cl)
{
    return cl == 16 ? k_af_cluster<M, 16> : cl == 8 ? k_af_cluster<M, 8> : k_af_cluster<M, 4>;
}

// The launch of one cluster of cl CTAs (the two attributes `at` must outlive
// the configuration).
template <int M>
static cudaLaunchConfig_t af_cluster_config(int cl, bool overlap, cudaStream_t st, cudaLaunchAttribute* at)
{
    cudaLaunchConfig_t cfg = {};
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = cl;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.gridDim = dim3(cl);
    cfg.blockDim = dim3(AFC<M>::THREADS);
    cfg.dynamicSmemBytes = AFC<M>::SMEM;
    cfg.stream = st;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 2 : 1;
    return cfg;
}

// Cluster engine set-up (once per device): shared-memory limit, non-portable
// cluster sizes, and the largest of 16/8/4 CTAs per cluster that can be
// resident.  Returns that size, 0 if none, or a negative cudaError_t.
template <int M>
static int af_cluster_probe()
{
    int best = 0;
    for (int cl : {16, 8, 4}) {
        const AfKernel k = af_kernel<M>(cl);
        cudaError_t e;
        if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AFC<M>::SMEM)))
            return -(int)e;
        if (cl > 8 && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))
            (void)cudaGetLastError();
        cudaLaunchAttribute at[2];
        const cudaLaunchConfig_t cfg = af_cluster_config<M>(cl, false, nullptr, at);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n > 0 && best == 0) best = cl;
        (void)cudaGetLastError();
    }
    return best;
}

template <int M>
static int af_cluster_setup()
{
    static PerDevice max_cl;
    return max_cl.get(af_cluster_probe<M>);
}

template <int M>
static cudaError_t af_cluster_launch(const FEArgs& a, int cl, int max_u, cudaStream_t st)
{
    const int mx = af_cluster_setup<M>();
    if (mx < 0) return (cudaError_t)(-mx);
    if (cl != 4 && cl != 8 && cl != 16) return cudaErrorInvalidValue;
    if (cl > mx) return cudaErrorInvalidClusterSize;
    cudaLaunchAttribute at[2];
    const cudaLaunchConfig_t cfg = af_cluster_config<M>(cl, a.overlap != 0, st, at);
    AFFrame fr{a.cut, a.bins, a.fdec, a.phase, a.af_stat, a.ws_w ? a.ws_phase : nullptr, a.gcol, a.bar + 3, max_u,
               a.bar_test.limit == kSpinLimit ? kMsgWaitLimit : (unsigned)a.bar_test.limit, a.bar_test.extra ? 16u : 0u};
    cudaError_t e = cudaLaunchKernelEx(&cfg, af_kernel<M>(cl), fr, a.iters, a.tol, a.tw);
    if (e == cudaSuccess) ISAR_COUNT(1);
    return e;
}

int af_cluster_max(int M)
{
    int r = 0;
    switch (M) {
    case 128: r = af_cluster_setup<128>(); break;
    case 256: r = af_cluster_setup<256>(); break;
    case 512: r = af_cluster_setup<512>(); break;
    case 1024: r = af_cluster_setup<1024>(); break;
    default: return 0;
    }
    return r < 0 ? 0 : r;
}

template <int M>
static cudaError_t fe_run_m(const FEArgs& a, cudaStream_t st)
{
    constexpr int CB = af_cb<M>();
    using F = FFTShape<M>;
    const size_t smem = ((size_t)CB * F::SMEM + TwShared<M>::kEntries) * sizeof(float2);
    const size_t smem_p = (size_t)4 * M * sizeof(float2) + (size_t)4 * F::SMEM * sizeof(float2) + M * sizeof(float2) +
                          TwShared<M>::kEntries * sizeof(float2);
    // per device: shared-memory limits, and whether the cooperative grid of
    // 128 CTAs (at most 4 of the <= 512 bins each) can be co-resident
    static PerDevice setup;
    const int su = setup.get([smem, smem_p]() -> int {
        cudaError_t e;
        if ((e = cudaFuncSetAttribute(k_fe_colfft<M, CB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)))
            return -(int)e;
        if ((e = cudaFuncSetAttribute(k_af_persist<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_p)))
            return -(int)e;
        int dev = 0, sms = 0, per_sm = 0;
        if ((e = cudaGetDevice(&dev))) return -(int)e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev))) return -(int)e;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_af_persist<M>, 4 * F::T, smem_p)))
            return -(int)e;
        return per_sm * sms;
    });
    if (su < 0) return (cudaError_t)(-su);
    constexpr int grid_p = 128;
    if (su < grid_p) return cudaErrorCooperativeLaunchTooLarge;
    const int rows_max = M < 256 ? M : 256;
    const int R = 8;
    const int nparts = (rows_max + R - 1) / R;
    cudaError_t e;
    if ((e = launch_after(a.overlap == 1, k_fe_stats, (M + R - 1) / R, 256, 0, st, a.cut, M, rows_max, R, a.cmax_part, a.dsum)))
        return e;
    if ((e = launch_after(a.overlap, k_fe_phase, M / 32, M, 0, st, a.cmax_part, nparts, a.dsum, M, a.phase, a.fdec)))
        return e;
    if ((e = launch_after(a.overlap, k_fe_colfft<M, CB>, C / CB, CB * F::T, smem, st, a.cut, a.phase, a.E, a.H, a.tw)))
        return e;
    if ((e = launch_after(a.overlap, k_fe_select, 1, C, 0, st, a.E, a.H, a.fdec, a.bins))) return e;
    if ((e = launch_after(a.overlap, k_af_doppler, (M * 32 + 255) / 256, 256, 0, st, a.cut, a.bins, a.fdec, M, a.dsum)))
        return e;
    if ((e = launch_after(a.overlap, k_fe_phase, M / 32, M, 0, st, nullptr, 0, a.dsum, M, a.phase, a.fdec))) return e;
    if (a.pre_only) return cudaGetLastError();
    if (a.ws_w && (a.af_cluster == 0 || a.iters == 0)) return cudaErrorInvalidValue;
    if (a.ws_w) {
        // learned warm start: features -> network -> second start phase
        if ((e = nn::features(a.cut, a.E, a.dsum, M, a.ws_a->act[0], a.ws_psi, st))) return e;
        if ((e = nn::forward(*a.ws_w, *a.ws_a, 1, M, a.ws_err, st))) return e;
        if ((e = nn::ws_phase(a.ws_psi, a.ws_a->out, M, a.ws_phase, st))) return e;
    }
    // The choice by bins (512 pulses): a cluster of 16 takes 2.8 us per iteration
    // at U = 64 and 6.0 at U = 256, the grid 7.6 and 7.8; only at the largest U,
    // 512 (profiles below one count: the integer mean of the threshold is 0), is
    // the grid ahead (8 against 10).  U is known on the device only: both kernels
    // are launched and the one that it does not select returns at once.
    const int cl = a.af_auto ? 16 : a.af_cluster;
    const int max_u = a.af_auto ? 256 : C;
    if (a.iters > 0 && cl > 0) {
        if ((e = af_cluster_launch<M>(a, cl, max_u, st))) return e;
    }
    if (a.iters > 0 && (cl == 0 || max_u < C)) {
        if ((e = cudaMemsetAsync(a.bar, 0, 2 * sizeof(unsigned), st))) return e;
        int min_u = cl == 0 ? 0 : max_u + 1;
        const float2* cut = a.cut;
        const int* bins = a.bins;
        const int* fdec = a.fdec;
        float2* phase = a.phase;
        float2* P = a.sig_part;
        unsigned* bar = a.bar;
        int* err = reinterpret_cast<int*>(a.bar + 1);
        int iters = a.iters;
        const float2* tw = a.tw;
        BarrierTest bt = a.bar_test;
        void* args[] = {(void*)&cut, (void*)&bins, (void*)&fdec, (void*)&phase, (void*)&P,
                        (void*)&bar, (void*)&err, (void*)&iters, (void*)&tw, (void*)&bt, (void*)&min_u};
        if ((e = cudaLaunchCooperativeKernel((const void*)k_af_persist<M>, dim3(grid_p), dim3(4 * F::T), args, smem_p,
                                             st)))
            return e;
        ISAR_COUNT(1);
    }
    if (a.defer_apply) return cudaGetLastError();   // the imaging applies the phase(s)
    if (a.ws_w && a.iters > 0 && a.af_cluster > 0) {
        k_af_apply2<<<M, 256, 0, st>>>(a.cut, a.phase, a.ws_phase, a.cut2, M);
        ISAR_COUNT(1);
        return cudaGetLastError();
    }
    return launch_after(a.overlap, k_af_apply, M, 256, 0, st, a.cut, a.phase, M);
}

cudaError_t fe_run(const FEArgs& a, cudaStream_t st)
{
    switch (a.M) {
    case 128: return fe_run_m<128>(a, st);
    case 256: return fe_run_m<256>(a, st);
    case 512: return fe_run_m<512>(a, st);
    case 1024: return fe_run_m<1024>(a, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace isar

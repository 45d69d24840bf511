// Windowed statistics of the stream and preparation of the query.
//
// Reference: include/stats.cuh.  The reference makes two FP64 prefix sums over
// the whole stream (CUB scans, 2 cudaMalloc + 5 kernels per 1e7-sample epoch,
// stats.cuh:85-142) and then takes the variance in FP32 (stats.cuh:49), which
// loses the variance of level-shifted signals.  Here one kernel reads the
// stream once per tile of kTileWindows windows: FP64 sums of (x-c) and
// (x-c)^2 per chunk of 16 samples, c the chunk's first one, joined over blocks
// of two, four, ... chunks, and per thread 16 windows slid from one that is
// put together from such blocks.  Output per window: mean (FP64) and sigma
// (FP32), 12 bytes.
#include "common.cuh"

#include <algorithm>

namespace cdtw {

namespace {

constexpr int kStatsRounds = 64;                 // rounds of 32 windows per warp
constexpr int kStatsWarpWindows = 32 * kStatsRounds;
constexpr int kStatsBlock = 128;                 // 4 warps per block
constexpr int kStatsSub = 4;                     // interleaved sub-runs per warp

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Windows of any length, a warp per run of kStatsWarpWindows: serves the
// lengths above kTileMaxM, whose tile would not fit shared memory.
template <class XT, class ST, bool INV>
__global__ void __launch_bounds__(kStatsBlock)
avg_std_long_kernel(const XT* __restrict__ x, int64_t N, int M, double* __restrict__ mu,
                    ST* __restrict__ sigma) {
    // The warp's run of kStatsWarpWindows windows is split into kStatsSub
    // sub-runs, each with its own shift c and starting sums; their scans are
    // interleaved round by round (independent shuffle / FP64 chains).
    const int64_t Nw = N - M + 1;
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t)blockIdx.x * (kStatsBlock / 32) + (threadIdx.x >> 5);
    const int64_t a = warp * kStatsWarpWindows;
    if (a >= Nw) return;
    constexpr int kSubRounds = kStatsRounds / kStatsSub;
    constexpr int kSubWindows = 32 * kSubRounds;
    double c[kStatsSub], s1[kStatsSub], s2[kStatsSub];
#pragma unroll
    for (int u = 0; u < kStatsSub; ++u) {
        const int64_t as = min(a + (int64_t)u * kSubWindows, Nw - 1);
        c[u] = (double)x[as];
        s1[u] = 0.0;
        s2[u] = 0.0;
    }
    // sums of the first window of every sub-run
    for (int k = lane; k < M; k += 32) {
#pragma unroll
        for (int u = 0; u < kStatsSub; ++u) {
            const int64_t as = min(a + (int64_t)u * kSubWindows, Nw - 1);
            const double v = (double)x[as + k] - c[u];
            s1[u] += v;
            s2[u] = fma(v, v, s2[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < kStatsSub; ++u) {
        s1[u] = warp_sum(s1[u]);
        s2[u] = warp_sum(s2[u]);
    }
    const double invM = 1.0 / (double)M;
    for (int r = 0; r < kSubRounds; ++r) {
        if (a + (int64_t)r * 32 >= Nw) break;  // warp-uniform (sub-run 0 ends first)
        double d1[kStatsSub], d2[kStatsSub];
        int64_t wv[kStatsSub];
#pragma unroll
        for (int u = 0; u < kStatsSub; ++u) {
            const int64_t w = a + (int64_t)u * kSubWindows + (int64_t)r * 32 + lane;
            wv[u] = w;
            d1[u] = 0.0;
            d2[u] = 0.0;
            if (w < Nw - 1) {
                // window w+1 = window w + x[w+M] - x[w]
                const double vin = (double)x[w + M] - c[u], vout = (double)x[w] - c[u];
                d1[u] = vin - vout;
                d2[u] = vin * vin - vout * vout;
            }
        }
        double i1[kStatsSub], i2[kStatsSub];
#pragma unroll
        for (int u = 0; u < kStatsSub; ++u) {
            i1[u] = d1[u];
            i2[u] = d2[u];
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int u = 0; u < kStatsSub; ++u) {
                const double t1 = __shfl_up_sync(0xffffffffu, i1[u], o);
                const double t2 = __shfl_up_sync(0xffffffffu, i2[u], o);
                if (lane >= o) {
                    i1[u] += t1;
                    i2[u] += t2;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kStatsSub; ++u) {
            // sums of window w: base + exclusive scan
            const double w1 = s1[u] + (i1[u] - d1[u]), w2 = s2[u] + (i2[u] - d2[u]);
            if (wv[u] < Nw) {
                const double m1 = w1 * invM;
                const double var = w2 * invM - m1 * m1;
                if (mu) mu[wv[u]] = c[u] + m1;
                const double sd = var > 0.0 ? sqrt(var) : 1.0;
                sigma[wv[u]] = INV ? (ST)(1.0 / sd) : (ST)sd;
            }
            s1[u] += __shfl_sync(0xffffffffu, i1[u], 31);
            s2[u] += __shfl_sync(0xffffffffu, i2[u], 31);
        }
    }
}

// Deviation of a positive variance.  For the FP32 result: an FP32 estimate
// (s0 = v * rsqrt(v)) and one Heron step whose residual v - s0^2 is taken in
// FP64, so the result is the FP64 root rounded to FP32 but for ties within
// 1e-6 ulp (an estimate within 2e-7 leaves 4e-14 of the root), at a fraction of
// the FP64 square root's instructions.
template <bool INV>
__device__ __forceinline__ double std_of(double var, double) {
    return var > 0.0 ? (INV ? rsqrt(var) : sqrt(var)) : 1.0;
}
template <bool INV>
__device__ __forceinline__ float std_of(double var, float) {
    static_assert(!INV, "the reciprocal is FP64 only");
    const float v = (float)var;
    if (!(v > 1e-30f && v < 1e30f)) return var > 0.0 ? (float)sqrt(var) : 1.0f;
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
    const float s0 = v * y;
    const double s = (double)s0;
    return fmaf((float)fma(-s, s, var), 0.5f * y, s0);
}

// One block per tile of kTileWindows windows, kTileR = 16 consecutive windows
// per thread.  The tile's kTileWindows + M samples are staged in shared memory
// with one 16-byte pad per 16 samples, so a warp's 16-byte accesses (lanes 16
// samples apart) fall on all banks; chunk c holds samples 16c .. 16c+15.  Blocks
// of 2^k chunks, from every chunk on, hold their sums about their first sample;
// a thread's first window is the sum of the blocks of M / 16's binary digits and
// the M mod 16 samples behind them, moved to its own first sample; the others
// follow by sliding, the leaving samples still in registers.  Results go out
// through shared memory in whole lines.
//
// No sum holds samples outside the thread's 16 windows, so nothing else in the
// tile (a level shift, a flat run, a bad sample) touches them: a constant window
// has variance exactly 0 (sigma 1).  What is left is the slide: where the
// variance is below kLost of the second moment it came from (a large sample that
// left), or a NaN or Inf sample left, the windows behind are summed again, the
// first by the warp in two passes, the next slid from it.  For M < 16 a sample
// may enter and leave within the 16 windows, so there the moment is that of all
// their samples, and such windows are summed one by one.
//
// Precision: with the sums as differences of prefixes over the tile, FP64
// sigmas were off by up to 9e-13 (ECG-like, M = 64; 8e-14 by the run of 512
// windows of avg_std_long_kernel), now 5e-14.
//
// Bound: HBM (16 bytes a window, 82 us at 2^25 windows and 6546 GB/s) if the
// latencies of a block's phases were hidden.  Six blocks per SM (80 registers,
// 84 bytes spilled) measured best at 2^25 windows, M = 512: 144 us, five 155;
// for FP64 sigmas four (no spills).  2^20 windows, M = 128: 10 us; a warp per
// 2048 windows and scans of 32 windows a round took 196 and 22.  A NaN every
// 3000 samples, M = 2000, 2^20 windows: 19 us, 12 without them.
constexpr int kTileThreads = 128;
constexpr int kTileR = 16;                                // windows per thread, samples per chunk
constexpr int kTileWindows = kTileThreads * kTileR;       // 2048
constexpr int kTileMaxM = 8192;

// Element i of an array of T with one 16-byte pad per 16 elements.
template <class T>
__host__ __device__ constexpr int tile_at(int i) {
    return i + (int)(16 / sizeof(T)) * (i >> 4);
}

template <class XT, class ST>
size_t tile_smem(int M) {
    const int S = (int)round_up(kTileWindows + M, kTileR), NC = S / kTileR;
    const size_t in = sizeof(XT) * (size_t)tile_at<XT>(S) + (2 * sizeof(double2) + sizeof(XT)) * (size_t)NC;
    return std::max(in, sizeof(double) * (size_t)tile_at<double>(kTileWindows));
}

// Elements 16c .. 16c+15 of a padded array, by 16-byte loads.
__device__ __forceinline__ void tile_load16(const float* p, float (&v)[16]) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const float4 a = reinterpret_cast<const float4*>(p)[g];
        v[4 * g] = a.x;
        v[4 * g + 1] = a.y;
        v[4 * g + 2] = a.z;
        v[4 * g + 3] = a.w;
    }
}
__device__ __forceinline__ void tile_load16(const double* p, double (&v)[16]) {
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        const double2 a = reinterpret_cast<const double2*>(p)[g];
        v[2 * g] = a.x;
        v[2 * g + 1] = a.y;
    }
}
__device__ __forceinline__ void tile_store16(float* p, const float (&v)[16]) {
#pragma unroll
    for (int g = 0; g < 4; ++g)
        reinterpret_cast<float4*>(p)[g] =
            make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
}
__device__ __forceinline__ void tile_store16(double* p, const double (&v)[16]) {
#pragma unroll
    for (int g = 0; g < 8; ++g)
        reinterpret_cast<double2*>(p)[g] = make_double2(v[2 * g], v[2 * g + 1]);
}

// The 16 samples that enter thread t's windows, 16t + M .. 16t + M + 15: the
// aligned vectors that cover them, shifted down by M mod V (the same for every
// thread).
__device__ __forceinline__ void tile_entering(const float* xs, int t, int M, float (&v)[16]) {
    float y[20];
    const int u0 = M & ~3;
#pragma unroll
    for (int g = 0; g < 5; ++g) {
        const int u = min(u0 + 4 * g, ((M + 15) & ~3));
        const float4 a = *reinterpret_cast<const float4*>(xs + 20 * t + tile_at<float>(u));
        y[4 * g] = a.x;
        y[4 * g + 1] = a.y;
        y[4 * g + 2] = a.z;
        y[4 * g + 3] = a.w;
    }
    const bool b1 = M & 1, b2 = M & 2;
#pragma unroll
    for (int k = 0; k < 18; ++k) y[k] = b2 ? y[k + 2] : y[k];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = b1 ? y[k + 1] : y[k];
}
__device__ __forceinline__ void tile_entering(const double* xs, int t, int M, double (&v)[16]) {
    double y[18];
    const int u0 = M & ~1;
#pragma unroll
    for (int g = 0; g < 9; ++g) {
        const int u = min(u0 + 2 * g, ((M + 15) & ~1));
        const double2 a = *reinterpret_cast<const double2*>(xs + 18 * t + tile_at<double>(u));
        y[2 * g] = a.x;
        y[2 * g + 1] = a.y;
    }
    const bool b1 = M & 1;
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = b1 ? y[k + 1] : y[k];
}

// Mean and variance of the window x[0 .. M) in two passes, the samples from
// `lane` on, `lanes` apart (1: by one thread; 32: by a warp, all of whose lanes
// get both).
template <int lanes, class XT>
__device__ __noinline__ double2 window_stats(const XT* __restrict__ x, int M, int lane) {
    const double f = (double)x[0], invM = 1.0 / (double)M;
    double m = 0.0, v = 0.0;
    for (int k = lane; k < M; k += lanes) m += (double)x[k] - f;
    m = f + (lanes == 32 ? warp_sum(m) : m) * invM;
    for (int k = lane; k < M; k += lanes) {
        const double d = (double)x[k] - m;
        v = fma(d, d, v);
    }
    return make_double2(m, (lanes == 32 ? warp_sum(v) : v) * invM);
}

// The sums (s1, s2) of n samples about g as part of sums about g - dl, added
// to (a1, a2).
__device__ __forceinline__ void tile_add(double& a1, double& a2, const double2& s, double dl,
                                         double n) {
    const double e = n * dl;
    a1 += s.x + e;
    a2 += fma(dl, fma(2.0, s.x, e), s.y);
}

// The tile's n results, 16 of them in each thread's v, to out through z (16-byte
// lines where out is aligned; the block's earlier accesses to z are done after
// the first barrier).
template <class T>
__device__ __forceinline__ void tile_out(T* z, const T (&v)[kTileR], T* __restrict__ out, int n) {
    constexpr int V = 16 / (int)sizeof(T);
    const int t = threadIdx.x;
    __syncthreads();
    tile_store16(z + tile_at<T>(kTileR * t), v);
    __syncthreads();
    if (n == kTileWindows && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
#pragma unroll
        for (int i = V * t; i < kTileWindows; i += V * kTileThreads)
            *reinterpret_cast<int4*>(out + i) = *reinterpret_cast<const int4*>(z + tile_at<T>(i));
    } else {
        for (int i = t; i < n; i += kTileThreads) out[i] = z[tile_at<T>(i)];
    }
}

// mu may be null (not wanted); INV: sigma takes 1 / sigma.
template <class XT, class ST, bool INV>
__global__ void __launch_bounds__(kTileThreads, sizeof(ST) == 8 ? 4 : 6)
avg_std_kernel(const XT* __restrict__ x, int64_t N, int M, double* __restrict__ mu,
               ST* __restrict__ sigma) {
    extern __shared__ __align__(16) unsigned char tsm[];
    constexpr int V = 16 / (int)sizeof(XT);  // samples of a 16-byte vector
    // variance, of the second moment it is left from, below which it is taken again
    constexpr unsigned kAll = (1u << kTileR) - 1u;
    constexpr double kLost = sizeof(ST) == 8 ? 0x1p-10 : 0x1p-22;
    const int64_t Nw = N - M + 1;
    const int64_t t0 = (int64_t)blockIdx.x * kTileWindows;
    const int t = threadIdx.x, lane = t & 31;
    const int S = (kTileWindows + M + kTileR - 1) / kTileR * kTileR, NC = S / kTileR;
    XT* xs = (XT*)tsm;
    double2* cur = (double2*)(xs + tile_at<XT>(S));  // sums of blocks of chunks from each chunk on
    double2* nxt = cur + NC;
    XT* fs = (XT*)(nxt + NC);  // first sample of every chunk
    const XT* __restrict__ xt = x + t0;
    if (M == 1) {  // every variance would be lost: 4 times the time
        for (int64_t i = t0 + t; i < min(t0 + kTileWindows, Nw); i += kTileThreads) {
            if (mu) mu[i] = (double)x[i];
            sigma[i] = (ST)1;
        }
        return;
    }
    // samples past the stream enter windows that are not stored only
    const int have = (int)min((int64_t)S, N - t0);
    int i0 = 0;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {  // t0 is a multiple of 2048
        i0 = have / V * V;
        for (int i = V * t; i < i0; i += V * kTileThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(xs + tile_at<XT>(i))),
                         "l"(xt + i)
                         : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    for (int i = i0 + t; i < S; i += kTileThreads) xs[tile_at<XT>(i)] = i < have ? xt[i] : XT(0);
    __syncthreads();
    // sums of every chunk about its first sample
    double v[kTileR], c = 0.0;  // the thread's own chunk, about c
    unsigned again = 0;         // windows to be summed again
    for (int ch = t; ch < NC; ch += kTileThreads) {
        XT xv[kTileR];
        tile_load16(xs + (kTileR + V) * ch, xv);
        const double f = (double)xv[0];
        double a1 = 0.0, a2 = 0.0;
#pragma unroll
        for (int k = 0; k < kTileR; ++k) {
            const double d = (double)xv[k] - f;
            if (ch == t) v[k] = d;
            a1 += d;
            a2 = fma(d, d, a2);
        }
        if (ch == t) {
            c = f;
            if (!(a2 < (double)CDTW_INF)) {  // bad samples spoil the slide behind them
                again = kAll;
                for (int k = 0; k < kTileR; ++k)
                    if (!(fabs((double)xs[(kTileR + V) * t + k]) < (double)CDTW_INF))
                        again = kAll & (kAll << (k + 1));
            }
        }
        cur[ch] = make_double2(a1, a2);
        fs[ch] = xv[0];
    }
    // sums of the thread's first window about its first sample: its n chunks as
    // blocks of the powers of two in n, then the samples of a part of a chunk
    const int n = M / kTileR, rest = M % kTileR;
    double w1 = 0.0, w2 = 0.0;
    for (int b = 1, len = 0; b <= n; b *= 2) {  // cur: blocks of b chunks
        __syncthreads();
        if (n & b) {
            tile_add(w1, w2, cur[t + len], (double)fs[t + len] - c, 16.0 * b);
            len += b;
        }
        if (2 * b <= n) {
            // from here on chunks t + (n mod 2b) and further are looked at
            for (int ch = t + (n & (2 * b - 1)); ch < kTileThreads + n - 2 * b;
                 ch += kTileThreads) {
                double2 a = cur[ch];
                tile_add(a.x, a.y, cur[ch + b], (double)fs[ch + b] - (double)fs[ch], 16.0 * b);
                nxt[ch] = a;
            }
            double2* const swap = cur;
            cur = nxt;
            nxt = swap;
        }
    }
    for (int k = 0; k < rest; ++k) {
        const double d = (double)xs[(kTileR + V) * (t + n) + k] - c;
        w1 += d;
        w2 = fma(d, d, w2);
    }
    const double invM = 1.0 / (double)M;
    double most = w2;  // the second moment that the slide's sums may have held
    if (n == 0) {      // a sample may enter and leave again: all of them
        for (int k = M; k < M + kTileR; ++k) {
            const double d = (double)xs[tile_at<XT>(kTileR * t + k)] - c;
            most = fma(d, d, most);
        }
        again = most < (double)CDTW_INF ? 0u : kAll;
    }
    const double lost = most * invM * kLost;
    XT in[kTileR];
    tile_entering(xs, t, M, in);
    double om[kTileR];
    ST os[kTileR];
#pragma unroll
    for (int r = 0; r < kTileR; ++r) {
        const double m1 = w1 * invM;
        const double var = fma(-m1, m1, w2 * invM);
        om[r] = c + m1;
        os[r] = std_of<INV>(var, ST());
        again |= var < lost ? 1u << r : 0u;
        const double vin = (double)in[r] - c, d = vin - v[r];
        w1 += d;
        w2 = fma(d, vin + v[r], w2);
    }
    // the samples and sums make room for the sigmas, these for the means
    tile_out(reinterpret_cast<ST*>(tsm), os, sigma + t0, (int)min((int64_t)kTileWindows, Nw - t0));
    if (mu)
        tile_out(reinterpret_cast<double*>(tsm), om, mu + t0,
                 (int)min((int64_t)kTileWindows, Nw - t0));
    // the windows to be summed again, from the stream
    const int left = (int)min(Nw - t0 - kTileR * t, (int64_t)kTileR);  // the thread's windows
    again &= left <= 0 ? 0u : kAll >> (kTileR - left);
    if (!__syncthreads_or((int)again)) return;
    auto put = [&](int r, double m, double var) {
        if (mu) mu[t0 + kTileR * t + r] = m;
        sigma[t0 + kTileR * t + r] = std_of<INV>(var, ST());
    };
    if (n == 0) {
        for (; again; again &= again - 1) {
            const int r = __ffs(again) - 1;
            const double2 q = window_stats<1>(xt + kTileR * t + r, M, 0);
            put(r, q.x, q.y);
        }
        return;
    }
    // a lane's first one by the warp; the lane slides on from there
    while (const unsigned need = __ballot_sync(0xffffffffu, again != 0)) {
        const int src = __ffs(need) - 1;
        const int r0 = __ffs(__shfl_sync(0xffffffffu, again, src)) - 1;
        const double2 q = window_stats<32>(xt + kTileR * (t - lane + src) + r0, M, lane);
        if (lane == src) {
            again = 0;
            w1 = 0.0;
            w2 = q.y * (double)M;
            const XT* xw = xt + kTileR * t;
            for (int r = r0;; ++r) {
                const double m1 = w1 * invM, var = fma(-m1, m1, w2 * invM);
                put(r, q.x + m1, var);
                if (var < q.y * kLost) again |= 1u << r;
                if (r + 1 >= left) break;
                const double vin = (double)xw[r + M] - q.x, out = (double)xw[r] - q.x;
                w1 += vin - out;
                w2 = fma(vin - out, vin + out, w2);
            }
        }
    }
}

// One block prepares the query pack: FP64 two-pass z-normalisation (the
// reference does this on the host in FP32, GPU-dtw.cu:67 / stats.cuh:8-28),
// the +inf-padded shifted copies read by the cDTW kernels, and the +-W
// envelope (same values as Lemire's filter, bounds.cuh:13-64).  Shared
// memory: M doubles (zs) and M floats behind them.
__device__ __forceinline__ void prepare_query_body(const float* __restrict__ qraw, int M, int W,
                                                   const QueryPack& p, double* zs) {
    float* zf = reinterpret_cast<float*>(zs + M);  // the z-values rounded to float
    __shared__ double red[2][8];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    double s = 0.0;
    for (int i = t; i < M; i += blockDim.x) {
        const double v = (double)qraw[i];
        zs[i] = v;
        s += v;
    }
    __syncthreads();  // qraw may be p.zq (a host query staged there)
    for (int i = t; p.qraw && i < M; i += blockDim.x) p.qraw[i] = (float)zs[i];
    s = warp_sum(s);
    if (lane == 0) red[0][wid] = s;
    __syncthreads();
    double tot = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) tot += red[0][k];
    const double mean = tot / M;
    double v2 = 0.0;
    for (int i = t; i < M; i += blockDim.x) {
        const double d = zs[i] - mean;
        v2 = fma(d, d, v2);
    }
    v2 = warp_sum(v2);
    if (lane == 0) red[1][wid] = v2;
    __syncthreads();
    double vt = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) vt += red[1][k];
    const double var = vt / M;
    const double sd = var > 0.0 ? sqrt(var) : 1.0;
    __syncthreads();
    for (int i = t; i < M; i += blockDim.x) {
        const double z = (zs[i] - mean) / sd;
        zs[i] = z;
        zf[i] = (float)z;
        p.zq64[i] = z;
        p.zq[i] = (float)z;
    }
    __syncthreads();
    // padded shifted copies: copy m, index a -> qp[a+m], qp[b] = zq[b-W]
    for (int e = t; p.qpad && e < 4 * p.lq; e += blockDim.x) {
        const int m = e / p.lq, a = e - m * p.lq;
        const int i = a + m - W;
        p.qpad[e] = (i >= 0 && i < M) ? (float)zs[i] : CDTW_INF;
    }
    // reversed extended copies for the strip kernel
    if (p.qrev) {
        const int lo = qrev_lo(W), A = p.qrev_base, len = qrev_hi(M, W) - lo + 1;
        for (int e = t; e < 4 * p.lqr; e += blockDim.x) {
            const int m = e / p.lqr, b = e - m * p.lqr + m;  // qr index
            float v = CDTW_INF;
            if (b < len) {
                const int i = A - b;
                v = (i < 0) ? CDTW_INF : (i < M ? (float)zs[i] : (float)i * 1e18f);
            }
            p.qrev[e] = v;
        }
    }
    // envelope over [k-W, k+W] clipped to the query, from the float values
    // (rounding is monotone: the extrema of the rounded values are the
    // rounded extrema); four independent min / max chains per window
    for (int k = t; k < M; k += blockDim.x) {
        const int a0 = max(0, k - W), a1 = min(M - 1, k + W);
        float lo[4], hi[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) lo[u] = hi[u] = zf[k];
        int i = a0;
        for (; i + 3 <= a1; i += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                lo[u] = fminf(lo[u], zf[i + u]);
                hi[u] = fmaxf(hi[u], zf[i + u]);
            }
        }
        for (; i <= a1; ++i) {
            lo[0] = fminf(lo[0], zf[i]);
            hi[0] = fmaxf(hi[0], zf[i]);
        }
        p.env[k] = make_float2(fminf(fminf(lo[0], lo[1]), fminf(lo[2], lo[3])),
                               fmaxf(fmaxf(hi[0], hi[1]), fmaxf(hi[2], hi[3])));
    }
}

__global__ void __launch_bounds__(256)
prepare_query_kernel(const float* __restrict__ qraw, int M, int W, QueryPack p) {
    extern __shared__ double zs[];  // M doubles, M floats
    prepare_query_body(qraw, M, W, p, zs);
}

__global__ void __launch_bounds__(256)
prepare_queries_kernel(const float* __restrict__ raw, const int64_t* __restrict__ offs,
                       const QueryPack* __restrict__ packs) {
    extern __shared__ double zs[];
    const QueryPack p = packs[blockIdx.x];
    prepare_query_body(raw + offs[blockIdx.x], p.M, p.W, p, zs);
}

}  // namespace

template <bool INV, class XT, class ST>
static int launch_stats(cdtw_handle h, const XT* x, int64_t N, int M, double* mu, ST* sigma) {
    const int64_t Nw = N - M + 1;
    if (M > kTileMaxM) {
        const int64_t blocks = div_up(div_up(Nw, kStatsWarpWindows), kStatsBlock / 32);
        avg_std_long_kernel<XT, ST, INV><<<(unsigned)blocks, kStatsBlock, 0, h->stream>>>(x, N, M, mu,
                                                                                    sigma);
        CDTW_LAUNCH(h, "avg_std_long_kernel");
        return CDTW_OK;
    }
    const size_t smem = tile_smem<XT, ST>(M);
    CDTW_TRY(allow_smem(h, (const void*)avg_std_kernel<XT, ST, INV>, smem));
    avg_std_kernel<XT, ST, INV>
        <<<(unsigned)div_up(Nw, kTileWindows), kTileThreads, smem, h->stream>>>(x, N, M, mu, sigma);
    CDTW_LAUNCH(h, "avg_std_kernel");
    return CDTW_OK;
}

int launch_avg_std(cdtw_handle h, const float* x, int64_t N, int M, double* mu, float* sigma) {
    return launch_stats<false>(h, x, N, M, mu, sigma);
}

// FP64 sigma (LDTW).
int launch_avg_std64(cdtw_handle h, const float* x, int64_t N, int M, double* mu, double* sigma) {
    return launch_stats<false>(h, x, N, M, mu, sigma);
}
// 1 / sigma alone (ED).
int launch_rstd64(cdtw_handle h, const double* x, int64_t N, int M, double* rs) {
    return launch_stats<true>(h, x, N, M, (double*)nullptr, rs);
}

int launch_prepare_queries(cdtw_handle h, const float* raw, const int64_t* offs,
                           const QueryPack* packs, int nq, int max_m) {
    const size_t smem = (size_t)max_m * (sizeof(double) + sizeof(float));
    CDTW_TRY(allow_smem(h, (const void*)prepare_queries_kernel, smem));
    prepare_queries_kernel<<<nq, 256, smem, h->stream>>>(raw, offs, packs);
    CDTW_LAUNCH(h, "prepare_queries_kernel");
    return CDTW_OK;
}

int launch_prepare_query(cdtw_handle h, const float* d_query_raw, int M, int W) {
    const size_t smem = (size_t)M * (sizeof(double) + sizeof(float));
    CDTW_TRY(allow_smem(h, (const void*)prepare_query_kernel, smem));
    prepare_query_kernel<<<1, 256, smem, h->stream>>>(d_query_raw, M, W, h->q);
    CDTW_LAUNCH(h, "prepare_query_kernel");
    return CDTW_OK;
}

}  // namespace cdtw

// Greedy locally-optimal warping path inside the Sakoe-Chiba band (LDTW),
// z-normalised, for every window: the GPU-LDTW path.
//
// Reference: ztsh2_ldtw (include/ldtw.cuh:294-391) and its serial twin
// z_serial_ldtw (ldtw.cuh:74-127): one path of at most 2M-2 steps per window;
// at (i, j) take the diagonal if it is strictly cheaper than both the cell
// below and the cell to the right, else "down" if the diagonal is not cheaper
// than it and it is cheaper than "right", else "right"; moves outside the
// matrix or the band cost INFTY = 1e10 (ldtw.cuh:8).  One thread per window
// here too (a path is inherently sequential), in FP64 so the branch decisions
// match the FP64 oracle; the four values a step reads (two query, two window
// samples) are carried in registers and only the entering ones are loaded.
#include "common.cuh"

#include <algorithm>

namespace cdtw {

namespace {

template <bool EU>
__device__ __forceinline__ double lcost(double d) { return EU ? d * d : fabs(d); }

template <bool EU>
__global__ void __launch_bounds__(128)
ldtw_kernel(const float* __restrict__ x, const double* __restrict__ mu,
            const double* __restrict__ sigma, const double* __restrict__ zq, int M, int W,
            int64_t Nw, double* __restrict__ out) {
    const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= Nw) return;
    const double INFTY = 1e10;
    const double m = mu[w], s = sigma[w];
    const float* __restrict__ xw = x + w;
    int i = 0, j = 0;
    double q0 = zq[0], q1 = (M > 1) ? zq[1] : 0.0;
    double s0 = ((double)xw[0] - m) / s, s1 = (M > 1) ? ((double)xw[1] - m) / s : 0.0;
    double d = lcost<EU>(q0 - s0);
    // every step advances i or j, so 2M-2 steps reach (M-1, M-1); the cap only
    // guards against non-finite input
    for (int it = 0; it < 2 * M && (i + 1 != M || j + 1 != M); ++it) {
        double diag = INFTY, rght = INFTY, down = INFTY;
        if (i + 1 < M && j + 1 < M) diag = lcost<EU>(q1 - s1);
        if (i + 1 < M && abs(i - j + 1) <= W) down = lcost<EU>(q1 - s0);
        if (j + 1 < M && abs(j - i + 1) <= W) rght = lcost<EU>(q0 - s1);
        const bool diagSdown = diag < down, diagSrght = diag < rght, downSrght = down < rght;
        bool mi, mj;
        if (diagSdown && diagSrght) {
            d += diag;
            mi = mj = true;
        } else if (!diagSdown && downSrght) {
            d += down;
            mi = true;
            mj = false;
        } else {
            d += rght;
            mi = false;
            mj = true;
        }
        if (mi) {
            ++i;
            q0 = q1;
            q1 = (i + 1 < M) ? zq[i + 1] : 0.0;
        }
        if (mj) {
            ++j;
            s0 = s1;
            s1 = (j + 1 < M) ? ((double)xw[j + 1] - m) / s : 0.0;
        }
    }
    out[w] = d;
}

// The reference's own FP32 arithmetic, for drop-in index parity with its
// GPU-LDTW.  The query is z-normalised as the reference driver does on the
// host (znormalize, stats.cuh:8-28: float sums in order, population sigma,
// (x - avg) / std), without fused multiply-adds.  The two ordered sums are a
// chain on one thread; their samples come from shared memory and the
// quotients are taken by the whole block (one thread for all of it, from
// global memory: 10.9 us at M = 128).
__global__ void __launch_bounds__(128)
ldtw_ref_query_kernel(const float* __restrict__ qraw, int M, float* __restrict__ zq) {
    extern __shared__ float qsm[];  // M floats
    __shared__ float stat[2];
    for (int i = threadIdx.x; i < M; i += blockDim.x) qsm[i] = qraw[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        float avg = 0.f, sd = 0.f;
#pragma unroll 8
        for (int i = 0; i < M; ++i) {
            avg = __fadd_rn(avg, qsm[i]);
            sd = __fadd_rn(sd, __fmul_rn(qsm[i], qsm[i]));
        }
        avg = __fdiv_rn(avg, (float)M);
        stat[0] = avg;
        stat[1] = __fsqrt_rn(__fsub_rn(__fdiv_rn(sd, (float)M), __fmul_rn(avg, avg)));
    }
    __syncthreads();
    const float avg = stat[0], sd = stat[1];
    for (int i = threadIdx.x; i < M; i += blockDim.x)
        zq[i] = __fdiv_rn(__fsub_rn(qsm[i], avg), sd);
}

template <bool EU>
__device__ __forceinline__ float lcost_ref(float d) {
    return EU ? __fmul_rn(d, d) : fabsf(d);
}

// Quotients a / sd of one window, all by the same sd, correctly rounded (the
// value of __fdiv_rn).  With y = RN(1 / sd) and q within one ulp of a / sd,
// the residual r = a - q sd is exact (fused) and RN(q + r y) is RN(a / sd):
// P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. R&D 34 (1990).  RN(a y) is within 1.5 ulp, so
// one such step brings it within one and the second gives the quotient (zero
// stays zero).  That holds while nothing under- or overflows, which `exact`
// grants for every sample of the window: sd in [2^-60, 2^40] and |avg| in
// [2^-60, 2^100], so a nonzero a = x - avg is at least 2^-84, q at least 2^-125
// and a residual a multiple of 2^-132.  The variance is the rounded difference
// of a 24-bit mean of squares and a 48-bit square, so where it is positive it is
// at least 2^-48 of that mean, sd at least 2^-25 max|x| / sqrt(M) and |q| below
// 2^33 (sd = 1 otherwise: |q| below 2^108).  Windows outside divide.
struct RefNorm {
    float avg, sd, y;
    bool exact;
};
__device__ __forceinline__ RefNorm make_ref_norm(float avg, float sd) {
    RefNorm n;
    n.avg = avg;
    n.sd = sd;
    n.y = __frcp_rn(sd);
    const float m = fabsf(avg);
    n.exact = sd >= 0x1p-60f && sd <= 0x1p40f && m >= 0x1p-60f && m <= 0x1p100f;
    return n;
}
template <bool EXACT>
__device__ __forceinline__ float ref_z(const RefNorm& n, float v) {
    const float a = __fsub_rn(v, n.avg);
    if (!EXACT) return __fdiv_rn(a, n.sd);
    const float q = __fmul_rn(a, n.y);
    const float p = __fmaf_rn(__fmaf_rn(-q, n.sd, a), n.y, q);
    return __fmaf_rn(__fmaf_rn(-p, n.sd, a), n.y, p);
}

// The choice of one step and its effects: costs diag / down / rght (INFTY
// where barred), the running cost d, byte addresses pq / px of q_i and x_j.
// The tests of ldtw.cuh:368-383 as three compares that chain their predicates
// (diag < down; then diag < rght, or down < rght); the cost is added by one of
// four predicated adds, which leaves the half-rate compare / select pipe to
// the compares.  Sets right when j advances.
__device__ __forceinline__ void ref_step(float diag, float down, float rght, float& d,
                                         unsigned& pq, unsigned& px, float& s0, float s1) {
    asm("{\n\t"
        ".reg .pred a, na, md, r1, dd, r2;\n\t"
        "setp.lt.f32 a, %4, %5;\n\t"
        "not.pred na, a;\n\t"
        "setp.lt.and.f32 md|r1, %4, %6, a;\n\t"
        "setp.lt.and.f32 dd|r2, %5, %6, na;\n\t"
        "@md add.rn.f32 %0, %0, %4;\n\t"
        "@dd add.rn.f32 %0, %0, %5;\n\t"
        "@r1 add.rn.f32 %0, %0, %6;\n\t"
        "@r2 add.rn.f32 %0, %0, %6;\n\t"
        "@md add.u32 %1, %1, 8;\n\t"
        "@dd add.u32 %1, %1, 8;\n\t"
        "@!dd add.u32 %2, %2, 4;\n\t"
        "@!dd mov.f32 %3, %7;\n\t"
        "}"
        : "+f"(d), "+r"(pq), "+r"(px), "+f"(s0)
        : "f"(diag), "f"(down), "f"(rght), "f"(s1));
}

// The walk of one window: xw its samples, qs the query as pairs
// (q_i, q_(i+1)), both with entries behind the last that no cost uses.  Bound
// by the half-rate pipe of compares, selects and integer adds, so a step
// holds as few of them as it can: the query pair is one shared load, the
// entering sample is loaded and normalised on the full-rate pipe, i and j are
// the two addresses (c = i - j + W from their difference; |i - j + 1| <= W is
// (unsigned)(c + 1) <= 2W), and as many steps as every lane of the warp
// surely has room for run without an end test.  act: the warp's lanes that
// call.
template <bool EU, bool ZN, bool EXACT>
__device__ __forceinline__ float ldtw_ref_walk(const float* xw, const float2* qs, int M, int W,
                                               const RefNorm& nm, unsigned act) {
    const float INFTY = 1e10f;
    auto sp = [&](float v) { return ZN ? ref_z<EXACT>(nm, v) : v; };
    const unsigned q00 = (unsigned)__cvta_generic_to_shared(qs);
    const unsigned x00 = (unsigned)__cvta_generic_to_shared(xw);
    const unsigned band = 2 * W;
    unsigned pq = q00, px = x00;
    float s0 = sp(xw[0]);
    float d = lcost_ref<EU>(__fsub_rn(qs[0].x, s0));
    int left = 2 * M - 2;  // relaxations left
    auto step = [&]() {
        float q0, q1, xv;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(q0), "=f"(q1) : "r"(pq));
        asm volatile("ld.shared.f32 %0, [%1+4];" : "=f"(xv) : "r"(px));
        const float s1 = sp(xv);
        const int c = (int)((pq - q00) >> 1) - (int)(px - x00) + 4 * W;  // 4 (i - j + W)
        const float diag = lcost_ref<EU>(__fsub_rn(q1, s1));
        const float dn = lcost_ref<EU>(__fsub_rn(q1, s0));
        const float rt = lcost_ref<EU>(__fsub_rn(q0, s1));
        const float down = (unsigned)(c + 4) <= 4 * band ? dn : INFTY;
        const float rght = (unsigned)(c - 4) <= 4 * band ? rt : INFTY;
        ref_step(diag, down, rght, d, pq, px, s0, s1);
    };
    auto room = [&]() {  // steps until i or j may be at its end
        return min(M - 1 - (int)((pq - q00) >> 3), M - 1 - (int)((px - x00) >> 2));
    };
    for (;;) {
        const int n = __reduce_min_sync(act, room());
        if (n < 4) break;
#pragma unroll 4
        for (int k = 0; k < n; ++k) step();
        left -= n;
    }
    for (int n = room(); n > 0; n = room()) {
        step();
        --left;
    }
    const int i0 = (int)((pq - q00) >> 3), j0 = (int)((px - x00) >> 2);
    float q0 = qs[i0].x, q1 = qs[i0].y, s1 = sp(xw[j0 + 1]);
    // one index is at its end: a move out of the matrix costs INFTY and, where
    // a cost above it makes that the choice, stays put
    int i = i0, j = j0;
    for (; left > 0 && (i + 1 < M || j + 1 < M); --left) {
        const bool vi = i + 1 < M, vj = j + 1 < M;
        const bool cd = abs(i - j + 1) <= W, cr = abs(j - i + 1) <= W;
        const float down = (vi && cd) ? lcost_ref<EU>(__fsub_rn(q1, s0)) : INFTY;
        const float rght = (vj && cr) ? lcost_ref<EU>(__fsub_rn(q0, s1)) : INFTY;
        // the diagonal costs INFTY here: it is never strictly the cheapest of
        // all, and "down" needs it not cheaper than down
        const bool mi = !(INFTY < down) && down < rght;
        const bool md = INFTY < down && INFTY < rght;
        d = __fadd_rn(d, md ? INFTY : (mi ? down : rght));
        if ((mi || md) && vi) {
            ++i;
            q0 = q1;
            q1 = qs[i].y;
        }
        if ((!mi || md) && vj) {
            ++j;
            s0 = s1;
            s1 = sp(xw[j + 1]);
        }
    }
    return d;
}

// One window per thread, the steps of ztsh2_ldtw (ZN) / tsh2_ldtw
// (ldtw.cuh:294-391 / :199-291) in FP32: at most 2M-2 relaxations, moves
// out of the matrix or the band cost INFTY = 1e10, the tie rule of
// ldtw.cuh:368-383, and nothing added once (M-1, M-1) is reached, where the
// walk ends (costs above INFTY can keep it from there: 2M-2 steps then).  ZN:
// the window statistics of avg_std<double> (stats.cuh:30-52): the window mean
// of x and of x^2 in FP64 rounded to float, variance E[x^2] - mu^2 in float
// (the fused multiply-add nvcc makes of stats.cuh:49), sigma = 1 where it is
// not positive; samples normalised as (s - avg) / std in float.  (The
// reference takes the window sums as differences of FP64 prefix sums; here
// they are summed directly, equal to a few FP64 ulps.)
//
// Bound by issue.  The block's samples (kRefWin + M) and the query sit in
// shared memory, since neighbouring lanes drift apart along their paths; a
// step takes one quotient by exact residuals where taking both window samples
// anew took two divisions.  The sums of the first kRefWin / 4 threads cover
// four windows each: a sample is converted to FP64 once for four windows (the
// conversions were the larger part of the statistics).  2^20 windows,
// M = 128, W = 12: 750 us with a division per sample and step and always 2M-2
// steps, 427 us with selects and an end test a step; now 335 us.
constexpr int kRefWin = 256;  // windows (and threads) per block

template <bool EU, bool ZN>
__global__ void __launch_bounds__(kRefWin)
ldtw_ref_kernel(const float* __restrict__ x, const float* __restrict__ zq, int M, int W,
                int64_t Nw, float* __restrict__ out) {
    extern __shared__ float rsm[];
    float2* qs = (float2*)rsm;  // M: (q_i, q_(i+1)), the last value repeated
    float* xs = rsm + 2 * M;    // kRefWin + M + 5: the block's samples (clamped at the end)
    __shared__ float2 st[kRefWin];
    const int t = threadIdx.x;
    const int64_t b0 = (int64_t)blockIdx.x * kRefWin;
    const int64_t xlast = Nw + M - 2;  // the stream's last sample
    for (int i = t; i < M; i += kRefWin) qs[i] = make_float2(zq[i], zq[min(i + 1, M - 1)]);
    for (int i = t; i < kRefWin + M + 5; i += kRefWin) xs[i] = x[min(b0 + i, xlast)];
    __syncthreads();
    if (ZN) {
        if (t < kRefWin / 4) {
            // windows 4t .. 4t + 3 of the block, each sum in sample order
            const float* xw = xs + 4 * t;
            double s1[4] = {0.0, 0.0, 0.0, 0.0}, s2[4] = {0.0, 0.0, 0.0, 0.0};
            double v[4];
#pragma unroll
            for (int r = 0; r < 3; ++r) v[r] = (double)xw[r];
            for (int k0 = 0; k0 < M; k0 += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (k0 + u < M) {
                        v[(u + 3) & 3] = (double)xw[k0 + u + 3];
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const double a = v[(u + r) & 3];
                            s1[r] += a;
                            s2[r] = fma(a, a, s2[r]);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float avg = (float)(s1[r] / M);
                const float ex2 = (float)(s2[r] / M);
                const float var = __fmaf_rn(-avg, avg, ex2);
                st[4 * t + r] = make_float2(avg, var > 0.f ? __fsqrt_rn(var) : 1.f);
            }
        }
        __syncthreads();
    }
    const int64_t w = b0 + t;
    const unsigned act = __ballot_sync(0xffffffffu, w < Nw);
    if (w >= Nw) return;
    const RefNorm nm = ZN ? make_ref_norm(st[t].x, st[t].y) : RefNorm();
    if (ZN && !__all_sync(act, nm.exact))
        out[w] = ldtw_ref_walk<EU, ZN, false>(xs + t, qs, M, W, nm, act);
    else
        out[w] = ldtw_ref_walk<EU, ZN, true>(xs + t, qs, M, W, nm, act);
}

// Packed (float bits, index) minimum; values are >= 0, so their bits order as
// unsigned ints, and ties keep the lowest index (determine_min's first strict
// minimum, ldtw.cuh:177-192).
__global__ void argmin_f32_kernel(const float* __restrict__ v, int64_t n,
                                  unsigned long long* __restrict__ key) {
    unsigned long long best = ~0ull;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float a = v[i];
        if (a == a) best = min(best, pack_key(a, (uint32_t)i));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0 && best != ~0ull) atomicMin(key, best);
}

}  // namespace

int launch_ldtw_ref(cdtw_handle h, const float* x, int64_t N, bool euclid, bool znorm,
                    float* qwork, float* out) {
    const QueryPack& q = h->q;
    if (!q.qraw) return set_error(h, CDTW_EINVAL, "query pack without the raw query");
    const int64_t Nw = N - q.M + 1;
    const float* zq = q.qraw;
    if (znorm) {
        ldtw_ref_query_kernel<<<1, 128, sizeof(float) * q.M, h->stream>>>(q.qraw, q.M, qwork);
        CDTW_LAUNCH(h, "ldtw_ref_query_kernel");
        zq = qwork;
    }
    const unsigned blocks = (unsigned)div_up(Nw, kRefWin);
    auto k = euclid ? (znorm ? ldtw_ref_kernel<true, true> : ldtw_ref_kernel<true, false>)
                    : (znorm ? ldtw_ref_kernel<false, true> : ldtw_ref_kernel<false, false>);
    // the query pairs and the block's samples
    const size_t smem = sizeof(float) * (size_t)(3 * q.M + kRefWin + 5);
    CDTW_TRY(allow_smem(h, (const void*)k, smem));
    k<<<blocks, kRefWin, smem, h->stream>>>(x, zq, q.M, q.W, Nw, out);
    CDTW_LAUNCH(h, "ldtw_ref_kernel");
    return CDTW_OK;
}

int launch_argmin_f32(cdtw_handle h, const float* v, int64_t n, unsigned long long* key) {
    const unsigned blocks = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>(div_up(n, 256), (int64_t)h->sm_count * 8));
    argmin_f32_kernel<<<blocks, 256, 0, h->stream>>>(v, n, key);
    CDTW_LAUNCH(h, "argmin_f32_kernel");
    return CDTW_OK;
}

int launch_ldtw(cdtw_handle h, const float* x, int64_t N, const double* mu, const double* sigma,
                bool euclid, double* out) {
    const QueryPack& q = h->q;
    const int64_t Nw = N - q.M + 1;
    const unsigned blocks = (unsigned)div_up(Nw, 128);
    if (euclid)
        ldtw_kernel<true><<<blocks, 128, 0, h->stream>>>(x, mu, sigma, q.zq64, q.M, q.W, Nw, out);
    else
        ldtw_kernel<false><<<blocks, 128, 0, h->stream>>>(x, mu, sigma, q.zq64, q.M, q.W, Nw, out);
    CDTW_LAUNCH(h, "ldtw_kernel");
    return CDTW_OK;
}

}  // namespace cdtw

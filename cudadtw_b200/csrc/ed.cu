// z-normalised Euclidean distance of a query to every window of a float64
// series, and its argmin: the GPU-ED path.
//
// Reference: calculate_ed (include/ed.cuh:71-153) zero-pads query and series
// to a multiple of 1e4, runs three cuFFT transforms for the correlation,
// scales it by -2/(sigma*NN) and argsorts all windows with a radix sort,
// printing sqrt(2M + min).  Since sum_k zq_k = 0, the same value is
//   d^2(w) = 2M - 2 * (sum_k zq_k * x_{w+k}) / sigma_w,
// computed here directly in FP64: each thread owns 8 consecutive windows and
// slides them over the query with the window samples in registers (one new
// sample load per query step for 8 FMAs), the query and the series tile staged
// in shared memory (padded one double per eight so the eight-apart thread
// reads do not collide in banks), with 1 / sigma from the statistics kernel,
// then an exact FP64 argmin.  No FFT, no sort.
#include "common.cuh"

#include <algorithm>

namespace cdtw {

namespace {

constexpr int kEdThreads = 128;
constexpr int kEdR = 8;                            // windows per thread
constexpr int kEdTile = kEdThreads * kEdR;         // windows per block
constexpr int kEdK = 256;                          // query positions per chunk
constexpr int kEdSpan = kEdTile + kEdK + kEdR;     // samples staged per chunk
constexpr int kEdXs = kEdSpan + (kEdSpan >> 3) + 1;  // with one pad per eight
constexpr int kEdStage = kEdXs + kEdK;               // doubles of a stage: samples, query chunk

__device__ __forceinline__ int pad8(int i) { return i + (i >> 3); }

// dst = *src, or 0 without reading where !in (8 bytes, asynchronously).
__device__ __forceinline__ void copy8(double* dst, const double* src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src),
                 "r"(in ? 8 : 0)
                 : "memory");
}

// rs: 1 / sigma per window.  Bound by the FP64 pipe (2^21 windows, M = 256:
// 5.4e8 multiply-adds, 29 us at 64 a cycle and SM).  Persistent blocks go
// through (tile, query chunk) stages with the next stage's copies in flight
// under the current one's arithmetic: with a block per tile every wave of
// blocks loaded together, computed together and divided by sigma together (60
// us; with the statistics pass 81, now 57 and 71).
__global__ void __launch_bounds__(kEdThreads)
ed_kernel(const double* __restrict__ x, int64_t N, const double* __restrict__ zq, int M,
          int64_t Nw, const double* __restrict__ rs, double* __restrict__ out) {
    extern __shared__ double esm[];  // two stages
    const int t = threadIdx.x;
    const int64_t tiles = (Nw + kEdTile - 1) / kEdTile;
    const int chunks = (M + kEdK - 1) / kEdK;
    auto stage_in = [&](int64_t tile, int chunk, double* xs) {
        const int64_t g0 = tile * kEdTile + (int64_t)chunk * kEdK;
        for (int i = t; i < kEdSpan; i += kEdThreads) {
            const bool in = g0 + i < N;
            copy8(xs + pad8(i), x + (in ? g0 + i : 0), in);
        }
        double* qs = xs + kEdXs;
        for (int i = t; i < kEdK; i += kEdThreads) {
            const int k = chunk * kEdK + i;
            copy8(qs + i, zq + (k < M ? k : 0), k < M);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int64_t tile = blockIdx.x;
    if (tile >= tiles) return;
    stage_in(tile, 0, esm);
    int buf = 0;
    for (; tile < tiles; tile += gridDim.x) {
        double acc[kEdR], rsv[kEdR];
        const int64_t w0 = tile * kEdTile + (int64_t)t * kEdR;
#pragma unroll
        for (int r = 0; r < kEdR; ++r) acc[r] = 0.0;
        for (int chunk = 0; chunk < chunks; ++chunk) {
            const bool last = chunk + 1 == chunks;
            const int64_t next = last ? tile + gridDim.x : tile;
            __syncthreads();  // the other buffer is read
            if (next < tiles) {
                stage_in(next, last ? 0 : chunk + 1, esm + (buf ^ 1) * kEdStage);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            if (last) {
#pragma unroll
                for (int r = 0; r < kEdR; ++r) rsv[r] = rs[min(w0 + r, Nw - 1)];
            }
            __syncthreads();
            const double* xs = esm + buf * kEdStage;
            const double* qs = xs + kEdXs;
            const int kn = min(kEdK, M - chunk * kEdK);
            const double* xb = xs + (kEdR + 1) * t;  // pad8(8 t)
            double xr[kEdR];
#pragma unroll
            for (int r = 0; r < kEdR; ++r) xr[r] = xb[r];
            for (int k = 0; k < kn; k += kEdR) {
                xb += kEdR + 1;
#pragma unroll
                for (int u = 0; u < kEdR; ++u) {
                    const double q = qs[k + u];  // zero beyond kn
#pragma unroll
                    for (int r = 0; r < kEdR; ++r) acc[r] = fma(q, xr[(r + u) % kEdR], acc[r]);
                    xr[u] = xb[u];  // sample 8t + k + 8 + u replaces 8t + k + u
                }
            }
            buf ^= 1;
        }
#pragma unroll
        for (int r = 0; r < kEdR; ++r)
            if (w0 + r < Nw) out[w0 + r] = fma(-2.0 * acc[r], rsv[r], 2.0 * M);
    }
}

__device__ __forceinline__ bool better(double av, long long ai, double bv, long long bi) {
    return av < bv || (av == bv && ai < bi);
}

__global__ void __launch_bounds__(256)
argmin64_kernel(const double* __restrict__ d, int64_t n, ArgMin64* __restrict__ out) {
    __shared__ ArgMin64 red[8];
    double bv = CDTW_INF;
    long long bi = 0x7fffffffffffffffll;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double v = d[i];
        if (better(v, i, bv, bi)) {
            bv = v;
            bi = i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const long long oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (better(ov, oi, bv, bi)) {
            bv = ov;
            bi = oi;
        }
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ArgMin64{bv, bi};
    __syncthreads();
    if (threadIdx.x == 0) {
        ArgMin64 b = red[0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k)
            if (better(red[k].v, red[k].i, b.v, b.i)) b = red[k];
        out[blockIdx.x] = b;
    }
}

__global__ void argmin64_final_kernel(const ArgMin64* __restrict__ p, int n,
                                      ArgMin64* __restrict__ res) {
    __shared__ ArgMin64 red[32];
    ArgMin64 b{CDTW_INF, 0x7fffffffffffffffll};
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (better(p[i].v, p[i].i, b.v, b.i)) b = p[i];
    red[threadIdx.x] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < (int)blockDim.x; ++k)
            if (better(red[k].v, red[k].i, b.v, b.i)) b = red[k];
        *res = b;
    }
}

constexpr int kArgminBlocks = 1024;

// z-normalise a float64 query in FP64 (GPU-ed.cu:88 znormalize on the host).
__global__ void __launch_bounds__(256) znorm64_kernel(const double* __restrict__ q, int M,
                                                      double* __restrict__ zq) {
    __shared__ double red[8];
    __shared__ double stat[2];
    const int t = threadIdx.x;
    double s = 0.0;
    for (int i = t; i < M; i += blockDim.x) s += q[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((t & 31) == 0) red[t >> 5] = s;
    __syncthreads();
    if (t == 0) {
        double a = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) a += red[k];
        stat[0] = a / M;
    }
    __syncthreads();
    const double mean = stat[0];
    double v = 0.0;
    for (int i = t; i < M; i += blockDim.x) v = fma(q[i] - mean, q[i] - mean, v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((t & 31) == 0) red[t >> 5] = v;
    __syncthreads();
    if (t == 0) {
        double a = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) a += red[k];
        const double var = a / M;
        stat[1] = var > 0.0 ? sqrt(var) : 1.0;
    }
    __syncthreads();
    for (int i = t; i < M; i += blockDim.x) zq[i] = (q[i] - mean) / stat[1];
}

}  // namespace

size_t argmin64_partials(int64_t n) { return (size_t)std::min<int64_t>(kArgminBlocks, div_up(n, 256)); }

int launch_argmin64(cdtw_handle h, const double* d, int64_t n, ArgMin64* partial,
                    ArgMin64* res) {
    const int blocks = (int)argmin64_partials(n);
    argmin64_kernel<<<blocks, 256, 0, h->stream>>>(d, n, partial);
    CDTW_LAUNCH(h, "argmin64_kernel");
    argmin64_final_kernel<<<1, 32, 0, h->stream>>>(partial, blocks, res);
    CDTW_LAUNCH(h, "argmin64_final_kernel");
    return CDTW_OK;
}

int launch_znorm64(cdtw_handle h, const double* q, int M, double* zq) {
    znorm64_kernel<<<1, 256, 0, h->stream>>>(q, M, zq);
    CDTW_LAUNCH(h, "znorm64_kernel");
    return CDTW_OK;
}

int launch_ed(cdtw_handle h, const double* x, int64_t N, const double* zq, int M,
              const double* rs, double* out) {
    const int64_t Nw = N - M + 1;
    const size_t smem = 2 * kEdStage * sizeof(double);
    CDTW_TRY(allow_smem(h, (const void*)ed_kernel, smem));
    int per_sm = 0;
    CDTW_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)ed_kernel,
                                                               kEdThreads, smem));
    const unsigned blocks = (unsigned)std::min<int64_t>(
        div_up(Nw, kEdTile), (int64_t)std::max(per_sm, 1) * h->sm_count);
    ed_kernel<<<blocks, kEdThreads, smem, h->stream>>>(x, N, zq, M, Nw, rs, out);
    CDTW_LAUNCH(h, "ed_kernel");
    return CDTW_OK;
}

}  // namespace cdtw

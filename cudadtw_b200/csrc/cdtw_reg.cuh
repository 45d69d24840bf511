// Banded DTW with the whole band of one window in registers ("register band").
//
// Reference: sparse_block_cdtw / dense_block_cdtw (include/cdtw.cuh:164-363),
// which spread one window over W+2 threads and step the anti-diagonals through
// shared memory with a __syncthreads per step.  Windows are independent and
// there are millions of them, so here one thread owns one window and keeps
// the 2W+1 band cells of the current row in registers; the 32 lanes of a warp
// run 32 neighbouring windows in lockstep, so all lanes read the same query
// values (a shared-memory broadcast) and consecutive stream samples (one
// coalesced 128-byte load per row).
//
// Orientation: rows are window (data) positions j = 0..M-1, columns are query
// positions i, band coordinate k = i - j + W in [0, 2W].  The cell update
//   D[j][k] = cost(z_j, q_{j-W+k}) + min(D[j-1][k], D[j-1][k+1], D[j][k-1])
// is one FADD, one three-input FMNMX and one FFMA.  Query positions outside
// [0, M) are padded with +inf, which makes out-of-matrix cells +inf without
// any per-cell test.  The result D[M-1][W] equals the reference's
// penalty[...][M] (cdtw.cuh:83).
//
// What bounds a cell is the register file: about two operands a cycle and
// scheduler (measured: FFMA with two distinct registers 1.07 cycles a warp,
// with three 1.60; FADD + two-input FMNMX + FFMA 3.26, with a three-input
// FMNMX 4.13), and 4.2 is what a row at a time ran at.  So four rows go
// together, each a cell behind the one above (reg_rows4): rows j .. j+3 then
// stand on the same query value q_{j-W+s} at step s, a row's diagonal and upper
// inputs are the two newest values of the row above, still in registers, and
// the differences z - q of two neighbouring steps come from one packed
// subtraction (z twice, the query pair as loaded).  A group of four rows loads
// the query once, from one copy of it.  All windows, M = 128, in cycles a warp
// and computed cell (2^22 windows: us), row at a time -> now: W = 12 4.19 ->
// 3.87 (1395), W = 25 4.19 -> 3.77 (2773), W = 55 3.69 now.  Scalar
// subtractions 4.2 to 4.4; rows in pairs 3.95 to 3.99, in eights 3.84 to 3.89;
// the pair over rows instead of steps 3.96 to 4.08; subtraction and
// multiply-add packed over two windows 4.7 to 5.1 (the three minimum operands
// then share a register bank).
#pragma once

#include "common.cuh"

#include <algorithm>

namespace cdtw {

namespace {

constexpr int kRegBlock = 128;
constexpr int kMaxRegW = 106;  // the widest band that 255 registers hold without spills

// Rows j .. j+3 of NW windows: p holds row j-1 (p[v][B] = +inf) and becomes
// row j+3; z[v][r] is window v's sample of row j + r, qr the padded query from
// element j (16-byte aligned; reads up to 2W + 7 further).  Step s takes row r
// to its cell s - r, whose query value is element s for every row.  CAP: res[v]
// takes D[j + last][W] for last in 0..3.
template <int W, bool EU, int NW, bool CAP>
__device__ __forceinline__ void reg_rows4(float (&p)[NW][2 * W + 2], const float (&z)[NW][4],
                                          const float4* qr, int last, float (&res)[NW]) {
    constexpr int B = 2 * W + 1;
    constexpr int kSteps = B + 3;
    float l[NW][4], d1[NW][4];  // rows' newest cells and the ones before
#pragma unroll
    for (int v = 0; v < NW; ++v) {
#pragma unroll
        for (int r = 0; r < 4; ++r) l[v][r] = d1[v][r] = CDTW_INF;
    }
#pragma unroll
    for (int s4 = 0; s4 < (kSteps + 3) / 4; ++s4) {
        const float4 q4 = qr[s4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const unsigned long long q2 = h ? pack2(q4.z, q4.w) : pack2(q4.x, q4.y);
            float df[NW][4][2];
#pragma unroll
            for (int v = 0; v < NW; ++v) {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    sub2(pack2(z[v][r], z[v][r]), q2, df[v][r][0], df[v][r][1]);
            }
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const int s = 4 * s4 + 2 * h + g;
#pragma unroll
                for (int v = 0; v < NW; ++v) {
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int k = s - r;  // row j + r's cell
                        if (k >= 0 && k < B) {
                            const float diag = r == 0 ? p[v][k < B ? k : 0] : d1[v][r > 0 ? r - 1 : 0];
                            const float up = r == 0 ? p[v][k < B ? k + 1 : B]
                                                    : (k + 1 < B ? l[v][r > 0 ? r - 1 : 0] : CDTW_INF);
                            const float c = cell<EU>(df[v][r][g], min3f(diag, l[v][r], up));
                            d1[v][r] = l[v][r];
                            l[v][r] = c;
                            if (r == 3) p[v][k] = c;
                            if (CAP && k == W) res[v] = r == last ? c : res[v];
                        } else if (k == B) {
                            d1[v][r] = l[v][r];  // the row below's last diagonal
                        }
                    }
                }
            }
        }
    }
}

// Samples j .. j+3 of xw, those past `last` clamped to it (one branch instead
// of four clamps; it is the same for the whole warp but at a stream's end).
__device__ __forceinline__ void reg_load4(float* v, const float* __restrict__ xw, int j,
                                          int last) {
    if (j + 3 <= last) {
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __ldg(xw + j + u);
    } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __ldg(xw + min(j + u, last));
    }
}

// The query envelope in shared memory, as the search reads it: four rows a
// group, (-inf, +inf) past the query (no bound there).  Holds reg_env_len(M).
__host__ __device__ inline int reg_env_len(int M) { return (M + 3) / 4 * 4; }
__device__ __forceinline__ void reg_stage_env(float2* senv, const float2* __restrict__ qenv,
                                              int M) {
    for (int e = threadIdx.x; e < reg_env_len(M); e += blockDim.x)
        senv[e] = e < M ? qenv[e] : make_float2(-CDTW_INF, CDTW_INF);
}

template <int W, int NW>
__device__ __forceinline__ void reg_init(float (&p)[NW][2 * W + 2]) {
#pragma unroll
    for (int v = 0; v < NW; ++v) {
#pragma unroll
        for (int k = 0; k <= 2 * W + 1; ++k) p[v][k] = CDTW_INF;
        p[v][W] = 0.0f;  // virtual D[-1][-1] = 0 (cdtw.cuh:35, :191)
    }
}

// Windows per thread: as many as the shortest rows need to overlap their
// chains, no more (cycles a cell with 1 / 2 / 3 windows: W = 6 4.6 / 4.15 /
// 3.99, W = 12 4.32 / 3.87 / 3.89, W = 25 3.84 / 3.77 / 3.79, W = 30 3.76 /
// 3.82, W = 46 3.72 / 3.78): fewer registers leave more warps to a scheduler
// and a finer split of short streams.
constexpr int kMaxReg3W = 7;
constexpr int kMaxReg2W = 28;
constexpr int reg_per_thread(int W) { return W <= kMaxReg3W ? 3 : (W <= kMaxReg2W ? 2 : 1); }

// Listed windows (all in order without idx), NW per thread; a window past the
// list repeats its last and is not stored.  A group's samples are loaded one
// group ahead.
template <int W, bool EU, int NW>
__global__ void __launch_bounds__(kRegBlock, 1)
cdtw_reg_kernel(const float* __restrict__ x, const double* __restrict__ mu,
                const float* __restrict__ sigma, const float4* __restrict__ qpad4, int lq4,
                int M, int Nw, const int32_t* __restrict__ idx, int L, float* __restrict__ out) {
    extern __shared__ float4 sq4[];
    for (int e = threadIdx.x; e < lq4; e += blockDim.x) sq4[e] = qpad4[e];
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((int64_t)NW * t >= L) return;
    Norm nm[NW];
    const float* xw[NW];
    bool ok[NW];
    float xn[NW][4], res[NW];
#pragma unroll
    for (int v = 0; v < NW; ++v) {
        const int tv = min(NW * t + v, L - 1);
        int w = idx ? idx[tv] : tv;
        ok[v] = w >= 0 && w < Nw;
        if (!ok[v]) w = 0;  // a listed window outside the subject: NaN, no access
        nm[v] = make_norm(mu[w], sigma[w]);
        xw[v] = x + w;
        res[v] = CDTW_INF;
        reg_load4(xn[v], xw[v], 0, M - 1);
    }
    float p[NW][2 * W + 2];
    reg_init<W, NW>(p);
    for (int j0 = 0; j0 < M; j0 += 4) {
        float z[NW][4];
#pragma unroll
        for (int v = 0; v < NW; ++v) {
#pragma unroll
            for (int r = 0; r < 4; ++r) z[v][r] = znorm(nm[v], xn[v][r]);
            reg_load4(xn[v], xw[v], j0 + 4, M - 1);
        }
        reg_rows4<W, EU, NW, true>(p, z, sq4 + (j0 >> 2), M - 1 - j0, res);
    }
#pragma unroll
    for (int v = 0; v < NW; ++v)
        if (NW * t + v < L) out[NW * t + v] = ok[v] ? res[v] : __int_as_float(0x7fc00000);
}

// All windows, NW consecutive ones per thread (windows NW t .. NW t + NW - 1,
// no index list): window v's sample at row j is x[NW t + v + j], so the NW
// windows of a thread read one sliding run of the stream.  A group of four
// rows needs NW + 3 consecutive samples, of which four are new: they are
// loaded one group ahead and the run is shifted by four at the end of the
// group.  Every group but the last runs without result tests; the last (one to
// four rows) ends at row M - 1.
template <int W, bool EU, int NW>
__global__ void __launch_bounds__(kRegBlock, 1)
cdtw_regc_kernel(const float* __restrict__ x, const double* __restrict__ mu,
                 const float* __restrict__ sigma, const float4* __restrict__ qpad4, int lq4,
                 int M, int Nw, float* __restrict__ out) {
    extern __shared__ float4 sq4[];
    for (int e = threadIdx.x; e < lq4; e += blockDim.x) sq4[e] = qpad4[e];
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int w0 = t * NW;
    if (w0 >= Nw) return;
    constexpr int NX = NW + 3;  // samples of a group of four rows
    // the last thread's missing windows repeat window Nw - 1's statistics and
    // read clamped samples; they are not stored
    const int rem = Nw - 1 - w0;                 // windows after w0 (>= 0)
    const int xlast = rem + M - 1;               // last sample index from w0
    const float* __restrict__ xb = x + w0;
    Norm nm[NW];
#pragma unroll
    for (int v = 0; v < NW; ++v) {
        const int w = w0 + min(v, rem);
        nm[v] = make_norm(mu[w], sigma[w]);
    }
    float p[NW][2 * W + 2], res[NW];
    reg_init<W, NW>(p);
#pragma unroll
    for (int v = 0; v < NW; ++v) res[v] = CDTW_INF;
    float xs[NX];
#pragma unroll
    for (int i = 0; i < NX; ++i) xs[i] = __ldg(xb + min(i, xlast));
    auto samples = [&](float (&z)[NW][4]) {
#pragma unroll
        for (int v = 0; v < NW; ++v) {
#pragma unroll
            for (int r = 0; r < 4; ++r) z[v][r] = znorm(nm[v], xs[r + v]);
        }
    };
    int j0 = 0;
    for (; j0 + 4 < M; j0 += 4) {
        float nx[4], z[NW][4];
        reg_load4(nx, xb, j0 + NX, xlast);
        samples(z);
        reg_rows4<W, EU, NW, false>(p, z, sq4 + (j0 >> 2), 0, res);
#pragma unroll
        for (int i = 0; i + 4 < NX; ++i) xs[i] = xs[i + 4];
#pragma unroll
        for (int i = 0; i < 4; ++i) xs[NX - 4 + i] = nx[i];
    }
    float z[NW][4];
    samples(z);
    reg_rows4<W, EU, NW, true>(p, z, sq4 + (j0 >> 2), M - 1 - j0, res);
#pragma unroll
    for (int v = 0; v < NW; ++v)
        if (v <= rem) out[w0 + v] = res[v];
}

using RegCKernel = void (*)(const float*, const double*, const float*, const float4*, int, int,
                            int, float*);

template <int LO, int HI>
struct RegCRange {
    static void fill(RegCKernel* eu, RegCKernel* mh) {
        if constexpr (LO <= HI) {
            eu[LO] = cdtw_regc_kernel<LO, true, reg_per_thread(LO)>;
            mh[LO] = cdtw_regc_kernel<LO, false, reg_per_thread(LO)>;
            RegCRange<LO + 1, HI>::fill(eu, mh);
        }
    }
};

// cDTW of one window (xw, normalisation nm) against the query whose padded
// copy sits in shared memory (sq4) with its envelope senv, abandoning once the
// last row minimum plus the remaining suffix of the window's forward LB_Keogh
// lbk (the cumulative bound cb of UCR_DTW_BIN.cpp:666-677, :336) reaches the
// best-so-far in *key.  alive marks lanes still worth finishing; the warp stops
// when no lane is.  All 32 lanes call together.  Returns +inf if the warp
// stopped early.
template <int W, bool EU>
__device__ __forceinline__ float reg_window_dtw(const float4* sq4, const float2* senv, int M,
                                                const float* __restrict__ xw, const Norm& nm,
                                                float lbk, bool& alive,
                                                const unsigned long long* key) {
    constexpr int B = 2 * W + 1;
    float p[1][B + 1], z[1][4], res[1] = {CDTW_INF};
    reg_init<W, 1>(p);
    float pre = 0.f;
    // W <= 64: the samples of the next 4-row group are loaded one group ahead
    // (with few windows in flight their latency is not hidden by other warps;
    // wider bands leave no registers for it)
    constexpr bool kAhead = W <= 64;
    float xn[4];
    if (kAhead) reg_load4(xn, xw, 0, M - 1);
    for (int j0 = 0; j0 < M; j0 += 4) {
        float xc[4];
        if constexpr (kAhead) {
#pragma unroll
            for (int u = 0; u < 4; ++u) xc[u] = xn[u];
            reg_load4(xn, xw, j0 + 4, M - 1);
        } else {
            reg_load4(xc, xw, j0, M - 1);
        }
        const bool check = (j0 & 7) == 4 && j0 + 3 < M - 1;  // rows j0..j0+3 are all real rows
        // W <= 64: the best-so-far is read before the group's cells
        const float bsf_early = (kAhead && check) ? load_bsf(key) : 0.f;
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
            // forward LB_Keogh terms of these data rows (query envelope there;
            // (-inf, +inf) past row M - 1)
            const float4 e = reinterpret_cast<const float4*>(senv)[(j0 + u) >> 1];
            z[0][u] = znorm(nm, xc[u]);
            z[0][u + 1] = znorm(nm, xc[u + 1]);
            const float d0 = max3f(z[0][u] - e.y, e.x - z[0][u], 0.f);
            const float d1 = max3f(z[0][u + 1] - e.w, e.z - z[0][u + 1], 0.f);
            pre += EU ? d0 * d0 : d0;
            pre += EU ? d1 * d1 : d1;
        }
        reg_rows4<W, EU, 1, true>(p, z, sq4 + (j0 >> 2), M - 1 - j0, res);
        if (check) {
            float rmin = p[0][0];
#pragma unroll
            for (int k = 1; k < B; k += 2) rmin = min3f(rmin, p[0][k], p[0][k + 1]);
            alive = alive && (rmin + lb_suffix(lbk, pre, M) * kLbSlack <
                              (kAhead ? bsf_early : load_bsf(key)));
            if (!__any_sync(0xffffffffu, alive)) return CDTW_INF;
        }
    }
    return res[0];
}

// Search variant: persistent warps take 32 candidates at a time from a device
// list, skip those whose lower bound already exceeds the best-so-far, run the
// register-band DTW with early abandoning, and fold results into *key by a
// packed (distance, window) atomicMin, so ties keep the lowest window (or
// append them to a hit list, report_window).  One block an SM in the launch
// bounds: left to itself the compiler holds the registers down for more warps
// and the rows' chains no longer overlap (W = 60, 168 registers instead of 180:
// 4 candidates of M = 300 151 us and 95, 100000 351 and 249; W = 25 78 and 50,
// 160 and 159).
template <int W, bool EU>
__global__ void __launch_bounds__(kRegBlock, 1)
cdtw_reg_search_kernel(const float* __restrict__ x, const double* __restrict__ mu,
                       const float* __restrict__ sigma, const float4* __restrict__ qpad4, int lq4,
                       const float2* __restrict__ qenv, int M, const Cand* __restrict__ cands,
                       const int* __restrict__ count, int* __restrict__ work,
                       unsigned long long* __restrict__ key, const HitSink sink, int nsm,
                       int gate) {
    extern __shared__ float4 sq4[];
    const int n = *(const volatile int*)count;
    if (n <= gate) return;  // the lane groups take them
    float2* senv = (float2*)(sq4 + lq4);
    for (int e = threadIdx.x; e < lq4; e += blockDim.x) sq4[e] = qpad4[e];
    reg_stage_env(senv, qenv, M);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int base = first_batch(work, 32, nsm); base < n; base = next_batch(work, 32)) {
        const int i = base + lane;
        Cand c;
        c.w = 0;
        c.lb = CDTW_INF;
        c.lbk = 0.f;
        if (i < n) c = cands[i];
        bool alive = (i < n) && (c.lb * kLbSlack < load_bsf(key));
        if (!__any_sync(0xffffffffu, alive)) continue;
        const Norm nm = make_norm(mu[c.w], sigma[c.w]);
        const float res = reg_window_dtw<W, EU>(sq4, senv, M, x + c.w, nm, c.lbk, alive, key);
        if (i < n && res < CDTW_INF) report_window(key, sink, res, (uint32_t)c.w);
    }
}

using RegKernel = void (*)(const float*, const double*, const float*, const float4*, int, int,
                           int, const int32_t*, int, float*);
using RegSearchKernel = void (*)(const float*, const double*, const float*, const float4*, int,
                                 const float2*, int, const Cand*, const int*, int*,
                                 unsigned long long*, const HitSink, int, int);

// Instantiates the one-window and the search kernels for bands LO..HI into the
// dispatch tables.
template <int LO, int HI>
struct RegRange {
    static void fill(RegKernel* eu, RegKernel* mh, RegSearchKernel* seu, RegSearchKernel* smh) {
        if constexpr (LO <= HI) {
            eu[LO] = cdtw_reg_kernel<LO, true, 1>;
            mh[LO] = cdtw_reg_kernel<LO, false, 1>;
            seu[LO] = cdtw_reg_search_kernel<LO, true>;
            smh[LO] = cdtw_reg_search_kernel<LO, false>;
            RegRange<LO + 1, HI>::fill(eu, mh, seu, smh);
        }
    }
};

// Several windows per thread, where the band leaves the registers for it.
template <int LO, int HI>
struct RegNRange {
    static void fill(RegKernel* eu, RegKernel* mh) {
        if constexpr (LO <= HI) {
            eu[LO] = cdtw_reg_kernel<LO, true, reg_per_thread(LO)>;
            mh[LO] = cdtw_reg_kernel<LO, false, reg_per_thread(LO)>;
            RegNRange<LO + 1, HI>::fill(eu, mh);
        }
    }
};

}  // namespace

// Defined in cdtw_reg_part*.cu: each fills its range of bands.
void reg_fill_part0(void** eu, void** mh, void** seu, void** smh);
void reg_fill_part1(void** eu, void** mh, void** seu, void** smh);
void reg_fill_part2(void** eu, void** mh, void** seu, void** smh);
void reg_fill_part3(void** eu, void** mh, void** seu, void** smh);
void reg_fill_part4(void** eu, void** mh, void** seu, void** smh);
void reg_fill_part5(void** eu, void** mh, void** seu, void** smh);
void reg_fill_part6(void** eu, void** mh, void** seu, void** smh);
void reg_fill_part7(void** eu, void** mh, void** seu, void** smh);
void regn_fill_part0(void** eu, void** mh);  // several windows, cdtw_regn_part0.cu
// all-windows kernels over consecutive windows (cdtw_regc_part*.cu)
void regc_fill_part0(void** eu, void** mh);
void regc_fill_part1(void** eu, void** mh);
void regc_fill_part2(void** eu, void** mh);
void regc_fill_part3(void** eu, void** mh);
void regc_fill_part4(void** eu, void** mh);
void regc_fill_part5(void** eu, void** mh);

}  // namespace cdtw

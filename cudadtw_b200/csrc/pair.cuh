// Differentiable pairwise cDTW, forward device code (no reference
// counterpart; the DP is the
// banded recurrence of include/cdtw.cuh:24-88 / UCR_DTW_BIN.cpp:288-354 on
// two series of equal length L).
//
// Forward: one group of G lanes (a power of two) per pair walks the band
// anti-diagonal by anti-diagonal.  Anti-diagonal k = i + j holds the band
// cells d = j - i with d = k (mod 2), |d| <= W; slot p = (d + W - e) / 2 with
// e = (k + W) & 1, so every anti-diagonal has W + 1 slots and lane l owns
// slots [l*C, l*C + C).  A cell needs slot p (diag) from k-2 and slots p, p-1
// (e = 0) or p+1, p (e = 1) from k-1: one shuffle per step.  The query values
// of a lane's cells move by one position every second step and the subject
// values every other step; the windows are rotated by index (the step loop
// is unrolled 2C times) and refilled by a shuffle from the neighbouring lane,
// the edge lanes reading the pair's series from global memory (L2-resident).
//
// With a path record the forward also stores 2 bits per band cell (diagonal
// predecessor is the minimum; up <= left) in device scratch, one element of
// 2C bits per lane and anti-diagonal (a byte for C <= 4, 16 bits for C <= 8,
// else 32), and, once the pair is done, one lane backtracks from (L-1, L-1)
// to (0, 0) and writes the warping path as row runs [a_i, b_i] and column
// runs [c_j, d_j]; or it stores two anti-diagonals every few, from which
// another kernel recomputes the band around the path.  Backward
// sums the cost derivatives over those runs and applies the z-normalisation
// Jacobian (I - 11'/L - zz'/L) / sigma.
#pragma once

#include "common.cuh"

#include <algorithm>
#include <type_traits>
#include <utility>

namespace cdtw {

constexpr int kPairThreads = 128;
// Thin checkpoints: anti-diagonals between them (at most kThinSeg, even).
// Lanes of up to kThinBody slots write them wherever they fall due; wider
// lanes, whose unrolled steps hold the instruction cache as they are, at the
// start of a body of 2C steps only.
constexpr int kThinSeg = 30;
constexpr int kThinBody = 8;
constexpr int thin_seg(int C) { return C <= kThinBody ? kThinSeg : 2 * C; }
constexpr int kWalkChunk = 64;  // bytes of direction record per lane in one backtracking chunk
constexpr unsigned kFull = 0xffffffffu;

struct PairArgs {
    const float* zq;      // DP inputs: n x L (z-normalised copies or the raw series);
    const float* zs;      // pair p's query starts at zq + p * qstride (0: one shared query)
    int64_t qstride;
    int64_t n;
    int L, W, G, lgG;
    float* D;             // n outputs
    uint32_t* dirs;       // per pair dstride words: 2L-1 rows of G lane elements (path record)
    int dstride;
    int recb, logb;       // shared-record mode: bytes of record and move log per group
    const int* gate;      // when set: a device count of the pairs present (at most n);
    int gate_max;         // the launch does nothing when it exceeds gate_max
    int gate_min;         // or when it is at most gate_min
    uint32_t* rows;       // per pair L words: a_i | b_i << 16
    uint32_t* cols;       // per pair L words: c_j | d_j << 16
    float* ckpt;          // checkpointed mode: per pair nseg x 2C x G floats
    int seg;              // anti-diagonals per segment (a multiple of 2C)
    int nseg;             // segments per pair
    int C;                // band slots per lane of the forward (corridor walk)
};

namespace {


// z-value of one sample with the pair header's mean and sigma (shared by the
// forward preparation and the backward pass, so both see the same floats).
__device__ __forceinline__ float pair_z(float x, double mu, double inv) {
    return (float)(((double)x - mu) * inv);
}

// Direction bits of one cell, as predicated ORs of immediates: bit SH when
// the diagonal is the minimum, bit SH+1 when up <= left.
template <int SH>
__device__ __forceinline__ void dir_bits(uint32_t& w, float diag, float m, float up, float left) {
    asm("{\n\t.reg .pred p;\n\tsetp.eq.f32 p, %1, %2;\n\t@p or.b32 %0, %0, %3;\n\t}"
        : "+r"(w) : "f"(diag), "f"(m), "n"(1u << SH));
    asm("{\n\t.reg .pred p;\n\tsetp.le.f32 p, %1, %2;\n\t@p or.b32 %0, %0, %3;\n\t}"
        : "+r"(w) : "f"(up), "f"(left), "n"(2u << SH));
}

// Direction element of one lane and anti-diagonal: 2 bits per slot.
template <int C>
using DirT = std::conditional_t<(C <= 4), uint8_t, std::conditional_t<(C <= 8), uint16_t, uint32_t>>;

// One cell (compile-time slot c) of an anti-diagonal of parity E.
template <int C, bool EU, bool DIRS, int E, int RQ, int RS, int c>
__device__ __forceinline__ void dp_cell(float (&X)[C], const float (&Y)[C], const float (&Q)[C],
                                        const float (&Sv)[C], const float (&lim)[C], float nb,
                                        uint32_t& nbits) {
    const float up = (E == 0) ? Y[c] : (c == C - 1 ? nb : Y[c + 1 < C ? c + 1 : c]);
    const float left = (E == 0) ? (c == 0 ? nb : Y[c > 0 ? c - 1 : 0]) : Y[c];
    const float diag = X[c];
    const float m = min3f(diag, up, left);
    const float df = __fsub_rn(Q[(c - RQ % C + C) % C], Sv[(c + RS) % C]);
    float v = EU ? __fmaf_rn(df, df, m) : __fadd_rn(fabsf(df), m);
    if (E == 1) v = fmaxf(v, lim[c]);  // d = W + 1 lies outside the band
    X[c] = v;
    if constexpr (DIRS) dir_bits<2 * c>(nbits, diag, m, up, left);
}

template <int C, bool EU, bool DIRS, int E, int RQ, int RS, int... Cs>
__device__ __forceinline__ void dp_cells_seq(float (&X)[C], const float (&Y)[C],
                                             const float (&Q)[C], const float (&Sv)[C],
                                             const float (&lim)[C], float nb, uint32_t& nbits,
                                             std::integer_sequence<int, Cs...>) {
    (dp_cell<C, EU, DIRS, E, RQ, RS, Cs>(X, Y, Q, Sv, lim, nb, nbits), ...);
}

// One anti-diagonal of parity E: X (slots of k-2) becomes k from Y (k-1).
// Logical query value of slot c is Q[(c - RQ) mod C], subject value
// Sv[(c + RS) mod C].
template <int C, bool EU, bool DIRS, int E, int RQ, int RS>
__device__ __forceinline__ void dp_cells(float (&X)[C], const float (&Y)[C], const float (&Q)[C],
                                         const float (&Sv)[C], const float (&lim)[C], float nb,
                                         uint32_t& bits) {
    uint32_t nbits = 0;
    dp_cells_seq<C, EU, DIRS, E, RQ, RS>(X, Y, Q, Sv, lim, nb, nbits,
                                         std::make_integer_sequence<int, C>{});
    if (DIRS) bits = nbits;
}

// State of one lane of a pair's group during the forward DP.
template <int C>
struct PairLane {
    float A[C], B[C], Q[C], Sv[C], lim[C];
    uint32_t bits;  // direction bits of the last anti-diagonal
    int iq, js;    // lane 0's slot-0 query index, lane G-1's last-slot subject index
    float pq, ps;  // the values at iq + 1 / js + 1 (the next shift's)
};

// Direction element of anti-diagonal k: to the pair's global record (DM 1,
// live groups only) or to the group's shared-memory record (DM 2).
template <int C, int DM>
__device__ __forceinline__ void store_dirs(const PairLane<C>& st, uint32_t* drow, int G, int l,
                                           int k, bool live) {
    if constexpr (DM == 1 || DM == 2) {
        if (DM == 2 || live) ((DirT<C>*)drow)[(size_t)k * G + l] = (DirT<C>)st.bits;
    }
}

// The sample entering at the group's edge, loaded by every lane: one address a
// group, no branch around the load (a step without the edge lanes' branches:
// 512 pairs of 2048, W = 409, 345 -> 232 us).  Past the series' ends a lane
// holds cells outside the matrix, which no cell inside takes a value from: any
// sample will do.
__device__ __forceinline__ float edge_sample(const float* x, int i, int L) {
    return __ldg(x + min(max(i, 0), L - 1));
}
// The same where only the edge lane takes it: stored directions of wide lanes
// (C > 4), whose unrolled body is the larger for the others' loads (4096 pairs
// of 2048, W = 409: 4.1 ms so, 5.7 ms with edge_sample).
template <int C, bool DIRS>
__device__ __forceinline__ void edge_next(float& v, int& i, const float* x, int L, bool edge) {
    if constexpr (DIRS && C > 4) {
        if (edge) {
            ++i;
            v = i + 1 < L ? __ldg(x + i + 1) : 0.f;
        }
    } else {
        ++i;
        v = edge_sample(x, i + 1, L);
    }
}

// Checkpoint of the two newest anti-diagonals (A = k-1, B = k-2) before the
// odd step k.  Wide layout: slot-major over the group's G x C slots, so a
// group's lanes write adjacent words.  Thin layout: the W + 1 band slots
// alone, slot c of lane l at c q + min(c, r) + l with q, r the quotient and
// remainder of (W + 1) / C (the lanes that have a band slot c are the first
// q + (c < r)).
template <int C>
__device__ __forceinline__ void ckpt_store(const PairLane<C>& st, float* ck, int G, int l,
                                           bool live) {
    if (!live) return;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        ck[(size_t)c * G + l] = st.A[c];
        ck[(size_t)(C + c) * G + l] = st.B[c];
    }
}
template <int C>
__device__ __forceinline__ void ckpt_store_thin(const PairLane<C>& st, float* ck, int W, int l,
                                                bool live) {
    const int q = (W + 1) / C, r = (W + 1) % C;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        if (live && l * C + c <= W) {
            const int at = c * q + min(c, r) + l;
            ck[at] = st.A[c];
            ck[W + 1 + at] = st.B[c];
        }
    }
}

// Where a pair's next checkpoint goes and the anti-diagonal it is due before.
struct NextCkpt {
    float* to;
    int due;
};

// Step with parity 1 (subject window shifts first; post-shift rotation RS)
// writing B from A; step with parity 0 (query window shifts; rotation RQ)
// writing A from B.
template <int C, bool EU, bool DIRS, int RQ, int RS>
__device__ __forceinline__ void step_odd(PairLane<C>& st, const float* ss, int L, int G, int l,
                                         bool shift) {
    if (shift) {
        constexpr int slot = (RS - 1 + C) % C;
        const float v = __shfl_down_sync(kFull, st.Sv[slot], 1, G);
        st.Sv[slot] = (l == G - 1) ? st.ps : v;
        edge_next<C, DIRS>(st.ps, st.js, ss, L, l == G - 1);
    }
    float nb = __shfl_down_sync(kFull, st.A[0], 1, G);
    if (l == G - 1) nb = CDTW_INF;
    dp_cells<C, EU, DIRS, 1, RQ, RS>(st.B, st.A, st.Q, st.Sv, st.lim, nb, st.bits);
}

template <int C, bool EU, bool DIRS, int RQ, int RS>
__device__ __forceinline__ void step_even(PairLane<C>& st, const float* sq, int L, int G, int l,
                                          bool shift) {
    if (shift) {
        constexpr int slot = (C - RQ) % C;  // = (C - 1 - (RQ - 1)) mod C
        const float v = __shfl_up_sync(kFull, st.Q[slot], 1, G);
        st.Q[slot] = (l == 0) ? st.pq : v;
        edge_next<C, DIRS>(st.pq, st.iq, sq, L, l == 0);
    }
    float nb = __shfl_up_sync(kFull, st.B[C - 1], 1, G);
    if (l == 0) nb = CDTW_INF;
    dp_cells<C, EU, DIRS, 0, RQ, RS>(st.A, st.B, st.Q, st.Sv, st.lim, nb, st.bits);
}

// 2C steps (C odd/even pairs) starting with an odd step at k; rotations
// return to 0 at the end.  CHK: stop at K (else the caller guarantees
// k + 2C <= K).
template <int C, bool EU, int DM, bool CHK, int R>
__device__ __forceinline__ void body(PairLane<C>& st, const float* sq, const float* ss,
                                     uint32_t* drow, int L, int G, int l, int& k, int K,
                                     bool live, NextCkpt& nc, int seg, int W) {
    if constexpr (R < C) {
        constexpr bool DIRS = DM == 1 || DM == 2;
        if (CHK && k >= K) return;
        if constexpr (DM == 5 && C <= kThinBody) {
            if (k == nc.due) {  // uniform
                ckpt_store_thin<C>(st, nc.to, W, l, live);
                nc.due += seg;
                nc.to += 2 * (W + 1);
            }
        }
        step_odd<C, EU, DIRS, R, R + 1>(st, ss, L, G, l, true);
        store_dirs<C, DM>(st, drow, G, l, k, live);
        ++k;
        if (CHK && k >= K) return;
        step_even<C, EU, DIRS, R + 1, R + 1>(st, sq, L, G, l, true);
        store_dirs<C, DM>(st, drow, G, l, k, live);
        ++k;
        body<C, EU, DM, CHK, R + 1>(st, sq, ss, drow, L, G, l, k, K, live, nc, seg, W);
    }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

constexpr int kWalkStages = 4;            // direction chunks in flight during backtracking
constexpr int kMoveLog = 256;             // bytes: the moves of one chunk (<= kWalkChunk)
constexpr size_t kSharedRecMax = 76 * 1024;  // shared-record mode: bytes per block (3 per SM)

// Row runs (a_i, b_i) and column runs (c_j, d_j) of the moves mlog[m0 ..
// m0 + nmax) of the group, lane l taking V consecutive moves; (gi, gj) is the
// (group-uniform) cell before move m0 and is advanced past the moves.  Every
// lane of the warp calls with the same nmax (full-mask shuffles).
template <int V>
__device__ __forceinline__ void runs_from_moves(const uint8_t* mlog, int nm, int nmax, int G,
                                                int l, bool live, int L, uint16_t* r16,
                                                uint16_t* c16, int& gi, int& gj) {
    for (int m0 = 0; m0 < nmax; m0 += V * G) {
        uint32_t bv[V];
        int nr = 0, nc = 0;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int m = m0 + V * l + v;
            bv[v] = m < nm ? mlog[m] : 4u;  // 4: no move
            nr += (bv[v] != 0u && bv[v] != 4u) ? 1 : 0;  // leaves its row
            nc += (bv[v] != 2u && bv[v] != 4u) ? 1 : 0;  // leaves its column
        }
        int sr = nr, sc = nc;  // inclusive scans over the group
        for (int o = 1; o < G; o <<= 1) {
            const int tr = __shfl_up_sync(kFull, sr, o, G);
            const int tc = __shfl_up_sync(kFull, sc, o, G);
            if (l >= o) {
                sr += tr;
                sc += tc;
            }
        }
        int ib = gi - (sr - nr), jb = gj - (sc - nc);  // cell before this lane's first move
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const uint32_t b = bv[v];
            const int lr = (b != 0u && b != 4u) ? 1 : 0;
            const int lc = (b != 2u && b != 4u) ? 1 : 0;
            const bool inside = live && (unsigned)ib < (unsigned)L && (unsigned)jb < (unsigned)L;
            if (inside && lr) {
                r16[2 * ib] = (uint16_t)jb;                               // a_i
                if (ib > 0) r16[2 * (ib - 1) + 1] = (uint16_t)(jb - lc);  // b_(i-1)
            }
            if (inside && lc) {
                c16[2 * jb] = (uint16_t)ib;                               // c_j
                if (jb > 0) c16[2 * (jb - 1) + 1] = (uint16_t)(ib - lr);  // d_(j-1)
            }
            ib -= lr;
            jb -= lc;
        }
        gi -= __shfl_sync(kFull, sr, G - 1, G);
        gj -= __shfl_sync(kFull, sc, G - 1, G);
    }
}

// Bytes in front of a shared-memory record: two anti-diagonals and an element,
// which the walk's loads may touch.
template <int C>
__host__ __device__ constexpr int shared_pad(int G) {
    return ((2 * G + 1) * (int)sizeof(DirT<C>) + 3) / 4 * 4;
}

// One walker move from slot c of lane lw on anti-diagonal kw (parity e) by
// code b: diagonal keeps the slot, up (d + 1) / left (d - 1) move to slot
// c + e / c + e - 1 of the other parity.  Branch-free (the walkers of a warp
// take different moves).
template <int C>
__device__ __forceinline__ void walk_move(uint32_t b, int& kw, int& e, int& lw, int& c) {
    const bool dg = b & 1u;
    int cn = c + (dg ? 0 : (b ? e : e - 1));
    kw -= dg ? 2 : 1;
    e ^= dg ? 0 : 1;
    const bool hi = cn >= C, lo = cn < 0;
    cn += hi ? -C : (lo ? C : 0);
    lw += hi ? 1 : (lo ? -1 : 0);
    c = cn;
}

// Backtracking with the record in shared memory (DM 2): lane 0 of the group
// walks the whole record into the move log, reading the three possible next
// elements while it decodes the current one; then the group builds the runs.
template <int C>
__device__ __forceinline__ void walk_shared(const PairArgs& a, unsigned char* smem,
                                            const uint32_t* drow, int64_t pr, int L, int K,
                                            int G, int l, int gib, int e0, int porg, bool live) {
    using DT = DirT<C>;
    const DT* rec = (const DT*)drow;
    uint8_t* mlog = smem + (size_t)(blockDim.x >> a.lgG) * a.recb + (size_t)gib * a.logb;
    uint16_t* r16 = (uint16_t*)(a.rows + pr * L);  // [2i] = a_i, [2i+1] = b_i
    uint16_t* c16 = (uint16_t*)(a.cols + pr * L);  // [2j] = c_j, [2j+1] = d_j
    __syncwarp();  // the group's record is visible to its walker
    int nm = 0;
    if (l == 0 && live) {
        r16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
        c16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
        int e = e0, lw = porg / C, c = porg - lw * C;
        int at = (K - 1) * G + lw;  // element of the walker's anti-diagonal and lane
        uint32_t cur = rec[at];
        // every move lowers the anti-diagonal, so at most K moves (the log holds
        // K bytes); the loads before anti-diagonal 0 fall into the record's pad
        while (at >= 0 && (unsigned)lw < (unsigned)G) {
            const DT* below = rec + at - G;
            const uint32_t n2 = below[-G], n1 = below[0], n1m = below[-1], n1p = below[1];
            const uint32_t b = (cur >> (2 * c)) & 3u;
            mlog[nm++] = (uint8_t)b;
            const bool dg = b & 1u;
            const int cn = c + (dg ? 0 : (b ? e : e - 1));  // up keeps or raises the slot
            const bool hi = cn >= C, lo = cn < 0;
            const int dl = hi ? 1 : (lo ? -1 : 0);
            at += dg ? -2 * G : dl - G;
            c = cn + (hi ? -C : (lo ? C : 0));
            lw += dl;
            e ^= dg ? 0 : 1;
            cur = dg ? n2 : (hi ? n1p : (lo ? n1m : n1));
        }
    }
    nm = __shfl_sync(kFull, nm, 0, G);
    const int nmax = __reduce_max_sync(kFull, (unsigned)nm);
    __syncwarp();
    int gi = L - 1, gj = L - 1;
    runs_from_moves<4>(mlog, nm, nmax, G, l, live, L, r16, c16, gi, gj);
}

// Backtracking with the record in global scratch (DM 1): the record streams
// into a kWalkStages-deep shared-memory ring in chunks of R anti-diagonals
// (kWalkChunk bytes per lane, 16-byte cp.async copies), last chunk first;
// lane 0 of the group decodes a chunk's moves into a byte log (2-bit codes: 1
// or 3 diagonal, 2 up (i-1, j), 0 left (i, j-1)) and the group turns the log
// into runs.  Cell (0, 0) always records a diagonal move (its diagonal is the
// origin, the other predecessors are +inf): it writes the last runs and ends
// the walk.
template <int C>
__device__ __forceinline__ void walk_ring(const PairArgs& a, unsigned char* smem,
                                          const uint32_t* drow, int64_t pr, int L, int K, int G,
                                          int l, int gib, int e0, int porg, bool live) {
    using DT = DirT<C>;
    constexpr int R = kWalkChunk / (int)sizeof(DT);  // anti-diagonals per chunk
    unsigned char* ring = smem + (size_t)gib * kWalkStages * kWalkChunk * G;
    uint8_t* mlog = smem + (size_t)blockDim.x * kWalkStages * kWalkChunk + gib * kMoveLog;
    const int nch = (K + R - 1) / R;  // the record holds nch whole chunks per pair
    const unsigned char* rec = (const unsigned char*)drow;
    auto issue = [&](int ch) {
        if (ch < nch) {
            unsigned char* dst = ring + (ch % kWalkStages) * kWalkChunk * G;
            const unsigned char* src = rec + (size_t)(nch - 1 - ch) * kWalkChunk * G;
#pragma unroll 4
            for (int t = l; t < kWalkChunk / 16 * G; t += G) cp_async16(dst + 16 * t, src + 16 * t);
        }
        cp_async_commit();
    };
    __syncwarp();  // the group's direction elements are visible to all its lanes
#pragma unroll
    for (int ch = 0; ch < kWalkStages - 1; ++ch) issue(ch);
    uint16_t* r16 = (uint16_t*)(a.rows + pr * L);  // [2i] = a_i, [2i+1] = b_i
    uint16_t* c16 = (uint16_t*)(a.cols + pr * L);  // [2j] = c_j, [2j+1] = d_j
    if (l == 0 && live) {
        r16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
        c16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
    }
    int kw = K - 1, e = e0;                  // walker: anti-diagonal and its parity
    int lw = porg / C, c = porg - lw * C;    // slot c of lane lw
    int gi = L - 1, gj = L - 1;  // (group-uniform) cell before the chunk's first move
    for (int ch = 0; ch < nch; ++ch) {  // same trip count in every group of the warp
        issue(ch + kWalkStages - 1);
        cp_async_wait<kWalkStages - 1>();
        __syncwarp();
        int nm = 0;
        if (l == 0 && live) {  // groups past the last pair do not walk
            const DT* buf = (const DT*)(ring + (ch % kWalkStages) * kWalkChunk * G);
            const int rlo = (nch - 1 - ch) * R;
            // every move lowers kw: at most R (<= kMoveLog) moves per chunk
            while (kw >= rlo && (unsigned)lw < (unsigned)G) {
                const uint32_t b = ((uint32_t)buf[(kw - rlo) * G + lw] >> (2 * c)) & 3u;
                mlog[nm++] = (uint8_t)b;
                walk_move<C>(b, kw, e, lw, c);
            }
        }
        nm = __shfl_sync(kFull, nm, 0, G);
        // every lane of the warp runs the same number of scan rounds (the
        // groups' move counts differ): the full-mask shuffles below need it
        const int nmax = __reduce_max_sync(kFull, (unsigned)nm);
        __syncwarp();
        runs_from_moves<1>(mlog, nm, nmax, G, l, live, L, r16, c16, gi, gj);
        __syncwarp();
    }
    cp_async_wait<0>();
}

// Lane state at anti-diagonal 0 (D[-1][-1] = 0 under d = 0; the group's lanes
// hold the band slots from pb) and the first one or two steps, up to the first step of parity 1 (k0 = 1 or 2), where the
// bodies of 2C steps begin.  Returns k0.
template <int C, bool EU, int DM>
__device__ __forceinline__ int pair_begin(PairLane<C>& st, const float* sq, const float* ss,
                                          uint32_t* drow, int L, int W, int G, int l, int K,
                                          bool live, int pb = 0) {
    constexpr bool DIRS = DM == 1 || DM == 2;
    const int e0 = W & 1;
    const int p0 = pb + l * C;
    const int porg = W >> 1;  // slot of d = 0 on every anti-diagonal of parity e0
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int p = p0 + c;
        st.lim[c] = (p == W) ? CDTW_INF : -CDTW_INF;
        const float org = (p == porg) ? 0.f : CDTW_INF;  // D[-1][-1] = 0 at k = -2
        st.A[c] = e0 == 0 ? org : CDTW_INF;
        st.B[c] = e0 == 0 ? CDTW_INF : org;
        const int d = -W + 2 * p + e0;
        const int i = -d / 2, j = d / 2;  // k = 0
        st.Q[c] = (i >= 0 && i < L) ? __ldg(sq + i) : 0.f;
        st.Sv[c] = (j >= 0 && j < L) ? __ldg(ss + j) : 0.f;
    }
    st.bits = 0;
    st.iq = (W - e0) / 2 - pb;                        // lane 0's slot-0 query index at k = 0
    st.js = (-W + 2 * (pb + G * C - 1) + e0) / 2;  // lane G-1's last-slot subject index
    st.pq = edge_sample(sq, st.iq + 1, L);
    st.ps = edge_sample(ss, st.js + 1, L);
    int k = 0;
    if (e0 == 0) {
        step_even<C, EU, DIRS, 0, 0>(st, sq, L, G, l, false);
        store_dirs<C, DM>(st, drow, G, l, k, live);
        k = 1;
    } else {
        step_odd<C, EU, DIRS, 0, 0>(st, ss, L, G, l, false);
        store_dirs<C, DM>(st, drow, G, l, k, live);
        k = 1;
        if (k < K) {
            // query shift with the rotation kept at 0: move the window down
            const float v = __shfl_up_sync(kFull, st.Q[C - 1], 1, G);
#pragma unroll
            for (int c = C - 1; c > 0; --c) st.Q[c] = st.Q[c - 1];
            st.Q[0] = (l == 0) ? st.pq : v;
            ++st.iq;
            st.pq = edge_sample(sq, st.iq + 1, L);
            step_even<C, EU, DIRS, 0, 0>(st, sq, L, G, l, false);
            store_dirs<C, DM>(st, drow, G, l, k, live);
            k = 2;
        }
    }
    return k;
}

// Lane state at the start of the body whose first step is k (parity 1),
// from checkpoint ck, written by G0 lanes of C0 slots each: the DP values of
// the slots from pb (+inf past the last), and the query / subject windows of
// step k-1 (rotation 0) rebuilt from the series -- the values the forward held
// there, so the recomputation is bit-identical.
template <int C>
__device__ __forceinline__ void ckpt_restore(PairLane<C>& st, const float* ck, const float* sq,
                                             const float* ss, int L, int W, int G, int l, int k,
                                             int G0, int C0, int pb) {
    const int p0 = pb + l * C;
    const int km = k - 1;                 // last anti-diagonal computed (parity 0)
    const int em = (km + W) & 1;          // = 0
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int p = p0 + c;
        st.lim[c] = (p == W) ? CDTW_INF : -CDTW_INF;
        const int l0 = p / C0, c0 = p - l0 * C0;
        const bool in = l0 < G0;
        st.A[c] = in ? ck[(size_t)c0 * G0 + l0] : CDTW_INF;
        st.B[c] = in ? ck[(size_t)(C0 + c0) * G0 + l0] : CDTW_INF;
        const int d = -W + 2 * p + em;
        const int i = (km - d) / 2, j = (km + d) / 2;
        st.Q[c] = (i >= 0 && i < L) ? __ldg(sq + i) : 0.f;
        st.Sv[c] = (j >= 0 && j < L) ? __ldg(ss + j) : 0.f;
    }
    st.bits = 0;
    st.iq = (km + W - em) / 2 - pb;                       // lane 0, slot 0 at k-1
    st.js = (km - W + 2 * (pb + G * C - 1) + em) / 2;     // lane G-1, last slot at k-1
    st.pq = edge_sample(sq, st.iq + 1, L);
    st.ps = edge_sample(ss, st.js + 1, L);
}

// DM: 0 distance only; 1 path record in global scratch, walked through a
// shared-memory ring; 2 path record in shared memory (short pairs, C <= 4);
// 3 distance plus checkpoints every a.seg anti-diagonals (the path is then
// recovered by pair_ckpt_walk_kernel or pair_corridor_kernel); 5 the same
// with checkpoints every thin_seg(C) (pair_thin_kernel).
template <int C, bool EU, int DM>
__global__ void __launch_bounds__(kPairThreads, 4) pair_fwd_kernel(const PairArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    int64_t np = a.n;  // pairs present
    if (a.gate) {
        const int c = *a.gate;
        if (c > a.gate_max || c <= a.gate_min) return;  // uniform for the whole launch
        np = min(np, (int64_t)max(c, 0));
    }
    const int G = a.G, L = a.L, W = a.W;
    const int tid = threadIdx.x;
    const int l = tid & (G - 1);
    const int gib = tid >> a.lgG;  // group in block
    const int64_t grp = (int64_t)blockIdx.x * (blockDim.x >> a.lgG) + gib;
    // a warp whose groups all lie past the pairs present has nothing to do
    // (groups never straddle warps: G is a power of two <= 32)
    if ((int64_t)blockIdx.x * (blockDim.x >> a.lgG) + ((tid & ~31) >> a.lgG) >= np) return;
    const bool live = grp < np;
    const int64_t pr = live ? grp : np - 1;
    const float* sq = a.zq + pr * a.qstride;  // the pair's series (L2-resident; edge lanes read them)
    const float* ss = a.zs + pr * L;

    const int K = 2 * L - 1;
    const int e0 = W & 1;
    const int p0 = l * C;
    const int porg = W >> 1;  // slot of d = 0 on every anti-diagonal of parity e0
    PairLane<C> st;
    uint32_t* drow = DM == 1   ? a.dirs + (size_t)pr * a.dstride
                     : DM == 2 ? (uint32_t*)(smem + (size_t)gib * a.recb + shared_pad<C>(G))
                               : nullptr;
    int k = pair_begin<C, EU, DM>(st, sq, ss, drow, L, W, G, l, K, live);
    NextCkpt nc{nullptr, K};
    if constexpr (DM == 3) {  // the place of checkpoint 0 stays unused
        nc.to = a.ckpt + (size_t)(pr * a.nseg + 1) * 2 * C * G;
        nc.due = k + a.seg;
    } else if constexpr (DM == 5) {
        nc.to = a.ckpt + (size_t)pr * (a.nseg - 1) * 2 * (C <= kThinBody ? W + 1 : C * G);
        nc.due = k + a.seg;
    }
    auto at_body = [&]() {  // checkpoints at body starts
        if constexpr (DM == 3 || (DM == 5 && C > kThinBody)) {
            if (k == nc.due) {
                ckpt_store<C>(st, nc.to, G, l, live);
                nc.due += a.seg;
                nc.to += 2 * C * G;
            }
        }
    };
    while (k + 2 * C <= K) {
        at_body();
        body<C, EU, DM, false, 0>(st, sq, ss, drow, L, G, l, k, K, live, nc, a.seg, W);
    }
    if (k < K) {
        at_body();
        body<C, EU, DM, true, 0>(st, sq, ss, drow, L, G, l, k, K, live, nc, a.seg, W);
    }

    // D[L-1][L-1]: slot porg of the last anti-diagonal (parity e0)
    float dval = CDTW_INF;
#pragma unroll
    for (int c = 0; c < C; ++c)
        if (p0 + c == porg) dval = (e0 == 0) ? st.A[c] : st.B[c];
    if (live && p0 <= porg && porg < p0 + C) a.D[pr] = dval;
    if constexpr (DM == 1) {
        walk_ring<C>(a, smem, drow, pr, L, K, G, l, gib, e0, porg, live);
    } else if constexpr (DM == 2) {
        walk_shared<C>(a, smem, drow, pr, L, K, G, l, gib, e0, porg, live);
    }
}

// Path recovery of the checkpointed mode: per pair, the segments of a.seg
// anti-diagonals from the last to the first are recomputed from their
// checkpoints (segment 0 from the start) with direction bits into shared
// memory, and lane 0 of the group walks the path back through each segment
// as walk_ring does through its chunks; the group turns each segment's moves
// into row and column runs.  Shared memory per group: a.recb bytes of
// directions (seg x G elements) and a.logb bytes of move log (>= seg).
template <int C, bool EU>
__global__ void __launch_bounds__(kPairThreads, 4) pair_ckpt_walk_kernel(const PairArgs a) {
    using DT = DirT<C>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int64_t np = a.n;
    const int G = a.G, L = a.L, W = a.W;
    const int tid = threadIdx.x;
    const int l = tid & (G - 1);
    const int gib = tid >> a.lgG;
    const int64_t grp = (int64_t)blockIdx.x * (blockDim.x >> a.lgG) + gib;
    if ((int64_t)blockIdx.x * (blockDim.x >> a.lgG) + ((tid & ~31) >> a.lgG) >= np) return;
    const bool live = grp < np;
    const int64_t pr = live ? grp : np - 1;
    const float* sq = a.zq + pr * a.qstride;
    const float* ss = a.zs + pr * L;
    const int K = 2 * L - 1;
    const int e0 = W & 1;
    const int porg = W >> 1;
    const int k0 = (e0 == 0) ? 1 : 2;
    const float* ck = a.ckpt + (size_t)pr * a.nseg * 2 * C * G;
    DT* rec = (DT*)(smem + (size_t)gib * a.recb);
    uint8_t* mlog = smem + (size_t)(blockDim.x >> a.lgG) * a.recb + (size_t)gib * a.logb;
    uint16_t* r16 = (uint16_t*)(a.rows + pr * L);  // [2i] = a_i, [2i+1] = b_i
    uint16_t* c16 = (uint16_t*)(a.cols + pr * L);  // [2j] = c_j, [2j+1] = d_j
    if (l == 0 && live) {
        r16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
        c16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
    }
    int kw = K - 1, e = e0;                // walker: anti-diagonal and its parity
    int lw = porg / C, c = porg - lw * C;  // slot c of lane lw
    int gi = L - 1, gj = L - 1;            // cell before the segment's first move
    for (int s = a.nseg - 1; s >= 0; --s) {
        const int kA = s == 0 ? 0 : k0 + s * a.seg;
        const int kB = min(k0 + (s + 1) * a.seg, K);
        // the record holds rows kA .. kB-1: store index k maps to row k - kA
        uint32_t* drow = (uint32_t*)((char*)rec - (ptrdiff_t)kA * G * (ptrdiff_t)sizeof(DT));
        PairLane<C> st;
        int k;
        if (s == 0) {
            k = pair_begin<C, EU, 2>(st, sq, ss, drow, L, W, G, l, K, live);
        } else {
            ckpt_restore<C>(st, ck + (size_t)s * 2 * C * G, sq, ss, L, W, G, l, kA, G, C, 0);
            k = kA;
        }
        NextCkpt none{nullptr, K};
        while (k + 2 * C <= kB)
            body<C, EU, 2, false, 0>(st, sq, ss, drow, L, G, l, k, kB, live, none, 0, W);
        if (k < kB) body<C, EU, 2, true, 0>(st, sq, ss, drow, L, G, l, k, kB, live, none, 0, W);
        __syncwarp();  // the segment's directions are visible to the walker
        int nm = 0;
        if (l == 0 && live) {
            // every move lowers kw: at most kB - kA (<= a.logb) moves here
            while (kw >= kA && (unsigned)lw < (unsigned)G) {
                const uint32_t b = ((uint32_t)rec[(size_t)(kw - kA) * G + lw] >> (2 * c)) & 3u;
                mlog[nm++] = (uint8_t)b;
                walk_move<C>(b, kw, e, lw, c);
            }
        }
        nm = __shfl_sync(kFull, nm, 0, G);
        const int nmax = __reduce_max_sync(kFull, (unsigned)nm);
        __syncwarp();
        runs_from_moves<4>(mlog, nm, nmax, G, l, live, L, r16, c16, gi, gj);
        __syncwarp();  // the record and the log are rewritten by the next segment
    }
}

// Path recovery of the checkpointed mode for bands wider than the path can
// stray within a segment: a warp per pair recomputes, per segment of a.seg
// anti-diagonals (last first), only the 32 CW band slots around the cell where
// the path enters it.  A cell of anti-diagonal k depends on the cells of
// anti-diagonal k - r within r of its diagonal, so of the checkpoint the
// a.seg + 1 slots around that cell decide every cell the path can reach
// (a.seg + 1 <= 32 CW); the others of the window may lack a neighbour and
// hold values that no cell of that cone takes.  The first segment starts at
// the origin, whose cone meets the wedge |d| <= k in half as many slots.
// Directions go to shared memory and are walked as in pair_ckpt_walk_kernel.
//
// Bound: the chain of 2L - 1 dependent anti-diagonals and the walk, per warp;
// the work is 32 CW / (W + 1) of a second forward.  CW = 4 (a byte of
// directions a lane) covers segments up to 127, CW = 5 those of 128.  512
// pairs of 2048, W = 409, with the forward: 1810 us recomputing the whole
// band, now 612.
template <int CW, bool EU>
__global__ void __launch_bounds__(kPairThreads, 4) pair_corridor_kernel(const PairArgs a) {
    using DT = DirT<CW>;
    constexpr int G = 32;
    extern __shared__ __align__(16) unsigned char smem[];
    const int L = a.L, W = a.W;
    const int l = threadIdx.x & 31, gib = threadIdx.x >> 5;
    const int64_t pr = (int64_t)blockIdx.x * (blockDim.x >> 5) + gib;
    if (pr >= a.n) return;  // whole warps
    const float* sq = a.zq + pr * a.qstride;
    const float* ss = a.zs + pr * L;
    const int K = 2 * L - 1;
    const int k0 = (W & 1) ? 2 : 1;
    const int pmax = max(a.G * a.C - 32 * CW, 0);  // last window start
    const float* ck = a.ckpt + (size_t)pr * a.nseg * 2 * a.C * a.G;
    DT* rec = (DT*)(smem + (size_t)gib * a.recb);
    uint8_t* mlog = smem + (size_t)(blockDim.x >> 5) * a.recb + (size_t)gib * a.logb;
    uint16_t* r16 = (uint16_t*)(a.rows + pr * L);  // [2i] = a_i, [2i+1] = b_i
    uint16_t* c16 = (uint16_t*)(a.cols + pr * L);  // [2j] = c_j, [2j+1] = d_j
    if (l == 0) {
        r16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
        c16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
    }
    int kw = K - 1, pw = W >> 1;  // walker: anti-diagonal and band slot
    int gi = L - 1, gj = L - 1;   // cell before the segment's first move
    for (int s = a.nseg - 1; s >= 0; --s) {
        const int kA = s == 0 ? 0 : k0 + s * a.seg;
        const int kB = min(k0 + (s + 1) * a.seg, K);
        // lowest slot of the cone at anti-diagonal kA - 1 (s > 0), or where it
        // meets the wedge of the origin
        const int dw = -W + 2 * pw + ((kw + W) & 1);
        const int dlo = s == 0 ? -((kw - dw) >> 1) - 2 : dw - (kw - kA + 1);
        const int pb = min(max((dlo + W) >> 1, 0), pmax);
        uint32_t* drow = (uint32_t*)((char*)rec - (ptrdiff_t)kA * G * (ptrdiff_t)sizeof(DT));
        PairLane<CW> st;
        int k;
        if (s == 0) {
            k = pair_begin<CW, EU, 2>(st, sq, ss, drow, L, W, G, l, K, true, pb);
        } else {
            ckpt_restore<CW>(st, ck + (size_t)s * 2 * a.C * a.G, sq, ss, L, W, G, l, kA, a.G,
                             a.C, pb);
            k = kA;
        }
        NextCkpt none{nullptr, K};
        while (k + 2 * CW <= kB)
            body<CW, EU, 2, false, 0>(st, sq, ss, drow, L, G, l, k, kB, true, none, 0, W);
        if (k < kB) body<CW, EU, 2, true, 0>(st, sq, ss, drow, L, G, l, k, kB, true, none, 0, W);
        __syncwarp();  // the segment's directions are visible to the walker
        int nm = 0;
        if (l == 0) {
            // every move lowers kw: at most kB - kA (<= a.logb) moves here.  The
            // three possible next elements are loaded while the current one is
            // decoded (as in walk_shared)
            int e = (kw + W) & 1, lw = (pw - pb) / CW, c = pw - pb - lw * CW;
            uint32_t cur = kw >= kA ? rec[(kw - kA) * G + lw] : 0u;
            while (kw >= kA && (unsigned)lw < (unsigned)G) {
                const int r1 = max(kw - 1 - kA, 0) * G + lw, r2 = max(kw - 2 - kA, 0) * G + lw;
                const uint32_t n2 = rec[r2];
                const uint32_t n1 = rec[r1];
                const uint32_t n1m = rec[max(r1 - 1, 0)];
                const uint32_t n1p = rec[r1 + 1];
                const uint32_t b = (cur >> (2 * c)) & 3u;
                mlog[nm++] = (uint8_t)b;
                const int lw0 = lw;
                walk_move<CW>(b, kw, e, lw, c);
                cur = (b & 1u) ? n2 : (lw > lw0 ? n1p : (lw < lw0 ? n1m : n1));
            }
            pw = pb + lw * CW + c;
        }
        nm = __shfl_sync(kFull, nm, 0);
        kw = __shfl_sync(kFull, kw, 0);
        pw = __shfl_sync(kFull, pw, 0);
        __syncwarp();
        runs_from_moves<4>(mlog, nm, nm, G, l, true, L, r16, c16, gi, gj);
        __syncwarp();  // the record and the log are rewritten by the next segment
    }
}

// Path recovery from checkpoints every a.seg <= kThinSeg anti-diagonals, a warp
// per pair: per segment (last first) the 32 band slots, one per lane, around
// the cell where the path enters it.  The cells the path can reach depend on
// a.seg + 1 slots of the checkpoint (see pair_corridor_kernel), so they all
// lie in the window.  A lane carries, with its cell's value, the moves of the
// cell's best path back to the start of the segment's half (kHalf
// anti-diagonals), two bits each, newest lowest: the cell takes the chosen
// predecessor's moves with its own shifted in, and the entry cell's lane holds
// the whole path through the half when its last anti-diagonal is done, with no
// walk over stored bits.  Lane t then takes move t, finds its cell from the
// moves before it by population counts and writes the row and column runs it
// ends; the cell the path leaves the upper half by picks the lower half's
// moves.
//
// Bound: with few pairs the latency of the chain, a shuffle, a min, a compare,
// two selects and a multiply-add per anti-diagonal; with many the half-rate
// compares and selects.  The window starts at slot -1 at the least, so the
// band's edges need no select (slot -1 and, on odd anti-diagonals, slot W are
// raised to +inf; a lane at the window's other edges reads its own value, in a
// cell outside the cone).  The next segment's checkpoint and samples are
// loaded a segment ahead for every window the path can enter it by.
//
// Measured with the forward before it (L = 2048, W = 409; direction bits for
// the whole band and a walk over them -> this): 512 pairs 1447 -> 483 us (238
// of them here), 4096 pairs 4.12 -> 1.83 ms; 1024 pairs of 1024, W = 102: 449
// -> 260 us.  With the bits of each anti-diagonal as two ballots in shared
// memory and a walk over those 388 us here, with 64-bit moves 260.
template <bool EU>
__global__ void __launch_bounds__(kPairThreads) pair_thin_kernel(const PairArgs a) {
    constexpr int kRows = kThinSeg + 2;    // the first segment holds k0 more
    constexpr int kHalf = 16;              // anti-diagonals of a lower half: 32 bits of moves
    constexpr int kSpan = 32 + kRows / 2;  // samples of each series a segment reads
    constexpr int kAhead = 3 * 32;         // samples loaded ahead: kSpan + 32 needed
    static_assert(kSpan + 32 <= kAhead && kRows <= 32, "segment sizes");
    __shared__ float qsm[kPairThreads / 32][kAhead], ssm[kPairThreads / 32][kAhead];
    const int L = a.L, W = a.W, seg = a.seg;
    const int l = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t pr = (int64_t)blockIdx.x * (kPairThreads / 32) + wib;
    if (pr >= a.n) return;  // whole warps
    const float* sq = a.zq + pr * a.qstride;
    const float* ss = a.zs + pr * L;
    const int K = 2 * L - 1, e0 = W & 1, k0 = e0 ? 2 : 1;
    // checkpoint layout: slot c of lane l at c cq + min(c, cr) + l
    const bool thin = a.C <= kThinBody;
    const int cq = thin ? (W + 1) / a.C : a.G, cr = thin ? (W + 1) % a.C : 0;
    const int half = thin ? W + 1 : a.C * a.G;
    const float* ck = a.ckpt + (size_t)pr * (a.nseg - 1) * 2 * half;
    const unsigned invC = 65536u / a.C + 1;  // p / C for p C < 65536
    float* qw = qsm[wib];
    float* sw = ssm[wib];
    uint16_t* r16 = (uint16_t*)(a.rows + pr * L);  // [2i] = a_i, [2i+1] = b_i
    uint16_t* c16 = (uint16_t*)(a.cols + pr * L);  // [2j] = c_j, [2j+1] = d_j
    if (l == 0) {
        r16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
        c16[2 * (L - 1) + 1] = (uint16_t)(L - 1);
    }
    const int pmax = max(W + 1 - 32, -1);  // last window start
    int kw = K - 1, pw = W >> 1;           // entry cell: anti-diagonal and band slot
    int gi = L - 1, gj = L - 1;            // and its indices
    // loaded ahead: checkpoint slots pa .. pa + 63 of both anti-diagonals,
    // samples from ia / ja
    float cA[2], cB[2], xq[3], xs[3];
    int pa = 0, ia = 0, ja = 0;
    auto ahead = [&](int s, int p0, int kA) {  // for segment s > 0 starting at kA
        pa = p0;
        ia = (kA + W - 1) / 2 - (pa + 32) - 31;
        ja = (kA - W + 1) / 2 + pa;
        const float* cs = ck + (size_t)(s - 1) * 2 * half;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int p = pa + 32 * v + l;
            const bool in = p >= 0 && p <= W;
            const int pc = in ? p : 0;
            const int l0 = (int)(pc * invC >> 16), c0 = pc - l0 * a.C;
            const int at = c0 * cq + min(c0, cr) + l0;
            cA[v] = in ? cs[at] : CDTW_INF;
            cB[v] = in ? cs[half + at] : CDTW_INF;
        }
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            xq[v] = edge_sample(sq, ia + 32 * v + l, L);
            xs[v] = edge_sample(ss, ja + 32 * v + l, L);
        }
    };
    // lowest slot of the window of segment s from its entry cell: the cone at
    // anti-diagonal kA - 1 (s > 0), or where it meets the wedge of the origin
    auto window = [&](int s, int kA) {
        const int dw = -W + 2 * pw + ((kw + W) & 1);
        const int dlo = s == 0 ? -((kw - dw) >> 1) - 2 : dw - (kw - kA + 1);
        return min(max((dlo + W) >> 1, -1), pmax);
    };
    // the moves h of a path from the entry cell down to anti-diagonal klo: runs
    // written, the entry cell moved to where the path leaves
    auto follow = [&](unsigned h, int klo) {
        const unsigned code = l < 16 ? h >> (2 * l) & 3u : 0u;
        const unsigned pd = __ballot_sync(kFull, code & 1u), pu = __ballot_sync(kFull, code == 2u);
        const unsigned below = (1u << l) - 1u;
        // anti-diagonal before the move; the moves that start in the half
        const int kt = kw - l - __popc(pd & below);
        const unsigned on = __ballot_sync(kFull, l < 16 && kt >= klo);
        const unsigned leave_row = (pd | pu) & on, leave_col = ~pu & on;
        if (on >> l & 1u) {
            const int ib = gi - __popc(leave_row & below), jb = gj - __popc(leave_col & below);
            const int lr = leave_row >> l & 1u, lc = leave_col >> l & 1u;
            if ((unsigned)ib < (unsigned)L && (unsigned)jb < (unsigned)L) {
                if (lr) {
                    r16[2 * ib] = (uint16_t)jb;                               // a_i
                    if (ib > 0) r16[2 * (ib - 1) + 1] = (uint16_t)(jb - lc);  // b_(i-1)
                }
                if (lc) {
                    c16[2 * jb] = (uint16_t)ib;                               // c_j
                    if (jb > 0) c16[2 * (jb - 1) + 1] = (uint16_t)(ib - lr);  // d_(j-1)
                }
            }
        }
        // k = i + j, d = j - i
        gi -= __popc(leave_row);
        gj -= __popc(leave_col);
        kw = gi + gj;
        pw = (gj - gi + W - ((kw + W) & 1)) / 2;
    };
    if (a.nseg > 1) ahead(a.nseg - 1, window(a.nseg - 1, k0 + (a.nseg - 1) * seg) - 16,
                          k0 + (a.nseg - 1) * seg);
    for (int s = a.nseg - 1; s >= 0; --s) {
        const int kA = s == 0 ? 0 : k0 + s * seg;
        const int kB = min(k0 + (s + 1) * seg, K);
        const int pb = window(s, kA), p = pb + l;
        const int eA = (kA + W) & 1;
        // cell of anti-diagonal k, parity e: i = (k + W - e) / 2 - p and
        // j = (k - W + e) / 2 + p
        const int iA = (kA + W - eA) / 2 - pb - 31, jA = (kA - W + eA) / 2 + pb;
        // E1 / E0: the newest anti-diagonals of parity 1 / 0; H1 / H0 the moves
        float E0, E1;
        const float *qp, *sp;
        __syncwarp();  // the previous segment's samples are read
        if (s == 0) {
            const float org = p == (W >> 1) ? 0.f : CDTW_INF;  // D[-1][-1] = 0 at k = -2
            E0 = e0 == 0 ? org : CDTW_INF;
            E1 = e0 == 0 ? CDTW_INF : org;
            for (int u = l; u < kSpan; u += 32) {
                qw[u] = edge_sample(sq, iA + u, L);
                sw[u] = edge_sample(ss, jA + u, L);
            }
            qp = qw + 31 - l;
            sp = sw + l;
        } else {
            // a path moves at most a.seg + 1 diagonals per segment, so this
            // window starts within 16 slots of the one before
            const int o = pb - pa + l;  // 0 .. 63
            const float a0 = __shfl_sync(kFull, cA[0], o & 31), a1 = __shfl_sync(kFull, cA[1], o & 31);
            const float b0 = __shfl_sync(kFull, cB[0], o & 31), b1 = __shfl_sync(kFull, cB[1], o & 31);
            E0 = o < 32 ? a0 : a1;
            E1 = o < 32 ? b0 : b1;
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                qw[32 * v + l] = xq[v];
                sw[32 * v + l] = xs[v];
            }
            qp = qw + (iA - ia) + 31 - l;
            sp = sw + (jA - ja) + l;
            if (s > 1) ahead(s - 1, pb - 16, kA - seg);
        }
        __syncwarp();
        // moves: 3 diagonal, 2 up (i-1, j), 0 left
        unsigned H0 = 0, H1 = 0;
        const float lim = p == W || p < 0 ? CDTW_INF : -CDTW_INF;
        float qv = qp[0], sv = sp[0];
        auto cost = [&](float m) {
            const float df = __fsub_rn(qv, sv);
            return EU ? __fmaf_rn(df, df, m) : __fadd_rn(fabsf(df), m);
        };
        auto even = [&]() {
            const float left = __shfl_up_sync(kFull, E1, 1);
            const unsigned hl = __shfl_up_sync(kFull, H1 * 4u, 1);
            const float m = min3f(E0, E1, left);
            const unsigned h = E1 <= left ? H1 * 4u + 2u : hl;
            H0 = E0 == m ? H0 * 4u + 3u : h;
            E0 = cost(m);
        };
        auto odd = [&]() {
            const float up = __shfl_down_sync(kFull, E0, 1);
            const unsigned hu = __shfl_down_sync(kFull, H0 * 4u + 2u, 1);
            const float m = min3f(E1, up, E0);
            const unsigned h = up <= E0 ? hu : H0 * 4u;
            H1 = E1 == m ? H1 * 4u + 3u : h;
            E1 = fmaxf(cost(m), lim);  // d = W + 1 lies outside the band
        };
        // the lower half, then, if the path enters above it, the upper one
        const int T = min(kB, kw + 1) - kA;
        int t = 0;
        if (eA == 0) {  // the first segment of an even band starts on parity 0
            if (T > 0) even();
            t = 1;
            sv = sp[1];  // j advances towards parity 1, i towards parity 0
            ++sp;
        }
        auto rows = [&](int end) {
            for (; t + 2 <= end; t += 2) {
                odd();
                qv = *++qp;
                even();
                sv = *++sp;
            }
        };
        rows(min(T, kHalf));
        unsigned L0 = 0, L1 = 0;  // the lower half's moves
        const bool upper = t + 2 <= T || (t < T && t >= kHalf - 1);
        const int kH = kA + t;  // first anti-diagonal of the upper half
        if (upper) {
            L0 = H0;
            L1 = H1;
            H0 = H1 = 0;
            rows(T);
        }
        if (t < T) odd();
        auto at_entry = [&](unsigned h0, unsigned h1) {
            return __shfl_sync(kFull, ((kw + W) & 1) ? h1 : h0, min(max(pw - pb, 0), 31));
        };
        if (upper) {
            follow(at_entry(H0, H1), kH);
            if (kw >= kA) follow(at_entry(L0, L1), kA);
        } else {
            follow(at_entry(H0, H1), kA);
        }
    }
}

using PairFwdK = void (*)(const PairArgs);

// dm 2 (shared record) is instantiated for C <= 4 only: the host selects it
// for records of at most 512 bytes per lane, which needs C <= 4.  dm 3 (the
// checkpointed forward) and dm 4 (its path recovery) for C >= 2: the host
// selects them only for pairs outside shared-record mode; wider lanes (C > 4)
// recover the path by pair_corridor_kernel.
template <int C>
PairFwdK pick_fwd(bool eu, int dm) {
    if constexpr (C <= 4) {
        if (dm == 2) return eu ? pair_fwd_kernel<C, true, 2> : pair_fwd_kernel<C, false, 2>;
    }
    if constexpr (C >= 2) {
        if (dm == 3) return eu ? pair_fwd_kernel<C, true, 3> : pair_fwd_kernel<C, false, 3>;
        if (dm == 5) return eu ? pair_fwd_kernel<C, true, 5> : pair_fwd_kernel<C, false, 5>;
    }
    if constexpr (C >= 2 && C <= 4) {
        if (dm == 4) return eu ? pair_ckpt_walk_kernel<C, true> : pair_ckpt_walk_kernel<C, false>;
    }
    if (eu) return dm ? pair_fwd_kernel<C, true, 1> : pair_fwd_kernel<C, true, 0>;
    return dm ? pair_fwd_kernel<C, false, 1> : pair_fwd_kernel<C, false, 0>;
}

}  // namespace

// Forward kernels by lane width C, instantiated in pair_part0..3.cu (C 1-4,
// 5-8, 9-12, 13-16) for a parallel build.
PairFwdK pair_fwd_part0(int C, bool eu, int dm);
PairFwdK pair_fwd_part1(int C, bool eu, int dm);
PairFwdK pair_fwd_part2(int C, bool eu, int dm);
PairFwdK pair_fwd_part3(int C, bool eu, int dm);

}  // namespace cdtw

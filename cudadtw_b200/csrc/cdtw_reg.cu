// Launchers and kernel choice of the register-band cDTW; the device code and
// its description are in cdtw_reg.cuh.
#include "cdtw_reg.cuh"

namespace cdtw {

namespace {

struct RegKernels {
    RegKernel eu[kMaxRegW + 1];
    RegKernel mh[kMaxRegW + 1];
    RegSearchKernel seu[kMaxRegW + 1];
    RegSearchKernel smh[kMaxRegW + 1];
    RegKernel eun[kMaxReg2W + 1];  // several windows per thread
    RegKernel mhn[kMaxReg2W + 1];
    RegCKernel euc[kMaxRegW + 1];  // consecutive windows, all of them
    RegCKernel mhc[kMaxRegW + 1];
    RegKernels() {
        void** a = (void**)eu;
        void** b = (void**)mh;
        void** c = (void**)seu;
        void** d = (void**)smh;
        reg_fill_part0(a, b, c, d);
        reg_fill_part1(a, b, c, d);
        reg_fill_part2(a, b, c, d);
        reg_fill_part3(a, b, c, d);
        reg_fill_part4(a, b, c, d);
        reg_fill_part5(a, b, c, d);
        reg_fill_part6(a, b, c, d);
        reg_fill_part7(a, b, c, d);
        regn_fill_part0((void**)eun, (void**)mhn);
        regc_fill_part0((void**)euc, (void**)mhc);
        regc_fill_part1((void**)euc, (void**)mhc);
        regc_fill_part2((void**)euc, (void**)mhc);
        regc_fill_part3((void**)euc, (void**)mhc);
        regc_fill_part4((void**)euc, (void**)mhc);
        regc_fill_part5((void**)euc, (void**)mhc);
    }
};

const RegKernels& reg_kernels() {
    static RegKernels k;
    return k;
}

}  // namespace

int choose_variant(cdtw_handle h, int W) {
    int v = (W >= 0 && W < CDTW_MAX_QUERY) ? h->band_variant[W] : 0;
    int G, B;
    const bool lane = lane_shape(W, &G, &B) && h->q.lq >= lane_qpad_min(h->q.M, W);
    if (v == CDTW_VARIANT_REGISTER && W > kMaxRegW) v = 0;
    if (v == CDTW_VARIANT_STRIP16 && W < 15) v = 0;
    if (v == CDTW_VARIANT_STRIP32 && W < 31) v = 0;
    if (v == CDTW_VARIANT_LANE && !lane) v = 0;
    if (v == 0)
        v = (W <= kMaxRegW) ? CDTW_VARIANT_REGISTER
                            : (lane ? CDTW_VARIANT_LANE : CDTW_VARIANT_STRIP16);
    return v;
}

// Bands that both the register band and the lane groups take, whose windows
// take the lanes less time each: few of them are faster there.
static bool few_on_lanes(cdtw_handle h, int W, int64_t windows, int64_t few) {
    constexpr int kLaneMinW = 96;
    int G, B;
    return W > kLaneMinW && windows <= few && h->band_variant[W] == CDTW_VARIANT_AUTO &&
           lane_shape(W, &G, &B) && h->q.lq >= lane_qpad_min(h->q.M, W);
}

// Candidates of a search up to which the lane groups are the faster (M = 1000,
// W = 100: 9827 survivors of 300k windows 800 us on the register band and 460 on
// lane groups, 32k windows 1060 and 1000, 262k 2800 and 4100).
constexpr int kLaneCandidates = 1 << 15;

int search_variant(cdtw_handle h, int W, int64_t Nw) {
    const int v = choose_variant(h, W);
    return v == CDTW_VARIANT_REGISTER && few_on_lanes(h, W, Nw, kLaneCandidates)
               ? CDTW_VARIANT_LANE
               : v;
}

// The kernel of L listed windows, or of all L of them: the lane groups as long
// as they need no more than a block an SM, two for the widest bands.  M = 1024,
// us on the register band / lane groups, all windows (148 SMs: a block each up
// to 9472 windows):
//   windows  9000         10000        18000        19500         41000
//   W = 97   495 / 401    494 / 608    505 / 606    790 / 941     1551 / 1492
//   W = 102  591 / 435    592 / 638    619 / 640    841 / 1001    1656 / 1577
//   W = 106  713 / 466    716 / 713    767 / 714    900 / 1102    1779 / 1746
// (at 41000 the register band starts its second wave; M = 300 has it faster
// there, 395 / 531.)
static int windows_variant(cdtw_handle h, int W, int64_t L) {
    constexpr int kTwoBlocksW = 105;
    const int v = choose_variant(h, W);
    const int64_t few =
        (int64_t)h->sm_count * lane_block_windows(W) * (W >= kTwoBlocksW ? 2 : 1);
    return v == CDTW_VARIANT_REGISTER && few_on_lanes(h, W, L, few) ? CDTW_VARIANT_LANE : v;
}

int launch_cdtw_strip_search(cdtw_handle h, const float* x, int64_t N, const double* mu,
                             const float* sigma, const Cand* cands, const int* count, int* work,
                             int max_count, bool euclid, int R, unsigned long long* key,
                             const HitSink& sink);

int launch_cdtw_search(cdtw_handle h, const float* x, int64_t N, const double* mu,
                       const float* sigma, const Cand* cands, const int* count, int* work,
                       int max_count, bool euclid, unsigned long long* key,
                       const HitSink& sink) {
    const QueryPack& q = h->q;
    if (max_count <= 0) return CDTW_OK;
    const int variant = search_variant(h, q.W, N - q.M + 1);
    if (variant == CDTW_VARIANT_LANE)
        return launch_cdtw_lane_search(h, x, N, mu, sigma, cands, count, work, max_count, euclid,
                                       key, sink);
    if (variant != CDTW_VARIANT_REGISTER)
        return launch_cdtw_strip_search(h, x, N, mu, sigma, cands, count, work, max_count,
                                        euclid, variant == CDTW_VARIANT_STRIP16 ? 16 : 32, key,
                                        sink);
    // their number is known on the device only: both are launched, each returns
    // at once where the other takes them
    int gate = -1;
    if (few_on_lanes(h, q.W, 0, 0)) {
        gate = kLaneCandidates;
        CDTW_TRY(launch_cdtw_lane_search(h, x, N, mu, sigma, cands, count, work,
                                         std::min(max_count, gate), euclid, key, sink, gate));
    }
    RegSearchKernel k = euclid ? reg_kernels().seu[q.W] : reg_kernels().smh[q.W];
    const int lq4 = q.lq / 4;
    const size_t smem = (size_t)q.lq * sizeof(float) + (size_t)reg_env_len(q.M) * sizeof(float2);
    CDTW_TRY(allow_smem(h, (const void*)k, smem));
    int per_sm = 0;
    CDTW_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k, kRegBlock,
                                                               smem));
    const int64_t want = div_up(max_count, kRegBlock);
    const unsigned blocks = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>(want, (int64_t)std::max(per_sm, 1) * h->sm_count));
    k<<<blocks, kRegBlock, smem, h->stream>>>(x, mu, sigma, (const float4*)q.qpad, lq4, q.env,
                                              q.M, cands, count, work, key, sink, h->sm_count,
                                              gate);
    CDTW_LAUNCH(h, "cdtw_reg_search_kernel");
    return CDTW_OK;
}

int launch_cdtw_windows(cdtw_handle h, const float* x, int64_t N, const double* mu,
                        const float* sigma, const int32_t* idx, int64_t L, bool euclid,
                        float* out) {
    const QueryPack& q = h->q;
    const int Nw = (int)(N - q.M + 1);
    const int variant = q.qrev ? windows_variant(h, q.W, L) : CDTW_VARIANT_REGISTER;
    if (variant == CDTW_VARIANT_LANE)
        return launch_cdtw_lane(h, x, N, mu, sigma, idx, L, euclid, out);
    if (variant != CDTW_VARIANT_REGISTER || q.W > kMaxRegW) {
        if (!q.qrev)
            return set_error(h, CDTW_EUNSUPPORTED, "band W=%d above the register-band limit %d",
                             q.W, kMaxRegW);
        return launch_cdtw_strip(h, x, N, mu, sigma, idx, L, euclid,
                                 variant == CDTW_VARIANT_STRIP16 ? 16 : 32, out);
    }
    if (L <= 0) return CDTW_OK;
    const int lq4 = q.lq / 4;
    const size_t smem = (size_t)q.lq * sizeof(float);
    auto prepare = [&](const void* k) -> int {
        CDTW_TRY(allow_smem(h, k, smem));
        return CDTW_OK;
    };
    if (!idx && L == Nw) {
        // every window: the consecutive-window kernels (one sliding run of
        // the stream per thread)
        RegCKernel kc = euclid ? reg_kernels().euc[q.W] : reg_kernels().mhc[q.W];
        CDTW_TRY(prepare((const void*)kc));
        const unsigned blocks = (unsigned)div_up(div_up(L, reg_per_thread(q.W)), kRegBlock);
        kc<<<blocks, kRegBlock, smem, h->stream>>>(x, mu, sigma, (const float4*)q.qpad, lq4, q.M,
                                                   Nw, out);
        CDTW_LAUNCH(h, "cdtw_regc_kernel");
        return CDTW_OK;
    }
    // listed windows: several per thread when that still gives every scheduler
    // a warp, else one, in blocks of a warp
    const int per = reg_per_thread(q.W);
    const bool many = per > 1 && L >= (int64_t)per * 128 * h->sm_count;
    RegKernel k = many ? (euclid ? reg_kernels().eun[q.W] : reg_kernels().mhn[q.W])
                       : (euclid ? reg_kernels().eu[q.W] : reg_kernels().mh[q.W]);
    CDTW_TRY(prepare((const void*)k));
    const int threads = L >= (int64_t)128 * h->sm_count ? kRegBlock : 32;
    const unsigned blocks = (unsigned)div_up(div_up(L, many ? per : 1), threads);
    k<<<blocks, threads, smem, h->stream>>>(x, mu, sigma, (const float4*)q.qpad, lq4, q.M, Nw,
                                            idx, (int)L, out);
    CDTW_LAUNCH(h, "cdtw_reg_kernel");
    return CDTW_OK;
}

}  // namespace cdtw

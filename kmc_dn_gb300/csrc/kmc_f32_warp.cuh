// kmc_f32_warp.cuh -- the batched FP32 hop loop for chains run by a slice of a
// warp: G = 4, 8, 16 or 32 lanes per chain, 32/G chains side by side.
//
// The chains of a warp go through the hop's phases together and every warp
// collective names all 32 lanes: a collective whose member mask differs
// between the halves of a warp runs once per half (measured: ballot 165
// cycles against 28, redux 175 against 23).  A chain that has ended takes
// part with no pairs and no sites.  Loop ends, re-anchors, host polls and the
// draw of new uniforms are found once for up to G hops at a time.  4096 N=30
// chains (G = 16), 10240 hops: 32.6 ms, 39.1 with per-slice masks; a hop's
// scan 499 cycles (1077), uniforms 41 (288), loop checks 132 (285).
#pragma once
#include "kmc_f32_engine.cuh"

namespace kmc {
namespace {

constexpr unsigned kAll = 0xffffffffu;

// A slice of PL lanes; collectives run for all slices of the warp at once.
template <int PL>
struct Slice {
    static constexpr int kSlices = 32 / PL;
    int g;      // lane within the slice
    int sub;    // slice within the warp
    __device__ __forceinline__ void init()
    {
        const int lane = threadIdx.x & 31;
        sub = lane / PL;
        g = lane % PL;
    }
    __device__ __forceinline__ unsigned bits(bool p) const
    {
        const unsigned b = __ballot_sync(kAll, p);
        return PL == 32 ? b : (b >> (sub * PL)) & ((1u << (PL & 31)) - 1u);
    }
    // lowest / highest lane of the slice with p true, or -1
    __device__ __forceinline__ int first(bool p) const { return __ffs(static_cast<int>(bits(p))) - 1; }
    __device__ __forceinline__ int last(bool p) const { return 31 - __clz(static_cast<int>(bits(p))); }
    template <typename V>
    __device__ __forceinline__ V bcast(V v, int src) const { return __shfl_sync(kAll, v, src, PL); }
    __device__ __forceinline__ uint32_t max_u32(uint32_t v) const
    {
        if constexpr (PL == 32) {
            return __reduce_max_sync(kAll, v);
        } else if constexpr (PL >= 8) {
            // one warp-wide reduction a slice (they overlap)
            uint32_t m = 0;
#pragma unroll
            for (int k = 0; k < kSlices; ++k) {
                const uint32_t w = __reduce_max_sync(kAll, sub == k ? v : 0u);
                if (sub == k) m = w;
            }
            return m;
        } else {
#pragma unroll
            for (int d = PL / 2; d >= 1; d >>= 1) v = max(v, __shfl_xor_sync(kAll, v, d, PL));
            return v;
        }
    }
    // inclusive scans over the slice
    __device__ __forceinline__ float scanf(float x) const
    {
#pragma unroll
        for (int d = 1; d < PL; d <<= 1) {
            const float o = __shfl_up_sync(kAll, x, d, PL);
            if (g >= d) x += o;
        }
        return x;
    }
    __device__ __forceinline__ uint64_t scan_u64(uint64_t x) const
    {
#pragma unroll
        for (int d = 1; d < PL; d <<= 1) {
            const uint64_t o = __shfl_up_sync(kAll, x, d, PL);
            if (g >= d) x += o;
        }
        return x;
    }
};

// kLean: the 80-register kernel, whose list rebuild takes one site a step
// (two or four spill).
template <int G, typename Pairs, bool kLean>
__device__ void run_warp(const kmc_batch &B, const Slice<G> &sl, ChainSmem<typename Pairs::Rec> sm, int c,
                         const float2 *shared_tab)
{
    static_assert(!Pairs::kPairedTgt, "plain target records");
    constexpr int kLogG = FixShift<G>::kLog;
    constexpr int RS = RateStride<G>::kValue;   // row stride of the stored running sums
    using Rec = typename Pairs::Rec;
    const int g = sl.g;
    bool ok = c >= 0;
    const int t_id = ok ? B.chain_tab[c] : 0;
    int N = ok ? B.tab_N[t_id] : 0, P = ok ? B.tab_P[t_id] : 0;
    if (ok && (P > kMaxElectrodes || N + P > B.max_sites || N < 0 ||
               (Pairs::kUniformTable && !(B.chain_kT[c] == B.uniform_kT)))) {
        // sizes beyond the launch's, or a table staged for another temperature
        if (g == 0) B.status[c] = KMC_ERR_INVALID;
        ok = false;
    }
    if (!ok) N = P = 0;
    const int S = N + P;
    Pairs pairs{};
    if (ok) pairs.init(B, t_id, S, shared_tab);
    const int64_t so = ok ? B.chain_site_off[c] : 0;
    const int64_t eoff = ok ? B.chain_el_off[c] : 0;
    const float *Ec = B.E_constant + so;
    const float *Vel = B.el_energy + eoff;
    uint8_t *occ_g = B.occupation + so;
    const float cs = ok ? kLog2e / B.chain_kT[c] : 0.0f;
    const int64_t hops_done0 = ok ? B.hops_done[c] : 0;
    int64_t todo = ok ? B.hops_total[c] - hops_done0 : 0;
    if (todo > B.max_hops_per_launch) todo = B.max_hops_per_launch;
    const uint64_t stream = ok ? B.stream[c] : 0;
    const uint32_t k0 = static_cast<uint32_t>(B.seed), k1 = static_cast<uint32_t>(B.seed >> 32);
    const int record = B.record;
    const int reanchor = B.reanchor > 0 ? B.reanchor : 1024;
    const int W = (N + 31) / 32;
    // the buffer of a launch that has one takes the running sums of every
    // state (rate_buffer_words): all chains of the launch keep them, or none
    const bool stored = sm.rate_words > 0;

    // ---- load state ----
    for (int w = g; w < W; w += G) {
        uint32_t bits = 0;
        for (int b = 0; b < 32; ++b) {
            const int j = w * 32 + b;
            if (j < N && occ_g[j]) bits |= 1u << b;
        }
        sm.occw[w] = bits;
    }
    for (int e = g; e < P; e += G) sm.eo[e] = 0;
    __syncwarp();
    int h = 0;
    for (int w = 0; w < W; ++w) h += __popc(sm.occw[w]);

    double t = ok ? B.time[c] : 0.0;   // the clock: FP64
    int64_t hop = hops_done0;
#ifdef KMC_DEBUG_CHECKS
    int dbg_bad = 0;
#endif
    const uint64_t t_launch = B.time_budget_ns > 0 ? globaltimer_ns() : 0;
    const int64_t hop_end = hops_done0 + (todo > 0 ? todo : 0);
    int status = KMC_OK;
    unsigned long long npairs = 0;
    const double *replay = B.replay && ok ? B.replay + B.replay_off[c] : nullptr;
    double *occ_time = record ? B.occ_time + so : nullptr;
    double *occ_since = record ? B.occ_since + so : nullptr;
    int32_t *traffic = record && ok ? B.traffic + B.chain_pair_off[c] : nullptr;
    if (record)
        for (int j = g; j < N; j += G) occ_since[j] = t;

    // Energies carry one rounding per increment: these networks are small and
    // drift ~1e-3 kT between re-anchors (block groups compensate; that cost
    // 2.5 % of the N=30 ensemble's throughput here).
    float drift_max = 0.0f;
    Rec el_rec{};
    auto anchor_and_build = [&](bool mine, bool drift) {
        const int n = mine ? N : 0;
        for (int j = g; j < n; j += G) {
            float e = Ec[j];
            for (int k = 0; k < N; ++k)
                if (!((sm.occw[k >> 5] >> (k & 31)) & 1u)) e -= pairs.coulomb(j, k);
            if (drift) drift_max = fmaxf(drift_max, fabsf(e - sm.E[j]));
            sm.E[j] = e;
        }
        const int z = N - h;
        int wcur = 0, cum = 0;
        for (int j = g; j < n; j += G) {
            const int w = j >> 5;
            while (wcur < w) { cum += __popc(sm.occw[wcur]); ++wcur; }
            const uint32_t word = sm.occw[w];
            const int below = cum + __popc(word & ((1u << (j & 31)) - 1u));
            const Rec r = pairs.rec(j, cs * sm.E[j]);
            if ((word >> (j & 31)) & 1u) {
                sm.src[below] = r;
                if (!Pairs::kSiteInRec) sm.src_id[below] = j;
            } else {
                sm.tgt[j - below] = r;
                if (!Pairs::kSiteInRec) sm.tgt_id[j - below] = j;
            }
        }
        if (mine)
            for (int e = g; e < P; e += G) {
                const Rec r = pairs.rec(N + e, cs * Vel[e]);
                if (e == g) el_rec = r;   // kept for the list rebuilds of later hops
                sm.src[h + e] = r;
                sm.tgt[z + e] = r;
                if (!Pairs::kSiteInRec) {
                    sm.src_id[h + e] = N + e;
                    sm.tgt_id[z + e] = N + e;
                }
            }
        __syncwarp();
    };
    anchor_and_build(ok, false);
    int until_anchor = reanchor - static_cast<int>(hop % reanchor);
    const bool polls = B.cancel || B.time_budget_ns > 0;
    bool run = ok && hop < hop_end;

#ifdef KMC_SECTION_CLOCKS
    uint32_t sec_cycles[kSections] = {};
    uint32_t sec_last = static_cast<uint32_t>(clock());
#endif
    while (__any_sync(kAll, run)) {
        if (polls) {
            // the host's cancel word, then the launch's wall-clock budget
            const bool due = run && (hop & 1023) == 0 && (B.cancel || hop != hops_done0);
            if (__any_sync(kAll, due)) {
                int stop = 0;
                if (due && g == 0) {
                    if (B.cancel && *B.cancel) stop = KMC_ERR_CANCELLED;
                    else if (B.time_budget_ns > 0 && hop != hops_done0 &&
                             static_cast<int64_t>(globaltimer_ns() - t_launch) > B.time_budget_ns)
                        stop = KMC_ERR_TIMEOUT;
                }
                stop = sl.bcast(stop, 0);
                if (due && stop) { status = stop; run = false; }
            }
        }
        const bool anchor = run && until_anchor == 0;
        if (__any_sync(kAll, anchor)) {
            __syncwarp();      // the last hop's bits are visible: a vote orders no memory
            anchor_and_build(anchor, B.energy_drift != nullptr);
            if (anchor) until_anchor = reanchor;
        }
        // hops before any chain of the warp ends, re-anchors, polls or needs
        // new draws
        int steps = G;
        if (run) {
            steps = min(steps, until_anchor);
            if (hop_end - hop < steps) steps = static_cast<int>(hop_end - hop);
            if (polls) steps = min(steps, 1024 - static_cast<int>(hop & 1023));
        }
        if (G < 32) steps = __reduce_min_sync(kAll, steps);
        // lane g draws (and maps) the uniforms of hop + g
        float rnd_e1 = 0.0f;
        uint64_t rnd_u = 0;
        if (replay) {
            if (run && g < steps) {
                rnd_e1 = -log1pf(-static_cast<float>(replay[2 * (hop + g)]));
                rnd_u = u01_fixed_from_double(replay[2 * (hop + g) + 1]);
            }
        } else {
            const uint64_t ctr = static_cast<uint64_t>(hop + g);
            const u32x4 w = philox4x32_10(u32x4{static_cast<uint32_t>(ctr), static_cast<uint32_t>(ctr >> 32),
                                                static_cast<uint32_t>(stream), static_cast<uint32_t>(stream >> 32)},
                                          k0, k1);
            rnd_e1 = -logf(u01_tail32(w.x));
            rnd_u = u01_fixed(w.y, w.z);
        }
        int done = 0;
        for (int step = 0; step < steps; ++step) {
            KMC_SECTION(0);
            // ---- pair phase: the A allowed pairs in G runs of M ----
            const int z = N - h;
            const int T1 = z + P, T2 = z;
            int A1 = h * T1;
            int A = A1 + P * T2;
            if (run && A <= 0) { status = KMC_ERR_NONFINITE; run = false; }
            if (!run) A = A1 = 0;      // no pairs: nothing below touches the lists or the buffer
            const float inv1 = T1 > 0 ? rcp_approx(static_cast<float>(T1)) : 0.0f;
            const float inv2 = T2 > 0 ? rcp_approx(static_cast<float>(T2)) : 0.0f;
            const int M = (A + G - 1) >> kLogG;
            const int kb = min(g * M, A), ke = min(kb + M, A);
            const PairRange range{h, z, P, T1, T2, A1, A, inv1, inv2};
            float lsum = 0.0f;
            if (kb < ke) {
                [[maybe_unused]] const bool in_range =
                    stored ? walk_pairs<true, RS, kPairStep>(pairs, sm.src, sm.tgt, range, kb, ke, cs, sm.rates + g, lsum)
                           : walk_pairs<false, RS, kPairStep>(pairs, sm.src, sm.tgt, range, kb, ke, cs, nullptr, lsum);
                KMC_DCHECK(in_range);
            }
            npairs += static_cast<unsigned>(A);
            KMC_SECTION(1);
            const float e1 = sl.bcast(rnd_e1, step);
            const uint64_t u_ev = sl.bcast(rnd_u, step);
            __syncwarp();      // stored sums visible to the whole slice
            KMC_SECTION(2);
            // ---- exact fixed-point scan of the runs' sums: the event is the
            // first pair whose cumulative rate reaches u*total ----
            Selection sel;
            {
                constexpr int kShift = FixShift<G>::kShift;
                bool good = sel.scale(sl.max_u32(__float_as_uint(lsum)));
                const uint64_t own = to_fixed(lsum, sel.emax, kShift);
                const uint64_t incl = sl.scan_u64(own);
                const uint64_t tot = sl.bcast(incl, G - 1);
                good = sel.total(tot, kShift) && good;
                if (run && !good) { status = KMC_ERR_NONFINITE; run = false; }
                const uint64_t target = fixed_target(u_ev, tot);
                // (the total reaches the target, so some lane does)
                const int at = max(sl.first(incl >= target), 0);
                sel.L = at;
                // what remains of u*total beyond the runs before L, in FP32
                sel.rem = sl.bcast(from_fixed(target - (incl - own), sel.emax, kShift), at);
            }
            const float totf = sel.totf;
            const int L = sel.L;
            float rem = sel.rem;
            KMC_SECTION(3);
            // ---- find the event inside run L ----
            int chosen = -1, last_pos = -1;
            if (!(rem > 0.0f)) rem = 1.0e-38f;   // first pair with a positive rate
            const int kbL = min(L * M, A), keL = min(kbL + M, A);
            const int len = run ? keL - kbL : 0;
            if (stored) {
                // lane L kept its running sums (element i at i*RS + L): the
                // event is the first that reaches rem
                const float *sums = sm.rates + L;
                int idx = -1;
                if constexpr (G == 32) {
                    // narrow the range 32-fold a round
                    int lo = 0, n = len;
                    bool in = true;
                    while (n > 32) {
                        const int q = (n + 31) >> 5;
                        const float v = sums[(lo + min((g + 1) * q, n) - 1) * RS];
                        const unsigned b = __ballot_sync(kAll, v >= rem);
                        if (!b) { in = false; break; }
                        const int skip = (__ffs(b) - 1) * q;
                        lo += skip;
                        n = min(q, n - skip);
                    }
                    if (in) {
                        const float v = g < n ? sums[(lo + g) * RS] : -1.0f;
                        const unsigned b = __ballot_sync(kAll, v >= rem);
                        if (b) idx = lo + __ffs(b) - 1;
                    }
                } else {
                    // chunks of 2 G elements, both loads issued first; the
                    // sums do not decrease, so the lowest element of the
                    // first chunk with a hit is the event
                    int i0 = 0;
                    do {
                        const int ia = i0 + g, ib = i0 + G + g;
                        const float va = ia < len ? sums[ia * RS] : -1.0f;
                        const float vb = ib < len ? sums[ib * RS] : -1.0f;
                        const unsigned ha = sl.bits(va >= rem), hb = sl.bits(vb >= rem);
                        if (idx < 0) {
                            if (ha) idx = i0 + __ffs(ha) - 1;
                            else if (hb) idx = i0 + G + __ffs(hb) - 1;
                        }
                        i0 += 2 * G;
                    } while (__any_sync(kAll, idx < 0 && i0 < len));
                }
                if (idx >= 0) chosen = kbL + idx;
                const bool beyond = run && idx < 0;
                if (__any_sync(kAll, beyond)) {
                    // rem rounded above the run's total: the run's last pair
                    // with a positive rate
                    int lp = -1;
                    if (beyond)
                        for (int i = g; i < len; i += G)
                            if (sums[i * RS] > (i > 0 ? sums[(i - 1) * RS] : 0.0f)) lp = i;
                    const int ll = static_cast<int>(sl.max_u32(static_cast<uint32_t>(lp + 1))) - 1;
                    if (beyond && ll >= 0) chosen = kbL + ll;
                }
            } else {
                // no stored sums: the run's rates again, G at a time
                int i0 = 0;
                do {
                    float r = 0.0f;
                    if (chosen < 0 && i0 + g < len) {
                        int row, col;
                        decode_pair(kbL + i0 + g, h, A1, T1, T2, inv1, inv2, row, col);
                        r = pairs.rate(sm.src[row], sm.tgt[col], row < h && col < z, cs);
                    }
                    const bool pos = r > 0.0f;
                    const float x = sl.scanf(r);
                    const float tot = sl.bcast(x, G - 1);
                    const int hit = sl.first(pos && x >= rem), lp = sl.last(pos);
                    if (chosen < 0 && i0 < len) {
                        if (hit >= 0) chosen = kbL + i0 + hit;
                        else if (lp >= 0) last_pos = kbL + i0 + lp;
                    }
                    rem -= tot;
                    i0 += G;
                } while (__any_sync(kAll, chosen < 0 && i0 < len));
            }
            if (chosen < 0) chosen = last_pos;
            if (run && chosen < 0) { status = KMC_ERR_NONFINITE; run = false; }
            if (chosen < 0) chosen = 0;
#if defined(KMC_DEBUG_CHECKS)
            if (B.select_mismatch) {
                // the same selection with an FP64 scan and compare over the
                // same FP32 sums: count the hops where it picks another pair
                double x = static_cast<double>(lsum);
                for (int d = 1; d < G; d <<= 1) {
                    const double o = __shfl_up_sync(kAll, x, d, G);
                    if (g >= d) x += o;
                }
                const double dtot = sl.bcast(x, G - 1), dtarget = __ull2double_rn(u_ev) * 0x1.0p-64 * dtot;
                int L64 = sl.first(x >= dtarget);
                if (L64 < 0) L64 = max(sl.last(ke > kb), 0);
                const float rem64 = sl.bcast(static_cast<float>(dtarget - (x - static_cast<double>(lsum))), L64);
                if (run && stored && g == 0) {
                    const int kb64 = min(L64 * M, A), len64 = min(kb64 + M, A) - kb64;
                    const float *s64 = sm.rates + L64;
                    int c64 = -1, lp = -1;
                    for (int i = 0; i < len64; ++i) {
                        const float ri = s64[i * RS];
                        if (c64 < 0 && ri >= (rem64 > 0.0f ? rem64 : 1.0e-38f)) c64 = i;
                        if (ri > (i > 0 ? s64[(i - 1) * RS] : 0.0f)) lp = i;
                    }
                    if (c64 < 0) c64 = lp;
                    if (kb64 + c64 != chosen) B.select_mismatch[c] += 1ull;
                }
            }
            if (run) KMC_DCHECK(chosen < A && L >= 0 && L < G && chosen >= kbL && chosen < keL);
#endif
            int row, col;
            decode_pair(chosen, h, A1, T1, T2, inv1, inv2, row, col);
#ifdef KMC_DEBUG_CHECKS
            if (run) KMC_DCHECK(row >= 0 && row < h + P && col >= 0 && col < (row < h ? T1 : T2));
            if (sl.first(dbg_bad != 0) >= 0 && run) { status = KMC_ERR_INVALID; run = false; }
            if (!run) row = col = 0;
#endif
            const int from = Pairs::kSiteInRec ? Pairs::site(sm.src[row]) : sm.src_id[row];
            const int to = Pairs::kSiteInRec ? Pairs::site(sm.tgt[col]) : sm.tgt_id[col];
#ifdef KMC_DEBUG_CHECKS
            if (run) KMC_DCHECK(from >= 0 && from < S && to >= 0 && to < S && from != to && (from < N || to < N));
            if (sl.first(dbg_bad != 0) >= 0 && run) { status = KMC_ERR_INVALID; run = false; }
#endif
            if (B.hop_log && run && g == 0) {
                const int64_t li = B.hop_log_off[c] + hop + step;
                B.hop_log[2 * li] = from;
                B.hop_log[2 * li + 1] = to;
                if (B.hop_rates) {
                    B.hop_rates[2 * li] = totf;
                    B.hop_rates[2 * li + 1] = pairs.rate(sm.src[row], sm.tgt[col], row < h && col < z, cs);
                }
            }
            KMC_SECTION(4);
            // (record: when the hole that leaves came, read while the lists are
            // rebuilt)
            double since = 0.0;
            if (record && run && g == 0 && from < N) since = occ_since[from];
            // ---- clock ----
            const float dt = e1 * rcp_approx(totf);
            const double t_before = t;
            if (run) t += widen(dt);
            if (B.flux_time) {
                // Expected net hole flow into each electrode in this state
                // times the time spent in it (run_chain has the reasons).
                for (int e = 0; __any_sync(kAll, run && e < P); ++e) {
                    const bool mine = run && e < P;
                    Rec er{};
                    if (mine) er = sm.src[h + e];
                    float J = 0.0f;
                    if (mine)
                        for (int k = g; k < N; k += G)
                            J += (k < h) ? pairs.rate(sm.src[k], er, false, cs)
                                         : -pairs.rate(er, sm.tgt[k - h], false, cs);
#pragma unroll
                    for (int d = G / 2; d >= 1; d >>= 1) J += __shfl_xor_sync(kAll, J, d, G);
                    if (mine && g == 0) B.flux_time[eoff + e] += static_cast<double>(J) * static_cast<double>(dt);
                }
            }
            __syncwarp();   // every lane is done reading the lists and rates
            KMC_SECTION(5);
            // ---- apply the hop and rebuild the lists in one pass ----
            const bool fa = from < N, tb = to < N;
            const int h_new = h + (tb ? 1 : 0) - (fa ? 1 : 0);
            const int z_new = N - h_new;
            if (run) {
                // tables read from L2: as many sites a step as the slice has,
                // up to four a lane (rebuild_sites)
                constexpr bool kMany = Pairs::kFarTable && !kLean;
                constexpr int kTwo = kMany ? 2 : 1, kFour = kMany ? 4 : 1;
                [[maybe_unused]] const int reb =
                    kFour > 1 && N > 2 * G ? rebuild_sites<G, kFour, false>(pairs, sm, g, N, cs, from, to, h_new)
                    : kTwo > 1 && N > G    ? rebuild_sites<G, kTwo, false>(pairs, sm, g, N, cs, from, to, h_new)
                                           : rebuild_sites<G, 1, false>(pairs, sm, g, N, cs, from, to, h_new);
#ifdef KMC_DEBUG_CHECKS
                dbg_bad |= reb;
#endif
                if (h_new != h) {
                    for (int e = g; e < P; e += G) {
                        const Rec r = (e == g) ? el_rec : pairs.rec(N + e, cs * Vel[e]);
                        sm.src[h_new + e] = r;
                        if (!Pairs::kSiteInRec) sm.src_id[h_new + e] = N + e;
                        sm.tgt[z_new + e] = r;
                        if (!Pairs::kSiteInRec) sm.tgt_id[z_new + e] = N + e;
                    }
                }
            }
            KMC_SECTION(6);
            __syncwarp();   // lists complete; the bitmask is read no more this hop
            if (run) {
                if (g == 0) {
                    if (fa) sm.occw[from >> 5] &= ~(1u << (from & 31));
                    else sm.eo[from - N] -= 1;
                    if (tb) sm.occw[to >> 5] |= 1u << (to & 31);
                    else sm.eo[to - N] += 1;
                    if (record) {
                        // fire and forget: this thread alone updates the chain's
                        // entries, and nothing waits for them
                        atomicAdd(&traffic[from * S + to], 1);
                        if (record == KMC_RECORD_GO) atomicAdd(&traffic[to * S + from], -1);
                        const double tx = (record == KMC_RECORD_GO) ? t : t_before;
                        if (fa) atomicAdd(&occ_time[from], tx - since);
                        if (tb) occ_since[to] = tx;
                    }
                }
                h = h_new;
                ++done;
            }
            KMC_SECTION(7);
#ifdef KMC_DEBUG_CHECKS
            if (sl.first(dbg_bad != 0) >= 0 && run) { status = KMC_ERR_INVALID; run = false; }
#endif
        }
        hop += done;
        until_anchor -= done;
        if (hop >= hop_end) run = false;
    }
    __syncwarp();

#ifdef KMC_SECTION_CLOCKS
    if (g == 0 && ok) {
        for (int k = 0; k < kSections; ++k) atomicAdd(&g_section_clocks[k], static_cast<unsigned long long>(sec_cycles[k]));
        atomicAdd(&g_section_clocks[kSections], static_cast<unsigned long long>(hop - hops_done0));
    }
#endif
    // ---- write back ----
    const float dm = B.energy_drift
                         ? __uint_as_float(sl.max_u32(__float_as_uint(drift_max * (cs / kLog2e)))) : 0.0f;
    if (!ok) return;
    if (record) {
        for (int j = g; j < N; j += G)
            if ((sm.occw[j >> 5] >> (j & 31)) & 1u) {
                occ_time[j] += t - occ_since[j];
                occ_since[j] = t;
            }
    }
    for (int j = g; j < N; j += G) occ_g[j] = static_cast<uint8_t>((sm.occw[j >> 5] >> (j & 31)) & 1u);
    for (int e = g; e < P; e += G) B.electrode_occupation[eoff + e] += sm.eo[e];
    if (g == 0) {
        // largest drift of the chain, in kT
        if (B.energy_drift) B.energy_drift[c] = fmaxf(B.energy_drift[c], dm);
        B.time[c] = t;
        B.hops_done[c] = hop;
        B.status[c] = status;
        if (B.n_pairs) B.n_pairs[c] += npairs;
    }
}

// Stage the one pair table of a launch whose chains all have kT = kT_u as
// (L, fma(c, B, L)) pairs followed by the B values, c = log2(e)/kT_u.
__device__ __forceinline__ const float2 *stage_table_uniform(const kmc_batch &B, uint32_t *smem, int table_words)
{
    if (table_words <= 0) return nullptr;
    const int S = B.tab_N[0] + B.tab_P[0];
    if (S > B.max_sites) return nullptr;   // invalid launch: chains report it
    const float cu = kLog2e / B.uniform_kT;
    const float2 *src = reinterpret_cast<const float2 *>(B.tab_LB + B.tab_off[0]);
    float2 *dst = reinterpret_cast<float2 *>(smem);
    float *bdst = reinterpret_cast<float *>(dst + S * S);
    for (int i = threadIdx.x; i < S * S; i += blockDim.x) {
        const float2 lb = __ldg(&src[i]);
        dst[i] = make_float2(lb.x, fmaf(cu, lb.y, lb.x));
        bdst[i] = lb.y;
    }
    __syncthreads();
    return reinterpret_cast<const float2 *>(smem);
}


// 32/G chains a warp, blockDim.x / 32 warps a block.  Two register budgets:
// MinBlocks = 2 allows 128 registers (two blocks of 256 threads, 16 warps an
// SM), which the pair walk uses without spills; MinBlocks = 3 allows 80 (24
// warps an SM).  4096 N = 100 chains with tables in memory: 31.7 ms in two
// waves at 128 registers, 51 in one and a part at 80 (launch_warp_kernel
// chooses).  table_words > 0: every chain of the launch uses table 0, staged
// in shared memory ahead of the per-chain areas.
template <int G, typename Pairs, int MinBlocks>
__global__ void __launch_bounds__(256, MinBlocks) warp_engine_kernel(const kmc_batch B, int rate_words,
                                                                     int table_words)
{
    constexpr int CPW = 32 / G;
    extern __shared__ __align__(16) uint32_t smem[];
    const float2 *stab = Pairs::kUniformTable ? stage_table_uniform(B, smem, table_words)
                                              : stage_table(B, smem, table_words);
    Slice<G> sl;
    sl.init();
    const int warp = threadIdx.x >> 5;
    using Rec = typename Pairs::Rec;
    const int words = chain_list_words<Rec>(B.max_sites) + rate_words;
    ChainSmem<Rec> sm = carve<Rec>(smem + table_words + (warp * CPW + sl.sub) * words, B.max_sites, rate_words);
    // the chain of this slice in item `item`, -1: none
    auto chain_of = [&](int item) {
        const int c = item < B.n_work ? B.work[item * CPW + sl.sub] : -1;
        return c < B.n_chains ? c : -1;
    };
    if (B.work_counter) {
        // Persistent launch: each warp claims the next unclaimed item when
        // the chains of its last one are done, so a warp whose chains end
        // early takes more work instead of idling until its block ends.  The
        // loop ends for the whole warp at once, when the list is used up.
        for (;;) {
            int item = 0;
            if ((threadIdx.x & 31) == 0) item = atomicAdd(B.work_counter, 1);
            item = __shfl_sync(kAll, item, 0);
            if (item >= B.n_work) break;
            run_warp<G, Pairs, (MinBlocks > 2)>(B, sl, sm, chain_of(item), stab);
            __syncwarp();
        }
        return;
    }
    const int item = blockIdx.x * (blockDim.x >> 5) + warp;
    if (item >= B.n_work) return;      // the whole warp
    run_warp<G, Pairs, (MinBlocks > 2)>(B, sl, sm, chain_of(item), stab);
}

// Whether a launch may take the 80-register kernel.  Not whole warps a chain,
// nor slices of 16 with tables in memory: there its 24 warps an SM are slower
// than two waves of 16 (N = 60, 3648 chains, tables in memory: 22.4 ms against
// 10.4; N = 30 in slices of 16, 6000 chains: 6.8 against 5.9).
template <int G, typename Pairs>
constexpr bool lean_warps()
{
    return G <= (Pairs::kFarTable ? 8 : 16);
}

template <int G, typename Pairs>
int launch_warp_kernel(const kmc_batch &b, cudaStream_t st, size_t smem, int rw, int tw)
{
    const int wpb = b.warps_per_block, sms = sm_count();
    int blocks = (b.n_work + wpb - 1) / wpb;
    if (blocks <= 0) return KMC_OK;
    auto *kernel = warp_engine_kernel<G, Pairs, 2>;
    static int configured_rich = 0;
    int rc = set_smem(kernel, smem, configured_rich);
    if (rc != KMC_OK) return rc;
    const bool crowded = blocks > (16 / wpb) * sms;      // more than the SMs hold at once
    if (b.work_counter || (crowded && lean_warps<G, Pairs>())) {
        int rich = 0, lean = 0;      // resident blocks an SM
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&rich, kernel, wpb * 32, smem);
        if (e != cudaSuccess) return fail_cuda(e, "engine occupancy");
        rich = max(1, rich);
        if (b.work_counter) {
            // persistent: as many blocks as stay resident at once, no more
            // than the work needs
            blocks = min(blocks, rich * sms);
            if (b.max_grid > 0) blocks = min(blocks, b.max_grid);
        } else if constexpr (lean_warps<G, Pairs>()) {
            // The 80-register kernel where its residency saves more waves than
            // its warps are slower: a wave of 24 takes 1/0.6 of one of 16
            // (N = 12 in slices of 8, 12000 chains: 4.5 ms in one wave, 5.3 in
            // two; N = 30 in slices of 16, positions, 6000: 5.5 and 6.1; N =
            // 40, where shared memory holds no more than 16 warps: 10.1 and 8.2).
            static int configured_lean = 0;
            auto *small = warp_engine_kernel<G, Pairs, 3>;
            if ((rc = set_smem(small, smem, configured_lean)) != KMC_OK) return rc;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&lean, small, wpb * 32, smem);
            if (e != cudaSuccess) return fail_cuda(e, "engine occupancy");
            lean = max(1, lean);
            const int q = (blocks + sms - 1) / sms, waves = (q + rich - 1) / rich, waves_lean = (q + lean - 1) / lean;
            if (5 * waves_lean < 3 * waves) kernel = small;
        }
    }
    kernel<<<blocks, wpb * 32, smem, st>>>(b, rw, tw);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KMC_OK : fail_cuda(e, "engine launch");
}

template <int G, typename Pairs>
int preload_warp_kernels()
{
    int rc = touch_kernel(warp_engine_kernel<G, Pairs, 2>);
    if constexpr (lean_warps<G, Pairs>())
        if (rc == KMC_OK) rc = touch_kernel(warp_engine_kernel<G, Pairs, 3>);
    return rc;
}

template <int G, typename Pairs>
int launch_warp(const kmc_batch &b, cudaStream_t st)
{
    constexpr int CPW = 32 / G;
    const int wpb = b.warps_per_block;
    const int lw = chain_list_words<typename Pairs::Rec>(b.max_sites);
    int rw = rate_buffer_words(b.max_sites, G);
    // Pad each chain's area to G words modulo 32: the 32/G chains of a warp
    // then write their rates to disjoint banks.
    if (G < 32) rw += ((G - (lw + rw)) % 32 + 32) % 32;
    if (static_cast<size_t>(wpb) * CPW * (lw + rw) * 4 > kSmemBudget) rw = 0;   // recompute instead
    const size_t chains = static_cast<size_t>(wpb) * CPW * (lw + rw) * 4;
    const int tw = table_stage_words<Pairs>(b, chains);
    const size_t smem = chains + static_cast<size_t>(tw) * 4;
    if (smem > kSmemBudget)
        return fail(KMC_ERR_INVALID, "engine: %zu bytes of shared memory per block (max_sites %d, G %d, %d warps) exceeds the budget",
                    smem, b.max_sites, G, wpb);
    if (tw > 0 && b.uniform_kT > 0.0f) {
        // every chain has kT = uniform_kT: stage (L, L + c B) and B (3 S^2 words)
        const int tw3 = ((3 * b.max_sites * b.max_sites) + 3) & ~3;
        const size_t smem3 = chains + static_cast<size_t>(tw3) * 4;
        if (smem3 <= kSmemBudget && static_cast<size_t>(tw3) * 4 <= 96 * 1024)
            return launch_warp_kernel<G, TablePairs<true, true>>(b, st, smem3, rw, tw3);
    }
    if (tw > 0) return launch_warp_kernel<G, TablePairs<true>>(b, st, smem, rw, tw);
    return launch_warp_kernel<G, Pairs>(b, st, smem, rw, tw);
}

}  // namespace
}  // namespace kmc

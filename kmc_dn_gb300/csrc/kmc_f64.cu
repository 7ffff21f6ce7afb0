// kmc_f64.cu -- plain FP64 hop loop for sm_103a, one thread block per chain.
//
// The semantics of the reference's numba loop _simulate_discrete_record
// (kmc_dopant_networks.py:33-135) in FP64, so that fed the same uniform
// stream it makes the same hop sequence:
//
//   energies   E_i = Ec_i + (-I_0 R) * sum_{j empty} 1/d_ij, summed in
//              ascending j (:59-66); 1/d_ij is tabulated once (the same
//              correctly rounded quotient the loop divides out each hop)
//   rates      tc_ij * (dE > 0 ? nu*exp(-dE/kT) : nu),
//              dE = E_j - E_i - (I_0 R)/d_ij for acceptor pairs (:69-87)
//   cumulative row-major running sum (:91-97)
//   clock      dt = -log(1 - u1) * (1/total) (:100)
//   event      first k with cum_k/total >= u2 (:103-110)
//   record     traffic[from,to] += 1, post-hop occupancy credit (:126-130)
//
// Only the allowed transitions are visited, A(h) = h(N-h) + hP + P(N-h) of
// the S^2 pairs, in the dense loop's row-major order (a forbidden pair has
// rate 0 and leaves every running sum as it is).  Thread g owns M
// consecutive allowed pairs and continues the running sum from the FP64
// prefix of the threads before it.  That prefix is a tree sum, not the
// reference's strictly left-to-right sum, and the exponential is taken as a
// product (below), so cum_k and the total may differ in the last bits: the
// hop sequence is the reference's except where u2 lies within a few ulp of a
// boundary cum_k/total.
//
// What bounds it is the FP64 pipe: a warp instruction holds its SM quarter's
// unit for 64 cycles whatever its neighbours do (64.3 measured for dependent
// and for independent chains; 128 with two warps on a quarter), so the count
// of FP64 instructions is the time.  So:
//   * exp(-dE/kT) is the product exp(E_i/kT) exp(-E_j/kT) exp(I_0R/d_ij/kT):
//     one exponential a site and hop, the third factor tabulated together
//     with tc, and a pair costs two multiplications and an integer minimum
//     against tc*nu instead of two subtractions, a comparison and an
//     exponential.  Mantissa and exponent are kept apart, so no factor can
//     overflow, and no difference of large energies is rounded;
//   * comparisons are integer compares of the bit patterns;
//   * after the warps' scans one warp picks the event while another divides
//     for the clock, and the uniforms' logarithms are taken for 32 hops at
//     once: three block barriers a hop;
//   * four warps, one a quarter of the SM: more would wait for the same pipe.
// One N = 30, P = 8 chain: 4.0 us a hop (18.8 us with S^2 dense rates and
// running sums in global memory, 6.1 us with the pairs' exponentials queued
// 32 at a time); 256 chains of N = 60, P = 8, 300 hops with occupancy and
// flux: 3.8 ms (28.9 ms, 6.6 ms).  Time against the same hop sequences in
// 113-bit arithmetic, rms relative error over 40 networks: N = 30 1.3e-14
// (dense rates 1.4e-14), N = 60 1.96e-13 (1.89e-13): the energies' rounding.
#include <algorithm>
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

#include "kmc_common.cuh"
#include "kmc_exp64.cuh"
#include "kmc_internal.h"

namespace kmc {
namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kDirectHops = 3;     // runs this short build no table of factors (f64_chain)
// A site in a list: exp(+-E/kT) = m 2^k (a source's +, a target's -).
struct __align__(16) Site {
    double m;
    int id;
    int k;
};

// Exact n / T for 0 <= n < 2^22 from inv ~ 1/T: float quotient, one
// correction step.
__device__ __forceinline__ int div_small(int n, int T, float inv, int &rem)
{
    int q = __float2int_rz(__int2float_rn(n) * inv);
    int r = n - q * T;
    if (r < 0) { --q; r += T; } else if (r >= T) { ++q; r -= T; }
    rem = r;
    return q;
}

// Shared memory of one chain.  The three optional parts go to shared memory
// when the launch gives them room (f64_layout), else they stay in the
// caller's arrays and the workspace.
struct Layout {
    int S;                  // sites the lists are sized for
    int tab, rates, invd;   // entries reserved, 0: not in shared memory
};

__host__ __device__ inline size_t layout_bytes(const Layout &l)
{
    return 20 * static_cast<size_t>(l.tab) + 8 * static_cast<size_t>(l.rates + l.invd) + 16 * kExpTable +
           (2 * sizeof(Site) + 2 * 8) * static_cast<size_t>(l.S) + 8 * (kThreads + 64 + 128) + 4 * 64 + 32;
}

// One chain run by the whole block (the body of both kernels below).
// kTab: tc and (I_0 R)/d are read from shared memory; kRate: the rates of a
// hop sit there; kReplay: the uniforms are the caller's (apart, because the
// test for those that Philox does not draw costs 2 % of a run).
template <bool kTab, bool kRate, bool kReplay>
__device__ __forceinline__ void f64_chain(
    const Layout &lay, int N, int P, double nu, double kT, double I0, double R, uint8_t *occ_g, const double *d,
    const double *Ec, const double *se_in, const double *tc, int64_t *eo, int64_t hops,
    int record, double *traffic, double *oit, const double *uniforms, uint64_t seed,
    int32_t *hop_log, double *time_out, int32_t *status_out, double *ws, double *flux_time)
{
    extern __shared__ __align__(16) unsigned char sraw[];
    const int S = N + P;
    double2 *tab = reinterpret_cast<double2 *>(sraw);              // [S*S] tc*nu, mantissa of tc*nu*exp(I_0R/d/kT)
    double2 *exp_tab = tab + lay.tab;                              // [kExpTable]
    Site *src = reinterpret_cast<Site *>(exp_tab + kExpTable);     // [S] holes at 0.., electrode e at N + e
    Site *tgt = src + lay.S;                                       // [S] empty acceptors at 0.., electrodes as there
    double *rate_s = reinterpret_cast<double *>(tgt + lay.S);      // [A] this hop's rates
    double *invd_s = rate_s + lay.rates;                           // [N*N] 1/d_ij at j*N + i
    double *src_e = invd_s + lay.invd;                             // [S] energies of the sources
    double *tgt_e = src_e + lay.S;                                 // [S] energies of the targets
    double *incl = tgt_e + lay.S;                                  // [kThreads] warp-inclusive sums
    double *u_ev = incl + kThreads;                                // [32] event uniforms
    double *u_cl = u_ev + 32;                                      // [32] -log(1 - u1)
    double *sh_J = u_cl + 32;                                      // [64] expected net inflow
    double *sh_fx = sh_J + 64;                                     // [64] its time integral
    int *tab_k = reinterpret_cast<int *>(sh_fx + 64);              // [S*S] exponents beside tab
    uint32_t *occw = reinterpret_cast<uint32_t *>(tab_k + lay.tab);   // [64] occupancy bits
    __shared__ int wide_always, wide_now[2];   // energies or couplings beyond the split exponential
    __shared__ int ev_from, ev_to;
    __shared__ double sh_dt;

    // workspace: mantissas and exponents of the table, 1/d, rates
    const size_t SS = (size_t)S * S;
    double *W_g = ws;
    int *k_g = reinterpret_cast<int *>(ws + SS);
    double *invd_g = ws + SS + (SS + 1) / 2;
    double *rates = kRate ? rate_s : invd_g + (size_t)N * N;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool unit = (kT == 1.0), nu_is_one = (nu == 1.0);
    const double inv_kT = 1.0 / kT;
    const double IR = I0 * R;
    const double mIR = -I0 * R;
    // A run of a few hops evaluates its pairs by the reference's expression:
    // the table's exponentials, one a pair of acceptors, are 38 FP64
    // instructions for N^2 pairs, the expression's 45 for at most N^2/4 + N P a
    // hop (a call of one hop at N = 200: 1.02 ms with the table, 0.73).
    const bool direct = hops <= kDirectHops;
    double *invd = lay.invd > 0 ? invd_s : invd_g;
    for (int j = tid; j < kExpTable; j += kThreads) exp_tab[j] = exp_table_entry(j);
    if (tid == 0) {
        wide_always = direct;
        wide_now[0] = wide_now[1] = 0;
    }
    for (int k = tid; k < N * N; k += kThreads) {
        const int i = k / N, j = k - (k / N) * N;
        const double dij = d[(size_t)i * S + j];
        invd[(size_t)j * N + i] = (i != j) ? 1.0 / dij : 0.0;
    }
    __syncthreads();
    for (int k = tid; k < S * S; k += kThreads) {
        const int i = k / S, j = k - (k / S) * S;
        const double cap = tc[k] * nu;
        double rest, m = 1.0;
        int e = 0;
        if (i < N && j < N && i != j && !direct) {
            const double x = over_kT(IR / d[k], unit, kT, inv_kT, rest);
            if (splittable(x)) m = exp_split(x, rest, exp_tab, e);
            else wide_always = 1;
        }
        // tc*nu in range: keep the factor's exponent apart from it
        if (kTab) {
            tab[k] = make_double2(cap, cap * m);
            tab_k[k] = e;
        } else {
            W_g[k] = cap * m;
            k_g[k] = e;
        }
    }
    const int W = (N + 31) >> 5;
    for (int w = tid; w < W; w += kThreads) {
        uint32_t bits = 0;
        for (int b = 0; b < 32 && w * 32 + b < N; ++b)
            if (occ_g[w * 32 + b]) bits |= 1u << b;
        occw[w] = bits;
    }
    if (flux_time)
        for (int e = tid; e < P; e += kThreads) sh_fx[e] = flux_time[e];
    // the electrodes' list entries, the same every hop
    for (int i = N + tid; i < S; i += kThreads) {
        const double e = se_in[i];
        double rest;
        const double x = over_kT(e, unit, kT, inv_kT, rest);
        src_e[i] = tgt_e[i] = e;
        Site a{1.0, i, 0}, b{1.0, i, 0};
        if (splittable(x)) {
            a.m = exp_split(x, rest, exp_tab, a.k);
            b.m = exp_split(-x, -rest, exp_tab, b.k);
        } else {
            wide_always = 1;
        }
        src[i] = a;
        tgt[i] = b;
    }
    __syncthreads();
    int h = 0;
    for (int w = 0; w < W; ++w) h += __popc(occw[w]);

    double time = 0.0, dt = 0.0;     // (the clock: warp 1)
    // this thread's first site: occupied time and constant energy
    double oit0 = (record && tid < N) ? oit[tid] : 0.0;
    const double Ec0 = tid < N ? Ec[tid] : 0.0;
    int status = KMC_OK;
    int from = S, to = S;      // the last hop, not yet in occw (none before the first)

    for (int64_t hop = 0;; ++hop) {
        // ---- lists of the current state: the last hop applied to the bits ----
        const int wf = from < N ? from >> 5 : -1, wt = to < N ? to >> 5 : -1;
        const uint32_t bf = from < N ? 1u << (from & 31) : 0u, bt = to < N ? 1u << (to & 31) : 0u;
        const int z = N - h;
        for (int i = tid; i < N; i += kThreads) {
            double acc = 0.0, next = 0.0;
            int below = 0, n_empty = 0;
            bool occ_i = false;
            for (int w = 0; w < W; ++w) {
                uint32_t word = occw[w];
                if (w == wf) word &= ~bf;
                if (w == wt) word |= bt;
                const int left = N - w * 32;
                uint32_t empty = ~word & (left >= 32 ? 0xffffffffu : (1u << left) - 1u);
                if ((i >> 5) == w) {
                    below += __popc(word & ((1u << (i & 31)) - 1u));
                    occ_i = (word >> (i & 31)) & 1u;
                } else if ((i >> 5) > w) {
                    below += __popc(word);
                }
                // ascending j, each entry loaded ahead of the add before it
                // (the diagonal entry is 0)
                const double *col = invd + (size_t)w * 32 * N + i;
                while (empty) {
                    const double v = col[(size_t)(__ffs(empty) - 1) * N];
                    empty &= empty - 1;
                    if (n_empty > 1) acc += next;
                    else acc = next;
                    ++n_empty;
                    next = v;
                }
            }
            if (n_empty > 1) acc += next;
            else acc = next;
            double e = i == tid ? Ec0 : Ec[i];
            e += mIR * acc;
            double rest;
            const double y = over_kT(e, unit, kT, inv_kT, rest);
            Site a{1.0, i, 0};
            if (splittable(y)) a.m = exp_split(occ_i ? y : -y, occ_i ? rest : -rest, exp_tab, a.k);
            else wide_now[hop & 1] = 1;
            if (occ_i) {
                src[below] = a;
                src_e[below] = e;
                if (record && hop > 0) {
                    if (i == tid) oit0 += dt;
                    else oit[i] += dt;
                }
            } else {
                tgt[i - below] = a;
                tgt_e[i - below] = e;
            }
        }
        if (hop >= hops) break;
        if ((hop & 31) == 0 && warp == kWarps - 1) {
            // the uniforms of the next 32 hops, mapped
            const int64_t hh = hop + lane;
            double u1 = 0.5, u2 = 0.5;
            if constexpr (kReplay) {
                if (hh < hops) {
                    u1 = uniforms[2 * hh];
                    u2 = uniforms[2 * hh + 1];
                }
            } else {
                const u32x4 r = philox4x32_10(u32x4{static_cast<uint32_t>(hh), static_cast<uint32_t>(hh >> 32), 0u, 0u},
                                              static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32));
                u1 = u01_from64(r.x, r.y);
                u2 = u01_from64(r.z, r.w);
            }
            // (a replay may hold 0; what is not in (0, 1] passes at k = 0, or never)
            if (kReplay && static_cast<unsigned long long>(__double_as_longlong(u2)) - 1ull >= 0x3ff0000000000000ull)
                u2 = NAN;
            u_ev[lane] = u2;
            u_cl[lane] = -log(1.0 - u1);
        }
        __syncthreads();
        const bool wide = wide_always | wide_now[hop & 1];
        if (tid == 0) {      // every thread has read the bits: take the last hop in
            wide_now[(hop + 1) & 1] = 0;
            if (wf >= 0) occw[wf] &= ~bf;
            if (wt >= 0) occw[wt] |= bt;
        }

        // ---- rates of the allowed pairs ----
        const int T1 = z + P, T2 = z;
        const int A1 = h * T1, A = A1 + P * T2;
        const float inv1 = T1 > 0 ? __fdividef(1.0f, static_cast<float>(T1)) : 0.0f;
        const float inv2 = T2 > 0 ? __fdividef(1.0f, static_cast<float>(T2)) : 0.0f;
        const int M = (A + kThreads - 1) / kThreads;      // pairs per thread
        const int kw = warp * 32 * M, kwe = min(kw + 32 * M, A);
        // kAhead rounds of 32 pairs load together
        constexpr int kAhead = 4;
        for (int k0 = kw; k0 < kwe; k0 += 32 * kAhead) {
            double cap[kAhead], g[kAhead];
            int ex[kAhead];
#pragma unroll
            for (int a = 0; a < kAhead; ++a) {
                const int k = k0 + 32 * a + lane;
                cap[a] = g[a] = 0.0;
                ex[a] = 0;
                if (k < kwe) {
                    int row, col;
                    if (k < A1) row = div_small(k, T1, inv1, col);
                    else row = N + div_small(k - A1, T2, inv2, col);
                    if (col >= z) col += N - z;
                    const Site f = src[row], t = tgt[col];
                    const size_t at = (size_t)f.id * S + t.id;
                    double w;
                    if (kTab) {
                        const double2 T = tab[at];
                        cap[a] = T.x;
                        w = T.y;
                        ex[a] = tab_k[at];
                    } else {
                        cap[a] = nu_is_one ? tc[at] : tc[at] * nu;
                        w = W_g[at];
                        ex[a] = k_g[at];
                    }
                    ex[a] += f.k + t.k;
                    g[a] = w * (f.m * t.m);
                    if (wide) {
                        // the reference's expression
                        double dE = tgt_e[col] - src_e[row];
                        if (row < N && col < N) dE -= IR / d[at];
                        g[a] = tc[at] * (dE > 0 ? nu * exp(-dE / kT) : nu);
                        ex[a] = INT_MIN;
                    }
                }
            }
#pragma unroll
            for (int a = 0; a < kAhead; ++a) {
                const int k = k0 + 32 * a + lane;
                if (k < kwe) {
                    const double r = ex[a] == INT_MIN ? g[a] : scaled_min(g[a], ex[a], cap[a]);
                    rates[k] = r;
                }
            }
        }
        __syncwarp();
        const int kb = min(kw + lane * M, kwe), ke = min(kb + M, kwe);
        double lsum = kb < ke ? rates[kb] : 0.0;
        for (int k = kb + 1; k < ke; ++k) lsum += rates[k];
        double x = lsum;
        if (kw < kwe) {
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const double o = __shfl_up_sync(0xffffffffu, x, s);
                if (lane >= s) x += o;
            }
        }
        incl[tid] = x;
        __syncthreads();

        // ---- warp 0: the event; warp 1: the clock; then the flux ----
        if (warp < 2) {
            double upto[kWarps];      // sums up to the end of each warp
            upto[0] = incl[31];
#pragma unroll
            for (int w = 1; w < kWarps; ++w) upto[w] = upto[w - 1] + incl[w * 32 + 31];
            const double total = upto[kWarps - 1];
            if (warp == 1) {
                const double scale = 1.0 / total;
                const double step = u_cl[hop & 31] * scale;
                if (lane == 0) sh_dt = step;
                if (positive(total) && !not_less(total, __double_as_longlong(1.0e300))) time += step;
            } else if (!positive(total) || not_less(total, __double_as_longlong(1.0e300))) {
                if (lane == 0) ev_from = -1;      // zero, negative, infinite or NaN
            } else {
                const double u2 = u_ev[hop & 31];
                // First k with cum_k/total >= u2 (the reference's test).
                // Where cum_k is 2^13 units in the last place or more away
                // from u2*total (over 1e-12 relative, far more than the
                // rounding of either side), the product decides it, else a
                // division.
                const long long ut = __double_as_longlong(u2 * total), lo = ut - 8192, hi = ut + 8192;
                // the first warp, then the first thread, whose last sum may pass
                int w = 0;
                double before = 0.0;
#pragma unroll
                for (int v = 0; v < kWarps - 1; ++v)
                    if (!not_less(upto[v], lo)) { w = v + 1; before = upto[v]; }
                double sums = before + incl[w * 32 + lane];     // up to each thread's end
                const unsigned b = __ballot_sync(0xffffffffu, not_less(sums, lo));
                int g = w * 32 + (b ? __ffs(b) - 1 : 31);
                int ev = -1, last = 0;
                double run = __shfl_sync(0xffffffffu, sums, (g - 1) & 31);
                if (!(g & 31)) run = before;
                for (;;) {
                    // 32 pairs of thread g's run at a time, a lane each
                    const int gb = g * M, ge = min(gb + M, A);
                    for (int k0 = gb; k0 < ge && ev < 0; k0 += 32) {
                        const int k = k0 + lane;
                        const double r = k < ge ? rates[k] : 0.0;
                        double x = r;
                        const int n = min(32, ge - k0);
                        for (int s = 1; s < n; s <<= 1) {
                            const double o = __shfl_up_sync(0xffffffffu, x, s);
                            if (lane >= s) x += o;
                        }
                        const double cum = run + x;
                        const bool hit = k < ge && (not_less(cum, hi) || (not_less(cum, lo) && cum / total >= u2));
                        const unsigned hits = __ballot_sync(0xffffffffu, hit);
                        if (hits) {
                            ev = k0 + __ffs(hits) - 1;
                        } else {
                            const unsigned some = __ballot_sync(0xffffffffu, positive(r));
                            if (some) last = k0 + 31 - __clz(some);
                            run = __shfl_sync(0xffffffffu, cum, 31);
                        }
                    }
                    if (ev >= 0 || ++g >= kThreads || g * M >= A) break;
                    // not in that run after all: the next thread's, from the
                    // prefix it has
                    if ((g >> 5) != w) before += incl[w++ * 32 + 31];
                    run = (g & 31) ? before + incl[g - 1] : before;
                }
                int f = 0, t = 0;
                if (kReplay && ev < 0 && (__double2hiint(u2) & 0x7ff00000) == 0x7ff00000) {
                    // NaN: the dense loop's first entry, pair (0, 0), which
                    // fills site 0: a hole from nowhere if it was empty
                    if (lane == 0) ev_from = (occw[0] & 1u) ? 0 : S;
                } else {
                    // u2 within the rounding of 1: the last pair that can hop
                    if (ev < 0) ev = last;
                    int row, col;
                    if (ev < A1) row = div_small(ev, T1, inv1, col);
                    else row = N + div_small(ev - A1, T2, inv2, col);
                    if (col >= z) col += N - z;
                    f = src[row].id;
                    t = tgt[col].id;
                    if (lane == 0) ev_from = f;
                }
                if (lane == 0) {
                    ev_to = t;
                    // fire and forget: nothing of this launch reads them
                    if (f >= N) atomicAdd(reinterpret_cast<unsigned long long *>(&eo[f - N]), ~0ull);
                    if (t >= N) atomicAdd(reinterpret_cast<unsigned long long *>(&eo[t - N]), 1ull);
                    if (record) atomicAdd(&traffic[(size_t)f * S + t], 1.0);
                    if (hop_log) { hop_log[2 * hop] = f; hop_log[2 * hop + 1] = t; }
                }
            }
        }
        if (flux_time) {
            // expected net hole flow into each electrode: its column of the
            // rate matrix minus its row
            for (int e = kWarps - 1 - warp; e < P; e += kWarps) {
                double in = 0.0, out = 0.0;
                for (int r = lane; r < h; r += 32) in += rates[r * T1 + z + e];
                for (int c = lane; c < z; c += 32) out += rates[A1 + e * T2 + c];
                double J = in - out;
#pragma unroll
                for (int s = 16; s > 0; s >>= 1) J += __shfl_xor_sync(0xffffffffu, J, s);
                if (lane == 0) sh_J[e] = J;
            }
        }
        __syncthreads();
        from = ev_from;
        if (from < 0) {
            status = KMC_ERR_NONFINITE;
            break;
        }
        to = ev_to;
        dt = sh_dt;
        h += (to < N ? 1 : 0) - (from < N ? 1 : 0);
        if (flux_time)
            for (int e = tid; e < P; e += kThreads) sh_fx[e] += sh_J[e] * dt;
    }
    __syncthreads();
    // the loop ends with the last hop not yet in the bits (an error: with
    // the bits up to date)
    if (status == KMC_OK && tid == 0) {
        if (from < N) occw[from >> 5] &= ~(1u << (from & 31));
        if (to < N) occw[to >> 5] |= 1u << (to & 31);
    }
    __syncthreads();
    for (int i = tid; i < N; i += kThreads) occ_g[i] = (occw[i >> 5] >> (i & 31)) & 1u;
    if (record && tid < N) oit[tid] = oit0;
    if (flux_time)
        for (int e = tid; e < P; e += kThreads) flux_time[e] = sh_fx[e];
    if (tid == 32) *time_out = time;
    if (tid == 0) *status_out = status;
}

template <bool kTab, bool kRate, bool kReplay>
__global__ void __launch_bounds__(kThreads, 1) f64_chain_kernel(
    const Layout lay, int N, int P, double nu, double kT, double I0, double R, uint8_t *occ_g, const double *d,
    const double *Ec, const double *se_in, const double *tc, int64_t *eo, int64_t hops,
    int record, double *traffic, double *oit, const double *uniforms, uint64_t seed,
    int32_t *hop_log, double *time_out, int32_t *status_out, double *ws, double *flux_time)
{
    f64_chain<kTab, kRate, kReplay>(lay, N, P, nu, kT, I0, R, occ_g, d, Ec, se_in, tc, eo, hops, record, traffic, oit,
                           uniforms, seed, hop_log, time_out, status_out, ws, flux_time);
}

// Many independent chains in one launch, one block each (Philox streams
// keyed by each chain's own seed).
template <bool kTab, bool kRate>
__global__ void __launch_bounds__(kThreads, 1) f64_batch_kernel(const Layout lay, const kmc_f64_batch B,
                                                             size_t ws_doubles)
{
    const int c = blockIdx.x;
    const int N = B.N[c], P = B.P[c];
    // a chain whose sizes do not fit the launch (shared memory is sized for
    // max_sites, the flux buffer for 64 electrodes) stops before any access
    if (N < 0 || P < 0 || N + P <= 0 || N + P > B.max_sites || (B.flux_time && P > 64) || !(B.kT[c] > 0.0) ||
        B.hops[c] < 0) {
        if (threadIdx.x == 0) {
            B.status_out[c] = KMC_ERR_INVALID;
            B.time_out[c] = 0.0;
        }
        return;
    }
    const int64_t so = B.site_off[c], eo = B.el_off[c], po = B.pair_off[c], vo = B.se_off[c];
    double *fx = B.flux_time ? B.flux_time + eo : nullptr;
    double *tr = B.record ? B.traffic + B.traffic_off[c] : nullptr;
    double *oit = B.record ? B.occupations_in_time + so : nullptr;
    f64_chain<kTab, kRate, false>(lay, N, P, B.nu[c], B.kT[c], B.I_0[c], B.R[c], B.occupation + so, B.distances + po,
                           B.E_constant + so, B.site_energies + vo, B.transitions_constant + po,
                           B.electrode_occupation + eo, B.hops[c], B.record, tr, oit, nullptr, B.seeds[c], nullptr,
                           B.time_out + c, B.status_out + c, B.workspace + (size_t)c * ws_doubles, fx);
}

// Where a launch's arrays go: `budget` bytes of shared memory a block, for at
// most A_max allowed pairs.  The rates first (written and read twice a hop),
// then the pair table (two reads a pair), then 1/d (z reads a site).
Layout f64_layout(int S, int N, int64_t A_max, size_t budget)
{
    Layout l{S, 0, 0, 0};
    auto take = [&](int Layout::*part, int64_t entries) {
        Layout t = l;
        if (entries > (1 << 20)) return;
        t.*part = static_cast<int>((entries + 1) & ~static_cast<int64_t>(1));
        if (layout_bytes(t) <= budget) l = t;
    };
    take(&Layout::rates, A_max);
    if (l.rates > 0) take(&Layout::tab, static_cast<int64_t>(S) * S);
    take(&Layout::invd, static_cast<int64_t>(N) * N);
    return l;
}

constexpr size_t kBlockSmem = 220 * 1024;    // dynamic shared memory of one block
constexpr size_t kSmSmem = 227 * 1024;       // shared by the blocks of an SM (1 KB of each is the system's)

template <typename K>
int allow_smem(K *kernel, size_t smem)
{
    if (smem <= 48 * 1024) return KMC_OK;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kBlockSmem));
    return e == cudaSuccess ? KMC_OK : fail_cuda(e, "cudaFuncSetAttribute(f64)");
}

}  // namespace

size_t f64_workspace_size(int S)
{
    return sizeof(double) * (2 * (size_t)S * S + (size_t)S * S);
}

int simulate_f64(int N, int P, double nu, double kT, double I0, double R, uint8_t *occ,
                 const double *d, const double *Ec, const double *se, const double *tc,
                 int64_t *eo, int64_t hops, int record, double *traffic, double *oit,
                 const double *uniforms, uint64_t seed, int32_t *hop_log, double *time_out,
                 int32_t *status_out, void *ws, size_t ws_bytes, cudaStream_t st, double *flux_time)
{
    const int S = N + P;
    if (N < 0 || P < 0 || S <= 0 || S > kMaxSitesF64 || hops < 0)
        return fail(KMC_ERR_INVALID, "simulate_f64: bad sizes N=%d P=%d hops=%lld", N, P, (long long)hops);
    if (!occ && N > 0) return fail(KMC_ERR_INVALID, "simulate_f64: occupation is NULL");
    if (!d || !Ec || !se || !tc || (!eo && P > 0) || !time_out || !status_out || !ws)
        return fail(KMC_ERR_INVALID, "simulate_f64: a required pointer is NULL");
    if (record && (!traffic || (!oit && N > 0)))
        return fail(KMC_ERR_INVALID, "simulate_f64: record needs traffic and occupations_in_time");
    if (ws_bytes < f64_workspace_size(S))
        return fail(KMC_ERR_INVALID, "simulate_f64: workspace %zu bytes < %zu", ws_bytes, f64_workspace_size(S));
    if (!(kT > 0)) return fail(KMC_ERR_INVALID, "simulate_f64: kT must be positive");
    if (flux_time && P > 64) return fail(KMC_ERR_INVALID, "simulate_f64: flux_time supports at most 64 electrodes");
    // A(h) = h(N - h) + N P is largest at h = N/2
    const Layout lay = f64_layout(S, N, static_cast<int64_t>(N) * N / 4 + static_cast<int64_t>(N) * P, kBlockSmem);
    const size_t smem = layout_bytes(lay);
    auto launch = [&](auto *kernel) -> int {
        const int rc = allow_smem(kernel, smem);
        if (rc != KMC_OK) return rc;
        kernel<<<1, kThreads, smem, st>>>(lay, N, P, nu, kT, I0, R, occ, d, Ec, se, tc, eo, hops, record, traffic,
                                          oit, uniforms, seed, hop_log, time_out, status_out,
                                          static_cast<double *>(ws), flux_time);
        return KMC_OK;
    };
    const int rc = uniforms ? (lay.tab > 0     ? launch(f64_chain_kernel<true, true, true>)
                               : lay.rates > 0 ? launch(f64_chain_kernel<false, true, true>)
                                               : launch(f64_chain_kernel<false, false, true>))
                            : (lay.tab > 0     ? launch(f64_chain_kernel<true, true, false>)
                               : lay.rates > 0 ? launch(f64_chain_kernel<false, true, false>)
                                               : launch(f64_chain_kernel<false, false, false>));
    if (rc != KMC_OK) return rc;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail_cuda(e, "f64 launch");
    return KMC_OK;
}


size_t f64_batch_workspace_size(int n_chains, int max_sites)
{
    return (size_t)n_chains * f64_workspace_size(max_sites);
}

int simulate_f64_batch(const kmc_f64_batch &B, cudaStream_t st)
{
    if (B.n_chains < 0 || B.max_sites <= 0 || B.max_sites > kMaxSitesF64)
        return fail(KMC_ERR_INVALID, "simulate_f64_batch: bad sizes (n_chains %d, max_sites %d)", B.n_chains,
                    B.max_sites);
    if (B.n_chains == 0) return KMC_OK;
    if (!B.N || !B.P || !B.nu || !B.kT || !B.I_0 || !B.R || !B.pair_off || !B.distances ||
        !B.transitions_constant || !B.site_off || !B.E_constant || !B.se_off || !B.site_energies ||
        !B.occupation || !B.el_off || !B.electrode_occupation || !B.hops || !B.seeds || !B.time_out ||
        !B.status_out || !B.workspace)
        return fail(KMC_ERR_INVALID, "simulate_f64_batch: a required pointer is NULL");
    if (B.record && (!B.traffic || !B.traffic_off || !B.occupations_in_time))
        return fail(KMC_ERR_INVALID, "simulate_f64_batch: record needs traffic, traffic_off, occupations_in_time");
    if (B.workspace_bytes < f64_batch_workspace_size(B.n_chains, B.max_sites))
        return fail(KMC_ERR_INVALID, "simulate_f64_batch: workspace %zu bytes < %zu", B.workspace_bytes,
                    f64_batch_workspace_size(B.n_chains, B.max_sites));
    // per-chain sizes are checked by each block (KMC_ERR_INVALID in status_out)
    const int S = B.max_sites;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return fail_cuda(e, "simulate_f64_batch: device query");
    // Blocks that share an SM overlap their serial phases, so a launch of
    // more chains than SMs divides an SM's shared memory among up to three:
    // 150 registers a thread hold no more (304 chains of N = 60, 100 hops 2.2
    // ms, 152 1.7; 512, the last 56 in a second wave, 4.1).
    const int per_sm = std::max(1, std::min(3, (B.n_chains + sms - 1) / std::max(sms, 1)));
    // A(h) <= S^2/3 for any split of S sites into acceptors and electrodes
    const Layout lay = f64_layout(S, S, static_cast<int64_t>(S) * S / 3 + 1,
                                  std::min(kBlockSmem, kSmSmem / per_sm - 1280));
    const size_t smem = layout_bytes(lay);
    auto launch = [&](auto *kernel) -> int {
        const int rc = allow_smem(kernel, smem);
        if (rc != KMC_OK) return rc;
        kernel<<<B.n_chains, kThreads, smem, st>>>(lay, B, f64_workspace_size(S) / sizeof(double));
        return KMC_OK;
    };
    const int rc = lay.tab > 0 ? launch(f64_batch_kernel<true, true>)
                   : lay.rates > 0 ? launch(f64_batch_kernel<false, true>) : launch(f64_batch_kernel<false, false>);
    if (rc != KMC_OK) return rc;
    e = cudaGetLastError();
    return e == cudaSuccess ? KMC_OK : fail_cuda(e, "f64 batch launch");
}

// ---------------------------------------------------------------------------
// Allocation-free variant
//
// Some callers of this kernel cannot allocate device memory when they call
// it: a host that owns every byte of the device through its own memory pool
// and hands plugins only the buffers it placed, or a latency-bound loop in
// which a cudaMalloc / cudaFree (which may synchronise the whole device)
// would stall other work.  For them the workspace is a fixed array in this
// library's device memory instead of a caller-provided buffer.
// ---------------------------------------------------------------------------

// Largest network the static workspace holds: S = N + P <= 128 sites, i.e.
// 3 * 128^2 doubles = 384 KiB, resident on every device that loads the
// library until the process exits.
constexpr int kStaticWorkspaceSites = 128;
static __device__ __align__(256) double g_f64_static_workspace[3 * kStaticWorkspaceSites * kStaticWorkspaceSites];

// Device address of the static workspace in the current context.  The
// array's name is only a host-side stand-in in host code, so its address is
// looked up on every call (cheap once the module is loaded).  It is not
// cached: after a cudaDeviceReset, or in another context on the same device,
// the module is loaded again at a different address.
static int static_workspace(double **out)
{
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_f64_static_workspace);
    if (e != cudaSuccess) return fail_cuda(e, "simulate_f64_static: cudaGetSymbolAddress");
    *out = static_cast<double *>(p);
    return KMC_OK;
}

}  // namespace kmc

extern "C" int kmc_simulate_f64_static(int32_t n_acceptors, int32_t n_electrodes, double nu,
                                       double kT, double I_0, double R, uint8_t *occupation,
                                       const double *distances, const double *E_constant,
                                       const double *site_energies,
                                       const double *transitions_constant,
                                       int64_t *electrode_occupation, int64_t hops, int32_t record,
                                       double *traffic, double *occupations_in_time,
                                       const double *uniforms, uint64_t seed, int32_t *hop_log,
                                       double *time_out, int32_t *status_out, void *stream)
{
    using namespace kmc;
    const int S = n_acceptors + n_electrodes;
    if (n_acceptors < 0 || n_electrodes < 0 || S <= 0 || S > kStaticWorkspaceSites)
        return fail(KMC_ERR_INVALID,
                    "kmc_simulate_f64_static: %d sites (N=%d, P=%d); the fixed workspace holds at most %d "
                    "(use kmc_simulate_f64 with a caller workspace for larger networks)",
                    S, n_acceptors, n_electrodes, kStaticWorkspaceSites);
    double *ws = nullptr;
    const int rc = static_workspace(&ws);
    if (rc != KMC_OK) return rc;
    // The kernel writes every workspace entry it reads within the call
    // (the pairs' factors, 1/d and the rates), so the contents a previous call
    // left behind need no clearing.
    return simulate_f64(n_acceptors, n_electrodes, nu, kT, I_0, R, occupation, distances, E_constant,
                        site_energies, transitions_constant, electrode_occupation, hops, record,
                        traffic, occupations_in_time, uniforms, seed, hop_log, time_out, status_out,
                        ws, sizeof(double) * 3 * (size_t)kStaticWorkspaceSites * kStaticWorkspaceSites,
                        static_cast<cudaStream_t>(stream), nullptr);
}

namespace kmc {

int preload_f64()
{
    int rc;
    if ((rc = touch_kernel(f64_chain_kernel<true, true, false>)) != KMC_OK) return rc;
    if ((rc = touch_kernel(f64_chain_kernel<true, true, true>)) != KMC_OK) return rc;
    if ((rc = touch_kernel(f64_chain_kernel<false, true, false>)) != KMC_OK) return rc;
    if ((rc = touch_kernel(f64_chain_kernel<false, true, true>)) != KMC_OK) return rc;
    if ((rc = touch_kernel(f64_chain_kernel<false, false, false>)) != KMC_OK) return rc;
    if ((rc = touch_kernel(f64_chain_kernel<false, false, true>)) != KMC_OK) return rc;
    if ((rc = touch_kernel(f64_batch_kernel<true, true>)) != KMC_OK) return rc;
    if ((rc = touch_kernel(f64_batch_kernel<false, true>)) != KMC_OK) return rc;
    return touch_kernel(f64_batch_kernel<false, false>);
}

}  // namespace kmc

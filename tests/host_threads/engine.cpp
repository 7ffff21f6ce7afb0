// The FP32 hop loops (warp slices and block groups) on host threads: a few
// chains of one small network over several re-anchors.  One argument, the
// launch; exits non-zero when a chain does not make its hops.
#include <cstdlib>

#include "device.h"
#include "kmc_f32_warp.cuh"

namespace kmc {
int fail(int code, const char *, ...) { return code; }
int fail_cuda(cudaError_t, const char *) { return 1; }
}
using namespace kmc;

namespace {

uint64_t rng_state;
double uniform()
{
    rng_state = rng_state * 6364136223846793005ull + 1442695040888963407ull;
    return static_cast<double>(rng_state >> 11) * 0x1p-53;
}

// a rate of 1 for every pair
struct PairPlace : PositionPairs {
    float rate(float4, float4, bool, float) const { return 1.0f; }
};

// record: the Go convention with flux, drift and log; stored: with the buffer
// of running sums; two: two tables (read from memory, not staged).
template <int G, typename Pairs>
int launch(int N, int P, int reanchor, int hops, int chains, bool record, bool stored, bool two)
{
    constexpr bool kBlock = G > 32;
    const int S = N + P;
    rng_state = 1000 * static_cast<uint64_t>(N) + P;
    const double L = std::sqrt(N / 0.075), a = 1.8, IR = 18.0;
    std::vector<float> pos, tab(2 * S * S), coef, Ec, Vel;
    for (int i = 0; i < S; ++i) {
        double x = L * uniform(), y = L * uniform();
        if (i >= N) (i & 1 ? x : y) = (i & 2) ? L : 0.0;
        for (double v : {x, y, 0.0, 0.0}) pos.push_back(static_cast<float>(v));
    }
    for (int i = 0; i < S; ++i)
        for (int j = 0; j < S; ++j) {
            const double d = std::hypot(pos[4 * i] - pos[4 * j], pos[4 * i + 1] - pos[4 * j + 1]);
            tab[2 * (i * S + j)] = static_cast<float>(-2.0 * d / a * kLog2e);
            tab[2 * (i * S + j) + 1] = i < N && j < N && i != j ? static_cast<float>(IR / d) : 0.0f;
        }
    std::vector<int32_t> n_of{N, N}, p_of{P, P}, tab_of, status(chains, -1), traffic(chains * S * S), work;
    std::vector<int64_t> zero{0, 0}, so, eo, po, lo, net(chains * P), done(chains), budget;
    std::vector<uint64_t> stream;
    std::vector<uint8_t> occ;
    std::vector<double> time(chains), occ_time(chains * N), since(chains * N), flux(chains * P);
    std::vector<float> kT(chains, 1.0f), drift(chains);
    std::vector<int32_t> log(2 * chains * hops);
    for (int k = 0; k < 2; ++k)
        for (double v : {-2.0 / a * kLog2e, 0.0, IR, 0.0}) coef.push_back(static_cast<float>(v));
    for (int c = 0; c < chains; ++c) {
        tab_of.push_back(two ? c & 1 : 0);
        so.push_back(c * N);
        eo.push_back(c * P);
        po.push_back(static_cast<int64_t>(c) * S * S);
        lo.push_back(static_cast<int64_t>(c) * hops);
        budget.push_back(hops - 3 * c);         // the chains of a warp end one after another
        stream.push_back(c);
        work.push_back(c);
        for (int i = 0; i < N; ++i) {
            Ec.push_back(static_cast<float>(4.0 * uniform() - 2.0));
            occ.push_back(i > N / 10);
        }
        for (int e = 0; e < P; ++e) Vel.push_back(static_cast<float>(2.0 * uniform() - 1.0));
    }
    constexpr int kPerItem = kBlock ? 1 : 32 / G;
    while (work.size() % kPerItem) work.push_back(-1);
    kmc_batch B{};
    B.n_tables = two ? 2 : 1;
    B.max_sites = S;
    B.tab_N = n_of.data();
    B.tab_P = p_of.data();
    B.tab_off = B.tab_pos_off = zero.data();
    B.tab_LB = tab.data();
    B.tab_pos = pos.data();
    B.tab_coef = coef.data();
    B.n_chains = chains;
    B.lanes_per_chain = G;
    B.chain_tab = tab_of.data();
    B.chain_kT = kT.data();
    B.uniform_kT = 1.0f;
    B.chain_site_off = so.data();
    B.chain_el_off = eo.data();
    B.chain_pair_off = po.data();
    B.E_constant = Ec.data();
    B.el_energy = Vel.data();
    B.occupation = occ.data();
    B.electrode_occupation = net.data();
    B.time = time.data();
    B.hops_done = done.data();
    B.hops_total = budget.data();
    B.stream = stream.data();
    B.status = status.data();
    B.energy_drift = drift.data();
    B.hop_log = log.data();
    B.hop_log_off = lo.data();
    if (record) {
        B.record = KMC_RECORD_GO;
        B.occ_time = occ_time.data();
        B.occ_since = since.data();
        B.traffic = traffic.data();
        B.flux_time = flux.data();
    }
    B.work = work.data();
    B.n_work = static_cast<int32_t>(work.size()) / kPerItem;
    B.reanchor = reanchor;
    B.warps_per_block = 1;
    B.max_hops_per_launch = 1 << 20;
    B.seed = 5;
    const int rate_words = stored ? rate_buffer_words(S, G) : 0;
    const int table_words = Pairs::kUniformTable ? (3 * S * S + 3) & ~3 : 0;
    for (int item = 0; item < B.n_work; ++item)
        run_block(kBlock ? G : 32, [&] {
            blockIdx.x = static_cast<unsigned>(item);
            if constexpr (kBlock) block_engine_kernel<G, Pairs, 512 / G>(B, rate_words, table_words);
            else warp_engine_kernel<G, Pairs, 2>(B, rate_words, table_words);
        });
    for (int c = 0; c < chains; ++c)
        if (status[c] != KMC_OK || done[c] != budget[c]) return 1;
    return 0;
}

#ifdef KMC_DEBUG_CHECKS
// Runs of two holes, three empty acceptors and one electrode (11 pairs): 0
// where those within are walked and those beyond are refused.
int runs()
{
    const PairPlace place{};
    std::vector<float4> rec(8, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
    const PairRange range{2, 3, 1, 4, 3, 8, 11, 0.25f, 1.0f / 3.0f};
    float kept[16], sum = 0.0f;
    auto walk = [&](int b, int e) { return walk_pairs<true, 1, 4>(place, rec.data(), rec.data(), range, b, e, 1.0f, kept, sum); };
    return walk(0, 11) && walk(3, 9) && sum == 17.0f && !walk(0, 12) && !walk(10, 12) && !walk(11, 12) && !walk(-1, 3) ? 0 : 1;
}
#endif

}  // namespace

int main(int, char **argv)
{
    using Far = TablePairs<false>;
    using Uniform = TablePairs<true, true>;
    switch (std::atoi(argv[1])) {
    case 0: return launch<4, Uniform>(12, 3, 4, 40, 6, false, true, false);
    case 1: return launch<8, PositionPairs>(30, 4, 7, 40, 3, true, false, false);
    case 2: return launch<64, Far>(40, 6, 5, 30, 1, true, true, true);
    case 3: return launch<64, PairedPositionPairs>(90, 6, 9, 20, 1, true, false, false);
    case 4: return launch<256, PairedPositionPairs>(70, 6, 5, 10, 1, true, true, false);
    case 5: return launch<16, Far>(40, 4, 5, 40, 2, true, true, true);
    case 6: return launch<32, Far>(40, 4, 9, 40, 1, false, true, true);
#ifdef KMC_DEBUG_CHECKS
    case 7: return runs();
#endif
    }
    return 2;
}

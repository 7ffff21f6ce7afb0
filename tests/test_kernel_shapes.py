"""Kernels and dispatch branches at the sizes where they change: edges of
warps, tiles and shared-memory layouts, launches of one chain and of many."""
import ctypes as C

import numpy as np
import pytest

from kmc_dn_gb300 import workloads
from kmc_dn_gb300.rng import replay_uniforms


def _net(N, P, seed=0, kT=1.0, nu=1.0, volts=1.0):
    L = float(np.sqrt(N / workloads.DENSITY))
    rng = np.random.Generator(np.random.PCG64(1000 * seed + N))
    return workloads.make_network(rng, N, N // 10, L, L, workloads.perimeter_electrodes(L, P),
                                  voltages=volts * rng.uniform(-1, 1, P), kT=kT, nu=nu, cells=40)


def _batch(nets, hops, seed=3, chain_table=None, streams=None, **kw):
    from kmc_dn_gb300.engine import Batch, TableSpec
    specs = [TableSpec.from_network(n) for n in nets]
    ct = np.arange(len(nets)) if chain_table is None else np.asarray(chain_table)
    of = [nets[k] for k in ct]
    return Batch(specs, ct, [n.kT for n in of], [n.E_constant() for n in of], [n.electrodes[:, 3] for n in of],
                 [n.occupation.astype(np.uint8) for n in of], hops, seed=seed, streams=streams, **kw)


def _same(a, b):
    """Equal results of one chain (bit for bit): (result, index) pairs."""
    (ra, i), (rb, j) = a, b
    for k in ("time", "hops_done", "status", "n_pairs", "occupation", "electrode_occupation", "hop_log"):
        if k in ra:
            np.testing.assert_array_equal(ra[k][i], rb[k][j], err_msg=k)


# ---- FP64 hop kernel ------------------------------------------------------
# Tolerance of the time: each total is a sum of at most A = N^2/4 + N P rates
# (relative error A eps at worst), each rate's exponent carries the rounding
# of an energy of size x/kT: a few eps x.  A = 43000, x = 1e3 at N = 400:
# 1e-11 + 1e-12.  With voltages of 1e6 kT the exponents carry eps 1e6 =
# 2e-10.
@pytest.mark.gpu
@pytest.mark.parametrize("N,P,kT,nu,volts,rtol", [
    (1, 2, 1.0, 1.0, 1.0, 1e-11), (31, 1, 0.7, 1.0, 1.0, 1e-11), (32, 8, 1.0, 2.5, 1.0, 1e-11),
    (33, 4, 2.3, 0.3, 1.0, 1e-11),
    (90, 8, 1.0, 1.0, 1.0, 1e-11),       # the largest tables in shared memory
    (100, 8, 1.0, 1.0, 1.0, 1e-11),      # rates and 1/d there
    (160, 8, 0.7, 1.0, 1.0, 1e-11),      # rates only
    (400, 8, 1.0, 1.0, 1.0, 1e-10),      # nothing there
    (33, 8, 1.0, 1.0, 1.0e6, 1e-9)])     # beyond the split exponential
def test_f64_layouts_match_oracle(engine_lib, oracle_mod, N, P, kT, nu, volts, rtol):
    from kmc_dn_gb300.engine import simulate_f64
    n, hops = _net(N, P, kT=kT, nu=nu, volts=volts), 200
    u = replay_uniforms(7, 2 * hops)
    args = (n.N, n.P, n.nu, n.kT, n.I_0, n.R)
    r = simulate_f64(*args, n.occupation.astype(np.uint8), n.distances, n.E_constant(), n.site_energies(),
                     n.transitions_constant, hops, record=True, uniforms=u, hop_log=True)
    o = oracle_mod.numba_replay(*args, n.occupation.astype(np.uint8), n.distances, n.E_constant(),
                                n.site_energies(), n.transitions_constant, u, record=True)
    assert r["status"] == 0
    np.testing.assert_array_equal(r["hop_log"], o["hop_log"])
    np.testing.assert_array_equal(r["traffic"], o["traffic"])
    assert abs(r["time"] - o["time"]) <= rtol * o["time"]
    np.testing.assert_allclose(r["occupations_in_time"], o["occupations_in_time"], rtol=rtol, atol=rtol * o["time"])


@pytest.mark.gpu
@pytest.mark.parametrize("N", [30, 60, 110])
def test_f64_batch_matches_single_chains(engine_lib, N):
    """Many chains share an SM's memory and get other layouts than one."""
    from kmc_dn_gb300.engine import simulate_f64, simulate_f64_many
    n, hops, seeds = _net(N, 8), 150, [11 + k for k in range(320)]
    c = dict(N=n.N, P=n.P, nu=n.nu, kT=n.kT, I_0=n.I_0, R=n.R, occupation=n.occupation.astype(np.uint8),
             distances=n.distances, E_constant=n.E_constant(), site_energies=n.site_energies(),
             transitions_constant=n.transitions_constant)
    t, eo, status = simulate_f64_many([c] * len(seeds), hops, seeds)[:3]
    assert not np.any(status)
    for k in (0, 151, 319):
        r = simulate_f64(*(c[x] for x in ("N", "P", "nu", "kT", "I_0", "R", "occupation", "distances", "E_constant",
                                          "site_energies", "transitions_constant")), hops, seed=seeds[k])
        np.testing.assert_array_equal(r["electrode_occupation"], eo[k])
        assert abs(r["time"] - t[k]) <= 1e-11 * t[k]


# ---- FP32 engine ----------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("lanes,N", [(8, 8), (8, 9), (8, 16), (8, 17), (8, 33), (16, 31), (16, 65), (32, 32),
                                     (32, 33), (32, 64), (32, 65), (32, 80)])
def test_rebuild_from_l2_equals_staged(engine_lib, lanes, N):
    """Two tables in a launch are read from L2 and the lists rebuilt several
    sites a lane a step; one table is staged and rebuilt site by site."""
    a, b = _net(N, 5, seed=1), _net(N, 5, seed=2)
    both = _batch([a, b], [1500, 1500], lanes=lanes, hop_log=True).run().results()
    for k, n in enumerate((a, b)):
        _same((both, k), (_batch([n], [1500], lanes=lanes, hop_log=True, streams=[k]).run().results(), 0))


@pytest.mark.gpu
@pytest.mark.parametrize("lanes,N,P", [(64, 40, 2), (64, 60, 8), (64, 61, 7), (64, 90, 1), (64, 120, 8), (128, 150, 9),
                                       (64, 200, 5)])
def test_runs_of_rows_in_part_replay(engine_lib, oracle_mod, lanes, N, P):
    """Positions, block groups, balanced runs of at least a row.  The oracle's hops on a stream that keeps 1e-4 of the
    total rate away from every boundary (the FP32 cumulative sums are within
    2e-5 of it); odd rows, odd starts, few electrodes."""
    n, hops = _net(N, P, seed=4), 400
    occ = n.occupation.astype(np.uint8)
    net = (n.N, n.P, n.nu, n.kT, n.I_0, n.R, occ, n.distances, n.E_constant(), n.site_energies(), n.transitions_constant)
    u, _ = oracle_mod.clear_stream(*net, hops, 9)
    o = oracle_mod.numba_replay(*net, u)
    r = _batch([n], [hops], lanes=lanes, pair_mode="positions", replay=[u], hop_log=True).run().results()
    np.testing.assert_array_equal(r["hop_log"][0], o["hop_log"])
    assert abs(r["time"][0] - o["time"]) <= 1e-4 * o["time"]


@pytest.mark.gpu
@pytest.mark.parametrize("mode,lanes,N", [("table", 4, 120), ("table", 4, 80), ("positions", 4, 80), ("table", 32, 120),
                                          ("positions", 32, 120), ("table", 4, 10), ("positions", 16, 30)])
def test_slices_of_a_warp_end_alone(engine_lib, mode, lanes, N):
    """Chains of one warp with other budgets (none, one hop, across an anchor),
    with and without a rate buffer (none at 4 lanes and N >= 80)."""
    n, hops = _net(N, 8), [700, 0, 1, 33, 1024, 1025, 5, 700, 300]
    r = _batch([n], hops, chain_table=[0] * 9, lanes=lanes, pair_mode=mode, hop_log=True).run().results()
    assert r["hops_done"].tolist() == hops
    for k in range(9):
        alone = _batch([n], hops[k:k + 1], chain_table=[0], streams=[k], lanes=lanes, pair_mode=mode, hop_log=True)
        _same((r, k), (alone.run().results(), 0))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["table", "positions"])
@pytest.mark.parametrize("lanes,N", [(64, 200), (64, 203), (128, 240)])
def test_block_search_without_stored_sums(engine_lib, lanes, N, mode):
    """A launch of more chains than fit beside their running sums drops these
    and re-evaluates the chosen run; alone a chain keeps them.  The two search
    the same rates in sums that associate differently (1e-7 of a run), so the
    hops of a few short chains are the same."""
    import torch
    n, count = _net(N, 7), 5 * torch.cuda.get_device_properties(0).multi_processor_count
    many = _batch([n], [60] * count, chain_table=[0] * count, lanes=lanes, pair_mode=mode, hop_log=True).run().results()
    assert not np.any(many["status"])
    for k in (0, 1, count // 2, count - 1):
        alone = _batch([n], [60], chain_table=[0], streams=[k], lanes=lanes, pair_mode=mode, hop_log=True).run().results()
        np.testing.assert_array_equal(many["hop_log"][k], alone["hop_log"][0])


@pytest.mark.gpu
def test_bins_side_by_side(engine_lib):
    """Size bins on streams of their own give what they give one after the
    other, and budgets changed after construction are kept to."""
    import torch
    nets = [_net(N, 6) for N in (5, 40, 150, 12, 90, 200)]
    side, serial = _batch(nets, [300] * 6), _batch(nets, [300] * 6)
    assert len(side._bins) > 1
    side.launch()
    serial.launch(bin_streams=[torch.cuda.current_stream()])
    for b in (side, serial):
        b.hops_total += 500
    side.launch()
    serial.launch(bin_streams=[torch.cuda.current_stream()])
    ra, rb = side.results(), serial.results()
    assert ra["hops_done"].tolist() == [800] * 6
    for k in range(6):
        _same((ra, k), (rb, k))


@pytest.mark.gpu
def test_tables_of_a_batch_equal_single_builds(engine_lib):
    import torch
    from kmc_dn_gb300._native import check, lib
    rng = np.random.default_rng(5)
    sizes = [(1, 0), (1, 2), (16, 1), (31, 8), (90, 8)]
    d = [rng.uniform(0.1, 3.0, (N + P, N + P)) for N, P in sizes]        # asymmetric
    tc = [rng.uniform(0.0, 1.0, x.shape) * (rng.random(x.shape) < 0.9) for x in d]
    k = np.arange(1.0, 6.0)
    N, P = (np.array(x, np.int32) for x in zip(*sizes))
    off = np.concatenate([[0], np.cumsum([2 * x.size for x in d])]).astype(np.int64)
    tab = torch.zeros(int(off[-1]), dtype=torch.float32, device="cuda")
    ptrs = [np.array([a.ctypes.data for a in x], np.uint64) for x in (d, tc)]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    nu, I0, R = k / 2, 10 * k, 1 / k
    check(lib().kmc_build_tables(5, *(C.c_void_p(a.ctypes.data) for a in (N, P, nu, I0, R, *ptrs, off)),
                                 C.c_void_p(tab.data_ptr()), st))
    for t in range(5):
        one = torch.zeros(2 * d[t].size, dtype=torch.float32, device="cuda")
        dd, tt = torch.as_tensor(d[t]).cuda(), torch.as_tensor(tc[t]).cuda()
        check(lib().kmc_build_table(int(N[t]), int(P[t]), nu[t], I0[t], R[t], C.c_void_p(dd.data_ptr()),
                                    C.c_void_p(tt.data_ptr()), C.c_void_p(one.data_ptr()), st))
        np.testing.assert_array_equal(tab[int(off[t]):int(off[t + 1])].cpu().numpy(), one.cpu().numpy())


# ---- mean field -----------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.parametrize("rates", ["f64", "f32"])
@pytest.mark.parametrize("N,P", [(1, 2), (30, 8), (32, 1), (63, 8), (87, 8), (88, 8)])
def test_mean_field_wide_and_narrow_blocks(engine_lib, rates, N, P):
    """Launches of few networks run wider FP64 blocks, and above 95 sites
    there is no room for the queue of exponentials: the same numbers."""
    from kmc_dn_gb300 import meanfield
    n = _net(N, P)
    V = np.random.default_rng(N).uniform(-1, 1, (200, P))
    nets = [meanfield.Network(N, P, n.nu, n.kT, n.I_0, n.R, n.distances, n.transitions_constant, n.E_constant(v), v)
            for v in V]
    many = meanfield.run(nets, 60, rates=rates)
    few = meanfield.run(nets[:3], 60, rates=rates)
    for k in range(3):
        assert many["status"][k] == 0 and many["time"][k] == few["time"][k]
        for key in ("occupation", "electrode_occupation", "site_energies"):
            np.testing.assert_array_equal(many[key][k], few[key][k])


# ---- Laplace basis --------------------------------------------------------
# Both solvers are direct, in FP64, on values in [0, 1]: the rounding of a
# system of n cells a side is a few n^2 eps (1e-10 at 600), observed far less.
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,P", [(2, 2, 1), (3, 5, 2), (7, 2, 3), (31, 33, 4), (64, 65, 8), (129, 31, 5),
                                     (600, 3, 2)])
def test_laplace_meshes(engine_lib, nx, ny, P):
    import torch
    from kmc_dn_gb300._native import check, lib
    from kmc_dn_gb300.laplace import boundary_grids, solve_basis_fields, solve_basis_fields_gpu
    X, Y = 3.0, 2.0
    el = np.array(workloads.perimeter_electrodes(1.0, P)) * (X, Y)
    for surplus in (None, 0.7):
        xy, g = torch.as_tensor(el).cuda(), torch.full((P + 1, ny + 1, nx + 1), -1.0, dtype=torch.float64, device="cuda")
        check(lib().kmc_laplace_boundary(nx, ny, X, Y, X / 10 if surplus is None else surplus, P,
                                         C.c_void_p(xy.data_ptr()), C.c_void_p(g.data_ptr()),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        np.testing.assert_array_equal(g.cpu().numpy(), boundary_grids(X, Y, el, nx, ny, surplus))
        gpu, cpu = (f(X, Y, el, nx, ny, surplus) for f in (solve_basis_fields_gpu, solve_basis_fields))
        np.testing.assert_allclose(gpu.fields, cpu.fields, atol=max(1e-12, max(nx, ny) ** 2 * 2.2e-16), rtol=0)


# ---- one buffer for a launch's arrays -------------------------------------
def test_pack_places_uploads_and_downloads():
    import torch
    from kmc_dn_gb300.engine import _Pack
    pk = _Pack()
    ins = {"a": (np.arange(7), torch.int32), "b": (np.arange(12.0).reshape(3, 4)[:, ::2], torch.float64),
           "c": (np.zeros(0), torch.float32), "d": (np.array([1, 0, 1]), torch.uint8)}
    for k, (a, dt) in ins.items():
        pk.add(k, a, dt)
    pk.zeros("z", (2, 5), torch.int64)
    pk.zeros("y", 3, torch.float64)
    t = pk.upload(torch.device("cpu"))
    for k, (a, dt) in ins.items():
        assert t[k].dtype == dt and tuple(t[k].shape) == a.shape
        np.testing.assert_array_equal(t[k].numpy(), a)
    assert t["z"].shape == (2, 5) and not t["z"].any() and not t["y"].any()
    t["z"][1, 2] = 9
    t["y"][2] = 0.5
    r = pk.download("d", "y")
    assert list(r) == ["d", "z", "y"] and r["z"][1, 2] == 9 and r["y"][2] == 0.5
    np.testing.assert_array_equal(r["d"], [1, 0, 1])

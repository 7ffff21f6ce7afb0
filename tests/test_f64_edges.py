"""The FP64 hop loop at the edges of its inputs: very short runs, uniforms on
the ends of their interval, electrode counts beyond 32 bits, energies and
rates at the ends of the exponent range."""
import numpy as np
import pytest

from kmc_dn_gb300 import workloads
from kmc_dn_gb300.rng import replay_uniforms

pytestmark = pytest.mark.gpu


def _net(N, P, seed=0, kT=1.0, nu=1.0, volts=1.0):
    L = float(np.sqrt(N / workloads.DENSITY))
    rng = np.random.Generator(np.random.PCG64(1000 * seed + N))
    return workloads.make_network(rng, N, N // 10, L, L, workloads.perimeter_electrodes(L, P),
                                  voltages=volts * rng.uniform(-1, 1, P), kT=kT, nu=nu, cells=30)


def _args(n, **kw):
    a = dict(N=n.N, P=n.P, nu=n.nu, kT=n.kT, I_0=n.I_0, R=n.R, occupation=n.occupation.astype(np.uint8),
             distances=n.distances, E_constant=n.E_constant(), site_energies=n.site_energies(),
             transitions_constant=n.transitions_constant)
    a.update(kw)
    return list(a.values())


def _replay(oracle_mod, args, u, rtol, **kw):
    """The kernel's run and the oracle's on one stream."""
    from kmc_dn_gb300.engine import simulate_f64
    hops = len(u) // 2
    r = simulate_f64(*args, hops, record=True, uniforms=u, hop_log=True, **kw)
    o = oracle_mod.numba_replay(*args, u, record=True, **kw)
    assert r["status"] == 0
    for k in ("hop_log", "traffic", "occupation", "electrode_occupation"):
        np.testing.assert_array_equal(r[k], o[k], err_msg=k)
    np.testing.assert_allclose(r["time"], o["time"], rtol=rtol)
    np.testing.assert_allclose(r["occupations_in_time"], o["occupations_in_time"], rtol=rtol, atol=rtol * o["time"])
    return r


# (Tolerances of the times: test_kernel_shapes.py.)
@pytest.mark.parametrize("hops", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,P,kT", [(1, 2, 1.0), (33, 8, 0.7), (100, 8, 1.0), (160, 8, 1.0), (400, 8, 2.0)])
def test_short_runs(engine_lib, oracle_mod, N, P, kT, hops):
    """Runs of up to three hops take every pair's own exponential."""
    _replay(oracle_mod, _args(_net(N, P, kT=kT)), replay_uniforms(11 + hops, 2 * hops), 1e-10)


@pytest.mark.parametrize("N,P", [(5, 3), (33, 8), (100, 8)])
def test_event_uniforms_at_the_ends(engine_lib, oracle_mod, N, P):
    """An event uniform of 0 takes the dense loop's first entry, pair (0, 0),
    which fills site 0; one outside [0, 1] never passes and ends there too.
    (1 itself is the boundary of every pair whose successors are lost in the
    total's rounding: which of them is first depends on the sums' order.)"""
    for fill in (False, True):
        n = _net(N, P, seed=2)
        n.occupation[0] = fill
        u = replay_uniforms(5, 160)
        u[[1, 3, 41, 159]] = 0.0
        u[81], u[101], u[121], u[131] = -0.0, 1.5, np.nan, 5e-324
        r = _replay(oracle_mod, _args(n), u, 1e-11)
        assert r["traffic"][0, 0] >= 6 and r["hop_log"][0].tolist() == [0, 0]


def test_electrode_counts_beyond_32_bits(engine_lib, oracle_mod):
    """The counters are the caller's 64-bit ones throughout the run."""
    n = _net(30, 6, seed=3)
    edge = 2**31
    start = np.array([edge - 1, -edge, edge, -edge - 1, 2**62, 0], np.int64)
    u = replay_uniforms(8, 2 * 2500)
    r = _replay(oracle_mod, _args(n), u, 1e-11, electrode_occupation=start)
    moved = r["electrode_occupation"] - start
    assert moved[0] or moved[1] or moved[2] or moved[3]

"""The mean field at the edges of its constants."""
import numpy as np
import pytest

from kmc_dn_gb300 import workloads

pytestmark = pytest.mark.gpu


def _run(n, hops, rates, **kw):
    from kmc_dn_gb300 import meanfield
    c = dict(nu=n.nu, kT=n.kT, I_0=n.I_0, R=n.R)
    c.update(kw)
    return meanfield.run([meanfield.Network(n.N, n.P, c["nu"], c["kT"], c["I_0"], c["R"], n.distances,
                                            n.transitions_constant, n.E_constant(), n.electrodes[:, 3])], hops, rates=rates)


@pytest.mark.parametrize("rates,tol", [("f64", 1e-9), ("f32", 2e-4)])
@pytest.mark.parametrize("I_0", [-5.0, -0.01, 0.0, 5.0])
def test_sites_that_attract(engine_lib, oracle_mod, rates, tol, I_0):
    """With I_0 < 0 a site's rate onto itself is 0, not K: it counts in the
    total, so in the clock and the step.  (Tolerances: test_meanfield.py.)"""
    n = workloads.plain_network(2)
    r = _run(n, 12, rates, I_0=I_0)
    o = oracle_mod.prob_simulate(n.N, n.P, n.nu, n.kT, I_0, n.R, np.full(n.N, 0.5), n.distances, n.E_constant(),
                                 n.site_energies(), n.transitions_constant, 12)
    assert r["status"][0] == 0
    np.testing.assert_allclose(r["time"][0], o["time"], rtol=tol)
    np.testing.assert_allclose(r["occupation"][0], o["occupation"], atol=tol, rtol=0)
    np.testing.assert_allclose(r["electrode_occupation"][0], o["electrode_occupation"],
                               atol=tol * max(1.0, np.abs(o["electrode_occupation"]).max()), rtol=0)


@pytest.mark.parametrize("rates", ["f64", "f32"])
@pytest.mark.parametrize("kT", [0.0, -0.0, np.nan, 5e-324])
def test_no_temperature_no_result(engine_lib, rates, kT):
    from kmc_dn_gb300._native import KMC_ERR_NONFINITE
    r = _run(workloads.plain_network(2), 12, rates, kT=kT)
    assert r["status"][0] == KMC_ERR_NONFINITE and r["iterations"][0] == 0

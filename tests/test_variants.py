"""Launch shapes that take the engine's other register variants: every chain
runs as it does alone."""
import numpy as np
import pytest

from kmc_dn_gb300 import workloads

pytestmark = pytest.mark.gpu


def _net(N, P, seed):
    L = float(np.sqrt(N / workloads.DENSITY))
    rng = np.random.Generator(np.random.PCG64(1000 * seed + N))
    return workloads.make_network(rng, N, max(1, N // 10), L, L, workloads.perimeter_electrodes(L, P),
                                  voltages=rng.uniform(-1, 1, P), cells=30)


def _same_as_alone(per_sm, N, P, lanes, mode, two, hops=40, **kw):
    """per_sm warps or blocks an SM, their chains from one network or two."""
    import torch
    from kmc_dn_gb300.engine import Batch, TableSet, TableSpec
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = per_sm * sms * max(1, 32 // lanes)
    nets = [_net(N, P, s) for s in range(2 if two else 1)]
    tables = TableSet([TableSpec.from_network(x) for x in nets], pair_mode=mode)
    E = [x.E_constant() for x in nets]

    def run(streams, **kw):
        of = [int(s) % len(nets) for s in streams]
        b = Batch(tables, of, [nets[t].kT for t in of], [E[t] for t in of], [nets[t].electrodes[:, 3] for t in of],
                  [nets[t].occupation.astype(np.uint8) for t in of], hops, seed=9, lanes=lanes, reanchor=16,
                  streams=np.asarray(streams), hop_log=True, **kw)
        return b.run().results()

    many = run(range(n), **kw)
    assert not many["status"].any()
    for c in (0, 1, n // 2, n - 1):
        one = run([c])
        for k in ("time", "n_pairs", "occupation", "electrode_occupation", "hop_log"):
            np.testing.assert_array_equal(many[k][c], one[k][0], err_msg=k)


@pytest.mark.parametrize("per_sm,N,P,lanes,mode,two", [
    (5, 30, 8, 128, "table", False),       # staged table, five chains an SM
    (5, 100, 8, 128, "table", True),       # tables in memory, sums stored
    (5, 200, 5, 128, "table", True), (7, 200, 8, 128, "table", True),      # and not stored
    (8, 200, 8, 128, "table", True),       # two full waves
    (5, 150, 3, 128, "positions", False), (10, 60, 8, 64, "positions", False), (14, 121, 8, 64, "table", True),
    (1, 100, 8, 512, "positions", False), (2, 100, 8, 512, "positions", False), (3, 240, 8, 256, "positions", False)])
def test_block_groups_in_a_crowd(engine_lib, per_sm, N, P, lanes, mode, two):
    _same_as_alone(per_sm, N, P, lanes, mode, two)


@pytest.mark.parametrize("per_sm,N,lanes,mode,two,kw", [
    (20, 12, 8, "table", True, {}), (20, 12, 8, "table", False, {}), (20, 30, 16, "positions", False, {}),
    (20, 40, 16, "positions", False, {}), (20, 30, 16, "table", True, {}), (17, 60, 32, "table", True, {}),
    (20, 12, 8, "table", True, {"persistent": True}), (17, 60, 32, "positions", False, {"persistent": True})])
def test_warp_slices_in_a_crowd(engine_lib, per_sm, N, lanes, mode, two, kw):
    """More warps than the SMs hold at 128 registers."""
    _same_as_alone(per_sm, N, 8, lanes, mode, two, **kw)

"""A batch's device state: complete when the constructor returns, and read as
it is when a launch starts."""
import types

import numpy as np
import pytest
import torch

from kmc_dn_gb300 import _native, engine, workloads


def _positions_spec(N, P, seed=0):
    L = float(np.sqrt(N / workloads.DENSITY))
    rng = np.random.Generator(np.random.PCG64(seed))
    return workloads.make_network(rng, N, N // 10, L, L, workloads.perimeter_electrodes(L, P),
                                  voltages=rng.uniform(-1, 1, P), cells=30)


def _make(net, hops, tables, **kw):
    n = len(hops)
    return engine.Batch(tables, [0] * n, [net.kT] * n, [net.E_constant()] * n, [net.electrodes[:, 3]] * n,
                        [net.occupation.astype(np.uint8)] * n, hops, seed=3, **kw)


def _on_cpu(monkeypatch):
    """Batches of plain CPU tensors (nothing can be launched)."""
    monkeypatch.setattr(engine, "device", lambda dev=None: torch.device("cpu"))
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: types.SimpleNamespace(multi_processor_count=152))


EVERYTHING = dict(record=_native.RECORD_GO, hop_log=True, hop_rates=True, count_select_mismatch=True,
                  measure_drift=True, persistent=True, flux=True)


def test_fills_come_before_the_blocking_copy(monkeypatch):
    """Every fill of optional state is queued before the one copy that waits
    for the stream (here: plain tensors, calls in order)."""
    _on_cpu(monkeypatch)
    net = _positions_spec(12, 4)
    tables = engine.TableSet([engine.TableSpec.from_network(net)], pair_mode="positions")
    calls = []

    def logged(owner, name):
        f = getattr(owner, name)
        monkeypatch.setattr(owner, name, lambda *a, **k: (calls.append(name), f(*a, **k))[1])

    for owner, name in ((torch, "zeros"), (torch, "full"), (torch, "ones"), (engine._Pack, "upload")):
        logged(owner, name)
    u = np.full(40, 0.5)
    b = _make(net, [20, 20], tables, replay=[u, u], **EVERYTHING)
    assert calls.count("zeros") >= 8 and "full" in calls
    assert calls[-1] == "upload" and calls.count("upload") == 1
    assert torch.all(b.hop_log == -1) and not b.traffic.any() and not b.flux_time.any()


def test_launch_covers_budgets_as_they_are(monkeypatch):
    """Budgets written after construction count, also by a writer that torch
    does not see (a kernel, another library, the tensor's .data)."""
    _on_cpu(monkeypatch)
    net = _positions_spec(12, 4)
    tables = engine.TableSet([engine.TableSpec.from_network(net)], pair_mode="positions")
    for reanchor in (1024, 700):
        b = _make(net, [20, 30], tables, reanchor=reanchor)
        segs = []
        monkeypatch.setattr(b, "_launch_bins", lambda seg, streams: segs.append(b._struct(b._bins[0], seg)))
        for write in (lambda: None, lambda: b.hops_total.data.fill_(10**6), lambda: b.hops_total.numpy().fill(10**7)):
            write()
            b.launch()
            assert segs[-1].max_hops_per_launch >= b.hops_total.max()
            assert segs[-1].max_hops_per_launch % reanchor == 0
        b.launch(5000)
        assert segs[-1].max_hops_per_launch == -(-5000 // reanchor) * reanchor


def test_pack_sends_large_arrays_from_where_they_are():
    """Large arrays between small ones, first and last; read-only ones too."""
    big = np.arange(engine._Pack._LARGE // 8 + 3, dtype=np.float64)
    frozen = big[::-1].copy()
    frozen.setflags(write=False)
    for order in ("Bsb", "sBs", "BbB", "sss", "B", "bs"):
        pk, want = engine._Pack(), {}
        for k, c in enumerate(order):
            a = {"B": big + k, "b": frozen, "s": np.arange(5 + k, dtype=np.int32)}[c]
            want[f"a{k}"] = a
            pk.add(f"a{k}", a, torch.float64 if c in "Bb" else torch.int32)
        pk.zeros("z", 7, torch.int64)
        t = pk.upload(torch.device("cpu"))
        for k, a in want.items():
            np.testing.assert_array_equal(t[k].numpy(), a)
        assert not t["z"].any()
        host = pk.download("a0", "z")
        np.testing.assert_array_equal(host["a0"], want["a0"])


@pytest.mark.gpu
def test_budgets_raised_in_place_are_run(engine_lib):
    net = _positions_spec(24, 5, seed=1)
    tables = engine.TableSet([engine.TableSpec.from_network(net)])
    want = _make(net, [3000, 1500], tables).run().results()
    b = _make(net, [40, 20], tables)
    b.hops_total.data.copy_(torch.tensor([3000, 1500]))
    got = b.run().results()
    assert got["hops_done"].tolist() == [3000, 1500] and not got["status"].any()
    np.testing.assert_array_equal(got["time"], want["time"])


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [8, 32, 64])
def test_batch_built_on_one_stream_runs_on_another(engine_lib, lanes, monkeypatch):
    """With work queued on the constructing stream behind the upload, a launch
    on a stream of its own keeps what it records."""
    net, hops = _positions_spec(24, 5, seed=1), [300, 200]
    tables = engine.TableSet([engine.TableSpec.from_network(net)])
    want = _make(net, hops, tables, lanes=lanes, **EVERYTHING).run().results()
    upload = engine._Pack.upload

    def slow(self, dev):
        t = upload(self, dev)
        torch.cuda._sleep(40_000_000)       # 20 ms on the current stream
        return t

    monkeypatch.setattr(engine._Pack, "upload", slow)
    build, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(build):
        b = _make(net, hops, tables, lanes=lanes, **EVERYTHING)
    b.launch(stream=other)
    got = b.results()
    for k in ("time", "hops_done", "n_pairs", "status", "energy_drift"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    for k in ("occupation", "electrode_occupation", "traffic", "occ_time", "flux_time", "hop_log", "hop_rates"):
        for c in range(2):
            np.testing.assert_array_equal(got[k][c], want[k][c], err_msg=k)


@pytest.mark.gpu
def test_table_build_stages_a_bounded_part(engine_lib):
    """The FP64 tables of a set pass through a staging buffer whose size does
    not grow with their number (the high-water mark of the device's memory
    pool), and each comes out as if it were built alone."""
    import ctypes as C
    cu = C.CDLL("libcuda.so.1")
    pool, high, zero = C.c_void_p(), C.c_uint64(), C.c_uint64(0)
    USED_MEM_HIGH = 8
    S, n = 900, 16                              # 13 MB of FP64 tables a geometry, 207 MB in all
    rng = np.random.default_rng(2)
    N, P = S - 7, 7
    d = [rng.uniform(0.1, 3.0, (S, S)) for _ in range(3)]
    tc = [rng.uniform(0.0, 1.0, (S, S)) for _ in range(3)]
    specs = [engine.TableSpec(N, P, 0.5 + k, 3.0, 0.25, d[k % 3], tc[(k + 1) % 3]) for k in range(n)]
    specs.insert(5, engine.TableSpec(1, 2, 1.0, 1.0, 1.0, d[0][:3, :3], tc[0][:3, :3]))
    engine.TableSet(specs[:1])
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), torch.cuda.current_device()) == 0
    assert cu.cuMemPoolSetAttribute(pool, USED_MEM_HIGH, C.byref(zero)) == 0
    ts = engine.TableSet(specs)
    assert cu.cuMemPoolGetAttribute(pool, USED_MEM_HIGH, C.byref(high)) == 0
    assert 16 * S * S <= high.value <= 70 << 20
    off = ts.tab_off.cpu().numpy()
    for k in (0, 4, 5, 6, 9, 16):
        one = engine.TableSet(specs[k:k + 1]).tab_LB
        assert torch.equal(ts.tab_LB[int(off[k]):int(off[k]) + one.numel()], one)

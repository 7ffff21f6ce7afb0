"""Mean-field relaxation on the device: the Go library's ``probSimulate``
(goSimulation/probabilitySimulation.go:53-157), reached from the reference as
``kmc.go_simulation(hops=1000, goSpecificFunction="wrapperSimulateProbability")``
(dn_search.py:49-52 uses it as the cheapest first search stage).

The state is the occupation probability of every acceptor; each iteration
moves the expected charge along the expected rates and advances the time by
0.98 of the largest admissible step.  ``run`` relaxes a batch of networks in
one launch (one thread block per network, kmc_mf_run); ``simulate_probability``
takes ``callGoSimulation``'s keyword set and returns what it returns.
"""
from __future__ import annotations

import ctypes as C

import numpy as np

from . import _native
from ._native import KmcMfBatch, check, lib
from .engine import _Pack

__all__ = ["Network", "MeanFieldBatch", "run", "simulate_probability", "max_sites"]

RATES = {"f64": _native.MF_RATES_F64, "f32": _native.MF_RATES_F32}


class Network:
    """One network's inputs: sizes, constants, S x S distances and
    transition constants, N constant energies, P electrode voltages."""

    def __init__(self, N, P, nu, kT, I_0, R, distances, transitions_constant, E_constant, voltages):
        self.N, self.P = int(N), int(P)
        self.nu, self.kT, self.I_0, self.R = float(nu), float(kT), float(I_0), float(R)
        S = self.N + self.P

        def as_shape(a, shape):
            # the caller's own array where it has the form: networks given the
            # same arrays keep sharing them
            a = np.ascontiguousarray(a, np.float64)
            return a if a.shape == shape else a.reshape(shape)

        self.distances = as_shape(distances, (S, S))
        self.transitions_constant = as_shape(transitions_constant, (S, S))
        self.E_constant = as_shape(E_constant, (self.N,))
        self.voltages = as_shape(voltages, (self.P,))


def max_sites(rates="f64"):
    """Largest network (acceptors + electrodes) one block holds."""
    return int(lib().kmc_mf_max_sites(RATES[rates]))


class MeanFieldBatch:
    """Device buffers of one batch of networks, launched with ``launch`` as
    often as wanted (each launch restarts from ``start``)."""

    def __init__(self, networks, hops, *, rates="f64", record=False, start=0.5, dev=None):
        import torch
        nets = list(networks)
        n = len(nets)
        if n == 0:
            raise ValueError("no networks")
        h = np.broadcast_to(np.asarray(hops, dtype=np.int64), (n,)).copy()
        if (h < 0).any():
            raise ValueError("hops must be >= 0")
        self.nets, self.n, self.record = nets, n, bool(record)
        self.mode = RATES[rates]
        Ns = np.array([x.N for x in nets], np.int32)
        Ps = np.array([x.P for x in nets], np.int32)
        Ss = Ns.astype(np.int64) + Ps
        lim = max_sites(rates)
        if Ss.max() > lim:
            raise ValueError(f"a network has {int(Ss.max())} sites; the {rates} kernel holds at most {lim}")
        # pair blocks, shared by identity
        pair_off = np.zeros(n, np.int64)
        blocks, seen, off = [], {}, 0
        for c, x in enumerate(nets):
            key = (id(x.distances), id(x.transitions_constant))
            at = seen.get(key)
            if at is None:
                seen[key] = at = off
                blocks.append((x.distances, x.transitions_constant))
                off += x.distances.size
            pair_off[c] = at
        self.site_off = np.concatenate([[0], np.cumsum(Ss)[:-1]]).astype(np.int64)
        self.el_off = np.concatenate([[0], np.cumsum(Ps.astype(np.int64))[:-1]]).astype(np.int64)
        self.tr_off = np.concatenate([[0], np.cumsum(Ss * Ss)[:-1]]).astype(np.int64)
        self.S = Ss
        n_sites = int(Ss.sum())
        # site pools: acceptors, then electrodes, of each network
        acceptor = np.arange(n_sites) - np.repeat(self.site_off, Ss) < np.repeat(Ns, Ss)
        ec = np.zeros(n_sites)
        se = np.zeros(n_sites)
        ec[acceptor] = np.concatenate([x.E_constant for x in nets])
        se[~acceptor] = np.concatenate([x.voltages for x in nets])
        occ = np.zeros(n_sites)
        if np.ndim(start) == 0:
            occ[acceptor] = start
        else:                     # a vector for every network
            for o, x in zip(self.site_off, nets):
                occ[o:o + x.N] = start
        self.dev = d = torch.device(dev if dev is not None else "cuda")
        f64, i64, i32 = torch.float64, torch.int64, torch.int32
        pk = self._pack = _Pack()
        for k, a, dt in (("N", Ns, i32), ("P", Ps, i32), *((k, [getattr(x, k) for x in nets], f64)
                                                           for k in ("nu", "kT", "I_0", "R")),
                         ("pair_off", pair_off, i64), ("distances", np.concatenate([b[0].ravel() for b in blocks]), f64),
                         ("transitions_constant", np.concatenate([b[1].ravel() for b in blocks]), f64),
                         ("site_off", self.site_off, i64), ("E_constant", ec, f64), ("el_off", self.el_off, i64),
                         ("hops", h, i64), ("traffic_off", self.tr_off, i64), ("se0", se, f64), ("occ0", occ, f64),
                         # results from here on
                         ("site_energies", se, f64), ("occupation", occ, f64)):
            pk.add(k, a, dt)
        pk.zeros("electrode_occupation", max(int(Ps.sum()), 1), f64)
        pk.zeros("time", n, f64)
        pk.zeros("iterations_done", n, i64)
        pk.zeros("status", n, i32)
        if record:
            pk.zeros("average_occupation", n_sites, f64)
            pk.zeros("traffic", int((Ss * Ss).sum()), f64)
        self.t = t = pk.upload(d)
        self._se0, self._occ0 = t.pop("se0"), t.pop("occ0")
        if not record:
            t.pop("traffic_off")
        self._last = "traffic" if record else "status"
        b = KmcMfBatch()
        b.n_chains, b.max_sites, b.rates, b.record = n, int(Ss.max()), self.mode, int(self.record)
        for name, _ in KmcMfBatch._fields_[4:]:
            v = t.get(name)
            setattr(b, name, v.data_ptr() if v is not None else None)
        self.b = b
        self.pairs_per_iteration = int((Ss * Ss).sum())

    def reset(self):
        """Back to the starting probabilities (the traffic and occupancy sums
        of record mode are zeroed too)."""
        t = self.t
        t["occupation"].copy_(self._occ0)
        t["site_energies"].copy_(self._se0)
        if self.record:
            t["traffic"].zero_()
            t["average_occupation"].zero_()

    def launch(self, stream=None):
        import torch
        st = stream if stream is not None else torch.cuda.current_stream(self.dev)
        check(lib().kmc_mf_run(C.byref(self.b), C.c_void_p(st.cuda_stream)))

    def results(self):
        import torch
        torch.cuda.synchronize(self.dev)
        r = self._pack.download("site_energies", self._last)
        nets, so, eo_off = self.nets, self.site_off, self.el_off
        occ_h, se_h, eo_h = r["occupation"], r["site_energies"], r["electrode_occupation"]
        out = dict(time=r["time"], status=r["status"], iterations=r["iterations_done"],
                   occupation=[occ_h[o:o + x.N] for o, x in zip(so, nets)],
                   site_energies=[se_h[o:o + x.N] for o, x in zip(so, nets)],
                   electrode_occupation=[eo_h[o:o + x.P] for o, x in zip(eo_off, nets)])
        if self.record:
            tr_h, avg_h = r["traffic"], r["average_occupation"]
            out["traffic"] = [tr_h[o:o + s * s].reshape(s, s) for o, s in zip(self.tr_off, self.S)]
            out["average_occupation"] = [avg_h[o:o + x.N] for o, x in zip(so, nets)]
        return out


def run(networks, hops, *, rates="f64", record=False, start=0.5, dev=None, stream=None):
    """Relax every network for ``hops`` iterations (int or one per network).

    Networks that share the same ``distances`` and ``transitions_constant``
    arrays (the same objects) share one pair block on the device.  Returns a
    dict of host arrays: time[C], occupation (list of N-vectors),
    electrode_occupation (list of P-vectors), site_energies (list of
    N-vectors), status[C], iterations[C] and, with record, traffic (list of
    S x S) and average_occupation (list of N-vectors, time-weighted sums)."""
    b = MeanFieldBatch(networks, hops, rates=rates, record=record, start=start, dev=dev)
    b.launch(stream)
    return b.results()


def simulate_probability(N_acceptors, N_electrodes, nu, kT, I_0, R, time, occupation, distances,
                         E_constant, site_energies, transitions_constant, transitions=None,
                         problist=None, electrode_occupation=None, hops=1000, record=False,
                         goSpecificFunction="wrapperSimulateProbability", prune_threshold=0.0,
                         rates="f64", **_ignored):
    """Drop-in for ``callGoSimulation(..., goSpecificFunction=
    "wrapperSimulateProbability")`` (goSimulation/pythonBind.py:49-92).

    The relaxation starts from 0.5 on every acceptor
    (simulationWrapper.go:229-232).  As through the ctypes bridge, the
    returned occupation and electrode_occupation are the Go slices' values
    truncated to int (pythonBind.py:85-86); the time and, with record, the
    traffic and time-weighted occupation sums are returned as floats."""
    N, P = int(N_acceptors), int(N_electrodes)
    S = N + P
    se = np.asarray(site_energies, np.float64).reshape(S)
    net = Network(N, P, nu, kT, I_0, R, distances, transitions_constant, E_constant, se[N:])
    r = run([net], int(hops), rates=rates, record=record)
    if r["status"][0] != 0:
        raise _native.KmcError(int(r["status"][0]), "mean-field relaxation stopped: total rate zero or non-finite")
    t = float(r["time"][0])
    occ = np.array([int(x) for x in r["occupation"][0]])
    eo = np.array([int(x) for x in r["electrode_occupation"][0]])
    if not record:
        return t, occ, eo
    return t, occ, eo, r["traffic"][0], r["average_occupation"][0]

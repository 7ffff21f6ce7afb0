"""The work a user has this framework do, as cases that can be timed.

Each case is one call (or one short sequence of calls) through the public
Python API, on seeded synthetic networks with the shapes and value
distributions of the workloads in ``kmc_dn_gb300/workloads.py``: 20 x 20
boxes of 30 acceptors and boxes of the same density, 10 % donors, electrodes
on the boundary, I_0 = 50 kT, ab = R.  ``kind`` says which calls:

one       one network simulated by its own ``kmc_dn`` object: what the class
          is for, and what an interactive user or a sequential search does.
          ``how``: "cuda" (FP32 engine), "go" (the Go library's semantics),
          "python" (the numba loop's semantics, FP64 kernel).
many64    FP64 reference statistics: ``simulate_f64_many``, independent
          chains of one network.
ensemble  a voltage ensemble on one resident geometry: constant energies
          superposed on the device, one ``Batch``, results left on the device.
search    a dopant search's population: one network per candidate, all with
          their own geometry, through ``parrallelSimulation``.
serve     a voltage-search population sent to a ``serving.Server``.
large     N ~ 1000 networks in positions mode, one geometry per chain.
relax     the mean-field relaxation of a population (``meanfield.run``),
          FP64 rates (the reference's arithmetic) or FP32 rates.
basis     the Laplace basis fields of a new electrode layout on the device,
          sampled at the acceptors.
"""
import copy
import math

import numpy as np
import torch

from kmc_dn_gb300 import _native, engine, meanfield, workloads
from kmc_dn_gb300.kmc_dn import kmc_dn
from kmc_dn_gb300.laplace import BasisFields, solve_basis_fields_gpu
from kmc_dn_gb300.parallel import parrallelSimulation
from kmc_dn_gb300.serving import Server


def listed():
    return [
        # a first look at one small network: few hops, so what the call itself costs counts
        {"name": "one_n30", "kind": "one", "how": "cuda", "N": 30, "P": 8, "hops": 1000, "record": False},
        # one mid-size network with traffic and occupancy recorded, the Go library's semantics
        {"name": "one_n100_go_record", "kind": "one", "how": "go", "N": 100, "P": 8, "hops": 10000, "record": True},
        # the reference's own loop semantics (python_simulation) on the plain network
        {"name": "one_n30_fp64", "kind": "one", "how": "python", "N": 30, "P": 8, "hops": 2000, "record": True},
        # FP64 statistics with the flux companion estimate, as the precision comparison takes them
        {"name": "many_fp64_n60", "kind": "many64", "N": 60, "P": 8, "chains": 256, "hops": 300, "flux": True},
        # the benchmark's ensemble: 4096 voltage vectors on the plain network, one temperature
        {"name": "ensemble_n30", "kind": "ensemble", "N": 30, "P": 8, "chains": 4096, "hops": 10240,
         "spread_kT": False, "record": False, "pair_mode": "table"},
        # a population of candidate networks of uneven size
        {"name": "search_uneven", "kind": "search", "chains": 384, "N_lo": 10, "N_hi": 200, "hops": 2000},
        # short serving requests: a small population on a small geometry, a full one on the largest
        {"name": "serve_n60", "kind": "serve", "N": 60, "P": 8, "chains": 64, "hops": 10000},
        {"name": "serve_n240", "kind": "serve", "N": 240, "P": 8, "chains": 512, "hops": 4000},
        # large networks, each with its own geometry
        {"name": "large_n1000", "kind": "large", "N": 1000, "chains": 256, "hops": 1024},
        # the search's first stage: mean field in the reference's precision, a small population
        {"name": "relax_fp64", "kind": "relax", "N": 30, "P": 8, "networks": 64, "iterations": 1000, "rates": "f64"},
        # a large population with FP32 rates
        {"name": "relax_fp32", "kind": "relax", "N": 30, "P": 8, "networks": 2048, "iterations": 1000, "rates": "f32"},
        # a new electrode layout on the reference's default mesh (99 cells a side)
        {"name": "basis_99", "kind": "basis", "P": 8, "N": 30, "nx": 99, "ny": 99},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "one", "many64", "ensemble", "ensemble", "search", "serve", "serve", "large",
                       "relax", "relax", "basis"])
    P = rng.randint(4, 12)
    if kind == "one":
        how = rng.choice(["cuda", "go", "python"])
        N = _log_int(rng, 10, 240)
        hops = _log_int(rng, 300, 10000 if how != "python" else min(2000, max(301, 4000000 // (N + P) ** 2)))
        return {"kind": kind, "how": how, "N": N, "P": P, "hops": hops, "record": rng.random() < 0.5}
    if kind == "many64":
        N, n = _log_int(rng, 10, 120), _log_int(rng, 16, 512)
        return {"kind": kind, "N": N, "P": P, "chains": n,
                "hops": rng.randint(50, max(60, min(300, 300000000 // (n * (N + P) ** 2)))), "flux": rng.random() < 0.5}
    if kind == "ensemble":
        N = rng.randint(10, 100)
        return {"kind": kind, "N": N, "P": P, "chains": _log_int(rng, 100, 8192 if N <= 40 else 1024),
                "hops": 1024 * rng.randint(1, 6), "spread_kT": rng.random() < 0.5,
                "record": rng.random() < 0.25, "pair_mode": rng.choice(["table", "table", "positions"])}
    if kind == "search":
        lo = _log_int(rng, 10, 100)
        return {"kind": kind, "chains": _log_int(rng, 20, 400), "N_lo": lo, "N_hi": rng.randint(lo, 200),
                "hops": _log_int(rng, 300, 3000)}
    if kind == "serve":
        N = _log_int(rng, 30, 240)
        hops = _log_int(rng, 2000, 30000 if N <= 60 else 8000)
        return {"kind": kind, "N": N, "P": 8, "chains": rng.randint(32, 512 if N <= 120 else 256), "hops": hops}
    if kind == "large":
        return {"kind": kind, "N": _log_int(rng, 400, 1000), "chains": _log_int(rng, 8, 256),
                "hops": rng.randint(200, 1024)}
    if kind == "relax":
        rates = rng.choice(["f64", "f32"])
        return {"kind": kind, "N": rng.randint(10, 80), "P": P, "networks": _log_int(rng, 1, 512),
                "iterations": _log_int(rng, 100, 1000), "rates": rates}
    return {"kind": kind, "P": P, "N": _log_int(rng, 10, 240), "nx": rng.randint(30, 150), "ny": rng.randint(30, 150)}


# ---------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------

_BASES = {}


def _layout(P):
    """P electrodes on the unit square: two per edge for 8, else evenly spaced."""
    return np.asarray(workloads.edge_thirds(1.0) if P == 8 else workloads.perimeter_electrodes(1.0, P), np.float64)


def _base(P):
    """One ``kmc_dn`` per electrode layout on the unit square: the Laplace
    problem is scale invariant, so every candidate network of that layout
    shares its basis fields."""
    if P not in _BASES:
        el = np.zeros((P, 4))
        el[:, :2] = _layout(P)
        _BASES[P] = kmc_dn(10, 1, 1.0, 1.0, 0, electrodes=el, I_0=50, a=1, seed=0)
    return _BASES[P]


def _candidate(rng, N, P):
    """A ``kmc_dn`` with new random dopants and voltages, as the searches make
    them: a copy with other acceptors, donors and electrode voltages."""
    base = _base(P)
    L = float(np.sqrt(N / workloads.DENSITY))
    dn = copy.copy(base)
    dn.calc_E_constant = dn.calc_E_constant_V_comp      # the copy's own method
    dn.rng = rng
    dn.xdim = dn.ydim = L
    bf = base.basis_fields
    dn.basis_fields = BasisFields(bf.fields, L, L, bf.nx, bf.ny, 2)
    dn.electrodes = np.zeros((P, 4))
    dn.electrodes[:, :2] = L * _layout(P)
    dn.electrodes[:, 3] = rng.uniform(-1.0, 1.0, P)
    dn.M = max(1, int(round(0.1 * N)))
    dn.donors = L * rng.random((dn.M, 3)) * np.array([1.0, 1.0, 0.0])
    dn.load_acceptors(L * rng.random((N, 3)) * np.array([1.0, 1.0, 0.0]))
    dn.update_V()
    return dn


def _network(rng, N, P):
    L = float(np.sqrt(N / workloads.DENSITY))
    return workloads.make_network(rng, N, max(1, int(round(0.1 * N))), L, L, L * _layout(P),
                                  voltages=rng.uniform(-1.0, 1.0, P), I_0=50.0)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    kind = case["kind"]
    st = {"case": case, "kind": kind, "seed": seed + 1}
    if kind == "one":
        st["dn"] = _candidate(rng, case["N"], case["P"])
        st["occupation"] = st["dn"].occupation.copy()
    elif kind == "many64":
        net = _network(rng, case["N"], case["P"])
        st["chains"] = [dict(N=net.N, P=net.P, nu=net.nu, kT=net.kT, I_0=net.I_0, R=net.R, occupation=net.occupation,
                             distances=net.distances, transitions_constant=net.transitions_constant,
                             E_constant=net.E_constant(), site_energies=net.site_energies())
                        for _ in range(case["chains"])]
        st["seeds"] = [int(s) for s in rng.integers(0, 2 ** 62, case["chains"])]
    elif kind == "ensemble":
        n = case["chains"]
        st["net"] = net = _network(rng, case["N"], case["P"])
        st["V"] = rng.uniform(-1.0, 1.0, (n, net.P))
        st["kT"] = np.exp(rng.uniform(np.log(0.5), np.log(5.0), n)) if case["spread_kT"] else np.ones(n)
        st["occupation"] = np.tile(net.occupation.astype(np.uint8), (n, 1))
        st["tables"] = engine.TableSet([engine.TableSpec.from_network(net)], pair_mode=case["pair_mode"])
    elif kind == "search":
        # the sizes are the case's, spread evenly over its range in no order
        lo, hi = case["N_lo"], case["N_hi"]
        sizes = np.random.Generator(np.random.PCG64(1)).permutation(
            np.linspace(lo, hi, case["chains"]).round().astype(int))
        st["dns"] = [_candidate(rng, int(N), 4 + k % 9) for k, N in enumerate(sizes)]
    elif kind == "serve":
        net = _network(rng, case["N"], case["P"])
        st["server"] = Server([net])
        st["V"] = rng.uniform(-1.0, 1.0, (case["chains"], net.P))
    elif kind == "large":
        # a few geometries, each with several voltage vectors
        nets = [_network(rng, case["N"], 8) for _ in range(4)]
        n = case["chains"]
        st["tab"] = np.arange(n) % len(nets)
        st["tables"] = engine.TableSet([engine.TableSpec.from_network(net) for net in nets], pair_mode="positions")
        V = rng.uniform(-1.0, 1.0, (n, 8))
        st["E"] = [nets[t].E_constant(v) for t, v in zip(st["tab"], V)]
        st["V"] = V
        st["occupation"] = [nets[t].occupation.astype(np.uint8) for t in st["tab"]]
    elif kind == "relax":
        net = _network(rng, case["N"], case["P"])
        V = rng.uniform(-1.0, 1.0, (case["networks"], net.P))
        st["nets"] = [meanfield.Network(net.N, net.P, net.nu, net.kT, net.I_0, net.R, net.distances,
                                        net.transitions_constant, net.E_constant(v), v) for v in V]
    elif kind == "basis":
        el = np.zeros((case["P"], 4))
        L = 20.0
        # the layout turned along the edges a little, so that every seed is another layout
        s = (np.arange(case["P"]) + rng.uniform(0.3, 0.7, case["P"])) * 4.0 / case["P"]
        el[:, :2] = [[(t, 0.0), (1.0, t), (1.0 - t, 1.0), (0.0, 1.0 - t)][e]
                     for e, t in ((int(x), x - int(x)) for x in s)]
        el[:, :2] *= L
        st["L"], st["electrodes"] = L, el
        st["points"] = L * rng.random((case["N"], 2))
    else:
        raise ValueError(kind)
    return st


def run(st):
    case, kind = st["case"], st["kind"]
    if kind == "one":
        dn = st["dn"]
        dn.occupation = st["occupation"].copy()
        if case["how"] == "cuda":
            dn.cuda_simulation(hops=case["hops"], record=case["record"], seed=st["seed"])
        elif case["how"] == "go":
            dn.go_simulation(hops=case["hops"], record=case["record"], seed=st["seed"])
        else:
            dn.python_simulation(hops=case["hops"], record=case["record"], seed=st["seed"])
        out = {"time": float(dn.time), "occupation": np.asarray(dn.occupation),
               "electrode_occupation": np.asarray(dn.electrode_occupation), "current": np.asarray(dn.current)}
        if case["record"]:
            out["traffic"] = np.asarray(dn.traffic)
            out["average_occupation"] = np.asarray(dn.average_occupation)
        return out
    if kind == "many64":
        r = engine.simulate_f64_many(st["chains"], case["hops"], st["seeds"], record=True, flux=case["flux"])
        out = {"time": r[0], "electrode_occupation": np.stack(r[1]), "status": r[2], "occupations_in_time": np.stack(r[3])}
        if case["flux"]:
            out["flux"] = np.stack(r[4])
        return out
    if kind == "ensemble":
        net, n = st["net"], case["chains"]
        ec, ve = engine.superpose(net.basis, net.comp, st["V"], net.mu)
        b = engine.Batch(st["tables"], np.zeros(n, np.int32), st["kT"], None, None, st["occupation"],
                         np.full(n, case["hops"]), seed=st["seed"], E_constant_dev=ec, el_energy_dev=ve,
                         record=_native.RECORD_NUMBA if case["record"] else _native.RECORD_NONE)
        b.run()
        out = {"time": b.time, "electrode_occupation": b.electrode_occupation, "occupation": b.occupation,
               "status": b.status, "hops_done": b.hops_done, "n_pairs": b.n_pairs, "E_constant": ec}
        if case["record"]:
            out["occ_time"], out["traffic"] = b.occ_time, b.traffic
        return out
    if kind == "search":
        p = parrallelSimulation(seed=st["seed"])
        for dn in st["dns"]:
            p.addSimulation(dn, case["hops"])
        r = p.runSimulation()
        return {"time": np.array([dn.parrallel_results[0][0] for dn in st["dns"]]),
                "electrode_occupation": np.concatenate(r["electrode_occupation"]),
                "current": np.concatenate([dn.parrallel_results[0][2] for dn in st["dns"]]),
                "occupation": np.concatenate(r["occupation"]), "status": r["status"], "hops_done": r["hops_done"]}
    if kind == "serve":
        server = st["server"]
        req = server.submit(0, st["V"], case["hops"], st["seed"])
        server.run_sync()
        r = req.future.result()
        return {k: r[k] for k in ("currents", "time", "electrode_occupation", "status", "hops_done")}
    if kind == "large":
        b = engine.Batch(st["tables"], st["tab"], np.ones(case["chains"]), st["E"], st["V"], st["occupation"],
                         np.full(case["chains"], case["hops"]), seed=st["seed"])
        r = b.run().results()
        return {"time": r["time"], "electrode_occupation": np.stack(r["electrode_occupation"]),
                "occupation": np.stack(r["occupation"]), "status": r["status"], "n_pairs": r["n_pairs"]}
    if kind == "relax":
        r = meanfield.run(st["nets"], case["iterations"], rates=case["rates"])
        return {"time": r["time"], "occupation": np.stack(r["occupation"]), "status": r["status"],
                "electrode_occupation": np.stack(r["electrode_occupation"]), "iterations": r["iterations"],
                "site_energies": np.stack(r["site_energies"])}
    bf = solve_basis_fields_gpu(st["L"], st["L"], st["electrodes"], case["nx"], case["ny"])
    return {"fields": bf.fields, "basis": bf.sample(st["points"])}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def work(case):
    """Pair rates: one per allowed transition and hop (h = 0.9 N holes, the
    mean of these networks), about 12 operations each (energy difference,
    Coulomb term, exponential, running sum), plus the O(N) energy update;
    bytes: tables or positions, energies and state once in, results once out."""
    kind = case["kind"]
    if kind == "basis":
        m = (case["nx"] + 1) * (case["ny"] + 1) * (case["P"] + 1)
        return {"bytes": 8.0 * 2 * m, "flops": 10.0 * m * math.log2(m)}   # two fast sine transforms each way
    if kind == "relax":
        S = case["N"] + case["P"]
        return {"bytes": 8.0 * (2 * S * S + 5 * S * case["networks"]),
                "flops": 14.0 * S * S * case["networks"] * case["iterations"]}
    P = case.get("P", 8)
    if kind == "search":
        lo, hi, n = case["N_lo"], case["N_hi"], case["chains"]
        Ns = np.linspace(lo, hi, 64)
    else:
        n = case.get("chains", 1)
        Ns = np.array([float(case["N"])])
    h = 0.9 * Ns
    pairs = h * (Ns - h) + h * P + P * (Ns - h)
    S = Ns + P
    rec = case.get("record", False)
    per_chain = 5 * Ns + 16 * P + 64 + (8 * S * S if rec else 0)
    tables = {"search": n, "large": 0}.get(kind, 1)
    return {"bytes": float(np.mean(n * per_chain + tables * 16 * S * S + (16 * S * 4 if kind == "large" else 0))),
            "flops": float(n * case["hops"] * np.mean(12 * pairs + 6 * Ns))}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------

def _philox(hop, seeds):
    """Philox4x32-10 words of counter (hop, 0, 0) under 64-bit keys (Salmon et
    al., SC'11): the uniforms the FP64 loop draws for one hop of each chain."""
    m32 = np.uint64(0xFFFFFFFF)
    seeds = np.asarray(seeds, np.uint64)
    k0, k1 = seeds & m32, seeds >> np.uint64(32)
    c = [np.full(seeds.shape, hop, np.uint64)] + [np.zeros(seeds.shape, np.uint64) for _ in range(3)]
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & m32, (a >> np.uint64(32)) ^ c[3] ^ k1, a & m32]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m32, (k1 + np.uint64(0xBB67AE85)) & m32
    u = [(((x << np.uint64(32)) | y) >> np.uint64(11)).astype(np.float64) for x, y in ((c[0], c[1]), (c[2], c[3]))]
    return (u[0] + 0.5) * 2.0 ** -53, (u[1] + 0.5) * 2.0 ** -53


def _hops_64(N, P, nu, kT, I_0, R, occ, d, Ec, Ve, tc, hops, seeds):
    """The hop loop of C chains of one network, dense, in FP64."""
    S, C = N + P, len(seeds)
    ar = np.arange(C)
    with np.errstate(divide="ignore"):
        inv = 1.0 / d[:N, :N]
    np.fill_diagonal(inv, 0.0)
    coul = np.zeros((S, S))
    coul[:N, :N] = I_0 * R * inv
    occ = np.tile(np.asarray(occ, bool), (C, 1))
    e = np.zeros((C, S))
    e[:, N:] = Ve
    full = np.zeros((C, S), bool)       # may be left; electrodes always
    room = np.zeros((C, S), bool)
    full[:, N:] = room[:, N:] = True
    t, eo = np.zeros(C), np.zeros((C, P), np.int64)
    oit, flux, traffic = np.zeros((C, N)), np.zeros((C, P)), np.zeros((C, S, S))
    for hop in range(hops):
        e[:, :N] = Ec - (I_0 * R) * ((~occ).astype(np.float64) @ inv)
        full[:, :N], room[:, :N] = occ, ~occ
        dE = e[:, None, :] - e[:, :, None] - coul
        r = tc * nu * np.exp(-np.maximum(dE, 0.0) / kT)
        r *= full[:, :, None] & room[:, None, :]
        r[:, N:, N:] = 0.0
        cum = np.cumsum(r.reshape(C, -1), axis=1)
        u1, u2 = _philox(hop, seeds)
        ev = np.argmax(cum / cum[:, -1:] >= u2[:, None], axis=1)
        i, j = ev // S, ev % S
        dt = -np.log(1.0 - u1) / cum[:, -1]
        flux += (r[:, :N, N:].sum(1) - r[:, N:, :N].sum(2)) * dt[:, None]
        a = i < N
        occ[ar[a], i[a]] = False
        eo[ar[~a], i[~a] - N] -= 1
        a = j < N
        occ[ar[a], j[a]] = True
        eo[ar[~a], j[~a] - N] += 1
        traffic[ar, i, j] += 1.0
        oit += occ * dt[:, None]
        t += dt
    return t, occ, eo, oit, flux, traffic


def exact(case, seed):
    kind = case["kind"]
    S = case.get("N", 0) + case.get("P", 0)
    if kind == "one" and case["how"] == "python" and S * S * case["hops"] <= 4e7:
        st = prepare(case, seed)
        dn = st["dn"]
        t, occ, eo, oit, _, tr = _hops_64(dn.N, dn.P, dn.nu, dn.kT, dn.I_0, dn.R, st["occupation"], dn.distances,
                                          dn.E_constant, dn.electrodes[:, 3], dn.transitions_constant, case["hops"],
                                          [st["seed"]])
        out = {"time": float(t[0]), "occupation": occ[0], "electrode_occupation": eo[0], "current": eo[0] / t[0]}
        if case["record"]:
            out["traffic"], out["average_occupation"] = tr[0], oit[0] / t[0]
        return out
    if kind == "many64" and S * S * case["hops"] * case["chains"] <= 5e8:
        st = prepare(case, seed)
        c = st["chains"][0]
        t, occ, eo, oit, flux, _ = _hops_64(c["N"], c["P"], c["nu"], c["kT"], c["I_0"], c["R"], c["occupation"],
                                            c["distances"], c["E_constant"], c["site_energies"][c["N"]:],
                                            c["transitions_constant"], case["hops"], st["seeds"])
        out = {"time": t, "electrode_occupation": eo, "status": None, "occupations_in_time": oit}
        if case["flux"]:
            out["flux"] = flux
        return out
    if kind == "relax":
        return _relax_64(case, seed)
    if kind == "basis":
        return _basis_64(case, seed)
    return None     # FP32 trajectories: a rounding decides a hop


def _relax_64(case, seed):
    """The mean-field iteration of all networks at once, in FP64."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nets = prepare(case, seed)["nets"]
    x = nets[0]
    N, P = x.N, x.P
    S, C = N + P, len(nets)
    T = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    d, tc = T(x.distances), T(x.transitions_constant)
    coul = torch.zeros(S, S, dtype=torch.float64, device=dev)
    coul[:N, :N] = x.I_0 * x.R / d[:N, :N].clone().fill_diagonal_(math.inf)
    K = (x.nu * tc).fill_diagonal_(0.0)     # no acceptor hops onto itself
    K[N:, N:] = 0.0
    Ec, V = T([n.E_constant for n in nets]), T([n.voltages for n in nets])
    o = torch.full((C, N), 0.5, dtype=torch.float64, device=dev)
    one = torch.ones(C, P, dtype=torch.float64, device=dev)
    t, eo = torch.zeros(C, dtype=torch.float64, device=dev), torch.zeros(C, P, dtype=torch.float64, device=dev)
    for _ in range(case["iterations"]):
        e = torch.cat([Ec - (1.0 - o) @ coul[:N, :N], V], 1)
        w = torch.cat([o, one], 1)[:, :, None] * torch.cat([1.0 - o, one], 1)[:, None, :]
        r = w * K * torch.exp(-torch.clamp(e[:, None, :] - e[:, :, None] - coul, min=0.0) / x.kT)
        out, inn = r.sum(2), r.sum(1)
        tot = out.sum(1, keepdim=True)
        q = (inn - out)[:, :N] / tot
        nv = o + q
        m = torch.where(nv < 0, o / -q, torch.where(nv > 1, (1.0 - o) / q, torch.ones_like(o))).amin(1, keepdim=True)
        m = torch.clamp(m, max=1.0)
        t += (0.98 * m / tot)[:, 0]
        f = m / tot
        net = (inn - out) * f
        o = torch.clamp(o + net[:, :N], 0.0, 1.0)
        eo += net[:, N:]
    return {"time": t.cpu().numpy(), "occupation": o.cpu().numpy(), "status": None,
            "electrode_occupation": eo.cpu().numpy(), "iterations": None, "site_energies": e[:, :N].cpu().numpy()}


def _basis_64(case, seed):
    """The 5-point system by its sine transforms, and P1 interpolation."""
    st = prepare(case, seed)
    nx, ny, L, el = case["nx"], case["ny"], st["L"], st["electrodes"]
    hx, hy = L / nx, L / ny
    # boundary data: a node belongs to the first electrode whose segment (a
    # tenth of the side either way along its edge) holds it, else to mu
    X, Y = np.meshgrid(np.arange(nx + 1) * hx, np.arange(ny + 1) * hy)
    free = np.zeros(X.shape, bool)
    free[[0, -1]] = free[:, [0, -1]] = True
    grids = np.zeros((len(el) + 1,) + X.shape)
    for k, (ex, ey) in enumerate(el[:, :2]):
        if ex in (0.0, L):
            mine = free & (X == ex) & (Y >= ey - L / 10) & (Y <= ey + L / 10)
        else:
            mine = free & (Y == ey) & (X >= ex - L / 10) & (X <= ex + L / 10)
        grids[k][mine] = 1.0
        free &= ~mine
    grids[-1][free] = 1.0
    cx, cy = hy / hx, hx / hy

    def modes(n):
        k = np.arange(1, n)
        return np.sqrt(2.0 / n) * np.sin(np.pi * ((k[:, None] * k[None, :]) % (2 * n)) / n), 2 - 2 * np.cos(np.pi * k / n)

    Qx, lx = modes(nx)
    Qy, ly = modes(ny)
    F = np.zeros((grids.shape[0], ny - 1, nx - 1))
    F[:, :, 0] += cx * grids[:, 1:-1, 0]
    F[:, :, -1] += cx * grids[:, 1:-1, -1]
    F[:, 0, :] += cy * grids[:, 0, 1:-1]
    F[:, -1, :] += cy * grids[:, -1, 1:-1]
    U = Qy @ ((Qy @ F @ Qx) / (cx * lx[None, :] + cy * ly[:, None])) @ Qx
    f = grids.copy()
    f[:, 1:-1, 1:-1] = U
    sx, sy = st["points"][:, 0] / hx, st["points"][:, 1] / hy
    ix, iy = np.clip(sx.astype(int), 0, nx - 1), np.clip(sy.astype(int), 0, ny - 1)
    xi, et = sx - ix, sy - iy
    f00, f10, f01, f11 = f[:, iy, ix], f[:, iy, ix + 1], f[:, iy + 1, ix], f[:, iy + 1, ix + 1]
    basis = np.where(xi >= et, f00 + xi * (f10 - f00) + et * (f11 - f10), f00 + et * (f01 - f00) + xi * (f11 - f01))
    return {"fields": f, "basis": basis}

"""The simulator's work as its users have it done, as a list of timed cases.

A case is a simulation (or a batch, or a served stream of simulations): topologies, transports and
traffic of the kinds that the tests, the configurations of workloads.py and bench.py use, each run
through the Python entry points a program calls and returned whole: every flow's established and
completed time (or start and completion time), every world's counters.

Kinds:
    one     run_world: a program that asks for one simulation and is given its results (world
            building, upload, run and download are all in the call)
    static  run_world_static: the same for callers that may not allocate device memory
    batch   a Simulator that holds its worlds and runs them: one world, the TCPs of one workload,
            or a parameter sweep over many worlds
    rdma    the same with RDMA worlds
    serve   a Server that is given a stream of requests at once and steps until all are done
"""
from __future__ import annotations

import math

import numpy as np

from twins_b200 import api, workloads

US = 1000  # ns
LINK = workloads.LINK_BYTES_PER_NS
TCPS = ("newreno", "dctcp", "cubic")
CCS = ("dcqcn", "hpcc", "dctcp")


# ------------------------------------------------------------------ the cases
def _case(name, kind, **kw):
    c = {"name": name, "kind": kind, "topo": "fattree", "k": 8, "leaves": 0, "spines": 0, "hpl": 0, "worlds": 1, "flows": 100, "load": 0.5,
         "cap": 1_000_000, "tcp": "dctcp", "ecn_k": 30, "queue": 200, "fin": False, "spray": False, "reuse": 0.0, "incasts": 0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a handful of short flows, in the fixed device area
        _case("static_k4", "static", k=4, flows=24, load=0.3, cap=100_000, tcp="newreno", fin=True),
        # a one-shot simulation of the smallest FatTree (the C1 shape: DCTCP, 30% load, 1 ms of arrivals)
        _case("one_k4_dctcp", "one", k=4, flows=240, load=0.3, tcp="dctcp"),
        # one k=8 world kept and run again: per-flow ECMP, losses and recovery (NewReno)
        _case("k8_newreno", "batch", flows=401, load=0.5, tcp="newreno"),
        # a k=8 world of the headline's shape with the whole size distribution: long flows, messages
        # over kept connections, FIN, per-packet spraying, Cubic
        _case("k8_cubic_spray", "batch", flows=200, load=0.5, cap=30_000_000, tcp="cubic", fin=True, spray=True, reuse=0.25),
        # a leaf-spine world: switches of 22 ports, whose ports are the critical path
        _case("leafspine12", "batch", topo="leafspine", leaves=12, spines=6, hpl=16, flows=613, load=0.6, tcp="newreno", queue=100),
        # the largest single world: FatTree k=16, 1,024 hosts and 320 switches
        _case("k16_dctcp", "batch", k=16, flows=2253, load=0.3, tcp="dctcp"),
        # the headline's batch: one workload under the three TCPs
        _case("k8_three_tcps", "batch", worlds=3, flows=1000, load=0.5, cap=3_000_000, tcp="each", fin=True, spray=True, reuse=0.25),
        # a mixed batch: leaf-spine worlds of different sizes and parameters
        _case("mixed_leafspines", "batch", topo="leafspines", worlds=12, flows=500, load=0.5, tcp="any"),
        # a parameter sweep: many small worlds of one topology
        _case("sweep_k8", "batch", worlds=96, flows=273, load=0.3, cap=300_000, tcp="any"),
        # RDMA: the largest single world, HPCC with PFC, incasts among all-to-all traffic
        _case("rdma_k16_hpcc", "rdma", k=16, flows=1500, load=0.4, tcp="hpcc", incasts=2),
        # RDMA: a sweep over congestion controls and buffers on k=8
        _case("rdma_sweep_k8", "rdma", worlds=8, flows=600, load=0.4, tcp="any", cap=500_000, incasts=1),
        # a served stream: requests on FatTrees, a Jellyfish and a Dragonfly, some with link failures
        _case("serve_mixed", "serve", topo="mixed", worlds=20, flows=150, load=0.4, cap=300_000, tcp="any"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["static", "one", "batch", "batch", "many", "many", "rdma", "rdma", "serve"])
    load = round(rng.uniform(0.2, 0.7), 2)
    c = {"load": load, "ecn_k": rng.choice([10, 20, 30, 40, 80]), "queue": rng.choice([100, 200, 400]), "fin": rng.random() < 0.5,
         "spray": rng.random() < 0.4, "reuse": rng.choice([0.0, 0.0, 0.25]), "tcp": rng.choice(TCPS), "cap": log(100_000, 1_000_000)}
    if kind == "static":
        c = _case("", "static", **{**c, "k": 4, "flows": log(8, 60), "cap": log(20_000, 200_000)})
    elif kind in ("one", "batch"):
        shape = rng.choice(["k4", "k8", "k16", "leafspine", "leafspine"])
        if shape == "leafspine":
            leaves, spines, hpl = rng.randint(3, 32), rng.randint(1, 8), rng.randint(3, 16)
            c = _case("", kind, **{**c, "topo": "leafspine", "leaves": leaves, "spines": spines, "hpl": hpl, "flows": log(30, 900)})
        else:
            c = _case("", kind, **{**c, "k": int(shape[1:]), "flows": log(30, {"k4": 250, "k8": 700, "k16": 2000}[shape])})
    elif kind == "many":
        topo = rng.choice(["fattree", "leafspines"])
        worlds = log(2, 40) if topo == "fattree" else log(2, 10)
        c = _case("", "batch", **{**c, "topo": topo, "k": rng.choice([4, 8]), "worlds": worlds, "flows": log(40, 300), "tcp": rng.choice(["any", "each"]),
                                  "cap": log(100_000, 500_000)})
    elif kind == "rdma":
        worlds = rng.choice([1, 1, log(2, 8)])
        c = _case("", "rdma", **{**c, "k": rng.choice([4, 8]) if worlds > 1 else rng.choice([4, 8, 16]), "worlds": worlds, "flows": log(40, 700),
                                 "tcp": rng.choice(CCS) if worlds == 1 else "any", "incasts": rng.randint(0, 2), "cap": log(100_000, 500_000)})
    else:
        c = _case("", "serve", **{**c, "topo": "mixed", "worlds": log(3, 20), "flows": log(30, 150), "tcp": "any", "cap": log(100_000, 300_000)})
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _traffic(rng, hosts, n, load, cap, reuse=0.0, incasts=0):
    """n messages between uniform random distinct hosts, web-search-like sizes up to `cap`, Poisson
    starts at `load` of the hosts' links; a share `reuse` of the connections carries four messages;
    `incasts` bursts of up to 32 senders x 64 KB to one host."""
    size = np.minimum(workloads.web_sizes(rng, n), cap)
    rate = load * hosts * LINK / _mean_size(cap)
    start = np.cumsum(rng.exponential(1.0 / rate, n)).astype(np.int64) + US
    src = rng.integers(0, hosts, n)
    dst = (src + rng.integers(1, hosts, n)) % hosts
    conn = np.full(n, -1, dtype=np.int64)
    if reuse > 0:
        # four messages apart in time share a connection
        m = int(n * reuse) // 4
        rows = rng.permutation(n)[:4 * m].reshape(m, 4)
        for i, r in enumerate(np.sort(rows, axis=1)):
            conn[r] = i
            src[r], dst[r] = src[r[0]], dst[r[0]]
    parts = [(src, dst, size, start, conn)]
    for _ in range(incasts):
        to = int(rng.integers(hosts))
        k = min(32, hosts - 1)
        snd = (to + 1 + rng.permutation(hosts - 1)[:k]) % hosts
        at = int(rng.integers(US, max(int(start[-1]), 2 * US)))
        parts.append((snd, np.full(k, to), np.full(k, 65_536), np.full(k, at), np.full(k, -1)))
    a = [np.concatenate(x) for x in zip(*parts)]
    order = np.argsort(a[3], kind="stable")
    return api.Flows.from_arrays(*(x[order] for x in a))


def _mean_size(cap):
    """The mean of the web-search-like distribution cut at `cap`."""
    s = np.array([p[0] for p in workloads.WEB_CDF])
    p = np.array([p[1] for p in workloads.WEB_CDF])
    u = (np.arange(4096) + 0.5) / 4096
    return float(np.minimum(np.interp(u, p, s), cap).mean())


def _topologies(case, rng):
    """Each world's topology."""
    kind, n = case["topo"], case["worlds"]
    if kind == "fattree":
        return [api.Topology.fattree(case["k"])] * n
    if kind == "leafspine":
        return [api.Topology.leafspine(case["leaves"], case["spines"], case["hpl"])] * n
    if kind == "leafspines":
        # (from 4 leaves to 32, each size once around: a batch's work hardly depends on the seed)
        leaves = [4 + 2 * ((5 * i) % 15) for i in range(n)]
        return [api.Topology.leafspine(x, x // 2, 16) for x in leaves]
    out = []
    for i in range(n):
        t = ("k4", "k8", "k4", "jf", "k8", "k4", "df", "k8", "k4", "k16")[i % 10]
        if t[0] == "k":
            out.append(api.Topology.fattree(int(t[1:])))
            continue
        g = workloads.jellyfish(seed=int(rng.integers(1000))) if t == "jf" else workloads.dragonfly()
        sw = [(a, b) for a, b in g.links if a < 0 and b < 0]
        a, b = sw[int(rng.integers(len(sw)))]
        at = int(rng.integers(20 * US, 60 * US))
        g.fails = [(at, -1 - a, -1 - b, 0), (at + 100 * US, -1 - a, -1 - b, 1)]
        out.append(g)
    return out


def _tcp_worlds(case, seed):
    rng = np.random.default_rng([seed, 17])
    topos = _topologies(case, rng)
    shared = None
    worlds = []
    for i, topo in enumerate(topos):
        tcp, ecn_k, queue, spray = case["tcp"], case["ecn_k"], case["queue"], case["spray"]
        n = case["flows"]
        if tcp == "each":
            tcp = TCPS[i % 3]
            shared = shared if shared is not None else _traffic(rng, topo.hosts, n, case["load"], case["cap"], case["reuse"])
        elif tcp == "any":
            # (a sweep's grid)
            tcp, ecn_k, queue = TCPS[i % 3], (10, 20, 40, 80)[i % 4], (100, 200, 400)[i // 4 % 3]
        if case["kind"] == "serve":
            spray = topo.kind == api.TOPO_GRAPH
        same = shared is not None and topo.hosts == topos[0].hosts
        flows = shared if same else _traffic(rng, topo.hosts, n, case["load"], case["cap"], case["reuse"])
        worlds.append((topo, flows, api.TcpParams(tcp, ecn_k, queue, fin=case["fin"], spray=spray, rng_seed=1 + seed % 1000, rng_run=1)))
    return worlds


def _rdma_worlds(case, seed):
    rng = np.random.default_rng([seed, 23])
    text = workloads.fattree_text(case["k"])
    hosts = case["k"] ** 3 // 4
    out = []
    for i in range(case["worlds"]):
        cc, over = case["tcp"], {}
        if cc == "any":
            kmin = (20, 50, 100, 400)[i % 4]
            cc, over = CCS[i % 3], {"BUFFER_SIZE": (2, 32)[i // 2 % 2], "KMIN_MAP": f"1 100000000000 {kmin}", "KMAX_MAP": f"1 100000000000 {4 * kmin}"}
        out.append((workloads.rdma_config(cc, **over), text, _traffic(rng, hosts, case["flows"], case["load"], case["cap"], 0.0, case["incasts"])))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rdma":
        worlds = _rdma_worlds(case, seed)
        sim = api.Simulator()
        for w in worlds:
            sim.add_rdma_world(*w)
        sim.prepare()
        return {"case": case, "worlds": worlds, "sim": sim}
    worlds = _tcp_worlds(case, seed)
    if kind in ("one", "static"):
        return {"case": case, "worlds": worlds}
    if kind == "batch":
        sim = api.Simulator()
        for w in worlds:
            sim.add_world(*w)
        sim.prepare()
        return {"case": case, "worlds": worlds, "sim": sim}
    srv = api.Server(worlds=12, hosts=4096, switches=1024, ports=16384, connections=1 << 15, messages=1 << 15, sent_list_entries=1 << 23,
                     ooo_blocks=1 << 22, active_per_host=256)
    return {"case": case, "worlds": worlds, "srv": srv}


# ------------------------------------------------------------------ a pass
def _counters(c):
    return np.array([c[k] for k in api.COUNTERS], dtype=np.int64)


def run(state):
    kind, worlds = state["case"]["kind"], state["worlds"]
    if kind == "one":
        est, done, ctr, _ = api.run_world(*worlds[0])
        return {"established": est, "completed": done, "counters": _counters(ctr)}
    if kind == "static":
        est, done, status = api.run_world_static(*worlds[0])
        return {"established": est, "completed": done, "status": status}
    if kind == "batch":
        sim = state["sim"]
        status = sim.run()
        got = [sim.results(w) for w in range(len(worlds))]
        return {"established": np.concatenate([g[0] for g in got]), "completed": np.concatenate([g[1] for g in got]),
                "counters": np.stack([_counters(sim.counters(w)) for w in range(len(worlds))]), "status": status}
    if kind == "rdma":
        sim = state["sim"]
        status = sim.run()
        got = [sim.rdma_results(w) for w in range(len(worlds))]
        # (the reference's counters, as its counters line prints them)
        return {"start": np.concatenate([g[0] for g in got]), "fct": np.concatenate([g[1] for g in got]),
                "counters": np.array(sim.rdma_counters()[:13], dtype=np.int64), "status": status}
    srv = state["srv"]
    ids = [srv.submit(*w) for w in worlds]
    while srv.step() or srv.stats()["queued"]:
        pass
    got = [srv.results(i) for i in ids]
    for i in ids:
        srv.release(i)
    return {"established": np.concatenate([g[0] for g in got]), "completed": np.concatenate([g[1] for g in got]),
            "counters": np.stack([_counters(g[2]) for g in got])}


# ------------------------------------------------------------------ what a pass is
def work(case):
    """Every frame is handed from node to node: written once by its sender and read once by the next
    node, 64 bytes each time (an RDMA frame with its INT words: 144), over the path's links; an ACK
    for every second TCP segment, for every RDMA frame. Inputs and results are small beside it."""
    rdma = case["kind"] == "rdma"
    links = {"fattree": 5.7, "leafspine": 3.9, "leafspines": 3.9, "mixed": 5.5}[case["topo"]]
    flow = max(_mean_size(case["cap"]) / (1000 if rdma else 1448), 1.0) * (2.0 if rdma else 1.5) + (0 if rdma else 4)
    frames = case["worlds"] * case["flows"] * flow + case["worlds"] * case["incasts"] * 32 * 66 * 2
    n = case["worlds"] * case["flows"]
    return {"bytes": frames * links * 2 * (144 if rdma else 64) + n * (28 + 16), "flops": 0}


def tolerance(case):
    """Times are whole nanoseconds and counters whole numbers: the same events in the same order."""
    return "exact"


def exact(case, seed):
    """The results are times of simulated events, whole numbers: no 64-bit arithmetic stands beside
    them (the packet-level oracles are programs of their own, which the tests compare with)."""
    return None

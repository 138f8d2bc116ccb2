"""A switch's slot staged in shared memory (a frame or a port per lane) against the same slot in phases
through L2, where the two can part: arrivals at one instant (their order and the draws' order fall to
the event chains, and undecided ties are counted), more frames than the staging area holds,
interfaces that go down, ports of every count up to 32.
"""
import ctypes

import numpy as np
import pytest

from twins_b200 import api, build, workloads

pytestmark = pytest.mark.gpu


def waves(hosts, n, seed, size):
    """Flows that start at one instant per wave and are of one size: frames meet at the switches in
    the same picosecond."""
    rng = np.random.default_rng(seed)
    src = np.concatenate([rng.permutation(hosts) for _ in range(n)])
    dst = (src + rng.integers(1, hosts, len(src))) % hosts
    start = np.repeat(np.arange(n) * 20_000 + 1000, hosts)
    return api.Flows.from_arrays(src, dst, np.full(len(src), size), start)


def worlds():
    df = workloads.dragonfly()
    sw = [(a, b) for a, b in df.links if a < 0 and b < 0]
    df.fails = [(15_000, -1 - sw[3][0], -1 - sw[3][1], 0), (60_000, -1 - sw[3][0], -1 - sw[3][1], 1)]
    for tag, topo in [("k4", api.Topology.fattree(4)), ("ls7x3x5", api.Topology.leafspine(7, 3, 5)), ("ls3x1x31", api.Topology.leafspine(3, 1, 31)),
                      ("df", df)]:
        for spray in (False, True):
            yield pytest.param(topo, spray, id=f"{tag}{'_spray' if spray else ''}")


@pytest.mark.parametrize("topo,spray", list(worlds()))
def test_staged_slots_equal_unstaged(native_lib, topo, spray):
    flows = waves(topo.hosts, 3, 5, 14_600)
    params = api.TcpParams("dctcp", 5, 20, spray=spray, rng_seed=3)
    got = {}
    # 384: every slot staged; 1: those of one frame; 20 and 97 (not a multiple of four): some
    # (test_a_shape_stages_the_frames_it_asks_for counts them)
    for stage in (384, 97, 20, 1):
        est, done, ctr, _ = api.run_world(topo, flows, params, host_lanes=1, stage_frames=stage)
        assert (done >= 0).all()
        got[stage] = (est, done, ctr)
    for stage in (97, 20, 1):
        assert (got[stage][0] == got[384][0]).all() and (got[stage][1] == got[384][1]).all(), stage
        assert got[stage][2] == got[384][2], stage
    assert got[384][2]["switch_events"] > 0 and got[384][2]["marks"] > 0


UNSTAGED = 15  # (the trace build's counter of switch slots beyond the staging area)


def unstaged_slots(topo, flows, params, stage):
    with api.Simulator(host_lanes=1, stage_frames=stage) as sim:
        w = sim.add_world(topo, flows, params)
        assert sim.run() == api.TB_OK
        out = (ctypes.c_ulonglong * 16)()
        assert sim.lib.tb_counters(sim.ctx, w, out, 16) == 0
        return out[UNSTAGED]


def test_a_shape_stages_the_frames_it_asks_for(native_lib, monkeypatch):
    """The switch slots that a launch shape's staging area does not hold, counted by the trace build. 31 hosts of
    one leaf open connections to each other at one instant: three of the leaf's slots have 31 frames (the
    SYNs first) and one has more, up to 62. In the waves above an area of 384 frames holds every slot, one
    of a frame only the slots of one frame, and areas between some."""
    monkeypatch.setattr(api, "_lib", api.load_library(build.SO_TRACE))
    leaf, i = api.Topology.leafspine(1, 1, 31), np.arange(31)
    syns = api.Flows.from_arrays(i, (i + 1) % 31, np.full(31, 1), np.full(31, 1000))
    got = {n: unstaged_slots(leaf, syns, api.TcpParams("newreno", 30, 200), n) for n in (384, 62, 31, 30)}
    assert got == {384: 0, 62: 0, 31: 1, 30: 4}
    for topo, some in ((api.Topology.leafspine(3, 1, 31), (97, 20)), (api.Topology.fattree(4), (20,))):
        flows = waves(topo.hosts, 3, 5, 14_600)
        n = {stage: unstaged_slots(topo, flows, api.TcpParams("dctcp", 5, 20), stage) for stage in (384, 97, 20, 1)}
        assert n[384] == 0 and all(0 < n[x] < n[1] for x in some), (topo, n)

"""A switch's slot staged in shared memory (a frame or a port per lane) against the same slot in phases
through L2, where the two can part: arrivals at one instant (their order and the draws' order fall to
the event chains, and undecided ties are counted), more frames than the staging area holds,
interfaces that go down, ports of every count up to 32.
"""
import numpy as np
import pytest

from twins_b200 import api, workloads

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
    # 384: every slot staged; 1: none; 20 and 97 (not a multiple of four): some
    for stage in (384, 97, 20, 1):
        est, done, ctr, _ = api.run_world(topo, flows, params, host_lanes=1, stage_frames=stage)
        assert (done >= 0).all()
        got[stage] = (est, done, ctr)
    for stage in (97, 20, 1):
        assert (got[stage][0] == got[384][0]).all() and (got[stage][1] == got[384][1]).all(), stage
        assert got[stage][2] == got[384][2], stage
    assert got[384][2]["switch_events"] > 0 and got[384][2]["marks"] > 0

"""The day kernel's segments against the oracle, bit for bit (gpu).

A segment draws all its timesteps at once and replays the locations where
somebody is infected: populations where a location holds one agent, a warp and
a few warps of agents, few and most of them infected within a day, one and
several variants; curfews that begin at the edges of the words of the
decision mask.
"""
import numpy as np
import pytest

from oracle import binding as ob
from tests.helpers import diff_state, small_snapshot, stats_rows

pytestmark = pytest.mark.gpu


def _equal_days(s_cpu, days=2):
    from pansim_gb300.native import GpuSim
    s_gpu = s_cpu.copy()
    o, g = ob.Oracle(s_cpu), GpuSim(s_gpu)
    for d in range(days):
        assert stats_rows(o.run_day(d)) == stats_rows(g.run_day(d)), d
    g.download()
    assert diff_state(s_cpu, s_gpu) == []
    off_o, ag_o = o.csr()
    off_g, ag_g = g.csr(canonical=True)
    assert np.array_equal(off_o, off_g) and np.array_equal(ag_o, ag_g)


@pytest.mark.parametrize("variants", [1, 3])
@pytest.mark.parametrize("n,locs,k", [(3000, 12, 3.74e-4), (3000, 12, 2e-2), (4097, 200, 5e-3), (511, 300, 0.5)])
def test_replayed_locations(gpu_lib, n, locs, k, variants):
    s = small_snapshot(n=n, locs=locs, k=k, initial_infected_frac=0.05, n_variants=variants)
    ill = np.nonzero(s.agents["st_infected_count"])[0]
    s.agents["variant"][ill] = np.arange(len(ill)) % variants
    _equal_days(s)


@pytest.mark.parametrize("begin", [1, 31, 32, 33, 95, 143])
def test_curfew_at_the_edges_of_the_decision_mask(gpu_lib, begin):
    s = small_snapshot(n=2000, locs=500, initial_infected_frac=0.05)
    s.params.update(enable_curfew=1, curfew_begin=begin, curfew_end=30)
    _equal_days(s)

"""Events at the ends of the range the kernels are written for, bit for bit the oracle's: nearly
empty events, and events above what a block holds in shared memory of super pixels, clusters,
used flags and tracks to follow."""
import pytest

import parity
from allen_b200 import generator
from allen_b200.chain import upload

pytestmark = pytest.mark.gpu

EVENTS = {
    "empty": dict(n_events=9, mean_pileup=0.05, noise_rate=1e-8),
    "sparse": dict(n_events=65, mean_pileup=0.4, noise_rate=1e-7),
    "noise_only": dict(n_events=17, mean_pileup=0.01, noise_rate=2e-4),
    "dense": dict(n_events=6, mean_pileup=40.0),
    "dense_noise": dict(n_events=3, mean_pileup=25.0, noise_rate=3e-4, hit_efficiency=0.9),
}


@pytest.mark.parametrize("version", [2, 4])
@pytest.mark.parametrize("name", list(EVENTS))
def test_event_sizes(chain, oracle, geometry, name, version):
    g = generator.generate(seed=300 + version, bank_version=version, **EVENTS[name])
    chain.reserve_for(g.raw)
    chain.run(upload(g.raw), use_graph=version == 2)
    totals = chain.synchronize()
    assert totals["device_flags"] == 0
    assert parity.compare(chain.outputs_to_host(totals), oracle.run(g.raw, geometry), g.raw.n_events) == []

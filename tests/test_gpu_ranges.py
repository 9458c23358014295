"""Events at the ends of the range the kernels are written for, bit for bit the oracle's: nearly
empty events, and events above what a block holds in shared memory of super pixels, clusters,
used flags and tracks to follow.  And slices of more than eight events per SM, which run other
kernels than smaller ones."""
import pytest

import parity
from allen_b200 import generator, seed_pruner
from allen_b200.chain import VeloChain, upload
from allen_b200.rawbanks import super_pixels_per_event, to_mep

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


MANY = 1301
SLICES = {
    "version_3": dict(bank_version=3),
    "version_4": dict(bank_version=4, pileup_min=1.0, pileup_max=15.0),
    "mep": dict(mep=True, bank_version=4),
    "retina": dict(raw_format=1, pileup_min=1.0, pileup_max=15.0),
    "retina_mep": dict(raw_format=1, mep=True, bank_version=4),
    "dense": dict(pileup_min=1.0, pileup_max=40.0),
    "dense_version_4": dict(bank_version=4, pileup_min=1.0, pileup_max=30.0, noise_rate=1e-4, hit_efficiency=0.95),
}


def _many(name):
    import torch
    assert MANY > 8 * torch.cuda.get_device_properties(0).multi_processor_count
    cfg = dict(SLICES[name])
    mep = cfg.pop("mep", False)
    s = generator.generate(MANY, seed=320 + len(name), **cfg).raw
    return s, to_mep(s) if mep else s


@pytest.mark.parametrize("name", list(SLICES))
def test_slices_of_many_events(chain, oracle, geometry, name):
    """The kernels of large slices, in the tuned configuration, on every kind of input: bit for bit
    the oracle's.  The dense slices hold events above what a block keeps in shared memory (3584
    super pixels, 8192 hits)."""
    s, given = _many(name)
    assert not name.startswith("dense") or super_pixels_per_event(s).max() > 10000
    assert chain.get_config()["persistent"] and chain.get_config()["search_ring_global"]
    chain.reserve_for(given)
    chain.run(upload(given), use_graph=True)
    totals = chain.synchronize()
    assert totals["device_flags"] == 0
    assert parity.compare(chain.outputs_to_host(totals), oracle.run(s, geometry), MANY) == []


@pytest.mark.parametrize("name", ["version_4", "dense"])
def test_learned_search_of_many_events(geometry, name):
    """The learned search on a large slice in its tuned configuration, against one block per event with
    rings in shared memory: bit for bit the same."""
    s, _ = _many(name)
    c = VeloChain(geometry)
    try:
        seed_pruner.use_learned(c)
        assert c.get_config()["persistent"] and c.get_config()["search_ring_global"]
        c.reserve_for(s)
        outs = []
        for cfg in (dict(), dict(search_threads=256, search_lanes_per_seed=0, search_ring_global=0, persistent=0)):
            c.configure(**cfg)
            c.run(upload(s))
            totals = c.synchronize()
            assert totals["device_flags"] == 0
            outs.append((totals, c.outputs_to_host(totals), c.seed_stats(MANY)))
        assert outs[0][0] == outs[1][0]
        assert (outs[0][2] == outs[1][2]).all() and (outs[0][2][:, 2] == 1).any()
        assert parity.compare(outs[0][1], outs[1][1], MANY) == []
    finally:
        c.close()

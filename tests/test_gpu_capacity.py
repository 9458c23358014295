"""Capacity limits and the less-travelled code paths of the chain, through the C ABI.

Every input here is well formed: the slices are generated, and the paths they take are the
kernels' own bounds-checked ones (a workspace reserved too small makes each stage return
before writing, a dense event overflows the 2048-entry ring of tracks to follow, which the
kernel indexes modulo its size and flags).  Parity cases force the fallbacks that typical
events never reach: the retina decoder's full key comparison and the Kalman filter's
in-place hit reads.
"""
import numpy as np
import pytest

import parity
from allen_b200 import generator
from allen_b200 import seed_pruner
from allen_b200.chain import COORDINATES_FP16, COORDINATES_FP32, OutputBuffersC, VeloChain, VeloError, upload
from allen_b200.rawbanks import RawSlice, super_pixels_per_event, to_mep

pytestmark = pytest.mark.gpu

VELO_ERR_CAPACITY = 3
VELO_ERR_DEVICE_FLAGS = 4
ERR_TTF_OVERFLOW = 1 << 2
ERR_INPUT_CAPACITY = 1 << 6


def run_chain(chain, s, use_graph=False):
    chain.reserve_for(s)
    chain.run(upload(s), use_graph=use_graph)
    totals = chain.synchronize()
    return totals, chain.outputs_to_host(totals)


@pytest.mark.parametrize("capacity", [0, 256])
def test_retina_full_comparison_rank(chain, oracle, geometry, capacity):
    """Retina clusters ranked by comparing every pair of keys (events above the bucket
    order's capacity take that path) give the oracle's sorted container, bit for bit."""
    g = generator.generate(60, seed=140 + capacity, raw_format=1, bank_version=3, pileup_min=1.0,
                           pileup_max=15.0)
    saved = chain.get_config()
    try:
        chain.configure(retina_order_capacity=capacity)
        totals, out = run_chain(chain, g.raw, use_graph=True)
        assert totals["device_flags"] == 0
        assert parity.compare(out, oracle.run(g.raw, geometry), g.raw.n_events) == []
    finally:
        chain.configure(**saved)


@pytest.mark.parametrize("warp_hits", [0, 64])
def test_kalman_hits_read_in_place(chain, oracle, geometry, warp_hits):
    """The Kalman filter with its per-warp staging capped (0: every span read in place; 64:
    most spans of 32 tracks exceed it) gives the oracle's states, bit for bit."""
    g = generator.generate(80, seed=57, pileup_min=5.0, pileup_max=15.0)
    saved = chain.get_config()
    chain.reserve_for(g.raw)
    chain.set_kalman(True, (0.1, -0.05))
    try:
        chain.configure(kalman_warp_hits=warp_hits)
        chain.run(upload(g.raw), use_graph=True)
        totals = chain.synchronize()
        got = chain.kalman_outputs(totals)
    finally:
        chain.set_kalman(False)
        chain.configure(**saved)
    ref = oracle.run(g.raw, geometry, beamline=(0.1, -0.05))
    reco = totals["host_number_of_reconstructed_velo_tracks"]
    assert reco == int(ref["dev_offsets_all_velo_tracks"][-1])
    assert np.array_equal(got["dev_is_backward"], ref["dev_is_backward"])
    w = parity.kalman_written_words(reco)
    for k in ("dev_velo_kalman_beamline_states", "dev_velo_kalman_endvelo_states"):
        assert np.array_equal(got[k].view(np.uint32)[w], ref[k].view(np.uint32)[w]), k
    with pytest.raises(VeloError):
        chain.configure(kalman_warp_hits=369)


def test_workspace_too_small(chain, oracle, geometry):
    """More events than reserved: VELO_ERR_CAPACITY before anything is queued.  More super
    pixels than reserved: the stages find the slice too large, write nothing, and the run
    ends in VELO_ERR_DEVICE_FLAGS with err_input_capacity; the chain then runs a slice that
    fits as before."""
    small = generator.generate(20, seed=61, mean_pileup=2.0).raw
    big = generator.generate(20, seed=62, mean_pileup=15.0, noise_rate=1e-4).raw
    # the reservation holds 2 estimated clusters per reserved super pixel: exceed that
    assert super_pixels_per_event(big).sum() > 3 * super_pixels_per_event(small).sum()
    chain.reserve_for(small)
    chain.set_kalman(True, (0.0, 0.0))
    try:
        more = generator.generate(21, seed=63).raw
        with pytest.raises(VeloError) as e:
            chain.run(upload(more))
        assert e.value.status == VELO_ERR_CAPACITY
        chain.run(upload(big))
        with pytest.raises(VeloError) as e:
            chain.synchronize()
        assert e.value.status == VELO_ERR_DEVICE_FLAGS
        assert e.value.flags & ERR_INPUT_CAPACITY
    finally:
        chain.set_kalman(False)
    totals, out = run_chain(chain, small)
    assert totals["device_flags"] == 0
    assert parity.compare(out, oracle.run(small, geometry), small.n_events) == []


@pytest.mark.parametrize("version", [2, 4])
def test_more_super_pixels_than_reserved(chain, oracle, geometry, version):
    """A slice of more super pixels than reserved whose clusters fit (two are reserved per super
    pixel, 0.9 made) runs like any other: bit for bit the oracle's, no flag."""
    s = generator.generate(60, seed=68 + version, bank_version=version, pileup_min=1.0, pileup_max=15.0).raw
    chain.reserve(s.n_events, int(0.6 * super_pixels_per_event(s).sum()))
    chain.run(upload(s), use_graph=version == 4)
    totals = chain.synchronize()
    assert totals["device_flags"] == 0
    assert parity.compare(chain.outputs_to_host(totals), oracle.run(s, geometry), s.n_events) == []


def event_words(s, raw, e):
    """(u32 view of event e's words in raw, word index of each bank's source ID)"""
    w = raw[int(s.offsets[e]):int(s.offsets[e + 1])].view(np.uint32)
    n_banks = int(w[0])
    return w, 2 + n_banks + w[1:1 + n_banks] // 4


def with_source_id_bit_9(s, every=1):
    """The slice with bit 9 set in the source IDs of every `every`-th event: the channel IDs of
    version 2 and 3 banks carry it, and it is the one bit of them that a cluster item does not hold."""
    raw = s.raw.copy()
    for e in range(0, s.n_events, every):
        w, source = event_words(s, raw, e)
        w[source] |= 0x200
    return RawSlice(raw, s.offsets, s.sizes, s.types, s.bank_version)


def with_two_banks_of_a_sensor(s):
    """(The slice with a bank of isolated super pixels, in each event that has one, renamed to the
    last bank's sensor with bit 9 set, the number of such events): the one sensor then has banks
    with and without the bit, which an item list cannot tell apart.  (No candidates, which would be
    looked up in the sensor's last bank.)"""
    raw, renamed = s.raw.copy(), 0
    for e in range(s.n_events):
        w, source = event_words(s, raw, e)
        for at in source[:-1]:
            words = w[at + 2:at + 2 + w[at + 1]]
            if len(words) and bool((words >> 31).all()) and w[source[-1] + 1]:
                w[at] = w[source[-1]] | 0x200
                renamed += 1
                break
    return RawSlice(raw, s.offsets, s.sizes, s.types, s.bank_version), renamed


@pytest.mark.parametrize("version,every,mep,gen", [
    (2, 1, False, dict(n_events=40, pileup_min=1.0, pileup_max=15.0)),
    (3, 2, False, dict(n_events=41, sp_order=1)),
    (2, 1, True, dict(n_events=20)),
    (2, 2, False, dict(n_events=4, mean_pileup=40.0)),
    (3, 1, False, dict(n_events=30, mean_pileup=0.05, noise_rate=1e-7)),
    (2, 0, False, dict(n_events=40, pileup_min=0.5, pileup_max=3.0)),
    (3, 0, False, dict(n_events=41, mean_pileup=1.0))])
@pytest.mark.parametrize("threads", [128, 256])
def test_source_id_bit_9(chain, oracle, geometry, version, every, mep, gen, threads):
    """Source IDs with bit 9 set, in all events and beside events without, in both bank layouts,
    sparse, and above what is held and staged in shared memory; and (every = 0) a sensor with banks of
    both kinds, whose event has no item list: bit for bit the oracle's."""
    s = generator.generate(seed=70 + version, bank_version=version, **gen).raw
    if every:
        s = with_source_id_bit_9(s, every)
    else:
        s, renamed = with_two_banks_of_a_sensor(s)
        assert renamed > s.n_events // 4
    saved = chain.get_config()
    try:
        chain.configure(cluster_threads=threads, cluster_stage_capacity=1024)
        totals, out = run_chain(chain, to_mep(s) if mep else s)
        assert totals["device_flags"] == 0
        assert parity.compare(out, oracle.run(s, geometry), s.n_events) == []
    finally:
        chain.configure(**saved)


@pytest.mark.parametrize("cfg", [dict(), dict(version=4, layout=COORDINATES_FP16), dict(retina=1), dict(learned=True)])
def test_too_many_clusters_write_nothing(geometry, cfg):
    """The first run on caller memory, with more clusters than it was sized for: every stage stops
    on this run's total (the clustering has written no offsets that the later ones could read), so
    all outputs stay as they were.  (Offsets and counts start at zero: a stage that trusted
    them would see empty events, and write that.)"""
    import torch
    gen = dict(bank_version=cfg.get("version", 2), raw_format=cfg.get("retina", 0))
    small = generator.generate(20, seed=66, mean_pileup=2.0, **gen).raw
    big = generator.generate(20, seed=67, mean_pileup=15.0, noise_rate=1e-4, **gen).raw
    sp = int(super_pixels_per_event(small).sum())
    assert super_pixels_per_event(big).sum() > 3 * sp
    layout = cfg.get("layout", COORDINATES_FP32)
    c = VeloChain(geometry)
    try:
        if cfg.get("learned"):
            seed_pruner.use_learned(c)
        z = c.sizes(20, sp, layout)
        ws = torch.zeros(z["workspace_bytes"] + 256, dtype=torch.uint8, device="cuda")
        bytes_of = {
            "dev_offsets_estimated_input_size": 4 * z["offsets_estimated_input_size"],
            "dev_module_cluster_num": 4 * z["module_cluster_num"],
            "dev_sorted_velo_cluster_container": z["sorted_velo_cluster_container_bytes"],
            "dev_offsets_all_velo_tracks": 4 * z["offsets_all_velo_tracks"],
            "dev_velo_track_hit_number": 4 * z["velo_track_hit_number"],
            "dev_offsets_velo_track_hit_number": 4 * z["offsets_velo_track_hit_number"],
            "dev_velo_track_hits": z["velo_track_hits_bytes"], "dev_accepted_velo_tracks": z["accepted_velo_tracks"]}
        empty = ("dev_offsets_estimated_input_size", "dev_module_cluster_num")
        fill = {k: 0 if k in empty else 0x5A for k in bytes_of}
        out = {k: torch.full((n,), fill[k], dtype=torch.uint8, device="cuda") for k, n in bytes_of.items()}
        c.bind((ws.data_ptr() + 255) & ~255, z["workspace_bytes"], 20, sp,
               {f: out[f].data_ptr() for f, _ in OutputBuffersC._fields_}, layout)
        c.run(upload(big))
        with pytest.raises(VeloError) as e:
            c.synchronize()
        assert e.value.status == VELO_ERR_DEVICE_FLAGS and e.value.flags == ERR_INPUT_CAPACITY
        torch.cuda.synchronize()
        assert [k for k, t in out.items() if not bool((t == fill[k]).all())] == []
    finally:
        c.close()


def test_ring_overflow_is_flagged(chain):
    """Events dense enough to hold more than 2048 tracks to follow at once (the reference
    overwrites ring entries it has not read yet): the run reports err_ttf_overflow through
    VELO_ERR_DEVICE_FLAGS instead of returning silently different tracks."""
    g = generator.generate(2, seed=64, mean_pileup=150.0)
    chain.reserve_for(g.raw)
    chain.run(upload(g.raw))
    with pytest.raises(VeloError) as e:
        chain.synchronize()
    assert e.value.status == VELO_ERR_DEVICE_FLAGS
    assert e.value.flags & ERR_TTF_OVERFLOW
    # the chain stays usable
    s = generator.generate(10, seed=65).raw
    totals, _ = run_chain(chain, s)
    assert totals["device_flags"] == 0

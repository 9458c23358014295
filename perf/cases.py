"""The work that a program using this package gives it, as cases that can be timed.

One pass of a chain case is what the package's own front end documents: VeloChain.run on a
device-resident slice of raw banks, VeloChain.synchronize, and the consolidated outputs in the
caller's buffers (VeloChain.bind), sized for the slices a program expects rather than for the one it gets.  The slices are the ones of the benchmark and the tests: synthetic
events of the package's generator, from a handful to 16000 per slice, at the nominal pileup of 7.6,
uneven pileup, and the high-occupancy stress setting; super-pixel banks of both layouts, MEPs and
retina-cluster banks; FP32 and FP16 coordinate containers; plain and learned search.  The other cases
are the end-to-end pipeline on host buffers, the Kalman filter on its own and the gradient of the
seed gate's training.
"""
from __future__ import annotations

import numpy as np
import torch

from allen_b200 import generator, seed_pruner
from allen_b200 import chain as vc
from allen_b200.rawbanks import RawSlice, super_pixels_per_event, to_mep

BEAMLINE = (0.35, -0.2)  # mm, the displaced beamline of the Kalman tests
UNIQUE_EVENTS = 1000     # larger slices hold these events again, each at its own place in memory


def _case(name=None, **fields):
    """A case: the fields given over the nominal slice's."""
    c = {"kind": "chain", "events": 1000, "pileup": 7.6, "pileup_max": 0.0, "noise": 1e-5, "efficiency": 0.98,
         "version": 2, "retina": False, "mep": False, "half": False, "learned": False, "graph": True}
    c.update(fields)
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        # the smallest call: a monitoring or test job with as many events as the committed samples hold
        _case("few_events", events=10),
        # a small production slice, launched kernel by kernel (the default of VeloChain.run)
        _case("slice_1000", events=1000, graph=False),
        # the benchmark's slice: the throughput setting of a farm node
        _case("slice_16000", events=16000),
        # uneven pileup, one to fifteen interactions per event, an odd number of events
        _case("uneven_8191", events=8191, pileup=1.0, pileup_max=15.0),
        # high occupancy: pileup 15, ten times the noise, inefficient sensors, one bank per sensor pair
        _case("stress_2000", events=2000, pileup=15.0, noise=1e-4, efficiency=0.95, version=4),
        # a MEP as it arrives, into the FP16 containers of a CUDA build of the consumer
        _case("mep_half_501", events=501, mep=True, half=True, version=4),
        # the default front end of the experiment: clusters found by the readout, small and large slices
        _case("retina_1000", events=1000, retina=True, graph=False),
        _case("retina_16000", events=16000, retina=True),
        # the search behind the learned seed gate
        _case("learned_4000", events=4000, learned=True),
        # end to end: three slices of page-locked raw banks in, consolidated tracks out on the host
        _case("host_3x2000", kind="host", events=2000),
        # the Kalman filter alone on the consolidated tracks of a slice
        _case("kalman_8000", kind="kalman", events=8000),
        # one training batch of the seed gate: loss and gradients
        _case("train_65536", kind="train", events=150, batch=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["chain"] * 7 + ["host", "kalman", "train"])
    if kind == "train":
        batch = _log_int(rng, 4096, 65536)
        return _case(kind="train", events=batch // 512 + 20, batch=batch)
    pileup, pileup_max, noise, efficiency = 7.6, 0.0, 1e-5, 0.98
    shape = rng.randrange(4)
    if shape == 1:
        pileup, pileup_max = 1.0, 15.0
    elif shape == 2:
        pileup, noise, efficiency = round(rng.uniform(1.0, 15.0), 1), 10 ** rng.uniform(-5, -4), 0.95
    elif shape == 3:
        pileup = round(rng.uniform(1.0, 15.0), 1)
    per_event = _super_pixels({"pileup": pileup, "pileup_max": pileup_max, "noise": noise})
    most = min(16000, int(16000 * 2500 / per_event))
    fields = dict(kind=kind, pileup=pileup, pileup_max=pileup_max, noise=noise, efficiency=efficiency,
                  version=rng.choice([2, 2, 3, 4]))
    if kind == "host":
        return _case(events=_log_int(rng, 100, min(most, 2000)), **fields)
    if kind == "kalman":
        return _case(events=_log_int(rng, 10, min(most, 8000)), **fields)
    fields.update(retina=rng.random() < 0.3, half=rng.random() < 0.2, graph=rng.random() < 0.6)
    fields["learned"] = rng.random() < 0.15
    fields["mep"] = rng.random() < 0.15
    return _case(events=_log_int(rng, 10, min(most, 600 if fields["mep"] else 16000)), **fields)


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _repeat(s: RawSlice, n_events: int, seed: int) -> RawSlice:
    """A slice of n_events events, the events of `s` in a random order, each repeated in full."""
    n = s.n_events
    order = np.concatenate([np.random.default_rng([seed, r]).permutation(n) for r in range(-(-n_events // n))])[:n_events]
    lengths = np.diff(s.offsets.astype(np.int64))
    offsets = np.zeros(n_events + 1, np.uint32)
    offsets[1:] = np.cumsum(lengths[order])
    raw = np.concatenate([s.raw[s.offsets[e]:s.offsets[e + 1]] for e in order])

    def column(a, dtype, unit):
        # [n + 1] u32 offsets in units of dtype from the array's start, then the values per bank
        start = a[:n + 1].astype(np.int64)
        values = a.view(dtype)
        first = (n_events + 1) * unit
        out_start = first + np.concatenate([[0], np.cumsum(np.diff(start)[order])])
        parts = [out_start.astype(np.uint32).view(dtype)] + [values[start[e]:start[e + 1]] for e in order]
        flat = np.concatenate(parts).view(np.uint8)
        return np.concatenate([flat, np.zeros((-flat.size) % 4 + 4, np.uint8)]).view(np.uint32)

    return RawSlice(raw, offsets, column(s.sizes, np.uint16, 2), column(s.types, np.uint8, 4), s.bank_version)


def _slice(case, seed) -> RawSlice:
    n = case["events"]
    g = generator.generate(min(n, UNIQUE_EVENTS), seed=1000 + seed, mean_pileup=case["pileup"],
                           pileup_min=case["pileup"] if case["pileup_max"] else 0.0, pileup_max=case["pileup_max"],
                           noise_rate=case["noise"], hit_efficiency=case["efficiency"], bank_version=case["version"],
                           raw_format=1 if case["retina"] else 0)
    s = g.raw if n <= UNIQUE_EVENTS else _repeat(g.raw, n, seed)
    return to_mep(s) if case["mep"] else s


def _bound_chain(case):
    """A chain that runs into buffers of the caller, sized for the case's slices, and those buffers."""
    chain = vc.VeloChain()
    if case["learned"]:
        seed_pruner.use_learned(chain)
    n, n_sp = case["events"], _super_pixel_bound(case)
    layout = vc.COORDINATES_FP16 if case["half"] else vc.COORDINATES_FP32
    z = chain.sizes(n, n_sp, layout)

    def words(k):
        return torch.zeros(int(k), dtype=torch.int32, device="cuda")

    def octets(k):
        return torch.zeros(int(k), dtype=torch.uint8, device="cuda")

    out = {"dev_offsets_estimated_input_size": words(z["offsets_estimated_input_size"]),
           "dev_module_cluster_num": words(z["module_cluster_num"]),
           "dev_sorted_velo_cluster_container": octets(z["sorted_velo_cluster_container_bytes"]),
           "dev_offsets_all_velo_tracks": words(z["offsets_all_velo_tracks"]),
           "dev_velo_track_hit_number": words(z["velo_track_hit_number"]),
           "dev_offsets_velo_track_hit_number": words(z["offsets_velo_track_hit_number"]),
           "dev_velo_track_hits": octets(z["velo_track_hits_bytes"]),
           "dev_accepted_velo_tracks": octets(z["accepted_velo_tracks"])}
    workspace = torch.empty(int(z["workspace_bytes"]), dtype=torch.uint8, device="cuda")
    chain.bind(workspace.data_ptr(), workspace.numel(), n, n_sp, {k: t.data_ptr() for k, t in out.items()}, layout)
    return chain, out, workspace


def prepare(case, seed):
    if case["kind"] == "train":
        return _prepare_train(case, seed)
    if case["kind"] == "host":
        return _prepare_host(case, seed)
    s = _slice(case, seed)
    assert int(super_pixels_per_event(s).sum()) <= _super_pixel_bound(case)
    chain, out, workspace = _bound_chain(case)
    dev = vc.upload(s)
    state = {"kind": case["kind"], "chain": chain, "out": out, "workspace": workspace, "dev": dev,
             "half": case["half"], "graph": case["graph"]}
    if case["kind"] == "kalman":
        chain.run(dev)
        totals = chain.synchronize()
        # states for as many tracks as such slices may have
        capacity = int(0.13 * _super_pixel_bound(case))
        assert totals["host_number_of_reconstructed_velo_tracks"] <= capacity
        state = {"kind": "kalman", "chain": chain, "n": s.n_events, "capacity": capacity, "totals": totals, "out": out,
                 "workspace": workspace, "backward": torch.zeros(capacity, dtype=torch.uint8, device="cuda"),
                 "beamline": torch.zeros(14 * capacity, dtype=torch.float32, device="cuda"),
                 "endvelo": torch.zeros(14 * capacity, dtype=torch.float32, device="cuda"),
                 "status": torch.zeros(1, dtype=torch.int32, device="cuda")}
    torch.cuda.synchronize()
    return state


def _prepare_host(case, seed):
    """Page-locked slices and a pipeline with room for them."""
    slices = [vc.pin_slice(_slice(case, 3 * seed + i)) for i in range(3)]
    pipe = vc.HostPipeline()
    pipe.reserve(case["events"], _super_pixel_bound(case), max(s.raw.nbytes for s in slices),
                 max(s.sizes.size for s in slices), max(s.types.size for s in slices))
    for buffers in pipe.host_out:
        for b in buffers:
            b.zero_()
    return {"kind": "host", "pipe": pipe, "slices": slices}


def _prepare_train(case, seed):
    """Training records of the plain search over generated events, in a fixed order, and a trainer
    with freshly initialised weights."""
    chain = vc.VeloChain()
    s = generator.generate(case["events"], seed=1000 + seed).raw
    chain.reserve_for(s)
    records, n, counted = seed_pruner.collect(chain, [vc.upload(s)], capacity=1200 * case["events"])
    assert n == counted and n >= case["batch"], (n, counted, case["batch"])
    rows = records[:seed_pruner.RECORD_BYTES * n].view(torch.int32).view(n, 16)
    order = torch.argsort(rows[:, 15].long() + (rows[:, 13].long() << 32))  # by event, then hit
    rows = rows[order][torch.from_numpy(np.random.default_rng(seed).permutation(n)).cuda()][:case["batch"]].contiguous()
    records = rows.view(torch.uint8).view(-1)
    model = seed_pruner.initial_model(records, case["batch"], seed=seed)
    trainer = seed_pruner.Trainer(model, pos_weight=2.0)
    torch.cuda.synchronize()
    chain.close()
    return {"kind": "train", "trainer": trainer, "model": model, "records": records, "batch": case["batch"]}


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def run(state):
    if state["kind"] == "train":
        loss, grads = state["trainer"].gradients(state["records"], 0, state["batch"])
        return {"loss": loss, "gradients": grads}
    if state["kind"] == "host":
        pipe = state["pipe"]
        totals, _ = pipe.run(state["slices"])
        # the results of each slice lie in the pipeline's page-locked buffers
        return {"totals": [list(t.values()) for t in totals], "out": [list(pipe.host_out[k]) for k in range(3)]}
    chain, out = state["chain"], state["out"]
    if state["kind"] == "kalman":
        st = chain.lib.velo_run_kalman_filter(
            state["n"], out["dev_offsets_all_velo_tracks"].data_ptr(), out["dev_offsets_velo_track_hit_number"].data_ptr(),
            out["dev_velo_track_hits"].data_ptr(), state["capacity"], BEAMLINE[0], BEAMLINE[1],
            state["backward"].data_ptr(), state["beamline"].data_ptr(), state["endvelo"].data_ptr(),
            state["status"].data_ptr(), vc._current_stream())
        if st:
            raise RuntimeError(f"velo_run_kalman_filter: {st}")
        return {"backward": state["backward"], "beamline": state["beamline"], "endvelo": state["endvelo"]}
    chain.run(state["dev"], use_graph=state["graph"])
    totals = chain.synchronize()
    # the containers mix 32- and 16-bit columns whose places depend on the totals: whole words
    return {"totals": list(totals.values()), **{k: v.view(torch.int32) if v.numel() % 4 == 0 else v for k, v in out.items()}}


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _pileup(case):
    return 0.5 * (case["pileup"] + case["pileup_max"]) if case["pileup_max"] else case["pileup"]


def _super_pixels(case):
    """Super pixels of an average event (the generator's: 280 per interaction, 409 noise pixels at 1e-5)."""
    return 280.0 * _pileup(case) + 409.0 * case["noise"] / 1e-5


def _super_pixel_bound(case):
    """Super pixels that a slice of the case is not expected to exceed."""
    mean = _super_pixels(case) * case["events"]
    spread = 300.0 * (case["events"] * (_pileup(case) + 17.0)) ** 0.5
    return int(1.1 * mean + 6.0 * spread) // 2 * 2


def work(case):
    if case["kind"] == "train":
        b = case["batch"]
        return {"bytes": 64 * b, "flops": 6 * b * (12 * 32 + 32 * 32 + 32)}
    n, nu = case["events"], _pileup(case)
    tracks, track_hits = 25.0 * nu * n, 233.0 * nu * n
    if case["kind"] == "kalman":
        # coordinates and offsets in; flag and two states (11 of 14 words each) out
        return {"bytes": int(12 * track_hits + 4 * tracks + tracks + 2 * 44 * tracks), "flops": int(2 * 30 * track_hits)}
    sps = _super_pixels(case) * n
    banks = (104 if case["version"] == 4 else 208) * n
    clusters = (1.0 if case["retina"] else 0.85) * sps
    element, track_element = (12, 10) if case["half"] else (18, 16)
    raw = 4 * sps + (11 if case["version"] == 4 else 15) * banks
    tracks_out = track_element * track_hits + 9 * tracks + 4 * n
    if case["kind"] == "host":
        return {"bytes": int(3 * (raw + tracks_out)), "flops": 0}
    return {"bytes": int(raw + element * clusters + 8 * 26 * n + tracks_out), "flops": 0}


# ---------------------------------------------------------------------------------------
# the computed numbers in 64 bits
# ---------------------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(prepare(case, seed))
    if case["kind"] == "kalman":
        return _exact_kalman(prepare(case, seed))
    # the chain's numbers are table lookups and selections, equal bit for bit or wrong
    return None


def _exact_train(state):
    """Binary cross-entropy of the 12-32-32-1 network and its gradient, in float64."""
    rows = state["records"].cpu().numpy().view(seed_pruner.RECORD_DTYPE)
    d = seed_pruner.model_dict(state["model"])
    f = torch.from_numpy(rows["f"].astype(np.float64))
    y = torch.from_numpy(rows["label"].astype(np.float64))
    x = ((f - torch.from_numpy(d["mean"].astype(np.float64))) * torch.from_numpy(d["inv_std"].astype(np.float64))).clamp(-8, 8)
    p = torch.from_numpy(d["params"].astype(np.float64)).requires_grad_()
    w1, b1, w2, b2, w3, b3 = torch.split(p, [384, 32, 1024, 32, 32, 1])
    h1 = torch.relu(x @ w1.view(32, 12).T + b1)
    h2 = torch.relu(h1 @ w2.view(32, 32).T + b2)
    z = h2 @ w3 + b3
    weight = torch.where(y > 0.5, 2.0, 1.0)
    loss = (weight * torch.nn.functional.binary_cross_entropy_with_logits(z, y, reduction="none")).mean()
    loss.backward()
    return {"loss": float(loss), "gradients": p.grad.numpy()}


def _exact_kalman(state):
    """The simplified Kalman fit of every track, in float64, all tracks at once."""
    t, o = state["totals"], state["out"]
    reco, TH = t["host_number_of_reconstructed_velo_tracks"], t["host_accumulated_number_of_hits_in_velo_tracks"]
    first = o["dev_offsets_velo_track_hit_number"][:reco + 1].long()
    xyz = o["dev_velo_track_hits"][4 * TH:16 * TH].view(torch.float32).view(TH, 3).double()
    capacity = state["capacity"]
    lo, hi = first[:-1], first[1:] - 1
    bx, by = (torch.tensor(b, dtype=torch.float32).double().item() for b in BEAMLINE)
    a, b = xyz[lo], xyz[hi]
    tx, ty = (b[:, 0] - a[:, 0]) / (b[:, 2] - a[:, 2]), (b[:, 1] - a[:, 1]) / (b[:, 2] - a[:, 2])
    lin_z = b[:, 2] + (tx * (bx - b[:, 0]) + ty * (by - b[:, 1])) / (tx * tx + ty * ty)
    backward = lin_z > a[:, 2]

    def fit(tx, ty, upstream):
        direction = torch.where(backward, 1.0, -1.0) * (1.0 if upstream else -1.0)
        reverse = (b[:, 2] - a[:, 2]) * direction < 0
        noise = 1e-8 + 7e-6 * (tx * tx + ty * ty)
        start, step = torch.where(reverse, hi, lo), torch.where(reverse, -1, 1)
        x, y, z = xyz[start].unbind(1)
        tx, ty = tx.clone(), ty.clone()
        c00, c20, c22 = torch.full_like(x, 0.00015625), torch.zeros_like(x), torch.ones_like(x)
        for i in range(1, int((hi - lo).max()) + 1):
            on = i <= hi - lo
            hx, hy, hz = xyz[torch.where(on, start + i * step, start)].unbind(1)
            v = c22 + noise
            dz = hz - z
            px, py, p20, p00 = x + dz * tx, y + dz * ty, c20 + dz * v, c00 + 2 * dz * c20 + dz * dz * v
            r = 1.0 / (1.0 / 6400.0 + p00)
            kx, kt = p00 * r, p20 * r
            new = (px + kx * (hx - px), py + kx * (hy - py), hz, tx + kt * (hx - px), ty + kt * (hy - py),
                   (1 - kx) * p00, (1 - kx) * p20, v - kt * p20)
            x, y, z, tx, ty, c00, c20, c22 = (torch.where(on, w, u) for w, u in zip(new, (x, y, z, tx, ty, c00, c20, c22)))
        c22 = c22 + noise
        dz = (tx * (bx - x) + ty * (by - y)) / (tx * tx + ty * ty) if upstream else 770.0 - z
        c00, c20 = c00 + dz * dz * c22 + 2 * dz * c20, c20 + c22 * dz
        zero = torch.zeros_like(x)
        parameters = torch.stack([x + tx * dz, y + ty * dz, z + dz, tx, ty, zero], 1)
        cov = torch.stack([c00, c20, c22, c00, c20, c22, zero, zero], 1)
        rest = torch.zeros(14 * (capacity - reco), dtype=torch.float64, device=x.device)
        return torch.cat([parameters.reshape(-1), cov.reshape(-1), rest]), tx, ty

    up, utx, uty = fit(tx, ty, True)
    down, _, _ = fit(utx, uty, False)
    return {"backward": None, "beamline": up, "endvelo": down}

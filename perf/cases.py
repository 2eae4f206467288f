"""Performance cases of the VELO chain, through the package's public entry points.

A case is one call a user of the framework makes: a batch of raw events through
`VeloChain` (plain, pruned, with the beamline PV stage, behind the global event cut, from
device or from host memory), or a call of the scorer's trainer. `listed()` holds the fixed
cases, `draw(rng)` makes more of the same ranges.

Event batches are the seeded synthetic workloads of `cuda_hlt_b200.events` (straight tracks
through the real geometry, encoded as raw banks), the seed of a case in the place of the
workload's own. Results of the chain are whole numbers and single-precision values that the
reference kernels define bit for bit, so their tolerance is "exact".
"""
import ctypes as C

import numpy as np
import torch

from cuda_hlt_b200 import chain, events, mlp, train_scorer

# workload -> generator settings (events.CONFIGS without seed and count)
WORKLOADS = {
    "nu7.6": dict(nu_min=7.6, nu_max=7.6),
    "nu2-15": dict(nu_min=2.0, nu_max=15.0),
    "nu2-20": dict(nu_min=2.0, nu_max=20.0),
    "nu15-noisy": dict(nu_min=15.0, nu_max=15.0, noisy_event_fraction=0.1, noisy_factor=3.0),
}
# distinct events generated per batch; a larger batch repeats them at other addresses
DISTINCT = 16384
# capacity of the consolidated outputs (VeloConfig.max_tracks): the mean of the workload's fullest
# events and room for a single one; track hits: 8 a track on average
HITS_PER_TRACK = 10
READBACK = ("atomics", "track_hit_number", "track_hits", "kalman")


def _case(name, n, workload, kind="device", mode="plain", mapping="auto", graphs=False, pv=False, gec=False):
    return dict(name=name, kind=kind, n=n, workload=workload, mode=mode, mapping=mapping, graphs=graphs, pv=pv, gec=gec)


def listed():
    return [
        # one event handed over by a host program, default settings: the latency of a call
        _case("one_event_host", 1, "nu7.6", kind="host"),
        # a thousand events of the smallest benchmark workload, default search mapping
        _case("plain_1k", 1000, "nu7.6", graphs=True),
        # the same size from pinned host memory with all consolidated results read back, the
        # program of a host trigger: run_host, sync, velo_download_async
        _case("host_readback_1k", 1000, "nu2-15", kind="readback", mapping="warp"),
        # an ordinary device-resident batch with the reference's own u32 offsets, ragged size
        _case("batched_4k_u32", 4001, "nu2-15", kind="device_u32", mapping="warp"),
        # high occupancy: nu = 15, a tenth of the events with three times the noise
        _case("noisy_3k", 3000, "nu15-noisy", mapping="warp", graphs=True),
        # primary vertices behind the chain
        _case("pv_4k", 4096, "nu2-20", mapping="warp", graphs=True, pv=True),
        # the global event cut in front of the chain
        _case("gec_8k", 8192, "nu2-20", mapping="warp", graphs=True, gec=True),
        # the learned scorer at its committed operating point
        _case("pruned_16k", 16384, "nu2-20", mode="pruned", mapping="warp", graphs=True),
        # the learned scorer on every seeding candidate (the quality operating point)
        _case("every_candidate_8k", 8191, "nu2-20", mode="every", mapping="warp", graphs=True),
        # the benchmark's batch size
        _case("plain_64k", 65536, "nu2-20", mapping="warp", graphs=True),
        # one epoch of the scorer's training on held samples: forward, backward, Adam
        dict(name="scorer_train", kind="train", n=200000, batch=16384),
        # logits of host feature rows
        dict(name="scorer_infer", kind="infer", n=100001),
    ]


def draw(rng):
    r = rng.random()
    if r < 0.08:
        return dict(kind="train", n=int(2 ** rng.uniform(13, 17.6)), batch=rng.choice([1000, 4096, 16384]))
    if r < 0.16:
        return dict(kind="infer", n=int(2 ** rng.uniform(3, 17)))
    workload = rng.choice(list(WORKLOADS))
    gec = rng.random() < 0.12
    c = _case("", int(2 ** rng.uniform(0, 12.5 if gec else 14)), workload,
              kind="device" if gec else rng.choice(["device", "device", "device_u32", "host", "readback"]),
              mode=rng.choice(["plain", "plain", "pruned", "every"]),
              mapping=rng.choice(["auto", "warp", "warp"]), graphs=rng.random() < 0.6, pv=rng.random() < 0.2, gec=gec)
    if c["kind"] == "readback":
        c["n"] = min(c["n"], 2048)
    del c["name"]
    return c


# ---- event batches ----
def _batch(case, seed):
    n = case["n"]
    return events.generate(min(n, DISTINCT), seed=int(seed), with_mc=False, **WORKLOADS[case["workload"]])


def _tiled(b, n):
    """(raw uint8 tensor, offsets int64 tensor) on the GPU of n events, the batch repeated."""
    raw, off = torch.from_numpy(b.raw).cuda(), torch.from_numpy(b.offsets.astype(np.int64)).cuda()
    reps = -(-n // b.n_events)
    if reps > 1:
        size = int(b.raw.size)
        off = torch.cat([off[:-1] + k * size for k in range(reps)] + [off[-1:] + (reps - 1) * size])[:n + 1].contiguous()
        raw = raw.repeat(reps)[:int(off[-1])].contiguous()
    return raw, off


def _max_tracks(case):
    return int(18.0 * _nu(case) * case["n"]) + 1200


def prepare(case, seed):
    if case["kind"] in ("train", "infer"):
        return _prepare_scorer(case, seed)
    b = _batch(case, seed)
    n, s = case["n"], dict(case=case)
    if case["kind"] in ("host", "readback"):
        pinned = torch.empty(b.raw.size, dtype=torch.uint8, pin_memory=True)
        pinned.copy_(torch.from_numpy(b.raw))
        s.update(batch=events.EventBatch(pinned.numpy(), b.offsets), pinned=pinned)
        raw_bytes = int(b.raw.size)
    else:
        raw, off = _tiled(b, n)
        if case["kind"] == "device_u32":
            off = off.to(torch.int32)
        s.update(raw=raw, off=off)
        raw_bytes = raw.numel()
    if case["gec"]:
        ut, sf = events.generate_ut_scifi(b, seed=int(seed))
        s["gec"] = [torch.from_numpy(a).cuda() for a in (ut.raw, ut.offsets.view(np.int64), sf.raw,
                                                         sf.offsets.view(np.int64))]
    T = s["max_tracks"] = _max_tracks(case)
    vc = chain.VeloChain(max_events=n, max_raw_bytes=raw_bytes + 4096, use_graphs=case["graphs"], max_tracks=T,
                         max_track_hits=HITS_PER_TRACK * T,
                         mapping=chain.MAP_WARP if case["mapping"] == "warp" else chain.MAP_AUTO)
    if case["pv"]:
        vc.set_pv(True)
    if case["mode"] != "plain":
        w = mlp.load_weights(train_scorer.DEFAULT_WEIGHTS)
        if case["mode"] == "every":
            w.min_pairs = 0
            w.min_event_clusters = 0
        vc.set_mlp(w)
        vc.set_mode(chain.MODE_PRUNED)
    s["vc"] = vc
    # an empty run fills in the addresses of the outputs; zeros stand past the run's own totals
    stream = torch.cuda.current_stream().cuda_stream
    if case["gec"]:
        vc.run_gec_device(0, 0, *[g.data_ptr() for g in s["gec"]], 0, stream=stream)
    else:
        vc.run_device(0, 0, 0, stream)
    for t in _outputs(vc, n, T).values():
        t.zero_()
    if case["kind"] == "readback":
        s["pinned_out"] = {k: torch.zeros(v.shape, dtype=v.dtype, pin_memory=True)
                           for k, v in _outputs(vc, n, T).items() if k in READBACK}
    return s


class _DeviceArray:
    """A device address of a context as torch reads it (no copy); a tensor made from it keeps
    this object, and so the context that owns the memory."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=kind, data=(int(ptr), False), version=3, strides=None)


def _view(owner, ptr, shape, kind):
    return torch.as_tensor(_DeviceArray(owner, ptr, tuple(shape), kind), device="cuda")


def _outputs(vc, n, T):
    """The context's own output buffers at their whole capacity: T tracks."""
    o = vc.out
    r = dict(atomics=_view(vc, o.atomics, (2 * n + 1,), "<i4"), status=_view(vc, o.status, (n,), "<i4"),
             track_hit_number=_view(vc, o.track_hit_number, (T + 1,), "<i4"),
             module_hit_num=_view(vc, o.module_hit_num, (n, chain.N_MODULES), "<i4"),
             # x, y, z and LHCb id of the hits, as bit patterns
             track_hits=_view(vc, o.track_hits, (4 * HITS_PER_TRACK * T,), "<i4"),
             states=_view(vc, o.states, (13 * T,), "<f4"), kalman=_view(vc, o.kalman_states, (13 * T,), "<f4"))
    if o.pv_vertices:
        M = chain.PV_MAX_VERTICES
        v = _view(vc, o.pv_vertices, (n, M, 13), "<f4")
        r.update(pv_position=v[..., 0:4], pv_cov=v[..., 6:12],
                 pv_n_tracks=_view(vc, o.pv_vertices, (n, M, 13), "<i4")[..., 5],
                 pv_count=_view(vc, o.pv_count, (n,), "<i4"), pv_npeaks=_view(vc, o.pv_npeaks, (n,), "<i4"),
                 pv_zpeaks=_view(vc, o.pv_zpeaks, (n, M), "<f4"))
    if o.event_list:
        r.update(n_selected=_view(vc, o.n_selected, (1,), "<i4"), event_list=_view(vc, o.event_list, (n,), "<i4"),
                 gec_counts=_view(vc, o.gec_counts, (n, 2), "<i4"), gec_flags=_view(vc, o.gec_flags, (n,), "|u1"))
    return r


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        t = state["trainer"]
        t.set_weights(state["weights"])
        loss = t.train(1, batch=case["batch"])
        d = mlp.weights_to_dict(t.weights())
        return dict(loss=loss, w1=d["w1"], w2=d["w2"], w3=d["w3"])
    if kind == "infer":
        return dict(logits=state["trainer"].infer(state["features"]))
    vc, n = state["vc"], case["n"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind in ("host", "readback"):
        vc.run_host(state["batch"], stream)
    elif kind == "device_u32":
        vc.run_device_u32(state["raw"].data_ptr(), state["off"].data_ptr(), n, stream)
    elif case["gec"]:
        vc.run_gec_device(state["raw"].data_ptr(), state["off"].data_ptr(), *[g.data_ptr() for g in state["gec"]], n,
                          stream=stream)
    else:
        vc.run_device(state["raw"].data_ptr(), state["off"].data_ptr(), n, stream)
    # the layout of the outputs depends on the totals: every program waits for them
    n_tracks, n_hits, _ = vc.sync(clusters=False)
    if kind == "readback":
        out, o = state["pinned_out"], vc.out
        for key, ptr, size in (("atomics", o.atomics, 8 * n + 4),
                               ("track_hit_number", o.track_hit_number, 4 * n_tracks + 4),
                               ("track_hits", o.track_hits, 16 * n_hits),
                               ("kalman", o.kalman_states, 49 * n_tracks)):
            rc = vc.lib.velo_download_async(vc.ctx, C.c_void_p(out[key].data_ptr()), C.c_void_p(ptr), size,
                                            C.c_void_p(stream))
            if rc != 0:
                raise chain.VeloError(f"velo_download_async failed with code {rc}")
        torch.cuda.current_stream().synchronize()  # the program reads them on the host
        return dict(out, n_tracks=n_tracks, n_hits=n_hits)
    return dict(_outputs(vc, n, state["max_tracks"]), n_tracks=n_tracks, n_hits=n_hits)


# ---- the scorer's trainer ----
def _features(n, seed):
    """Feature rows with the ranges of seeding candidates (mlp.FEATURES)."""
    g = np.random.default_rng(seed)
    f = np.empty((n, 12), np.float32)
    f[:, 0:2] = g.normal(0, 0.12, (n, 2))                    # slopes
    f[:, 2] = np.log1p(g.exponential(30.0, n))               # log scatter
    f[:, 3:5] = g.uniform(-0.062, 0.062, (n, 2))             # phi differences
    f[:, 5] = g.integers(2, 50, n)                           # module
    f[:, 6:8] = g.integers(1, 30, (n, 2))                    # window sizes
    f[:, 8] = g.uniform(5.0, 45.0, n)                        # radius
    f[:, 9:12] = g.integers(1, 4, (n, 3))                    # pixels
    return f


def _prepare_scorer(case, seed):
    s = dict(case=case)
    n = case["n"]
    t = mlp.MlpTrainer(max(n, 1), seed=int(seed))
    s["trainer"] = t
    if case["kind"] == "infer":
        t.set_weights(mlp.load_weights(train_scorer.DEFAULT_WEIGHTS))
        s["features"] = _features(n, int(seed))
        return s
    # candidates of plain runs, as the training pipeline collects them (about 2,200 an event)
    b = events.generate(n // 1200 + 16, seed=int(seed), with_mc=False, **WORKLOADS["nu2-15"])
    vc = chain.VeloChain(max_events=b.n_events, max_raw_bytes=int(b.raw.size) + 4096, mapping=chain.MAP_WARP)
    vc.run_host(b)
    vc.sync()
    t.collect(vc)
    vc.close()
    t.normalize()
    s["weights"] = t.weights()
    return s


# ---- what a pass cannot do without ----
def _nu(case):
    lo, hi = WORKLOADS[case["workload"]]["nu_min"], WORKLOADS[case["workload"]]["nu_max"]
    return 0.5 * (lo + hi)


def work(case):
    n = case["n"]
    if case["kind"] == "infer":  # 12 features in, 2 logits out
        return dict(bytes=56.0 * n, flops=2.0 * n * (12 * 64 + 64 * 64 + 64 * 2))
    if case["kind"] == "train":  # features and label of each sample; forward and twice that backward
        return dict(bytes=49.0 * n + 3 * 4 * 5122.0, flops=6.0 * n * (12 * 64 + 64 * 64 + 64 * 2))
    nu = _nu(case)
    # averages of the generator: raw bytes, tracks and track hits per event
    raw, tracks, hits = 2650.0 + 1385.0 * nu, 15.2 * nu, 122.0 * nu
    per = raw + 16 * hits + 98 * tracks + 4 * (tracks + 1) + 8
    # seeding and forwarding triplets (about 30 operations each) and the two fits of each hit
    flops = 30 * 2400.0 * nu + 90 * hits
    if case["pv"]:
        per += 49 * tracks + chain.PV_MAX_VERTICES * 56
        flops += 60 * tracks * 7
    if case["gec"]:
        per = per * 0.6 + 2429.0  # the cut keeps the emptier events
        flops *= 0.6
    if case["mode"] == "every":  # the scorer on every candidate, 1,900 at nu = 11
        flops += 172 * nu * 2.0 * (12 * 64 + 64 * 64 + 64 * 2)
    return dict(bytes=per * n, flops=flops * n)


def tolerance(case):
    if case["kind"] == "infer":
        # bf16 weights and activations, 32-bit sums: only the order of a sum is free
        return {"rel": 2e-3, "max": 0.05}
    if case["kind"] == "train":
        # bf16 products; the order of the sums travels through the epoch's Adam steps
        return {"rel": 1e-2, "max": 0.2}
    if case["pv"]:
        # the vertex sums of a track fit have no defined order; everything else is exact
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.0}
    return "exact"


def exact(case, seed):
    """Logits in 64 bits. The other cases have no 64-bit value: which hits make a track is
    decided by comparisons of single-precision values that the reference defines, and the
    sample order of a training epoch is the trainer's own."""
    if case["kind"] != "infer":
        return None
    w = mlp.weights_to_dict(mlp.load_weights(train_scorer.DEFAULT_WEIGHTS))
    w = {k: v.astype(np.float64) for k, v in w.items() if isinstance(v, np.ndarray)}
    x = (_features(case["n"], int(seed)).astype(np.float64) - w["mean"]) * w["inv_std"]
    h = np.maximum(x @ w["w1"][:, :12].T + w["w1"][:, 12], 0.0)
    h = np.maximum(h @ w["w2"][:, :64].T + w["w2"][:, 64], 0.0)
    return dict(logits=h @ w["w3"][:, :64].T + w["w3"][:, 64])

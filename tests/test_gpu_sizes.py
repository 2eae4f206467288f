"""The launch shapes and paths that a batch's size, an event's occupancy or a module's size
chooses, at the sizes where one takes over from the next: every event's result is the same
whatever the batch it comes in."""
import numpy as np
import pytest

import oracle
from cuda_hlt_b200 import chain, events, mlp, train_scorer
from conftest import golden_batch
from test_gpu_windows import PHI_CAP, windows_of

pytestmark = pytest.mark.gpu


def run(b, max_tracks=0, max_track_hits=0, **kw):
    vc = chain.VeloChain(max_events=b.n_events, max_raw_bytes=int(b.raw.size) + 4096, max_tracks=max_tracks,
                         max_track_hits=max_track_hits, **kw)
    vc.run_host(b)
    totals = vc.sync()
    res = vc.results()
    vc.close()
    return res, totals


def bits(parts):
    return b"".join(np.ascontiguousarray(p).tobytes() for p in parts)


def track_bits(res, e):
    """The tracks of one event, their states and, behind the vertex stage, its vertices."""
    t0, t1 = int(res["track_offsets"][e]), int(res["track_offsets"][e + 1])
    h0, h1 = int(res["track_hit_number"][t0]), int(res["track_hit_number"][t1])
    parts = [res["status"][e], res["track_hit_number"][t0:t1 + 1] - h0, res["hit_id"][h0:h1]]
    parts += [res[k][h0:h1] for k in ("hit_x", "hit_y", "hit_z")]
    parts += [res[s][k][t0:t1] for s in ("states", "kalman") for k in chain.STATE_FIELDS + ("backward",)]
    if "pv_count" in res:
        parts += [res["pv_count"][e], res["pv_vertices"][e, :res["pv_count"][e]], res["pv_npeaks"][e],
                  res["pv_zpeaks"][e, :res["pv_npeaks"][e]]]
    return bits(parts)


def event_bits(res, e):
    """Everything the chain says of one event, as comparable bytes."""
    parts = [m[k] for m in chain.event_clusters(res, e) for k in ("id", "phi", "x", "y", "z", "size")]
    return track_bits(res, e) + bits(parts)


@pytest.fixture(scope="module")
def batch_700():
    import torch
    b = events.generate_config("pruned_1m", n_events=700, first_event=40_000, with_mc=False)
    # one block an event in the search, four warps an event in the decode
    ref, _ = run(b, mapping=chain.MAP_BLOCK, decode_warps=4)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return b, [event_bits(ref, e) for e in range(b.n_events)], sms


# up to 2 events per SM the decode takes 16 warps, up to 4 the search takes eight
@pytest.mark.parametrize("per_sm, more", [(0, 1), (0, 2), (2, 0), (2, 1), (4, 0), (4, 1)])
def test_events_do_not_depend_on_the_batch_size(batch_700, per_sm, more):
    b, want, sms = batch_700
    n = per_sm * sms + more
    res, totals = run(b.subset(0, n))
    assert totals[0] == int(res["atomics"][2 * n]) and totals[1] == int(res["track_hit_number"][totals[0]])
    for e in range(n):
        assert event_bits(res, e) == want[e], e


def sp_event(rng, counts):
    """A raw event with counts[m] isolated one-pixel SPs in module m, in address order."""
    payload, offs = [], [0]
    for sensor in range(208):
        n = counts[sensor // 4] // 4 + (sensor % 4 < counts[sensor // 4] % 4)
        # distinct addresses with an empty SP between any two
        addr = np.sort(rng.choice(128 * 3 * 16, n, replace=False))
        words = [0x80000000 | ((((int(a) // 16) << 6) | (int(a) % 16) * 4) << 8) | 1 << int(rng.integers(8)) for a in addr]
        payload += [sensor, n] + words
        offs.append(4 * len(payload))
    return np.array([208] + offs + payload, np.uint32).view(np.uint8)


# blocks of 4 warps hold 6,144 phi, of 8 warps (more events than the wide decode takes) 8,192
@pytest.mark.parametrize("copies, warps", [(2, 4), (330, 8)])
@pytest.mark.parametrize("large", [0, 1])
def test_modules_of_a_parity_beyond_the_shared_phi(copies, warps, large):
    """The windows of an event whose modules of one parity hold more phi than the block's shared
    memory: they are searched in the cluster records, the other parity's as ever."""
    rng = np.random.default_rng(11)
    counts = np.where(np.arange(52) % 2 == large, PHI_CAP[warps] // 26 + 5, 60)
    ev = sp_event(rng, counts)
    b = events.EventBatch(np.tile(ev, copies), np.arange(copies + 1, dtype=np.uint64) * np.uint64(ev.size))
    vc = chain.VeloChain(max_events=copies, max_raw_bytes=int(b.raw.size) + 4096, max_tracks=1200 * copies,
                         decode_warps=warps)
    vc.run_host(b)
    vc.sync()
    res = vc.results()
    assert np.array_equal(res["module_num"][:52], counts)
    per_parity = res["module_num"][:52].reshape(26, 2).sum(0)
    assert per_parity[large] > PHI_CAP[warps] > per_parity[1 - large] and per_parity.sum() <= 16384
    windows_of(vc, res, 2)
    vc.close()
    assert event_bits(res, 0) == event_bits(res, copies - 1)


@pytest.mark.parametrize("copies", [1, 330])
def test_module_sizes_at_the_edges_of_the_sorts(geometry, copies):
    """32, 64, 128 and 256 clusters are the widths of the register sorts, 500 is past them all."""
    rng = np.random.default_rng(5)
    sizes = [0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 500]
    evs = [sp_event(rng, np.resize(np.roll(sizes, k), 52)) for k in (0, 5)] * copies
    off = np.concatenate([[0], np.cumsum([e.size for e in evs])]).astype(np.uint64)
    b = events.EventBatch(np.concatenate(evs), off)
    res, _ = run(b)
    r = oracle.run(b.subset(0, 2), geometry)
    for e in (0, 1, b.n_events - 1):
        assert not res["status"][e] & chain.STATUS["bad_raw"]
        want = r.event_clusters(e % 2)
        got = chain.event_clusters(res, e)
        assert [len(m["id"]) for m in got] == list(np.resize(np.roll(sizes, (0, 5)[e % 2]), 52))
        assert np.array_equal(np.sort(np.concatenate([m["id"] for m in got])), np.sort(want["id"]))
        for m in got:  # on (phi, id)
            order = np.lexsort((m["id"], m["phi"]))
            assert np.array_equal(order, np.arange(len(order)))
    assert event_bits(res, 0) == event_bits(res, b.n_events - 2)


@pytest.fixture(scope="module")
def full_run():
    """Batches of n events, their results with the vertex stage and nothing left out, and their
    events as bytes."""
    cache = {}

    def get(n):
        if n not in cache:
            b = events.generate(n, seed=9, nu_min=0.6, nu_max=0.6, with_mc=False)
            vc = chain.VeloChain(max_events=n, max_raw_bytes=int(b.raw.size) + 4096)
            vc.set_pv(True)
            vc.run_host(b)
            T, H, _ = vc.sync()
            res = vc.results()
            vc.close()
            assert T > 2 * n and H == res["track_hit_number"][T]
            assert np.array_equal(res["track_offsets"], np.concatenate([[0], np.cumsum(res["n_tracks"])]))
            res["n_hits"] = np.diff(res["track_hit_number"][res["track_offsets"]].astype(np.int64))
            cache[n] = b, res, T, H, [track_bits(res, e) for e in range(n)]
        return cache[n]
    return get


# 4,096 events and less are scanned by one block, more by many
@pytest.mark.parametrize("n", [5, 1025, 4096, 4097, 5121])
@pytest.mark.parametrize("tracks, hits", [(1.0, 1.0), (0.97, 1.0), (0.4, 1.0), (1.0, 0.97), (1.0, 0.4), (0.4, 0.97)])
@pytest.mark.parametrize("pv", [False, True])
def test_event_scan_and_output_capacity(full_run, n, tracks, hits, pv):
    """Of a batch beyond the output capacity every event is that of the full run, byte for byte,
    or flagged and without tracks, whatever an earlier run left in the buffers. The rule of the
    scan: 1,024 runs of events, each from the sum of all events before it; an event that does not
    fit keeps no tracks; what is kept lies packed."""
    b, full, T, H, want = full_run(n)
    cap_t, cap_h = int(T * tracks), int(H * hits)
    vc = chain.VeloChain(max_events=n, max_raw_bytes=2 * int(b.raw.size) + 4096, max_tracks=cap_t, max_track_hits=cap_h)
    vc.set_pv(pv)
    vc.run_host(events.generate(n, seed=10, nu_min=0.9, nu_max=0.9, with_mc=False))
    vc.sync()
    vc.run_host(b)
    totals = vc.sync()
    res = vc.results()
    vc.close()

    nt, nh = full["n_tracks"].astype(np.int64), full["n_hits"]
    st, sh = (np.concatenate([[0], np.cumsum(v)]) for v in (nt, nh))
    per = -(-n // 1024)
    over = np.zeros(n, bool)
    for a in range(0, n, per):
        t, h = st[a], sh[a]
        for e in range(a, min(n, a + per)):
            over[e] = t + nt[e] > cap_t or h + nh[e] > cap_h
            t, h = (t, h) if over[e] else (t + nt[e], h + nh[e])
    assert over.any() == (tracks < 1 or hits < 1) and not over.all()
    kept = np.where(over, 0, nt)
    assert np.array_equal(res["n_tracks"], kept)
    assert np.array_equal(res["track_offsets"], np.concatenate([[0], np.cumsum(kept)]))
    assert totals[:2] == (kept.sum(), np.where(over, 0, nh).sum()) and totals[0] <= cap_t and totals[1] <= cap_h
    assert np.array_equal((res["status"] & chain.STATUS["track_overflow"]) != 0, over)
    if not pv:
        full = {k: v for k, v in full.items() if not k.startswith("pv_")}
        want = [track_bits(full, e) for e in range(n)]
    for e in range(n):
        assert track_bits(res, e) == want[e] or over[e], e
    if pv:
        assert not res["pv_count"][over].any()


def tiled(b, n):
    """n copies of a batch, one after the other."""
    size = int(b.offsets[-1])
    off = np.concatenate([b.offsets[:-1] + np.uint64(k * size) for k in range(n)] + [[np.uint64(n * size)]])
    return events.EventBatch(np.tile(b.raw, n), off.astype(np.uint64))


def overfull_event(rng, modules):
    """125 clusters a sensor over the same 64 x 64 SPs of each: everything near everything, so that
    more tracks are followed than the ring holds."""
    payload, offs = [], [0]
    for sensor in range(208):
        n = 125 if sensor // 4 in modules else 0
        a = np.sort(rng.choice(64 * 64, n, replace=False))
        payload += [sensor, n] + [0x80000000 | ((int(x) // 64) << 6 | int(x) % 64) << 8 | 1 << int(rng.integers(8)) for x in a]
        offs.append(4 * len(payload))
    return np.array([208] + offs + payload, np.uint32).view(np.uint8)


def test_ring_overflow_does_not_depend_on_the_batch():
    """Events that overflow the ring of tracks to follow, which the reference leaves undefined: the
    same tracks on one warp, on four and on eight, whatever the batch."""
    import torch
    rng = np.random.default_rng(1)
    few = [overfull_event(rng, range(a, a + k)) for a, k in ((10, 8), (25, 8), (38, 14))]
    off = np.concatenate([[0], np.cumsum([e.size for e in few])]).astype(np.uint64)
    b = events.EventBatch(np.concatenate(few), off)
    # eight warps an event
    vc = chain.VeloChain(max_events=3, max_raw_bytes=int(b.raw.size) + 4096, max_tracks=3600)
    vc.run_host(b)
    vc.sync()
    res = vc.results()
    assert np.all(res["status"] & chain.STATUS["ttf_overflow"]) and res["n_tracks"].min() > 100
    want = [track_bits(res, e) for e in range(3)]
    # one warp an event, windows computed in place
    track_n, track_hits = (torch.zeros(3 * 1200 * k, dtype=torch.int16, device="cuda") for k in (1, 26))
    n_tracks, status = (torch.zeros(3, dtype=torch.int32, device="cuda") for _ in range(2))
    status_in = torch.from_numpy(res["status"].astype(np.int32) & chain.STATUS["candidate_overflow"]).cuda()
    o = vc.out
    assert vc.lib.velo_search_static(o.hit_xyzp, o.module_hit_start, o.module_hit_num, status_in.data_ptr(), 3,
                                     track_n.data_ptr(), track_hits.data_ptr(), n_tracks.data_ptr(), status.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    vc.close()
    assert np.array_equal(n_tracks.cpu().numpy(), res["n_tracks"]) and np.array_equal(status.cpu().numpy(), res["status"])
    tn, th = track_n.cpu().numpy().reshape(3, 1200), track_hits.cpu().numpy().view(np.uint16).reshape(3, 1200, 26)
    for e in range(3):
        ids = res["cluster_id"][int(res["module_start"][52 * e]):]
        assert [tuple(ids[th[e, t, :tn[e, t]]]) for t in range(n_tracks[e])] == chain.event_tracks(res, e)
    # four warps an event, each event a large one of its batch
    small = events.generate(700, seed=3, nu_min=2.0, nu_max=4.0, with_mc=False)
    mixed = events.EventBatch(np.concatenate([b.raw, small.raw]), np.concatenate([b.offsets, small.offsets[1:] + b.offsets[3]]))
    got, _ = run(mixed)
    assert [track_bits(got, e) for e in range(3)] == want
    # one warp an event in a full device (the third, the larger one, takes a block)
    n = 1600
    got, _ = run(tiled(b, n), max_tracks=1200 * 3 * n)
    assert all(track_bits(got, e) == want[e % 3] for e in range(3 * n))


def warp_events(hits, sms):
    """Events that the order kernel's rule leaves a warp each: up to 12,288 clusters, and no longer
    than a warp's share of the batch."""
    mid = (np.asarray(hits, np.int64) // 16) * 16 + 8.0
    cost = mid * (mid + 2000.0)
    return (np.asarray(hits) < 12288) & (cost * (32 * sms) <= cost.sum())


@pytest.mark.parametrize("mode", ["plain", "extension"])
def test_one_warp_an_event_in_a_full_device(mode, batch_700):
    """A batch that fills the device: most events take a warp each, the largest a block, and every
    copy equals the event in a small batch of one block an event, whose tracks other tests compare
    with the reference's. In the pruned mode every candidate is scored and forwarding is pruned too."""
    sms = batch_700[2]
    b = golden_batch("batched")
    w = None
    if mode == "extension":
        w = mlp.load_weights(train_scorer.DEFAULT_WEIGHTS)
        w.min_pairs = w.min_event_clusters = 0
        w.ext_threshold = 0.3
    small, full = [], []
    for batch, mapping, out in ((b, chain.MAP_BLOCK, small), (tiled(b, 280), chain.MAP_WARP, full)):
        vc = chain.VeloChain(max_events=batch.n_events, max_raw_bytes=int(batch.raw.size) + 4096, mapping=mapping)
        if w is not None:
            vc.set_mlp(w)
            vc.set_mode(chain.MODE_PRUNED)
        vc.run_host(batch)
        vc.sync()
        res = vc.results()
        vc.close()
        out += [track_bits(res, e) for e in range(batch.n_events)]
    warp = warp_events(res["module_num"].reshape(-1, 52).sum(1), sms)
    assert warp.sum() > 4000 and (~warp).sum() > 500
    if w is not None:
        assert not (res["status"] & chain.STATUS["mlp_fallback"]).any() and (res["cluster_keep"] & 2 == 0).any()
    for e, got in enumerate(full):
        assert got == small[e % 32], e


def test_largest_events_of_one_warp():
    """A warp's used-hit bits hold 12,288 clusters: events of 12,272 to 12,287 take one in a batch
    that fills the device, those above a block, and each equals itself in a small batch."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(7)
    sizes = [12272, 12286, 12287, 12288, 12289, 12304]
    few = [sp_event(rng, np.full(52, n // 52) + (np.arange(52) < n % 52)) for n in sizes]
    off = np.concatenate([[0], np.cumsum([e.size for e in few])]).astype(np.uint64)
    b = events.EventBatch(np.concatenate(few), off)
    ref, _ = run(b, max_tracks=1200 * 6)
    assert ref["module_num"].reshape(-1, 52).sum(1).tolist() == sizes and ref["n_tracks"].min() > 0
    want = [track_bits(ref, e) for e in range(6)]
    n = 6 * (7 * 32 * sms // 36)
    assert warp_events(sizes * (n // 6), sms).tolist() == [True, True, True, False, False, False] * (n // 6)
    many = tiled(b, n // 6)
    vc = chain.VeloChain(max_events=n, max_raw_bytes=int(many.raw.size) + 4096, max_tracks=1200 * n, max_track_hits=6000 * n)
    vc.run_host(many)
    vc.sync()
    res = vc.results(clusters=False)
    vc.close()
    for e in range(n):
        assert track_bits(res, e) == want[e % 6], e

"""The launch shapes and paths that a batch's size, an event's occupancy or a module's size
chooses, at the sizes where one takes over from the next: every event's result is the same
whatever the batch it comes in."""
import numpy as np
import pytest

import oracle
from cuda_hlt_b200 import chain, events
from test_gpu_windows import windows_of

pytestmark = pytest.mark.gpu


def run(b, max_tracks=0, max_track_hits=0, **kw):
    vc = chain.VeloChain(max_events=b.n_events, max_raw_bytes=int(b.raw.size) + 4096, max_tracks=max_tracks,
                         max_track_hits=max_track_hits, **kw)
    vc.run_host(b)
    totals = vc.sync()
    res = vc.results()
    vc.close()
    return res, totals


def event_bits(res, e):
    """Everything the chain says of one event, as comparable bytes."""
    t0, t1 = int(res["track_offsets"][e]), int(res["track_offsets"][e + 1])
    h0, h1 = int(res["track_hit_number"][t0]), int(res["track_hit_number"][t1])
    parts = [res["status"][e], res["track_hit_number"][t0:t1 + 1] - h0, res["hit_id"][h0:h1]]
    parts += [res[k][h0:h1] for k in ("hit_x", "hit_y", "hit_z")]
    parts += [res[s][k][t0:t1] for s in ("states", "kalman") for k in chain.STATE_FIELDS]
    for m in chain.event_clusters(res, e):
        parts += [m[k] for k in ("id", "phi", "x", "y", "z", "size")]
    return b"".join(np.ascontiguousarray(p).tobytes() for p in parts)


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


def test_large_events_search_their_windows_by_parity():
    """More events than the wide decode takes, some above the 8,192 clusters whose phi fit the
    shared memory together."""
    b = events.generate_config("high_occupancy_200k", n_events=330, first_event=0, with_mc=False)
    vc = chain.VeloChain(max_events=330, max_raw_bytes=int(b.raw.size) + 4096)
    vc.run_host(b)
    vc.sync()
    res = vc.results()
    assert res["module_num"].reshape(-1, 52).sum(1).max() > 8192
    windows_of(vc, res, 330)
    vc.close()


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


@pytest.mark.parametrize("n", [4096, 4097, 5121])
@pytest.mark.parametrize("capacity", [1.0, 0.97])
def test_event_scan_and_output_capacity(n, capacity):
    """Above 4,096 events the scan runs over many blocks. In a batch beyond the output capacity
    the rule of the one-block scan holds: 1,024 runs of events, each from the sum of all events
    before it, an event that does not fit keeps no tracks and is flagged."""
    b = events.generate(n, seed=9, nu_min=0.6, nu_max=0.6, with_mc=False)
    full, (T, H, _) = run(b)
    assert T > 2 * n
    nt = full["n_tracks"].astype(np.int64)
    starts = np.concatenate([[0], np.cumsum(nt)])
    assert np.array_equal(full["track_offsets"], starts) and full["track_hit_number"][T] == H
    cap_t = int(T * capacity)
    vc = chain.VeloChain(max_events=n, max_raw_bytes=int(b.raw.size) + 4096, max_tracks=cap_t, max_track_hits=16 * T)
    vc.run_host(b)
    totals = vc.sync()
    atomics, status = (vc._down(p, np.uint32, k) for p, k in ((vc.out.atomics, 2 * n + 1), (vc.out.status, n)))
    vc.close()
    per = -(-n // 1024)
    kept, over, offsets = np.zeros(n, np.int64), np.zeros(n, bool), np.zeros(n + 1, np.int64)
    for a in range(0, n, per):
        at = starts[a]
        for e in range(a, min(n, a + per)):
            over[e] = at + nt[e] > cap_t
            kept[e] = 0 if over[e] else nt[e]
            offsets[e] = at
            at += kept[e]
        offsets[n] = at
    assert np.array_equal(atomics[:n], kept) and np.array_equal(atomics[n:], offsets) and totals[0] == offsets[n]
    assert np.array_equal((status & chain.STATUS["track_overflow"]) != 0, over) and over.any() == (capacity < 1)

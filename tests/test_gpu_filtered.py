"""The filtered mixed-precision paths and the ZHS deposits as differences, where
their bins sit on an edge: traces of one, two and odd numbers of bins, cut
through the pulse at either end, samples at whole and half bins, and antennas
inside a track's reach.  FP64 traces equal the oracle's bit for bit; mixed
precision's sample counts per bin and counters equal the oracle's, and its
amplitudes are the oracle's to FP32."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

COUNTERS = ("coreas_contributions", "zhs_contributions", "zhs_subtracks", "valid_tracks", "fixed_point_overflows")


def project(pkg, config, records, tuning=None):
    import torch

    raw = torch.from_numpy(np.ascontiguousarray(records).view(np.uint8).reshape(-1)).cuda()
    acc = pkg.RadioAccumulator(config, tuning)
    acc.accumulate_lepton_tracks(raw.data_ptr(), records.size)
    got = acc.download_fixed()
    acc.close()
    return got


# Mixed against FP64 traces, relative to a trace's 2-norm and to its peak: a sample's
# amplitude takes a dozen FP32 roundings (2^-24 each: 7e-7 in all) and, where the Doppler
# factor is as small as the filtered paths take it (1e-6), 2^-43 of that factor, 1.2e-7;
# samples of opposite sign cancel in a bin.  Measured up to 1.1e-6 and 1.7e-6.  Not
# where a track's two CoREAS samples share their bin and all but cancel
# (amplitudes=False): what is left of 1e11 units is then their rounding.
MIXED_BOUND = 5e-6


def check(pkg, oracle, showers, workload, records, tuning=None, amplitudes=True, **extra):
    for precision, counting in ((0, False), (0, True), (1, True)) + (((1, False),) if amplitudes else ()):
        config = showers.make_config(workload, precision=precision, kernel=2, count_samples=counting, **extra)
        got = project(pkg, config, records, tuning)
        want = oracle.restatement().project(showers.make_config(workload, count_samples=counting, **extra), records,
                                            threads=16)
        for k in range(2):
            if precision == 0 or counting:
                assert np.array_equal(got[k], want[k]), (precision, counting, k, np.count_nonzero(got[k] != want[k]))
                continue
            ends = np.cumsum(workload["observers"]["number_of_bins"].astype(int))
            for g, w in zip(np.split(got[k], ends[:-1], axis=1), np.split(want[k], ends[:-1], axis=1)):
                error, w = g.astype(np.float64) - w, w.astype(np.float64)
                units = len(records)  # a sample's conversion rounds by half a unit
                assert np.linalg.norm(error) <= MIXED_BOUND * np.linalg.norm(w) + units, k
                assert np.abs(error).max() <= MIXED_BOUND * np.abs(w).max() + units, k
        for key in COUNTERS:
            assert got[2][key] == want[2][key], (precision, counting, key)


@pytest.mark.parametrize("bins", [1, 2, 31, 32, 33, 97, 1023, 4099])
def test_traces_cut_through_the_pulse(pkg, oracle, showers, bins):
    wl, gen, _ = showers.workload_config("plain_c0", bins=bins)
    records = showers.shower_records(20_003, seed=17 + bins, **gen)
    observers = wl["observers"].copy()
    observers["start_time_s"] += np.linspace(30e-9, 70e-9, len(observers))  # from before the pulse into it
    wl["observers"] = observers
    check(pkg, oracle, showers, wl, records, pkg.TuningParameters(track_tile_size=4000))


def test_samples_at_whole_and_half_bins(pkg, oracle, showers):
    """Tracks along one line towards an antenna in vacuum: every arrival is a
    whole or half number of bins, so no guard can decide and each pair takes the
    exact evaluation."""
    c = showers.SPEED_OF_LIGHT
    count = 4096
    step = c / 1e10  # one bin of path
    start = np.zeros((count, 3))
    start[:, 2] = 1000.0 + 0.5 * step * np.arange(count)
    direction = np.tile([0.0, 0.0, -1.0], (count, 1))
    length = np.full(count, 8 * step)
    t0 = np.zeros(count)
    seg = dict(start=start, end=start + length[:, None] * direction, t_start=t0, t_end=t0 + length / (0.5 * c),
               pid=np.where(np.arange(count) % 2, 11, -11).astype(np.int32), energy_gev=np.full(count, 1e-3),
               direction=direction, weight=np.ones(count))
    observers = np.zeros(3, pkg.abi.OBSERVER)
    observers["position_m"][1] = (3.0, 0.0, 0.0)
    observers["position_m"][2] = (0.0, 0.0, 1200.0)  # between the tracks
    observers["start_time_s"] = (1000.0 / c, 1000.0 / c, 0.0)
    observers["duration_s"] = 2047 / 1e10
    observers["sample_rate_hz"] = 1e10
    observers["number_of_bins"] = 2048
    wl = dict(observers=observers, homogeneous=1.0, table=None)
    check(pkg, oracle, showers, wl, showers.to_records(seg))


@pytest.mark.parametrize("edge,duration", [("end", 1e-3), ("end", 1.3), ("start", 1e-3), ("start", 1.1), ("start", 2.7)])
def test_detection_time_just_below_the_first_half_bin(pkg, oracle, showers, edge, duration):
    """The one detection time x (in bins) whose floor(x + 1/2) is not its nearest
    bin: 1/2 less a unit in the last place, at which x + 1/2 rounds to 1.  The
    track passes its antenna at a right angle (k.beta = 0), so a detection time is
    a track time plus the travel time and can be placed there exactly."""
    below = np.nextafter(0.5, 0.0)
    height = 1.0e6
    travel = height / showers.SPEED_OF_LIGHT
    if edge == "end":
        t_end = below - travel
        t_start = t_end - duration
        t_end = t_start + (t_end - t_start)
        assert t_end + travel == below
    else:
        t_start = below - travel
        t_end = t_start + duration
        assert t_start + travel == below
    seg = dict(start=np.array([[-500.0, 0.0, height]]), end=np.array([[500.0, 0.0, height]]),
               t_start=np.array([t_start]), t_end=np.array([t_end]), pid=np.array([11], np.int32),
               energy_gev=np.array([1e-3]), direction=np.array([[1.0, 0.0, 0.0]]), weight=np.array([1e18]))
    observers = np.zeros(1, pkg.abi.OBSERVER)
    observers["duration_s"] = 7.0
    observers["sample_rate_hz"] = 1.0
    observers["number_of_bins"] = 8
    wl = dict(observers=observers, homogeneous=1.0, table=None)
    check(pkg, oracle, showers, wl, showers.to_records(seg), amplitudes=False)


def test_divided_tracks_above_the_table_beside_the_antenna_height(pkg, oracle, showers):
    """Divided tracks past the table's upper end, a few nanometres above the
    antenna: the travel time's factor 1 + (I - I_antenna) / height then turns on
    differences at the rounding of the height itself."""
    count = 3000
    rng = np.random.default_rng(8)
    table = vars(cases.uniform_table(1.0003, 0.0, 2000.0, 1.0))
    z = 2000.0 + rng.uniform(1e-9, 8e-9, count)
    start = np.stack([np.zeros(count), np.full(count, -50.0), z], axis=1)
    end = np.stack([np.zeros(count), np.full(count, 50.0), z + rng.uniform(-1e-9, 1e-9, count)], axis=1)
    t0 = rng.uniform(0.0, 100e-9, count)
    observers = np.zeros(1, pkg.abi.OBSERVER)
    observers["position_m"][0] = (3.0e4, 0.0, 2000.0 - 1e-9)
    observers["start_time_s"] = 3.0e4 / showers.SPEED_OF_LIGHT
    observers["duration_s"] = 8191 / 1e10
    observers["sample_rate_hz"] = 1e10
    observers["number_of_bins"] = 8192
    seg = dict(start=start, end=end, t_start=t0, t_end=t0 + 100.0 / (0.99 * showers.SPEED_OF_LIGHT),
               pid=np.full(count, 11, np.int32), energy_gev=np.full(count, 1e-3),
               direction=np.tile([0.0, 1.0, 0.0], (count, 1)), weight=np.ones(count))
    wl = dict(observers=observers, homogeneous=0.0, table=table)
    check(pkg, oracle, showers, wl, showers.to_records(seg), amplitudes=False)


@pytest.mark.parametrize("name,refinement,shift", [("ice_c2", 1, 0.0), ("ice_c2", 3, 0.0), ("plain_c0", 1, 52e-9), ("plain_c0", 2, 0.0)])
@pytest.mark.parametrize("precision", [0, 1])
def test_items_run_again_give_the_same_bits(pkg, oracle, showers, name, refinement, shift, precision):
    """A sample's fixed-point value does not depend on the way its item went: one
    item an antenna near the fixed-point limit, run again with checked adds,
    against items so small that none is (which items are depends on the order that
    the ingest's atomics leave the tracks in, so else the traces would too)."""
    import torch

    wl, gen, _ = showers.workload_config(name, bins=1001)
    records = (showers.ice_records if gen.get("ice") else showers.shower_records)(6_000, seed=3, **gen)
    wl["observers"] = wl["observers"][::5].copy()
    wl["observers"]["start_time_s"] += shift  # into the pulse: the trace's start cuts segments
    extra = dict(zhs_subtrack_refinement=refinement)
    floating = showers.make_config(wl, deterministic=False, **extra)
    coreas, zhs, _ = oracle.restatement().project(floating, records, threads=16)
    peak = max(np.abs(coreas).max(), 1e10 * np.abs(zhs).max())
    config = showers.make_config(wl, precision=precision, kernel=2, **extra)
    config.fixed_point_field_limit_v_per_m = 1.5 * peak
    raw = torch.from_numpy(records.view(np.uint8).reshape(-1)).cuda()
    got = []
    for tracks in (8192, 32):
        acc = pkg.RadioAccumulator(config, pkg.TuningParameters(track_tile_size=tracks))
        acc.accumulate_lepton_tracks(raw.data_ptr(), records.size)
        got.append(acc.download_fixed() + (acc.statistics().window_reruns,))
        acc.close()
    assert got[0][3] > 0
    for k in range(2):
        assert np.array_equal(got[0][k], got[1][k]), (k, np.count_nonzero(got[0][k] != got[1][k]))


@pytest.mark.parametrize("refinement", [1, 3, 64])
def test_divided_tracks_inside_the_cone(pkg, oracle, showers, refinement):
    """Tracks in ice seen from inside and outside the Cherenkov cone (Doppler factors
    of both signs), divided for the antennas, then refined as well."""
    wl, gen, _ = showers.workload_config("ice_c2", bins=1000)
    records = showers.ice_records(4_001, seed=5, **gen)
    wl["observers"] = wl["observers"][::5].copy()
    check(pkg, oracle, showers, wl, records, zhs_subtrack_refinement=refinement)


@pytest.mark.parametrize("scale", [1e-6, 1e3, 1e6])
def test_times_outside_the_guards_reach(pkg, oracle, showers, scale):
    """Track times shifted until the filtered paths' bounds no longer cover them
    (the last scales): those tracks are evaluated exactly."""
    wl, gen, _ = showers.workload_config("ice_c2", bins=1000)
    records = showers.ice_records(6_001, seed=5, **gen)
    shift = 3.7e-6 * scale
    records["start"]["time_s"] += shift
    records["end"]["time_s"] += shift
    wl["observers"] = wl["observers"][::5].copy()
    wl["observers"]["start_time_s"] += shift
    check(pkg, oracle, showers, wl, records)


@pytest.mark.parametrize("count", [1, 255, 256, 257, 1500, 16_385])
@pytest.mark.parametrize("deterministic", [True, False])
def test_automatic_route_at_every_size(pkg, oracle, showers, count, deterministic):
    """The automatic choice (direct below 256 tracks, windowed above, items cut
    evenly over the GPU) gives the oracle's traces: bit for bit in fixed point, to
    the order of FP64 sums in floating point."""
    wl, gen, _ = showers.workload_config("plain_c0", bins=1500)
    wl["observers"] = wl["observers"][:5].copy()
    records = showers.shower_records(count, seed=91, **gen)
    config = showers.make_config(wl, deterministic=deterministic)
    want = oracle.restatement().project(config, records, threads=8)
    if deterministic:
        got = project(pkg, config, records)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        counters = got[2]
    else:
        import torch

        raw = torch.from_numpy(records.view(np.uint8).reshape(-1)).cuda()
        acc = pkg.RadioAccumulator(config)
        acc.accumulate_lepton_tracks(raw.data_ptr(), records.size)
        waveforms = acc.download()
        acc.close()
        for g, w in ((waveforms.coreas, want[0]), (waveforms.zhs, want[1])):
            assert np.abs(g - w).max(initial=0.0) <= 1e-28 + 2e-12 * np.abs(w).max(initial=0.0)
        counters = waveforms.counters
    for key in COUNTERS:
        assert counters[key] == want[2][key], key


@pytest.mark.parametrize("sizes", [(20_011,), (100, 9_000, 4_096, 1), (70_003,)])
def test_pageable_host_calls_of_many_records(pkg, oracle, showers, sizes):
    """Host calls that fill several batches (ingested as they fill, projected
    together) and calls that leave a batch part full."""
    wl, gen, _ = showers.workload_config("plain_c0", bins=2048)
    records = showers.shower_records(sum(sizes), seed=95, **gen)
    config = showers.make_config(wl)
    want = oracle.restatement().project(config, records, threads=16)
    acc = pkg.RadioAccumulator(config)
    begin = 0
    for size in sizes:
        acc.enqueue_host_lepton_tracks(records[begin:begin + size])
        begin += size
    got = acc.download_fixed()
    stats = acc.statistics()
    acc.close()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert stats.host_tracks_enqueued == records.size
    assert stats.host_track_batches == -(-records.size // 4096)

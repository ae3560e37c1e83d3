"""The work a user of the radio library has it do, as measurable cases.

A case is one or several showers projected from their track records to the
downloaded antenna traces through the package's public classes: a fresh event
on a kept accumulator (or batch, or server) -- reset, hand over the tracks,
project, download.  The listed cases go from a shower of a thousand segments
to the 1e7-segment, 160-antenna workload, in both precisions, with fixed-point
and floating traces, from host records, pinned host records, device records
and device columns, in air and ice, and over the batched and served forms.

Segments are drawn on the GPU from the seed with the distributions of the
package's shower generator (Gaisser-Hillas profile, exponential lateral
spread and lengths, Gaussian angles, log-uniform energies).
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
PACKAGE = "corsika8_kokkos_b200"
C = 299792458.0
ELECTRON_MASS_GEV = 5.109989e-4
GROUND = 1400.0
RATE = 1e10


def package():
    """The repository's package (its folder's name carries a hyphen)."""
    if PACKAGE not in sys.modules:
        folder = ROOT / "corsika8-kokkos_b200"
        spec = importlib.util.spec_from_file_location(PACKAGE, folder / "__init__.py",
                                                      submodule_search_locations=[str(folder)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[PACKAGE] = module
        spec.loader.exec_module(module)
    return sys.modules[PACKAGE]


def showers():
    package()
    return importlib.import_module(PACKAGE + ".showers")


# Every key a case has, with its ordinary value.
#   medium     air (refractivity table) or ice (uniform n = 1.78)
#   precision  fp64 (the bit-exact drop-in) or mixed (FP64 times, FP32 amplitudes)
#   traces     fixed (int64, the production default) or float
#   input      host (pageable records, default host batches), pinned, device or columns
#   output     download (decoded traces), fixed (int64 traces), pinned (decoded into pinned memory)
#   form       alone, batch (events projected together, graph replay) or served
#   terrain    1: every antenna at a height of its own
DEFAULTS = dict(medium="air", segments=100_000, antennas=16, bins=4096, zenith=30.0, precision="fp64",
                traces="fixed", input="device", output="download", form="alone", events=1,
                algorithms="both", refinement=1, diagnostics=False, terrain=False, pre_trigger_ns=50.0)


def case(**kw):
    return {**DEFAULTS, **kw}


def listed():
    return [
        # one small shower handed over by a CPU cascade: latency and launches
        case(name="small_event_host", segments=1_500, antennas=16, zenith=0.0, input="host"),
        # the plain drop-in: host records through the default 4096-record batches
        case(name="host_batches_fp64", segments=60_001, antennas=48, bins=4096, input="host"),
        # the small plain workload: 1e5 segments x 16 antennas, device records
        case(name="plain_c0_fp64", segments=100_000, antennas=16, zenith=0.0, output="fixed"),
        # device steps as columns with track diagnostics, mixed precision
        case(name="columns_mixed", segments=262_147, antennas=40, precision="mixed", input="columns",
             diagnostics=True, zenith=45.0),
        # the production workload: 1e7 segments x 160 antennas x 8192 bins
        case(name="shower_1e7_mixed", segments=10_000_000, antennas=160, bins=8192, precision="mixed"),
        # the same geometry as the FP64 drop-in, 1e6 segments
        case(name="shower_1e6_fp64", segments=1_000_000, antennas=160, bins=8192),
        # in-ice cascade on the Cherenkov cone: near-cone branch and subdivision count here
        case(name="ice_mixed", medium="ice", segments=5_000_000, antennas=64, precision="mixed"),
        # antennas on a slope (no shared destination row), ragged sizes, floating traces
        case(name="terrain_float_fp64", segments=333_333, antennas=61, bins=3001, zenith=55.0,
             traces="float", terrain=True),
        # ZHS potential only, tracks refined threefold (the convergence study's option)
        case(name="zhs_refined_mixed", segments=150_001, antennas=24, precision="mixed", algorithms="zhs",
             refinement=3),
        # 2 us traces: longer than one shared-memory window holds
        case(name="long_traces_mixed", segments=250_000, antennas=30, bins=20_000, precision="mixed",
             zenith=0.0, pre_trigger_ns=800.0),
        # several showers in one call, records staged, graph replay
        case(name="batch_mixed", form="batch", events=6, segments=400_000, antennas=96, precision="mixed",
             zenith=40.0),
        # showers arriving at the server together
        case(name="served_mixed", form="served", events=5, segments=600_000, antennas=120, precision="mixed",
             zenith=20.0),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kw = dict(zenith=round(rng.uniform(0.0, 60.0), 2), precision=rng.choice(["fp64", "mixed"]),
              antennas=size(5, 240), bins=rng.choice([rng.randint(900, 8400), 4096, 8192]))
    kind = rng.choice(["host", "device", "device", "columns", "ice", "float", "zhs", "long", "pinned", "batch",
                       "served"])
    pairs = 2.5e8  # at most this many track-antenna pairs
    lo, hi = 3_000, 3_000_000
    if kind == "host":
        kw.update(input="host")
        pairs, lo, hi = 6e6, 700, 100_000
    elif kind == "columns":
        kw.update(input="columns", diagnostics=rng.choice([True, False]), terrain=rng.choice([True, False]))
    elif kind == "pinned":
        kw.update(input="pinned", output="pinned")
        hi = 300_000
    elif kind == "ice":
        kw.update(medium="ice", antennas=rng.randint(4, 64), bins=rng.randint(1500, 4096))
    elif kind == "float":
        kw.update(traces="float", terrain=rng.choice([True, False]))
        pairs = 5e7
    elif kind == "zhs":
        kw.update(algorithms=rng.choice(["zhs", "zhs", "coreas"]), refinement=rng.randint(1, 4))
        pairs = 3e7
    elif kind == "long":
        kw.update(bins=rng.randint(9_000, 24_000), pre_trigger_ns=round(rng.uniform(50.0, 900.0), 1))
        pairs, hi = 2e7, 400_000
    elif kind in ("batch", "served"):
        kw.update(form=kind, events=rng.randint(2, 7), output="download")
        pairs, hi = 4e7, 600_000
    kw["segments"] = max(lo, min(size(lo, hi), int(pairs / kw["antennas"])))
    return case(**kw)


# ------------------------------------------------------------------ inputs
def event_cases(c):
    """The events of a case: one, or for batch and served several of different sizes."""
    if c["form"] == "alone":
        return [c]
    share = [1.0, 0.31, 0.08, 0.55, 0.17, 0.74, 0.044]
    return [dict(c, segments=max(64, int(c["segments"] * share[k % 7]) | 1),
                 antennas=max(3, int(c["antennas"] * share[(3 * k + 1) % 7])),
                 zenith=(c["zenith"] + 7.0 * k) % 60.0) for k in range(c["events"])]


def air_observers(c):
    s = showers()
    arms = 8
    radii = list(np.linspace(25.0, 500.0, max(1, -(-c["antennas"] // arms))))
    pre = c["pre_trigger_ns"] * 1e-9
    out = s.star_antennas(arms, radii, GROUND, c["bins"], RATE, zenith_deg=c["zenith"],
                          pre_trigger_s=pre)[: c["antennas"]].copy()
    if c["terrain"]:
        up, _, _ = s.shower_axis(c["zenith"], 0.0)
        height = np.random.default_rng(11).uniform(0.0, 250.0, out.size)
        for k in range(out.size):
            out[k]["position_m"][2] += height[k]
            offset = np.array(out[k]["position_m"]) - np.array([0.0, 0.0, GROUND])
            out[k]["start_time_s"] = float(np.dot(offset, -up)) / C - pre
    return out


def workload(c):
    s = showers()
    if c["medium"] == "ice":
        wl, _, _ = s.workload_config("ice_c2", segments=c["segments"], bins=c["bins"])
        order = np.random.default_rng(5).permutation(len(wl["observers"]))
        wl["observers"] = wl["observers"][order][: c["antennas"]].copy()
        return wl
    return dict(observers=air_observers(c), homogeneous=0.0,
                table=s.flat_atmosphere_table(s.AtmosphereModel(), GROUND, 30000.0, 1.0))


def config(c):
    return showers().make_config(
        workload(c), precision=1 if c["precision"] == "mixed" else 0, deterministic=c["traces"] == "fixed",
        coreas=c["algorithms"] in ("both", "coreas"), zhs=c["algorithms"] in ("both", "zhs"),
        track_diagnostics=c["diagnostics"], zhs_subtrack_refinement=c["refinement"])


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def depths(u, w, lam, xmax, stop):
    """Gaisser-Hillas depths by the inverse of the profile's running integral
    (summed on the host: a parallel running sum has no fixed order)."""
    x = np.linspace(0.0, stop, 20000)
    logn = w * np.log(np.maximum(x / xmax, 1e-300)) + (xmax - x) / lam
    pdf = np.exp(logn - logn.max())
    cdf = np.concatenate([[0.0], np.cumsum(0.5 * (pdf[1:] + pdf[:-1]) * (x[1] - x[0]))])
    cdf, x = (torch.from_numpy(v).to(u.device) for v in (cdf / cdf[-1], x))
    k = torch.clamp(torch.searchsorted(cdf, u), 1, x.numel() - 1)
    step = torch.clamp(cdf[k] - cdf[k - 1], min=1e-300)
    return x[k - 1] + (u - cdf[k - 1]) / step * (x[k] - x[k - 1])


def segments(c, seed):
    """Columns of one shower's track segments on the GPU, FP64."""
    s = showers()
    dev, n, air = device(), c["segments"], c["medium"] == "air"
    g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 13)

    def uniform():
        return torch.rand(n, generator=g, dtype=torch.float64, device=dev)

    def exponential(mean):
        return -mean * torch.log1p(-uniform())

    zenith = c["zenith"] if air else 50.0
    up, e1, e2 = s.shower_axis(zenith, 0.0)
    if air:
        model = s.AtmosphereModel()
        cos_z = math.cos(math.radians(zenith))
        ground = float(model.vertical_depth(GROUND)) / cos_z
        depth = torch.clamp(depths(uniform(), 700.0 / 70.0, 70.0, 700.0, ground), min=1e-3)
        top = model.rho0_g_cm3 * model.scale_height_m * 100.0
        height = -model.scale_height_m * torch.log(depth * cos_z / top)
        along = (height - GROUND) / cos_z  # above the core, against the shower direction
        lateral, mean, longest = 30.0, 1.0, 10.0
    else:
        xmax = 7.6 * 0.92 * 100.0
        along = -(depths(uniform(), xmax / 70.0, 70.0, xmax, 4.0 * xmax) / 92.0 - 7.6)
        lateral, mean, longest = 0.1, 0.05, 0.5
    r, phi = exponential(lateral), 2.0 * math.pi * uniform()
    k1 = torch.randn(n, generator=g, dtype=torch.float64, device=dev) * math.radians(5.0)
    k2 = torch.randn(n, generator=g, dtype=torch.float64, device=dev) * math.radians(5.0)
    core = (0.0, 0.0, GROUND if air else 0.0)
    start = [core[a] + along * up[a] + r * torch.cos(phi) * e1[a] + r * torch.sin(phi) * e2[a] for a in range(3)]
    direction = [k1 * e1[a] + k2 * e2[a] - up[a] for a in range(3)]
    norm = torch.sqrt(sum(d * d for d in direction))
    direction = [d / norm for d in direction]
    length = torch.clamp(exponential(mean), min=1e-9, max=longest)
    kinetic = torch.exp(math.log(1e-3) + uniform() * math.log(1e3))
    gamma = 1.0 + kinetic / ELECTRON_MASS_GEV
    beta = torch.sqrt(1.0 - 1.0 / (gamma * gamma))
    t0 = -along / C + (r * r / (2.0 * C * 5000.0) if air else 0.0)
    pid = torch.where(uniform() < 0.6, 11, -11)
    pid = torch.where(uniform() < 0.01, 22, pid).to(torch.int32)  # a few photons, which radio skips
    return dict(pid=pid, weight=1.0 + 4.0 * (uniform() < 0.1).double(), energy=kinetic + ELECTRON_MASS_GEV,
                start=start, end=[start[a] + length * direction[a] for a in range(3)], direction=direction,
                t0=t0, t1=t0 + length / (beta * C))


def records(seg):
    """LeptonTransportRecords (752 bytes each) as a (n, 94) FP64 tensor on the GPU."""
    abi = package().abi
    raw = torch.zeros(seg["pid"].numel(), abi.LEPTON_RECORD.itemsize // 8, dtype=torch.float64, device=seg["t0"].device)
    at = {name: abi.PARTICLE_STATE.fields[name][1] // 8 for name in abi.PARTICLE_STATE.names}
    for state, position, time in (("start", "start", "t0"), ("end", "end", "t1")):
        base = abi.LEPTON_RECORD.fields[state][1] // 8
        raw.view(torch.int32)[:, 2 * (base + at["pid"])] = seg["pid"]
        raw[:, base + at["energy_gev"]] = seg["energy"]
        raw[:, base + at["time_s"]] = seg[time]
        raw[:, base + at["weight"]] = seg["weight"]
        for a in range(3):
            raw[:, base + at["position_m"] + a] = seg[position][a]
            raw[:, base + at["direction"] + a] = seg["direction"][a]
    return raw


def prepare(c, seed):
    pkg = package()
    events = event_cases(c)
    segs = [segments(e, seed * 101 + k) for k, e in enumerate(events)]
    state = {"case": c, "counts": [e["segments"] for e in events]}
    stream = None
    if c["form"] == "batch":
        state["stream"] = torch.cuda.Stream()
        stream = state["stream"].cuda_stream
    tuning = pkg.TuningParameters(batch_size=65536) if c["input"] == "pinned" else None
    configs = [config(e) for e in events]
    if c["form"] == "served":
        bytes_ = sum(2 * 128 * e["segments"] + 6 * 16 * e["antennas"] * e["bins"] for e in events)
        state["server"] = pkg.RadioServer(2 * bytes_ + (1 << 30))
        state["configs"] = configs
    else:
        state["events"] = [pkg.RadioAccumulator(g, tuning, stream) for g in configs]
    if c["form"] == "batch":
        state["batch"] = pkg.RadioBatch(stream)
    if c["input"] == "columns":
        state["keep"] = segs
        state["columns"] = [
            dict(pid=s["pid"].data_ptr(), weight=s["weight"].data_ptr(), start_time_s=s["t0"].data_ptr(),
                 end_time_s=s["t1"].data_ptr(), start_energy_gev=s["energy"].data_ptr(),
                 start_position_m=tuple(t.data_ptr() for t in s["start"]),
                 end_position_m=tuple(t.data_ptr() for t in s["end"]),
                 start_direction=tuple(t.data_ptr() for t in s["direction"]),
                 end_direction=tuple(t.data_ptr() for t in s["direction"])) for s in segs]
    else:
        state["records"] = [records(s) for s in segs]
        if c["input"] in ("host", "pinned"):
            host = []
            for raw in state["records"]:
                copy = torch.empty(raw.shape, dtype=raw.dtype, pin_memory=c["input"] == "pinned")
                copy.copy_(raw)
                host.append(copy)
            state["records"] = host
            state["host"] = [h.numpy().view(pkg.LEPTON_RECORD).reshape(-1) for h in host]
    if c["output"] == "pinned":
        state["out"] = [tuple(torch.empty(3 * b, dtype=torch.float64, pin_memory=True).numpy()
                              for b in (e.coreas_bins, e.zhs_bins)) for e in state["events"]]
    return state


# --------------------------------------------------------------------- run
COUNTS = ("coreas_contributions", "zhs_contributions", "zhs_subtracks", "valid_tracks", "fixed_point_overflows")
DIAGNOSTICS = ("weighted_segment_count", "track_length_m", "weighted_track_length_m",
               "electron_weighted_track_length_m", "positron_weighted_track_length_m",
               "energy_weighted_track_length_gev_m", "maximum_segment_length_m",
               "weighted_beta_deficit_track_length_m")


def outputs(c, coreas, zhs, counters):
    out = {"coreas": coreas, "zhs": zhs, "counts": [int(counters[k]) for k in COUNTS]}
    if c["diagnostics"]:
        out["diagnostics"] = [float(counters[k]) for k in DIAGNOSTICS]
    return out


def run(state):
    c = state["case"]
    if c["form"] == "served":
        return run_served(state)
    if c["form"] == "batch":
        for k, acc in enumerate(state["events"]):
            acc.reset()
            acc.stage_lepton_tracks(state["records"][k].data_ptr(), state["counts"][k])
        state["batch"].project(state["events"], graph=True)
        got = [acc.download() for acc in state["events"]]
        return [outputs(c, w.coreas, w.zhs, w.counters) for w in got]
    acc = state["events"][0]
    acc.reset()
    if c["input"] == "columns":
        acc.accumulate_columns(state["columns"][0], state["counts"][0])
    elif c["input"] in ("host", "pinned"):
        acc.enqueue_host_lepton_tracks(state["host"][0])
    else:
        acc.accumulate_lepton_tracks(state["records"][0].data_ptr(), state["counts"][0])
    if c["output"] == "fixed":
        return outputs(c, *acc.download_fixed())
    if c["output"] == "pinned":
        coreas, zhs = state["out"][0]
        counters = acc.download_into(coreas, zhs)
        return outputs(c, coreas.reshape(3, -1), zhs.reshape(3, -1), counters)
    w = acc.download()
    return outputs(c, w.coreas, w.zhs, w.counters)


def run_served(state):
    server, c = state["server"], state["case"]
    ids = []
    for k, cfg in enumerate(state["configs"]):
        event = server.open(cfg)
        server.add_device(event, state["records"][k].data_ptr(), state["counts"][k])
        server.close_event(event)
        ids.append(event)
    out = []
    for event in ids:
        w, _ = server.fetch(event)
        out.append(outputs(c, w.coreas, w.zhs, w.counters))
    return out


# ---------------------------------------------------------- bytes and flops
def work(c):
    """Each track's used fields read once (76 bytes, with diagnostics 132) and
    each trace value written once; FP64 operations of one pair: two
    propagations, two Doppler factors, two fields and two samples (CoREAS,
    152), the Fraunhofer test (52) and per segment a propagation, two detection
    times, the potential and two samples (ZHS, 116)."""
    algorithms = 2 if c["algorithms"] == "both" else 1
    bytes_ = flops = 0.0
    for e in event_cases(c):
        bytes_ += e["segments"] * (132.0 if c["diagnostics"] else 76.0)
        bytes_ += algorithms * 3 * 8.0 * e["antennas"] * e["bins"]
        pair = (152.0 if c["algorithms"] in ("both", "coreas") else 0.0)
        pair += (52.0 + 116.0 * c["refinement"] if c["algorithms"] in ("both", "zhs") else 0.0)
        flops += e["segments"] * float(e["antennas"]) * pair
    return {"bytes": bytes_, "flops": flops}


def tolerance(c):
    """FP64 with fixed-point traces is exact: integer sums of the same IEEE
    values in any order.  Floating traces (and the diagnostics' sums) differ by
    the order of FP64 operations: two passes by 1e-15, one from exact() by
    3e-11 (samples near the cone cancel).  Mixed precision rounds directions
    and amplitudes to FP32: measured against exact() up to 7.3e-7 (CoREAS,
    k x (k x beta) of nearly parallel vectors)."""
    if c["precision"] == "mixed":
        return {"rel": 3e-6, "max": 4e-4}
    if c["traces"] == "float" or c["diagnostics"]:
        return {"rel": 1.2e-10, "max": 8e-9}
    return "exact"


# ------------------------------------------------------------------- exact
def source(p, z, observer_z):
    """Refractive index at the source, at the observer and the time factor."""
    if p["homogeneous"] > 0:
        n = torch.full_like(z, p["homogeneous"])
        return n, n, n
    low, inv, step, last = p["minimum"], p["inverse"], p["step"], p["n"].numel() - 1
    oh = (observer_z - low) * inv
    oi = int(oh + 0.5)
    h = (z - low) * inv
    inside = (h + 0.5 < last) & (h > 0)
    if not bool(inside.all()):
        raise ValueError("a source point outside the table")
    i = torch.clamp((h + 0.5).long(), 0, last)
    rise = (i - oi).double() * step
    rise = torch.where(rise == 0, torch.ones_like(rise), rise)
    factor = 1.0 + (p["integral"][i] - p["integral"][oi]) / rise
    return p["n"][i] + 1.0, torch.full_like(z, float(p["n"][oi]) + 1.0), factor


def path(p, o, pos):
    d = [o["position"][a] - pos[a] for a in range(3)]
    dist = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    n_src, n_dst, factor = source(p, pos[2], o["position"][2])
    return dict(k=[x / dist for x in d], dist=dist, n=n_src, n_dst=n_dst, time=factor * dist / C)


def dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def nearest(x):
    f = torch.floor(x)
    return f + (x - f >= 0.5).double()


def add(trace, o, t, value, gate, mask):
    """Adds the samples whose bin lies on the trace; returns how many."""
    b = nearest((t - o["start"]) * o["rate"])
    mask = mask & (b >= 0) & (b < o["bins"])
    if gate:
        mask = mask & ~((t < o["start"]) | (t > o["stop"]))
    b = b[mask].long()
    for a in range(3):
        trace[a].index_add_(0, b, value[a][mask])
    return int(b.numel())


def separate(s, e, res, signed):
    """Start and end times moved into neighbouring bins where they share one."""
    same = nearest(s / res) == nearest(e / res)
    sf, ef = s / res - torch.floor(s / res), e / res - torch.floor(e / res)
    forward = (e >= s) if signed else torch.ones_like(same)
    up, down = (sf >= 0.5) & (ef >= 0.5), (sf < 0.5) & (ef < 0.5)
    to_end = down | (~up & (ef >= 1.0 - sf))       # forward: the end moves on, else the start back
    to_start = down | (~up & (sf >= 1.0 - ef))     # backward: the start moves on, else the end back
    s2 = torch.where(same & forward & ~to_end, s - res, torch.where(same & ~forward & to_start, s + res, s))
    e2 = torch.where(same & forward & to_end, e + res, torch.where(same & ~forward & ~to_start, e - res, e))
    return s2, e2


def exact_coreas(p, o, t, trace):
    res = 1.0 / o["rate"]
    ps, pe = path(p, o, t["start"]), path(p, o, t["end"])
    pre, post = 1.0 - ps["n"] * dot(t["beta"], ps["k"]), 1.0 - pe["n"] * dot(t["beta"], pe["k"])
    sr, er = t["t0"] + ps["time"], t["t1"] + pe["time"]
    scale = t["constant"] * o["rate"]
    near = (ps["n_dst"] > 1) & ((pre.abs() < 1e-3) | (post.abs() < 1e-3))
    fs = [x * (scale / (pre * ps["dist"])) for x in cross(ps["k"], cross(ps["k"], t["beta"]))]
    fe = [x * (-scale / (post * pe["dist"])) for x in cross(pe["k"], cross(pe["k"], t["beta"]))]
    dt = er - sr
    close = ~near & ((pre < 1e-9) | (post < 1e-9)) & (dt.abs() < res)
    shrink = torch.where(close, (dt / res).abs(), torch.ones_like(dt))
    s2, e2 = separate(sr, er, res, False)
    s2, e2 = torch.where(close, s2, sr), torch.where(close, e2, er)
    count = add(trace, o, s2, [x * shrink for x in fs], True, ~near)
    count += add(trace, o, e2, [x * shrink for x in fe], True, ~near)
    if bool(near.any()):
        u = {k: ([x[near] for x in v] if isinstance(v, list) else v[near]) for k, v in t.items()}
        pm = path(p, o, [(u["start"][a] + u["end"][a]) * 0.5 for a in range(3)])
        mr = (u["t0"] + u["t1"]) * 0.5 + pm["time"]
        md = 1.0 - pm["n"] * dot(u["beta"], pm["k"])
        f = [x * (scale[near] / (md * pm["dist"])) for x in cross(pm["k"], cross(pm["k"], u["beta"]))]
        half = 0.5 * (u["length"] / (C * u["module"]) * md.abs())
        order = torch.where(sr[near] < er[near], 1.0, -1.0).double()
        s3, e3 = mr - order * half, mr + order * half
        dt = e3 - s3
        close = dt.abs() < res
        shrink = torch.where(close, (dt / res).abs(), torch.ones_like(dt))
        a3, b3 = separate(s3, e3, res, True)
        f = [x * shrink for x in f]
        every = torch.ones_like(close)
        count += add(trace, o, torch.where(close, a3, s3), f, True, every)
        count += add(trace, o, torch.where(close, b3, e3), [-x for x in f], True, every)
    return count


def exact_segment(p, o, p1, p2, t1, t2, beta, constant, divided, trace):
    m = path(p, o, [(p1[a] + p2[a]) * 0.5 for a in range(3)])
    nbk = m["n"] * dot(beta, m["k"])
    mt = (t1 + t2) * 0.5
    a, b = t1 + m["time"] - nbk * (t1 - mt), t2 + m["time"] - nbk * (t2 - mt)
    swap = a > b
    d1, d2 = torch.where(swap, b, a), torch.where(swap, a, b)
    sign = torch.where(swap, -1.0, 1.0).double()
    fs = o["rate"]
    x1, x2 = (d1 - o["start"]) * fs, (d2 - o["start"]) * fs
    sb, eb = torch.floor(x1 + 0.5), torch.floor(x2 + 0.5)
    perp = cross(m["k"], cross(beta, m["k"]))
    den = 1.0 - nbk
    tiny, single = ~(den.abs() > 1e-15), sb == eb
    dd = den * m["dist"]
    last = torch.where(single, torch.where(tiny, (t2 - t1) * fs, (d2 * fs - d1 * fs).abs()), (x2 + 0.5 - eb).abs())
    below = torch.where(single & tiny, m["dist"], dd)
    every = torch.ones_like(single)
    count = add(trace, o, d2, [x * (sign * constant * last / below) for x in perp], False, every)
    first = (sb + 0.5 - x1).abs()
    count += add(trace, o, d1, [x * (sign * constant * first / dd) for x in perp], False, ~single)
    # the bins between: only the indices that can reach the trace
    nb = eb - sb
    lo = torch.clamp(torch.floor(-x1 - 3.0), min=1.0)
    hi = torch.minimum(nb, torch.ceil(o["bins"] - x1 + 3.0))
    runs = torch.clamp(torch.where(single, torch.zeros_like(hi), hi - lo), min=0.0).long()
    if int(runs.sum()) == 0:
        return count
    owner = torch.repeat_interleave(torch.arange(runs.numel(), device=runs.device), runs)
    begin = torch.cumsum(runs, 0) - runs
    index = (torch.arange(owner.numel(), device=runs.device) - begin[owner]).double() + lo[owner]
    scale = torch.where(divided, constant, sign * constant) / dd
    value = [(x * scale)[owner] for x in perp]
    return count + add(trace, o, d1[owner] + index / fs, value, False, torch.ones_like(owner, dtype=torch.bool))


def exact_zhs(p, o, t, refinement, trace):
    mid = [(t["start"][a] + t["end"][a]) * 0.5 for a in range(3)]
    d = [o["position"][a] - mid[a] for a in range(3)]
    dist = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    uk = dot(t["beta"], [x / dist for x in d]) / t["module"]
    f = (1.0 - uk * uk) * t["length"] * t["length"] / dist / (C / o["rate"]) * 2.0 * math.pi
    divisor = torch.where(f > 1, torch.sqrt(torch.clamp(f, min=0.0)) + 1.0, torch.ones_like(f))
    parts = torch.ceil(divisor).long()
    steps = [(t["end"][a] - t["start"][a]) / divisor / refinement for a in range(3)]
    dt = (t["t1"] - t["t0"]) / divisor / refinement
    total = parts * refinement
    at, when, count = [x.clone() for x in t["start"]], t["t0"].clone(), 0
    rows = torch.arange(total.numel(), device=total.device)
    for k in range(int(total.max())):
        rows = rows[total[rows] > k]
        p1 = [x[rows] for x in at]
        p2 = [p1[a] + steps[a][rows] for a in range(3)]
        t1 = when[rows]
        t2 = t1 + dt[rows]
        count += exact_segment(p, o, p1, p2, t1, t2, [x[rows] for x in t["beta"]], t["constant"][rows],
                               total[rows] > 1, trace)
        for a in range(3):
            at[a][rows] = p2[a]
        when[rows] = t2
    return count, int(parts.sum()) + (int((parts * (refinement - 1)).sum()) if refinement > 1 else 0)


def exact_event(c, seed):
    wl, dev = workload(c), device()
    seg = segments(c, seed)
    valid = seg["pid"].abs() == 11
    pick = {k: ([x[valid] for x in v] if isinstance(v, list) else v[valid]) for k, v in seg.items()}
    delta = [pick["end"][a] - pick["start"][a] for a in range(3)]
    duration = pick["t1"] - pick["t0"]
    length = torch.sqrt(delta[0] * delta[0] + delta[1] * delta[1] + delta[2] * delta[2])
    charge = 1.6021766208e-19 * torch.where(pick["pid"] == 11, -1.0, 1.0).double()
    constant = charge * (1.0 / (4.0 * math.pi * 8.8541878128e-12 * C)) * pick["weight"]
    track = dict(start=pick["start"], end=pick["end"], t0=pick["t0"], t1=pick["t1"], length=length,
                 beta=[x / (C * duration) for x in delta], module=length / (C * duration), constant=constant)
    p = dict(homogeneous=wl["homogeneous"])
    if not p["homogeneous"] > 0:
        t = wl["table"]
        p.update(minimum=t["minimum_height_m"], inverse=t["inverse_step_per_m"], step=t["step_m"],
                 n=torch.from_numpy(t["refractivity"]).to(dev), integral=torch.from_numpy(t["integrated_refractivity"]).to(dev))
    coreas, zhs, counts, subtracks = [], [], [0, 0], 0
    n = length.numel()
    for row in wl["observers"]:
        o = dict(position=[float(x) for x in row["position_m"]], start=float(row["start_time_s"]),
                 stop=float(row["start_time_s"]) + float(row["duration_s"]), rate=float(row["sample_rate_hz"]),
                 bins=float(row["number_of_bins"]))
        tc, tz = (torch.zeros(3, int(row["number_of_bins"]), dtype=torch.float64, device=dev) for _ in range(2))
        for begin in range(0, n, 1 << 20):
            part = slice(begin, min(n, begin + (1 << 20)))
            t = {k: ([x[part] for x in v] if isinstance(v, list) else v[part]) for k, v in track.items()}
            if c["algorithms"] in ("both", "coreas"):
                counts[0] += exact_coreas(p, o, t, tc)
            if c["algorithms"] in ("both", "zhs"):
                a, b = exact_zhs(p, o, t, c["refinement"], tz)
                counts[1] += a
                subtracks += b
        coreas.append(tc)
        zhs.append(tz)
    on = [torch.cat(x, 1).cpu().numpy() if c["algorithms"] in ("both", name) else np.zeros((3, 0))
          for name, x in (("coreas", coreas), ("zhs", zhs))]
    out = {"coreas": on[0], "zhs": on[1], "counts": [counts[0], counts[1], subtracks, n, 0]}
    if c["diagnostics"]:
        w, e = pick["weight"], pick["energy"] - ELECTRON_MASS_GEV
        sums = [w.sum(), length.sum(), (w * length).sum(), (w * length)[pick["pid"] == 11].sum(),
                (w * length)[pick["pid"] != 11].sum(), (w * length * e).sum(), length.max(),
                (w * length * (1.0 - track["module"])).sum()]
        out["diagnostics"] = [float(x) for x in sums]
    return out


def exact(c, seed):
    events = event_cases(c)
    if sum(e["segments"] * e["antennas"] * c["refinement"] for e in events) > 4e8:
        return None  # takes too long
    got = [exact_event(e, seed * 101 + k) for k, e in enumerate(events)]
    if c["output"] == "fixed":
        got[0]["coreas"] = got[0]["zhs"] = None
    return got if c["form"] != "alone" else got[0]

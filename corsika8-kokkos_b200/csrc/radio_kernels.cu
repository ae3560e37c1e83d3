// radio_kernels.cu — sm_100a kernels of the radio projection.
//
// Compiled with -fmad=false (see build.py): FP64 time/bin/branch arithmetic is
// the IEEE result of the reference's expressions, so fixed-point traces in the
// FP64 path are bit-identical to the reference's, and bin indices and branch
// decisions are identical in the mixed path too.
//
//   ingest_kernel    LeptonTransportRecord (752 B AoS) -> compacted SoA
//                    kinematics + counters (record_track, RadioProjection.inl:541-611)
//   direct_kernel    one thread per (track, antenna) pair, 64-bit global
//                    atomics per sample (RadioAccumulator.inl:663-697 shape)
//   windowed_kernel  persistent CTAs over a work list of (event, chunk,
//                    algorithm, antenna) items; the CTA owns that antenna's
//                    trace as an int64 window in shared memory, deposits with
//                    shared atomics and flushes non-zero bins with checked
//                    global atomics
//   tiled_kernel     the reference's large-batch tile shape
//   decode_kernel    int64 fixed point -> V/m (V s/m) (RadioAccumulator.inl:849-898)
#include "radio_kernels.cuh"

#include <cuda_runtime.h>

#include <cstddef>
#include <cstring>

#include "../../include/c8radio.h"

namespace c8r {
namespace {

constexpr double kEmConstant = 1. / (4. * kPi * kVacuumPermittivity * kSpeedOfLight);

// ---------------------------------------------------------------- fixed point
// add_radio_fixed_point, RadioProjection.inl:254-260.
// `mag` gains |v scale| (an upper bound of |out| up to half a unit) when the
// conversion succeeds.
__device__ __forceinline__ bool to_fixed(double v, ObserverCache const& o, long long& out,
                                         float& mag) {
  if (o.count_samples) {
    out = 1;
    mag += 1.f;
    return true;
  }
  double const s = v * o.fixed_scale;
  if (!(fabs(s) < kSignedLimit)) return false;  // also rejects NaN and infinities
  out = __double2ll_rn(s);
  mag += static_cast<float>(fabs(s));
  return true;
}
__device__ __forceinline__ bool to_fixed(float v, ObserverCache const& o, long long& out,
                                         float& mag) {
  if (o.count_samples) {
    out = 1;
    mag += 1.f;
    return true;
  }
  float const s = v * o.fixed_scale_f;
  if (!(fabsf(s) < 9223372036854775808.f)) return false;  // also rejects NaN and infinities
  out = __float2ll_rn(s);
  mag += fabsf(s);
  return true;
}

// checked_radio_atomic_add's overflow test on the returned previous value
// (RadioProjection.inl:246-251).
__device__ __forceinline__ bool checked(unsigned long long previous_bits, long long inc) {
  long long const previous = static_cast<long long>(previous_bits);
  return !((inc > 0 && previous > LLONG_MAX - inc) || (inc < 0 && previous < LLONG_MIN - inc));
}

__device__ __forceinline__ double amp_div(double a, double b) { return a / b; }
__device__ __forceinline__ float amp_div(float a, float b) { return __fdividef(a, b); }

template <class T>
__device__ __forceinline__ Vec3<T> scaled(Vec3<T> v, T s) {
  return {v.x * s, v.y * s, v.z * s};
}

__device__ __forceinline__ void add_counts(Counts& c, Counts const& d) {
  c.coreas += d.coreas;
  c.zhs += d.zhs;
  c.subtracks += d.subtracks;
  c.overflows += d.overflows;
  c.mag += d.mag;
}

// A thread's counts within one work item in 32 bits, which the track loops hold
// in fewer registers: CoREAS adds two samples a track (2^30 tracks an item at
// most), and a ZHS item whose threads might pass 2^32 samples is not given to
// the loop that uses them (kPass 1).
struct Tally {
  unsigned coreas = 0, zhs = 0, overflows = 0;
  float mag = 0.f;
};
__device__ __forceinline__ Counts counts_of(Tally const& t) {
  Counts c;
  c.coreas = t.coreas;
  c.zhs = t.zhs;
  c.overflows = t.overflows;
  c.mag = t.mag;
  return c;
}

// Signed overflow of the three adds previous + increment (two's complement),
// the condition checked_radio_atomic_add tests; increments whose conversion
// failed are passed as 0 and cannot overflow.
__device__ __forceinline__ bool no_overflow3(unsigned long long px, long long x,
                                             unsigned long long py, long long y,
                                             unsigned long long pz, long long z) {
  long long const sx = static_cast<long long>(px + static_cast<unsigned long long>(x));
  long long const sy = static_cast<long long>(py + static_cast<unsigned long long>(y));
  long long const sz = static_cast<long long>(pz + static_cast<unsigned long long>(z));
  long long const bad = ((static_cast<long long>(px) ^ sx) & (x ^ sx)) |
                        ((static_cast<long long>(py) ^ sy) & (y ^ sy)) |
                        ((static_cast<long long>(pz) ^ sz) & (z ^ sz));
  return bad >= 0;
}

// ---------------------------------------------------------------- sinks
// Trace rows of one observer: global X|Y|Z rows already offset to the
// observer's first bin.
struct GlobalSink {
  unsigned long long* row[3];
  double* frow[3];
  // All three components at one bin; false if a conversion failed or an add overflowed.
  __device__ __forceinline__ bool add3(uint64_t bin, long long x, long long y, long long z,
                                       bool ox, bool oy, bool oz, float mag, float& bound) {
    (void)mag;
    (void)bound;
    unsigned long long const px = ox ? atomicAdd(row[0] + bin, static_cast<unsigned long long>(x)) : 0ull;
    unsigned long long const py = oy ? atomicAdd(row[1] + bin, static_cast<unsigned long long>(y)) : 0ull;
    unsigned long long const pz = oz ? atomicAdd(row[2] + bin, static_cast<unsigned long long>(z)) : 0ull;
    return ox && oy && oz && no_overflow3(px, x, py, y, pz, z);
  }
  __device__ __forceinline__ void addf3(uint64_t bin, double x, double y, double z) {
    atomicAdd(frow[0] + bin, x);
    atomicAdd(frow[1] + bin, y);
    atomicAdd(frow[2] + bin, z);
  }
};

// Bins past a shared-memory window: checked global adds.  Inline: a call in
// the track loops costs the loop registers.
__device__ __forceinline__ bool spill3(unsigned long long* r0, unsigned long long* r1,
                                    unsigned long long* r2, long long x, long long y, long long z,
                                    bool ox, bool oy, bool oz) {
  unsigned long long const px = ox ? atomicAdd(r0, static_cast<unsigned long long>(x)) : 0ull;
  unsigned long long const py = oy ? atomicAdd(r1, static_cast<unsigned long long>(y)) : 0ull;
  unsigned long long const pz = oz ? atomicAdd(r2, static_cast<unsigned long long>(z)) : 0ull;
  return ox && oy && oz && no_overflow3(px, x, py, y, pz, z);
}

__device__ __forceinline__ void spillf3(double* r0, double* r1, double* r2, double x, double y,
                                     double z) {
  atomicAdd(r0, x);
  atomicAdd(r1, y);
  atomicAdd(r2, z);
}

// Shared-memory window of `width` bins starting at bin 0, with bins past the
// window spilled to the global rows.  A bin's three components are neighbours
// (word 3 bin + component), so that a deposit forms one address and reaches the
// others by immediate offsets.
struct WindowSink {
  unsigned long long* win;
  double* fwin;
  uint32_t width;
  bool unchecked;
  unsigned long long* row[3];
  double* frow[3];
  // unchecked: window adds whose results are not read; `bound` then gains
  // |x| + |y| + |z| (as `mag`), and the kernel checks afterwards that no
  // partial sum of the window can have left the int64 range.
  __device__ __forceinline__ bool add3(uint64_t bin, long long x, long long y, long long z,
                                       bool ox, bool oy, bool oz, float mag, float& bound) {
    if (bin >= width)
      return spill3(row[0] + bin, row[1] + bin, row[2] + bin, x, y, z, ox, oy, oz);
    unsigned long long* const w = win + 3u * static_cast<uint32_t>(bin);
    if (unchecked) {
      if (ox) atomicAdd(w, static_cast<unsigned long long>(x));
      if (oy) atomicAdd(w + 1, static_cast<unsigned long long>(y));
      if (oz) atomicAdd(w + 2, static_cast<unsigned long long>(z));
      bound += mag;
      return ox && oy && oz;
    }
    unsigned long long const px = ox ? atomicAdd(w, static_cast<unsigned long long>(x)) : 0ull;
    unsigned long long const py = oy ? atomicAdd(w + 1, static_cast<unsigned long long>(y)) : 0ull;
    unsigned long long const pz = oz ? atomicAdd(w + 2, static_cast<unsigned long long>(z)) : 0ull;
    return ox && oy && oz && no_overflow3(px, x, py, y, pz, z);
  }
  __device__ __forceinline__ void addf3(uint64_t bin, double x, double y, double z) {
    if (bin >= width) {
      spillf3(frow[0] + bin, frow[1] + bin, frow[2] + bin, x, y, z);
      return;
    }
    double* const w = fwin + 3u * static_cast<uint32_t>(bin);
    atomicAdd(w, x);
    atomicAdd(w + 1, y);
    atomicAdd(w + 2, z);
  }
};

// A window of differences (see deposit_differences) that holds the whole
// trace: a value at one bin is that value there and its negative at the next.
struct DifferenceSink {
  unsigned long long* win;
  uint32_t width;
  __device__ __forceinline__ void add(uint32_t bin, long long x, long long y, long long z) {
    unsigned long long* w = win + 3u * bin;
    asm volatile("" : "+l"(w));
    atomicAdd(w, static_cast<unsigned long long>(x));
    atomicAdd(w + 1, static_cast<unsigned long long>(y));
    atomicAdd(w + 2, static_cast<unsigned long long>(z));
  }
  __device__ __forceinline__ bool add3(uint64_t bin, long long x, long long y, long long z,
                                       bool ox, bool oy, bool oz, float mag, float& bound) {
    uint32_t const b = static_cast<uint32_t>(bin);
    add(b, x, y, z);
    if (b + 1u < width) add(b + 1u, -x, -y, -z);
    bound += mag;
    return ox && oy && oz;
  }
  __device__ __forceinline__ void addf3(uint64_t, double, double, double) {}  // fixed point only
};

// ---------------------------------------------------------------- add_sample
// RadioProjection.inl:263-301.  kPotential selects the ZHS overload (no time
// gate).
template <bool kPotential>
__device__ __forceinline__ bool sample_bin(ObserverCache const& o, double t, uint64_t& bin) {
  if (!kPotential) {
    if (t < o.start_time || t > o.end_time) return false;
  }
  double const bv = nearest_bin((t - o.start_time) * o.sample_rate);
  if (!(bv >= 0. && bv < o.bins_d)) return false;
  bin = static_cast<uint64_t>(bv);
  return bin < o.bins;
}

template <class Amp>
struct Deposit {
  Vec3<Amp> value;
  long long ix, iy, iz;
  bool okx, oky, okz;
  float mag;  // |scaled components| that converted
};

template <bool kFixed, class Amp>
__device__ __forceinline__ Deposit<Amp> make_deposit(ObserverCache const& o, Vec3<Amp> v) {
  Deposit<Amp> d;
  d.value = v;
  d.mag = 0.f;
  if (kFixed) {
    d.okx = to_fixed(v.x, o, d.ix, d.mag);
    d.oky = to_fixed(v.y, o, d.iy, d.mag);
    d.okz = to_fixed(v.z, o, d.iz, d.mag);
  }
  return d;
}

template <bool kPotential, bool kFixed, class Amp, class Sink>
__device__ __forceinline__ void deposit(ObserverCache const& o, Sink& sink, double t,
                                        Deposit<Amp> const& d, unsigned long long& contributions,
                                        unsigned long long& overflows, float& bound) {
  uint64_t bin;
  if (!sample_bin<kPotential>(o, t, bin)) return;
  if (kFixed) {
    if (!sink.add3(bin, d.okx ? d.ix : 0, d.oky ? d.iy : 0, d.okz ? d.iz : 0, d.okx, d.oky, d.okz,
                   d.mag, bound)) {
      ++overflows;
      return;
    }
  } else {
    sink.addf3(bin, static_cast<double>(d.value.x), static_cast<double>(d.value.y),
               static_cast<double>(d.value.z));
  }
  ++contributions;
}

template <bool kPotential, bool kFixed, class Amp, class Sink>
__device__ __forceinline__ void add_sample(ObserverCache const& o, Sink& sink, double t,
                                           Vec3<Amp> v, unsigned long long& contributions,
                                           unsigned long long& overflows, float& bound) {
  uint64_t bin;
  if (!sample_bin<kPotential>(o, t, bin)) return;
  Deposit<Amp> const d = make_deposit<kFixed>(o, v);
  if (kFixed) {
    if (!sink.add3(bin, d.okx ? d.ix : 0, d.oky ? d.iy : 0, d.okz ? d.iz : 0, d.okx, d.oky, d.okz,
                   d.mag, bound)) {
      ++overflows;
      return;
    }
  } else {
    sink.addf3(bin, static_cast<double>(v.x), static_cast<double>(v.y), static_cast<double>(v.z));
  }
  ++contributions;
}

// A deposit at a bin already known to lie in [0, bins).
template <bool kFixed, class Amp, class Sink>
__device__ __forceinline__ void deposit_bin(Sink& sink, uint64_t bin, Deposit<Amp> const& d,
                                            unsigned long long& contributions,
                                            unsigned long long& overflows, float& bound) {
  if (kFixed) {
    if (!sink.add3(bin, d.okx ? d.ix : 0, d.oky ? d.iy : 0, d.okz ? d.iz : 0, d.okx, d.oky, d.okz,
                   d.mag, bound)) {
      ++overflows;
      return;
    }
  } else {
    sink.addf3(bin, static_cast<double>(d.value.x), static_cast<double>(d.value.y),
               static_cast<double>(d.value.z));
  }
  ++contributions;
}

// Near-Cherenkov branch of accumulate_co_reas (RadioProjection.inl:352-387):
// midpoint field over the Doppler-compressed duration.  Kept out of line: it
// is taken by a minority of pairs, and its third propagation would otherwise
// grow the hot loop's instruction footprint.  Returns the counts it adds.
template <bool kFixed, class Amp, bool kPre, bool kDivide = false, class Sink>
__device__ __noinline__ Counts coreas_near_cone(Track const t, Propagation const& p,
                                                ObserverCache const& o, Sink sink,
                                                bool start_before_end, SourceTerms const pre_mid) {
  Counts c;
  Vec3<Amp> const beta{static_cast<Amp>(t.bx), static_cast<Amp>(t.by), static_cast<Amp>(t.bz)};
  double const cf = t.constant * o.sample_rate;
  double const mx = (t.sx + t.ex) * 0.5, my = (t.sy + t.ey) * 0.5, mz = (t.sz + t.ez) * 0.5;
  double const mt = (t.ts + t.te) * 0.5;
  Path const pm =
      kPre ? propagate_with<true, kDivide>(pre_mid, o, mx, my, mz) : propagate<true, kDivide>(p, o, mx, my, mz);
  double const mr = mt + pm.time;
  double const md = doppler(pm.n_src, t.bx, t.by, t.bz, pm.kx, pm.ky, pm.kz);
  Vec3<Amp> const k{static_cast<Amp>(pm.kx), static_cast<Amp>(pm.ky), static_cast<Amp>(pm.kz)};
  Vec3<Amp> fstart =
      scaled(cross(k, cross(k, beta)), amp_div(static_cast<Amp>(cf), static_cast<Amp>(md * pm.dist)));
  Vec3<Amp> fend = scaled(fstart, static_cast<Amp>(-1.));
  Track whole = t;
  derive_track(whole);
  double dt = whole.length / (kSpeedOfLight * whole.beta_module) * fabs(md);
  double sr, er;
  if (start_before_end) {
    sr = mr - 0.5 * dt;
    er = mr + 0.5 * dt;
  } else {
    sr = mr + 0.5 * dt;
    er = mr - 0.5 * dt;
  }
  double const res = o.resolution;
  dt = er - sr;
  if (fabs(dt) < res) {
    Amp const s = static_cast<Amp>(fabs(dt / res));
    fstart = scaled(fstart, s);
    fend = scaled(fend, s);
    separate_same_bin(sr, er, res, true);
  }
  add_sample<false, kFixed>(o, sink, sr, fstart, c.coreas, c.overflows, c.mag);
  add_sample<false, kFixed>(o, sink, er, fend, c.coreas, c.overflows, c.mag);
  return c;
}

// ---------------------------------------------------------------- CoREAS
// accumulate_co_reas, RadioProjection.inl:339-409, every decision and (FP64
// path) every amplitude evaluated exactly as the reference.
// kPre: the start, end and midpoint source terms are `terms` (precomputed at
// ingest for the event's shared destination row), else looked up.
// kDivide: see propagate_with (the plain shapes).
template <bool kFixed, class Amp, class Sink, bool kPre = false, bool kDivide = false>
__device__ __forceinline__ void coreas_pair(Track const& t, Propagation const& p,
                                            ObserverCache const& o, Sink& sink, Counts& c,
                                            SourceTerms const* terms = nullptr) {
  Path const ps = kPre ? propagate_with<true, kDivide>(terms[0], o, t.sx, t.sy, t.sz)
                       : propagate<true, kDivide>(p, o, t.sx, t.sy, t.sz);
  Path const pe = kPre ? propagate_with<true, kDivide>(terms[1], o, t.ex, t.ey, t.ez)
                       : propagate<true, kDivide>(p, o, t.ex, t.ey, t.ez);
  double const pre = doppler(ps.n_src, t.bx, t.by, t.bz, ps.kx, ps.ky, ps.kz);
  double const post = doppler(pe.n_src, t.bx, t.by, t.bz, pe.kx, pe.ky, pe.kz);
  double sr = t.ts + ps.time;
  double er = t.te + pe.time;
  double const cf = t.constant * o.sample_rate;
  Vec3<Amp> const beta{static_cast<Amp>(t.bx), static_cast<Amp>(t.by), static_cast<Amp>(t.bz)};

  if (ps.n_dst > 1. && (fabs(pre) < kCoreasThreshold || fabs(post) < kCoreasThreshold)) {
    Counts const d = coreas_near_cone<kFixed, Amp, kPre, kDivide>(t, p, o, sink, sr < er, kPre ? terms[2] : SourceTerms{});
    c.coreas += d.coreas;
    c.overflows += d.overflows;
    c.mag += d.mag;
    return;
  }

  Vec3<Amp> const ks{static_cast<Amp>(ps.kx), static_cast<Amp>(ps.ky), static_cast<Amp>(ps.kz)};
  Vec3<Amp> const ke{static_cast<Amp>(pe.kx), static_cast<Amp>(pe.ky), static_cast<Amp>(pe.kz)};
  Vec3<Amp> fstart =
      scaled(cross(ks, cross(ks, beta)), amp_div(static_cast<Amp>(cf), static_cast<Amp>(pre * ps.dist)));
  Vec3<Amp> fend =
      scaled(cross(ke, cross(ke, beta)), amp_div(static_cast<Amp>(-cf), static_cast<Amp>(post * pe.dist)));
  if (pre < 1.e-9 || post < 1.e-9) {
    double const res = o.resolution;
    double const dt = er - sr;
    if (fabs(dt) < res) {
      Amp const s = static_cast<Amp>(fabs(dt / res));
      fstart = scaled(fstart, s);
      fend = scaled(fend, s);
      separate_same_bin(sr, er, res, false);
    }
  }
  add_sample<false, kFixed>(o, sink, sr, fstart, c.coreas, c.overflows, c.mag);
  add_sample<false, kFixed>(o, sink, er, fend, c.coreas, c.overflows, c.mag);
}

// What became of a pair in the windowed CoREAS track loop: deposited, or
// deferred to coreas_drain_pair -- kCoreasExact, or kCoreasNearCone with bit 0
// the branch's start-before-end order (sr < er), both decided exactly, so the
// drain evaluates only the near-Cherenkov branch itself.
constexpr int kCoreasDeposited = 0, kCoreasExact = 1, kCoreasNearCone = 2;

// The common CoREAS pair of the windowed kernel (RadioProjection.inl:339-409
// without its near-Cherenkov branch), evaluated exactly.  Deposits nothing
// when it defers.
template <bool kFixed, bool kPre, class Amp, class Sink>
__device__ __forceinline__ int coreas_common(Track const& t, Propagation const& p,
                                              ObserverCache const& o, Sink& sink, Counts& c,
                                              SourceTerms const& pre_start, SourceTerms const& pre_end) {
  Path const ps = kPre ? propagate_with<true>(pre_start, o, t.sx, t.sy, t.sz) : propagate<true>(p, o, t.sx, t.sy, t.sz);
  Path const pe = kPre ? propagate_with<true>(pre_end, o, t.ex, t.ey, t.ez) : propagate<true>(p, o, t.ex, t.ey, t.ez);
  double const pre = doppler(ps.n_src, t.bx, t.by, t.bz, ps.kx, ps.ky, ps.kz);
  double const post = doppler(pe.n_src, t.bx, t.by, t.bz, pe.kx, pe.ky, pe.kz);
  double sr = t.ts + ps.time;
  double er = t.te + pe.time;
  if (ps.n_dst > 1. && (fabs(pre) < kCoreasThreshold || fabs(post) < kCoreasThreshold))
    return kCoreasNearCone | (sr < er ? 1 : 0);
  Vec3<Amp> const beta{static_cast<Amp>(t.bx), static_cast<Amp>(t.by), static_cast<Amp>(t.bz)};
  Vec3<Amp> const ks{static_cast<Amp>(ps.kx), static_cast<Amp>(ps.ky), static_cast<Amp>(ps.kz)};
  Vec3<Amp> const ke{static_cast<Amp>(pe.kx), static_cast<Amp>(pe.ky), static_cast<Amp>(pe.kz)};
  double const cf = t.constant * o.sample_rate;
  Vec3<Amp> fstart =
      scaled(cross(ks, cross(ks, beta)), amp_div(static_cast<Amp>(cf), static_cast<Amp>(pre * ps.dist)));
  Vec3<Amp> fend =
      scaled(cross(ke, cross(ke, beta)), amp_div(static_cast<Amp>(-cf), static_cast<Amp>(post * pe.dist)));
  if (pre < 1.e-9 || post < 1.e-9) {
    double const res = o.resolution;
    double const dt = er - sr;
    if (fabs(dt) < res) {
      Amp const s = static_cast<Amp>(fabs(dt / res));
      fstart = scaled(fstart, s);
      fend = scaled(fend, s);
      separate_same_bin(sr, er, res, false);
    }
  }
  add_sample<false, kFixed>(o, sink, sr, fstart, c.coreas, c.overflows, c.mag);
  add_sample<false, kFixed>(o, sink, er, fend, c.coreas, c.overflows, c.mag);
  return kCoreasDeposited;
}

// The windowed kernels' work item in shared memory: its observer, the filtered
// paths' constants of it, and the number of its deferred pairs.  At namespace
// scope, so that the track loops, functions of their own, address them directly.
__shared__ ObserverCache s_observer;
__shared__ LeanObserver s_lean;
__shared__ unsigned s_deferred_total;
__shared__ unsigned* s_deferred_list;  // this CTA's list (global memory)

// The packed word's flags (kTrackRegular, ...) and FP32 constant.
__device__ __forceinline__ unsigned pack_flags(double pack) {
  return static_cast<unsigned>(__double2hiint(pack));
}
// n_dst as the projection looks at it: above 1 or not.
__device__ __forceinline__ double dense_index(unsigned flags) { return (flags & kTrackDense) ? 2. : 1.; }
__device__ __forceinline__ float pack_constant(double pack) { return __int_as_float(__double2loint(pack)); }

// One endpoint (or midpoint) of a track seen from an observer, for the
// filtered paths: distance, detection time in bins, Doppler factor 1 - n w and
// w / |d|, from which k (k.beta) - beta = d (w / |d|) - beta.
struct LeanPoint {
  double dx, dy, dz, dist, inverse, x, w, factor, along;
  bool ok;
};
__device__ __forceinline__ LeanPoint lean_point(LeanObserver const& l, double sx, double sy, double sz,
                                                double t, double bx, double by, double bz,
                                                double factor, double index) {
  LeanPoint r;
  r.dx = l.px - sx;
  r.dy = l.py - sy;
  r.dz = l.pz - sz;
  double const s2 = fma(r.dz, r.dz, fma(r.dy, r.dy, r.dx * r.dx));
  r.ok = lean_rsqrt(s2, r.inverse);
  r.dist = s2 * r.inverse;
  r.x = fma(r.dist, factor * l.rate_over_c, (t - l.start_time) * l.rate);
  r.w = fma(bz, r.dz, fma(by, r.dy, bx * r.dx)) * r.inverse;
  r.factor = fma(-index, r.w, 1.);
  r.along = r.w * r.inverse;
  return r;
}

// separate_same_bin_endpoints (RadioProjection.inl:303-336) in bins.  `u` =
// x + t0 fs is the absolute time start / res; with the fraction of `u` at or
// above one half exactly when its nearest-integer remainder r is negative, the
// reference's cases reduce to the sign of the two remainders' sum: `high`
// (the end in forward order) moves on where it is not negative, else `low`
// moves back.  False when a guard cannot decide.
__device__ __forceinline__ bool lean_separate(double& low, double& high, LeanObserver const& l) {
  double const ul = low + l.start_bins, uh = high + l.start_bins;
  int bl, bh;
  double const rl = lean_nearest(ul, bl), rh = lean_nearest(uh, bh);
  if (!(fabs(ul) < 0x1p30 && fabs(uh) < 0x1p30 && fabs(rl) < 0.5 - kBinGuard && fabs(rh) < 0.5 - kBinGuard))
    return false;
  if (bl != bh) return true;
  double const sum = rl + rh;
  if (fabs(sum) < 2. * kBinGuard) return false;
  if (sum > 0.)
    high += 1.;
  else
    low -= 1.;
  return true;
}

// Where a CoREAS sample at x bins goes: its bin, no bin (`in` false), or
// undecided (returns false).
__device__ __forceinline__ bool lean_gate(double x, LeanObserver const& l, int& bin, bool& in) {
  double const r = lean_nearest(x, bin);
  in = (x > kBinGuard) & (x < l.gate_in) & (fabs(r) < 0.5 - kBinGuard);
  return in | (x < -kBinGuard) | (x > l.gate_out);
}

// Adds one filtered sample, (vx, vy, vz) a in fixed-point units (1 per
// component when counting samples).  Every component is below 2^61.
template <bool kUnchecked>
__device__ __forceinline__ void lean_add(WindowSink& sink, LeanObserver const& l, int bin, float vx, float vy,
                                         float vz, float a, Tally& c) {
  long long const x = __float2ll_rn(fmaf(vx, a, l.bias)), y = __float2ll_rn(fmaf(vy, a, l.bias)),
                  z = __float2ll_rn(fmaf(vz, a, l.bias));
  if (kUnchecked) {
    // through a generic pointer (see deposit_differences)
    unsigned long long* w = sink.win + 3u * static_cast<unsigned>(bin);
    asm volatile("" : "+l"(w));
    atomicAdd(w, static_cast<unsigned long long>(x));
    atomicAdd(w + 1, static_cast<unsigned long long>(y));
    atomicAdd(w + 2, static_cast<unsigned long long>(z));
    ++c.coreas;
  } else {
    float const mag = (fabsf(vx) + fabsf(vy) + fabsf(vz)) * fabsf(a) + 3.f * l.bias;
    if (sink.add3(static_cast<uint64_t>(bin), x, y, z, true, true, true, mag, c.mag))
      ++c.coreas;
    else
      ++c.overflows;
  }
}

// The two samples of a CoREAS pair, fields (s) as and (e) ae, at xs and xe
// bins.  False, having added nothing, when a bin is undecided or a component
// might not convert.  kUnchecked: the window bound gains an upper bound of the
// |components| (each factor's roundings inside 2^-20).
template <bool kUnchecked>
__device__ __forceinline__ bool lean_samples(WindowSink& sink, LeanObserver const& l, double xs, double xe,
                                             Vec3<float> s, float as, Vec3<float> e, float ae, Tally& c) {
  int bs, be;
  bool ins, ine;
  bool decided = lean_gate(xs, l, bs, ins);
  decided = lean_gate(xe, l, be, ine) & decided;
  float const ms = (fabsf(s.x) + fabsf(s.y) + fabsf(s.z)) * fabsf(as);
  float const me = (fabsf(e.x) + fabsf(e.y) + fabsf(e.z)) * fabsf(ae);
  if (!(decided & (ms + me < 0x1p60f))) return false;  // also NaN and infinities
  if (ins) lean_add<kUnchecked>(sink, l, bs, s.x, s.y, s.z, as, c);
  if (ine) lean_add<kUnchecked>(sink, l, be, e.x, e.y, e.z, ae, c);
  if (kUnchecked) c.mag = fmaf(ms + me, 1.f + 0x1p-20f, c.mag) + 6.f * l.bias;
  return true;
}

// The common CoREAS pair of the windowed kernel in mixed precision and fixed
// point (RadioProjection.inl:339-409 without its near-Cherenkov branch), from
// the track's columns `r`: detection times and Doppler factors in FP64 by the
// filtered arithmetic above, transverse vectors k (k.beta) - beta in FP64
// (k x (k x beta) of FP32 vectors cancels when they are nearly parallel),
// amplitudes in FP32.  Returns one of the codes above; a deferred pair has
// deposited nothing.  kPre: the points' source terms are the track's columns.
//
// Against exact times (a square root and four divisions an endpoint) and an
// FP32 cross product the pair takes 344 instead of 621 warp instructions:
// 1e7 x 160 x 8192 CoREAS 41.6 -> 22.5 ms, 5e6 x 64 in ice 9.0 -> 3.9 ms, and the
// traces' relative error falls from 6e-7 to 1.1e-7.  What bounds it now is the
// L1 data pipe (79% busy: track columns, observer constants and, two fifths of it, the
// six 64-bit shared atomics) beside 61% of the issue slots.
template <bool kPre, bool kUnchecked>
__device__ __forceinline__ int coreas_lean(double2 const* __restrict__ r, Propagation const& p,
                                           LeanObserver const& l, WindowSink& sink, Tally& c) {
  constexpr unsigned T = kTrackTile;
  double2 const ca = __ldg(r), cb = __ldg(r + T), cc = __ldg(r + 2 * T), ct = __ldg(r + 3 * T),
                cd = __ldg(r + 4 * T), ce = __ldg(r + 5 * T);
  unsigned const flags = pack_flags(ce.y);
  SourceTerms ts, te;
  bool ok = (flags & kTrackRegular & l.usable) != 0u;
  if (kPre) {
    double2 const s = __ldg(r + kFactorStart / 2 * T), e = __ldg(r + kFactorEnd / 2 * T);
    ts = SourceTerms{s.x, s.y, dense_index(flags)};
    te = SourceTerms{e.x, e.y, 0.};
  } else {
    Destination const d = destination_of(s_observer);
    ts = source_terms(p, d, cb.x);
    te = source_terms(p, d, cc.y);
    ok = ok & lean_terms(ts) & lean_terms(te);
  }
  LeanPoint const s = lean_point(l, ca.x, ca.y, cb.x, ct.x, cd.x, cd.y, ce.x, ts.factor, ts.n_src);
  LeanPoint const e = lean_point(l, cb.y, cc.x, cc.y, ct.y, cd.x, cd.y, ce.x, te.factor, te.n_src);
  bool const dense = ts.n_dst > 1.;
  ok = ok & s.ok & e.ok;
  double const least = fmin(fabs(s.factor), fabs(e.factor));
  // below 1e-3 the near-Cherenkov branch (n_dst > 1); below 1e-6 the factor's
  // own error counts
  if (!(ok & (least >= (dense ? kCoreasThreshold + kDopplerGuard : 1.e-6)))) {
    if (ok && dense && least < kCoreasThreshold - kDopplerGuard && fabs(s.x - e.x) > 2. * kBinGuard &&
        fabs(s.x) < 0x1p27 && fabs(e.x) < 0x1p27)
      return kCoreasNearCone | (s.x < e.x ? 1 : 0);
    return kCoreasExact;
  }
  float const constant = pack_constant(ce.y) * l.scale;
  float as = __fdividef(constant, static_cast<float>(s.factor * s.dist));
  float ae = __fdividef(-constant, static_cast<float>(e.factor * e.dist));
  double xs = s.x, xe = e.x;
  if ((s.factor < 0.) | (e.factor < 0.)) {  // |factor| >= 1e-6: the reference's "< 1e-9"
    double const dt = fabs(xe - xs);
    if (dt < 1. + kBinGuard) {
      if (!(dt < 1. - kBinGuard && lean_separate(xs, xe, l))) return kCoreasExact;
      as *= static_cast<float>(dt);
      ae *= static_cast<float>(dt);
    }
  }
  Vec3<float> const vs{static_cast<float>(fma(s.dx, s.along, -cd.x)), static_cast<float>(fma(s.dy, s.along, -cd.y)),
                       static_cast<float>(fma(s.dz, s.along, -ce.x))};
  Vec3<float> const ve{static_cast<float>(fma(e.dx, e.along, -cd.x)), static_cast<float>(fma(e.dy, e.along, -cd.y)),
                       static_cast<float>(fma(e.dz, e.along, -ce.x))};
  return lean_samples<kUnchecked>(sink, l, xs, xe, vs, as, ve, ae, c) ? kCoreasDeposited : kCoreasExact;
}

// The near-Cherenkov branch of a deferred pair (RadioProjection.inl:352-387)
// by the filtered arithmetic: the midpoint field over the Doppler-compressed
// duration |1 - n w| (t_end - t_start).  False, having added nothing, when a
// guard cannot decide.
template <bool kPre>
__device__ __forceinline__ bool near_cone_lean(double2 const* __restrict__ r, bool start_before_end,
                                               Propagation const& p, LeanObserver const& l, WindowSink& sink,
                                               Tally& c) {
  constexpr unsigned T = kTrackTile;
  double2 const ca = __ldg(r), cb = __ldg(r + T), cc = __ldg(r + 2 * T), ct = __ldg(r + 3 * T),
                cd = __ldg(r + 4 * T), ce = __ldg(r + 5 * T);
  unsigned const flags = pack_flags(ce.y);
  double const mz = (cb.x + cc.y) * 0.5;
  SourceTerms m;
  if (kPre && (flags & kTrackOneMid)) {
    double2 const mid = __ldg(r + kFactorMid / 2 * T);
    m = SourceTerms{mid.x, mid.y, 0.};
  } else {
    m = source_terms(p, destination_of(s_observer), mz);
  }
  LeanPoint const s = lean_point(l, (ca.x + cb.y) * 0.5, (ca.y + cc.x) * 0.5, mz, (ct.x + ct.y) * 0.5, cd.x,
                                 cd.y, ce.x, m.factor, m.n_src);
  double const dt = (ct.y - ct.x) * l.rate * fabs(s.factor);
  // |factor| > 8 guards: its sign and the field's are the reference's.  Where
  // the samples share a bin the field is scaled by dt, which carries the
  // same factor, so a small one costs no precision.
  if (!((flags & kTrackRegular) && l.usable && s.ok && lean_terms(m) && fabs(s.factor) > 8. * kDopplerGuard &&
        fabs(dt - 1.) > 2. * kBinGuard && dt > 2. * kBinGuard))
    return false;
  double low = fma(-0.5, dt, s.x), high = fma(0.5, dt, s.x);
  float a = __fdividef(pack_constant(ce.y) * l.scale, static_cast<float>(s.factor * s.dist));
  if (dt < 1.) {
    if (!lean_separate(low, high, l)) return false;
    a *= static_cast<float>(dt);
  }
  Vec3<float> const v{static_cast<float>(fma(s.dx, s.along, -cd.x)), static_cast<float>(fma(s.dy, s.along, -cd.y)),
                      static_cast<float>(fma(s.dz, s.along, -ce.x))};
  return lean_samples<false>(sink, l, start_before_end ? low : high, start_before_end ? high : low, v, a, v, -a, c);
}

// Intermediate ZHS bins binned index by index with the reference's own
// expression (RadioProjection.inl:465-472).  Samples of index i land in bin
// nearest((d1 + i/fs - t0) fs), monotone in i and within a hundredth of a bin
// of x1 + i while all magnitudes stay below 2^40 bins; indices whose bin is
// surely outside [0, bins) are skipped, which changes no sum and no counter.
template <bool kFixed, class Amp, class Sink>
__device__ __noinline__ Counts zhs_indexed_bins(ObserverCache const& o, Sink sink, double d1,
                                                double x1, int nb, Deposit<Amp> const mid) {
  Counts c;
  double const fs = o.sample_rate;
  int lo = 1, hi = nb;
  double const span = 1099511627776.0;  // 2^40
  if (fabs(x1) < span && fabs(o.start_time * fs) < span && fabs(d1 * fs) < span &&
      static_cast<double>(nb) < span) {
    double const first = -x1 - 3.;
    double const last = o.bins_d - x1 + 3.;
    if (first > 1.) lo = first >= static_cast<double>(nb) ? nb : static_cast<int>(first);
    if (last < static_cast<double>(nb)) hi = last <= 1. ? 1 : static_cast<int>(last) + 1;
    if (hi > nb) hi = nb;
  }
  for (int index = lo; index < hi; ++index)
    deposit<true, kFixed>(o, sink, d1 + static_cast<double>(index) / fs, mid, c.zhs, c.overflows, c.mag);
  return c;
}

// ---------------------------------------------------------------- ZHS
// The multi-bin tail of a ZHS segment (first sample and intermediate bins,
// RadioProjection.inl:457-472), out of line: about half the segments take it,
// and keeping it out of the common path saves registers and instruction fetch.
template <bool kFixed, bool kRuns, class Amp, class Sink>
__device__ __noinline__ Counts zhs_multi_tail(ObserverCache const& o, Sink sink, double d1,
                                              double x1, double sb, int nb, Vec3<Amp> perp,
                                              double sc, double dd, double mc, bool run_ok) {
  Counts c;
  double const frac_first = fabs(sb + 0.5 - x1);
  add_sample<true, kFixed>(o, sink, d1,
                           scaled(perp, amp_div(static_cast<Amp>(sc * frac_first), static_cast<Amp>(dd))),
                           c.zhs, c.overflows, c.mag);
  if (nb > 1) {
    Deposit<Amp> const mid =
        make_deposit<kFixed>(o, scaled(perp, amp_div(static_cast<Amp>(mc), static_cast<Amp>(dd))));
    if (kRuns && run_ok) {
      long long const b1 = static_cast<long long>(floor(x1)) + (x1 - floor(x1) >= 0.5 ? 1 : 0);
      long long lo = 1, hi = nb;
      if (-b1 > lo) lo = -b1;
      long long const top = static_cast<long long>(o.bins) - b1;
      if (top < hi) hi = top;
      if (hi > lo) {
        uint64_t const first = static_cast<uint64_t>(b1 + lo);
        uint32_t const count = static_cast<uint32_t>(hi - lo);
        for (uint32_t j = 0; j < count; ++j)
          deposit_bin<kFixed>(sink, first + j, mid, c.zhs, c.overflows, c.mag);
      }
    } else {
      Counts const d = zhs_indexed_bins<kFixed, Amp>(o, sink, d1, x1, nb, mid);
      c.zhs += d.zhs;
      c.overflows += d.overflows;
      c.mag += d.mag;
    }
  }
  return c;
}

// accumulate_zhs_segment, RadioProjection.inl:412-480, every decision exact.
//
// kRuns = true (windowed kernel): the intermediate bins of a segment are the
// consecutive bins nearest(x1) + i whenever x1 lies farther than a rounding
// bound from a half bin (checked below); they are then deposited as one run,
// without the per-index division.  Otherwise, and always for kRuns = false
// (the reference-shaped direct kernel), each index is binned by the
// reference's own expression.
//
template <bool kFixed, bool kRuns, class Amp, bool kDivide = false, class Sink>
__device__ __forceinline__ void zhs_segment(double p1x, double p1y, double p1z, double p2x,
                                            double p2y, double p2z, double t1, double t2,
                                            Track const& t, Propagation const& p,
                                            ObserverCache const& o, Sink& sink, Counts& c,
                                            bool subdivided) {
  double const mx = (p1x + p2x) * 0.5, my = (p1y + p2y) * 0.5, mz = (p1z + p2z) * 0.5;
  Path const path = propagate<true, kDivide>(p, o, mx, my, mz);
  double const bk = t.bx * path.kx + t.by * path.ky + t.bz * path.kz;
  double const nbk = path.n_src * bk;
  double const mt = (t1 + t2) * 0.5;
  double d1 = t1 + path.time - nbk * (t1 - mt);
  double d2 = t2 + path.time - nbk * (t2 - mt);
  double sign = 1.;
  if (d1 > d2) {
    double const swap = d1;
    d1 = d2;
    d2 = swap;
    sign = -1.;
  }
  double const fs = o.sample_rate;
  double const x1 = (d1 - o.start_time) * fs;
  double const x2 = (d2 - o.start_time) * fs;
  double const sb = floor(x1 + 0.5);
  double const eb = floor(x2 + 0.5);
  double const den = 1. - nbk;
  int const nb = x86_int(eb - sb);
  // consecutive-run test for the intermediate bins.  Index i is binned at
  // y_i = RN(RN(RN(d1 + RN(i/fs)) - t0) fs); with u = 2^-53,
  // |y_i - (x1 + i)| <= 6 u M (1 + u)^4 < 2^-50 M for M = |x1| + i + |d1 fs|
  // + |t0 fs| + 2.  The nearest bin changes only at half-integers, which sit
  // at integer offsets from each other, so if x1 is farther than that bound
  // (plus, filtered, x1's own error) from a half-integer, nearest(y_i) =
  // nearest(x1) + i for every i < nb.
  double const f1 = fabs(x1 - floor(x1) - 0.5);
  double const mag = fabs(x1) + static_cast<double>(nb) + fabs(d1 * fs) + fabs(o.start_time * fs) + 2.;
  bool const run_ok = mag < 0x1p50 && f1 > mag * 0x1p-48;
  Vec3<Amp> const k{static_cast<Amp>(path.kx), static_cast<Amp>(path.ky), static_cast<Amp>(path.kz)};
  Vec3<Amp> const beta{static_cast<Amp>(t.bx), static_cast<Amp>(t.by), static_cast<Amp>(t.bz)};
  Vec3<Amp> const perp = cross(k, cross(beta, k));
  double const sc = sign * t.constant;
  double const dd = den * path.dist;

  // The last sample (detection_time2) and, when both times share a bin, the
  // only one (:441-455); fraction and denominator selected, not branched.
  bool const single = sb == eb;
  bool const tiny = !(fabs(den) > 1.e-15);
  double const frac_last = single ? (tiny ? (t2 - t1) * fs : fabs(d2 * fs - d1 * fs))
                                  : fabs(x2 + 0.5 - eb);
  double const den_last = single && tiny ? path.dist : dd;
  add_sample<true, kFixed>(o, sink, d2,
                           scaled(perp, amp_div(static_cast<Amp>(sc * frac_last),
                                                static_cast<Amp>(den_last))),
                           c.zhs, c.overflows, c.mag);
  if (single) return;
  Counts const d = zhs_multi_tail<kFixed, kRuns, Amp>(
      o, sink, d1, x1, sb, nb, perp, sc, dd, (subdivided ? 1. : sign) * t.constant, run_ok);
  c.zhs += d.zhs;
  c.overflows += d.overflows;
  c.mag += d.mag;
}

// The samples of one ZHS segment, staged for the warp (windowed kernel): the
// in-range bins [start, start + count) of its first sample and intermediate
// bins (value perp * first at `start` when flag bit 0, perp * mid elsewhere)
// and its last sample at last_bin (flag bit 1).  Bins are consecutive there
// because the segment is staged only when its intermediate bins are
// nearest(x1) + i (the consecutive-run test of zhs_segment).
template <class Amp>
struct StagedSegment {
  Vec3<Amp> perp;
  Amp first, mid, last;
  uint32_t start, count, last_bin, flags;
};
// FP64 amplitudes: slots of 72 bytes (18 banks) rather than 64, which spreads
// the lanes' loads of different slots over the shared-memory banks (11% off
// the FP64 ZHS kernel; the same padding of the 40-byte FP32 slot cost 10%).
template <>
struct StagedSegment<double> {
  Vec3<double> perp;
  double first, mid, last;
  uint32_t start, count, last_bin, flags;
  uint32_t pad_[2];
};

// accumulate_zhs_segment (RadioProjection.inl:412-480) evaluated exactly, as
// zhs_segment<kRuns = true>, its samples staged instead of deposited.  The
// segment's midpoint, its times and the time between them come from the
// caller; kPre: the midpoint's source terms are `pre`, else they are looked
// up.  Returns false when the segment needs the per-index binning, when the
// trace has 2^26 bins or more (staged counts then stay far inside 32 bits per
// warp), or when a detection time's nearest bin is not the floor(x + 1/2) that
// counts the bins between (x just below 1/2, where x + 1/2 rounds to 1): the
// last sample then would not be in the bin after the run, as
// deposit_differences takes it.  The caller discards whatever `out` holds.
template <class Amp, bool kPre = false>
__device__ __forceinline__ bool zhs_stage(double mx, double my, double mz, double t1, double t2, double mt,
                                          Track const& t, Propagation const& p,
                                          ObserverCache const& o, bool subdivided,
                                          StagedSegment<Amp>& out,
                                          SourceTerms const& pre = SourceTerms{}) {
  if (!(o.bins_d < kMaxLeanBins)) return false;
  Path const path = kPre ? propagate_with<true>(pre, o, mx, my, mz) : propagate<true>(p, o, mx, my, mz);
  double const bk = t.bx * path.kx + t.by * path.ky + t.bz * path.kz;
  double const nbk = path.n_src * bk;
  double d1 = t1 + path.time - nbk * (t1 - mt);
  double d2 = t2 + path.time - nbk * (t2 - mt);
  double sign = 1.;
  if (d1 > d2) {
    double const swap = d1;
    d1 = d2;
    d2 = swap;
    sign = -1.;
  }
  double const fs = o.sample_rate;
  double const x1 = (d1 - o.start_time) * fs;
  double const x2 = (d2 - o.start_time) * fs;
  double const sb = floor(x1 + 0.5);
  double const eb = floor(x2 + 0.5);
  double const den = 1. - nbk;
  int const nb = x86_int(eb - sb);
  double const f1 = fabs(x1 - floor(x1) - 0.5);
  double const mag = fabs(x1) + static_cast<double>(nb) + fabs(d1 * fs) + fabs(o.start_time * fs) + 2.;
  bool const run_ok = mag < 0x1p50 && f1 > mag * 0x1p-48;
  if (nb > 1 && !run_ok) return false;
  Vec3<Amp> const k{static_cast<Amp>(path.kx), static_cast<Amp>(path.ky), static_cast<Amp>(path.kz)};
  Vec3<Amp> const beta{static_cast<Amp>(t.bx), static_cast<Amp>(t.by), static_cast<Amp>(t.bz)};
  out.perp = cross(k, cross(beta, k));
  double const sc = sign * t.constant;
  double const dd = den * path.dist;
  bool const single = sb == eb;
  bool const tiny = !(fabs(den) > 1.e-15);
  double const frac_last = single ? (tiny ? (t2 - t1) * fs : fabs(d2 * fs - d1 * fs))
                                  : fabs(x2 + 0.5 - eb);
  double const den_last = single && tiny ? path.dist : dd;
  out.last = amp_div(static_cast<Amp>(sc * frac_last), static_cast<Amp>(den_last));
  out.flags = 0u;
  out.start = 0u;
  out.count = 0u;
  out.last_bin = 0u;
  // last sample, add_sample(detection_time2): bin nearest((d2 - t0) fs) = nearest(x2)
  double const bv2 = nearest_bin(x2);
  if (bv2 != eb) return false;
  if (bv2 >= 0. && bv2 < o.bins_d) {
    out.last_bin = static_cast<uint32_t>(bv2);
    out.flags = 2u;
  }
  if (single) return true;
  double const frac_first = fabs(sb + 0.5 - x1);
  out.first = amp_div(static_cast<Amp>(sc * frac_first), static_cast<Amp>(dd));
  double const mc = (subdivided ? 1. : sign) * t.constant;
  out.mid = amp_div(static_cast<Amp>(mc), static_cast<Amp>(dd));
  // first sample, add_sample(detection_time1): bin nearest(x1)
  double const bv1 = nearest_bin(x1);
  if (bv1 != sb) return false;
  bool const first_in = bv1 >= 0. && bv1 < o.bins_d;
  if (first_in) {
    out.start = static_cast<uint32_t>(bv1);
    out.count = 1u;
    out.flags |= 1u;
  }
  if (nb > 1) {  // intermediate bins b1 + i, i in [1, nb), clipped to the trace
    long long const b1 = static_cast<long long>(floor(x1)) + (x1 - floor(x1) >= 0.5 ? 1 : 0);
    long long lo = 1, hi = nb;
    if (-b1 > lo) lo = -b1;
    long long const top = static_cast<long long>(o.bins) - b1;
    if (top < hi) hi = top;
    if (hi > lo) {
      if (first_in) {  // b1 = nearest(x1) >= 0, so lo = 1: one run from the first sample
        out.count = static_cast<uint32_t>(1 + (hi - lo));
      } else {
        out.start = static_cast<uint32_t>(b1 + lo);
        out.count = static_cast<uint32_t>(hi - lo);
      }
    }
  }
  return true;
}

// The Fraunhofer number of an undivided track, (|beta|^2 - w^2) (h fs)^2 / |d|
// times 8 pi c^2 / (wavelength fs^2) for the half duration h, surely below 1:
// accumulate_zhs (RadioProjection.inl:483-503) then takes one segment.  The
// difference |beta|^2 - w^2 is within 2^-46 of the reference's, so for a factor
// below 2^18 the number is within 2^-26 of its FP64 value (the guard is
// 2^-20); above it the caller defers.
__device__ __forceinline__ bool surely_undivided(LeanPoint const& m, LeanObserver const& l, double half_bins,
                                                 double bx, double by, double bz) {
  double const square = fma(bz, bz, fma(by, by, bx * bx));
  double const factor = half_bins * half_bins * (m.inverse * l.fraunhofer);
  return (factor < 0x1p18) & (fma(-m.w, m.w, square) * factor < 1. - 0x1p-20);
}

// One ZHS segment (RadioProjection.inl:412-480) by the filtered arithmetic,
// staged: `m` is its midpoint with the time in its middle, half_bins half its
// duration in bins, `constant` the charge constant in the observer's units.
// Its detection times are m.x -+ |half_bins (1 - n w)|, in time order, and the
// potential's sign times 1 / (1 - n w) is 1 / |1 - n w|.  False when a guard
// cannot decide (the caller evaluates the segment exactly).  `cut`: an end of the
// trace cuts the segment.
__device__ __forceinline__ bool zhs_lean(LeanPoint const& m, double half_bins, float constant, double bx, double by,
                                         double bz, LeanObserver const& l, bool subdivided,
                                         StagedSegment<float>& out, bool& cut) {
  double const reach = fabs(half_bins * m.factor);
  double const x1 = m.x - reach, x2 = m.x + reach;
  out.flags = 0u;
  out.start = 0u;
  out.count = 0u;
  out.last_bin = 0u;
  int b1, b2;
  double const r1 = lean_nearest(x1, b1), r2 = lean_nearest(x2, b2);
  bool const decided = (fabs(r1) < 0.5 - kBinGuard) & (fabs(r2) < 0.5 - kBinGuard) & (reach > kBinGuard) &
                       (fabs(m.factor) >= 1.e-6);
  cut = false;
  if ((x2 < -1.) | (x1 > l.past)) return m.ok;  // off the trace
  cut = (static_cast<unsigned>(b1) >= l.bins) | (static_cast<unsigned>(b2) >= l.bins);
  // from here |x1|, |x2| < 2^27: reach is below 2^25 and one of them is near the trace
  float const amplitude = __fdividef(constant, static_cast<float>(fabs(m.factor) * m.dist));
  out.perp = Vec3<float>{static_cast<float>(fma(-m.dx, m.along, bx)), static_cast<float>(fma(-m.dy, m.along, by)),
                         static_cast<float>(fma(-m.dz, m.along, bz))};
  bool const single = b1 == b2;
  out.last = amplitude * static_cast<float>(single ? 2. * reach : r2 + 0.5);
  out.first = amplitude * static_cast<float>(0.5 - r1);
  out.mid = (subdivided & (m.factor < 0.)) ? -amplitude : amplitude;
  unsigned const bins = l.bins;
  if (static_cast<unsigned>(b2) < bins) {
    out.last_bin = static_cast<unsigned>(b2);
    out.flags = 2u;
  }
  if (!single) {
    bool const first_in = static_cast<unsigned>(b1) < bins;
    int const low = b1 + 1 > 0 ? b1 + 1 : 0;
    int const high = b2 < static_cast<int>(bins) ? b2 : static_cast<int>(bins);
    int const mids = high > low ? high - low : 0;
    out.start = static_cast<unsigned>(first_in ? b1 : low);
    out.count = static_cast<unsigned>(mids) + (first_in ? 1u : 0u);
    out.flags |= first_in ? 1u : 0u;
  }
  return decided & m.ok;
}

// Deposits the staged segments of a warp: every lane takes two bins of the
// flattened list (lane order, then bin order) per step, their owner searches
// interleaved.  Every lane of the
// warp calls it; `staging` is the warp's 32 slots in shared memory.
template <bool kFixed, class Amp, class Sink>
__device__ __forceinline__ void deposit_staged(StagedSegment<Amp>* staging,
                                               StagedSegment<Amp> const& seg,
                                               ObserverCache const& o, Sink& sink, Counts& c) {
  unsigned const lane = threadIdx.x & 31u;
  uint32_t const cnt = seg.count + ((seg.flags >> 1) & 1u);
  uint32_t incl = cnt;
#pragma unroll
  for (unsigned d = 1; d < 32u; d <<= 1) {
    uint32_t const v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  uint32_t const total = __shfl_sync(0xffffffffu, incl, 31);
  if (total == 0u) return;
  staging[lane] = seg;
  __syncwarp();
  uint32_t const before_mine = incl - cnt;
  // the converting fields in registers: `o` lives in shared memory, which the
  // window atomics below might alias as far as the compiler can tell
  ObserverCache grid;
  grid.fixed_scale = o.fixed_scale;
  grid.fixed_scale_f = 1.f;  // staged FP32 values are in fixed-point units
  grid.count_samples = o.count_samples;
  for (uint32_t base = 0; base < total; base += 64u) {
    uint32_t const j0 = base + lane, j1 = j0 + 32u;
    uint32_t owner0 = 0, owner1 = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1u; step >>= 1) {
      uint32_t const v0 = __shfl_sync(0xffffffffu, incl, owner0 + step - 1u);
      uint32_t const v1 = __shfl_sync(0xffffffffu, incl, owner1 + step - 1u);
      if (v0 <= j0) owner0 += step;
      if (v1 <= j1) owner1 += step;
    }
    uint32_t const before0 = __shfl_sync(0xffffffffu, before_mine, owner0 & 31u);
    uint32_t const before1 = __shfl_sync(0xffffffffu, before_mine, owner1 & 31u);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t const j = u ? j1 : j0;
      uint32_t const owner = u ? owner1 : owner0;
      uint32_t const before = u ? before1 : before0;
      if (j < total) {
        StagedSegment<Amp> const& g = staging[owner];
        uint32_t const k = j - before;
        uint32_t bin;
        Amp scale;
        if (k < g.count) {
          bin = g.start + k;
          scale = (k == 0u && (g.flags & 1u)) ? g.first : g.mid;
        } else {
          bin = g.last_bin;
          scale = g.last;
        }
        deposit_bin<kFixed>(sink, bin, make_deposit<kFixed>(grid, scaled(g.perp, scale)), c.zhs,
                            c.overflows, c.mag);
      }
    }
  }
  __syncwarp();
}

// The owner's half of the unchecked deposit of its staged segment (fixed
// point, the whole trace in the window, whose adds are not checked): shows
// once for the segment that every sample converts -- each component's
// |(p_c scale) fixed_scale| is at most max|p_c| max|scale| fixed_scale (1 +
// 2^-22), kept below 2^62 -- counts the samples as contributions and adds
// an upper bound of their |components| to the window bound (each factor's
// roundings, at most nine of 2^-24, inside the 2^-20 margin).  The deposit
// then converts and adds each sample with no check.  Returns false when a
// sample might not convert (huge or non-finite values): the pair then goes to
// the checked drain.
template <class Amp, class Tallies>
__device__ __forceinline__ bool account_staged(StagedSegment<Amp> const& seg, LeanObserver const& l,
                                               Tallies& c) {
  uint32_t const samples = seg.count + ((seg.flags >> 1) & 1u);
  if (samples == 0u) return true;
  bool const has_first = (seg.flags & 1u) != 0u;
  uint32_t const mids = seg.count - (has_first ? 1u : 0u);
  Amp const zero = static_cast<Amp>(0);
  Amp const af = has_first ? fabs(seg.first) : zero;
  Amp const am = mids ? fabs(seg.mid) : zero;
  Amp const al = (seg.flags & 2u) ? fabs(seg.last) : zero;
  // staged FP32 values are in fixed-point units; when counting samples each component adds 1
  Amp const fs = sizeof(Amp) == sizeof(float) ? static_cast<Amp>(1) : static_cast<Amp>(l.fixed_scale);
  Amp const width = (fabs(seg.perp.x) + fabs(seg.perp.y) + fabs(seg.perp.z)) * fs;
  if (!(width * fmax(fmax(af, am), al) < static_cast<Amp>(0x1p62))) return false;  // also NaN and infinities
  Amp const sum = (af + am * static_cast<Amp>(mids) + al) * width +
                  static_cast<Amp>(3u * samples) * static_cast<Amp>(l.bias);
  c.zhs += samples;
  Amp const bound = sum * static_cast<Amp>(1. + 0x1p-20);
  c.mag += sizeof(Amp) == sizeof(float) ? static_cast<float>(bound)
                                        : __double2float_ru(static_cast<double>(bound));
  return true;
}

// The fixed-point value of one staged component, as to_fixed computes it; 1
// when counting samples (the amplitude or the scale is 0 then, the bias 1).
__device__ __forceinline__ long long fixed_value(float v, float amplitude, float, float bias) {
  return __float2ll_rn(fmaf(v, amplitude, bias));
}
__device__ __forceinline__ long long fixed_value(double v, double amplitude, double scale, double bias) {
  return __double2ll_rn(fma(v * amplitude, scale, bias));
}

// Adds a bin's three components to its words of a window (a generic pointer).
__device__ __forceinline__ void add_words(unsigned long long* words, Vec3<long long> v) {
  atomicAdd(words, static_cast<unsigned long long>(v.x));
  atomicAdd(words + 1, static_cast<unsigned long long>(v.y));
  atomicAdd(words + 2, static_cast<unsigned long long>(v.z));
}

// The unchecked deposit of a staged segment as differences: the window holds
// the differences of consecutive bins and difference_window sums them before
// the flush.  A segment's samples are constant between its first and its last
// bin, so it touches at most four bins -- start, start + 1, the bin after the
// run (its last sample) and the next -- whatever its length, each lane on its
// own: no redistribution over the warp (a prefix sum, searches by shuffle and
// 40 bytes staged a lane in the former version, 764 and 143 warp instructions per
// 32 pairs with the drain; with the filtered segment it takes 370 in all, ZHS of
// the 1e7 x 160 workload 59.4 -> 23.0 ms).  On the 1e7 x 160 workload 55% of the
// segments have one sample, 26% two, 17% more (2.0 samples a pair, 2.6
// differences).  The sums of differences are exact modulo 2^64, and the
// item's bound (account_staged) shows that no bin's value leaves the int64
// range.  The adds go through a generic pointer: where the compiler can tell
// the window is shared memory it emits shared-space 64-bit atomics, which this
// GPU executes as about one instruction per active lane (twice the atomic
// wavefronts of generic adds on the same samples).
template <class Amp>
__device__ __forceinline__ void deposit_differences(StagedSegment<Amp> const& seg, LeanObserver const& l,
                                                    unsigned long long* win, uint32_t width) {
  bool const last = (seg.flags & 2u) != 0u;
  if (seg.count == 0u && !last) return;
  // FP32 values are staged in fixed-point units, 0 when counting samples
  Amp const bias = static_cast<Amp>(l.bias);
  Amp const scale = sizeof(Amp) == sizeof(float) ? static_cast<Amp>(1) : static_cast<Amp>(l.fixed_scale);
  asm volatile("" : "+l"(win));
  auto value = [&](Amp amplitude) {
    return Vec3<long long>{fixed_value(seg.perp.x, amplitude, scale, bias),
                           fixed_value(seg.perp.y, amplitude, scale, bias),
                           fixed_value(seg.perp.z, amplitude, scale, bias)};
  };
  auto add = [&](uint32_t bin, Vec3<long long> v) { add_words(win + 3u * bin, v); };
  Vec3<long long> run{0, 0, 0};  // the value up to the bin before `end`
  uint32_t const end = seg.start + seg.count;
  if (seg.count != 0u) {
    bool const first = (seg.flags & 1u) != 0u;
    run = value(first ? seg.first : seg.mid);
    add(seg.start, run);
    if (first && seg.count > 1u) {
      Vec3<long long> const mid = value(seg.mid);
      add(seg.start + 1u, Vec3<long long>{mid.x - run.x, mid.y - run.y, mid.z - run.z});
      run = mid;
    }
  }
  // the last sample is in the bin after the run (staged runs are clipped to
  // the trace only at its start when the last sample is on it)
  if (last) {
    Vec3<long long> const v = value(seg.last);
    add(seg.last_bin, Vec3<long long>{v.x - run.x, v.y - run.y, v.z - run.z});
    run = v;
  }
  uint32_t const after = last ? seg.last_bin + 1u : end;
  if (after < width) add(after, Vec3<long long>{-run.x, -run.y, -run.z});
}

// The samples of a staged segment one by one, each component converted only if
// it can be (fixed point).
template <class Amp, class Sink>
__device__ __noinline__ Counts deposit_samples(StagedSegment<Amp> const seg, ObserverCache const& o, Sink sink) {
  Counts c;
  ObserverCache grid;
  grid.fixed_scale = o.fixed_scale;
  grid.fixed_scale_f = 1.f;  // staged FP32 values are in fixed-point units
  grid.count_samples = o.count_samples;
  for (uint32_t k = 0; k < seg.count; ++k) {
    Amp const amplitude = k == 0u && (seg.flags & 1u) ? seg.first : seg.mid;
    deposit_bin<true>(sink, seg.start + k, make_deposit<true>(grid, scaled(seg.perp, amplitude)), c.zhs, c.overflows,
                      c.mag);
  }
  if (seg.flags & 2u)
    deposit_bin<true>(sink, seg.last_bin, make_deposit<true>(grid, scaled(seg.perp, seg.last)), c.zhs, c.overflows,
                      c.mag);
  return c;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  return v;
}

// Turns a window of differences into the bins' values: a running sum of each
// component over the bins.  Every thread of the CTA calls it.  Out of line, so
// that its registers do not count in the track loops.
__device__ __noinline__ void difference_window(unsigned long long* win, uint32_t width) {
  __shared__ unsigned long long totals[32];  // of each warp's bins, one component at a time
  unsigned const lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t per = (width + blockDim.x - 1) / blockDim.x;
  per |= 1u;  // an odd stride keeps the lanes' 64-bit words on different banks
  uint32_t const first = threadIdx.x * per < width ? threadIdx.x * per : width;
  uint32_t const stop = first + per < width ? first + per : width;
  __syncthreads();
  unsigned long long sum[3] = {0, 0, 0};
  for (uint32_t j = first; j < stop; ++j)
#pragma unroll
    for (int k = 0; k < 3; ++k) sum[k] += win[3u * j + k];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    unsigned long long incl = sum[k];
    for (unsigned d = 1; d < 32u; d <<= 1) {
      unsigned long long const v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31u) totals[warp] = incl;
    __syncthreads();
    // the warps before this one: a lane takes one total, the warp adds them
    sum[k] = incl - sum[k] + __shfl_sync(0xffffffffu, warp_sum(lane < warp ? totals[lane] : 0ull), 0);
    __syncthreads();
  }
  for (uint32_t j = first; j < stop; ++j)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      sum[k] += win[3u * j + k];
      win[3u * j + k] = sum[k];
    }
  __syncthreads();
}

// An undivided segment evaluated and deposited as differences in one go, in mixed
// precision with the whole trace in the window: zhs_lean and
// deposit_differences without the staged form between them, for segments that
// lie on the trace whole (or off it whole).  The amplitudes and conversions are
// those of zhs_lean's segments.  False, having deposited nothing, when a guard
// cannot decide, an end of the trace cuts the segment or a value might not
// convert.
__device__ __forceinline__ bool zhs_lean_differences(LeanPoint const& m, double half_bins, float constant, double bx,
                                                     double by, double bz, LeanObserver const& l,
                                                     unsigned long long* win, Tally& c) {
  double const reach = fabs(half_bins * m.factor);
  double const x1 = m.x - reach, x2 = m.x + reach;
  if ((x2 < -1.) | (x1 > l.past)) return m.ok;  // off the trace
  int b1, b2;
  double const r1 = lean_nearest(x1, b1), r2 = lean_nearest(x2, b2);
  bool const decided = (fabs(r1) < 0.5 - kBinGuard) & (fabs(r2) < 0.5 - kBinGuard) & (reach > kBinGuard) &
                       (fabs(m.factor) >= 1.e-6) & (static_cast<unsigned>(b1) < l.bins) &
                       (static_cast<unsigned>(b2) < l.bins) & m.ok;
  float const amplitude = __fdividef(constant, static_cast<float>(fabs(m.factor) * m.dist));
  Vec3<float> const perp{static_cast<float>(fma(-m.dx, m.along, bx)), static_cast<float>(fma(-m.dy, m.along, by)),
                         static_cast<float>(fma(-m.dz, m.along, bz))};
  int const bins = b2 - b1;  // after the first
  float const first = amplitude * static_cast<float>(0.5 - r1);
  float const last = amplitude * static_cast<float>(bins == 0 ? 2. * reach : r2 + 0.5);
  // every |sample| is at most |perp|_1 |amplitude|; the roundings lie inside 2^-20
  float const width = fabsf(perp.x) + fabsf(perp.y) + fabsf(perp.z);
  if (!(decided & (width * fabsf(amplitude) < 0x1p60f))) return false;  // also NaN and infinities
  unsigned const samples = static_cast<unsigned>(bins) + 1u;
  float const between = bins == 0 ? fabsf(last) : fabsf(first) + fabsf(last) + static_cast<float>(bins - 1) * fabsf(amplitude);
  c.zhs += samples;
  c.mag = fmaf(between * width, 1.f + 0x1p-20f, c.mag) + static_cast<float>(3u * samples) * l.bias;
  auto value = [&](float a) {
    return Vec3<long long>{fixed_value(perp.x, a, 1.f, l.bias), fixed_value(perp.y, a, 1.f, l.bias),
                           fixed_value(perp.z, a, 1.f, l.bias)};
  };
  // through a generic pointer (see deposit_differences)
  unsigned long long* w = win + 3u * static_cast<unsigned>(b1);
  asm volatile("" : "+l"(w));
  Vec3<long long> run{0, 0, 0};
  if (bins > 0) {
    run = value(first);
    add_words(w, run);
    if (bins > 1) {
      Vec3<long long> const mid = value(amplitude);
      add_words(w + 3, Vec3<long long>{mid.x - run.x, mid.y - run.y, mid.z - run.z});
      run = mid;
    }
  }
  Vec3<long long> const v = value(last);
  unsigned long long* const end = w + 3 * bins;
  add_words(end, Vec3<long long>{v.x - run.x, v.y - run.y, v.z - run.z});
  if (static_cast<unsigned>(b2) + 1u < l.bins) add_words(end + 3, Vec3<long long>{-v.x, -v.y, -v.z});
  return true;
}

// The FP64 counterpart: an undivided segment evaluated exactly (zhs_stage's
// operations and decisions) and deposited as differences in one go.  Its fields
// are formed one at a time as they are deposited, where a staged segment holds
// six FP64 values a lane at once (which spilled the track loop at 640 threads).
__device__ __forceinline__ bool zhs_exact_differences(Path const& path, double t1, double t2, double mt, double bx,
                                                      double by, double bz, double constant, ObserverCache const& o,
                                                      LeanObserver const& l, unsigned long long* win, Tally& c) {
  double const bk = bx * path.kx + by * path.ky + bz * path.kz;
  double const nbk = path.n_src * bk;
  double d1 = t1 + path.time - nbk * (t1 - mt);
  double d2 = t2 + path.time - nbk * (t2 - mt);
  double sign = 1.;
  if (d1 > d2) {
    double const swap = d1;
    d1 = d2;
    d2 = swap;
    sign = -1.;
  }
  double const fs = o.sample_rate;
  double const x1 = (d1 - o.start_time) * fs;
  double const x2 = (d2 - o.start_time) * fs;
  if ((x2 < -1.) | (x1 > l.past)) return true;  // off the trace
  // on the trace whole (an end that cuts the segment is left to the drain); then
  // floor(x + 0.5) is an int
  double const sb = floor(x1 + 0.5), eb = floor(x2 + 0.5);
  if (!((sb >= 0.) & (eb < o.bins_d) & (x1 >= -0.5) & (nearest_bin(x1) == sb) & (nearest_bin(x2) == eb))) return false;
  int const b1 = static_cast<int>(sb), bins = static_cast<int>(eb) - b1;
  double const f1 = fabs(x1 - floor(x1) - 0.5);
  double const mag = fabs(x1) + static_cast<double>(bins) + fabs(d1 * fs) + fabs(l.start_bins) + 2.;
  // the consecutive-run test of zhs_segment
  if (bins > 1 && !(mag < 0x1p50 && f1 > mag * 0x1p-48)) return false;
  double const den = 1. - nbk;
  Vec3<double> const k{path.kx, path.ky, path.kz};
  Vec3<double> const perp = cross(k, cross(Vec3<double>{bx, by, bz}, k));
  double const sc = sign * constant;
  double const dd = den * path.dist;
  bool const tiny = !(fabs(den) > 1.e-15);
  double const frac_last = bins == 0 ? (tiny ? (t2 - t1) * fs : fabs(d2 * fs - d1 * fs)) : fabs(x2 + 0.5 - eb);
  double const last = sc * frac_last / (bins == 0 && tiny ? path.dist : dd);
  double first = 0., mid = 0.;
  if (bins > 0) first = sc * fabs(sb + 0.5 - x1) / dd;
  if (bins > 1) mid = sc / dd;
  double const width = (fabs(perp.x) + fabs(perp.y) + fabs(perp.z)) * l.fixed_scale;
  if (!(width * fmax(fmax(fabs(first), fabs(mid)), fabs(last)) < 0x1p60)) return false;  // also NaN and infinities
  unsigned const samples = static_cast<unsigned>(bins) + 1u;
  c.zhs += samples;
  c.mag += __double2float_ru((fabs(first) + fabs(last) + fabs(mid) * static_cast<double>(bins > 1 ? bins - 1 : 0)) *
                                 width * (1. + 0x1p-20) +
                             static_cast<double>(3u * samples) * static_cast<double>(l.bias));
  double const bias = static_cast<double>(l.bias);
  auto value = [&](double a) {
    return Vec3<long long>{fixed_value(perp.x, a, l.fixed_scale, bias), fixed_value(perp.y, a, l.fixed_scale, bias),
                           fixed_value(perp.z, a, l.fixed_scale, bias)};
  };
  unsigned long long* w = win + 3u * static_cast<unsigned>(b1);
  asm volatile("" : "+l"(w));
  Vec3<long long> run{0, 0, 0};
  if (bins > 0) {
    run = value(first);
    add_words(w, run);
    if (bins > 1) {
      Vec3<long long> const v = value(mid);
      add_words(w + 3, Vec3<long long>{v.x - run.x, v.y - run.y, v.z - run.z});
      run = v;
    }
  }
  Vec3<long long> const v = value(last);
  unsigned long long* const end = w + 3 * bins;
  add_words(end, Vec3<long long>{v.x - run.x, v.y - run.y, v.z - run.z});
  if (static_cast<unsigned>(b1 + bins) + 1u < l.bins) add_words(end + 3, Vec3<long long>{-v.x, -v.y, -v.z});
  return true;
}

// The subdivision of a track seen from an observer (accumulate_zhs,
// RadioProjection.inl:483-503), every operation exact.
struct Subdivision {
  double divisor;
  int subtracks;
};
template <bool kDivide = false>
__device__ __forceinline__ Subdivision subdivide(Track t, Propagation const& p, ObserverCache const& o) {
  derive_track(t);
  double const mx = (t.sx + t.ex) * 0.5, my = (t.sy + t.ey) * 0.5, mz = (t.sz + t.ez) * 0.5;
  Path const pm = propagate<false, kDivide>(p, o, mx, my, mz);
  double const uk = (t.bx * pm.kx + t.by * pm.ky + t.bz * pm.kz) / t.beta_module;
  double const s2 = 1. - uk * uk;
  double const fraunhofer = s2 * t.length * t.length / pm.dist / o.wavelength * 2. * kPi;
  Subdivision d{1., 1};
  if (fraunhofer > 1.) {
    d.divisor = sqrt(fraunhofer) + 1.;
    d.subtracks = x86_int(ceil(d.divisor));
  }
  return d;
}
// Whether a track seen from an observer is surely one segment: the Fraunhofer
// number as surely_undivided estimates it, 8 pi c^2 / (wavelength fs^2) being
// 8 pi wavelength (wavelength = c / fs).
__device__ __forceinline__ bool surely_one_segment(Track const& t, ObserverCache const& o) {
  double const dx = o.px - (t.sx + t.ex) * 0.5, dy = o.py - (t.sy + t.ey) * 0.5, dz = o.pz - (t.sz + t.ez) * 0.5;
  double inverse;
  bool const ok = lean_rsqrt(fma(dz, dz, fma(dy, dy, dx * dx)), inverse);
  double const w = fma(t.bz, dz, fma(t.by, dy, t.bx * dx)) * inverse;
  double const square = fma(t.bz, t.bz, fma(t.by, t.by, t.bx * t.bx));
  double const half_bins = (t.te - t.ts) * 0.5 * o.sample_rate;
  double const factor = half_bins * half_bins * (inverse * (8. * kPi) * o.wavelength);
  return ok & (fabs(t.bx) + fabs(t.by) + fabs(t.bz) <= 4.) & (factor < 0x1p18) &
         (fma(-w, w, square) * factor < 1. - 0x1p-20);
}

// accumulate_zhs, RadioProjection.inl:483-529, every decision exact (the plain
// shapes: kDivide, see propagate_with).
template <bool kFixed, class Amp, class Sink>
__device__ __forceinline__ void zhs_pair(Track const& t, Propagation const& p,
                                         ObserverCache const& o, Sink& sink, Counts& c) {
  double divisor = 1.;
  int subtracks = 1;
  if (!surely_one_segment(t, o)) {
    Subdivision const d = subdivide<true>(t, p, o);
    divisor = d.divisor;
    subtracks = d.subtracks;
  }
  c.subtracks += static_cast<unsigned long long>(static_cast<long long>(subtracks));
  int const refinement = static_cast<int>(p.refinement);
  // One segment when undivided: the loop below then evaluates
  // point2 = start + (end - start) / 1 / 1, exactly the reference's values.
  bool const subdivided = subtracks > 1 || refinement > 1;
  double rx = t.ex - t.sx, ry = t.ey - t.sy, rz = t.ez - t.sz, rt = t.te - t.ts;
  if (refinement > 1) {  // x / 1 == x exactly: undivided tracks skip the divisions
    double const rd = static_cast<double>(refinement);
    rx = rx / divisor / rd;
    ry = ry / divisor / rd;
    rz = rz / divisor / rd;
    rt = rt / divisor / rd;
  } else if (subdivided) {
    rx = rx / divisor;
    ry = ry / divisor;
    rz = rz / divisor;
    rt = rt / divisor;
  }
  double p1x = t.sx, p1y = t.sy, p1z = t.sz, t1 = t.ts;
  // subtrack-major, refinement-minor order of the reference's nested loops
  long long const segments = static_cast<long long>(subtracks) * refinement;
#pragma unroll 1
  for (long long index = 0; index < segments; ++index) {
    double const p2x = p1x + rx, p2y = p1y + ry, p2z = p1z + rz, t2 = t1 + rt;
    zhs_segment<kFixed, false, Amp, true>(p1x, p1y, p1z, p2x, p2y, p2z, t1, t2, t, p, o, sink, c, subdivided);
    p1x = p2x;
    p1y = p2y;
    p1z = p2z;
    t1 = t2;
  }
  if (refinement > 1)
    c.subtracks += static_cast<unsigned long long>(
        static_cast<long long>(subtracks * (refinement - 1)));
}

// The segment of an undivided track seen from the item's observer, from the
// track's columns `r`, by the filtered arithmetic.  `one`: the track is surely
// one segment but for refinement (the Fraunhofer number surely below 1) and inside
// the filtered paths' bounds.
struct ZhsPoint {
  LeanPoint m;
  double half_bins, bx, by, bz;
  float constant;
  SourceTerms terms;
  bool one;
};
template <bool kPre>
__device__ __forceinline__ ZhsPoint zhs_point(double2 const* __restrict__ r, Propagation const& p,
                                              LeanObserver const& l) {
  constexpr unsigned T = kTrackTile;
  double2 const cd = __ldg(r + 4 * T), ce = __ldg(r + 5 * T), cm = __ldg(r + 9 * T), cn = __ldg(r + 10 * T);
  double const half = __ldg(reinterpret_cast<double const*>(r + kHalf / 2 * T));
  unsigned const flags = pack_flags(ce.y);
  ZhsPoint z;
  if (kPre) {
    double2 const m = __ldg(r + kFactorMid / 2 * T);
    z.terms = SourceTerms{m.x, m.y, 0.};
  } else {
    z.terms = source_terms(p, destination_of(s_observer), cn.x);
  }
  z.bx = cd.x;
  z.by = cd.y;
  z.bz = ce.x;
  z.m = lean_point(l, cm.x, cm.y, cn.x, cn.y, cd.x, cd.y, ce.x, z.terms.factor, z.terms.n_src);
  z.half_bins = half * l.rate;
  z.constant = pack_constant(ce.y) * l.scale;
  z.one = ((flags & kTrackRegular & l.usable) != 0u) & z.m.ok &
          surely_undivided(z.m, l, z.half_bins, cd.x, cd.y, ce.x);
  if (!kPre) z.one = z.one & lean_terms(z.terms);
  return z;
}

// The common ZHS pair of the windowed kernel: one undivided segment, staged.
// Returns false, staging nothing (`seg` cleared), when the track is or might be
// subdivided or when the segment cannot be staged; the kernel then defers the
// pair to a drain.  Mixed precision (Amp = float) stages by the filtered
// arithmetic, FP64 exactly; both decide "one segment" from the filtered
// midpoint, which spares FP64 the exact Fraunhofer number (a square root and
// seven divisions).
template <bool kFixed, bool kPre, class Amp>
__device__ __forceinline__ bool zhs_common(double2 const* __restrict__ r, Propagation const& p,
                                           LeanObserver const& l, StagedSegment<Amp>& seg) {
  constexpr unsigned T = kTrackTile;
  ZhsPoint const z = zhs_point<kPre>(r, p, l);
  bool staged = z.one;
  if constexpr (sizeof(Amp) == sizeof(float)) {
    // in fixed point a cut segment is the drain's, as in zhs_lean_differences: a sample's
    // FP32 value is then the same bits whether its item runs with checked adds or without
    bool cut;
    staged = zhs_lean(z.m, z.half_bins, z.constant, z.bx, z.by, z.bz, l, false, seg, cut) & staged &
             !(kFixed && cut);
  } else if (staged) {
    double2 const cm = __ldg(r + 9 * T), cn = __ldg(r + 10 * T), ct = __ldg(r + 3 * T);
    Track t;
    t.bx = z.bx;
    t.by = z.by;
    t.bz = z.bz;
    t.constant = __ldg(r + kConst / 2 * T).y;
    staged = zhs_stage<Amp, true>(cm.x, cm.y, cn.x, ct.x, ct.x + (ct.y - ct.x), cn.y, t, p,
                                          copy_words(s_observer), false, seg, z.terms);
  }
  if (!staged) {
    seg.count = 0u;
    seg.flags = 0u;
  }
  return staged;
}

// ---------------------------------------------------------------- helpers
// The fields of a track, its columns read by `load`; length and |beta| are left
// to derive_track, where an exact evaluation needs them.
template <class Load>
__device__ __forceinline__ Track unpack_track(Load load) {
  double2 const a = load(0), b = load(1), c = load(2), d = load(3);
  double2 const e = load(4), f = load(5), g = load(kConst / 2);
  Track t;
  t.sx = a.x;
  t.sy = a.y;
  t.sz = b.x;
  t.ex = b.y;
  t.ey = c.x;
  t.ez = c.y;
  t.ts = d.x;
  t.te = d.y;
  t.bx = e.x;
  t.by = e.y;
  t.bz = f.x;
  t.constant = g.y;
  return t;
}

__device__ __forceinline__ Track load_track(const double* __restrict__ base, uint64_t i) {
  double2 const* r = track_ref(base, i);
  return unpack_track([&](unsigned k) { return __ldg(r + k * kTrackTile); });
}

// A track staged in shared memory as one interleaved 192-byte record (plain
// loads: __ldg reads the global space only).
__device__ __forceinline__ Track load_staged_track(double const* base, unsigned i) {
  double2 const* r = reinterpret_cast<double2 const*>(base + i * kTrackDoubles);
  return unpack_track([&](unsigned k) { return r[k]; });
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int d = 16; d > 0; d >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, d));
  return v;
}

// Adds per-thread counts into the event counters: one atomic per warp.
// Every lane of the warp must call it.
__device__ __forceinline__ void flush_counts(Counts& c, DeviceCounters* counters) {
  unsigned long long const a = warp_sum(c.coreas), b = warp_sum(c.zhs),
                           s = warp_sum(c.subtracks), f = warp_sum(c.overflows);
  if ((threadIdx.x & 31) == 0) {
    if (a) atomicAdd(&counters->coreas_contributions, a);
    if (b) atomicAdd(&counters->zhs_contributions, b);
    if (s) atomicAdd(&counters->zhs_subtracks, s);
    if (f) atomicAdd(&counters->fixed_point_overflows, f);
  }
  c = Counts{};
}

// RadioAtomicOperations::maximum (RadioAtomicOperations.inl:46-56): finite,
// non-negative maxima compare as their bit patterns.
__device__ __forceinline__ void atomic_max_nonnegative(double* address, double value) {
  atomicMax(reinterpret_cast<unsigned long long*>(address),
            static_cast<unsigned long long>(__double_as_longlong(value)));
}

// diagnostic_energy_bin, RadioProjection.inl:531-538.
__device__ __forceinline__ int energy_bin(double kinetic) {
  double const edges[14] = {1.e-3, 2.e-3, 5.e-3, 1.e-2, 2.e-2, 5.e-2, 1.e-1,
                            2.e-1, 5.e-1, 1.,    2.,    5.,    10.,   100.};
  int index = 0;
  while (index < 14 && kinetic > edges[index]) ++index;
  return index;
}

// ---------------------------------------------------------------- ingest
// The fields radio reads from a track step, from 752-byte records or from
// columns (one device array per field): the same arithmetic follows.
struct RecordSource {
  const unsigned char* starts;  // the first record's start state, its end state after it
  uint64_t pitch;               // bytes from one record's to the next's
  __device__ const c8r_particle_state& start(uint64_t i) const {
    return *reinterpret_cast<const c8r_particle_state*>(starts + i * pitch);
  }
  __device__ const c8r_particle_state& end(uint64_t i) const { return (&start(i))[1]; }
  __device__ int pid(uint64_t i) const { return start(i).pid; }
  __device__ double weight(uint64_t i) const { return start(i).weight; }
  __device__ double start_energy(uint64_t i) const { return start(i).energy_gev; }
  __device__ double start_position(uint64_t i, int a) const { return start(i).position_m[a]; }
  __device__ double end_position(uint64_t i, int a) const { return end(i).position_m[a]; }
  __device__ double start_time(uint64_t i) const { return start(i).time_s; }
  __device__ double end_time(uint64_t i) const { return end(i).time_s; }
  __device__ double start_direction(uint64_t i, int a) const { return start(i).direction[a]; }
  __device__ double end_direction(uint64_t i, int a) const { return end(i).direction[a]; }
};
static_assert(offsetof(c8r_lepton_transport_record, end) ==
                  offsetof(c8r_lepton_transport_record, start) + sizeof(c8r_particle_state),
              "a record's end state follows its start state");

struct ColumnSource {
  c8r_track_columns columns;
  __device__ int pid(uint64_t i) const { return columns.pid[i]; }
  __device__ double weight(uint64_t i) const { return columns.weight[i]; }
  __device__ double start_energy(uint64_t i) const { return columns.start_energy_gev[i]; }
  __device__ double start_position(uint64_t i, int a) const { return columns.start_position_m[a][i]; }
  __device__ double end_position(uint64_t i, int a) const { return columns.end_position_m[a][i]; }
  __device__ double start_time(uint64_t i) const { return columns.start_time_s[i]; }
  __device__ double end_time(uint64_t i) const { return columns.end_time_s[i]; }
  __device__ double start_direction(uint64_t i, int a) const { return columns.start_direction[a][i]; }
  __device__ double end_direction(uint64_t i, int a) const { return columns.end_direction[a][i]; }
};

template <class Source>
__global__ void __launch_bounds__(256) ingest_kernel(
    const __grid_constant__ Source src, uint64_t count, double* __restrict__ tracks, uint64_t stride,
    unsigned long long* slot, DeviceCounters* counters, int diagnostics,
    const __grid_constant__ IngestTerms terms) {
  uint64_t const i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  bool valid = false;
  Track t;
  double duration = 0.;
  int pid = 0;
  if (i < count) {
    pid = src.pid(i);
    // make_radio_track_kinematics, RadioProjection.inl:145-168
    if (pid == 11 || pid == -11) {
      t.sx = src.start_position(i, 0);
      t.sy = src.start_position(i, 1);
      t.sz = src.start_position(i, 2);
      t.ex = src.end_position(i, 0);
      t.ey = src.end_position(i, 1);
      t.ez = src.end_position(i, 2);
      t.ts = src.start_time(i);
      t.te = src.end_time(i);
      duration = t.te - t.ts;
      double const dx = t.ex - t.sx, dy = t.ey - t.sy, dz = t.ez - t.sz;
      t.length = sqrt(dx * dx + dy * dy + dz * dz);
      if (duration > 0. && t.length > 0.) {
        double const denominator = kSpeedOfLight * duration;
        t.bx = dx / denominator;
        t.by = dy / denominator;
        t.bz = dz / denominator;
        t.beta_module = t.length / (kSpeedOfLight * duration);
        double const charge = pid == 11 ? -kElementaryCharge : kElementaryCharge;
        t.constant = charge * kEmConstant * src.weight(i);
        valid = true;
      }
    }
  }
  unsigned const ballot = __ballot_sync(0xffffffffu, valid);
  unsigned const lane = threadIdx.x & 31;
  unsigned long long base = 0;
  if (lane == 0 && ballot) base = atomicAdd(slot, static_cast<unsigned long long>(__popc(ballot)));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (valid) {
    uint64_t const j = base + __popc(ballot & ((1u << lane) - 1u));
    double2* r = track_ref(tracks, j);
    constexpr unsigned T = kTrackTile;
    // the ZHS segment of an undivided track, with the reference's own
    // arithmetic (RadioProjection.inl:418-425, :505-512): it ends at
    // start + (end - start)
    double const mx = (t.sx + (t.sx + (t.ex - t.sx))) * 0.5, my = (t.sy + (t.sy + (t.ey - t.sy))) * 0.5,
                 mz = (t.sz + (t.sz + (t.ez - t.sz))) * 0.5;
    double const t2 = t.ts + (t.te - t.ts);
    double const tm = (t.ts + t2) * 0.5;
    bool regular = regular_track(t, duration, terms.limits);
    unsigned flags = 0u;
    if (terms.enabled) {
      // the source points of the windowed kernels
      Propagation const& p = terms.propagation;
      Destination const& d = terms.destination;
      SourceTerms const s = source_terms(p, d, t.sz);
      SourceTerms const e = source_terms(p, d, t.ez);
      SourceTerms const m = source_terms(p, d, mz);
      // the CoREAS near-cone midpoint is (start + end) / 2 (:357-359)
      SourceTerms const mc = source_terms(p, d, (t.sz + t.ez) * 0.5);
      r[6 * T] = make_double2(s.factor, s.n_src);
      r[7 * T] = make_double2(e.factor, e.n_src);
      r[8 * T] = make_double2(m.factor, m.n_src);
      regular = regular && lean_terms(s) && lean_terms(e) && lean_terms(m);
      if (s.n_dst > 1.) flags |= kTrackDense;
      if (mc.factor == m.factor && mc.n_src == m.n_src) flags |= kTrackOneMid;
    }
    if (regular) flags |= kTrackRegular;
    double const pack = __hiloint2double(
        static_cast<int>(flags), __float_as_int(static_cast<float>(t.constant * kConstantShift)));
    r[0 * T] = make_double2(t.sx, t.sy);
    r[1 * T] = make_double2(t.sz, t.ex);
    r[2 * T] = make_double2(t.ey, t.ez);
    r[3 * T] = make_double2(t.ts, t.te);
    r[4 * T] = make_double2(t.bx, t.by);
    r[5 * T] = make_double2(t.bz, pack);
    r[9 * T] = make_double2(mx, my);
    r[10 * T] = make_double2(mz, tm);
    r[11 * T] = make_double2((t2 - t.ts) * 0.5, t.constant);
  }
  if (lane == 0 && ballot) atomicAdd(&counters->valid_tracks, static_cast<unsigned long long>(__popc(ballot)));
  if (!diagnostics) return;

  // record_track diagnostics, RadioProjection.inl:553-610 (warp-reduced).
  double w = 0., len = 0., wl = 0., ewl = 0., el = 0., pl = 0., sl = 0., dchg = 0., dchg2 = 0.,
         bdef = 0., tres = 0., maxlen = 0., maxchg = 0., sdx = 0., sdy = 0., sdz = 0.;
  int ebin = -1;
  double ebin_value = 0.;
  if (valid) {
    double const weight = src.weight(i);
    double const kinetic = src.start_energy(i) - kElectronMassGeV;
    if (isfinite(t.length) && t.length > 0. && isfinite(weight) && !(weight < 0.) &&
        isfinite(kinetic) && !(kinetic < 0.)) {
      double const weighted_length = weight * t.length;
      w = weight;
      len = t.length;
      wl = weighted_length;
      ewl = weighted_length * kinetic;
      maxlen = t.length;
      if (pid == 11) {
        el = weighted_length;
        sl = -weighted_length;
      } else {
        pl = weighted_length;
        sl = weighted_length;
      }
      ebin = energy_bin(kinetic);
      ebin_value = weighted_length;
      double direction_dot = 0.;
      double delta[3];
      for (int axis = 0; axis < 3; ++axis) {
        double const pre = src.start_direction(i, axis);
        double const post = src.end_direction(i, axis);
        direction_dot += pre * post;
        delta[axis] = post - pre;
      }
      double clamped = -1. > direction_dot ? -1. : direction_dot;
      clamped = 1. < clamped ? 1. : clamped;
      double const change = acos(clamped);
      double const residual = duration - t.length / kSpeedOfLight;
      dchg = weight * change;
      dchg2 = weight * change * change;
      bdef = weighted_length * (1. - t.beta_module);
      tres = weight * residual;
      maxchg = change;
      double const charge_sign = pid == 11 ? -1. : 1.;
      sdx = charge_sign * weight * delta[0];
      sdy = charge_sign * weight * delta[1];
      sdz = charge_sign * weight * delta[2];
    }
  }
  w = warp_sum(w);
  len = warp_sum(len);
  wl = warp_sum(wl);
  ewl = warp_sum(ewl);
  el = warp_sum(el);
  pl = warp_sum(pl);
  sl = warp_sum(sl);
  dchg = warp_sum(dchg);
  dchg2 = warp_sum(dchg2);
  bdef = warp_sum(bdef);
  tres = warp_sum(tres);
  sdx = warp_sum(sdx);
  sdy = warp_sum(sdy);
  sdz = warp_sum(sdz);
  maxlen = warp_max(maxlen);
  maxchg = warp_max(maxchg);
  if (lane == 0 && ballot) {
    atomicAdd(&counters->weighted_segment_count, w);
    atomicAdd(&counters->track_length_m, len);
    atomicAdd(&counters->weighted_track_length_m, wl);
    atomicAdd(&counters->energy_weighted_track_length_gev_m, ewl);
    atomicAdd(&counters->electron_weighted_track_length_m, el);
    atomicAdd(&counters->positron_weighted_track_length_m, pl);
    atomicAdd(&counters->signed_charge_weighted_track_length_m, sl);
    atomicAdd(&counters->weighted_direction_change_rad, dchg);
    atomicAdd(&counters->weighted_direction_change_squared_rad2, dchg2);
    atomicAdd(&counters->weighted_beta_deficit_track_length_m, bdef);
    atomicAdd(&counters->weighted_time_residual_s, tres);
    atomicAdd(&counters->signed_charge_weighted_direction_change[0], sdx);
    atomicAdd(&counters->signed_charge_weighted_direction_change[1], sdy);
    atomicAdd(&counters->signed_charge_weighted_direction_change[2], sdz);
    atomic_max_nonnegative(&counters->maximum_segment_length_m, maxlen);
    atomic_max_nonnegative(&counters->maximum_direction_change_rad, maxchg);
  }
  if (ebin >= 0) atomicAdd(&counters->weighted_track_length_by_kinetic_energy_m[ebin], ebin_value);
}

// ---------------------------------------------------------------- direct
template <bool kFixed, class Amp, bool kCoreas, bool kZhs>
__global__ void __launch_bounds__(256) direct_kernel(const __grid_constant__ EventPlan ev) {
  uint64_t const tracks = *ev.valid_tracks;
  uint32_t const observers =
      ev.observer_count[0] > ev.observer_count[1] ? ev.observer_count[0] : ev.observer_count[1];
  uint64_t const pairs = tracks * observers;
  Counts c;
  for (uint64_t pair = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; pair < pairs;
       pair += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    uint64_t const ti = pair / observers;
    uint32_t const oi = static_cast<uint32_t>(pair - ti * observers);
    Track const t = load_track(ev.tracks, ti);
    if (kCoreas && oi < ev.observer_count[0]) {
      ObserverCache const& o = ev.observers[0][oi];
      GlobalSink sink;
      for (int r = 0; r < 3; ++r) {
        sink.row[r] = kFixed ? ev.fixed[0] + r * ev.total_bins[0] + o.offset : nullptr;
        sink.frow[r] = kFixed ? nullptr : ev.floating[0] + r * ev.total_bins[0] + o.offset;
      }
      coreas_pair<kFixed, Amp, GlobalSink, false, true>(t, ev.propagation, o, sink, c);
    }
    if (kZhs && oi < ev.observer_count[1]) {
      ObserverCache const& o = ev.observers[1][oi];
      GlobalSink sink;
      for (int r = 0; r < 3; ++r) {
        sink.row[r] = kFixed ? ev.fixed[1] + r * ev.total_bins[1] + o.offset : nullptr;
        sink.frow[r] = kFixed ? nullptr : ev.floating[1] + r * ev.total_bins[1] + o.offset;
      }
      zhs_pair<kFixed, Amp>(t, ev.propagation, o, sink, c);
    }
  }
  flush_counts(c, ev.counters);
}

// ---------------------------------------------------------------- tiled
// The reference's large-batch launch shape (RadioTileProjection,
// RadioAccumulator.inl:13-85, launched by project(), :699-847, for batches
// of 16384 tracks or more on a GPU): one 256-thread CTA per tile of
// kTileTracks tracks x kTileObservers observers, the tile's track kinematics
// and observer constants staged in shared memory, one thread per pair (lane
// l takes track l / 32 at observer l % 32, so a warp holds one track at 32
// observers), every sample a checked 64-bit global atomic.  Tiles are taken
// by a grid-stride loop over track tile x observer tile.
constexpr int kTileTracks = 8;      // RadioAccumulator.hpp:61 (TrackTileSize)
constexpr int kTileObservers = 32;  // RadioAccumulator.hpp:62 (ObserverTileSize)
constexpr int kTileThreads = kTileTracks * kTileObservers;
static_assert(sizeof(ObserverCache) % sizeof(double2) == 0, "observer constants in 16-byte words");

template <bool kFixed, class Amp, bool kCoreas, bool kZhs>
__global__ void __launch_bounds__(kTileThreads) tiled_kernel(const __grid_constant__ EventPlan ev,
                                                              uint64_t track_tiles) {
  __shared__ __align__(16) double tracks[kTileTracks * kTrackDoubles];
  __shared__ ObserverCache observers[2][kTileObservers];
  uint64_t const valid = *ev.valid_tracks;
  uint32_t const observer_count =
      ev.observer_count[0] > ev.observer_count[1] ? ev.observer_count[0] : ev.observer_count[1];
  uint64_t const observer_tiles = (observer_count + kTileObservers - 1) / kTileObservers;
  uint64_t const tiles = track_tiles * observer_tiles;
  unsigned const track_lane = threadIdx.x / kTileObservers;
  unsigned const observer_lane = threadIdx.x % kTileObservers;
  Counts c;
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint64_t const track_base = (tile / observer_tiles) * kTileTracks;
    uint64_t const observer_base = (tile % observer_tiles) * kTileObservers;
    __syncthreads();  // the previous tile's reads are done
    // column-major over the tile's tracks: consecutive threads read
    // consecutive tracks of one column (kTileTracks divides kTrackTile)
    for (unsigned i = threadIdx.x; i < kTileTracks * kTrackColumns; i += blockDim.x) {
      unsigned const k = i / kTileTracks, lane = i % kTileTracks;
      uint64_t const row = track_base + lane;
      reinterpret_cast<double2*>(tracks)[lane * kTrackColumns + k] =
          row < valid ? __ldg(track_ref(ev.tracks, row) + k * kTrackTile) : make_double2(0., 0.);
    }
    constexpr unsigned kWords = sizeof(ObserverCache) / sizeof(double2);
    for (int a = 0; a < 2; ++a) {
      if (!(a == 0 ? kCoreas : kZhs)) continue;
      for (unsigned i = threadIdx.x; i < kTileObservers * kWords; i += blockDim.x) {
        uint64_t const index = observer_base + i / kWords;
        if (index < ev.observer_count[a])
          reinterpret_cast<double2*>(observers[a])[i] =
              __ldg(reinterpret_cast<double2 const*>(ev.observers[a] + observer_base) + i);
      }
    }
    __syncthreads();
    uint64_t const ti = track_base + track_lane;
    uint64_t const oi = observer_base + observer_lane;
    if (ti < valid) {
      Track const t = load_staged_track(tracks, track_lane);
      if (kCoreas && oi < ev.observer_count[0]) {
        ObserverCache const& o = observers[0][observer_lane];
        GlobalSink sink;
        for (int r = 0; r < 3; ++r) {
          sink.row[r] = kFixed ? ev.fixed[0] + r * ev.total_bins[0] + o.offset : nullptr;
          sink.frow[r] = kFixed ? nullptr : ev.floating[0] + r * ev.total_bins[0] + o.offset;
        }
        coreas_pair<kFixed, Amp, GlobalSink, false, true>(t, ev.propagation, o, sink, c);
      }
      if (kZhs && oi < ev.observer_count[1]) {
        ObserverCache const& o = observers[1][observer_lane];
        GlobalSink sink;
        for (int r = 0; r < 3; ++r) {
          sink.row[r] = kFixed ? ev.fixed[1] + r * ev.total_bins[1] + o.offset : nullptr;
          sink.frow[r] = kFixed ? nullptr : ev.floating[1] + r * ev.total_bins[1] + o.offset;
        }
        zhs_pair<kFixed, Amp>(t, ev.propagation, o, sink, c);
      }
    }
  }
  flush_counts(c, ev.counters);
}

// ---------------------------------------------------------------- windowed
// Threads of a CTA of the ZHS kernels that stage: of one pass (floating traces, the
// no-allocation entry point, launches past the two-pass storage cap) and of the last
// of two (items handed back: refined tracks, long traces, items near the fixed-point
// limit).  Their drain's live state needs more registers than their track loop, which
// gains from the warps.  us, FP64 at 384 / 480 threads: 262144 x 24 floating 519 / 478,
// refined twice 1453 / 1259, handed back in 24000 bins 927 / 776 but 60000 x 16 refined
// fourfold 586 / 745 (CoREAS included); mixed at 768 / 640 / 512: floating 329 / 339 /
// 343, handed back in 24000 bins 788 / 731 / 696, 60000 x 160 refined twice 3804 / 3416 /
// 3165.  480 threads' FP64 staging leaves room for 8202 bins; a longer window takes 384.
constexpr int kZhsThreadsFloat = 768;
constexpr int kZhsHandedThreadsFloat = 512;
constexpr int kZhsThreadsDouble = 480;
constexpr int kZhsHandedThreadsDouble = 384;
// Two passes (fixed point): the first, whose track loop is a function of its own,
// runs larger CTAs.  FP32 1024 threads (1e7 x 160 workload: 23.0 ms, 24.0 at 896),
// FP64 640.
constexpr int kZhsLoopThreadsFloat = 1024;
constexpr int kZhsLoopThreadsDouble = 640;
// kPass: 0 one pass; of a two-pass launch 1 the first, 3 the handed-back items
// in full (as one pass).
template <class Amp, int kPass = 0>
constexpr int zhs_threads_max() {
  return kPass == 1 ? (sizeof(Amp) == sizeof(float) ? kZhsLoopThreadsFloat : kZhsLoopThreadsDouble)
         : kPass == 3 ? (sizeof(Amp) == sizeof(float) ? kZhsHandedThreadsFloat : kZhsHandedThreadsDouble)
                      : (sizeof(Amp) == sizeof(float) ? kZhsThreadsFloat : kZhsThreadsDouble);
}
// Dynamic shared memory of a CTA (227 KB less the static part and a kilobyte's room).
constexpr size_t kSharedBytes = 227u * 1024u - 1024u;
// Dynamic shared memory of a launch: the window and, for a ZHS kernel that stages, 32
// staging slots a warp of its `block` threads.
template <class Amp>
constexpr size_t windowed_smem_bytes(uint32_t window, int algorithm, int pass, int block) {
  return static_cast<size_t>(window) * 3 * sizeof(unsigned long long) +
         (algorithm == 1 && pass != 1 ? static_cast<size_t>(block) * sizeof(StagedSegment<Amp>) : 0);
}
// The ZHS block for a team of `threads` and a window: the team when it is smaller than
// the default team, else the largest block of the amplitude type and pass whose
// staging fits beside the window.
template <class Amp, int kPass = 0>
constexpr int zhs_block(int threads, uint32_t window) {
  int most = zhs_threads_max<Amp, kPass>();
  if (windowed_smem_bytes<Amp>(window, 1, kPass, most) > kSharedBytes && most == kZhsThreadsDouble)
    most = kZhsHandedThreadsDouble;
  return threads < kWindowThreads && threads < most ? threads : most;
}
// CoREAS in mixed precision and fixed point: ms of the 1e7 x 160 workload at 640 /
// 768 / 896 / 1024 threads 26.4 / 24.3 / 23.9 / 22.5, in ice (5e6 x 64) 5.1 / 4.4 /
// 4.2 / 3.9.  Where each endpoint looks its source terms up (no shared
// destination row) 1024 threads spill the loop.
constexpr int kCoreasLeanThreads = 1024, kCoreasLeanLookupThreads = 768;
template <bool kFixed, class Amp, bool kPre>
constexpr int coreas_threads_max() {
  return kFixed && sizeof(Amp) == sizeof(float) ? (kPre ? kCoreasLeanThreads : kCoreasLeanLookupThreads)
                                                : kWindowThreads;
}
// The CoREAS block for a team of `threads`, by the same rule.
template <bool kFixed, class Amp, bool kPre>
constexpr int coreas_block(int threads) {
  return threads < kWindowThreads ? threads : coreas_threads_max<kFixed, Amp, kPre>();
}
static_assert(windowed_smem_bytes<double>(kPartialWindowBins, 1, 0, kZhsThreadsDouble) <= kSharedBytes &&
                  windowed_smem_bytes<float>(kPartialWindowBins, 0, 0, 0) + 2048 <= 196u * 1024u,
              "the window of longer traces");
// The staging that every window leaves room for.
constexpr size_t kStagingBytes = kZhsThreadsFloat * sizeof(StagedSegment<float>) >
                                         kZhsHandedThreadsDouble * sizeof(StagedSegment<double>)
                                     ? kZhsThreadsFloat * sizeof(StagedSegment<float>)
                                     : kZhsHandedThreadsDouble * sizeof(StagedSegment<double>);

__device__ __forceinline__ uint32_t find_event(EventPlan const* events, uint32_t n, uint64_t item) {
  uint32_t lo = 0, hi = n;  // last event with first_item <= item
  while (hi - lo > 1) {
    uint32_t const mid = (lo + hi) >> 1;
    if (events[mid].first_item <= item)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// The step of a divided track's sequential additions (RadioProjection.inl:505-512).
struct Steps {
  double x, y, z, t;
};
__device__ __forceinline__ Steps subtrack_steps(Track const& t, double divisor, int refinement) {
  Steps r{t.ex - t.sx, t.ey - t.sy, t.ez - t.sz, t.te - t.ts};
  if (divisor != 1. || refinement > 1) {  // x / 1 == x exactly: undivided tracks skip the divisions
    r.x = r.x / divisor;
    r.y = r.y / divisor;
    r.z = r.z / divisor;
    r.t = r.t / divisor;
  }
  if (refinement > 1) {
    double const rd = static_cast<double>(refinement);
    r.x = r.x / rd;
    r.y = r.y / rd;
    r.z = r.z / rd;
    r.t = r.t / rd;
  }
  return r;
}

// Segments from, from + stride, .. of a divided track (`from` alone for a stride of 0)
// evaluated exactly and deposited sample by sample, as zhs_drain does: what the
// filtered drain leaves undecided.
template <class Amp>
__device__ __noinline__ Counts zhs_exact_segments(const double* __restrict__ tracks, uint64_t row, unsigned from,
                                                  unsigned stride, Propagation const& p, ObserverCache const& o,
                                                  DifferenceSink sink) {
  Counts c;
  Track const t = load_track(tracks, row);
  Subdivision const d = subdivide(t, p, o);
  int const refinement = static_cast<int>(p.refinement);
  Steps const r = subtrack_steps(t, d.divisor, refinement);
  bool const subdivided = d.subtracks > 1 || refinement > 1;
  double x = t.sx, y = t.sy, z = t.sz, time = t.ts;
  long long const segments = static_cast<long long>(d.subtracks) * refinement;
  long long const stop = stride != 0u || segments <= from ? segments : static_cast<long long>(from) + 1;
  long long due = from;
#pragma unroll 1
  for (long long s = 0; s < stop; ++s) {
    double const nx = x + r.x, ny = y + r.y, nz = z + r.z, next = time + r.t;
    if (s == due) {
      due += stride;
      zhs_segment<true, true, Amp>(x, y, z, nx, ny, nz, time, next, t, p, o, sink, c, subdivided);
    }
    x = nx;
    y = ny;
    z = nz;
    time = next;
  }
  return c;
}

// Whether a track's `segments` may be evaluated by lean_segment below, which takes a
// segment's middle at start + (index + 1/2) (end - start) / divisor where the
// reference adds up s segments.  With u = 2^-53, the two differ by less than (s + 4) u
// of the largest coordinate and of the largest time, so the detection time by (s + 4) u
// (4 sqrt(3) |coordinate| fs / c + |time| fs), which has to stay below 2^-20 bins, a part
// of kBinGuard (s up to 60 at the filtered paths' limits, 300 in a shower of 100 km);
// at most kLeanSegments whatever the magnitudes, so that a warp's segments count in 32
// bits.
constexpr long long kLeanSegments = 4096;
__device__ __forceinline__ bool lean_divisible(Track const& t, double pack, long long segments, LeanObserver const& l) {
  double const furthest = fmax(fmax(fmax(fabs(t.sx), fabs(t.sy)), fmax(fabs(t.sz), fabs(t.ex))),
                               fmax(fabs(t.ey), fabs(t.ez)));
  double const bins = 7. * furthest * l.rate_over_c + fmax(fabs(t.ts), fabs(t.te)) * l.rate;
  return (segments <= kLeanSegments) & (static_cast<double>(segments + 4) * bins <= 0x1p33) &
         ((pack_flags(pack) & kTrackRegular & l.usable) != 0u);
}
// Whether the source terms at height z decide what the terms at the reference's
// own height, within `z_error` m of z, would.  In the table they are the same when
// no row lies within kBinGuard bins.  Past its ends (out of line: rare) they are
// linear in z: factor - 1 = (I - I_antenna) / rise with the rise in steps to the
// antenna's height, so an error e of the rise and one of I move the travel time by
// (dI + |factor - 1| e) / (|rise| - e) of `path_bins`; that and the index's change
// over half the segment have to stay below 2^-22 bins, which kBinGuard leaves over.
__device__ __noinline__ bool terms_decided_past_table(Propagation const& p, double height, double factor,
                                                      double z_error, double path_bins, double half_bins) {
  bool const above = height > 0.;
  double const steps = z_error * p.inv_step, antenna = s_observer.dest_height;
  double const rise = fabs(above ? height - antenna : antenna - fabs(height));
  double const rise_error = steps + 0x1p-50 * (fabs(height) + fabs(antenna));
  double const excess = fabs(factor - 1.) + 0x1p-52;
  double const integral_error = (above ? fabs(p.slope_i_upper) * z_error : fabs(p.slope_i_lower) * steps) +
                                0x1p-50 * (fabs(s_observer.dest_integral) + excess * rise);
  double const index_error = fabs(above ? p.slope_n_upper : p.slope_n_lower) * steps;
  return ((integral_error + excess * rise_error) * path_bins <
          (0x1p-22 - 4. * index_error * half_bins) * (rise - rise_error)) & (rise > rise_error);
}
__device__ __forceinline__ bool terms_decided(Propagation const& p, LeanObserver const& l, double factor, double z,
                                              double z_error, double path_bins, double half_bins) {
  if (p.homogeneous > 0.) return true;
  double const height = (z - p.min_height) * p.inv_step, guard = l.bin_guard_m * p.inv_step;
  int row;
  if (!((fabs(lean_nearest(height + 0.5, row)) > guard) & (fabs(height) > guard))) return false;
  if ((height > 0.) & (height + 0.5 < static_cast<double>(p.table_size - 1))) return true;
  return terms_decided_past_table(p, height, factor, z_error, path_bins, half_bins);
}
// A deferred track's division seen from the item's observer, out of line.  Refined
// tracks are all deferred, most of them undivided but for that: their Fraunhofer
// number is surely below 1.
struct Division {
  double divisor;
  int subtracks;
  bool lean;  // lean_divisible
};
__device__ __noinline__ Division divide_row(const double* __restrict__ tracks, uint64_t row, Propagation const& p) {
  int const refinement = static_cast<int>(p.refinement);
  Track const t = load_track(tracks, row);
  Subdivision d{1., 1};
  if (refinement == 1 || !surely_one_segment(t, s_observer)) d = subdivide(t, p, s_observer);
  double const pack = __ldg(track_ref(tracks, row) + kPack / 2 * kTrackTile).y;
  return {d.divisor, d.subtracks, lean_divisible(t, pack, static_cast<long long>(d.subtracks) * refinement, s_lean)};
}

// Segment `index` of a divided track (lean_divisible) by the filtered arithmetic,
// staged.  Both drains evaluate a segment by this function first.  False when a
// guard cannot decide.
__device__ __forceinline__ bool lean_segment(double2 const* __restrict__ r, unsigned index, bool subdivided,
                                             double fraction, Propagation const& p, LeanObserver const& l,
                                             StagedSegment<float>& seg) {
  constexpr unsigned T = kTrackTile;
  double2 const ca = __ldg(r), cb = __ldg(r + T), cc = __ldg(r + 2 * T), ct = __ldg(r + 3 * T);
  double2 const cd = __ldg(r + 4 * T), ce = __ldg(r + 5 * T);
  double const at = (static_cast<double>(index) + 0.5) * fraction;
  double const z = fma(cc.y - cb.x, at, cb.x), duration = ct.y - ct.x;
  double const half_bins = duration * fraction * l.half_rate;
  SourceTerms const st = source_terms(p, destination_of(s_observer), z);
  LeanPoint const m = lean_point(l, fma(cb.y - ca.x, at, ca.x), fma(cc.x - ca.y, at, ca.y), z,
                                 fma(duration, at, ct.x), cd.x, cd.y, ce.x, st.factor, st.n_src);
  bool cut;
  return zhs_lean(m, half_bins, pack_constant(ce.y) * l.scale, cd.x, cd.y, ce.x, l, subdivided, seg, cut) &
         lean_terms(st) & (m.dist * l.rate_over_c >= 4. * half_bins) &
         terms_decided(p, l, st.factor, z, 0x1p-46 * (fabs(cb.x) + fabs(cc.y)), m.dist * l.rate_over_c, half_bins);
}

// Deferred ZHS pairs in mixed precision and fixed point, the whole trace in the
// window: the warp's pairs (a lane each, below `count`) are divided exactly,
// then their segments are dealt out to the lanes in turn -- lane j of a step
// takes segment base + j of the flattened list, its owner found by shuffles --
// and each lane evaluates and deposits its segment on its own by lean_segment.
// Longer divisions, irregular tracks and segments that a guard cannot decide are
// evaluated exactly, the tracks by the whole warp, every 32nd segment a lane (each lane adds up the
// points in between: 128 additions where a segment is 900 operations; by its own lane
// alone 262144 tracks x 24 antennas refined 64 fold took 41.6 ms in 8192 bins).
// Little is held per lane (a row, an index, one FP64 number), so the function fits
// the registers of the track loop's kernel: the pair-per-lane drain it replaces there
// spilled 1700 words a pair at 64 registers.
__device__ __noinline__ Counts zhs_drain_lean(const double* __restrict__ tracks, uint64_t begin, unsigned const* list,
                                              unsigned count, Propagation const& p, unsigned long long* win,
                                              uint32_t width) {
  Tally c;
  Counts rare;  // counts of the exact evaluations, and the subtracks
  unsigned const lane = threadIdx.x & 31u;
  uint64_t row = 0;
  double fraction = 1.;
  unsigned mine = 0;
  bool exact = false;
  if (lane < count) {
    row = begin + list[lane];
    int const refinement = static_cast<int>(p.refinement);
    Division const d = divide_row(tracks, row, p);
    // both products as the reference forms them (RadioProjection.inl:503, :527)
    rare.subtracks = static_cast<unsigned long long>(static_cast<long long>(d.subtracks));
    if (refinement > 1)
      rare.subtracks += static_cast<unsigned long long>(static_cast<long long>(d.subtracks * (refinement - 1)));
    fraction = 1. / (d.divisor * static_cast<double>(refinement));
    exact = !d.lean;
    if (d.lean && d.subtracks > 0) mine = static_cast<unsigned>(d.subtracks * refinement);
  }
  unsigned incl = mine;
#pragma unroll
  for (unsigned d = 1; d < 32u; d <<= 1) {
    unsigned const v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  unsigned const total = __shfl_sync(0xffffffffu, incl, 31);
  for (unsigned base = 0; base < total; base += 32u) {
    unsigned const j = base + lane;
    unsigned owner = 0;
#pragma unroll
    for (unsigned step = 16; step >= 1u; step >>= 1) {
      unsigned const v = __shfl_sync(0xffffffffu, incl, owner + step - 1u);
      if (v <= j) owner += step;
    }
    owner &= 31u;
    unsigned const index = j - __shfl_sync(0xffffffffu, incl - mine, owner);
    uint64_t const its_row = __shfl_sync(0xffffffffu, row, owner);
    double const its_fraction = __shfl_sync(0xffffffffu, fraction, owner);
    bool const subdivided = __shfl_sync(0xffffffffu, mine, owner) > 1u;
    bool deposited = true;
    if (j < total) {
      LeanObserver const l = copy_words(s_lean);
      StagedSegment<float> seg;
      deposited = lean_segment(track_ref(tracks, its_row), index, subdivided, its_fraction, p, l, seg) &&
                  account_staged(seg, l, c);
      if (deposited) deposit_differences(seg, l, win, width);
    }
    if (__any_sync(0xffffffffu, !deposited) && !deposited)
      add_counts(rare, zhs_exact_segments<float>(tracks, its_row, index, 0u, p, s_observer,
                                                 DifferenceSink{win, width}));
  }
  for (unsigned left = __ballot_sync(0xffffffffu, exact); left != 0u; left &= left - 1u)
    add_counts(rare, zhs_exact_segments<float>(tracks, __shfl_sync(0xffffffffu, row, __ffs(static_cast<int>(left)) - 1),
                                               lane, 32u, p, s_observer, DifferenceSink{win, width}));
  add_counts(rare, counts_of(c));
  return rare;
}

// Deferred ZHS pairs of the windowed kernel, drained by the whole warp
// (accumulate_zhs, RadioProjection.inl:483-529).  Lanes below `count` take
// one deferred pair each and evaluate its Fraunhofer number and subdivision
// exactly; the warp then steps through segment index s = 0, 1, ...: every lane
// whose pair has a segment s forms its endpoints by the reference's
// sequential additions, stages it (FP64: exactly; mixed precision: by the filtered
// arithmetic), and the warp deposits the staged samples together.  A segment that
// cannot be staged is evaluated exactly and deposited on its own lane.  In mixed
// precision and fixed point these are zhs_drain_lean's steps (lean_segment, else
// zhs_segment), so that a pair's FP32 values are the same bits whether its item runs
// with checked adds or without.  Every lane of the warp calls it.
template <bool kFixed, bool kDifferences, class Amp, class Sink>
__device__ __noinline__ Counts zhs_drain(const double* __restrict__ tracks, uint64_t begin,
                                         unsigned const* list, unsigned count,
                                         Propagation const& p, ObserverCache const& o, LeanObserver const& l, Sink sink,
                                         StagedSegment<Amp>* staging) {
  Counts c;
  unsigned const lane = threadIdx.x & 31u;
  uint64_t row = 0;
  long long segments = 0;
  bool subdivided = false;
  double p1x = 0., p1y = 0., p1z = 0., t1 = 0., rx = 0., ry = 0., rz = 0., rt = 0.;
  double fraction = 1.;  // mixed precision, fixed point: of the track, a segment
  bool lean = false;     // and whether lean_segment may evaluate it
  if (lane < count) {
    row = begin + list[lane];
    Track const t = load_track(tracks, row);
    Subdivision const d = subdivide(t, p, o);
    int const refinement = static_cast<int>(p.refinement);
    c.subtracks += static_cast<unsigned long long>(static_cast<long long>(d.subtracks));
    if (refinement > 1)
      c.subtracks += static_cast<unsigned long long>(static_cast<long long>(d.subtracks * (refinement - 1)));
    subdivided = d.subtracks > 1 || refinement > 1;
    Steps const step = subtrack_steps(t, d.divisor, refinement);
    rx = step.x;
    ry = step.y;
    rz = step.z;
    rt = step.t;
    segments = static_cast<long long>(d.subtracks) * refinement;
    if constexpr (kFixed && sizeof(Amp) == sizeof(float)) {
      fraction = 1. / (d.divisor * static_cast<double>(refinement));
      lean = lean_divisible(t, __ldg(track_ref(tracks, row) + kPack / 2 * kTrackTile).y, segments, l);
    }
    p1x = t.sx;
    p1y = t.sy;
    p1z = t.sz;
    t1 = t.ts;
  }
#pragma unroll 1
  for (long long s = 0; __any_sync(0xffffffffu, s < segments); ++s) {
    StagedSegment<Amp> seg;
    seg.count = 0u;
    seg.flags = 0u;
    if (s < segments) {
      // velocity and charge constant read again each step (L1): fewer
      // registers held across the warp's steps
      double2 const* r = track_ref(tracks, row);
      asm volatile("" : "+l"(r));
      double2 const e = __ldg(r + 4 * kTrackTile), f = __ldg(r + 5 * kTrackTile);
      double const p2x = p1x + rx, p2y = p1y + ry, p2z = p1z + rz, t2 = t1 + rt;
      Track t;
      t.bx = e.x;
      t.by = e.y;
      t.bz = f.x;
      t.constant = __ldg(r + kConst / 2 * kTrackTile).y;
      double const mx = (p1x + p2x) * 0.5, my = (p1y + p2y) * 0.5, mz = (p1z + p2z) * 0.5, mt = (t1 + t2) * 0.5;
      bool staged = false;
      if constexpr (sizeof(Amp) == sizeof(float)) {
        if constexpr (kFixed) {
          staged = lean && lean_segment(r, static_cast<unsigned>(s), subdivided, fraction, p, l, seg);
        } else {  // the sums' order decides the last bits anyway: at the sequential points
          SourceTerms const st = source_terms(p, destination_of(o), mz);
          LeanPoint const m = lean_point(l, mx, my, mz, mt, e.x, e.y, f.x, st.factor, st.n_src);
          bool cut;
          staged = zhs_lean(m, (t2 - t1) * l.half_rate, pack_constant(f.y) * l.scale, e.x, e.y, f.x, l, subdivided, seg,
                            cut) &
                   ((pack_flags(f.y) & kTrackRegular & l.usable) != 0u) & lean_terms(st);
        }
      }
      if (!staged && !(kFixed && sizeof(Amp) == sizeof(float)))
        staged = zhs_stage<Amp>(mx, my, mz, t1, t2, mt, t, p, o, subdivided, seg);
      if (!staged) {
        seg.count = 0u;
        seg.flags = 0u;
        zhs_segment<kFixed, true, Amp>(p1x, p1y, p1z, p2x, p2y, p2z, t1, t2, t, p, o, sink,
                                              c, subdivided);
      }
      p1x = p2x;
      p1y = p2y;
      p1z = p2z;
      t1 = t2;
    }
    if constexpr (kDifferences) {
      // a segment whose values might not convert: sample by sample, checked
      if (!account_staged(seg, l, c))
        add_counts(c, deposit_samples(seg, o, sink));
      else
        deposit_differences(seg, l, sink.win, sink.width);
    } else {
      deposit_staged<kFixed>(staging, seg, o, sink, c);
    }
  }
  return c;
}

// A deferred CoREAS pair of the windowed kernel, loaded and evaluated exactly
// out of line (the caller passes the row, not the 112-byte track).  `hint`
// (kCoreasNearCone, as the track loop decided it, else 0): the pair takes the
// near-Cherenkov branch in the order of bit 0, evaluated here directly.
template <bool kFixed, class Amp, bool kPre, class Sink>
__device__ __noinline__ Counts coreas_drain_pair(const double* __restrict__ tracks, uint64_t row,
                                                 unsigned hint, Propagation const& p,
                                                 ObserverCache const& o, Sink sink) {
  Counts c;
  double2 const* r = track_ref(tracks, row);
  if constexpr (kFixed && sizeof(Amp) == sizeof(float)) {
    Tally t;
    if ((hint & static_cast<unsigned>(kCoreasNearCone)) &&
        near_cone_lean<kPre>(r, (hint & 1u) != 0u, p, s_lean, sink, t))
      return counts_of(t);
  }
  constexpr unsigned T = kTrackTile;
  unsigned const flags = pack_flags(__ldg(r + kPack / 2 * T).y);
  Track const t = load_track(tracks, row);
  if (kPre) {
    // the near-cone midpoint's terms are the ZHS midpoint's (kTrackOneMid) or looked up
    double2 const m = __ldg(r + kFactorMid / 2 * T);
    SourceTerms const mid = (flags & kTrackOneMid) ? SourceTerms{m.x, m.y, 0.}
                                                   : source_terms(p, destination_of(o), (t.sz + t.ez) * 0.5);
    if (hint & static_cast<unsigned>(kCoreasNearCone))
      return coreas_near_cone<kFixed, Amp, true>(t, p, o, sink, (hint & 1u) != 0u, mid);
    double2 const s = __ldg(r + kFactorStart / 2 * T), e = __ldg(r + kFactorEnd / 2 * T);
    SourceTerms const pre[3] = {{s.x, s.y, dense_index(flags)}, {e.x, e.y, 0.}, mid};
    coreas_pair<kFixed, Amp, Sink, true>(t, p, o, sink, c, pre);
  } else {
    if (hint & static_cast<unsigned>(kCoreasNearCone))
      return coreas_near_cone<kFixed, Amp, false>(t, p, o, sink, (hint & 1u) != 0u, SourceTerms{});
    coreas_pair<kFixed, Amp>(t, p, o, sink, c);
  }
  return c;
}

// The precomputed source terms of a track's end points (with the start's n_dst
// as far as the path looks at it: above 1 or not).
__device__ __forceinline__ void load_endpoint_terms(const double* __restrict__ base, uint64_t i, SourceTerms& start,
                                                    SourceTerms& end) {
  double2 const* r = track_ref(base, i);
  constexpr unsigned T = kTrackTile;
  double2 const s = __ldg(r + kFactorStart / 2 * T), e = __ldg(r + kFactorEnd / 2 * T);
  start = SourceTerms{s.x, s.y, dense_index(pack_flags(__ldg(r + kPack / 2 * T).y))};
  end = SourceTerms{e.x, e.y, 0.};
}

// A deferred-list entry: the track's offset in the item and, for CoREAS, the
// track loop's decision in the top bits.
__device__ __forceinline__ unsigned deferred_entry(uint32_t offset, int code) {
  return offset | (code >= kCoreasNearCone ? static_cast<unsigned>(code) << kDeferredHintShift : 0u);
}

// Appends a warp's deferred pairs to its CTA's list: `entry` of the lanes with
// `deferred` set, one atomic on the shared counter.
__device__ __forceinline__ void push_deferred(bool deferred, unsigned entry) {
  unsigned const ballot = __ballot_sync(0xffffffffu, deferred);
  if (!ballot) return;
  unsigned const lane = threadIdx.x & 31u;
  unsigned slot = 0;
  if (lane == 0) slot = atomicAdd(&s_deferred_total, static_cast<unsigned>(__popc(ballot)));
  slot = __shfl_sync(0xffffffffu, slot, 0);
  if (deferred) s_deferred_list[slot + __popc(ballot & ((1u << lane) - 1u))] = entry;
}

// The track loops run out of line, each a function of its own: what the kernel
// holds across an item (the plan, the calls of the drain and the flush) then
// takes no registers from the loop, whose speed turns on its register
// allocation (inlined beside them, the loops of the 1e7 x 160 workload ran 31.1
// (CoREAS) and 42.7 ms (ZHS) where they run 26.8 and 34.3 as functions).  `count` tracks from `begin`, a
// thread each; a thread's track advances by whole tiles, so its columns'
// address is one running pointer.  Deferred pairs go to `list`.

// CoREAS in mixed precision and fixed point.
template <bool kPre, bool kUnchecked>
__device__ __noinline__ Counts coreas_lean_loop(const double* __restrict__ tracks, uint64_t begin, uint32_t count,
                                                Propagation const& p, WindowSink sink) {
  Tally c;
  double2 const* r = track_ref(tracks, begin + threadIdx.x);
  uint32_t const step = blockDim.x / kTrackTile * (kTrackTile * kTrackColumns);
  for (uint32_t base = 0; base < count; base += blockDim.x, r += step) {
    uint32_t const k = base + threadIdx.x;
    int code = kCoreasDeposited;
    if (k < count) code = coreas_lean<kPre, kUnchecked>(r, p, copy_words(s_lean), sink, c);
    push_deferred(code != kCoreasDeposited, deferred_entry(k, code));
  }
  return counts_of(c);
}

// CoREAS in FP64 or with floating traces.
template <bool kFixed, bool kPre, class Amp>
__device__ __noinline__ Counts coreas_loop(const double* __restrict__ tracks, uint64_t begin, uint32_t count,
                                           Propagation const& p, WindowSink sink) {
  Counts c;
  for (uint32_t base = 0; base < count; base += blockDim.x) {
    uint32_t const k = base + threadIdx.x;
    int code = kCoreasDeposited;
    if (k < count) {
      Track const t = load_track(tracks, begin + k);
      SourceTerms start{}, end{};
      if (kPre) load_endpoint_terms(tracks, begin + k, start, end);
      code = coreas_common<kFixed, kPre, Amp>(t, p, s_observer, sink, c, start, end);
    }
    push_deferred(code != kCoreasDeposited, deferred_entry(k, code));
  }
  return c;
}

// ZHS in fixed point with the whole trace in the window: deposited lane by lane
// as differences.
template <bool kPre, bool kMayRefine, class Amp>
__device__ __noinline__ Counts zhs_difference_loop(const double* __restrict__ tracks, uint64_t begin,
                                                   uint32_t count, Propagation const& p, unsigned long long* win,
                                                   uint32_t width) {
  Tally c;
  double2 const* r = track_ref(tracks, begin + threadIdx.x);
  uint32_t const step = blockDim.x / kTrackTile * (kTrackTile * kTrackColumns);
  for (uint32_t base = 0; base < count; base += blockDim.x, r += step) {
    uint32_t const k = base + threadIdx.x;
    bool deferred = kMayRefine && k < count && p.refinement != 1u;  // refined: the drain divides it
    LeanObserver const l = copy_words(s_lean);
    if constexpr (sizeof(Amp) == sizeof(float)) {
      if (k < count && !deferred) {
        ZhsPoint const z = zhs_point<kPre>(r, p, l);
        deferred = !(z.one && zhs_lean_differences(z.m, z.half_bins, z.constant, z.bx, z.by, z.bz, l, win, c));
      }
    } else if (k < count && !deferred) {
      ZhsPoint const z = zhs_point<kPre>(r, p, l);
      deferred = !z.one;
      if (z.one) {
        constexpr unsigned T = kTrackTile;
        ObserverCache const o = copy_words(s_observer);
        double2 const cm = __ldg(r + 9 * T), cn = __ldg(r + 10 * T), ct = __ldg(r + 3 * T);
        deferred = !zhs_exact_differences(propagate_with<true>(z.terms, o, cm.x, cm.y, cn.x), ct.x,
                                          ct.x + (ct.y - ct.x), cn.y, z.bx, z.by, z.bz,
                                          __ldg(r + kConst / 2 * T).y, o, l, win, c);
      }
    }
    push_deferred(deferred, k);
  }
  return counts_of(c);
}

// ZHS with the segments staged for the warp (floating traces, checked runs).
template <bool kFixed, bool kPre, class Amp>
__device__ __noinline__ Counts zhs_staged_loop(const double* __restrict__ tracks, uint64_t begin, uint32_t count,
                                               Propagation const& p, WindowSink sink,
                                               StagedSegment<Amp>* staging) {
  Counts c;
  double2 const* r = track_ref(tracks, begin + threadIdx.x);
  uint32_t const step = blockDim.x / kTrackTile * (kTrackTile * kTrackColumns);
  for (uint32_t base = 0; base < count; base += blockDim.x, r += step) {
    uint32_t const k = base + threadIdx.x;
    bool deferred = false;
    StagedSegment<Amp> seg;
    seg.count = 0u;
    seg.flags = 0u;
    if (k < count) deferred = p.refinement != 1u || !zhs_common<kFixed, kPre, Amp>(r, p, s_lean, seg);
    deposit_staged<kFixed>(staging, seg, s_observer, sink, c);
    push_deferred(deferred, k);
  }
  return c;
}

// No thread of the CTA can count 2^32 samples in an item of `count` tracks.
__device__ __forceinline__ bool tally_fits(uint64_t count, uint32_t width) {
  return (count / blockDim.x + 1u) * width < 0xffffffffull;
}

// Notes an item for the second pass (kPass 3); one thread of the CTA writes it.
__device__ __forceinline__ void hand_back(WorkPlan const& plan, uint64_t item) {
  if (threadIdx.x != 0) return;
  plan.item_state[atomicAdd(plan.drain_next_item, 1u)] = {item};
  if (plan.handbacks) atomicAdd(plan.handbacks, 1ull);
}

// Zeroes 3 * width words of the window.  Every thread of the CTA calls it.
__device__ __forceinline__ void zero_window(unsigned long long* win, uint32_t width) {
  uint32_t const words = 3u * width;
  for (uint32_t j = threadIdx.x; j < words / 2u; j += blockDim.x)
    reinterpret_cast<ulonglong2*>(win)[j] = make_ulonglong2(0ull, 0ull);
  if (threadIdx.x == 0 && (words & 1u)) win[words - 1u] = 0ull;
}

// Adds the window's non-zero bins to the observer's trace rows with checked
// global atomics; returns this thread's overflows.  A thread issues the adds
// of four bins' three components before it looks at what they returned: one
// add at a time waits for the L2 at every bin (24576 adds an item of 8192
// bins).  Out of line, so that its registers do not count in the track loops.
__device__ __noinline__ unsigned flush_window(unsigned long long const* win, uint32_t width,
                                              unsigned long long* row0, unsigned long long* row1,
                                              unsigned long long* row2) {
  constexpr uint32_t kDepth = 4;
  unsigned overflows = 0;
  for (uint32_t base = threadIdx.x; base < width; base += kDepth * blockDim.x) {
    unsigned long long v[kDepth][3], before[kDepth][3];
#pragma unroll
    for (uint32_t d = 0; d < kDepth; ++d) {
      uint32_t const j = base + d * blockDim.x;
#pragma unroll
      for (uint32_t row = 0; row < 3; ++row) v[d][row] = j < width ? win[3u * j + row] : 0ull;
    }
#pragma unroll
    for (uint32_t d = 0; d < kDepth; ++d) {
      uint32_t const j = base + d * blockDim.x;
      before[d][0] = v[d][0] ? atomicAdd(row0 + j, v[d][0]) : 0ull;
      before[d][1] = v[d][1] ? atomicAdd(row1 + j, v[d][1]) : 0ull;
      before[d][2] = v[d][2] ? atomicAdd(row2 + j, v[d][2]) : 0ull;
    }
#pragma unroll
    for (uint32_t d = 0; d < kDepth; ++d)
#pragma unroll
      for (uint32_t row = 0; row < 3; ++row)
        overflows += checked(before[d][row], static_cast<long long>(v[d][row])) ? 0u : 1u;
  }
  return overflows;
}

__device__ __noinline__ void flush_window_floating(double const* win, uint32_t width, double* row0, double* row1,
                                                   double* row2) {
  for (uint32_t j = threadIdx.x; j < width; j += blockDim.x) {
    double const x = win[3u * j], y = win[3u * j + 1u], z = win[3u * j + 2u];
    if (x != 0.) atomicAdd(row0 + j, x);
    if (y != 0.) atomicAdd(row1 + j, y);
    if (z != 0.) atomicAdd(row2 + j, z);
  }
}

// kPass 0: every item in one pass.  Two passes (fixed-point ZHS): kPass 1
// projects an item's tracks and then its deferred pairs with unchecked window
// adds, all as differences (deposit_differences), and hands back, unflushed and
// uncounted, the items it cannot: traces longer than the window, refined
// tracks (each pair is divided) and items whose window bound does not hold;
// kPass 3 projects those in full, as kPass 0 does.  With the general path in a
// kernel of its own, the first pass holds nothing but the track loop and runs
// it without spills in larger CTAs.
template <bool kFixed, class Amp, int kAlgorithm, bool kPre, int kPass = 0>
__global__ void __launch_bounds__(kAlgorithm == 1 ? zhs_threads_max<Amp, kPass>() : coreas_threads_max<kFixed, Amp, kPre>(), 1)
    windowed_kernel(const __grid_constant__ WorkPlan plan) {
  static_assert(kPass == 0 || (kFixed && kAlgorithm == 1), "two passes: fixed-point ZHS");
  extern __shared__ __align__(16) unsigned long long window[];
  __shared__ unsigned long long item_shared;
  __shared__ float window_bound;
  // this CTA's list of the deferred pairs of its current item
  if (threadIdx.x == 0)
    s_deferred_list = (kPass == 3 ? plan.drain_deferred : plan.deferred) +
                      static_cast<size_t>(blockIdx.x) * plan.deferred_stride;
  Counts c;
  for (;;) {
    // the next item: of the plan, or of those that the first pass handed back (most
    // launches have none: the last pass then ends without a turn taken)
    unsigned const handed = kPass == 3 ? plan.drain_next_item[0] : 0u;
    if (kPass == 3 && handed == 0u) break;
    __syncthreads();
    if (threadIdx.x == 0) item_shared = atomicAdd(kPass == 3 ? plan.drain_next_item + 1 : plan.next_item, 1u);
    __syncthreads();
    uint64_t item = item_shared;
    if (item >= (kPass == 3 ? handed : plan.total_items)) break;
    if constexpr (kPass == 3) item = plan.item_state[item].item;
    EventPlan const& ev = plan.events[find_event(plan.events, plan.event_count, item)];
    constexpr int algorithm = kAlgorithm;
    uint64_t const local = item - ev.first_item;
    uint32_t const per_chunk = ev.observer_count[algorithm];
    uint64_t const slice_chunk = local / per_chunk;
    uint32_t const oi = static_cast<uint32_t>(local - slice_chunk * per_chunk);
    uint64_t const valid = *ev.valid_tracks;
    uint64_t const track_count = valid < ev.last_track ? valid : ev.last_track;
    uint64_t const begin = ev.first_track + slice_chunk * ev.chunk_size;
    if (begin >= track_count) continue;
    uint64_t const end = begin + ev.chunk_size < track_count ? begin + ev.chunk_size : track_count;
    uint64_t const bins = ev.observers[algorithm][oi].bins;
    uint32_t const width = static_cast<uint32_t>(bins < ev.window ? bins : ev.window);
    if (kPass == 1 && (bins > width || ev.propagation.refinement != 1u || !tally_fits(end - begin, width))) {
      hand_back(plan, item);
      continue;
    }
    if (threadIdx.x == 0) {
      s_observer = ev.observers[algorithm][oi];
      if (kAlgorithm == 1 || sizeof(Amp) == sizeof(float)) make_lean_observer<kAlgorithm>(s_observer, s_lean);
    }

    // zero the window (3 words for each of width bins); the barrier also publishes the observer
    zero_window(window, width);
    if (threadIdx.x == 0) window_bound = 0.f;
    __syncthreads();

    constexpr bool kFilter = sizeof(Amp) == sizeof(float);  // mixed precision
    // Deferred pairs (track offsets in the chunk: CoREAS pairs for the
    // near-Cherenkov branch or an exact evaluation, ZHS pairs with subdivided
    // tracks or an exact evaluation) leave the common path, so rare paths do
    // not hold up the other lanes: they go to the CTA's list in global memory
    // and all warps drain it, 32 pairs at a time, after the item's tracks.
    // per-warp staging slots of the ZHS kernel's cooperative deposit
    StagedSegment<Amp>* const staging =
        reinterpret_cast<StagedSegment<Amp>*>(window + 3 * static_cast<size_t>(plan.window)) +
        (threadIdx.x >> 5) * 32u;
    unsigned const lane = threadIdx.x & 31u;
    uint32_t const count = static_cast<uint32_t>(end - begin);
    bool handed_back = false, whole = false;  // whole: the window's adds were unchecked
    // The trace rows' addresses are formed again wherever they are used
    // (`fresh` hides that they are the same), not held across the track loop.
    auto make_sink = [&](bool unchecked) {
      uint64_t offset = s_observer.offset;
      asm volatile("" : "+l"(offset));  // fresh
      WindowSink k;
      k.win = window;
      k.fwin = reinterpret_cast<double*>(window);
      k.width = width;
      k.unchecked = unchecked;
      for (int row = 0; row < 3; ++row) {
        uint64_t const at = row * ev.total_bins[algorithm] + offset;
        k.row[row] = kFixed ? ev.fixed[algorithm] + at : nullptr;
        k.frow[row] = kFixed ? nullptr : ev.floating[algorithm] + at;
      }
      return k;
    };
    // Fixed point, whole trace in the window: the window takes unchecked
    // adds, and `c.mag` bounds the sum of |increments| of this thread.  If the
    // block's bound stays below 2^61, no partial sum of any bin can have left
    // the int64 range in any order, so no add overflowed; else the item is
    // run again with checked adds (kPass 1: handed back).  An FP32 sum of n
    // terms is off by a factor below 1 + n 2^-24, so a thread's sum counts only
    // while the thread made fewer than 2^22 adds (factor below 1 + 2^-2); a
    // thread with more (its deposits since the attempt began: contributions
    // plus failed conversions, an upper bound of its window adds) sends the
    // item to the checked run.  Bins past the window and the flush below are
    // always checked.
    for (int attempt = 0;; ++attempt) {
      if (attempt > 0) {
        zero_window(window, width);
        __syncthreads();
      }
      bool const unchecked = kFixed && attempt == 0 && bins <= width && (kAlgorithm == 0 || tally_fits(count, width));
      c = Counts{};
      if (threadIdx.x == 0) s_deferred_total = 0u;
      __syncthreads();
      Propagation const& p = ev.propagation;
      if constexpr (kAlgorithm == 0 && kFixed && kFilter) {
        c = unchecked ? coreas_lean_loop<kPre, true>(ev.tracks, begin, count, p, make_sink(true))
                      : coreas_lean_loop<kPre, false>(ev.tracks, begin, count, p, make_sink(false));
      } else if constexpr (kAlgorithm == 0) {
        c = coreas_loop<kFixed, kPre, Amp>(ev.tracks, begin, count, p, make_sink(unchecked));
      } else if (kFixed && (kPass == 1 || unchecked)) {
        c = zhs_difference_loop<kPre, kPass != 1, Amp>(ev.tracks, begin, count, p, window, width);
      } else if constexpr (kPass != 1) {
        c = zhs_staged_loop<kFixed, kPre, Amp>(ev.tracks, begin, count, p, make_sink(false), staging);
      }
      __syncthreads();
      unsigned const n = s_deferred_total;  // at most end - begin <= deferred_stride
      // one subtrack for each pair that the track loop deposited; the drain counts the others'
      if (kAlgorithm == 1 && threadIdx.x == 0) c.subtracks += count - n;
      for (unsigned from = (threadIdx.x >> 5) * 32u; from < n; from += (blockDim.x >> 5) * 32u) {
        unsigned const left = n - from < 32u ? n - from : 32u;
        Counts d;
        if constexpr (kAlgorithm == 1) {
          if (kFixed && (kPass == 1 || unchecked)) {
            if constexpr (sizeof(Amp) == sizeof(float))
              d = zhs_drain_lean(ev.tracks, begin, s_deferred_list + from, left, p, window, width);
            else
              d = zhs_drain<kFixed, true, Amp>(ev.tracks, begin, s_deferred_list + from, left, p, s_observer, s_lean,
                                               DifferenceSink{window, width}, staging);
          }
          else if constexpr (kPass != 1)
            d = zhs_drain<kFixed, false, Amp>(ev.tracks, begin, s_deferred_list + from, left, p, s_observer, s_lean,
                                              make_sink(false), staging);
        } else if (lane < left) {
          unsigned const entry = s_deferred_list[from + lane];
          d = coreas_drain_pair<kFixed, Amp, kPre>(ev.tracks, begin + (entry & kDeferredOffsetMask),
                                                   entry >> kDeferredHintShift, p, s_observer,
                                                   make_sink(unchecked));
        }
        add_counts(c, d);
        __syncwarp();
      }
      __syncthreads();
      if (!unchecked) break;
      whole = true;
      unsigned long long const adds = c.coreas + c.zhs + c.overflows;
      double const mine = adds < (1ull << 22) ? static_cast<double>(c.mag) : static_cast<double>(INFINITY);
      float const thread_bound = static_cast<float>(warp_sum(mine));
      if (lane == 0) atomicAdd(&window_bound, thread_bound);
      __syncthreads();
      float const block_bound = window_bound;
      __syncthreads();
      if (block_bound < 0x1p61f) break;
      whole = false;
      if (kPass == 1) {
        handed_back = true;
        break;
      }
      if (threadIdx.x == 0 && plan.reruns) atomicAdd(plan.reruns, 1ull);
    }
    if (kPass == 1 && handed_back) {
      hand_back(plan, item);
      continue;
    }
    if (kAlgorithm == 1 && kFixed && whole) difference_window(window, width);
    WindowSink const sink = make_sink(false);
    if (kFixed)
      c.overflows += flush_window(window, width, sink.row[0], sink.row[1], sink.row[2]);
    else
      flush_window_floating(sink.fwin, width, sink.frow[0], sink.frow[1], sink.frow[2]);
    flush_counts(c, ev.counters);
  }
}

// ---------------------------------------------------------------- decode
__global__ void decode_kernel(const long long* __restrict__ fixed, double* __restrict__ out,
                              uint64_t total_bins, const uint64_t* __restrict__ offsets,
                              const double* __restrict__ factors) {
  uint32_t const o = blockIdx.y;
  uint64_t const begin = offsets[o], end = offsets[o + 1];
  double const f = factors[o];
  for (uint64_t i = begin + static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < end;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    out[i] = static_cast<double>(fixed[i]) * f;
    out[total_bins + i] = static_cast<double>(fixed[total_bins + i]) * f;
    out[2 * total_bins + i] = static_cast<double>(fixed[2 * total_bins + i]) * f;
  }
}

// The output step on the device: CoREAS fields added as they are, ZHS
// potentials differentiated into fields E_i = -(A_{i+1} - A_i) fs at the bin
// midpoints (RadioProcess.inl:213-223; one sample fewer per observer), both
// added into `out` (the observer add of CorsikaOutputSink.inl:255-278).
// Values are the decoded traces: fixed x factor of the observer, or the FP64
// traces.  `out` rows are [X | Y | Z] of total_bins - observers (ZHS) or
// total_bins (CoREAS) values.
__global__ void output_kernel(const long long* __restrict__ fixed, const double* __restrict__ floating,
                              double* __restrict__ out, uint64_t total_bins,
                              const ObserverCache* __restrict__ observers, const double* __restrict__ factors,
                              uint32_t observer_count, int differentiate) {
  uint32_t const o = blockIdx.y;
  ObserverCache const& oc = observers[o];
  double const f = fixed ? factors[o] : 1.;
  uint64_t const bins = oc.bins;
  uint64_t const samples = differentiate ? (bins > 0 ? bins - 1 : 0) : bins;
  uint64_t const out_total = differentiate ? total_bins - observer_count : total_bins;
  uint64_t const out_offset = differentiate ? oc.offset - o : oc.offset;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < samples;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    for (int r = 0; r < 3; ++r) {
      uint64_t const j = r * total_bins + oc.offset + i;
      double const a = fixed ? static_cast<double>(fixed[j]) * f : floating[j];
      double value = a;
      if (differentiate) {
        double const b = fixed ? static_cast<double>(fixed[j + 1]) * f : floating[j + 1];
        value = -(b - a) * oc.sample_rate;
      }
      out[r * out_total + out_offset + i] += value;
    }
  }
}

template <bool kFixed, class Amp>
cudaError_t direct_dispatch(EventPlan const& ev, uint64_t bound, bool coreas, bool zhs,
                            cudaStream_t stream) {
  uint32_t const observers =
      ev.observer_count[0] > ev.observer_count[1] ? ev.observer_count[0] : ev.observer_count[1];
  uint64_t const pairs = bound * observers;
  if (pairs == 0) return cudaSuccess;
  int device = 0, sms = 148;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  uint64_t blocks = (pairs + 255) / 256;
  uint64_t const cap = static_cast<uint64_t>(sms) * 16;
  if (blocks > cap) blocks = cap;
  unsigned const grid = static_cast<unsigned>(blocks);
  if (coreas && zhs)
    direct_kernel<kFixed, Amp, true, true><<<grid, 256, 0, stream>>>(ev);
  else if (coreas)
    direct_kernel<kFixed, Amp, true, false><<<grid, 256, 0, stream>>>(ev);
  else if (zhs)
    direct_kernel<kFixed, Amp, false, true><<<grid, 256, 0, stream>>>(ev);
  return cudaGetLastError();
}

template <bool kFixed, class Amp>
cudaError_t tiled_dispatch(EventPlan const& ev, uint64_t bound, bool coreas, bool zhs, cudaStream_t stream) {
  uint32_t const observers =
      ev.observer_count[0] > ev.observer_count[1] ? ev.observer_count[0] : ev.observer_count[1];
  if (bound == 0 || observers == 0) return cudaSuccess;
  uint64_t const track_tiles = (bound + kTileTracks - 1) / kTileTracks;
  uint64_t const tiles = track_tiles * ((observers + kTileObservers - 1) / kTileObservers);
  int device = 0, sms = 148;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  uint64_t const cap = static_cast<uint64_t>(sms) * 64;
  unsigned const grid = static_cast<unsigned>(tiles < cap ? tiles : cap);
  if (coreas && zhs)
    tiled_kernel<kFixed, Amp, true, true><<<grid, kTileThreads, 0, stream>>>(ev, track_tiles);
  else if (coreas)
    tiled_kernel<kFixed, Amp, true, false><<<grid, kTileThreads, 0, stream>>>(ev, track_tiles);
  else if (zhs)
    tiled_kernel<kFixed, Amp, false, true><<<grid, kTileThreads, 0, stream>>>(ev, track_tiles);
  return cudaGetLastError();
}

// Every event of the plan carries precomputed source terms.
bool plan_precomputed(WorkPlan const& plan) {
  if (plan.event_count == 0) return false;
  for (uint32_t e = 0; e < plan.event_count; ++e)
    if (!plan.events[e].precomputed) return false;
  return true;
}

template <bool kFixed, class Amp, int kAlgorithm, bool kPre, int kPass = 0>
cudaError_t windowed_launch(WorkPlan const& plan, int ctas, int threads, cudaStream_t stream) {
  int const block =
      kAlgorithm == 1 ? zhs_block<Amp, kPass>(threads, plan.window) : coreas_block<kFixed, Amp, kPre>(threads);
  size_t const bytes = windowed_smem_bytes<Amp>(plan.window, kAlgorithm, kPass, block);
  cudaError_t err = cudaFuncSetAttribute(windowed_kernel<kFixed, Amp, kAlgorithm, kPre, kPass>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(bytes));
  if (err != cudaSuccess) return err;
  windowed_kernel<kFixed, Amp, kAlgorithm, kPre, kPass><<<ctas, block, bytes, stream>>>(plan);
  return cudaGetLastError();
}

// The passes of a two-pass fixed-point ZHS launch, one after the other on
// the stream; drain_next_item counts the items handed back and those taken up.
template <class Amp, bool kPre>
cudaError_t windowed_two_pass(WorkPlan const& plan, int ctas, int threads, cudaStream_t stream) {
  cudaError_t err = cudaMemsetAsync(plan.drain_next_item, 0, 2 * sizeof(unsigned), stream);
  if (err != cudaSuccess) return err;
  err = windowed_launch<true, Amp, 1, kPre, 1>(plan, ctas, threads, stream);
  if (err != cudaSuccess) return err;
  return windowed_launch<true, Amp, 1, kPre, 3>(plan, ctas, threads, stream);
}

template <bool kFixed, class Amp, int kAlgorithm>
cudaError_t windowed_dispatch_algorithm(WorkPlan const& plan, int ctas, int threads,
                                        cudaStream_t stream) {
  if (plan.deferred == nullptr || plan.deferred_stride < deferred_list_stride(plan))
    return cudaErrorInvalidValue;
  bool const pre = plan_precomputed(plan);
  if (plan.item_state != nullptr) {
    if constexpr (kFixed && kAlgorithm == 1) {
      if (plan.drain_deferred == nullptr || plan.drain_next_item == nullptr) return cudaErrorInvalidValue;
      return pre ? windowed_two_pass<Amp, true>(plan, ctas, threads, stream)
                 : windowed_two_pass<Amp, false>(plan, ctas, threads, stream);
    } else {
      return cudaErrorInvalidValue;
    }
  }
  return pre ? windowed_launch<kFixed, Amp, kAlgorithm, true>(plan, ctas, threads, stream)
             : windowed_launch<kFixed, Amp, kAlgorithm, false>(plan, ctas, threads, stream);
}

template <bool kFixed, class Amp>
cudaError_t windowed_dispatch(WorkPlan const& plan, int ctas, int threads, cudaStream_t stream) {
  return plan.algorithm == 0
             ? windowed_dispatch_algorithm<kFixed, Amp, 0>(plan, ctas, threads, stream)
             : windowed_dispatch_algorithm<kFixed, Amp, 1>(plan, ctas, threads, stream);
}

template <bool kFixed, class Amp>
int ctas_per_sm(int window, int threads) {
  int worst = 1 << 30;
  uint32_t const bins = static_cast<uint32_t>(window);
  auto probe = [&](auto kernel, int block, int algorithm, int pass = 0) {
    size_t const bytes = windowed_smem_bytes<Amp>(static_cast<uint32_t>(window), algorithm, pass, block);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, block, bytes) != cudaSuccess)
      blocks = 0;
    worst = blocks < worst ? blocks : worst;
  };
  probe(windowed_kernel<kFixed, Amp, 0, false>, coreas_block<kFixed, Amp, false>(threads), 0);
  probe(windowed_kernel<kFixed, Amp, 0, true>, coreas_block<kFixed, Amp, true>(threads), 0);
  probe(windowed_kernel<kFixed, Amp, 1, false>, zhs_block<Amp>(threads, bins), 1);
  probe(windowed_kernel<kFixed, Amp, 1, true>, zhs_block<Amp>(threads, bins), 1);
  if constexpr (kFixed) {  // the two passes
    probe(windowed_kernel<true, Amp, 1, false, 1>, zhs_block<Amp, 1>(threads, bins), 1, 1);
    probe(windowed_kernel<true, Amp, 1, true, 1>, zhs_block<Amp, 1>(threads, bins), 1, 1);
    probe(windowed_kernel<true, Amp, 1, false, 3>, zhs_block<Amp, 3>(threads, bins), 1, 3);
    probe(windowed_kernel<true, Amp, 1, true, 3>, zhs_block<Amp, 3>(threads, bins), 1, 3);
  }
  return worst;
}

}  // namespace

cudaError_t launch_ingest_spans(const void* starts, uint64_t pitch, uint64_t count, double* tracks,
                                uint64_t stride, unsigned long long* slot, DeviceCounters* counters,
                                bool diagnostics, IngestTerms const& terms, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  uint64_t const blocks = (count + 255) / 256;
  ingest_kernel<RecordSource><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
      RecordSource{static_cast<const unsigned char*>(starts), pitch}, count, tracks, stride, slot, counters,
      diagnostics, terms);
  return cudaGetLastError();
}

cudaError_t launch_ingest(const c8r_lepton_transport_record* records, uint64_t count,
                          double* tracks, uint64_t stride, unsigned long long* slot,
                          DeviceCounters* counters, bool diagnostics, IngestTerms const& terms,
                          cudaStream_t stream) {
  return launch_ingest_spans(reinterpret_cast<const unsigned char*>(records) +
                                 offsetof(c8r_lepton_transport_record, start),
                             sizeof(c8r_lepton_transport_record), count, tracks, stride, slot, counters, diagnostics,
                             terms, stream);
}

cudaError_t launch_ingest_columns(c8r_track_columns const& columns, uint64_t count, double* tracks,
                                  uint64_t stride, unsigned long long* slot, DeviceCounters* counters,
                                  bool diagnostics, IngestTerms const& terms, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  uint64_t const blocks = (count + 255) / 256;
  ingest_kernel<ColumnSource><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
      ColumnSource{columns}, count, tracks, stride, slot, counters, diagnostics, terms);
  return cudaGetLastError();
}

bool shared_destination(ObserverCache const* observers, std::size_t count, Destination& out) {
  if (count == 0) return false;
  Destination const first = destination_of_host(observers[0]);
  for (std::size_t i = 1; i < count; ++i) {
    Destination const d = destination_of_host(observers[i]);
    if (std::memcmp(&d.height, &first.height, sizeof(double)) != 0 || d.index != first.index ||
        std::memcmp(&d.n, &first.n, sizeof(double)) != 0 ||
        std::memcmp(&d.integral, &first.integral, sizeof(double)) != 0)
      return false;
  }
  out = first;
  return true;
}

cudaError_t launch_direct(EventPlan const& event, uint64_t track_bound, bool coreas, bool zhs,
                          bool fixed, Precision precision, cudaStream_t stream) {
  if (fixed) {
    return precision == Precision::kFP64
               ? direct_dispatch<true, double>(event, track_bound, coreas, zhs, stream)
               : direct_dispatch<true, float>(event, track_bound, coreas, zhs, stream);
  }
  return precision == Precision::kFP64
             ? direct_dispatch<false, double>(event, track_bound, coreas, zhs, stream)
             : direct_dispatch<false, float>(event, track_bound, coreas, zhs, stream);
}

cudaError_t launch_tiled(EventPlan const& event, uint64_t track_bound, bool coreas, bool zhs,
                         bool fixed, Precision precision, cudaStream_t stream) {
  if (fixed) {
    return precision == Precision::kFP64
               ? tiled_dispatch<true, double>(event, track_bound, coreas, zhs, stream)
               : tiled_dispatch<true, float>(event, track_bound, coreas, zhs, stream);
  }
  return precision == Precision::kFP64
             ? tiled_dispatch<false, double>(event, track_bound, coreas, zhs, stream)
             : tiled_dispatch<false, float>(event, track_bound, coreas, zhs, stream);
}

cudaError_t launch_windowed(WorkPlan const& plan, bool fixed, Precision precision, int ctas,
                            int threads, cudaStream_t stream) {
  if (plan.total_items == 0) return cudaSuccess;
  if (fixed)
    return precision == Precision::kFP64 ? windowed_dispatch<true, double>(plan, ctas, threads, stream)
                                         : windowed_dispatch<true, float>(plan, ctas, threads, stream);
  return precision == Precision::kFP64 ? windowed_dispatch<false, double>(plan, ctas, threads, stream)
                                       : windowed_dispatch<false, float>(plan, ctas, threads, stream);
}

int windowed_max_bins(int device) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  // static shared memory of the kernel is a few hundred bytes; keep 1 KiB spare
  int const usable = optin - 1024 - static_cast<int>(kStagingBytes);
  return usable > 0 ? usable / static_cast<int>(3 * sizeof(unsigned long long)) : 0;
}

int windowed_ctas_per_sm(int window, int threads, bool fixed, Precision precision) {
  if (fixed)
    return precision == Precision::kFP64 ? ctas_per_sm<true, double>(window, threads)
                                         : ctas_per_sm<true, float>(window, threads);
  return precision == Precision::kFP64 ? ctas_per_sm<false, double>(window, threads)
                                       : ctas_per_sm<false, float>(window, threads);
}

cudaError_t launch_output(const long long* fixed, const double* floating, double* out, uint64_t total_bins,
                          const ObserverCache* observers, const double* factors, uint32_t observer_count,
                          uint64_t max_bins, bool differentiate, cudaStream_t stream) {
  if (observer_count == 0 || total_bins == 0) return cudaSuccess;
  uint64_t bx = (max_bins + 255) / 256;
  if (bx > 64) bx = 64;
  if (bx == 0) bx = 1;
  dim3 const grid(static_cast<unsigned>(bx), observer_count);
  output_kernel<<<grid, 256, 0, stream>>>(fixed, floating, out, total_bins, observers, factors,
                                          observer_count, differentiate ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t launch_decode(const long long* fixed, double* out, uint64_t total_bins,
                          const uint64_t* observer_offsets, const double* factors,
                          uint32_t observer_count, uint64_t max_bins, cudaStream_t stream) {
  if (observer_count == 0 || total_bins == 0) return cudaSuccess;
  uint64_t bx = (max_bins + 255) / 256;
  if (bx > 64) bx = 64;
  if (bx == 0) bx = 1;
  dim3 const grid(static_cast<unsigned>(bx), observer_count);
  decode_kernel<<<grid, 256, 0, stream>>>(fixed, out, total_bins, observer_offsets, factors);
  return cudaGetLastError();
}

}  // namespace c8r

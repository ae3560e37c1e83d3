// radio_device.cuh — device arithmetic of the radio projection (sm_100a).
//
// Every FP64 expression that decides a time bin, a branch or (in the FP64
// path) an amplitude is written with the reference's association order
// (corsika/detail/kokkos/radio/algorithms/RadioProjection.inl) and this file
// is compiled with -fmad=false, so no multiply-add is contracted: results are
// the IEEE-754 results the x86-64 host produces for the same source.
// Amplitudes take the type `Amp`: double for the FP64 drop-in, float for the
// mixed-precision path.
#pragma once

#include <cstdint>
#include <climits>
#include <cmath>
#include <cstring>

namespace c8r {

// corsika/kokkos/ScalarPhysicalConstants.hpp:18-20, RadioProjectionData.hpp:21-37
constexpr double kSpeedOfLight = 299792458.;
constexpr double kElementaryCharge = 1.6021766208e-19;
constexpr double kVacuumPermittivity = 8.8541878128e-12;
constexpr double kPi = 3.141592653589793238462643383279502884;
constexpr double kCoreasThreshold = 1.e-3;
constexpr double kHeadroom = 4611686018427387904.0;     // 2^62
constexpr double kSignedLimit = 9223372036854775808.0;  // 2^63
constexpr double kElectronMassGeV = 5.109989e-4;        // TransportMass.hpp:20

// Per-observer constants, derived on the host with the same IEEE operations
// the reference evaluates inline (destination bin of propagate, window end of
// add_sample, grid resolution and wavelength).
struct alignas(16) ObserverCache {
  double px, py, pz;
  double start_time;     // startTimeS_
  double end_time;       // startTimeS_ + durationS_   (RadioProjection.inl:273)
  double sample_rate;    // sampleRateHz_
  double resolution;     // 1. / sampleRateHz_         (:374, :396)
  double wavelength;     // c / sampleRateHz_          (:492)
  double fixed_scale;    // fixedPointScale_
  double bins_d;         // (double) numberOfBins_     (:280)
  uint64_t bins;
  uint64_t offset;       // waveformOffset_
  double dest_height;    // (z - minimumHeightM_) * inverseStepPerM_   (:184-185)
  double dest_n;         // refractivity_[dest] + 1.                   (:191)
  double dest_integral;  // integratedRefractivity_[dest]              (:192)
  uint64_t dest_index;   // static_cast<size_t>(dest_height + 0.5)      (:187)
  float fixed_scale_f;
  uint32_t count_samples;  // diagnostic: deposit 1 per component instead of the amplitude
};

// RadioPropagationView with the two tables interleaved as {n-1, integral}.
struct Propagation {
  double homogeneous;
  double min_height;
  double max_height;
  double step;
  double inv_step;
  double slope_n_lower;
  double slope_i_lower;
  double slope_n_upper;
  double slope_i_upper;
  const double2* table;  // .x = refractivity, .y = integrated refractivity
  uint64_t table_size;
  uint32_t refinement;
  uint32_t pad_;
};

// Track kinematics in registers (RadioTrackKinematics minus derived vectors).
struct Track {
  double sx, sy, sz, ex, ey, ez;
  double ts, te;
  double bx, by, bz;
  double length, beta_module, constant;
};

// Track workspace: a record of 24 doubles (192 bytes) per track: start xyz,
// end xyz, t_start, t_end, beta xyz, a packed word (below), the propagation
// terms (factor, n_src; SourceTerms below) of the start, the end and the ZHS
// segment midpoint when every observer of the event shares one destination
// row, that midpoint (start + (start + (end - start))) / 2, the time in the
// middle of the segment, half its duration, and the charge constant.  The
// length and |beta| are recomputed from the fields where an exact evaluation
// needs them (load_track: the same IEEE operations as at ingest).  Records are
// stored in tiles (track_column below).
enum TrackField : int {
  kSx = 0, kSy, kSz, kEx, kEy, kEz, kTs, kTe, kBx, kBy, kBz, kPack,
  kFactorStart, kNsrcStart, kFactorEnd, kNsrcEnd, kFactorMid, kNsrcMid,
  kMx, kMy, kMz, kTm, kHalf, kConst, kTrackDoubles
};
static_assert(kTrackDoubles == 24, "192-byte track records");

// The packed word: the charge constant rounded to FP32 in its low half, and
// in its high half what ingest found out about the track:
//   kTrackRegular  the magnitudes for which the error bounds of the filtered
//                  decisions below are written out hold (regular_track)
//   kTrackDense    n_dst > 1 at the start point (shared destination row only)
//   kTrackOneMid   the CoREAS near-cone midpoint (start + end) / 2 has the
//                  source terms of the ZHS segment midpoint
constexpr unsigned kTrackRegular = 1u, kTrackDense = 2u, kTrackOneMid = 4u;

// The workspace holds tiles of kTrackTile consecutive tracks (6144 bytes): in
// a tile, column k of the records (doubles 2k and 2k + 1, one 16-byte double2)
// is contiguous over the tile's 32 tracks.  The 32 lanes of a warp that read
// one column of 32 consecutive tracks then read 512 contiguous bytes (4 cache
// lines) where interleaved 192-byte records put every lane on its own line;
// the projection kernels' track loads were bound by the L1 data pipe's
// wavefronts with interleaved records.  A workspace is a whole number of tiles
// (track_capacity), so every column of a track below the capacity is inside it.
constexpr unsigned kTrackTile = 32;
constexpr unsigned kTrackColumns = kTrackDoubles / 2;

// Index (in double2 units) of column k of track i.
__host__ __device__ __forceinline__ uint64_t track_column(uint64_t i, unsigned k) {
  return (i / kTrackTile) * (kTrackTile * kTrackColumns) + k * kTrackTile + (i % kTrackTile);
}
// Column 0 of track i; column k is at [k * kTrackTile].
__host__ __device__ __forceinline__ double2 const* track_ref(double const* base, uint64_t i) {
  return reinterpret_cast<double2 const*>(base) + track_column(i, 0);
}
__host__ __device__ __forceinline__ double2* track_ref(double* base, uint64_t i) {
  return reinterpret_cast<double2*>(base) + track_column(i, 0);
}
// Field f of track i.
__host__ __device__ __forceinline__ double track_field(double const* base, uint64_t i, int f) {
  return base[2 * track_column(i, static_cast<unsigned>(f) / 2) + (f & 1)];
}
// Tracks a workspace for n tracks holds: n rounded up to whole tiles.
__host__ __device__ constexpr uint64_t track_capacity(uint64_t n) {
  return (n + kTrackTile - 1) / kTrackTile * kTrackTile;
}

// Length and |beta| as make_radio_track_kinematics evaluates them
// (RadioProjection.inl:145-168), from the track's other fields.
__device__ __forceinline__ void derive_track(Track& t) {
  double const dx = t.ex - t.sx, dy = t.ey - t.sy, dz = t.ez - t.sz;
  t.length = sqrt(dx * dx + dy * dy + dz * dz);
  t.beta_module = t.length / (kSpeedOfLight * (t.te - t.ts));
}

struct Path {
  double time, n_src, n_dst, dist, kx, ky, kz;
};

// static_cast<int>(double) as x86-64 executes it (cvttsd2si): out of range and
// NaN give INT_MIN.  The reference's host build relies on it for ZHS bin spans
// and subtrack counts (RadioProjection.inl:457, :502).
__device__ __forceinline__ int x86_int(double v) {
  if (!(v > -2147483649.0 && v < 2147483648.0)) return INT_MIN;
  return static_cast<int>(v);
}

// static_cast<long long>(double) as x86-64 executes it (cvttsd2si, 64-bit).
__device__ __forceinline__ long long x86_ll(double v) {
  if (!(v >= -9223372036854775808.0 && v < 9223372036854775808.0)) return LLONG_MIN;
  return static_cast<long long>(v);
}

// observer_nearest_bin, RadioProjection.inl:75-82.
__device__ __forceinline__ double nearest_bin(double scaled) {
  double const integral = floor(scaled);
  return integral + (scaled - integral >= 0.5 ? 1. : 0.);
}

// co_reas_doppler, RadioProjection.inl:113-143 (device branch).
__device__ __forceinline__ double doppler(double index, double bx, double by, double bz,
                                          double kx, double ky, double kz) {
  double const ordinary = 1. - index * (bx * kx + by * ky + bz * kz);
  if (ordinary != 0.) return ordinary;
  double const px = bx * kx, py = by * ky, pz = bz * kz;
  double const ex = fma(bx, kx, -px), ey = fma(by, ky, -py), ez = fma(bz, kz, -pz);
  double const xy = px + py;
  double const xy_virtual = xy - px;
  double const xy_error = (px - (xy - xy_virtual)) + (py - xy_virtual);
  double const xyz = xy + pz;
  double const xyz_virtual = xyz - xy;
  double const xyz_error = (xy - (xyz - xyz_virtual)) + (pz - xyz_virtual);
  double const low = ex + ey + ez + xy_error + xyz_error;
  double const product = index * xyz;
  double const product_error = fma(index, xyz, -product) + index * low;
  return (1. - product) - product_error;
}

// The destination row of propagate (RadioProjection.inl:184-192) as the
// projection sees it: the observer's height in table steps, its table index,
// n and integrated refractivity there.  Observers with the same four values
// give the same source terms for a source point.
struct Destination {
  double height;
  uint64_t index;
  double n;
  double integral;
};

__device__ __forceinline__ Destination destination_of(ObserverCache const& o) {
  return Destination{o.dest_height, o.dest_index, o.dest_n, o.dest_integral};
}
inline Destination destination_of_host(ObserverCache const& o) {
  return Destination{o.dest_height, o.dest_index, o.dest_n, o.dest_integral};
}

// The part of propagate (RadioProjection.inl:170-238) that depends on the
// source's height and the destination row only: the travel time is
// factor * |d| / c, with factor = 1 + (I_src - I_dst) / height from the table
// (n for a homogeneous medium), and the refractive indices at both ends.
struct SourceTerms {
  double factor, n_src, n_dst;
};

__device__ __forceinline__ SourceTerms source_terms(Propagation const& p, Destination const& d, double sz) {
  if (p.homogeneous > 0.) return SourceTerms{p.homogeneous, p.homogeneous, p.homogeneous};
  double const sh = (sz - p.min_height) * p.inv_step;
  double const dh = d.height;
  uint64_t const last = p.table_size - 1;
  double n_src = 1., i_src = 1., n_dst = d.n, height = 1.;
  if (sh + 0.5 >= static_cast<double>(last)) {
    double2 const t = __ldg(p.table + last);
    n_src = t.x + p.slope_n_upper * fabs((sz - p.max_height) * p.inv_step) + 1.;
    i_src = t.y + p.slope_i_upper * fabs(p.max_height - sz);
    height = sh - dh;
  } else if (sh + 0.5 < static_cast<double>(last) && sh > 0.) {
    uint64_t const si = static_cast<uint64_t>(sh + 0.5);
    double2 const t = __ldg(p.table + si);
    n_src = t.x + 1.;
    i_src = t.y;
    height = static_cast<double>(static_cast<int64_t>(si) - static_cast<int64_t>(d.index)) * p.step;
    if (height == 0.) height = 1.;
  } else if (sh == 0.) {
    n_src = 1.;
    n_dst = 1.;
    i_src = __ldg(p.table).y;
    height = dh - sh;
  } else {
    double2 const t0 = __ldg(p.table);
    n_src = t0.x + p.slope_n_lower * fabs(sh) + 1.;
    i_src = t0.y + p.slope_i_lower * fabs(sh);
    n_dst = 1.;
    height = dh - fabs(sh);
  }
  return SourceTerms{1. + (i_src - d.integral) / height, n_src, n_dst};
}

// The high word of |x|: sign cleared, exponent on top.
__host__ __device__ __forceinline__ unsigned magnitude_word(double x) {
#ifdef __CUDA_ARCH__
  return static_cast<unsigned>(__double2hiint(x)) & 0x7fffffffu;
#else
  uint64_t bits;
  std::memcpy(&bits, &x, sizeof bits);
  return static_cast<unsigned>(bits >> 32) & 0x7fffffffu;
#endif
}

// The operands of the quotients below lie in [2^-400, 2^400): a quotient is then
// a normal number above 2^-801, and its remainder, a multiple of 2^-1000, exact.  Outside (zeros, infinities and NaN among them) the division is used.
constexpr unsigned kQuotientLow = 0x26f00000u, kQuotientHigh = 0x58f00000u;  // 2^-400, 2^400

// x / c, correctly rounded, without a division (P. Markstein, IBM J. Res. Dev. 34,
// 1990): with z = RN(1/c), q = RN(x z) and the exact remainder r = x - q c,
// RN(q + r z) is RN(x / c) when q is within one unit in the last place of x / c.
// z is within 0.187 2^-53 of 1/c here, so q is within 0.69 units.
__host__ __device__ __forceinline__ double over_light_speed(double x) {
  constexpr double z = 1. / kSpeedOfLight;
  if (magnitude_word(x) - kQuotientLow >= kQuotientHigh - kQuotientLow) return x / kSpeedOfLight;
  double const q = x * z;
  return fma(fma(-q, kSpeedOfLight, x), z, q);
}

// (x, y, z) / d for d = |(x, y, z)|, each correctly rounded, from one reciprocal
// (the same theorem):
// r = RN(1/d); a r is within 1.5 units in the last place of a / d, one
// correction by its remainder brings it within one, and the second one rounds
// correctly.
__host__ __device__ __forceinline__ void divide3(double& x, double& y, double& z, double d) {
  unsigned const hx = magnitude_word(x), hy = magnitude_word(y), hz = magnitude_word(z);
  unsigned const least = min(min(hx, hy), hz);
  if (least < kQuotientLow || magnitude_word(d) >= kQuotientHigh) {
    x = x / d;
    y = y / d;
    z = z / d;
    return;
  }
  double const r = 1. / d;
  auto quotient = [&](double a) {
    double const q0 = a * r;
    double const q1 = fma(fma(-q0, d, a), r, q0);
    return fma(fma(-q1, d, a), r, q1);
  };
  x = quotient(x);
  y = quotient(y);
  z = quotient(z);
}

// propagate, RadioProjection.inl:170-238, given the source terms of the
// point: the reference's (1 + (I_src - I_dst) / height) * dist / c with the
// parenthesised factor taken from `st` (the same IEEE value), or n dist / c.
// kTime = false skips the refractive index and travel time (the Fraunhofer
// midpoint uses only k and distance).  kDivide takes the three quotients by the
// distance as divisions: the plain shapes, which wait for their atomics and not for
// the FP64 pipe, lose more to the written-out form's range checks and registers than
// they save (3e5 x 160, direct shape, written-out / divisions: FP64 25.6 / 24.6 ms,
// mixed 24.8 / 23.2, floating 16.7 / 15.6; the travel time divided too, 200 mixed
// tracks x 16 antennas refined fourfold take 152 us for 131; the windowed FP64 CoREAS
// kernel 4.6 written out, 5.0 divided, at 1e6 x 160).
template <bool kTime, bool kDivide = false>
__device__ __forceinline__ Path propagate_with(SourceTerms const& st, ObserverCache const& o,
                                               double sx, double sy, double sz) {
  Path r;
  double const dx = o.px - sx, dy = o.py - sy, dz = o.pz - sz;
  double const dist = sqrt(dx * dx + dy * dy + dz * dz);
  r.kx = dx;
  r.ky = dy;
  r.kz = dz;
  if (kDivide) {
    r.kx = dx / dist;
    r.ky = dy / dist;
    r.kz = dz / dist;
  } else {
    divide3(r.kx, r.ky, r.kz, dist);
  }
  r.dist = dist;
  if (!kTime) return r;
  r.time = over_light_speed(st.factor * dist);
  r.n_src = st.n_src;
  r.n_dst = st.n_dst;
  return r;
}

// propagate, RadioProjection.inl:170-238: the source terms looked up in the
// table for this observer, then the path.
template <bool kTime, bool kDivide = false>
__device__ __forceinline__ Path propagate(Propagation const& p, ObserverCache const& o,
                                          double sx, double sy, double sz) {
  SourceTerms const st = kTime ? source_terms(p, destination_of(o), sz) : SourceTerms{0., 0., 0.};
  return propagate_with<kTime, kDivide>(st, o, sx, sy, sz);
}

// ---------------------------------------------------------------- filtered paths
// The mixed-precision kernels evaluate distances, detection times and Doppler
// factors with a few FP64 operations each, in units of the observer's bins,
// and take a decision (a bin, a branch, an order) only where a fixed guard
// shows that the reference's own arithmetic takes the same one; any other pair
// or segment is evaluated exactly, operation by operation.  The guards hold
// for "regular" tracks, whose magnitudes ingest has checked (regular_track):
//
//   |beta|_1 <= 4; 0 < n <= 4 and |factor| <= 4 at the source points; every time
//   t of the track has (|t| + |t0|) fs <= 2^24 bins and every coordinate x has
//   |x| fs / c <= 2^24 at every observer of the event, and the track lasts at
//   most 2^21 bins (TrackLimits).
//
// With u = 2^-53, for a source point at displacement d from the observer
// (the reference's own subtractions):
//   s2 = d.d (one product, two fused adds) is within 2u of |d|^2 where the
//   reference's is within 3u; y from lean_rsqrt is within 4u of 1/sqrt(s2);
//   so |d| = RN(s2 y) is within 7u of the reference's and k = d y within 8u.
//   w = beta.k and n w lie within 16 u n |beta|_1 <= 2^-45 of the reference's,
//   hence 1 - n w within kDopplerGuard = 2^-43.
//   A detection time in bins, x = (t - t0) fs + |d| factor fs / c, lies within
//   32u (|t| + |t0| + time) fs of the reference's (t + time - t0) fs; where x
//   falls on the trace (fewer than 2^26 bins) that is below 32u 2^27 = 2^-21,
//   and the ZHS term n w (t - t_mid) adds at most 2^-43 2^20; kBinGuard =
//   2^-19 covers both, the 2^-20 of a divided track's segments
//   (lean_divisible) and the 2^-22 of their source terms (terms_decided).  Where |x| is larger the error grows like 2^-46 |x|, so
//   such an x is off the trace in the reference as well.
constexpr double kDopplerGuard = 0x1p-43;
constexpr double kBinGuard = 0x1p-19;
constexpr double kMaxLeanBins = 67108864.0;   // 2^26
constexpr double kMaxLeanTime = 16777216.0;   // 2^24 bins

// Limits on a track's times (s), from every observer of the event.
struct TrackLimits {
  double time = 0.;      // |t_start|, |t_end| at most this
  double duration = 0.;  // t_end - t_start at most this
  double length = 0.;    // |coordinates| (m) at most this
};

__device__ __forceinline__ bool lean_terms(SourceTerms const& st) {
  return (st.n_src > 0.) & (st.n_src <= 4.) & (fabs(st.factor) <= 4.);
}

// Whether the track's own magnitudes are covered by the bounds above.
__device__ __forceinline__ bool regular_track(Track const& t, double duration, TrackLimits const& limits) {
  double const furthest = fmax(fmax(fmax(fabs(t.sx), fabs(t.sy)), fmax(fabs(t.sz), fabs(t.ex))),
                               fmax(fabs(t.ey), fabs(t.ez)));
  return fabs(t.bx) + fabs(t.by) + fabs(t.bz) <= 4. && fabs(t.ts) <= limits.time && fabs(t.te) <= limits.time &&
         duration <= limits.duration && furthest <= limits.length;
}

// 1/sqrt(s2) from the hardware's approximate reciprocal square root (about 20
// bits) and one third-order step (the binomial series of (1 - r)^(-1/2), Householder's
// iteration of order 2): with r = 1 - s2 y0^2 and |r| <= 2^-17
// (checked, so the seed's accuracy is not relied on), y0 (1 + r/2 + 3 r^2/8)
// is within (5/16) 2^-51 + 3u < 4u of it.  False when s2 lies outside
// [2^-100, 2^100] or is not a number.
__device__ __forceinline__ bool lean_rsqrt(double s2, double& y) {
  double seed;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(seed) : "d"(s2));
  double const r = fma(-(s2 * seed), seed, 1.);
  y = fma(seed * r, fma(r, 0.375, 0.5), seed);
  unsigned const high = static_cast<unsigned>(__double2hiint(s2)) - 0x39b00000u;  // 2^-100
  return (fabs(r) <= 0x1p-17) & (high <= 0x46300000u - 0x39b00000u);               // 2^100
}

// The nearest integer of x (|x| < 2^31 where the result is used) as `bin`, and
// x minus it, in [-1/2, 1/2]: x + 1.5 2^52 rounds to an integer whose low word
// is the integer's.
__device__ __forceinline__ double lean_nearest(double x, int& bin) {
  constexpr double kRound = 6755399441055744.0;  // 1.5 2^52
  double const shifted = x + kRound;
  bin = __double2loint(shifted);
  return x - (shifted - kRound);
}

// The FP32 charge constants carry 2^60 and the observers' scales 2^-60, so
// that neither leaves the FP32 range for any field limit whose fixed-point
// scale is an FP32 number itself.
constexpr double kConstantShift = 0x1p60;

// Constants of the item's observer for the filtered paths, derived once per
// work item from its ObserverCache.  In 16-byte groups of what is used together:
// the track loops read them from shared memory once a track, 16 bytes a load
// (copy_words; as 8-byte loads they took a third of the ZHS loop's
// shared-memory wavefronts).
struct alignas(16) LeanObserver {
  double px, py;
  double pz, start_time;
  double rate;         // fs
  double rate_over_c;  // fs / c
  double gate_in;      // CoREAS: a sample at kBinGuard < x < gate_in is recorded,
  double gate_out;     // one at x < -kBinGuard or x > gate_out is not
  double fraunhofer;   // ZHS: 8 pi c^2 / (wavelength fs^2)
  double past;         // number of bins + 1: a segment that starts later is off the trace
  float scale;         // 2^-60 x fixed-point scale (x fs, CoREAS); 0 when counting samples
  float bias;          // 1 when counting samples, else 0
  uint32_t usable;     // the filtered paths may be used for this observer
  uint32_t bins;
  double start_bins;   // t0 fs
  double half_rate;    // fs / 2
  double bin_guard_m;  // kBinGuard bins of path
  double fixed_scale;  // fixed-point scale; 0 when counting samples
};

template <int kAlgorithm>
__device__ __forceinline__ void make_lean_observer(ObserverCache const& o, LeanObserver& l) {
  double const fs = o.sample_rate;
  l.px = o.px;
  l.py = o.py;
  l.pz = o.pz;
  l.start_time = o.start_time;
  l.rate = fs;
  l.rate_over_c = fs / kSpeedOfLight;
  l.half_rate = 0.5 * fs;
  l.bin_guard_m = kBinGuard * kSpeedOfLight / fs;
  double const end = (o.end_time - o.start_time) * fs;
  double const last = o.bins_d - 0.5;
  double const gate = end < last ? end : last;
  l.gate_in = gate - kBinGuard;
  l.gate_out = gate + kBinGuard;
  l.start_bins = o.start_time * fs;
  l.fraunhofer = 8. * kPi * (kSpeedOfLight / fs) * (kSpeedOfLight / fs) / o.wavelength;
  l.past = o.bins_d + 1.;
  double const scale = (kAlgorithm == 0 ? fs * o.fixed_scale : o.fixed_scale) / kConstantShift;
  l.scale = o.count_samples ? 0.f : static_cast<float>(scale);
  l.fixed_scale = o.count_samples ? 0. : o.fixed_scale;
  l.bias = o.count_samples ? 1.f : 0.f;
  l.usable = o.bins_d < kMaxLeanBins && fs < 0x1p200 ? 1u : 0u;
  l.bins = static_cast<uint32_t>(o.bins);
}

// A copy in registers, read from shared memory 16 bytes at a time.
template <class T>
__device__ __forceinline__ T copy_words(T const& shared) {
  static_assert(sizeof(T) % sizeof(double2) == 0 && alignof(T) >= sizeof(double2), "16-byte words");
  T copy;
#pragma unroll
  for (unsigned i = 0; i < sizeof(T) / sizeof(double2); ++i)
    reinterpret_cast<double2*>(&copy)[i] = reinterpret_cast<double2 const*>(&shared)[i];
  return copy;
}

// separate_same_bin_endpoints, RadioProjection.inl:303-336.
__device__ __forceinline__ void separate_same_bin(double& start, double& end, double res,
                                                  bool signed_order) {
  long long const sb = x86_ll(nearest_bin(start / res));
  long long const eb = x86_ll(nearest_bin(end / res));
  if (sb != eb) return;
  double const sf = start / res - floor(start / res);
  double const ef = end / res - floor(end / res);
  bool const forward = !signed_order || end >= start;
  if (forward) {
    if (sf >= 0.5 && ef >= 0.5) start -= res;
    else if (sf < 0.5 && ef < 0.5) end += res;
    else if (ef >= 1. - sf) end += res;
    else start -= res;
  } else {
    if (sf >= 0.5 && ef >= 0.5) end -= res;
    else if (sf < 0.5 && ef < 0.5) start += res;
    else if (sf >= 1. - ef) start += res;
    else end -= res;
  }
}

template <class T>
struct Vec3 {
  T x, y, z;
};

// k x (k x beta) (transverse_endpoint, :240-243) and k x (beta x k) (:438).
template <class T>
__device__ __forceinline__ Vec3<T> cross(Vec3<T> a, Vec3<T> b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// Per-thread event counters (RadioCounters' projection fields).
struct Counts {
  unsigned long long coreas = 0, zhs = 0, subtracks = 0, overflows = 0;
  float mag = 0.f;  // sum of |fixed-point increments| added to a window without checks
};

}  // namespace c8r

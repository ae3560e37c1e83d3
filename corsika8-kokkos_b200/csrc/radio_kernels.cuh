// radio_kernels.cuh — launch-side declarations shared by the host library.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "radio_device.cuh"

struct c8r_lepton_transport_record;
struct c8r_counters;
struct c8r_track_columns;

namespace c8r {

// Device-side counters of one event (the layout of RadioCounters).
struct alignas(8) DeviceCounters {
  unsigned long long coreas_contributions;
  unsigned long long zhs_contributions;
  unsigned long long zhs_subtracks;
  unsigned long long valid_tracks;
  unsigned long long fixed_point_overflows;
  double weighted_segment_count;
  double track_length_m;
  double weighted_track_length_m;
  double electron_weighted_track_length_m;
  double positron_weighted_track_length_m;
  double signed_charge_weighted_track_length_m;
  double energy_weighted_track_length_gev_m;
  double maximum_segment_length_m;
  double weighted_direction_change_rad;
  double weighted_direction_change_squared_rad2;
  double weighted_beta_deficit_track_length_m;
  double weighted_time_residual_s;
  double maximum_direction_change_rad;
  double signed_charge_weighted_direction_change[3];
  double weighted_track_length_by_kinetic_energy_m[15];
};
static_assert(sizeof(DeviceCounters) == 288, "RadioCounters layout");

// One event of a projection launch: its tracks (SoA, `stride` doubles per
// row), observers, traces and counters.  Algorithm 0 = CoREAS field,
// algorithm 1 = ZHS potential.  Trace rows are [X | Y | Z] of total_bins each.
struct EventPlan {
  const double* tracks;
  uint64_t stride;
  const unsigned long long* valid_tracks;  // device: tracks written by ingest
  const ObserverCache* observers[2];
  uint32_t observer_count[2];
  unsigned long long* fixed[2];  // int64 fixed-point traces (deterministic)
  double* floating[2];           // FP64 traces (floating mode)
  uint64_t total_bins[2];
  Propagation propagation;
  DeviceCounters* counters;
  uint64_t first_item;           // work-list offset of this event (in its algorithm's list)
  uint32_t chunk_size;           // tracks per work item
  uint32_t chunks;
  uint32_t window;               // shared-memory bins per item (<= kernel window)
  uint64_t first_track;          // chunk c covers first_track + c * chunk_size onwards,
  uint64_t last_track;           // clipped to [.., last_track) and the valid tracks
  uint32_t precomputed;          // tracks carry their source terms (every observer shares
                                 // one destination row; see IngestTerms)
  uint32_t pad_;
};

// Source terms written at ingest: when every observer of an event shares one
// destination row (always in a homogeneous medium), each track record gets
// the propagation terms of its start, end and midpoint for that row,
// and the windowed kernels read them instead of looking them up per pair.
struct IngestTerms {
  int32_t enabled;
  int32_t pad_;
  Propagation propagation;
  Destination destination;
  TrackLimits limits;  // times for which the filtered paths' error bounds hold
};
// The destination row shared by all `count` observers, if they share one.
bool shared_destination(ObserverCache const* observers, std::size_t count, Destination& out);
// The track limits of the filtered paths over `count` observers, narrowed from
// `limits` (start from widest_limits()).
inline TrackLimits widest_limits() { return TrackLimits{1e300, 1e300, 1e300}; }
inline void narrow_limits(ObserverCache const* observers, std::size_t count, TrackLimits& limits) {
  for (std::size_t i = 0; i < count; ++i) {
    ObserverCache const& o = observers[i];
    double const start = o.start_time < 0. ? -o.start_time : o.start_time;
    double const time = kMaxLeanTime / o.sample_rate - start, duration = 0x1p21 / o.sample_rate;
    double const length = kMaxLeanTime * kSpeedOfLight / o.sample_rate;
    if (!(time >= limits.time)) limits.time = time;  // may be negative: no track then
    if (!(duration >= limits.duration)) limits.duration = duration;
    if (!(length >= limits.length)) limits.length = length;
  }
}

// Persistent windowed launch over a work list of (event, chunk, algorithm,
// observer) items drawn from an atomic counter.  Passed as a __grid_constant__
// kernel parameter (no host-to-device copy; graph-capturable).
constexpr int kMaxEventsPerLaunch = 64;
constexpr int kPlanEntries = kMaxEventsPerLaunch + 1;  // + the short-chunk tail of the last event
constexpr int kWindowThreads = 640;  // upper bound (and default) of the windowed block size
// A work item that the first pass of a two-pass ZHS launch handed back.
struct ItemState {
  uint64_t item;
};

struct WorkPlan {
  EventPlan events[kPlanEntries];
  int32_t algorithm;        // 0: CoREAS items, 1: ZHS items
  uint32_t event_count;
  uint32_t window;          // shared-memory bins per CTA (max over events)
  uint64_t total_items;
  unsigned int* next_item;  // zeroed before each launch
  // Each CTA's list of the deferred pairs of its current item,
  // `deferred_stride` entries from deferred + blockIdx.x * deferred_stride
  // (at least the longest chunk of the plan; deferred_list_stride below).
  unsigned int* deferred;
  uint32_t deferred_stride;
  // Items run again with checked window adds (the unchecked run's bound did
  // not hold); counted when not null.
  unsigned long long* reruns;
  // Items the first pass of two handed to the second; counted when not null.
  unsigned long long* handbacks;
  // Two-pass ZHS (fixed point), when item_state is set: the first pass projects
  // the items it can with unchecked window adds and appends the others to
  // item_state, counted by drain_next_item[0]; the second takes those in turn,
  // counted by drain_next_item[1], and projects them in full, with its own lists
  // (`drain_deferred`, deferred_stride entries a CTA).  attach_deferred sets these.
  ItemState* item_state;
  unsigned int* drain_deferred;
  unsigned int* drain_next_item;
};

// A work item spans at most kMaxChunkTracks tracks: a deferred-list entry is
// the pair's track offset in the item (its low 30 bits) and two bits of the
// track loop's decision (CoREAS: the near-Cherenkov branch and its order).
constexpr uint32_t kMaxChunkTracks = 1u << 30;
constexpr unsigned kDeferredHintShift = 30;
constexpr unsigned kDeferredOffsetMask = (1u << kDeferredHintShift) - 1u;

// Entries per CTA of a launch's deferred lists: the plan's longest chunk.
inline uint32_t deferred_list_stride(WorkPlan const& plan) {
  uint32_t stride = 0;
  for (uint32_t e = 0; e < plan.event_count; ++e)
    if (plan.events[e].chunk_size > stride) stride = plan.events[e].chunk_size;
  return stride;
}

// Launches whose two-pass storage would pass 2^30 words (4 GiB) run one pass.
constexpr uint64_t kTwoPassMaxWords = 1ull << 30;

inline uint64_t two_pass_words(WorkPlan const& plan, uint64_t ctas) {
  return 2 * ctas * plan.deferred_stride +
         plan.total_items * (sizeof(ItemState) / sizeof(unsigned)) + 2;
}

// ZHS launches in fixed point run in two passes when their storage fits.
inline bool two_pass(WorkPlan const& plan, uint64_t ctas, bool fixed) {
  return fixed && plan.algorithm == 1 && two_pass_words(plan, ctas) <= kTwoPassMaxWords;
}

// 32-bit words of deferred-list storage a launch of `plan` (deferred_stride
// and total_items set) over `ctas` CTAs needs: its CTAs' lists, and for two
// passes the second pass's lists, the handed-back items and their two counters.
inline uint64_t deferred_words(WorkPlan const& plan, uint64_t ctas, bool fixed) {
  if (!two_pass(plan, ctas, fixed)) return ctas * plan.deferred_stride;
  return two_pass_words(plan, ctas);
}

// Points the plan's deferred-list storage into `words` (deferred_words of it).
inline void attach_deferred(WorkPlan& plan, unsigned* words, uint64_t ctas, bool fixed) {
  plan.deferred = words;
  plan.item_state = nullptr;
  plan.drain_deferred = nullptr;
  plan.drain_next_item = nullptr;
  if (!two_pass(plan, ctas, fixed)) return;
  uint64_t const first = ctas * plan.deferred_stride;
  plan.drain_deferred = words + first;
  plan.item_state = reinterpret_cast<ItemState*>(words + first + ctas * plan.deferred_stride);
  plan.drain_next_item = reinterpret_cast<unsigned*>(plan.item_state + plan.total_items);
}

// How append_work divides `chunks` long chunks of `big` tracks when it ends the
// list on short items: the first `head` stay long, the rest of the tracks go in
// chunks of `small`, a quarter as long (at least 8192 tracks), about two items for
// each of the `ctas` persistent CTAs.
struct TailSplit {
  uint64_t head, small;
};
inline TailSplit split_tail(uint64_t chunks, uint64_t big, uint64_t per, uint64_t ctas) {
  constexpr uint64_t kSplit = 4, kMinTailChunk = 8192;
  uint64_t const quarter = (big + kSplit - 1) / kSplit;
  // whole track tiles, so that short items start on a tile as long ones do
  uint64_t const small = track_capacity(quarter > kMinTailChunk ? quarter : kMinTailChunk);
  if (small >= big) return {chunks, small};
  uint64_t const short_items = (2 * ctas + per - 1) / per;
  uint64_t const replaced = (short_items * small + big - 1) / big;  // long chunks they cover
  return {replaced >= chunks ? 0 : chunks - replaced, small};
}

// Appends the (chunk, observer) work items of `ev` for plan.algorithm to
// `plan` (first_item, event_count and total_items follow).  With `fine_tail`
// and a free event slot, the last chunks go in as a second entry of short chunks
// (split_tail): the launch then ends on short items instead of one CTA finishing a
// long item while the others wait.  Every track stays in exactly one item.
// Returns the number of items appended.
inline uint64_t append_work(WorkPlan& plan, EventPlan ev, uint64_t ctas, bool fine_tail) {
  uint64_t const per = ev.observer_count[plan.algorithm];
  if (per == 0 || ev.chunks == 0 || plan.event_count >= kPlanEntries) return 0;
  uint64_t const big = ev.chunk_size;
  TailSplit split{ev.chunks, 0};
  if (fine_tail && plan.event_count + 2 <= kPlanEntries) split = split_tail(ev.chunks, big, per, ctas);
  uint64_t const head = split.head, small = split.small;
  uint64_t const before = plan.total_items;
  if (head > 0) {
    EventPlan e = ev;
    e.chunks = static_cast<uint32_t>(head);
    e.first_item = plan.total_items;
    plan.events[plan.event_count++] = e;
    plan.total_items += head * per;
  }
  if (head < ev.chunks) {
    uint64_t const stop = ev.first_track + ev.chunks * big;
    EventPlan e = ev;
    e.first_track = ev.first_track + head * big;
    e.last_track = stop < ev.last_track ? stop : ev.last_track;
    e.chunk_size = static_cast<uint32_t>(small);
    e.chunks = static_cast<uint32_t>(((ev.chunks - head) * big + small - 1) / small);
    e.first_item = plan.total_items;
    plan.events[plan.event_count++] = e;
    plan.total_items += static_cast<uint64_t>(e.chunks) * per;
  }
  return plan.total_items - before;
}

// What an item costs beside its tracks, in tracks: the window zeroed, summed and
// flushed, a part of it whatever the window's size; relative to the tracks' own
// time, which is 2.2 times as long in FP64 and grows with the subtrack refinement (of
// ZHS, half of the tracks' time).
// Fitted, with the two margins of plan_cost, to 2044 timed launches (1 to 300
// antennas, 1500 to 9.5e6 tracks, windows of 900 to 8192 bins, 1 to 296 chunks with
// and without a short tail): the plan of least cost is within 0.6% of the fastest
// timed one in the mean, 6.8% at worst.
inline double item_cost(uint32_t window, bool fp64, uint32_t refinement) {
  return (2000. + 1.5 * window) * (fp64 ? 0.4 : 1.) * 2. / (1. + (refinement > 1 ? refinement : 1u));
}

// Length of a launch over `count` tracks at `per` observers in chunks of `chunk`
// tracks, in tracks: without a tail as many rounds as the busiest CTA has items,
// and a fifth more, since the antennas' loads differ; with a short tail, which
// evens that out, the mean load and half a short item.  (A list of short items
// alone is one without a tail.)
inline double plan_cost(uint64_t count, uint64_t per, uint64_t ctas, uint64_t chunk, bool tail, double item) {
  uint64_t const chunks = (count + chunk - 1) / chunk;
  TailSplit const split = tail ? split_tail(chunks, chunk, per, ctas) : TailSplit{chunks, 0};
  uint64_t const left = count - (split.head * chunk < count ? split.head * chunk : count);
  uint64_t const short_chunks = split.head < chunks && left > 0 ? (left + split.small - 1) / split.small : 0;
  double const longest = static_cast<double>(chunk < count ? chunk : count);
  double const rounds = static_cast<double>((split.head * per + ctas - 1) / ctas) * (item + longest);
  if (short_chunks == 0) return 1.2 * rounds;
  double const shortest = static_cast<double>(split.small < count ? split.small : count);
  if (split.head == 0)
    return 1.2 * static_cast<double>((short_chunks * per + ctas - 1) / ctas) * (item + shortest);
  double const mean = (static_cast<double>((split.head + short_chunks) * per) * item +
                       static_cast<double>(count) * static_cast<double>(per)) / static_cast<double>(ctas);
  double const even = mean + 0.5 * (item + shortest);
  return 1.1 * (rounds > even ? rounds : even);
}

// Whether a launch of one algorithm's items of `ev` alone ends sooner on short items.
inline bool tail_pays(EventPlan const& ev, int algorithm, uint64_t ctas, double item) {
  uint64_t const per = ev.observer_count[algorithm], count = static_cast<uint64_t>(ev.chunks) * ev.chunk_size;
  if (count == 0 || per == 0 || ctas == 0) return false;
  return plan_cost(count, per, ctas, ev.chunk_size, true, item) < plan_cost(count, per, ctas, ev.chunk_size, false, item);
}

// The least number of chunks whose deferred lists, an item for each CTA, stay small:
// at least 16 items a CTA, or items of 262144 tracks.
inline uint64_t fewest_chunks(uint64_t count, uint64_t per, uint64_t ctas) {
  constexpr uint64_t kLongest = 262144;
  uint64_t const share = (count * per + 16 * ctas - 1) / (16 * ctas);
  uint64_t const longest = share > kLongest ? share : kLongest;
  return (count + longest - 1) / longest;
}

// Tracks per work item for `count` tracks at `per` observers of one algorithm's
// launch on `ctas` persistent CTAs: of the plans that fill 1, 2, .. rounds, with or
// without a tail, the one of least cost.
// (The former rule took at most 64 chunks and no tail below four rounds: 9.5e6
// tracks at 1 / 5 antennas, 6e6 at 8, CoREAS and ZHS together, FP64 1800 / 5545 / 5415
// -> 922 / 3624 / 3479 us, mixed 828 / 2513 / 2461 -> 516 / 1706 / 1617.)
inline uint64_t auto_chunk(uint64_t count, uint64_t per, uint64_t ctas, double item) {
  constexpr uint64_t kRounds = 32;
  if (count == 0 || per == 0 || ctas == 0) return kTrackTile;
  uint64_t const fewest = fewest_chunks(count, per, ctas);
  uint64_t best = 0;
  double least = 0.;
  auto consider = [&](uint64_t chunks) {
    if (chunks < fewest) return;
    uint64_t const chunk = track_capacity((count + chunks - 1) / chunks);
    if (chunk == best) return;
    for (bool tail : {false, true}) {
      double const cost = plan_cost(count, per, ctas, chunk, tail, item);
      if (best == 0 || cost < least) {
        least = cost;
        best = chunk;
      }
    }
  };
  consider(fewest);
  uint64_t const first = (fewest * per + ctas - 1) / ctas;
  for (uint64_t round = first; round < first + kRounds; ++round) consider(round * ctas / per);
  return best;
}

// The same for an event of a batched launch, whose items fill the GPU together: the
// more chunks, the more windows its `share` of the CTAs passes over (the event's
// part of the launch's work, `total`), the fewer, the longer the launch waits for
// its last items (half an item; a whole one or two cost up to 27%: 3 events of 20000
// tracks at 100 antennas); the number with the least of both.  Cut for the whole GPU each, 64
// events of 1500 tracks at 16 antennas took 1738 us in FP64, 604 in chunks of 8192
// tracks at least, 437 so.
inline uint64_t batch_chunk(uint64_t count, uint64_t per, uint64_t ctas, double item, double total) {
  if (count == 0 || per == 0 || ctas == 0) return kTrackTile;
  double const work = static_cast<double>(per) * (static_cast<double>(count) + item);
  double const window = static_cast<double>(per) * item / (static_cast<double>(ctas) * (work / total));
  uint64_t chunks = fewest_chunks(count, per, ctas);
  auto cost = [&](uint64_t c) {
    return static_cast<double>(c) * window + 0.5 * static_cast<double>(count) / static_cast<double>(c);
  };
  uint64_t const most = (count + kTrackTile - 1) / kTrackTile;
  while (chunks < most && cost(chunks + 1) < cost(chunks)) ++chunks;
  return track_capacity((count + chunks - 1) / chunks);
}

// Whether `count` tracks at `observers` antennas go to the direct kernel where the
// choice is automatic; `whole`: the longest trace fits a window.  The windowed launches
// cost 25 us an algorithm whatever their size, the direct kernel waits for its serial
// chain of atomics (longest for ZHS's many samples at few antennas).  Timed on 7560
// launches of 64 to 16000 tracks at 1 to 300 antennas; of the two kernels the rule
// takes the slower one by 0.2 to 3% in the mean of each class below.  us, direct /
// windowed, 8192 bins x 160 antennas unless given:
//   below 256 tracks       direct; 128 tracks FP64 210 / 67, but 33 / 57 where few samples meet the trace
//   both algorithms        windowed; FP64 256 tracks 202 / 89, 4096 393 / 153
//   CoREAS alone           FP64 512 tracks 30 / 47, 16000 219 / 155; floating 600 bins 4096 tracks 44 / 55
//   refined (not mixed in fixed point in one window: there the drain is windowed's
//                          fastest)   FP64 fourfold 16 antennas 4096 tracks 241 / 149,
//                          160 antennas 4096 tracks 470 / 719
// From 16384 tracks (the reference's threshold, RadioAccumulator.hpp:101) windowed.
inline bool direct_pays(uint64_t count, uint64_t observers, bool zhs, uint32_t refinement, bool fixed, bool fp64,
                        bool whole) {
  constexpr uint64_t kFewest = 256, kMost = 16384;
  if (count < kFewest || count >= kMost) return count < kFewest;
  double const n = static_cast<double>(count), antennas = static_cast<double>(observers);
  if (!zhs) return !fixed || n * n * antennas < 26000. * 26000.;
  if (refinement <= 1 || (fixed && !fp64 && whole)) return false;
  double const refined = antennas * refinement * refinement;
  return n * refined * refined >= 40000. * 40000.;
}

enum class Precision : int { kFP64 = 0, kMixed = 1 };

// Record ingest: LeptonTransportRecord AoS -> compacted SoA kinematics
// (make_radio_track_kinematics + record_track).  `slot` receives the number of
// valid tracks written.
cudaError_t launch_ingest(const c8r_lepton_transport_record* records, uint64_t count,
                          double* tracks, uint64_t stride, unsigned long long* slot,
                          DeviceCounters* counters, bool diagnostics, IngestTerms const& terms,
                          cudaStream_t stream);

// The same from records' start and end states `pitch` bytes apart, the first
// record's at `starts`.
cudaError_t launch_ingest_spans(const void* starts, uint64_t pitch, uint64_t count, double* tracks,
                                uint64_t stride, unsigned long long* slot, DeviceCounters* counters,
                                bool diagnostics, IngestTerms const& terms, cudaStream_t stream);

// The same ingest from a structure-of-arrays view of the steps.
cudaError_t launch_ingest_columns(c8r_track_columns const& columns, uint64_t count, double* tracks,
                                  uint64_t stride, unsigned long long* slot, DeviceCounters* counters,
                                  bool diagnostics, IngestTerms const& terms, cudaStream_t stream);

// Direct pair kernel: one thread per (track, observer) pair, global atomics.
// The valid-track count is read on the device; `track_bound` (the record
// count) bounds the grid on the host.
cudaError_t launch_direct(EventPlan const& event, uint64_t track_bound, bool coreas, bool zhs,
                          bool fixed, Precision precision, cudaStream_t stream);

// The reference's large-batch tile shape: 256-thread CTAs over tiles of 8
// tracks x 32 observers staged in shared memory, one thread per pair, global
// atomics (RadioTileProjection, RadioAccumulator.inl:13-85).
cudaError_t launch_tiled(EventPlan const& event, uint64_t track_bound, bool coreas, bool zhs,
                         bool fixed, Precision precision, cudaStream_t stream);

// Persistent windowed kernel.  `ctas` persistent CTAs of `threads` threads.
// The plan needs plan.deferred with ctas * deferred_stride entries and
// deferred_stride >= deferred_list_stride(plan) (else cudaErrorInvalidValue).
cudaError_t launch_windowed(WorkPlan const& plan, bool fixed, Precision precision, int ctas,
                            int threads, cudaStream_t stream);
// Largest window (bins) that fits the opt-in shared memory of this device.
int windowed_max_bins(int device);
// The window of a launch whose longest trace has `longest` bins, `max_bins` the
// largest that fits: the whole trace, or a part of it that leaves the CoREAS kernel
// inside 196 KB of shared memory and the ZHS kernels room for their FP64 staging.  The
// next configuration, 228 KB, halves the L1 cache that the tracks, the table and the
// bins past the window go through: CoREAS of 262144 tracks x 24 antennas x 24000
// bins ran 617 us with 8362 bins and 372 with 8202 in FP64, 609 and 322 in mixed
// precision, also where every sample lies past both.
constexpr uint64_t kPartialWindowBins = 8192;
inline uint32_t window_for(uint64_t longest, int max_bins) {
  uint64_t const most = max_bins > 0 ? static_cast<uint64_t>(max_bins) : 0;
  if (longest <= most) return static_cast<uint32_t>(longest > 0 ? longest : 1);
  uint64_t const part = most < kPartialWindowBins ? most : kPartialWindowBins;
  return static_cast<uint32_t>(part > 0 ? part : 1);
}
// Resident CTAs per SM of the windowed kernel for a window and block size.
int windowed_ctas_per_sm(int window, int threads, bool fixed, Precision precision);

// The precision study's kernel (precision_study.cu): one thread per pair,
// arrival-time arithmetic in FP64, compensated double-FP32 or FP32,
// amplitudes in FP32.
enum class TimeArithmetic : int { kDouble = 0, kDoubleFloat = 1, kFloat = 2 };
cudaError_t launch_study(EventPlan const& event, uint64_t track_bound, bool coreas, bool zhs,
                         bool fixed, TimeArithmetic arithmetic, cudaStream_t stream);

// Output step: decoded CoREAS fields, or ZHS fields -(A[i+1] - A[i]) fs,
// added into `out` (fixed traces when `fixed` is non-null, else `floating`).
cudaError_t launch_output(const long long* fixed, const double* floating, double* out, uint64_t total_bins,
                          const ObserverCache* observers, const double* factors, uint32_t observer_count,
                          uint64_t max_bins, bool differentiate, cudaStream_t stream);

// Fixed-point decode on the device: out[r*bins + i] = in[r*bins + i] * factor(observer).
cudaError_t launch_decode(const long long* fixed, double* out, uint64_t total_bins,
                          const uint64_t* observer_offsets, const double* factors,
                          uint32_t observer_count, uint64_t max_bins, cudaStream_t stream);

}  // namespace c8r

// Host-side checks of the windowed launch plans (no GPU): the work list of
// append_work and the deferred-list storage of deferred_words /
// attach_deferred, the arithmetic that keeps every kernel access of a launch
// inside its buffers.  Prints "ok" or the first failed check; exit status 1
// on a failure.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <utility>
#include <vector>

#include "radio_kernels.cuh"

using namespace c8r;

namespace {

int failures = 0;

void expect(bool ok, char const* what, unsigned long long a = 0, unsigned long long b = 0) {
  if (ok) return;
  std::printf("FAIL %s (%llu, %llu)\n", what, a, b);
  ++failures;
}

EventPlan event(uint32_t chunk, uint32_t chunks, uint32_t observers) {
  EventPlan e;
  std::memset(&e, 0, sizeof e);
  e.chunk_size = chunk;
  e.chunks = chunks;
  e.observer_count[0] = observers;
  e.observer_count[1] = observers;
  e.first_track = 0;
  e.last_track = ~0ull;
  return e;
}

WorkPlan plan_of(std::vector<EventPlan> const& events, int algorithm, uint64_t ctas) {
  WorkPlan plan;
  std::memset(&plan, 0, sizeof plan);
  plan.algorithm = algorithm;
  for (std::size_t i = 0; i < events.size(); ++i) append_work(plan, events[i], ctas, i + 1 == events.size());
  plan.deferred_stride = deferred_list_stride(plan);
  return plan;
}

// Every track of every event falls in exactly one item of the plan, and the
// items' chunks lie inside [first_track, first_track + chunks * chunk_size).
void check_work_list(std::vector<EventPlan> const& events, WorkPlan const& plan) {
  uint64_t items = 0;
  for (uint32_t e = 0; e < plan.event_count; ++e) {
    EventPlan const& p = plan.events[e];
    expect(p.first_item == items, "entries' items are consecutive", p.first_item, items);
    items += static_cast<uint64_t>(p.chunks) * p.observer_count[plan.algorithm];
    expect(p.chunk_size <= kMaxChunkTracks, "chunk within the deferred-entry offset bits", p.chunk_size);
    expect(p.chunk_size <= plan.deferred_stride, "list stride holds a chunk", p.chunk_size, plan.deferred_stride);
  }
  expect(items == plan.total_items, "total items", items, plan.total_items);
  uint64_t want_tracks = 0, got_tracks = 0;
  for (auto const& e : events) want_tracks += static_cast<uint64_t>(e.chunks) * e.chunk_size;
  for (uint32_t e = 0; e < plan.event_count; ++e) {
    EventPlan const& p = plan.events[e];
    uint64_t const stop = p.first_track + static_cast<uint64_t>(p.chunks) * p.chunk_size;
    uint64_t const end = stop < p.last_track ? stop : p.last_track;
    got_tracks += end - p.first_track;
  }
  expect(got_tracks == want_tracks, "every track in one item", got_tracks, want_tracks);
}

// The storage of a launch: the regions the kernels index are disjoint and
// inside deferred_words words.
void check_storage(WorkPlan plan, uint64_t ctas, bool fixed) {
  uint64_t const words = deferred_words(plan, ctas, fixed);
  // only addresses are compared: nothing is read or written through them
  unsigned* const base = reinterpret_cast<unsigned*>(uintptr_t{1} << 20);  // a 16-byte aligned stand-in
  attach_deferred(plan, base, ctas, fixed);
  uint64_t const lists = ctas * plan.deferred_stride;
  if (!two_pass(plan, ctas, fixed)) {
    expect(plan.item_state == nullptr && plan.drain_deferred == nullptr, "one pass: no second-pass storage");
    expect(words == lists, "one pass: the CTAs' lists", words, lists);
    return;
  }
  uint64_t const first = lists;
  expect(plan.drain_deferred == base + first, "second-pass lists follow the first pass's");
  unsigned* const states = reinterpret_cast<unsigned*>(plan.item_state);
  expect(states == base + first + lists, "item states follow the lists");
  expect(plan.drain_next_item == states + plan.total_items * (sizeof(ItemState) / sizeof(unsigned)),
         "counters follow the states");
  expect(static_cast<uint64_t>(plan.drain_next_item - base) + 2 == words, "storage ends at the counters",
         static_cast<uint64_t>(plan.drain_next_item - base) + 2, words);
  expect(reinterpret_cast<uintptr_t>(plan.item_state) % alignof(ItemState) == 0, "item states aligned");
  expect(words <= kTwoPassMaxWords, "two passes within the cap", words, kTwoPassMaxWords);
  // the kernels' last indices: first-pass list of the last CTA, its last
  // entry; second-pass list likewise; the last item's state
  expect((ctas - 1) * plan.deferred_stride + plan.deferred_stride - 1 < first, "first-pass index");
  expect(first + (ctas - 1) * plan.deferred_stride + plan.deferred_stride - 1 < first + lists, "second-pass index");
}

// Length of a launch, in tracks, on CTAs that take items in order as they come
// free: groups of equal items, one group after the other.
struct Items {
  uint64_t count;
  double length;
};
double launch_length(std::vector<Items> const& groups, uint64_t ctas) {
  std::vector<double> busy(ctas, 0.);
  bool first = true;
  for (Items const& g : groups) {
    uint64_t n = g.count;
    if (first) {
      for (double& b : busy) b = static_cast<double>(n / ctas) * g.length;
      n %= ctas;
      std::make_heap(busy.begin(), busy.end(), std::greater<double>());
    }
    first = false;
    for (uint64_t i = 0; i < n; ++i) {
      std::pop_heap(busy.begin(), busy.end(), std::greater<double>());
      busy.back() += g.length;
      std::push_heap(busy.begin(), busy.end(), std::greater<double>());
    }
  }
  return *std::max_element(busy.begin(), busy.end());
}

// Chunks of `chunk` tracks over `count`, the last one perhaps shorter.
void append_chunks(std::vector<Items>& groups, uint64_t count, uint64_t chunk, uint64_t per, double item) {
  if (count == 0) return;
  groups.push_back({count / chunk * per, item + static_cast<double>(chunk)});
  if (count % chunk) groups.push_back({per, item + static_cast<double>(count % chunk)});
}

double planned_length(uint64_t count, uint64_t per, uint64_t ctas, uint64_t chunk, bool tail, double item) {
  uint64_t const chunks = (count + chunk - 1) / chunk;
  TailSplit const split = tail ? split_tail(chunks, chunk, per, ctas) : TailSplit{chunks, 0};
  uint64_t const head = split.head < chunks ? split.head * chunk : count;
  std::vector<Items> groups;
  append_chunks(groups, head, chunk, per, item);
  append_chunks(groups, count - head, split.small, per, item);
  return launch_length(groups, ctas);
}

// The automatic chunks of 1 to 300 antennas and 1e3 to 4e7 tracks: the launch is
// within 15% and one item's window of the shortest one over every number of chunks
// that the deferred lists allow, and its lists hold no more than 16 items a CTA
// would or 262144 tracks.
void check_auto_chunk(uint64_t ctas) {
  for (uint64_t per : {1, 2, 3, 5, 8, 16, 30, 48, 64, 100, 147, 148, 149, 160, 240, 300})
    for (uint64_t count : {1000, 4097, 20000, 100003, 300000, 1000000, 2000000, 4000000, 6000000, 9500000, 40000000})
      for (double item : {item_cost(900, true, 1), item_cost(8192, false, 1), item_cost(4096, true, 4)}) {
        uint64_t const chunk = auto_chunk(count, per, ctas, item);
        uint64_t const share = (count * per + 16 * ctas - 1) / (16 * ctas);
        uint64_t const longest = share > 262144 ? share : 262144;
        expect(chunk >= kTrackTile && chunk % kTrackTile == 0, "whole track tiles", chunk, count);
        expect(chunk <= track_capacity(longest), "a chunk the deferred lists allow", chunk, longest);
        uint64_t const chunks = (count + chunk - 1) / chunk;
        double const length =
            planned_length(count, per, ctas, chunk,
                                             tail_pays(event(static_cast<uint32_t>(chunk), static_cast<uint32_t>(chunks),
                                                             static_cast<uint32_t>(per)), 0, ctas, item), item);
        double shortest = 1e300;
        for (uint64_t c = (count + longest - 1) / longest; c <= 600; c += c < 200 ? 1 : 10) {
          uint64_t const other = track_capacity((count + c - 1) / c);
          if (other < 256) break;
          for (bool tail : {false, true}) {
            double const l = planned_length(count, per, ctas, other, tail, item);
            if (l < shortest) shortest = l;
          }
        }
        if (shortest == 1e300) continue;
        expect(length <= 1.15 * shortest + item, "launch length within 15% and a window of the shortest",
               count * 1000 + per, chunk);
      }
}

// Events of a batched launch, cut for their share of the GPU: the items' windows add
// at most a third to the work that one item an antenna would be, or an item's
// length a CTA in all where few events share the launch, and no chunk passes what
// the whole launch's lists are sized for.
void check_batch(std::vector<std::pair<uint64_t, uint64_t>> const& events, double item, uint64_t ctas) {
  double work = 0., planned = 0.;
  for (auto const& e : events) work += static_cast<double>(e.second) * (static_cast<double>(e.first) + item);
  for (auto const& e : events) {
    uint64_t const chunk = batch_chunk(e.first, e.second, ctas, item, work);
    uint64_t const share = (e.first * e.second + 16 * ctas - 1) / (16 * ctas);
    expect(chunk <= track_capacity(share > 262144 ? share : 262144), "a batched chunk the lists allow", chunk);
    planned += static_cast<double>((e.first + chunk - 1) / chunk * e.second) * item +
               static_cast<double>(e.first * e.second);
  }
  expect(planned <= 4. / 3. * work + static_cast<double>(8 * ctas) * item, "windows of a batched launch",
         static_cast<uint64_t>(planned), static_cast<uint64_t>(work));
}

// The automatic kernel at measured points (us of the direct and of the windowed kernel):
// the choice is within a quarter of the faster one, and never changes from 16384 tracks on.
void check_kernel_choice() {
  struct Point {
    uint64_t tracks, antennas;
    bool zhs;
    uint32_t refinement;
    bool fixed, fp64, whole;
    double direct, windowed;
  };
  Point const points[] = {
      {4096, 16, true, 1, true, true, true, 175., 78.},
      {256, 160, true, 1, true, true, true, 221., 88.},
      {1024, 300, true, 1, true, false, true, 105., 71.},
      {512, 48, true, 1, false, true, true, 98., 57.},
      {512, 160, false, 1, true, true, true, 29., 45.},
      {16000, 160, false, 1, true, true, true, 227., 156.},
      {4096, 48, false, 1, false, false, true, 34., 36.},
      {4096, 16, true, 4, true, true, true, 259., 161.},
      {4096, 160, true, 4, true, true, true, 472., 781.},
      {16000, 300, true, 16, true, true, true, 3594., 6497.},
      {8192, 160, true, 16, true, false, true, 1753., 1706.},
      {8192, 160, true, 16, true, false, false, 1854., 4120.},
      {4096, 160, true, 3, false, true, true, 228., 412.},
      {2048, 16, true, 2, false, false, true, 75., 60.},
      {16000, 5, true, 3, true, true, false, 278., 156.},
  };
  for (Point const& p : points) {
    double const chosen =
        direct_pays(p.tracks, p.antennas, p.zhs, p.refinement, p.fixed, p.fp64, p.whole) ? p.direct : p.windowed;
    expect(chosen <= 1.25 * (p.direct < p.windowed ? p.direct : p.windowed), "the faster kernel", p.tracks, p.antennas);
  }
  for (uint64_t tracks : {16384, 100000, 10000000})
    for (uint32_t refinement : {1, 4, 64})
      for (int flags = 0; flags < 16; ++flags)
        expect(!direct_pays(tracks, 300, flags & 1, refinement, flags & 2, flags & 4, flags & 8), "windowed", tracks);
  expect(direct_pays(1, 1, true, 1, true, true, true) && direct_pays(255, 300, false, 1, false, false, false), "direct");
}

// The window is the whole trace while it fits; of a longer one the part that leaves
// the kernel inside the shared memory that does not cut into the L1 cache.
void check_windows() {
  for (int most : {1, 4096, 8277, 8362, 9000})
    for (uint64_t longest : {1, 2, 4096, 8192, 8277, 8278, 8362, 8363, 24000, 1 << 20}) {
      uint32_t const window = window_for(longest, most);
      expect(window >= 1 && window <= static_cast<uint64_t>(most) && window <= longest, "window fits", window, most);
      if (longest <= static_cast<uint64_t>(most))
        expect(window == longest, "the whole trace", window, longest);
      else
        expect(24ull * window + 2048 <= 196 * 1024, "a part beside the full L1", window, longest);
    }
}

}  // namespace

int main() {
  check_kernel_choice();
  check_windows();
  for (double item : {item_cost(900, true, 1), item_cost(8192, false, 1)}) {
    check_batch(std::vector<std::pair<uint64_t, uint64_t>>(64, {1500, 16}), item, 148);
    check_batch(std::vector<std::pair<uint64_t, uint64_t>>(64, {300, 16}), item, 148);
    check_batch(std::vector<std::pair<uint64_t, uint64_t>>(32, {5000, 40}), item, 148);
    check_batch(std::vector<std::pair<uint64_t, uint64_t>>(16, {1000000, 160}), item, 148);
    check_batch({{5000000, 160}, {1000, 16}, {20000, 300}, {300, 5}}, item, 148);
    check_batch({{100000, 16}}, item, 148);
  }
  check_auto_chunk(148);
  // the 1e7 x 160 workload's ZHS launch, a served round, a batched launch of
  // several events, small launches, and one past the two-pass cap
  struct Case {
    std::vector<EventPlan> events;
    uint64_t ctas;
  };
  std::vector<Case> cases = {
      {{event(666688, 15, 160)}, 148},
      {{event(131072, 8, 64), event(131072, 3, 300), event(131072, 1, 16)}, 148},
      {{event(524288, 20, 300), event(524288, 4, 16), event(524288, 39, 120)}, 148},
      {{event(8192, 1, 16)}, 148},
      {{event(256, 79, 16)}, 148},
      {{event(1u << 30, 64, 300)}, 148},  // 2e13 pairs: one pass
  };
  for (auto const& c : cases) {
    for (int algorithm = 0; algorithm < 2; ++algorithm) {
      uint64_t ctas = c.ctas;
      WorkPlan plan = plan_of(c.events, algorithm, ctas);
      if (ctas > plan.total_items) ctas = plan.total_items;
      check_work_list(c.events, plan);
      for (bool fixed : {false, true}) {
        check_storage(plan, ctas, fixed);
        bool const expect_two = fixed && algorithm == 1 && two_pass_words(plan, ctas) <= kTwoPassMaxWords;
        expect(two_pass(plan, ctas, fixed) == expect_two, "two passes exactly for fixed ZHS within the cap");
      }
    }
  }
  {
    WorkPlan huge = plan_of({event(1u << 30, 64, 300)}, 1, 148);
    expect(!two_pass(huge, 148, true), "a launch past the cap runs one pass");
  }
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}

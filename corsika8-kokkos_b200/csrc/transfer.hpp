// transfer.hpp — device results into pageable host memory through a ring of
// pinned slots, emptied by several host threads.
//
// A caller's fresh output arrays are pageable and mostly untouched: a plain
// cudaMemcpy into them runs at the speed of one thread that copies out of the
// driver's staging buffer and takes every page fault (63 MB of traces: 14.3 ms).
// Here the copy engine fills slots while up to kWorkers threads copy the filled
// ones out, so the faults and the copies run in parallel (the same 63 MB: 4.8
// ms).  A call's threads end with it.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <memory>
#include <system_error>
#include <thread>
#include <vector>

namespace c8r {
namespace {

// Where a caller's result buffer lies: ordinary host memory (through the slots),
// memory that the copy engine writes (page-locked, managed), or device memory,
// which no result is copied to.
enum class ResultMemory { kPageable, kDirect, kDevice };
inline ResultMemory result_memory(void const* p) {
  cudaPointerAttributes attributes{};
  if (cudaPointerGetAttributes(&attributes, p) != cudaSuccess) {
    cudaGetLastError();
    return ResultMemory::kPageable;
  }
  if (attributes.type == cudaMemoryTypeDevice) return ResultMemory::kDevice;
  return attributes.type == cudaMemoryTypeUnregistered ? ResultMemory::kPageable : ResultMemory::kDirect;
}

class SlotRing {
 public:
  static constexpr std::size_t kSlotBytes = std::size_t{1} << 19;
  static constexpr std::size_t kSlots = 8;
  static constexpr unsigned kWorkers = 6;
  // below this much a call copies on its own thread (2.4 MB took 180 us longer with
  // threads, 9.4 MB 2 ms less); above it, one for each kBytesPerWorker
  static constexpr std::size_t kThreadedBytes = 5u << 20, kBytesPerWorker = 2u << 20;

  struct Segment {
    void* destination;
    std::size_t bytes;
  };

  SlotRing() = default;
  SlotRing(SlotRing const&) = delete;
  SlotRing& operator=(SlotRing const&) = delete;
  ~SlotRing() {
    for (cudaEvent_t e : filled_) cudaEventDestroy(e);
  }

  // Page-locked memory for the slots; the owner keeps it and leaves it alone
  // while run() is under way.
  cudaError_t use(void* pinned, std::size_t bytes) {
    for (std::size_t at = 0; at + kSlotBytes <= bytes && slots_.size() < kSlots; at += kSlotBytes) {
      cudaEvent_t e = nullptr;
      cudaError_t const err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
      if (err != cudaSuccess) return err;
      filled_.push_back(e);
      slots_.push_back(static_cast<unsigned char*>(pinned) + at);
    }
    return cudaSuccess;
  }
  bool usable() const { return !slots_.empty(); }

  // Fills the segments in order: issue(segment, offset, bytes, slot) queues on
  // `stream` the work that writes bytes [offset, offset + bytes) of a segment
  // into `slot`, emit(segment, offset, bytes, slot) moves them on to the segment's
  // destination.  Returns once everything has been copied out.  Only the calling
  // thread calls the CUDA runtime: a new thread's device is 0, whatever the owner's,
  // and its first call costs as much as the copy of a megabyte.
  template <class Issue, class Emit>
  cudaError_t run(std::vector<Segment> const& segments, cudaStream_t stream, Issue issue, Emit emit) {
    std::vector<Piece> pieces;
    std::size_t total = 0;
    for (std::size_t s = 0; s < segments.size(); ++s)
      for (std::size_t at = 0; at < segments[s].bytes; at += kSlotBytes) {
        pieces.push_back({s, at, std::min(kSlotBytes, segments[s].bytes - at)});
        total += pieces.back().bytes;
      }
    std::size_t const n = pieces.size(), depth = slots_.size();
    auto fill = [&](std::size_t i) {
      Piece const& p = pieces[i];
      cudaError_t const err = issue(p.segment, p.offset, p.bytes, slots_[i % depth]);
      return err != cudaSuccess ? err : cudaEventRecord(filled_[i % depth], stream);
    };
    auto empty = [&](std::size_t i) {
      Piece const& p = pieces[i];
      emit(p.segment, p.offset, p.bytes, static_cast<void const*>(slots_[i % depth]));
    };
    unsigned const cores = std::max(1u, std::thread::hardware_concurrency() / 2);
    Shared shared(n);
    Workers workers(shared);
    if (total >= kThreadedBytes && depth > 1) {
      std::size_t const wanted = std::min<std::size_t>({kWorkers, cores, total / kBytesPerWorker});
      for (std::size_t k = 0; k < wanted; ++k)
        if (!workers.start([&] { drain(shared, n, empty); })) break;
    }
    for (std::size_t issued = 0, filled = 0; filled < n;) {
      // a slot takes its next piece when its last one is out
      if (issued < n && (issued < depth || shared.done[issued - depth].load(std::memory_order_acquire))) {
        if (cudaError_t const err = fill(issued)) return err;
        ++issued;
      } else if (filled < issued) {
        if (cudaError_t const err = cudaEventSynchronize(filled_[filled % depth])) return err;
        if (workers.none()) {
          empty(filled);
          shared.done[filled].store(true, std::memory_order_relaxed);
        }
        shared.filled.store(++filled, std::memory_order_release);
      } else {
        std::this_thread::yield();
      }
    }
    workers.join();
    return cudaSuccess;
  }
  // The same, the bytes copied as they are.
  template <class Issue>
  cudaError_t run(std::vector<Segment> const& segments, cudaStream_t stream, Issue issue) {
    return run(segments, stream, issue, [&](std::size_t k, std::size_t offset, std::size_t bytes, void const* slot) {
      std::memcpy(static_cast<unsigned char*>(segments[k].destination) + offset, slot, bytes);
    });
  }

 private:
  struct Piece {
    std::size_t segment, offset, bytes;
  };
  struct Shared {
    explicit Shared(std::size_t n) : done(new std::atomic<bool>[n ? n : 1]) {
      for (std::size_t i = 0; i < n; ++i) done[i].store(false);
    }
    std::atomic<std::size_t> filled{0}, next{0};
    std::atomic<bool> stop{false};
    std::unique_ptr<std::atomic<bool>[]> done;
  };
  // Joins its threads on every way out; what has not been filled by then never is.
  class Workers {
   public:
    explicit Workers(Shared& shared) : shared_(shared) {}
    ~Workers() {
      shared_.stop.store(true);
      join();
    }
    template <class F>
    bool start(F body) {
      try {
        threads_.emplace_back(body);
        return true;
      } catch (std::system_error const&) {
        return false;  // fewer threads
      }
    }
    bool none() const { return threads_.empty(); }
    void join() {
      for (std::thread& t : threads_) t.join();
      threads_.clear();
    }

   private:
    Shared& shared_;
    std::vector<std::thread> threads_;
  };
  template <class Empty>
  static void drain(Shared& shared, std::size_t n, Empty const& empty) {
    for (;;) {
      std::size_t const i = shared.next.fetch_add(1);
      if (i >= n) return;
      while (shared.filled.load(std::memory_order_acquire) <= i) {
        if (shared.stop.load()) return;
        std::this_thread::yield();
      }
      empty(i);
      shared.done[i].store(true, std::memory_order_release);
    }
  }

  std::vector<unsigned char*> slots_;
  std::vector<cudaEvent_t> filled_;
};

// One result: device memory and where it goes.
struct ResultCopy {
  void* to;
  void const* from;
  std::size_t bytes;
};
// Copies results after the stream's earlier work: page-locked and managed
// destinations each by one copy (in flight on return), pageable ones through the
// slots.  Device memory is refused: the slots are emptied by host threads.
inline cudaError_t copy_results(SlotRing& ring, std::vector<ResultCopy> const& results, cudaStream_t stream) {
  std::vector<SlotRing::Segment> pageable;
  std::vector<unsigned char const*> from;
  for (ResultCopy const& r : results) {
    ResultMemory const memory = result_memory(r.to);
    if (memory == ResultMemory::kDevice) return cudaErrorInvalidValue;
    if (memory == ResultMemory::kPageable && ring.usable()) {
      pageable.push_back({r.to, r.bytes});
      from.push_back(static_cast<unsigned char const*>(r.from));
    } else if (cudaError_t const err = cudaMemcpyAsync(r.to, r.from, r.bytes, cudaMemcpyDeviceToHost, stream)) {
      return err;
    }
  }
  if (pageable.empty()) return cudaSuccess;
  return ring.run(pageable, stream, [&](std::size_t k, std::size_t offset, std::size_t bytes, void* slot) {
    return cudaMemcpyAsync(slot, from[k] + offset, bytes, cudaMemcpyDeviceToHost, stream);
  });
}

}  // namespace
}  // namespace c8r

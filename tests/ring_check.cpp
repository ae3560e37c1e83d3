// Host-side check (no GPU, no CUDA library) of the result copies of transfer.hpp
// against a runtime of its own: "device" buffers are host memory, copies happen
// when the stream's events are waited for, and every call notes the device of the
// thread that made it.  Prints "ok" or the first failed check; exit status 1 on a
// failure.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <vector>

namespace {

constexpr int kOwner = 3;  // the device of the accumulator or server
thread_local int t_device = 0;
std::atomic<int> wrong_device{0}, event_waits{0}, runtime_copies{0};
std::mutex mu;
struct Copy {
  void* to;
  void const* from;
  std::size_t bytes;
};
std::deque<Copy> queued;
std::map<void const*, cudaMemoryType> kinds;  // pointers that are not pageable

void note_device() {
  if (t_device != kOwner) ++wrong_device;
}
void finish_queued() {
  std::lock_guard<std::mutex> lock(mu);
  for (; !queued.empty(); queued.pop_front()) std::memcpy(queued.front().to, queued.front().from, queued.front().bytes);
}

}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* device) {
  *device = t_device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int device) {
  t_device = device;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* event, unsigned) {
  *event = reinterpret_cast<cudaEvent_t>(new char);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t event) {
  delete reinterpret_cast<char*>(event);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) {
  note_device();
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) {
  note_device();
  ++event_waits;
  finish_queued();
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, void const* from, std::size_t bytes, cudaMemcpyKind, cudaStream_t) {
  note_device();
  ++runtime_copies;
  std::lock_guard<std::mutex> lock(mu);
  queued.push_back({to, from, bytes});
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* attributes, void const* p) {
  *attributes = {};
  auto const it = kinds.find(p);
  attributes->type = it == kinds.end() ? cudaMemoryTypeUnregistered : it->second;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

#include "transfer.hpp"

using c8r::SlotRing;

namespace {

int failures = 0;
void expect(bool ok, char const* what) {
  if (ok) return;
  std::printf("FAIL %s\n", what);
  ++failures;
}

std::vector<unsigned char> pattern(std::size_t n, unsigned seed) {
  std::vector<unsigned char> out(n);
  for (std::size_t i = 0; i < n; ++i) out[i] = static_cast<unsigned char>((i * 2654435761u + seed) >> 13);
  return out;
}

// Copies of several sizes reach their destinations whole, and every runtime call is
// made on the owner's device (the copying threads, whose device is 0, make none).
// A copy that fails on its way ends the call with its error.
void check_copies(SlotRing& ring) {
  for (std::size_t bytes : {std::size_t{1}, SlotRing::kSlotBytes, SlotRing::kSlotBytes + 1, std::size_t{23} << 20}) {
    std::vector<unsigned char> const a = pattern(bytes, 1), b = pattern(bytes / 2 + 1, 2);
    std::vector<unsigned char> x(a.size()), y(b.size());
    std::vector<SlotRing::Segment> const out{{x.data(), x.size()}, {y.data(), y.size()}};
    unsigned char const* const from[] = {a.data(), b.data()};
    cudaError_t const err = ring.run(out, nullptr, [&](std::size_t k, std::size_t at, std::size_t n, void* slot) {
      return cudaMemcpyAsync(slot, from[k] + at, n, cudaMemcpyDeviceToHost, nullptr);
    });
    expect(err == cudaSuccess, "copy returns success");
    expect(x == a && y == b, "copies arrive whole");
  }
  for (std::size_t bad : {0, 3, 20, 45}) {
    std::vector<unsigned char> const a = pattern(std::size_t{23} << 20, 5);
    std::vector<unsigned char> x(a.size());
    std::size_t pieces = 0;
    cudaError_t const err = ring.run({{x.data(), x.size()}}, nullptr,
                                     [&](std::size_t, std::size_t at, std::size_t n, void* slot) {
                                       if (pieces++ == bad) return cudaErrorUnknown;
                                       return cudaMemcpyAsync(slot, a.data() + at, n, cudaMemcpyDeviceToHost, nullptr);
                                     });
    expect(err == cudaErrorUnknown, "a failed copy ends the call");
    finish_queued();
  }
  expect(event_waits > 0, "the copies waited for their slots");
  expect(wrong_device == 0, "every call on the owner's device");
}

// Page-locked results take one copy each, straight to them; pageable ones go
// through the slots; a device pointer among them is an error.
void check_routes(SlotRing& ring) {
  std::size_t const bytes = 3 * SlotRing::kSlotBytes + 5;
  std::vector<unsigned char> const a = pattern(bytes, 3), b = pattern(bytes, 4);
  std::vector<unsigned char> x(bytes), y(bytes);
  kinds[x.data()] = cudaMemoryTypeHost;
  runtime_copies = 0;
  expect(c8r::copy_results(ring, {{x.data(), a.data(), bytes}}, nullptr) == cudaSuccess, "page-locked result");
  expect(runtime_copies == 1, "page-locked: one copy");
  finish_queued();
  expect(x == a, "page-locked result arrives");
  runtime_copies = 0;
  expect(c8r::copy_results(ring, {{x.data(), b.data(), bytes}, {y.data(), a.data(), bytes}}, nullptr) == cudaSuccess,
         "results of both kinds");
  expect(runtime_copies == 1 + 4, "one copy and four slots");
  finish_queued();
  expect(x == b && y == a, "results of both kinds arrive");
  kinds[x.data()] = cudaMemoryTypeDevice;
  expect(c8r::copy_results(ring, {{x.data(), a.data(), bytes}}, nullptr) == cudaErrorInvalidValue, "device memory");
  expect(x == b, "device memory untouched");
  kinds.clear();
}

// A result buffer's memory decides its route.
void check_memory() {
  char pageable, locked, managed, device;
  kinds[&locked] = cudaMemoryTypeHost;
  kinds[&managed] = cudaMemoryTypeManaged;
  kinds[&device] = cudaMemoryTypeDevice;
  expect(c8r::result_memory(&pageable) == c8r::ResultMemory::kPageable, "ordinary memory through the slots");
  expect(c8r::result_memory(&locked) == c8r::ResultMemory::kDirect, "page-locked memory directly");
  expect(c8r::result_memory(&managed) == c8r::ResultMemory::kDirect, "managed memory directly");
  expect(c8r::result_memory(&device) == c8r::ResultMemory::kDevice, "device memory refused");
}

}  // namespace

int main() {
  cudaSetDevice(kOwner);
  check_memory();
  std::vector<unsigned char> slots(4 * SlotRing::kSlotBytes);
  {
    SlotRing ring;
    expect(ring.use(slots.data(), slots.size()) == cudaSuccess, "slots");
    check_copies(ring);
    check_routes(ring);
  }
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}

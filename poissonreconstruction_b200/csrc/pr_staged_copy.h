// Copies between pageable host memory and the device through pinned slots, by several host threads.
// Host code only.
//
// The driver's own path is one thread that stages through a pinned buffer; out of the device it also faults
// in the pages of a fresh destination.  Here host threads copy pieces to and from pinned slots
// while the DMAs of other slots run.  The calling thread issues every DMA; the helpers call no CUDA
// function, since a stream handle can name another stream in another thread (cudaStreamPerThread).  Beside
// helpers the calling thread copies nothing itself: they would wait for it (134 MB out in 13.8 ms, not 9.9).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <memory>
#include <thread>
#include <vector>

namespace pr {

constexpr size_t kStageSlot = size_t(1) << 20;
constexpr int kStageThreads = 4, kStageSlots = 2 * kStageThreads;

// Slots with an event each, made by the first copy that uses them: eight of 1 MiB in memory of their own, or
// up to eight of another size in memory of the owner's.
struct StageSlots {
  unsigned char* mem = nullptr;
  size_t size = 0;   // of a slot
  size_t count = 0;  // of slots
  bool lent = false;
  std::vector<cudaEvent_t> events;
  // false: there is no pinned memory (or no event) for them
  bool make() {
    if (!mem && cudaMallocHost(reinterpret_cast<void**>(&mem), kStageSlots * kStageSlot) != cudaSuccess) mem = nullptr;
    size = kStageSlot;
    count = kStageSlots;
    return make_events();
  }
  // the same in pinned memory that outlives them
  bool lend(unsigned char* memory, size_t slot, size_t slots) {
    mem = memory;
    size = slot;
    count = slots;
    lent = true;
    return make_events();
  }
  bool make_events() {
    cudaEvent_t e = nullptr;
    while (mem && events.size() < count && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess)
      events.push_back(e);
    if (mem && events.size() == count) return true;
    cudaGetLastError();
    return false;
  }
  void free() {
    if (mem && !lent) cudaFreeHost(mem);
    for (cudaEvent_t e : events) cudaEventDestroy(e);
    mem = nullptr;
    lent = false;
    events.clear();
  }
};

// The pieces of one copy between host memory and the slots (piece k in slot k mod their number), shared by
// the copying threads: pieces [0, avail) may be moved, next is the first that no thread has taken.
struct StagedPieces {
  const size_t pieces;
  std::atomic<size_t> avail{0}, next{0};
  std::atomic<bool> stop{false};
  std::unique_ptr<std::atomic<bool>[]> moved;
  explicit StagedPieces(size_t n) : pieces(n), moved(new std::atomic<bool>[n]) {
    for (size_t k = 0; k < n; ++k) moved[k].store(false, std::memory_order_relaxed);
  }
  // takes a piece and moves it; false if there is none for now
  template <typename F>
  bool move_one(F move) {
    size_t k = next.load(std::memory_order_relaxed);
    do {
      if (k >= avail.load(std::memory_order_acquire)) return false;
    } while (!next.compare_exchange_weak(k, k + 1, std::memory_order_relaxed));
    move(k);
    moved[k].store(true, std::memory_order_release);
    return true;
  }
  bool is_moved(size_t k) const { return moved[k].load(std::memory_order_acquire); }
  // a helper thread's work
  template <typename F>
  void help(F move) {
    while (!stop.load(std::memory_order_relaxed) && next.load(std::memory_order_relaxed) < pieces)
      if (!move_one(move)) std::this_thread::yield();
  }
};

// Runs drive(whether this thread is alone) in this thread, beside nt helpers that move pieces (none for one).
template <typename Drive, typename Move>
cudaError_t with_helpers(StagedPieces& q, int nt, Drive drive, Move move) {
  std::vector<std::thread> th;
  try {
    for (int i = 0; nt > 1 && i < nt; ++i) th.emplace_back([&q, move] { q.help(move); });
  } catch (...) {  // no more threads: those that there are share the pieces
  }
  const cudaError_t e = drive(th.empty());
  q.stop = true;
  for (auto& t : th) t.join();
  return e;
}

// Copies in pieces through the slots (`out`: device to host) with nt copying threads, one: the calling thread
// by itself.  When it returns the destination is complete (out), or the source may be reused while the last
// DMAs still run on the stream (in).  After an error DMAs may still run, to or from the slots.
inline cudaError_t staged_copy(cudaStream_t stream, StageSlots& st, unsigned char* dev, unsigned char* host,
                               size_t bytes, int nt, bool out) {
  const size_t size = st.size, count = st.count;
  StagedPieces q((bytes + size - 1) / size);
  unsigned char* const slots = st.mem;
  auto length = [bytes, size](size_t k) { return std::min(size, bytes - k * size); };
  auto slot = [slots, size, count](size_t k) { return slots + (k % count) * size; };
  auto move = [=](size_t k) {
    if (out) std::memcpy(host + k * size, slot(k), length(k));
    else std::memcpy(slot(k), host + k * size, length(k));
  };
  auto drive = [&](bool alone) -> cudaError_t {
    size_t issued = 0;  // pieces whose DMA was issued
    size_t done = 0;    // out: pieces whose DMA has arrived; in: pieces whose slot is free of earlier DMAs
    for (;;) {
      if (issued < q.pieces && (out ? issued < count || q.is_moved(issued - count) : q.is_moved(issued))) {
        const size_t k = issued % count, at = issued * size;
        cudaError_t e = cudaSuccess;
        if (out && issued < count) e = cudaEventSynchronize(st.events[k]);  // an earlier copy's DMA from the slot
        if (e == cudaSuccess)
          e = out ? cudaMemcpyAsync(slot(issued), dev + at, length(issued), cudaMemcpyDeviceToHost, stream)
                  : cudaMemcpyAsync(dev + at, slot(issued), length(issued), cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaEventRecord(st.events[k], stream);
        if (e != cudaSuccess) return e;
        ++issued;
        continue;
      }
      if (out ? done < issued : done < q.pieces && done < issued + count) {
        const cudaError_t e = cudaEventQuery(st.events[done % count]);
        if (e == cudaSuccess) {
          q.avail.store(++done, std::memory_order_release);
          continue;
        }
        if (e != cudaErrorNotReady) return e;
        cudaGetLastError();
      }
      if (alone && q.move_one(move)) continue;
      if (!out && issued == q.pieces) return cudaSuccess;
      if (out && done == q.pieces) {
        size_t k = q.pieces > count ? q.pieces - count : 0;  // the earlier ones' slots were reused
        while (k < q.pieces && q.is_moved(k)) ++k;
        if (k == q.pieces) return cudaSuccess;
      }
      std::this_thread::yield();
    }
  };
  return with_helpers(q, nt, drive, move);
}

}  // namespace pr

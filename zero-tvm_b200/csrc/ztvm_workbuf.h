// Work buffers of the calls that need device memory of their own (the expert-sorted plan of the grouped MoE matmul, the f32
// rows of the fused FFN's two-launch form, the counters of a step's matmuls in one launch), host side.
//
// Calls that may overlap never share a buffer:
//   * a call outside any capture uses its stream's buffer (at most kWorkStreams of them per purpose; a further stream takes
//     the one that was used least recently, after a device synchronisation);
//   * a captured call uses a buffer that belongs to the graph being captured (one per stream of the capture). Later calls
//     neither free, grow nor write it, so the graph stays valid whatever the context does next, and two graphs may be
//     replayed side by side. The first kKeptBytes of such buffers stay with their graphs for the context's life. A further
//     one goes back to the context when the graph and every executable made from it are gone, and the next capture takes it
//     over: a user object of the graph says so, which costs each replay some 2 to 5 us (recorded 3-bit MoE blocks, 8 tokens of
//     54 experts: 72.6 us a step without, 76.9 us with), so the few graphs that most programs have are spared it.
// Nothing has to be allocated ahead of a capture: allocations are made in relaxed capture mode.
#pragma once
#include <atomic>
#include <cstdint>
#include <memory>
#include <new>
#include <vector>

#include <cuda_runtime.h>

namespace ztvm {

// What the plan in a buffer was built from.
struct PlanKey {
  const void *ids = nullptr, *segs = nullptr;
  uint32_t tokens = 0, slots = 0, stride = 0, tile_rows = 0, experts = 0;
  bool operator==(const PlanKey& o) const {
    return ids == o.ids && segs == o.segs && tokens == o.tokens && slots == o.slots && stride == o.stride && tile_rows == o.tile_rows &&
           experts == o.experts;
  }
};

struct WorkBuf {
  void* p = nullptr;
  size_t bytes = 0;
  int purpose = 0;
  unsigned long long capture = 0;   // capture it was made for, 0: calls outside captures
  unsigned long long stream = 0;    // stream id, inside a capture the handle
  std::atomic<bool> held{false};    // a graph refers to it, or did: `held` falls only for those with a user object
  uint64_t last_use = 0;
  PlanKey plan;                     // plan.ids == nullptr: no plan
  bool fresh = false;               // (re)allocated since its user last looked
};

class WorkBufs {
 public:
  static constexpr int kWorkStreams = 4;
  static constexpr size_t kKeptBytes = 64u << 20;
  enum Purpose { kPlan, kFfnRows, kStep };

  // A buffer of at least `need` bytes for a call on `st`.
  cudaError_t get(Purpose purpose, size_t need, cudaStream_t st, WorkBuf** out) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0, stream = reinterpret_cast<uintptr_t>(st);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamGetCaptureInfo(st, &status, &capture, &graph, nullptr, nullptr);
    if (e != cudaSuccess) return e;
    if (status == cudaStreamCaptureStatusInvalidated) return cudaErrorStreamCaptureInvalidated;
    if (status == cudaStreamCaptureStatusActive) return get_captured(purpose, need, stream, capture, graph, out);
    if ((e = cudaStreamGetId(st, &stream)) != cudaSuccess) return e;     // (a handle may come back as another stream)
    WorkBuf *mine = nullptr, *oldest = nullptr;
    int streams = 0;
    for (auto& b : bufs_) {
      if (b->purpose != purpose || b->capture) continue;
      ++streams;
      if (b->stream == stream) mine = b.get();
      if (!oldest || b->last_use < oldest->last_use) oldest = b.get();
    }
    if (!mine && streams >= kWorkStreams) {
      if ((e = cudaDeviceSynchronize()) != cudaSuccess) return e;
      mine = oldest;
      mine->plan = PlanKey();
    }
    if (!mine) {
      mine = add(purpose);
      if (!mine) return cudaErrorMemoryAllocation;
    }
    mine->stream = stream;
    mine->last_use = ++uses_;
    if (mine->bytes < need) {
      if (mine->p && (e = cudaStreamSynchronize(st)) != cudaSuccess) return e;     // only calls on this stream use it
      // half as much again as asked for, so that a slowly growing size does not allocate every time
      if ((e = renew(mine, need + need / 2)) != cudaSuccess) return e;
    }
    *out = mine;
    return cudaSuccess;
  }

  void drop_plans() {
    for (auto& b : bufs_) b->plan.ids = nullptr;
  }

  void free_all() {
    for (auto& b : bufs_)
      if (b->p) cudaFree(b->p);
    bufs_.clear();
  }

 private:
  cudaError_t get_captured(Purpose purpose, size_t need, unsigned long long stream, unsigned long long capture, cudaGraph_t graph, WorkBuf** out) {
    WorkBuf* idle = nullptr;                 // the smallest that fits of those whose graphs are gone, else any of them
    for (auto& b : bufs_) {
      if (b->purpose != purpose || !b->capture) continue;
      if (b->held.load(std::memory_order_acquire)) {
        if (b->capture == capture && b->stream == stream && b->bytes >= need) { *out = b.get(); return cudaSuccess; }
      } else if (!idle || (idle->bytes < need ? b->bytes > idle->bytes : b->bytes >= need && b->bytes < idle->bytes)) {
        idle = b.get();
      }
    }
    cudaError_t e = cudaSuccess;
    if (!idle) {
      idle = add(purpose);
      if (!idle) return cudaErrorMemoryAllocation;
      idle->capture = capture;               // (also where the allocation fails: never a buffer of plain calls)
    }
    if (idle->bytes < need) {
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      if ((e = cudaThreadExchangeStreamCaptureMode(&mode)) != cudaSuccess) return e;
      e = renew(idle, (need + 4095) / 4096 * 4096);
      cudaThreadExchangeStreamCaptureMode(&mode);
      if (e != cudaSuccess) return e;
    }
    if (kept_ + idle->bytes <= kKeptBytes) {
      kept_ += idle->bytes;
      idle->held.store(true, std::memory_order_release);
    } else if ((e = let_go_with(graph, idle)) != cudaSuccess) {
      return e;
    }
    idle->capture = capture;
    idle->stream = stream;
    idle->plan = PlanKey();
    *out = idle;
    return cudaSuccess;
  }

  // The buffer is let go by whatever thread destroys the last of the graph and its executables, possibly after the
  // context, so the note outlives both.
  cudaError_t let_go_with(cudaGraph_t graph, WorkBuf* buf) {
    std::shared_ptr<WorkBuf>* hold = nullptr;
    for (auto& b : bufs_)
      if (b.get() == buf) hold = new (std::nothrow) std::shared_ptr<WorkBuf>(b);
    if (!hold) return cudaErrorMemoryAllocation;
    buf->held.store(true, std::memory_order_release);
    cudaUserObject_t obj = nullptr;
    cudaError_t e = cudaUserObjectCreate(&obj, hold, &WorkBufs::let_go, 1, cudaUserObjectNoDestructorSync);
    if (e != cudaSuccess) { let_go(hold); return e; }
    e = cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove);
    if (e != cudaSuccess) cudaUserObjectRelease(obj, 1);
    return e;
  }
  static void CUDART_CB let_go(void* hold) {
    auto* b = static_cast<std::shared_ptr<WorkBuf>*>(hold);
    (*b)->held.store(false, std::memory_order_release);
    delete b;
  }

  WorkBuf* add(Purpose purpose) try {
    bufs_.push_back(std::make_shared<WorkBuf>());
    bufs_.back()->purpose = purpose;
    return bufs_.back().get();
  } catch (const std::bad_alloc&) {
    return nullptr;
  }

  static cudaError_t renew(WorkBuf* b, size_t bytes) {
    if (b->p) cudaFree(b->p);
    b->p = nullptr;
    b->bytes = 0;
    b->plan = PlanKey();
    const cudaError_t e = cudaMalloc(&b->p, bytes);
    if (e == cudaSuccess) b->bytes = bytes;
    b->fresh = true;
    return e;
  }

  std::vector<std::shared_ptr<WorkBuf>> bufs_;
  uint64_t uses_ = 0;
  size_t kept_ = 0;
};

}  // namespace ztvm

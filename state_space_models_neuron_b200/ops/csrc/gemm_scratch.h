// Scratch of the GEMM's split tail: fp32 partial sums and arrival counters (zero between launches).  Launches that may run at
// once never share one: every stream has its own, and so has every stream of every graph capture, because a graph is replayed
// on whichever stream its owner likes.
//   eager     kept per stream (by the runtime's id, which is not used again for a later stream), at most EAGER per device; the
//             one that was used longest ago is freed for the next, which waits for the device
//   captured  belongs to the graph: it comes back when the graph and what was instantiated from it are gone.  The first launch of
//             the capture clears the counters inside the graph, so that every replay begins with zeros.
// Locked from the look-up to the launch: a scratch is not freed between the two.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace ssm {

struct Scratch { float* ws; int* counters; };

class ScratchPool {
 public:
  static constexpr int EAGER = 16, SPARE = 4;                // per device
  // one for all callers, never destroyed: graphs may outlive the library's statics
  static ScratchPool& get() { static ScratchPool* pool = new ScratchPool; return *pool; }
  std::mutex lock;                                 // held by the caller until its launch is in the stream

  // ws_bytes, counters: the same at every call.  False: no scratch (the caller launches without split tiles).
  bool take(cudaStream_t stream, size_t ws_bytes, int counters, Scratch* out) {
    int dev = 0;
    cudaStreamCaptureStatus state = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    cudaGraph_t graph = nullptr;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaStreamGetCaptureInfo_v2(stream, &state, &id, &graph, nullptr, nullptr) != cudaSuccess) return false;
    const bool captured = state == cudaStreamCaptureStatusActive;
    if (!captured && cudaStreamGetId(stream, &id) != cudaSuccess) return false;
    const Key key{dev, captured, id, captured ? stream : nullptr};
    const auto known = kept_.find(key);
    if (known != kept_.end()) {
      known->second.used = ++clock_;
      *out = split(known->second.memory, ws_bytes);
      return true;
    }
    Relaxed relaxed;                                         // allocating is no part of anybody's capture
    void* memory = nullptr;
    collect();
    std::vector<void*>& spare = spare_[dev];
    if (!captured) drop_oldest(dev);
    while ((int)spare.size() > SPARE) { cudaFree(spare.back()); spare.pop_back(); }
    if (!spare.empty()) {
      memory = spare.back();
      spare.pop_back();
    } else if (cudaMalloc(&memory, ws_bytes + counters * sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    *out = split(memory, ws_bytes);
    if (captured && !give_to(graph, key, memory)) { spare.push_back(memory); cudaGetLastError(); return false; }
    kept_[key] = Entry{memory, ++clock_};
    if (cudaMemsetAsync(out->counters, 0, counters * sizeof(int), stream) != cudaSuccess) {
      cudaGetLastError();
      if (!captured) { kept_.erase(key); spare.push_back(memory); }       // a captured one comes back with its graph
      return false;
    }
    return true;
  }
  // scratches of streams, of graphs, and spare ones
  void count(int* out) {
    std::lock_guard<std::mutex> hold(lock);
    collect();
    out[0] = out[1] = out[2] = 0;
    for (const auto& e : kept_) ++out[std::get<1>(e.first) ? 1 : 0];
    for (const auto& s : spare_) out[2] += (int)s.second.size();
  }

 private:
  using Key = std::tuple<int, bool, unsigned long long, cudaStream_t>;   // device, captured, stream's or capture's id, its stream
  struct Entry { void* memory; unsigned long long used; };
  struct Held { Key key; void* memory; Held* next; };
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  };
  static Scratch split(void* memory, size_t ws_bytes) {
    return Scratch{reinterpret_cast<float*>(memory), reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(memory) + ws_bytes)};
  }
  void drop_oldest(int dev) {
    int n = 0;
    auto oldest = kept_.end();
    for (auto e = kept_.begin(); e != kept_.end(); ++e) {
      if (std::get<0>(e->first) != dev || std::get<1>(e->first)) continue;
      ++n;
      if (oldest == kept_.end() || e->second.used < oldest->second.used) oldest = e;
    }
    if (n < EAGER) return;
    cudaFree(oldest->second.memory);                         // waits for the device
    kept_.erase(oldest);
  }
  // Called by the runtime when no graph uses the memory any more, perhaps under locks of its own: it neither calls CUDA nor
  // waits for a thread that does.
  static void returned(void* p) {
    Held* h = reinterpret_cast<Held*>(p);
    std::atomic<Held*>& top = get().returned_;
    h->next = top.load(std::memory_order_relaxed);
    while (!top.compare_exchange_weak(h->next, h, std::memory_order_release, std::memory_order_relaxed)) {}
  }
  void collect() {
    for (Held* h = returned_.exchange(nullptr, std::memory_order_acquire); h != nullptr;) {
      if (h->memory != nullptr) {
        kept_.erase(h->key);
        spare_[std::get<0>(h->key)].push_back(h->memory);
      }
      Held* next = h->next;
      delete h;
      h = next;
    }
  }
  static bool give_to(cudaGraph_t graph, const Key& key, void* memory) {
    Held* h = new Held{key, memory, nullptr};
    cudaUserObject_t object = nullptr;
    if (cudaUserObjectCreate(&object, h, returned, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) { delete h; return false; }
    if (cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove) == cudaSuccess) return true;
    h->memory = nullptr;                                     // stays with the caller
    cudaUserObjectRelease(object, 1);
    return false;
  }
  std::atomic<Held*> returned_{nullptr};                     // given back by graphs, not yet collected
  std::map<Key, Entry> kept_;
  std::map<int, std::vector<void*>> spare_;
  unsigned long long clock_ = 0;
};

}  // namespace ssm

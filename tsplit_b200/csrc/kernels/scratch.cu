// Registry of the library-owned device scratch buffers (see scratch.h).
#include "scratch.h"

#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

namespace {

struct Buf {
  void* ptr = nullptr;
  size_t bytes = 0;
};
typedef std::shared_ptr<std::remove_pointer_t<cudaEvent_t>> Event;
struct Idle {
  int device, tag;
  Buf buf;
  Event done;               // behind the last launch that may use it
};
std::mutex g_mu;
std::map<std::tuple<int, cudaStream_t, int>, Buf> g_table;
std::vector<std::pair<int, Buf>> g_parked;        // (device, replaced buffer)
std::vector<Idle> g_idle;
long long g_total = 0;

// The smallest given-back buffer for the purpose that is large enough and whose last launch has run.
bool take_idle(int device, int tag, size_t bytes, Buf* out) {
  int best = -1;
  for (int i = 0; i < (int)g_idle.size(); ++i) {
    const Idle& f = g_idle[i];
    if (f.device != device || f.tag != tag || f.buf.bytes < bytes || (best >= 0 && f.buf.bytes >= g_idle[best].buf.bytes)) continue;
    if (cudaEventQuery(f.done.get()) == cudaSuccess) best = i;
    else cudaGetLastError();
  }
  if (best < 0) return false;
  *out = g_idle[best].buf;
  g_idle.erase(g_idle.begin() + best);
  return true;
}

}  // namespace

namespace tsb_scratch {

void* get(cudaStream_t stream, int tag, size_t bytes, size_t floor_bytes) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> g(g_mu);
  Buf& b = g_table[std::make_tuple(dev, stream, tag)];
  if (b.bytes >= bytes && b.ptr) return b.ptr;
  Buf fresh;
  if (!take_idle(dev, tag, bytes, &fresh)) {
    fresh.bytes = bytes < floor_bytes ? floor_bytes : bytes;
    if (cudaMalloc(&fresh.ptr, fresh.bytes) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    g_total += (long long)fresh.bytes;
  }
  if (b.ptr) g_parked.push_back({dev, b});         // work queued on the stream may still use it
  b = fresh;
  return b.ptr;
}

}  // namespace tsb_scratch

extern "C" {

long long tsb_scratch_bytes() {
  std::lock_guard<std::mutex> g(g_mu);
  return g_total;
}

long long tsb_scratch_trim() {
  std::lock_guard<std::mutex> g(g_mu);
  int cur = 0;
  cudaGetDevice(&cur);
  long long freed = 0;
  for (auto& p : g_parked) {
    cudaSetDevice(p.first);
    if (cudaFree(p.second.ptr) == cudaSuccess) freed += (long long)p.second.bytes;
  }
  g_parked.clear();
  for (auto& f : g_idle) {
    cudaSetDevice(f.device);
    if (cudaFree(f.buf.ptr) == cudaSuccess) freed += (long long)f.buf.bytes;
  }
  g_idle.clear();
  cudaSetDevice(cur);
  g_total -= freed;
  return freed;
}

int tsb_scratch_give_back(int device, void* stream) {
  std::lock_guard<std::mutex> g(g_mu);
  int cur = 0;
  if (cudaGetDevice(&cur) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) {
    cudaGetLastError();
    return 0;                // (the process is ending)
  }
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  Event done;
  cudaEvent_t e = nullptr;
  if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess) {
    done.reset(e, cudaEventDestroy);
    if (cudaEventRecord(e, st) != cudaSuccess) done.reset();
  }
  cudaGetLastError();
  for (auto it = g_table.begin(); it != g_table.end();) {
    if (std::get<0>(it->first) != device || std::get<1>(it->first) != st || !it->second.ptr) {
      ++it;
      continue;
    }
    if (done) g_idle.push_back({device, std::get<2>(it->first), it->second, done});
    else g_parked.push_back({device, it->second});        // (nobody can tell when it is free)
    it = g_table.erase(it);
  }
  cudaSetDevice(cur);
  return 0;
}

}  // extern "C"

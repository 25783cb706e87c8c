// A stand-in for the CUDA runtime and the library's kernels, so that the host orchestration
// (ooc_api.cu, compiled as plain C++) runs without a GPU.  Work queued on a stream runs as late
// as CUDA allows: when the host waits for it, or when work that waits for it runs.  What the
// library leaves unfinished is therefore still in a queue, and what it takes for finished too
// early has not happened.
//
// The kernels' model: every stripe with items has one voxel, its first.  The voxelization sets its
// bit and lists one large item, and reports bits and list entries that it finds there already; the
// emission clears both, or (raise_flag) fails its layout check and leaves the bit.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <memory>
#include <vector>

#include "ooc_internal.h"

namespace fake {

using Op = std::function<void()>;
struct Stream {
  std::deque<Op> queue;
  std::vector<Op>* capture = nullptr;
};
struct Event {
  Stream* on = nullptr;
  uint64_t recorded = 0, done = 0;
};
struct Graph {
  std::vector<Op> ops;
};

inline std::vector<std::unique_ptr<Stream>> streams;
inline std::map<char*, size_t> device, pinned;  // allocations
inline size_t device_bytes = 0, device_peak = 0;
inline long events = 0, execs = 0;
inline cudaError_t last = cudaSuccess;
inline long fail_after = -1;  // allocations until one fails (-1: none does)
inline bool raise_flag = false;
inline long dirty = 0;  // voxelizations that began with set bits or a list that was not empty

inline cudaError_t fails(cudaError_t e) { return last = e; }
inline bool run_one(Stream* s) {
  if (s->queue.empty()) return false;
  Op op = std::move(s->queue.front());
  s->queue.pop_front();
  op();
  return true;
}
inline void drain(Stream* s) {
  while (run_one(s)) {
  }
}
inline void drain_all() {
  for (auto& s : streams) drain(s.get());
}
inline size_t queued() {
  size_t n = 0;
  for (auto& s : streams) n += s->queue.size();
  return n;
}
inline Stream* of(cudaStream_t st) { return reinterpret_cast<Stream*>(st); }
inline void put(cudaStream_t st, Op op) {
  Stream* s = of(st);
  if (s->capture) s->capture->push_back(std::move(op));
  else s->queue.push_back(std::move(op));
}
inline cudaStream_t new_stream() {
  streams.push_back(std::make_unique<Stream>());
  return reinterpret_cast<cudaStream_t>(streams.back().get());
}
inline bool is_pinned(const void* p) {
  const char* c = static_cast<const char*>(p);
  auto it = pinned.upper_bound(const_cast<char*>(c));
  return it != pinned.begin() && c < std::prev(it)->first + std::prev(it)->second;
}
inline bool out_of_memory() { return fail_after >= 0 && fail_after-- == 0; }

}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  if (fake::out_of_memory()) return fake::fails(cudaErrorMemoryAllocation);
  char* c = static_cast<char*>(std::calloc(n, 1));
  if (n < (16u << 20)) std::memset(c, 0xab, n);
  fake::device[c] = n;
  fake::device_bytes += n;
  fake::device_peak = std::max(fake::device_peak, fake::device_bytes);
  *p = c;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  fake::drain_all();
  auto it = fake::device.find(static_cast<char*>(p));
  fake::device_bytes -= it->second;
  fake::device.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (fake::out_of_memory()) return fake::fails(cudaErrorMemoryAllocation);
  char* c = static_cast<char*>(std::malloc(n));
  fake::pinned[c] = n;
  *p = c;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  fake::drain_all();
  fake::pinned.erase(static_cast<char*>(p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = *t = 64ull << 30;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
  if (kind == cudaMemcpyHostToDevice && !fake::is_pinned(s)) {  // pageable memory is read before the call returns
    auto copy = std::make_shared<std::vector<char>>(static_cast<const char*>(s), static_cast<const char*>(s) + n);
    fake::put(st, [=] { std::memcpy(d, copy->data(), n); });
  } else {
    fake::put(st, [=] { std::memcpy(d, s, n); });
  }
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  fake::drain_all();
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  fake::put(st, [=] { std::memset(d, v, n); });
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = fake::new_stream();
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  for (size_t i = 0; i < fake::streams.size(); i++)
    if (fake::streams[i].get() == fake::of(s)) fake::streams.erase(fake::streams.begin() + (long)i);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  fake::drain(fake::of(s));
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t s) { return fake::run_one(fake::of(s)) ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  fake::events++;
  *e = reinterpret_cast<cudaEvent_t>(new fake::Event);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  fake::events--;
  delete reinterpret_cast<fake::Event*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t st) {
  auto* e = reinterpret_cast<fake::Event*>(ev);
  e->on = fake::of(st);
  const uint64_t r = ++e->recorded;
  fake::put(st, [=] { e->done = r; });
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t ev, unsigned) {
  auto* e = reinterpret_cast<fake::Event*>(ev);
  fake::Stream* on = e->on;
  const uint64_t r = e->recorded;
  fake::put(st, [=] {
    while (e->done < r && fake::run_one(on)) {
    }
  });
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t ev) {
  auto* e = reinterpret_cast<fake::Event*>(ev);
  while (e->done < e->recorded && fake::run_one(e->on)) {
  }
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t ev) {
  auto* e = reinterpret_cast<fake::Event*>(ev);
  if (e->done < e->recorded) fake::run_one(e->on);
  return e->done < e->recorded ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  fake::of(s)->capture = new std::vector<fake::Op>;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  std::unique_ptr<std::vector<fake::Op>> ops(fake::of(s)->capture);
  fake::of(s)->capture = nullptr;
  *g = reinterpret_cast<cudaGraph_t>(new fake::Graph{*ops});
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) {
  *n = 0;
  return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType*) { return cudaErrorInvalidValue; }
cudaError_t cudaGraphKernelNodeGetParams(cudaGraphNode_t, cudaKernelNodeParams*) { return cudaErrorInvalidValue; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  fake::execs++;
  *x = reinterpret_cast<cudaGraphExec_t>(new fake::Graph(*reinterpret_cast<fake::Graph*>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t x, cudaGraph_t g, cudaGraphExecUpdateResultInfo*) {
  reinterpret_cast<fake::Graph*>(x)->ops = reinterpret_cast<fake::Graph*>(g)->ops;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<fake::Graph*>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  fake::execs--;
  delete reinterpret_cast<fake::Graph*>(x);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  for (const fake::Op& op : reinterpret_cast<fake::Graph*>(x)->ops) fake::put(s, op);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
}  // extern "C"

namespace ooc {

namespace {
LaunchState* t_state = nullptr;
}
LaunchState* current_launch_state() { return t_state; }
LaunchScope::LaunchScope(LaunchState* s) : prev(t_state) { t_state = s; }
LaunchScope::~LaunchScope() { t_state = prev; }

uint64_t scan_partials_needed(uint64_t n) { return n / 4096 + 2; }
uint32_t stream_ctas(uint64_t n) { return (uint32_t)(n / 64 + 1); }
int persist_ctas_per_sm() { return 0; }

void launch_copy_words(const uint32_t* src, uint64_t n, uint32_t* dst, cudaStream_t st) {
  fake::put(st, [=] { std::memcpy(dst, src, n * 4); });
}
void launch_part_count(const float*, int, uint64_t n_tris, const float*, const float*, int, uint64_t n_parts, uint32_t* hist,
                       int, cudaStream_t st) {
  fake::put(st, [=] {
    for (uint64_t p = 0; p < n_parts; p++) hist[p] += (uint32_t)n_tris;  // every triangle in every partition
  });
}
void launch_part_emit(const float*, int, uint64_t, const float*, const float*, int, uint64_t, uint32_t*, uint32_t*,
                      int, cudaStream_t st) {
  fake::put(st, [] {});
}
void launch_stream_bases(const uint32_t*, uint32_t, uint32_t, uint64_t*, cudaStream_t) {}
void launch_stream_group_chunk(const float*, int, uint64_t, const float*, const float*, int, uint32_t, uint32_t, uint32_t*,
                               uint32_t*, uint64_t*, float*, cudaStream_t) {}

void launch_b_vox_small(const VoxJob* jobs, const uint64_t*, uint32_t n, uint64_t, int pass, const VoxJob* single,
                        cudaStream_t st) {
  if (pass != 0) return;
  const bool lone = single != nullptr;
  const VoxJob j0 = lone ? *single : VoxJob();
  fake::put(st, [=] {
    for (uint32_t s = 0; s < n; s++) {
      const VoxJob& j = lone ? j0 : jobs[s];
      bool clean = s > 0 || j.ctr[kCtrLarge] == 0;
      for (int k = 0; k < 8; k++) clean = clean && j.leafbits[k] == 0;
      if (j.leaftouch) clean = clean && j.leaftouch[0] == 0;
      fake::dirty += !clean;
      j.leafbits[0] |= 1u;
      if (j.leaftouch) j.leaftouch[0] = 1;
      j.ctr[kCtrLarge]++;
    }
  });
}
void launch_b_vox_large(const VoxJob*, const LargeLists&, int, const VoxJob*, cudaStream_t st, int, int, int) {
  fake::put(st, [] {});
}
void launch_b_persist(const PersistJob&, int, int, cudaStream_t) {}
void launch_b_bricks(const Stripe*, const uint64_t*, uint32_t, uint64_t, const Stripe*, cudaStream_t st) {
  fake::put(st, [] {});
}
void launch_b_upper(const Stripe* stripes, uint32_t n, int, uint32_t* counts, const unsigned long long* large_ctr,
                    uint64_t* large_out, const uint64_t*, uint64_t*, const Stripe* single, cudaStream_t st) {
  const bool lone = single != nullptr;
  const Stripe p0 = lone ? *single : Stripe();
  fake::put(st, [=] {
    for (uint32_t s = 0; s < n; s++) {
      const Stripe& p = lone ? p0 : stripes[s];
      uint32_t* o = counts + (uint64_t)s * kCountWords;
      o[0] = p.leaf[0] & 1u;
      o[1] = p.K > 1 ? (uint32_t)p.K - 1u : 0u;
      for (int l = 0; l <= p.U; l++) o[2 + l] = 1;
      o[kRootWord] = 1;
    }
    *large_out = large_ctr[kCtrLarge];
  });
}
void launch_b_leaf_payload(const Stripe*, const EmitJob*, const uint64_t*, uint32_t, uint64_t, uint32_t, const Stripe*,
                           const EmitJob*, cudaStream_t st) {
  fake::put(st, [] {});
}
void launch_b_emit(const Stripe* stripes, const EmitJob* emits, const uint64_t*, uint32_t n, uint64_t, bool, int,
                   unsigned long long* large_ctr, const Stripe* sp, const EmitJob* se, cudaStream_t st) {
  const bool lone = sp != nullptr;
  const Stripe p0 = lone ? *sp : Stripe();
  const EmitJob e0 = lone ? *se : EmitJob();
  fake::put(st, [=] {
    for (uint32_t s = 0; s < n; s++) {
      const Stripe& p = lone ? p0 : stripes[s];
      if (fake::raise_flag) {
        *(lone ? e0 : emits[s]).flag = 1;
        continue;
      }
      p.leaf[0] = 0;
      if (p.touch) p.touch[0] = 0;
    }
    for (uint32_t k = 0; k < kLargeCtrWords; k++) large_ctr[k] = 0;
  });
}
void launch_b_upper_levels(const Stripe*, const EmitJob*, uint32_t, int, const Stripe*, const EmitJob*, cudaStream_t st) {
  fake::put(st, [] {});
}
void launch_scatter_records(const uint64_t*, uint64_t, uint64_t, uint64_t*, uint64_t*, cudaStream_t st) {
  fake::put(st, [] {});
}

}  // namespace ooc

// The host side of a build on the stand-in runtime of fake_cuda.h (test_host_build.py).  One
// argument: the property to check.
#include <algorithm>
#include <string>

#include "fake_cuda.h"
#include "ooc_admission.h"

namespace {

int bad = 0;
void expect(bool ok, const std::string& what) {
  if (ok) return;
  if (bad++ < 10) std::printf("%s\n", what.c_str());
}

ooc_build_params params(uint64_t grid, uint64_t limit, bool levels = false) {
  ooc_build_params p;
  std::memset(&p, 0, sizeof(p));
  p.gridsize = grid;
  p.memory_limit_mb = limit;
  p.geometry_only = 1;
  p.generate_levels = levels;
  for (int a = 0; a < 3; a++) p.bbox_max[a] = 1.0f;
  return p;
}

// What a call's callbacks do: the `left`-th from now on refuses.
struct Callbacks {
  long left = -1;
  ooc_device_arena arena{};
  int next() { return left >= 0 && left-- == 0 ? 1 : 0; }
};
int on_sink(void* u, int32_t, const void*, uint64_t) { return static_cast<Callbacks*>(u)->next(); }
int on_batch_sink(void* u, uint64_t, int32_t, const void*, uint64_t) { return static_cast<Callbacks*>(u)->next(); }
int on_alloc(void* u, uint64_t m, uint64_t nb, uint64_t db, void* st, void** n, void** d) {
  Callbacks* c = static_cast<Callbacks*>(u);
  return c->next() ? 1 : ooc_arena_alloc(&c->arena, m, nb, db, st, n, d);
}
int on_ready(void* u, uint64_t) { return static_cast<Callbacks*>(u)->next(); }

// The calls: octree on the device, to a sink, batches to a sink and to device destinations; one stripe or
// 64 in several sub-batches.
constexpr int kCalls = 6;
const char* const kNames[kCalls] = {"device", "device, 64 partitions", "device, 64 partitions, levels",
                                    "sink, 64 partitions", "batch", "batch to device memory"};
char arena_mem[1 << 20];

int call(int which, ooc_ctx* c, cudaStream_t st, Callbacks& cb) {
  static float tri[9] = {0.0f, 0.0f, 0.0f, 0.1f, 0.0f, 0.0f, 0.0f, 0.1f, 0.0f};
  ooc_mesh m[3];
  for (ooc_mesh& x : m) x.tris = tri, x.n_tris = 1, x.params = params(64, 2048);
  m[1].params = params(256, 1);
  ooc_set_batch_budget(c, 8 * 40000);  // about eight stripes of 64^3
  cb.arena = ooc_device_arena{arena_mem, sizeof(arena_mem), 0};
  const ooc_build_params one = params(64, 2048), many = params(256, 1), lev = params(256, 1, true);
  switch (which) {
    case 0: return ooc_build_device(c, &one, tri, 1, st, nullptr);
    case 1: return ooc_build_device(c, &many, tri, 1, st, nullptr);
    case 2: return ooc_build_device(c, &lev, tri, 1, st, nullptr);
    case 3: return ooc_build(c, &many, tri, 1, on_sink, &cb, nullptr);
    case 4: return ooc_build_batch(c, m, 3, on_batch_sink, &cb, nullptr);
    default: return ooc_build_batch_device(c, m, 3, on_alloc, on_ready, &cb, nullptr);
  }
}

// After a failure at every point of every call: `check(name of the point, context)`.
template <typename F>
void each_failure(F check) {
  for (int which = 0; which < kCalls; which++)
    for (int kind = 0; kind < 2; kind++) {  // allocations, callbacks
      long at = 0;
      for (;; at++) {
        fake::last = cudaSuccess;
        const cudaStream_t user = fake::new_stream();
        ooc_ctx* c = nullptr;
        expect(ooc_ctx_create(0, &c) == OOC_OK, "ooc_ctx_create");
        Callbacks cb;
        if (kind == 0) fake::fail_after = at;
        else cb.left = at;
        const int rc = call(which, c, user, cb);
        const bool reached = (kind == 0 ? fake::fail_after : cb.left) < 0;
        fake::fail_after = -1;
        if (reached) {
          expect(rc != OOC_OK, "a failure was not reported");
          check(std::string(kNames[which]) + (kind ? ", callback " : ", allocation ") + std::to_string(at), c);
        } else {
          expect(rc == OOC_OK, std::string(kNames[which]) + " without a failure: " + ooc_last_error(c));
        }
        ooc_ctx_destroy(c);
        cudaStreamDestroy(user);
        if (!reached) break;
      }
      expect(at > (kind == 0 || which > 2 ? 3 : -1), std::string(kNames[which]) + ": too few points of failure");
    }
}

void check_drained() {
  each_failure([](const std::string& at, ooc_ctx*) {
    expect(fake::queued() == 0, at + ": " + std::to_string(fake::queued()) + " operations still queued");
  });
}

// A build that fails its layout check leaves the bits of what it did not write: the next one, whatever it
// returns to, starts from clean buffers.
void check_clean() {
  for (int which = 0; which < kCalls; which++) {
    const cudaStream_t user = fake::new_stream();
    ooc_ctx* c = nullptr;
    expect(ooc_ctx_create(0, &c) == OOC_OK, "ooc_ctx_create");
    Callbacks cb;
    fake::raise_flag = true;
    expect(call(which, c, user, cb) == OOC_ERR_DEVICE, std::string(kNames[which]) + ": the flag was not reported");
    fake::raise_flag = false;
    for (int next = 0; next < kCalls; next++) {
      fake::dirty = 0;
      expect(call(next, c, user, cb) == OOC_OK, std::string(kNames[next]) + ": " + ooc_last_error(c));
      expect(fake::dirty == 0, std::string(kNames[next]) + " after " + kNames[which] + " with its flag raised: " +
                                   std::to_string(fake::dirty) + " stripes began with bits set");
    }
    ooc_ctx_destroy(c);
    cudaStreamDestroy(user);
  }
}

// The build after a failed one succeeds: the failure's error is not met again as that build's own.
void check_recovered() {
  each_failure([](const std::string& at, ooc_ctx* c) {
    expect(fake::last == cudaSuccess, at + ": the error is still the thread's last one");
    Callbacks cb;
    for (int next = 0; next < kCalls; next++)
      expect(call(next, c, nullptr, cb) == OOC_OK, std::string(kNames[next]) + " after " + at + ": " + ooc_last_error(c));
  });
}

// A destroyed context has given back its memory, streams, events and graphs.
void check_freed() {
  const cudaStream_t user = fake::new_stream();
  ooc_ctx* c = nullptr;
  expect(ooc_ctx_create(0, &c) == OOC_OK, "ooc_ctx_create");
  Callbacks cb;
  for (int which = 0; which < kCalls; which++) expect(call(which, c, user, cb) == OOC_OK, kNames[which]);
  static float tri[9] = {0.0f, 0.0f, 0.0f, 0.1f, 0.0f, 0.0f, 0.0f, 0.1f, 0.0f};
  const ooc_mesh m = {tri, 1, params(64, 2048)};
  expect(ooc_autotune(c, &m, 1, nullptr) == OOC_OK, "ooc_autotune");
  ooc_ctx_destroy(c);
  cudaStreamDestroy(user);
  expect(fake::device.empty(), std::to_string(fake::device.size()) + " device allocations left");
  expect(fake::pinned.empty(), std::to_string(fake::pinned.size()) + " pinned allocations left");
  expect(fake::streams.empty() && fake::events == 0 && fake::execs == 0, "streams, events or graphs left");
}

// Destinations of a batch: `nodes` needs 8 bytes, `data` 16 where the file holds more than header records.
struct Offsets {
  uint64_t nodes, data;
};
int offset_alloc(void* u, uint64_t, uint64_t nb, uint64_t, void*, void** n, void** d) {
  const Offsets* o = static_cast<Offsets*>(u);
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(arena_mem) + 255) / 256 * 256);
  *n = base + o->nodes;
  *d = base + (nb + 511) / 256 * 256 + o->data;
  return 0;
}
void check_aligned() {
  static float tri[21] = {0.0f, 0.0f, 0.0f, 0.1f, 0.0f, 0.0f, 0.0f, 0.1f, 0.0f};
  for (int payload = 0; payload < 2; payload++)
    for (int levels = 0; levels < 2; levels++)
      for (uint64_t count = 0; count < 2; count++)
        for (uint64_t nodes : {0, 4, 8, 16})
          for (uint64_t data : {0, 4, 8, 16}) {
            ooc_ctx* c = nullptr;
            expect(ooc_ctx_create(0, &c) == OOC_OK, "ooc_ctx_create");
            ooc_mesh m = {tri, count, params(64, 2048, levels)};
            m.params.geometry_only = !payload;
            Offsets o{nodes, data};
            const bool records = count && (payload || levels);
            const int want = nodes % 8 || data % (records ? 16 : 8) ? OOC_ERR_INVALID : OOC_OK;
            const int got = ooc_build_batch_device(c, &m, 1, offset_alloc, nullptr, &o, nullptr);
            expect(got == want, "payload " + std::to_string(payload) + ", levels " + std::to_string(levels) + ", " +
                                    std::to_string(count) + " triangles, nodes at " + std::to_string(nodes) + ", data at " +
                                    std::to_string(data) + ": status " + std::to_string(got));
            ooc_ctx_destroy(c);
          }
}

// What the serving loop admits a request for covers what a build of it allocates and its result.
int sized_alloc(void* u, uint64_t, uint64_t nb, uint64_t db, void*, void** n, void** d) {
  *static_cast<uint64_t*>(u) = nb + db;
  *n = arena_mem;
  *d = arena_mem + (nb + 255) / 256 * 256;
  return 0;
}
void check_admitted() {
  static float small[21] = {0.5f, 0.5f, 0.5f, 0.505f, 0.5f, 0.5f, 0.5f, 0.505f, 0.5f};
  static float wide[21] = {0.0f, 0.0f, 0.0f, 1.0f, 1.0f, 0.9f, 0.1f, 1.0f, 1.0f};
  for (int payload = 0; payload < 2; payload++)
    for (int levels = 0; levels < 2; levels++)
      for (const auto& [grid, limit] : {std::pair<uint64_t, uint64_t>{1, 2048}, {8, 2048}, {64, 2048}, {256, 2048}, {512, 2048},
                                        {1024, 2048}, {2048, 16384}, {64, 1}, {128, 1}, {256, 1}, {512, 17}}) {
        const bool parts = ooc_estimate_partitions(grid, limit) > 1;
        ooc_ctx* c = nullptr;
        expect(ooc_ctx_create(0, &c) == OOC_OK, "ooc_ctx_create");
        ooc_mesh m = {parts ? wide : small, 1, params(grid, limit, levels)};  // the stand-in bins it everywhere
        m.params.geometry_only = !payload;
        ooc_set_batch_budget(c, 64 << 20);  // the octree of several stripes is parked
        uint64_t files = 0;
        fake::device_peak = fake::device_bytes;
        expect(ooc_build_batch_device(c, &m, 1, sized_alloc, nullptr, &files, nullptr) == OOC_OK, ooc_last_error(c));
        const uint64_t held = fake::device_peak + files, admitted = ooc::footprint(m);
        const std::string at = "gridsize " + std::to_string(grid) + ", payload " + std::to_string(payload) + ", levels " +
                               std::to_string(levels) + ": " + std::to_string(held) + " bytes held, admitted for " +
                               std::to_string(admitted);
        expect(held <= admitted, at);
        if (grid == 1024) expect(admitted <= held + held / 16, at + ", far more");
        ooc_ctx_destroy(c);
      }
  // the bound on a triangle's partitions against the test that bins it
  std::srand(1);
  const uint64_t N = 512, per = 8, side = N / per;
  const float u = 1.0f / (float)N;
  for (int k = 0; k < 20000; k++) {
    float v[9];
    for (float& x : v) {
      x = (float)std::rand() / (float)RAND_MAX * 1.4f - 0.2f;
      if (std::rand() % 3 == 0) x = (float)(std::rand() % (int)(per + 1)) * (float)side * u;  // on a slab's bound
    }
    if (k % 2)  // a small box
      for (int q = 3; q < 9; q++) v[q] = v[q % 3] + (float)(std::rand() % 257 - 128) / 128.0f * u * (float)(1 + 30 * (q % 3 == k % 3));
    uint64_t n = 1;
    for (int a = 0; a < 3; a++) {
      const float lo = std::min(v[a], std::min(v[3 + a], v[6 + a])), hi = std::max(v[a], std::max(v[3 + a], v[6 + a]));
      uint64_t on = 0;
      for (uint64_t j = 0; j < per; j++) on += !(hi < (float)(j * side) * u) && !(lo > (float)((j + 1) * side) * u);
      n *= on;
    }
    expect((double)n <= ooc::pair_bound(1.0, ooc::box_voxels(v, 1.0f / u, N), side, per * per * per), "pair_bound");
  }
}

}  // namespace

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "drained") check_drained();
  else if (what == "clean") check_clean();
  else if (what == "recovered") check_recovered();
  else if (what == "freed") check_freed();
  else if (what == "aligned") check_aligned();
  else if (what == "admitted") check_admitted();
  else return 2;
  std::printf("%d failures\n", bad);
  return bad ? 1 : 0;
}

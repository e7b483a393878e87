// A CUDA runtime for host tests of the renderer's runtime: device memory is
// host memory, kernels are hooks.  Include it after renderer.cpp.
//
// Work on a created stream runs at once; work on the legacy default stream
// waits until something has to wait for it (a synchronous copy, a blocking
// stream), as it does when another thread keeps that stream busy.  A
// synchronous copy waits for what lies before it; one to the device then returns
// once it has read the host's memory and writes the device's later, as it may.
// Work that relies on an order between the two streams then runs out of order.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <vector>

namespace fake {

struct Stream {
  bool blocking;
};
struct Graph {
  std::vector<std::function<void()>> ops;
};

inline std::deque<std::function<void()>> legacy;
inline Graph* capture = nullptr;
inline cudaStream_t capture_stream = nullptr;
inline std::map<cudaEvent_t, cudaStream_t> recorded;            // the stream of an event's last record
inline std::vector<std::pair<cudaStream_t, cudaStream_t>> waits;  // (waiting stream, stream waited for)
inline int captures = 0, instantiations = 0, sms = 152, occupancy = 2;
inline std::function<void(const gbr::PrepareParams&, uint32_t scenes)> on_prepare;
inline std::function<void(const gbr::RasterParams&, uint32_t scenes, uint32_t* done)> on_order;
inline std::function<void(const gbr::RasterParams&, int threads, uint32_t grid, size_t smem)> on_raster;

inline void run_legacy() {
  while (!legacy.empty()) {
    auto op = legacy.front();
    legacy.pop_front();
    op();
  }
}
inline void enqueue(cudaStream_t s, std::function<void()> op) {
  if (capture && s == capture_stream) {
    capture->ops.push_back(op);
  } else if (!s) {
    legacy.push_back(op);
  } else {
    if (reinterpret_cast<Stream*>(s)->blocking) run_legacy();
    op();
  }
}
inline cudaStream_t stream(bool blocking) { return reinterpret_cast<cudaStream_t>(new Stream{blocking}); }

}  // namespace fake

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? fake::sms
       : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472
       : a == cudaDevAttrReservedSharedMemoryPerBlock ? 1024 : 0;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind) {
  fake::run_legacy();
  if (kind == cudaMemcpyDeviceToHost) {
    std::memcpy(d, s, n);
  } else {
    const std::vector<char> staged(static_cast<const char*>(s), static_cast<const char*>(s) + n);
    fake::enqueue(nullptr, [=] { std::memcpy(d, staged.data(), staged.size()); });
  }
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  fake::enqueue(st, [=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
  fake::run_legacy();
  for (size_t y = 0; y < h; ++y) std::memcpy(static_cast<char*>(d) + y * dp, static_cast<const char*>(s) + y * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k,
                              cudaStream_t st) {
  fake::enqueue(st, [=] { cudaMemcpy2D(d, dp, s, sp, w, h, k); });
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  fake::enqueue(nullptr, [=] { std::memset(d, v, n); });
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  fake::enqueue(st, [=] { std::memset(d, v, n); });
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  *a = cudaPointerAttributes{};
  return cudaSuccess;
}
cudaError_t cudaStreamCreate(cudaStream_t* s) {
  *s = fake::stream(true);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags) {
  *s = fake::stream(flags != cudaStreamNonBlocking);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  delete reinterpret_cast<fake::Stream*>(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (!s || reinterpret_cast<fake::Stream*>(s)->blocking) fake::run_legacy();
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  fake::run_legacy();
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  fake::waits.push_back({s, fake::recorded[e]});
  return fake::capture && s == fake::capture_stream ? cudaErrorStreamCaptureIsolation : cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* out) {
  *out = fake::capture && s == fake::capture_stream ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  fake::recorded[e] = s;
  return cudaSuccess;
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  fake::capture = new fake::Graph;
  fake::capture_stream = s;
  ++fake::captures;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(fake::capture);
  fake::capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(new fake::Graph(*reinterpret_cast<fake::Graph*>(g)));
  ++fake::instantiations;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<fake::Graph*>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete reinterpret_cast<fake::Graph*>(e);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
  for (const auto& op : reinterpret_cast<fake::Graph*>(e)->ops) fake::enqueue(s, op);
  return cudaSuccess;
}
}  // extern "C"

namespace gbr {
cudaError_t launch_prepare(const PrepareParams& p, uint32_t scenes, cudaStream_t s) {
  fake::enqueue(s, [=] { if (fake::on_prepare) fake::on_prepare(p, scenes); });
  return cudaSuccess;
}
cudaError_t launch_order(const RasterParams& p, uint32_t scenes, WorkItem*, uint32_t*, uint32_t* done, uint32_t, bool,
                         cudaStream_t s) {
  fake::enqueue(s, [=] { if (fake::on_order) fake::on_order(p, scenes, done); });
  return cudaSuccess;
}
cudaError_t launch_raster(const RasterParams& p, int threads, uint32_t grid, size_t smem, bool, cudaStream_t s) {
  fake::enqueue(s, [=] { if (fake::on_raster) fake::on_raster(p, threads, grid, smem); });
  return cudaSuccess;
}
cudaError_t launch_gather_tiles(const void*, int64_t, int, int, int, uint32_t, uint32_t, void*, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t raster_configure(int, size_t* max_dynamic, size_t* static_bytes) {
  *max_dynamic = 232448 - 2048;
  *static_bytes = 2048;
  return cudaSuccess;
}
cudaError_t raster_max_ctas_per_sm(int threads, size_t, int* out) {
  *out = fake::occupancy * 512 / threads > 0 ? fake::occupancy * 512 / threads : 1;
  return cudaSuccess;
}
cudaError_t hbao_launch(const HbaoScene*, const HbaoScene&, int, int, int, const float*, uint32_t*, void*,
                        const HbaoParams&, cudaStream_t) {
  return cudaSuccess;
}
}  // namespace gbr

namespace fake {

inline int failures = 0;
#define CHECK(c)                                                   \
  do {                                                             \
    if (!(c)) {                                                    \
      std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c); \
      ++fake::failures;                                            \
    }                                                              \
  } while (0)

// A renderer of `scenes` viewports of w x h, each with `draws` triangles of its own.
inline gbr::Renderer* renderer(uint32_t scenes, int w, int h, uint32_t draws = 1) {
  gbr_config cfg{};
  std::vector<int32_t> viewports;
  for (uint32_t s = 0; s < scenes; ++s) viewports.insert(viewports.end(), {w, h});
  cfg.scene_count = scenes;
  cfg.viewports = viewports.data();
  cfg.planes = GBR_PLANE_ALL;
  std::string err;
  gbr::Renderer* r = gbr::Renderer::create(cfg, err);
  if (!r) {
    std::fprintf(stderr, "%s\n", err.c_str());
    std::exit(1);
  }
  const float pos[9] = {0, 0, -1, 1, 0, -1, 0, 1, -1};
  const uint32_t idx[3] = {0, 1, 2};
  gbr_mesh_data m{};
  m.vertex_count = 3;
  m.positions = pos;
  m.index_count = 3;
  m.indices = idx;
  uint32_t id = 0;
  CHECK(r->add_mesh(m, &id) == GBR_OK);
  gbr_mesh_view v{};
  v.mesh = id;
  v.index_count = 3;
  for (int i = 0; i < 4; ++i) v.transform[5 * i] = 1.0f;
  CHECK(r->add_template("t", 1, &v) == GBR_OK);
  uint64_t node;
  for (uint32_t s = 0; s < scenes; ++s)
    for (uint32_t d = 0; d < draws; ++d) CHECK(r->add_node_hierarchy(s, "t", nullptr, &node) == GBR_OK);
  return r;
}

inline int finish() {
  if (failures) return 1;
  std::printf("ok\n");
  return 0;
}

}  // namespace fake

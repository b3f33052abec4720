// Lifetimes of the scratch buffers of the C++ host mirror (csrc/host/direct_gpu_backend.cpp), without a GPU: the few CUDA
// runtime calls and library entry points that the mirror makes are the fakes below.  A "graph" is the list of workspace
// addresses recorded while the fake stream was capturing; every one of them has to stay allocated as long as the graph
// lives, and no two live graphs may share one.  Exit code 0 = all cases passed.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>
#include <vector>

#include "../../aidotnet/tensors_b200/csrc/host/direct_gpu_backend.hpp"

using aidn::host::CudaBackend;
using aidn::host::GpuBuffer;

static std::map<void*, size_t> g_live;
static size_t g_limit = ~(size_t)0;              // device memory left to allocate
static unsigned long long g_capture = 0;         // id of the running capture, 0 = none
static cudaStreamCaptureMode g_mode = cudaStreamCaptureModeGlobal;
static std::map<unsigned long long, std::vector<std::pair<cudaHostFn_t, void*>*>> g_objects;   // user objects by graph
static std::vector<std::pair<void*, int64_t>> g_launches;
static int64_t g_need = 0;

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_capture && g_mode != cudaStreamCaptureModeRelaxed) return cudaErrorStreamCaptureUnsupported;
  if (n > g_limit) return cudaErrorMemoryAllocation;
  *p = std::malloc(16);
  g_live[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) { return g_live.erase(p) ? cudaSuccess : cudaErrorInvalidValue; }   // (never given back: an address is used once)
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
  std::swap(*m, g_mode);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = g_capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus* s, unsigned long long* id, cudaGraph_t* graph,
                                        const cudaGraphNode_t**, size_t*) {
  *s = g_capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  if (id) *id = g_capture;
  if (graph) *graph = reinterpret_cast<cudaGraph_t>(g_capture);
  return cudaSuccess;
}
cudaError_t cudaUserObjectCreate(cudaUserObject_t* out, void* ptr, cudaHostFn_t destroy, unsigned, unsigned) {
  *out = reinterpret_cast<cudaUserObject_t>(new std::pair<cudaHostFn_t, void*>(destroy, ptr));
  return cudaSuccess;
}
cudaError_t cudaGraphRetainUserObject(cudaGraph_t graph, cudaUserObject_t object, unsigned, unsigned) {
  g_objects[reinterpret_cast<unsigned long long>(graph)].push_back(reinterpret_cast<std::pair<cudaHostFn_t, void*>*>(object));
  return cudaSuccess;
}

const char* aidn_sdpa_last_error(void) { return "fake"; }
int aidn_sdpa_device_supported(int32_t) { return 1; }
int aidn_sdpa_create(const aidn_sdpa_desc*, aidn_sdpa_t* out) {
  static int h;
  *out = reinterpret_cast<aidn_sdpa_t>(&h);
  return AIDN_OK;
}
int aidn_sdpa_destroy(aidn_sdpa_t) { return AIDN_OK; }
int64_t aidn_sdpa_workspace_bytes(aidn_sdpa_t, int64_t, int64_t, int64_t) { return g_need; }
int64_t aidn_sdpa_backward_workspace_bytes(aidn_sdpa_t, int64_t, int64_t) { return g_need; }
int64_t aidn_mha_workspace_bytes(aidn_sdpa_t, int64_t, int64_t, int32_t, int32_t) { return g_need; }
int aidn_sdpa_launch(aidn_sdpa_t, const aidn_sdpa_args* a, void*) {
  g_launches.push_back({a->workspace, a->workspace_bytes});
  return AIDN_OK;
}
int aidn_sdpa_backward(aidn_sdpa_t, const aidn_sdpa_bwd_args* a, void*) {
  g_launches.push_back({a->fwd.workspace, a->fwd.workspace_bytes});
  return AIDN_OK;
}
int aidn_mha_forward(aidn_sdpa_t, const aidn_mha_args* a, void*) {
  g_launches.push_back({a->workspace, a->workspace_bytes});
  return AIDN_OK;
}
int aidn_sdpa_last_path(aidn_sdpa_t) { return 0; }
int aidn_sdpa_last_launch_count(aidn_sdpa_t) { return 1; }
}

static int g_failed = 0;
#define EXPECT(cond)                                                              \
  do {                                                                            \
    if (!(cond)) {                                                                \
      std::printf("FAILED %s:%d: %s\n", __FILE__, __LINE__, #cond);               \
      ++g_failed;                                                                 \
    }                                                                             \
  } while (0)

static GpuBuffer buffer(int64_t n) {
  static char memory[16];
  GpuBuffer b;
  b.Handle = memory;
  b.Size = n;
  return b;
}

// One launch that asks for `need` bytes: decode (one query row) cannot run without them, a prefill can.
static void* attention(CudaBackend& be, int64_t need, int rows) {
  g_need = need;
  const GpuBuffer q = buffer(64 * rows), kv = buffer(64 * 128);
  be.ScaledDotProductAttention(q, kv, kv, q, nullptr, nullptr, 1, 1, rows, 128, 64, 0.125f, false, 0.f, 1);
  EXPECT(g_launches.back().second >= need || g_launches.back().first == nullptr);
  return g_launches.back().first;
}
static void* backward(CudaBackend& be, int64_t need) {
  g_need = need;
  const GpuBuffer b = buffer(64 * 4);
  be.FlashAttentionBackward(b, b, b, b, b, b, b, b, b, 1, 1, 4, 4, 64, 0.125f, false);
  EXPECT(g_launches.back().second >= need);
  return g_launches.back().first;
}
static void* layer(CudaBackend& be, int64_t need) {
  g_need = need;
  const GpuBuffer x = buffer(64 * 4), w = buffer(64 * 64);
  be.MultiHeadAttentionForward(x, w, w, w, w, x, 1, 4, 64, 1);
  EXPECT(g_launches.back().second >= need);
  return g_launches.back().first;
}
static bool live(void* p) { return g_live.count(p) == 1; }

static void destroy_graph(unsigned long long id) {
  for (auto* o : g_objects[id]) {
    o->first(o->second);
    delete o;
  }
  g_objects.erase(id);
}

static void graphs_keep_their_buffers() {
  CudaBackend be(0, nullptr);
  void* eager = attention(be, 100, 1);
  g_capture = 7;
  void* first = attention(be, 100, 1);
  EXPECT(attention(be, 50, 4) == first);          // the layers of one graph take turns with one buffer
  void* grown = attention(be, 300, 4);
  EXPECT(live(first));
  g_capture = 8;                                  // a second graph on the same stream: may be replayed beside the first
  void* second = attention(be, 100, 1);
  g_capture = 0;
  std::set<void*> recorded = {first, grown, second};
  EXPECT(recorded.size() == 3 && recorded.count(eager) == 0);
  // growth by every kind of call
  attention(be, 1000, 1);
  attention(be, 2000, 4);
  backward(be, 3000);
  void* last = layer(be, 4000);
  for (void* p : recorded) EXPECT(live(p) && p != last);
  EXPECT(!live(eager) && g_live.size() == 4);     // what no graph knows is given back
  destroy_graph(7);
  attention(be, 10, 1);
  EXPECT(live(second) && live(last) && g_live.size() == 2);
}

static void graphs_give_back() {
  {
    CudaBackend be(0, nullptr);
    for (unsigned long long id = 1; id <= 50; ++id) {   // a program that captures again and again
      g_capture = id;
      attention(be, 100, 1);
      g_capture = 0;
      if (id > 1) destroy_graph(id - 1);
    }
    EXPECT(g_live.size() <= 3);
  }
  EXPECT(g_live.empty());
  destroy_graph(50);                                    // the graph may outlive the backend
}

// A prefill that finds no memory for its optional buffer runs without one; the buffer that is there stays for decode calls.
static void optional_buffers() {
  CudaBackend be(0, nullptr);
  void* eager = attention(be, 100, 1);
  g_limit = 1000;
  EXPECT(attention(be, 2000, 4) == nullptr && live(eager) && attention(be, 100, 1) == eager);
  g_capture = 9;
  EXPECT(attention(be, 2000, 4) == nullptr);
  EXPECT(live(attention(be, 100, 1)));
  g_capture = 0;
  bool threw = false;
  try { attention(be, 2000, 1); } catch (const std::runtime_error&) { threw = true; }
  EXPECT(threw);
  EXPECT(live(attention(be, 500, 1)));
  g_limit = ~(size_t)0;
}

int main() {
  optional_buffers();
  EXPECT(g_live.empty());
  graphs_keep_their_buffers();
  EXPECT(g_live.empty());
  destroy_graph(8);
  graphs_give_back();
  std::printf(g_failed ? "%d checks failed\n" : "all cases passed\n", g_failed);
  return g_failed != 0;
}

// A stand-in for the CUDA runtime under the library's own host code: no GPU, kernels do nothing, device
// memory is host memory.  What it keeps of the runtime is the order that the documentation promises and no
// more: work on a stream happens when something waits for that stream, and cudaMemcpy from pageable memory
// returns once the bytes are staged -- they reach the device in the order of the legacy stream, which
// non-blocking streams do not follow.  Two devices; attributes of kernels belong to a device.
// Linked with the objects of epic_gb300/_lib by tests/host_library.py.
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

#define API extern "C" __attribute__((visibility("default")))

namespace {
struct Launch { std::string name; dim3 grid, block; size_t smem; unsigned cluster; };
struct Op { bool write; std::function<void()> run; };
struct Stream { int device = 0; std::vector<Op> ops; };
struct Event { double at = 0.; };
struct Graph { std::vector<Launch> nodes; };
struct Exec { std::vector<Launch> nodes; };

Stream legacy;
std::set<Stream *> streams;
std::map<const void *, std::string> names;
std::map<std::pair<int, std::string>, std::map<int, int>> attributes;   // of a device and kernel
std::vector<Launch> launches;
Graph *capturing = nullptr;
int device = 0, sms[2] = {152, 148}, cluster16[2] = {1, 1};
int streams_left = 1 << 30;
long graph_launches = 0, direct_launches = 0;
double clock_ms = 0.;   // what the GPU has done: a microsecond a kernel of a graph, ten of a direct launch

Stream *of(cudaStream_t s) { return s ? reinterpret_cast<Stream *>(s) : &legacy; }
void drain(Stream *s) {
  for (auto &o : s->ops) o.run();
  s->ops.clear();
}
cudaError_t launch(const std::string &name, dim3 g, dim3 b, size_t smem, unsigned cluster) {
  const auto &a = attributes[{device, name}];
  const auto at = [&](int k) { const auto i = a.find(k); return i == a.end() ? 0 : i->second; };
  if (cluster > 8 && !at(cudaFuncAttributeNonPortableClusterSizeAllowed)) return cudaErrorInvalidClusterSize;
  if (smem > 48 * 1024 && (int)smem > at(cudaFuncAttributeMaxDynamicSharedMemorySize)) return cudaErrorInvalidValue;
  const Launch l = {name, g, b, smem, cluster};
  launches.push_back(l);
  if (capturing) capturing->nodes.push_back(l);
  else { direct_launches++; clock_ms += .01; }
  return cudaSuccess;
}
std::vector<Launch> pushed;
std::vector<cudaStream_t> pushed_streams;
cudaError_t last = cudaSuccess;
cudaError_t note(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
}  // namespace

// ---- what a test asks ----
// copies and sets on other streams than s that nothing has waited for yet
API long fake_unordered_writes(void *s) {
  long n = 0;
  auto count = [&](Stream *t) { if (t != s) for (auto &o : t->ops) n += o.write; };
  count(&legacy);
  for (auto *t : streams) count(t);
  return n;
}
API void fake_reset_counts() { graph_launches = direct_launches = 0; launches.clear(); }
API long fake_graph_launches() { return graph_launches; }
API long fake_direct_launches() { return direct_launches; }
// launches whose kernel's name contains `part`; the cluster size, threads and grid of the last of them
API long fake_launches(const char *part, unsigned *cluster, unsigned *threads, unsigned *gx, unsigned *gy) {
  long n = 0;
  for (auto &l : launches)
    if (l.name.find(part) != std::string::npos) {
      n++;
      *cluster = l.cluster; *threads = l.block.x; *gx = l.grid.x; *gy = l.grid.y;
    }
  return n;
}
API void fake_streams_left(int n) { streams_left = n; }   // cudaStreamCreate fails after n more
API void fake_device(int d, int sm_count, int clusters_of_16) { sms[d] = sm_count; cluster16[d] = clusters_of_16; }

// ---- registration and launches ----
API void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
API void __cudaRegisterFatBinaryEnd(void **) {}
API void __cudaUnregisterFatBinary(void **) {}
API void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
API void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
  names[host] = name;
}
API cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *s) {
  pushed.push_back({"", g, b, smem, 1});
  pushed_streams.push_back(s);
  return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = pushed.back().grid; *b = pushed.back().block; *smem = pushed.back().smem;
  *(cudaStream_t *)s = pushed_streams.back();
  pushed.pop_back();
  pushed_streams.pop_back();
  return cudaSuccess;
}
API cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **, size_t smem, cudaStream_t) {
  return note(launch(names[(const void *)k], g, b, smem, 1));
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  unsigned cluster = 1;
  for (unsigned q = 0; q < c->numAttrs; q++)
    if (c->attrs[q].id == cudaLaunchAttributeClusterDimension)
      cluster = c->attrs[q].val.clusterDim.x * c->attrs[q].val.clusterDim.y * c->attrs[q].val.clusterDim.z;
  return note(launch(names[f], c->gridDim, c->blockDim, c->dynamicSmemBytes, cluster));
}
API cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) { attributes[{device, names[f]}][a] = v; return cudaSuccess; }
API cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) { *n = cluster16[device]; return cudaSuccess; }

// ---- devices, errors, memory ----
API cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
API cudaError_t cudaSetDevice(int d) { if (d < 0 || d > 1) return note(cudaErrorInvalidDevice); device = d; return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int d) { *v = a == cudaDevAttrMultiProcessorCount ? sms[d] : 0; return cudaSuccess; }
API cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
API const char *cudaGetErrorString(cudaError_t) { return "fake runtime error"; }
API cudaError_t cudaMalloc(void **p, size_t n) { *p = aligned_alloc(4096, (n + 4095) / 4096 * 4096); memset(*p, 0xAB, n); return cudaSuccess; }
API cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
API cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
API cudaError_t cudaFreeAsync(void *p, cudaStream_t) { free(p); return cudaSuccess; }
API cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
API cudaError_t cudaMallocHost(void **p, size_t n) { *p = malloc(n); return cudaSuccess; }
API cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
API cudaError_t cudaGetSymbolAddress(void **p, const void *) { static double table[1 << 16]; *p = table; return cudaSuccess; }
static cudaError_t copy(void *d, const void *s, size_t n, cudaMemcpyKind kind, Stream *t) {
  if (kind == cudaMemcpyHostToDevice) {   // pageable: the source is staged at once
    auto *b = new std::vector<char>((const char *)s, (const char *)s + n);
    t->ops.push_back({true, [=] { memcpy(d, b->data(), n); delete b; }});
  } else {
    t->ops.push_back({true, [=] { memcpy(d, s, n); }});
  }
  return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t t) { return copy(d, s, n, k, of(t)); }
API cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  copy(d, s, n, k, &legacy);
  if (k != cudaMemcpyHostToDevice) drain(&legacy);
  return cudaSuccess;
}
API cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t t) {
  of(t)->ops.push_back({true, [=] { memset(d, v, n); }});
  return cudaSuccess;
}

// ---- streams, events, graphs ----
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  if (streams_left-- <= 0) return note(cudaErrorMemoryAllocation);
  auto *t = new Stream;
  t->device = device;
  streams.insert(t);
  *s = reinterpret_cast<cudaStream_t>(t);
  return cudaSuccess;
}
API cudaError_t cudaStreamDestroy(cudaStream_t s) { drain(of(s)); streams.erase(of(s)); delete of(s); return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t s) { drain(of(s)); return cudaSuccess; }
API cudaError_t cudaStreamQuery(cudaStream_t s) { drain(of(s)); return cudaSuccess; }
API cudaError_t cudaStreamGetDevice(cudaStream_t s, int *d) { *d = of(s)->device; return cudaSuccess; }
API cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
API cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(new Event); return cudaSuccess; }
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
API cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event *>(e); return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { reinterpret_cast<Event *>(e)->at = clock_ms; return cudaSuccess; }
API cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
API cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(reinterpret_cast<Event *>(b)->at - reinterpret_cast<Event *>(a)->at);
  return cudaSuccess;
}
API cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = new Graph; return cudaSuccess; }
API cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = reinterpret_cast<cudaGraph_t>(capturing);
  capturing = nullptr;
  return cudaSuccess;
}
API cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t *n, size_t *count) {
  auto &v = reinterpret_cast<Graph *>(g)->nodes;
  if (n) for (size_t q = 0; q < v.size(); q++) n[q] = reinterpret_cast<cudaGraphNode_t>(&v[q]);
  *count = v.size();
  return cudaSuccess;
}
API cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType *t) { *t = cudaGraphNodeTypeKernel; return cudaSuccess; }
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
  *x = reinterpret_cast<cudaGraphExec_t>(new Exec{reinterpret_cast<Graph *>(g)->nodes});
  return cudaSuccess;
}
API cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph *>(g); return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete reinterpret_cast<Exec *>(x); return cudaSuccess; }
API cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  graph_launches++;
  clock_ms += .001 * (double)reinterpret_cast<Exec *>(x)->nodes.size();
  return cudaSuccess;
}

// the one driver function the library asks for
static CUresult encode_tiled(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
API cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **f, unsigned, unsigned long long, cudaDriverEntryPointQueryResult *r) {
  *f = (void *)encode_tiled;
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

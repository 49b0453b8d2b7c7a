// A CUDA runtime without a GPU, for tests of libtpo's host code on the CPU: the
// runtime calls libtpo makes, over host memory. Launches run nothing; they are
// checked against the rules a device enforces (function attributes belong to the
// current device) and written to a log that the test reads.
#include <cuda_runtime.h>
#include <cxxabi.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

namespace {
constexpr int kDevices = 2;
constexpr int kSms = 148;
constexpr size_t kSmemDefault = 48 * 1024, kSmemOptIn = 227 * 1024;

thread_local int t_dev = 0;
thread_local cudaError_t t_err = cudaSuccess;
std::mutex g_mu;
std::map<const void *, std::string> g_names;
std::map<std::tuple<int, const void *, int>, int> g_attr;  // device, function, attribute
int g_max_cluster[kDevices] = {16, 16};                    // CTAs a cluster can have
size_t g_max_smem[kDevices] = {kSmemOptIn, kSmemOptIn};    // dynamic shared memory a block can have
std::string g_log;

struct Call { dim3 grid, block; size_t smem; cudaStream_t stream; };
thread_local std::vector<Call> t_calls;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) t_err = e;
  return e;
}

int attr(const void *f, cudaFuncAttribute a) {
  auto it = g_attr.find({t_dev, f, (int)a});
  return it == g_attr.end() ? 0 : it->second;
}

// the launch's error, or none
cudaError_t check(const void *f, dim3 grid, dim3 block, size_t smem, int cluster, bool coop) {
  const size_t threads = (size_t)block.x * block.y * block.z;
  if (!grid.x || !grid.y || !grid.z || !threads || threads > 1024)
    return cudaErrorInvalidConfiguration;
  if (smem > std::max(kSmemDefault, (size_t)attr(f, cudaFuncAttributeMaxDynamicSharedMemorySize)))
    return cudaErrorInvalidValue;
  if (cluster > 1 && grid.x % cluster) return cudaErrorInvalidClusterSize;
  if (cluster > 8 && (!attr(f, cudaFuncAttributeNonPortableClusterSizeAllowed) ||
                      cluster > g_max_cluster[t_dev]))
    return cudaErrorInvalidClusterSize;
  if (coop && (size_t)grid.x * grid.y * grid.z > (size_t)kSms)
    return cudaErrorCooperativeLaunchTooLarge;
  return cudaSuccess;
}

cudaError_t launch(const void *f, dim3 grid, dim3 block, size_t smem, int cluster, bool coop) {
  std::lock_guard<std::mutex> lk(g_mu);
  const cudaError_t e = check(f, grid, block, smem, cluster, coop);
  char line[512];
  auto it = g_names.find(f);
  snprintf(line, sizeof line, "%d %s grid=%u threads=%u smem=%zu cluster=%d coop=%d err=%d\n", t_dev,
           it == g_names.end() ? "?" : it->second.c_str(), grid.x * grid.y * grid.z, block.x, smem,
           cluster, (int)coop, (int)e);
  g_log += line;
  return ret(e);
}
}  // namespace

extern "C" {
// ------------------------------------------------------------- the test's side
int fake_set_device(int d) { return cudaSetDevice(d); }
void fake_limits(int d, int max_cluster, size_t max_smem) {
  g_max_cluster[d] = max_cluster;
  g_max_smem[d] = max_smem;
}
const char *fake_log(void) {
  static std::string out;
  std::lock_guard<std::mutex> lk(g_mu);
  out.swap(g_log);
  g_log.clear();
  return out.c_str();
}

// ------------------------------------------------------------- registration
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 0; }
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *,
                            uint3 *, dim3 *, dim3 *, int *) {
  int st = 0;
  char *d = abi::__cxa_demangle(name, nullptr, nullptr, &st);
  std::string s = st == 0 ? d : name;
  free(d);
  s = s.substr(0, s.find('('));
  if (s.rfind("void ", 0) == 0) s = s.substr(5);
  s.erase(std::remove(s.begin(), s.end(), ' '), s.end());
  std::string bare;
  for (size_t i = 0; i < s.size(); ++i) {
    if (s.compare(i, 5, "tpo::") == 0) { i += 4; continue; }
    bare += s[i];
  }
  g_names[host] = bare;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st *s) {
  t_calls.push_back({g, b, smem, (cudaStream_t)s});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  const Call c = t_calls.back();
  t_calls.pop_back();
  *g = c.grid;
  *b = c.block;
  *smem = c.smem;
  *(cudaStream_t *)s = c.stream;
  return cudaSuccess;
}

// ------------------------------------------------------------- devices, functions
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= kDevices) return ret(cudaErrorInvalidDevice);
  t_dev = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = t_dev; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? kSms : a == cudaDevAttrL2CacheSize ? 126 << 20 : 1;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = t_err; t_err = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError(void) { return t_err; }
const char *cudaGetErrorString(cudaError_t e) {
  static thread_local char s[32];
  snprintf(s, sizeof s, "error %d", (int)e);
  return s;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && (size_t)v > g_max_smem[t_dev])
    return ret(cudaErrorInvalidValue);
  g_attr[{t_dev, f, (int)a}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int threads,
                                                                   size_t smem, unsigned) {
  *n = std::max(1, std::min(2048 / std::max(1, threads), (int)(kSmemOptIn / std::max<size_t>(1, smem))));
  *n = std::min(*n, 4);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c) {
  std::lock_guard<std::mutex> lk(g_mu);
  int cl = 1;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cl = c->attrs[i].val.clusterDim.x;
  *n = 0;
  const cudaError_t e = check(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, cl, false);
  if (e == cudaSuccess) *n = 4;
  return ret(e);
}

// ------------------------------------------------------------- launches
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t smem, cudaStream_t) {
  return launch(f, g, b, smem, 1, false);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **, size_t smem,
                                        cudaStream_t) {
  return launch(f, g, b, smem, 1, true);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  int cl = 1;
  bool coop = false;
  for (unsigned i = 0; i < c->numAttrs; ++i) {
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cl = c->attrs[i].val.clusterDim.x;
    if (c->attrs[i].id == cudaLaunchAttributeCooperative) coop = c->attrs[i].val.cooperative != 0;
  }
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, cl, coop);
}

// ------------------------------------------------------------- memory (the host's)
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  static char room[1 << 20];
  *p = room;
  return cudaSuccess;
}

// ------------------------------------------------------------- streams, events
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)malloc(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)malloc(8); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

// ------------------------------------------------------------- graphs
static char g_graph[8], g_node[8], g_body[8], g_exec[8];
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *,
                                          const cudaGraphEdgeData *, size_t, cudaStreamCaptureMode) {
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = (cudaGraph_t)g_graph; return cudaSuccess; }
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus *st, unsigned long long *,
                                        cudaGraph_t *g, const cudaGraphNode_t **deps, size_t *n) {
  *st = cudaStreamCaptureStatusActive;
  if (g) *g = (cudaGraph_t)g_graph;
  if (deps) *deps = nullptr;
  if (n) *n = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t *, size_t, unsigned) {
  return cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) { *g = (cudaGraph_t)g_graph; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphAddNode(cudaGraphNode_t *n, cudaGraph_t, const cudaGraphNode_t *, size_t,
                             cudaGraphNodeParams *p) {
  static cudaGraph_t body = (cudaGraph_t)g_body;
  *n = (cudaGraphNode_t)g_node;
  if (p->type == cudaGraphNodeTypeConditional) p->conditional.phGraph_out = &body;
  return cudaSuccess;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned,
                                             unsigned) {
  *h = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)g_exec;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
}

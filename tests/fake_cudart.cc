// fake_cudart.cc -- a CUDA runtime without a device, for CPU tests of the
// library's host path: linked in place of libcudart with the library's own,
// unchanged sources.
//
// Device memory is addresses only: allocations are counted against a settable
// capacity, so that out-of-memory paths and tables of any size can be driven
// here.  A kernel launch runs nothing; its parameters are searched for device
// addresses outside every live allocation.  A captured graph keeps copies of
// its launches' parameters and is searched again each time it is launched.
// Events complete at once and copies from the device give zeros.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

// Only the parameter structs are used of the device header; its device code
// wants these names declared.
#define __ldg(p) (*(p))
inline uint32_t __byte_perm(uint32_t, uint32_t, uint32_t) { return 0; }
inline uint32_t __funnelshift_l(uint32_t, uint32_t, uint32_t) { return 0; }
inline uint32_t __dp2a_lo(uint32_t, uint32_t, uint32_t) { return 0; }
inline uint32_t __dp4a(uint32_t, uint32_t, uint32_t) { return 0; }
inline uint32_t __shfl_sync(uint32_t, uint32_t, int, int) { return 0; }
#include "mg_device.cuh"

namespace {

constexpr uint64_t kBase = 0x700000000000ull, kSpan = 1ull << 46;
constexpr int kSms = 148;
constexpr size_t kSmemOptin = 227 * 1024, kSmemSm = 228 * 1024;

struct Launch {
  std::string kernel;
  std::vector<uint64_t> words;  // parameters, 8 bytes at a time
};

std::mutex mu;
uint64_t capacity = 178ull << 30, used = 0, peak = 0, next_addr = kBase;
bool reuse = false;                                  // freed addresses are handed out again (exact size)
std::map<uint64_t, uint64_t> live;                   // address -> bytes
std::map<uint64_t, std::vector<uint64_t>> freed;     // bytes -> addresses
uint64_t fail_mask = 0;                              // bit i: the i-th next allocation (device or pinned) fails
std::map<const void*, std::string>& kernels() {  // filled by other files' static initialisers
  static std::map<const void*, std::string> m;
  return m;
}
std::vector<Launch> graph_being_captured;
bool capturing = false;
uint64_t dead_launches = 0, graphs = 0, last_delta[4];
cudaError_t last_error = cudaSuccess;

bool alive(uint64_t a) {
  auto it = live.upper_bound(a);
  if (it == live.begin()) return false;
  --it;
  return a <= it->first + it->second;  // one past the end is a valid bound
}

// Parameter words of a kernel of the library, by its name.
std::vector<uint64_t> words_of(const std::string& name, void** args) {
  std::vector<uint64_t> w;
  auto add = [&](int i, size_t n) {
    for (size_t o = 0; o + 8 <= n; o += 8) {
      uint64_t v;
      std::memcpy(&v, (const char*)args[i] + o, 8);
      w.push_back(v);
    }
  };
  auto is = [&](const char* s) { return name.find(s) != std::string::npos; };
  if (is("scan_pair_kernel") || is("scan_block_kernel")) add(0, sizeof(mg::WarpScanParams));
  else if (is("scan_kernel")) add(0, sizeof(mg::ScanParams));
  else if (is("frontier_kernel")) add(0, sizeof(mg::FrontierStep));
  else if (is("delta_kernel")) {
    for (int i = 0; i < 7; ++i) add(i, 8);
    add(9, 8);
  } else if (is("reduce_kernel")) {
    add(0, 8);
    add(4, 8);
  } else if (is("copy_u4_kernel")) {
    add(0, 8);
    add(1, 8);
    add(3, 8);
  }
  return w;
}

void execute(const Launch& l) {
  bool ok = true;
  for (uint64_t v : l.words) ok = ok && !(v >= kBase && v < kBase + kSpan && !alive(v));
  dead_launches += ok ? 0 : 1;
  if (l.kernel.find("delta_kernel") != std::string::npos) {
    // keys, jobs, fr_seed, fr_t, idx, diffs, count, out
    last_delta[0] = l.words[1];
    for (int i = 1; i < 4; ++i) last_delta[i] = l.words[3 + i];
  }
}

cudaError_t launch(const void* f, void** args) {
  std::lock_guard<std::mutex> lk(mu);
  Launch l{kernels()[f], {}};
  l.words = words_of(l.kernel, args);
  if (capturing) graph_being_captured.push_back(l);
  else execute(l);
  return cudaSuccess;
}

cudaError_t fail(cudaError_t e) { return last_error = e; }

bool fail_now() {
  const bool f = fail_mask & 1u;
  fail_mask >>= 1;
  return f;
}

dim3 cfg_grid, cfg_block;
size_t cfg_smem;
cudaStream_t cfg_stream;

}  // namespace

// ---- controls for the tests ------------------------------------------------
extern "C" {
void fake_reset(uint64_t bytes, int reuse_addresses) {
  std::lock_guard<std::mutex> lk(mu);
  capacity = bytes;
  reuse = reuse_addresses != 0;
  fail_mask = dead_launches = graphs = 0;
  peak = used;
}
void fake_fail(uint64_t mask) { fail_mask = mask; }
uint64_t fake_used() { return used; }
uint64_t fake_peak() { return peak; }
uint64_t fake_dead_launches() { return dead_launches; }
uint64_t fake_graphs() { return graphs; }
void fake_last_delta(uint64_t out[4]) { std::memcpy(out, last_delta, sizeof last_delta); }

// ---- the runtime -----------------------------------------------------------
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  kernels()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  cfg_grid = g;
  cfg_block = b;
  cfg_smem = smem;
  cfg_stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = cfg_grid;
  *b = cfg_block;
  *smem = cfg_smem;
  *(cudaStream_t*)st = cfg_stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) { return launch(f, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void** args) { return launch(f, args); }

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = kSms;
  p->sharedMemPerBlockOptin = kSmemOptin;
  p->unifiedAddressing = p->canMapHostMemory = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? kSms : (int)kSmemOptin;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
  return v <= (int)kSmemOptin ? cudaSuccess : fail(cudaErrorInvalidValue);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int threads, size_t smem, unsigned) {
  *n = std::min((int)(kSmemSm / (smem + 1024)), 768 / threads > 0 ? 768 / threads : 1);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return fail(cudaErrorInvalidSymbol); }
cudaError_t cudaGetLastError() { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake CUDA error"; }

cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> lk(mu);
  if (fail_now() || n > capacity - used) return fail(cudaErrorMemoryAllocation);
  uint64_t a = 0;
  auto it = freed.find(n);
  if (reuse && it != freed.end() && !it->second.empty()) {
    a = it->second.back();
    it->second.pop_back();
  } else {
    a = next_addr;
    next_addr += (n + 4096) / 512 * 512;  // a gap behind every allocation
  }
  live[a] = n;
  used += n;
  peak = std::max(peak, used);
  *p = (void*)a;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> lk(mu);
  auto it = live.find((uint64_t)p);
  if (!p) return cudaSuccess;
  if (it == live.end()) return fail(cudaErrorInvalidValue);
  used -= it->second;
  freed[it->second].push_back(it->first);
  live.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  std::lock_guard<std::mutex> lk(mu);
  if (fail_now()) return fail(cudaErrorMemoryAllocation);
  *p = std::calloc(1, n ? n : 1);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  std::lock_guard<std::mutex> lk(mu);
  *f = capacity - used;
  *t = capacity;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind k, cudaStream_t) {
  if (n && (!dst || !src)) return fail(cudaErrorInvalidValue);
  if (k == cudaMemcpyDeviceToHost) std::memset(dst, 0, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(dst, src, n, k, nullptr); }
cudaError_t cudaMemset(void* p, int, size_t n) { return n && !p ? fail(cudaErrorInvalidValue) : cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.01f; return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  graph_being_captured.clear();
  capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capturing = false;
  *g = (cudaGraph_t) new std::vector<Launch>(graph_being_captured);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  ++graphs;
  *x = (cudaGraphExec_t) new std::vector<Launch>(*(std::vector<Launch>*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  std::lock_guard<std::mutex> lk(mu);
  for (const Launch& l : *(std::vector<Launch>*)x) execute(l);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (std::vector<Launch>*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete (std::vector<Launch>*)x; return cudaSuccess; }
}

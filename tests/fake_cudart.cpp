// A CUDA runtime without a GPU, for the host side of libgb300fea.so: kernels
// are recorded instead of run, "device" memory is host memory, and a launch is
// refused as the real runtime refuses it (dynamic shared memory above 48 KB
// without the kernel's attribute on the current device, a cooperative grid
// larger than the device).  The test sets the current device and its SMs, and
// may have a resident solve report a wait that ran out.
#include <cuda_runtime_api.h>
#include <cxxabi.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <set>
#include <string>
#include <utility>

namespace {

int g_device = 0, g_sms = 152, g_coop_limit = 152;
cudaError_t g_last = cudaSuccess;
std::map<const void*, std::string> g_names;
std::map<std::pair<int, const void*>, size_t> g_smem;  // (device, kernel): opted-in bytes
std::string g_log;

// The multi-kernel solve's scalar record: a residual of norm 1 after every
// residual kernel, and an iteration that ends at its first product.
struct Scalars {
  double rz, rr, pap, alpha, beta, bb, tol2, rr_true, absAx, ry;
  int32_t done, iters, status, max_iters;
};
Scalars* g_scalars = nullptr;

bool g_timed_out = false;  // the next resident solve reports a wait that ran out

struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_config;

std::string short_name(const char* mangled) {
  int st = 0;
  char* d = abi::__cxa_demangle(mangled, nullptr, nullptr, &st);
  std::string s = st == 0 ? d : mangled;
  free(d);
  if (s.rfind("void ", 0) == 0) s = s.substr(5);
  const std::string anon = "(anonymous namespace)::";
  for (size_t p; (p = s.find(anon)) != std::string::npos;) s.erase(p, anon.size());
  s = s.substr(0, s.find_first_of("<("));
  const size_t c = s.rfind("::");
  return c == std::string::npos ? s : s.substr(c + 2);
}

cudaError_t fail(cudaError_t e) { return g_last = e; }

cudaError_t record(const void* k, dim3 grid, dim3 block, size_t smem, bool coop, void** args) {
  const std::string name = g_names.count(k) ? g_names[k] : "?";
  const auto it = g_smem.find({g_device, k});
  const size_t limit = it == g_smem.end() ? 40 * 1024 : it->second;  // 48 KB with a static part of up to 8
  const size_t ctas = (size_t)grid.x * grid.y * grid.z;
  cudaError_t e = cudaSuccess;
  if (smem > limit) e = cudaErrorInvalidValue;
  if (coop && ctas > (size_t)g_coop_limit) e = cudaErrorCooperativeLaunchTooLarge;
  g_log += name + " grid " + std::to_string(ctas) + " block " + std::to_string(block.x) + " smem " +
           std::to_string(smem) + " device " + std::to_string(g_device) + (coop ? " cooperative" : "") +
           (e ? " refused" : "") + "\n";
  if (e) return fail(e);
  if (name == "bbox_kernel") {  // bounding box of a 100 x 20 x 20 box, from every block
    double* p = *static_cast<double**>(args[2]);
    for (unsigned b = 0; b < grid.x; ++b)
      for (int i = 0; i < 6; ++i) p[6 * b + i] = i < 3 ? 0.0 : (i == 3 ? 100.0 : 20.0);
  }
  if (name == "resid_comp_kernel" || name == "resid_kernel") {
    g_scalars = *static_cast<Scalars**>(args[7]);
    g_scalars->bb = g_scalars->rr_true = 1;
  }
  if (name.rfind("apply_", 0) == 0 && g_scalars) {
    g_scalars->done = 1;
    g_scalars->status = 5;
  }
  return cudaSuccess;
}

}  // namespace

extern "C" {

void fake_device(int device, int sms, int coop_limit) {
  g_device = device;
  g_sms = sms;
  g_coop_limit = coop_limit;
}
void fake_timed_out(int v) { g_timed_out = v != 0; }
void fake_clear() { g_log.clear(); }
const char* fake_log() { return g_log.c_str(); }

void** __cudaRegisterFatBinary(void*) {
  static void* h = nullptr;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  g_names[host] = short_name(name);
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = (cudaKernel_t)host;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  g_config = Config{grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = g_config.grid;
  *block = g_config.block;
  *smem = g_config.smem;
  *static_cast<cudaStream_t*>(stream) = g_config.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t) {
  return record((const void*)k, grid, block, smem, false, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* k, void** args) {
  bool coop = false;
  for (unsigned i = 0; i < c->numAttrs; ++i)
    coop |= c->attrs[i].id == cudaLaunchAttributeCooperative && c->attrs[i].val.cooperative;
  return record(k, c->gridDim, c->blockDim, c->dynamicSmemBytes, coop, args);
}
cudaError_t cudaFuncSetAttribute(const void* k, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_smem[{g_device, k}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = g_device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  if (a != cudaDevAttrMultiProcessorCount) return fail(cudaErrorInvalidValue);
  *v = g_sms;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = g_sms / 8;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  memmove(dst, src, n);
  if (kind == cudaMemcpyDeviceToHost && (n == 32 || n == 40) && g_timed_out) {  // a result, alone or with its flag
    const int32_t status = 9, flag = 1;
    memcpy(dst, &status, sizeof(status));
    if (n == 40) memcpy(static_cast<char*>(dst) + 32, &flag, sizeof(flag));
    g_timed_out = false;
  }
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbolAsync(void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static char scratch[16 << 20] __attribute__((aligned(256)));
  *p = scratch;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)1;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)2;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = nullptr;  // nothing captured: the solve launches directly
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return fail(cudaErrorInvalidValue); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return fail(cudaErrorInvalidValue); }

}  // extern "C"

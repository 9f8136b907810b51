// A stand-in for the CUDA runtime (and the cuBLAS handle calls) for tests of
// the library's host code without a GPU: device memory is host memory, kernels
// do not run, and every launch, copy and free is checked against the live
// allocations of the current device instead.  An allocation can be made to
// fail.  Linked with the library's objects into one shared object.
#include <cublas_v2.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

// the launch structs, from the kernels' header: device functions in it only
// have to compile
#include <algorithm>
#include <cmath>
using std::max;
static const uint3 threadIdx{};
template <class T>
T atomicAdd(T *, T);
template <class T>
T __shfl_sync(unsigned, T, int);
template <class T>
T __ldg(const T *);
int __double2loint(double);
double __hiloint2double(int, int);
double rsqrt(double);
#include "../hartreefock_b200/csrc/hfg_internal.cuh"

namespace {
constexpr int kDevices = 2;
constexpr int kDynamicShared = 48 * 1024;  // more needs the kernel's attribute on the device
struct Block {
  size_t bytes;
  int device;
};
struct Use {  // what a launch reads: [p, p + bytes)
  const void *p;
  size_t bytes;
  std::string what;
};
std::map<const char *, Block> blocks;
std::map<const void *, std::string> kernels;
std::map<const void *, std::pair<void *, size_t>> vars;
std::set<std::pair<const void *, int>> attributed;
std::map<const void *, int> stream_device, handle_device;
std::vector<Use> captured;
bool capturing = false;
int current = 0, fail_in = 0, allocations = 0, launches = 0;
size_t total_live = 0, peak_live = 0;
cudaError_t last = cudaSuccess;
std::string bad, log_;
struct Config {
  dim3 grid, block;
  size_t smem;
  void *stream;
} pushed;

void complain(const std::string &s) {
  if (bad.size() < 4000) bad += s + "\n";
}
cudaError_t error(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
void check(const Use &u) {
  const char *p = static_cast<const char *>(u.p);
  auto it = blocks.upper_bound(p);
  if (!p || it == blocks.begin()) return complain(u.what + ": not an allocation");
  --it;
  if (p + u.bytes > it->first + it->second.bytes) complain(u.what + ": outside its allocation, or freed");
  else if (it->second.device != current) complain(u.what + ": on another device");
}
void use(const void *p, size_t bytes, const std::string &what) {
  const Use u{p, bytes, what};
  if (capturing) captured.push_back(u);
  check(u);
}

// Entries of the allocation from p on.
template <class T>
long long entries(const T *p) {
  const char *q = reinterpret_cast<const char *>(p);
  auto it = blocks.upper_bound(q);
  if (it == blocks.begin()) return 0;
  --it;
  return (it->first + it->second.bytes - q) / (long long)sizeof(T);
}
int longest_run = 0;
// Every range of a grouped launch's tasks lies in its lists.
void check_group_tasks(const hfg::ClassLaunch &cl, const std::string &name) {
  if (cl.ntasks_dev || entries(cl.tasks) < cl.task_offset + cl.ntasks) return;
  for (int t = cl.task_offset; t < cl.task_offset + cl.ntasks; ++t) {
    const hfg::GroupTask g = hfg::group_task(cl.tasks[t]);
    longest_run = std::max(longest_run, g.nbra);
    if (g.nbra < 1 || g.nbra > hfg::kGroupMaxBras || g.nket < 1 || g.nket << g.lg > 32 ||
        g.bra_start + g.nbra > entries(cl.bra_list) || g.ket_start + g.nket > entries(cl.ket_list) ||
        (long long)g.mask_off + g.nbra > entries(cl.masks))
      complain(name + ": task outside its lists");
  }
}
}  // namespace

extern "C" {
// --- controls of the tests
void fake_fail_allocation(int n) { fail_in = n; }
int fake_allocations() { return allocations; }
int fake_launches() { return launches; }
long long fake_live_bytes() { return (long long)total_live; }
long long fake_peak_bytes(int restart) {
  if (restart) peak_live = total_live;
  return (long long)peak_live;
}
const char *fake_complaints() { return bad.c_str(); }
int fake_longest_run() {
  const int r = longest_run;
  longest_run = 0;
  return r;
}
const char *fake_log() { return log_.c_str(); }
long long fake_prim_pair_bytes() {
  return sizeof(hfg::PrimPair) + sizeof(hfg::PrimPairF) + hfg::kKetFields * sizeof(double);
}
double fake_far_T(int L) { return hfg::far_T(L); }
void fake_clear() {
  bad.clear();
  log_.clear();
}
void fake_set_device(int d) { current = d; }

// --- registration
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  kernels[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) {
  vars[host] = {nullptr, size};
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *s) {
  pushed = {g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = pushed.grid;
  *b = pushed.block;
  *smem = pushed.smem;
  *static_cast<void **>(s) = pushed.stream;
  return cudaSuccess;
}

// --- devices
cudaError_t cudaGetDeviceCount(int *n) {
  *n = kDevices;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  current = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = current;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *t = size_t(180) << 30;
  *f = *t - total_live;
  return cudaSuccess;
}

// --- memory
cudaError_t cudaMalloc(void **p, size_t n) {
  ++allocations;
  if (fail_in > 0 && --fail_in == 0) return error(cudaErrorMemoryAllocation);
  // every byte 0x3f: doubles of 4.8e-4, so that no quartet is screened
  char *q = static_cast<char *>(std::malloc(n ? n : 1));
  if (n <= (size_t(64) << 20)) std::memset(q, 0x3f, n);
  blocks[q] = {n, current};
  total_live += n;
  peak_live = total_live > peak_live ? total_live : peak_live;
  *p = q;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  auto it = blocks.find(static_cast<char *>(p));
  if (it == blocks.end()) {
    complain("cudaFree: not an allocation");
    return error(cudaErrorInvalidValue);
  }
  total_live -= it->second.bytes;
  blocks.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  if (k == cudaMemcpyHostToDevice) use(d, n, "copy to the device");
  if (k == cudaMemcpyDeviceToHost) use(s, n, "copy from the device");
  if (d && s) std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  use(d, n, "memset");
  if (n <= (size_t(64) << 20)) std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
  auto &v = vars[sym];
  if (!v.first) {
    const int keep = fail_in;
    fail_in = 0;
    cudaMalloc(&v.first, v.second);
    fail_in = keep;
  }
  *p = v.first;
  return cudaSuccess;
}

// --- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(new char[16]);
  stream_device[*s] = current;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  stream_device.erase(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new char[16]);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = true;
  captured.clear();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  capturing = false;
  *g = reinterpret_cast<cudaGraph_t>(new std::vector<Use>(captured));
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
  *x = reinterpret_cast<cudaGraphExec_t>(new std::vector<Use>(*reinterpret_cast<std::vector<Use> *>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<std::vector<Use> *>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  delete reinterpret_cast<std::vector<Use> *>(x);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  ++launches;
  for (Use u : *reinterpret_cast<std::vector<Use> *>(x)) {
    u.what = "graph replay: " + u.what;
    check(u);
  }
  return cudaSuccess;
}

// --- kernels
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int) {
  attributed.insert({f, current});
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t smem, cudaStream_t s) {
  using namespace hfg;
  ++launches;
  const std::string &name = kernels[f];
  if (smem > kDynamicShared && !attributed.count({f, current}))
    complain(name + ": more shared memory than the kernel is set to on this device");
  if (stream_device.count(s) && stream_device[s] != current) complain(name + ": stream of another device");
  const auto has = [&](const char *k) { return name.find(k) != std::string::npos; };
  if (has("eri_group_kernel") || has("eri_class_kernel") || has("eri_warp_kernel") || has("eri_prim_split_kernel") ||
      has("eri_hrr_")) {
    const ClassLaunch &cl = *static_cast<const ClassLaunch *>(args[1]);
    log_ += name + (cl.queue ? " queue\n" : "\n");
    use(cl.tasks, sizeof(Task) * (size_t)(cl.task_offset + cl.ntasks), name + " tasks");
    use(cl.bra_list, 4, name + " bra list");
    use(cl.ket_list, 4, name + " ket list");
    if (cl.queue) use(cl.queue, 4, name + " queue");
    if (cl.ntasks_dev) use(cl.ntasks_dev, 4, name + " task count");
    if (has("eri_group_kernel")) {
      use(cl.masks, sizeof(uint2), name + " masks");
      use(cl.ket_blocks, kKetStride * sizeof(double), name + " ket blocks");
      use(cl.ket_block_off, 4, name + " ket block offsets");
      check_group_tasks(cl, name);
    }
  } else if (has("group_masks_kernel")) {
    for (int a : {1, 2, 3, 4, 9}) use(*static_cast<void **>(args[a]), 4, name + " argument " + std::to_string(a));
  }
  return cudaSuccess;
}

// --- cuBLAS calls of the MO transforms
cublasStatus_t cublasCreate_v2(cublasHandle_t *h) {
  *h = reinterpret_cast<cublasHandle_t>(new char[16]);
  handle_device[*h] = current;
  return CUBLAS_STATUS_SUCCESS;
}
cublasStatus_t cublasDestroy_v2(cublasHandle_t h) {
  handle_device.erase(h);
  return CUBLAS_STATUS_SUCCESS;
}
cublasStatus_t cublasSetStream_v2(cublasHandle_t h, cudaStream_t) {
  if (handle_device.at(h) != current) complain("cuBLAS handle of another device");
  return CUBLAS_STATUS_SUCCESS;
}
static cublasStatus_t gemm(cublasHandle_t h, int m, int n, int k, const double *A, const double *B, double *C) {
  if (handle_device.at(h) != current) complain("cuBLAS handle of another device");
  use(A, 8, "GEMM A");
  use(B, 8, "GEMM B");
  use(C, 8, "GEMM C");
  return m > 0 && n > 0 && k > 0 ? CUBLAS_STATUS_SUCCESS : CUBLAS_STATUS_INVALID_VALUE;
}
cublasStatus_t cublasDgemm_v2(cublasHandle_t h, cublasOperation_t, cublasOperation_t, int m, int n, int k,
                              const double *, const double *A, int, const double *B, int, const double *, double *C,
                              int) {
  return gemm(h, m, n, k, A, B, C);
}
cublasStatus_t cublasDgemmStridedBatched(cublasHandle_t h, cublasOperation_t, cublasOperation_t, int m, int n, int k,
                                         const double *, const double *A, int, long long, const double *B, int,
                                         long long, const double *, double *C, int, long long, int) {
  return gemm(h, m, n, k, A, B, C);
}
}  // extern "C"

// A CUDA runtime without a GPU, for tests of the library's launch code: two devices of
// 148 SMs, device memory on the host, launches that are checked against the shared-memory
// limit of the current device and counted but run nothing, and cooperative launches that
// are refused beyond the SMs a test leaves free.
#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>

#include <cuda_runtime_api.h>
#include <cufft.h>

namespace {
constexpr int kSms = 148, kOptin = 227 * 1024, kDefault = 48 * 1024;
int device = 0, free_sms = kSms, launches = 0, refusals = 0, shared = 0,
    allocations = 0;
bool capturing = false;
cudaError_t last = cudaSuccess;
std::map<std::pair<int, const void*>, int> limit;  // raised limits: (device, kernel)
std::map<const void*, const char*>& names() {
  static std::map<const void*, const char*> m;  // filled while the library is loaded
  return m;
}
const char* last_kernel = "";
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} pending;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}

cudaError_t launch(const void* kernel, dim3 grid, size_t smem, bool cooperative) {
  const auto it = limit.find({device, kernel});
  cudaError_t e = cudaSuccess;
  if (smem > (size_t)(it == limit.end() ? kDefault : it->second)) e = cudaErrorInvalidValue;
  if (cooperative && (int)grid.x > free_sms) e = cudaErrorCooperativeLaunchTooLarge;
  ++(e == cudaSuccess ? launches : refusals);
  shared = (int)smem;
  last_kernel = names()[kernel];
  return ret(e);
}
}  // namespace

extern "C" {
int fake_launches() { return launches; }
int fake_allocations() { return allocations; }
void fake_capture(int on) { capturing = on; }
int fake_refusals() { return refusals; }
const char* fake_last_kernel() { return last_kernel; }
int fake_dynamic_smem() { return shared; }  // of the last launch
int fake_last_error() { return last; }
void fake_free_sms(int n) { free_sms = n; }
void fake_reset() {
  device = launches = refusals = 0;
  free_sms = kSms;
  capturing = false;
  last = cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? kSms : kOptin;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
  ++allocations;
  *p = calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) {
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void*, const void*, size_t, size_t, cudaMemcpyKind) {
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static int word;
  *p = &word;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return std::exchange(last, cudaSuccess); }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  memset(a, 0, sizeof *a);
  a->numRegs = 128;
  a->sharedSizeBytes = 128;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute, int v) {
  limit[{device, kernel}] = v;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* k, dim3 g, dim3, void**, size_t smem, cudaStream_t) {
  return launch(k, g, smem, false);
}
cudaError_t cudaLaunchCooperativeKernel(const void* k, dim3 g, dim3, void**, size_t smem,
                                        cudaStream_t) {
  return launch(k, g, smem, true);
}

// what compiled launches and kernels register with
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  pending = {g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = pending.grid;
  *b = pending.block;
  *smem = pending.smem;
  *(cudaStream_t*)s = pending.stream;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*,
                            void*, void*, int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

cufftResult cufftDestroy(cufftHandle) { return CUFFT_SUCCESS; }
cufftResult cufftSetStream(cufftHandle, cudaStream_t) { return CUFFT_SUCCESS; }
cufftResult cufftExecR2C(cufftHandle, cufftReal*, cufftComplex*) { return CUFFT_SUCCESS; }
cufftResult cufftExecC2R(cufftHandle, cufftComplex*, cufftReal*) { return CUFFT_SUCCESS; }
cufftResult cufftExecZ2D(cufftHandle, cufftDoubleComplex*, cufftDoubleReal*) {
  return CUFFT_SUCCESS;
}
cufftResult cufftPlan3d(cufftHandle* p, int, int, int, cufftType) { *p = 1; return CUFFT_SUCCESS; }
cufftResult cufftPlanMany(cufftHandle* p, int, int*, int*, int, int, int*, int, int, cufftType,
                          int) {
  *p = 1;
  return CUFFT_SUCCESS;
}
}

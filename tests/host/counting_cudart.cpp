// A CUDA runtime without a device: device memory is host memory, streams and
// events are handles, graph launches are counted.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

cudaError_t g_last = cudaSuccess;
int g_launched = 0;
// the one page-locked range and its place on the device
char *g_pin = nullptr, *g_pin_dev = nullptr;
size_t g_pin_bytes = 0;

static CUresult pointer_attributes(unsigned n, CUpointer_attribute* a, void** out, CUdeviceptr p) {
  char* c = (char*)p;
  const bool in = c >= g_pin && c < g_pin + g_pin_bytes;
  for (unsigned i = 0; i < n; ++i)
    if (a[i] == CU_POINTER_ATTRIBUTE_DEVICE_POINTER) *(CUdeviceptr*)out[i] = in ? (CUdeviceptr)(g_pin_dev + (c - g_pin)) : 0;
    else if (a[i] == CU_POINTER_ATTRIBUTE_RANGE_START_ADDR) *(CUdeviceptr*)out[i] = in ? (CUdeviceptr)g_pin : 0;
    else if (a[i] == CU_POINTER_ATTRIBUTE_RANGE_SIZE) *(size_t*)out[i] = in ? g_pin_bytes : 0;
    else return CUDA_ERROR_INVALID_VALUE;
  return CUDA_SUCCESS;
}

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 0; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) { *a = *b = 0; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free((void*)e); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidConfiguration ? "refused" : "other"; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free((void*)g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { free((void*)g); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)malloc(1); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { ++g_launched; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { *a = cudaPointerAttributes{}; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return cudaStreamCreateWithFlags(s, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free((void*)s); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusActive; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long, cudaDriverEntryPointQueryResult* st) {
  const bool known = !std::strcmp(name, "cuPointerGetAttributes");
  *f = known ? (void*)pointer_attributes : nullptr;
  *st = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
}

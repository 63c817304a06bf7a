// fake_cuda.cpp -- the runtime calls of fake_cuda.h.
#include "fake_cuda.h"

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { fake::work("memset", nullptr); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t st) { fake::work("memset", st); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    fake::work("memcpy", nullptr);   // (from pageable memory it may return before the copy is done)
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    fake::work("memcpy", st);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *st, unsigned)
{
    *st = (cudaStream_t)(fake::next += 16);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) { fake::wait("sync", st); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t st)
{
    ++fake::queries;
    if (fake::on_query) fake::on_query();
    return fake::left(st) ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaDeviceSynchronize()
{
    for (auto &p : fake::outstanding) p.second = 0;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)(fake::next += 16); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st)
{
    fake::log.push_back("record " + std::to_string((uintptr_t)e) + " " + std::to_string((uintptr_t)st));
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned)
{
    fake::log.push_back("wait " + std::to_string((uintptr_t)e) + " " + std::to_string((uintptr_t)st));
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = nullptr; return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceFlags(unsigned *f) { *f = fake::device_flags | cudaDeviceMapHost; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
}

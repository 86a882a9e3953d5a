// The functions of the fake CUDA runtime (fake_cuda.h).
#include "fake_cuda.h"

#include <chrono>

#define FAKE_CALL(name) \
    if (fake::fails(name)) return cudaErrorUnknown; \
    fake::State& s = fake::state();                \
    std::lock_guard<std::recursive_mutex> lock(s.mu)

extern "C" {

cudaError_t cudaMalloc(void** p, size_t n) {
    FAKE_CALL("cudaMalloc");
    s.mallocs++;
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    s.device[(char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    FAKE_CALL("cudaFree");
    s.device.erase((char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* p, size_t n, cudaMemcpyKind k) {
    FAKE_CALL("cudaMemcpy");
    fake::copy("cudaMemcpy", d, p, n, nullptr);
    if (k != cudaMemcpyHostToDevice) s.host |= s.stream[nullptr];
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* p, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (fake::state().pause_us) std::this_thread::sleep_for(std::chrono::microseconds(fake::state().pause_us));
    FAKE_CALL("cudaMemcpyAsync");
    fake::copy("cudaMemcpyAsync", d, p, n, st);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    FAKE_CALL("cudaMemset");
    memset(d, v, n);
    fake::enqueue("cudaMemset", nullptr, {{(char*)d, n, true}});
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) {
    FAKE_CALL("cudaStreamCreateWithFlags");
    *st = (cudaStream_t)malloc(64);
    s.live_streams.insert(*st);
    s.stream[*st] = fake::Ops();
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t st) {
    FAKE_CALL("cudaStreamDestroy");
    s.live_streams.erase(st);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    FAKE_CALL("cudaStreamSynchronize");
    s.host |= s.stream[st == cudaStreamLegacy ? nullptr : st];
    fake::waited();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
    FAKE_CALL("cudaStreamWaitEvent");
    s.stream[st] |= s.event[e];
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus* c) {
    FAKE_CALL("cudaStreamIsCapturing");
    *c = s.capturing.count(st) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* mode) {
    FAKE_CALL("cudaThreadExchangeStreamCaptureMode");
    static thread_local cudaStreamCaptureMode now = cudaStreamCaptureModeGlobal;
    std::swap(now, *mode);
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t st, cudaStreamCaptureMode) {
    FAKE_CALL("cudaStreamBeginCapture");
    s.capturing.insert(st);
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t* g) {
    FAKE_CALL("cudaStreamEndCapture");
    s.capturing.erase(st);
    *g = (cudaGraph_t)malloc(64);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    FAKE_CALL("cudaGraphInstantiate");
    *e = (cudaGraphExec_t)malloc(64);
    return cudaSuccess;
}
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) {
    FAKE_CALL("cudaGraphUpload");
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
    FAKE_CALL("cudaGraphLaunch");
    fake::enqueue("graph", st, {});
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    free(g);
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof(*p));
    strcpy(p->name, "fake GPU");
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    FAKE_CALL("cudaEventCreateWithFlags");
    *e = (cudaEvent_t)malloc(64);
    s.live_events.insert(*e);
    s.event[*e] = fake::Ops();
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    FAKE_CALL("cudaEventDestroy");
    s.live_events.erase(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    FAKE_CALL("cudaEventRecord");
    s.event[e] = s.stream[st];
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* kernel, void** args) {
    FAKE_CALL("cudaLaunchKernelExC");
    bool cooperative = false, overlap = false;
    for (unsigned i = 0; i < c->numAttrs; i++)
        cooperative = cooperative || (c->attrs[i].id == cudaLaunchAttributeCooperative && c->attrs[i].val.cooperative);
    for (unsigned i = 0; i < c->numAttrs; i++)
        overlap = overlap || (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
                              c->attrs[i].val.programmaticStreamSerializationAllowed);
    fake::enqueue("launch", c->stream, s.kernel_spans ? s.kernel_spans(kernel, args) : std::vector<fake::Span>(),
                  cooperative, overlap);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* k, cudaFuncAttribute a, int) {
    FAKE_CALL("cudaFuncSetAttribute");
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) s.attributes.insert({k, s.current_device});
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
    FAKE_CALL("cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    FAKE_CALL("cudaGetDevice");
    *d = s.current_device;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    FAKE_CALL("cudaDeviceGetAttribute");
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    FAKE_CALL("cudaGetSymbolAddress");
    static char area[65536];
    *p = area;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    FAKE_CALL("cudaPointerGetAttributes");
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    for (auto& r : s.pinned)
        if ((const char*)p >= r.first && (const char*)p < r.first + r.second) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
static int fake_address_range(unsigned long long* base, size_t* size, unsigned long long p) {
    fake::State& s = fake::state();
    std::lock_guard<std::recursive_mutex> lock(s.mu);
    auto it = s.device.upper_bound((char*)p);
    if (it == s.device.begin()) return 1;
    --it;
    *base = (unsigned long long)it->first;
    *size = it->second;
    return 0;
}
// a query of a stream under capture would end the capture
static int fake_stream_query(cudaStream_t st) {
    if (fake::state().capturing.count(st)) abort();
    return fake::state().busy.count(st) ? 600 : 0;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
    if (fake::state().pause_us) std::this_thread::sleep_for(std::chrono::microseconds(fake::state().pause_us));
    *f = !strcmp(name, "cuMemGetAddressRange") ? (void*)fake_address_range
         : !strcmp(name, "cuStreamQuery")      ? (void*)fake_stream_query
                                               : nullptr;
    *q = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the fake runtime"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }

// what compiled kernels register with
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

}  // extern "C"

// A CUDA runtime that runs nothing: device memory is host memory, a kernel launch is a line in a list. Linked with the library's
// objects in place of the real one it shows on the CPU which kernels a call launches, with which grid, and which of them may start
// ahead of their predecessor's end.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string name;
    dim3 grid, block;
    size_t smem;
    bool dependent;  // may start before the kernel ahead of it has ended
};
std::vector<Launch> launches;
std::map<const void*, std::string>& kernels() {  // registered by static constructors of the objects
    static std::map<const void*, std::string> names;
    return names;
}
Launch pushed;
int sms = 148;
bool capturing = false;
int handle;
int encode_nothing(...) { return 0; }
void record(const void* f, dim3 grid, dim3 block, size_t smem, bool dependent) {
    launches.push_back(Launch{kernels()[f], grid, block, smem, dependent});
}
}  // namespace

extern "C" {

// ---- the list
void seen_clear() { launches.clear(); }
unsigned seen_count() { return (unsigned)launches.size(); }
const char* seen_name(unsigned i) { return launches[i].name.c_str(); }
void seen_shape(unsigned i, unsigned* out) {
    const Launch& l = launches[i];
    const unsigned v[6] = {l.grid.x, l.grid.y, l.grid.z, l.block.x, (unsigned)l.smem, l.dependent};
    memcpy(out, v, sizeof(v));
}
void set_sms(int n) { sms = n; }
void set_capturing(int on) { capturing = on; }

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(&handle); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void*) {
    pushed.grid = grid;
    pushed.block = block;
    pushed.smem = smem;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = pushed.grid;
    *block = pushed.block;
    *smem = pushed.smem;
    *static_cast<void**>(stream) = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
    record(f, grid, block, smem, false);
    return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
    record(f, grid, block, smem, false);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    bool dependent = false;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
            dependent = c->attrs[i].val.programmaticStreamSerializationAllowed;
    record(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, dependent);
    return cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = nullptr;
    if (posix_memalign(p, 256, n ? n : 1)) return cudaErrorMemoryAllocation;
    memset(*p, 0, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static unsigned long long words[64];
    *p = words;
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, size_t n, size_t, cudaMemcpyKind) {
    memset(d, 0, n);
    return cudaSuccess;
}

// ---- the rest
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? sms : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 1;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = reinterpret_cast<void*>(&encode_nothing);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = reinterpret_cast<cudaGraph_t>(&handle);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) {
    *g = reinterpret_cast<cudaGraphExec_t>(&handle);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    launches.push_back(Launch{"graph", dim3(1), dim3(1), 0, false});
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
}

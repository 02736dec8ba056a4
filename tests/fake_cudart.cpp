// A CUDA runtime on the host for the tests of the network entries' workspace:
// device memory is host memory, kernels do not run, and every allocation and
// event belongs to the context it was made in.  A context ends with a reset of
// its device; a use of what it held is counted (fake_errors), not made.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

namespace {
struct Obj {
    int dev;
    unsigned long long ctx;
    size_t bytes;
};
std::mutex mu;
std::map<void*, Obj> objs;                // live
std::map<void*, Obj> dead;                // ended with their context
unsigned long long ctx_of[2] = {0, 0};    // 0: no context on the device
unsigned long long next_ctx = 1;
int errors = 0, fail_attribute = 0;
thread_local int cur_dev = 0;

unsigned long long context() {   // the device's context, made at its first use
    if (!ctx_of[cur_dev]) ctx_of[cur_dev] = next_ctx++;
    return ctx_of[cur_dev];
}
cudaError_t make(void** p, size_t bytes) {
    std::lock_guard<std::mutex> g(mu);
    *p = std::calloc(1, bytes ? bytes : 1);
    objs[*p] = Obj{cur_dev, context(), bytes};
    return cudaSuccess;
}
cudaError_t end(void* p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> g(mu);
    if (!objs.erase(p)) {
        errors++;
        return cudaErrorInvalidValue;
    }
    std::free(p);
    return cudaSuccess;
}
// p lies in an object that ended with its context
bool stale(const void* p) {
    for (auto& o : dead)
        if (p >= o.first && (const char*)p < (const char*)o.first + o.second.bytes) return true;
    return false;
}
cudaError_t use(const void* p) {
    std::lock_guard<std::mutex> g(mu);
    if (!stale(p)) return cudaSuccess;
    errors++;
    return cudaErrorInvalidValue;
}

// driver entries: a context handle is the address of its device's id
CUresult ctx_current(CUcontext* c) {
    std::lock_guard<std::mutex> g(mu);
    *c = ctx_of[cur_dev] ? (CUcontext)&ctx_of[cur_dev] : nullptr;
    return CUDA_SUCCESS;
}
CUresult ctx_id(CUcontext c, unsigned long long* id) {
    std::lock_guard<std::mutex> g(mu);
    *id = c ? *(unsigned long long*)c : 0;
    return *id ? CUDA_SUCCESS : CUDA_ERROR_CONTEXT_IS_DESTROYED;
}
CUresult primary_state(CUdevice d, unsigned* flags, int* active) {
    std::lock_guard<std::mutex> g(mu);
    *flags = 0;
    *active = ctx_of[d] != 0;
    return CUDA_SUCCESS;
}
CUresult primary_retain(CUcontext* c, CUdevice d) {
    *c = (CUcontext)&ctx_of[d];
    return CUDA_SUCCESS;
}
CUresult primary_release(CUdevice) { return CUDA_SUCCESS; }
}  // namespace

extern "C" {
// ---- the tests' handles -------------------------------------------------
void fake_device(int d) { cur_dev = d; }
void fake_fail_attribute(int on) { fail_attribute = on; }
int fake_errors() { return errors; }
int fake_live(int dev) {
    std::lock_guard<std::mutex> g(mu);
    int n = 0;
    for (auto& o : objs) n += o.second.dev == dev;
    return n;
}
void fake_reset() {   // cudaDeviceReset of the current device
    std::lock_guard<std::mutex> g(mu);
    for (auto it = objs.begin(); it != objs.end();)
        if (it->second.dev == cur_dev) {
            dead.insert(*it);
            it = objs.erase(it);
        } else {
            ++it;
        }
    ctx_of[cur_dev] = 0;
}

// ---- the runtime ------------------------------------------------------------
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
static thread_local struct {
    dim3 g, b;
    size_t s;
    void* st;
} conf;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
    conf.g = g;
    conf.b = b;
    conf.s = s;
    conf.st = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
    *g = conf.g;
    *b = conf.b;
    *s = conf.s;
    *(void**)st = conf.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = cur_dev;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 4;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return make(p, n); }
cudaError_t cudaFree(void* p) {
    if (!p) {
        std::lock_guard<std::mutex> g(mu);
        context();
        return cudaSuccess;
    }
    return end(p);
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return make(p, n); }
cudaError_t cudaFreeHost(void* p) { return end(p); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return make((void**)e, 8); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return end(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return use(e); }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t a, cudaEvent_t b) {
    *t = 1.f;
    const cudaError_t ra = use(a), rb = use(b);
    return ra ? ra : rb;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
    if (cudaError_t e = use(p)) return e;
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (cudaError_t e = use(d)) return e;
    if (cudaError_t e = use(s)) return e;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
    return fail_attribute ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    struct {
        const char* n;
        void* f;
    } t[] = {{"cuCtxGetCurrent", (void*)ctx_current},
             {"cuCtxGetId", (void*)ctx_id},
             {"cuDevicePrimaryCtxGetState", (void*)primary_state},
             {"cuDevicePrimaryCtxRetain", (void*)primary_retain},
             {"cuDevicePrimaryCtxRelease", (void*)primary_release}};
    *f = nullptr;
    for (auto& e : t)
        if (!std::strcmp(e.n, name)) *f = e.f;
    if (q) *q = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
}

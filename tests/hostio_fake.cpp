// The host-side transfers (csrc/hostio.cu) over a CUDA runtime of plain memory:
// "device" arrays are host arrays, copies happen at once, and every call that
// pins memory or copies is counted.  Built by tests/test_hostio.py.
#include "hostio.cu"

#include <cstdlib>
#include <map>

namespace {
std::mutex g;
std::map<void*, size_t> g_pinned;  // start -> bytes
size_t g_pinned_now = 0, g_pinned_sum = 0, g_pins = 0;
size_t g_copies = 0, g_pinned_copies = 0;  // copies; of them through pinned memory
int g_refuse_pins = 0;                     // pinned memory is not to be had

bool is_pinned(const void* p) {
    auto it = g_pinned.upper_bound(const_cast<void*>(p));
    if (it == g_pinned.begin()) return false;
    --it;
    return (const char*)p < (const char*)it->first + it->second;
}
cudaError_t pin(void* p, size_t bytes) {
    std::lock_guard<std::mutex> lk(g);
    g_pinned[p] = bytes;
    g_pinned_now += bytes;
    g_pinned_sum += bytes;
    g_pins++;
    return cudaSuccess;
}
cudaError_t unpin(void* p) {
    std::lock_guard<std::mutex> lk(g);
    auto it = g_pinned.find(p);
    if (it == g_pinned.end()) return cudaErrorInvalidValue;
    g_pinned_now -= it->second;
    g_pinned.erase(it);
    return cudaSuccess;
}
}  // namespace

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    if (g_refuse_pins) return cudaErrorMemoryAllocation;
    *p = aligned_alloc(4096, (bytes + 4095) / 4096 * 4096);
    return pin(*p, bytes);
}
cudaError_t cudaFreeHost(void* p) {
    const cudaError_t e = unpin(p);
    free(p);
    return e;
}
cudaError_t cudaHostRegister(void* p, size_t bytes, unsigned) {
    return g_refuse_pins ? cudaErrorMemoryAllocation : pin(p, bytes);
}
cudaError_t cudaHostUnregister(void* p) { return unpin(p); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = (cudaEvent_t)1;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> lk(g);
    a->type = is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t bytes, cudaMemcpyKind kind, cudaStream_t) {
    {
        std::lock_guard<std::mutex> lk(g);
        g_copies++;
        g_pinned_copies += is_pinned(kind == cudaMemcpyHostToDevice ? s : d);
    }
    memcpy(d, s, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind kind, cudaStream_t st) {
    for (size_t k = 0; k < h; k++)
        cudaMemcpyAsync((char*)d + k * dp, (const char*)s + k * sp, w, kind, st);
    return cudaSuccess;
}

// ---- for the test --------------------------------------------------------
#define API __attribute__((visibility("default")))
API void* t_open(int rows, size_t bytes) {
    nb::HostIO* io = new nb::HostIO();
    if (!nb::hostio_init(*io, 0, rows, bytes)) {
        nb::hostio_free(*io);
        delete io;
        return nullptr;
    }
    memset(io->extra(), 1, nb::kHostExtra);
    return io;
}
API void t_close(void* h) {
    nb::hostio_free(*(nb::HostIO*)h);
    delete (nb::HostIO*)h;
}
API int t_up(void* h, int n, void** dst, void** src, size_t bytes) {
    std::vector<nb::CopySeg> seg;
    for (int k = 0; k < n; k++) seg.push_back({dst[k], src[k], bytes});
    return (int)nb::copy_up(*(nb::HostIO*)h, nullptr, seg.data(), n);
}
API int t_down(void* h, int n, void** dst, void** src, size_t bytes) {
    std::vector<nb::CopySeg> seg;
    for (int k = 0; k < n; k++) seg.push_back({dst[k], src[k], bytes});
    bool queued = false;
    cudaError_t e = nb::start_down(*(nb::HostIO*)h, nullptr, seg.data(), n, &queued);
    if (e == cudaSuccess) e = nb::finish_down(*(nb::HostIO*)h, nullptr, seg.data(), n, queued);
    return (int)e;
}
// pinned now, pinned ever, pins, copies, copies through pinned memory
API void t_counts(size_t* out) {
    std::lock_guard<std::mutex> lk(g);
    const size_t c[5] = {g_pinned_now, g_pinned_sum, g_pins, g_copies, g_pinned_copies};
    memcpy(out, c, sizeof(c));
}
// The start of some pinned memory, and its bytes.
API void t_some_pinned(size_t* out) {
    std::lock_guard<std::mutex> lk(g);
    out[0] = (size_t)g_pinned.begin()->first;
    out[1] = g_pinned.begin()->second;
}
API void t_refuse_pins(int on) { g_refuse_pins = on; }
}

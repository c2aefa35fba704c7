// csrc/stride_api.cu's host code on a fake CUDA runtime: memory is the host's
// and freed blocks are only marked, events know whether a capture recorded
// them, and the launches write what the test says.  For the lifetimes of
// handles, which a failing launch or allocation tests without a GPU.
#include "../meshpress_gb300/csrc/stride_api.cu"

#include <map>
#include <set>

namespace {

struct Ev {
    bool recorded = false, captured = false;
};
std::map<void*, size_t> g_bytes;  // of every block ever
std::set<void*> g_freed;
size_t g_most = ~size_t(0);  // cudaMalloc fails above
void* g_capturing = nullptr; // the stream in capture
int g_decode_rc = 0;
unsigned long long g_decode_err = 0;
uint32_t g_scans = 0, g_outputs = 0;  // launches that read or wrote a handle's records
bool g_freed_used = false;            // ... of memory that had been given back
std::set<void*> g_pending;            // streams with work that no one has waited for
Status* g_status = nullptr;
uint8_t* g_arena = nullptr;

Ev* ev(cudaEvent_t e) { return reinterpret_cast<Ev*>(e); }

bool freed(const void* p) {
    for (void* q : g_freed)
        if (p >= q && p < static_cast<uint8_t*>(q) + g_bytes[q]) return true;
    return false;
}

void records(const void* p) {
    g_freed_used = g_freed_used || freed(p);
    g_outputs++;
}

}  // namespace

extern "C" {

cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMalloc(void** p, size_t n) {
    if (n > g_most) return *p = nullptr, cudaErrorMemoryAllocation;
    *p = std::calloc(1, n);
    g_bytes[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p) g_freed.insert(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    return *e = reinterpret_cast<cudaEvent_t>(new Ev), cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete ev(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    ev(e)->recorded = true;
    ev(e)->captured = s != nullptr && s == g_capturing;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return ev(e)->captured ? cudaErrorCapturedEvent : cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.0f, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(new int), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return delete reinterpret_cast<int*>(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return g_pending.erase(s), cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
    *c = s != nullptr && s == g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    const bool cap = s != nullptr && s == g_capturing;
    if (ev(e)->captured && !cap) return cudaErrorCapturedEvent;
    return cap && !ev(e)->captured ? cudaErrorStreamCaptureIsolation : cudaSuccess;
}

// ---- the test's side
void fake_reset() {
    g_most = ~size_t(0);
    g_capturing = nullptr;
    g_decode_rc = 0;
    g_decode_err = 0;
    g_scans = g_outputs = 0;
    g_freed_used = false;
    g_pending.clear();
}
void fake_most(size_t n) { g_most = n; }
void fake_capture(void* s) { g_capturing = s; }
void fake_decode(int rc, unsigned long long err) { g_decode_rc = rc, g_decode_err = err; }
void fake_replay(unsigned long long err) { g_status->err = err; }  // of the last decode that was enqueued
uint32_t fake_outputs() { return g_outputs; }
int fake_pending(void* s) { return static_cast<int>(g_pending.count(s)); }
int fake_freed_used() { return g_freed_used ? 1 : 0; }
// whether the last decode's status word and bytes have gone back to the driver
int fake_returned() { return freed(g_status) && freed(g_arena) ? 1 : 0; }

}  // extern "C"

namespace stride {

int device_sm_count() { return 152; }
int check_config(const LaunchCfg&, bool) { return STRIDE_OK; }
LaunchCfg default_config(uint32_t, uint64_t, uint32_t, bool) {
    LaunchCfg c;
    c.persistent = 4;
    return c;
}
void last_launch(uint32_t* smem, uint32_t* grid) { *smem = *grid = 0; }
int enqueue_decode(const DecodeArgs& a, const LaunchCfg&, void* s, void* const*) {
    g_scans++;  // queued, whatever becomes of the kernel behind it
    g_pending.insert(s);
    g_status = a.status;
    g_arena = const_cast<uint8_t*>(a.arena);
    a.status->err = g_decode_err;
    return g_decode_rc;
}
int enqueue_part(const DecodeArgs&, const LaunchCfg&, void*, uint32_t, uint32_t, bool, void*, void*, void*) { return 0; }
int enqueue_parts_begin(const DecodeArgs&, const LaunchCfg&, void*) { return 0; }
int enqueue_parts_end(const DecodeArgs&, const LaunchCfg&, void*, void*) { return 0; }
int enqueue_cull(const float*, uint32_t, const Planes&, uint32_t*, uint32_t*, void*) { return 0; }
int enqueue_normalise(const int32_t*, unsigned long long, const NormAxes&, float*, void*) { return 0; }
int enqueue_side_table(const MeshletDesc* d, uint32_t, unsigned long long*, uint16_t*, void*) { return records(d), 0; }
int enqueue_meshlet_bounds(const MeshletDesc* d, const BlockPrefix*, uint32_t, const float*, float*, void*) {
    return records(d), 0;
}
int enqueue_meshlet_ranges(const MeshletDesc* d, const BlockPrefix*, uint32_t, unsigned long long*,
                           unsigned long long*, void*) {
    return records(d), 0;
}

}  // namespace stride

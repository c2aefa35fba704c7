// C ABI of the single-mesh decoder (include/stride_gb300.h): host header
// parse, device buffers, enqueue and status.
#include <cuda_runtime.h>

#include <algorithm>
#include <bitset>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <unordered_map>
#include <vector>

#include "stride_common.cuh"
#include "stride_gb300.h"
#include "stride_internal.h"

namespace stride {

thread_local std::string g_last_error;

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    return fail(STRIDE_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

static uint32_t be32(const uint8_t* p) {
    return (static_cast<uint32_t>(p[0]) << 24) | (static_cast<uint32_t>(p[1]) << 16) |
           (static_cast<uint32_t>(p[2]) << 8) | p[3];
}

static float bef32(const uint8_t* p) {
    const uint32_t u = be32(p);
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

// Global header of a DPR4 v3 stream (encoder/paradelta_v5_dup.py:412-447,
// read back at :472-501).
int parse_header(const uint8_t* data, size_t len, MeshParams* p, char* why, size_t why_len) {
    auto say = [&](int code, const char* msg) {
        if (why && why_len) snprintf(why, why_len, "%s", msg);
        return code;
    };
    std::memset(p, 0, sizeof(*p));
    if (!data) return say(STRIDE_ERR_ARG, "null stream");
    if (len < kHeaderBytes) return say(STRIDE_ERR_TRUNCATED, "stream shorter than the 86-byte DPR4 header");
    if (be32(data) != kMagic) {
        char m[96];
        snprintf(m, sizeof(m), "bad magic 0x%08X (expected DPR4 0x44505234)", be32(data));
        return say(STRIDE_ERR_MAGIC, m);
    }
    if (data[4] != kVersion) {
        char m[64];
        snprintf(m, sizeof(m), "DPR4 version %u (expected 3)", data[4]);
        return say(STRIDE_ERR_VERSION, m);
    }
    float center[3], gmin[3], grange[3];
    for (int i = 0; i < 3; i++) center[i] = bef32(data + 6 + 4 * i);
    const float scale = bef32(data + 18);
    for (int i = 0; i < 3; i++) gmin[i] = bef32(data + 26 + 4 * i);
    for (int i = 0; i < 3; i++) grange[i] = bef32(data + 38 + 4 * i);
    for (int i = 0; i < 3; i++) p->g_bits[i] = data[50 + i];
    for (int i = 0; i < 9; i++) {
        const uint32_t v = (static_cast<uint32_t>(data[53 + 2 * i]) << 8) | data[54 + 2 * i];
        p->pred_n[i] = (v & 0x8000u) ? static_cast<int32_t>(v) - 0x10000 : static_cast<int32_t>(v);
    }
    for (int i = 0; i < 3; i++) p->pred_k[i] = data[71 + i];
    p->n_v = be32(data + 74);
    p->n_t = be32(data + 78);
    p->n_meshlets = be32(data + 82);
    const unsigned long long table_end = kHeaderBytes + 4ull * p->n_meshlets;
    if (table_end > len) return say(STRIDE_ERR_TRUNCATED, "offset table runs past the end of the stream");
    if (len * 8ull >= (1ull << 32) - 4096) return say(STRIDE_ERR_UNSUPPORTED, "stream longer than 512 MB");
    if (p->n_meshlets == 0) return say(STRIDE_ERR_CORRUPT, "stream has no meshlets");
    for (int d = 0; d < 3; d++) {
        if (p->g_bits[d] > static_cast<uint32_t>(kMaxGBits))
            return say(STRIDE_ERR_UNSUPPORTED, "more than 24 bits per axis");
        if (p->pred_k[d] > 30) return say(STRIDE_ERR_UNSUPPORTED, "predictor shift K above 30");
        p->code_max[d] = (1u << p->g_bits[d]) - 1u;
        p->pred_half[d] = p->pred_k[d] ? (1 << (p->pred_k[d] - 1)) : 0;
        // the int32 IRLP sum of in-range codes must not overflow
        long long bound = 0;
        for (int j = 0; j < 3; j++) bound += std::llabs(static_cast<long long>(p->pred_n[3 * d + j]));
        bound = bound * static_cast<long long>(p->code_max[d]) + p->pred_half[d];
        if (bound >= (1ll << 31)) return say(STRIDE_ERR_UNSUPPORTED, "IRLP weights overflow int32 arithmetic");
        stride_dequant_setup(&p->dq[d], center[d], scale, gmin[d], grange[d], p->g_bits[d]);
    }
    p->nbits = len * 8ull;
    p->body_bit = static_cast<uint32_t>(table_end * 8ull);
    p->anchor_bits = p->g_bits[0] + p->g_bits[1] + p->g_bits[2];
    p->meshlet_begin = 0;
    p->blob_off = 0;
    p->v_offset = 0;
    p->t_offset = 0;
    return STRIDE_OK;
}

size_t blob_alloc_bytes(size_t len) { return (len + kBlobPad + 255) & ~static_cast<size_t>(255); }

int status_to_code(const Status& st, uint32_t* bad_meshlet) {
    if (st.err == 0ull) return STRIDE_OK;
    const int code = static_cast<int>(st.err >> 32);
    if (bad_meshlet) *bad_meshlet = static_cast<uint32_t>(st.err & 0xFFFFFFFFull);
    switch (code) {
        case kErrOffset: return STRIDE_ERR_OFFSET;
        case kErrCorrupt: return STRIDE_ERR_CORRUPT;
        case kErrUnsupported: return STRIDE_ERR_UNSUPPORTED;
        case kErrTimeout: return STRIDE_ERR_TIMEOUT;
        default: return STRIDE_ERR_CORRUPT;
    }
}

const char* status_message(int code) {
    switch (code) {
        case STRIDE_ERR_OFFSET: return "meshlet offset table out of order or out of range";
        case STRIDE_ERR_CORRUPT: return "meshlet payload inconsistent with its header or the offset table";
        case STRIDE_ERR_UNSUPPORTED: return "meshlet outside this decoder's limits (>256 vertices/triangles, k>24)";
        case STRIDE_ERR_TIMEOUT: return "a bounded device wait gave up";
        default: return "decode failed";
    }
}

}  // namespace stride

using namespace stride;

namespace stride {

unsigned long long plan_luts(MeshParams* p, uint32_t n, uint32_t* meshes, uint32_t max_meshes, uint32_t* n_lut,
                             uint32_t* lut_max, bool alone) {
    unsigned long long total = 0;
    uint32_t k = 0, mx = 0;
    for (uint32_t i = 0; i < n; i++) {
        p[i].has_lut = 0;
        p[i].lut_off = 0;
        const unsigned long long e = lut_entries(p[i], alone);
        if (!e || k >= max_meshes || k >= 65535u) continue;  // bounds the table blocks of the scan launch
        p[i].has_lut = 1;
        p[i].lut_off = total;
        total += e;
        if (meshes) meshes[k] = i;
        k++;
        mx = std::max<uint32_t>(mx, static_cast<uint32_t>(e));
    }
    *n_lut = k;
    *lut_max = mx;
    return total;
}

}  // namespace stride

// What a handle keeps on the device whatever its stream: uploaded at once.
struct HandleFixed {
    MeshParams params;
    alignas(16) Status status;
    uint32_t lut_mesh;  // the one-entry mesh list {0}
};

struct stride_handle {
    int device = 0;
    size_t len = 0, cap_bytes = 0;
    uint32_t cap_meshlets = 0;
    HandleFixed* d_fixed = nullptr;
    uint8_t* d_mem = nullptr;  // the buffers below
    uint8_t* d_blob = nullptr;
    MeshParams params;
    MeshletDesc* d_descs = nullptr;
    uint4* d_blk_sums = nullptr;
    BlockPrefix* d_blk_prefix = nullptr;
    uint32_t* d_walk_scratch = nullptr;
    unsigned long long walk_cap = 0;
    float* d_lut = nullptr;             // dequantisation tables
    unsigned long long lut_cap = 0;     // floats
    uint32_t n_lut = 0, lut_max = 0;
    uint8_t* d_out = nullptr;           // stride_decode_host's outputs: triangles, positions
    size_t cap_v = 0, cap_t = 0;
    cudaEvent_t done = nullptr;
    Status* h_status = nullptr;         // pinned: stride_finish's copy
    cudaEvent_t used = nullptr;         // behind the last use of the buffers that `done` does not cover
    bool launched = false;
    bool in_use = false;                // `used` is recorded
    bool unseen = false;                // work that no event of the handle covers (a capture's replays, a failed call's)
    bool known = false;                 // last: the last decode's status
    Status last;
    LaunchCfg cfg;
    bool cfg_set = false;               // stride_set_config called: keep cfg across reloads
    long long wait_clocks = 1ll << 31;  // DecodeArgs::wait_clocks of this handle's decodes
    uint32_t launch_smem = 0, launch_grid = 0;  // the last decode's main kernel
    HostLink link;          // stride_decode_host, and a reload that uploads by parts
    bool up_parts = false;  // the last reload uploaded by parts (link.bytes_in)
};

// A reload that uploaded by parts: the decode stream waits for all of it
// (decodes that do not go by parts).
static cudaError_t wait_upload(stride_handle* h, cudaStream_t s) {
    return h->up_parts ? cudaStreamWaitEvent(s, h->link.bytes_in[kHostParts - 1], 0) : cudaSuccess;
}

namespace stride {

namespace {
// Pinned memory for status words and part ends: cudaHostAlloc and
// cudaFreeHost take 100 and 150 us a piece.  One slab of 64 KB, pinned on
// first use and kept; slots go back to it, and what it has no room for is
// pinned by itself.
struct PinnedSlab {
    static constexpr size_t kSlot = 256, kSlots = 256;
    std::mutex mu;
    uint8_t* base = nullptr;
    std::bitset<kSlots> used;
};
PinnedSlab& pinned_slab() {
    static PinnedSlab* s = new PinnedSlab;  // never destroyed: handles may outlive static objects
    return *s;
}
}  // namespace

cudaError_t pinned_take(size_t bytes, void** out) {
    *out = nullptr;
    if (bytes <= PinnedSlab::kSlot) {
        PinnedSlab& s = pinned_slab();
        std::lock_guard<std::mutex> g(s.mu);
        if (!s.base && cudaHostAlloc(reinterpret_cast<void**>(&s.base), PinnedSlab::kSlot * PinnedSlab::kSlots,
                                     cudaHostAllocPortable) != cudaSuccess) {
            s.base = nullptr;
            cudaGetLastError();
        }
        for (size_t i = 0; s.base && i < PinnedSlab::kSlots; i++) {
            if (s.used[i]) continue;
            s.used[i] = true;
            *out = s.base + PinnedSlab::kSlot * i;
            return cudaSuccess;
        }
    }
    return cudaHostAlloc(out, bytes, cudaHostAllocPortable);
}

void pinned_give(void* p) {
    if (!p) return;
    PinnedSlab& s = pinned_slab();
    {
        std::lock_guard<std::mutex> g(s.mu);
        const uint8_t* b = static_cast<uint8_t*>(p);
        if (s.base && b >= s.base && b < s.base + PinnedSlab::kSlot * PinnedSlab::kSlots) {
            s.used[static_cast<size_t>(b - s.base) / PinnedSlab::kSlot] = false;
            return;
        }
    }
    cudaFreeHost(p);
}

namespace {
// Device blocks of closed handles for the next ones: a cudaMalloc and its
// cudaFree take 60 us.  At most kBlocks blocks and kBytes bytes per process;
// the oldest go back to the driver beyond that, all of them when an allocation
// fails.  A block comes in once everything its handle has enqueued is over
// (handle_idle), so whoever takes it, on whatever stream, finds it unused.
struct DeviceBlocks {
    static constexpr size_t kBlocks = 16, kBytes = size_t(32) << 20;
    struct Block {
        void* p;
        size_t bytes;
        int device;
    };
    std::mutex mu;
    std::vector<Block> free;               // the oldest first
    std::unordered_map<void*, Block> out;  // in use
    size_t bytes = 0;                      // of the free ones
};
DeviceBlocks& device_blocks() {
    static DeviceBlocks* b = new DeviceBlocks;  // never destroyed: handles may outlive static objects
    return *b;
}
}  // namespace

static cudaError_t block_take(size_t bytes, void** out) {
    *out = nullptr;
    bytes = (std::max<size_t>(bytes, 1) + 255) & ~static_cast<size_t>(255);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    DeviceBlocks& B = device_blocks();
    try {
        std::lock_guard<std::mutex> g(B.mu);
        size_t best = B.free.size();
        for (size_t i = 0; i < B.free.size(); i++) {
            const DeviceBlocks::Block& b = B.free[i];
            // not more than twice what is asked for, and 4 KB
            if (b.device == dev && b.bytes >= bytes && b.bytes <= 2 * bytes + 4096 &&
                (best == B.free.size() || b.bytes < B.free[best].bytes))
                best = i;
        }
        if (best < B.free.size()) {
            const DeviceBlocks::Block b = B.free[best];
            B.out.emplace(b.p, b);
            B.free.erase(B.free.begin() + static_cast<std::ptrdiff_t>(best));
            B.bytes -= b.bytes;
            *out = b.p;
            return cudaSuccess;
        }
        void* p = nullptr;
        e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess && !B.free.empty()) {
            cudaGetLastError();
            for (const DeviceBlocks::Block& b : B.free) cudaFree(b.p);
            B.free.clear();
            B.bytes = 0;
            e = cudaMalloc(&p, bytes);
        }
        if (e != cudaSuccess) return e;
        try {
            B.out.emplace(p, DeviceBlocks::Block{p, bytes, dev});
        } catch (const std::bad_alloc&) {
            cudaFree(p);
            return cudaErrorMemoryAllocation;
        }
        *out = p;
        return cudaSuccess;
    } catch (const std::bad_alloc&) {
        return cudaErrorMemoryAllocation;
    }
}

// `idle`: the caller has waited for whatever was to use the block; else cudaFree
// does.
static void block_give(void* p, bool idle) {
    if (!p) return;
    DeviceBlocks& B = device_blocks();
    std::lock_guard<std::mutex> g(B.mu);
    const auto it = B.out.find(p);
    bool kept = false;
    if (it != B.out.end()) {
        const DeviceBlocks::Block b = it->second;
        B.out.erase(it);
        if (idle && b.bytes <= DeviceBlocks::kBytes) {
            try {
                B.free.push_back(b);
                B.bytes += b.bytes;
                kept = true;
            } catch (const std::bad_alloc&) {
            }
            while (B.free.size() > DeviceBlocks::kBlocks || B.bytes > DeviceBlocks::kBytes) {
                cudaFree(B.free.front().p);
                B.bytes -= B.free.front().bytes;
                B.free.erase(B.free.begin());
            }
        }
    }
    if (!kept) cudaFree(p);
}

static void for_link_events(HostLink& L, void (*f)(cudaEvent_t*, cudaError_t*), cudaError_t* e) {
    for (cudaEvent_t* ev : {&L.conn_done, &L.vert_done, &L.done, &L.copied[0], &L.copied[1], &L.before_up})
        f(ev, e);
    for (int p = 0; p < kHostParts; p++)
        for (cudaEvent_t* ev : {&L.part_done[p], &L.scan_done[p], &L.end_in[p], &L.bytes_in[p]}) f(ev, e);
}

void host_link_free(HostLink& L) {
    for (cudaStream_t* c : {&L.copy[0], &L.copy[1], &L.up})
        if (*c) cudaStreamDestroy(*c), *c = nullptr;
    for_link_events(L, [](cudaEvent_t* ev, cudaError_t*) { if (*ev) cudaEventDestroy(*ev), *ev = nullptr; }, nullptr);
    pinned_give(L.h_end);
    L.h_end = nullptr;
    pinned_give(L.h_status);
    L.h_status = nullptr;
}

cudaError_t host_link_init(HostLink& L) {
    if (L.copy[0]) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    for (cudaStream_t* c : {&L.copy[0], &L.copy[1], &L.up})
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(c, cudaStreamNonBlocking);
    for_link_events(L, [](cudaEvent_t* ev, cudaError_t* err) {
        if (*err == cudaSuccess) *err = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    }, &e);
    if (e == cudaSuccess && !L.h_status) e = pinned_take(sizeof(Status), reinterpret_cast<void**>(&L.h_status));
    if (e == cudaSuccess) e = pinned_take(kHostParts * sizeof(PartEnd), reinterpret_cast<void**>(&L.h_end));
    if (e != cudaSuccess) host_link_free(L);
    return e;
}

void host_part_groups(uint32_t total_meshlets, uint32_t* part_g) {
    const uint32_t n_groups = (total_meshlets + 31u) / 32u;
    const uint32_t n_win = (n_groups + 7u) / 8u;
    for (int p = 0; p < kHostParts; p++)
        part_g[p] = 8u * static_cast<uint32_t>(static_cast<uint64_t>(n_win) * p / kHostParts);
    part_g[kHostParts] = n_groups;
}

int decode_to_host(HostLink& L, const DecodeArgs& a, LaunchCfg cfg, void* stream, uint64_t n_t, uint64_t n_v,
                   uint32_t* h_idx, float* h_pos, const cudaEvent_t* bytes_in, uint32_t* bad, bool* ran) {
    *ran = false;
    cudaError_t e;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t ib = 12 * n_t, pb = 12 * n_v;
    // a failure once work is queued: nothing may still run on the buffers
    // or write the host outputs when this returns
    auto drain = [&]() {
        cudaStreamSynchronize(s);
        for (cudaStream_t c : L.copy)
            if (c) cudaStreamSynchronize(c);
        // parts may have ended half-way: the next scan finds its counter at zero
        if (cudaMemsetAsync(a.status, 0, sizeof(Status), s) == cudaSuccess) cudaStreamSynchronize(s);
    };
    auto bail = [&](cudaError_t err, const char* what) {
        drain();
        return cuda_fail(err, what);
    };
    auto not_launched = [&](int rc) {  // the scan may be queued
        const char* why = cudaGetErrorString(cudaGetLastError());
        drain();
        return fail(rc, "decode launch failed: %s", why);
    };
    if (cfg.persistent == 2) cfg.persistent = 1;
    if (cfg.persistent == 4 && a.total_meshlets > kHostTeam) {
        LaunchCfg two = cfg;
        two.persistent = 1;
        if (check_config(two, a.wide_codes) == STRIDE_OK) cfg = two;
    }
    if (cfg.persistent >= 2) {
        // One kernel, so nothing to copy beside it: everything on the decode's
        // own stream (14-bit heightfields into pageable memory, 10 / 336 / 1,295
        // / 2,631 meshlets: 73 / 79 / 102 / 143 us, by two copy streams 98 / 105
        // / 128 / 168; pinned 64 / 70 / 92 / 136 and 71 / 78 / 98 / 139).
        if (!L.h_status && (e = pinned_take(sizeof(Status), reinterpret_cast<void**>(&L.h_status))) != cudaSuccess)
            return cuda_fail(e, "pinned status");
        if (bytes_in && (e = cudaStreamWaitEvent(s, bytes_in[kHostParts - 1], 0)) != cudaSuccess)
            return cuda_fail(e, "decode to host: upload");
        const int rc = enqueue_decode(a, cfg, stream);
        if (rc) return not_launched(rc);
        e = cudaMemcpyAsync(L.h_status, a.status, sizeof(Status), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && ib) e = cudaMemcpyAsync(h_idx, a.idx, ib, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && pb) e = cudaMemcpyAsync(h_pos, a.pos, pb, cudaMemcpyDeviceToHost, s);
        const cudaError_t e2 = cudaStreamSynchronize(s);  // in any case: nothing may still write the host outputs
        if (e != cudaSuccess || (e = e2) != cudaSuccess) return cuda_fail(e, "decode to host: copies");
        *ran = true;
        return status_to_code(*L.h_status, bad);
    }
    if ((e = host_link_init(L)) != cudaSuccess) return cuda_fail(e, "copy streams");
    const bool parts = cfg.persistent < 2 && host_parts(n_t, a.total_meshlets);
    if (parts) {
        // Part by part: its scan, the read-back of its end (the next part's
        // first triangle row), its connectivity; then, once its end is
        // known, the copy of its triangles, queued before the next part's
        // kernels so that it starts as soon as the part's connectivity ends.
        // A corrupt stream's ends are clamped (its status reports it).
        uint32_t part_g[kHostParts + 1];
        host_part_groups(a.total_meshlets, part_g);
        int rc = enqueue_parts_begin(a, cfg, stream);
        size_t from = 0;
        for (int p = 0; p < kHostParts && rc == STRIDE_OK && e == cudaSuccess; p++) {
            rc = enqueue_part(a, cfg, stream, part_g[p], part_g[p + 1], p == 0, bytes_in ? bytes_in[p] : nullptr,
                              L.scan_done[p], L.part_done[p]);
            if (rc) break;
            size_t to = ib;
            if (p + 1 < kHostParts) {
                const uint32_t last = part_g[p + 1] / 8u - 1u;  // the part's last window
                if ((e = cudaStreamWaitEvent(L.copy[1], L.scan_done[p], 0)) != cudaSuccess ||
                    (e = cudaMemcpyAsync(&L.h_end[p].prefix, a.blk_prefix + last, sizeof(BlockPrefix),
                                         cudaMemcpyDeviceToHost, L.copy[1])) != cudaSuccess ||
                    (e = cudaMemcpyAsync(&L.h_end[p].sums, a.blk_sums + last, sizeof(uint4), cudaMemcpyDeviceToHost,
                                         L.copy[1])) != cudaSuccess ||
                    (e = cudaEventRecord(L.end_in[p], L.copy[1])) != cudaSuccess ||
                    (e = cudaEventSynchronize(L.end_in[p])) != cudaSuccess)
                    break;
                const PartEnd& pe = L.h_end[p];
                to = std::max(from, 12 * std::min<size_t>(pe.prefix.t + pe.sums.y, n_t));
            }
            if ((e = cudaStreamWaitEvent(L.copy[0], L.part_done[p], 0)) == cudaSuccess && to > from)
                e = cudaMemcpyAsync(reinterpret_cast<uint8_t*>(h_idx) + from,
                                    reinterpret_cast<const uint8_t*>(a.idx) + from, to - from,
                                    cudaMemcpyDeviceToHost, L.copy[0]);
            from = to;
        }
        if (rc == STRIDE_OK && e == cudaSuccess) rc = enqueue_parts_end(a, cfg, stream, L.vert_done);
        if (e != cudaSuccess) return bail(e, "decode to host: parts");
        if (rc) return not_launched(rc);
    } else {
        if (bytes_in && (e = cudaStreamWaitEvent(s, bytes_in[kHostParts - 1], 0)) != cudaSuccess)
            return cuda_fail(e, "decode to host: upload");
        void* ev[4] = {nullptr, nullptr, L.conn_done, L.vert_done};
        const int rc = enqueue_decode(a, cfg, stream, ev);
        if (rc) return not_launched(rc);
    }
    // each output (the triangles unless they went by parts) in two halves,
    // one per copy stream
    const size_t ih = (ib / 2) & ~size_t(15), ph = (pb / 2) & ~size_t(15);
    const size_t ioff[2] = {0, ih}, ilen[2] = {ih, ib - ih};
    const size_t poff[2] = {0, ph}, plen[2] = {ph, pb - ph};
    for (int k = 0; k < 2 && e == cudaSuccess; k++) {
        cudaStream_t c = L.copy[k];
        if (!parts && (e = cudaStreamWaitEvent(c, L.conn_done, 0)) == cudaSuccess && ilen[k])
            e = cudaMemcpyAsync(reinterpret_cast<uint8_t*>(h_idx) + ioff[k],
                                reinterpret_cast<const uint8_t*>(a.idx) + ioff[k], ilen[k], cudaMemcpyDeviceToHost, c);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(c, L.vert_done, 0);
        if (e == cudaSuccess && plen[k])
            e = cudaMemcpyAsync(reinterpret_cast<uint8_t*>(h_pos) + poff[k],
                                reinterpret_cast<const uint8_t*>(a.pos) + poff[k], plen[k], cudaMemcpyDeviceToHost, c);
        // the status is final with the vertex kernel: it comes back with the
        // positions, and no synchronous read follows the decode
        if (e == cudaSuccess && k == 1)
            e = cudaMemcpyAsync(L.h_status, a.status, sizeof(Status), cudaMemcpyDeviceToHost, c);
        if (e == cudaSuccess) e = cudaEventRecord(L.copied[k], c);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s, L.copied[k], 0);
    }
    if (e == cudaSuccess) e = cudaEventRecord(L.done, s);
    if (e == cudaSuccess) e = cudaEventSynchronize(L.done);
    if (e != cudaSuccess) return bail(e, "decode to host: copies");
    *ran = true;
    return status_to_code(*L.h_status, bad);
}

}  // namespace stride

// Waits for everything the handle has enqueued; false when that cannot be
// told.  (Not by a device synchronisation, which would end another thread's
// stream capture.)
static bool handle_idle(stride_handle* h) {
    bool ok = !h->unseen;
    if (h->launched) ok = cudaEventSynchronize(h->done) == cudaSuccess && ok;
    if (h->in_use) ok = cudaEventSynchronize(h->used) == cudaSuccess && ok;
    if (h->up_parts) ok = cudaEventSynchronize(h->link.bytes_in[kHostParts - 1]) == cudaSuccess && ok;
    if (!ok) cudaGetLastError();
    return ok;
}

// Behind work on `stream` that reads or writes the handle's buffers and that
// stride_decode's event does not cover.
static cudaError_t mark_use(stride_handle* h, cudaStream_t s) {
    const cudaError_t e = cudaEventRecord(h->used, s);
    if (e == cudaSuccess) h->in_use = true;
    if (e != cudaSuccess) h->unseen = true;
    return e;
}

static bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess) return cap != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;  // the legacy stream while a stream captures
}

// Before such work: behind the one before it, so that one event covers both.
static cudaError_t chain_use(stride_handle* h, cudaStream_t s) {
    return h->in_use ? cudaStreamWaitEvent(s, h->used, 0) : cudaSuccess;
}

static void free_buffers(stride_handle* h, bool idle) {
    block_give(h->d_fixed, idle);
    block_give(h->d_mem, idle);
    block_give(h->d_out, idle);
    pinned_give(h->h_status);
}

// Buffers for a stream of this size, in one block; also plans the
// dequantisation tables of `p` (has_lut, lut_off).  (A mesh of 23,254 triangles
// decoded once, from open to close: 833 us with nine allocations, pinned words
// and copy streams of its own, 124 now.)
static int ensure_capacity(stride_handle* h, size_t len, MeshParams& p) {
    const unsigned long long lut = plan_luts(&p, 1, nullptr, 1, &h->n_lut, &h->lut_max, true);
    const unsigned long long ww = walk_scratch_words(p.n_v, p.n_meshlets);
    const size_t blob = blob_alloc_bytes(len);
    if (h->d_mem && lut <= h->lut_cap && ww <= h->walk_cap && blob <= h->cap_bytes && p.n_meshlets <= h->cap_meshlets)
        return STRIDE_OK;
    const unsigned long long c_lut = std::max(lut, h->lut_cap), c_ww = std::max(ww, h->walk_cap);
    const size_t c_blob = std::max(blob, h->cap_bytes);
    const uint32_t c_m = std::max(p.n_meshlets, h->cap_meshlets), nb = scan_blocks(c_m);
    size_t total = 0;
    auto place = [&](unsigned long long bytes) {
        const size_t at = total;
        total += (static_cast<size_t>(bytes) + 255) & ~static_cast<size_t>(255);
        return at;
    };
    const size_t o_blob = place(c_blob), o_descs = place(sizeof(MeshletDesc) * static_cast<unsigned long long>(c_m)),
                 o_sums = place(sizeof(uint4) * static_cast<unsigned long long>(nb)),
                 o_prefix = place(sizeof(BlockPrefix) * static_cast<unsigned long long>(nb)), o_walk = place(4ull * c_ww),
                 o_lut = place(4ull * c_lut);
    block_give(h->d_mem, false);  // cudaFree: after the work queued on it
    h->d_mem = h->d_blob = nullptr;
    h->d_descs = nullptr;
    h->d_blk_sums = nullptr;
    h->d_blk_prefix = nullptr;
    h->d_walk_scratch = nullptr;
    h->d_lut = nullptr;
    h->cap_bytes = 0;
    h->cap_meshlets = 0;
    h->walk_cap = h->lut_cap = 0;
    const cudaError_t e = block_take(total, reinterpret_cast<void**>(&h->d_mem));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(stream, scratch)");
    h->d_blob = h->d_mem + o_blob;
    h->d_descs = reinterpret_cast<MeshletDesc*>(h->d_mem + o_descs);
    h->d_blk_sums = reinterpret_cast<uint4*>(h->d_mem + o_sums);
    h->d_blk_prefix = reinterpret_cast<BlockPrefix*>(h->d_mem + o_prefix);
    h->d_walk_scratch = reinterpret_cast<uint32_t*>(h->d_mem + o_walk);
    h->d_lut = reinterpret_cast<float*>(h->d_mem + o_lut);
    h->cap_bytes = c_blob;
    h->cap_meshlets = c_m;
    h->walk_cap = c_ww;
    h->lut_cap = c_lut;
    return STRIDE_OK;
}

extern "C" {

const char* stride_last_error_message(void) { return g_last_error.c_str(); }

const char* stride_error_string(int code) {
    switch (code) {
        case STRIDE_OK: return "ok";
        case STRIDE_ERR_ARG: return "bad argument";
        case STRIDE_ERR_MAGIC: return "bad magic";
        case STRIDE_ERR_VERSION: return "unsupported version";
        case STRIDE_ERR_TRUNCATED: return "truncated stream";
        case STRIDE_ERR_OFFSET: return "bad meshlet offset table";
        case STRIDE_ERR_CORRUPT: return "corrupt meshlet payload";
        case STRIDE_ERR_UNSUPPORTED: return "unsupported stream parameters";
        case STRIDE_ERR_CUDA: return "CUDA error";
        case STRIDE_ERR_TIMEOUT: return "timeout";
        case STRIDE_ERR_NOMEM: return "out of memory";
        case STRIDE_ERR_BUSY: return "busy";
        default: return "unknown error";
    }
}

int stride_device_info(int* sm_count, int* arch) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (sm_count) *sm_count = device_sm_count();
    if (arch) *arch = 103;
    return STRIDE_OK;
}

static bool wide_codes(const MeshParams& p) { return p.g_bits[0] > 16 || p.g_bits[1] > 16 || p.g_bits[2] > 16; }

static void fill_info(const MeshParams& p, size_t len, int persistent, stride_info_t* info) {
    std::memset(info, 0, sizeof(*info));
    info->n_meshlets = p.n_meshlets;
    for (int i = 0; i < 3; i++) {
        info->g_bits[i] = p.g_bits[i];
        info->center[i] = static_cast<float>(p.dq[i].center);
        info->g_min[i] = static_cast<float>(p.dq[i].gmin);
        info->g_range[i] = static_cast<float>(p.dq[i].grange);
        info->pred_k[i] = p.pred_k[i];
    }
    for (int i = 0; i < 9; i++) info->pred_n[i] = p.pred_n[i];
    info->scale = static_cast<float>(p.dq[0].scale);
    info->n_v = p.n_v;
    info->n_t = p.n_t;
    info->nbytes = len;
    // scan (+ tables), then one kernel (group or fused) or the connectivity and vertex kernels
    info->kernels = p.n_meshlets ? (persistent >= 2 ? 2u : 3u) : 0u;
}

int stride_inspect(const uint8_t* data, size_t len, stride_info_t* info) {
    if (!info) return fail(STRIDE_ERR_ARG, "null info");
    MeshParams p;
    char why[256] = {0};
    const int rc = parse_header(data, len, &p, why, sizeof(why));
    if (rc) return fail(rc, "%s", why);
    fill_info(p, len, default_config(p.n_meshlets, p.n_t, 1u, wide_codes(p)).persistent, info);
    return STRIDE_OK;
}

int stride_open(const uint8_t* data, size_t len, stride_handle** out) {
    if (!out) return fail(STRIDE_ERR_ARG, "null output handle");
    *out = nullptr;
    MeshParams p;
    char why[256] = {0};
    int rc = parse_header(data, len, &p, why, sizeof(why));
    if (rc) return fail(rc, "%s", why);
    stride_handle* h = new stride_handle();
    cudaGetDevice(&h->device);
    h->len = len;
    cudaError_t e;
    rc = ensure_capacity(h, len, p);
    h->params = p;
    h->cfg = default_config(p.n_meshlets, p.n_t, 1u, wide_codes(p));
    if (rc != STRIDE_OK) {
        free_buffers(h, false);
        delete h;
        return rc;
    }
    HandleFixed fixed;
    std::memset(&fixed, 0, sizeof(fixed));
    fixed.params = h->params;
    if ((e = block_take(sizeof(HandleFixed), reinterpret_cast<void**>(&h->d_fixed))) != cudaSuccess ||
        (e = pinned_take(sizeof(Status), reinterpret_cast<void**>(&h->h_status))) != cudaSuccess ||
        (e = cudaMemcpy(h->d_blob, data, len, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemset(h->d_blob + len, 0, h->cap_bytes - len)) != cudaSuccess ||
        (e = cudaMemcpy(h->d_fixed, &fixed, sizeof(HandleFixed), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&h->done, cudaEventDisableTiming)) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&h->used, cudaEventDisableTiming)) != cudaSuccess) {
        if (h->done) cudaEventDestroy(h->done);
        free_buffers(h, false);
        delete h;
        return cuda_fail(e, "stride_open");
    }
    *out = h;
    return STRIDE_OK;
}

int stride_reload(stride_handle* h, const uint8_t* data, size_t len, void* stream) {
    if (!h) return fail(STRIDE_ERR_ARG, "null handle");
    MeshParams p;
    char why[256] = {0};
    int rc = parse_header(data, len, &p, why, sizeof(why));
    if (rc) return fail(rc, "%s", why);
    if ((rc = ensure_capacity(h, len, p)) != STRIDE_OK) return rc;
    h->params = p;
    h->len = len;
    if (!h->cfg_set) h->cfg = default_config(p.n_meshlets, p.n_t, 1u, wide_codes(p));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    const size_t pad = std::min<size_t>(h->cap_bytes - len, kBlobPad);
    const bool cap = capturing(s), unseen = h->unseen;
    h->unseen = true;  // until all of it is enqueued
    // an earlier upload by parts may still be writing the arena
    if ((e = wait_upload(h, s)) != cudaSuccess) return cuda_fail(e, "stride_reload");
    h->up_parts = false;
    if (host_parts(p.n_t, p.n_meshlets) && host_link_init(h->link) == cudaSuccess) {
        // A stream large enough for a host decode by parts goes up in the
        // same parts (whole windows of meshlets, cut where the offset table
        // says the part's first meshlet starts), one event per part, on
        // the handle's upload stream after the work already queued on
        // `stream` (a decode there may still read the arena).
        uint32_t part_g[kHostParts + 1];
        host_part_groups(p.n_meshlets, part_g);
        size_t cut[kHostParts + 1];
        cut[0] = 0;
        cut[kHostParts] = len;
        for (int q = 1; q < kHostParts; q++) {
            const uint8_t* t = data + kHeaderBytes + 4ull * (32ull * part_g[q]);  // inside the table
            const uint64_t bit = (uint64_t(t[0]) << 24) | (uint64_t(t[1]) << 16) | (uint64_t(t[2]) << 8) | t[3];
            cut[q] = std::min(len, std::max(cut[q - 1], static_cast<size_t>((bit + 7) / 8)));
        }
        HostLink& L = h->link;
        if ((e = cudaEventRecord(L.before_up, s)) != cudaSuccess || (e = cudaStreamWaitEvent(L.up, L.before_up, 0)))
            return cuda_fail(e, "stride_reload");
        // the mesh record first: a copy queued on `stream` would go after
        // every part on the copy engine, and the first part's scan needs it
        if ((e = cudaMemcpyAsync(&h->d_fixed->params, &h->params, sizeof(MeshParams), cudaMemcpyHostToDevice, L.up)) !=
            cudaSuccess)
            return cuda_fail(e, "stride_reload");
        for (int q = 0; q < kHostParts; q++) {
            if (cut[q + 1] > cut[q] &&
                (e = cudaMemcpyAsync(h->d_blob + cut[q], data + cut[q], cut[q + 1] - cut[q], cudaMemcpyHostToDevice,
                                     L.up)) != cudaSuccess)
                return cuda_fail(e, "stride_reload");
            if (q + 1 == kHostParts && (e = cudaMemsetAsync(h->d_blob + len, 0, pad, L.up)) != cudaSuccess)
                return cuda_fail(e, "stride_reload");
            if ((e = cudaEventRecord(L.bytes_in[q], L.up)) != cudaSuccess) return cuda_fail(e, "stride_reload");
        }
        h->up_parts = true;
    } else if ((e = cudaMemcpyAsync(h->d_blob, data, len, cudaMemcpyHostToDevice, s)) != cudaSuccess ||
               (e = cudaMemsetAsync(h->d_blob + len, 0, pad, s)) != cudaSuccess ||
               (e = cudaMemcpyAsync(&h->d_fixed->params, &h->params, sizeof(MeshParams), cudaMemcpyHostToDevice, s)) !=
                   cudaSuccess ||
               (!cap && ((e = chain_use(h, s)) != cudaSuccess || (e = mark_use(h, s)) != cudaSuccess))) {
        return cuda_fail(e, "stride_reload");
    }
    h->unseen = unseen || cap;
    return STRIDE_OK;
}

int stride_info(const stride_handle* h, stride_info_t* info) {
    if (!h || !info) return fail(STRIDE_ERR_ARG, "null argument");
    fill_info(h->params, h->len, h->cfg.persistent, info);
    info->shared_bytes = h->launch_smem;
    info->persistent_blocks = h->launch_grid;
    return STRIDE_OK;
}

static DecodeArgs handle_args(stride_handle* h, uint32_t* d_idx, float* d_pos, int32_t* d_codes) {
    DecodeArgs a;
    a.wait_clocks = h->wait_clocks;
    a.status_kept = true;
    a.arena = h->d_blob;
    a.meshes = &h->d_fixed->params;
    a.meshlet_mesh = nullptr;
    a.total_meshlets = h->params.n_meshlets;
    a.n_meshes = 1;
    a.descs = h->d_descs;
    a.blk_sums = h->d_blk_sums;
    a.blk_prefix = h->d_blk_prefix;
    a.walk_scratch = h->d_walk_scratch;
    a.walk_cap = h->walk_cap;
    a.status = &h->d_fixed->status;
    a.idx = d_idx;
    a.pos = d_pos;
    a.codes = d_codes;
    a.wide_codes = wide_codes(h->params);
    a.lut = h->d_lut;
    a.lut_meshes = &h->d_fixed->lut_mesh;
    a.n_lut_meshes = h->n_lut;
    a.lut_max = h->lut_max;
    a.hint_bytes = h->len;
    a.hint_v = h->params.n_v;
    a.hint_t = h->params.n_t;
    return a;
}

// After a reload that could not allocate, until one that could.
static int no_buffers() { return fail(STRIDE_ERR_CUDA, "the last reload could not allocate the handle's buffers"); }

int stride_decode_timed(stride_handle* h, void* stream, uint32_t* d_idx, float* d_pos, float* kernel_ms) {
    if (!h || !d_idx || !d_pos) return fail(STRIDE_ERR_ARG, "null argument");
    if (!h->d_mem) return no_buffers();
    if ((reinterpret_cast<uintptr_t>(d_idx) & 15u) || (reinterpret_cast<uintptr_t>(d_pos) & 3u))
        return fail(STRIDE_ERR_ARG, "index output must be 16-byte aligned, positions 4-byte aligned");
    cudaEvent_t ev[4];
    for (auto& e : ev) cudaEventCreate(&e);
    void* evp[4] = {ev[0], ev[1], ev[2], ev[3]};
    h->known = false;
    const bool unseen = h->unseen || capturing(static_cast<cudaStream_t>(stream));
    h->unseen = true;  // as in stride_decode
    int rc = wait_upload(h, static_cast<cudaStream_t>(stream)) == cudaSuccess
                 ? enqueue_decode(handle_args(h, d_idx, d_pos, nullptr), h->cfg, stream, evp)
                 : STRIDE_ERR_CUDA;
    if (rc == STRIDE_OK) {
        last_launch(&h->launch_smem, &h->launch_grid);
        if (cudaEventRecord(h->done, static_cast<cudaStream_t>(stream)) == cudaSuccess) h->unseen = unseen;
        h->launched = true;
        cudaError_t e = cudaEventSynchronize(ev[3]);
        if (e != cudaSuccess) {
            rc = cuda_fail(e, "stride_decode_timed");
        } else if (kernel_ms) {
            for (int i = 0; i < 3; i++) cudaEventElapsedTime(&kernel_ms[i], ev[i], ev[i + 1]);
        }
    } else {
        rc = fail(rc, "decode launch failed");
    }
    for (auto& e : ev) cudaEventDestroy(e);
    return rc;
}

int stride_decode(stride_handle* h, void* stream, uint32_t* d_idx, float* d_pos, int32_t* d_codes) {
    if (!h) return fail(STRIDE_ERR_ARG, "null handle");
    if ((!d_idx && h->params.n_t) || (!d_pos && h->params.n_v)) return fail(STRIDE_ERR_ARG, "null output pointer");
    if (!h->d_mem) return no_buffers();
    if ((reinterpret_cast<uintptr_t>(d_idx) & 15u) || (reinterpret_cast<uintptr_t>(d_pos) & 3u) ||
        (reinterpret_cast<uintptr_t>(d_codes) & 3u))
        return fail(STRIDE_ERR_ARG, "index output must be 16-byte aligned, positions and codes 4-byte aligned");
    if (wait_upload(h, static_cast<cudaStream_t>(stream)) != cudaSuccess)
        return fail(STRIDE_ERR_CUDA, "decode launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    h->known = false;
    const bool unseen = h->unseen || capturing(static_cast<cudaStream_t>(stream));
    h->unseen = true;  // until all of it is enqueued, and the event behind it
    const int rc = enqueue_decode(handle_args(h, d_idx, d_pos, d_codes), h->cfg, stream);
    if (rc) return fail(rc, "decode launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    last_launch(&h->launch_smem, &h->launch_grid);
    cudaError_t e = cudaEventRecord(h->done, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
    h->launched = true;
    h->unseen = unseen;
    return STRIDE_OK;
}

static int say_status(const Status& st, uint32_t* bad_meshlet) {
    uint32_t bad = 0;
    const int rc = status_to_code(st, &bad);
    if (bad_meshlet) *bad_meshlet = bad;
    return rc ? fail(rc, "%s (meshlet %u)", status_message(rc), bad) : STRIDE_OK;
}

// Whether `last` is the last decode's status: a captured one's replays run
// without a call.
static bool seen(const stride_handle* h) { return h->known && !h->unseen; }

static int read_status(stride_handle* h, int wait, uint32_t* bad_meshlet, bool kept) {
    if (!h->launched) return STRIDE_OK;
    if (kept && seen(h)) return say_status(h->last, bad_meshlet);
    cudaError_t e = wait ? cudaEventSynchronize(h->done) : cudaEventQuery(h->done);
    if (e == cudaErrorNotReady) return STRIDE_ERR_BUSY;
    if (e != cudaSuccess) return cuda_fail(e, "decode");
    Status st;
    if ((e = cudaMemcpy(&st, &h->d_fixed->status, sizeof(st), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(e, "cudaMemcpy(status)");
    return say_status(st, bad_meshlet);
}

int stride_status(stride_handle* h, int wait, uint32_t* bad_meshlet) {
    if (!h) return fail(STRIDE_ERR_ARG, "null handle");
    return read_status(h, wait, bad_meshlet, true);
}

// The status comes back on the decode's stream, queued behind it: a copy
// that starts when the host has seen the decode's end costs 11 us more.
int stride_finish(stride_handle* h, void* stream, uint32_t* bad_meshlet) {
    if (!h) return fail(STRIDE_ERR_ARG, "null handle");
    if (!h->launched) return STRIDE_OK;
    if (seen(h)) return say_status(h->last, bad_meshlet);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaStreamWaitEvent(s, h->done, 0);  // another stream's decode
    if (e == cudaSuccess) e = cudaMemcpyAsync(h->h_status, &h->d_fixed->status, sizeof(Status), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaEventRecord(h->done, s);
    if (e == cudaSuccess) e = cudaEventSynchronize(h->done);
    if (e != cudaSuccess) return cuda_fail(e, "decode");
    h->last = *h->h_status;
    h->known = true;
    return say_status(h->last, bad_meshlet);
}

// Before work on `stream` that reads the last decode's records: its status, and
// the order behind the work before it, so that one event covers both.  No event
// covers a captured call's replays (an event recorded in a capture cannot be
// waited for outside it, nor the handle's eager ones inside), and its status is
// read, not taken from an earlier call.
static int begin_use(stride_handle* h, cudaStream_t s, bool* cap, const char* what) {
    *cap = capturing(s);
    const int rc = read_status(h, 1, nullptr, !*cap);
    if (rc) return rc;
    if (*cap) h->unseen = true;
    if (!*cap && chain_use(h, s) != cudaSuccess) return fail(STRIDE_ERR_CUDA, "%s launch failed", what);
    return STRIDE_OK;
}

int stride_side_table(stride_handle* h, void* stream, uint64_t* d_resid_bit, uint16_t* d_sub_offs) {
    if (!h) return fail(STRIDE_ERR_ARG, "null handle");
    const uint32_t n = h->params.n_meshlets;
    if (n && (!d_resid_bit || !d_sub_offs)) return fail(STRIDE_ERR_ARG, "null output pointer");
    if (!h->launched) return fail(STRIDE_ERR_ARG, "no decode yet");
    if (!h->d_mem) return no_buffers();
    bool cap = false;
    const int rc = begin_use(h, static_cast<cudaStream_t>(stream), &cap, "side table");
    if (rc) return rc;
    const int r2 = enqueue_side_table(h->d_descs, n, reinterpret_cast<unsigned long long*>(d_resid_bit), d_sub_offs,
                                      stream);
    if (!cap) mark_use(h, static_cast<cudaStream_t>(stream));
    return r2 ? fail(r2, "side table launch failed") : STRIDE_OK;
}

int stride_meshlet_ranges(stride_handle* h, void* stream, uint64_t* d_v_first, uint64_t* d_t_first) {
    if (!h || !d_v_first || !d_t_first) return fail(STRIDE_ERR_ARG, "null argument");
    if (!h->launched) return fail(STRIDE_ERR_ARG, "no decode yet");
    if (!h->d_mem) return no_buffers();
    bool cap = false;
    const int rc = begin_use(h, static_cast<cudaStream_t>(stream), &cap, "meshlet ranges");
    if (rc) return rc;
    const uint32_t n = h->params.n_meshlets;
    if (n == 0u) {
        const uint64_t z[1] = {0};
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        if (cudaMemcpyAsync(d_v_first, z, 8, cudaMemcpyHostToDevice, s) != cudaSuccess ||
            cudaMemcpyAsync(d_t_first, z, 8, cudaMemcpyHostToDevice, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return cuda_fail(cudaGetLastError(), "meshlet ranges");
        return STRIDE_OK;
    }
    const int r2 = enqueue_meshlet_ranges(h->d_descs, h->d_blk_prefix, n,
                                          reinterpret_cast<unsigned long long*>(d_v_first),
                                          reinterpret_cast<unsigned long long*>(d_t_first), stream);
    if (!cap) mark_use(h, static_cast<cudaStream_t>(stream));
    return r2 ? fail(r2, "meshlet ranges launch failed") : STRIDE_OK;
}

int stride_meshlet_bounds(stride_handle* h, void* stream, const float* d_pos, float* d_bounds) {
    if (!h || (!d_pos && h->params.n_v) || (!d_bounds && h->params.n_meshlets)) return fail(STRIDE_ERR_ARG, "null argument");
    if ((reinterpret_cast<uintptr_t>(d_pos) & 3u) || (reinterpret_cast<uintptr_t>(d_bounds) & 3u))
        return fail(STRIDE_ERR_ARG, "positions and bounds must be 4-byte aligned");
    if (!h->launched) return fail(STRIDE_ERR_ARG, "no decode yet");
    if (!h->d_mem) return no_buffers();
    bool cap = false;
    const int rc = begin_use(h, static_cast<cudaStream_t>(stream), &cap, "meshlet bounds");
    if (rc) return rc;
    const int r2 = enqueue_meshlet_bounds(h->d_descs, h->d_blk_prefix, h->params.n_meshlets, d_pos, d_bounds, stream);
    if (!cap) mark_use(h, static_cast<cudaStream_t>(stream));
    return r2 ? fail(r2, "meshlet bounds launch failed") : STRIDE_OK;
}

int stride_normalise_codes(const stride_handle* h, void* stream, const int32_t* d_codes, float* d_norm) {
    if (!h || ((!d_codes || !d_norm) && h->params.n_v)) return fail(STRIDE_ERR_ARG, "null argument");
    if ((reinterpret_cast<uintptr_t>(d_codes) & 3u) || (reinterpret_cast<uintptr_t>(d_norm) & 3u))
        return fail(STRIDE_ERR_ARG, "codes and positions must be 4-byte aligned");
    NormAxes c;
    // placed by the identity: a centre of -0 leaves every value, a -0 too, as it is
    for (int d = 0; d < 3; d++)
        stride_dequant_setup(&c.d[d], -0.0f, 1.0f, static_cast<float>(h->params.dq[d].gmin),
                             static_cast<float>(h->params.dq[d].grange), h->params.g_bits[d]);
    const int rc = enqueue_normalise(d_codes, 3ull * h->params.n_v, c, d_norm, stream);
    return rc ? fail(rc, "normalise launch failed") : STRIDE_OK;
}

int stride_cull_meshlets(const float* d_bounds, uint32_t n, const float* planes, void* stream, uint32_t* d_visible,
                         uint32_t* d_count) {
    if (!planes || !d_count || (n && (!d_bounds || !d_visible))) return fail(STRIDE_ERR_ARG, "null argument");
    if ((reinterpret_cast<uintptr_t>(d_bounds) & 3u) || (reinterpret_cast<uintptr_t>(d_visible) & 3u) ||
        (reinterpret_cast<uintptr_t>(d_count) & 3u))
        return fail(STRIDE_ERR_ARG, "bounds, visibility and count must be 4-byte aligned");
    Planes pl;
    for (int i = 0; i < 24; i++) pl.p[i] = planes[i];
    const int r2 = enqueue_cull(d_bounds, n, pl, d_visible, d_count, stream);
    return r2 ? fail(r2, "cull launch failed") : STRIDE_OK;
}

int stride_decode_host(stride_handle* h, void* stream, uint32_t* h_idx, float* h_pos) {
    if (!h || (!h_idx && h->params.n_t) || (!h_pos && h->params.n_v)) return fail(STRIDE_ERR_ARG, "null argument");
    if (!h->d_mem) return no_buffers();
    if (h->params.n_v > h->cap_v || h->params.n_t > h->cap_t) {
        const size_t cv = std::max<size_t>(h->params.n_v, h->cap_v), ct = std::max<size_t>(h->params.n_t, h->cap_t);
        block_give(h->d_out, false);
        h->d_out = nullptr;
        h->cap_v = h->cap_t = 0;
        const cudaError_t e = block_take(((12 * ct + 255) & ~static_cast<size_t>(255)) + 12 * cv,
                                         reinterpret_cast<void**>(&h->d_out));
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(outputs)");
        h->cap_v = cv;
        h->cap_t = ct;
    }
    uint32_t* d_idx = reinterpret_cast<uint32_t*>(h->d_out);
    float* d_pos = reinterpret_cast<float*>(h->d_out + ((12 * h->cap_t + 255) & ~static_cast<size_t>(255)));
    uint32_t bad = 0;
    bool ran = false;
    // after a reload by parts, each part of the decode starts when its
    // bytes are in.  With a valid offset table a part's meshlets lie inside
    // the bytes up to its cut; a table that decreases is rejected by the
    // scan, whatever the bytes not yet in hold (which of its faults the
    // error names can then differ from a decode after the whole upload)
    const cudaEvent_t* bytes_in = h->up_parts ? h->link.bytes_in : nullptr;
    const int rc = decode_to_host(h->link, handle_args(h, d_idx, d_pos, nullptr), h->cfg, stream,
                                  h->params.n_t, h->params.n_v, h_idx, h_pos, bytes_in, &bad, &ran);
    if (!ran) {  // what was enqueued before the failure may still run
        h->known = false;
        h->unseen = true;
        return rc;
    }
    h->last = *h->link.h_status;
    h->known = true;
    h->launched = true;  // later status queries see this decode
    cudaEventRecord(h->done, static_cast<cudaStream_t>(stream));
    return rc ? fail(rc, "%s (meshlet %u)", status_message(rc), bad) : STRIDE_OK;
}

int stride_set_wait_limit(stride_handle* h, uint64_t clocks) {
    if (!h) return fail(STRIDE_ERR_ARG, "null handle");
    h->wait_clocks = static_cast<long long>(clocks > (1ull << 62) ? (1ull << 62) : clocks);
    return STRIDE_OK;
}

int stride_set_config(stride_handle* h, const stride_launch_cfg* c) {
    if (!h || !c) return fail(STRIDE_ERR_ARG, "null argument");
    LaunchCfg cfg;
    cfg.warps_per_cta = c->warps_per_cta;
    cfg.persistent = c->persistent;
    cfg.ctas_per_sm = c->ctas_per_sm;
    cfg.stage_bytes = c->stage_bytes;
    cfg.code_bytes = c->code_bytes;
    const bool wide = wide_codes(h->params);
    if (check_config(cfg, wide)) return fail(STRIDE_ERR_ARG, "launch configuration not launchable");
    h->cfg = cfg;
    h->cfg_set = true;
    return STRIDE_OK;
}

int stride_get_config(const stride_handle* h, stride_launch_cfg* c) {
    if (!h || !c) return fail(STRIDE_ERR_ARG, "null argument");
    c->warps_per_cta = h->cfg.warps_per_cta;
    c->persistent = h->cfg.persistent;
    c->ctas_per_sm = h->cfg.ctas_per_sm;
    c->stage_bytes = h->cfg.stage_bytes;
    c->code_bytes = h->cfg.code_bytes;
    return STRIDE_OK;
}

void stride_close(stride_handle* h) {
    if (!h) return;
    const bool idle = handle_idle(h);
    cudaEventDestroy(h->done);
    cudaEventDestroy(h->used);
    host_link_free(h->link);
    free_buffers(h, idle);
    delete h;
}

}  // extern "C"

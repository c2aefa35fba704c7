// PLDT v5 decoding on the GPU: the format the reference's CuPy decoder
// ParaDeltaV5GpuDecoder reads (utils/paradelta_v5_cuda.py:515-718), decoded
// bit-exactly like its CPU decoder decode_paradelta_v5
// (encoder/paradelta_v5.py:286-462; the CuPy kernel computes in float32).
//
// Split as in the reference: the host parses the global header and the
// boundary table (parse_globals_v5, :515-577) and reads every meshlet's
// four-field header from the offset table (the reference's sizes kernel and
// cumulative sums, :640-660); the device decodes the meshlets: the team kernel
// from their bytes to float32 world positions in one launch, or, for streams
// with a meshlet too large for it, the general kernel, one thread per meshlet,
// into float64 normalised rows, which a second kernel turns into positions.
//
// Rows: the boundary vertices, then every meshlet's interior vertices in
// meshlet order.  A meshlet's triangles go to its rows of the index output
// as global row numbers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <new>
#include <stdexcept>
#include <vector>

#include "stride_common.cuh"
#include "stride_device.cuh"
#include "stride_gb300.h"
#include "stride_internal.h"
#include "stride_team.cuh"

namespace stride {
namespace {

constexpr uint32_t kP5Magic = 0x504C4454u;  // MAGIC (encoder/paradelta_codec.py:101)
constexpr uint32_t kP5Version = 5u;         // VERSION_V5 (encoder/paradelta_v5.py:27)
constexpr uint32_t kP5HeaderBits = 32 + 8 + 8 + 32 * 11 + 8 * 3 + 32 * 4 + 32 * 3;
constexpr int kP5MaxLocal = 256;  // local ids are bytes in the walk scratch
constexpr int kP5MaxK = 24;       // largest Rice / Exp-Golomb parameter accepted (the encoder writes <= 11)
constexpr int kP5MaxWidth = 32;   // largest fixed-width residual accepted

struct P5Args {
    const uint8_t* blob;       // stream bytes (64 zero bytes after the end)
    unsigned long long nbits;  // valid bits of the stream
    const uint32_t* start;     // meshlet m starts at start[m]; start[n] = stream end
    const uint32_t* row_base;  // first row of meshlet m's interior vertices
    const uint32_t* tri_base;  // first triangle of meshlet m
    const uint32_t* ref_base;  // first boundary reference of meshlet m
    uint32_t n_meshlets, n_boundary;
    double* rows;              // normalised positions (n_rows x 3)
    uint32_t* refs;            // boundary references of every meshlet
    uint32_t* walk;            // first-reach order per interior row: v | a << 8 | b << 16 | c << 24
    uint32_t* idx;             // output triangles (n_t x 3)
    double w0, w1, w2, delta;
    double scale, center[3];   // to world positions
    float* pos;                // output (n_rows x 3)
    Status* status;
};

// row -> f32(row * scale + center)
__device__ __forceinline__ float p5_world(const P5Args& a, double x, uint32_t d) {
    const double c = d == 0u ? a.center[0] : (d == 1u ? a.center[1] : a.center[2]);
    return __double2float_rn(__dadd_rn(__dmul_rn(x, a.scale), c));
}

__device__ __forceinline__ void p5_report(Status* st, int code, uint32_t m) {
    const unsigned long long v = (static_cast<unsigned long long>(static_cast<unsigned>(code)) << 32) | m;
    atomicCAS(&st->err, 0ull, v);
}

// MSB-first reads from global memory (through L2, as every global read of
// the library) through a three-word register window: a read costs a funnel
// shift, and the word load that refills the window is issued a word ahead
// of its use.  The stream is read as big-endian 32-bit words (its device
// copy is 256-byte aligned and followed by 64 zero bytes, so the window
// never reads past the padding); a read never passes `limit`.
struct P5Bits {
    const uint32_t* w;
    unsigned long long pos, limit, wi;  // wi: word index of w0
    uint32_t w0, w1, w2;
    bool bad;
    __device__ __forceinline__ static uint32_t ld(const uint32_t* w, unsigned long long i) {
        return bswap32(__ldcg(w + i));
    }
    __device__ __forceinline__ void seek(unsigned long long p) {
        pos = p;
        wi = p >> 5;
        w0 = ld(w, wi);
        w1 = ld(w, wi + 1ull);
        w2 = ld(w, wi + 2ull);
    }
    __device__ __forceinline__ uint32_t peek() const {
        return __funnelshift_l(w1, w0, static_cast<uint32_t>(pos & 31ull));
    }
    // n <= 32: crosses at most one word boundary
    __device__ __forceinline__ void skip(uint32_t n) {
        pos += n;
        const unsigned long long ni = pos >> 5;
        if (ni != wi) {
            wi = ni;
            w0 = w1;
            w1 = w2;
            w2 = ld(w, wi + 2ull);
        }
    }
    __device__ __forceinline__ uint32_t bits(int n) {  // n <= 32
        if (n <= 0) return 0u;
        if (pos + static_cast<unsigned>(n) > limit) {
            bad = true;
            return 0u;
        }
        const uint32_t v = peek() >> (32 - n);
        skip(static_cast<uint32_t>(n));
        return v;
    }
    // zeros before the next one bit, and the one bit (BitReader unary prefix;
    // any length up to the end of the stream)
    __device__ __forceinline__ uint32_t unary() {
        uint32_t q = 0u;
        for (;;) {
            if (pos >= limit) {
                bad = true;
                return 0u;
            }
            const uint32_t x = peek();
            if (x) {
                const uint32_t z = static_cast<uint32_t>(__clz(x));
                q += z;
                skip(z + 1u);
                if (pos > limit) bad = true;
                return q;
            }
            q += 32u;
            skip(32u);
        }
    }
    // Rice(k) (BitReader.read_rice); q < 2^32 and k <= 24 fit 64 bits
    __device__ __forceinline__ unsigned long long rice(int k) {
        const uint32_t q = unary();
        const uint32_t low = bits(k);
        return (static_cast<unsigned long long>(q) << k) | low;
    }
    // Exp-Golomb(k) (BitReader.read_exp_golomb); a prefix above 32 bits (a
    // value of at least 2^32, never a residual of a valid stream) is rejected
    __device__ __forceinline__ unsigned long long eg(int k) {
        const uint32_t lb = unary();
        if (lb > 32u) {
            bad = true;
            return 0ull;
        }
        const uint32_t off = bits(static_cast<int>(lb));
        const unsigned long long s = ((1ull << lb) - 1ull) + off;
        const uint32_t low = bits(k);
        return (s << k) | low;
    }
};

// n <= 32 bits at an arbitrary position (fixed-width codes), 0 past `limit`
__device__ __forceinline__ uint32_t p5_bits_at(const uint32_t* w, unsigned long long pos, int n,
                                               unsigned long long limit, bool& bad) {
    if (n <= 0) return 0u;
    if (pos + static_cast<unsigned>(n) > limit) {
        bad = true;
        return 0u;
    }
    const unsigned long long i = pos >> 5;
    const uint32_t x = __funnelshift_l(P5Bits::ld(w, i + 1ull), P5Bits::ld(w, i), static_cast<uint32_t>(pos & 31ull));
    return x >> (32 - n);
}

__device__ __forceinline__ long long unzig(unsigned long long u) {
    return static_cast<long long>((u >> 1) ^ (0ull - (u & 1ull)));
}

// One axis' residual substream: tag 0 fixed width (random access), 1 Rice,
// 2 Exp-Golomb (paradelta_v5.py:405-424); tags 1 and 2 read through their
// own window.
struct P5Axis {
    int tag, k, bw;
    long long mn;
    unsigned long long base;  // first code (tag 0)
    P5Bits r;                 // the next code (tags 1, 2)
};


// One codeword of a Rice (eg false) or Exp-Golomb substream through its
// window: a straight-line read when prefix, terminator and value fit the
// 32-bit window, the general reader otherwise (rare; a branch taken by
// single lanes).  u is the codeword's value.
__device__ __forceinline__ unsigned long long p5_codeword(P5Bits& r, bool eg, int k) {
    const uint32_t x = r.peek();
    const uint32_t z = static_cast<uint32_t>(__clz(x));
    const uint32_t nb = (eg ? z : 0u) + static_cast<uint32_t>(k);
    const uint32_t len = z + 1u + nb;
    if (len > 32u || r.pos + len > r.limit) return eg ? r.eg(k) : r.rice(k);
    const uint32_t t = __funnelshift_lc(0u, x, z + 1u);      // bits after the terminator
    const uint32_t val = nb ? (t >> (32u - nb)) : 0u;        // the top nb of them
    const unsigned long long base = eg ? ((1ull << z) - 1ull) : static_cast<unsigned long long>(z);
    r.skip(len);
    return (base << k) + val;
}

constexpr int kP5Threads = 64;     // meshlets (lanes) per block
constexpr int kP5RefCache = 128;   // a lane's first boundary references kept in shared memory

// The general kernel, for streams that the team kernel does not take (p5_plan).
// One lane per meshlet, 32 meshlets per warp, every phase a loop that the
// whole warp runs to its longest lane's count (no branch per token: the
// lanes stay together), as in the DPR4 kernels:
//  1. the meshlet header and its boundary references (:350-361), the first
//     kP5RefCache of them into shared memory;
//  2. connectivity, one token per iteration (strip header, roots, strip
//     bodies; the FIFO as a move-to-front register), triangles written as
//     rows, first-reach order of the interior vertices (:371-400);
//  3. the three residual substreams' starts (:403-424);
//  4. the float64 reconstruction in walk order (:426-445).
// Validity is checked lazily: running extremes and counts compared once per
// meshlet, ids clamped below n_local and writes bounded by the header's
// counts until then, so a corrupt lane runs on harmlessly and is reported.
__global__ void __launch_bounds__(kP5Threads) p5_decode_kernel(P5Args a) {
    __shared__ uint4 masks[17];
    __shared__ uint32_t seen_all[8 * kP5Threads];           // word i of lane t at [i * kP5Threads + t]
    __shared__ uint32_t ref_all[kP5RefCache * kP5Threads];  // reference l of lane t at [l * kP5Threads + t]
    if (threadIdx.x < 17u) masks[threadIdx.x] = threadIdx.x < 16u ? mtf_mask_row(threadIdx.x) : make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const uint32_t m = blockIdx.x * kP5Threads + threadIdx.x;
    bool act = m < a.n_meshlets;
    const uint32_t mm = act ? m : 0u;
    const unsigned long long s0 = a.start[mm], s1 = a.start[mm + 1u];
    const bool last = mm + 1u == a.n_meshlets;
    const uint32_t* words = reinterpret_cast<const uint32_t*>(a.blob);
    P5Bits b;
    b.w = words;
    b.limit = a.nbits;
    b.bad = false;
    b.seek(act ? s0 : 0ull);
    uint32_t n_bnd = b.bits(16), n_int = b.bits(16), n_tris = b.bits(16), n_strips = b.bits(16);
    uint32_t n_local = n_bnd + n_int;
    bool bad = b.bad;
    if (act && n_local > static_cast<uint32_t>(kP5MaxLocal)) {
        p5_report(a.status, kErrUnsupported, m);
        act = false;
    }
    bad = bad || n_strips > n_tris;  // every strip emits a triangle
    if (!act || bad) n_bnd = n_int = n_tris = n_strips = n_local = 0u;
    const uint32_t rb = act ? a.ref_base[m] : 0u;
    const uint32_t row0 = act ? a.row_base[m] : 0u;
    uint32_t* tri = a.idx + 3ull * (act ? a.tri_base[m] : 0u);
    uint32_t* refc = ref_all + threadIdx.x;
    // 1. boundary references; the decoder reads them as rows of the boundary
    // table (a stream whose references point past it is rejected)
    if (n_bnd > 0u) {
        unsigned long long prev = b.bits(32);
        bad = bad || prev >= a.n_boundary;
        a.refs[rb] = static_cast<uint32_t>(prev);
        refc[0] = static_cast<uint32_t>(prev);
        const int k = n_bnd > 1u ? static_cast<int>(b.bits(8)) : 0;
        bad = bad || k > kP5MaxK;
        for (uint32_t i = 1; i < n_bnd && !bad; i++) {
            prev = prev + p5_codeword(b, false, k) + 1ull;
            bad = bad || b.bad || prev >= a.n_boundary;
            a.refs[rb + i] = static_cast<uint32_t>(prev);
            if (i < static_cast<uint32_t>(kP5RefCache)) refc[i * kP5Threads] = static_cast<uint32_t>(prev);
        }
    }
    auto row_of = [&](uint32_t l) -> uint32_t {
        if (l >= n_bnd) return row0 + (l - n_bnd);
        return l < static_cast<uint32_t>(kP5RefCache) ? refc[l * kP5Threads] : __ldcg(a.refs + rb + l);
    };
    // 2. connectivity
    uint32_t* seen = seen_all + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t lo = 32u * i;
        seen[i * kP5Threads] = n_bnd >= lo + 32u ? 0xFFFFFFFFu : (n_bnd > lo ? (1u << (n_bnd - lo)) - 1u : 0u);
    }
    const uint32_t idx_bits = max(1u, 32u - __clz(n_local));  // max(1, ceil(log2(n_local + 1)))
    const uint32_t rsh = 32u - idx_bits, vmax = n_local ? n_local - 1u : 0u;
    MtfFifo f;
    uint32_t sl = n_strips, tl = 0u, tx = 0u, P = 0u, n_t = 0u, n_emit = 0u, ridmax = 0u;
    int32_t smin = 0;
    bool live = act && !bad && sl > 0u;
    const uint32_t iters = __reduce_max_sync(0xFFFFFFFFu, live ? n_tris + 2u * n_strips : 0u);
    for (uint32_t it = 0; it < iters; it++) {
        const uint32_t x0 = b.peek();
        const bool hdr = tl == 0u;                     // strip header (:376)
        const uint32_t sb = max(x0 >> 16, 1u) - 1u;   // body tokens of the strip
        tl = hdr ? sb + 3u : tl;
        sl -= hdr ? 1u : 0u;
        const uint32_t tix = hdr ? 0u : tx;
        uint32_t x = hdr ? (x0 << 16) : x0;
        uint32_t used = hdr ? 16u : 0u;
        const bool body = tix == 3u;
        const uint32_t ec = x >> 31;  // edge bit of a strip-body token
        x = body ? (x << 1) : x;
        used += body ? 1u : 0u;
        const bool raw = static_cast<int32_t>(x) < 0;  // _read_vert's flag
        const uint32_t y = x << 1;
        const uint32_t rid = y >> rsh;
        const uint32_t fi = y >> 27;
        used += raw ? 1u + idx_bits : 6u;
        // IndexError on a FIFO index past the entries or an id past n_local
        const int32_t sd = static_cast<int32_t>(f.len) - 1 - static_cast<int32_t>(fi);
        smin = min(smin, (raw | !live) ? 0 : sd);
        ridmax = max(ridmax, (raw & live) ? rid + 1u : 0u);
        const uint32_t sdep = static_cast<uint32_t>(sd) & 15u;
        const uint32_t v = raw ? (rid & 0xFFu) : f.at(sdep);
        const uint32_t at = raw ? f.find(v) : sdep;
        const bool fresh = at == 16u;
        f.mtf_masked(v, masks[live ? (fresh ? min(f.len, 15u) : at) : 16u]);  // row 16: no change
        f.len += (live & fresh & (f.len < 16u)) ? 1u : 0u;
        if (live) {
            const uint32_t u = min(v, vmax);
            // edge 0 -> (p1, p2 | p0), 1 -> (p0, p2 | p1) (:386-391); a root
            // token puts u at its position
            const uint32_t sel = body ? (ec ? 0x7420u : 0x7421u) : (0x7210u + ((4u - tix) << (4u * tix)));
            const uint32_t cref = ec ? ((P >> 8) & 0xFFu) : (P & 0xFFu);
            const uint32_t Pn = __byte_perm(P, u, sel);
            if ((body | (tix == 2u)) && n_t < n_tris) {
                tri[3u * n_t] = row_of(Pn & 0xFFu);
                tri[3u * n_t + 1u] = row_of((Pn >> 8) & 0xFFu);
                tri[3u * n_t + 2u] = row_of((Pn >> 16) & 0xFFu);
            }
            n_t += (body | (tix == 2u)) ? 1u : 0u;
            // first reach of an interior vertex (boundary bits are preset)
            uint32_t* sp = seen + (u >> 5) * kP5Threads;
            const uint32_t sw = *sp;
            const uint32_t bit = 1u << (u & 31u);
            if ((sw & bit) == 0u) {
                *sp = sw | bit;
                if (n_emit < n_int)
                    a.walk[row0 + n_emit] = body ? (u | ((Pn & 0xFFFFu) << 8) | (cref << 24)) : u * 0x01010101u;
                n_emit++;
            }
            P = Pn;
        }
        tl--;
        tx = min(tix + 1u, 3u);
        b.skip(live ? used : 0u);
        live = live & ((tl | sl) != 0u) & (b.pos <= b.limit);
    }
    bad = bad || live || b.pos > b.limit || smin < 0 || ridmax > n_local || n_t != n_tris || n_emit > n_int;
    // 3. residual substreams: tag, then fixed width (tag 0: minimum and width,
    // random access) or Rice / Exp-Golomb (tags 1, 2: k); each axis' start
    P5Axis ax[3];
    const bool vx = act && !bad && n_int > 0u;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        ax[d].tag = vx ? static_cast<int>(b.bits(8)) : 1;
        ax[d].k = 0;
        ax[d].bw = 0;
        ax[d].mn = 0;
        ax[d].base = 0ull;
        ax[d].r.w = words;
        ax[d].r.limit = a.nbits;
        ax[d].r.bad = false;
        if (ax[d].tag == 0) {
            const uint32_t mn_u = b.bits(16);
            ax[d].mn = (mn_u & 0x8000u) ? static_cast<long long>(mn_u) - 0x10000 : mn_u;
            ax[d].bw = static_cast<int>(b.bits(8));
            bad = bad || ax[d].bw > kP5MaxWidth;
            ax[d].base = b.pos;
            const unsigned long long e = b.pos + static_cast<unsigned long long>(n_int) * static_cast<unsigned>(ax[d].bw);
            bad = bad || e > b.limit;
            if (vx && !bad) b.seek(e);
        } else if (ax[d].tag == 1 || ax[d].tag == 2) {
            ax[d].k = vx ? static_cast<int>(b.bits(8)) : 0;
            bad = bad || ax[d].k > kP5MaxK;
            ax[d].r.seek(vx ? b.pos : 0ull);
        } else {
            bad = true;  // ValueError("bad tag")
        }
        // the substream's codewords, skipped (every lane of the warp takes
        // part in the count)
        const bool skipping = vx && !bad && (ax[d].tag == 1 || ax[d].tag == 2);
        const uint32_t n = __reduce_max_sync(0xFFFFFFFFu, skipping ? n_int : 0u);
        for (uint32_t i = 0; i < n; i++)
            if (skipping && i < n_int) (void)p5_codeword(b, ax[d].tag == 2, ax[d].k);
        bad = bad || b.bad;
    }
    // meshlets lie back to back, as the CPU decoder reads them
    if (act) {
        bad = bad || (last ? b.pos > a.nbits : b.pos != s1);
        if (bad) p5_report(a.status, kErrCorrupt, m);
    }
    // 4. reconstruction in float64, in the reference's operation order, no
    // contraction (:426-445).  A strip-body vertex is predicted from the
    // previous triangle, whose interior vertices were reconstructed a step
    // or two before: the last four interior rows stay in registers, so those
    // references do not wait for a store to come back from L2.
    const bool rec = act && !bad && n_int > 0u;
    double fb[3] = {0.0, 0.0, 0.0};
    if (rec && n_bnd > 0u) {
        for (int d = 0; d < 3; d++) {
            double s = __ldcg(a.rows + 3ull * row_of(0u) + d);
#pragma unroll 4
            for (uint32_t i = 1; i < n_bnd; i++) s = __dadd_rn(s, __ldcg(a.rows + 3ull * row_of(i) + d));
            fb[d] = __ddiv_rn(s, static_cast<double>(n_bnd));
        }
    }
    uint32_t cid[4] = {0xFFFFu, 0xFFFFu, 0xFFFFu, 0xFFFFu};  // local ids of the cached rows (newest first)
    double cx[4][3];
#pragma unroll
    for (int j = 0; j < 4; j++) cx[j][0] = cx[j][1] = cx[j][2] = 0.0;
    // coordinate d of local vertex l: a cached row or the rows array
    auto coord = [&](uint32_t l, unsigned long long o, int d) -> double {
        double r = 0.0;
        bool hit = false;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const bool h = cid[j] == l;
            r = h ? cx[j][d] : r;
            hit = hit || h;
        }
        return hit ? r : __ldcg(a.rows + o + d);
    };
    const uint32_t ne = __reduce_max_sync(0xFFFFFFFFu, rec ? n_emit : 0u);
    uint32_t e_next = (rec && n_emit > 0u) ? __ldcg(a.walk + row0) : 0u;
    for (uint32_t i = 0; i < ne; i++) {
        if (!rec || i >= n_emit) continue;
        const uint32_t e = e_next;
        if (i + 1u < n_emit) e_next = __ldcg(a.walk + row0 + i + 1u);  // the next entry, a step ahead
        const uint32_t v = e & 0xFFu, ra = (e >> 8) & 0xFFu, rbv = (e >> 16) & 0xFFu, rc = e >> 24;
        const bool para = ra != v;  // roots are stored as (v, v, v, v)
        const unsigned long long out = 3ull * row_of(v);
        const unsigned long long oa = 3ull * row_of(ra), ob = 3ull * row_of(rbv), oc = 3ull * row_of(rc);
        double nr[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            long long code;
            if (ax[d].tag == 0) {
                code = ax[d].mn + static_cast<long long>(p5_bits_at(words, ax[d].base + static_cast<unsigned long long>(i) *
                                                                               static_cast<unsigned>(ax[d].bw),
                                                                    ax[d].bw, a.nbits, bad));
            } else {
                code = unzig(p5_codeword(ax[d].r, ax[d].tag == 2, ax[d].k));
            }
            double pred = fb[d];
            if (para) {
                const double t0 = __dmul_rn(a.w0, coord(ra, oa, d));
                const double t1 = __dmul_rn(a.w1, coord(rbv, ob, d));
                const double t2 = __dmul_rn(a.w2, coord(rc, oc, d));
                pred = __dadd_rn(__dadd_rn(t0, t1), t2);
            }
            nr[d] = __dadd_rn(pred, __dmul_rn(static_cast<double>(code), a.delta));
            a.rows[out + d] = nr[d];
        }
#pragma unroll
        for (int j = 3; j > 0; j--) {
            cid[j] = cid[j - 1];
            cx[j][0] = cx[j - 1][0];
            cx[j][1] = cx[j - 1][1];
            cx[j][2] = cx[j - 1][2];
        }
        cid[0] = v;
        cx[0][0] = nr[0];
        cx[0][1] = nr[1];
        cx[0][2] = nr[2];
    }
}

// ---- team kernel ------------------------------------------------------------
// A CTA takes up to M consecutive meshlets from their bytes to world positions
// in shared memory, as in stride_team.cu (whose parser, FIFO and assembly it
// shares): only what is serial stays on one lane per meshlet.
//
//  1. stage    a warp per meshlet: its bytes into shared memory, in bit order;
//              the parser warp then reads the boundary references.
//  2. connect  parser, FIFO and eight assembler warps, a chunk behind one
//              another; beside them the predictor warps sum the boundary rows
//              (the roots' prediction).
//  3. walk     a decoder lane per meshlet reads the three residual substreams
//              one after the other; two warps behind it scale the residuals
//              into their vertices' places; a predictor lane per (meshlet,
//              axis) follows on the last axis, in float64 and the reference's
//              operation order; three warps behind it put out float32 world
//              positions.
//
// What bounds it are the chains: 2.5K cycles to stage, 4.5K for the references,
// 31K for 280 tokens, 21K for the first two substreams of 120 residuals, 39K
// for 120 float64 predictions (a 33 x 33 terrain).  The general kernel, whose
// one lane has all of it, tokens one by one, takes eight times as long: 361 x 361
// terrain, 1,295 meshlets, 714 us against 90.
//
// The host knows every meshlet's size: a CTA's shared memory is what the
// stream's largest group of M needs, and each meshlet gets the room of its own
// (the room of the largest kept CTAs of sixteen from sharing an SM: 9,921
// meshlets 251 us, now 217).
struct P5Room {
    uint32_t bits = 0u;  // staged bytes (odd in units of 16)
    uint32_t loc = 0u;   // words of the walk, of the row table, and doubles of an axis (odd)
    uint32_t tok = 0u, asm_w = 0u;  // words of the token records and of the assembly
    __host__ __device__ void add(uint32_t bytes, uint32_t n_local, uint32_t n_tris, uint32_t n_tok) {
        bits += bytes | 16u;
        loc += n_local | 1u;
        tok += team_tok_words(n_tok);
        asm_w += team_asm_words(n_tris);
    }
};

constexpr int32_t kP5Zigzag = 1 << 30;  // in place of a minimum (16 bits): zigzag values
constexpr uint32_t kP5Res = 16u;  // residuals between hand-overs from the decoder to the predictor warps
constexpr uint32_t kP5MaxStage = 16384u;  // most staged bytes of a meshlet

template <uint32_t M>
__host__ __device__ constexpr uint32_t p5_pred_warps() {
    return (3u * M + 31u) / 32u;
}
template <uint32_t M>
__host__ __device__ constexpr uint32_t p5_team_threads() {
    return 32u * (kTeamAsm + 2u + p5_pred_warps<M>());
}
// Shared memory: staged bytes, then (also where a corrupt lane's reads end)
// walks and row tables, then the token records (read up to 31 past the last)
// and the assembly, whose place the planes take when the walk starts.
__host__ __device__ inline uint32_t p5_tables(const P5Room& t) {  // bytes before that
    return (t.bits + 8u * t.loc + 15u) & ~15u;
}
__host__ __device__ inline uint32_t p5_records(const P5Room& t) {  // their words
    return (t.tok + 3u) & ~3u;
}
inline uint32_t p5_team_bytes(const P5Room& t) {
    const uint32_t both = std::max(24u * t.loc, 4u * (p5_records(t) + t.asm_w));
    return (std::max(p5_tables(t) + both, t.bits + kTeamSlack) + 15u) & ~15u;
}

struct P5Facts : TeamSize {
    unsigned long long row0, tri0;
    uint32_t m, n_bnd, n_int, n_strips;
    uint32_t loc_off, tok_off, asm_off;  // words (doubles of an axis)
    uint32_t axis;       // doubles of an axis
    uint32_t at, end;    // bits of the staged words: after the header, the meshlet's end
    uint32_t conn;       // where the connectivity starts
    uint32_t anchor;     // ... and ends
    uint32_t n_walk;
    uint32_t bad;
    int32_t mn[3];       // a fixed-width substream's minimum, or kP5Zigzag
};

template <uint32_t M>
struct P5Shared {
    uint4 masks[17];
    P5Facts f[M];
    // parser steps of three chunks (being written; with the FIFO; with the assemblers)
    union {
        struct {
            uint32_t x[3][kTeamSteps * M];
            uint32_t step[3][kTeamSteps * M];
        };
        unsigned long long res[2][kP5Res * M];  // in the walk: codeword values of two chunks
    };
    uint8_t meta[3][kTeamSteps * M];
    double mean[3 * M];  // the roots' prediction, by (axis, meshlet)
    uint32_t more[2];  // the parser has tokens left after its last chunk
    uint32_t rmask;    // meshlets to decode
    uint32_t redo;     // decode the connectivity again, with the exact FIFO
};

// One codeword from bit `pos` of staged words, of any length below `limit`
// (the general reader, for the codewords longer than a window).
__device__ __noinline__ bool p5_long(const uint32_t* w, uint32_t& pos, uint32_t tag, uint32_t k, uint32_t limit,
                                     unsigned long long& u) {
    uint32_t q = 0u;
    if (tag != 0u) {
        for (;;) {
            if (pos >= limit) return false;
            const uint32_t x = peek32<true>(w, pos);
            const uint32_t z = static_cast<uint32_t>(__clz(x));
            q += z;
            pos += z;
            if (x) break;
        }
        pos++;
        if (tag == 2u && q > 32u) return false;  // (see P5Bits::eg)
    }
    auto take = [&](uint32_t n) -> uint32_t {
        if (n == 0u) return 0u;
        const uint32_t v = peek32<true>(w, pos) >> (32u - n);
        pos += n;
        return v;
    };
    unsigned long long head = q;
    if (tag == 2u) {
        if (pos + q > limit) return false;
        head = ((1ull << q) - 1ull) + take(q);
    }
    if (pos + k > limit) return false;
    const uint32_t low = take(k);
    u = (head << k) + low;
    return true;
}

// Four codewords of a substream (tag 0: fixed width k) from bit `pos` of the
// words at shared address `base`, the first n of them, as values into u.
// `far` when one is longer than 32 bits or starts beyond the window, or a fixed
// width is above 30: its lane then takes them again by the general reader.
// Bound by the chain from one codeword to the next: a 96-bit window read once
// for four leaves on it the leading zeros, a multiply-add and a funnel shift
// (45 cycles a codeword on one warp; with a window refilled at each one, 100).
__device__ __forceinline__ bool p5_four(uint32_t base, uint32_t& pos, uint32_t tag, uint32_t k, int n, uint32_t (&u)[4]) {
    const uint32_t em = tag, k1 = tag ? k + 1u : k, pow = tag ? 1u << (k & 31u) : 0u;
    const uint32_t zmul = tag == 1u ? pow : 0u, most = tag ? 32u : 30u;
    const uint32_t a = mad_u32(pos >> 5, 4u, base), o = pos & 31u;
    uint32_t w0, w1, w2, w3;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w0) : "r"(a));
    asm volatile("ld.shared.u32 %0, [%1+4];" : "=r"(w1) : "r"(a));
    asm volatile("ld.shared.u32 %0, [%1+8];" : "=r"(w2) : "r"(a));
    asm volatile("ld.shared.u32 %0, [%1+12];" : "=r"(w3) : "r"(a));
    uint32_t hi = __funnelshift_l(w1, w0, o), mid = __funnelshift_l(w2, w1, o), lo = __funnelshift_l(w3, w2, o);
    uint32_t used = 0u, longest = 0u, before = 0u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t len = __clz(hi) * em + k1;
        // with the terminator as the value bits' leading one: 2^nb + value
        u[i] = __clz(hi) * zmul + (__funnelshift_rc(hi, 0u, 32u - len) - pow);
        const uint32_t take = i < n ? len : 0u;
        longest = max(longest, take);
        before = used;
        used += take;
        hi = __funnelshift_lc(mid, hi, take);
        mid = __funnelshift_lc(lo, mid, take);
        lo = __funnelshift_lc(0u, lo, take);
    }
    pos += used;
    return (longest > most) | (before > 64u);
}

// A double from 32 bits by integer instructions: a float64 instruction takes a
// warp 64 cycles, a conversion 100.
__device__ __forceinline__ double p5_double(uint32_t q) {
    const uint32_t neg = sign_mask(q), u = (q ^ neg) - neg;
    const uint32_t z = __clz(u), m = __funnelshift_lc(0u, u, z);  // leading one on top
    const uint32_t top = u ? (neg & 0x80000000u) + ((1053u - z) << 20) + (m >> 11) : 0u;
    return __hiloint2double(static_cast<int>(top), static_cast<int>(m << 21));
}

__device__ __forceinline__ double ld_shared_f64(uint32_t a) {
    double x;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(a) : "memory");
    return x;
}

// Predictions of parallelogram entries of the walk, [h, h + 8) below n_walk, in
// the reference's order and without contraction (encoder/paradelta_v5.py:
// 426-445); a vertex's scaled residual is in its place of the plane, where the
// roots' rows are already.  Bound by the chain of float64 instructions, 64
// cycles each whatever their lanes: three an entry with the canonical weights
// 1, 1, -1 (kUnit: their products are exact), six with others.  Addresses are
// formed for all eight first, and no select is on the chain (one on a float64
// result costs it 50 cycles; rows through shared memory, 35): 256 cycles an
// entry on one warp, 342 with the last row kept in registers and the roots here.
template <bool kUnit>
__device__ __forceinline__ void p5_predict(uint32_t plane, const uint32_t* __restrict__ walk, uint32_t h, uint32_t n_walk,
                                           double w0, double w1, double w2) {
    uint32_t av[8], aa[8], ab[8], ac[8];
    double r[8];
#pragma unroll
    for (uint32_t i = 0; i < 8u; i++) {
        const uint32_t e = h + i < n_walk ? walk[h + i] : 0u;
        av[i] = mad_u32(__byte_perm(e, 0u, 0x4440u), 8u, plane);
        aa[i] = mad_u32(__byte_perm(e, 0u, 0x4441u), 8u, plane);
        ab[i] = mad_u32(__byte_perm(e, 0u, 0x4442u), 8u, plane);
        ac[i] = mad_u32(e >> 24, 8u, plane);
        r[i] = ld_shared_f64(av[i]);
    }
#pragma unroll
    for (uint32_t i = 0; i < 8u; i++) {
        const double a = ld_shared_f64(aa[i]), b = ld_shared_f64(ab[i]), c = ld_shared_f64(ac[i]);
        const double p = kUnit ? __dadd_rn(__dadd_rn(a, b), -c)
                               : __dadd_rn(__dadd_rn(__dmul_rn(w0, a), __dmul_rn(w1, b)), __dmul_rn(w2, c));
        const double x = __dadd_rn(p, r[i]);
        // roots, and entries past the end, are (v, v, v, v)
        asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %0, %2;\n@p st.shared.f64 [%0], %1;\n}" ::"r"(av[i]), "d"(x), "r"(aa[i])
                     : "memory");
    }
}

template <uint32_t M>
__global__ void __launch_bounds__(p5_team_threads<M>(), 2) p5_team_kernel(P5Args a) {
    constexpr uint32_t kThreads = p5_team_threads<M>(), kPred = p5_pred_warps<M>();
    constexpr uint32_t kPer = (M + kTeamAsm - 1u) / kTeamAsm;  // meshlets of an assembler warp
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ P5Shared<M> s;
    const uint32_t warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const bool predictor = warp >= kTeamAsm + 2u;
    const bool assembler = warp != kTeamParser && warp != kTeamFifo && !predictor;
    const uint32_t aw0 = team_asm_index(warp);  // an assembler's first meshlet
    const uint32_t n_here = min(M, a.n_meshlets - blockIdx.x * M);
    const uint32_t* words = reinterpret_cast<const uint32_t*>(smem);
    // 1. facts (lane j of every warp: meshlet j) and layout; stage.  The header
    // (:350-353), inside the stream as the host has checked, may end past the
    // meshlet.
    const bool have = static_cast<uint32_t>(lane) < n_here;
    const uint32_t lm = blockIdx.x * M + (have ? lane : 0);
    const uint32_t ls0 = __ldcg(a.start + lm), ls1 = __ldcg(a.start + lm + 1u);
    const uint32_t lrow = __ldcg(a.row_base + lm), ltri = __ldcg(a.tri_base + lm);
    const uint32_t lfrom = (ls0 >> 3) & ~15u;  // the first byte staged
    const uint32_t ln16 = ((ls1 - 8u * lfrom) + 127u) >> 7;
    uint32_t lh0, lh1;
    {
        const uint32_t* g = reinterpret_cast<const uint32_t*>(a.blob) + (ls0 >> 5);
        const uint32_t x = bswap32(__ldcg(g)), y = bswap32(__ldcg(g + 1)), z = bswap32(__ldcg(g + 2));
        lh0 = __funnelshift_l(y, x, ls0 & 31u);
        lh1 = __funnelshift_l(z, y, ls0 & 31u);
    }
    const uint32_t lloc = (lh0 >> 16) + (lh0 & 0xFFFFu), ltok = (lh1 >> 16) + 2u * (lh1 & 0xFFFFu);
    P5Room mine, all;
    if (have) mine.add(16u * ln16, lloc, lh1 >> 16, ltok);
    all = mine;
#pragma unroll
    for (uint32_t o = 1; o < M; o <<= 1) {
        const uint32_t b0 = __shfl_up_sync(kFull, all.bits, o), b1 = __shfl_up_sync(kFull, all.loc, o);
        const uint32_t b2 = __shfl_up_sync(kFull, all.tok, o), b3 = __shfl_up_sync(kFull, all.asm_w, o);
        if (static_cast<uint32_t>(lane) >= o) {
            all.bits += b0;
            all.loc += b1;
            all.tok += b2;
            all.asm_w += b3;
        }
    }
    P5Room off;  // exclusive
    off.bits = all.bits - mine.bits;
    off.loc = all.loc - mine.loc;
    off.tok = all.tok - mine.tok;
    off.asm_w = all.asm_w - mine.asm_w;
    all.bits = __shfl_sync(kFull, all.bits, M - 1u);
    all.loc = __shfl_sync(kFull, all.loc, M - 1u);
    all.tok = __shfl_sync(kFull, all.tok, M - 1u);
    uint32_t* walks = reinterpret_cast<uint32_t*>(smem + all.bits);
    uint32_t* tabs = walks + all.loc;
    double* planes = reinterpret_cast<double*>(smem + p5_tables(all));
    uint32_t* toks = reinterpret_cast<uint32_t*>(planes);
    uint32_t* asms = toks + p5_records(all);
    if (threadIdx.x < 17u) s.masks[threadIdx.x] = threadIdx.x < 16u ? mtf_mask_row(threadIdx.x) : make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0u && have) {
        P5Facts& F = s.f[lane];
        F.m = lm;
        F.n_bnd = lh0 >> 16;
        F.n_int = lh0 & 0xFFFFu;
        F.n_local = lloc;
        F.n_tris = lh1 >> 16;
        F.n_strips = lh1 & 0xFFFFu;
        F.n_tok = ltok;
        F.idsh = 9u - max(1u, 32u - __clz(lloc));
        F.loc_off = off.loc;
        F.tok_off = off.tok;
        F.asm_off = off.asm_w;
        F.axis = lloc | 1u;
        F.row0 = lrow;
        F.tri0 = ltri;
        F.end = ls1 - 8u * lfrom + 8u * off.bits;
        F.at = ls0 + 64u - 8u * lfrom + 8u * off.bits;
    }
    if (assembler) {
        for (uint32_t j = aw0; j < M; j += kTeamAsm) {
            const uint32_t from = __shfl_sync(kFull, lfrom, j), n16 = __shfl_sync(kFull, ln16, j);
            const uint32_t boff = __shfl_sync(kFull, off.bits, j), loff = __shfl_sync(kFull, off.loc, j);
            const uint32_t row0 = __shfl_sync(kFull, lrow, j), h0 = __shfl_sync(kFull, lh0, j);
            if (j >= n_here) continue;  // warp-uniform
            const uint4* src = reinterpret_cast<const uint4*>(a.blob + from);
            uint4* dst = reinterpret_cast<uint4*>(smem + boff);
            for (uint32_t i = lane; i < n16; i += 32u) {
                uint4 q = __ldcg(src + i);
                q.x = bswap32(q.x);
                q.y = bswap32(q.y);
                q.z = bswap32(q.z);
                q.w = bswap32(q.w);
                dst[i] = q;
            }
            const uint32_t n_bnd = h0 >> 16, n_int = h0 & 0xFFFFu;
            // rows of the interior vertices
            for (uint32_t i = lane; i < n_int; i += 32u) tabs[loff + n_bnd + i] = row0 + i;
        }
    }
    __syncthreads();
    // boundary references: the first in 32 bits, then Rice codewords of the
    // differences less one (:354-361); rows of the boundary table
    if (warp == kTeamParser) {
        const bool act = static_cast<uint32_t>(lane) < n_here;
        P5Facts& F = s.f[act ? lane : 0];
        const uint32_t n = act ? F.n_bnd : 0u;
        uint32_t* tab = tabs + (act ? F.loc_off : 0u);
        bool bad = act && (F.n_strips > F.n_tris || F.at > F.end);  // every strip emits a triangle
        const uint32_t limit = act ? F.end : 0u;
        const uint32_t base = smem_addr(words);
        uint32_t pos = act ? min(F.at, F.end) : 0u;
        unsigned long long prev = peek_shared(base, pos);
        pos += n > 0u ? 32u : 0u;
        uint32_t k = n > 1u ? peek_shared(base, pos) >> 24 : 0u;
        pos += n > 1u ? 8u : 0u;
        bad = bad || k > static_cast<uint32_t>(kP5MaxK) || pos > limit;
        if (n > 0u && !bad) {
            tab[0] = static_cast<uint32_t>(prev);
            bad = prev >= a.n_boundary;
        }
        k = bad ? 0u : k;
        const uint32_t most = __reduce_max_sync(kFull, bad ? 0u : n);
#pragma unroll 1
        for (uint32_t i0 = 1u; i0 < most; i0 += 8u) {
            const int left = bad ? 0 : static_cast<int>(n) - static_cast<int>(i0);
            uint32_t u[8], at = pos;
            bool far = false;
#pragma unroll
            for (int h = 0; h < 8; h += 4)
                far = p5_four(base, pos, 1u, k, left - h, *reinterpret_cast<uint32_t(*)[4]>(u + h)) | far;
            if (far) {
                for (int i = 0; i < 8; i++) {
                    if (i >= left || bad) continue;
                    unsigned long long v = 0ull;
                    if (!p5_long(words, at, 1u, k, limit, v) || v >= a.n_boundary) bad = true;
                    u[i] = static_cast<uint32_t>(v);
                }
                pos = at;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                prev += i < left ? u[i] + 1ull : 0ull;
                if (i < left) tab[i0 + i] = static_cast<uint32_t>(prev);
            }
            bad = bad || (left > 0 && (pos > limit || prev >= a.n_boundary));
            pos = min(pos, limit);
            __syncwarp();
        }
        if (act) F.conn = pos;
        if (bad) p5_report(a.status, kErrCorrupt, F.m);
        const uint32_t mask = __ballot_sync(kFull, act && !bad);
        if (lane == 0) s.rmask = mask;
    } else {
        // meanwhile the others: this CTA's share of the boundary rows' positions
        const uint32_t t = threadIdx.x < 32u * kTeamParser ? threadIdx.x : threadIdx.x - 32u;
        const unsigned long long all = static_cast<unsigned long long>(gridDim.x) * (kThreads - 32u);
        for (unsigned long long e = static_cast<unsigned long long>(blockIdx.x) * (kThreads - 32u) + t;
             e < 3ull * a.n_boundary; e += all)
            a.pos[e] = p5_world(a, __ldcg(a.rows + e), static_cast<uint32_t>(e % 3ull));
    }
    __syncthreads();
    const uint32_t rmask = s.rmask;
    // a predictor's (meshlet, axis)
    const uint32_t pid = (warp - kTeamAsm - 2u) * 32u + lane;
    const uint32_t pj = pid % M, pd = pid / M < 3u ? pid / M : 2u;
    const bool pon = predictor && pid < 3u * M && ((rmask >> pj) & 1u);
    double* pplane = planes + (pon ? 3u * s.f[pj].loc_off + pd * s.f[pj].axis : 0u);
    // 2. connectivity, in step: chunk c with the parser, c - 1 with the FIFO
    // warp, c - 2 with the assemblers
    for (uint32_t pass = 0; pass < 2u; pass++) {  // the second one with the exact FIFO, rarely
        const bool exact = pass != 0u;
        if (threadIdx.x == 0) s.redo = 0u;
        if (threadIdx.x < M) s.f[threadIdx.x].bad = 0u;
        __syncthreads();
        if (predictor) {
            // the roots' prediction: the mean of the boundary rows, summed in
            // order (:362-365)
            const uint32_t n = pon && !exact ? s.f[pj].n_bnd : 0u;
            const uint32_t most = __reduce_max_sync(kFull, n);
            const uint32_t* tab = tabs + (pon ? s.f[pj].loc_off : 0u);
            double mean = 0.0;
            uint32_t at = 0u;
            auto sum = [&](uint32_t upto) {
                for (; at < upto; at += 8u) {
                    double r[8];
#pragma unroll
                    for (uint32_t i = 0; i < 8u; i++) r[i] = at + i < n ? __ldcg(a.rows + 3ull * tab[at + i] + pd) : 0.0;
                    if (at == 0u) mean = n ? -0.0 : 0.0;  // the first sum is the first row
#pragma unroll
                    for (uint32_t i = 0; i < 8u; i++)
                        if (at + i < n) mean = __dadd_rn(mean, r[i]);
                }
            };
            bool more = true;
            for (uint32_t c = 0;; c++) {
                sum(min(at + 16u, most));
                team_all_bar<kThreads>();
                if (!more) break;
                more = s.more[c & 1u] != 0u;
            }
            sum(most);
            if (n) mean = __ddiv_rn(mean, static_cast<double>(n));
            if (pon && !exact) s.mean[pid] = mean;
            if (exact) {
                team_all_bar<kThreads>();
                team_all_bar<kThreads>();
            }
        } else if (!assembler) {
            const bool act = (rmask >> lane) & 1u;
            P5Facts& F = s.f[act ? lane : 0];
            const uint32_t n_tok = act ? F.n_tok : 0u;
            const uint32_t sl = act ? lane : 0u;  // an idle lane repeats the first one's steps
            const uint32_t ib = act ? 9u - F.idsh : 1u;
            uint16_t* row = reinterpret_cast<uint16_t*>(toks + (act ? F.tok_off : 0u)) + 2;
            TeamParse T;
            MtfFifo fifo;
            uint32_t t = 0u;
            uint32_t past = 0u;  // negative: a FIFO index named no entry
            T.strips = F.n_strips;
            T.pos = act ? F.conn : 0u;
            fifo.f0 = fifo.f1 = fifo.f2 = fifo.f3 = 0xFFFFFFFFu;
            if (warp == kTeamParser && act) row[-2] = row[-1] = 0;
            bool more = true;
            for (uint32_t c = 0;; c++) {
                if (warp == kTeamParser) {
                    const uint32_t b = c % 3u;
                    if (act) team_parse<true, M>(T, words, n_tok, ib, 0u, s.x[b] + lane, s.meta[b] + lane);
                    __syncwarp();
                    const bool m = __any_sync(kFull, T.t < n_tok);
                    if (lane == 0) s.more[c & 1u] = m ? 1u : 0u;
                } else if (c > 0u) {
                    const uint32_t b = (c - 1u) % 3u;
                    if (act) team_fifo<M>(fifo, t, s.x[b] + sl, s.meta[b] + sl, s.step[b] + sl, ib, s.masks, past);
                }
                __syncwarp();
                team_all_bar<kThreads>();
                if (!more) break;  // this was the chunk after the parser's last
                more = s.more[c & 1u] != 0u;
            }
            if (act && warp == kTeamParser) {
                F.anchor = T.pos;
                // every strip read, inside the meshlet
                if (T.t != n_tok || T.strips != 0u || T.left != 0u || T.pos > F.end) atomicOr(&F.bad, 1u);
            }
            if (exact) team_all_bar<kThreads>();  // the records are there
            if (act && warp == kTeamFifo) {
                if (exact ? !team_fifo_exact(row, n_tok, F.idsh, s.masks) : sign_mask(past) != 0u) atomicOr(&F.bad, 1u);
            }
            __syncwarp();
            if (exact) team_all_bar<kThreads>();
        } else {
            TeamAsm S[kPer];
            auto mine = [&](uint32_t q) { return aw0 + q * kTeamAsm < M && ((rmask >> (aw0 + q * kTeamAsm)) & 1u); };
            // the windows that the records fill (or end)
            auto windows = [&](TeamAsm& A, uint32_t j) {
                const P5Facts& F = s.f[j];
                uint32_t* last = asms + F.asm_off;
                const uint32_t have = A.t >= F.n_tok ? F.n_tok + 31u : A.t;
                for (; A.t0 + 32u <= have; A.t0 += 32u)
                    team_window<false>(A, F, F.n_bnd, exact, A.t0, reinterpret_cast<const uint16_t*>(toks + F.tok_off) + 2,
                                       walks + F.loc_off, nullptr, last, last + 256, lane);
            };
            auto chunk = [&](uint32_t c) {
#pragma unroll
                for (uint32_t q = 0; q < kPer; q++) {
                    const uint32_t j = aw0 + q * kTeamAsm;
                    if (!mine(q) || S[q].t >= s.f[j].n_tok) continue;  // warp-uniform, here and below
                    team_records<M>(S[q], s.f[j], exact, reinterpret_cast<uint16_t*>(toks + s.f[j].tok_off) + 2,
                                    s.x[c % 3u] + j, s.step[c % 3u] + j, lane);
                    if (!exact) windows(S[q], j);
                }
            };
#pragma unroll
            for (uint32_t q = 0; q < kPer; q++) {
                const uint32_t j = aw0 + q * kTeamAsm;
                if (!mine(q)) continue;
                uint4* last = reinterpret_cast<uint4*>(asms + s.f[j].asm_off);
                last[lane] = last[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
            }
            __syncwarp();
            bool more = true;
            uint32_t c = 0u;
            for (;; c++) {
                if (c > 1u) chunk(c - 2u);
                team_all_bar<kThreads>();
                if (!more) break;
                more = s.more[c & 1u] != 0u;
            }
            chunk(c - 1u);  // the parser's last chunk
            if (exact) {
                __syncwarp();
                team_all_bar<kThreads>();
                team_all_bar<kThreads>();  // the FIFO warp has resolved the records
#pragma unroll
                for (uint32_t q = 0; q < kPer; q++)
                    if (mine(q)) windows(S[q], aw0 + q * kTeamAsm);
            }
#pragma unroll
            for (uint32_t q = 0; q < kPer; q++) {
                const uint32_t j = aw0 + q * kTeamAsm;
                if (!mine(q)) continue;
                P5Facts& F = s.f[j];
                const uint32_t* tab = tabs + F.loc_off;
                // ids of a valid meshlet lie in the table; an invalid one's are cut to it
                const uint32_t vmax = F.n_local ? F.n_local - 1u : 0u;
                uint32_t* out = a.idx + 3ull * F.tri0;
                const uint32_t ph = (0u - static_cast<uint32_t>(reinterpret_cast<uintptr_t>(out) >> 2)) & 3u;
                team_triangles(out, asms + F.asm_off + 256, ph, min(S[q].tcnt, F.n_tris),
                               [&](uint32_t v) { return tab[min(v, vmax)]; }, lane);
                const bool bad = __any_sync(kFull, S[q].out) || S[q].tcnt != F.n_tris;
                if (lane == 0) {
                    F.n_walk = min(S[q].wcnt, F.n_int);
                    if (bad || S[q].wcnt > F.n_int) atomicOr(&F.bad, 1u);
                    if (S[q].redo && !exact) s.redo = 1u;
                }
            }
        }
        __syncthreads();
        if (s.redo == 0u || exact) break;
        __syncthreads();  // everyone has read it
    }
    // 3. walk, in step: chunk g with the decoder, g - 1 with the warps that
    // put its residuals, scaled, and the roots' rows into the plane, and of
    // the last axis g - 2 with the predictors and g - 3 with the warps that put
    // positions out (on schedulers that the predictors do not use).
    constexpr uint32_t kScalers = 2u, kEmitters = 3u;
    const uint32_t scaler = warp == 1u ? 0u : (warp == 4u ? 1u : kScalers);
    const uint32_t emitter = warp == 5u ? 0u : (warp == 8u || warp == 9u ? warp - 7u : kEmitters);
    const bool lon = static_cast<uint32_t>(lane) < M && ((rmask >> lane) & 1u) && s.f[lane].bad == 0u;
    const uint32_t on_mask = __ballot_sync(kFull, lon);
    if (warp == 0u || scaler < kScalers || predictor || emitter < kEmitters) {
        constexpr uint32_t kBar = 32u * (1u + kScalers + kPred + kEmitters);
        auto bar = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(kBar) : "memory"); };
        const uint32_t chunks = (__reduce_max_sync(kFull, lon ? s.f[lane].n_int : 0u) + kP5Res - 1u) / kP5Res;
        const uint32_t steps = 3u * chunks + 3u;
        if (predictor) {
            const bool on = pon && ((on_mask >> pj) & 1u);
            const P5Facts& F = s.f[on ? pj : 0u];
            const uint32_t n_walk = on ? F.n_walk : 0u;
            if (on && n_walk < F.n_int)  // vertices that the walk never reaches keep row 0
                for (uint32_t i = 0; i < F.n_int; i++) pplane[F.n_bnd + i] = 0.0;
            __syncwarp();
            bar();
            const uint32_t* walk = walks + (on ? F.loc_off : 0u);
            const uint32_t plane_addr = smem_addr(pplane);
            const bool unit = a.w0 == 1.0 && a.w1 == 1.0 && a.w2 == -1.0;
            for (uint32_t g = 0; g < steps; g++) {
                if (g >= 2u * chunks + 2u && g < 3u * chunks + 2u) {
                    const uint32_t h0 = (g - 2u - 2u * chunks) * kP5Res;
#pragma unroll 1
                    for (uint32_t h = h0; h < h0 + kP5Res; h += 8u) {
                        if (unit) {
                            p5_predict<true>(plane_addr, walk, h, n_walk, a.w0, a.w1, a.w2);
                        } else {
                            p5_predict<false>(plane_addr, walk, h, n_walk, a.w0, a.w1, a.w2);
                        }
                    }
                }
                __syncwarp();
                bar();
            }
        } else if (scaler < kScalers) {
            bar();
            uint32_t d = 0u, c = 0u;
            for (uint32_t g = 0; g < steps; g++) {
                if (g > 0u && g <= 3u * chunks) {
                    constexpr uint32_t kIts = M * kP5Res / 64u;
                    double* slot[kIts];
                    double x[kIts], mean[kIts];
                    long long r[kIts];
                    bool in[kIts], wide = false;
#pragma unroll
                    for (uint32_t q = 0; q < kIts; q++) {
                        const uint32_t it = 64u * q + 32u * scaler + lane, j = it % M, i = c * kP5Res + it / M;
                        in[q] = ((on_mask >> j) & 1u) && i < s.f[j].n_walk;
                        const int32_t mn = s.f[j].mn[d];
                        const unsigned long long u = s.res[(g - 1u) & 1u][it];
                        r[q] = mn == kP5Zigzag ? unzig(u) : mn + static_cast<long long>(u);
                        const uint32_t e = walks[(in[q] ? s.f[j].loc_off + i : 0u)], v = e & 0xFFu;
                        // roots are (v, v, v, v); a residual that is added to nothing is added to -0
                        mean[q] = v == ((e >> 8) & 0xFFu) ? s.mean[d * M + j] : -0.0;
                        slot[q] = planes + (in[q] ? 3u * s.f[j].loc_off + d * s.f[j].axis : 0u) + v;
                        x[q] = p5_double(static_cast<uint32_t>(r[q]));
                        wide = wide | (r[q] != static_cast<int32_t>(r[q]));
                    }
                    if (__any_sync(kFull, wide)) {
#pragma unroll
                        for (uint32_t q = 0; q < kIts; q++) x[q] = static_cast<double>(r[q]);
                    }
#pragma unroll
                    for (uint32_t q = 0; q < kIts; q++) {
                        x[q] = __dadd_rn(mean[q], __dmul_rn(x[q], a.delta));
                        if (in[q]) *slot[q] = x[q];
                    }
                    c++;
                    if (c == chunks) c = 0u, d++;
                }
                __syncwarp();
                bar();
            }
        } else if (warp == 0u) {
            // (lanes from M on repeat the first M)
            const uint32_t j = lane % M;
            const bool on = (on_mask >> j) & 1u;
            P5Facts& F = s.f[on ? j : 0u];
            const uint32_t n = on ? F.n_int : 0u;
            const uint32_t limit = on ? F.end : 0u;
            const uint32_t base = smem_addr(words);
            uint32_t pos = on ? F.anchor : 0u;
            bool bad = false;
            bar();
            uint32_t g = 0u;
#pragma unroll 1
            for (uint32_t d = 0; d < 3u; d++) {
                // tag, then fixed width (tag 0: minimum and width) or Rice /
                // Exp-Golomb (tags 1, 2: k) (:403-424)
                uint32_t tag = 1u, k = 0u;
                if (n) {
                    const uint32_t x = peek_shared(base, pos), y = peek_shared(base, pos + 24u);
                    tag = x >> 24;
                    k = tag ? (x >> 16) & 0xFFu : y >> 24;
                    F.mn[d] = tag ? kP5Zigzag : static_cast<int32_t>(x << 8) >> 16;
                    pos += tag ? 16u : 32u;
                    bad = bad || tag > 2u || k > static_cast<uint32_t>(tag ? kP5MaxK : kP5MaxWidth);
                    tag = bad ? 1u : tag;
                    k = bad ? 0u : k;
                }
                __syncwarp();
#pragma unroll 1
                for (uint32_t c = 0; c < chunks; c++, g++) {
                    unsigned long long* res = s.res[g & 1u] + j;
                    const int left = bad ? 0 : static_cast<int>(n) - static_cast<int>(c * kP5Res);
                    uint32_t at = pos;
                    bool far = false;
#pragma unroll
                    for (uint32_t h = 0; h < kP5Res; h += 4u) {
                        uint32_t u[4];
                        far = p5_four(base, pos, tag, k, left - static_cast<int>(h), u) | far;
                        pos = min(pos, limit + 128u);  // inside what a corrupt lane may read
#pragma unroll
                        for (uint32_t i = 0; i < 4u; i++) res[(h + i) * M] = u[i];
                    }
                    if (far) {
                        for (int i = 0; i < static_cast<int>(kP5Res); i++) {
                            unsigned long long v = 0ull;
                            if (i < left && !bad) bad = !p5_long(words, at, tag, k, limit, v);
                            res[i * M] = v;
                        }
                        pos = at;
                    }
                    bad = bad || pos > limit;
                    pos = min(pos, limit);
                    __syncwarp();
                    bar();
                }
            }
            // meshlets lie back to back, as the CPU decoder reads them
            const bool last = F.m + 1u == a.n_meshlets;
            if (on && (bad || (!last && pos != limit))) F.bad = 1u;
            bar();
            bar();
            bar();
        } else {
            // f32(row * scale + center)
            bar();
            uint32_t rows = 0u;  // meshlets whose boundary rows are in the planes
            for (uint32_t g = 0; g < steps; g++) {
                // first, before the predictors start, the boundary rows of a
                // meshlet a step (through L2, as every global read: a handle
                // may have another's memory)
                const uint32_t upto = g < 2u * chunks ? min(rows + 1u, n_here) : n_here;
                for (; g < 2u * chunks + 2u && rows < upto; rows++) {
                    if (!((on_mask >> rows) & 1u)) continue;
                    const P5Facts& F = s.f[rows];
#pragma unroll 4
                    for (uint32_t e = 32u * emitter + lane; e < 3u * F.n_bnd; e += 32u * kEmitters) {
                        const uint32_t i = e / 3u, d = e - 3u * i;
                        planes[3u * F.loc_off + d * F.axis + i] = __ldcg(a.rows + 3ull * tabs[F.loc_off + i] + d);
                    }
                }
                if (g >= 2u * chunks + 3u) {
                    const uint32_t c = g - 3u - 2u * chunks;
#pragma unroll 2
                    for (uint32_t it = 32u * emitter + lane; it < 3u * M * kP5Res; it += 32u * kEmitters) {
                        const uint32_t d = it % 3u, j = it / (3u * kP5Res), i = c * kP5Res + it / 3u % kP5Res;
                        const P5Facts& F = s.f[j];
                        if (!((on_mask >> j) & 1u) || i >= F.n_walk) continue;
                        const uint32_t v = walks[F.loc_off + i] & 0xFFu;
                        a.pos[3ull * (F.row0 + (v - F.n_bnd)) + d] = p5_world(a, planes[3u * F.loc_off + d * F.axis + v], d);
                    }
                }
                __syncwarp();
                bar();
            }
        }
    }
    __syncthreads();
    // invalid meshlets, and those with vertices that the walk never reaches
    if (assembler) {
        for (uint32_t j = aw0; j < n_here; j += kTeamAsm) {
            if (!((rmask >> j) & 1u)) continue;
            const P5Facts& F = s.f[j];
            if (F.bad) {
                if (lane == 0) p5_report(a.status, kErrCorrupt, F.m);
            } else if (F.n_walk < F.n_int) {
                for (uint32_t e = lane; e < 3u * F.n_int; e += 32u) {
                    const uint32_t i = e / 3u, d = e - 3u * i;
                    a.pos[3ull * F.row0 + e] = p5_world(a, planes[3u * F.loc_off + d * F.axis + F.n_bnd + i], d);
                }
            }
        }
    }
}

__global__ void p5_world_kernel(P5Args a, unsigned long long n) {
    const unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
    if (i < 3ull * n) a.pos[i] = p5_world(a, a.rows[i], static_cast<uint32_t>(i % 3ull));
}

constexpr uint32_t kP5Eight = 8u * 2u * 152u * 9u / 8u;  // about as many as CTAs of eight take at once on a GB300
constexpr uint32_t kP5Most = 44u << 10;        // meshlets of a stream
constexpr uint32_t kP5Two = 102u << 10;        // two CTAs to an SM
// eight meshlets of the largest size that is accepted (197 KB) and the static part, in an SM's 227 KB
constexpr uint32_t kP5MaxSmem = 200u << 10;

template <uint32_t M>
cudaError_t p5_team_prepare() {
    cudaError_t e = cudaFuncSetAttribute(p5_team_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kP5MaxSmem));
    if (e != cudaSuccess) return e;
    // global data is read through L2 only
    return cudaFuncSetAttribute(p5_team_kernel<M>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared);
}

template <uint32_t M>
cudaError_t p5_team_launch(const P5Args& a, uint32_t smem, cudaStream_t s) {
    p5_team_kernel<M><<<(a.n_meshlets + M - 1u) / M, p5_team_threads<M>(), smem, s>>>(a);
    return cudaGetLastError();
}

// ---- host side ------------------------------------------------------------
struct HostBits {
    const uint8_t* p;
    unsigned long long nbits, pos;
    bool bad;
    uint64_t read(int n) {  // n <= 64
        if (n <= 0) return 0;
        if (pos + static_cast<unsigned>(n) > nbits) {
            bad = true;
            pos = nbits;
            return 0;
        }
        uint64_t v = 0;
        for (int i = 0; i < n; i++, pos++) v = (v << 1) | ((p[pos >> 3] >> (7 - (pos & 7))) & 1u);
        return v;
    }
    uint64_t rice(int k) {  // q < 2^32 (the stream length) and k <= 24 fit 64 bits
        uint64_t q = 0;
        for (;;) {
            if (pos >= nbits) {
                bad = true;
                return 0;
            }
            const unsigned bit = (p[pos >> 3] >> (7 - (pos & 7))) & 1u;
            pos++;
            if (bit) break;
            q++;
        }
        if (k > kP5MaxK) {
            bad = true;
            return 0;
        }
        return (q << k) | read(k);
    }
    float f32() {
        const uint32_t u = static_cast<uint32_t>(read(32));
        float f;
        std::memcpy(&f, &u, 4);
        return f;
    }
};

}  // namespace
}  // namespace stride

using namespace stride;

struct pldt5_handle {
    pldt5_info_t info;
    size_t len = 0;
    uint8_t* d_blob = nullptr;
    uint32_t* d_meta = nullptr;  // start (n + 1) | row_base (n) | tri_base (n) | ref_base (n)
    uint32_t* d_refs = nullptr;  // refs, walk: the general kernel's
    uint32_t* d_walk = nullptr;
    double* d_rows = nullptr;    // the boundary's, and for the general kernel all
    uint32_t team = 0;           // meshlets per CTA of the team kernel, 0: the general kernel
    uint32_t team_smem = 0;      // its dynamic shared memory
    Status* d_status = nullptr;
    Status* h_status = nullptr;
    cudaEvent_t done = nullptr;
    bool launched = false;
    double w[3], delta, scale, center[3];
};

static void pldt5_free(pldt5_handle* h) {
    cudaFree(h->d_blob);
    cudaFree(h->d_meta);
    cudaFree(h->d_refs);
    cudaFree(h->d_walk);
    cudaFree(h->d_rows);
    cudaFree(h->d_status);
    pinned_give(h->h_status);
    if (h->done) cudaEventDestroy(h->done);
    delete h;
}

// Host parse shared by pldt5_open and pldt5_inspect: header, boundary rows
// (float64), every meshlet's start bit and output placement.  STRIDE_OK or
// a STRIDE_ERR_* with the message set.
struct P5Host {
    pldt5_info_t info;
    float per_coord_err;
    std::vector<double> rows0;    // boundary rows, n_boundary x 3
    std::vector<uint32_t> meta;   // start (M + 1) | row_base (M) | tri_base (M) | ref_base (M)
    uint64_t refs = 0;
    // the largest meshlet's
    uint32_t most_tokens = 0, most_bytes = 0;
    // shared memory of the largest group of eight and of sixteen meshlets
    uint32_t smem8 = 0, smem16 = 0;
};

static int p5_host_parse_sized(const uint8_t* data, size_t len, P5Host& H);

// The host parse with its host allocations' failures turned into an error
// code (no exception may cross the C ABI).
static int p5_host_parse(const uint8_t* data, size_t len, P5Host& H) {
    try {
        return p5_host_parse_sized(data, len, H);
    } catch (const std::bad_alloc&) {
        return fail(STRIDE_ERR_NOMEM, "host memory for the PLDT v5 tables");
    } catch (const std::length_error&) {
        return fail(STRIDE_ERR_NOMEM, "host memory for the PLDT v5 tables");
    }
}

static int p5_host_parse_sized(const uint8_t* data, size_t len, P5Host& H) {
    pldt5_info_t& info = H.info;
    HostBits r{data, 8ull * len, 0, false};
    if (8ull * len < kP5HeaderBits) return fail(STRIDE_ERR_TRUNCATED, "PLDT v5 header past the end");
    std::memset(&info, 0, sizeof(info));
    const uint32_t magic = static_cast<uint32_t>(r.read(32));
    if (magic != kP5Magic) return fail(STRIDE_ERR_MAGIC, "bad magic 0x%08X (PLDT v5 expected)", magic);
    const uint32_t version = static_cast<uint32_t>(r.read(8));
    if (version != kP5Version) return fail(STRIDE_ERR_VERSION, "expected v5, got v%u", version);
    (void)r.read(8);  // code width: a shared-memory hint of the reference kernel
    for (int d = 0; d < 3; d++) info.center[d] = r.f32();
    info.scale = r.f32();
    const float per_coord_err = r.f32();
    H.per_coord_err = per_coord_err;
    float g_min[3], g_range[3];
    for (int d = 0; d < 3; d++) g_min[d] = r.f32();
    for (int d = 0; d < 3; d++) g_range[d] = r.f32();
    for (int d = 0; d < 3; d++) info.g_bits[d] = static_cast<uint32_t>(r.read(8));
    (void)r.read(32);  // n_v and n_t of the source mesh: the decoder counts its own
    (void)r.read(32);
    info.n_boundary = static_cast<uint32_t>(r.read(32));
    info.n_meshlets = static_cast<uint32_t>(r.read(32));
    for (int d = 0; d < 3; d++) info.lin3_w[d] = r.f32();
    for (int d = 0; d < 3; d++)
        if (info.g_bits[d] > 32) return fail(STRIDE_ERR_UNSUPPORTED, "g_bits %u above 32", info.g_bits[d]);
    // boundary table (parse_globals_v5, :538-560), positions in float64 like
    // the CPU decoder (:322-336)
    const uint64_t nb = info.n_boundary;
    // every row after the first takes at least one bit per axis (a Rice
    // codeword's terminator): the header's count is bounded by the bits
    // left before anything is sized from it
    if (nb > (8ull * len - r.pos) / 3ull + 1ull) return fail(STRIDE_ERR_TRUNCATED, "boundary table past the end");
    std::vector<double>& rows0 = H.rows0;
    rows0.assign(3 * nb, 0.0);
    {
        std::vector<int64_t> code(3 * nb, 0);
        for (int d = 0; d < 3 && nb > 0; d++) {
            code[d] = static_cast<int64_t>(r.read(static_cast<int>(info.g_bits[d])));
            if (nb > 1) {
                const int k = static_cast<int>(r.read(8));
                for (uint64_t i = 1; i < nb && !r.bad; i++) {
                    const uint64_t u = r.rice(k);
                    code[3 * i + d] = code[3 * (i - 1) + d] + static_cast<int64_t>((u >> 1) ^ (0ull - (u & 1ull)));
                }
            }
        }
        if (r.bad) return fail(STRIDE_ERR_TRUNCATED, "boundary table past the end or malformed");
        for (uint64_t i = 0; i < nb; i++)
            for (int d = 0; d < 3; d++) {
                const uint64_t mx = (1ull << info.g_bits[d]) - 1ull;
                if (mx == 0) {
                    rows0[3 * i + d] = static_cast<double>(g_min[d]);
                } else {
                    const double q = static_cast<double>(code[3 * i + d]) / static_cast<double>(mx);
                    rows0[3 * i + d] = static_cast<double>(g_min[d]) + q * static_cast<double>(g_range[d]);
                }
            }
    }
    // offset table, then every meshlet's header (the reference's sizes pass)
    r.pos += (0ull - r.pos) & 7ull;
    const uint64_t M = info.n_meshlets;
    if (r.pos + 32ull * M > r.nbits) return fail(STRIDE_ERR_TRUNCATED, "offset table past the end");
    std::vector<uint32_t>& meta = H.meta;
    meta.assign(4 * M + 1, 0u);
    uint32_t* start = meta.data();
    uint32_t* row_base = start + M + 1;
    uint32_t* tri_base = row_base + M;
    uint32_t* ref_base = tri_base + M;
    for (uint64_t m = 0; m < M; m++) start[m] = static_cast<uint32_t>(r.read(32));
    const uint64_t body = r.pos;
    start[M] = static_cast<uint32_t>(std::min<uint64_t>(8ull * len, 0xFFFFFFFFull));
    if (8ull * len > 0xFFFFFFFFull) return fail(STRIDE_ERR_UNSUPPORTED, "stream above 512 MiB");
    uint64_t rows = nb, tris = 0, refs = 0;
    P5Room r8, r16;  // of the group so far
    for (uint64_t m = 0; m < M; m++) {
        // the CPU decoder reads meshlets back to back from the end of the table
        if ((m == 0 && start[0] != body) || start[m] < body || start[m] + 64ull > 8ull * len ||
            (m > 0 && start[m] <= start[m - 1]))
            return fail(STRIDE_ERR_OFFSET, "meshlet %llu offset out of order or range", (unsigned long long)m);
        HostBits hb{data, 8ull * len, start[m], false};
        const uint32_t n_bnd = static_cast<uint32_t>(hb.read(16));
        const uint32_t n_int = static_cast<uint32_t>(hb.read(16));
        const uint32_t n_tris = static_cast<uint32_t>(hb.read(16));
        const uint32_t n_strips = static_cast<uint32_t>(hb.read(16));
        H.most_tokens = std::max(H.most_tokens, n_tris + 2u * n_strips);
        // staged: from the 16 bytes of its first bit to those of its last
        const uint64_t first = (start[m] >> 3) & ~15ull, end = ((start[m + 1] + 127ull) >> 7) << 4;
        const uint32_t staged = static_cast<uint32_t>(std::min<uint64_t>(end - first, 0xFFFFFFF0u));
        H.most_bytes = std::max(H.most_bytes, staged);
        if (m % 8 == 0) r8 = P5Room{};
        if (m % 16 == 0) r16 = P5Room{};
        if (H.most_tokens <= kTeamTokens && H.most_bytes <= kP5MaxStage) {  // else there is no team
            r8.add(staged, n_bnd + n_int, n_tris, n_tris + 2u * n_strips);
            r16.add(staged, n_bnd + n_int, n_tris, n_tris + 2u * n_strips);
            H.smem8 = std::max(H.smem8, p5_team_bytes(r8));
            H.smem16 = std::max(H.smem16, p5_team_bytes(r16));
        }
        if (n_bnd + n_int > static_cast<uint32_t>(kP5MaxLocal))
            return fail(STRIDE_ERR_UNSUPPORTED, "meshlet %llu has %u local vertices (at most 256)",
                        (unsigned long long)m, n_bnd + n_int);
        row_base[m] = static_cast<uint32_t>(rows);
        tri_base[m] = static_cast<uint32_t>(tris);
        ref_base[m] = static_cast<uint32_t>(refs);
        rows += n_int;
        tris += n_tris;
        refs += n_bnd;
        if (rows > 0xFFFFFFFFull || tris > 0x55555555ull || refs > 0xFFFFFFFFull)
            return fail(STRIDE_ERR_UNSUPPORTED, "more than 2^32 rows, indices or boundary references");
    }
    info.n_v = rows;
    info.n_t = tris;
    info.nbytes = len;
    H.refs = refs;
    return STRIDE_OK;
}

// Room and launch shape for a stream: the team kernel takes meshlets of up to
// kTeamTokens tokens and kP5MaxStage bytes (encoded meshlets of 256 vertices
// have half as many and a tenth), in streams of up to kP5Most meshlets; the
// general kernel the others.  Its time hardly grows with the meshlets, the
// team's does: up to 256 vertices, 21,307 / 43,086 meshlets 778 / 895 us and 383
// / 721; up to 64 vertices, 23,843 / 50,955 meshlets 302 / 376 and 228 / 445.
static cudaError_t p5_plan(const P5Host& H, uint32_t& team, uint32_t& smem) {
    team = smem = 0;
    if (H.info.n_meshlets == 0 || H.info.n_meshlets > kP5Most || H.most_tokens > kTeamTokens ||
        H.most_bytes > kP5MaxStage)
        return cudaSuccess;
    // Eight meshlets per CTA as long as the CTAs are on the chip at once, two
    // to an SM (or all but a few); above, sixteen where two such CTAs fit an SM:
    // a decode then takes the CTAs' waves, and a CTA's chains hardly depend on
    // its number of meshlets (sixteen against eight: meshlets of up to 64
    // vertices, 3,072 of them, 65 us against 79, 23,843 228 against 289; of up to
    // 199 vertices, 10 78 against 76, 2,451 102 against 90, 4,913 141 against 149,
    // 9,921 217 against 252).
    team = H.info.n_meshlets > kP5Eight && H.smem16 <= kP5Two ? 16u : 8u;
    smem = team == 8u ? H.smem8 : H.smem16;
    return team == 8u ? p5_team_prepare<8>() : p5_team_prepare<16>();
}

extern "C" {

int pldt5_open(const uint8_t* data, size_t len, pldt5_handle** out) {
    if (!out || (!data && len)) return fail(STRIDE_ERR_ARG, "null argument");
    *out = nullptr;
    P5Host H;
    const int prc = p5_host_parse(data, len, H);
    if (prc) return prc;
    const pldt5_info_t& info = H.info;
    const uint64_t nb = info.n_boundary, rows = info.n_v, refs = H.refs;
    const float per_coord_err = H.per_coord_err;
    const std::vector<double>& rows0 = H.rows0;
    const std::vector<uint32_t>& meta = H.meta;

    pldt5_handle* h = new pldt5_handle();
    h->info = info;
    h->len = len;
    for (int d = 0; d < 3; d++) {
        h->w[d] = static_cast<double>(info.lin3_w[d]);
        h->center[d] = static_cast<double>(info.center[d]);
    }
    h->scale = static_cast<double>(info.scale);
    h->delta = 2.0 * static_cast<double>(per_coord_err);
    cudaError_t e = p5_plan(H, h->team, h->team_smem);
    if (e != cudaSuccess) {
        pldt5_free(h);
        return cuda_fail(e, "pldt5_open");
    }
    const uint64_t gen = h->team ? 0 : 1;  // buffers of the general kernel
    const size_t blob = blob_alloc_bytes(len);
    if ((e = cudaMalloc(&h->d_blob, blob)) != cudaSuccess ||
        (e = cudaMalloc(&h->d_meta, 4 * meta.size())) != cudaSuccess ||
        (e = cudaMalloc(&h->d_refs, 4 * std::max<uint64_t>(gen * refs, 1))) != cudaSuccess ||
        (e = cudaMalloc(&h->d_walk, 4 * std::max<uint64_t>(gen * rows, 1))) != cudaSuccess ||
        (e = cudaMalloc(&h->d_rows, 24 * std::max<uint64_t>(gen ? rows : nb, 1))) != cudaSuccess ||
        (e = cudaMalloc(&h->d_status, sizeof(Status))) != cudaSuccess ||
        (e = pinned_take(sizeof(Status), reinterpret_cast<void**>(&h->h_status))) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&h->done, cudaEventDisableTiming)) != cudaSuccess) {
        pldt5_free(h);
        return cuda_fail(e, "pldt5_open");
    }
    if ((e = cudaMemset(h->d_blob, 0, blob)) != cudaSuccess ||
        (len && (e = cudaMemcpy(h->d_blob, data, len, cudaMemcpyHostToDevice)) != cudaSuccess) ||
        (e = cudaMemcpy(h->d_meta, meta.data(), 4 * meta.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (nb && (e = cudaMemcpy(h->d_rows, rows0.data(), 24 * nb, cudaMemcpyHostToDevice)) != cudaSuccess)) {
        pldt5_free(h);
        return cuda_fail(e, "pldt5_open upload");
    }
    *out = h;
    return STRIDE_OK;
}

int pldt5_inspect(const uint8_t* data, size_t len, pldt5_info_t* info) {
    if (!info || (!data && len)) return fail(STRIDE_ERR_ARG, "null argument");
    P5Host H;
    const int rc = p5_host_parse(data, len, H);
    if (rc) return rc;
    *info = H.info;
    return STRIDE_OK;
}

int pldt5_info(const pldt5_handle* h, pldt5_info_t* info) {
    if (!h || !info) return fail(STRIDE_ERR_ARG, "null argument");
    *info = h->info;
    return STRIDE_OK;
}

int pldt5_meshlets_per_cta(const pldt5_handle* h) { return h ? static_cast<int>(h->team) : 0; }

int pldt5_decode(pldt5_handle* h, void* stream, uint32_t* d_idx, float* d_pos) {
    if (!h || (!d_idx && h->info.n_t) || (!d_pos && h->info.n_v)) return fail(STRIDE_ERR_ARG, "null argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint64_t M = h->info.n_meshlets, nb = h->info.n_boundary, rows = h->info.n_v;
    cudaError_t e;
    P5Args a;
    a.blob = h->d_blob;
    a.nbits = 8ull * h->len;
    a.start = h->d_meta;
    a.row_base = h->d_meta + M + 1;
    a.tri_base = a.row_base + M;
    a.ref_base = a.tri_base + M;
    a.n_meshlets = static_cast<uint32_t>(M);
    a.n_boundary = static_cast<uint32_t>(nb);
    a.rows = h->d_rows;
    a.refs = h->d_refs;
    a.walk = h->d_walk;
    a.idx = d_idx;
    a.pos = d_pos;
    a.w0 = h->w[0];
    a.w1 = h->w[1];
    a.w2 = h->w[2];
    a.delta = h->delta;
    a.scale = h->scale;
    for (int d = 0; d < 3; d++) a.center[d] = h->center[d];
    a.status = h->d_status;
    if ((e = cudaMemsetAsync(h->d_status, 0, sizeof(Status), s)) != cudaSuccess) return cuda_fail(e, "pldt5_decode");
    if (h->team) {
        e = h->team == 8 ? p5_team_launch<8>(a, h->team_smem, s) : p5_team_launch<16>(a, h->team_smem, s);
        if (e != cudaSuccess) return cuda_fail(e, "p5_team_kernel");
    } else {
        if (rows > nb && (e = cudaMemsetAsync(h->d_rows + 3 * nb, 0, 24 * (rows - nb), s)) != cudaSuccess)
            return cuda_fail(e, "pldt5_decode");
        if (M) {
            // one lane per meshlet (kP5Threads per block)
            p5_decode_kernel<<<static_cast<uint32_t>((M + kP5Threads - 1) / kP5Threads), kP5Threads, 0, s>>>(a);
            if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "p5_decode_kernel");
        }
        if (rows) {
            p5_world_kernel<<<static_cast<uint32_t>((3 * rows + 255) / 256), 256, 0, s>>>(a, rows);
            if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "p5_world_kernel");
        }
    }
    if ((e = cudaMemcpyAsync(h->h_status, h->d_status, sizeof(Status), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaEventRecord(h->done, s)) != cudaSuccess)
        return cuda_fail(e, "pldt5_decode");
    h->launched = true;
    return STRIDE_OK;
}

int pldt5_status(pldt5_handle* h, int wait) {
    if (!h) return fail(STRIDE_ERR_ARG, "null handle");
    if (!h->launched) return STRIDE_OK;
    cudaError_t e = wait ? cudaEventSynchronize(h->done) : cudaEventQuery(h->done);
    if (e == cudaErrorNotReady) return STRIDE_ERR_BUSY;
    if (e != cudaSuccess) return cuda_fail(e, "pldt5_status");
    uint32_t bad = 0;
    const int rc = status_to_code(*h->h_status, &bad);
    if (rc) return fail(rc, "%s (meshlet %u)", status_message(rc), bad);
    return STRIDE_OK;
}

void pldt5_close(pldt5_handle* h) {
    if (!h) return;
    if (h->launched) cudaEventSynchronize(h->done);
    pldt5_free(h);
}

}  // extern "C"

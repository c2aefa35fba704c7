// Team kernel (launch shape 4): a CTA of ten warps decodes M consecutive
// meshlets (M = 4, 8 or 16) from their bytes to positions, in shared memory.
//
// What bounds a decode is the length of one meshlet's serial chains: token
// widths depend on flag bits, the FIFO on every earlier token, codewords on
// the ones before them, IRLP on earlier codes.  The team keeps on those
// chains only what is serial, one lane per meshlet, and spreads the rest over
// whole warps:
//
//  1. stage    a warp per meshlet: its bytes into shared memory, in bit order.
//  2. parse    a warp, lane per meshlet: token boundaries.  Six tokens of
//              seven are raw, so a step takes up to three raw tokens and the
//              FIFO token after them.
//     FIFO     a warp, lane per meshlet, a chunk of steps behind: the
//              move-to-front FIFO, once per step; ids of the FIFO tokens.
//     assemble eight warps, a warp per meshlet, a chunk behind the FIFO: steps
//              to token records (lane per step), then windows of 32 tokens
//              (lane per token): strip state by ballots (a strip-body
//              triangle is the previous two ids and the id two before the
//              last edge-code-0 token), triangles, first occurrences, walk.
//  3. walk     lane per (meshlet, axis): a decoder warp finds the substreams
//              and reads residuals, a predictor warp behind it runs IRLP.
//              The other warps meanwhile put out the triangles.
//  4. emit     a warp per meshlet, lane per vertex: exact positions.
//
// Loops that carry a chain are unrolled, free of branches and of the same
// length in every lane where they can be: a taken branch costs a lone warp
// about 20 cycles, a diverged one twice that.  Groups are independent: no
// work queue, no waits between CTAs; several CTAs per SM overlap one
// another's phases.
//
// The scan (output placement, tables, the offset table's checks) runs beside
// the first half: connectivity needs only the stream, so the kernel is
// launched as the scan's programmatic dependent, reads the meshlet headers
// itself and waits for the scan before it writes anything.
#include <cuda_runtime.h>

#include <algorithm>

#include "stride_common.cuh"
#include "stride_device.cuh"
#include "stride_gb300.h"
#include "stride_team.cuh"

namespace stride {
namespace {

constexpr uint32_t kTeamThreads = 32u * (kTeamAsm + 2u);
constexpr uint32_t kTeamRes = 16u;    // residuals between hand-overs from decoder to predictor warps

// Shared memory of a round: staged bytes, walks, then the token records and
// each id's last token, whose place the code planes take when the walk starts,
// then the triangles.  Laid out by what the round's meshlets need.
__host__ __device__ inline uint32_t team_bytes(uint32_t bits, uint32_t walk, uint32_t tok, uint32_t last,
                                               uint32_t plane, uint32_t tri) {
    const uint32_t uni = tok + last > plane ? tok + last : plane;
    const uint32_t rest = 4u * (walk + uni + tri);
    return bits + (rest > kTeamSlack ? rest : kTeamSlack);
}
// A meshlet's words in each.
__host__ __device__ inline uint32_t team_walk_words(uint32_t n_local) {  // entries, then the vertex list
    return (n_local + ((n_local + 3u) >> 2)) | 1u;
}
__host__ __device__ inline uint32_t team_axis_words(uint32_t n_local, uint32_t code_size) {
    return ((n_local * code_size + 3u) >> 2) | 1u;
}

// Decoder warps for M meshlets (a lane per meshlet and axis), each with a
// predictor warp behind it.
template <uint32_t M>
__host__ __device__ constexpr uint32_t team_dec_warps() {
    return (3u * M + 31u) / 32u;
}

// Barriers of two warps; ids are immediates (see pair_bar).
template <int kId>
__device__ __forceinline__ void team_bar() {
    asm volatile("bar.sync %0, 64;" ::"n"(kId) : "memory");
}
__device__ __forceinline__ void team_dec_bar(uint32_t k) {  // warp-uniform
    if (k == 0u) {
        team_bar<1>();
    } else if (k == 1u) {
        team_bar<2>();
    } else {
        team_bar<3>();
    }
}

// A round's meshlet as every warp sees it, in shared memory.
struct TeamFacts : TeamSize {
    MeshParams P;
    unsigned long long src16;           // arena offset of its bytes (16-byte aligned)
    unsigned long long v_base, t_base;  // its first output rows (from the scan)
    uint32_t placed;                    // ... which lie inside its mesh's
    uint32_t m;                         // meshlet, or none when not in the round
    uint32_t mi;                        // its mesh
    uint32_t n_strips;
    uint32_t start_bit, end_bit, ssz;   // ssz: bytes staged
    uint32_t bit_off, walk_off, tok_off, last_off, plane_off, tri_off;  // bytes, then words
    uint32_t axis_words;                // one axis' code plane
    // found on the way
    uint32_t anchor;                    // the stream bit after the connectivity
    uint32_t walk;                      // n_kind0 | n_walk << 16
    uint32_t tcnt;                      // triangles
    uint32_t bad;                       // invalid connectivity: reported, the later phases skip it
    uint32_t wbad;                      // invalid walk
    uint32_t slow[3];                   // the axis is decoded by team_walk_slow
};

// A lane's 96 bits at bit `pos` of the words at shared address `base`.
__device__ __forceinline__ void team_window96(uint32_t base, uint32_t pos, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint32_t a = mad_u32(pos >> 5, 4u, base), o = pos & 31u;
    uint32_t w0, w1, w2, w3;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w0) : "r"(a));
    asm volatile("ld.shared.u32 %0, [%1+4];" : "=r"(w1) : "r"(a));
    asm volatile("ld.shared.u32 %0, [%1+8];" : "=r"(w2) : "r"(a));
    asm volatile("ld.shared.u32 %0, [%1+12];" : "=r"(w3) : "r"(a));
    hi = __funnelshift_l(w1, w0, o);
    mid = __funnelshift_l(w2, w1, o);
    lo = __funnelshift_l(w3, w2, o);
}

// Four codewords from bit `pos`, the first n of them, as zigzag values; true
// when one is longer than 32 bits or starts beyond the window (the caller then
// takes them again by the general reader).  A window read once for four leaves
// the leading zeros, a multiply-add and a funnel shift between one codeword and
// the next: 73 cycles a residual on one warp, with its store, against 87 with a
// window refilled at each codeword.
struct TeamCode {
    uint32_t em, k1, zmul, pow;  // a codeword of z leading zeros has z * em + k1 bits
    __device__ __forceinline__ explicit TeamCode(uint32_t tk) {
        const uint32_t k = tk & 0x3Fu;
        const bool eg = (tk & 0x80u) != 0u;
        em = eg ? 2u : 1u;
        k1 = k + 1u;
        pow = 1u << k;
        zmul = eg ? 0u : pow;
    }
};
__device__ __forceinline__ bool team_four(uint32_t base, uint32_t& pos, const TeamCode& C, int n, uint32_t* u) {
    uint32_t hi, mid, lo;
    team_window96(base, pos, hi, mid, lo);
    uint32_t used = 0u, longest = 0u, before = 0u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t z = __clz(hi), len = mad_u32(z, C.em, C.k1);
        // the value bits with the terminator as their leading one: 2^nb + value
        u[i] = mad_u32(z, C.zmul, __funnelshift_rc(hi, 0u, 32u - len) - C.pow);
        const uint32_t take = i < n ? len : 0u;
        longest = max(longest, take);
        before = used;
        used += take;
        hi = __funnelshift_lc(mid, hi, take);
        mid = __funnelshift_lc(lo, mid, take);
        lo = __funnelshift_lc(0u, lo, take);
    }
    pos += used;
    return (longest > 32u) | (before > 64u);
}

// Skip n codewords of one substream from bit `pos` of w (their lengths are
// not stored), n its own in every lane of the warp (0: none).  Unary
// (Rice(0)) codewords end at a one bit each: when every lane's are, whole
// windows by their count of one bits, then the last word by halving.  Others
// eight at a time; a lane that met one longer than the window takes its eight
// again by the general reader.  False for a malformed one.
__device__ __forceinline__ bool team_skip(const uint32_t* __restrict__ w, uint32_t& pos, uint32_t tk, uint32_t n,
                                          uint32_t limit) {
    const uint32_t most = __reduce_max_sync(kFull, n);
    if (most == 0u) return true;
    const uint32_t base = smem_addr(w);
    bool ok = true;
    if (__all_sync(kFull, tk == 0u || n == 0u)) {
        uint32_t hi, mid, lo, c0, c1, c2;  // one bits up to each word's end
        for (;;) {
            team_window96(base, pos, hi, mid, lo);
            c0 = __popc(hi);
            c1 = c0 + __popc(mid);
            c2 = c1 + __popc(lo);
            if (c2 >= n) break;
            pos += 96u;
            n -= c2;
            if (pos > limit) break;  // only a corrupt stream runs past its meshlet
        }
        __syncwarp();
        uint32_t y = n > c1 ? lo : (n > c0 ? mid : hi), need = n - (n > c1 ? c1 : (n > c0 ? c0 : 0u));
        uint32_t at = n > c1 ? 64u : (n > c0 ? 32u : 0u);
#pragma unroll
        for (uint32_t wd = 16u; wd >= 1u; wd >>= 1) {
            const uint32_t t = __popc(y >> (32u - wd));  // ones in the top wd bits
            const bool more = t < need;
            need -= more ? t : 0u;
            y = more ? (y << wd) : y;
            at += more ? wd : 0u;
        }
        pos += n ? at + 1u : 0u;
    } else {
        const TeamCode C(tk);
        for (uint32_t i0 = 0; i0 < most; i0 += 8u) {
            const int left = static_cast<int>(n) - static_cast<int>(i0);
            uint32_t from = pos, u[4];
            bool far = team_four(base, pos, C, left, u);
            far = team_four(base, pos, C, left - 4, u) | far;
            if (far) {
                const int m = min(8, left);
                int32_t r;
                for (int i = 0; i < m; i++) ok = residual<true>(w, 0u, from, tk, limit, r) & ok;
                pos = from;
            }
            ok = ok & (pos <= limit);
            pos = min(pos, limit);
            __syncwarp();
        }
    }
    return ok & (pos <= limit);
}

// One (meshlet, axis) of the residual decoder: a lane of a decoder warp.
struct TeamAxis {
    uint32_t pos0;         // the first substream's bit, after the (tag, k) pairs
    uint32_t cp, cdd;      // parallelogram and delta cursors (bits of w)
    uint32_t tp, td;       // their (tag, k)
    uint32_t tk[6];
    uint32_t n_para, n_delta;
    int32_t anc;
    bool bad, slow;
};

// Anchor codes and (tag, k) pairs (paradelta_v5_dup.py:544-557); `act`: the
// lane has a meshlet.
template <bool kShared>
__device__ __forceinline__ void team_axis_open(TeamAxis& X, const MeshParams* __restrict__ P, uint32_t d, bool act,
                                               uint32_t anchor_bit, uint32_t end, uint32_t wk,
                                               const uint32_t* __restrict__ w, uint32_t rbase) {
    uint32_t pos = anchor_bit + rbase;
    X.bad = !act;
    X.slow = !kShared;
    X.anc = 0;
#pragma unroll
    for (int i = 0; i < 6; i++) X.tk[i] = 0u;
    if (act) {
#pragma unroll
        for (uint32_t e = 0; e < 3u; e++) {
            const uint32_t gb = P->g_bits[e];
            const int32_t v = gb ? static_cast<int32_t>(peek32<kShared>(w, pos) >> (32u - gb)) : 0;
            X.anc = e == d ? v : X.anc;
            pos += gb;
        }
#pragma unroll
        for (int i = 0; i < 6; i++) {
            const uint32_t t = peek32<kShared>(w, pos) >> 16;
            pos += 16u;
            const uint32_t k = t & 0xFFu;
            X.bad = X.bad || k > static_cast<uint32_t>(kMaxResidK);
            X.tk[i] = ((t >> 8) == 1u ? 0u : 0x80u) | (k & 0x3Fu);
        }
        X.bad = X.bad || pos > end + rbase;
    }
    const uint32_t n_kind0 = wk & 0xFFFFu;
    X.n_delta = n_kind0 ? n_kind0 - 1u : 0u;  // the anchor has no delta
    X.n_para = (wk >> 16) - n_kind0;
    X.pos0 = X.cp = X.cdd = pos;
    X.td = d == 0u ? X.tk[0] : (d == 1u ? X.tk[1] : X.tk[2]);
    X.tp = d == 0u ? X.tk[3] : (d == 1u ? X.tk[4] : X.tk[5]);
}

// kN codewords (8 or 16) of a substream as residuals into the code plane at
// their vertices, the first n of the kN bytes at `list`.  A lane that met one
// longer than the window takes all of them again by the general reader.  A
// residual that does not fit the plane sets `slow`; false for a malformed
// codeword.  kDown: the list runs backwards; store false: only skipped.
template <uint32_t kN, bool kWide, bool kDown>
__device__ __forceinline__ bool team_decode(const uint32_t* __restrict__ w, uint32_t& pos, uint32_t tk, uint32_t limit,
                                            const uint8_t* __restrict__ list, int n, bool store, uint32_t plane,
                                            bool& slow) {
    constexpr uint32_t kSize = sizeof(PlaneT<kWide>);
    const TeamCode C(tk);
    const uint32_t base = smem_addr(w);
    uint32_t l[kN / 4u];
    if constexpr (!kDown) {
#pragma unroll
        for (uint32_t q = 0; q < kN / 4u; q++) l[q] = reinterpret_cast<const uint32_t*>(list)[q];
    }
    uint32_t from = pos, big = 0u;
    bool far = false;
    auto put = [&](int i, uint32_t u, bool on) {
        uint32_t v;
        if constexpr (kDown) {
            v = on ? list[-i] : 0u;
        } else {
            v = __byte_perm(l[i / 4], 0u, 0x4440u | (i & 3));
        }
        const uint32_t at = mad_u32(v, kSize, plane), act = static_cast<uint32_t>(on);
        const int32_t r = unzigzag(u);
        if constexpr (kWide) {
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.u32 [%0], %1;\n}" ::"r"(at), "r"(r), "r"(act)
                         : "memory");
        } else {
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.u16 [%0], %1;\n}" ::"r"(at),
                         "h"(static_cast<short>(r)), "r"(act)
                         : "memory");
            big |= on ? u : 0u;
        }
    };
#pragma unroll
    for (int h = 0; h < static_cast<int>(kN); h += 4) {
        uint32_t u[4];
        far = team_four(base, pos, C, n - h, u) | far;
#pragma unroll
        for (int i = 0; i < 4; i++) put(h + i, u[i], store & (h + i < n));
    }
    bool ok = true;
    if (far) {  // (what was put is put again)
        big = 0u;
        for (int i = 0; i < min(static_cast<int>(kN), n); i++) {
            int32_t r;
            ok = residual<true>(w, 0u, from, tk, limit, r) & ok;
            const uint32_t u = (static_cast<uint32_t>(r) << 1) ^ static_cast<uint32_t>(r >> 31);
            if (store) {
                const uint32_t v = kDown ? list[-i] : list[i];
                reinterpret_cast<PlaneT<kWide>*>(__cvta_shared_to_generic(plane))[v] = static_cast<PlaneT<kWide>>(r);
                big |= u;
            }
        }
        pos = from;
    }
    slow = slow | (!kWide && big > 0xFFFFu);  // outside 16 bits
    ok = ok & (pos <= limit);
    pos = min(pos, limit);
    return ok;
}

// IRLP of walk entries [h, h + 8) below n_walk (paradelta_v5_dup.py:91-104,
// 581-600): a vertex's residual is in its place of the code plane.  The
// plane's addresses are formed for all eight entries first, with multiply-adds
// (the integer ALU, which issues every other cycle, has the byte extractions),
// so that only loads, arithmetic and the store are between one code and the
// next, and an entry's codes are loaded before the one before it is stored and
// taken from its register where they are that one: 59 cycles an entry on one
// warp, 86 through shared memory, 143 with the addresses where they are used.
template <bool kWide>
__device__ __forceinline__ void team_predict(uint32_t plane, const uint32_t* __restrict__ walk, uint32_t h,
                                             uint32_t n_walk, int32_t n0, int32_t n1, int32_t n2, int32_t K,
                                             int32_t half, int32_t& prev, uint32_t& codes) {
    constexpr uint32_t kSize = sizeof(PlaneT<kWide>);
    uint32_t av[8], aa[8], ab[8], ac[8];
    bool para[8];
#pragma unroll
    for (uint32_t i = 0; i < 8u; i++) {
        const uint32_t e = h + i < n_walk ? walk[h + i] : 0u;
        av[i] = mad_u32(__byte_perm(e, 0u, 0x4440u), kSize, plane);
        aa[i] = mad_u32(__byte_perm(e, 0u, 0x4441u), kSize, plane);
        ab[i] = mad_u32(__byte_perm(e, 0u, 0x4442u), kSize, plane);
        ac[i] = mad_u32(e >> 24, kSize, plane);
        para[i] = av[i] != aa[i];  // roots are stored as (v, v, v, v)
    }
    auto ld = [](uint32_t at) -> int32_t {  // a code
        int32_t c;
        if constexpr (kWide) {
            asm volatile("ld.shared.s32 %0, [%1];" : "=r"(c) : "r"(at) : "memory");
        } else {
            asm volatile("ld.shared.u16 %0, [%1];" : "=r"(c) : "r"(at) : "memory");
        }
        return c;
    };
    int32_t r[8];
#pragma unroll
    for (uint32_t i = 0; i < 8u; i++) {
        if constexpr (kWide) {
            asm volatile("ld.shared.s32 %0, [%1];" : "=r"(r[i]) : "r"(av[i]) : "memory");
        } else {
            asm volatile("ld.shared.s16 %0, [%1];" : "=r"(r[i]) : "r"(av[i]) : "memory");
            if (i == 0u) r[i] = h == 0u ? r[i] & 0xFFFF : r[i];  // the first entry is the anchor, a code
        }
    }
    int32_t ca = ld(aa[0]), cb = ld(ab[0]), cc = ld(ac[0]);
#pragma unroll
    for (uint32_t i = 0; i < 8u; i++) {
        const uint32_t act = static_cast<uint32_t>(h + i < n_walk);
        int32_t na = 0, nb = 0, nc = 0;
        if (i < 7u) {
            na = ld(aa[i + 1u]);
            nb = ld(ab[i + 1u]);
            nc = ld(ac[i + 1u]);
        }
        const int32_t code = (para[i] ? (n0 * ca + n1 * cb + n2 * cc + half) >> K : prev) + r[i];
        if constexpr (kWide) {
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.u32 [%0], %1;\n}" ::"r"(av[i]), "r"(code),
                         "r"(act)
                         : "memory");
        } else {
            asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.u16 [%0], %1;\n}" ::"r"(av[i]),
                         "h"(static_cast<short>(code)), "r"(act)
                         : "memory");
        }
        codes |= act ? static_cast<uint32_t>(code) : 0u;
        prev = code;
        if (i < 7u) {
            const int32_t kept = kWide ? code : code & 0xFFFF;  // as the plane keeps it
            ca = aa[i + 1u] == av[i] ? kept : na;
            cb = ab[i + 1u] == av[i] ? kept : nb;
            cc = ac[i + 1u] == av[i] ? kept : nc;
        }
    }
}

// The whole axis by the general reader, one lane: substream starts,
// residuals and IRLP together.  For residuals wider than the plane and
// meshlets read in place.
template <bool kShared, bool kWide>
__device__ __noinline__ bool team_walk_slow(TeamAxis& X, const MeshParams* P, uint32_t d, const uint32_t* w,
                                            uint32_t limit, const uint32_t* walk, uint32_t n_walk,
                                            PlaneT<kWide>* plane) {
    uint32_t pos = X.pos0;
    X.cdd = pos;
    for (uint32_t e = 0; e < 3u + d; e++) {
        if (e == d && e < 3u) X.cdd = pos;
        if (!skip_codes<kShared>(w, 0u, pos, X.tk[e], e < 3u ? X.n_delta : X.n_para, limit)) return false;
    }
    X.cp = pos;
    uint32_t cp = pos, cdd = X.cdd;
    const int32_t n0 = P->pred_n[3 * d], n1 = P->pred_n[3 * d + 1], n2 = P->pred_n[3 * d + 2];
    const int32_t K = P->pred_k[d], half = P->pred_half[d];
    const uint32_t cmax = P->code_max[d];
    int32_t prev = X.anc;
    bool ok = true;
    for (uint32_t i = 0; i < n_walk; i++) {
        const uint32_t e = walk[i], v = e & 0xFFu, ra = (e >> 8) & 0xFFu;
        const bool para = ra != v;
        int32_t code = prev;  // the anchor's
        if (i) {
            int32_t r;
            uint32_t p = para ? cp : cdd;
            ok = residual<kShared>(w, 0u, p, para ? X.tp : X.td, limit, r) & ok;
            cp = para ? p : cp;
            cdd = para ? cdd : p;
            const int32_t ca = static_cast<int32_t>(plane[ra]), cb = static_cast<int32_t>(plane[(e >> 16) & 0xFFu]),
                          cc = static_cast<int32_t>(plane[e >> 24]);
            code = (para ? (n0 * ca + n1 * cb + n2 * cc + half) >> K : prev) + r;
        }
        ok = ok & (static_cast<uint32_t>(code) <= cmax);
        plane[v] = static_cast<PlaneT<kWide>>(code);
        prev = code;
    }
    X.pos0 = cp;  // where the axis' parallelogram codewords end
    return ok;
}

// Positions (and codes) of one meshlet: lane per vertex.
template <bool kWide>
__device__ __forceinline__ void team_emit(const DecodeArgs& a, const MeshParams* __restrict__ P, uint32_t nv,
                                          unsigned long long vb, const PlaneT<kWide>* __restrict__ plane,
                                          uint32_t stride, int lane) {
    float* __restrict__ dst = a.pos + 3ull * vb;
    if (P->has_lut) {
        const uint32_t g0 = P->g_bits[0], g1 = P->g_bits[1];
        const float* __restrict__ l0 = a.lut + P->lut_off;
        const float* __restrict__ l1 = l0 + (1u << g0);
        const float* __restrict__ l2 = l1 + (1u << g1);
        // codes lie inside the tables: an invalid meshlet is not written
#pragma unroll 4
        for (uint32_t v = lane; v < nv; v += 32u) {
            const float x = __ldcg(l0 + plane[v]), y = __ldcg(l1 + plane[v + stride]),
                        z = __ldcg(l2 + plane[v + 2u * stride]);
            dst[3u * v] = x;
            dst[3u * v + 1u] = y;
            dst[3u * v + 2u] = z;
        }
    } else {
#pragma unroll
        for (uint32_t d = 0; d < 3u; d++) {
            stride_dequant_axis c;
            c.a_hi = P->dq[d].a_hi;
            c.a_lo = P->dq[d].a_lo;
            c.b_hi = P->dq[d].b_hi;
            c.b_lo = P->dq[d].b_lo;
            c.err = P->dq[d].err;
            const bool zero_bits = P->dq[d].zero_bits != 0;
            for (uint32_t v = lane; v < nv; v += 32u) {
                const uint32_t q = static_cast<uint32_t>(plane[v + d * stride]);
                float y;
                const bool fast = stride_dequant_fast(&c, q, &y) != 0;
                if (!fast || zero_bits) y = dequant_slow(P, d, q);
                dst[3u * v + d] = y;
            }
        }
    }
    if (a.codes) {
        int32_t* cd = a.codes + 3ull * vb;
        for (uint32_t v = lane; v < nv; v += 32u) {
            cd[3u * v] = static_cast<int32_t>(plane[v]);
            cd[3u * v + 1u] = static_cast<int32_t>(plane[v + stride]);
            cd[3u * v + 2u] = static_cast<int32_t>(plane[v + 2u * stride]);
        }
    }
}

template <uint32_t M>
struct TeamShared {
    uint4 masks[17];
    TeamFacts f[M];
    // parser steps of three chunks (being written; with the FIFO; with the assemblers)
    uint32_t x[3][kTeamSteps * M];
    uint32_t step[3][kTeamSteps * M];
    uint8_t meta[3][kTeamSteps * M];
    uint32_t more[2];  // the parser has tokens left after its last chunk
    uint32_t rmask;   // meshlets of the round
    uint32_t walk_base, uni_base;  // bytes
    uint32_t staged;
    uint32_t redo;    // decode the connectivity again, with the exact FIFO
};

// The meshlets of a round from their bytes to positions.
template <uint32_t M, bool kShared, bool kWide>
__device__ __forceinline__ void team_round(const DecodeArgs& a, TeamShared<M>& s, uint8_t* bits, uint32_t warp,
                                           int lane) {
    const uint32_t rmask = s.rmask;
    uint32_t* walks = reinterpret_cast<uint32_t*>(bits + s.walk_base);
    uint32_t* uni = reinterpret_cast<uint32_t*>(bits + s.uni_base);
    constexpr uint32_t kPer = (M + kTeamAsm - 1u) / kTeamAsm;  // meshlets of an assembler warp
    const bool assembler = warp != kTeamParser && warp != kTeamFifo;
    const uint32_t aw0 = team_asm_index(warp);  // an assembler's first meshlet
    const uint32_t* bit_words = reinterpret_cast<const uint32_t*>(bits);
    // 1. stage; the mesh records' loads on their way beside the bytes' (a trip to
    // L2 less per meshlet of a warp: sixteen to a CTA, 55 -> 53 and 96 -> 94 us for
    // 4,090 and 7,503 meshlets)
    if (assembler) {
        constexpr uint32_t kWords = sizeof(MeshParams) / 4u, kP = (kWords + 31u) / 32u;
        uint32_t pv[kPer][kP];
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            const uint32_t j = aw0 + q * kTeamAsm;
            const bool in = j < M && ((rmask >> (j & 31u)) & 1u);  // warp-uniform
            const uint32_t* ps = reinterpret_cast<const uint32_t*>(a.meshes + (in ? s.f[j].mi : 0u));
#pragma unroll
            for (uint32_t r = 0; r < kP; r++) pv[q][r] = __ldcg(ps + min(lane + 32u * r, kWords - 1u));
        }
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            const uint32_t j = aw0 + q * kTeamAsm;
            if (j >= M || !((rmask >> j) & 1u)) continue;
            TeamFacts& F = s.f[j];
            if constexpr (kShared) {
                const uint32_t n16 = F.ssz >> 4;
                const uint4* src = reinterpret_cast<const uint4*>(a.arena + F.src16);
                uint4* dst = reinterpret_cast<uint4*>(bits + F.bit_off);
                for (uint32_t i = lane; i < n16; i += 32u) {
                    uint4 v = __ldcg(src + i);
                    v.x = bswap32(v.x);
                    v.y = bswap32(v.y);
                    v.z = bswap32(v.z);
                    v.w = bswap32(v.w);
                    dst[i] = v;
                }
            }
            uint32_t* pd = reinterpret_cast<uint32_t*>(&F.P);
#pragma unroll
            for (uint32_t r = 0; r < kP; r++)
                if (lane + 32u * r < kWords) pd[lane + 32u * r] = pv[q][r];
        }
    }
    // bit p of the stream is bit p + rbase of w
    auto base_of = [&](const TeamFacts& F, const uint32_t*& w) -> uint32_t {
        w = kShared ? bit_words : reinterpret_cast<const uint32_t*>(a.arena + F.P.blob_off);
        return kShared ? static_cast<uint32_t>((F.P.blob_off - F.src16 + F.bit_off) * 8ull) : 0u;
    };
    // Output rows of a meshlet, once the scan has ended: inside its mesh's (header n_v_total, n_t), and the last meshlet's end exactly there
    // (see placement_ok).
    auto place = [&](TeamFacts& F) {
        if (lane == 0) {
            const MeshletDesc* D = a.descs + F.m;
            const BlockPrefix* bp = a.blk_prefix + F.m / kScanThreads;
            const bool failed = *reinterpret_cast<volatile unsigned long long*>(&a.status->err) != 0ull;
            F.v_base = __ldcg(&bp->v) + __ldcg(&D->v_pref);
            F.t_base = __ldcg(&bp->t) + __ldcg(&D->t_pref);
            const unsigned long long v0 = F.P.v_offset, v1 = v0 + F.P.n_v, t0 = F.P.t_offset, t1 = t0 + F.P.n_t;
            const unsigned long long ve = F.v_base + F.n_local, te = F.t_base + F.n_tris;
            bool ok = F.v_base >= v0 && ve <= v1 && F.t_base >= t0 && te <= t1;
            if (ok && F.m - F.P.meshlet_begin + 1u == F.P.n_meshlets) ok = ve == v1 && te == t1;
            F.placed = ok && !failed ? 1u : 0u;
        }
        __syncwarp();
    };
    for (uint32_t pass = 0; pass < 2u; pass++) {  // the second one with the exact FIFO, rarely
        const bool exact = pass != 0u;
        if (threadIdx.x == 0) s.redo = 0u;
        if (threadIdx.x < M) {
            TeamFacts& F = s.f[threadIdx.x];
            F.bad = F.wbad = F.slow[0] = F.slow[1] = F.slow[2] = 0u;
        }
        __syncthreads();
        // 2. connectivity, in step: chunk c with the parser, c - 1 with the
        // FIFO warp, c - 2 with the assemblers
        if (!assembler) {
            const bool act = (rmask >> lane) & 1u;
            TeamFacts& F = s.f[act ? lane : 0];
            const uint32_t* w;
            const uint32_t rbase = base_of(F, w);
            const uint32_t n_tok = act ? F.n_tok : 0u;
            const uint32_t ib = 9u - F.idsh;
            uint16_t* row = reinterpret_cast<uint16_t*>(uni + F.tok_off) + 2;
            const uint32_t sl = act ? lane : 0u;  // an idle lane repeats the first one's steps
            TeamParse T;
            MtfFifo fifo;
            uint32_t t = 0u;
            uint32_t past = 0u;  // negative: a FIFO index named no entry
            T.strips = F.n_strips;
            T.pos = act ? F.start_bit + 48u + rbase : 0u;
            fifo.f0 = fifo.f1 = fifo.f2 = fifo.f3 = 0xFFFFFFFFu;
            if (warp == kTeamParser && act) {
                row[-2] = row[-1] = 0;
            }
            bool more = true;
            for (uint32_t c = 0;; c++) {
                if (warp == kTeamParser) {
                    const uint32_t b = c % 3u;
                    if (act) team_parse<kShared, M>(T, w, n_tok, ib, F.end_bit + rbase + 1u, s.x[b] + lane, s.meta[b] + lane);
                    __syncwarp();
                    const bool m = __any_sync(kFull, T.t < n_tok);
                    if (lane == 0) s.more[c & 1u] = m ? 1u : 0u;
                } else if (c > 0u) {
                    const uint32_t b = (c - 1u) % 3u;
                    if (act) team_fifo<M>(fifo, t, s.x[b] + sl, s.meta[b] + sl, s.step[b] + sl, ib, s.masks, past);
                }
                __syncwarp();
                team_all_bar<kTeamThreads>();
                if (!more) break;  // this was the chunk after the parser's last
                more = s.more[c & 1u] != 0u;
            }
            if (act && warp == kTeamParser) {
                const uint32_t pos = T.pos - rbase;  // the stream bit after the last token
                F.anchor = pos;
                // every strip read, inside the meshlet
                if (T.t != n_tok || T.strips != 0u || T.left != 0u || pos > F.end_bit) atomicOr(&F.bad, 1u);
            }
            if (exact) team_all_bar<kTeamThreads>();  // the records are there
            if (act && warp == kTeamFifo) {
                if (exact ? !team_fifo_exact(row, n_tok, F.idsh, s.masks) : sign_mask(past) != 0u) atomicOr(&F.bad, 1u);
            }
            __syncwarp();
            if (exact) team_all_bar<kTeamThreads>();
        } else {
            TeamAsm S[kPer];
#pragma unroll
            for (uint32_t q = 0; q < kPer; q++) {
                const uint32_t j = aw0 + q * kTeamAsm;
                if (j >= M || !((rmask >> j) & 1u)) continue;
                uint4* last = reinterpret_cast<uint4*>(uni + s.f[j].last_off);
                last[lane] = last[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
            }
            __syncwarp();
            // the windows that the records fill (or end)
            auto windows = [&](TeamAsm& A, const TeamFacts& F) {
                uint32_t* walk = walks + F.walk_off;
                uint32_t* last = uni + F.last_off;
                const uint32_t have = A.t >= F.n_tok ? F.n_tok + 31u : A.t;
                for (; A.t0 + 32u <= have; A.t0 += 32u)
                    team_window<true>(A, F, 0u, exact, A.t0, reinterpret_cast<const uint16_t*>(uni + F.tok_off) + 2, walk,
                                reinterpret_cast<uint8_t*>(walk + F.n_local), last, uni + F.tri_off, lane);
            };
            auto chunk = [&](uint32_t c) {
#pragma unroll
                for (uint32_t q = 0; q < kPer; q++) {
                    const uint32_t j = aw0 + q * kTeamAsm;
                    if (j >= M || !((rmask >> j) & 1u)) continue;
                    const TeamFacts& F = s.f[j];
                    if (S[q].t >= F.n_tok) continue;
                    team_records<M>(S[q], F, exact, reinterpret_cast<uint16_t*>(uni + F.tok_off) + 2,
                                    s.x[c % 3u] + j, s.step[c % 3u] + j, lane);
                    if (!exact) windows(S[q], F);
                }
            };
            bool more = true;
            uint32_t c = 0u;
            for (;; c++) {
                if (c > 1u) chunk(c - 2u);
                team_all_bar<kTeamThreads>();
                if (!more) break;
                more = s.more[c & 1u] != 0u;
            }
            chunk(c - 1u);  // the parser's last chunk
            if (exact) {
                __syncwarp();
                team_all_bar<kTeamThreads>();
                team_all_bar<kTeamThreads>();  // the FIFO warp has resolved the records
#pragma unroll
                for (uint32_t q = 0; q < kPer; q++) {
                    const uint32_t j = aw0 + q * kTeamAsm;
                    if (j < M && ((rmask >> j) & 1u)) windows(S[q], s.f[j]);
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < kPer; q++) {
                const uint32_t j = aw0 + q * kTeamAsm;
                if (j >= M || !((rmask >> j) & 1u)) continue;
                TeamFacts& F = s.f[j];
                const bool bad = __any_sync(kFull, S[q].out) || S[q].tcnt != F.n_tris;
                if (lane == 0) {
                    F.walk = S[q].kind0 | (min(S[q].wcnt, F.n_local) << 16);
                    F.tcnt = min(S[q].tcnt, F.n_tris);
                    if (bad) atomicOr(&F.bad, 1u);
                    if (S[q].redo && !exact) s.redo = 1u;
                }
            }
        }
        __syncthreads();
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (threadIdx.x < M && ((rmask >> threadIdx.x) & 1u)) a.descs[s.f[threadIdx.x].m].anchor_bit = s.f[threadIdx.x].anchor;
        if (s.redo == 0u || exact) break;
        __syncthreads();  // everyone has read it
    }
    // 3. walk: lane (axis, meshlet) of a decoder warp and of the predictor
    // warp a chunk behind it, so that the chains of the bit cursor and of the
    // codes run side by side.  A residual waits in its vertex's own place of
    // the code plane, which nothing reads before the vertex is reached.
    constexpr uint32_t kDec = team_dec_warps<M>();
    if (warp < 2u * kDec) {
        const uint32_t k = warp % kDec;
        const uint32_t tid = 32u * k + lane;
        const uint32_t d = tid / M < 3u ? tid / M : 2u, j = tid % M;
        TeamFacts& F = s.f[j];
        const MeshParams& P = F.P;
        const bool on = tid < 3u * M && ((rmask >> j) & 1u) && F.bad == 0u;
        const uint32_t nl = on ? F.n_local : 0u;
        const uint32_t wk = on ? F.walk : 0u;
        const uint32_t n_walk = wk >> 16;
        // (a lane without a meshlet reads the front of each array)
        const uint32_t* __restrict__ walk = walks + (on ? F.walk_off : 0u);
        const uint8_t* __restrict__ vlist = reinterpret_cast<const uint8_t*>(walk + nl);
        PlaneT<kWide>* __restrict__ plane = reinterpret_cast<PlaneT<kWide>*>(uni + (on ? F.plane_off + d * F.axis_words : 0u));
        const uint32_t chunks = (__reduce_max_sync(kFull, n_walk) + kTeamRes - 1u) / kTeamRes;
        const bool decoder = warp < kDec;
        if (!decoder && n_walk < nl && on) {  // vertices the walk never reaches keep code 0
            uint32_t* z = reinterpret_cast<uint32_t*>(plane);
            const uint32_t nz = (nl * static_cast<uint32_t>(sizeof(PlaneT<kWide>)) + 3u) >> 2;
            for (uint32_t i = 0; i < nz; i++) z[i] = 0u;
        }
        __syncwarp();
        team_dec_bar(k);
        if (decoder) {
            const uint32_t* w;
            const uint32_t rbase = base_of(F, w);
            const uint32_t limit = on ? F.end_bit + rbase : 0u;
            TeamAxis X;
            team_axis_open<kShared>(X, &P, d, on, F.anchor, F.end_bit, wk, w, rbase);
            uint32_t pos = 0u;
            const uint32_t plane_addr = smem_addr(plane);
            bool run = kShared && !X.bad;
            if constexpr (kShared) {
                // dx dy dz, the lane's own one into its roots' places; then the
                // parallelogram substreams before its own
                const uint32_t nd = run ? X.n_delta : 0u;
                const uint32_t most = __reduce_max_sync(kFull, nd);
                pos = run ? X.pos0 : 0u;
#pragma unroll
                for (uint32_t e = 0; e < 3u; e++) {
                    X.cdd = e == d ? pos : X.cdd;
#pragma unroll 1
                    for (uint32_t i = 0; i < most; i += 8u) {
                        run = team_decode<8u, kWide, true>(w, pos, X.tk[e], limit, vlist + nl - 2u - i,
                                                       run ? static_cast<int>(nd) - static_cast<int>(i) : 0, e == d,
                                                       plane_addr, X.slow) & run;
                        __syncwarp();
                    }
                }
#pragma unroll
                for (uint32_t e = 0; e < 2u; e++) {
                    run = team_skip(w, pos, X.tk[3 + e], run && e < d ? X.n_para : 0u, limit) & run;
                    __syncwarp();
                }
                X.cp = pos;
                run = run && n_walk;
                if (run) plane[vlist[nl - 1u]] = static_cast<PlaneT<kWide>>(X.anc);  // the first root is the anchor
                X.bad = X.bad || (n_walk && !run);
                pos = run ? X.cp : 0u;
            }
            const uint32_t np = run ? X.n_para : 0u;
            for (uint32_t c = 0; c <= chunks; c++) {
                if constexpr (kShared) {
                    if (c < chunks) {
                        const uint32_t i0 = c * kTeamRes;
                        if (!team_decode<kTeamRes, kWide, false>(w, pos, X.tp, limit, vlist + i0,
                                                                 static_cast<int>(np) - static_cast<int>(i0), true,
                                                                 plane_addr, X.slow))
                            X.bad = true;
                    }
                }
                if (c == chunks && on) F.slow[d] = X.slow ? 1u : 0u;
                __syncwarp();
                team_dec_bar(k);
            }
            uint32_t cend = run ? pos : X.cp;
            team_dec_bar(k);  // the predictor has left the planes
            if (on && X.slow) {
                TeamAxis Y = X;  // a copy: only this path keeps it in memory
                // (what the header's checks refused stays refused: the walk knows only the low bits of k)
                X.bad = X.bad || !team_walk_slow<kShared, kWide>(Y, &P, d, w, limit, walk, n_walk, plane);
                cend = Y.pos0;
                X.cp = Y.cp;
                X.cdd = Y.cdd;
            }
            if (on) {
                // pz, the last substream, must end where the next meshlet starts (:507)
                const bool last = F.m - P.meshlet_begin + 1u == P.n_meshlets;
                const bool ends = (d != 2u || last) ? cend <= limit : cend == limit;
                if (X.bad || !ends) atomicOr(&F.wbad, 1u);
                // the side table: this axis' substream starts after the anchor
                const uint32_t a0 = F.anchor + rbase;
                const uint32_t rp = min(X.cp - a0, 0xFFFFu), rd = min(X.cdd - a0, 0xFFFFu);
                uint16_t* so = a.descs[F.m].sub_offs;
                if (d != 0u) so[d - 1u] = static_cast<uint16_t>(rd);
                so[2u + d] = static_cast<uint16_t>(rp);
            }
        } else {
            const int32_t n0 = P.pred_n[3 * d], n1 = P.pred_n[3 * d + 1], n2 = P.pred_n[3 * d + 2];
            const int32_t K = P.pred_k[d], half = P.pred_half[d];
            const uint32_t cmax = P.code_max[d];
            int32_t prev = 0;
            uint32_t codes = 0u;  // every code, or-ed
            const uint32_t plane_addr = smem_addr(plane);
            for (uint32_t c = 0; c <= chunks; c++) {
                if (c > 0u) {
                    const uint32_t i0 = (c - 1u) * kTeamRes;
#pragma unroll 1
                    for (uint32_t h = i0; h < i0 + kTeamRes; h += 8u)
                        team_predict<kWide>(plane_addr, walk, h, n_walk, n0, n1, n2, K, half, prev, codes);
                }
                __syncwarp();
                team_dec_bar(k);
            }
            // codes of a valid stream lie in [0, 2^g_bits)
            if (on && (codes & ~cmax) != 0u && F.slow[d] == 0u) atomicOr(&F.wbad, 1u);
            __syncwarp();
            team_dec_bar(k);
        }
    } else {
        // beside it the other warps: the rows that the scan gave the meshlets,
        // and the triangles
        for (uint32_t j = warp - 2u * kDec; j < M; j += kTeamAsm + 2u - 2u * kDec) {
            if (!((rmask >> j) & 1u)) continue;
            TeamFacts& F = s.f[j];
            place(F);
            // triangle indices are relative to the mesh's first vertex
            const uint32_t vloc = static_cast<uint32_t>(F.v_base - F.P.v_offset);
            if (F.placed)
                team_triangles(a.idx + 3ull * F.t_base, uni + F.tri_off, static_cast<uint32_t>(F.t_base) & 3u, F.tcnt,
                               [&](uint32_t v) { return vloc + v; }, lane);
        }
    }
    __syncthreads();
    // 4. emit
    if (assembler) {
        for (uint32_t j = aw0; j < M; j += kTeamAsm) {
            const TeamFacts& F = s.f[j];
            if (!((rmask >> j) & 1u)) continue;
            if (F.bad | F.wbad | (F.placed ^ 1u)) {
                if (lane == 0) report(a.status, kErrCorrupt, F.m);
                continue;
            }
            team_emit<kWide>(a, &F.P, F.n_local, F.v_base,
                             reinterpret_cast<const PlaneT<kWide>*>(uni + F.plane_off),
                             F.axis_words * 4u / static_cast<uint32_t>(sizeof(PlaneT<kWide>)), lane);
        }
    }
    __syncthreads();  // the next round overwrites the shared memory
}

template <uint32_t M, bool kWide>
__global__ void __launch_bounds__(kTeamThreads, 2) team_kernel(DecodeArgs a, uint32_t smem_bytes) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ TeamShared<M> s;
    if (threadIdx.x < 17u)
        s.masks[threadIdx.x] = threadIdx.x < 16u ? mtf_mask_row(threadIdx.x) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    uint32_t todo = 0u, nb = 0u, nw = 0u, nt = 0u, nr = 0u, np = 0u;
    if (warp == 0u) {
        bool ok = false;
        if (static_cast<uint32_t>(lane) < M) {
            TeamFacts& F = s.f[lane];
            MeshletDesc D;
            memset(&D, 0, sizeof(D));
            F.m = blockIdx.x * M + lane;
            F.mi = 0u;
            F.ssz = 0u;
            if (F.m < a.total_meshlets) {
                F.mi = a.meshlet_mesh ? __ldcg(a.meshlet_mesh + F.m) : 0u;
                const MeshParams& P = a.meshes[F.mi];
                ok = scan_meshlet(a.arena, P, F.m - P.meshlet_begin, D) == 0;  // the scan reports an error
                const unsigned long long blob = P.blob_off;
                F.src16 = (blob + (D.start_bit >> 3)) & ~15ull;
                const unsigned long long end16 = (blob + ((D.end_bit + 7u) >> 3) + 15ull) & ~15ull;
                F.ssz = ok ? staged_bytes(F.src16, end16) : 0u;
            }
            F.n_local = ok ? D.counts0 & 0xFFFFu : 0u;
            F.n_tris = ok ? D.counts0 >> 16 : 0u;
            F.n_strips = ok ? D.n_strips : 0u;
            F.n_tok = F.n_tris + 2u * F.n_strips;
            F.start_bit = D.start_bit;
            F.end_bit = D.end_bit;
            F.idsh = 9u - max(1u, 32u - __clz(F.n_local));
            // odd strides (in words; the staged bytes in 16-byte units): lanes
            // work at about the same offsets of their meshlets at the same time
            F.axis_words = team_axis_words(F.n_local, sizeof(PlaneT<kWide>));
            nb = F.ssz + ((F.ssz & 16u) ? 0u : 16u);
            nw = team_walk_words(F.n_local);
            nt = team_tok_words(F.n_tok);
            nr = (F.n_tris + 3u) & ~3u;
            np = 3u * F.axis_words;
        }
        todo = __ballot_sync(kFull, ok);
    }
    for (;;) {  // rounds of as many meshlets as fit, in slot order (nearly always one)
        if (warp == 0u) {
            const bool in = (todo >> lane) & 1u;
            uint32_t cb = in ? nb : 0u, cw = in ? nw : 0u, ct = in ? nt : 0u, cr = in ? nr : 0u, cp = in ? np : 0u;
            const uint32_t cl = 256u * __popc(todo & ((2u << lane) - 1u));
#pragma unroll
            for (uint32_t o = 1; o < M; o <<= 1) {
                const uint32_t t0 = __shfl_up_sync(kFull, cb, o), t1 = __shfl_up_sync(kFull, cw, o);
                const uint32_t t2 = __shfl_up_sync(kFull, ct, o), t3 = __shfl_up_sync(kFull, cr, o);
                const uint32_t t4 = __shfl_up_sync(kFull, cp, o);
                if (static_cast<uint32_t>(lane) >= o) {
                    cb += t0;
                    cw += t1;
                    ct += t2;
                    cr += t3;
                    cp += t4;
                }
            }
            // (ten words: alignments)
            const bool fit = in && team_bytes(cb, cw, ct, cl, cp, cr) + 40u <= smem_bytes;
            uint32_t rmask = __ballot_sync(kFull, fit);
            const bool staged = rmask != 0u;
            // one meshlet whose bytes exceed the stage: read in place
            if (!staged && todo) rmask = 1u << (__ffs(todo) - 1);
            todo &= ~rmask;
            const int end = rmask ? 31 - __clz(rmask) : 0;  // the round's last meshlet
            const uint32_t walk_base = staged ? __shfl_sync(kFull, cb, end) : 0u;
            const uint32_t tw = staged ? __shfl_sync(kFull, cw, end) : 0u, tt = staged ? __shfl_sync(kFull, ct, end) : 0u;
            const uint32_t tp = staged ? __shfl_sync(kFull, cp, end) : 0u, tl = staged ? __shfl_sync(kFull, cl, end) : 0u;
            // the words after the walks, the records and the planes start on 16 bytes
            const uint32_t uni_base = staged ? (walk_base + 4u * tw + 15u) & ~15u : 0u;
            const uint32_t last_base = (tt + 3u) & ~3u;
            const uint32_t tri_base = max(last_base + tl, (tp + 3u) & ~3u);
            const bool mine = (rmask >> lane) & 1u;
            if (mine) {
                TeamFacts& F = s.f[lane];
                F.bit_off = staged ? cb - nb : 0u;
                F.walk_off = staged ? cw - nw : 0u;
                F.tok_off = staged ? ct - nt : 0u;
                F.last_off = staged ? last_base + cl - 256u : (nt + 3u) & ~3u;
                F.plane_off = staged ? cp - np : 0u;
                F.tri_off = staged ? tri_base + cr - nr : max(F.last_off + 256u, (np + 3u) & ~3u);
                if (!staged) {
                    s.walk_base = 0u;
                    s.uni_base = (4u * nw + 15u) & ~15u;
                }
            }
            if (lane == 0 && staged) {
                s.walk_base = walk_base;
                s.uni_base = uni_base;
            }
            if (lane == 0) {
                s.rmask = rmask;
                s.staged = staged ? 1u : 0u;
            }
        }
        __syncthreads();
        if (s.rmask == 0u) {  // CTA-uniform
            // what follows this kernel on the stream must find the scan ended
            asm volatile("griddepcontrol.wait;" ::: "memory");
            return;
        }
        if (s.staged) {
            team_round<M, true, kWide>(a, s, smem, warp, lane);
        } else {
            team_round<M, false, kWide>(a, s, smem, warp, lane);
        }
    }
}

// Dynamic shared memory of a team CTA: room for M meshlets 2/5 above the
// average of what is decoded (consecutive meshlets are about equally large);
// a group that needs more goes in rounds.  Never less than one meshlet of the
// largest size read in place.
uint32_t team_smem(const DecodeArgs& a, uint32_t m, bool wide) {
    const unsigned long long n = std::max<uint32_t>(1u, a.total_meshlets);
    auto avg = [&](unsigned long long total, unsigned long long most) {
        return static_cast<uint32_t>(std::min<unsigned long long>(total / n + 1ull, most)) * 7u / 5u;
    };
    const uint32_t size = wide ? 4u : 2u;
    const uint32_t by = (avg(a.hint_bytes, 1024u) + 63u) & ~31u;
    const uint32_t nv = std::min(avg(a.hint_v, 256u) + 4u, 256u), nt = std::min(avg(a.hint_t, 256u) + 8u, 256u);
    const uint32_t b = team_bytes(m * by, m * team_walk_words(nv), m * team_tok_words(nt + nt / 12u),
                                  m * 256u, m * 3u * team_axis_words(nv, size), m * ((nt + 3u) & ~3u)) + 48u;
    const uint32_t least = team_bytes(0u, team_walk_words(256u), team_tok_words(kTeamTokens), 256u,
                                      3u * team_axis_words(256u, size), 256u) + 48u;
    return (std::max(b, least) + 15u) & ~15u;
}

template <uint32_t M, bool kWide>
cudaError_t launch_team_m(const DecodeArgs& a, cudaStream_t s, bool after_scan) {
    static size_t configured[64] = {0};
    const uint32_t smem = team_smem(a, M, kWide);
    cudaError_t e = opt_in_smem(team_kernel<M, kWide>, smem, configured);
    if (e != cudaSuccess) return e;
    const uint32_t grid = (a.total_meshlets + M - 1u) / M;
    if (grid == 0u) return cudaSuccess;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(kTeamThreads);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = after_scan ? 1 : 0;
    e = cudaLaunchKernelEx(&lc, team_kernel<M, kWide>, a, smem);
    note_launch(smem, grid);
    return e;
}

}  // namespace

cudaError_t launch_team(const DecodeArgs& a, const LaunchCfg& cfg, cudaStream_t s, bool after_scan) {
    const bool w = a.wide_codes;
    switch (team_meshlets(cfg)) {
        case 4: return w ? launch_team_m<4, true>(a, s, after_scan) : launch_team_m<4, false>(a, s, after_scan);
        case 8: return w ? launch_team_m<8, true>(a, s, after_scan) : launch_team_m<8, false>(a, s, after_scan);
        default: return w ? launch_team_m<16, true>(a, s, after_scan) : launch_team_m<16, false>(a, s, after_scan);
    }
}

}  // namespace stride

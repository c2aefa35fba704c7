// The connectivity of meshlets by a team of warps, in shared memory: parser and
// FIFO warps (lane per meshlet) and assembler warps (warp per meshlet, lane per
// token), and their bit reader.  The two formats' decoders (stride_team.cu,
// pldt5.cu) share it: strips, tokens and the FIFO are the same in both.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "stride_device.cuh"

namespace stride {
namespace {

constexpr uint32_t kTeamAsm = 8u;  // assembler warps, beside the parser and the FIFO warp
// Warps w, w + 4 and w + 8 share one of the SM's four schedulers, whose
// integer ALU the parser and the FIFO warp keep busy by themselves: they are
// warps 2 and 3, with one assembler each beside them (and none up to M = 4),
// the other six three to a scheduler.
constexpr uint32_t kTeamParser = 2u, kTeamFifo = 3u;
__device__ __forceinline__ uint32_t team_asm_index(uint32_t warp) {  // 0 1 4 5 8 9 6 7 -> 0..7
    return warp < 2u ? warp : (warp < 6u ? warp - 2u : (warp < 8u ? warp : warp - 4u));
}
constexpr uint32_t kTeamSteps = 20u;  // parser steps between hand-overs
constexpr uint32_t kTeamTokens = 768u;  // most tokens of a meshlet: n_tris + 2 n_strips
// Token records: bits 0..8 the nine bits after the flag (a raw token's id on
// top, or a FIFO index in bits 4..8, replaced by the field of the id it
// names), bit 9 raw, bit 10 the edge code of a strip-body token, bit 11 the
// first token of a strip.
constexpr uint32_t kTokRaw = 1u << 9, kTokEdge = 1u << 10, kTokHead = 1u << 11;
// A corrupt lane's cursor runs on past its meshlet until its loop ends: at
// most 768 steps of 32 bits, or 256 codewords of 32 bits and a window.
constexpr uint32_t kTeamSlack = 5120u;

__host__ __device__ inline uint32_t team_tok_words(uint32_t n_tok) { return ((n_tok + 6u) >> 1) | 1u; }
__host__ __device__ inline uint32_t team_asm_words(uint32_t n_tris) { return 256u + ((n_tris + 3u) & ~3u); }

template <uint32_t kThreads>
__device__ __forceinline__ void team_all_bar() {  // every warp, from its own loop
    asm volatile("bar.sync 4, %0;" ::"n"(kThreads) : "memory");
}

// A parser step: what it read (32 bits from its first token's edge code or
// flag) and, for the FIFO warp and the assembler, bits 0..1 the raw tokens,
// bit 2 a FIFO token after them, bit 3 strip-body tokens (each with its edge
// code before the flag), bit 4 the strip's first tokens; the FIFO warp adds
// the FIFO token's id in bits 8..15 and the step's first token in bits
// 16..25.  A strip header is a step without tokens.
constexpr uint32_t kStepFifo = 1u << 2, kStepBody = 1u << 3, kStepHead = 1u << 4;

struct TeamParse {
    uint32_t pos;         // bit of w
    uint32_t t = 0u;      // tokens read
    uint32_t left = 0u;   // tokens left in the strip
    uint32_t roots = 0u;  // of which roots
    uint32_t strips;      // strips to read
    uint32_t head = 0u;   // kStepHead after a header
};

// All ones when x is negative.
__device__ __forceinline__ uint32_t sign_mask(uint32_t x) { return static_cast<uint32_t>(static_cast<int32_t>(x) >> 31); }

// kTeamSteps parser steps of a lane (x and meta: its slots, M apart).  A
// strip of length len takes max(len, 1) + 2 tokens, so a valid meshlet's
// strips end with its n_tris + 2 n_strips tokens; a corrupt one's cursor
// runs on until the count is reached and its strips do not come out (checked
// by the caller).  All a step may take is laid out before its flag bits are
// known (tokens at 0, L, 2 L).  Conditions are masks: what the compiler made
// branches of cost a lane that took them 40 cycles (170 cycles a step on one
// warp against 128 without any taken).
template <bool kShared, uint32_t M>
__device__ __forceinline__ void team_parse(TeamParse& T, const uint32_t* __restrict__ w, uint32_t n_tok, uint32_t ib,
                                           uint32_t limit, uint32_t* __restrict__ x_out, uint8_t* __restrict__ meta_out) {
    const uint32_t most = ib <= 8u ? 3u : 2u;  // three tokens of 1 + 1 + ib bits in a window
    const uint32_t p1 = 2u << ib;
    const uint32_t ws = kShared ? smem_addr(w) : 0u;
#pragma unroll 4
    for (uint32_t i = 0; i < kTeamSteps; i++) {
        uint32_t x;
        if constexpr (kShared) {
            x = peek_shared(ws, T.pos);
        } else {
            x = peek32<false>(w, T.pos);
        }
        const uint32_t on = sign_mask(T.t - n_tok);
        const uint32_t hdr = sign_mask(T.left - 1u);    // strip header (paradelta_v5_dup.py:519)
        const uint32_t body = sign_mask(T.roots - 1u);
        const uint32_t L = ib + 1u - body, pl = p1 + (p1 & body);  // 2^L
        const uint32_t lim = min((T.left & body) | T.roots, most);  // none for a header
        const uint32_t x0 = x * (1u - body), x1 = x0 * pl, x2 = x1 * pl;  // flags on top (shifts on the multiplier)
        const uint32_t s0 = sign_mask(x0), s1 = s0 & sign_mask(x1), s2 = s1 & sign_mask(x2);
        const uint32_t r = min(0u - (s0 + s1 + s2), lim);
        const uint32_t f = sign_mask(r - lim);  // then the next token is a FIFO token
        const uint32_t k = (r - f) & on;
        const uint32_t used = r * L + (f & (6u - body)) + (hdr & 16u);
        x_out[i * M] = x;
        meta_out[i * M] = static_cast<uint8_t>((r | (f & kStepFifo) | (body & kStepBody) | T.head) & on);
        T.pos += used & on;
        if constexpr (!kShared) T.pos = min(T.pos, limit);  // reads stay inside the stream (a staged lane's, the stage)
        const uint32_t open = hdr & on;
        const uint32_t len = max(x >> 16, 1u) + 2u;
        T.t += k;
        T.strips += open;  // minus one
        T.left = ((T.left - k) & ~open) | (len & open);
        T.roots = (T.roots - (k & ~body)) | (open & 3u);
        T.head = open & kStepHead;
    }
}

// The FIFO over kTeamSteps steps of a lane.  Raw ids are taken as new to the
// FIFO (an encoder writes an index for an id it still holds; the assembly
// checks it).
template <uint32_t M>
__device__ __forceinline__ void team_fifo(MtfFifo& fifo, uint32_t& t, const uint32_t* __restrict__ xs,
                                          const uint8_t* __restrict__ meta, uint32_t* __restrict__ out, uint32_t ib,
                                          const uint4* __restrict__ masks, uint32_t& past) {
    const uint32_t ish = 32u - ib, p1 = 2u << ib;
#pragma unroll 4
    for (uint32_t i = 0; i < kTeamSteps; i++) {
        const uint32_t x = xs[i * M], me = meta[i * M];
        const uint32_t body = (me >> 3) & 1u, r = me & 3u, f = 0u - ((me >> 2) & 1u);
        const uint32_t L = ib + 1u + body, pl = p1 << body;
        const uint32_t y = x << (1u + body);  // the first token's id on top
        const uint32_t y1 = y * pl, y2 = y1 * pl;
        // push the first r ids: depths 0..15 move r deeper
        const uint32_t ids = __byte_perm(__byte_perm(y2 >> ish, y1 >> ish, 0x0400u), y >> ish, 0x4210u) & 0xFFFFFF00u;
        const uint32_t sh = 8u * r;
        fifo.f3 = __funnelshift_l(fifo.f2, fifo.f3, sh);
        fifo.f2 = __funnelshift_l(fifo.f1, fifo.f2, sh);
        fifo.f1 = __funnelshift_l(fifo.f0, fifo.f1, sh);
        fifo.f0 = __funnelshift_l(ids, fifo.f0, sh);
        fifo.len = min(fifo.len + r, 16u);
        // the FIFO token: its entry moves to the front
        const uint32_t fi = (y << (r * L)) >> 27;
        const uint32_t sd = fifo.len - 1u - fi;
        past |= sd & f;  // negative: past the entries
        const uint32_t d = sd & 15u;
        const uint32_t h = 0u - (d >> 3);
        const uint32_t a0 = fifo.f0 ^ ((fifo.f0 ^ fifo.f2) & h), a1 = fifo.f1 ^ ((fifo.f1 ^ fifo.f3) & h);
        const uint32_t v = __byte_perm(a0, a1, d & 7u) & 0xFFu;
        fifo.mtf_masked(v, masks[(d & f) | (16u & ~f)]);  // row 16 changes nothing
        out[i * M] = me | (v << 8) | (t << 16);
        t += r - f;
    }
}

// A token's local id: the top bits of its field (idsh = 9 - the id width).
__device__ __forceinline__ uint32_t tok_id(uint32_t rec, uint32_t idsh) { return (rec & 0x1FFu) >> idsh; }

// All of a lane's records with the exact FIFO (a raw id is searched for and
// moved from where it is, as in conn_parse); whether every FIFO index named
// an entry.
__device__ __noinline__ bool team_fifo_exact(uint16_t* row, uint32_t n, uint32_t idsh, const uint4* masks) {
    MtfFifo fifo;
    fifo.f0 = fifo.f1 = fifo.f2 = fifo.f3 = 0xFFFFFFFFu;
    int32_t smin = 0;
    for (uint32_t i = 0; i < n; i++) {
        const uint32_t rec = row[i];
        const bool raw = (rec & kTokRaw) != 0u;
        const int32_t sd = static_cast<int32_t>(fifo.len) - 1 - static_cast<int32_t>((rec >> 4) & 31u);
        smin = min(smin, raw ? 0 : sd);
        const uint32_t s = static_cast<uint32_t>(sd) & 15u;
        const uint32_t v = raw ? (tok_id(rec, idsh) & 0xFFu) : fifo.at(s);
        const uint32_t at = raw ? fifo.find(v) : 16u;
        const bool fresh = raw & (at == 16u);
        fifo.mtf_masked(v, masks[raw ? (fresh ? min(fifo.len, 15u) : at) : s]);
        fifo.len += (fresh & (fifo.len < 16u)) ? 1u : 0u;
        if (!raw) row[i] = static_cast<uint16_t>((rec & ~0x1FFu) | ((v << idsh) & 0x1FFu));
    }
    return smin >= 0;
}

// What the assembly needs to know of a meshlet.
struct TeamSize {
    uint32_t n_local, n_tris, n_tok;
    uint32_t idsh;  // 9 - id width (_idx_bits_for, paradelta_codec.py:124-125)
};

// One meshlet's assembly: a warp's state between windows of 32 tokens.
struct TeamAsm {
    uint32_t heads = 0u;    // heads of the window before
    uint32_t last0 = 2u;    // the last token that reset p0 (edge code 0 or a strip's third root)
    uint32_t tcnt = 0u, wcnt = 0u, kind0 = 0u, n_raw = 0u;
    uint32_t t = 0u;        // records written
    uint32_t t0 = 0u;       // the next window
    uint32_t tp_prev = 0u;  // lane's token of the window before: its id's token before it, + 1
    bool out = false;       // an id outside the meshlet (lane's)
    bool redo = false;      // needs the exact FIFO
};

// A meshlet's token records from a chunk of steps, a lane per step (xs and
// steps: its slots, M apart).  FIFO tokens get the field of their id, or keep
// their index when `exact` (the exact FIFO resolves them).
template <uint32_t M>
__device__ __forceinline__ void team_records(TeamAsm& S, const TeamSize& F, bool exact, uint16_t* __restrict__ row,
                                             const uint32_t* __restrict__ xs, const uint32_t* __restrict__ steps,
                                             int lane) {
    const bool has = static_cast<uint32_t>(lane) < kTeamSteps;
    const uint32_t x = has ? xs[lane * M] : 0u, st = has ? steps[lane * M] : 0u;
    const bool body = (st & kStepBody) != 0u;
    const uint32_t L = 9u - F.idsh + (body ? 2u : 1u), s = body ? 21u : 22u;
    const uint32_t r = st & 3u, f = (st >> 2) & 1u, t = st >> 16;
    if (r + f > 0u) row[t] = static_cast<uint16_t>((x >> s) | ((st & kStepHead) ? kTokHead : 0u));
    if (r + f > 1u) row[t + 1u] = static_cast<uint16_t>((x << L) >> s);
    if (r + f > 2u) row[t + 2u] = static_cast<uint16_t>((x << (2u * L)) >> s);
    if (f && !exact) {
        const uint32_t rec = ((x << (r * L)) >> s) & ~0x1FFu;
        row[t + r] = static_cast<uint16_t>(rec | ((((st >> 8) & 0xFFu) << F.idsh) & 0x1FFu) |
                                           (r == 0u && (st & kStepHead) ? kTokHead : 0u));
    }
    S.t = __shfl_sync(kFull, t + r + f, kTeamSteps - 1);
    __syncwarp();
}

// Tokens [t0, t0 + 32) of a meshlet.  `row` has two readable entries before
// it.  The walk (first occurrences of ids from `first` on) goes out as entries
// in walk order and, when kList, as bytes, the vertices of the parallelogram
// entries from the front of `vlist` and of the roots from its end.  `exact`:
// by the exact FIFO, raw ids need no check.
template <bool kList>
__device__ __forceinline__ void team_window(TeamAsm& S, const TeamSize& F, uint32_t first, bool exact, uint32_t t0,
                                            const uint16_t* __restrict__ row, uint32_t* __restrict__ walk,
                                            uint8_t* __restrict__ vlist, uint32_t* __restrict__ last,
                                            uint32_t* __restrict__ tri, int lane) {
    const uint32_t me = 1u << lane, lt = me - 1u, le = lt | me;
    const uint32_t n_tok = F.n_tok, n_local = F.n_local, idsh = F.idsh;
    const uint32_t t = t0 + lane;
    const bool in = t < n_tok;
    const uint32_t rec = in ? row[t] : 0u;
    const bool raw = (rec & kTokRaw) != 0u;
    const uint32_t lm = __ballot_sync(kFull, in);
    const uint32_t rm = __ballot_sync(kFull, raw);
    const uint32_t hm = __ballot_sync(kFull, (rec & kTokHead) != 0u);
    const uint32_t em = __ballot_sync(kFull, (rec & kTokEdge) != 0u);
    const uint32_t id = tok_id(rec, idsh), v = id & 0xFFu;
    const uint32_t v1 = tok_id(row[static_cast<int>(t) - 1], idsh) & 0xFFu;
    const uint32_t v2 = tok_id(row[static_cast<int>(t) - 2], idsh) & 0xFFu;
    // the id's token before this one, and the raw tokens up to it
    const uint32_t same = __match_any_sync(kFull, in ? v : 256u + lane);
    const uint32_t lw = last[v];  // (token + 1) << 16 | raw tokens up to it, 0: none
    const uint32_t pm = same & lt;
    const uint32_t pl = 31u - __clz(pm);
    const bool seen = (pm | lw) != 0u;
    const uint32_t raws = S.n_raw + __popc(rm & le);
    const uint32_t raws_to = pm ? S.n_raw + __popc(rm & ((2u << (pl & 31u)) - 1u)) : lw & 0xFFFFu;
    const uint32_t tp1 = in & seen ? (pm ? t0 + pl + 1u : lw >> 16) : 0u;
    const bool isnew = raw & !seen & (v >= first);  // first occurrences are raw
    __syncwarp();
    if (in && (same & ~le) == 0u) last[v] = ((t + 1u) << 16) | raws;
    const uint32_t nm = __ballot_sync(kFull, isnew);
    const uint32_t r2 = ((hm << 2) | (S.heads >> 30)) & lm;  // third roots
    const uint32_t rootm = hm | (hm << 1) | (S.heads >> 31) | r2;
    const uint32_t bodym = lm & ~rootm;
    const uint32_t emit = bodym | r2;
    const uint32_t zm = r2 | (bodym & ~em);  // tokens that reset p0
    const bool body = (bodym & me) != 0u;
    S.out = S.out | (in & (id >= n_local));
    // p0 before this token: the id two before the last reset
    const uint32_t m = zm & lt;
    const uint32_t l0 = m ? t0 + 31u - __clz(m) : S.last0;
    const uint32_t p0p = tok_id(row[static_cast<int>(l0) - 2], idsh) & 0xFFu;
    // edge code 0 -> (p1, p2 | p0), 1 -> (p0, p2 | p1) (:530-535)
    const bool ec = body & ((em & me) != 0u);
    const uint32_t p0 = ec ? p0p : v2;
    const uint32_t cref = ec ? v2 : p0p;
    const uint32_t ts = S.tcnt + __popc(emit & lt);
    if ((emit & me) && ts < F.n_tris) tri[ts] = p0 | (v1 << 8) | (v << 16);
    const uint32_t wi = S.wcnt + __popc(nm & lt);
    if (isnew && wi < n_local) {
        walk[wi] = body ? (v | (p0 << 8) | (v1 << 16) | (cref << 24)) : v * 0x01010101u;
        if constexpr (kList) {
            const uint32_t rk = S.kind0 + __popc(nm & rootm & lt);  // roots before this entry
            vlist[body ? wi - rk : n_local - 1u - rk] = static_cast<uint8_t>(v);
        }
    }
    // The raw ids must be new to the FIFO.  Sixteen raw tokens since the id's
    // token pushed it out; with fewer, sixteen distinct ids did: tokens since
    // whose own predecessor lies before it.  (Counted as far back as the
    // window before this one: a lower bound.)
    if (!exact) {
        for (uint32_t mb = __ballot_sync(kFull, raw & seen & (raws - raws_to <= 16u)); mb; mb &= mb - 1u) {
            const uint32_t b = 31u - __clz(mb & (0u - mb));
            const uint32_t from = __shfl_sync(kFull, tp1, b);  // that token + 1
            const uint32_t now = __ballot_sync(kFull, in & (t >= from) & (tp1 < from)) & ((1u << b) - 1u);
            const uint32_t before = __ballot_sync(kFull, t >= from + 32u && S.tp_prev < from);
            S.redo = S.redo | (__popc(now) + __popc(before) < 16);
        }
        S.tp_prev = tp1;
    }
    S.kind0 += __popc(nm & rootm);
    S.wcnt += __popc(nm);
    S.tcnt += __popc(emit);
    S.n_raw += __popc(rm);
    S.last0 = zm ? t0 + 31u - __clz(zm) : S.last0;
    S.heads = hm;
    __syncwarp();
}

// A meshlet's first n triangles out to its index rows (out = idx + 3 *
// t_base, ph = t_base & 3; row(v): the row of local id v): whole quads as 48 bytes from a 16-byte boundary,
// then the up to three triangles before the first and after the last.
template <typename Row>
__device__ __forceinline__ void team_triangles(uint32_t* __restrict__ out, const uint32_t* __restrict__ tri, uint32_t ph,
                                               uint32_t n, Row row, int lane) {
    auto id = [&](uint32_t p, uint32_t k) { return row((p >> (8u * k)) & 0xFFu); };
    const uint32_t h = min((4u - ph) & 3u, n);   // head: [0, h)
    const uint32_t q = h + ((n - h) & ~3u);      // whole quads: [h, q)
    for (uint32_t l = h + 4u * lane; l < q; l += 128u) {
        const uint32_t x = tri[l], y = tri[l + 1u], z = tri[l + 2u], w = tri[l + 3u];
        uint4* o = reinterpret_cast<uint4*>(out + 3u * l);
        o[0] = make_uint4(id(x, 0), id(x, 1), id(x, 2), id(y, 0));
        o[1] = make_uint4(id(y, 1), id(y, 2), id(z, 0), id(z, 1));
        o[2] = make_uint4(id(z, 2), id(w, 0), id(w, 1), id(w, 2));
    }
    const uint32_t odd = h + (n - q);
    if (static_cast<uint32_t>(lane) < odd) {
        const uint32_t l = static_cast<uint32_t>(lane) < h ? lane : q + (lane - h);
        const uint32_t p = tri[l];
        out[3u * l] = id(p, 0);
        out[3u * l + 1u] = id(p, 1);
        out[3u * l + 2u] = id(p, 2);
    }
}

}  // namespace
}  // namespace stride

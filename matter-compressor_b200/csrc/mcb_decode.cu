// mcb_decode.cu -- sm_100a block decode: entropy stage + reconstruction stage.
//
// Stage 1, k_entropy: one LANE per block. The adaptive binary range decoder
// is a serial dependency chain per block (src/mc_codec.c:197-226), so the
// parallelism is across blocks: every lane of a warp runs its own decoder and
// the loop body advances every lane by up to a whole coefficient -- a run of
// zeros, a significance bin, a magnitude rung and a sign -- in straight-line
// code, so lanes never wait on each other inside a block. The per-bin chain is
// kept short: the significance band is tracked by scan-position boundaries and
// the density by the positions at which the last three ones leave its window,
// so the only shared-memory read on the chain is the context itself. The lane's adaptive contexts sit
// in shared memory as 32-bit words (context j of lane l at word j*32+l:
// conflict-free). Output per block: a small header (dc, flags) and a list of
// nonzero levels plus corrections.
//
// Stage 2, k_reconstruct: one CTA (64 threads) per block. Dequantise into a
// dense coefficient box bounded by the block's extents, then the three
// separable DCT-III passes along x, y, z, each output accumulated over
// ascending k in single precision with explicit round-to-nearest adds and
// multiplies (no FMA), exactly the order of src/mc_codec_float.h:98-105.
// Coefficients outside the extent box are zero and the reference skips them;
// including zero terms inside the box adds +/-0 to an accumulator that can
// never be -0, so the dense box sum is bit-identical to the sparse one.
// Then lrint + dc, clamp to u8 (src/mc_codec.c:766-769), the sparse
// corrections in stream order (:770-782), and the clipped store.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mcb_devinfo.h"
#include "mcb_f32x2.cuh"
#include "mcb_format.h"
#include "mcb_kernels.h"
#include "mcb_rowstore.cuh"

namespace mcb {

__constant__ float c_cos[16][16];
// {c[k][m], c[k][m], c[k][m+1], c[k][m+1]} at [k][m/2]: weights of packed pairs
__constant__ float4 c_cos2[16][8];
// c_bend[b]: the first scan position past band b (b < 7), then kN3 and a
// sentinel; kernels copy it into shared memory at start
__constant__ uint16_t c_bend[9];

// ---------------------------------------------------------------- stage 1
// Lane states. A lane that decodes significance and magnitude bins takes part
// in the step that every lane of a warp runs together; the slow states occur a
// few times per block and are worked off by the lanes that hold them while the
// rest of the warp waits (see run_lanes). The block header and EOB are decoded
// when a lane starts its block.
enum : uint32_t {
    F_RUN = 0,   // k == 0: significance of scan position p, context sigb + min(ones among the last 16
                 // flags, 3); k in 1..11: magnitude rung k of the coefficient at p - 1, context 56 + k;
                 // k >= 12: a bit of the Exp-Golomb prefix behind the twelfth rung, 12 + the ones so far
    S_IDLE,      // no more blocks for this lane
    S_LAST,      // the coefficient at the last position before the EOB, significant by definition
    S_END,       // scan done: corrections, then the block is finished
    S_DONE
};
// Context slots per lane: the 68 adaptive contexts plus one that follows the
// magnitude ladder and holds 1: a bypass bin splits at (range >> 1) * 1 where a
// rung splits at (range >> 12) * p. A parked lane uses it as a scratch slot.
constexpr int kCtxSlots = kNumCtx + 1;
constexpr uint32_t kScr = kNumCtx;
static_assert(kScr == kCtxMag + 12, "scratch slot follows the 12 magnitude rungs");
// The range is renormalised when it falls below this (src/mc_codec.c:202).
constexpr uint32_t kTop = 1u << 24;

struct LaneState {
    const uint8_t *abase;      // payload start rounded down to 4 bytes
    uint32_t *ent;             // the block's entries in the arena (first cap of them)
    uint32_t len, off0;        // payload length, payload start - abase
    uint32_t w, w2, used;      // two payload words, first byte highest; bits of w already read (0, 8, 16, 24)
    uint32_t nxt, nmask, jn;   // the word after them (raw), its payload bytes, its index
    uint32_t code, range;
    uint32_t st, p, eob, sigb, band, bend, stop;   // p: next scan position to decode a significance flag of
    uint32_t e1, e2, e3;       // the last three significant positions (newest first) + 17: the position
                               // from which each has left the 16-flag density window
    uint32_t cs, ps, lim;      // significance context slot at p, its probability, and the position from
                               // which another slot (or a position event) is due
    uint32_t k, pm;            // next magnitude rung (0 at a significance bin), its probability
    uint32_t hdr;              // flag0, flag1, dc bits 7..0 (10 bits, first bin highest)
    uint32_t nent, cap, ovf, bad, ccount;
    int item;
};

// Payload word j (bytes 4j-off0 .. 4j-off0+3 of the payload), bytes past the
// payload read as zero (src/mc_codec.c:96). Loads are 4-byte aligned and never
// start past the word holding the payload's last byte. The raw load and the
// mask of its payload bytes are kept apart: the next word is loaded a refill
// ahead and masked only when it enters the window, so nothing waits on the
// load until then.
__device__ __forceinline__ uint32_t word_mask(const LaneState &L, uint32_t j) {
    const int avail = (int)L.len - ((int)(4 * j) - (int)L.off0);
    return avail >= 4 ? 0xFFFFFFFFu : (avail <= 0 ? 0u : (1u << (8 * avail)) - 1u);
}
__device__ __forceinline__ uint32_t word_raw(const LaneState &L, uint32_t j) {
    uint32_t v = 0;
    if ((int)(4 * j) - (int)L.off0 < (int)L.len) v = __ldg(reinterpret_cast<const uint32_t *>(L.abase) + j);
    return v;
}
__device__ __forceinline__ uint32_t load_word(const LaneState &L, uint32_t j) {
    return __byte_perm(word_raw(L, j) & word_mask(L, j), 0, 0x0123);
}

// The window's first word is read to its end: the second takes its place.
__device__ __forceinline__ void refill(LaneState &L) {
    L.w = L.w2;
    L.w2 = __byte_perm(L.nxt & L.nmask, 0, 0x0123);
    L.used -= 32;
    ++L.jn;
    L.nmask = word_mask(L, L.jn);
    L.nxt = word_raw(L, L.jn);
}

// One payload byte (slow paths).
__device__ __forceinline__ uint32_t next_byte(LaneState &L) {
    const uint32_t b = (L.w >> (24 - L.used)) & 0xFFu;
    L.used += 8;
    if (L.used == 32) refill(L);
    return b;
}

// Renormalise (src/mc_codec.c:202).
__device__ __forceinline__ void renorm(LaneState &L) {
    while (L.range < kTop) { L.code = (L.code << 8) | next_byte(L); L.range <<= 8; }
}

// One adaptive bin (src/mc_codec.c:198-204).
__device__ __forceinline__ uint32_t ctx_bin(LaneState &L, uint32_t *cp) {
    const uint32_t p0 = *cp;
    const uint32_t r0 = (L.range >> 12) * p0;
    const uint32_t bit = L.code >= r0 ? 1u : 0u;
    L.code -= bit ? r0 : 0u;
    L.range = bit ? L.range - r0 : r0;
    *cp = bit ? p0 - (p0 >> 4) : p0 + ((4096u - p0) >> 4);
    renorm(L);
    return bit;
}

// nb bypass bits read as one batch, 1 <= nb <= 16 (src/mc_codec.c:205,216-226).
__device__ __forceinline__ uint32_t bypass_bits(LaneState &L, uint32_t nb) {
    L.range >>= nb;
    uint32_t q;
    if (nb == 1) {
        q = L.code >= L.range ? 1u : 0u;
    } else {
        q = L.code / L.range;
        const uint32_t mx = (1u << nb) - 1u;
        q = q > mx ? mx : q;
    }
    L.code -= q * L.range;
    renorm(L);
    return q;
}

// Any number of bypass bits: pieces of 16, most significant first
// (src/mc_codec.c:219-220).
__device__ __forceinline__ uint32_t bypass_long(LaneState &L, uint32_t nb) {
    uint32_t v = 0;
    while (nb > 16) { v = (v << 16) | bypass_bits(L, 16); nb -= 16; }
    return nb ? (v << nb) | bypass_bits(L, nb) : v;
}

// Exp-Golomb value in bypass bins (src/mc_codec.c:234-238); a prefix of
// kEgCap one-bits marks the stream bad and yields 0.
__device__ __forceinline__ uint32_t eg_value(LaneState &L) {
    uint32_t nb = 0;
    while (bypass_bits(L, 1)) {
        if (++nb >= (uint32_t)kEgCap) { L.bad = 1; return 0; }
    }
    if (!nb) return 0;
    return ((1u << (nb & 31)) | bypass_long(L, nb)) - 1u;
}

// Appends one entry; false (stream cut short) when a corrupt stream also
// exhausts the shared overflow pool.
__device__ __forceinline__ bool put_entry(LaneState &L, const EntParams &P, uint32_t v) {
    const uint32_t j = L.nent;
    if (j < L.cap) {
        L.ent[j] = v;
    } else {   // only corrupt streams get here
        if (L.ovf == 0xFFFFFFFFu) {
            const uint32_t need = kEntryMax - L.cap;
            const uint32_t off = atomicAdd(P.pool_used, need);
            if ((uint64_t)off + need > P.pool_cap) { L.bad = 1; L.st = S_DONE; return false; }
            L.ovf = off;
        }
        P.pool[L.ovf + (j - L.cap)] = v;
    }
    L.nent = j + 1;
    return true;
}

// The density class at position p, min(ones among the last 16 flags, 3)
// (src/mc_codec.c:249-259), from the expiries of the last three ones: its
// context slot, and the position up to which slot and band stay the same.
__device__ __forceinline__ void density(LaneState &L) {
    const bool a3 = L.p < L.e3, a2 = L.p < L.e2, a1 = L.p < L.e1;   // e1 >= e2 >= e3
    L.cs = L.sigb + (a3 ? 3u : (a2 ? 2u : (a1 ? 1u : 0u)));
    L.lim = min(L.stop, a3 ? L.e3 : (a2 ? L.e2 : (a1 ? L.e1 : 0xFFFFFFFFu)));
}

// flags bit 1 (has corrections) is the second header bin
__device__ __forceinline__ bool has_corr(const LaneState &L) { return (L.hdr >> 8) & 1; }

// A lane with no more work: an endless run of zeros over an empty payload, in
// the scratch context (code 0 is below every split; p stays far from stop).
__device__ __forceinline__ void park(LaneState &L) {
    L.st = S_IDLE;
    L.item = -1;
    L.code = 0;
    L.range = 0xFFFFFFFFu;
    L.sigb = L.cs = kScr;
    L.ps = L.pm = 2048;
    L.p = 0;
    L.lim = L.stop = 0xFFFFFFFFu;
    L.e1 = L.e2 = L.e3 = 0;
    L.len = L.off0 = L.jn = 0;
    L.w = L.w2 = L.nxt = L.nmask = L.used = 0;
    L.k = 0;
}

// Scan position L.p is next and L.p >= L.stop: a band change and/or the
// end of the scan. The last position before the EOB is significant by
// definition and costs no bin (src/mc_codec.c:364); past the EOB the
// coefficient loop ends.
__device__ __forceinline__ void position_event(LaneState &L, const uint32_t *ctx, const uint16_t *s_bend) {
    while (L.p >= L.bend) { L.band++; L.sigb += 4; L.bend = s_bend[L.band]; }
    if (L.p + 1 >= L.eob) {
        if (L.p + 1 == L.eob) {
            L.p++;
            L.st = S_LAST;
        } else {
            L.st = S_END;
        }
    }
    L.stop = min(L.bend, L.eob - 1);   // eob >= 1 here (eob == 0 never enters the scan)
    density(L);
    L.ps = ctx[L.cs * 32];
}

// Starts block `slot`: contexts from the quality table, range decoder,
// header bins, EOB (src/mc_codec.c:739-757, 321-327).
__device__ __forceinline__ void lane_begin(LaneState &L, const EntParams &P, uint32_t *ctx, const uint16_t *s_bend,
                                           int slot) {
    const DecItem &it = P.items[slot];
    L.item = slot;
    const uintptr_t src = (uintptr_t)it.src;
    L.abase = reinterpret_cast<const uint8_t *>(src & ~(uintptr_t)3);
    L.off0 = (uint32_t)(src & 3);
    L.len = it.len;
    ctx[kScr * 32] = 1;
    L.ent = P.arena + P.base[slot];
    L.cap = entry_cap(L.len);
    L.ovf = 0xFFFFFFFFu;
    L.bad = 0;
    L.nent = 0;
    L.ccount = 0;
    L.hdr = 0;
    L.p = 0; L.eob = 0; L.k = 0;
    L.e1 = 0; L.e2 = 0; L.e3 = 0;
    L.band = 0; L.sigb = kCtxSig; L.bend = s_bend[0]; L.stop = 0;
    if (L.len == 0) { L.st = S_DONE; return; }   // absent block: zeros
    const uint4 *q = reinterpret_cast<const uint4 *>(P.qtab[it.qslot].ctx);
#pragma unroll
    for (int j = 0; j < 9; ++j) {               // 72 u16 initial contexts
        const uint4 v = __ldg(q + j);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int c = j * 8 + h * 2;
            if (c < kNumCtx) ctx[c * 32] = w[h] & 0xFFFFu;
            if (c + 1 < kNumCtx) ctx[(c + 1) * 32] = w[h] >> 16;
        }
    }
    L.w = load_word(L, 0);
    L.w2 = load_word(L, 1);
    L.used = 8 * L.off0;
    L.jn = 2;
    L.nmask = word_mask(L, 2);
    L.nxt = word_raw(L, 2);
    L.range = 0xFFFFFFFFu;
    L.code = 0;
    for (int i = 0; i < 5; ++i) L.code = (L.code << 8) | next_byte(L);
    for (int i = 0; i < 10; ++i) L.hdr = (L.hdr << 1) | ctx_bin(L, ctx + (kCtxFlag + i) * 32);
    uint32_t k = 0;
    while (k < 13 && ctx_bin(L, ctx + (kCtxEob + k) * 32)) k++;
    const uint32_t eob = k < 2 ? k : (1u << (k - 1)) | bypass_bits(L, k - 1);
    L.eob = eob > (uint32_t)kN3 ? (uint32_t)kN3 : eob;
    if (L.eob == 0) { L.st = S_END; return; }
    L.st = F_RUN;
    L.pm = ctx[kCtxMag * 32];
    position_event(L, ctx, s_bend);
}

__device__ __forceinline__ void lane_finish(LaneState &L, const EntParams &P) {
    EntHdr h;
    h.dc = (uint8_t)(L.hdr & 0xFF);
    h.flags = (uint8_t)(((L.hdr >> 9) & 1) | (((L.hdr >> 8) & 1) << 1));
    h.bad = (uint8_t)L.bad;
    h.pad = 0;
    h.ez = h.ey = h.ex = -1;    // extents are taken from the entries by k_reconstruct
    h.pad2 = 0;
    h.nnz = (uint16_t)(L.nent - 2 * L.ccount);
    h.ncorr = (uint16_t)L.ccount;
    h.ovf = L.ovf;
    P.hdr[L.item] = h;
    if (L.bad) atomicAdd(P.status, 1u);
}

// The sparse max-error corrections after the scan (src/mc_codec.c:770-782):
// count, then per correction a position gap, a sign and a magnitude, each
// gap and magnitude an Exp-Golomb value. Recorded as entry pairs (position,
// wrapping delta) after the coefficients.
__device__ __forceinline__ void decode_corrections(LaneState &L, const EntParams &P) {
    uint32_t n = eg_value(L) + 1u;
    if (L.bad) return;
    if (n > (uint32_t)kN3) n = kN3;
    uint32_t pos = 0;
    for (uint32_t c = 0; c < n; ++c) {
        pos += eg_value(L);
        if (L.bad) return;
        const uint32_t neg = bypass_bits(L, 1);
        const uint32_t m = eg_value(L) + 1u;
        if (L.bad || pos >= (uint32_t)kN3) return;
        if (!put_entry(L, P, pos) || !put_entry(L, P, neg ? 0u - m : m)) return;
        L.ccount++;
    }
}

// Bits that a renormalisation shifts in (src/mc_codec.c:202): two bytes at
// most, since the range is at least 2^24 before a bin and a split leaves at
// least 15 * 2^12 of it (p <= 4081 once adapted).
__device__ __forceinline__ uint32_t renorm_bits(uint32_t range) {
    return range < (1u << 16) ? 16u : (range < kTop ? 8u : 0u);
}

// The rest of the coefficient at p - 1: for m > 12 the Exp-Golomb suffix of
// m - 12 bits (the magnitude is 11 + (1 << nb | suffix), src/mc_codec.c:234-238,
// 268-275), then sign and entry; false when the block ends (overflow pool
// exhausted: corrupt streams only). A suffix of nb <= 16 bits, the batched read
// range >>= nb, q = min(code / range, 2^nb - 1), code -= q * range (:216-226), and
// the sign take at most 24 bits of the window, so both go straight through (see
// renorm_bits): where many coefficients have a suffix, some lane of the warp is
// here at every step (12 chunks at q=1 3.62 ms bit by bit with a renormalisation
// loop each, 3.33 so; 10 chunks of noise at q=0.25 27.9 and 24.7).
__device__ __forceinline__ bool finish_coef(LaneState &L, const EntParams &P, uint32_t m) {
    const uint32_t nb = m > 12u ? m - 12u : 0u;
    uint32_t neg;
    if (nb <= 16u) {
        uint32_t x = funnel_left(L.w2, L.w, L.used), code = L.code, r = L.range >> nb;
        const uint32_t q = min(code / r, (1u << nb) - 1u);   // 0 without a suffix
        code -= q * r;
        m = nb ? 11u + ((1u << nb) | q) : m;
        const uint32_t s1 = renorm_bits(r);
        code = funnel_left(x, code, s1);
        x <<= s1;
        r = (r << s1) >> 1;
        neg = code >= r ? 1u : 0u;
        code = neg ? code - r : code;
        const uint32_t s2 = r < kTop ? 8u : 0u;
        L.code = funnel_left(x, code, s2);
        L.range = r << s2;
        L.used += s1 + s2;
        if (L.used >= 32u) refill(L);
    } else {
        m = 11u + ((1u << (nb & 31u)) | bypass_long(L, nb));
        neg = bypass_bits(L, 1);
    }
    return put_entry(L, P, (L.p - 1u) | ((neg ? 0u - m : m) << 16));
}

// The same with the suffix as nb halvings: with the range's low nb bits cleared
// first they are that long division bit by bit, clamp included, and leave the same
// code and range.
__device__ __forceinline__ bool finish_coef_bits(LaneState &L, const EntParams &P, uint32_t m) {
    if (m > 12u) {
        const uint32_t nb = m - 12u;
        uint32_t acc = 1u << (nb & 31u);
        if (nb <= 16u) {
            uint32_t r = L.range & (0xFFFFFFFFu << nb);
            acc = 1;
            for (uint32_t i = 0; i < nb; ++i) {
                r >>= 1;
                const bool b = L.code >= r;
                L.code = b ? L.code - r : L.code;
                acc = 2u * acc + (b ? 1u : 0u);
            }
            L.range = r;
            renorm(L);
        } else {
            acc |= bypass_long(L, nb);
        }
        m = 11u + acc;
    }
    const uint32_t neg = bypass_bits(L, 1);
    return put_entry(L, P, (L.p - 1u) | ((neg ? 0u - m : m) << 16));
}

// The slow states of one lane, run while the rest of its warp waits. ALONE: of a
// single-thread kernel, which gets here for S_END only; with finish_coef in its
// place they still took 1 % longer (one chunk at q=0.5 2035 us, 2016 so).
template <bool ALONE>
__device__ __forceinline__ void slow_work(LaneState &L, const EntParams &P, uint32_t *ctx, const uint16_t *s_bend) {
    if (L.st == S_LAST) {
        uint32_t k = 0;
        while (k < 12 && ctx_bin(L, ctx + (kCtxMag + k) * 32)) ++k;
        if (k == 12) {
            while (bypass_bits(L, 1)) {
                if (++k >= 12u + (uint32_t)kEgCap) { L.bad = 1; L.st = S_DONE; return; }
            }
        }
        const uint32_t m = k < 12u ? k + 1u : k;
        if (ALONE ? finish_coef_bits(L, P, m) : finish_coef(L, P, m)) L.st = S_END;
        return;
    }
    // S_END
    if (has_corr(L)) decode_corrections(L, P);
    L.st = S_DONE;
}

// Predicated global store (the compiler turns this into one predicated
// instruction, no branch).
__device__ __forceinline__ void stg_if(bool pred, uint32_t *p, uint32_t v) {
    if (pred) *p = v;
}

// p + ((4096 - p) >> 4) and p - (p >> 4) (src/mc_codec.c:198-204) as one
// multiply-add and a shift: equal for every p in 0..4096
__device__ __forceinline__ uint32_t prob_after0(uint32_t p) { return (15u * p + 4096u) >> 4; }
__device__ __forceinline__ uint32_t prob_after1(uint32_t p) { return (15u * p + 15u) >> 4; }

// The rare events of a fast step: a coefficient that goes on in finish_coef
// (an Exp-Golomb suffix, or a sign that the step had no bytes left for), a
// prefix at its cap and an entry past the block's arena share (corrupt streams
// only), and a scan position at a band change or the end of the scan.
enum : uint32_t { EV_COEF = 1, EV_CAP = 2, EV_OVF = 4, EV_POS = 8 };
__device__ __forceinline__ void fast_event(LaneState &L, const EntParams &P, const uint32_t *ctx,
                                           const uint16_t *s_bend, uint32_t why, uint32_t v) {
    if ((why & EV_COEF) && !finish_coef(L, P, v >> 16)) return;
    if (why & EV_CAP) { L.bad = 1; L.st = S_DONE; return; }
    if ((why & EV_OVF) && !put_entry(L, P, v)) return;   // pool exhausted, block ends
    if (L.p >= L.stop && L.k == 0) position_event(L, ctx, s_bend);
}

// One step of every lane: up to a whole coefficient, by the same straight-line
// code of selects and predicated accesses for every lane.
//  1. A lane at a significance bin first takes a run of one or four
//     insignificant positions. While bins are 0 the code does not change and
//     the range only falls, so a run needs no compare per bin: its last split
//     above both the code and the renormalisation bound (one compare with the
//     larger) says that all its bins are 0 and none renormalises. Its length
//     leaves room for a bin in the same context after it.
//  2. Then one significance bin (src/mc_codec.c:353-375).
//  3. A significant position goes on with magnitude rung 0 at once, a lane at
//     a later rung or in an Exp-Golomb prefix with its next bin
//     (src/mc_codec.c:268-275).
//  4. A magnitude that closes takes its sign at once (:205).
// A lane without a bin of a kind keeps its range by splitting at the range
// itself. The context values come from shared memory a step ahead (ps, pm):
// loaded as soon as the next position's density class and the next rung are
// known, after the store of the context just used.
// The bins of a step could take 40 bits (see renorm_bits), and the window always
// holds as many; the 32 extracted here serve all but a sign after more than 24 bits,
// which is left to fast_event. Returns the events of the lane; v is its entry (for
// EV_COEF, the argument of finish_coef in the high half).
// What bounds it: integer issue, most of it on the ALU pipe at half rate. Runs
// of length 1 or 4: allowing 1 to 4 takes 6 % fewer steps (a q=6 block of the bench
// volumes 701 against 743, 1643 without runs) of a tenth more instructions. A step of one
// bin per lane took 2041 steps a block at q=6 and 9870 at q=1; 64 chunks at
// q=6: 2.68 ms with it, 1.54 ms with this one.
__device__ __forceinline__ uint32_t fast_step(LaneState &L, const EntParams &P, uint32_t *ctx, uint32_t &v) {
    const uint32_t k0 = L.k;
    const bool is_sig = k0 == 0u;
    uint32_t code = L.code, range = L.range, pr = L.ps, p = L.p;
    uint32_t x = funnel_left(L.w2, L.w, L.used);   // the next 32 payload bits
    // 1. zeros
    {
        const uint32_t floor1 = code >= kTop ? code : kTop - 1u;
        const uint32_t room = is_sig ? L.lim - p : 0u;   // > 0 at a significance bin
        const uint32_t r1 = (range >> 12) * pr, q1 = prob_after0(pr);
        const uint32_t r2 = (r1 >> 12) * q1, q2 = prob_after0(q1);
        const uint32_t r3 = (r2 >> 12) * q2, q3 = prob_after0(q2);
        const uint32_t r4 = (r3 >> 12) * q3, q4 = prob_after0(q3);
        const bool z1 = (r1 > floor1) & (room > 1u), z4 = (r4 > floor1) & (room > 4u);
        range = z4 ? r4 : (z1 ? r1 : range);
        pr = z4 ? q4 : (z1 ? q1 : pr);
        p += z4 ? 4u : (z1 ? 1u : 0u);
    }
    // 2. one significance bin
    const uint32_t r1 = is_sig ? (range >> 12) * pr : range;
    const bool one = is_sig & (code >= r1);
    code = one ? code - r1 : code;
    range = one ? range - r1 : r1;
    pr = (15u * pr + (one ? 15u : 4096u)) >> 4;
    if (is_sig) ctx[L.cs * 32] = pr;
    const uint32_t s1 = renorm_bits(range);
    code = funnel_left(x, code, s1);
    x <<= s1;
    range <<= s1;
    // the next position, its density class and context
    p += is_sig ? 1u : 0u;
    L.p = p;
    L.e3 = one ? L.e2 : L.e3;
    L.e2 = one ? L.e1 : L.e2;
    L.e1 = one ? p + 16u : L.e1;
    density(L);
    L.ps = ctx[L.cs * 32];
    // 3. one magnitude rung
    const bool act = one | !is_sig;
    const uint32_t pm = L.pm;
    const bool pfx = k0 >= 12u;
    const uint32_t r2 = act ? (range >> (pfx ? 1u : 12u)) * pm : range;
    const bool up = act & (code >= r2);
    code = up ? code - r2 : code;
    range = up & !pfx ? range - r2 : r2;   // a bypass bin leaves the half either way
    uint32_t *cm = ctx + (kCtxMag + k0) * 32;
    if (act & !pfx) *cm = (15u * pm + (up ? 15u : 4096u)) >> 4;
    const uint32_t kn = up ? k0 + 1u : 0u;
    L.k = kn;
    L.pm = ctx[(kCtxMag + min(kn, 12u)) * 32];   // the next rung's
    const uint32_t s2 = renorm_bits(range);
    code = funnel_left(x, code, s2);
    x <<= s2;
    range <<= s2;
    // 4. the sign of a magnitude that closed, and the entry of the coefficient at p - 1
    const bool closed = act & !up;
    const bool sign = closed & (k0 <= 12u) & (s1 + s2 <= 24u);
    const uint32_t r3 = sign ? range >> 1 : range;
    const bool neg = sign & (code >= r3);
    code = neg ? code - r3 : code;
    const uint32_t s3 = r3 < kTop ? 8u : 0u;
    L.code = funnel_left(x, code, s3);
    L.range = r3 << s3;
    const uint32_t m = pfx ? k0 : k0 + 1u;
    v = (p - 1u) | ((neg ? 0u - m : m) << 16);
    const bool room_e = L.nent < L.cap;
    stg_if(sign & room_e, L.ent + L.nent, v);
    L.nent += (sign & room_e) ? 1u : 0u;
    // the window
    const uint32_t u = L.used + s1 + s2 + s3;
    L.used = u;
    if (u >= 32u) refill(L);
    return ((closed & !sign) ? (uint32_t)EV_COEF : 0u) |
           ((kn >= 12u + (uint32_t)kEgCap) ? (uint32_t)EV_CAP : 0u) |
           ((sign & !room_e) ? (uint32_t)EV_OVF : 0u) | (((kn == 0u) & (p >= L.stop)) ? (uint32_t)EV_POS : 0u);
}

// Work queue of a launch: the first ncoded entries of the processing order
// (longest payload first). Lane g starts with entry g; later entries are
// claimed from the launch's counter in runs of P.claim consecutive entries.
struct Claim {
    int next, end;
};
__device__ __forceinline__ int claim_next(Claim &c, const EntParams &P, int nlanes) {
    if (c.next >= c.end) {
        const uint32_t run = P.claim > 0 ? (uint32_t)P.claim : 1u;
        c.next = nlanes + (int)atomicAdd(P.counter, run);
        c.end = c.next + (int)run;
    }
    return c.next++;
}

// Every lane of the warp decodes blocks until the queue is empty. Lane gtid
// starts with entry gtid (none when gtid < 0), then claims from the counter. Fast steps
// run while every lane runs or is parked; when a lane reaches a slow state the
// warp leaves the loop, that lane works its slow states off (finishing its
// block and starting the next one), and the loop resumes. Every block ends
// after a bounded number of bins (finite scan, capped Exp-Golomb prefixes,
// bounded correction count) and every lane claims at most ncoded blocks, so
// the loop ends. on_done(item) runs for every finished block.
template <class OnDone>
__device__ __forceinline__ void run_lanes(LaneState &L, const EntParams &P, uint32_t *ctx, const uint16_t *s_bend,
                                          int gtid, int nlanes, OnDone on_done) {
    memset(&L, 0, sizeof L);
    park(L);
    L.st = S_DONE;
    Claim c = gtid >= 0 ? Claim{gtid, gtid + 1} : Claim{0, 0};   // gtid < 0: queue claims only
    for (;;) {
        while (L.st >= S_LAST) {
            if (L.st != S_DONE) {
                slow_work<false>(L, P, ctx, s_bend);
                continue;
            }
            if (L.item >= 0) {
                lane_finish(L, P);
                on_done(L.item);
            }
            const int nx = claim_next(c, P, nlanes);
            if (nx < P.ncoded) lane_begin(L, P, ctx, s_bend, P.order ? (int)P.order[nx] : nx);
            else park(L);
        }
        if (__all_sync(0xFFFFFFFFu, L.st == S_IDLE)) break;
        for (;;) {
            uint32_t v;
            const uint32_t why = fast_step(L, P, ctx, v);
            if (__any_sync(0xFFFFFFFFu, why != 0)) {
                if (why) fast_event(L, P, ctx, s_bend, why, v);
                if (__any_sync(0xFFFFFFFFu, L.st >= S_LAST)) break;
            }
        }
    }
}

// The whole stream of one block on one thread, after lane_begin, written for
// the latency of one thread alone on its warp (no other lane shares its
// instructions). What bounds it: the chain of dependent instructions (five
// cycles each) and the branches, a third of the cycles. So every decision jumps
// straight to where the next bin is decoded: with the same work in nested loops
// whose flags were tested again at each level it took a fifth longer (48 blocks
// at q=6: 5.76 against 4.66 ms), and a renormalisation decided by a branch, not
// by selects, took another 4 % off (4.50; 5.94 before runs of zeros).
// All contexts of the coefficient loop that the common bins use are held in
// registers: the four significance contexts of the current band and the twelve
// magnitude rungs. Bands only advance, so a band's register contexts are never
// written back to shared memory, and the magnitude rungs are used by nothing
// else.
// Where three or more of the last 16 positions were significant (density class
// 3), half of the positions are, and bins go one at a time, their probability in
// the class's own register. In the sparser classes runs of zeros are long and go
// four at a time: while bins are 0 the code does not change and the range only
// falls, so four splits are computed straight through and one compare of the
// last with the code and the renormalisation bound decides them all.
// Band changes, Exp-Golomb tails and the corrections take the shared functions
// (position_event, eg_value, put_entry, slow_work).

// The window while the thread is alone: w shifted to its next byte, `used` bits
// gone from it; shifted back for the shared functions that read bytes.
__device__ __forceinline__ void window_in(LaneState &L) { L.w <<= L.used; }
__device__ __forceinline__ void window_out(LaneState &L) { L.w >>= L.used; }
__device__ __forceinline__ void solo_norm(LaneState &L) {
    while (L.range < kTop) {
        L.code = funnel_left(L.w, L.code, 8);
        L.w <<= 8;
        L.range <<= 8;
        L.used += 8;
        if (L.used == 32) refill(L);
    }
}
// One adaptive bin on a register context.
__device__ __forceinline__ bool reg_bin(LaneState &L, uint32_t &g) {
    const uint32_t r = (L.range >> 12) * g;
    const bool b = L.code >= r;
    L.code = b ? L.code - r : L.code;
    L.range = b ? L.range - r : r;
    g = (15u * g + (b ? 15u : 4096u)) >> 4;
    solo_norm(L);
    return b;
}
// One magnitude rung on a register context; after a 1 the range is
// renormalised here, after the closing 0 by the caller.
__device__ __forceinline__ bool rung(LaneState &L, uint32_t &g) {
    const uint32_t r = (L.range >> 12) * g;
    if (L.code < r) {
        L.range = r;
        g = prob_after0(g);
        return false;
    }
    L.code -= r;
    L.range -= r;
    g = prob_after1(g);
    solo_norm(L);
    return true;
}
// One bypass bin (src/mc_codec.c:205).
__device__ __forceinline__ bool reg_bypass(LaneState &L) {
    L.range >>= 1;
    const bool b = L.code >= L.range;
    L.code = b ? L.code - L.range : L.code;
    solo_norm(L);
    return b;
}

__device__ __forceinline__ void solo_entropy(LaneState &L, const EntParams &P, uint32_t *ctx,
                                             const uint16_t *s_bend) {
    uint32_t sigb = L.sigb;
    uint32_t s0 = ctx[(sigb + 0) * 32], s1 = ctx[(sigb + 1) * 32];
    uint32_t s2 = ctx[(sigb + 2) * 32], s3 = ctx[(sigb + 3) * 32];
    uint32_t g0 = ctx[(kCtxMag + 0) * 32], g1 = ctx[(kCtxMag + 1) * 32], g2 = ctx[(kCtxMag + 2) * 32];
    uint32_t g3 = ctx[(kCtxMag + 3) * 32], g4 = ctx[(kCtxMag + 4) * 32], g5 = ctx[(kCtxMag + 5) * 32];
    uint32_t g6 = ctx[(kCtxMag + 6) * 32], g7 = ctx[(kCtxMag + 7) * 32], g8 = ctx[(kCtxMag + 8) * 32];
    uint32_t g9 = ctx[(kCtxMag + 9) * 32], g10 = ctx[(kCtxMag + 10) * 32], g11 = ctx[(kCtxMag + 11) * 32];
    uint32_t pc, m;
    window_in(L);
    if (L.st == S_LAST) goto coef;   // the implicit last position is all there is
    if (L.st != F_RUN) goto done;
next:   // a significance bin at p < stop
    if (L.p < L.e3) {   // density class 3
        const uint32_t r = (L.range >> 12) * s3;
        ++L.p;
        if (L.code >= r) {   // significant
            L.code -= r;
            L.range -= r;
            s3 = prob_after1(s3);
            solo_norm(L);
            goto one;
        }
        L.range = r;
        s3 = prob_after0(s3);
        if ((r < kTop) | (L.p >= L.stop)) {
            solo_norm(L);
            if (L.p >= L.stop) goto position;
        }
        goto next;
    } else {
        const bool a2 = L.p < L.e2, a1 = L.p < L.e1;
        const uint32_t end = min(L.stop, a2 ? L.e2 : (a1 ? L.e1 : 0xFFFFFFFFu));
        pc = a2 ? s2 : (a1 ? s1 : s0);
    run:
        {
            const uint32_t floor1 = L.code >= kTop ? L.code : kTop - 1u;
            while (L.p + 4u <= end) {
                const uint32_t r1 = (L.range >> 12) * pc, q1 = prob_after0(pc);
                const uint32_t r2 = (r1 >> 12) * q1, q2 = prob_after0(q1);
                const uint32_t r3 = (r2 >> 12) * q2, q3 = prob_after0(q2);
                const uint32_t r4 = (r3 >> 12) * q3;
                if (r4 <= floor1) break;
                L.range = r4;
                pc = prob_after0(q3);
                L.p += 4;
            }
        }
        if (L.p < end) {
            const uint32_t r = (L.range >> 12) * pc;
            ++L.p;
            if (L.code >= r) {
                L.code -= r;
                L.range -= r;
                pc = prob_after1(pc);
                solo_norm(L);
                s0 = a1 ? s0 : pc;
                s1 = a1 & !a2 ? pc : s1;
                s2 = a2 ? pc : s2;
                goto one;
            }
            L.range = r;
            pc = prob_after0(pc);
            solo_norm(L);
            if (L.p < end) goto run;
        }
        s0 = a1 ? s0 : pc;
        s1 = a1 & !a2 ? pc : s1;
        s2 = a2 ? pc : s2;
        if (L.p >= L.stop) goto position;
        goto next;
    }
one:
    L.e3 = L.e2;
    L.e2 = L.e1;
    L.e1 = L.p + 16u;
coef:   // the coefficient at p - 1: the unary magnitude (src/mc_codec.c:268-275), the sign, the entry
    m = 1;
    if (rung(L, g0)) {
        if (!rung(L, g1)) m = 2;
        else if (!rung(L, g2)) m = 3;
        else if (!rung(L, g3)) m = 4;
        else if (!rung(L, g4)) m = 5;
        else if (!rung(L, g5)) m = 6;
        else if (!rung(L, g6)) m = 7;
        else if (!rung(L, g7)) m = 8;
        else if (!rung(L, g8)) m = 9;
        else if (!rung(L, g9)) m = 10;
        else if (!rung(L, g10)) m = 11;
        else if (!rung(L, g11)) m = 12;
        else {   // the twelfth rung set: 12 + an Exp-Golomb value
            window_out(L);
            m = 12u + eg_value(L);
            window_in(L);
            if (L.bad) { L.st = S_DONE; goto done; }   // prefix cap (corrupt streams only)
        }
    }
    solo_norm(L);
    {
        const bool neg = reg_bypass(L);
        const uint32_t v = (L.p - 1u) | ((neg ? 0u - m : m) << 16);
        if (L.nent < L.cap) L.ent[L.nent++] = v;
        else if (!put_entry(L, P, v)) goto done;   // overflow pool exhausted (corrupt streams only)
    }
    if (L.p < L.stop) goto next;
position:
    L.st = F_RUN;
    position_event(L, ctx, s_bend);
    if (L.sigb != sigb) {   // the band's contexts come into registers when it changes
        sigb = L.sigb;
        s0 = ctx[(sigb + 0) * 32]; s1 = ctx[(sigb + 1) * 32];
        s2 = ctx[(sigb + 2) * 32]; s3 = ctx[(sigb + 3) * 32];
    }
    if (L.st == F_RUN) goto next;
    if (L.st == S_LAST) goto coef;
done:
    window_out(L);
    while (L.st != S_DONE) slow_work<true>(L, P, ctx, s_bend);
}

template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 20 / WARPS) k_entropy(EntParams P) {
    // s_bend[b]: first scan position past band b; then the lanes' contexts,
    // context j of lane l of warp w at word (w * kCtxSlots + j) * 32 + l
    extern __shared__ uint32_t s_ent[];
    uint16_t *s_bend = reinterpret_cast<uint16_t *>(s_ent);
    if (threadIdx.x < 9) s_bend[threadIdx.x] = c_bend[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *ctx = s_ent + 8 + warp * kCtxSlots * 32 + lane;
    LaneState L;
    // warps 0..nsolo-1 of the grid: order entry `warp` on the warp's first
    // thread alone, then the queue
    const int gwarp = blockIdx.x * WARPS + warp;
    if (gwarp < P.nsolo) {
        if (lane == 0) {
            memset(&L, 0, sizeof L);
            lane_begin(L, P, ctx, s_bend, (int)P.order[gwarp]);
            solo_entropy(L, P, ctx, s_bend);
            lane_finish(L, P);
        }
        __syncwarp();
    }
    EntParams F = P;   // the rest of the order, one lane per block
    F.order = P.order ? P.order + P.nsolo : nullptr;
    F.ncoded = P.ncoded - P.nsolo;
    const int gtid = (int)(blockIdx.x * blockDim.x + threadIdx.x) - 32 * P.nsolo;
    run_lanes(L, F, ctx, s_bend, gtid, (int)(gridDim.x * blockDim.x) - 32 * P.nsolo, [](int) {});
}
// dynamic shared memory of k_entropy<W>
constexpr size_t entropy_smem(int warps) { return 32 + sizeof(uint32_t) * kCtxSlots * 32 * (size_t)warps; }

// The entropy stage with every block on a single thread: each warp's first
// thread decodes blocks of the order one after another (its own entry first,
// then claims from the counter), the other 31 threads leave at once. First
// entries go to the CTAs in turn, and the second half of the CTAs starts at its
// third warp, so that a small batch spreads over all SMs and their schedulers
// (with entries 0..15 on the first CTA and so on, the stage at q=6 took 16 %
// longer at 1 chunk and 15 % at 2). A block then costs a few times fewer cycles
// per bin than as a lane of k_entropy, at several times the issue slots per bin,
// which pays where a batch is too
// small to fill the machine and its longest blocks set the stage's time. The
// threads' contexts share one 32-column region of shared memory (column =
// warp index), conflict-free like k_entropy's. Two CTAs of 16 warps per SM
// fit the register file at 64 registers a thread.
constexpr int kSoloWarps = 16;
__global__ void __launch_bounds__(kSoloWarps * 32, 2) k_entropy_solo(EntParams P) {
    __shared__ uint32_t s_ctx[kCtxSlots * 32];
    __shared__ uint16_t s_bend[9];
    if (threadIdx.x < 9) s_bend[threadIdx.x] = c_bend[threadIdx.x];
    __syncthreads();
    if (threadIdx.x & 31) return;
    const int warp = threadIdx.x >> 5;
    uint32_t *ctx = s_ctx + warp;
    const int nwarps = gridDim.x * kSoloWarps;
    const int turn = (warp + (2 * blockIdx.x >= gridDim.x ? kSoloWarps - 2 : 0)) % kSoloWarps;
    for (int j = blockIdx.x + turn * gridDim.x; j < P.ncoded; j = nwarps + (int)atomicAdd(P.counter, 1u)) {
        LaneState L;
        memset(&L, 0, sizeof L);
        lane_begin(L, P, ctx, s_bend, P.order ? (int)P.order[j] : j);
        solo_entropy(L, P, ctx, s_bend);
        lane_finish(L, P);
    }
}

// ---------------------------------------------------------------- stage 2
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }

// acc + w*v per lane with two roundings (see mcb_f32x2.cuh)
__device__ __forceinline__ float2 madd2(float2 acc, float2 w, float2 v) {
    const float2 p = mul2(w, v);
    return make_float2(__fadd_rn(acc.x, p.x), __fadd_rn(acc.y, p.y));
}
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// 4 adjacent lines x 2 outputs (m, m+1): even-k and odd-k halves, each a
// sequential sum over ascending k (src/mc_codec_float.h:102-104). in[k*ks]
// holds the 4 lines' k-th inputs, W[k*16 + m/2] = {c[k][m], c[k][m], c[k][m+1], c[k][m+1]}.
struct Acc4 { float2 e0a, e0b, e1a, e1b, o0a, o0b, o1a, o1b; };
// From four terms on, each sum starts from its first product rather than
// from 0 plus it: equal, except that 0 + (-0) is +0 where the product alone
// keeps -0; a zero of either sign stays a zero through every later add and
// multiply and rounds to the same voxel, and every nonzero sum is unchanged.
// With fewer terms a half-sum could be a bare product, which the packed e +/- o
// below would take into one fused rounding (see madd2), so those start at 0.
__device__ __forceinline__ Acc4 lines4(const float4 *in, int ks, int K, const float4 *W, int mh) {
    Acc4 a;
    int k;
    if (K >= 4) {
        const float4 v = in[0], w = W[mh];
        const float2 w0 = lo2(w), w1 = hi2(w);
        a.e0a = mul2(w0, lo2(v)); a.e0b = mul2(w0, hi2(v));
        a.e1a = mul2(w1, lo2(v)); a.e1b = mul2(w1, hi2(v));
        const float4 u = in[ks], x = W[8 + mh];
        const float2 x0 = lo2(x), x1 = hi2(x);
        a.o0a = mul2(x0, lo2(u)); a.o0b = mul2(x0, hi2(u));
        a.o1a = mul2(x1, lo2(u)); a.o1b = mul2(x1, hi2(u));
        k = 2;
    } else {
        const float2 z = make_float2(0.f, 0.f);
        a.e0a = a.e0b = a.e1a = a.e1b = a.o0a = a.o0b = a.o1a = a.o1b = z;
        k = 0;
    }
    // (even, odd) pairs of k without a per-step guard, then the last even k
#pragma unroll 2
    for (; k + 1 < K; k += 2) {
        const float4 v = in[k * ks], w = W[k * 8 + mh];
        const float2 w0 = lo2(w), w1 = hi2(w);
        a.e0a = madd2(a.e0a, w0, lo2(v)); a.e0b = madd2(a.e0b, w0, hi2(v));
        a.e1a = madd2(a.e1a, w1, lo2(v)); a.e1b = madd2(a.e1b, w1, hi2(v));
        const float4 u = in[(k + 1) * ks], x = W[(k + 1) * 8 + mh];
        const float2 x0 = lo2(x), x1 = hi2(x);
        a.o0a = madd2(a.o0a, x0, lo2(u)); a.o0b = madd2(a.o0b, x0, hi2(u));
        a.o1a = madd2(a.o1a, x1, lo2(u)); a.o1b = madd2(a.o1b, x1, hi2(u));
    }
    if (k < K) {
        const float4 v = in[k * ks], w = W[k * 8 + mh];
        const float2 w0 = lo2(w), w1 = hi2(w);
        a.e0a = madd2(a.e0a, w0, lo2(v)); a.e0b = madd2(a.e0b, w0, hi2(v));
        a.e1a = madd2(a.e1a, w1, lo2(v)); a.e1b = madd2(a.e1b, w1, hi2(v));
    }
    return a;
}

// Entry j of a block. CG: read through L2 only (__ldcg), for entries that
// another SM may have written during this kernel (the fused decode): a line
// this SM cached earlier for a neighbouring block must not be reused.
template <bool CG>
__device__ __forceinline__ uint32_t entry_at(const RecParams &P, uint64_t base, uint32_t cap, uint32_t ovf, uint32_t j) {
    if (j < cap) return CG ? __ldcg(P.arena + base + j) : P.arena[base + j];
    if (ovf == 0xFFFFFFFFu) return 0u;
    return CG ? __ldcg(P.pool + ovf + (j - cap)) : P.pool[ovf + (j - cap)];
}
template <bool CG>
__device__ __forceinline__ EntHdr load_hdr(const EntHdr *h) {
    if (!CG) return *h;
    const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(h));
    EntHdr r;
    memcpy(&r, &v, sizeof r);
    return r;
}

// (int)lrintf(v) + dc clamped to u8 (src/mc_codec.c:766-769). Adding 1.5*2^23
// rounds to an integer half-to-even for |v| < 2^22, which is exactly lrintf;
// larger values (only from corrupt streams) take the 64-bit conversion.
__device__ __forceinline__ uint32_t to_u8(float v, int dc) {
    int r;
    if (fabsf(v) < 4194304.0f) {
        r = __float_as_int(fadd(v, 12582912.0f)) - 0x4B400000;
    } else {
        r = (int)(uint32_t)(unsigned long long)__float2ll_rn(v);
    }
    const int s = r + dc;
    return (uint32_t)(s < 0 ? 0 : s > 255 ? 255 : s);
}
// four voxels (x, x+1 | x+2, x+3) -> little-endian u8x4
__device__ __forceinline__ uint32_t pack4(float2 a, float2 b, int dc) {
    return to_u8(a.x, dc) | (to_u8(a.y, dc) << 8) | (to_u8(b.x, dc) << 16) | (to_u8(b.y, dc) << 24);
}
// The same for a block whose voxels are all known to satisfy |v| < 2^21:
// round half to even by the magic add, + dc, and a saturating pack (four
// ints to u8, s0 in the low byte).
__device__ __forceinline__ int rint_dc(float v, int dc) {
    return __float_as_int(fadd(v, 12582912.0f)) - 0x4B400000 + dc;
}
__device__ __forceinline__ uint32_t pack4_fast(float2 a, float2 b, int dc) {
    uint32_t t, d;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, 0;" : "=r"(t) : "r"(rint_dc(b.y, dc)), "r"(rint_dc(b.x, dc)));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(rint_dc(a.y, dc)), "r"(rint_dc(a.x, dc)), "r"(t));
    return d;
}
// Every output voxel is a sum of at most 4096 terms coef * c[kz][z]c[ky][y]c[kx][x]
// with |c| <= sqrt(2/16), so |v| <= L1(coef) * 0.0442; below this L1 norm
// (with a factor-2 margin for rounding) every voxel takes the fast rounding.
constexpr float kFastL1 = 2097152.0f / 0.04419417f;

// Shared-memory layouts. A (pass-1 output) rows of 16 floats are padded to
// kRowF so that the lanes of a warp that write the four outputs
// (m, m+1, 15-m, 14-m) of a line hit different banks. B (pass-2 output) rows
// are not padded: float4 group g of row y (in every cz plane) sits at group
// g ^ bswz(y), so pass-3 loads (rows y, y+1 of one plane) are conflict-free
// and pass-2 stores at most 2-way, in 4 KB less shared memory per CTA.
constexpr int kRowF = 20;            // A rows of 16 floats
constexpr int kRowB = 16;            // B rows
constexpr int kPlaneB = 16 * kRowB;  // one cz plane of B
__device__ __forceinline__ int bswz(int y) { return (y >> 1) & 3; }
// The coefficient box in B: coefficient (cz, cy, cx) at cz*kBoxPlane + cx*16 + cy.
// For one (cz, cx) the 16 cy values are contiguous, so pass 1 reads the k-th
// inputs of 4 adjacent x-lines as one float4; planes are padded by 16 floats
// so that the two planes a warp reads sit in different banks. B holds kBoxB
// floats (the pass-2 output uses the first 16 * kPlaneB).
constexpr int kBoxPlane = 16 * 16 + 16;
constexpr int kBoxB = 16 * kBoxPlane;
constexpr int kStageZ = 272;         // stage: one z slice of 16 rows of 16 bytes
constexpr int kStageBytes = 16 * kStageZ;

// Per-CTA state of the block being reconstructed: extents and L1 norm. Both
// are zero when a block starts, like the coefficient box (rec_init, then
// every block puts them back).
__shared__ int s_rec_ext[3];
__shared__ float s_rec_l1;

// Before a CTA's first block: an all-zero coefficient box, zero extents and
// L1 norm. The caller synchronises before the first block.
__device__ __forceinline__ void rec_init(float *sB) {
    for (int i = threadIdx.x; i < kBoxB / 4; i += blockDim.x)
        reinterpret_cast<float4 *>(sB)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (threadIdx.x < 3) s_rec_ext[threadIdx.x] = 0;
    if (threadIdx.x == 3) s_rec_l1 = 0.0f;
}

// Reconstruct one block into a stage (z slices of kStageZ bytes). Thread t owns the
// output pair (m, m+1) = 2*(t&3) of every line it touches; its cosine weights
// come from the shared table W.
// On entry the coefficient box in sB, s_rec_ext and s_rec_l1 are zero; the
// block leaves them zero again.
template <bool CG>
__device__ __forceinline__ void reconstruct_block(const RecParams &P, int item, float *sA, float *sB,
                                                  uint8_t *stage, const float4 *W) {
    const int tid = threadIdx.x;
    const int m = (tid & 3) * 2;
    const DecItem it = P.items[item];
    const EntHdr h = load_hdr<CG>(P.hdr + item);
    const uint64_t base = P.base[item];
    const uint32_t cap = entry_cap(it.len);
    // the header comes from k_entropy; the guards keep every index below
    // inside shared memory whatever its contents
    const bool sane = h.nnz <= kN3 && h.ncorr <= kN3;
    const int dc = it.len && sane ? h.dc : 0;
    const int nnz = it.len && sane ? h.nnz : 0;
    const int ncorr = it.len && sane ? h.ncorr : 0;
    int E = 0;   // cz planes of the box this block wrote

    if (nnz == 0) {
        // constant block (src/mc_codec.c:757-759) or absent block (zeros)
        const uint32_t w = (uint32_t)dc * 0x01010101u;
        const uint4 v = make_uint4(w, w, w, w);
        for (int i = tid; i < kStageBytes / 16; i += 128) reinterpret_cast<uint4 *>(stage)[i] = v;
    } else {
        // One pass over the entries: the extents of the coefficient box
        // (largest cz, cy, cx of any entry, src/mc_codec.c:371-372), the
        // dequantised coefficients (src/mc_codec_float.h:185-190) straight
        // into the zeroed box, and the L1 norm. Four entries per thread are
        // in flight at a time.
        const QTab &qt = P.qtab[it.qslot];
        int mz = 0, my = 0, mx = 0;
        float l1 = 0.0f;
        for (int j0 = tid; j0 < nnz; j0 += 512) {
            uint32_t e[4], ix[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) e[k] = j0 + 128 * k < nnz ? entry_at<CG>(P, base, cap, h.ovf, j0 + 128 * k) : 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) ix[k] = j0 + 128 * k < nnz ? __ldg(P.scan + (e[k] & 0xFFFu)) & 0xFFFu : 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (j0 + 128 * k >= nnz) break;
                const int idx = (int)ix[k];
                const int cz = idx >> 8, cy = (idx >> 4) & 15, cx = idx & 15;
                mz = max(mz, cz);
                my = max(my, cy);
                mx = max(mx, cx);
                const int lv = (int16_t)(e[k] >> 16);
                if (lv) {
                    const int f = cz + cy + cx;
                    const float a = (float)(lv < 0 ? -lv : lv);
                    const float r = fadd(fadd(fmul(fsub(a, 1.0f), qt.step[f]), qt.dz8[f]), qt.dz4[f]);
                    sB[cz * kBoxPlane + cx * 16 + cy] = lv < 0 ? -r : r;
                    l1 = fadd(l1, r);
                }
            }
        }
        // one shared-memory atomic per warp and value; the L1 norm only
        // bounds the voxels, so any summation order will do
        mz = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)mz);
        my = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)my);
        mx = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)mx);
        for (int o = 16; o > 0; o >>= 1) l1 += __shfl_xor_sync(0xFFFFFFFFu, l1, o);
        if ((tid & 31) == 0) {
            atomicMax(&s_rec_ext[0], mz);
            atomicMax(&s_rec_ext[1], my);
            atomicMax(&s_rec_ext[2], mx);
            atomicAdd(&s_rec_l1, l1);
        }
        __syncthreads();
        E = s_rec_ext[0] + 1;
        const int Y = s_rec_ext[1] + 1, X = s_rec_ext[2] + 1;
        const bool fast = s_rec_l1 < kFastL1;
        // pass 1: lines along x for 4 adjacent cy at once, box[cz][k][cy..cy+3]
        // -> A[cz*Y + cy][x]. Group g of plane cz holds lines cy = 4g..4g+3;
        // lines at cy >= Y are zero and not stored. gi < 64, so
        // gi * ceil(2^16 / G) >> 16 is exactly gi / G.
        const int mh = tid & 3;   // this thread's output pair (m, m+1) = (2mh, 2mh+1)
        const int G = (Y + 3) >> 2;
        const int invG = (65536 + G - 1) / G;
        for (int t = tid; t < E * G * 4; t += 128) {
            const int gi = t >> 2;
            const int cz = (gi * invG) >> 16;
            const int cy0 = (gi - cz * G) << 2;
            const Acc4 a = lines4(reinterpret_cast<const float4 *>(sB + cz * kBoxPlane + cy0), 4, X, W, mh);
            // line i of the group: outputs m, m+1 (e + o) and 15-m, 14-m (e - o)
            const float2 p0 = add2(a.e0a, a.o0a), p1 = add2(a.e0b, a.o0b);
            const float2 q0 = add2(a.e1a, a.o1a), q1 = add2(a.e1b, a.o1b);
            const float2 r0 = sub2(a.e0a, a.o0a), r1 = sub2(a.e0b, a.o0b);
            const float2 s0 = sub2(a.e1a, a.o1a), s1 = sub2(a.e1b, a.o1b);
            float *out = sA + (cz * Y + cy0) * kRowF;
            const int nl = min(Y - cy0, 4);
            *reinterpret_cast<float2 *>(out + m) = make_float2(p0.x, q0.x);
            *reinterpret_cast<float2 *>(out + 14 - m) = make_float2(s0.x, r0.x);
            if (nl > 1) {
                *reinterpret_cast<float2 *>(out + kRowF + m) = make_float2(p0.y, q0.y);
                *reinterpret_cast<float2 *>(out + kRowF + 14 - m) = make_float2(s0.y, r0.y);
            }
            if (nl > 2) {
                *reinterpret_cast<float2 *>(out + 2 * kRowF + m) = make_float2(p1.x, q1.x);
                *reinterpret_cast<float2 *>(out + 2 * kRowF + 14 - m) = make_float2(s1.x, r1.x);
            }
            if (nl > 3) {
                *reinterpret_cast<float2 *>(out + 3 * kRowF + m) = make_float2(p1.y, q1.y);
                *reinterpret_cast<float2 *>(out + 3 * kRowF + 14 - m) = make_float2(s1.y, r1.y);
            }
        }
        __syncthreads();
        // every thread has read the extents and the norm: zero for the next block
        if (tid < 3) s_rec_ext[tid] = 0;
        if (tid == 3) s_rec_l1 = 0.0f;
        // pass 2: lines along y for 4 adjacent x at once, A[cz][k][x..x+3] -> B[cz][y][x..x+3]
        for (int t = tid; t < E * 16; t += 128) {
            const int xg = (t >> 2) & 3, cz = t >> 4;
            const Acc4 a = lines4(reinterpret_cast<const float4 *>(sA + cz * Y * kRowF + xg * 4), kRowF / 4, Y,
                                  W, mh);
            // rows m, m+1 swizzle by bswz(m) = mh, rows 15-m, 14-m by 3 - mh
            float *ob = sB + cz * kPlaneB;
            const int ga = (xg ^ mh) << 2, gb = (xg ^ (3 - mh)) << 2;
            const float2 p0 = add2(a.e0a, a.o0a), p1 = add2(a.e0b, a.o0b);
            const float2 q0 = add2(a.e1a, a.o1a), q1 = add2(a.e1b, a.o1b);
            const float2 r0 = sub2(a.e0a, a.o0a), r1 = sub2(a.e0b, a.o0b);
            const float2 s0 = sub2(a.e1a, a.o1a), s1 = sub2(a.e1b, a.o1b);
            *reinterpret_cast<float4 *>(ob + m * kRowB + ga) = make_float4(p0.x, p0.y, p1.x, p1.y);
            *reinterpret_cast<float4 *>(ob + (m + 1) * kRowB + ga) = make_float4(q0.x, q0.y, q1.x, q1.y);
            *reinterpret_cast<float4 *>(ob + (15 - m) * kRowB + gb) = make_float4(r0.x, r0.y, r1.x, r1.y);
            *reinterpret_cast<float4 *>(ob + (14 - m) * kRowB + gb) = make_float4(s0.x, s0.y, s1.x, s1.y);
        }
        __syncthreads();
        // pass 3: lines along z for 4 adjacent x, B[k][y][x..x+3] -> voxels
        for (int t = tid; t < 256; t += 128) {
            const int xg = (t >> 2) & 3, y = t >> 4;
            const Acc4 a = lines4(reinterpret_cast<const float4 *>(sB + y * kRowB + ((xg ^ bswz(y)) << 2)), kPlaneB / 4,
                                  E, W, mh);
            uint32_t *row = reinterpret_cast<uint32_t *>(stage + y * 16 + xg * 4);
            constexpr int Z = kStageZ / 4;
            if (fast) {
                row[m * Z] = pack4_fast(add2(a.e0a, a.o0a), add2(a.e0b, a.o0b), dc);
                row[(m + 1) * Z] = pack4_fast(add2(a.e1a, a.o1a), add2(a.e1b, a.o1b), dc);
                row[(15 - m) * Z] = pack4_fast(sub2(a.e0a, a.o0a), sub2(a.e0b, a.o0b), dc);
                row[(14 - m) * Z] = pack4_fast(sub2(a.e1a, a.o1a), sub2(a.e1b, a.o1b), dc);
            } else {
                row[m * Z] = pack4(add2(a.e0a, a.o0a), add2(a.e0b, a.o0b), dc);
                row[(m + 1) * Z] = pack4(add2(a.e1a, a.o1a), add2(a.e1b, a.o1b), dc);
                row[(15 - m) * Z] = pack4(sub2(a.e0a, a.o0a), sub2(a.e0b, a.o0b), dc);
                row[(14 - m) * Z] = pack4(sub2(a.e1a, a.o1a), sub2(a.e1b, a.o1b), dc);
            }
        }
    }
    __syncthreads();
    // the box planes this block wrote (coefficients and pass-2 output) back to zero
    for (int i = tid; i < E * (kBoxPlane / 4); i += 128)
        reinterpret_cast<float4 *>(sB)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ncorr && tid == 0) {
        // corrections in stream order: a position may repeat, each
        // application clamps (src/mc_codec.c:775-781)
        for (int c = 0; c < ncorr; ++c) {
            const uint32_t pos = entry_at<CG>(P, base, cap, h.ovf, nnz + 2 * c);
            const uint32_t d = entry_at<CG>(P, base, cap, h.ovf, nnz + 2 * c + 1);
            if (pos >= (uint32_t)kN3) break;
            uint8_t &vox = stage[(pos >> 8) * kStageZ + (pos & 255)];
            const int v = (int)((uint32_t)vox + d);
            vox = (uint8_t)(v < 0 ? 0 : v > 255 ? 255 : v);
        }
    }
    __syncthreads();
}

struct StageRows {   // z slices of kStageZ bytes
    const uint8_t *p;
    __device__ const uint8_t *operator()(int z, int y) const { return p + z * kStageZ + y * 16; }
};
// Clipped store of one staged block (row (z, y) at stage_row(z, y)) by nthr
// threads, this one thread `tid` of them: one 16-voxel row per thread step.
template <class Row>
__device__ __forceinline__ void store_block(const DecItem &it, Row stage_row, int tid, int nthr) {
    uint8_t *dst = reinterpret_cast<uint8_t *>(it.dst);
    if (it.clip_lo == kClipFullLo && it.clip_hi == kClipFullHi) {
        for (int r = tid; r < 256; r += nthr) {
            const int z = r >> 4, y = r & 15;
            store_row16(dst + z * it.sz + y * it.sy, *reinterpret_cast<const uint4 *>(stage_row(z, y)));
        }
        return;
    }
    const int z0 = it.clip_lo >> 8, y0 = (it.clip_lo >> 4) & 15, x0 = it.clip_lo & 15;
    const int z1 = it.clip_hi >> 8, y1 = (it.clip_hi >> 4) & 15, x1 = it.clip_hi & 15;
    const int ny = y1 - y0 + 1, nrows = (z1 - z0 + 1) * ny;
    for (int r = tid; r < nrows; r += nthr) {
        const int z = z0 + r / ny, y = y0 + r % ny;
        uint8_t *row = dst + z * it.sz + y * it.sy;
        const uint8_t *srow = stage_row(z, y);
        if (x0 == 0 && x1 == 15) {
            store_row16(row, *reinterpret_cast<const uint4 *>(srow));
        } else {
            for (int x = x0; x <= x1; ++x) row[x] = srow[x];
        }
    }
}

// Two blocks that sit side by side in x in the same output: one 32-byte
// row per step, so every DRAM sector is written whole (16-byte halves of a
// sector written apart cost a read-modify-write).
__device__ __forceinline__ bool pairable(const DecItem &a, const DecItem &b) {
    return a.clip_lo == kClipFullLo && a.clip_hi == kClipFullHi && b.clip_lo == kClipFullLo &&
           b.clip_hi == kClipFullHi && b.dst == a.dst + 16 && a.sz == b.sz && a.sy == b.sy && (a.dst & 31) == 0 &&
           (a.sy & 31) == 0 && (a.sz & 31) == 0;
}

// One line-group step of the warp-wide passes: 4 adjacent lines x 2 outputs,
// like lines4, with packed adds. A product must not reach a packed add inside
// one basic block (see madd2), so the loop is software-pipelined: an iteration
// adds the products of the previous one and computes its own, and the products
// pass through the loop's back edge. #pragma unroll 1 keeps it so. K is even
// and at least 4: a sum over fewer inputs takes zeros up to that, which add
// +/-0, and starts from its first products (see lines4).
__device__ __forceinline__ void mul_even(Acc4 &q, float4 v, float4 w) {
    q.e0a = mul2(lo2(w), lo2(v)); q.e0b = mul2(lo2(w), hi2(v));
    q.e1a = mul2(hi2(w), lo2(v)); q.e1b = mul2(hi2(w), hi2(v));
}
__device__ __forceinline__ void mul_odd(Acc4 &q, float4 v, float4 w) {
    q.o0a = mul2(lo2(w), lo2(v)); q.o0b = mul2(lo2(w), hi2(v));
    q.o1a = mul2(hi2(w), lo2(v)); q.o1b = mul2(hi2(w), hi2(v));
}
__device__ __forceinline__ void add_pending(Acc4 &a, const Acc4 &q) {
    a.e0a = add2(a.e0a, q.e0a); a.e0b = add2(a.e0b, q.e0b);
    a.e1a = add2(a.e1a, q.e1a); a.e1b = add2(a.e1b, q.e1b);
    a.o0a = add2(a.o0a, q.o0a); a.o0b = add2(a.o0b, q.o0b);
    a.o1a = add2(a.o1a, q.o1a); a.o1b = add2(a.o1b, q.o1b);
}
__device__ __forceinline__ Acc4 lines4p(const float4 *in, int ks, int K, const float4 *W) {
    Acc4 a, q;
    mul_even(a, in[0], W[0]);
    mul_odd(a, in[ks], W[8]);
    mul_even(q, in[2 * ks], W[16]);
    mul_odd(q, in[3 * ks], W[24]);
    if (K > 4) {
        // inputs and weights are loaded an iteration ahead
        float4 v = in[4 * ks], w = W[32], u = in[5 * ks], x = W[40];
#pragma unroll 1
        for (int k = 6;; k += 2) {
            add_pending(a, q);
            mul_even(q, v, w);
            mul_odd(q, u, x);
            if (k >= K) break;
            in += 2 * ks;
            W += 16;
            v = in[4 * ks]; w = W[32]; u = in[5 * ks]; x = W[40];
        }
    }
    add_pending(a, q);
    return a;
}

// Four voxels of a fast block: x, x + 1 | x + 2, x + 3 rounded by a packed magic add.
__device__ __forceinline__ uint32_t pack4_fast2(float2 a, float2 b, int bias) {
    const float2 mg = make_float2(12582912.0f, 12582912.0f);
    const float2 fa = add2(a, mg), fb = add2(b, mg);
    uint32_t t, d;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, 0;" : "=r"(t) : "r"(__float_as_int(fb.y) + bias), "r"(__float_as_int(fb.x) + bias));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(__float_as_int(fa.y) + bias), "r"(__float_as_int(fa.x) + bias), "r"(t));
    return d;
}

// The same for voxels of any size (corrupt streams only).
__device__ __noinline__ uint32_t pack4_slow(float2 a, float2 b, int dc) { return pack4(a, b, dc); }

// Shared memory of k_reconstruct: the weights ([k][m/2], as c_cos2), the
// coefficient box, whose planes become the pass-2 output in place (kBoxPlane
// floats each), and for each of the two warps the pass-1 output of the planes it
// works on, later the stage of its half of the rows (warp w: y >> 3 == w,
// [z][y & 7][x]).
struct RecSmem {
    float4 W[16 * 8];
    float box[kBoxB];
    float a[2][32 * kRowF];
    uint32_t ext[2];    // per warp: largest cz << 8 | cy << 4 | cx, each coordinate on its own
    float l1[2];
};
constexpr int kStageHalf = sizeof(float) * 32 * kRowF;   // bytes from row 0's slice to row 8's
__device__ __forceinline__ int stage_at(int z, int y) { return (y >> 3) * kStageHalf + z * 128 + (y & 7) * 16; }

// Pass 3 of the warp's 32 line groups, outputs m = 4 half + j and 15 - m of 4
// adjacent z-lines: in[k * kBoxPlane/4] the k-th inputs; the four voxels at z =
// m to word j, at z = 15 - m to word 4 + j.
struct Acc8 { float2 ea[4], eb[4], oa[4], ob[4]; };   // even and odd sums, lines 0-1 and 2-3
__device__ __forceinline__ void mul8(float2 *a, float2 *b, float4 v, const float4 *w) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float4 c = w[j];
        a[2 * j] = mul2(lo2(c), lo2(v)); b[2 * j] = mul2(lo2(c), hi2(v));
        a[2 * j + 1] = mul2(hi2(c), lo2(v)); b[2 * j + 1] = mul2(hi2(c), hi2(v));
    }
}
__device__ __forceinline__ void add_pending8(Acc8 &a, const Acc8 &q) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        a.ea[j] = add2(a.ea[j], q.ea[j]); a.eb[j] = add2(a.eb[j], q.eb[j]);
        a.oa[j] = add2(a.oa[j], q.oa[j]); a.ob[j] = add2(a.ob[j], q.ob[j]);
    }
}
__device__ __forceinline__ void pass3(const float4 *in, int E, int half, int dc, bool fast, uint32_t word[8]) {
    constexpr int ks = kBoxPlane / 4;
    const float4 *w = c_cos2[0] + 2 * half;
    Acc8 a, q;
    mul8(a.ea, a.eb, in[0], w);
    mul8(a.oa, a.ob, in[ks], w + 8);
    mul8(q.ea, q.eb, in[2 * ks], w + 16);
    mul8(q.oa, q.ob, in[3 * ks], w + 24);
    if (E > 4) {
        float4 v = in[4 * ks], u = in[5 * ks];   // loaded an iteration ahead
#pragma unroll 1
        for (int k = 6;; k += 2) {
            add_pending8(a, q);
            w += 16;
            mul8(q.ea, q.eb, v, w + 16);
            mul8(q.oa, q.ob, u, w + 24);
            if (k >= E) break;
            in += 2 * ks;
            v = in[4 * ks];
            u = in[5 * ks];
        }
    }
    add_pending8(a, q);
    const int bias = dc - 0x4B400000;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 p0 = add2(a.ea[j], a.oa[j]), p1 = add2(a.eb[j], a.ob[j]);
        const float2 q0 = sub2(a.ea[j], a.oa[j]), q1 = sub2(a.eb[j], a.ob[j]);
        word[j] = fast ? pack4_fast2(p0, p1, bias) : pack4_slow(p0, p1, dc);
        word[4 + j] = fast ? pack4_fast2(q0, q1, bias) : pack4_slow(q0, q1, dc);
    }
}

// The reconstruction stage of a batch: two warps per block. The first two
// passes go a few planes at a time (as many as fill a warp's 32 lanes with pass-1
// groups), plane groups in turn to the two warps, each through its own small
// pass-1 buffer, and leave their output in the box's own planes. So a block
// needs 25 KB of shared memory instead of the 43 KB of the CTA-wide routine
// (reconstruct_block, for the kernels that decode few blocks or hold one CTA's
// memory for both stages): nine blocks at a time on an SM instead of five, with
// half the warps issuing the work outside the transforms (headers, entry
// scatter, reductions, stores). The last pass gives a lane 8 of a line group's 16
// outputs at a time and takes its weights from constant memory by a warp-uniform
// index; all sums are packed adds (see lines4p).
// What bounds it: latency, at 18 warps an SM and 0.43 instructions a cycle and
// scheduler (3130 a block at q=6, 3960 before). 64 chunks at q=6 1.55 ms, at q=12
// 1.15 (1.61 and 1.16 without the pairs of launch_reconstruct); with reconstruct_block on
// 4-warp CTAs 1.87 and 1.51. Tried and dropped:
// one warp per block without barriers (10 warps an SM, 1.87), pairs of blocks
// with 32-byte row stores (16 registers held over a block, spills: 1.70).
__global__ void __launch_bounds__(64, 9) k_reconstruct(RecParams P) {
    extern __shared__ __align__(16) uint8_t s_rec[];
    RecSmem &S = *reinterpret_cast<RecSmem *>(s_rec);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < 16 * 8; i += 64) S.W[i] = c_cos2[i >> 3][i & 7];
    for (int i = tid; i < kBoxB / 4; i += 64) reinterpret_cast<float4 *>(S.box)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    const int nb = gridDim.x;
    // blocks dealt to the CTAs in turn; in a large batch two adjacent ones at a
    // time, so that the two halves of a 32-byte sector of the output are written
    // soon after one another (see launch_reconstruct)
    auto after = [&P, nb](int j) { return !P.pairs ? j + nb : (j & 1 ? j + 2 * nb - 1 : j + 1); };
    const int mh = lane & 3, m = mh * 2;
    float *const A = S.a[warp];
    uint8_t *const stage = reinterpret_cast<uint8_t *>(S.a);
    // the next block's header, entry offset and payload length, loaded while
    // this one is transformed; then its first 256 entries, while pass 3 runs
    int i = P.pairs ? 2 * blockIdx.x : blockIdx.x;
    EntHdr hn = {};
    uint64_t basen = 0;
    uint32_t lenn = 0, slotn = 0, en[4] = {0, 0, 0, 0};
    auto next_head = [&](int j) {
        const int item = P.idx ? (int)__ldg(P.idx + j) : j;
        hn = load_hdr<false>(P.hdr + item);
        basen = P.base[item];
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(&P.items[item].len));
        lenn = v.x;
        slotn = v.y & 0xFFFFu;
    };
    auto next_entries = [&]() {
        const int lim = lenn && hn.nnz <= kN3 ? min((int)hn.nnz, (int)entry_cap(lenn)) : 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (tid + 64 * k < lim) en[k] = P.arena[basen + tid + 64 * k];
    };
    if (i < P.n) {
        next_head(i);
        next_entries();
    }
    for (int nx; i < P.n; i = nx) {
        nx = after(i);
        const int item = P.idx ? (int)__ldg(P.idx + i) : i;
        const DecItem it = P.items[item];
        const EntHdr h = hn;
        const uint64_t base = basen;
        const uint32_t len = lenn, cap = entry_cap(lenn), nslot = slotn;
        if (nx < P.n) next_head(nx);
        // the header comes from k_entropy; the guards keep every index below
        // inside shared memory whatever its contents
        const bool sane = h.nnz <= kN3 && h.ncorr <= kN3;
        const int dc = len && sane ? h.dc : 0;
        const int nnz = len && sane ? h.nnz : 0;
        const int ncorr = len && sane ? h.ncorr : 0;
        int E = 0;   // box planes that this block wrote
        if (nnz == 0) {
            // constant block (src/mc_codec.c:757-759) or absent block (zeros)
            const uint32_t w = (uint32_t)dc * 0x01010101u;
            if (!ncorr && it.clip_lo == kClipFullLo && it.clip_hi == kClipFullHi) {
                uint8_t *dst = reinterpret_cast<uint8_t *>(it.dst) + (tid & 15) * it.sy + (tid >> 4) * it.sz;
#pragma unroll
                for (int j = 0; j < 4; ++j) store_row16(dst + 4 * j * it.sz, make_uint4(w, w, w, w));
                if (nx < P.n) next_entries();
                continue;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                reinterpret_cast<uint4 *>(stage + warp * kStageHalf)[j * 32 + lane] = make_uint4(w, w, w, w);
            if (nx < P.n) next_entries();
        } else {
            // one pass over the entries, as in reconstruct_block
            const QTab &qt = P.qtab[nslot];
            int mz = 0, my = 0, mx = 0;
            float l1 = 0.0f;
            for (int j0 = tid; j0 < nnz; j0 += 256) {
                uint32_t e[4], ix[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int j = j0 + 64 * k;
                    e[k] = j < nnz ? (j0 < 64 && j < (int)cap ? en[k] : entry_at<false>(P, base, cap, h.ovf, j)) : 0u;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) ix[k] = j0 + 64 * k < nnz ? __ldg(P.scan + (e[k] & 0xFFFu)) & 0xFFFu : 0u;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (j0 + 64 * k >= nnz) break;
                    const int idx = (int)ix[k];
                    const int cz = idx >> 8, cy = (idx >> 4) & 15, cx = idx & 15;
                    mz = max(mz, cz);
                    my = max(my, cy);
                    mx = max(mx, cx);
                    const int lv = (int16_t)(e[k] >> 16);
                    if (lv) {
                        const int f = cz + cy + cx;
                        const float a = (float)(lv < 0 ? -lv : lv);
                        const float r = fadd(fadd(fmul(fsub(a, 1.0f), qt.step[f]), qt.dz8[f]), qt.dz4[f]);
                        S.box[cz * kBoxPlane + cx * 16 + cy] = lv < 0 ? -r : r;
                        l1 = fadd(l1, r);
                    }
                }
            }
            mz = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)mz);
            my = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)my);
            mx = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)mx);
            for (int o = 16; o > 0; o >>= 1) l1 += __shfl_xor_sync(0xFFFFFFFFu, l1, o);
            if (lane == 0) {
                S.ext[warp] = (uint32_t)(mz << 8 | my << 4 | mx);
                S.l1[warp] = l1;
            }
            __syncthreads();   // the box is complete
            const uint32_t x0 = S.ext[0], x1 = S.ext[1];
            E = (int)max(x0 >> 8, x1 >> 8) + 1;
            const int Y = (int)max((x0 >> 4) & 15u, (x1 >> 4) & 15u) + 1, X = (int)max(x0 & 15u, x1 & 15u) + 1;
            const bool fast = S.l1[0] + S.l1[1] < kFastL1;
            // even numbers of inputs, at least 4 (see lines4p)
            const int Ee = max((E + 1) & ~1, 4), Ye = max((Y + 1) & ~1, 4), Xe = max((X + 1) & ~1, 4);
            // passes 1 and 2 over np planes at a time: G groups of 4 lines a plane
            const int G = (Y + 3) >> 2;
            const int np = G == 1 ? 8 : (G == 2 ? 4 : 2);
            const int gi = lane >> 2;
            const int lp = G == 1 ? gi : (G == 2 ? gi >> 1 : (G == 3 ? (gi * 11) >> 5 : gi >> 2));   // gi / G
            const int cy0 = (gi - lp * G) << 2;
            for (int c0 = warp * np; c0 < E; c0 += 2 * np) {
                if (lp < np && c0 + lp < E) {
                    const Acc4 a = lines4p(reinterpret_cast<const float4 *>(S.box + (c0 + lp) * kBoxPlane + cy0), 4, Xe,
                                           S.W + mh);
                    // line i of the group: outputs m, m+1 (e + o) and 15-m, 14-m (e - o)
                    const float2 p0 = add2(a.e0a, a.o0a), p1 = add2(a.e0b, a.o0b);
                    const float2 q0 = add2(a.e1a, a.o1a), q1 = add2(a.e1b, a.o1b);
                    const float2 r0 = sub2(a.e0a, a.o0a), r1 = sub2(a.e0b, a.o0b);
                    const float2 s0 = sub2(a.e1a, a.o1a), s1 = sub2(a.e1b, a.o1b);
                    float *out = A + (lp * (4 * G) + cy0) * kRowF;
                    *reinterpret_cast<float2 *>(out + m) = make_float2(p0.x, q0.x);
                    *reinterpret_cast<float2 *>(out + 14 - m) = make_float2(s0.x, r0.x);
                    *reinterpret_cast<float2 *>(out + kRowF + m) = make_float2(p0.y, q0.y);
                    *reinterpret_cast<float2 *>(out + kRowF + 14 - m) = make_float2(s0.y, r0.y);
                    *reinterpret_cast<float2 *>(out + 2 * kRowF + m) = make_float2(p1.x, q1.x);
                    *reinterpret_cast<float2 *>(out + 2 * kRowF + 14 - m) = make_float2(s1.x, r1.x);
                    *reinterpret_cast<float2 *>(out + 3 * kRowF + m) = make_float2(p1.y, q1.y);
                    *reinterpret_cast<float2 *>(out + 3 * kRowF + 14 - m) = make_float2(s1.y, r1.y);
                }
                __syncwarp();
                // A[plane][k][x..x+3] -> box plane [y][x..x+3], float4 groups swizzled (see bswz)
                const int npl = min(np, E - c0);
                for (int t = lane; t < npl * 16; t += 32) {
                    const int xg = (t >> 2) & 3, pl = t >> 4;
                    const Acc4 a = lines4p(reinterpret_cast<const float4 *>(A + pl * (4 * G) * kRowF + xg * 4), kRowF / 4,
                                           Ye, S.W + mh);
                    float *ob = S.box + (c0 + pl) * kBoxPlane;
                    const int ga = (xg ^ mh) << 2, gb = (xg ^ (3 - mh)) << 2;
                    const float2 p0 = add2(a.e0a, a.o0a), p1 = add2(a.e0b, a.o0b);
                    const float2 q0 = add2(a.e1a, a.o1a), q1 = add2(a.e1b, a.o1b);
                    const float2 r0 = sub2(a.e0a, a.o0a), r1 = sub2(a.e0b, a.o0b);
                    const float2 s0 = sub2(a.e1a, a.o1a), s1 = sub2(a.e1b, a.o1b);
                    *reinterpret_cast<float4 *>(ob + m * kRowB + ga) = make_float4(p0.x, p0.y, p1.x, p1.y);
                    *reinterpret_cast<float4 *>(ob + (m + 1) * kRowB + ga) = make_float4(q0.x, q0.y, q1.x, q1.y);
                    *reinterpret_cast<float4 *>(ob + (15 - m) * kRowB + gb) = make_float4(r0.x, r0.y, r1.x, r1.y);
                    *reinterpret_cast<float4 *>(ob + (14 - m) * kRowB + gb) = make_float4(s0.x, s0.y, s1.x, s1.y);
                }
                __syncwarp();
            }
            if (nx < P.n) next_entries();
            __syncthreads();   // every plane has its pass-2 output
            // pass 3: lane l of warp w takes the group (y, xg) = (8 w + (l >> 2), l & 3)
            const int y = 8 * warp + (lane >> 2);
            const float4 *in = reinterpret_cast<const float4 *>(S.box + y * kRowB + (((lane & 3) ^ bswz(y)) << 2));
            uint32_t *out = reinterpret_cast<uint32_t *>(A) + lane;   // the pass-1 buffer is free
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                uint32_t word[8];
                pass3(in, Ee, half, dc, fast, word);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    out[(4 * half + j) * 32] = word[j];
                    out[(15 - 4 * half - j) * 32] = word[4 + j];
                }
            }
        }
        if (ncorr) {
            __syncthreads();
            if (tid == 0) {
                // corrections in stream order: a position may repeat, each
                // application clamps (src/mc_codec.c:775-781)
                for (int c = 0; c < ncorr; ++c) {
                    const uint32_t pos = entry_at<false>(P, base, cap, h.ovf, nnz + 2 * c);
                    const uint32_t d = entry_at<false>(P, base, cap, h.ovf, nnz + 2 * c + 1);
                    if (pos >= (uint32_t)kN3) break;
                    uint8_t &vox = stage[stage_at(pos >> 8, (pos >> 4) & 15) + (pos & 15)];
                    const int v = (int)((uint32_t)vox + d);
                    vox = (uint8_t)(v < 0 ? 0 : v > 255 ? 255 : v);
                }
            }
            __syncthreads();
        }
        __syncwarp();
        if (it.clip_lo == kClipFullLo && it.clip_hi == kClipFullHi) {
            // each warp the rows it staged
            uint8_t *dst = reinterpret_cast<uint8_t *>(it.dst) + (8 * warp + (lane & 7)) * it.sy + (lane >> 3) * it.sz;
            const uint4 *row = reinterpret_cast<const uint4 *>(stage + warp * kStageHalf) + lane;
#pragma unroll
            for (int j = 0; j < 4; ++j) store_row16(dst + 4 * j * it.sz, row[32 * j]);
            __syncthreads();   // the box is read
        } else {
            __syncthreads();
            store_block(it, [&](int z, int yy) { return stage + stage_at(z, yy); }, tid, 64);
        }
        for (int j = tid; j < E * (kBoxPlane / 4); j += 64)
            reinterpret_cast<float4 *>(S.box)[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
    }
}


// ---------------------------------------------------------------- fused decode
// One persistent kernel for both stages. Every CTA first runs entropy lanes
// (the k_entropy loop) until the shared block queue is drained. Blocks are
// reconstructed in pairs (items 2j, 2j+1, x-neighbours
// inside a chunk): the block that completes a pair -- an absent block at
// kernel start, a coded one when its lane finishes -- appends the pair to a
// completion list. A CTA whose lanes are all idle reconstructs pairs in list
// order, while CTAs that still hold long blocks finish their entropy decode:
// the tail of the entropy stage overlaps the reconstruction of everything
// else, and the entries of a finished block are read back while still in L2.
// A CTA that claims a list position not yet written polls with a bounded
// backoff; if the bound runs out it records the position and leaves, and
// k_fused_tail (launched after, stream-ordered) reconstructs whatever was
// recorded or never claimed. No wait is unbounded.
struct FusedSmem {
    union {
        struct {
            uint16_t bend[9];
            uint32_t ctx[4][kCtxSlots][32];
        } e;
        struct {
            float A[16 * 16 * kRowF];
            float B[kBoxB];
            uint8_t stage0[kStageBytes];
        } r;
    } u;
    float4 W[16 * 8];
    int pair;
};

// Item `item` is ready for reconstruction; the last of its pair appends the pair.
__device__ __forceinline__ void pair_ready(const FusedParams &F, int item) {
    const uint32_t j = (uint32_t)item >> 1;
    const uint32_t size = 2u * j + 1u < (uint32_t)F.r.n ? 2u : 1u;
    __threadfence();   // this block's header and entries before the pair's count
    if (atomicAdd(F.pair_cnt + j, 1u) + 1u == size) {
        const uint32_t pos = atomicAdd(F.ws + kFusedDone, 1u);
        __threadfence();   // the other block's results, seen through the count, before the list entry
        atomicExch(F.rlist + pos, j + 1u);
    }
}

// Pair at completion-list position p, or -1 if not written yet.
__device__ __forceinline__ int list_pair(const FusedParams &F, uint32_t p) {
    const uint32_t v = *reinterpret_cast<const volatile uint32_t *>(F.rlist + p);
    return (int)v - 1;
}

template <bool CG>
__device__ __forceinline__ void reconstruct_pair(const RecParams &P, int j, float *sA, float *sB, uint8_t *stage0,
                                                 const float4 *W) {
    const int tid = threadIdx.x;
    uint8_t *const stage1 = reinterpret_cast<uint8_t *>(sA);   // sA is free once a block is staged
    const int i0 = 2 * j, i1 = 2 * j + 1;
    reconstruct_block<CG>(P, i0, sA, sB, stage0, W);
    const DecItem a = P.items[i0];
    if (i1 < P.n) {
        reconstruct_block<CG>(P, i1, sA, sB, stage1, W);
        const DecItem b = P.items[i1];
        if (pairable(a, b)) {
            uint8_t *dst = reinterpret_cast<uint8_t *>(a.dst);
            for (int r = tid; r < 256; r += 128) {
                const int z = r >> 4, y = r & 15;
                uint4 *row = reinterpret_cast<uint4 *>(dst + z * a.sz + y * a.sy);
                row[0] = *reinterpret_cast<const uint4 *>(stage0 + z * kStageZ + y * 16);
                row[1] = *reinterpret_cast<const uint4 *>(stage1 + z * kStageZ + y * 16);
            }
        } else {
            store_block(a, StageRows{stage0}, tid, 128);
            store_block(b, StageRows{stage1}, tid, 128);
        }
    } else {
        store_block(a, StageRows{stage0}, tid, 128);
    }
}

__global__ void __launch_bounds__(128, 4) k_decode_fused(FusedParams F) {
    extern __shared__ __align__(16) uint8_t s_raw[];
    FusedSmem &S = *reinterpret_cast<FusedSmem *>(s_raw);
    const EntParams &P = F.e;
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nlanes = gridDim.x * blockDim.x;
    // absent blocks are ready at once
    for (int q = P.ncoded + gtid; q < P.n; q += nlanes) pair_ready(F, (int)P.order[q]);
    if (threadIdx.x < 9) S.u.e.bend[threadIdx.x] = c_bend[threadIdx.x];
    for (int i = threadIdx.x; i < 16 * 8; i += blockDim.x) {
        const int k = i >> 3, mm = (i & 7) * 2;
        S.W[i] = make_float4(c_cos[k][mm], c_cos[k][mm], c_cos[k][mm + 1], c_cos[k][mm + 1]);
    }
    __syncthreads();

    // ---- entropy: the k_entropy loop, each finished block marked ready;
    // warps 0..nsolo-1 of the grid first decode order entry `warp` on their
    // first thread alone, as in k_entropy
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        uint32_t *ctx = &S.u.e.ctx[warp][0][lane];
        LaneState L;
        const int gwarp = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        if (gwarp < P.nsolo) {
            if (lane == 0) {
                memset(&L, 0, sizeof L);
                lane_begin(L, P, ctx, S.u.e.bend, (int)P.order[gwarp]);
                solo_entropy(L, P, ctx, S.u.e.bend);
                lane_finish(L, P);
                pair_ready(F, L.item);
            }
            __syncwarp();
        }
        EntParams E = P;   // the rest of the order, one lane per block
        E.order = P.order + P.nsolo;
        E.ncoded = P.ncoded - P.nsolo;
        run_lanes(L, E, ctx, S.u.e.bend, gtid - 32 * P.nsolo, nlanes - 32 * P.nsolo,
                  [&F](int item) { pair_ready(F, item); });
    }
    __syncthreads();   // the shared memory changes hands
    rec_init(S.u.r.B);
    __syncthreads();

    // ---- reconstruction over the completion list, one pair per claim
    const uint32_t npairs = ((uint32_t)F.r.n + 1u) >> 1;
    for (;;) {
        if (threadIdx.x == 0) {
            int j = -1;
            const uint32_t p = atomicAdd(F.ws + kFusedClaim, 1u);
            if (p < npairs) {
                j = list_pair(F, p);
                uint32_t ns = 32;
                for (uint32_t tries = 0; j < 0 && tries < F.spin_limit; ++tries) {
                    __nanosleep(ns);
                    if (ns < 1024) ns <<= 1;
                    j = list_pair(F, p);
                }
                if (j < 0) F.ws[kFusedSkip0 + atomicAdd(F.ws + kFusedNSkip, 1u)] = p;   // k_fused_tail takes it
                __threadfence();   // the pair's results after its list entry
            }
            S.pair = j;
        }
        __syncthreads();
        const int j = S.pair;
        if (j < 0) break;
        reconstruct_pair<true>(F.r, j, S.u.r.A, S.u.r.B, S.u.r.stage0, S.W);
        __syncthreads();
    }
}

// List positions that k_decode_fused recorded as given up or never claimed
// (normally none): one pair per CTA step. Runs after it, stream-ordered, so
// every pair is in the list.
__global__ void __launch_bounds__(128) k_fused_tail(FusedParams F) {
    __shared__ __align__(16) float sA[16 * 16 * kRowF];
    __shared__ __align__(16) float sB[kBoxB];
    __shared__ __align__(16) uint8_t sStage0[kStageBytes];
    __shared__ __align__(16) float4 sW[16 * 8];
    const uint32_t npairs = ((uint32_t)F.r.n + 1u) >> 1;
    const uint32_t claimed = min(F.ws[kFusedClaim], npairs);
    const uint32_t nsk = min(F.ws[kFusedNSkip], (uint32_t)kFusedMaxSkip);
    const uint32_t work = nsk + (npairs - claimed);
    if (blockIdx.x >= work) return;
    for (int i = threadIdx.x; i < 16 * 8; i += blockDim.x) {
        const int k = i >> 3, mm = (i & 7) * 2;
        sW[i] = make_float4(c_cos[k][mm], c_cos[k][mm], c_cos[k][mm + 1], c_cos[k][mm + 1]);
    }
    rec_init(sB);
    __syncthreads();
    for (uint32_t w = blockIdx.x; w < work; w += gridDim.x) {
        const uint32_t p = w < nsk ? F.ws[kFusedSkip0 + w] : claimed + (w - nsk);
        const int j = p < npairs ? list_pair(F, p) : -1;
        if (j < 0 || (uint32_t)j >= npairs) continue;   // every pair is listed by now
        reconstruct_pair<false>(F.r, j, sA, sB, sStage0, sW);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- one block
// The single-block calls (mc_archive_decode_block, mc_dec_block): one CTA
// decodes one block end to end in one launch, with the work item as a kernel
// argument -- no batch layout, no host-to-device copies, no second launch.
// Thread 0 runs the entropy decode (solo_entropy), the CTA then reconstructs
// the block.

static_assert(sizeof(DecItem) % 16 == 0, "SoloScratch::hdr must sit on a 16-byte boundary");

__global__ void __launch_bounds__(128) k_decode_one(DecItem it, SoloScratch *S, const QTab *qtab,
                                                    const uint16_t *scan, uint32_t *status) {
    // sA holds thread 0's entropy contexts (one column of 32-word rows, the
    // layout k_entropy uses) until the entropy decode is done, then the
    // pass-1 output
    __shared__ __align__(16) float sA[16 * 16 * kRowF];
    __shared__ __align__(16) float sB[kBoxB];
    __shared__ __align__(16) uint8_t sStage[kStageBytes];
    __shared__ __align__(16) float4 sW[16 * 8];
    __shared__ uint16_t s_bend[9];
    static_assert(sizeof(sA) >= sizeof(uint32_t) * kCtxSlots * 32, "contexts fit in sA");
    const int tid = threadIdx.x;
    if (tid < 9) s_bend[tid] = c_bend[tid];
    for (int i = tid; i < 16 * 8; i += blockDim.x) {
        const int k = i >> 3, mm = (i & 7) * 2;
        sW[i] = make_float4(c_cos[k][mm], c_cos[k][mm], c_cos[k][mm + 1], c_cos[k][mm + 1]);
    }
    rec_init(sB);
    const uint32_t cap = entry_cap(it.len);
    if (tid == 0) {
        S->item = it;
        S->base = 0;
        S->pool_used = 0;
        status[0] = 0;
    }
    __syncthreads();
    if (tid == 0) {
        EntParams P;
        P.items = &S->item;
        P.order = nullptr;
        P.n = 1;
        P.ncoded = 1;
        P.base = &S->base;
        P.arena = S->entries;
        P.hdr = &S->hdr;
        P.pool = S->entries + cap;       // the overflow continues the list
        P.pool_cap = kEntryMax - cap;    // what one block may ask of the pool
        P.pool_used = &S->pool_used;
        P.qtab = qtab;
        P.scan = scan;
        P.status = status;
        P.counter = nullptr;
        P.claim = 1;
        uint32_t *ctx = reinterpret_cast<uint32_t *>(sA);
        LaneState L;
        memset(&L, 0, sizeof L);
        lane_begin(L, P, ctx, s_bend, 0);
        solo_entropy(L, P, ctx, s_bend);
        lane_finish(L, P);
    }
    __syncthreads();   // thread 0's header and entries are visible to the CTA
    RecParams R;
    R.items = &S->item;
    R.idx = nullptr;
    R.n = 1;
    R.hdr = &S->hdr;
    R.base = &S->base;
    R.arena = S->entries;
    R.pool = S->entries + cap;
    R.qtab = qtab;
    R.scan = scan;
    reconstruct_block<true>(R, 0, sA, sB, sStage, sW);   // written in this kernel: read through L2
    store_block(it, StageRows{sStage}, tid, 128);
}

// ---------------------------------------------------------------- launchers
cudaError_t preload_decode_kernels() {
    // under lazy module loading a kernel's code is loaded at its first launch,
    // which would put a few milliseconds into the first call that uses it
    cudaFuncAttributes fa;
    const void *fns[] = {(const void *)k_entropy<2>, (const void *)k_entropy<4>, (const void *)k_entropy<8>,
                         (const void *)k_entropy_solo, (const void *)k_reconstruct, (const void *)k_decode_fused,
                         (const void *)k_fused_tail, (const void *)k_decode_one};
    for (const void *f : fns) {
        const cudaError_t e = cudaFuncGetAttributes(&fa, f);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t upload_decode_tables(const float cmf[16][16], const uint16_t scan[kN3], cudaStream_t s) {
    // pageable sources: the copies are staged before these calls return
    static uint16_t bend[9];
    for (int i = 1; i < kN3; ++i) {
        const uint32_t b = scan[i] >> 12;
        if ((uint32_t)(scan[i - 1] >> 12) != b) bend[b - 1] = (uint16_t)i;
    }
    bend[7] = kN3;
    bend[8] = 0xFFFF;
    static float pairs[16][16][2];
    for (int k = 0; k < 16; ++k)
        for (int m = 0; m < 16; ++m) pairs[k][m][0] = pairs[k][m][1] = cmf[k][m];
    cudaError_t e = cudaMemcpyToSymbolAsync(c_cos, cmf, sizeof(float) * 256, 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(c_cos2, pairs, sizeof pairs, 0, cudaMemcpyHostToDevice, s);
    return e != cudaSuccess ? e : cudaMemcpyToSymbolAsync(c_bend, bend, sizeof bend, 0, cudaMemcpyHostToDevice, s);
}

static int num_sms() { return dev_sms(); }

template <int W>
static cudaError_t launch_entropy_w(const EntParams &p, int ctas_per_sm, cudaStream_t s) {
    // per device: the dynamic shared memory opt-in of this instantiation
    static std::atomic<int> attr[kMaxDevs];
    const int a = dev_once(attr, [] {
        const cudaError_t e = cudaFuncSetAttribute(k_entropy<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)entropy_smem(W));
        return e == cudaSuccess ? 1 : -(int)e;
    });
    if (a < 0) return (cudaError_t)(-a);
    // one warp per solo block, one lane per other block
    EntParams q = p;
    if (!q.order || q.nsolo < 0) q.nsolo = 0;
    if (q.nsolo > q.ncoded) q.nsolo = q.ncoded;
    int blocks = (q.nsolo + (q.ncoded - q.nsolo + 31) / 32 + W - 1) / W;
    const int cap = num_sms() * ctas_per_sm;
    if (blocks > cap) blocks = cap;
    if (q.nsolo > blocks * W / 2) q.nsolo = blocks * W / 2;   // at most half of the warps
    k_entropy<W><<<blocks, W * 32, entropy_smem(W), s>>>(q);
    return cudaGetLastError();
}

// The single-thread share when a launch configuration leaves it open, from
// the launch's coded blocks. Below about 5 chunks' worth the stage's time is the
// longest block's chain, which a single thread runs fastest (q=6: 2 chunks 352
// us against 723 with lanes alone, 4 chunks 461 against 745; q=12: 244 against
// 399). Up to about 40 chunks' worth the longest blocks, four for each SM (one
// for each of its schedulers), run on single threads beside the lanes (8 chunks
// 637 us against 770 with lanes alone and 791 on single threads; 16: 745 / 850
// / 1583; 32: 940 / 1055). Beyond that the lanes are issue-bound and the single
// threads' extra instructions cost more than their chains save: 40 chunks of noise
// at q=0.25 68.8 ms with them, 63.4 without (q=0.1: 104 and 90), 48 chunks a third
// air at q=1 12.1 and 11.9, at q=6 4.19 and 4.21.
constexpr int kSoloAllMax = 19 * 1024, kSoloShareMax = 90 * 1024;
static int auto_solo(int ncoded) {
    if (ncoded <= kSoloAllMax) return 1;
    return ncoded <= kSoloShareMax ? ncoded / (4 * num_sms()) : 0;
}

cudaError_t launch_entropy(const EntParams &p, const LaunchCfg &cfg, cudaStream_t s) {
    if (p.ncoded <= 0) return cudaSuccess;
    const int solo = cfg.ent_solo >= 0 ? cfg.ent_solo : auto_solo(p.ncoded);
    if (solo == 1) {   // every block on a single thread
        const int blocks = std::min(p.ncoded, 2 * num_sms());
        k_entropy_solo<<<blocks, kSoloWarps * 32, 0, s>>>(p);
        return cudaGetLastError();
    }
    EntParams q = p;
    q.claim = cfg.ent_claim > 0 ? cfg.ent_claim : 1;
    q.nsolo = solo > 0 ? p.ncoded / solo : 0;
    const int per_sm = cfg.ent_ctas_per_sm > 0 ? cfg.ent_ctas_per_sm : 5;
    switch (cfg.ent_warps) {
    case 2: return launch_entropy_w<2>(q, per_sm, s);
    case 8: return launch_entropy_w<8>(q, per_sm, s);
    default: return launch_entropy_w<4>(q, per_sm, s);
    }
}

int fused_grid(const LaunchCfg &cfg) {
    static std::atomic<int> occ_by_dev[kMaxDevs];
    const int occ = dev_once(occ_by_dev, [] {
        // dynamic shared memory above 48 KiB: opt in once per device
        int o = 0;
        if (cudaFuncSetAttribute(k_decode_fused, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(FusedSmem)) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_decode_fused, 128, sizeof(FusedSmem)) !=
                cudaSuccess || o < 1)
            o = -1;
        return o;
    });
    if (occ < 0) return 0;
    // every CTA resident at once: a CTA's waits are then on CTAs that run
    const int per_sm = std::min(cfg.fused_ctas_per_sm > 0 ? cfg.fused_ctas_per_sm : 4, occ);
    return std::min(num_sms() * per_sm, kFusedMaxSkip);
}

cudaError_t launch_fused(const FusedParams &f, const LaunchCfg &cfg, cudaStream_t s) {
    const int blocks = fused_grid(cfg);
    if (blocks <= 0) return cudaErrorInvalidConfiguration;
    // the single-thread share (all blocks is not a fused layout: at most half
    // of the warps, as in k_entropy)
    FusedParams g = f;
    const int solo = cfg.ent_solo >= 0 ? cfg.ent_solo : auto_solo(f.e.ncoded);
    g.e.nsolo = solo > 0 ? std::min(f.e.ncoded / solo, blocks * 4 / 2) : 0;
    k_decode_fused<<<blocks, 128, sizeof(FusedSmem), s>>>(g);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_fused_tail<<<num_sms(), 128, 0, s>>>(f);
    return cudaGetLastError();
}

cudaError_t launch_reconstruct(const RecParams &p, const LaunchCfg &cfg, cudaStream_t s) {
    if (p.n <= 0) return cudaSuccess;
    // the knob counts 128 threads per SM as one: two CTAs of 64, of which 9 fit
    const int per_sm = std::min(2 * (cfg.rec_ctas_per_sm > 0 ? cfg.rec_ctas_per_sm : 5), 9);
    const int blocks = std::min(p.n, num_sms() * per_sm);
    // per device: the dynamic shared memory opt-in and the largest carveout, so that 9 CTAs per SM fit
    static std::atomic<int> attr[kMaxDevs];
    const int a = dev_once(attr, [] {
        cudaError_t e = cudaFuncSetAttribute(k_reconstruct, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RecSmem));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_reconstruct, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared);
        return e == cudaSuccess ? 1 : -(int)e;
    });
    if (a < 0) return (cudaError_t)(-a);
    // From 64 blocks per CTA up, where the output is several times the L2 and a
    // CTA's turn comes round late: half-written sectors then leave the L2 and are
    // read back and written twice (16 chunks, 268 MB: 213 MB read and 380 written).
    // 64 chunks at q=6 1.55 ms against 1.61, q=1 3.52 against 3.63. Below that the
    // batch is cut less evenly than by single blocks: 8 chunks at q=3 350 us
    // against 336, 3 chunks at q=12 73 against 72.
    RecParams P = p;
    P.pairs = p.n >= 64 * blocks;
    k_reconstruct<<<blocks, 64, sizeof(RecSmem), s>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_decode_one(const DecItem &it, SoloScratch *scratch, const QTab *qtab, const uint16_t *scan,
                              uint32_t *status, cudaStream_t s) {
    k_decode_one<<<1, 128, 0, s>>>(it, scratch, qtab, scan, status);
    return cudaGetLastError();
}

}  // namespace mcb

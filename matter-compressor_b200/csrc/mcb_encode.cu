// mcb_encode.cu -- sm_100a block encode and chunk-blob assembly.
//
// k_encode: one CTA (128 threads) per 16^3 block (src/mc_codec.c:629-736).
//   gather + sum/count -> dc -> forward DCT-II along x, y, z
//   (each output a sequential single-precision sum over n of the even/odd
//   halves, src/mc_codec_float.h:83-95) -> fused dead-zone quantiser
//   (src/mc_codec.c:686-692) -> optional max-error pass: dequantise, inverse
//   transform, lrint + dc, list every voxel whose error exceeds tau
//   (:697-708) -> the block's symbols in scratch.
// k_encode_rc: range coding of header bins, coefficients and corrections, one
//   lane per block (the coder is a serial chain; src/mc_codec.c:178-233).
// k_frac_count / k_fracmap / k_blob_layout / k_blob_fill / k_blob_hash: per-chunk blob assembly
//   (src/mc_codec.c:809-845, src/mc_archive.c:861-901): bitmap + u16 lengths
//   in block order, fraction map range-coded (src/mc_codec.c:600-611),
//   payloads concatenated in block order, xxh64 chain over
//   fmap | bitmap | lengths | payloads (src/mc_archive.c:76-88).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "mcb_devinfo.h"
#include "mcb_f32x2.cuh"
#include "mcb_format.h"
#include "mcb_kernels.h"

namespace mcb {

// this translation unit's copies (no -rdc): the cosine basis c[k][n] with every
// value doubled, as [n][k] and as [k][n] for n < 8, and the first scan position past
// each band (b < 7), then kN3 and a sentinel
__constant__ float4 c_fwd[8][8];
__constant__ float4 c_inv[16][4];
__constant__ uint16_t c_bend[9];

namespace {

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }

// ------------------------------------------------------------ range encoder
struct Enc {
    uint8_t *out;
    uint32_t cap, len;
    uint64_t low;
    uint32_t range;
    uint32_t cache;
    uint32_t pending;   // bytes held back for carry propagation (cache + 0xFF run)
};

__device__ __forceinline__ void enc_emit(Enc &e, uint32_t b) {
    if (e.len < e.cap) e.out[e.len] = (uint8_t)b;
    e.len++;
}
// src/mc_codec.c:180-187
__device__ __forceinline__ void enc_shift(Enc &e) {
    uint32_t top = (uint32_t)(e.low >> 32);
    if (top != 0 || e.low < 0xFF000000ull) {
        enc_emit(e, (e.cache + top) & 0xFF);
        for (uint32_t i = 1; i < e.pending; ++i) enc_emit(e, (0xFF + top) & 0xFF);
        e.pending = 0;
        e.cache = (uint32_t)(e.low >> 24) & 0xFF;
    }
    e.pending++;
    e.low = (e.low << 8) & 0xFFFFFFFFull;
}
__device__ __forceinline__ void enc_norm(Enc &e) {
    while (e.range < (1u << 24)) { enc_shift(e); e.range <<= 8; }
}
__device__ __forceinline__ int bitlen32(uint32_t v) { return v ? 32 - __clz(v) : 0; }
// ------------------------------------------------------------ transforms
// Two adjacent lines per thread, packed: value n of both lines is in[n * st].
// Every sum runs over ascending n (forward) or k (inverse), as the reference's
// (src/mc_codec_float.h:70-158). The adds take the products of the iteration
// before, which reach them through the loop's back edge (see mcb_f32x2.cuh). A sum
// starts from its first product, not from 0 plus it: only the sign of a zero can
// differ, which no level and no voxel shows.
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
// forward DCT-II, all 16 outputs
__device__ __forceinline__ void dct_products(float2 q[16], float2 a, float2 b, const float4 *w) {
    const float2 s = add2(a, b), d = sub2(a, b);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        q[2 * k] = mul2(lo2(w[k]), s);
        q[2 * k + 1] = mul2(hi2(w[k]), d);
    }
}
__device__ __forceinline__ void dct_lines(const float2 *in, int st, float2 o[16]) {
    const float2 *end = in + 15 * st;
    const float4 *w = c_fwd[0];
    float2 q[16];
    dct_products(o, *in, *end, w);
    in += st; end -= st; w += 8;
    dct_products(q, *in, *end, w);
#pragma unroll 1
    for (int n = 2;; ++n) {
        in += st; end -= st; w += 8;
        const float2 a = *in, b = *end;
#pragma unroll
        for (int k = 0; k < 16; ++k) o[k] = add2(o[k], q[k]);
        dct_products(q, a, b, w);
        if (n == 7) break;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) o[k] = add2(o[k], q[k]);
}
// inverse DCT-III, all 16 outputs from all 16 inputs
__device__ __forceinline__ void idct_products(float2 q[16], float2 e, float2 o, const float4 *w) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        q[2 * m] = mul2(lo2(w[m]), e);
        q[2 * m + 1] = mul2(hi2(w[m]), e);
        q[8 + 2 * m] = mul2(lo2(w[4 + m]), o);
        q[8 + 2 * m + 1] = mul2(hi2(w[4 + m]), o);
    }
}
__device__ __forceinline__ void idct_lines(const float2 *in, int st, float2 o[16]) {
    const float4 *w = c_inv[0];
    float2 a[16], q[16];   // the even-k sums of outputs 0-7, then the odd-k ones
    idct_products(a, in[0], in[st], w);
    in += 2 * st; w += 8;
    idct_products(q, in[0], in[st], w);
#pragma unroll 1
    for (int k = 4;; k += 2) {
        in += 2 * st; w += 8;
        const float2 e = in[0], d = in[st];
#pragma unroll
        for (int m = 0; m < 16; ++m) a[m] = add2(a[m], q[m]);
        idct_products(q, e, d, w);
        if (k == 14) break;
    }
#pragma unroll
    for (int m = 0; m < 16; ++m) a[m] = add2(a[m], q[m]);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        o[n] = add2(a[n], a[8 + n]);
        o[15 - n] = sub2(a[n], a[8 + n]);
    }
}

// Three passes x, y, z over a block in `buf`, in place; 128 threads, two lines each.
// In: (z, y, x) at x * 256 + z * 16 + y, stored but not yet synchronised. Out: the
// thread's values o[z] at y = tid >> 3 and x = 2 * (tid & 7), + 1. The strides keep
// every load and store of the passes without bank conflicts, but for the x pass's
// stores (two ways).
constexpr int kRowX = 256, kRowY = 260, kRowZ = 272;
template <bool FWD>
__device__ __forceinline__ void transform3(float *buf, float2 o[16]) {
    const int tid = threadIdx.x;
    float2 *mine = reinterpret_cast<float2 *>(buf) + tid;
    auto lines = [&](const float2 *in, int st) {
        if (FWD) dct_lines(in, st, o);
        else idct_lines(in, st, o);
    };
    __syncthreads();
    lines(mine, kRowX / 2);             // x lines at z = tid >> 3, y = 2 * (tid & 7), + 1
    __syncthreads();
    float *to = buf + 2 * (tid & 7) * kRowY + (tid >> 3) * 16;
#pragma unroll
    for (int x = 0; x < 16; x += 4) {
        *reinterpret_cast<float4 *>(to + x) = make_float4(o[x].x, o[x + 1].x, o[x + 2].x, o[x + 3].x);
        *reinterpret_cast<float4 *>(to + kRowY + x) = make_float4(o[x].y, o[x + 1].y, o[x + 2].y, o[x + 3].y);
    }
    __syncthreads();
    lines(mine, kRowY / 2);             // y lines at z = tid >> 3, x = 2 * (tid & 7), + 1
    __syncthreads();
#pragma unroll
    for (int y = 0; y < 16; ++y) mine[y * (kRowZ / 2)] = o[y];
    __syncthreads();
    lines(reinterpret_cast<const float2 *>(buf + (tid >> 3) * kRowZ) + (tid & 7), 8);   // z lines
}

// dead-zone reconstruction (src/mc_codec_float.h:185-190)
__device__ __forceinline__ float dequant(int lv, int f, const QTab &qt) {
    if (!lv) return 0.0f;
    float a = (float)(lv < 0 ? -lv : lv);
    float r = fadd(fadd(fmul(fsub(a, 1.0f), qt.step[f]), qt.dz8[f]), qt.dz4[f]);
    return lv < 0 ? -r : r;
}

struct EncSmem {
    float a[16 * kRowZ];
    int16_t lv[kN3];
    uint8_t vox[kN3];
    uint32_t mask[4][32];   // entry list and max-error pass: hit masks per warp and step
    uint32_t red[8];
    uint32_t ncorr, nent;
    uint32_t eob;
    uint32_t used;   // words of the CTA's share of the pool that hold symbols
};

}  // namespace

// What bounds it: instruction issue (59 % of the cycles), a quarter of it the
// transform's packed multiplies and adds, and latency at 5 CTAs (20 warps) per SM. 8
// chunks at q=6: 0.50 ms; 0.73 ms with one output of one line per step (scalar
// multiplies and adds, weights indexed by lane, 4-way bank conflicts in the x
// pass, two 16 KB buffers and 4 CTAs per SM). With the max-error pass (tau=16) 1.04
// ms against 2.07.
__global__ void __launch_bounds__(128, 5) k_encode(EncParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    EncSmem &S = *reinterpret_cast<EncSmem *>(smem_raw);
    const int tid = threadIdx.x;
    // the CTA's share of the symbol pool, filled block after block. A block that
    // it has no room for is left out and counted in status[1]: the caller runs the
    // launch again with a larger pool.
    const uint32_t share = P.pool_words / gridDim.x, pool0 = blockIdx.x * share;
    if (tid == 0) S.used = 0;
    auto no_room = [&](int item) {
        if (tid == 0) {
            atomicAdd(P.status + 1, 1u);
            P.len[item] = 0;
            P.sym[item] = make_uint4(0, 0, 0, 0);
        }
        __syncthreads();
    };

    for (int item = blockIdx.x; item < P.n; item += gridDim.x) {
        const EncItem it = P.items[item];
        const QTab &qt = P.qtab[it.qslot];
        const uint8_t *src = reinterpret_cast<const uint8_t *>(it.src);
        // gather: two 16-voxel rows per thread
        uint32_t sum = 0, cnt = 0;
        uint4 rows[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = tid + 128 * h, z = r >> 4, y = r & 15;
            const uint8_t *row = src + z * it.sz + y * it.sy;
            uint4 &w = rows[h];
            if (((uintptr_t)row & 15) == 0) {
                w = *reinterpret_cast<const uint4 *>(row);
            } else {
                uint8_t b[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) b[x] = row[x];
                memcpy(&w, b, 16);
            }
            *reinterpret_cast<uint4 *>(S.vox + r * 16) = w;
            const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
#pragma unroll
                for (int bb = 0; bb < 4; ++bb) {
                    uint32_t v = (ws[q] >> (8 * bb)) & 0xFF;
                    sum += v;
                    cnt += v != 0;
                }
            }
        }
        // block reduce sum, count
        for (int o = 16; o; o >>= 1) {
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
            cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
        }
        if ((tid & 31) == 0) { S.red[tid >> 5] = sum; S.red[4 + (tid >> 5)] = cnt; }
        if (tid == 0) { S.ncorr = 0; S.eob = 0; }
        __syncthreads();
        sum = S.red[0] + S.red[1] + S.red[2] + S.red[3];
        cnt = S.red[4] + S.red[5] + S.red[6] + S.red[7];
        if (tid == 0 && !cnt) { P.len[item] = 0; P.sym[item] = make_uint4(0, 0, 0, 0); }
        if (!cnt) { __syncthreads(); continue; }       // all air: not coded
        const int dc = (int)((sum + kN3 / 2) / kN3);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t ws[4] = {rows[h].x, rows[h].y, rows[h].z, rows[h].w};
#pragma unroll
            for (int x = 0; x < 16; ++x)
                S.a[x * kRowX + tid + 128 * h] = (float)((int)((ws[x >> 2] >> (8 * (x & 3))) & 0xFF) - dc);
        }
        float2 o[16];
        transform3<true>(S.a, o);
        // fused quantiser: t = |c|*rstep + (1-0.8), clamp [0,32767], truncate
        const float bias = 1.0f - 0.80f;
        const int y0 = tid >> 3, x0 = 2 * (tid & 7);   // the thread's column of coefficients
        uint32_t last = 0;
        auto level = [&](float c, int f) -> uint32_t {
            float t = fadd(fmul(fabsf(c), qt.rstep[f]), bias);
            if (!(t > 0.0f)) t = 0.0f;
            if (!(t < 32767.0f)) t = 32767.0f;
            int v = (int)t;
            return (uint16_t)(int16_t)(c < 0.0f ? -v : v);
        };
#pragma unroll
        for (int z = 0; z < 16; ++z)
            reinterpret_cast<uint32_t *>(S.lv)[z * 128 + tid] =
                level(o[z].x, z + y0 + x0) | level(o[z].y, z + y0 + x0 + 1) << 16;
        __syncthreads();
        // the nonzero levels in scan order as one entry list (position | level
        // << 16) for k_encode_rc: warp w owns positions [1024w, 1024w + 1024) in
        // 32 steps of 32; a first pass counts (the step masks kept in shared
        // memory), one barrier gives every warp its start, a second pass writes
        {
            const int lane = tid & 31, w = tid >> 5;
            uint32_t cnt_w = 0;
            for (int k = 0; k < 32; ++k) {
                const uint32_t p0 = 1024u * w + 32u * k;
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, S.lv[__ldg(P.scan + p0 + lane) & 0xFFF] != 0);
                if (lane == 0) S.mask[w][k] = m;
                cnt_w += __popc(m);
                if (m) last = p0 + 32u - __clz(m);   // eob = 1 + last nonzero position
            }
            if (lane == 0) {
                S.red[w] = cnt_w;
                atomicMax(&S.eob, last);
            }
            __syncthreads();
            uint32_t at = 0;
            for (int ww = 0; ww < w; ++ww) at += S.red[ww];
            const uint32_t nent = S.red[0] + S.red[1] + S.red[2] + S.red[3];
            if (S.used + nent > share) {
                no_room(item);
                continue;
            }
            if (tid == 0) S.nent = nent;
            uint32_t *ent = P.pool + pool0 + S.used;
            for (int k = 0; k < 32; ++k) {
                const uint32_t m = S.mask[w][k], p = 1024u * w + 32u * k + lane;
                if ((m >> lane) & 1)
                    ent[at + __popc(m & ((1u << lane) - 1u))] =
                        p | (uint32_t)(uint16_t)S.lv[__ldg(P.scan + p) & 0xFFF] << 16;
                at += __popc(m);
            }
        }
        if (it.tau > 0) {
            // local reconstruction for the max-error pass
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = tid + 128 * h;
                const uint4 *row = reinterpret_cast<const uint4 *>(S.lv + 16 * r);
                const uint4 u = row[0], v = row[1];
                const uint32_t ws[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
                for (int x = 0; x < 16; ++x)
                    S.a[x * kRowX + r] =
                        dequant((int)(int16_t)(ws[x >> 1] >> (16 * (x & 1))), (r >> 4) + (r & 15) + x, qt);
            }
            transform3<false>(S.a, o);
            // voxel (z, y, x) to where the thread read (y, z, x) of its own lines
            float2 *mine = reinterpret_cast<float2 *>(S.a + y0 * kRowZ + x0);
#pragma unroll
            for (int z = 0; z < 16; ++z) mine[8 * z] = o[z];
            __syncthreads();
            // corrections in ascending voxel order, written straight to the
            // coder's scratch: warp w owns voxels [1024w, 1024w + 1024) in 32
            // steps of 32; a first pass counts its hits (the step masks kept
            // in shared memory), one barrier gives every warp its start, and a
            // second pass writes the entries
            const int lane = tid & 31, w = tid >> 5;
            auto hit_at = [&](int i, int &dl) {
                long long rr = __float2ll_rn(S.a[((i >> 4) & 15) * kRowZ + (i >> 8) * 16 + (i & 15)]);
                int v = (int)(uint32_t)(unsigned long long)rr + dc;
                v = v < 0 ? 0 : v > 255 ? 255 : v;
                const int err = (int)S.vox[i] - v;
                const int ae = err < 0 ? -err : err;
                dl = err < 0 ? -(ae - (int)it.tau) : (ae - (int)it.tau);
                return ae > (int)it.tau;
            };
            uint32_t cnt_w = 0;
            for (int k = 0; k < 32; ++k) {
                int dl;
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit_at(1024 * w + 32 * k + lane, dl));
                if (lane == 0) S.mask[w][k] = m;
                cnt_w += __popc(m);
            }
            if (lane == 0) S.red[w] = cnt_w;
            __syncthreads();
            uint32_t at = 0;
            for (int ww = 0; ww < w; ++ww) at += S.red[ww];
            const uint32_t ncorr = S.red[0] + S.red[1] + S.red[2] + S.red[3], cor0 = S.used + S.nent;
            if (cor0 + ncorr > share) {
                no_room(item);
                continue;
            }
            uint32_t *cor = P.pool + pool0 + cor0;
            for (int k = 0; k < 32; ++k) {
                const uint32_t m = S.mask[w][k];
                if ((m >> lane) & 1) {
                    int dl;
                    const int i = 1024 * w + 32 * k + lane;
                    hit_at(i, dl);
                    cor[at + __popc(m & ((1u << lane) - 1u))] = (uint32_t)i | ((uint32_t)(uint16_t)(int16_t)dl << 16);
                }
                at += __popc(m);
            }
            if (tid == 0) S.ncorr = ncorr;
        }
        __syncthreads();   // nent and ncorr complete, used read
        if (tid == 0) {
            const uint32_t at = pool0 + S.used;
            P.sym[item] = make_uint4(0x80000000u | (S.eob << 8) | (uint32_t)dc, S.ncorr, at, at + S.nent);
            S.used += S.nent + S.ncorr;
        }
        __syncthreads();
    }
}

// Range coding of every coded block, one lane per block (src/mc_codec.c:
// 330-350, 710-729): header bins, EOB, the coefficient loop and the
// corrections, in the order the reference writes them. The coder of a block is
// a serial chain; lanes in a warp code different blocks, with contexts in
// shared memory (one word per context per lane, context j of lane l at word
// j * 32 + l).
//
// The coefficient loop is the mirror of the decoder's (k_entropy in
// mcb_decode.cu): one step of straight-line code advances every lane by a run of
// one or four zeros, a significance bin, a magnitude rung and a sign. A run of
// zeros does not touch the code value and the range only falls, so the last
// split above the renormalisation bound says that none of the run renormalises.
//
// The code value is `low` with its not yet written bytes in front of it
// (ah:al, n of them, at least two), so that a carry ripples through by plain
// addition; the bytes go out two at a time, and a carry past all of them, about
// one in 65536 writes, walks back through the bytes already written.
namespace {
constexpr int kEncSlots = kNumCtx + 1;   // one more: 1, the "probability" of a bypass bin (see k_entropy)
constexpr uint32_t kEncScr = kNumCtx;
constexpr uint32_t kEncTop = 1u << 24;

struct EncLane {
    uint8_t *out;
    uint32_t len;                   // bytes written
    uint32_t n, ah, al, low, range;
    const uint32_t *ent;            // the block's entries
    uint32_t idx, ahead;            // next entry to load, the entry after the current one
    uint32_t pos, m, neg, kend;     // current coefficient: position, magnitude, sign, one-bits of its unary code
    uint32_t p, eob, sigb, band, bend, stop;
    uint32_t e1, e2, e3;            // the last three significant positions + 17, newest first
    uint32_t cs, ps, lim;           // context slot at p, its probability, where either changes
    uint32_t k, pm;                 // next rung (0 at a significance bin), its probability
    bool live;
};

__device__ __forceinline__ void code_add(EncLane &e, uint32_t v) {
    const uint32_t t = e.low + v, a = e.al + (t < v ? 1u : 0u);
    e.ah += a < e.al ? 1u : 0u;
    e.al = a;
    e.low = t;
}
// Bits that a renormalisation shifts out: 0, 8 or 16 (src/mc_codec.c:180-187)
__device__ __forceinline__ uint32_t code_norm(EncLane &e) {
    const uint32_t s = e.range < (1u << 16) ? 16u : (e.range < kEncTop ? 8u : 0u);
    e.ah = funnel_left(e.al, e.ah, s);
    e.al = funnel_left(e.low, e.al, s);
    e.low <<= s;
    e.range <<= s;
    e.n += s >> 3;
    return s;
}
// A carry past the held bytes: one more in the bytes already written.
__device__ __noinline__ void code_carry(uint8_t *out, uint32_t len) {
    uint32_t i = min(len, (uint32_t)kEncCap);
    while (i > 0 && ++out[i - 1] == 0) --i;
}
// Writes the two oldest of n >= 4 held bytes.
__device__ __forceinline__ void code_flush(EncLane &e) {
    uint64_t acc = (uint64_t)e.ah << 32 | e.al;
    const uint32_t sh = 8u * (e.n - 2u);   // 16..40
    const uint32_t v = (uint32_t)(acc >> sh);
    acc &= (1ull << sh) - 1u;
    e.ah = (uint32_t)(acc >> 32);
    e.al = (uint32_t)acc;
    e.n -= 2;
    if (v >> 16) code_carry(e.out, e.len);
    if (e.len + 2 <= (uint32_t)kEncCap)   // even offsets, even base
        *reinterpret_cast<uint16_t *>(e.out + e.len) = (uint16_t)((v >> 8 & 0xFFu) | (v & 0xFFu) << 8);
    e.len += 2;
}
__device__ __forceinline__ void code_settle(EncLane &e) {   // after a single operation
    code_norm(e);
    while (e.range < kEncTop) code_norm(e);
    while (e.n >= 4) code_flush(e);
}

// The coder of a thread that is alone on its warp: the held bytes and low in one
// 64-bit word, 1 to 3 bytes held, a byte at a time.
struct EncOne {
    uint8_t *out;
    uint32_t len, n, range;
    uint64_t code;   // n held bytes, low
};
__device__ __forceinline__ void code_add(EncOne &e, uint32_t v) { e.code += v; }
__device__ __forceinline__ void code_settle(EncOne &e) {
    while (e.range < kEncTop) {
        if (e.n == 3) {   // the two oldest go out
            const uint32_t v = (uint32_t)(e.code >> 40);
            e.code &= (1ull << 40) - 1u;
            e.n = 1;
            if (v >> 16) code_carry(e.out, e.len);
            if (e.len + 2 <= (uint32_t)kEncCap)   // even offsets, even base
                *reinterpret_cast<uint16_t *>(e.out + e.len) = (uint16_t)((v >> 8 & 0xFFu) | (v & 0xFFu) << 8);
            e.len += 2;
        }
        e.code <<= 8;
        e.range <<= 8;
        ++e.n;
    }
}

// Single bins of either coder.
__device__ __forceinline__ uint32_t after0(uint32_t p) { return p + ((4096u - p) >> 4); }
__device__ __forceinline__ uint32_t after1(uint32_t p) { return p - (p >> 4); }
template <class Coder>
__device__ __forceinline__ void code_bin(Coder &e, uint32_t &p0, uint32_t bit) {
    const uint32_t r0 = (e.range >> 12) * p0;
    if (!bit) { e.range = r0; p0 = after0(p0); }
    else { code_add(e, r0); e.range -= r0; p0 = after1(p0); }
    code_settle(e);
}
template <class Coder>
__device__ __forceinline__ void code_bypass(Coder &e, uint32_t bit) {
    e.range >>= 1;
    if (bit) code_add(e, e.range);
    code_settle(e);
}
// k bits MSB-first, 16 at a time from the top (src/mc_codec.c:209-215)
template <class Coder>
__device__ __forceinline__ void code_bits(Coder &e, uint32_t v, int k) {
    while (k > 0) {
        const int take = k > 16 ? 16 : k;
        e.range >>= take;
        code_add(e, ((v >> (k - take)) & ((1u << take) - 1u)) * e.range);
        code_settle(e);
        k -= take;
    }
}
// order-0 Exp-Golomb (src/mc_codec.c:229-233)
template <class Coder>
__device__ __forceinline__ void code_eg(Coder &e, uint32_t v) {
    const uint32_t t = v + 1u;
    const int nb = bitlen32(t) - 1;
    for (int i = 0; i < nb; ++i) code_bypass(e, 1);
    code_bypass(e, 0);
    if (nb > 0) code_bits(e, t & ((1u << nb) - 1u), nb);
}
// Header bins and EOB: its bit length prefix, then the bits below the MSB
// (src/mc_codec.c:314-320). No context occurs twice; p0(j) is context j's.
template <class Coder, class P0>
__device__ __forceinline__ void code_header(Coder &e, P0 p0, uint32_t dc, uint32_t eob, uint32_t ncorr) {
    auto bin = [&](int j, uint32_t bit) {
        uint32_t p = p0(j);
        code_bin(e, p, bit);
    };
    bin(kCtxFlag + 0, 0);                 // reserved
    bin(kCtxFlag + 1, ncorr > 0);
    for (int b = 0; b < 8; ++b) bin(kCtxDc + b, (dc >> (7 - b)) & 1);
    const int k = bitlen32(eob);
    for (int i = 0; i < k; ++i) bin(kCtxEob + i, 1);
    if (k < 13) bin(kCtxEob + k, 0);
    if (k > 1) code_bits(e, eob & ((1u << (k - 1)) - 1u), k - 1);
}
// What follows the scan (src/mc_codec.c:721-729).
template <class Coder>
__device__ __forceinline__ void code_corrections(Coder &e, const uint32_t *cor, uint32_t ncorr) {
    if (!ncorr) return;
    code_eg(e, ncorr - 1);
    uint32_t prev = 0;
    for (uint32_t c = 0; c < ncorr; ++c) {
        const uint32_t w = cor[c];
        const uint32_t pos = w & 0xFFFF;
        code_eg(e, pos - prev);
        prev = pos;
        const int d = (int16_t)(w >> 16);
        code_bypass(e, d < 0);
        code_eg(e, (uint32_t)(d < 0 ? -d : d) - 1u);
    }
}
// The n held bytes, then the four of low; the payload's length.
__device__ __forceinline__ void code_end(const EncParams &P, int item, uint8_t *out, uint32_t len, uint64_t held,
                                         uint32_t n, uint32_t low) {
    if ((held >> (8 * n)) & 1) code_carry(out, len);
    for (int i = (int)n + 3; i >= 0; --i, ++len) {
        const uint32_t b = i >= 4 ? (uint32_t)(held >> (8 * (i - 4))) : low >> (8 * i);
        if (len < (uint32_t)kEncCap) out[len] = (uint8_t)b;
    }
    if (len > (uint32_t)kEncCap) atomicAdd(P.status, 1u);
    P.len[item] = min(len, (uint32_t)kEncCap);
}

__device__ __forceinline__ void enc_density(EncLane &e) {
    const bool a3 = e.p < e.e3, a2 = e.p < e.e2, a1 = e.p < e.e1;
    e.cs = e.sigb + (a3 ? 3u : (a2 ? 2u : (a1 ? 1u : 0u)));
    e.lim = min(e.stop, a3 ? e.e3 : (a2 ? e.e2 : (a1 ? e.e1 : 0xFFFFFFFFu)));
}
__device__ __forceinline__ void set_entry(EncLane &e, uint32_t w) {
    const int lv = (int)w >> 16;
    e.pos = w & 0xFFFFu;
    e.neg = lv < 0 ? 1u : 0u;
    e.m = (uint32_t)(lv < 0 ? -lv : lv);
    // m - 1 ones and a zero up to m = 12; twelve ones and the prefix of the
    // Exp-Golomb code of m - 12 beyond (src/mc_codec.c:268-275)
    e.kend = e.m <= 12u ? e.m - 1u : 43u - (uint32_t)__clz(e.m - 11u);
}
__device__ __forceinline__ void next_entry(EncLane &e) {
    set_entry(e, e.ahead);
    e.ahead = e.ent[e.idx++];   // up to two entries past the block's last (EncParams::pool)
}
// p >= stop: a band change, or the last position, significant by definition:
// its coefficient without a significance bin (src/mc_codec.c:337-349); the
// coefficient loop is then over.
__device__ __forceinline__ void enc_position(EncLane &e, uint32_t *ctx, const uint16_t *s_bend) {
    while (e.p >= e.bend) { e.band++; e.sigb += 4; e.bend = s_bend[e.band]; }
    if (e.p + 1 >= e.eob) {
        for (uint32_t k = 0; k < 12u; ++k) {
            code_bin(e, ctx[(kCtxMag + k) * 32], k < e.kend);
            if (k >= e.kend) break;
        }
        if (e.m > 12u) code_eg(e, e.m - 12u);
        code_bypass(e, e.neg);
        e.live = false;
        e.lim = e.stop = 0xFFFFFFFFu;
        return;
    }
    e.stop = min(e.bend, e.eob - 1);
    enc_density(e);
    e.ps = ctx[e.cs * 32];
}

// One step of every live lane; returns whether enc_event has work for the lane.
__device__ __forceinline__ bool enc_step(EncLane &e, uint32_t *ctx, bool &rest) {
    const uint32_t k0 = e.k;
    const bool is_sig = e.live & (k0 == 0u);
    uint32_t pr = e.ps, p = e.p;
    {   // zeros
        const uint32_t gap = e.pos - p, room = is_sig ? min(e.lim - p, gap + 1u) : 0u;
        const uint32_t r1 = (e.range >> 12) * pr, q1 = (15u * pr + 4096u) >> 4;
        const uint32_t r2 = (r1 >> 12) * q1, q2 = (15u * q1 + 4096u) >> 4;
        const uint32_t r3 = (r2 >> 12) * q2, q3 = (15u * q2 + 4096u) >> 4;
        const uint32_t r4 = (r3 >> 12) * q3, q4 = (15u * q3 + 4096u) >> 4;
        const bool z1 = (r1 >= kEncTop) & (room > 1u), z4 = (r4 >= kEncTop) & (room > 4u);
        e.range = z4 ? r4 : (z1 ? r1 : e.range);
        pr = z4 ? q4 : (z1 ? q1 : pr);
        p += z4 ? 4u : (z1 ? 1u : 0u);
    }
    // the significance bin at p
    const bool one = is_sig & (p == e.pos);
    const uint32_t r1 = is_sig ? (e.range >> 12) * pr : e.range;
    code_add(e, one ? r1 : 0u);
    e.range = one ? e.range - r1 : r1;
    if (is_sig) ctx[e.cs * 32] = (15u * pr + (one ? 15u : 4096u)) >> 4;
    const uint32_t s1 = code_norm(e);
    p += is_sig ? 1u : 0u;
    e.p = p;
    e.e3 = one ? e.e2 : e.e3;
    e.e2 = one ? e.e1 : e.e2;
    e.e1 = one ? p + 16u : e.e1;
    enc_density(e);
    e.ps = ctx[e.cs * 32];
    // a rung, or a bit of the prefix behind the twelfth
    const bool act = one | (k0 != 0u), pfx = k0 >= 12u;
    const bool up = act & (k0 < e.kend);
    const uint32_t pm = e.pm;
    const uint32_t r2 = act ? (e.range >> (pfx ? 1u : 12u)) * pm : e.range;
    code_add(e, up ? r2 : 0u);
    e.range = up & !pfx ? e.range - r2 : r2;
    if (act & !pfx) ctx[(kCtxMag + k0) * 32] = (15u * pm + (up ? 15u : 4096u)) >> 4;
    const uint32_t kn = up ? k0 + 1u : 0u;
    e.k = kn;
    e.pm = ctx[(kCtxMag + min(kn, 12u)) * 32];
    const uint32_t s2 = code_norm(e);
    // the sign, unless a suffix comes first or the held bytes are many
    const bool closed = act & !up;
    const bool sign = closed & !pfx & (s1 + s2 <= 16u);
    const uint32_t r3 = sign ? e.range >> 1 : e.range;
    code_add(e, (sign & (e.neg != 0u)) ? r3 : 0u);
    e.range = r3;
    code_norm(e);
    if (sign) next_entry(e);
    while (e.n >= 4) code_flush(e);
    rest = closed & !sign;
    return rest | (e.live & (kn == 0u) & (p >= e.stop));
}
__device__ __forceinline__ void enc_event(EncLane &e, uint32_t *ctx, const uint16_t *s_bend, bool rest) {
    if (rest) {   // the suffix of an escape, the sign
        if (e.m > 12u) {
            const int nb = bitlen32(e.m - 11u) - 1;
            code_bits(e, (e.m - 11u) & ((1u << nb) - 1u), nb);
        }
        code_bypass(e, e.neg);
        next_entry(e);
    }
    if (e.p >= e.stop) enc_position(e, ctx, s_bend);
}
}  // namespace

// Warp groups of `lanes` blocks (the warp's other lanes idle): launches of few
// blocks spread them over more warps, since a warp's time is its longest
// block's chain and its lanes' rare events add up.
constexpr int kRcWarps = 4;
__global__ void __launch_bounds__(kRcWarps * 32) k_encode_rc(EncParams P, int lanes) {
    __shared__ uint32_t s_ctx[kRcWarps][kEncSlots][32];
    __shared__ uint16_t s_bend[9];
    if (threadIdx.x < 9) s_bend[threadIdx.x] = c_bend[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *ctx = &s_ctx[warp][0][lane];
    const int ngroups = (P.n + lanes - 1) / lanes;
    for (int g = blockIdx.x * kRcWarps + warp; g < ngroups; g += gridDim.x * kRcWarps) {
        const int item = g * lanes + lane;
        uint4 sy = make_uint4(0, 0, 0, 0);
        if (lane < lanes && item < P.n) sy = P.sym[item];
        const bool coded = (sy.x & 0x80000000u) != 0;   // an all-air block is not coded
        const uint32_t dc = sy.x & 0xFF, eob = (sy.x >> 8) & 0x1FFF, ncorr = sy.y;
        EncLane e;
        memset(&e, 0, sizeof e);
        e.range = 0xFFFFFFFFu;
        e.n = 1;   // the coder's leading byte
        e.cs = e.sigb = kEncScr;
        e.lim = e.stop = 0xFFFFFFFFu;
        e.pm = 1;
        if (coded) {
            const EncItem it = P.items[item];
            const QTab &qt = P.qtab[it.qslot];
            e.out = reinterpret_cast<uint8_t *>(it.out);
            for (int j = 0; j < kNumCtx; ++j) ctx[j * 32] = qt.ctx[j];
            ctx[kEncScr * 32] = 1;
            code_header(e, [ctx](int j) { return ctx[j * 32]; }, dc, eob, ncorr);
            if (eob) {
                e.ent = P.pool + sy.z;
                e.eob = eob;
                e.sigb = kCtxSig;
                e.bend = s_bend[0];
                e.ahead = e.ent[0];
                e.idx = 1;
                next_entry(e);
                e.live = true;
                e.pm = ctx[kCtxMag * 32];
                enc_position(e, ctx, s_bend);
            }
        }
        __syncwarp();
        while (__any_sync(0xFFFFFFFFu, e.live)) {
            bool rest;
            const bool ev = enc_step(e, ctx, rest);
            if (__any_sync(0xFFFFFFFFu, ev)) {
                if (ev) enc_event(e, ctx, s_bend, rest);
                __syncwarp();
            }
        }
        if (coded) {
            code_corrections(e, P.pool + sy.w, ncorr);
            code_end(P, item, e.out, e.len, (uint64_t)e.ah << 32 | e.al, e.n, e.low);
        }
        __syncwarp();
    }
}

// The coder of a few blocks, each by one thread alone on its warp: the mirror of
// the decoder's solo_entropy (mcb_decode.cu). The contexts of the scan are held in
// registers, the four of the current band and the twelve rungs, and every
// position jumps to where the next is coded; a run of zeros in a sparse density
// class goes four at a time, one compare of the last split deciding that none
// renormalises. What bounds it: the chain of dependent instructions through the
// range. A block of noise at q=0.5 takes 2.57 ms, 10.1 as the one live lane of
// k_encode_rc, which pays every lane's step for it (3.54 bin by bin from a list of
// levels); textured material at q=24 130 us, 204 and 500.
namespace {
__device__ __forceinline__ bool code_rung(EncOne &e, uint32_t &g, bool up) {
    code_bin(e, g, up);
    return up;
}
__device__ __forceinline__ void code_scan(EncOne &e, const QTab &qt, const uint32_t *ent, uint32_t eob) {
    uint32_t g0 = qt.ctx[kCtxMag + 0], g1 = qt.ctx[kCtxMag + 1], g2 = qt.ctx[kCtxMag + 2], g3 = qt.ctx[kCtxMag + 3];
    uint32_t g4 = qt.ctx[kCtxMag + 4], g5 = qt.ctx[kCtxMag + 5], g6 = qt.ctx[kCtxMag + 6], g7 = qt.ctx[kCtxMag + 7];
    uint32_t g8 = qt.ctx[kCtxMag + 8], g9 = qt.ctx[kCtxMag + 9], g10 = qt.ctx[kCtxMag + 10], g11 = qt.ctx[kCtxMag + 11];
    uint32_t s0 = 0, s1 = 0, s2 = 0, s3 = 0;   // the band's contexts
    uint32_t p = 0, e1 = 0, e2 = 0, e3 = 0, band = 0, bend = 0, stop = 0;
    uint32_t w = ent[0], ahead = ent[1], idx = 2, pos = w & 0xFFFFu;
    auto to_band = [&](uint32_t b) {
        band = b;
        bend = c_bend[b];
        const uint16_t *c = qt.ctx + kCtxSig + 4 * b;
        s0 = c[0]; s1 = c[1]; s2 = c[2]; s3 = c[3];
    };
    to_band(0);
position:   // a band change, or the last position, significant by definition
    while (p >= bend) to_band(band + 1);
    stop = min(bend, eob - 1);
    if (p + 1 == eob) {
        ++p;
        goto coef;
    }
next:       // a significance bin at p < stop
    if (p < e3) {   // density class 3: bins one at a time
        const bool sig = p == pos;
        code_bin(e, s3, sig);
        ++p;
        if (sig) goto one;
        if (p >= stop) goto position;
        goto next;
    } else {
        const bool a2 = p < e2, a1 = p < e1;
        const uint32_t lim = min(stop, a2 ? e2 : (a1 ? e1 : 0xFFFFFFFFu)), end = min(lim, pos);
        uint32_t pc = a2 ? s2 : (a1 ? s1 : s0);
        while (p < end) {
            if (p + 4u <= end) {
                const uint32_t r1 = (e.range >> 12) * pc, q1 = after0(pc);
                const uint32_t r2 = (r1 >> 12) * q1, q2 = after0(q1);
                const uint32_t r3 = (r2 >> 12) * q2, q3 = after0(q2);
                const uint32_t r4 = (r3 >> 12) * q3;
                if (r4 >= kEncTop) {
                    e.range = r4;
                    pc = after0(q3);
                    p += 4;
                    continue;
                }
            }
            code_bin(e, pc, 0);
            ++p;
        }
        const bool sig = p < lim;   // p is the next significant position
        if (sig) {
            code_bin(e, pc, 1);
            ++p;
        }
        s0 = a1 ? s0 : pc;
        s1 = a1 & !a2 ? pc : s1;
        s2 = a2 ? pc : s2;
        if (sig) goto one;
        if (p >= stop) goto position;
        goto next;
    }
one:
    e3 = e2;
    e2 = e1;
    e1 = p + 16u;
coef:       // the coefficient at p - 1 (src/mc_codec.c:268-275)
    {
        const int lv = (int)w >> 16;
        const uint32_t m = (uint32_t)(lv < 0 ? -lv : lv);
        w = ahead;
        pos = w & 0xFFFFu;
        ahead = ent[idx++];   // up to two entries past the block's last (EncParams::pool)
        if (code_rung(e, g0, m > 1) && code_rung(e, g1, m > 2) && code_rung(e, g2, m > 3) && code_rung(e, g3, m > 4) &&
            code_rung(e, g4, m > 5) && code_rung(e, g5, m > 6) && code_rung(e, g6, m > 7) && code_rung(e, g7, m > 8) &&
            code_rung(e, g8, m > 9) && code_rung(e, g9, m > 10) && code_rung(e, g10, m > 11) &&
            code_rung(e, g11, m > 12))
            code_eg(e, m - 12u);
        code_bypass(e, lv < 0);
    }
    if (p >= eob) return;
    if (p < stop) goto next;
    goto position;
}
}  // namespace
__global__ void __launch_bounds__(32) k_encode_rc_one(EncParams P) {
    const int item = blockIdx.x;
    if (threadIdx.x) return;
    const uint4 sy = P.sym[item];
    if (!(sy.x & 0x80000000u)) return;   // all air: not coded
    const uint32_t dc = sy.x & 0xFF, eob = (sy.x >> 8) & 0x1FFF, ncorr = sy.y;
    const EncItem it = P.items[item];
    const QTab &qt = P.qtab[it.qslot];
    EncOne e;
    e.out = reinterpret_cast<uint8_t *>(it.out);
    e.len = 0;
    e.n = 1;   // the coder's leading byte
    e.range = 0xFFFFFFFFu;
    e.code = 0;
    code_header(e, [&qt](int j) { return (uint32_t)qt.ctx[j]; }, dc, eob, ncorr);
    if (eob) code_scan(e, qt, P.pool + sy.z, eob);
    code_corrections(e, P.pool + sy.w, ncorr);
    code_end(P, item, e.out, e.len, e.code >> 32, e.n, (uint32_t)e.code);
}

// ------------------------------------------------------------ blob assembly
// Material nibble of every block (src/mc_codec.c:820-822), one warp per block:
// the voxels are read once more (20 us for 8 chunks) so that the fraction maps
// need not wait for the transform.
__global__ void __launch_bounds__(256) k_frac_count(EncParams P) {
    const int item = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (item >= P.n) return;   // whole warps leave together
    const EncItem it = P.items[item];
    const uint8_t *src = reinterpret_cast<const uint8_t *>(it.src);
    uint32_t cnt = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int r = j * 32 + lane;
        const uint8_t *row = src + (r >> 4) * it.sz + (r & 15) * it.sy;
        if (((uintptr_t)row & 15) == 0) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row));
            cnt += __popc(__vsetne4(v.x, 0)) + __popc(__vsetne4(v.y, 0)) + __popc(__vsetne4(v.z, 0)) +
                   __popc(__vsetne4(v.w, 0));
        } else {
            for (int x = 0; x < 16; ++x) cnt += row[x] != 0;
        }
    }
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    if (lane == 0) {
        uint32_t f = (cnt * 15u + 2048u) / 4096u;
        if (cnt && !f) f = 1;
        P.frac[item] = (uint8_t)f;
    }
}

// Fraction map of a chunk, range-coded by one thread (src/mc_codec.c:600-611):
// a chain of 16384 bins, which needs only the material nibbles, so it runs on a
// stream of its own beside the transform and the block coder. Most nibbles repeat
// one of the two extremes, air behind air (four 0 bins) or full behind full
// (four 1 bins); such a nibble is coded straight through, the four splits
// computed one from the other, when the last range shows that none of them
// renormalises. One chunk or many: 0.95 ms as the tail of the sizing pass with
// contexts in local memory, 0.75 ms here, hidden where the transform and the block
// coder take longer (not for the small levels of a pyramid).
__device__ __forceinline__ void frac_bit(Enc &e, uint32_t &p0, uint32_t bit) {
    const uint32_t r0 = (e.range >> 12) * p0;
    if (!bit) { e.range = r0; p0 = after0(p0); }
    else { e.low += r0; e.range -= r0; p0 = after1(p0); }
    enc_norm(e);
}
__device__ __forceinline__ void frac_nibble(Enc &e, uint32_t (&p)[4], uint32_t v) {
    frac_bit(e, p[3], (v >> 3) & 1);
    frac_bit(e, p[2], (v >> 2) & 1);
    frac_bit(e, p[1], (v >> 1) & 1);
    frac_bit(e, p[0], v & 1);
}
__global__ void __launch_bounds__(32) k_fracmap(BlobParams P) {
    if (threadIdx.x) return;
    const int c = blockIdx.x;
    Enc e;
    e.out = P.fmap + (size_t)c * kFmapCap;
    e.cap = kFmapCap; e.len = 0; e.low = 0; e.range = 0xFFFFFFFFu; e.cache = 0; e.pending = 1;
    uint32_t lo[4], mid[4], hi[4];   // contexts behind a nibble of 0, of 1..14, of 15
#pragma unroll
    for (int j = 0; j < 4; ++j) lo[j] = mid[j] = hi[j] = 2048;
    const uint4 *fr = reinterpret_cast<const uint4 *>(P.frac + (size_t)c * kGrid3);
    uint32_t prev = 0;
    uint4 ahead = fr[0];
    for (int i = 0; i < kGrid3 / 16; ++i) {
        const uint4 now = ahead;
        if (i + 1 < kGrid3 / 16) ahead = fr[i + 1];
        const uint32_t w[4] = {now.x, now.y, now.z, now.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t word = w[q];
#pragma unroll 1
            for (int b = 0; b < 4; ++b, word >>= 8) {
                const uint32_t v = word & 15u;
                if (prev == 0) {
                    const uint32_t r1 = (e.range >> 12) * lo[3], r2 = (r1 >> 12) * lo[2];
                    const uint32_t r3 = (r2 >> 12) * lo[1], r4 = (r3 >> 12) * lo[0];
                    if (v == 0 && r4 >= (1u << 24)) {
                        e.range = r4;
                        lo[3] = after0(lo[3]); lo[2] = after0(lo[2]); lo[1] = after0(lo[1]); lo[0] = after0(lo[0]);
                    } else {
                        frac_nibble(e, lo, v);
                    }
                } else if (prev == 15) {
                    const uint32_t s1 = (e.range >> 12) * hi[3], r1 = e.range - s1;
                    const uint32_t s2 = (r1 >> 12) * hi[2], r2 = r1 - s2;
                    const uint32_t s3 = (r2 >> 12) * hi[1], r3 = r2 - s3;
                    const uint32_t s4 = (r3 >> 12) * hi[0], r4 = r3 - s4;
                    if (v == 15 && r4 >= (1u << 24)) {
                        e.low += (uint64_t)s1 + s2 + s3 + s4;
                        e.range = r4;
                        hi[3] = after1(hi[3]); hi[2] = after1(hi[2]); hi[1] = after1(hi[1]); hi[0] = after1(hi[0]);
                    } else {
                        frac_nibble(e, hi, v);
                    }
                } else {
                    frac_nibble(e, mid, v);
                }
                prev = v;
            }
        }
    }
    for (int i = 0; i < 5; ++i) enc_shift(e);
    P.fml[c] = e.len > (uint32_t)kFmapCap ? (uint32_t)kFmapCap : e.len;
}

// Sizing pass, one CTA of 1024 threads per chunk: block-order exclusive scans
// of (present, bytes), the u16 length table and bitmap into side buffers, and
// the blob's total length (0 when every block is air). After k_fracmap.
__global__ void __launch_bounds__(1024) k_blob_layout(BlobParams P) {
    __shared__ uint32_t s_wnp[32], s_wby[32];
    const int c = blockIdx.x, tid = threadIdx.x;
    const int lane = tid & 31, w = tid >> 5;
    const uint32_t *len = P.len + (size_t)c * kGrid3;
    uint32_t *pref = P.scratch + (size_t)c * kGrid3;
    uint32_t l[4], np = 0, bytes = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) { l[i] = len[tid * 4 + i]; np += l[i] != 0; bytes += l[i]; }
    uint32_t snp = np, sby = bytes;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t a = __shfl_up_sync(0xFFFFFFFFu, snp, o);
        uint32_t b = __shfl_up_sync(0xFFFFFFFFu, sby, o);
        if (lane >= o) { snp += a; sby += b; }
    }
    if (lane == 31) { s_wnp[w] = snp; s_wby[w] = sby; }
    __syncthreads();
    if (w == 0) {
        uint32_t a = s_wnp[lane], b = s_wby[lane];
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t x = __shfl_up_sync(0xFFFFFFFFu, a, o);
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, b, o);
            if (lane >= o) { a += x; b += y; }
        }
        s_wnp[lane] = a; s_wby[lane] = b;
    }
    __syncthreads();
    uint32_t slot = snp - np + (w ? s_wnp[w - 1] : 0);
    uint32_t off = sby - bytes + (w ? s_wby[w - 1] : 0);
    const uint32_t np_total = s_wnp[31], by_total = s_wby[31];
    uint16_t *lens16 = P.lens16 + (size_t)c * kGrid3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        pref[tid * 4 + i] = off;
        if (l[i]) { lens16[slot] = (uint16_t)l[i]; slot++; off += l[i]; }
    }
    if (tid < kBitmapBytes) {
        uint32_t byte = 0;
        for (int b = 0; b < 8; ++b) byte |= (len[tid * 8 + b] != 0 ? 1u : 0u) << b;
        P.bitmap[(size_t)c * kBitmapBytes + tid] = (uint8_t)byte;
    }
    if (tid == 0) {
        P.np[c] = np_total;
        P.blob_len[c] = np_total ? (uint64_t)kBlobHdr + P.fml[c] + kBitmapBytes + 2ull * np_total + by_total : 0;
    }
}

// Write pass: header (the hash is k_blob_hash's, patched into the installed blob), fmap, bitmap, lengths and
// the payloads in block order. Grid (64, nchunks), a warp per block.
__global__ void __launch_bounds__(256) k_blob_fill(BlobParams P) {
    const int c = blockIdx.y;
    const uint64_t total = P.blob_len[c];
    if (!total) return;
    uint8_t *blob = P.blobs + P.blob_off[c];
    const uint32_t fml = P.fml[c], np = P.np[c];
    const int tid = threadIdx.x;
    if (blockIdx.x == 0) {
        if (tid == 0) {
            float q = P.header_q[c];
            memcpy(blob, &q, 4);
            for (int i = 4; i < 12; ++i) blob[i] = 0;
            blob[12] = (uint8_t)fml;
            blob[13] = (uint8_t)(fml >> 8);
        }
        const uint8_t *fm = P.fmap + (size_t)c * kFmapCap;
        for (uint32_t i = tid; i < fml; i += blockDim.x) blob[kBlobHdr + i] = fm[i];
        const uint8_t *bm = P.bitmap + (size_t)c * kBitmapBytes;
        for (int i = tid; i < kBitmapBytes; i += blockDim.x) blob[kBlobHdr + fml + i] = bm[i];
        const uint16_t *l16 = P.lens16 + (size_t)c * kGrid3;
        uint8_t *lens = blob + kBlobHdr + fml + kBitmapBytes;
        for (uint32_t i = tid; i < np; i += blockDim.x) {
            lens[2 * i] = (uint8_t)l16[i];
            lens[2 * i + 1] = (uint8_t)(l16[i] >> 8);
        }
    }
    uint8_t *pay = blob + kBlobHdr + fml + kBitmapBytes + 2ull * np;
    const int lane = tid & 31, w = tid >> 5;
    for (int b = blockIdx.x * 8 + w; b < kGrid3; b += gridDim.x * 8) {
        size_t item = (size_t)c * kGrid3 + b;
        uint32_t l = P.len[item];
        if (!l) continue;
        uint32_t off = P.scratch[item];
        const uint8_t *s = P.payload + item * (size_t)kEncCap;
        for (uint32_t i = lane; i < l; i += 32) pay[off + i] = s[i];
    }
}

// ------------------------------------------------------------ xxh64
namespace {
constexpr uint64_t XP1 = 0x9E3779B185EBCA87ull, XP2 = 0xC2B2AE3D27D4EB4Full,
                   XP3 = 0x165667B19E3779F9ull, XP4 = 0x85EBCA77C2B2AE63ull,
                   XP5 = 0x27D4EB2F165667C5ull;
__device__ __forceinline__ uint64_t rotl64(uint64_t x, int r) { return (x << r) | (x >> (64 - r)); }
__device__ __forceinline__ uint64_t xround(uint64_t acc, uint64_t in) { return rotl64(acc + in * XP2, 31) * XP1; }
__device__ __forceinline__ uint64_t ld64u(const uint8_t *p) {
    uint64_t v = 0;
    for (int i = 7; i >= 0; --i) v = (v << 8) | p[i];
    return v;
}

}  // namespace

// The chained hash of a blob (src/mc_archive.c:76-88), one CTA per blob.
//
// XXH64 keeps 4 serial accumulators, acc = rotl(acc + word * P2, 31) * P1, so
// four lanes of the first warp hash and the other warps feed them: they read
// the next tile's words (any alignment), multiply them by P2, which is off the
// chain, and leave the products in shared memory while the current tile is
// hashed. What is left on the chain is an add, a rotate and one multiply, and
// nothing waits on memory. A blob of 6.3 MB: 10.05 ms with one warp loading and
// hashing by turns, 4.2 ms so.
namespace {
constexpr int kHashThreads = 128;
constexpr int kTileStripes = 128;
struct HashSmem {
    uint64_t prod[2][kTileStripes * 4];
    uint64_t h;
};

// 8 little-endian bytes at q; aligned loads inside [base, limit), bytes
// outside it read 0.
__device__ __forceinline__ uint64_t word64(const uint8_t *base, const uint8_t *limit, const uint8_t *q) {
    const uint32_t a = (uint32_t)(uintptr_t)q & 7u;
    const uint8_t *w = q - a;
    if (w >= base && w + 16 <= limit) {
        const uint64_t lo = __ldg(reinterpret_cast<const unsigned long long *>(w));
        if (!a) return lo;
        const uint64_t hi = __ldg(reinterpret_cast<const unsigned long long *>(w) + 1);
        return (lo >> (8 * a)) | (hi << (64 - 8 * a));
    }
    uint64_t v = 0;
    for (int k = 7; k >= 0; --k) v = (v << 8) | (q + k >= base && q + k < limit ? q[k] : 0);
    return v;
}

// XXH64 of [p, p + len) by the whole CTA; the hash in every thread.
__device__ uint64_t xxh64_cta(const uint8_t *base, const uint8_t *limit, const uint8_t *p, uint64_t len, uint64_t seed,
                              HashSmem &S) {
    const int tid = threadIdx.x;
    const uint64_t nstripes = len / 32;
    const uint64_t ntiles = (nstripes + kTileStripes - 1) / kTileStripes;
    auto stripes_of = [&](uint64_t t) { return (int)min((uint64_t)kTileStripes, nstripes - t * kTileStripes); };
    auto fill = [&](uint64_t t, int first, int step) {
        const uint8_t *q = p + t * (kTileStripes * 32);
        const int n = stripes_of(t) * 4;
        for (int w = first; w < n; w += step) S.prod[t & 1][w] = word64(base, limit, q + 8 * w) * XP2;
    };
    uint64_t acc = tid == 0 ? seed + XP1 + XP2 : tid == 1 ? seed + XP2 : tid == 2 ? seed : seed - XP1;
    if (ntiles) fill(0, tid, kHashThreads);
    __syncthreads();
    for (uint64_t t = 0; t < ntiles; ++t) {
        if (tid < 4) {
            const uint64_t *pr = S.prod[t & 1] + tid;
            const int n = stripes_of(t);
#pragma unroll 8
            for (int s = 0; s < n; ++s) acc = rotl64(acc + pr[4 * s], 31) * XP1;
        } else if (tid >= 32 && t + 1 < ntiles) {
            fill(t + 1, tid - 32, kHashThreads - 32);
        }
        __syncthreads();
    }
    if (tid < 32) {
        const uint64_t a0 = __shfl_sync(0xFFFFFFFFu, acc, 0), a1 = __shfl_sync(0xFFFFFFFFu, acc, 1);
        const uint64_t a2 = __shfl_sync(0xFFFFFFFFu, acc, 2), a3 = __shfl_sync(0xFFFFFFFFu, acc, 3);
        if (tid == 0) {
            uint64_t h;
            if (nstripes) {
                h = rotl64(a0, 1) + rotl64(a1, 7) + rotl64(a2, 12) + rotl64(a3, 18);
                h = (h ^ xround(0, a0)) * XP1 + XP4;
                h = (h ^ xround(0, a1)) * XP1 + XP4;
                h = (h ^ xround(0, a2)) * XP1 + XP4;
                h = (h ^ xround(0, a3)) * XP1 + XP4;
            } else {
                h = seed + XP5;
            }
            h += len;
            const uint8_t *q = p + nstripes * 32, *end = p + len;
            for (; end - q >= 8; q += 8) h = rotl64(h ^ xround(0, word64(base, limit, q)), 27) * XP1 + XP4;
            if (end - q >= 4) {
                const uint64_t w = word64(base, limit, q) & 0xFFFFFFFFull;
                h = rotl64(h ^ (w * XP1), 23) * XP2 + XP3;
                q += 4;
            }
            for (; q < end; ++q) h = rotl64(h ^ ((word64(base, limit, q) & 0xFFull) * XP5), 11) * XP1;
            h ^= h >> 33; h *= XP2; h ^= h >> 29; h *= XP3; h ^= h >> 32;
            S.h = h;
        }
    }
    __syncthreads();
    const uint64_t h = S.h;
    __syncthreads();   // S is reused by the next call
    return h;
}

// Over fmap | bitmap | lengths | payloads of the blob at `blob`, len bytes, np
// present blocks.
__device__ uint64_t blob_hash_cta(const uint8_t *base, const uint8_t *limit, const uint8_t *blob, uint64_t len,
                                  uint32_t np, HashSmem &S) {
    const uint16_t fml = (uint16_t)(blob[12] | (blob[13] << 8));
    const uint8_t *fmap = blob + kBlobHdr, *bm = fmap + fml, *lens = bm + kBitmapBytes;
    const uint64_t pay = (uint64_t)kBlobHdr + fml + kBitmapBytes + 2ull * np;
    uint64_t h = xxh64_cta(base, limit, fmap, fml, kHashSeed, S);
    h ^= xxh64_cta(base, limit, bm, kBitmapBytes, h, S);
    h ^= xxh64_cta(base, limit, lens, 2ull * np, h, S);
    h ^= xxh64_cta(base, limit, blob + pay, len - pay, h, S);
    return h;
}
}  // namespace

// Device verify (src/mc_archive.c:1072-1111): the hash of every listed blob of
// an archive held in device memory, compared with the hash stored in the
// blob's header; bad[i] = 1 on a mismatch.
__global__ void __launch_bounds__(kHashThreads) k_verify_hash(const uint8_t *arc, uint64_t arc_len,
                                                              const VerifyItem *items, uint32_t *bad) {
    __shared__ HashSmem S;
    const VerifyItem it = items[blockIdx.x];
    const uint8_t *blob = arc + it.co;
    const uint64_t h = blob_hash_cta(arc, arc + arc_len, blob, it.len, it.np, S);
    if (threadIdx.x == 0) bad[blockIdx.x] = h != ld64u(blob + 4) ? 1u : 0u;
}

// The hash of each assembled blob, 0 for an all-air chunk.
__global__ void __launch_bounds__(kHashThreads) k_blob_hash(BlobParams P) {
    __shared__ HashSmem S;
    const int c = blockIdx.x;
    const uint64_t total = P.blob_len[c];
    uint64_t h = 0;
    if (total) {
        const uint8_t *blob = P.blobs + P.blob_off[c];
        h = blob_hash_cta(blob, blob + total, blob, total, P.np[c], S);
    }
    if (threadIdx.x == 0) P.hash[c] = h;
}

cudaError_t launch_verify_hash(const uint8_t *d_arc, uint64_t arc_len, const VerifyItem *d_items, int n,
                               uint32_t *d_bad, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_verify_hash<<<(unsigned)n, kHashThreads, 0, s>>>(d_arc, arc_len, d_items, d_bad);
    return cudaGetLastError();
}

cudaError_t upload_encode_tables(const float cmf[16][16], const uint16_t scan[kN3], cudaStream_t s) {
    // pageable sources: the copies are staged before these calls return
    uint16_t bend[9];
    for (int i = 1; i < kN3; ++i) {
        const uint32_t b = scan[i] >> 12;
        if ((uint32_t)(scan[i - 1] >> 12) != b) bend[b - 1] = (uint16_t)i;
    }
    bend[7] = kN3;
    bend[8] = 0xFFFF;
    float2 fwd[8][16], inv[16][8];
    for (int k = 0; k < 16; ++k)
        for (int n = 0; n < 8; ++n) fwd[n][k] = inv[k][n] = make_float2(cmf[k][n], cmf[k][n]);
    cudaError_t e = cudaMemcpyToSymbolAsync(c_fwd, fwd, sizeof fwd, 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(c_inv, inv, sizeof inv, 0, cudaMemcpyHostToDevice, s);
    return e != cudaSuccess ? e : cudaMemcpyToSymbolAsync(c_bend, bend, sizeof bend, 0, cudaMemcpyHostToDevice, s);
}

// The items of whole chunks, block by block: made where they are read, instead
// of 1.3 MB for 8 chunks built and uploaded by the host (0.2 ms of a call).
__global__ void __launch_bounds__(256) k_encode_items(EncChunks c, EncItem *items, uint8_t *pay) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x, k = i >> 12, b = i & 4095u;
    EncItem it;
    it.src = (uint64_t)(uintptr_t)(c.vox[k] + (size_t)((b >> 8) * 16) * 65536 + ((b >> 4) & 15) * (16 * 256) + (b & 15) * 16);
    it.sz = 65536;
    it.sy = 256;
    it.out = (uint64_t)(uintptr_t)(pay + (size_t)i * kEncCap);
    it.qslot = c.qslot[k];
    it.tau = c.tau[k];
    it.pad = 0;
    items[i] = it;
}

cudaError_t launch_encode_items(const EncChunks &c, EncItem *d_items, uint8_t *d_pay, cudaStream_t s) {
    if (c.n <= 0) return cudaSuccess;
    k_encode_items<<<c.n * (kGrid3 / 256), 256, 0, s>>>(c, d_items, d_pay);
    return cudaGetLastError();
}

// One wave of CTAs: as many per SM as fit. CTAs walk the blocks with a fixed
// stride, so CTAs beyond one wave would start their whole share late.
static int encode_ctas(int n) {
    static std::atomic<int> occ_by_dev[kMaxDevs];
    const int occ = dev_once(occ_by_dev, [] {
        int o = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_encode, 128, sizeof(EncSmem)) != cudaSuccess || o < 1) o = 1;
        return o;
    });
    return std::min(n, dev_sms() * occ);
}

uint32_t encode_pool_max(int n) {
    const uint32_t ctas = (uint32_t)encode_ctas(n);
    return ctas * (((uint32_t)n + ctas - 1) / ctas) * (2u * kN3);
}

cudaError_t launch_encode(const EncParams &p, cudaStream_t s) {
    if (p.n <= 0) return cudaSuccess;
    const int smem = (int)sizeof(EncSmem);
    // per device: the dynamic shared memory opt-in and the carveout (1), or
    // the error code of the attribute call that failed (negated)
    static std::atomic<int> attr[kMaxDevs];
    const int a = dev_once(attr, [smem] {
        cudaError_t e = cudaFuncSetAttribute(k_encode, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_encode, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared);
        return e == cudaSuccess ? 1 : -(int)e;
    });
    if (a < 0) return (cudaError_t)(-a);
    const int blocks = encode_ctas(p.n);
    k_encode<<<blocks, 128, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_encode_rc(const EncParams &p, cudaStream_t s) {
    if (p.n <= 0) return cudaSuccess;
    // otherwise at least one warp for each of the SMs' four schedulers while a warp
    // still has four blocks or more (8 chunks at q=6: 0.97 ms with 32 lanes, 1.36
    // with 16; 2 chunks at q=1 tau=4: 5.06, 4.41, and 4.39 with 8)
    const int sms = dev_sms();
    if (p.n <= sms) {   // as many blocks as SMs or fewer, the single-block call: a thread and a CTA each
        k_encode_rc_one<<<p.n, 32, 0, s>>>(p);
        return cudaGetLastError();
    }
    int lanes = 32;
    while (lanes > 4 && p.n < lanes * sms * 4) lanes >>= 1;
    const int blocks = ((p.n + lanes - 1) / lanes + kRcWarps - 1) / kRcWarps;
    k_encode_rc<<<blocks < sms * 16 ? blocks : sms * 16, kRcWarps * 32, 0, s>>>(p, lanes);
    return cudaGetLastError();
}

cudaError_t launch_fracmap(const EncParams &e, const BlobParams &p, cudaStream_t s) {
    if (p.nchunks <= 0) return cudaSuccess;
    k_frac_count<<<(unsigned)((e.n + 7) / 8), 256, 0, s>>>(e);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    k_fracmap<<<p.nchunks, 32, 0, s>>>(p);
    return cudaGetLastError();
}
cudaError_t launch_blob_layout(const BlobParams &p, cudaStream_t s) {
    if (p.nchunks <= 0) return cudaSuccess;
    k_blob_layout<<<p.nchunks, 1024, 0, s>>>(p);
    return cudaGetLastError();
}
cudaError_t launch_blob_fill(const BlobParams &p, cudaStream_t s) {
    if (p.nchunks <= 0) return cudaSuccess;
    k_blob_fill<<<dim3(64, p.nchunks), 256, 0, s>>>(p);
    return cudaGetLastError();
}
cudaError_t launch_blob_hash(const BlobParams &p, cudaStream_t s) {
    if (p.nchunks <= 0) return cudaSuccess;
    k_blob_hash<<<p.nchunks, kHashThreads, 0, s>>>(p);
    return cudaGetLastError();
}

}  // namespace mcb

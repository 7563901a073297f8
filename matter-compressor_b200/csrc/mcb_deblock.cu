// mcb_deblock.cu -- the decode-side deblocking filter on the device
// (src/mc_codec.c:561-595, declared at src/matter_compressor.h:106).
//
// The filter works in place, axis by axis: every x face, then every y face,
// then every z face between 16-aligned blocks. A face at coordinate f of its
// axis reads the voxels at f-2, f-1, f, f+1 along the axis and writes f-1 and
// f; faces of one axis sit 16 apart, so no two of them touch a common voxel
// and all faces of an axis run in parallel. One kernel per axis, in stream
// order, gives the reference's result: each axis sees the previous axes'
// output. Volumes of a batch are independent (grid.y).
//
// Neighbours are addressed linearly, like the reference's pointer arithmetic:
// a face in the last voxel of a row (or plane) reads the next row's (plane's)
// first voxel, which no face of the same axis writes. A read past the end of
// the volume -- undefined in the reference -- reads 0.
//
// Three kernels, one per axis in stream order, move the volume's sectors twice
// for the x pass (faces every 16 bytes) and a quarter of the rows and planes twice
// for y and z. k_deblock_tile does the same in one pass over memory wherever
// faces never read across the volume's far edges (see launch_deblock).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "mcb_devinfo.h"
#include "mcb_kernels.h"

namespace mcb {

struct DbParams {
    uint8_t *vol;
    size_t vstride;      // bytes between the volumes of a batch
    size_t total;        // voxels of one volume
    uint32_t nx, ny, nz;
    uint32_t sz;         // ny * nx
    uint32_t nf;         // faces of this pass's axis: (n - 1) / 16 for n > 16, else 0
    uint32_t work;       // face positions of this pass in one volume
    int beta, tc;
};

// One face: p1 p0 | q0 q1, q0 at index i, neighbours `step` apart
// (src/mc_codec.c:563-574).
__device__ __forceinline__ void db_face(uint8_t *v, size_t total, size_t i, size_t step, int beta, int tc) {
    const int p0 = v[i - step], q0 = v[i];
    if (p0 == 0 || q0 == 0) return;          // air is never touched
    const int d = q0 - p0;
    if (abs(d) >= beta) return;              // a real edge is kept
    const int p1 = v[i - 2 * step];
    const int q1 = i + step < total ? v[i + step] : 0;
    const int pn = p1 ? p1 : p0, qn = q1 ? q1 : q0;
    int delta = (4 * d + (pn - qn) + 4) >> 3;
    delta = delta > tc ? tc : delta;
    delta = delta < -tc ? -tc : delta;
    v[i - step] = (uint8_t)min(max(p0 + delta, 1), 255);
    v[i] = (uint8_t)min(max(q0 - delta, 1), 255);
}

// x faces: work = rows (nz*ny) x nf, the face index fastest.
__global__ void __launch_bounds__(256) k_deblock_x(DbParams P) {
    uint8_t *v = P.vol + (size_t)blockIdx.y * P.vstride;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < P.work; g += gridDim.x * blockDim.x) {
        const uint32_t row = g / P.nf, j = g - row * P.nf;
        db_face(v, P.total, (size_t)row * P.nx + 16u * (j + 1u), 1, P.beta, P.tc);
    }
}

// y faces: work = nz x nf x nx, x fastest (coalesced).
__global__ void __launch_bounds__(256) k_deblock_y(DbParams P) {
    uint8_t *v = P.vol + (size_t)blockIdx.y * P.vstride;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < P.work; g += gridDim.x * blockDim.x) {
        const uint32_t t = g / P.nx, x = g - t * P.nx;
        const uint32_t z = t / P.nf, k = t - z * P.nf;
        db_face(v, P.total, (size_t)z * P.sz + (size_t)(16u * (k + 1u)) * P.nx + x, P.nx, P.beta, P.tc);
    }
}

// z faces: work = nf x (ny*nx), the in-plane index fastest.
__global__ void __launch_bounds__(256) k_deblock_z(DbParams P) {
    uint8_t *v = P.vol + (size_t)blockIdx.y * P.vstride;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < P.work; g += gridDim.x * blockDim.x) {
        const uint32_t k = g / P.sz, r = g - k * P.sz;
        db_face(v, P.total, (size_t)(16u * (k + 1u)) * P.sz + r, P.sz, P.beta, P.tc);
    }
}

// The same filter on 16 faces side by side in x: rows p1, p0, q0, q1 as
// 16-byte vectors; p0 and q0 are filtered.
__device__ __forceinline__ void db_filter16(const uint4 P1, uint4 &P0, uint4 &Q0, const uint4 Q1, int beta, int tc) {
    const uint8_t *p1 = reinterpret_cast<const uint8_t *>(&P1), *q1 = reinterpret_cast<const uint8_t *>(&Q1);
    uint8_t *p0 = reinterpret_cast<uint8_t *>(&P0), *q0 = reinterpret_cast<uint8_t *>(&Q0);
#pragma unroll
    for (int b = 0; b < 16; ++b) {
        const int a = p0[b], c = q0[b];
        if (a == 0 || c == 0) continue;
        const int d = c - a;
        if (abs(d) >= beta) continue;
        const int pn = p1[b] ? p1[b] : a, qn = q1[b] ? q1[b] : c;
        int delta = (4 * d + (pn - qn) + 4) >> 3;
        delta = delta > tc ? tc : delta;
        delta = delta < -tc ? -tc : delta;
        p0[b] = (uint8_t)min(max(a + delta, 1), 255);
        q0[b] = (uint8_t)min(max(c - delta, 1), 255);
    }
}
// Used when rows are 16-byte aligned.
__device__ __forceinline__ void db_face16(uint8_t *v, size_t total, size_t i, size_t step, int beta, int tc) {
    const uint4 P1 = *reinterpret_cast<const uint4 *>(v + i - 2 * step);
    uint4 P0 = *reinterpret_cast<const uint4 *>(v + i - step);
    uint4 Q0 = *reinterpret_cast<const uint4 *>(v + i);
    const uint4 Q1 = i + step < total ? *reinterpret_cast<const uint4 *>(v + i + step) : make_uint4(0, 0, 0, 0);
    db_filter16(P1, P0, Q0, Q1, beta, tc);
    *reinterpret_cast<uint4 *>(v + i - step) = P0;
    *reinterpret_cast<uint4 *>(v + i) = Q0;
}

// y faces, 16 x at a time: work = nz x nf x (nx/16).
__global__ void __launch_bounds__(256) k_deblock_y16(DbParams P) {
    uint8_t *v = P.vol + (size_t)blockIdx.y * P.vstride;
    const uint32_t nxs = P.nx >> 4;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < P.work; g += gridDim.x * blockDim.x) {
        const uint32_t t = g / nxs, xs = g - t * nxs;
        const uint32_t z = t / P.nf, k = t - z * P.nf;
        db_face16(v, P.total, (size_t)z * P.sz + (size_t)(16u * (k + 1u)) * P.nx + 16u * xs, P.nx, P.beta, P.tc);
    }
}

// z faces, 16 x at a time: work = nf x (ny*nx/16).
__global__ void __launch_bounds__(256) k_deblock_z16(DbParams P) {
    uint8_t *v = P.vol + (size_t)blockIdx.y * P.vstride;
    const uint32_t s16 = P.sz >> 4;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < P.work; g += gridDim.x * blockDim.x) {
        const uint32_t k = g / s16, r = g - k * s16;
        db_face16(v, P.total, (size_t)(16u * (k + 1u)) * P.sz + 16u * r, P.sz, P.beta, P.tc);
    }
}

// Two faces at a time in packed half precision, where every value of the filter
// is an integer of at most 1024 (beta <= 192: |4d + (pn - qn) + 4| < 1024 for
// every face that passes the gate), so all of it is exact. Voxels are 1024 + v,
// the byte v under the high byte 0x64; differences lose the bias.
constexpr int kHalfBeta = 192;
struct Faces2 { __half2 p, q; };
__device__ __forceinline__ uint32_t h2bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __half2 bitsh2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t pick(uint32_t m, uint32_t a, uint32_t b) { return (a & m) | (b & ~m); }
__device__ __forceinline__ Faces2 db_faces2(uint32_t p1, uint32_t p0, uint32_t q0, uint32_t q1, __half2 beta, __half2 tc) {
    const __half2 zero = __float2half2_rn(1024.0f);   // the voxel 0
    const __half2 P0 = bitsh2(p0), Q0 = bitsh2(q0);
    const __half2 d = __hsub2(Q0, P0);
    const __half2 pn = bitsh2(pick(__hne2_mask(bitsh2(p1), zero), p1, p0));
    const __half2 qn = bitsh2(pick(__hne2_mask(bitsh2(q1), zero), q1, q0));
    // t = 4d + (pn - qn) + 4; floor(t / 8) as t / 8 - 7 / 16 to the nearest, which is never a tie
    const __half2 e = __hadd2(__hsub2(pn, qn), __float2half2_rn(0.5f));
    const __half2 u = __hfma2(d, __float2half2_rn(4.0f), e);
    const __half2 fl = __hfma2(u, __float2half2_rn(0.125f), __float2half2_rn(1536.0f));
    __half2 delta = __hsub2(fl, __float2half2_rn(1536.0f));
    delta = __hmin2(__hmax2(delta, __hneg2(tc)), tc);
    const uint32_t on = __hne2_mask(P0, zero) & __hne2_mask(Q0, zero) & __hlt2_mask(__habs2(d), beta);
    const __half2 lo = __float2half2_rn(1025.0f), hi = __float2half2_rn(1279.0f);
    Faces2 r;
    r.p = bitsh2(pick(on, h2bits(__hmin2(__hmax2(__hadd2(P0, delta), lo), hi)), p0));
    r.q = bitsh2(pick(on, h2bits(__hmin2(__hmax2(__hsub2(Q0, delta), lo), hi)), q0));
    return r;
}
// 16 faces side by side, as db_filter16.
__device__ __forceinline__ void db_filter16h(const uint4 P1, uint4 &P0, uint4 &Q0, const uint4 Q1, __half2 beta,
                                             __half2 tc) {
    constexpr uint32_t kHi = 0x64646464u;
    const uint32_t p1[4] = {P1.x, P1.y, P1.z, P1.w}, q1[4] = {Q1.x, Q1.y, Q1.z, Q1.w};
    uint32_t p0[4] = {P0.x, P0.y, P0.z, P0.w}, q0[4] = {Q0.x, Q0.y, Q0.z, Q0.w};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const Faces2 a = db_faces2(__byte_perm(p1[w], kHi, 0x4140), __byte_perm(p0[w], kHi, 0x4140),
                                   __byte_perm(q0[w], kHi, 0x4140), __byte_perm(q1[w], kHi, 0x4140), beta, tc);
        const Faces2 b = db_faces2(__byte_perm(p1[w], kHi, 0x4342), __byte_perm(p0[w], kHi, 0x4342),
                                   __byte_perm(q0[w], kHi, 0x4342), __byte_perm(q1[w], kHi, 0x4342), beta, tc);
        p0[w] = __byte_perm(h2bits(a.p), h2bits(b.p), 0x6420);
        q0[w] = __byte_perm(h2bits(a.q), h2bits(b.q), 0x6420);
    }
    P0 = make_uint4(p0[0], p0[1], p0[2], p0[3]);
    Q0 = make_uint4(q0[0], q0[1], q0[2], q0[3]);
}

// All three axes in one pass, for rows of whole aligned 16-byte vectors. Tiles
// of whole rows, 8 rows by 8 planes, start 4 voxels before the multiples of 8: a
// face at a multiple of 16 and the four voxels it reads (f - 2 .. f + 1) then lie
// inside one tile, a tile's x faces need no other tile, and neither does the
// order x, y, z. So a tile is read, filtered axis by axis and written back, in
// place, with nothing read that another tile writes.
// A thread holds 16 voxels of the tile's 8 rows of one plane in registers. x
// faces sit between vectors: each thread leaves the two bytes at either end of
// its rows in shared memory and filters the face on either side for its own
// byte. A y face lies between registers. The four planes around a z face go
// through shared memory, one row vector a thread.
// What bounds it: memory, one read and one write of the volume. 16 decoded
// chunks (268 MB): 85 us (a copy takes 86), 141 us as three passes (the x pass
// alone moves every sector both ways); with the faces in integers 122 us, the ALU
// pipe 82 % busy.
constexpr uint32_t kTileMaxVecs = 56;   // row vectors: 448 threads

__global__ void __launch_bounds__(kTileMaxVecs * 8) k_deblock_tile(DbParams P, uint32_t ty) {
    extern __shared__ __align__(16) uint8_t s_db[];
    const uint32_t nseg = P.nx >> 4, nthr = nseg * 8;
    uint4 *s_z = reinterpret_cast<uint4 *>(s_db);                        // [4 planes][8 rows][nseg]
    uint32_t *s_edge = reinterpret_cast<uint32_t *>(s_z + 4 * 8 * nseg);   // [8 rows][8 planes][nseg]
    uint8_t *v = P.vol + (size_t)blockIdx.y * P.vstride;
    const uint32_t tz = blockIdx.x / ty, tyi = blockIdx.x - tz * ty;
    const uint32_t tid = threadIdx.x, pl = tid / nseg, seg = tid - pl * nseg;
    // the tile's rows 8 tyi - 4 + r and planes 8 tz - 4 + pl, those inside the volume
    const int y0 = 8 * (int)tyi - 4, z = 8 * (int)tz - 4 + (int)pl;
    const bool in = z >= 0 && z < (int)P.nz;
    uint8_t *row0 = v + (ptrdiff_t)z * (ptrdiff_t)P.sz + (ptrdiff_t)y0 * (ptrdiff_t)P.nx + 16 * seg;
    uint4 r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int y = y0 + k;
        r[k] = in && y >= 0 && y < (int)P.ny ? *reinterpret_cast<const uint4 *>(row0 + (ptrdiff_t)k * P.nx)
                                             : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) s_edge[k * nthr + tid] = __byte_perm(r[k].x, r[k].w, 0x7610);   // bytes 0, 1, 14, 15
    __syncthreads();
    const __half2 beta = __float2half2_rn((float)P.beta), tc = __float2half2_rn((float)P.tc);
    constexpr uint32_t kHi = 0x64646464u;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {   // rows k and k + 1 at a time
        const uint32_t o0 = __byte_perm(r[k].x, r[k].w, 0x7610), o1 = __byte_perm(r[k + 1].x, r[k + 1].w, 0x7610);
        const uint32_t own01 = __byte_perm(o0, o1, 0x5140), own23 = __byte_perm(o0, o1, 0x7362);   // bytes 0 1, 14 15
        if (seg > 0) {
            const uint32_t l = __byte_perm(s_edge[k * nthr + tid - 1], s_edge[(k + 1) * nthr + tid - 1], 0x7362);
            const uint32_t q = h2bits(db_faces2(__byte_perm(l, kHi, 0x4140), __byte_perm(l, kHi, 0x4342),
                                                __byte_perm(own01, kHi, 0x4140), __byte_perm(own01, kHi, 0x4342), beta,
                                                tc).q);
            r[k].x = __byte_perm(r[k].x, q, 0x3214);
            r[k + 1].x = __byte_perm(r[k + 1].x, q, 0x3216);
        }
        if (seg + 1 < nseg) {
            const uint32_t n = __byte_perm(s_edge[k * nthr + tid + 1], s_edge[(k + 1) * nthr + tid + 1], 0x5140);
            const uint32_t p = h2bits(db_faces2(__byte_perm(own23, kHi, 0x4140), __byte_perm(own23, kHi, 0x4342),
                                                __byte_perm(n, kHi, 0x4140), __byte_perm(n, kHi, 0x4342), beta, tc).p);
            r[k].w = __byte_perm(r[k].w, p, 0x4210);
            r[k + 1].w = __byte_perm(r[k + 1].w, p, 0x6210);
        }
    }
    // the faces inside, at multiples of 16
    if (tyi && (tyi & 1) == 0 && 8 * tyi < P.ny) db_filter16h(r[2], r[3], r[4], r[5], beta, tc);
    if (tz && (tz & 1) == 0 && 8 * tz < P.nz) {
        if (pl >= 2 && pl < 6) {
#pragma unroll
            for (int k = 0; k < 8; ++k) s_z[((pl - 2) * 8 + k) * nseg + seg] = r[k];
        }
        __syncthreads();
        // thread (pl, seg) filters row pl of the face; past the last plane it reads 0
        uint4 *q = s_z + pl * nseg + seg;
        uint4 p0 = q[8 * nseg], q0 = q[16 * nseg];
        db_filter16h(q[0], p0, q0, q[24 * nseg], beta, tc);
        q[8 * nseg] = p0;
        q[16 * nseg] = q0;
        __syncthreads();
        if (pl == 3 || pl == 4) {
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = s_z[((pl - 2) * 8 + k) * nseg + seg];
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int y = y0 + k;
        if (in && y >= 0 && y < (int)P.ny) *reinterpret_cast<uint4 *>(row0 + (ptrdiff_t)k * P.nx) = r[k];
    }
}

static int db_sms() { return dev_sms(); }

static uint32_t faces(uint32_t n) { return n > 16 ? (n - 1) / 16 : 0; }

cudaError_t launch_deblock(uint8_t *d_vol, int count, size_t vstride, int nz, int ny, int nx, int beta, int tc,
                           cudaStream_t s) {
    if (count <= 0 || nz <= 0 || ny <= 0 || nx <= 0) return cudaSuccess;
    if (count > 65535) return cudaErrorInvalidValue;
    const uint64_t sz = (uint64_t)ny * (uint64_t)nx;
    const uint64_t rows = (uint64_t)nz * (uint64_t)ny;
    // every per-pass index of one volume in 32 bits
    if (sz >= (1ull << 32) || rows >= (1ull << 32) || rows * faces((uint32_t)nx) >= (1ull << 32) ||
        (uint64_t)nz * faces((uint32_t)ny) * (uint64_t)nx >= (1ull << 32) ||
        (uint64_t)faces((uint32_t)nz) * sz >= (1ull << 32))
        return cudaErrorInvalidValue;
    DbParams P;
    P.vol = d_vol;
    P.vstride = vstride;
    P.total = (size_t)rows * (size_t)nx;
    P.nx = (uint32_t)nx;
    P.ny = (uint32_t)ny;
    P.nz = (uint32_t)nz;
    P.sz = (uint32_t)sz;
    P.beta = beta;
    P.tc = tc;
    // rows of 16-byte vectors when every row of every volume starts on a 16-byte boundary
    const bool vec = nx % 16 == 0 && ((uintptr_t)d_vol & 15) == 0 && (count == 1 || vstride % 16 == 0);
    // One pass over tiles, unless a y face sits in a plane's last row (ny % 16 ==
    // 1): it reads the next plane's first row as the y pass finds it, which a
    // tile next door may have filtered along z by then. (A z face in the last
    // plane reads 0 either way, and whole vectors leave no x face in a row's last
    // voxel.)
    const uint32_t ty = (uint32_t)(((uint64_t)ny + 11) / 8), tz = (uint32_t)(((uint64_t)nz + 11) / 8);
    const uint64_t tiles = (uint64_t)ty * tz;
    // And where the tiles do not cost more than the passes they save. Without y and
    // z faces the passes leave most rows alone (4096 volumes of 512 x 1 x 16: 16 us,
    // 148 as tiles). Otherwise the tiles' work, warps filled up and rows beyond the
    // edges counted, may be 1.9 times the volume's at row lengths of 64 to 576 and 1.5
    // times elsewhere (400 MB of volumes, tiles / passes: 24 x 24 x 128 at 1.78 times
    // 0.94, 48 x 48 x 96 at 1.81 1.00, 24 x 24 x 96 at 2.37 1.17, 256 x 256 x 32 at 2.12
    // 1.20, 24 x 24 x 640 at 1.78 1.12, 40 x 40 x 640 at 1.44 0.95, 256 x 256 x 48 at
    // 1.41 0.91). CTAs for longer rows fit an SM one fewer at a time (256 x 256 x 896:
    // 0.78, 944: 1.06, 1024: 1.02; 40 x 40: 0.88, 1.26, 1.19).
    const uint32_t nseg = (uint32_t)nx / 16;
    const uint64_t work = tiles * 64 * (uint64_t)((nseg * 8 + 31) / 32 * 64);
    const bool pays = ny > 16 && nz > 16 && 10 * work <= (nx >= 64 && nx <= 576 ? 19u : 15u) * P.total;
    if (vec && beta <= kHalfBeta && nseg <= kTileMaxVecs && !(ny % 16 == 1) && pays && tiles < (1ull << 31)) {
        const size_t smem = (size_t)nseg * (4 * 8 * sizeof(uint4) + 8 * 8 * sizeof(uint32_t));   // 768 B a vector
        k_deblock_tile<<<dim3((unsigned)tiles, (unsigned)count), nseg * 8, smem, s>>>(P, ty);
        return cudaGetLastError();
    }
    const uint32_t cap = (uint32_t)db_sms() * 8u;
    auto grid = [&](uint32_t work) {
        uint32_t b = (work + 255u) / 256u;
        return dim3(b < cap ? b : cap, (unsigned)count);
    };
    P.nf = faces(P.nx);
    P.work = (uint32_t)(rows * P.nf);
    if (P.work) k_deblock_x<<<grid(P.work), 256, 0, s>>>(P);
    P.nf = faces(P.ny);
    P.work = P.nz * P.nf * (vec ? P.nx / 16 : P.nx);
    if (P.work) {
        if (vec) k_deblock_y16<<<grid(P.work), 256, 0, s>>>(P);
        else k_deblock_y<<<grid(P.work), 256, 0, s>>>(P);
    }
    P.nf = faces(P.nz);
    P.work = P.nf * (vec ? P.sz / 16 : P.sz);
    if (P.work) {
        if (vec) k_deblock_z16<<<grid(P.work), 256, 0, s>>>(P);
        else k_deblock_z<<<grid(P.work), 256, 0, s>>>(P);
    }
    return cudaGetLastError();
}

}  // namespace mcb

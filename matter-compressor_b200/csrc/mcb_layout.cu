// mcb_layout.cu -- the layout of a decode batch, made on the device from its
// work items: each item's arena offset and the entropy stage's processing order
// (longest payload first, absent blocks last).
//
// The offsets may be any disjoint ranges of entry_cap(len) entries, and the
// order only has to put similar lengths together (lanes of a warp then finish
// about together, and the longest chains start first), so neither needs a full
// scan or sort: a CTA reserves the entries of its 1024 items with one atomic, and
// the order is a counting sort by length class (see length_class), whose ranks inside
// a class fall as the CTAs arrive. On the host (a stable counting sort over 65536
// lengths, three more arrays built and uploaded) a batch of 46 K items took about
// 0.3 ms of every call that builds its work list; here 10 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mcb_devinfo.h"
#include "mcb_format.h"
#include "mcb_kernels.h"

namespace mcb {

namespace {
constexpr int kThreads = 1024;
constexpr int kClasses = kLayoutClasses;
static_assert(kClasses == kThreads, "one thread per class in the scans");
// Inclusive sum of v over the CTA's threads up to this one.
__device__ __forceinline__ uint32_t cta_scan(uint32_t v, uint32_t *s_warp) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) s_warp[w] = v;
    __syncthreads();
    if (w == 0) {
        uint32_t x = s_warp[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += u;
        }
        s_warp[lane] = x;
    }
    __syncthreads();
    return v + (w ? s_warp[w - 1] : 0);
}
}  // namespace

// Offsets, and how many items each class holds.
__global__ void __launch_bounds__(kThreads) k_layout_count(const DecItem *items, int n, uint64_t *base, uint32_t *ws) {
    __shared__ uint32_t s_cnt[kClasses], s_warp[32];
    __shared__ unsigned long long s_at;
    const int tid = threadIdx.x, i = blockIdx.x * kThreads + tid;
    s_cnt[tid] = 0;
    __syncthreads();
    const uint32_t len = i < n ? __ldg(&items[i].len) : 0u;
    const uint32_t cap = i < n ? entry_cap(len) : 0u;
    if (i < n) atomicAdd(&s_cnt[length_class(len)], 1u);
    const uint32_t upto = cta_scan(cap, s_warp);   // at most 1024 * 12288
    if (tid == kThreads - 1)
        s_at = atomicAdd(reinterpret_cast<unsigned long long *>(ws + 2 * kClasses), (unsigned long long)upto);
    __syncthreads();
    if (i < n) base[i] = (uint64_t)s_at + upto - cap;
    if (s_cnt[tid]) atomicAdd(ws + tid, s_cnt[tid]);
}

// The order: class c's items go to places [start of c, start of c + its count).
__global__ void __launch_bounds__(kThreads) k_layout_order(const DecItem *items, int n, uint32_t *order, uint32_t *ws) {
    __shared__ uint32_t s_cnt[kClasses], s_at[kClasses], s_warp[32];
    const int tid = threadIdx.x, i = blockIdx.x * kThreads + tid;
    s_cnt[tid] = 0;
    __syncthreads();
    const int c = length_class(i < n ? __ldg(&items[i].len) : 0u);
    uint32_t rank = 0;
    if (i < n) rank = atomicAdd(&s_cnt[c], 1u);
    const uint32_t total = ws[tid];
    const uint32_t start = cta_scan(total, s_warp) - total;   // its barriers order the counts too
    s_at[tid] = start + (s_cnt[tid] ? atomicAdd(ws + kClasses + tid, s_cnt[tid]) : 0u);
    __syncthreads();
    if (i < n) order[s_at[c] + rank] = (uint32_t)i;
}

cudaError_t launch_layout(const DecItem *d_items, int n, uint64_t *d_base, uint32_t *d_order, uint32_t *d_ws,
                          cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const cudaError_t e = cudaMemsetAsync(d_ws, 0, sizeof(uint32_t) * kLayoutWords, s);
    if (e != cudaSuccess) return e;
    const unsigned blocks = (unsigned)((n + kThreads - 1) / kThreads);
    k_layout_count<<<blocks, kThreads, 0, s>>>(d_items, n, d_base, d_ws);
    k_layout_order<<<blocks, kThreads, 0, s>>>(d_items, n, d_order, d_ws);
    return cudaGetLastError();
}

cudaError_t preload_layout_kernels() {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, k_layout_count);
    return e != cudaSuccess ? e : cudaFuncGetAttributes(&fa, k_layout_order);
}

}  // namespace mcb

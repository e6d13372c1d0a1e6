// Pieces that the graph kernels of small batches share: radius_graph.cu (lists for the caller) and small_route.cu (lists of an evaluation).
#pragma once
#include "common.cuh"

namespace mlcgb {

constexpr int64_t kMaskNodes = 2048;
constexpr int kMaskStructs = 2048;             // structure boundaries held in shared memory

// Where a kernel leaves {sequence number, edges, status word, another status word} for the waiting host (mapped pinned memory)
struct Publish {
    int64_t *host = nullptr;
    int64_t seq = 0;
    const int32_t *pending = nullptr;
    bool cells_known = false;                  // h[4] = 0: no structure of the batch belongs to the cell or warp kernels
};
__device__ __forceinline__ void publish(const Publish &p, int64_t edges, int status) {
    volatile int64_t *h = p.host;
    h[1] = edges;
    h[2] = status;
    if (!p.cells_known) h[4] = 1;
    h[3] = p.pending ? *reinterpret_cast<const volatile int32_t *>(p.pending) : 0;
    __threadfence_system();
    h[0] = p.seq;
}

// structure boundaries into shared memory: from the sizes (whose prefix sums block 0 also writes out) or from ptr
template <int NT /* threads of the block */>
__device__ __forceinline__ void load_boundaries(int *s_ptr, const int64_t *sizes, int64_t *ptr, int64_t B) {
    __shared__ int s_part[NT / 32];
    if (!sizes) {
        for (int b = threadIdx.x; b <= B; b += NT) s_ptr[b] = (int)ptr[b];
        __syncthreads();
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int64_t b0 = 0; b0 < B; b0 += NT) {
        const int64_t b = b0 + threadIdx.x;
        const int v = b < B ? (int)sizes[b] : 0;
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_part[warp] = inc;
        __syncthreads();
        int before = carry;
        for (int w = 0; w < warp; w++) before += s_part[w];
        if (b < B) s_ptr[b] = before + inc - v;
        for (int w = 0; w < NT / 32; w++) carry += s_part[w];
        __syncthreads();
    }
    if (threadIdx.x == 0) s_ptr[B] = carry;
    __syncthreads();
    if (blockIdx.x == 0)
        for (int b = threadIdx.x; b <= B; b += NT) ptr[b] = s_ptr[b];
}
__device__ __forceinline__ int structure_of(const int *s_ptr, int64_t B, int i) {     // last b with s_ptr[b] <= i (empty structures skipped)
    int lo = 0, hi = (int)B - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_ptr[mid] <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}


// radius_graph.cu: the calling thread's line of mapped memory for the next published result, and the wait for it
int publish_begin(Publish *p);
int publish_wait(const Publish &p, cudaStream_t st);

}  // namespace mlcgb

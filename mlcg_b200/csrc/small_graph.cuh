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

// A structure's size as the kernels take it.  Sizes that do not add up to the points are reported (kSizes), and the boundaries made of them
// are those of N points all the same, ascending: the last structure begins where the others end and takes what is left.
__device__ __forceinline__ int64_t usable_size(int64_t size, int64_t N) { return size < 0 ? 0 : size < N ? size : N; }

// structure boundaries into shared memory: from the sizes (whose prefix sums block 0 also writes out) or from ptr
template <int NT /* threads of the block */>
__device__ __forceinline__ void load_boundaries(int *s_ptr, const int64_t *sizes, int64_t *ptr, int64_t B, int N, int32_t *status) {
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
        const int64_t size = b < B ? sizes[b] : 0;
        const int v = (int)usable_size(size, N);
        if (v != size && blockIdx.x == 0) atomicOr(status, (int)kSizes);
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
        if (b < B) s_ptr[b] = min(before + inc - v, N);
        for (int w = 0; w < NT / 32; w++) carry += s_part[w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        s_ptr[B] = N;
        if (carry != N && blockIdx.x == 0) atomicOr(status, (int)kSizes);
    }
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

// ---- rows of bits: a warp tests the points of a centre's structure and keeps its hits, {hits before the word, word} per 32 points
struct RowHits {
    int total, before_own;                     // hits (without the centre unless `loop`), and those of points before it
    bool own;                                  // the centre is within its own cutoff
};
// centre ci of the structure [lo, lo + n), n <= 2048, by the whole warp
template <typename T>
__device__ __forceinline__ RowHits row_of_bits(const T *__restrict__ pos, int64_t ci, int lo, int n, T r2, bool loop, uint2 *__restrict__ row, int lane) {
    static_assert(kMaskNodes <= 64 * 32, "two words per lane");
    const T xi = pos[3 * ci], yi = pos[3 * ci + 1], zi = pos[3 * ci + 2];
    unsigned m0 = 0, m1 = 0;                   // words `lane` and `32 + lane` of the row
    for (int jb = 0; jb < n; jb += 32) {
        const int j = jb + lane;
        bool hit = false;
        if (j < n) {
            const T *q = pos + 3 * ((int64_t)lo + j);
            hit = dist2_rn(xi, yi, zi, q[0], q[1], q[2]) < r2;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        const int w = jb >> 5;
        if (w == lane) m0 = bal;
        if (w == lane + 32) m1 = bal;
    }
    const int il = (int)ci - lo, sw = il >> 5;         // the centre's own word and bit
    const unsigned own = sw < 32 ? __shfl_sync(0xffffffffu, m0, sw) : __shfl_sync(0xffffffffu, m1, sw & 31);
    const bool self_hit = own >> (il & 31) & 1;
    if (!loop && self_hit) {
        if (lane == sw) m0 &= ~(1u << (il & 31));
        if (lane + 32 == sw) m1 &= ~(1u << (il & 31));
    }
    int p0 = __popc(m0), p1 = __popc(m1);
    const int c0 = p0, c1 = p1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t0 = __shfl_up_sync(0xffffffffu, p0, o), t1 = __shfl_up_sync(0xffffffffu, p1, o);
        if (lane >= o) { p0 += t0; p1 += t1; }
    }
    const int first = __shfl_sync(0xffffffffu, p0, 31), total = first + __shfl_sync(0xffffffffu, p1, 31);
    p0 -= c0;                                          // hits before the word
    p1 += first - c1;
    const int nw = (n + 31) >> 5;
    if (lane < nw) row[lane] = make_uint2((unsigned)p0, m0);
    if (lane + 32 < nw) row[lane + 32] = make_uint2((unsigned)p1, m1);
    const unsigned below = (1u << (il & 31)) - 1u;
    const int nlo0 = p0 + __popc(m0 & below), nlo1 = p1 + __popc(m1 & below);
    const int nlo = sw < 32 ? __shfl_sync(0xffffffffu, nlo0, sw) : __shfl_sync(0xffffffffu, nlo1, sw & 31);
    return {total, nlo, self_hit};
}
constexpr int kDense = 16, kDensePlan = 24;        // of each_hit()
// The k-th set bit of a word that has more than k
__device__ __forceinline__ int nth_bit(unsigned bits, int k) {
    int at = 0;
#pragma unroll
    for (int half = 16; half; half >>= 1) {
        const int c = __popc(bits & ((1u << half) - 1u));
        const bool up = k >= c;
        k -= up ? c : 0;
        at += up ? half : 0;
        bits >>= up ? half : 0;
    }
    return at;
}
// f(rank, local index) for the first `kept` hits of a row of nw words, 32 consecutive ranks at a time: a lane looks for the word of its rank
// among the 32 of the warp, and for the bit in it.  (Word by word, the lanes of the word's bits at work, a row takes as many turns as it
// has words with a hit, most lanes idle: 37 structures of up to 700 points in float64 with distances 99 -> 81 us.)  Where the words
// are full the two take the same number of turns and the search is what is left over: rows of more than DENSE hits for each word with one go
// word by word.  64 structures of 1000 points, float32, us, by ranks alone : by words alone : these lines, a hit in so many of a word's 32,
//   edges alone (16)       9  297 : 326 : 292      18  469 : 432 : 433      23  555 : 501 : 503      all  728 : 661 : 665
//   with their plan (24)   9  287 : 381 : 284      18  490 : 579 : 490      23  605 : 672 : 612      all  872 : 850 : 855
// each_hit_of: of up to 32 words from w0 on, of which lane t holds word w0 + t (whatever it holds beyond the row).
template <int DENSE, typename F>
__device__ __forceinline__ void each_hit_of(uint2 mine, int w0, int nw, int kept, int lane, F &&f) {
    const bool there = w0 + lane < nw;
    if (!there) mine = make_uint2(0u, 0u);
    const int first = (int)__shfl_sync(0xffffffffu, mine.x, 0), last = min(nw - w0, 32) - 1;
    const int before = there ? (int)mine.x : 0x7fffffff;
    const int end = min(kept, (int)__shfl_sync(0xffffffffu, mine.x + (unsigned)__popc(mine.y), last));
    unsigned live = __ballot_sync(0xffffffffu, mine.y != 0u);
    if (end - first > DENSE * __popc(live)) {
        for (; live; live &= live - 1) {
            const int w = __ffs(live) - 1;
            const unsigned bits = __shfl_sync(0xffffffffu, mine.y, w);
            const int rank = (int)__shfl_sync(0xffffffffu, mine.x, w) + __popc(bits & lanemask_lt());
            if ((bits >> lane & 1u) && rank < kept) f(rank, (w0 + w) * 32 + lane);
        }
        return;
    }
    for (int k = first; k < end; k += 32) {
        const int rank = k + lane;
        int w = 0;                                 // the last word with no more hits before it than the rank
#pragma unroll
        for (int step = 16; step; step >>= 1) {
            const int b = __shfl_sync(0xffffffffu, before, w + step);
            if (b <= rank) w += step;
        }
        const unsigned bits = __shfl_sync(0xffffffffu, mine.y, w);
        const int b = __shfl_sync(0xffffffffu, before, w);
        if (rank < end) f(rank, (w0 + w) * 32 + nth_bit(bits, rank - b));
    }
}
template <int DENSE, typename F>
__device__ __forceinline__ void each_hit(const uint2 *__restrict__ row, int nw, int kept, int lane, F &&f) {
    for (int w0 = 0; w0 < nw; w0 += 32) each_hit_of<DENSE>(w0 + lane < nw ? row[w0 + lane] : make_uint2(0u, 0u), w0, nw, kept, lane, f);
}
// The reverse of the edge (i, j) that is hit `rank` of its row, and the pair of the two: from j's row at the word of i (local index il).
// `at`: first edge, kept edges, lower ones among them and pairs before of a row.  Not ok where the list holds no plan (cut short, or sizes
// that do not add up); every index is inside its array if it is.
template <typename I> struct PairPlace {
    I twin, pair;
    bool ok;
};
template <typename I, typename At>
__device__ __forceinline__ PairPlace<I> pair_place(const uint2 *__restrict__ masks, int words, int i, int il, int j, int rank, I P, const At &at) {
    const uint2 rev = masks[(int64_t)j * words + (il >> 5)];
    const int rank_j = (int)rev.x + __popc(rev.y & ((1u << (il & 31)) - 1u));
    const I p = j > i ? at.pairs(i) + (rank - at.lower(i)) : at.pairs(j) + (rank_j - at.lower(j));
    return {at.first(j) + rank_j, p, rank_j >= 0 && rank_j < at.kept(j) && (rev.y >> (il & 31) & 1u) && i != j && p >= 0 && p < P};
}

// radius_graph.cu: the calling thread's line of mapped memory for the next published result, and the wait for it
int publish_begin(Publish *p);
int publish_wait(const Publish &p, cudaStream_t st);

}  // namespace mlcgb

// The node side of the whole-model sequences for small batches (up to kSmallNodes beads).
//
// At these sizes an evaluation is a chain of dependent launches, and what counts is how long one link takes.  A tensor-core kernel
// over node rows takes 8-11 us for its only tile (a 128-row tile on one SM: fp16 conversion, two exchanges and 1400 cycles of
// issue per GEMM, and 32 columns of epilogue per thread), whatever the batch.  Here a CTA takes 1 to 8 rows (small_rows()),
// so the rows spread over the chip, and one kernel does a whole link: the aggregation of its
// nodes, the Linear layers behind it up to the next aggregation, activations and residuals between them, in plain fp32:
//   forward, block l   agg -> lin2, tanh -> lin, + x -> lin1 of block l+1       (last block: output network, its gradient and
//                                                                                 the first step of the force pass instead)
//   force pass         gagg -> aggregation + edge dot products -> lin1^T, + g -> lin^T, tanh' -> lin2^T of block l-1
// and the two along a tangent and back that a force-matching step adds.  Weights (three 64 KB matrices) are copied to shared
// memory while the kernel waits for its predecessor, each waited for in front of its layer (SmallTile says how a layer is split; a
// column and 32 k per thread over tiles of 4 or 8 rows: 61.4 us an evaluation of 64 x 10 beads, with the tiles below 52, and 49 with weights by the
// copy engine and the filters in two CTAs a tile).  Launches per evaluation of L blocks: 2 L + 3 where the tensor-core
// sequence takes 7 L + 7; one evaluation of 64 x 10 beads, two blocks: 154 us of kernels before.
// For many more rows per SM the tensor-core kernels are the faster ones (figures at kSmallNodes).
#include "schnet_internal.cuh"
#include "tc_common.cuh"

namespace mlcgb {

constexpr int kST = 512;                      // threads
constexpr int kWPitch = 132;                  // floats per weight row: 128-bit reads along k by neighbouring columns meet no bank twice

struct SmallNet {                             // pointers of one launch
    const float *w[3];                        // matrices in slots 0..2 ([128][128]; slot 2 of a last block: [Wh][128])
    const float *b2, *b3, *bh, *wo, *bo;      // biases; output layer
    int64_t N, B;
    int Wh;
    int32_t *status;
    const int64_t *ptr, *struct_ptr;
    const int32_t *nbr, *pair_of;
    const float *W, *Wd, *dd;
    float *s;
    int accumulate;
    // inputs and outputs by role (NULL: not wanted / zero)
    const float *in_a, *in_b;                 // gathered operands of the aggregation
    const float *res, *act, *gu, *q, *gE;
    float *o_agg, *o_act, *o_x, *o_next, *o_ah, *o_en, *o_g, *o_gu, *o_gagg, *o_q, *o_yb, *o_gy, *o_r;
    float *o_ub;
};

enum { kSmFwd = 0, kSmFwdLast = 1, kSmBwd = 2, kSmTan = 3, kSmTanLast = 4, kSmRev = 5, kSmRevFirst = 6 };

template <int RT>
struct SmallSmem {
    static constexpr int kW = 0, kWFloats = 128 * kWPitch;                  // three slots
    static constexpr int kS = 3 * kWFloats;                                 // two row tiles [RT][128]
    static constexpr int kX = kS + 2 * RT * 128;                            // partial sums [4][RT][128]; the aggregation's [16][128]
    static constexpr int kXFloats = 16 * 128 > 4 * RT * 128 ? 16 * 128 : 4 * RT * 128;
    static constexpr int kBar = kX + kXFloats;                              // a barrier per slot
    static constexpr size_t kBytes = sizeof(float) * (kBar + 6);
};

__device__ __forceinline__ void fma4s(float4 &acc, const float4 &a, const float4 &b) {
    acc.x = fmaf(a.x, b.x, acc.x); acc.y = fmaf(a.y, b.y, acc.y); acc.z = fmaf(a.z, b.z, acc.z); acc.w = fmaf(a.w, b.w, acc.w);
}
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// What a thread multiplies with in a layer: 16 k of two columns, w[4 i + j] and w[16 + 4 i + j] at k = 32 kq + 8 i + 4 kh + j
struct SmallWeights { float w[32]; };

// A layer over RT rows: warp = 32 columns (warp & 3) by a quarter of k (kq = warp >> 2); lane = two columns (lane & 15) by half of every
// eight k (kh = lane >> 4).  What bounds it is what shared memory hands to registers: a broadcast 128-bit read takes two cycles like any
// 256 bytes, so a second column per thread halves the rows' share (256 -> 128 cycles a row and layer), and the halves of k meet in one
// exchange a row.  (Measured on one SM: broadcast 128-bit reads 2.1 cycles a warp, full ones 4.0; packed multiplications no faster than plain.)
template <int RT>
struct SmallTile {
    static constexpr int RO = (RT + 3) / 4;   // rows a thread holds after a layer: rows rq + 4 i, column c
    float *smem, *x;
    int tid, c, rq, lane, warp;
    int64_t n0, N;
    bool failed = false;                      // a matrix did not arrive

    __device__ __forceinline__ SmallTile(float4 *base, int at_x, int64_t N_)
        : smem(reinterpret_cast<float *>(base)), x(smem + at_x), tid(threadIdx.x), c(threadIdx.x & 127), rq(threadIdx.x >> 7), lane(threadIdx.x & 31),
          warp(threadIdx.x >> 5), n0(0), N(N_) {}
    __device__ __forceinline__ float *slot(int i) const { return smem + SmallSmem<RT>::kW + i * SmallSmem<RT>::kWFloats; }
    __device__ __forceinline__ float *rows(int i) const { return smem + SmallSmem<RT>::kS + i * RT * 128; }
    // The matrices of a launch -> slots, by the copy engine, a row of 512 bytes at a time (by all threads; rows past the end zero).  (Copies of
    // 16 bytes by all lanes kept a CTA that had to wait for its SM, beside the last one's links, from its lists for 1 us: 64 x 10 beads replayed 50.3 -> 48.6 us.)
    __device__ __forceinline__ uint32_t bar(int i) const { return tc::smem_u32(smem + SmallSmem<RT>::kBar) + 8 * i; }
    __device__ __forceinline__ void fetch_all(const float *const (&src)[3], int last_rows) const {
        if (tid == 0) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                tc::mbar_init(bar(i), 1);
                if (src[i]) tc::mbar_expect_bytes(bar(i), (uint32_t)(i == 2 ? last_rows : 128) * 512u);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int row = warp * 8 + lane, rows = i == 2 ? last_rows : 128;
            if (!src[i] || lane >= 8) continue;
            if (row < rows) {
                tc::bulk_load(tc::smem_u32(slot(i) + row * kWPitch), src[i] + row * 128, 512, bar(i));
            } else {
                for (int k = 0; k < 32; k++) reinterpret_cast<float4 *>(slot(i) + row * kWPitch)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    __device__ __forceinline__ void arrived(int i) {
        if (!failed && !tc::mbar_wait(bar(i), 0)) failed = true;
    }
    // matrix [rows][128] -> slot, asynchronously, a group of copies of its own; rows past the end zero
    __device__ __forceinline__ void fetch(int i, const float *src, int nrows) const {
        const uint32_t base = tc::smem_u32(slot(i));
        if (src) {
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int idx = tid + u * kST, row = idx >> 5, ch = idx & 31;
                const int nbytes = row < nrows ? 16 : 0;
                const float *g = row < nrows ? src + row * 128 + ch * 4 : src;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + (row * kWPitch + ch * 4) * 4), "l"(g), "r"(nbytes) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // NT: columns lane & 15 and 16 more, W stored [c][k]; else neighbouring columns, W stored [k][c]: no bank is met twice either way
    template <bool NT> __device__ __forceinline__ int column() const { return (warp & 3) * 32 + (NT ? (lane & 15) : 2 * (lane & 15)); }
    template <bool NT>
    __device__ __forceinline__ SmallWeights weights(const float *Wm) const {
        SmallWeights r;
        const int c0 = column<NT>(), k0 = (warp >> 2) * 32 + (lane >> 4) * 4;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int k = k0 + 8 * i;
            if (NT) {
                const float4 a = *reinterpret_cast<const float4 *>(Wm + c0 * kWPitch + k), b = *reinterpret_cast<const float4 *>(Wm + (c0 + 16) * kWPitch + k);
                r.w[4 * i] = a.x; r.w[4 * i + 1] = a.y; r.w[4 * i + 2] = a.z; r.w[4 * i + 3] = a.w;
                r.w[16 + 4 * i] = b.x; r.w[17 + 4 * i] = b.y; r.w[18 + 4 * i] = b.z; r.w[19 + 4 * i] = b.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 a = *reinterpret_cast<const float2 *>(Wm + (k + j) * kWPitch + c0);
                    r.w[4 * i + j] = a.x;
                    r.w[16 + 4 * i + j] = a.y;
                }
            }
        }
        return r;
    }
    // v[i] = sum_k S[row][k] W(k, c).  Ends with every thread past its reads of S.
    template <bool NT>
    __device__ __forceinline__ void multiply(const float *S, const SmallWeights &m, float (&v)[RO]) const {
        const int kh = lane >> 4, k0 = (warp >> 2) * 32 + kh * 4;
        float acc[RT][2];
#pragma unroll
        for (int r = 0; r < RT; r++) acc[r][0] = acc[r][1] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
            for (int r = 0; r < RT; r++) {
                const float4 a = *reinterpret_cast<const float4 *>(S + r * 128 + k0 + 8 * i);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float *w = m.w + 16 * h + 4 * i;
                    acc[r][h] = fmaf(a.x, w[0], fmaf(a.y, w[1], fmaf(a.z, w[2], fmaf(a.w, w[3], acc[r][h]))));
                }
            }
        }
        const int col = column<NT>() + (NT ? 16 * kh : kh);
#pragma unroll
        for (int r = 0; r < RT; r++) {
            const float mine = kh ? acc[r][1] : acc[r][0], other = kh ? acc[r][0] : acc[r][1];
            x[((warp >> 2) * RT + r) * 128 + col] = mine + __shfl_xor_sync(0xffffffffu, other, 16);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < RO; i++) {
            const int r = rq + 4 * i;
            v[i] = 0.f;
            if (r < RT) v[i] = (x[r * 128 + c] + x[(RT + r) * 128 + c]) + (x[(2 * RT + r) * 128 + c] + x[(3 * RT + r) * 128 + c]);
        }
    }
    template <bool NT>
    __device__ __forceinline__ void layer(const float *S, const float *Wm, float (&v)[RO]) const {
        multiply<NT>(S, weights<NT>(Wm), v);
    }
    __device__ __forceinline__ int64_t node(int i) const { return rq + 4 * i < RT ? n0 + rq + 4 * i : N; }      // (N: none)
    __device__ __forceinline__ float get(const float *p, int i) const { return node(i) < N ? p[node(i) * 128 + c] : 0.f; }
    __device__ __forceinline__ void put(float *p, int i, float v) const {
        if (p && node(i) < N) p[node(i) * 128 + c] = v;
    }
    // values -> row tile for the next layer; every thread sees it after
    __device__ __forceinline__ void hand_on(float *S, const float (&v)[RO]) const {
#pragma unroll
        for (int i = 0; i < RO; i++)
            if (rq + 4 * i < RT) S[(rq + 4 * i) * 128 + c] = v[i];
        __syncthreads();
    }
};

// Aggregation of the tile's nodes, 16 / RT warps per node (a contiguous part of its edges each), eight edges in flight per lane:
//   FORCE    sum_j a[j] W[p], s[e] (+)= xi a[j] W'[p]        TANGENT  sum_j a[j] W[p] + b[j] dd W'[p]  (a NULL: zero)     PLAIN  sum_j a[j] W[p]
enum { kAggPlain = 0, kAggForce = 1, kAggTangent = 2 };

// A warp's part of its row's edges, and of the first 32 of them the neighbours and pairs
struct SmallEdges {
    int64_t k0, k1;
    int32_t j, p;
};
template <int RT>
__device__ __forceinline__ SmallEdges small_edges(const SmallNet &p, const SmallTile<RT> &t) {
    constexpr int WPR = 16 / RT;
    const int part = t.warp % WPR;
    const int64_t n = t.n0 + t.warp / WPR;
    SmallEdges e = {0, 0, 0, 0};
    if (n >= p.N || t.warp >= RT * WPR) return e;
    // (past the first-level cache: this may run before the wait for the kernel in front, where that cache may hold the lists of another call)
    const int64_t b0 = __ldcg(p.ptr + n), b1 = __ldcg(p.ptr + n + 1), per = (b1 - b0 + WPR - 1) / WPR;
    e.k0 = b0 + part * per;
    e.k1 = e.k0 + per < b1 ? e.k0 + per : b1;
    if (e.k0 + t.lane < e.k1) {
        e.j = __ldcg(p.nbr + e.k0 + t.lane);
        e.p = __ldcg(p.pair_of + e.k0 + t.lane);
    }
    return e;
}

template <int MODE, int RT>
__device__ __forceinline__ void small_aggregate(const SmallNet &p, const SmallTile<RT> &t, float *S, const SmallEdges &ed) {
    constexpr int WPR = 16 / RT;                                       // (warps that have no row are idle)
    const int row = t.warp / WPR, lane = t.lane;
    const int64_t n = t.n0 + row;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 *red = reinterpret_cast<float4 *>(t.x);                     // [16][32]
    if (n < p.N && row < RT) {
        const int64_t k0 = ed.k0, k1 = ed.k1;
        const float4 *a4 = reinterpret_cast<const float4 *>(p.in_a) + lane, *b4 = reinterpret_cast<const float4 *>(p.in_b) + lane;
        const float4 *W4 = reinterpret_cast<const float4 *>(p.W) + lane, *Wd4 = reinterpret_cast<const float4 *>(p.Wd) + lane;
        const float4 xi = MODE == kAggForce ? b4[n * 32] : acc;
        const bool with_a = MODE != kAggTangent || p.in_a;
        constexpr int U = MODE == kAggPlain ? 8 : 4;
        for (int64_t c0 = k0; c0 < k1; c0 += 32) {                     // lane t holds edge c0 + t
            const int len = (int)(k1 - c0 < 32 ? k1 - c0 : 32);
            int32_t my_j = ed.j, my_p = ed.p;
            float my_d = 0.f;
            if (lane < len) {
                if (c0 > k0) {
                    my_j = p.nbr[c0 + lane];
                    my_p = p.pair_of[c0 + lane];
                }
                if (MODE == kAggTangent) my_d = p.dd[c0 + lane];
            }
            for (int g = 0; g < len; g += U) {
                float4 va[U], vb[U], w[U], wd[U];
                float dv[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int e = g + u;
                    const int64_t j = __shfl_sync(0xffffffffu, my_j, e & 31), q = __shfl_sync(0xffffffffu, my_p, e & 31);
                    dv[u] = MODE == kAggTangent ? __shfl_sync(0xffffffffu, my_d, e & 31) : 0.f;
                    va[u] = vb[u] = w[u] = wd[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (e < len) {
                        if (with_a) {
                            va[u] = a4[j * 32];
                            w[u] = W4[q * 32];
                        }
                        if (MODE == kAggTangent) vb[u] = b4[j * 32];
                        if (MODE != kAggPlain) wd[u] = Wd4[q * 32];
                    }
                }
                float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int u = 0; u < U; u++) {
                    fma4s(acc, va[u], w[u]);
                    if (MODE == kAggTangent) fma4s(acc, make_float4(dv[u] * vb[u].x, dv[u] * vb[u].y, dv[u] * vb[u].z, dv[u] * vb[u].w), wd[u]);
                    if (MODE == kAggForce)
                        dot[u & 3] = fmaf(xi.x * va[u].x, wd[u].x, fmaf(xi.y * va[u].y, wd[u].y, fmaf(xi.z * va[u].z, wd[u].z, xi.w * va[u].w * wd[u].w)));
                }
                if (MODE == kAggForce) {
                    // four warp sums at once: lane group of eight (lane >> 3) is left with edge 2 (lane >> 4 & 1) + (lane >> 3 & 1)
                    const bool up = lane & 16, up2 = lane & 8;
                    const float d0 = (up ? dot[2] : dot[0]) + __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[2], 16);
                    const float d1 = (up ? dot[3] : dot[1]) + __shfl_xor_sync(0xffffffffu, up ? dot[1] : dot[3], 16);
                    float d = (up2 ? d1 : d0) + __shfl_xor_sync(0xffffffffu, up2 ? d0 : d1, 8);
                    d += __shfl_xor_sync(0xffffffffu, d, 4);
                    d += __shfl_xor_sync(0xffffffffu, d, 2);
                    d += __shfl_xor_sync(0xffffffffu, d, 1);
                    const int e = g + (lane >> 4) * 2 + ((lane >> 3) & 1);
                    if ((lane & 7) == 0 && e < len) p.s[c0 + e] = p.accumulate ? p.s[c0 + e] + d : d;
                }
            }
        }
    }
    red[t.warp * 32 + lane] = acc;
    __syncthreads();
    if (t.tid < RT * 32) {
        const int r = t.tid >> 5;
        float4 v = red[(r * WPR) * 32 + lane];
#pragma unroll
        for (int k = 1; k < WPR; k++) {
            const float4 o = red[(r * WPR + k) * 32 + lane];
            v = make_float4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
        }
        reinterpret_cast<float4 *>(S)[r * 32 + lane] = v;
        if (p.o_agg && t.n0 + r < p.N) reinterpret_cast<float4 *>(p.o_agg)[(t.n0 + r) * 32 + lane] = v;
    }
    __syncthreads();
}

template <int KIND, int RT>
__global__ void __launch_bounds__(kST, 1) small_block_kernel(const __grid_constant__ SmallNet p) {
    extern __shared__ float4 small_smem[];
    using T = SmallTile<RT>;
    constexpr int RO = T::RO;
    T t(small_smem, SmallSmem<RT>::kX, p.N);
    constexpr bool kLast = KIND == kSmFwdLast || KIND == kSmTanLast;
    t.fetch_all(p.w, kLast ? p.Wh : 128);
    // What does not come from the kernel in front is read before the wait for it, a latency of the second-level cache each (the first-level
    // cache may hold what lay there in a call before): biases and the
    // lists of the first tile (the kernel in front began behind those that made the lists).  What does, and is wanted after a layer,
    // is read under the aggregation (64 x 10 beads replayed: 64 -> 60.5 us).
    constexpr bool kForward = KIND == kSmFwd || KIND == kSmFwdLast;
    const float b2 = kForward ? __ldcg(p.b2 + t.c) : 0.f, b3 = kForward ? __ldcg(p.b3 + t.c) : 0.f;
    const float bh = KIND == kSmFwdLast && t.c < p.Wh ? __ldcg(p.bh + t.c) : 0.f, wo = kLast && t.c < p.Wh ? __ldcg(p.wo + t.c) : 0.f;
    t.n0 = (int64_t)blockIdx.x * RT;
    SmallEdges ed = small_edges(p, t);
    pdl_wait();
    pdl_launch_dependents();
    float *S0 = t.rows(0), *S1 = t.rows(1);
    bool ready = false;
    for (; t.n0 < p.N; t.n0 += (int64_t)gridDim.x * RT) {
        if (ready) ed = small_edges(p, t);
        float res[RO], act[RO];
#pragma unroll
        for (int i = 0; i < RO; i++) {
            res[i] = p.res ? t.get(p.res, i) : 0.f;
            act[i] = kForward || KIND == kSmRevFirst ? 0.f : t.get(p.act, i);
        }
        small_aggregate<kForward ? kAggPlain : (KIND == kSmBwd ? kAggForce : kAggTangent), RT>(p, t, S0, ed);
        t.arrived(0);                                                  // (a matrix is waited for in front of its layer)
        ready = true;
        float v[RO], a[RO], q[RO];
        if (KIND == kSmFwd || KIND == kSmFwdLast) {
            t.template layer<true>(S0, t.slot(0), v);                  // lin2 + tanh
#pragma unroll
            for (int i = 0; i < RO; i++) {
                a[i] = tc::tanh_ex2(v[i] + b2);
                t.put(p.o_act, i, a[i]);
            }
            t.arrived(1);
            t.hand_on(S1, a);
            t.template layer<true>(S1, t.slot(1), v);                  // lin + residual
#pragma unroll
            for (int i = 0; i < RO; i++) {
                v[i] += b3 + res[i];
                t.put(p.o_x, i, v[i]);
            }
            t.arrived(2);
            t.hand_on(S0, v);
            t.template layer<true>(S0, t.slot(2), v);                  // lin1 of the next block | output network
            if (KIND == kSmFwd) {
#pragma unroll
                for (int i = 0; i < RO; i++) t.put(p.o_next, i, v[i]);
            } else {
                float y[RO];
#pragma unroll
                for (int i = 0; i < RO; i++) {
                    v[i] = tc::tanh_ex2(v[i] + bh);
                    if (p.o_ah && t.c < p.Wh && t.node(i) < p.N) p.o_ah[t.node(i) * p.Wh + t.c] = v[i];
                    y[i] = v[i] * wo;
                }
                t.hand_on(S1, y);
                if (t.warp < RT && t.n0 + t.warp < p.N) {              // energy of a node
                    float e = (S1[t.warp * 128 + t.lane] + S1[t.warp * 128 + t.lane + 32]) + (S1[t.warp * 128 + t.lane + 64] + S1[t.warp * 128 + t.lane + 96]);
                    e = warp_sum(e);
                    if (t.lane == 0) p.o_en[t.n0 + t.warp] = e + (p.bo ? p.bo[0] : 0.f);
                }
                if (p.o_gagg) {
#pragma unroll
                    for (int i = 0; i < RO; i++) y[i] = wo * fmaf(-v[i], v[i], 1.f);
                    t.hand_on(S0, y);
                    t.template layer<false>(S0, t.slot(2), v);         // g = dE/dx of the last block's output
#pragma unroll
                    for (int i = 0; i < RO; i++) t.put(p.o_g, i, v[i]);
                    t.hand_on(S1, v);
                    t.template layer<false>(S1, t.slot(1), v);
#pragma unroll
                    for (int i = 0; i < RO; i++) {
                        v[i] *= fmaf(-a[i], a[i], 1.f);
                        t.put(p.o_gu, i, v[i]);
                    }
                    t.hand_on(S0, v);
                    t.template layer<false>(S0, t.slot(0), v);
#pragma unroll
                    for (int i = 0; i < RO; i++) t.put(p.o_gagg, i, v[i]);
                }
            }
        } else if (KIND == kSmBwd) {
            t.template layer<false>(S0, t.slot(0), v);                 // lin1^T + residual
#pragma unroll
            for (int i = 0; i < RO; i++) {
                v[i] += res[i];
                t.put(p.o_g, i, v[i]);
            }
            t.arrived(1);
            t.hand_on(S1, v);
            t.template layer<false>(S1, t.slot(1), v);                 // lin^T, tanh' of the block below
#pragma unroll
            for (int i = 0; i < RO; i++) {
                v[i] *= fmaf(-act[i], act[i], 1.f);
                t.put(p.o_gu, i, v[i]);
            }
            t.arrived(2);
            t.hand_on(S0, v);
            t.template layer<false>(S0, t.slot(2), v);                 // lin2^T
#pragma unroll
            for (int i = 0; i < RO; i++) t.put(p.o_gagg, i, v[i]);
        } else if (KIND == kSmTan || KIND == kSmTanLast) {
            t.template layer<true>(S0, t.slot(0), v);
#pragma unroll
            for (int i = 0; i < RO; i++) {
                a[i] = act[i];
                q[i] = -2.f * a[i] * v[i] * t.get(p.gu, i);
                v[i] *= fmaf(-a[i], a[i], 1.f);
                t.put(p.o_act, i, v[i]);
                if (KIND == kSmTan) t.put(p.o_q, i, q[i]);
            }
            t.arrived(1);
            t.hand_on(S1, v);
            t.template layer<true>(S1, t.slot(1), v);
#pragma unroll
            for (int i = 0; i < RO; i++) {
                v[i] += res[i];
                t.put(p.o_x, i, v[i]);
            }
            t.arrived(2);
            t.hand_on(S0, v);
            t.template layer<true>(S0, t.slot(2), v);
            if (KIND == kSmTan) {
#pragma unroll
                for (int i = 0; i < RO; i++) t.put(p.o_next, i, v[i]);
            } else {
#pragma unroll
                for (int i = 0; i < RO; i++) {
                    const int64_t n = t.node(i);
                    float yb = 0.f;
                    if (n < p.N && t.c < p.Wh) {
                        float ge = 0.f;
                        if (p.gE) {                                    // the structure of node n: last b with struct_ptr[b] <= n
                            int64_t lo = 0, hi = p.B - 1;
                            while (lo < hi) {
                                const int64_t mid = (lo + hi + 1) >> 1;
                                if (p.struct_ptr[mid] <= n) lo = mid;
                                else hi = mid - 1;
                            }
                            ge = p.gE[lo];
                        }
                        const float h = p.o_ah[n * p.Wh + t.c], s = fmaf(-h, h, 1.f);
                        yb = wo * s * fmaf(-2.f * h, v[i], ge);
                        p.o_yb[n * p.Wh + t.c] = yb;
                        p.o_gy[n * p.Wh + t.c] = wo * s;
                        p.o_r[n * p.Wh + t.c] = fmaf(ge, h, s * v[i]);
                    }
                    v[i] = yb;
                }
                t.hand_on(S1, v);
                t.template layer<false>(S1, t.slot(2), v);
#pragma unroll
                for (int i = 0; i < RO; i++) t.put(p.o_g, i, v[i]);
                t.hand_on(S0, v);
                t.template layer<false>(S0, t.slot(1), v);
#pragma unroll
                for (int i = 0; i < RO; i++) {
                    v[i] = fmaf(v[i], fmaf(-a[i], a[i], 1.f), q[i]);
                    t.put(p.o_ub, i, v[i]);
                }
                t.hand_on(S1, v);
                t.template layer<false>(S1, t.slot(0), v);
#pragma unroll
                for (int i = 0; i < RO; i++) t.put(p.o_gagg, i, v[i]);
            }
        } else {                                                       // kSmRev, kSmRevFirst
            t.template layer<false>(S0, t.slot(0), v);
#pragma unroll
            for (int i = 0; i < RO; i++) {
                v[i] += res[i];
                t.put(p.o_g, i, v[i]);
            }
            if (KIND == kSmRev) {
                t.arrived(1);
                t.hand_on(S1, v);
                t.template layer<false>(S1, t.slot(1), v);
#pragma unroll
                for (int i = 0; i < RO; i++) {
                    v[i] = fmaf(v[i], fmaf(-act[i], act[i], 1.f), t.get(p.q, i));
                    t.put(p.o_ub, i, v[i]);
                }
                t.arrived(2);
                t.hand_on(S0, v);
                t.template layer<false>(S0, t.slot(2), v);
#pragma unroll
                for (int i = 0; i < RO; i++) t.put(p.o_gagg, i, v[i]);
            }
        }
        __syncthreads();                                               // the tile buffers are free for the next rows
    }
    if (t.failed) atomicOr(p.status, (int)kTensorWait);
}

// Embedding rows and lin1 of the first block, eight nodes
__device__ __forceinline__ void embedding_rows(SmallTile<8> &t, float *S, const int64_t *types, int64_t num_types, const float *table, float *x, float *xl,
                                               int32_t *status) {
    const int64_t n = t.n0 + t.warp;
    if (t.warp < 8) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < t.N) {
            int64_t ty = types[n];
            if (ty < 0 || ty >= num_types) {
                if (t.lane == 0) atomicOr(status, (int)kBadIndex);
                ty = 0;
            }
            v = __ldg(reinterpret_cast<const float4 *>(table + ty * 128) + t.lane);
            reinterpret_cast<float4 *>(x)[n * 32 + t.lane] = v;
        }
        reinterpret_cast<float4 *>(S)[t.warp * 32 + t.lane] = v;
    }
    copies_wait<0>();                                                  // (the weight, under the two latencies of the rows)
    __syncthreads();
    float v[2];
    t.layer<true>(S, t.slot(0), v);
#pragma unroll
    for (int i = 0; i < 2; i++) t.put(xl, i, v[i]);
}

// Distances of the edges, embedding rows and lin1 of the first block (8 rows per CTA and step)
__global__ void __launch_bounds__(kST, 1)
small_start_kernel(const float *__restrict__ pos, const int64_t *__restrict__ types, const int32_t *__restrict__ row0, const int32_t *__restrict__ row1,
                   int64_t N, int64_t E, int64_t num_types, const float *__restrict__ table, const float *__restrict__ W1, float *__restrict__ d,
                   float *__restrict__ x, float *__restrict__ xl, int32_t *__restrict__ status) {
    extern __shared__ float4 small_smem[];
    constexpr int RT = 8;
    SmallTile<RT> t(small_smem, SmallSmem<RT>::kX, N);
    // (a CTA of edges alone, where there are more than 64 to a bead, brings nothing: nothing would wait for it before the CTA is gone)
    if ((int64_t)blockIdx.x * RT < N) t.fetch(0, W1, 128);
    pdl_wait();
    pdl_launch_dependents();
    for (int64_t e = (int64_t)blockIdx.x * kST + threadIdx.x; e < E; e += (int64_t)gridDim.x * kST) {
        const int64_t i = row0[e], j = row1[e];
        float v = 0.f;
        if (i < 0 || i >= N || j < 0 || j >= N) {
            atomicOr(status, (int)kBadIndex);
        } else {
            v = sqrtf(dist2_rn(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], pos[3 * j], pos[3 * j + 1], pos[3 * j + 2]));
        }
        d[e] = v;
    }
    for (t.n0 = (int64_t)blockIdx.x * RT; t.n0 < N; t.n0 += (int64_t)gridDim.x * RT) {
        __syncthreads();
        embedding_rows(t, t.rows(0), types, num_types, table, x, xl, status);
    }
}

// The first two launches of an evaluation that makes its own lists (SmallGraph).  The graph of a small batch used to be four links
// in front of the filters (clear, count with the last block scanning, a host read of the edge count, fill, distances with the embedding
// layer): of 85 us for 64 x 10 beads 20 were gone before its lists lay there, 7 of them waiting for the host.  Here the
// counting blocks share a launch with the embedding layer, every block of the second launch scans the at most 2048 degrees for
// itself, distances are written with the edges, the filters load their weights meanwhile, and the host looks at the count once
// everything is launched: 84 -> 68 us an evaluation of 64 x 10 beads, 89 -> 75 of 73 beads, 72 -> 64 replayed.  Above kMaskNodes the
// degrees no longer fit a block.
//   blocks [0, count_blocks): 16 beads each, a warp per bead: hits as bits with the hits before each word, degree (bit 30: cut short)
//   the others: embedding rows and lin1 of the first block, 8 rows at a time
constexpr int kDegCut = 1 << 30;
struct SmallStartSmem {
    static constexpr int kS = 128 * kWPitch, kX = kS + 8 * 128;            // one weight slot, one row tile, partial sums
    static constexpr size_t kBytes = sizeof(float) * (kX + 4 * 8 * 128);
};

__global__ void __launch_bounds__(kST, 2)
small_graph_count_kernel(const float *__restrict__ pos, const SmallGraph g, int64_t N, int64_t B, float r2, int count_blocks,
                         const int64_t *__restrict__ types, int64_t num_types, const float *__restrict__ table, const float *__restrict__ W1,
                         float *__restrict__ x, float *__restrict__ xl, int32_t *__restrict__ status) {
    extern __shared__ float4 small_smem[];
    __shared__ int s_ptr[kMaskStructs + 1];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x >= count_blocks) {
        SmallTile<8> t(small_smem, SmallStartSmem::kX, N);
        t.fetch(0, W1, 128);
        for (t.n0 = (int64_t)(blockIdx.x - count_blocks) * 8; t.n0 < N; t.n0 += (int64_t)(gridDim.x - count_blocks) * 8) {
            __syncthreads();
            embedding_rows(t, t.smem + SmallStartSmem::kS, types, num_types, table, x, xl, status);
        }
        return;
    }
    load_boundaries<kST>(s_ptr, g.sizes, g.ptr, B, (int)N, status);
    const int64_t ci = (int64_t)blockIdx.x * (kST / 32) + warp;
    if (ci >= N) return;
    const int i = (int)ci, b = structure_of(s_ptr, B, i), lo = s_ptr[b], n = min(s_ptr[b + 1], (int)N) - lo;
    const RowHits h = row_of_bits<float>(pos, ci, lo, n, r2, false, g.masks + ci * ((N + 31) >> 5), lane);
    if (lane == 0) {
        // (the cluster rule keeps max_nn + 1 of a bead whose own index comes after as many hits)
        const int64_t most = h.own && h.before_own >= g.max_nn + 1 ? g.max_nn + 1 : g.max_nn;
        const int k = h.total < most ? h.total : (int)most;
        g.deg[i] = k | (k < h.total ? kDegCut : 0);
        g.upper[i] = k > h.before_own ? k - h.before_own : 0;
    }
}

constexpr int kFillThreads = 1024;
__global__ void __launch_bounds__(kFillThreads, 1)
small_graph_fill_kernel(const float *__restrict__ pos, const SmallGraph g, int64_t N, int64_t B, float *__restrict__ d, int32_t *__restrict__ status) {
    __shared__ int s_ptr[kMaskStructs + 1], s_off[kMaskNodes + 1], s_uoff[kMaskNodes + 1];
    __shared__ uint64_t s_part[kFillThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_all = (int)N;
    pdl_launch_dependents();
    pdl_wait();
    // (the host's line is written by a block of its own: its system-wide fence held a block with edges up for 2.5 us)
    const bool publishes = g.pub.host && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0;
    const int sizes = publishes ? __ldcg(status) & kSizes : 0;                                // (what the count found)
    for (int b = threadIdx.x; b <= B; b += kFillThreads) s_ptr[b] = (int)g.ptr[b];
    static_assert(kMaskNodes == 2 * kFillThreads, "two beads per thread");
    const int i0 = 2 * threadIdx.x;
    const int d0 = i0 < n_all ? g.deg[i0] : 0, d1 = i0 + 1 < n_all ? g.deg[i0 + 1] : 0, u0 = i0 < n_all ? g.upper[i0] : 0, u1 = i0 + 1 < n_all ? g.upper[i0 + 1] : 0;
    const bool cut = __syncthreads_or((d0 | d1) & kDegCut);
    const int k0 = d0 & (kDegCut - 1), k1 = d1 & (kDegCut - 1);
    const uint64_t own = ((uint64_t)(uint32_t)(u0 + u1) << 32) | (uint32_t)(k0 + k1);      // (upper degrees above, degrees below: neither reaches 2^31)
    uint64_t inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_part[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint64_t v = s_part[lane];
        const uint64_t mine = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += t;
        }
        s_part[lane] = v - mine;
        if (lane == 31) s_off[kMaskNodes] = (int)(uint32_t)v;
    }
    __syncthreads();
    const int64_t total = s_off[kMaskNodes];
    const bool bad = cut || total > g.capacity || (total & 1);
    const uint64_t before = s_part[warp] + inc - own;
    const int e0 = (int)(uint32_t)before, p0 = (int)(before >> 32);
    __syncthreads();                                   // (the total has been read)
    s_off[i0] = e0; s_off[i0 + 1] = e0 + k0;
    s_uoff[i0] = p0; s_uoff[i0 + 1] = p0 + u0;
    if (threadIdx.x == kFillThreads - 1) { s_off[kMaskNodes] = (int)total; s_uoff[kMaskNodes] = p0 + u0 + u1; }
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            g.counts[0] = bad ? 0 : total;
            g.counts[1] = bad ? 0 : total >> 1;
            if (!g.pub.host && bad) atomicOr(status, (cut ? (int)kTruncated : 0) | (total > g.capacity ? (int)kCapacity : 0) | (total & 1 ? (int)kAsymmetric : 0));
        }
        if (i0 <= n_all) g.offsets[i0] = bad ? 0 : e0;
        if (i0 + 1 <= n_all) g.offsets[i0 + 1] = bad ? 0 : e0 + k0;
        if (i0 + 2 == n_all) g.offsets[n_all] = bad ? 0 : total;
    }
    if (publishes) publish(g.pub, total, (cut ? (int)kTruncated : 0) | sizes);
    if (bad) return;
    __syncthreads();
    const int words = (n_all + 31) >> 5, P = (int)(total >> 1);
    struct {
        const int *off, *uoff;
        __device__ int first(int k) const { return off[k]; }
        __device__ int kept(int k) const { return off[k + 1] - off[k]; }
        __device__ int lower(int k) const { return kept(k) - (uoff[k + 1] - uoff[k]); }
        __device__ int pairs(int k) const { return uoff[k]; }
    } const at = {s_off, s_uoff};
    for (int i = blockIdx.x * (kFillThreads / 32) + warp; i < n_all; i += gridDim.x * (kFillThreads / 32)) {
        const int b = structure_of(s_ptr, B, i), lo = s_ptr[b], n = min(s_ptr[b + 1], n_all) - lo, il = i - lo;
        const int off = s_off[i], kept = s_off[i + 1] - off;
        if (kept == 0) continue;
        const float xi = pos[3 * i], yi = pos[3 * i + 1], zi = pos[3 * i + 2];
        each_hit<kDensePlan>(g.masks + (int64_t)i * words, (n + 31) >> 5, kept, lane, [&](int rank, int jl) {
            const int slot = off + rank, j = lo + jl;
            const float d2 = dist2_rn(xi, yi, zi, pos[3 * j], pos[3 * j + 1], pos[3 * j + 2]);
            const auto place = pair_place(g.masks, words, i, il, j, rank, P, at);
            // (structure sizes that do not add up: reported, and every index written stays inside its array)
            if (!place.ok) atomicOr(status, (int)kAsymmetric);
            g.row1[slot] = j;
            g.twin[slot] = place.ok ? place.twin : slot;
            g.pair_of[slot] = place.ok ? place.pair : 0;
            const float r = sqrtf(d2);
            d[slot] = r;
            if (place.ok && j > i) g.pair_d[place.pair] = r;
        });
    }
}

// Forces and energies: the dot products of the first block taken here in both directions (a node's edges by WPN warps, so nothing is
// written per edge), those of the other blocks read from s.  A latency chain: with one warp per node, four edges at a time, it took
// 4.5-4.9 us behind the last link, most of it the later edges' turns.  Eight warps a node or four (small_finish()), an evaluation replayed, us:
//   beads   73    128    146    200    250    296    300    400    560    640 (10 a chain)   1000   1400   2000
//   8      41.1   45.1   49.2   49.2   57.4   55.2   57.1   59.1   61.6   60.1               84.0   119.3  135.4
//   4      43.0   45.6   50.8   51.0   58.0   55.5   57.5   60.0   61.6   58.0               82.2   116.8  131.4
// (two: 2-4 us more up to 640 beads, 129.3 at 2000.)  They meet between 300 and 640 beads, the sooner the fewer
// edges a bead has; the line lies at two beads an SM.
constexpr int kFinishThreads = 256;
template <int WPN>
__global__ void __launch_bounds__(kFinishThreads)
small_finish_kernel(const float *__restrict__ pos, const float *__restrict__ d, const float *__restrict__ gagg, const float *__restrict__ xl,
                    const float *__restrict__ Wd, const float *__restrict__ s, const int64_t *__restrict__ ptr, const int32_t *__restrict__ nbr,
                    const int32_t *__restrict__ pair_of, const int32_t *__restrict__ twin, int64_t N, int node_blocks, float *__restrict__ grad, float sign,
                    const float *__restrict__ en, const int64_t *__restrict__ struct_ptr, int64_t B, float *__restrict__ energy) {
    constexpr int kWarps = kFinishThreads / 32, kNodes = kWarps / WPN;
    __shared__ float s_sum[kWarps][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x >= node_blocks) {                                // energies, a warp per structure
        const int64_t b = (int64_t)((int)blockIdx.x - node_blocks) * kWarps + warp;
        if (b >= B) return;
        const int64_t n0 = __ldcg(struct_ptr + b), n1 = __ldcg(struct_ptr + b + 1);
        pdl_wait();
        float e = 0.f;
        for (int64_t k = n0 + lane; k < n1; k += 32) e += en[k];
        e = warp_sum(e);
        if (lane == 0) energy[b] = e;
        return;
    }
    const int64_t n = (int64_t)blockIdx.x * kNodes + warp / WPN;
    const bool mine = n < N;
    // (lists, distances and positions lie there long before the kernel in front is done.  All of them past the first-level cache, as in
    // small_edges(): a program that moves its positions in place leaves other coordinates at the same addresses)
    int64_t k0 = 0, k1 = 0;
    int32_t my_j = 0, my_p = 0, my_t = 0;
    float my_d = 0.f, x = 0.f, y = 0.f, z = 0.f;
    const auto edge = [&](int64_t k) {
        my_j = __ldcg(nbr + k);
        my_p = __ldcg(pair_of + k);
        if (s) my_t = __ldcg(twin + k);
        my_d = __ldcg(d + k);
        const float *pi = pos + 3 * n, *pj = pos + 3 * (int64_t)my_j;
        x = __ldcg(pi) - __ldcg(pj);
        y = __ldcg(pi + 1) - __ldcg(pj + 1);
        z = __ldcg(pi + 2) - __ldcg(pj + 2);
    };
    if (mine) {
        const int64_t b0 = __ldcg(ptr + n), b1 = __ldcg(ptr + n + 1), per = (b1 - b0 + WPN - 1) / WPN;
        k0 = b0 + (warp % WPN) * per;
        k1 = k0 + per < b1 ? k0 + per : b1;
        if (k0 + lane < k1) edge(k0 + lane);
    }
    pdl_wait();
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
    if (k0 < k1) {
        const float4 *g4 = reinterpret_cast<const float4 *>(gagg) + lane, *x4 = reinterpret_cast<const float4 *>(xl) + lane;
        const float4 *Wd4 = reinterpret_cast<const float4 *>(Wd) + lane;
        const float4 gi = g4[n * 32], xi = x4[n * 32];
        for (int64_t c0 = k0; c0 < k1; c0 += 32) {
            const int len = (int)(k1 - c0 < 32 ? k1 - c0 : 32);
            float my_s = 0.f;
            if (lane < len) {
                if (c0 > k0) edge(c0 + lane);
                if (s) my_s = s[c0 + lane] + s[my_t];
            }
            for (int g = 0; g < len; g += 4) {
                float dot[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int64_t j = __shfl_sync(0xffffffffu, my_j, (g + u) & 31), q = __shfl_sync(0xffffffffu, my_p, (g + u) & 31);
                    dot[u] = 0.f;
                    if (g + u < len) {
                        const float4 gj = g4[j * 32], xj = x4[j * 32], w = Wd4[q * 32];
                        dot[u] = fmaf(xi.x * gj.x + xj.x * gi.x, w.x, fmaf(xi.y * gj.y + xj.y * gi.y, w.y, fmaf(xi.z * gj.z + xj.z * gi.z, w.z,
                                      (xi.w * gj.w + xj.w * gi.w) * w.w)));
                    }
                }
                const bool up = lane & 16, up2 = lane & 8;
                const float d0 = (up ? dot[2] : dot[0]) + __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[2], 16);
                const float d1 = (up ? dot[3] : dot[1]) + __shfl_xor_sync(0xffffffffu, up ? dot[1] : dot[3], 16);
                float v = (up2 ? d1 : d0) + __shfl_xor_sync(0xffffffffu, up2 ? d0 : d1, 8);
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                // edge u of the four sits in lanes 8 (2 (u >> 1) + (u & 1)): to the lane that holds the edge
                const float got = __shfl_sync(0xffffffffu, v, (lane & 3) * 8);
                if (lane >= g && lane < g + 4 && lane < len) my_s += got;
            }
            if (lane < len) {
                const float w = my_d > 0.f ? sign * my_s / my_d : 0.f;
                s0 = fmaf(w, x, s0);
                s1 = fmaf(w, y, s1);
                s2 = fmaf(w, z, s2);
            }
        }
        s0 = warp_sum(s0); s1 = warp_sum(s1); s2 = warp_sum(s2);
    }
    if (lane == 0) { s_sum[warp][0] = s0; s_sum[warp][1] = s1; s_sum[warp][2] = s2; }
    __syncthreads();
    if (mine && warp % WPN == 0 && lane < 3) {
        float v = s_sum[warp][lane];
#pragma unroll
        for (int k = 1; k < WPN; k++) v += s_sum[warp + k][lane];
        grad[n * 3 + lane] = v;
    }
}

template <typename Kern>
static int small_configure(Kern kern, size_t bytes, bool *done) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return check_launch();
        done[dev] = true;
    }
    return MLCGB_OK;
}

// Rows of a tile.  Fewer rows make a link shorter while the chip has an SM for every tile (one pass), and while it has two, one for the
// link before, a tile's weights arrive under that link.  Chains of 12 A, three blocks, us an evaluation with tiles of
//   beads     73 (10 A)   146    200    270    400    560   640 (10 a chain)   800   1000   1400   1700   2000
//   1 row        46        59     67     73     91
//   2            48        48     57     61     74     79     89
//   3            50        50     53     59     65     75     76      90
//   4            52        53     55     57     65     65     78      94     88    126    133
//   6            57        59     61     67     72     67     67      81     97    121    124    160
//   8            62        63     65     71     78     67     69      83     77    130    135    141
// (9 of 640 beads, 72 tiles: 73; weights of two layers held in registers for one row a tile: 46.3 against 46.2)
// The links of a training step go by the same line.  Kernels of a step (forward and backward) of the same chains, us:
//   beads     73    146    200    270    400    560    640    800   1000   1184   1204   1400   1700   2000   2368
//   1 row    123    137    164    172    210    250    274    338    413    458    488    535    649    732    828
//   2        128    142    137    142    185    193    217    247    322    335    372    384    466    511    571
//   3        135    151    143    145    153    197    185    220    298    304    316    366    408    455    512
//   4        143    159    149    150    159    165    192    231    269    277    322    345    379    432    452
//   6        158    180    168    168    176    183    160    196    290    305    321    322    363    425    449
//   8        167    195    179    178    187    192    168    206    246    253    324    352    384    384    401
// Where the two disagree (146 to 400 beads: a row less) the line costs a step 3-5 % of its kernels, which take a third of its time there.
static int small_rows(int64_t N) {
    constexpr int64_t kHalf = kNumSM / 2;
    if (N <= 3 * kHalf) return (int)((N + kHalf - 1) / kHalf);
    if (N <= 4 * kNumSM) return 4;
    if (N <= 6 * kNumSM) return 6;
    if (N <= 8 * kNumSM) return 8;
    return N <= 12 * kNumSM ? 6 : 8;                                   // (two passes)
}
template <int KIND, int RT>
static int small_launch_rt(const SmallNet &p, bool early, cudaStream_t st) {
    static bool done[64] = {false};
    if (int rc = small_configure(small_block_kernel<KIND, RT>, SmallSmem<RT>::kBytes, done)) return rc;
    const int64_t tiles = (p.N + RT - 1) / RT;
    launch_early(early, small_block_kernel<KIND, RT>, dim3((unsigned)(tiles < kNumSM ? tiles : kNumSM)), dim3(kST), SmallSmem<RT>::kBytes, st, p);
    return check_launch();
}
template <int KIND>
static int small_launch(const SmallNet &p, cudaStream_t st, bool early = true) {
    TimelineScope timeline_scope("small_block", st);
    early = early && g_chain_depth > 0;                                // (weights are read before the wait, as launch_with_weights() has it)
    switch (small_rows(p.N)) {
        case 0: case 1: return small_launch_rt<KIND, 1>(p, early, st);
        case 2: return small_launch_rt<KIND, 2>(p, early, st);
        case 3: return small_launch_rt<KIND, 3>(p, early, st);
        case 4: return small_launch_rt<KIND, 4>(p, early, st);
        case 6: return small_launch_rt<KIND, 6>(p, early, st);
        default: return small_launch_rt<KIND, 8>(p, early, st);
    }
}

int small_start(const SmallForward &f, cudaStream_t st) {
    TimelineScope timeline_scope("small_start", st);
    static bool done[64] = {false};
    if (int rc = small_configure(small_start_kernel, SmallSmem<8>::kBytes, done)) return rc;
    int64_t grid = (f.N + 7) / 8;
    if (grid < (f.E + kST - 1) / kST) grid = (f.E + kST - 1) / kST;
    if (grid > kNumSM) grid = kNumSM;
    launch_with_weights(small_start_kernel, dim3((unsigned)grid), dim3(kST), SmallSmem<8>::kBytes, st, f.pos, f.types, f.row0, f.row1, f.N, f.E, f.w->num_types,
               (const float *)f.w->embedding, (const float *)f.w->blocks[0].lin1_w, f.d, f.x[0], f.xl[0], f.status);
    return check_launch();
}

int small_graph_start(const SmallForward &f, const SmallGraph &g, cudaStream_t st) {
    TimelineScope timeline_scope("small_graph_start", st);
    static bool done[64] = {false};
    if (int rc = small_configure(small_graph_count_kernel, SmallStartSmem::kBytes, done)) return rc;
    const int count_blocks = (int)((f.N + kST / 32 - 1) / (kST / 32)), tiles = (int)((f.N + 7) / 8);
    // (launched plainly: it writes what the call before may still read, and what follows may read weights behind it)
    small_graph_count_kernel<<<count_blocks + (tiles < kNumSM ? tiles : kNumSM), kST, SmallStartSmem::kBytes, st>>>(
        f.pos, g, f.N, f.B, (float)(g.r * g.r), count_blocks, f.types, f.w->num_types, (const float *)f.w->embedding, (const float *)f.w->blocks[0].lin1_w, f.x[0],
        f.xl[0], f.status);
    if (int rc = check_launch()) return rc;
    const unsigned fill_blocks = (unsigned)((f.N + kFillThreads / 32 - 1) / (kFillThreads / 32)) + (g.pub.host ? 1 : 0);
    launch_pdl(small_graph_fill_kernel, dim3(fill_blocks), dim3(kFillThreads), 0, st, f.pos, g, f.N, f.B, f.d,
               f.status);
    return check_launch();
}

static SmallNet small_net(const SmallForward &f, int64_t l) {
    SmallNet p = {};
    p.N = f.N;
    p.B = f.B;
    p.Wh = (int)f.w->head_width;
    p.status = f.status;
    p.ptr = f.ptr;
    p.nbr = f.row1;
    p.pair_of = f.pair_of;
    p.W = f.W + l * f.wstride;
    p.Wd = f.Wd ? f.Wd + l * f.wstride : nullptr;
    p.wo = (const float *)f.w->head_out;
    p.bo = (const float *)f.w->head_out_b;
    p.bh = (const float *)f.w->head_b;
    p.s = f.s;
    return p;
}

int small_forward(const SmallForward &f, cudaStream_t st) {
    const int64_t L = f.w->num_blocks;
    for (int64_t l = 0; l < L; l++) {
        const mlcgb_schnet_block &w = f.w->blocks[l];
        SmallNet p = small_net(f, l);
        p.w[0] = (const float *)w.lin2_w;
        p.w[1] = (const float *)w.lin_w;
        p.w[2] = (const float *)(l + 1 < L ? f.w->blocks[l + 1].lin1_w : f.w->head_W);
        p.b2 = (const float *)w.lin2_b;
        p.b3 = (const float *)w.lin_b;
        p.in_a = f.xl[l];
        p.res = f.x[l];
        p.o_agg = f.agg[l];
        p.o_act = f.a[l];
        p.o_x = f.x[l + 1];
        // The lists are read before the wait, which is sound behind a kernel that has waited for those that made them: the filters, or a
        // link.  Lists without room for an edge have no filters, and the first link would stand behind the kernel that writes the offsets.
        const bool early = l > 0 || f.E > 0;
        if (l + 1 < L) {
            p.o_next = f.xl[l + 1];
            if (int rc = small_launch<kSmFwd>(p, st, early)) return rc;
        } else {
            p.o_ah = f.ah;
            p.o_en = f.en;
            p.o_g = f.g[l];
            p.o_gu = f.gu[l];
            p.o_gagg = f.want_grad ? f.gagg[l] : nullptr;
            if (int rc = small_launch<kSmFwdLast>(p, st, early)) return rc;
        }
    }
    for (int64_t l = L - 1; l > 0 && f.want_grad; l--) {
        const mlcgb_schnet_block &below = f.w->blocks[l - 1];
        SmallNet p = small_net(f, l);
        p.w[0] = (const float *)f.w->blocks[l].lin1_w;
        p.w[1] = (const float *)below.lin_w;
        p.w[2] = (const float *)below.lin2_w;
        p.in_a = f.gagg[l];
        p.in_b = f.xl[l];
        p.accumulate = l != L - 1;
        p.res = f.g[l];
        p.act = f.a[l - 1];
        p.o_agg = f.gxl[l];
        p.o_g = f.g[l - 1];
        p.o_gu = f.gu[l - 1];
        p.o_gagg = f.gagg[l - 1];
        if (int rc = small_launch<kSmBwd>(p, st)) return rc;
    }
    return MLCGB_OK;
}

int small_finish(const SmallForward &f, const int32_t *twin, const int64_t *struct_ptr, float *energy, float *grad, float sign, cudaStream_t st) {
    TimelineScope timeline_scope("small_finish", st);
    const auto go = [&](auto kern, int nodes) {                          // nodes per block
        const int node_blocks = f.want_grad && grad ? (int)((f.N + nodes - 1) / nodes) : 0;
        launch_pdl(kern, dim3((unsigned)(node_blocks + (f.B + kFinishThreads / 32 - 1) / (kFinishThreads / 32))), dim3(kFinishThreads), 0, st, f.pos,
                   (const float *)f.d, (const float *)f.gagg[0], (const float *)f.xl[0], (const float *)f.Wd,
                   (const float *)(f.w->num_blocks > 1 ? f.s : nullptr), f.ptr, f.row1, f.pair_of, twin, f.N, node_blocks, grad, sign, (const float *)f.en,
                   struct_ptr, f.B, energy);
    };
    if (f.N <= 2 * kNumSM) go(small_finish_kernel<8>, kFinishThreads / 32 / 8);
    else go(small_finish_kernel<4>, kFinishThreads / 32 / 4);
    return check_launch();
}

int small_backward(const SmallForward &f, const SmallBackward &b, cudaStream_t st) {
    const int64_t L = f.w->num_blocks;
    for (int64_t l = 0; l < L; l++) {
        const mlcgb_schnet_block &w = f.w->blocks[l];
        SmallNet p = small_net(f, l);
        p.struct_ptr = b.struct_ptr;
        p.dd = b.dd;
        p.w[0] = (const float *)w.lin2_w;
        p.w[1] = (const float *)w.lin_w;
        p.w[2] = (const float *)(l + 1 < L ? f.w->blocks[l + 1].lin1_w : f.w->head_W);
        p.in_a = l > 0 ? b.xlt[l] : nullptr;
        p.in_b = f.xl[l];
        p.res = l > 0 ? b.xt[l - 1] : nullptr;
        p.act = f.a[l];
        p.gu = f.gu[l];
        p.o_agg = b.aggt[l];
        p.o_act = b.at[l];
        p.o_x = b.xt[l];
        if (l + 1 < L) {
            p.o_q = b.q[l];
            p.o_next = b.xlt[l + 1];
            if (int rc = small_launch<kSmTan>(p, st)) return rc;
        } else {
            p.gE = b.gE;
            p.o_ah = f.ah;
            p.o_yb = b.yb;
            p.o_gy = b.gy;
            p.o_r = b.r;
            p.o_g = b.xb[l + 1];
            p.o_ub = b.ub[l];
            p.o_gagg = b.agb[l];
            if (int rc = small_launch<kSmTanLast>(p, st)) return rc;
        }
    }
    for (int64_t l = L - 1; l >= 0; l--) {
        SmallNet p = small_net(f, l);
        p.dd = b.dd;
        p.w[0] = (const float *)f.w->blocks[l].lin1_w;
        p.in_a = b.agb[l];
        p.in_b = f.gagg[l];
        p.res = b.xb[l + 1];
        p.o_agg = b.xlb[l];
        p.o_g = b.xb[l];
        if (l > 0) {
            p.w[1] = (const float *)f.w->blocks[l - 1].lin_w;
            p.w[2] = (const float *)f.w->blocks[l - 1].lin2_w;
            p.act = f.a[l - 1];
            p.q = b.q[l - 1];
            p.o_ub = b.ub[l - 1];
            p.o_gagg = b.agb[l - 1];
            if (int rc = small_launch<kSmRev>(p, st)) return rc;
        } else {
            if (int rc = small_launch<kSmRevFirst>(p, st)) return rc;
        }
    }
    return MLCGB_OK;
}

}  // namespace mlcgb

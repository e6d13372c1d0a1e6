// Edge-sized GEMMs of the filter network on the sm_100a tensor cores, fp32-equivalent.
//
// The composable (training) path needs plain GEMMs whose tall dimension is the edge count and whose
// other two dimensions are the widths of the filter network (128 and at most 128):
//   NT  C[E,N] = A[E,K] B[N,K]^T (+ bias)     forward of a Linear layer
//   NN  C[E,N] = A[E,K] B[K,N]                gradient w.r.t. the layer input
//   TN  C[M,N] = A[E,M]^T B[E,N]              gradient w.r.t. the weight (contraction over edges)
// Every fp32 operand is carried as an fp16 pair (hi + lo, ~22 bits) and each product runs as
// hi*hi + hi*lo + lo*hi with fp32 accumulation in tensor memory, like the fused eval-mode kernels.
// Rows of A (NT/NN) are scaled by a power of two so that their largest magnitude sits in [8,16);
// TN scales each 128-edge tile of A and of B by one power of two and accumulates the tiles in registers.
#include "schnet_internal.cuh"
#include "tc_common.cuh"
#include "tensor_map.cuh"
#include "tn_jobs.cuh"

namespace mlcgb {

constexpr int kGT = 512;   // threads: thread = (row of the tile, 32-column quarter)

struct GemmTcSmem {
    static constexpr int kB = 0;                 // operand tile hi | lo (2 x 32 KB)
    static constexpr int kStageA = 65536;        // fp32 stage 64 KB
    static constexpr int kStageB = 131072;       // fp32 stage 64 KB (TN only)
    static constexpr int kMisc = 196608;         // exchange [4][128] f32, bias [128], barrier, TMEM slot, flags
    static constexpr int kTotal = kMisc + 4096 + 1024;
};

__device__ __forceinline__ float4 *gstage(uint8_t *stage, int row, int chunk) {
    return reinterpret_cast<float4 *>(stage + row * 512 + ((chunk ^ (row & 7)) << 4));
}
__device__ __forceinline__ float *gstage_elem(uint8_t *stage, int row, int col) {
    return reinterpret_cast<float *>(stage + row * 512 + ((((col >> 2) ^ (row & 7)) << 4) | ((col & 3) << 2)));
}

// rows [row0, row0+128) x cols [0, ncols) of a row-major [nrows_total, ncols] fp32 matrix -> stage, zero-filled
// outside; whole rows are read by consecutive lanes
__device__ __forceinline__ void load_tile_to_stage(uint8_t *stage, const float *__restrict__ src, int64_t row0, int64_t nrows_total,
                                                   int ncols) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool vec = (ncols & 3) == 0 && ((uintptr_t)src & 15) == 0;
#pragma unroll 1
    for (int i = 0; i < 8; i++) {
        const int row = warp * 8 + i;
        const int64_t gr = row0 + row;
        if (vec) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (gr < nrows_total && lane * 4 < ncols) v = __ldcs(reinterpret_cast<const float4 *>(src + gr * ncols) + lane);
            *gstage(stage, row, lane) = v;
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int col = lane + 32 * c;
                *gstage_elem(stage, row, col) = (gr < nrows_total && col < ncols) ? src[gr * ncols + col] : 0.f;
            }
        }
    }
}

// The same, asynchronously (cp.async, 16 bytes per lane) for rows whose length is a multiple of four floats: used to
// fetch the next tile while the current one is processed.  Out-of-range chunks are zero-filled by the copy itself.
__device__ __forceinline__ void prefetch_tile_to_stage(uint8_t *stage, const float *__restrict__ src, int64_t row0, int64_t nrows_total,
                                                       int ncols) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = warp * 8 + i;
        const int64_t gr = row0 + row;
        const bool ok = gr < nrows_total && lane * 4 < ncols;
        const float *g = ok ? src + gr * ncols + lane * 4 : src;
        const uint32_t dst = tc::smem_u32(gstage(stage, row, lane));
        const int nbytes = ok ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(g), "r"(nbytes) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// rows [row0, row0+128) of a row-major [nrows_total, ncols] fp32 matrix (ncols a multiple of four) -> 32-column boxes in
// the 128-byte swizzle, asynchronously; whole rows are read by consecutive lanes
__device__ __forceinline__ void prefetch_tile_to_boxes(uint8_t *stage, const float *__restrict__ src, int64_t row0, int64_t nrows_total,
                                                       int ncols) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = warp * 8 + i;
        const int64_t gr = row0 + row;
        const bool ok = gr < nrows_total && lane * 4 < ncols;
        const float *g = ok ? src + gr * ncols + lane * 4 : src;
        const uint32_t dst = tc::smem_u32(box_chunk(stage, lane >> 3, row, lane & 7));
        const int nbytes = ok ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(g), "r"(nbytes) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void wait_prefetch() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// ------------------------------------------------------------------------------------------------ NT / NN
template <int MODE>   // 0 NT, 1 NN
__global__ void __launch_bounds__(kGT, 1)
gemm_tc_rows_kernel(const float *__restrict__ A, const float *__restrict__ B, const float *__restrict__ bias, int64_t E, int N, int K,
                    float *__restrict__ C, int32_t *__restrict__ status) {
    using namespace tc;
    using L = GemmTcSmem;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *sB_hi = smem + L::kB, *sB_lo = sB_hi + 32768;
    uint8_t *stages[2] = {smem + L::kStageA, smem + L::kStageB};   // input tiles, double-buffered; outputs reuse the current one
    float *s_red = reinterpret_cast<float *>(smem + L::kMisc);
    float *s_bias = s_red + 512;
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_bias + 128);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 1);
    int *s_err = reinterpret_cast<int *>(s_tmem + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & 127, qt = tid >> 7, col0 = qt * 32;
    constexpr float kWS = 64.f;
    // operand tile of the weight: NT: rows = n, K-major;  NN: rows = k, read as an MN-major operand
    const int wrows = MODE == 0 ? N : K, wcols = MODE == 0 ? K : N;
    const int wpad = wcols <= 64 ? 64 : 128;
    if (load_weight_tile<true>(sB_hi, sB_lo, B, wrows, wcols, wpad, kWS) && blockIdx.x == 0) atomicOr(status, (int)kWeightRange);
    if (tid < 128) s_bias[tid] = (bias && tid < N) ? bias[tid] : 0.f;
    const uint32_t bar = smem_u32(s_bar);
    if (tid == 0) {
        mbar_init(bar, 1);
        *s_err = 0;
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_u32(s_tmem), 256);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const int ksteps = MODE == 0 ? wpad / 16 : (K + 15) / 16;
    const int nmma = MODE == 0 ? 128 : wpad;
    uint32_t phase = 0;

    const int64_t ntiles = (E + kRows - 1) / kRows;
    const bool async_in = (K & 3) == 0 && ((uintptr_t)A & 15) == 0;
    int sidx = 0;
    if (async_in && blockIdx.x < ntiles) prefetch_tile_to_stage(stages[0], A, (int64_t)blockIdx.x * kRows, E, K);
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, sidx ^= 1) {
        uint8_t *stage = stages[sidx];
        if (async_in) {
            wait_prefetch();
            __syncthreads();          // this tile has landed; the other stage was fully consumed one iteration ago
            const int64_t next = tile + gridDim.x;
            if (next < ntiles) prefetch_tile_to_stage(stages[sidx ^ 1], A, next * kRows, E, K);
        } else {
            load_tile_to_stage(stage, A, tile * kRows, E, K);
            __syncthreads();
        }
        float x[32];
        float rmax = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const float4 v = *gstage(stage, r, (col0 >> 2) + w);
            x[4 * w] = v.x; x[4 * w + 1] = v.y; x[4 * w + 2] = v.z; x[4 * w + 3] = v.w;
            rmax = fmaxf(fmaxf(rmax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
        s_red[qt * 128 + r] = rmax;
        __syncthreads();
        const float sc = row_scale(fmaxf(fmaxf(s_red[r], s_red[128 + r]), fmaxf(s_red[256 + r], s_red[384 + r])));
        if (col0 < ksteps * 16) store_a_tmem<true>(tmem + 128 + lane_off, col0, x, sc);
        tmem_wait_st();
        tc_fence_before();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after();
            issue_gemm_ts<true>(tmem, tmem + 128, smem_u32(sB_hi), smem_u32(sB_lo), ksteps, MODE, nmma);
            mma_commit(bar);
        }
        if (!mbar_wait(bar, phase)) *s_err = 1;
        phase ^= 1;
        tc_fence_after();
        if (col0 < nmma) {
            float v[32];
            tmem_ld32(tmem + lane_off + col0, v);
            const float inv = 1.f / (sc * kWS);
#pragma unroll
            for (int w = 0; w < 8; w++)
                *gstage(stage, r, (col0 >> 2) + w) = make_float4(fmaf(v[4 * w], inv, s_bias[col0 + 4 * w]), fmaf(v[4 * w + 1], inv, s_bias[col0 + 4 * w + 1]),
                                                                 fmaf(v[4 * w + 2], inv, s_bias[col0 + 4 * w + 2]), fmaf(v[4 * w + 3], inv, s_bias[col0 + 4 * w + 3]));
        }
        tc_fence_before();
        __syncthreads();
        if (*s_err) break;
        const bool vec = (N & 3) == 0 && ((uintptr_t)C & 15) == 0;
#pragma unroll 1
        for (int i = 0; i < 8; i++) {
            const int row = warp * 8 + i;
            const int64_t gr = tile * kRows + row;
            if (gr >= E) continue;
            if (vec) {
                if (lane * 4 < N) __stcs(reinterpret_cast<float4 *>(C + gr * N) + lane, *gstage(stage, row, lane));
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int col = lane + 32 * c;
                    if (col < N) C[gr * N + col] = *gstage_elem(stage, row, col);
                }
            }
        }
        __syncthreads();
    }
    tc_fence_before();
    __syncthreads();
    if (*s_err && tid == 0) atomicOr(status, 8);
    if (warp == 0) tmem_free(tmem, 256);
}

// ------------------------------------------------------------------------------------------------ NT / NN, pipelined
// Fast path of the two row-wise modes (K and N multiples of four, 16-byte aligned A and C, at least one full tile):
//  * input tiles arrive in one shared-memory stage by cp.async (whole rows per warp); the copy of tile i+2 is issued
//    as soon as tile i+1 has been read out of the stage;
//  * two operand blocks and two accumulators in tensor memory: the conversion of tile i+1 (row scale, fp16 hi/lo, store
//    to TMEM) and its MMAs are issued before the epilogue of tile i, so the tensor core works under both;
//  * the output tile goes to a second stage (32-column boxes, 128-byte swizzle) and leaves through tensor stores that
//    drain while the next tile is processed.
// Epilogues (EPI): 0 none; 1 tanh; 2 + aux; 3 * (1 - aux^2), the derivative of tanh given its output.  `aux` is a matrix
// shaped like C; its tile is copied into the output stage while the next tile is converted and combined there.
// EPI 4 is a transform of the input instead: A[m,k] <- aux[k] * (1 - A[m,k]^2) with a vector aux[K], applied as the tile is read
// (the derivative of a tanh layer followed by a dot product with aux, fed straight into the next GEMM).
enum { kEpiNone = 0, kEpiTanh = 1, kEpiAdd = 2, kEpiTanhGrad = 3, kProTanhGradVec = 4 };
template <int MODE>   // 0 NT, 1 NN
__global__ void __launch_bounds__(kGT, 1)
gemm_tc_rows_pipe_kernel(const float *__restrict__ A, const float *__restrict__ B, const float *__restrict__ bias, int64_t E, int N, int K,
                         const float *__restrict__ aux, int epi, const __grid_constant__ CUtensorMap cmap, const uint8_t *__restrict__ image,
                         int32_t *__restrict__ status) {
    using namespace tc;
    using L = GemmTcSmem;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *sB_hi = smem + L::kB, *sB_lo = sB_hi + 32768;
    uint8_t *s_in = smem + L::kStageA, *s_out = smem + L::kStageB;
    float *s_red = reinterpret_cast<float *>(smem + L::kMisc);
    float *s_bias = s_red + 512;
    float *s_vec = s_bias + 128;                                     // input-transform vector (EPI 4)
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_vec + 128);     // two barriers, one per accumulator; the weight's
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 3);
    int *s_err = reinterpret_cast<int *>(s_tmem + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int r = tid & 127, qt = tid >> 7, col0 = qt * 32;
    constexpr float kWS = 64.f;
    const int64_t ntiles = (E + kRows - 1) / kRows;
    const int64_t step = gridDim.x, t0 = blockIdx.x;
    const int wrows = MODE == 0 ? N : K, wcols = MODE == 0 ? K : N;
    const int wpad = wcols <= 64 ? 64 : 128;
    if (!image && load_weight_tile<true>(sB_hi, sB_lo, B, wrows, wcols, wpad, kWS) && blockIdx.x == 0) atomicOr(status, (int)kWeightRange);
    if (tid < 128) {
        s_bias[tid] = (bias && tid < N) ? bias[tid] : 0.f;
        s_vec[tid] = (epi == kProTanhGradVec && tid < K) ? aux[tid] : 0.f;      // (a parameter vector, not a result of the kernels before)
    }
    const uint32_t bar0 = smem_u32(s_bar);
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init(bar0 + 16, 1);
        *s_err = 0;
        if (image) fetch_image(smem_u32(sB_hi), image, bar0 + 16);
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_u32(s_tmem), 512);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();                                    // set-up done (weights only); A, aux and C belong to the kernels before
    pdl_launch_dependents();
    if (t0 < ntiles) prefetch_tile_to_stage(s_in, A, t0 * kRows, E, K);
    const uint32_t tmem = *s_tmem;                 // accumulators at columns [0,128) [128,256), operands at [256,384) [384,512)
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const int ksteps = MODE == 0 ? wpad / 16 : (K + 15) / 16;
    const int nmma = MODE == 0 ? 128 : wpad;
    const uint32_t b_hi = smem_u32(sB_hi), b_lo = smem_u32(sB_lo);
    uint32_t phase_bits = 0;          // bit b: parity the next wait on barrier b looks for
    bool have_weight = !image;

    // the tile that has landed in the input stage: row scale, operand store, MMAs into accumulator `buf`; then the copy of
    // tile `following` (if any) into the stage.  Returns the row's scale.
    auto convert_issue = [&](int buf, int64_t following) {
        wait_prefetch();
        __syncthreads();
        float x[32];
        float rmax = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            float4 v = *gstage(s_in, r, (col0 >> 2) + w);
            if (epi == kProTanhGradVec) {
                const float4 u = *reinterpret_cast<const float4 *>(s_vec + col0 + 4 * w);
                v = make_float4(u.x * fmaf(-v.x, v.x, 1.f), u.y * fmaf(-v.y, v.y, 1.f), u.z * fmaf(-v.z, v.z, 1.f), u.w * fmaf(-v.w, v.w, 1.f));
            }
            x[4 * w] = v.x; x[4 * w + 1] = v.y; x[4 * w + 2] = v.z; x[4 * w + 3] = v.w;
            rmax = fmaxf(fmaxf(rmax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
        s_red[qt * 128 + r] = rmax;
        __syncthreads();                            // also: everybody has read the stage
        if (following < ntiles) prefetch_tile_to_stage(s_in, A, following * kRows, E, K);
        const float sc = row_scale(fmaxf(fmaxf(s_red[r], s_red[128 + r]), fmaxf(s_red[256 + r], s_red[384 + r])));
        const uint32_t ta = tmem + 256 + buf * 128;
        if (col0 < ksteps * 16) store_a_tmem<true>(ta + lane_off, col0, x, sc);
        tmem_wait_st();
        tc_fence_before();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            if (!have_weight && !mbar_wait(bar0 + 16, 0)) *s_err = 1;
            have_weight = true;
            tc_fence_after();
            issue_gemm_ts<true>(tmem + buf * 128, ta, b_hi, b_lo, ksteps, MODE, nmma);
            mma_commit(bar0 + 8 * buf);
        }
        return sc;
    };

    float sc_cur = 1.f;
    if (t0 < ntiles) sc_cur = convert_issue(0, t0 + step);
    int buf = 0;
    const int nboxes = (N + 31) >> 5;
    for (int64_t tile = t0; tile < ntiles; tile += step, buf ^= 1) {
        float sc_next = 1.f;
        const bool with_aux = epi == kEpiAdd || epi == kEpiTanhGrad;
        if (with_aux) {                             // the aux tile travels to the output stage under the conversion below
            if (tid == 0) bulk_wait_read<0>();      // the stores of the previous tile have read the output stage
            __syncthreads();
            prefetch_tile_to_boxes(s_out, aux, tile * kRows, E, N);
        }
        if (tile + step < ntiles) sc_next = convert_issue(buf ^ 1, tile + 2 * step);
        if (!mbar_wait(bar0 + 8 * buf, (phase_bits >> buf) & 1u)) *s_err = 1;
        phase_bits ^= 1u << buf;
        tc_fence_after();
        if (with_aux) wait_prefetch();              // (also waits for the input tile just requested)
        else if (tid == 0) bulk_wait_read<0>();
        __syncthreads();
        if (col0 < nmma) {
            float v[32];
            tmem_ld32(tmem + buf * 128 + lane_off + col0, v);
            const float inv = 1.f / (sc_cur * kWS);
#pragma unroll
            for (int w = 0; w < 8; w++) {
                float4 o = make_float4(fmaf(v[4 * w], inv, s_bias[col0 + 4 * w]), fmaf(v[4 * w + 1], inv, s_bias[col0 + 4 * w + 1]),
                                       fmaf(v[4 * w + 2], inv, s_bias[col0 + 4 * w + 2]), fmaf(v[4 * w + 3], inv, s_bias[col0 + 4 * w + 3]));
                float4 *slot = box_chunk(s_out, qt, r, w);
                if (epi == kEpiTanh) {
                    o = make_float4(tanh_ex2(o.x), tanh_ex2(o.y), tanh_ex2(o.z), tanh_ex2(o.w));
                } else if (epi == kEpiAdd) {
                    const float4 a4 = *slot;
                    o = make_float4(o.x + a4.x, o.y + a4.y, o.z + a4.z, o.w + a4.w);
                } else if (epi == kEpiTanhGrad) {
                    const float4 a4 = *slot;
                    o = make_float4(o.x * fmaf(-a4.x, a4.x, 1.f), o.y * fmaf(-a4.y, a4.y, 1.f), o.z * fmaf(-a4.z, a4.z, 1.f), o.w * fmaf(-a4.w, a4.w, 1.f));
                }
                *slot = o;
            }
        }
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (*s_err) break;
        if (tid == 0) {
            for (int b = 0; b < nboxes; b++) tensor_store_box(&cmap, 32 * b, (int)(tile * kRows), s_out + b * 16384);
            bulk_commit();
        }
        sc_cur = sc_next;
    }
    wait_prefetch();
    bulk_wait_all();
    tc_fence_before();
    __syncthreads();
    if (*s_err && tid == 0) atomicOr(status, 8);
    if (warp == 0) tmem_free(tmem, 512);
}

// ------------------------------------------------------------------------------------------------ two Linear layers chained
// The two node-sized layers that follow the aggregation of an interaction block, and their counterparts in the force pass,
// as one kernel: the 128-row tile stays on the chip between the two GEMMs.
//   FWD (NT, NT):  mid = tanh(A Wa^T + ba)  (stored: the force pass reads it)      C = aux + mid Wb^T + bb
//   BWD (NN, NN):  mid = (A Wa) * (1 - aux^2)  (stored where wanted)                C = mid Wb
// and, for the weight gradients of a force-matching step, the same two along a tangent and back (a: the block's tanh outputs):
//   TAN (NT, NT):  u = A Wa^T,  mid = (1 - a^2) u,  q_out = -2 a u gu               C = aux + mid Wb^T      (ext0 = a, ext1 = gu)
//   REV (NN, NN):  mid = (A Wa) (1 - aux^2) + q                                     C = mid Wb              (ext0 = q)
// LINKED: a third layer on the tile while it is on the chip (ChainLink, schnet_internal.cuh): behind the forward kinds the next block's
// first layer or the output network's, in front of the backward ones the transpose of the same; its result, the gradient of the block's
// output, then leaves on the way.  There is no room for three weights: the first and the third take turns in one place, each fetched by
// bulk copy as soon as the other's GEMM is over.
// All widths are 128 (but the third layer's outer one).  Shared memory: two weight tiles as fp16 hi/lo pairs (2 x 64 KB) and 64 KB of
// boxes through which every tile enters and leaves.  One accumulator and one operand block of tensor memory, used by the
// GEMMs of a tile one after the other.
// Bound by latency: a tile's layers follow one another at one CTA per SM.  So nothing in a tile waits for more than it needs: a warp's
// 32 x 32 part of every tile comes and goes through a box of its own (asynchronous copies and whole 128-byte pieces by its lanes), the
// four warps of the same rows meet for the rows' largest entry, and all sixteen only at the operand, by arriving at a barrier that a
// warp waits for which issues the products and fetches the weights.  With the whole tile in one stage and barriers of the CTA at every
// turn of it (twelve a tile) a launch over 51200 rows (three tiles a CTA)
// took 45.6 us forward and 42 back; it takes 42.9 and 38.5.
// A layer in a kernel of its own pays for a launch, barriers and tensor memory, a tile's way in and out.
struct ChainSmem {
    static constexpr int kWa = 0, kWb = 65536, kStage = 131072, kMisc = 196608;
    static constexpr int kTotal = kMisc + 4352 + 1024;      // (exchange and four vectors, 4 KB, then barriers)
};
constexpr int kChainThreads = kGT + 32;                     // sixteen warps with a row and 32 columns a thread, and the issuing warp
enum { kMapA, kMapAux, kMapRes, kMapExt, kMapMid, kMapC, kMapOut, kMapQ, kChainMaps };
struct ChainMaps {
    CUtensorMap m[kChainMaps];             // of the matrices that a launch has, boxes of 32 columns by box_rows
    int box_rows;
};

enum { kChainFwd = 0, kChainBwd = 1, kChainTan = 2, kChainRev = 3 };
template <int KIND, bool LINKED>
__global__ void __launch_bounds__(kChainThreads, 1)
gemm_tc_chain2_kernel(const __grid_constant__ ChainMaps maps, const float *__restrict__ Wa, const float *__restrict__ ba, const float *__restrict__ Wb,
                      const float *__restrict__ bb, int64_t E, int with_aux, int with_mid, int32_t *__restrict__ status, const float *__restrict__ ext,
                      const uint8_t *__restrict__ image_a, const uint8_t *__restrict__ image_b, const ChainLink link) {
    using namespace tc;
    using L = ChainSmem;
    constexpr bool BWD = KIND == kChainBwd || KIND == kChainRev;
    constexpr int W = 128, MODE = BWD ? 1 : 0;
    const bool residual = !BWD && with_aux;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *sWa_hi = smem + L::kWa, *sWa_lo = sWa_hi + 32768, *sWb_hi = smem + L::kWb, *sWb_lo = sWb_hi + 32768;
    float *s_red = reinterpret_cast<float *>(smem + L::kMisc);
    float *s_ba = s_red + 512, *s_bb = s_ba + 128, *s_bc = s_bb + 128;         // biases; s_bc: of the third layer, or its vector
    float *s_dot = s_bc + 128;
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_dot + 128);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 4);
    int *s_err = reinterpret_cast<int *>(s_tmem + 1);
    // a GEMM is complete; the first and the second weight have arrived; an operand is written (one arrival per warp)
    const uint32_t done = smem_u32(s_bar), have_a = done + 8, have_b = done + 16, ready = done + 24;
    const uint32_t arrived = done + 48 + 8 * (threadIdx.x >> 5);               // a warp's box (behind the two words of s_tmem and s_err)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & 127, qt = (tid >> 7) & 3, col0 = qt * 32;
    constexpr float kWS = 64.f;
    if (!image_a) {
        bool range = load_weight_tile<true>(sWa_hi, sWa_lo, Wa, W, W, W, kWS);
        range = load_weight_tile<true>(sWb_hi, sWb_lo, Wb, W, W, W, kWS) || range;
        if (range && blockIdx.x == 0) atomicOr(status, (int)kWeightRange);
    }
    if (tid < 128) {
        s_ba[tid] = ba ? ba[tid] : 0.f;
        s_bb[tid] = bb ? bb[tid] : 0.f;
        if (LINKED) {
            const float *of = BWD ? link.vec : link.bias;
            s_bc[tid] = of && tid < link.width ? of[tid] : 0.f;
            s_dot[tid] = !BWD && link.dot && tid < link.width ? link.dot_w[tid] : 0.f;
        }
    }
    if (tid == 0) {
        mbar_init(done, 1);
        mbar_init(have_a, 1);
        mbar_init(have_b, 1);
        mbar_init(ready, kGT / 32);
        for (int w = 0; w < kGT / 32; w++) mbar_init(done + 48 + 8 * w, 1);
        *s_err = 0;
        if (image_a) {
            fetch_image(smem_u32(sWa_hi), LINKED && BWD ? link.image : image_a, have_a);
            fetch_image(smem_u32(sWb_hi), image_b, have_b);
        }
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_u32(s_tmem), 256);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();                                    // set-up done (weights only); A and aux belong to the kernels before
    pdl_launch_dependents();
    const uint32_t tmem = *s_tmem;                 // accumulator at columns [0,128), operand at [128,256)
    const int64_t ntiles = (E + kRows - 1) / kRows;
    bool failed = false;
    auto await = [&](uint32_t bar, uint32_t parity) {
        if (!failed && !mbar_wait(bar, parity)) failed = true;
        tc_fence_after();
    };

    if (warp == kGT / 32) {
        // ---- the issuing warp: products in the order of the layers.  The first place holds two weights in turn (LINKED), each fetched
        // when the product with the other is done; `parity` of the fetch that has to be over
        const bool elected = elect_one();
        uint32_t n = 0;                            // products issued
        auto gemm = [&](uint8_t *w_hi, uint32_t wbar, uint32_t parity) {
            if (image_a) await(wbar, parity);
            await(ready, n & 1);
            if (elected) {
                issue_gemm_ts<true>(tmem, tmem + 128, smem_u32(w_hi), smem_u32(w_hi) + 32768, W / 16, MODE, W);
                mma_commit(done);
            }
            __syncwarp();
            n++;
        };
        auto refill = [&](const uint8_t *image) {
            await(done, (n - 1) & 1);
            if (elected) fetch_image(smem_u32(sWa_hi), image, have_a);
            __syncwarp();
        };
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const bool more = tile + gridDim.x < ntiles;
            gemm(sWa_hi, have_a, 0);
            if (LINKED && BWD) {
                refill(image_a);
                gemm(sWa_hi, have_a, 1);
                if (more) refill(link.image);
            }
            if (LINKED && !BWD) refill(link.image);
            gemm(sWb_hi, have_b, 0);
            if (LINKED && !BWD) {
                gemm(sWa_hi, have_a, 1);
                if (more) refill(image_a);
            }
        }
    } else {
        const uint32_t acc = tmem + ((uint32_t)((warp & 3) * 32) << 16), ta = acc + 128;
        uint8_t *const box = smem + L::kStage + warp * 4096;                    // [32 rows][128 bytes], 16-byte pieces in the 128-byte swizzle
        const int row0 = 32 * (warp & 3);
        auto piece = [&](int row, int w) { return reinterpret_cast<float4 *>(box + row * 128 + ((w ^ (row & 7)) << 4)); };
        auto own = [&](int w) { return piece(lane, w); };                       // four columns of this thread's row
        // the warp's part of a tile into its box (zeros past the end), once all lanes are past what they had to do there and what leaves has
        // been read.  The fence is what keeps the copy behind the lanes' reads of what the box held: a __syncwarp() alone says that they
        // have been issued, and a copy out of the second-level cache can overtake them (one evaluation of 3000 beads in 400 had rows of
        // the wrong matrix)
        uint32_t loads = 0;
        auto load_box = [&](const CUtensorMap *map, int64_t tile) {
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                bulk_wait_read<0>();
                mbar_expect_bytes(arrived, (uint32_t)maps.box_rows * 128u);
                tensor_load_box(map, col0, (int)(tile * kRows) + row0, smem_u32(box), arrived);
            }
            loads++;
        };
        auto wait_box = [&]() { await(arrived, (loads - 1) & 1); };
        // the box to its place; the next to write there waits for box_left()
        auto store_box = [&](const CUtensorMap *map, int64_t tile) {
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (tile * kRows + row0 < E) tensor_store_box(map, col0, (int)(tile * kRows) + row0, box);
                bulk_commit();
            }
        };
        auto box_left = [&]() {
            if (lane == 0) bulk_wait_read<0>();
            __syncwarp();
        };
        auto row_group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp & 3)) : "memory"); };
        // this thread's 32 values -> operand block (row-scaled fp16 pairs); returns the row's scale.  (What the accumulator and the operand
        // block held has been read and consumed: by this warp, and by the product that it has waited for.)
        auto to_operand = [&](const float (&x)[32]) {
            float rmax = 0.f;
#pragma unroll
            for (int c = 0; c < 32; c++) rmax = fmaxf(rmax, fabsf(x[c]));
            s_red[qt * 128 + r] = rmax;
            row_group_sync();
            const float sc = row_scale(fmaxf(fmaxf(s_red[r], s_red[128 + r]), fmaxf(s_red[256 + r], s_red[384 + r])));
            store_a_tmem<true>(ta, col0, x, sc);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready);
            return sc;
        };
        uint32_t phase = 0;
        auto await_product = [&]() {
            await(done, phase);
            phase ^= 1;
        };
        // four columns of this thread's row of a matrix shaped like A (zero past the end); both halves of a 32-byte sector are used
        auto own_row = [&](const float *src, int64_t tile, int w) {
            const int64_t gr = tile * kRows + r;
            return gr < E ? __ldg(reinterpret_cast<const float4 *>(src + gr * W + col0) + w) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        if (blockIdx.x < ntiles) load_box(&maps.m[kMapA], blockIdx.x);

        // The box holds, in turn: the input; BWD: what the third layer adds, its result on its way out, the tanh outputs, mid on its way out;
        // TAN: a, then q on its way out; FWD: mid on its way out, then the residual; the output on its way out, and the third layer's.
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            float x[32];
            wait_box();
#pragma unroll
            for (int w = 0; w < 8; w++) {
                const float4 v = *own(w);
                x[4 * w] = v.x; x[4 * w + 1] = v.y; x[4 * w + 2] = v.z; x[4 * w + 3] = v.w;
            }
            if (LINKED && BWD) {
                if (link.vec) {
#pragma unroll
                    for (int c = 0; c < 32; c++) x[c] = s_bc[col0 + c] * fmaf(-x[c], x[c], 1.f);
                }
                const float sc0 = to_operand(x);
                if (link.res) load_box(&maps.m[kMapRes], tile);      // (behind the last use of what the box held)
                await_product();
                if (link.res) wait_box();
                float v[32];
                tmem_ld32(acc + col0, v);
                const float inv = 1.f / (sc0 * kWS);
#pragma unroll
                for (int w = 0; w < 8; w++) {
                    float4 o = make_float4(v[4 * w] * inv, v[4 * w + 1] * inv, v[4 * w + 2] * inv, v[4 * w + 3] * inv);
                    if (link.res) {
                        const float4 t4 = *own(w);
                        o = make_float4(o.x + t4.x, o.y + t4.y, o.z + t4.z, o.w + t4.w);
                    }
                    *own(w) = o;
                    x[4 * w] = o.x; x[4 * w + 1] = o.y; x[4 * w + 2] = o.z; x[4 * w + 3] = o.w;
                }
            }
            const float sc1 = to_operand(x);
            if (LINKED && BWD) store_box(&maps.m[kMapOut], tile);
            if (BWD) load_box(&maps.m[kMapAux], tile);
            if (KIND == kChainTan) load_box(&maps.m[kMapExt], tile);
            float4 e4[8];                            // (on their way under the product)
            if (KIND == kChainTan || KIND == kChainRev) {
#pragma unroll
                for (int w = 0; w < 8; w++) e4[w] = own_row(ext, tile, w);
            }
            await_product();
            if (BWD || KIND == kChainTan) wait_box();
            {
                float v[32];
                tmem_ld32(acc + col0, v);
                const float inv = 1.f / (sc1 * kWS);
#pragma unroll
                for (int w = 0; w < 8; w++) {
                    float4 o = make_float4(fmaf(v[4 * w], inv, s_ba[col0 + 4 * w]), fmaf(v[4 * w + 1], inv, s_ba[col0 + 4 * w + 1]),
                                           fmaf(v[4 * w + 2], inv, s_ba[col0 + 4 * w + 2]), fmaf(v[4 * w + 3], inv, s_ba[col0 + 4 * w + 3]));
                    if (BWD) {
                        const float4 t4 = *own(w);
                        o = make_float4(o.x * fmaf(-t4.x, t4.x, 1.f), o.y * fmaf(-t4.y, t4.y, 1.f), o.z * fmaf(-t4.z, t4.z, 1.f), o.w * fmaf(-t4.w, t4.w, 1.f));
                        if (KIND == kChainRev) o = make_float4(o.x + e4[w].x, o.y + e4[w].y, o.z + e4[w].z, o.w + e4[w].w);
                        if (with_mid) *own(w) = o;
                    } else if (KIND == kChainTan) {
                        const float4 a4 = *own(w), g4 = e4[w];
                        *own(w) = make_float4(-2.f * a4.x * o.x * g4.x, -2.f * a4.y * o.y * g4.y, -2.f * a4.z * o.z * g4.z, -2.f * a4.w * o.w * g4.w);
                        o = make_float4(o.x * fmaf(-a4.x, a4.x, 1.f), o.y * fmaf(-a4.y, a4.y, 1.f), o.z * fmaf(-a4.z, a4.z, 1.f), o.w * fmaf(-a4.w, a4.w, 1.f));
                    } else {
                        o = make_float4(tanh_ex2(o.x), tanh_ex2(o.y), tanh_ex2(o.z), tanh_ex2(o.w));
                        *own(w) = o;
                    }
                    x[4 * w] = o.x; x[4 * w + 1] = o.y; x[4 * w + 2] = o.z; x[4 * w + 3] = o.w;
                }
            }
            const float sc2 = to_operand(x);         // under the second product: mid leaves, the residual arrives
            if (KIND == kChainTan) {
                store_box(&maps.m[kMapQ], tile);
                box_left();
#pragma unroll
                for (int w = 0; w < 8; w++) *own(w) = make_float4(x[4 * w], x[4 * w + 1], x[4 * w + 2], x[4 * w + 3]);
            }
            if (!BWD || with_mid) store_box(&maps.m[kMapMid], tile);
            if (residual) load_box(&maps.m[kMapAux], tile);
            await_product();
            if (residual) wait_box();
            else box_left();
            {
                float v[32];
                tmem_ld32(acc + col0, v);
                const float inv = 1.f / (sc2 * kWS);
#pragma unroll
                for (int w = 0; w < 8; w++) {
                    float4 o = make_float4(fmaf(v[4 * w], inv, s_bb[col0 + 4 * w]), fmaf(v[4 * w + 1], inv, s_bb[col0 + 4 * w + 1]),
                                           fmaf(v[4 * w + 2], inv, s_bb[col0 + 4 * w + 2]), fmaf(v[4 * w + 3], inv, s_bb[col0 + 4 * w + 3]));
                    if (residual) {
                        const float4 t4 = *own(w);
                        o = make_float4(o.x + t4.x, o.y + t4.y, o.z + t4.z, o.w + t4.w);
                    }
                    *own(w) = o;
                    if (LINKED && !BWD) { x[4 * w] = o.x; x[4 * w + 1] = o.y; x[4 * w + 2] = o.z; x[4 * w + 3] = o.w; }
                }
            }
            if (LINKED && !BWD) {
                const float sc3 = to_operand(x);
                store_box(&maps.m[kMapC], tile);
                await_product();
                float dot = 0.f;
                if (col0 < link.width) {
                    box_left();
                    float v[32];
                    tmem_ld32(acc + col0, v);
                    const float inv = 1.f / (sc3 * kWS);
#pragma unroll
                    for (int w = 0; w < 8; w++) {
                        float4 o = make_float4(fmaf(v[4 * w], inv, s_bc[col0 + 4 * w]), fmaf(v[4 * w + 1], inv, s_bc[col0 + 4 * w + 1]),
                                               fmaf(v[4 * w + 2], inv, s_bc[col0 + 4 * w + 2]), fmaf(v[4 * w + 3], inv, s_bc[col0 + 4 * w + 3]));
                        if (link.tanh) o = make_float4(tanh_ex2(o.x), tanh_ex2(o.y), tanh_ex2(o.z), tanh_ex2(o.w));
                        *own(w) = o;
                        const float4 u = *reinterpret_cast<const float4 *>(s_dot + col0 + 4 * w);
                        dot = fmaf(o.x, u.x, fmaf(o.y, u.y, fmaf(o.z, u.z, fmaf(o.w, u.w, dot))));
                    }
                    store_box(&maps.m[kMapOut], tile);
                }
                if (link.dot) {
                    s_red[qt * 128 + r] = dot;
                    row_group_sync();
                    if (qt == 0 && tile * kRows + r < E)
                        link.dot[tile * kRows + r] = (s_red[r] + s_red[128 + r]) + (s_red[256 + r] + s_red[384 + r]) + (link.dot_b ? link.dot_b[0] : 0.f);
                    row_group_sync();                // (before the next tile's rows exchange anything there)
                }
            } else {
                store_box(&maps.m[kMapC], tile);
            }
            const int64_t next = tile + gridDim.x;
            if (next < ntiles) load_box(&maps.m[kMapA], next);
        }
        bulk_wait_all();
    }
    if (failed) *s_err = 1;
    tc_fence_before();
    __syncthreads();
    if (*s_err && tid == 0) atomicOr(status, 8);
    if (warp == 0) tmem_free(tmem, 256);
}

// ------------------------------------------------------------------------------------------------ TN
__device__ __forceinline__ float block_max_512(float v, float *s_red) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 8));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
    __syncthreads();
    float m = s_red[0];
#pragma unroll
    for (int i = 1; i < 16; i++) m = fmaxf(m, s_red[i]);
    __syncthreads();
    return m;
}

__global__ void __launch_bounds__(kGT, 1)
gemm_tc_tn_kernel(const float *__restrict__ A, const float *__restrict__ B, int64_t E, int M, int N, float *__restrict__ partial,
                  int32_t *__restrict__ status) {
    using namespace tc;
    using L = GemmTcSmem;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *sB_hi = smem + L::kB, *sB_lo = sB_hi + 32768, *stageA = smem + L::kStageA, *stageB = smem + L::kStageB;
    float *s_red = reinterpret_cast<float *>(smem + L::kMisc);
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_red + 640);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 1);
    int *s_err = reinterpret_cast<int *>(s_tmem + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int r = tid & 127, qt = tid >> 7, col0 = qt * 32;   // r: output row m (TMEM lane); col0: edge sub-range / output column range
    const int npad = N <= 64 ? 64 : 128;
    const uint32_t bar = smem_u32(s_bar);
    if (tid == 0) {
        mbar_init(bar, 1);
        *s_err = 0;
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_u32(s_tmem), 256);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t phase = 0;
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; j++) acc[j] = 0.f;

    const int64_t ntiles = (E + kRows - 1) / kRows;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        load_tile_to_stage(stageA, A, tile * kRows, E, M);
        load_tile_to_stage(stageB, B, tile * kRows, E, N);
        __syncthreads();
        // A operand: lane = output row m, K = edge: x[j] = A[edge col0 + j][m]
        float x[32];
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 32; j++) {
            x[j] = *gstage_elem(stageA, col0 + j, r);
            amax = fmaxf(amax, fabsf(x[j]));
        }
        float bmax = 0.f;
        for (int idx = tid; idx < kRows * 32; idx += kGT) {
            const float4 v = *reinterpret_cast<const float4 *>(stageB + idx * 16);
            bmax = fmaxf(fmaxf(bmax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
        const float sa = row_scale(block_max_512(amax, s_red));
        const float sb = row_scale(block_max_512(bmax, s_red));
        store_a_tmem<true>(tmem + 128 + lane_off, col0, x, sa);
        // B operand tile [edge rows][n cols], read MN-major
        for (int idx = tid; idx < kRows * npad; idx += kGT) {
            const int er = idx / npad, n = idx - er * npad;
            const float w = *gstage_elem(stageB, er, n) * sb;
            const uint32_t off = elem_offset(er, n);
            const __half a = __float2half_rn(w);
            *reinterpret_cast<__half *>(sB_hi + off) = a;
            *reinterpret_cast<__half *>(sB_lo + off) = __float2half_rn(w - __half2float(a));
        }
        tmem_wait_st();
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after();
            issue_gemm_ts<true>(tmem, tmem + 128, smem_u32(sB_hi), smem_u32(sB_lo), kRows / 16, 1, npad);
            mma_commit(bar);
        }
        if (!mbar_wait(bar, phase)) *s_err = 1;
        phase ^= 1;
        tc_fence_after();
        if (col0 < npad) {
            float v[32];
            tmem_ld32(tmem + lane_off + col0, v);
            const float inv = 1.f / (sa * sb);
#pragma unroll
            for (int j = 0; j < 32; j++) acc[j] = fmaf(v[j], inv, acc[j]);
        }
        tc_fence_before();
        __syncthreads();
        if (*s_err) break;
    }
    // this CTA's partial [M][N]
    if (r < M)
#pragma unroll
        for (int j = 0; j < 32; j++)
            if (col0 + j < N) partial[((int64_t)blockIdx.x * M + r) * N + col0 + j] = acc[j];
    tc_fence_before();
    __syncthreads();
    if (*s_err && tid == 0) atomicOr(status, 8);
    if (warp == 0) tmem_free(tmem, 256);
}

// ------------------------------------------------------------------------------------------------ TN, pipelined
// C[M,N] = A[E,M]^T B[E,N], the contraction runs over the edges.  Per 128-edge tile:
//  * A operand (lane = output row m, K = edge): every thread reads its 32 values A[e][m] straight from global memory —
//    for one edge the 128 threads of a lane quarter read 128 consecutive floats;
//  * B operand (rows = edges, read MN-major): float4 per thread from global memory, converted to fp16 hi/lo and written
//    as 8-byte pieces of the swizzled operand tile;
//  * both are scaled by one power of two per tile (largest magnitude to [8,16)), so every tile has its own scale and
//    its product is read out of tensor memory and added to an fp32 accumulator tile in shared memory;
//  * two operand buffers (TMEM for A, shared memory for B) and two accumulators: the loads and conversion of tile i+1
//    run under the MMAs of tile i.
// Needs N % 4 == 0 and a 16-byte aligned B; the one-tile-at-a-time kernel below takes everything else.
struct GemmTnSmem {
    static constexpr int kB0 = 0, kB1 = 65536;        // operand tiles hi | lo, two buffers
    static constexpr int kAcc = 131072;               // fp32 accumulators [128][128], chunk-swizzled
    static constexpr int kMisc = 196608;
    static constexpr int kTotal = kMisc + 1024 + 1024;
};

// A launch takes a list of such products over the same number of rows (tn_jobs.cuh), `parts` CTAs each; a product may be the sum of
// two (A0^T B0 + A1^T B1), whose tiles then follow one another.
__global__ void __launch_bounds__(kGT, 1)
gemm_tc_tn_pipe_kernel(const __grid_constant__ TnJobs jobs, int32_t *__restrict__ status) {
    using namespace tc;
    using L = GemmTnSmem;
    const TnJob &job = jobs.job[blockIdx.x / jobs.parts];
    const int part = blockIdx.x % jobs.parts, M = job.M, N = job.N;
    const int64_t E = jobs.E;
    float *partial = job.partial, *colsum_partial = job.colsum_partial;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *s_acc = smem + L::kAcc;
    float2 *s_red = reinterpret_cast<float2 *>(smem + L::kMisc);          // [16] per-warp maxima of (A, B)
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(smem + L::kMisc + 256);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 2);
    int *s_err = reinterpret_cast<int *>(s_tmem + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & 127, qt = tid >> 7, col0 = qt * 32;   // r: output row m (TMEM lane); col0: edge sub-range / output columns
    const int npad = N <= 64 ? 64 : 128;
    const int qpr = npad >> 2;                                  // float4 pieces per row of the B tile
    const uint32_t bar0 = smem_u32(s_bar);
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        *s_err = 0;
    }
#pragma unroll
    for (int w = 0; w < 8; w++) *gstage(s_acc, r, (col0 >> 2) + w) = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_u32(s_tmem), 512);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;                 // accumulators [0,128) [128,256); A operands [256,384) [384,512)
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t phase_bits = 0;

    const int64_t seg_tiles = (E + kRows - 1) / kRows, ntiles = job.segments * seg_tiles;
    const int64_t step = jobs.parts;
    float xa[32];
    float4 xb[8];
    bool first_segment = true;                      // of the tile held in xa / xb
    float csum = 0.f;                               // this thread's share of sum_e A[e][r]
    auto load_tile = [&](int64_t tile) {
        first_segment = tile < seg_tiles;
        const float *__restrict__ A = job.A[first_segment ? 0 : 1], *__restrict__ B = job.B[first_segment ? 0 : 1];
        const int64_t e0 = (first_segment ? tile : tile - seg_tiles) * kRows;
#pragma unroll
        for (int j = 0; j < 32; j++) {
            const int64_t e = e0 + col0 + j;
            xa[j] = (e < E && r < M) ? __ldg(A + e * M + r) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int idx = tid + u * kGT;
            const int er = idx / qpr, n4 = (idx - er * qpr) << 2;
            const int64_t e = e0 + er;
            xb[u] = (er < kRows && e < E && n4 < N) ? __ldg(reinterpret_cast<const float4 *>(B + e * N + n4)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    // scales, operand stores and MMAs of the tile held in xa / xb into buffer `buf`; returns 1 / (sa sb)
    auto convert_issue = [&](int buf) {
        float amax = 0.f, bmax = 0.f;
#pragma unroll
        for (int j = 0; j < 32; j++) {
            amax = fmaxf(amax, fabsf(xa[j]));
            if (first_segment) csum += xa[j];
        }
#pragma unroll
        for (int u = 0; u < 8; u++) bmax = fmaxf(fmaxf(bmax, fmaxf(fabsf(xb[u].x), fabsf(xb[u].y))), fmaxf(fabsf(xb[u].z), fabsf(xb[u].w)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
        }
        if (lane == 0) s_red[warp] = make_float2(amax, bmax);
        __syncthreads();
        if (*s_err) return -1.f;      // written before this barrier, so every thread takes the same branch
#pragma unroll
        for (int w = 0; w < 16; w++) {
            const float2 m = s_red[w];
            amax = fmaxf(amax, m.x);
            bmax = fmaxf(bmax, m.y);
        }
        const float sa = row_scale(amax), sb = row_scale(bmax);
        const uint32_t ta = tmem + 256 + buf * 128;
        store_a_tmem<true>(ta + lane_off, col0, xa, sa);
        uint8_t *b_hi = smem + (buf ? L::kB1 : L::kB0), *b_lo = b_hi + 32768;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int idx = tid + u * kGT;
            const int er = idx / qpr, n4 = (idx - er * qpr) << 2;
            if (er < kRows) {
                const float4 w = make_float4(xb[u].x * sb, xb[u].y * sb, xb[u].z * sb, xb[u].w * sb);
                const uint32_t off = elem_offset(er, n4);
                const __half2 a0 = __floats2half2_rn(w.x, w.y), a1 = __floats2half2_rn(w.z, w.w);
                const float2 f0 = __half22float2(a0), f1 = __half22float2(a1);
                const __half2 c0 = __floats2half2_rn(w.x - f0.x, w.y - f0.y), c1 = __floats2half2_rn(w.z - f1.x, w.w - f1.y);
                *reinterpret_cast<uint2 *>(b_hi + off) = make_uint2(*reinterpret_cast<const uint32_t *>(&a0), *reinterpret_cast<const uint32_t *>(&a1));
                *reinterpret_cast<uint2 *>(b_lo + off) = make_uint2(*reinterpret_cast<const uint32_t *>(&c0), *reinterpret_cast<const uint32_t *>(&c1));
            }
        }
        tmem_wait_st();
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after();
            issue_gemm_ts<true>(tmem + buf * 128, ta, smem_u32(b_hi), smem_u32(b_lo), kRows / 16, 1, npad);
            mma_commit(bar0 + 8 * buf);
        }
        return 1.f / (sa * sb);
    };
    // product of the tile in accumulator `buf` -> shared-memory accumulator
    auto collect = [&](int buf, float inv) {
        if (!mbar_wait(bar0 + 8 * buf, (phase_bits >> buf) & 1u)) *s_err = 1;
        phase_bits ^= 1u << buf;
        tc_fence_after();
        if (col0 < npad) {
#pragma unroll
            for (int half = 0; half < 2; half++) {
                float v[16];
                tmem_ld16(tmem + buf * 128 + lane_off + col0 + half * 16, v);
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    float4 *slot = gstage(s_acc, r, (col0 >> 2) + half * 4 + w);
                    float4 a4 = *slot;
                    a4.x = fmaf(v[4 * w], inv, a4.x); a4.y = fmaf(v[4 * w + 1], inv, a4.y);
                    a4.z = fmaf(v[4 * w + 2], inv, a4.z); a4.w = fmaf(v[4 * w + 3], inv, a4.w);
                    *slot = a4;
                }
            }
        }
        tc_fence_before();
    };

    const int64_t t0 = part;
    float inv_prev = 0.f;
    int buf = 0;
    if (t0 < ntiles) load_tile(t0);
    for (int64_t tile = t0; tile < ntiles; tile += step, buf ^= 1) {
        const float inv_cur = convert_issue(buf);
        if (inv_cur < 0.f) break;                                   // a wait ran out (all threads leave together)
        if (tile + step < ntiles) load_tile(tile + step);           // in flight under the MMAs just issued
        if (tile != t0) collect(buf ^ 1, inv_prev);
        inv_prev = inv_cur;
    }
    __syncthreads();
    if (t0 < ntiles && !*s_err) collect(buf ^ 1, inv_prev);
    __syncthreads();
    if (r < M)
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const float4 a4 = *gstage(s_acc, r, (col0 >> 2) + w);
            const float o[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (col0 + 4 * w + j < N) partial[((int64_t)part * M + r) * N + col0 + 4 * w + j] = o[j];
        }
    if (colsum_partial) {                           // the four edge sub-ranges of each output row, in a fixed order
        float *s_cs = reinterpret_cast<float *>(s_acc);
        __syncthreads();
        s_cs[qt * 128 + r] = csum;
        __syncthreads();
        if (qt == 0 && r < M) colsum_partial[(int64_t)part * M + r] = (s_cs[r] + s_cs[128 + r]) + (s_cs[256 + r] + s_cs[384 + r]);
    }
    tc_fence_before();
    __syncthreads();
    if (*s_err && tid == 0) atomicOr(status, 8);
    if (warp == 0) tmem_free(tmem, 512);
}

// C = the partials added in their order (eight loads in flight at a time; the additions stay in sequence, so the result does
// not depend on how the loop is unrolled)
__global__ void gemm_tc_reduce_kernel(const float *__restrict__ partial, int64_t MN, int parts, float *__restrict__ C) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < MN; i += (int64_t)gridDim.x * blockDim.x) {
        float s = 0.f;
        int z = 0;
        for (; z + 8 <= parts; z += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = __ldg(partial + (int64_t)(z + u) * MN + i);
#pragma unroll
            for (int u = 0; u < 8; u++) s += v[u];
        }
        for (; z < parts; z++) s += __ldg(partial + (int64_t)z * MN + i);
        C[i] = s;
    }
}

// The same for two sets of partials in one launch (a weight gradient and its bias gradient): element i < MN of the first,
// element i - MN of the second
__global__ void gemm_tc_reduce2_kernel(const float *__restrict__ partial, int64_t MN, const float *__restrict__ partial2, int64_t M2, int parts,
                                       float *__restrict__ C, float *__restrict__ C2) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < MN + M2; i += (int64_t)gridDim.x * blockDim.x) {
        const bool second = i >= MN;
        const float *src = second ? partial2 + (i - MN) : partial + i;
        const int64_t stride = second ? M2 : MN;
        float s = 0.f;
        int z = 0;
        for (; z + 8 <= parts; z += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = __ldg(src + (int64_t)(z + u) * stride);
#pragma unroll
            for (int u = 0; u < 8; u++) s += v[u];
        }
        for (; z < parts; z++) s += __ldg(src + (int64_t)z * stride);
        if (second) C2[i - MN] = s;
        else C[i] = s;
    }
}

// CTAs of the TN kernels (each writes one [M,N] partial): one per SM for edge-sized contractions; for short ones two tiles
// per CTA (one, two and four measured within a per cent of one another on a node-sized contraction)
static int tn_parts(int64_t K) {
    const int64_t ntiles = (K + tc::kRows - 1) / tc::kRows;
    int64_t parts = (ntiles + 1) / 2;
    if (parts > kNumSM) parts = kNumSM;
    return (int)(parts < 1 ? 1 : parts);
}

static TnJobs one_job(const void *A, const void *B, int64_t E, int64_t M, int64_t N, float *partial, float *colsum_partial, int parts) {
    TnJobs jobs;
    jobs.E = E;
    jobs.parts = parts;
    jobs.job[0] = {{(const float *)A, nullptr}, {(const float *)B, nullptr}, partial, colsum_partial, (int)M, (int)N, 1};
    return jobs;
}

static int tn_pipe_configure() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        if (cudaFuncSetAttribute(gemm_tc_tn_pipe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmTnSmem::kTotal) != cudaSuccess) return check_launch();
        done[dev] = true;
    }
    return MLCGB_OK;
}

// `n` products in one launch, jobs.parts CTAs each; the partials are the caller's to add up (launch_partial_sums)
int tn_jobs_launch(const TnJobs &jobs, int n, int32_t *status, cudaStream_t st) {
    if (int rc = tn_pipe_configure()) return rc;
    gemm_tc_tn_pipe_kernel<<<n * jobs.parts, kGT, GemmTnSmem::kTotal, st>>>(jobs, status);
    return check_launch();
}

// dst[i] = sum over parts of src[part * stride + i]; entry blockIdx.y.  A block takes 128 elements, four a lane, a warp an eighth of the
// parts, and the eighths are added in their order: bound by the latency of a thread's chain of loads, which is 592 parts long for the
// embedding table (one thread per element: 49 us for the sums of a 256 x 73 step, one element per lane 29, now 20, the
// longest chains first).
constexpr int kSumWarps = 8;
__global__ void __launch_bounds__(kSumWarps * 32) partial_sums_kernel(const __grid_constant__ PartialSums sums) {
    __shared__ float4 s_part[kSumWarps][32];
    const PartialSum &s = sums.sum[blockIdx.y];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, z0 = s.parts * warp / kSumWarps, z1 = s.parts * (warp + 1) / kSumWarps;
    const bool whole = ((uintptr_t)s.dst & 15) == 0;
    auto add = [](float4 &v, const float4 &x) { v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w; };
    for (int64_t i0 = (int64_t)blockIdx.x * 128; i0 < s.n; i0 += (int64_t)gridDim.x * 128) {
        const int64_t i = i0 + lane * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < s.n) {
            int z = z0;
            for (; z + 8 <= z1; z += 8) {
                float4 x[8];
#pragma unroll
                for (int u = 0; u < 8; u++) x[u] = __ldg(reinterpret_cast<const float4 *>(s.src + (z + u) * s.stride + i));
#pragma unroll
                for (int u = 0; u < 8; u++) add(v, x[u]);
            }
            float4 x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = z + u < z1 ? __ldg(reinterpret_cast<const float4 *>(s.src + (z + u) * s.stride + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 8; u++) add(v, x[u]);
        }
        s_part[warp][lane] = v;
        __syncthreads();
        if (warp == 0 && i < s.n) {
#pragma unroll
            for (int w = 1; w < kSumWarps; w++) add(v, s_part[w][lane]);
            if (whole) *reinterpret_cast<float4 *>(s.dst + i) = v;
            else { s.dst[i] = v.x; s.dst[i + 1] = v.y; s.dst[i + 2] = v.z; s.dst[i + 3] = v.w; }
        }
        __syncthreads();
    }
}
int partial_sums_launch(const PartialSums &sums, int n, cudaStream_t st) {
    partial_sums_kernel<<<dim3(128, n), kSumWarps * 32, 0, st>>>(sums);
    return check_launch();
}

template <typename Kern>
static int set_smem(Kern kern, bool *done) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmTcSmem::kTotal) != cudaSuccess) return check_launch();
        done[dev] = true;
    }
    return MLCGB_OK;
}

// Pipelined row-wise kernel; MLCGB_E_LIMIT when its conditions on shape and alignment do not hold.
static int rows_pipe_launch(int mode, const void *A, const void *B, const void *bias, const void *aux, int epi, int64_t M, int64_t N, int64_t K,
                            void *C, const uint8_t *image, int32_t *status, cudaStream_t st) {
    CUtensorMap cmap;
    if ((K & 3) != 0 || ((uintptr_t)A & 15) != 0 || (aux && epi != kProTanhGradVec && ((uintptr_t)aux & 15) != 0) || !make_rows_map(&cmap, (float *)C, M, N))
        return MLCGB_E_LIMIT;
    const int64_t ntiles = (M + tc::kRows - 1) / tc::kRows;
    const int grid = (int)(ntiles < kNumSM ? ntiles : kNumSM);
    static bool p0[64] = {false}, p1[64] = {false};
    if (mode == 0) {
        if (int rc = set_smem(gemm_tc_rows_pipe_kernel<0>, p0)) return rc;
        launch_with_weights(gemm_tc_rows_pipe_kernel<0>, dim3(grid), dim3(kGT), GemmTcSmem::kTotal, st, (const float *)A, (const float *)B, (const float *)bias, M,
                   (int)N, (int)K, (const float *)aux, epi, cmap, image, status);
    } else {
        if (int rc = set_smem(gemm_tc_rows_pipe_kernel<1>, p1)) return rc;
        launch_with_weights(gemm_tc_rows_pipe_kernel<1>, dim3(grid), dim3(kGT), GemmTcSmem::kTotal, st, (const float *)A, (const float *)B, (const float *)bias, M,
                   (int)N, (int)K, (const float *)aux, epi, cmap, image, status);
    }
    return check_launch();
}

template <int KIND, bool LINKED>
static int chain2_launch_as(const void *A, const void *Wa, const void *ba, const void *Wb, const void *bb, const void *aux, int64_t M, void *mid_out,
                            void *C, const void *ext0, const void *ext1, void *q_out, const uint8_t *image_a, const uint8_t *image_b,
                            const ChainLink &link, int32_t *status, cudaStream_t st) {
    const int64_t ntiles = (M + tc::kRows - 1) / tc::kRows;
    const int grid = (int)(ntiles < kNumSM ? ntiles : kNumSM);
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        if (cudaFuncSetAttribute(gemm_tc_chain2_kernel<KIND, LINKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, ChainSmem::kTotal) != cudaSuccess)
            return check_launch();
        done[dev] = true;
    }
    ChainMaps maps = {};
    maps.box_rows = (int)(M < 32 ? M : 32);
    const auto map = [&](int k, const void *p, int64_t cols = 128) { return !p || make_rows_map(&maps.m[k], (float *)p, M, cols, 32); };
    if (M >= (int64_t)1 << 31 || !map(kMapA, A, LINKED && (KIND == kChainBwd || KIND == kChainRev) ? link.width : 128) || !map(kMapAux, aux) ||
        !map(kMapRes, link.res) || !map(kMapExt, KIND == kChainTan ? ext0 : nullptr) || !map(kMapMid, mid_out) || !map(kMapC, C) ||
        !map(kMapOut, link.out, LINKED && KIND != kChainBwd && KIND != kChainRev ? link.width : 128) || !map(kMapQ, q_out))
        return MLCGB_E_LIMIT;
    launch_with_weights(gemm_tc_chain2_kernel<KIND, LINKED>, dim3(grid), dim3(kChainThreads), ChainSmem::kTotal, st, maps, (const float *)Wa, (const float *)ba,
               (const float *)Wb, (const float *)bb, M, aux ? 1 : 0, mid_out ? 1 : 0, status, (const float *)(KIND == kChainTan ? ext1 : ext0), image_a, image_b, link);
    return check_launch();
}
template <int KIND>
static int chain2_launch(const void *A, const void *Wa, const void *ba, const void *Wb, const void *bb, const void *aux, int64_t M, void *mid_out,
                         void *C, const void *ext0, const void *ext1, void *q_out, const uint8_t *image_a, const uint8_t *image_b,
                         const ChainLink *link, int32_t *status, cudaStream_t st) {
    if (link) {
        if (!link->image || !image_a || !image_b || !link->out) return MLCGB_E_ARG;
        return chain2_launch_as<KIND, true>(A, Wa, ba, Wb, bb, aux, M, mid_out, C, ext0, ext1, q_out, image_a, image_b, *link, status, st);
    }
    return chain2_launch_as<KIND, false>(A, Wa, ba, Wb, bb, aux, M, mid_out, C, ext0, ext1, q_out, image_a, image_b, ChainLink{}, status, st);
}

int gemm_fused(int mode, const void *A, const void *B, const void *bias, const void *aux, int epilogue, int64_t M, int64_t N, int64_t K, void *C,
               const uint8_t *image, int32_t *status, void *stream) {
    TimelineScope timeline_scope("gemm_tc_fused", stream);
    if ((mode != 0 && mode != 1) || epilogue < 0 || epilogue > 4 || !status) return MLCGB_E_ARG;
    if ((epilogue == kEpiAdd || epilogue == kEpiTanhGrad || epilogue == kProTanhGradVec) && !aux) return MLCGB_E_ARG;
    if (!mlcgb_gemm_tc_supported(mode, M, N, K)) return MLCGB_E_LIMIT;
    if (M == 0) return MLCGB_OK;
    if (!A || !B || !C) return MLCGB_E_ARG;
    return rows_pipe_launch(mode, A, B, bias, aux, epilogue, M, N, K, C, image, status, (cudaStream_t)stream);
}

int gemm_chain2(int backward, const void *A, const void *Wa, const void *ba, const void *Wb, const void *bb, const void *aux, int64_t M, void *mid_out,
                void *C, const uint8_t *image_a, const uint8_t *image_b, const ChainLink *link, int32_t *status, void *stream) {
    TimelineScope timeline_scope("gemm_tc_chain2", stream);
    if (M < 0 || !status) return MLCGB_E_ARG;
    if (M == 0) return MLCGB_OK;
    if (!A || !Wa || !Wb || !aux || !C || (!backward && !mid_out)) return MLCGB_E_ARG;
    if ((((uintptr_t)A | (uintptr_t)aux | (uintptr_t)C | (uintptr_t)mid_out) & 15) != 0) return MLCGB_E_LIMIT;
    const auto st = (cudaStream_t)stream;
    return backward ? chain2_launch<kChainBwd>(A, Wa, ba, Wb, bb, aux, M, mid_out, C, nullptr, nullptr, nullptr, image_a, image_b, link, status, st)
                    : chain2_launch<kChainFwd>(A, Wa, ba, Wb, bb, aux, M, mid_out, C, nullptr, nullptr, nullptr, image_a, image_b, link, status, st);
}

int gemm_chain2_tangent(int reverse, const void *A, const void *Wa, const void *Wb, const void *a, const void *gu, const void *aux, int64_t M, void *q,
                        void *mid_out, void *C, const uint8_t *image_a, const uint8_t *image_b, const ChainLink *link, int32_t *status, void *stream) {
    TimelineScope timeline_scope("gemm_tc_chain2_tangent", stream);
    if (M < 0 || !status) return MLCGB_E_ARG;
    if (M == 0) return MLCGB_OK;
    if (!A || !Wa || !Wb || !a || !q || !mid_out || !C || (!reverse && !gu)) return MLCGB_E_ARG;
    if ((((uintptr_t)A | (uintptr_t)a | (uintptr_t)gu | (uintptr_t)aux | (uintptr_t)q | (uintptr_t)mid_out | (uintptr_t)C) & 15) != 0) return MLCGB_E_LIMIT;
    const auto st = (cudaStream_t)stream;
    if (reverse) return chain2_launch<kChainRev>(A, Wa, nullptr, Wb, nullptr, a, M, mid_out, C, q, nullptr, nullptr, image_a, image_b, link, status, st);
    return chain2_launch<kChainTan>(A, Wa, nullptr, Wb, nullptr, aux, M, mid_out, C, a, gu, q, image_a, image_b, link, status, st);
}

}  // namespace mlcgb

using namespace mlcgb;

extern "C" {

int mlcgb_gemm_tc_fused(int mode, const void *A, const void *B, const void *bias, const void *aux, int epilogue, int64_t M, int64_t N,
                        int64_t K, void *C, int32_t *status, void *stream) {
    return gemm_fused(mode, A, B, bias, aux, epilogue, M, N, K, C, nullptr, status, stream);
}

int mlcgb_gemm_tc_chain2(int backward, const void *A, const void *Wa, const void *ba, const void *Wb, const void *bb, const void *aux,
                         int64_t M, void *mid_out, void *C, int32_t *status, void *stream) {
    return gemm_chain2(backward, A, Wa, ba, Wb, bb, aux, M, mid_out, C, nullptr, nullptr, nullptr, status, stream);
}

int mlcgb_gemm_tc_chain2_tangent(int reverse, const void *A, const void *Wa, const void *Wb, const void *a, const void *gu, const void *aux,
                                 int64_t M, void *q, void *mid_out, void *C, int32_t *status, void *stream) {
    return gemm_chain2_tangent(reverse, A, Wa, Wb, a, gu, aux, M, q, mid_out, C, nullptr, nullptr, nullptr, status, stream);
}

int mlcgb_gemm_tc_tn_colsum(const void *A, const void *B, int64_t K, int64_t M, int64_t N, void *C, void *colsum, void *workspace,
                            size_t workspace_bytes, int32_t *status, void *stream) {
    TimelineScope timeline_scope("gemm_tc_tn_colsum", stream);
    if (!A || !B || !C || !colsum || !status) return MLCGB_E_ARG;
    if (!mlcgb_gemm_tc_supported(2, M, N, K) || (N & 3) != 0 || ((uintptr_t)B & 15) != 0) return MLCGB_E_LIMIT;
    const int parts = tn_parts(K);
    if (!workspace || workspace_bytes < (size_t)parts * M * (N + 1) * sizeof(float)) return MLCGB_E_WORKSPACE;
    auto st = (cudaStream_t)stream;
    if (int rc = tn_pipe_configure()) return rc;
    float *part = (float *)workspace, *cpart = part + (size_t)parts * M * N;
    gemm_tc_tn_pipe_kernel<<<parts, kGT, GemmTnSmem::kTotal, st>>>(one_job(A, B, K, M, N, part, cpart, parts), status);
    gemm_tc_reduce2_kernel<<<grid_for(M * N + M, 256), 256, 0, st>>>(part, M * N, cpart, M, parts, (float *)C, (float *)colsum);
    return check_launch();
}

int mlcgb_gemm_tc_supported(int mode, int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if (mode == 0 || mode == 1) return N <= 128 && K <= 128;   // M = edges
    if (mode == 2) return M <= 128 && N <= 128;                // K = edges
    return 0;
}

size_t mlcgb_gemm_tc_workspace_bytes(int mode, int64_t M, int64_t N, int64_t K) {
    if (mode != 2 || !mlcgb_gemm_tc_supported(mode, M, N, K)) return 0;
    return (size_t)tn_parts(K) * (size_t)M * (size_t)(N + 1) * sizeof(float);   // partial products, and partial column sums
}

int mlcgb_gemm_tc(int mode, const void *A, const void *B, const void *bias, int64_t M, int64_t N, int64_t K, void *C, void *workspace,
                  size_t workspace_bytes, int32_t *status, void *stream) {
    TimelineScope timeline_scope("gemm_tc", stream);
    if (!A || !B || !C || !status) return MLCGB_E_ARG;
    if (!mlcgb_gemm_tc_supported(mode, M, N, K)) return MLCGB_E_LIMIT;
    auto st = (cudaStream_t)stream;
    static bool c0[64] = {false}, c1[64] = {false}, c2[64] = {false};
    if (mode == 0 || mode == 1) {
        const int64_t ntiles = (M + tc::kRows - 1) / tc::kRows;
        const int grid = (int)(ntiles < kNumSM ? ntiles : kNumSM);
        const int rc = rows_pipe_launch(mode, A, B, bias, nullptr, kEpiNone, M, N, K, C, nullptr, status, st);
        if (rc != MLCGB_E_LIMIT) return rc;            // else: shapes or alignment the pipelined kernel does not take
        if (mode == 0) {
            if (int rc = set_smem(gemm_tc_rows_kernel<0>, c0)) return rc;
            gemm_tc_rows_kernel<0><<<grid, kGT, GemmTcSmem::kTotal, st>>>((const float *)A, (const float *)B, (const float *)bias, M, (int)N, (int)K, (float *)C, status);
        } else {
            if (int rc = set_smem(gemm_tc_rows_kernel<1>, c1)) return rc;
            gemm_tc_rows_kernel<1><<<grid, kGT, GemmTcSmem::kTotal, st>>>((const float *)A, (const float *)B, nullptr, M, (int)N, (int)K, (float *)C, status);
        }
        return check_launch();
    }
    const int parts = tn_parts(K);
    if (!workspace || workspace_bytes < (size_t)parts * M * N * sizeof(float)) return MLCGB_E_WORKSPACE;
    if ((N & 3) == 0 && ((uintptr_t)B & 15) == 0) {
        if (int rc = tn_pipe_configure()) return rc;
        gemm_tc_tn_pipe_kernel<<<parts, kGT, GemmTnSmem::kTotal, st>>>(one_job(A, B, K, M, N, (float *)workspace, nullptr, parts), status);
    } else {
        if (int rc = set_smem(gemm_tc_tn_kernel, c2)) return rc;
        gemm_tc_tn_kernel<<<parts, kGT, GemmTcSmem::kTotal, st>>>((const float *)A, (const float *)B, K, (int)M, (int)N, (float *)workspace, status);
    }
    gemm_tc_reduce_kernel<<<grid_for(M * N, 256), 256, 0, st>>>((const float *)workspace, M * N, parts, (float *)C);
    return check_launch();
}

}  // extern "C"

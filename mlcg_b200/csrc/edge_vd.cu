// Aggregations of a symmetric list whose filters are stored per pair as value rows W and distance-derivative rows W'
// (filter_vd.cu), float32, 128 features.  A warp takes a destination node and walks its edges in list order, lane t four features
// of every row; the two filter rows of an edge come through a ring of asynchronous copies (a lane copies and reads its own
// 16 bytes of a row: no synchronisation beyond the copy groups), node rows through registers.  Sums in edge order, no atomics.
//
//   force    out[i] = sum_j a[j] W[p]          s[e] (+)= sum_f (x[i] a[j] W'[p])_f          e = (i, j), p = its pair
//   tangent  out[i] = sum_j a[j] W[p] + b[j] (dd[e] W'[p])
//
// `force` is the step of the force pass that used to be an aggregation and a backward pass of the filter network: gd of a pair is
// s[(i,j)] + s[(j,i)], with x = lin1 features and a = gradient of the aggregate.  Bound by rows in flight
// and the first-level path: per edge 1.5 KB (force) or 2 KB (tangent) of rows, of which W and W' come from HBM once (force, 1.1 M edges: first
// level 70 % of its throughput, L2 48 %, memory 65 %, issue slots 54 %).
#include "schnet_internal.cuh"

#include <type_traits>

namespace mlcgb {

enum { kSegForce = 0, kSegTangent = 1, kSegTangentRows = 2 };     // the last: tangent with a = 0
constexpr int kVdWarps = 8;
// Rows in flight per warp and blocks per SM.  The rings take first-level cache from the node rows, which are read again and again
// while a structure is worked on: eight rows (or pairs of rows) and three blocks took 313 us for three `force` launches over 1.1 M
// edges; four and four blocks 286.  A tangent holds too much in registers for four blocks (324 against 297).
template <int MODE> constexpr int kVdSlots = MODE == kSegForce ? 4 : 8;
template <int MODE> constexpr int kVdBlocks = MODE == kSegForce ? 4 : 3;

__device__ __forceinline__ void fma4(float4 &acc, const float4 &a, const float4 &b) {
    acc.x = fmaf(a.x, b.x, acc.x); acc.y = fmaf(a.y, b.y, acc.y); acc.z = fmaf(a.z, b.z, acc.z); acc.w = fmaf(a.w, b.w, acc.w);
}

template <int MODE>
__global__ void __launch_bounds__(kVdWarps * 32, kVdBlocks<MODE>)
seg_vd_kernel(const float *__restrict__ a, const float *__restrict__ x, const float *__restrict__ W, const float *__restrict__ Wd,
              const int64_t *__restrict__ ptr, const int32_t *__restrict__ nbr, const int32_t *__restrict__ pair_of, int64_t N,
              float *__restrict__ out, float *__restrict__ s, int accumulate) {
    extern __shared__ float4 vd_ring[];                            // [warps][slots][W | W'][32], then [warps][32] dot products
    constexpr int kSlots = kVdSlots<MODE>;
    constexpr bool kTan = MODE == kSegTangent || MODE == kSegTangentRows, kValue = MODE == kSegForce || MODE == kSegTangent;
    constexpr int kRows = kValue ? 2 : 1;                          // rows copied per edge
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4 *ring = vd_ring + wib * kSlots * kRows * 32 + lane;
    float *s_dot = reinterpret_cast<float *>(vd_ring + kVdWarps * kSlots * kRows * 32) + wib * 32;
    const uint32_t ring_addr = (uint32_t)__cvta_generic_to_shared(ring);
    const float4 *a4 = reinterpret_cast<const float4 *>(a) + lane, *x4 = reinterpret_cast<const float4 *>(x) + lane;
    const float4 *W4 = reinterpret_cast<const float4 *>(W) + lane, *Wd4 = reinterpret_cast<const float4 *>(Wd) + lane;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    pdl_wait();
    for (int64_t n = warp; n < N; n += nwarps) {
        const int64_t k0 = ptr[n], k1 = ptr[n + 1];
        float4 acc0 = make_float4(0.f, 0.f, 0.f, 0.f), acc1 = acc0;
        float4 xi = acc0;
        if (!kTan && k1 > k0) xi = __ldg(x4 + n * 32);
        for (int64_t c0 = k0; c0 < k1; c0 += 32) {                // the node's edges, 32 at a time: lane t holds edge c0 + t
            const int len = (int)(k1 - c0 < 32 ? k1 - c0 : 32);
            int32_t my_j = 0, my_p = 0;
            float my_s = 0.f;                                      // tangent: dd[e]
            if (lane < len) {
                my_j = nbr[c0 + lane];
                my_p = pair_of[c0 + lane];
                if (kTan) my_s = s[c0 + lane];
            }
            const int ngroups = (len + 1) >> 1;
            // group g = edges 2g, 2g+1 of the chunk -> slots (2g + u) % kSlots
            auto issue = [&](int g) {
                if (g < ngroups) {
                    const uint32_t to = ring_addr + (uint32_t)((2 * g % kSlots) * kRows * 512);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int t = 2 * g + u;
                        const int64_t p = __shfl_sync(0xffffffffu, my_p, t & 31);
                        if (t < len) {
                            const uint32_t dst = to + (uint32_t)(u * kRows * 512);
                            if (kValue) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(W4 + p * 32) : "memory");
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (kRows - 1) * 512), "l"(Wd4 + p * 32) : "memory");
                        }
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");   // (an empty group keeps the count of pending groups fixed)
            };
#pragma unroll
            for (int g = 0; g < kSlots / 2; g++) issue(g);
            // two groups (four edges) per step; of the last step perhaps some.  (Tangents: steps of whole groups without bounds, a step of
            // 256 x 73 beads 1380 -> 1350 us; the force pass has no registers for both kinds of step: 124 -> 129 us a launch.)
            auto step = [&](int g, auto whole) {
                constexpr bool ALL = decltype(whole)::value;
                float4 xa[4], xb[4];
                float dd[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int t = 2 * g + u;
                    const int64_t j = __shfl_sync(0xffffffffu, my_j, t & 31);
                    if (kTan) dd[u] = __shfl_sync(0xffffffffu, my_s, t & 31);
                    if (MODE != kSegTangentRows) xa[u] = ALL || t < len ? __ldg(a4 + j * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
                    if (kTan) xb[u] = ALL || t < len ? __ldg(x4 + j * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(kSlots / 2 - 1) : "memory");
                    const float4 *slots = ring + (2 * (g + h) % kSlots) * kRows * 32;
#pragma unroll
                    for (int v = 0; v < 2; v++) {
                        const int u = 2 * h + v, t = 2 * g + u;
                        if (ALL || t < len) {
                            const float4 *slot = slots + v * kRows * 32;
                            const float4 wd = slot[(kRows - 1) * 32];
                            if (kValue) {
                                const float4 w = slot[0];
                                if (v) fma4(acc1, xa[u], w);
                                else fma4(acc0, xa[u], w);
                            }
                            if (kTan) {
                                const float4 tb = make_float4(dd[u] * xb[u].x, dd[u] * xb[u].y, dd[u] * xb[u].z, dd[u] * xb[u].w);
                                if (v) fma4(acc1, tb, wd);
                                else fma4(acc0, tb, wd);
                            } else {
                                dot[u] = fmaf(xi.x * xa[u].x, wd.x, fmaf(xi.y * xa[u].y, wd.y, fmaf(xi.z * xa[u].z, wd.z, xi.w * xa[u].w * wd.w)));
                            }
                        }
                    }
                    issue(g + h + kSlots / 2);
                }
                if (!kTan) {
                    // the four edges' sums over the warp at once: after two exchanges a lane is left with one of them, edge
                    // 2 (lane >> 4 & 1) + (lane >> 3 & 1), and a sum over eight lanes
                    const bool up = lane & 16, up2 = lane & 8;
                    float d0 = (up ? dot[2] : dot[0]) + __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[2], 16);
                    float d1 = (up ? dot[3] : dot[1]) + __shfl_xor_sync(0xffffffffu, up ? dot[1] : dot[3], 16);
                    float d = (up2 ? d1 : d0) + __shfl_xor_sync(0xffffffffu, up2 ? d0 : d1, 8);
                    d += __shfl_xor_sync(0xffffffffu, d, 4);
                    d += __shfl_xor_sync(0xffffffffu, d, 2);
                    d += __shfl_xor_sync(0xffffffffu, d, 1);
                    if ((lane & 7) == 0) s_dot[(2 * g + (lane >> 4) * 2 + ((lane >> 3) & 1)) & 31] = d;
                }
            };
            int g = 0;
            if constexpr (kTan)
                for (; 2 * g + 4 <= len; g += 2) step(g, std::true_type{});
            for (; 2 * g < len; g += 2) step(g, std::false_type{});
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (!kTan) {
                __syncwarp();
                if (lane < len) {
                    const float v = s_dot[lane];
                    s[c0 + lane] = accumulate ? s[c0 + lane] + v : v;
                }
                __syncwarp();
            }
        }
        reinterpret_cast<float4 *>(out)[n * 32 + lane] = make_float4(acc0.x + acc1.x, acc0.y + acc1.y, acc0.z + acc1.z, acc0.w + acc1.w);
    }
}

// One dot product per pair (seg_pair_dot): a warp takes the upper edges of its node, whose pairs and rows of W' are consecutive, four
// at a time in registers.  Per pair one row of W' and two node rows cross the first-level pipe where the two directed edges of the
// kernel above took four, and the sums of the other blocks are added here, once per pair, instead of per edge with the forces.  Dot
// products of 545 k pairs inside an evaluation 114 us by edges, 94 like this; 128 k pairs 39 and 29; 94 k pairs 39 and 27.
constexpr int kPairWarps = 4;
__global__ void __launch_bounds__(kPairWarps * 32, 6)
seg_pair_dot_kernel(const float *__restrict__ a, const float *__restrict__ x, const float *__restrict__ Wd, const int64_t *__restrict__ ptr,
                    const int32_t *__restrict__ nbr, const int32_t *__restrict__ pair_of, const int32_t *__restrict__ twin, const float *__restrict__ s,
                    int64_t N, float *__restrict__ sp) {
    const int lane = threadIdx.x & 31;
    const char *a_lane = reinterpret_cast<const char *>(a) + lane * 16, *x_lane = reinterpret_cast<const char *>(x) + lane * 16,
               *w_lane = reinterpret_cast<const char *>(Wd) + lane * 16;
    auto row = [](const char *base, int64_t r) { return __ldg(reinterpret_cast<const float4 *>(base + r * 512)); };
    const int64_t n = (int64_t)blockIdx.x * kPairWarps + (threadIdx.x >> 5);
    if (n >= N) return;
    const int64_t k0 = ptr[n], k1 = ptr[n + 1];
    if (k0 == k1) return;
    const float4 xi = row(x_lane, n), ai = row(a_lane, n);
    for (int64_t c0 = k0; c0 < k1; c0 += 32) {
        const bool in = c0 + lane < k1;
        const int32_t my_j = in ? nbr[c0 + lane] : 0;
        const unsigned upper = __ballot_sync(0xffffffffu, in && my_j > n);
        if (!upper) continue;
        const int first = __ffs(upper) - 1, len = first + __popc(upper);       // (neighbours ascend)
        const bool mine = lane >= first && lane < len;
        int32_t my_p = 0;
        float my_s = 0.f;
        if (mine) {
            my_p = pair_of[c0 + lane];
            if (s) my_s = s[c0 + lane] + s[twin[c0 + lane]];
        }
        for (int g = first; g < len; g += 4) {
            float4 w[4], aj[4], xj[4];
            float dot[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int t = g + u < len ? g + u : len - 1;
                const int64_t j = __shfl_sync(0xffffffffu, my_j, t);
                w[u] = row(w_lane, __shfl_sync(0xffffffffu, my_p, t));
                aj[u] = row(a_lane, j);
                xj[u] = row(x_lane, j);
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                dot[u] = fmaf(fmaf(xi.x, aj[u].x, xj[u].x * ai.x), w[u].x, fmaf(fmaf(xi.y, aj[u].y, xj[u].y * ai.y), w[u].y,
                         fmaf(fmaf(xi.z, aj[u].z, xj[u].z * ai.z), w[u].z, fmaf(xi.w, aj[u].w, xj[u].w * ai.w) * w[u].w)));
            // (the four sums as in the kernel above: sum u is left in lanes 8 u .. 8 u + 7)
            const bool up = lane & 16, up2 = lane & 8;
            const float d0 = (up ? dot[2] : dot[0]) + __shfl_xor_sync(0xffffffffu, up ? dot[0] : dot[2], 16);
            const float d1 = (up ? dot[3] : dot[1]) + __shfl_xor_sync(0xffffffffu, up ? dot[1] : dot[3], 16);
            float d = (up2 ? d1 : d0) + __shfl_xor_sync(0xffffffffu, up2 ? d0 : d1, 8);
            d += __shfl_xor_sync(0xffffffffu, d, 4);
            d += __shfl_xor_sync(0xffffffffu, d, 2);
            d += __shfl_xor_sync(0xffffffffu, d, 1);
            const float got = __shfl_sync(0xffffffffu, d, ((lane - g) & 3) * 8);
            if (lane >= g && lane < g + 4) my_s += got;
        }
        if (mine) sp[my_p] = my_s;
    }
}

int seg_pair_dot(const float *a, const float *x, const float *Wd, const int64_t *ptr, const int32_t *nbr, const int32_t *pair_of, const int32_t *twin,
                 const float *s, int64_t N, float *sp, cudaStream_t st) {
    TimelineScope timeline_scope("seg_pair_dot", st);
    if (int rc = prefer_l1<seg_pair_dot_kernel>()) return rc;
    seg_pair_dot_kernel<<<(unsigned)((N + kPairWarps - 1) / kPairWarps), kPairWarps * 32, 0, st>>>(a, x, Wd, ptr, nbr, pair_of, twin, s, N, sp);
    return check_launch();
}

// dd[e] = d(distance of e)/dt when the positions move along sign v: (pos[j] - pos[i]) . (v[j] - v[i]) / d, zero where the beads coincide
__global__ void edge_tangent_kernel(const float *__restrict__ pos, const float *__restrict__ v, const float *__restrict__ d,
                                    const int32_t *__restrict__ row0, const int32_t *__restrict__ row1, int64_t E, float sign, float *__restrict__ dd) {
    pdl_wait();
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = row0[e], j = row1[e];
        const float s = (pos[3 * j] - pos[3 * i]) * (v[3 * j] - v[3 * i]) + (pos[3 * j + 1] - pos[3 * i + 1]) * (v[3 * j + 1] - v[3 * i + 1]) +
                        (pos[3 * j + 2] - pos[3 * i + 2]) * (v[3 * j + 2] - v[3 * i + 2]);
        dd[e] = d[e] > 0.f ? sign * s / d[e] : 0.f;
    }
}

template <int MODE>
static int seg_vd_launch(const void *a, const void *x, const void *W, const void *Wd, const int64_t *ptr, const int32_t *nbr, const int32_t *pair_of,
                         int64_t N, void *out, void *s, int accumulate, cudaStream_t st) {
    constexpr int kRows = MODE == kSegForce || MODE == kSegTangent ? 2 : 1;
    constexpr size_t smem = (size_t)kVdWarps * kVdSlots<MODE> * kRows * 512 + kVdWarps * 128;
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        if (cudaFuncSetAttribute(seg_vd_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return check_launch();
        done[dev] = true;
    }
    launch_pdl(seg_vd_kernel<MODE>, dim3(grid_for(N, kVdWarps, 24)), dim3(kVdWarps * 32), smem, st, (const float *)a, (const float *)x, (const float *)W,
               (const float *)Wd, ptr, nbr, pair_of, N, (float *)out, (float *)s, accumulate);
    return check_launch();
}

}  // namespace mlcgb

using namespace mlcgb;

extern "C" {

int mlcgb_seg_force(const void *a, const void *x, const void *W, const void *Wd, const int64_t *ptr, const int32_t *nbr, const int32_t *pair_of,
                    int64_t N, int64_t F, void *out, void *s, int accumulate, void *stream) {
    TimelineScope timeline_scope("seg_force", stream);
    if (N < 0) return MLCGB_E_ARG;
    if (F != 128) return MLCGB_E_LIMIT;
    if (N == 0) return MLCGB_OK;
    if (!a || !x || !ptr || !out) return MLCGB_E_ARG;
    return seg_vd_launch<kSegForce>(a, x, W, Wd, ptr, nbr, pair_of, N, out, s, accumulate, (cudaStream_t)stream);
}

int mlcgb_seg_tangent(const void *a, const void *b, const void *W, const void *Wd, const void *dd, const int64_t *ptr, const int32_t *nbr,
                      const int32_t *pair_of, int64_t N, int64_t F, void *out, void *stream) {
    TimelineScope timeline_scope("seg_tangent", stream);
    if (N < 0) return MLCGB_E_ARG;
    if (F != 128) return MLCGB_E_LIMIT;
    if (N == 0) return MLCGB_OK;
    if (!b || !ptr || !out) return MLCGB_E_ARG;
    if (!a) return seg_vd_launch<kSegTangentRows>(a, b, W, Wd, ptr, nbr, pair_of, N, out, const_cast<void *>(dd), 0, (cudaStream_t)stream);
    return seg_vd_launch<kSegTangent>(a, b, W, Wd, ptr, nbr, pair_of, N, out, const_cast<void *>(dd), 0, (cudaStream_t)stream);
}

int mlcgb_edge_tangent(const void *pos, const void *v, const void *d, const int32_t *row0, const int32_t *row1, int64_t E, int negate, void *dd,
                       void *stream) {
    TimelineScope timeline_scope("edge_tangent", stream);
    if (E < 0) return MLCGB_E_ARG;
    if (E == 0) return MLCGB_OK;
    if (!pos || !v || !d || !row0 || !row1 || !dd) return MLCGB_E_ARG;
    launch_pdl(edge_tangent_kernel, dim3(grid_for(E, 256)), dim3(256), 0, (cudaStream_t)stream, (const float *)pos, (const float *)v, (const float *)d,
               row0, row1, E, negate ? -1.f : 1.f, (float *)dd);
    return check_launch();
}

}  // extern "C"

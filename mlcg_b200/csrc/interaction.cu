// One interaction block per call: the kernel sequences of the eval-mode forward and force pass of
//   x_new = x + lin( tanh( lin2( sum_j lin1(x)_j * W(d_ij) ) ) )            src/mlcg/nn/schnet.py:150, 252-262, 340-350
// issued from C, so that a host in any language pays one foreign call per block and direction instead of one per kernel
// (for small systems the evaluation time is the host's launch path, not the GPU).  Symmetric edge lists only (one filter
// row per unordered pair); everything else goes through the individual entry points.
#include "common.cuh"
#include "schnet_internal.cuh"
#include "tc_common.cuh"

using namespace mlcgb;

extern "C" {

static int interaction_forward_counted(const void *x, const void *d, const int64_t *ptr_out, const int32_t *nbr_out, const int32_t *sel,
                                      const int32_t *pair_of, const int64_t *pairs_dev, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind,
                                      double conv_lower, double conv_upper, const void *W1, const void *fA1, const void *fb1,
                                      const void *fA2, const void *W2, const void *b2, const void *W3, const void *b3, int64_t N, int64_t E,
                                      int64_t P, int64_t H, int64_t F, int64_t H2, int precision, void *xl, void *Wp, void *hsave, void *agg, void *a,
                                      void *out, int32_t *status, void *stream);
static int interaction_backward_counted(const void *g, const void *a, const void *Wp, const void *xl, const void *hsave, const void *d, const int64_t *ptr_out,
                                       const int32_t *nbr_out, const int32_t *sel, const int32_t *pair_of, const int32_t *twin,
                                       const int64_t *pairs_dev, const int32_t *row0, const int32_t *row1, const mlcgb_rbf_spec *rbf,
                                       int conv_cutoff_kind, double conv_lower, double conv_upper, const void *W1, const void *fA1,
                                       const void *fb1, const void *fA2, const void *W2, const void *W3, int64_t N, int64_t E, int64_t P,
                                       int64_t H, int64_t F, int64_t H2, int precision, void *gy, void *gagg, void *gxl, void *gx,
                                       void *gd, int gd_accumulate, int32_t *status, void *stream);

int mlcgb_interaction_forward(const void *x, const void *d, const int64_t *ptr_out, const int32_t *nbr_out, const int32_t *sel,
                              const int32_t *pair_of, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower,
                              double conv_upper, const void *W1, const void *fA1, const void *fb1, const void *fA2, const void *W2,
                              const void *b2, const void *W3, const void *b3, int64_t N, int64_t E, int64_t P, int64_t H, int64_t F,
                              int64_t H2, int precision, void *xl, void *Wp, void *hsave, void *agg, void *a, void *out,
                              int32_t *status, void *stream) {
    return interaction_forward_counted(x, d, ptr_out, nbr_out, sel, pair_of, nullptr, rbf, conv_cutoff_kind, conv_lower, conv_upper, W1,
                                             fA1, fb1, fA2, W2, b2, W3, b3, N, E, P, H, F, H2, precision, xl, Wp, hsave, agg, a, out, status,
                                             stream);
}

// pairs_dev: NULL, or the number of pairs in device memory; P then only sizes the buffers (see mlcgb_filter_forward_counted)
static int interaction_forward_counted(const void *x, const void *d, const int64_t *ptr_out, const int32_t *nbr_out, const int32_t *sel,
                                      const int32_t *pair_of, const int64_t *pairs_dev, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind,
                                      double conv_lower, double conv_upper, const void *W1, const void *fA1, const void *fb1,
                                      const void *fA2, const void *W2, const void *b2, const void *W3, const void *b3, int64_t N, int64_t E,
                                      int64_t P, int64_t H, int64_t F, int64_t H2, int precision, void *xl, void *Wp, void *hsave, void *agg, void *a,
                                      void *out, int32_t *status, void *stream) {
    if (N < 0 || E < 0 || P < 0 || !status) return MLCGB_E_ARG;
    if (N == 0) return MLCGB_OK;
    if (!x || !ptr_out || !W1 || !W2 || !b2 || !W3 || !b3 || !xl || !agg || !a || !out) return MLCGB_E_ARG;
    if (P > 0 && (!d || !nbr_out || !sel || !pair_of || !Wp)) return MLCGB_E_ARG;
    if ((H & 3) || (F & 3) || (H2 & 3) || H > 128 || F != 128 || H2 > 128) return MLCGB_E_LIMIT;
    int rc = mlcgb_gemm_tc_fused(0, x, W1, nullptr, nullptr, 0, N, F, H, xl, status, stream);                 // lin1 (no bias)
    if (rc) return rc;
    ChainScope chain;
    rc = mlcgb_filter_forward_counted(d, P, pairs_dev, sel, nullptr, rbf, conv_cutoff_kind, conv_lower, conv_upper, fA1, fb1, fA2, F, precision,
                                      Wp, hsave, status, stream);
    if (rc) return rc;
    rc = mlcgb_seg_mul_sum(xl, Wp, MLCGB_F32, ptr_out, nbr_out, pair_of, N, P, F, agg, stream);                // aggregation
    if (rc) return rc;
    if (H == 128 && F == 128 && H2 == 128) {                                                                   // lin2 + tanh -> lin + residual, one kernel
        rc = mlcgb_gemm_tc_chain2(0, agg, W2, b2, W3, b3, x, N, a, out, status, stream);
        if (rc != MLCGB_E_LIMIT) return rc;
    }
    rc = mlcgb_gemm_tc_fused(0, agg, W2, b2, nullptr, 1, N, H2, F, a, status, stream);                         // lin2 + tanh
    if (rc) return rc;
    return mlcgb_gemm_tc_fused(0, a, W3, b3, x, 2, N, H, H2, out, status, stream);                             // lin + residual
}

int mlcgb_interaction_backward(const void *g, const void *a, const void *Wp, const void *xl, const void *hsave, const void *d, const int64_t *ptr_out,
                               const int32_t *nbr_out, const int32_t *sel, const int32_t *pair_of, const int32_t *twin,
                               const int32_t *row0, const int32_t *row1, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind,
                               double conv_lower, double conv_upper, const void *W1, const void *fA1, const void *fb1,
                               const void *fA2, const void *W2, const void *W3, int64_t N, int64_t E, int64_t P, int64_t H, int64_t F,
                               int64_t H2, int precision, void *gy, void *gagg, void *gxl, void *gx /* or NULL */,
                               void *gd /* [E] or NULL */, int32_t *status, void *stream) {
    return interaction_backward_counted(g, a, Wp, xl, hsave, d, ptr_out, nbr_out, sel, pair_of, twin, nullptr, row0, row1, rbf, conv_cutoff_kind,
                                              conv_lower, conv_upper, W1, fA1, fb1, fA2, W2, W3, N, E, P, H, F, H2, precision, gy, gagg, gxl,
                                              gx, gd, 0, status, stream);
}

static int interaction_backward_counted(const void *g, const void *a, const void *Wp, const void *xl, const void *hsave, const void *d, const int64_t *ptr_out,
                                       const int32_t *nbr_out, const int32_t *sel, const int32_t *pair_of, const int32_t *twin,
                                       const int64_t *pairs_dev, const int32_t *row0, const int32_t *row1, const mlcgb_rbf_spec *rbf,
                                       int conv_cutoff_kind, double conv_lower, double conv_upper, const void *W1, const void *fA1,
                                       const void *fb1, const void *fA2, const void *W2, const void *W3, int64_t N, int64_t E, int64_t P,
                                       int64_t H, int64_t F, int64_t H2, int precision, void *gy, void *gagg, void *gxl,
                                       void *gx /* or NULL */, void *gd /* [E] or NULL */, int gd_accumulate, int32_t *status,
                                       void *stream) {
    if (N < 0 || E < 0 || P < 0 || !status) return MLCGB_E_ARG;
    if (N == 0) return MLCGB_OK;
    if (!g || !a || !xl || !ptr_out || !W1 || !W2 || !W3 || !gy || !gagg || !gxl) return MLCGB_E_ARG;
    if (P > 0 && (!d || !nbr_out || !sel || !pair_of || !twin || !row0 || !row1 || !Wp)) return MLCGB_E_ARG;
    if ((H & 3) || (F & 3) || (H2 & 3) || H > 128 || F != 128 || H2 > 128) return MLCGB_E_LIMIT;
    int rc = MLCGB_E_LIMIT;
    if (H == 128 && F == 128 && H2 == 128)                                                                     // through lin, tanh and lin2, one kernel
        rc = mlcgb_gemm_tc_chain2(1, g, W3, nullptr, W2, nullptr, a, N, nullptr, gagg, status, stream);
    if (rc == MLCGB_E_LIMIT) {
        rc = mlcgb_gemm_tc_fused(1, g, W3, nullptr, a, 3, N, H2, H, gy, status, stream);                      // through lin and tanh
        if (rc) return rc;
        rc = mlcgb_gemm_tc_fused(1, gy, W2, nullptr, nullptr, 0, N, F, H2, gagg, status, stream);              // through lin2
    }
    if (rc) return rc;
    ChainScope chain;
    if (gx) {
        rc = mlcgb_seg_mul_sum(gagg, Wp, MLCGB_F32, ptr_out, nbr_out, pair_of, N, P, F, gxl, stream);          // to the gathered features
        if (rc) return rc;
        rc = mlcgb_gemm_tc_fused(1, gxl, W1, nullptr, g, 2, N, H, F, gx, status, stream);                     // through lin1, + residual branch
        if (rc) return rc;
    }
    if (gd && E > 0)
        rc = mlcgb_filter_backward_counted(d, P, pairs_dev, sel, twin, rbf, conv_cutoff_kind, conv_lower, conv_upper, fA1, fb1, fA2, F, precision,
                                           row0, row1, xl, gagg, N, hsave, gd, gd_accumulate, status, stream);
    return rc;
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// The whole SchNet evaluation — embedding, interaction blocks, output network, per-structure sum and the force pass — as
// one kernel sequence issued from C (src/mlcg/nn/schnet.py:116-162 and its derivative, src/mlcg/nn/gradients.py:191-230).
// ------------------------------------------------------------------------------------------------
namespace mlcgb {

// Rows of the embedding table, and in front of them eight blocks per weight image, 16 of its rows each
__global__ void __launch_bounds__(256)
embedding_rows_kernel(const float *__restrict__ table, const int64_t *__restrict__ types, int64_t N, int64_t H, int64_t T, float *__restrict__ x,
                      const __grid_constant__ WeightImages im, int32_t *__restrict__ status) {
    pdl_wait();
    if ((int)blockIdx.x < 8 * im.n) {
        const int k = blockIdx.x >> 3, cols = im.cols[k], pad = cols <= 64 ? 64 : 128;
        uint8_t *hi = im.dst + k * kWeightImage;
        float most = 0.f;
        const bool first_layer = k >= im.first_filter && ((k - im.first_filter) & 1) == 0;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int row = (blockIdx.x & 7) * 16 + u * 8 + (threadIdx.x >> 5), col = (threadIdx.x & 31) * 4;
            const float *src = im.src[k] + row * cols + col;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < im.rows[k] && col < pad) {
                if (col + 4 <= cols && ((uintptr_t)src & 15) == 0) v = *reinterpret_cast<const float4 *>(src);
                else
                    v = make_float4(col < cols ? src[0] : 0.f, col + 1 < cols ? src[1] : 0.f, col + 2 < cols ? src[2] : 0.f, col + 3 < cols ? src[3] : 0.f);
            }
            if (first_layer) v = tc::spread_nan(v, 32);
            if (col < pad) most = fmaxf(most, tc::put_weight4<true>(hi, hi + kWeightImage / 2, row, col, v, 64.f));
        }
        if (!(most * 64.f <= 32768.f)) atomicOr(status, (int)kWeightRange);
        return;
    }
    // a warp takes four nodes: their types, then their rows (a thread per quad of columns, its node from a 64-bit division, took 40 % of the
    // issue slots: 51 200 nodes 11.4 us, now 7.3, in the middle of an evaluation)
    const int64_t Hv = H >> 2, warp = ((blockIdx.x - 8 * im.n) * (int64_t)blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x - 8 * im.n) * (int64_t)blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    for (int64_t n0 = warp * 4; n0 < N; n0 += warps * 4) {
        const int nodes = N - n0 < 4 ? (int)(N - n0) : 4;
        int64_t ty[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            ty[u] = types[n0 + (u < nodes ? u : 0)];
            if (ty[u] < 0 || ty[u] >= T) {
                if (lane == 0) atomicOr(status, (int)kBadIndex);
                ty[u] = 0;
            }
        }
        for (int64_t c = lane; c < Hv; c += 32) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = __ldg(reinterpret_cast<const float4 *>(table + ty[u] * H) + c);
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (u < nodes) reinterpret_cast<float4 *>(x)[(n0 + u) * Hv + c] = v[u];
        }
    }
}

int embedding_launch(const mlcgb_schnet_weights *w, const int64_t *types, int64_t N, float *x, void *images, int num_rbf, int32_t *status, cudaStream_t st) {
    TimelineScope timeline_scope("embedding", st);
    WeightImages im;
    im.n = 0;
    im.first_filter = kMaxImages;
    im.dst = (uint8_t *)images;
    auto add = [&](const void *src, int64_t rows, int cols = 128) {          // (a weight that is not there is refused by the kernel that takes it)
        im.src[im.n] = (const float *)src;
        im.rows[im.n] = (int16_t)(src ? rows : 0);
        im.cols[im.n++] = (int16_t)cols;
    };
    if (images) {
        for (int64_t l = 0; l < w->num_blocks; l++) {
            add(w->blocks[l].lin1_w, 128);
            add(w->blocks[l].lin2_w, 128);
            add(w->blocks[l].lin_w, 128);
        }
        add(w->head_W, w->head_width);
        im.first_filter = im.n;
        for (int64_t l = 0; l < w->num_blocks && num_rbf; l++) {
            add(w->blocks[l].filter_w1, 128, num_rbf);
            add(w->blocks[l].filter_w2, 128);
        }
    }
    launch_pdl(embedding_rows_kernel, dim3(8 * im.n + grid_for(N * 8, 256)), dim3(256), 0, st, (const float *)w->embedding, types, N, w->hidden,
               w->num_types, x, im, status);
    return check_launch();
}

// e[n] = sum_f a[n,f] w[f] + b: the last Linear layer of the output network (one output); one warp per node
__global__ void head_out_kernel(const float *__restrict__ a, const float *__restrict__ w, const float *__restrict__ b, int64_t N, int64_t F,
                                float *__restrict__ e) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    pdl_wait();
    for (int64_t n = warp; n < N; n += nwarps) {
        float s = 0.f;
        for (int64_t f = lane; f < F; f += 32) s = fmaf(a[n * F + f], w[f], s);
        s = warp_sum(s);
        if (lane == 0) e[n] = s + (b ? b[0] : 0.f);
    }
}

// tanh(agg W2^T + b2) -> a,  x + a W3^T + b3 -> out; one kernel where all widths are 128
static int node_layers_forward(const float *agg, const mlcgb_schnet_block &w, const float *x, int64_t N, int64_t H, int64_t F, int64_t H2, float *a,
                               float *out, const uint8_t *images, const ChainLink *link, int32_t *status, void *stream) {
    if (H == 128 && F == 128 && H2 == 128)
        return gemm_chain2(0, agg, w.lin2_w, w.lin2_b, w.lin_w, w.lin_b, x, N, a, out, images ? images + kLin2 * kWeightImage : nullptr,
                           images ? images + kLin * kWeightImage : nullptr, link, status, stream);
    int rc = mlcgb_gemm_tc_fused(0, agg, w.lin2_w, w.lin2_b, nullptr, 1, N, H2, F, a, status, stream);
    return rc ? rc : mlcgb_gemm_tc_fused(0, a, w.lin_w, w.lin_b, x, 2, N, H, H2, out, status, stream);
}
// ((g W3) (1 - a^2)) W2 -> gagg
static int node_layers_backward(const float *g, const mlcgb_schnet_block &w, const float *a, int64_t N, int64_t H, int64_t F, int64_t H2, float *gy,
                                float *gagg, const uint8_t *images, const ChainLink *link, int32_t *status, void *stream) {
    if (H == 128 && F == 128 && H2 == 128)
        return gemm_chain2(1, g, w.lin_w, nullptr, w.lin2_w, nullptr, a, N, nullptr, gagg, images ? images + kLin * kWeightImage : nullptr,
                           images ? images + kLin2 * kWeightImage : nullptr, link, status, stream);
    int rc = mlcgb_gemm_tc_fused(1, g, w.lin_w, nullptr, a, 3, N, H2, H, gy, status, stream);
    return rc ? rc : mlcgb_gemm_tc_fused(1, gy, w.lin2_w, nullptr, nullptr, 0, N, F, H2, gagg, status, stream);
}

// Every array starts on a 256-byte boundary: a row of 512 bytes that does not start on a line takes five lines instead of four (with 16-byte
// boundaries, by luck of the edge count: 634 -> 616 us for 96 x 268 ragged, 1860 -> 1808 for 512 x 100, dot products by pairs included)
static inline int64_t up64(int64_t n) { return (n + 63) & ~(int64_t)63; }

struct SchnetLayout {                                                        // offsets in floats
    int64_t d, x[2], g[2], agg, gy, gxl, ah, en, gd, gp, images, W, Wd, wstride, block0, block_stride, xl_off, a_off, total;   // images -1: none
};
static SchnetLayout schnet_layout(int64_t N, int64_t E, int64_t P, int64_t H, int64_t F, int64_t H2, int64_t Wh, int64_t L) {
    SchnetLayout o;
    int64_t at = 0;
    auto take = [&](int64_t n) { const int64_t r = at; at += up64(n); return r; };
    o.d = take(E);                                                           // (first: schnet_eval_distances)
    o.x[0] = take(N * H); o.x[1] = take(N * H);
    o.g[0] = take(N * H); o.g[1] = take(N * H);
    o.agg = take(N * F); o.gy = take(N * H2); o.gxl = take(N * F);
    o.ah = take(N * Wh); o.en = take(N);
    o.gd = take(E); o.gp = take(P);
    o.images = N > kSmallNodes && H == 128 && F == 128 && H2 == 128 && L <= kMaxBlocks ? take(weight_images_floats(L)) : -1;
    o.wstride = padded_rows(P) * F;
    o.W = take(L * o.wstride); o.Wd = take(L * o.wstride);                   // filter rows of all blocks, and their distance derivatives
    o.xl_off = 0; o.a_off = up64(N * F);
    o.block_stride = o.a_off + up64(N * H2);
    o.block0 = at;
    at += L * o.block_stride;
    o.total = at;
    return o;
}

}  // namespace mlcgb

extern "C" {

size_t mlcgb_schnet_eval_workspace_bytes(int64_t N, int64_t E, int64_t P, int64_t H, int64_t F, int64_t H2, int64_t head_width,
                                         int64_t num_blocks) {
    if (N < 0 || E < 0 || P < 0 || H <= 0 || F <= 0 || H2 <= 0 || head_width <= 0 || num_blocks < 0) return 0;
    return (size_t)schnet_layout(N, E, P, H, F, H2, head_width, num_blocks).total * sizeof(float);
}

int mlcgb_schnet_eval(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0,
                      const int32_t *row1, const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin,
                      int64_t E, int64_t P, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                      const mlcgb_schnet_weights *w, int precision, void *workspace, size_t workspace_bytes, void *energy,
                      void *grad_pos, int32_t *status, void *stream) {
    return mlcgb_schnet_eval_counted(pos, types, struct_ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, P, nullptr, rbf,
                                     conv_cutoff_kind, conv_lower, conv_upper, w, precision, workspace, workspace_bytes, energy, grad_pos,
                                     status, stream);
}

// counts: NULL, or {edges, pairs} in device memory as mlcgb_radius_graph_capacity leaves them.  E and P are then the
// capacities of the index arrays (whose entries past the live ones must be valid node / edge indices, e.g. zero): the
// edge-sized elementwise kernels run over the capacity, the filter kernels over the live pairs, everything else over nodes.
static int schnet_eval_impl(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B,
                              const int32_t *row0, const int32_t *row1, const int64_t *offsets, const int32_t *sel,
                              const int32_t *pair_of, const int32_t *twin, int64_t E, int64_t P, const int64_t *counts,
                              const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                              const mlcgb_schnet_weights *w, int precision, void *workspace, size_t workspace_bytes, void *energy,
                              void *grad_pos, float grad_sign, int32_t *status, void *stream, const SmallGraph *graph = nullptr, bool have_distances = false) {
    const int64_t *pairs_dev = counts ? counts + 1 : nullptr;
    if (N < 0 || B < 0 || E < 0 || P < 0 || !w || !status || !energy || !struct_ptr) return MLCGB_E_ARG;
    if (B == 0) return MLCGB_OK;
    const int64_t H = w->hidden, F = w->filters, H2 = w->conv_out, Wh = w->head_width, L = w->num_blocks;
    if (F != 128 || H > 128 || H2 > 128 || Wh > 128 || (H & 3) || (H2 & 3) || (Wh & 3) || L < 1) return MLCGB_E_LIMIT;
    if (!pos || !types || !offsets || !w->embedding || !w->blocks || !w->head_W || !w->head_b || !w->head_out || !workspace) return MLCGB_E_ARG;
    if (E > 0 && ((!row0 && !graph) || !row1 || (!sel && !graph) || !pair_of || !twin || 2 * P != E)) return MLCGB_E_ARG;
    if ((uintptr_t)w->embedding & 15) return MLCGB_E_LIMIT;                  // (its rows are read in pieces of 16 bytes)
    const SchnetLayout lay = schnet_layout(N, E, P, H, F, H2, Wh, L);
    if (workspace_bytes < (size_t)lay.total * sizeof(float)) return MLCGB_E_WORKSPACE;
    float *ws = (float *)workspace;
    auto st = (cudaStream_t)stream;
    float *d = ws + lay.d;
    int rc;
    // (the kernel behind the one that makes them converts its weight itself: it reads it before it waits for that one)
    const uint8_t *images = lay.images >= 0 && ((uintptr_t)ws & 15) == 0 ? (const uint8_t *)(ws + lay.images) : nullptr;
    auto image = [&](int64_t k) { return images ? images + k * kWeightImage : nullptr; };
    const bool filter_images = images && grad_pos && P > 0 && precision == 0 && rbf && rbf->num_rbf <= 128;
    auto filters = [&](int64_t l, int64_t n) {                               // of blocks l .. l + n - 1, with derivatives where a force pass follows
        float *W = ws + lay.W + l * lay.wstride;
        if (grad_pos)
            return filter_vd_blocks(graph ? graph->pair_d : d, P, pairs_dev, graph ? nullptr : sel, rbf, conv_cutoff_kind, conv_lower, conv_upper, w->blocks + l, n, precision, W,
                                    ws + lay.Wd + l * lay.wstride, nullptr, nullptr, nullptr, filter_images ? image(3 * L + 1 + 2 * l) : nullptr, status, st);
        int rf = MLCGB_OK;
        for (int64_t k = l; k < l + n && !rf; k++)
            rf = mlcgb_filter_forward_counted(d, P, pairs_dev, sel, nullptr, rbf, conv_cutoff_kind, conv_lower, conv_upper, w->blocks[k].filter_w1,
                                              w->blocks[k].filter_b1, w->blocks[k].filter_w2, F, precision, W + (k - l) * lay.wstride, nullptr, status, stream);
        return rf;
    };
    if (H == 128 && H2 == 128 && small_route(N, w)) {                        // one launch per link of the chain (small_route.cu)
        SmallForward f = {};
        f.pos = (const float *)pos; f.types = types; f.row0 = row0; f.row1 = row1; f.pair_of = pair_of; f.ptr = offsets;
        f.N = N; f.E = E; f.B = B; f.w = w; f.d = d; f.W = ws + lay.W; f.Wd = grad_pos ? ws + lay.Wd : nullptr; f.wstride = lay.wstride;
        for (int64_t l = 0; l < L; l++) {
            float *blk = ws + lay.block0 + l * lay.block_stride;
            f.x[l] = ws + lay.x[l & 1];
            f.xl[l] = blk + lay.xl_off;
            f.a[l] = blk + lay.a_off;
            f.g[l] = ws + lay.g[l & 1];
            f.gagg[l] = ws + (l & 1 ? lay.agg : lay.gxl);
        }
        f.ah = nullptr; f.en = ws + lay.en; f.s = ws + lay.gd; f.want_grad = grad_pos != nullptr; f.status = status;
        if ((rc = graph ? small_graph_start(f, *graph, st) : small_start(f, st))) return rc;
        ChainScope chain;
        if ((rc = filters(0, L))) return rc;       // (of all blocks at once: they depend on the distances alone)
        if ((rc = small_forward(f, st))) return rc;
        return small_finish(f, twin, struct_ptr, (float *)energy, (float *)grad_pos, grad_sign, st);
    }
    if (!have_distances && (rc = mlcgb_edge_distance(pos, MLCGB_F32, row0, row1, E, N, d, status, stream))) return rc;
    if ((rc = embedding_launch(w, types, N, ws + lay.x[0], (void *)images, filter_images ? rbf->num_rbf : 0, status, st))) return rc;
    ChainScope chain;
    int cur = 0;
    for (int64_t l = 0; l < L; l++) {
        const mlcgb_schnet_block &bw = w->blocks[l];
        float *blk = ws + lay.block0 + l * lay.block_stride;
        float *xin = ws + lay.x[cur], *xout = ws + lay.x[cur ^ 1], *xl = blk + lay.xl_off, *a = blk + lay.a_off, *agg = ws + lay.agg;
        if (l == 0 || !images) {                    // (else it came with the block before)
            rc = gemm_fused(0, xin, bw.lin1_w, nullptr, nullptr, 0, N, F, H, xl, nullptr, status, stream);
            if (rc) return rc;
        }
        if ((rc = filters(l, 1))) return rc;        // (block by block: what is written last is read first, some of it out of the L2)
        rc = mlcgb_seg_mul_sum(xl, ws + lay.W + l * lay.wstride, MLCGB_F32, offsets, row1, pair_of, N, P, F, agg, stream);
        if (rc) return rc;
        // what follows on the same rows: the next block's first layer, or the output network's, tanh(x W^T + b)
        const ChainLink link = l + 1 < L ? ChainLink{image(3 * (l + 1) + kLin1), nullptr, nullptr, nullptr, blk + lay.block_stride + lay.xl_off, 128, 0}
                                         : ChainLink{image(3 * L), (const float *)w->head_b, nullptr, nullptr, ws + lay.ah, (int)Wh, 1, (const float *)w->head_out,
                                                     (const float *)w->head_out_b, ws + lay.en};
        rc = node_layers_forward(agg, bw, xin, N, H, F, H2, a, xout, image(3 * l), images ? &link : nullptr, status, stream);
        if (rc) return rc;
        cur ^= 1;
    }
    // output network: tanh(x W^T + b) . w_out (+ b_out), summed per structure
    if (!images) {
        rc = gemm_fused(0, ws + lay.x[cur], w->head_W, w->head_b, nullptr, 1, N, Wh, H, ws + lay.ah, nullptr, status, stream);
        if (rc) return rc;
        TimelineScope timeline_scope("head_out", stream);
        launch_pdl(head_out_kernel, dim3(grid_for(N * 32, 256)), dim3(256), 0, st, (const float *)(ws + lay.ah), (const float *)w->head_out, (const float *)w->head_out_b, N, Wh, ws + lay.en);
    }
    if (!grad_pos) return mlcgb_segment_sum(ws + lay.en, MLCGB_F32, struct_ptr, B, energy, stream);

    // force pass: d(sum of energies)/d(pos)
    // through the output network: g = (w_out * (1 - a^2)) head_W, the factor applied as the GEMM reads its input tile
    int gcur = 0;
    // (with images each block's node layers take the layer before them along, which makes their input g)
    ChainLink link = {image(3 * L), nullptr, (const float *)w->head_out, nullptr, ws + lay.g[gcur], (int)Wh, 0};
    if (!images) {
        rc = gemm_fused(1, ws + lay.ah, w->head_W, nullptr, w->head_out, 4, N, H, Wh, ws + lay.g[gcur], nullptr, status, stream);
        if (rc) return rc;
    }
    for (int64_t l = L - 1; l >= 0; l--) {
        const mlcgb_schnet_block &bw = w->blocks[l];
        float *blk = ws + lay.block0 + l * lay.block_stride;
        float *g = ws + lay.g[gcur], *gnext = ws + lay.g[gcur ^ 1], *gagg = ws + lay.agg, *gxl = ws + lay.gxl;
        rc = node_layers_backward(!images ? g : l == L - 1 ? ws + lay.ah : gxl, bw, blk + lay.a_off, N, H, F, H2, ws + lay.gy, gagg, image(3 * l),
                                  images ? &link : nullptr, status, stream);
        if (rc) return rc;
        // s[e] of every block adds up in one array: the last block sets it, the others add
        if (l == 0) {
            if ((rc = seg_pair_dot(gagg, blk + lay.xl_off, ws + lay.Wd, offsets, row1, pair_of, twin, L > 1 ? ws + lay.gd : nullptr, N, ws + lay.gp, st))) return rc;
            break;
        }
        rc = mlcgb_seg_force(gagg, blk + lay.xl_off, ws + lay.W + l * lay.wstride, ws + lay.Wd + l * lay.wstride, offsets, row1, pair_of, N, F, gxl, ws + lay.gd,
                             l != L - 1, stream);
        if (rc) return rc;
        if (!images && (rc = gemm_fused(1, gxl, bw.lin1_w, nullptr, g, 2, N, H, F, gnext, nullptr, status, stream))) return rc;
        link = {image(3 * l + kLin1), nullptr, nullptr, g, gnext, 128, 0};
        gcur ^= 1;
    }
    return finish_launch((const float *)pos, ws + lay.gp, d, row1, offsets, pair_of, N, (float *)grad_pos, grad_sign, ws + lay.en, struct_ptr, B, (float *)energy, st);
}

}  // extern "C"

int mlcgb::schnet_eval_distances(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0, const int32_t *row1,
                                 const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin, int64_t E, const mlcgb_rbf_spec *rbf,
                                 int conv_cutoff_kind, double conv_lower, double conv_upper, const mlcgb_schnet_weights *w, int precision, void *workspace,
                                 size_t workspace_bytes, void *energy, void *grad_pos, float grad_sign, int32_t *status, void *stream) {
    return schnet_eval_impl(pos, types, struct_ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, E / 2, nullptr, rbf, conv_cutoff_kind, conv_lower,
                            conv_upper, w, precision, workspace, workspace_bytes, energy, grad_pos, grad_sign, status, stream, nullptr, true);
}

int mlcgb::schnet_eval_small(const void *pos, const int64_t *types, int64_t N, int64_t B, const SmallGraph &g, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind,
                             double conv_lower, double conv_upper, const mlcgb_schnet_weights *w, int precision, void *workspace, size_t workspace_bytes,
                             void *energy, void *grad_pos, float grad_sign, int32_t *status, cudaStream_t st) {
    if (!grad_pos || !small_graph_ok(N, B, w)) return MLCGB_E_LIMIT;
    return schnet_eval_impl(pos, types, g.ptr, N, B, nullptr, g.row1, g.offsets, nullptr, g.pair_of, g.twin, g.capacity, g.capacity / 2, g.counts, rbf,
                            conv_cutoff_kind, conv_lower, conv_upper, w, precision, workspace, workspace_bytes, energy, grad_pos, grad_sign, status, st, &g);
}

extern "C" {

int mlcgb_schnet_eval_counted(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0,
                              const int32_t *row1, const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin, int64_t E,
                              int64_t P, const int64_t *counts, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                              const mlcgb_schnet_weights *w, int precision, void *workspace, size_t workspace_bytes, void *energy, void *grad_pos,
                              int32_t *status, void *stream) {
    return schnet_eval_impl(pos, types, struct_ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, P, counts, rbf, conv_cutoff_kind, conv_lower,
                            conv_upper, w, precision, workspace, workspace_bytes, energy, grad_pos, 1.f, status, stream);
}

int mlcgb_schnet_energy_forces(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0,
                               const int32_t *row1, const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin, int64_t E,
                               int64_t P, const int64_t *counts, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                               const mlcgb_schnet_weights *w, int precision, void *workspace, size_t workspace_bytes, void *energy, void *forces,
                               int32_t *status, void *stream) {
    if (!forces) return MLCGB_E_ARG;
    return schnet_eval_impl(pos, types, struct_ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, P, counts, rbf, conv_cutoff_kind, conv_lower,
                            conv_upper, w, precision, workspace, workspace_bytes, energy, forces, -1.f, status, stream);
}

}  // extern "C"

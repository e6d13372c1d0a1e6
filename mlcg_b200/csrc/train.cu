// A force-matching step of SchNet as two kernel sequences issued from C: energies and forces with what their derivative needs kept,
// and the gradient of a loss on them with respect to every weight.
//
// Forces are -dE/dpos, so the loss reaches the weights through a second derivative.  With u = dL/d(dE/dpos) as a displacement of the
// positions, dL/dtheta = d/dtheta [ sum_b gE_b E_b + (dE/dpos) . u ], and the second term is the tangent of the energy along u:
// the backward pass runs the model once along that tangent and once back through values and tangents together.  The gradients
// of the tangents (g, gagg, gxl, gu) are those of the force pass: kept by the forward, not computed again.  Notation, block l:
//   xl = x W1^T   agg_i = sum_j xl_j W   a = tanh(agg W2^T + b2)   x' = x + a W3^T + b3            tangents: suffix t
//   g = dE/dx'    gu = (g W3)(1 - a^2)   gagg = gu W2              gxl_j = sum_i gagg_i W           gradients of values: suffix b
// A weight gradient is then a sum of two row-contracting products, e.g. dW2 = ub^T agg + gu^T aggt; all of the node-sized ones are
// one launch at the end (tn_jobs.cuh), the filter networks' one per block (filter_wgrad.cu).
#include "schnet_internal.cuh"
#include "tn_jobs.cuh"

namespace mlcgb {

__global__ void head_out_kernel(const float *a, const float *w, const float *b, int64_t N, int64_t F, float *e);

// Output network e = wo . tanh(y), its tangent along yt, and gE (per structure, NULL: zero); one warp per node:
//   yb = dS/dy = wo (1 - t^2) (gE - 2 t yt)     gy = dS/dyt = wo (1 - t^2)     r = dS/dwo (one term of the sum over nodes) = gE t + (1 - t^2) yt
__global__ void __launch_bounds__(256)
head_grad_kernel(const float *__restrict__ ah, const float *__restrict__ yt, const float *__restrict__ wo, const float *__restrict__ gE,
                 const int64_t *__restrict__ struct_ptr, int64_t N, int64_t B, int64_t F, float *__restrict__ yb, float *__restrict__ gy,
                 float *__restrict__ r) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    pdl_wait();
    for (int64_t n = warp; n < N; n += nwarps) {
        float ge = 0.f;
        if (gE) {
            int64_t lo = 0, hi = B - 1;               // the structure of node n: last b with struct_ptr[b] <= n
            while (lo < hi) {
                const int64_t mid = (lo + hi + 1) >> 1;
                if (struct_ptr[mid] <= n) lo = mid;
                else hi = mid - 1;
            }
            ge = gE[lo];
        }
        for (int64_t f = lane; f < F; f += 32) {
            const float t = ah[n * F + f], s = fmaf(-t, t, 1.f), y = yt[n * F + f];
            yb[n * F + f] = wo[f] * s * fmaf(-2.f * t, y, ge);
            gy[n * F + f] = wo[f] * s;
            r[n * F + f] = fmaf(ge, t, s * y);
        }
    }
}

// Sums of the rows of xb[N][128] by type: each group of 128 threads (thread = column) adds its rows, in order, to a table of its
// own in shared memory; the tables are added up by partial_sums_kernel
__global__ void __launch_bounds__(512)
embedding_grad_kernel(const float *__restrict__ xb, const int64_t *__restrict__ types, int64_t N, int T, float *__restrict__ partial) {
    extern __shared__ float s_table[];                // [groups][T][128]
    const int groups = blockDim.x >> 7, g = threadIdx.x >> 7, c = threadIdx.x & 127;
    float *tab = s_table + (int64_t)g * T * 128 + c;
    for (int t = 0; t < T; t++) tab[t * 128] = 0.f;
    const int64_t total = (int64_t)gridDim.x * groups, me = (int64_t)blockIdx.x * groups + g;
    const int64_t chunk = (N + total - 1) / total, n0 = me * chunk, n1 = n0 + chunk < N ? n0 + chunk : N;
    pdl_wait();
    int64_t n = n0;
    for (; n + 8 <= n1; n += 8) {
        float v[8];
        int ty[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            v[u] = __ldg(xb + (n + u) * 128 + c);
            const int64_t t = types[n + u];
            ty[u] = t < 0 || t >= T ? 0 : (int)t;      // (as the forward took it; its status word reports the index)
        }
#pragma unroll
        for (int u = 0; u < 8; u++) tab[ty[u] * 128] += v[u];
    }
    for (; n < n1; n++) {
        const int64_t t = types[n];
        tab[(t < 0 || t >= T ? 0 : (int)t) * 128] += xb[n * 128 + c];
    }
    for (int t = 0; t < T; t++) partial[(me * T + t) * 128 + c] = tab[t * 128];
}

// Before anything else of a forward pass: the positions as the backward will want them (the caller may overwrite his), zmax cleared
__global__ void __launch_bounds__(256)
train_begin_kernel(const float *__restrict__ pos, int64_t n, float *__restrict__ kept, float *__restrict__ zmax, int64_t L) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < L) zmax[t] = 0.f;
    for (int64_t i = t; i < n; i += (int64_t)gridDim.x * blockDim.x) kept[i] = pos[i];
}

constexpr int64_t kH = 128;

struct TrainForward {                                 // offsets in floats
    int64_t pos, d, gd, gp, en, ah, zmax, images, W, Wd, Hs, Zs, wstride, hstride, block0, stride, total;      // W .. Zs: of all blocks
    int64_t x, xl, agg, a, gu, gagg, gxl, g;          // of a block; g: the gradient of the block's output
};
struct TrainBackward {
    int64_t dd, yt, yb, gy, r, node_part, pair_part, emb_part, block0, stride, total;
    int64_t xt, xlt, aggt, at, q, ub, agb, xlb, xb;   // of a block: xt, xb belong to its OUTPUT
    int64_t pair_stride;
    int node_parts, emb_grid, emb_groups;
};

static TrainForward train_forward_layout(int64_t N, int64_t E, int64_t P, int64_t Wh, int64_t L) {
    TrainForward o;
    int64_t at = 0;
    auto take = [&](int64_t n) { const int64_t r = at; at += (n + 63) & ~(int64_t)63; return r; };      // (arrays on 256-byte boundaries)
    const int64_t hidden = (int64_t)(mlcgb_filter_hidden_bytes(P) / sizeof(float));
    o.pos = take(3 * N);
    o.d = take(E); o.gd = take(E); o.gp = take(P); o.en = take(N); o.ah = take(N * Wh); o.zmax = take(L);
    o.images = N > kSmallNodes ? take(weight_images_floats(L)) : -1;
    o.wstride = padded_rows(P) * kH;
    o.hstride = hidden;
    o.W = take(L * o.wstride); o.Wd = take(L * o.wstride); o.Hs = take(L * hidden); o.Zs = take(L * hidden);
    o.block0 = at;
    at = 0;
    o.x = take(N * kH); o.xl = take(N * kH); o.agg = take(N * kH); o.a = take(N * kH); o.gu = take(N * kH); o.gagg = take(N * kH); o.gxl = take(N * kH); o.g = take(N * kH);
    o.stride = at;
    o.total = o.block0 + L * o.stride + N * kH;       // ... and the last block's output
    return o;
}
static TrainBackward train_backward_layout(int64_t N, int64_t E, int64_t P, int64_t R, int64_t Wh, int64_t L, int64_t T) {
    TrainBackward o;
    int64_t at = 0;
    auto take = [&](int64_t n) { const int64_t r = at; at += (n + 63) & ~(int64_t)63; return r; };      // (arrays on 256-byte boundaries)
    const int64_t jobs = 3 * L + 2;
    const int64_t tiles = 2 * ((N + 127) / 128);
    o.node_parts = (int)(kNumSM / jobs < 1 ? 1 : kNumSM / jobs);
    if (o.node_parts > tiles) o.node_parts = (int)tiles;
    o.emb_groups = T <= 96 ? 4 : 1;
    const int64_t emb_rows = (N + 31) / 32;           // at least 32 rows for a group
    o.emb_grid = (int)((emb_rows + o.emb_groups - 1) / o.emb_groups);
    if (o.emb_grid > kNumSM) o.emb_grid = kNumSM;
    o.pair_stride = kH * kH + kH * R + kH;
    o.dd = take(E); o.yt = take(N * Wh); o.yb = take(N * Wh); o.gy = take(N * Wh); o.r = take(N * Wh);
    o.node_part = take(jobs * o.node_parts * (kH * kH + kH));
    o.pair_part = take(L * filter_wgrad_parts(P, L) * o.pair_stride);
    o.emb_part = take((int64_t)o.emb_grid * o.emb_groups * T * kH);
    o.block0 = at;
    at = 0;
    o.xt = take(N * kH); o.xlt = take(N * kH); o.aggt = take(N * kH); o.at = take(N * kH); o.q = take(N * kH); o.ub = take(N * kH);
    o.agb = take(N * kH); o.xlb = take(N * kH); o.xb = take(N * kH);
    o.stride = at;
    o.total = o.block0 + L * o.stride + N * kH;       // ... and the gradient of the first block's input
    return o;
}
static int train_supported(const mlcgb_schnet_weights *w, int64_t R) {
    const int64_t jobs = 3 * w->num_blocks + 2, sums = 8 * w->num_blocks + 4;
    return w->hidden == kH && w->filters == kH && w->conv_out == kH && w->head_width >= 4 && w->head_width <= 128 && (w->head_width & 3) == 0 &&
           w->num_blocks >= 1 && w->num_blocks <= kMaxBlocks && jobs <= kMaxTnJobs && sums <= kMaxPartialSums && w->num_types <= 400 && R <= 128;
}

// what the small route (small_route.cu) reads and writes of a forward workspace
static SmallForward small_view(const TrainForward &o, float *ws, const void *pos, const int64_t *types, const int32_t *row0, const int32_t *row1,
                               const int32_t *pair_of, const int64_t *offsets, int64_t N, int64_t E, int64_t B, const mlcgb_schnet_weights *w,
                               int32_t *status) {
    SmallForward f = {};
    f.pos = (const float *)pos; f.types = types; f.row0 = row0; f.row1 = row1; f.pair_of = pair_of; f.ptr = offsets;
    f.N = N; f.E = E; f.B = B; f.w = w; f.d = ws + o.d; f.W = ws + o.W; f.Wd = ws + o.Wd; f.wstride = o.wstride;
    for (int64_t l = 0; l < w->num_blocks; l++) {
        float *b = ws + o.block0 + l * o.stride;
        f.x[l] = b + o.x; f.xl[l] = b + o.xl; f.agg[l] = b + o.agg; f.a[l] = b + o.a; f.gu[l] = b + o.gu; f.gagg[l] = b + o.gagg;
        f.gxl[l] = b + o.gxl; f.g[l] = b + o.g;
    }
    f.x[w->num_blocks] = ws + o.block0 + w->num_blocks * o.stride;
    f.ah = ws + o.ah; f.en = ws + o.en; f.s = ws + o.gd; f.want_grad = 1; f.status = status;
    return f;
}

size_t train_distances_at(int64_t N, int64_t E, int64_t head_width, int64_t num_blocks) {
    return sizeof(float) * (size_t)train_forward_layout(N, E, E / 2, head_width, num_blocks).d;
}

}  // namespace mlcgb

using namespace mlcgb;

extern "C" {

size_t mlcgb_schnet_train_workspace_bytes(int backward, int64_t N, int64_t E, int64_t P, int64_t num_rbf, int64_t head_width, int64_t num_blocks,
                                          int64_t num_types) {
    if (N < 0 || E < 0 || P < 0 || num_rbf <= 0 || head_width <= 0 || num_blocks < 1 || num_types < 1) return 0;
    return sizeof(float) * (size_t)(backward ? train_backward_layout(N, E, P, num_rbf, head_width, num_blocks, num_types).total
                                             : train_forward_layout(N, E, P, head_width, num_blocks).total);
}

}  // extern "C"

int mlcgb::schnet_train_forward(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0,
                               const int32_t *row1, const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin,
                               int64_t E, int64_t P, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                               const mlcgb_schnet_weights *w, int negate, bool have_distances, void *workspace, size_t workspace_bytes, void *energy,
                               void *grad_pos, int32_t *status, void *stream) {
    if (!rbf || !w || N <= 0 || B <= 0 || E <= 0 || 2 * P != E) return MLCGB_E_ARG;
    if (!pos || !types || !struct_ptr || !row0 || !row1 || !offsets || !sel || !pair_of || !twin || !workspace || !energy || !grad_pos || !status)
        return MLCGB_E_ARG;
    if (!train_supported(w, rbf->num_rbf) || ((uintptr_t)w->embedding & 15)) return MLCGB_E_LIMIT;      // (the table's rows are read in pieces of 16 bytes)
    const int64_t Wh = w->head_width, L = w->num_blocks;
    const TrainForward o = train_forward_layout(N, E, P, Wh, L);
    if (workspace_bytes < (size_t)o.total * sizeof(float)) return MLCGB_E_WORKSPACE;
    float *ws = (float *)workspace, *d = ws + o.d;
    auto st = (cudaStream_t)stream;
    auto blk = [&](int64_t l) { return ws + o.block0 + l * o.stride; };
    train_begin_kernel<<<grid_for(3 * N, 256), 256, 0, st>>>((const float *)pos, 3 * N, ws + o.pos, ws + o.zmax, L);
    ChainScope chain;
    const uint8_t *images = N > kSmallNodes && ((uintptr_t)ws & 15) == 0 ? (const uint8_t *)(ws + o.images) : nullptr;
    auto image = [&](int64_t k) { return images ? images + k * kWeightImage : nullptr; };
    auto filters = [&](int64_t l, int64_t n) {
        return filter_vd_blocks(d, P, nullptr, sel, rbf, conv_cutoff_kind, conv_lower, conv_upper, w->blocks + l, n, 0, ws + o.W + l * o.wstride,
                                ws + o.Wd + l * o.wstride, ws + o.Hs + l * o.hstride, ws + o.Zs + l * o.hstride, ws + o.zmax + l, image(3 * L + 1 + 2 * l), status, st);
    };
    if (small_route(N, w)) {
        const SmallForward f = small_view(o, ws, pos, types, row0, row1, pair_of, offsets, N, E, B, w, status);
        int rs = small_start(f, st);
        if (!rs) rs = filters(0, L);
        if (!rs) rs = small_forward(f, st);
        return rs ? rs : small_finish(f, twin, struct_ptr, (float *)energy, (float *)grad_pos, negate ? -1.f : 1.f, st);
    }
    int rc = have_distances ? MLCGB_OK : mlcgb_edge_distance(pos, MLCGB_F32, row0, row1, E, N, d, status, stream);
    if (rc) return rc;
    if ((rc = embedding_launch(w, types, N, blk(0) + o.x, (void *)images, rbf->num_rbf, status, st))) return rc;
    for (int64_t l = 0; l < L; l++) {
        const mlcgb_schnet_block &bw = w->blocks[l];
        float *b = blk(l), *xout = l + 1 < L ? blk(l + 1) + o.x : ws + o.block0 + L * o.stride;
        if ((l == 0 || !images) && (rc = gemm_fused(0, b + o.x, bw.lin1_w, nullptr, nullptr, 0, N, kH, kH, b + o.xl, nullptr, status, stream))) return rc;
        if ((rc = filters(l, 1))) return rc;
        if ((rc = mlcgb_seg_mul_sum(b + o.xl, ws + o.W + l * o.wstride, MLCGB_F32, offsets, row1, pair_of, N, P, kH, b + o.agg, stream))) return rc;
        // (with images the layer that follows on the same rows, the next block's first or the output network's, comes along)
        const ChainLink link = l + 1 < L ? ChainLink{image(3 * (l + 1) + kLin1), nullptr, nullptr, nullptr, blk(l + 1) + o.xl, (int)kH, 0}
                                         : ChainLink{image(3 * L), (const float *)w->head_b, nullptr, nullptr, ws + o.ah, (int)Wh, 1, (const float *)w->head_out,
                                                     (const float *)w->head_out_b, ws + o.en};
        if ((rc = gemm_chain2(0, b + o.agg, bw.lin2_w, bw.lin2_b, bw.lin_w, bw.lin_b, b + o.x, N, b + o.a, xout, image(3 * l + kLin2), image(3 * l + kLin),
                              images ? &link : nullptr, status, stream)))
            return rc;
    }
    float *xL = ws + o.block0 + L * o.stride, *ah = ws + o.ah;
    if (!images && (rc = gemm_fused(0, xL, w->head_W, w->head_b, nullptr, 1, N, Wh, kH, ah, nullptr, status, stream))) return rc;
    if (!images) {
        TimelineScope timeline_scope("head_out", stream);
        launch_pdl(head_out_kernel, dim3(grid_for(N * 32, 256)), dim3(256), 0, st, (const float *)ah, (const float *)w->head_out, (const float *)w->head_out_b, N,
                   Wh, ws + o.en);
    }
    // force pass; block l's g is the gradient of its output
    if (!images && (rc = gemm_fused(1, ah, w->head_W, nullptr, w->head_out, 4, N, kH, Wh, blk(L - 1) + o.g, nullptr, status, stream))) return rc;
    ChainLink link = {image(3 * L), nullptr, (const float *)w->head_out, nullptr, blk(L - 1) + o.g, (int)Wh, 0};      // (the layer in front of a block's, which makes its g)
    for (int64_t l = L - 1; l >= 0; l--) {
        const mlcgb_schnet_block &bw = w->blocks[l];
        float *b = blk(l);
        if ((rc = gemm_chain2(1, !images ? b + o.g : l == L - 1 ? ah : blk(l + 1) + o.gxl, bw.lin_w, nullptr, bw.lin2_w, nullptr, b + o.a, N, b + o.gu, b + o.gagg,
                              image(3 * l + kLin), image(3 * l + kLin2), images ? &link : nullptr, status, stream)))
            return rc;
        if (l == 0) {
            if ((rc = seg_pair_dot(b + o.gagg, b + o.xl, ws + o.Wd, offsets, row1, pair_of, twin, L > 1 ? ws + o.gd : nullptr, N, ws + o.gp, st))) return rc;
            break;
        }
        if ((rc = mlcgb_seg_force(b + o.gagg, b + o.xl, ws + o.W + l * o.wstride, ws + o.Wd + l * o.wstride, offsets, row1, pair_of, N, kH, b + o.gxl, ws + o.gd, l != L - 1,
                                  stream)))
            return rc;
        if (!images && (rc = gemm_fused(1, b + o.gxl, bw.lin1_w, nullptr, b + o.g, 2, N, kH, kH, blk(l - 1) + o.g, nullptr, status, stream))) return rc;
        link = {image(3 * l + kLin1), nullptr, nullptr, b + o.g, blk(l - 1) + o.g, (int)kH, 0};
    }
    return finish_launch((const float *)pos, ws + o.gp, d, row1, offsets, pair_of, N, (float *)grad_pos, negate ? -1.f : 1.f, ws + o.en, struct_ptr, B, (float *)energy, st);
}

extern "C" {

int mlcgb_schnet_train_forward(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0,
                               const int32_t *row1, const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin,
                               int64_t E, int64_t P, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                               const mlcgb_schnet_weights *w, int negate, void *workspace, size_t workspace_bytes, void *energy, void *grad_pos,
                               int32_t *status, void *stream) {
    return schnet_train_forward(pos, types, struct_ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, P, rbf, conv_cutoff_kind, conv_lower, conv_upper, w,
                                negate, false, workspace, workspace_bytes, energy, grad_pos, status, stream);
}

int mlcgb_schnet_train_backward(const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0,
                                const int32_t *row1, const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, int64_t E, int64_t P,
                                const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                                const mlcgb_schnet_weights *w, int negate, const void *gE, const void *gG, const void *forward_workspace, void *workspace,
                                size_t workspace_bytes, const mlcgb_schnet_weights *grads, int32_t *status, void *stream) {
    if (!rbf || !w || !grads || N <= 0 || B <= 0 || E <= 0 || 2 * P != E) return MLCGB_E_ARG;
    if (!types || !struct_ptr || !row0 || !row1 || !offsets || !sel || !pair_of || !gG || !forward_workspace || !workspace || !status) return MLCGB_E_ARG;
    const int64_t R = rbf->num_rbf, Wh = w->head_width, L = w->num_blocks, T = w->num_types;
    if (!train_supported(w, R)) return MLCGB_E_LIMIT;
    const TrainForward o = train_forward_layout(N, E, P, Wh, L);
    const TrainBackward v = train_backward_layout(N, E, P, R, Wh, L, T);
    if (workspace_bytes < (size_t)v.total * sizeof(float)) return MLCGB_E_WORKSPACE;
    const float *fw = (const float *)forward_workspace, *d = fw + o.d, *pos = fw + o.pos;
    float *ws = (float *)workspace, *dd = ws + v.dd;
    auto st = (cudaStream_t)stream;
    auto fblk = [&](int64_t l) { return fw + o.block0 + l * o.stride; };
    auto blk = [&](int64_t l) { return ws + v.block0 + l * v.stride; };
    const float *xL = fw + o.block0 + L * o.stride;
    float *xb0 = ws + v.block0 + L * v.stride;         // gradient of the first block's input
    int rc = mlcgb_edge_tangent(pos, gG, d, row0, row1, E, negate, dd, stream);
    if (rc) return rc;
    ChainScope chain;
    float *yb = ws + v.yb, *gy = ws + v.gy, *r = ws + v.r;
    if (small_route(N, w)) {
        const SmallForward f = small_view(o, const_cast<float *>(fw), pos, types, row0, row1, pair_of, offsets, N, E, B, w, status);
        SmallBackward sb = {};
        sb.dd = dd; sb.gE = (const float *)gE; sb.struct_ptr = struct_ptr; sb.yb = yb; sb.gy = gy; sb.r = r;
        for (int64_t l = 0; l < L; l++) {
            float *b = blk(l);
            sb.xt[l] = b + v.xt; sb.xlt[l] = b + v.xlt; sb.aggt[l] = b + v.aggt; sb.at[l] = b + v.at; sb.q[l] = b + v.q; sb.ub[l] = b + v.ub;
            sb.agb[l] = b + v.agb; sb.xlb[l] = b + v.xlb; sb.xb[l + 1] = b + v.xb;
        }
        sb.xb[0] = xb0;
        if ((rc = small_backward(f, sb, st))) return rc;
    } else {
        const uint8_t *images = N > kSmallNodes && ((uintptr_t)fw & 15) == 0 ? (const uint8_t *)(fw + o.images) : nullptr;
        auto image = [&](int64_t k) { return images ? images + k * kWeightImage : nullptr; };
        // ---- along the tangent
        for (int64_t l = 0; l < L; l++) {
            const mlcgb_schnet_block &bw = w->blocks[l];
            const float *f = fblk(l), *xt_in = l > 0 ? blk(l - 1) + v.xt : nullptr;
            float *b = blk(l);
            if (l > 0 && !images && (rc = gemm_fused(0, xt_in, bw.lin1_w, nullptr, nullptr, 0, N, kH, kH, b + v.xlt, nullptr, status, stream))) return rc;
            if ((rc = mlcgb_seg_tangent(l > 0 ? b + v.xlt : nullptr, f + o.xl, fw + o.W + l * o.wstride, fw + o.Wd + l * o.wstride, dd, offsets, row1, pair_of, N, kH, b + v.aggt, stream))) return rc;
            const ChainLink link = l + 1 < L ? ChainLink{image(3 * (l + 1) + kLin1), nullptr, nullptr, nullptr, blk(l + 1) + v.xlt, (int)kH, 0}
                                             : ChainLink{image(3 * L), nullptr, nullptr, nullptr, ws + v.yt, (int)Wh, 0};
            if ((rc = gemm_chain2_tangent(0, b + v.aggt, bw.lin2_w, bw.lin_w, f + o.a, f + o.gu, xt_in, N, b + v.q, b + v.at, b + v.xt, image(3 * l + kLin2),
                                          image(3 * l + kLin), images ? &link : nullptr, status, stream)))
                return rc;
        }
        // ---- output network
        const float *ah = fw + o.ah;
        float *yt = ws + v.yt;
        if (!images && (rc = gemm_fused(0, blk(L - 1) + v.xt, w->head_W, nullptr, nullptr, 0, N, Wh, kH, yt, nullptr, status, stream))) return rc;
        {
            TimelineScope timeline_scope("head_grad", stream);
            launch_pdl(head_grad_kernel, dim3(grid_for(N * 32, 256)), dim3(256), 0, st, ah, (const float *)yt, (const float *)w->head_out, (const float *)gE,
                       struct_ptr, N, B, Wh, yb, gy, r);
        }
        if (!images && (rc = gemm_fused(1, yb, w->head_W, nullptr, nullptr, 0, N, kH, Wh, blk(L - 1) + v.xb, nullptr, status, stream))) return rc;
        ChainLink link = {image(3 * L), nullptr, nullptr, nullptr, blk(L - 1) + v.xb, (int)Wh, 0};
        // ---- and back
        for (int64_t l = L - 1; l >= 0; l--) {
            const mlcgb_schnet_block &bw = w->blocks[l];
            const float *f = fblk(l);
            float *b = blk(l);
            if ((rc = gemm_chain2_tangent(1, !images ? b + v.xb : l == L - 1 ? yb : blk(l + 1) + v.xlb, bw.lin_w, bw.lin2_w, f + o.a, nullptr, nullptr, N, b + v.q,
                                          b + v.ub, b + v.agb, image(3 * l + kLin), image(3 * l + kLin2), images ? &link : nullptr, status, stream)))
                return rc;
            if ((rc = mlcgb_seg_tangent(b + v.agb, f + o.gagg, fw + o.W + l * o.wstride, fw + o.Wd + l * o.wstride, dd, offsets, row1, pair_of, N, kH, b + v.xlb, stream))) return rc;
            if ((l == 0 || !images) && (rc = gemm_fused(1, b + v.xlb, bw.lin1_w, nullptr, b + v.xb, 2, N, kH, kH, l > 0 ? blk(l - 1) + v.xb : xb0, image(3 * l + kLin1), status, stream))) return rc;
            if (l > 0) link = {image(3 * l + kLin1), nullptr, nullptr, b + v.xb, blk(l - 1) + v.xb, (int)kH, 0};
        }
    }
    // ---- the filter networks
    const int pair_parts = filter_wgrad_parts(P, L);
    float *pair_part = ws + v.pair_part;
    FilterGradBlock gb[kMaxBlocks];
    for (int64_t l = 0; l < L; l++)
        gb[l] = {(const float *)w->blocks[l].filter_w2, fblk(l) + o.xl, l > 0 ? blk(l) + v.xlt : nullptr, fblk(l) + o.gagg, blk(l) + v.agb};
    if ((rc = filter_wgrad_blocks(d, dd, P, sel, row0, row1, rbf, conv_cutoff_kind, conv_lower, conv_upper, gb, L, fw + o.Hs, fw + o.Zs, fw + o.zmax, pair_part,
                                  status, st)))
        return rc;
    // ---- weight gradients: node-sized products, embedding rows, then every sum of partials
    TnJobs jobs;
    PartialSums sums;
    int nj = 0, ns = 0;
    sums.sum[ns++] = {ws + v.emb_part, (float *)grads->embedding, T * kH, (int)(T * kH), v.emb_grid * v.emb_groups};   // (the longest chains first)
    jobs.E = N;
    jobs.parts = v.node_parts;
    float *part = ws + v.node_part;
    auto job = [&](const float *A0, const float *B0, const float *A1, const float *B1, int M, const void *dst, const void *dst_bias) {
        float *cs = part + (int64_t)v.node_parts * M * kH;
        jobs.job[nj++] = {{A0, A1}, {B0, B1}, part, dst_bias ? cs : nullptr, M, (int)kH, A1 ? 2 : 1};
        if (dst) sums.sum[ns++] = {part, (float *)dst, M * kH, (int)(M * kH), v.node_parts};
        if (dst_bias) sums.sum[ns++] = {cs, (float *)dst_bias, M, M, v.node_parts};
        part += (int64_t)v.node_parts * (kH * kH + kH);
    };
    for (int64_t l = 0; l < L; l++) {
        const mlcgb_schnet_block &gw = grads->blocks[l];
        const float *f = fblk(l), *b = blk(l);
        job(b + v.xlb, f + o.x, l > 0 ? f + o.gxl : nullptr, l > 0 ? blk(l - 1) + v.xt : nullptr, kH, gw.lin1_w, nullptr);
        job(b + v.ub, f + o.agg, f + o.gu, b + v.aggt, kH, gw.lin2_w, gw.lin2_b);
        job(b + v.xb, f + o.a, f + o.g, b + v.at, kH, gw.lin_w, gw.lin_b);
        const float *pp = pair_part + l * pair_parts * v.pair_stride;
        sums.sum[ns++] = {pp, (float *)gw.filter_w2, v.pair_stride, (int)(kH * kH), pair_parts};
        sums.sum[ns++] = {pp + kH * kH, (float *)gw.filter_w1, v.pair_stride, (int)(kH * R), pair_parts};
        sums.sum[ns++] = {pp + kH * kH + kH * R, (float *)gw.filter_b1, v.pair_stride, (int)kH, pair_parts};
    }
    job(yb, xL, gy, blk(L - 1) + v.xt, (int)Wh, grads->head_W, grads->head_b);
    job(r, xL, nullptr, nullptr, (int)Wh, nullptr, grads->head_out);
    {
        TimelineScope timeline_scope("weight_gradients", stream);
        static bool done[64] = {false};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 0 && dev < 64 && !done[dev]) {
            if (cudaFuncSetAttribute(embedding_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 400 * 512) != cudaSuccess) return check_launch();
            done[dev] = true;
        }
        launch_pdl(embedding_grad_kernel, dim3(v.emb_grid), dim3(128 * v.emb_groups), (size_t)v.emb_groups * T * 512, st, (const float *)xb0, types, N, (int)T,
                   ws + v.emb_part);
        if ((rc = tn_jobs_launch(jobs, nj, status, st))) return rc;
        if ((rc = partial_sums_launch(sums, ns, st))) return rc;
    }
    return check_launch();
}

}  // extern "C"

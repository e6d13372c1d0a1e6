// Energies and forces from positions in one library call: radius graph with its pair plan, then the SchNet evaluation, with the edge
// count handed to the host in between by the graph's mapped line.  The lists never leave the workspace, so nothing is allocated and
// no caller's code runs between the count's arrival and the launches that need it: for a single small structure that gap was as
// long as all of its kernels (127 -> 99 us per evaluation of 73 beads).
#include "common.cuh"
#include "schnet_internal.cuh"

using namespace mlcgb;

namespace {

inline size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

struct GraphPart {
    size_t graph, offsets, ptr, total;
};
inline GraphPart graph_part(int64_t N, int64_t B) {
    GraphPart p;
    p.graph = mlcgb_graph_workspace_bytes(N, B, MLCGB_F32);
    p.offsets = up256(p.graph);
    p.ptr = p.offsets + up256((size_t)(N + 1) * 8);
    p.total = p.ptr + up256((size_t)(B + 1) * 8);
    return p;
}
inline size_t list_bytes(int64_t E) { return 4 * up256((size_t)E * 4) + up256((size_t)(E / 2) * 4); }

// the graph of a small batch with lists of `capacity` edges, and the evaluation behind it
int evaluate_small(const void *pos, const int64_t *types, const int64_t *n_atoms, int64_t *ptr, int64_t N, int64_t B, double r, int64_t max_nn,
                   const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper, const mlcgb_schnet_weights *w, int precision,
                   int negate, int64_t capacity, int32_t *row1, char *g, const GraphPart &G, char *at, size_t bytes, void *energy, void *grad_pos, const Publish &pub,
                   int32_t *status, cudaStream_t st) {
    if (G.graph < small_graph_scratch(N) || ((uintptr_t)at & 255) || ((uintptr_t)g & 15)) return MLCGB_E_ARG;
    const size_t row = up256((size_t)capacity * 4), lists = list_bytes(capacity);
    SmallGraph s = {};
    s.sizes = n_atoms;
    s.ptr = ptr;
    s.r = r;
    s.max_nn = max_nn;
    s.capacity = capacity;
    s.counts = (int64_t *)g;
    s.masks = (uint2 *)(g + 256);
    s.deg = (int32_t *)(g + 256 + (size_t)N * ((N + 31) / 32) * 8);
    s.upper = s.deg + N;
    s.row1 = row1 ? row1 : (int32_t *)(at + row);      // (places as below, without row0)
    s.twin = (int32_t *)(at + 2 * row);
    s.pair_of = (int32_t *)(at + 3 * row);
    s.pair_d = (float *)(at + 4 * row);
    s.offsets = (int64_t *)(g + G.offsets);
    s.pub = pub;
    return schnet_eval_small(pos, types, N, B, s, rbf, conv_cutoff_kind, conv_lower, conv_upper, w, precision, at + lists, bytes - lists, energy, grad_pos,
                             negate ? -1.f : 1.f, status, st);
}

}  // namespace

extern "C" {

int mlcgb_schnet_evaluate_fixed_ok(int64_t N, int64_t B, const mlcgb_schnet_weights *w) { return w && small_graph_ok(N, B, w); }

int mlcgb_schnet_evaluate_fixed(const void *pos, const int64_t *types, const int64_t *n_atoms, const int64_t *struct_ptr, int64_t N, int64_t B, double r,
                                int64_t max_nn, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                                const mlcgb_schnet_weights *w, int precision, int negate, int64_t capacity, int32_t *neighbours, void *graph_workspace,
                                size_t graph_bytes,
                                void *workspace, size_t workspace_bytes, void *energy, void *grad_pos, int32_t *status, void *stream) {
    if (N <= 0 || B <= 0 || max_nn < 0 || capacity < 0 || (capacity & 1) || !pos || !types || !w || !rbf || !energy || !grad_pos || !status || !graph_workspace ||
        !workspace || (!n_atoms && !struct_ptr))
        return MLCGB_E_ARG;
    if (!small_graph_ok(N, B, w)) return MLCGB_E_LIMIT;
    const GraphPart G = graph_part(N, B);
    if (graph_bytes < G.total || workspace_bytes < mlcgb_schnet_evaluate_workspace_bytes(N, B, capacity, rbf->num_rbf, w, 0)) return MLCGB_E_WORKSPACE;
    char *g = (char *)graph_workspace;
    return evaluate_small(pos, types, n_atoms, n_atoms ? (int64_t *)(g + G.ptr) : const_cast<int64_t *>(struct_ptr), N, B, r, max_nn, rbf, conv_cutoff_kind,
                          conv_lower, conv_upper, w, precision, negate, capacity, neighbours, g, G, (char *)workspace, workspace_bytes, energy, grad_pos, Publish{}, status,
                          (cudaStream_t)stream);
}

size_t mlcgb_schnet_evaluate_workspace_bytes(int64_t N, int64_t B, int64_t E, int64_t num_rbf, const mlcgb_schnet_weights *w, int training) {
    if (N <= 0 || B <= 0 || !w) return 0;
    if (E < 0) return graph_part(N, B).total;
    if (training) return list_bytes(E) + mlcgb_schnet_train_workspace_bytes(0, N, E, E / 2, num_rbf, w->head_width, w->num_blocks, w->num_types);
    return list_bytes(E) + mlcgb_schnet_eval_workspace_bytes(N, E, E / 2, w->hidden, w->filters, w->conv_out, w->head_width, w->num_blocks);
}

int mlcgb_schnet_evaluate(const void *pos, const int64_t *types, const int64_t *n_atoms, const int64_t *struct_ptr, int64_t N, int64_t B, double r,
                          int64_t max_nn, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper,
                          const mlcgb_schnet_weights *w, int precision, int negate, int training, void *graph_workspace, size_t graph_bytes,
                          void *workspace, size_t workspace_bytes, void *energy, void *grad_pos, const int32_t *pending_status, int32_t *status,
                          int64_t *host, void *stream) {
    if (N <= 0 || B <= 0 || !pos || !types || !w || !rbf || !energy || !grad_pos || !status || !host || !graph_workspace || (!n_atoms && !struct_ptr))
        return MLCGB_E_ARG;
    const GraphPart G = graph_part(N, B);
    if (graph_bytes < G.total) return MLCGB_E_WORKSPACE;
    char *g = (char *)graph_workspace;
    auto *offsets = (int64_t *)(g + G.offsets);
    auto *ptr = n_atoms ? (int64_t *)(g + G.ptr) : const_cast<int64_t *>(struct_ptr);
    if (!training && workspace && max_nn >= 0 && small_graph_ok(N, B, w)) {
        // as many edges as the workspace has room for (none on a first call without a guess); the host looks at the count last
        auto bytes = [&](int64_t pairs) { return mlcgb_schnet_evaluate_workspace_bytes(N, B, 2 * pairs, rbf->num_rbf, w, 0); };
        int64_t lo = 0, hi = N * (N - 1) / 2;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (bytes(mid) <= workspace_bytes) lo = mid;
            else hi = mid - 1;
        }
        if (lo > 0) {
            Publish pub;
            int rc = publish_begin(&pub);
            if (rc) return rc;
            pub.pending = pending_status;
            rc = evaluate_small(pos, types, n_atoms, ptr, N, B, r, max_nn, rbf, conv_cutoff_kind, conv_lower, conv_upper, w, precision, negate, 2 * lo, nullptr, g, G,
                                (char *)workspace, workspace_bytes, energy, grad_pos, pub, status, (cudaStream_t)stream);
            if (rc || (rc = publish_wait(pub, (cudaStream_t)stream))) return rc;
            for (int i = 0; i < 4; i++) host[i] = pub.host[1 + i];
            host[4] = (host[1] & (kTruncated | kSizes)) || host[0] <= 0 || (host[0] & 1) ? MLCGB_EVALUATE_NO_PLAN : host[0] > 2 * lo ? MLCGB_EVALUATE_MORE : MLCGB_EVALUATE_DONE;
            return MLCGB_OK;
        }
    }
    if (host[4] != MLCGB_EVALUATE_MORE) {
        if (int rc = mlcgb_graph_begin(pos, MLCGB_F32, n_atoms, ptr, N, B, r, max_nn, 0, MLCGB_RULE_CLUSTER, nullptr, nullptr, g, G.graph, offsets,
                                       pending_status, host, stream))
            return rc;
    }
    const int64_t E = host[0];
    host[4] = MLCGB_EVALUATE_NO_PLAN;
    if ((host[1] & (kTruncated | kSizes)) || E <= 0 || (E & 1) || E >= (int64_t)1 << 31) return MLCGB_OK;
    host[4] = MLCGB_EVALUATE_MORE;
    if (!workspace || workspace_bytes < mlcgb_schnet_evaluate_workspace_bytes(N, B, E, rbf->num_rbf, w, training)) return MLCGB_OK;
    if ((uintptr_t)workspace & 255) return MLCGB_E_ARG;
    const size_t row = up256((size_t)E * 4);
    char *at = (char *)workspace;
    auto *row0 = (int32_t *)at, *row1 = (int32_t *)(at + row), *twin = (int32_t *)(at + 2 * row), *pair_of = (int32_t *)(at + 3 * row),
         *sel = (int32_t *)(at + 4 * row);
    const size_t lists = list_bytes(E);
    // (the distances go straight to where the evaluation wants them)
    char *distances = at + lists + (training ? train_distances_at(N, E, w->head_width, w->num_blocks) : 0);
    int rc = mlcgb_graph_finish(pos, MLCGB_F32, ptr, N, B, r, 0, nullptr, nullptr, g, G.graph, offsets, E, nullptr, distances, nullptr, row0, row1, twin, sel,
                                pair_of, host[3] != 0, status, stream);
    if (rc) return rc;
    ChainScope chain;
    if (training)
        rc = precision ? MLCGB_E_ARG
                       : schnet_train_forward(pos, types, ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, E / 2, rbf, conv_cutoff_kind, conv_lower, conv_upper,
                                              w, negate, true, at + lists, workspace_bytes - lists, energy, grad_pos, status, stream);
    else
        rc = schnet_eval_distances(pos, types, ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, rbf, conv_cutoff_kind, conv_lower, conv_upper, w, precision,
                                   at + lists, workspace_bytes - lists, energy, grad_pos, negate ? -1.f : 1.f, status, stream);
    if (rc == MLCGB_OK) host[4] = MLCGB_EVALUATE_DONE;
    return rc;
}

void mlcgb_schnet_evaluate_lists(int64_t N, int64_t B, int64_t E, int64_t *at) {
    const GraphPart G = graph_part(N, B);
    at[0] = (int64_t)G.ptr;
    at[1] = (int64_t)G.offsets;
    for (int i = 0; i < 5; i++) at[2 + i] = (int64_t)(i * up256((size_t)E * 4));
    at[7] = (int64_t)list_bytes(E);
}

}  // extern "C"

// Energies and forces from positions in one library call: radius graph with its pair plan, then the SchNet evaluation, with the edge
// count handed to the host in between by the graph's mapped line.  The lists never leave the workspace, so nothing is allocated and
// no caller's code runs between the count's arrival and the launches that need it: for a single small structure that gap was as
// long as all of its kernels (127 -> 99 us per evaluation of 73 beads).
#include "common.cuh"

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

}  // namespace

extern "C" {

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
    if (host[4] != MLCGB_EVALUATE_MORE) {
        if (int rc = mlcgb_graph_begin(pos, MLCGB_F32, n_atoms, ptr, N, B, r, max_nn, 0, MLCGB_RULE_CLUSTER, nullptr, nullptr, g, G.graph, offsets,
                                       pending_status, host, stream))
            return rc;
    }
    const int64_t E = host[0];
    host[4] = MLCGB_EVALUATE_NO_PLAN;
    if ((host[1] & kTruncated) || E <= 0 || (E & 1) || E >= (int64_t)1 << 31) return MLCGB_OK;
    host[4] = MLCGB_EVALUATE_MORE;
    if (!workspace || workspace_bytes < mlcgb_schnet_evaluate_workspace_bytes(N, B, E, rbf->num_rbf, w, training)) return MLCGB_OK;
    if ((uintptr_t)workspace & 255) return MLCGB_E_ARG;
    const size_t row = up256((size_t)E * 4);
    char *at = (char *)workspace;
    auto *row0 = (int32_t *)at, *row1 = (int32_t *)(at + row), *twin = (int32_t *)(at + 2 * row), *pair_of = (int32_t *)(at + 3 * row),
         *sel = (int32_t *)(at + 4 * row);
    const size_t lists = list_bytes(E);
    int rc = mlcgb_graph_finish(pos, MLCGB_F32, ptr, N, B, r, 0, nullptr, nullptr, g, G.graph, offsets, E, nullptr, nullptr, nullptr, row0, row1, twin, sel,
                                pair_of, host[3] != 0, status, stream);
    if (rc) return rc;
    ChainScope chain;
    if (training)
        rc = precision ? MLCGB_E_ARG
                       : mlcgb_schnet_train_forward(pos, types, ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, E / 2, rbf, conv_cutoff_kind,
                                                    conv_lower, conv_upper, w, negate, at + lists, workspace_bytes - lists, energy, grad_pos, status, stream);
    else
        rc = (negate ? mlcgb_schnet_energy_forces : mlcgb_schnet_eval_counted)(pos, types, ptr, N, B, row0, row1, offsets, sel, pair_of, twin, E, E / 2,
                                                                               nullptr, rbf, conv_cutoff_kind, conv_lower, conv_upper, w, precision, at + lists,
                                                                               workspace_bytes - lists, energy, grad_pos, status, stream);
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

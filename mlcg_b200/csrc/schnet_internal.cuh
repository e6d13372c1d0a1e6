// Pieces of the whole-model sequences (interaction.cu, train.cu) that live in files of their own.
#pragma once
#include "common.cuh"
#include "small_graph.cuh"

namespace mlcgb {

constexpr int kMaxBlocks = 10;             // interaction blocks of the whole-model calls that run several blocks per launch

// rows kept per block where all blocks' filter rows share one matrix: whole 128-row tiles
inline int64_t padded_rows(int64_t P) { return (P + 127) / 128 * 128; }

// Weights as the tensor-core kernels hold them: fp16 pairs in the layout of a 128-row operand tile (high part, low part), 64 KB each.
// Made once per evaluation or step beside the embedding (interaction.cu); a kernel then fetches them with bulk copies that arrive under
// its first tile instead of 64 KB of loads, conversions and stores per weight in every one of its CTAs.
constexpr int64_t kWeightImage = 65536;
enum { kLin1 = 0, kLin2 = 1, kLin = 2 };   // image 3 l + one of these: of block l; 3 L: the output network's first layer; 3 L + 1 + 2 l: filter_w1, filter_w2
constexpr int kMaxImages = 5 * kMaxBlocks + 1;
struct WeightImages {
    const float *src[kMaxImages];
    int16_t rows[kMaxImages], cols[kMaxImages];
    int n, first_filter;                   // (of the filters' weights; every other one from there on is a filter_w1)
    uint8_t *dst;
};
inline int64_t weight_images_floats(int64_t num_blocks) { return (5 * num_blocks + 1) * (kWeightImage / 4); }
// embedding rows of all nodes and, unless images is NULL (16-byte aligned, all widths 128 but the output network's), the weight images,
// the filter networks' (of num_rbf basis functions) too unless num_rbf is 0
int embedding_launch(const mlcgb_schnet_weights *w, const int64_t *types, int64_t N, float *x, void *images, int num_rbf, int32_t *status, cudaStream_t st);
// gemm_tc.cu: mlcgb_gemm_tc_fused, _chain2 and _chain2_tangent with the images of their weights (NULL: converted by the kernel)
int gemm_fused(int mode, const void *A, const void *B, const void *bias, const void *aux, int epilogue, int64_t M, int64_t N, int64_t K, void *C,
               const uint8_t *image, int32_t *status, void *stream);
// A third layer on the same tile (needs the images of all three).  Forward kinds: behind the two, out[M][width] = C image^T + bias, through
// tanh if wanted, and dot[M] = out . dot_w + dot_b (the output network's last layer) where dot is given.  Backward kinds: in front of them, out = A image + res, A[M][width] replaced by vec (1 - A^2) where vec is given.
struct ChainLink {
    const uint8_t *image;
    const float *bias, *vec, *res;         // NULL: none
    float *out;
    int width, tanh;
    const float *dot_w, *dot_b;            // dot_b NULL: zero
    float *dot;
};
int gemm_chain2(int backward, const void *A, const void *Wa, const void *ba, const void *Wb, const void *bb, const void *aux, int64_t M, void *mid_out,
                void *C, const uint8_t *image_a, const uint8_t *image_b, const ChainLink *link, int32_t *status, void *stream);
int gemm_chain2_tangent(int reverse, const void *A, const void *Wa, const void *Wb, const void *a, const void *gu, const void *aux, int64_t M, void *q,
                        void *mid_out, void *C, const uint8_t *image_a, const uint8_t *image_b, const ChainLink *link, int32_t *status, void *stream);

// filter_vd.cu: filter rows and their derivatives of `num_blocks` blocks in one launch.  Block l's rows start at row
// l * padded_rows(P) of W and Wd, its kept rows (or NULL) at l * mlcgb_filter_hidden_bytes(P) of hs and zs, its zmax at l.
int filter_vd_blocks(const float *d, int64_t P, const int64_t *rows_dev, const int32_t *sel, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind,
                     double conv_lower, double conv_upper, const mlcgb_schnet_block *blocks, int64_t num_blocks, int precision, float *W, float *Wd,
                     float *hs, float *zs, float *zmax, const uint8_t *images, int32_t *status, cudaStream_t st);    // images: of blocks[0], NULL: none

// filter_wgrad.cu: the weight gradients of all of them in one launch; xl, xt, gagg, agb per block
struct FilterGradBlock {
    const float *A2, *xl, *xt, *gagg, *agb;
};
int filter_wgrad_blocks(const float *d, const float *dd, int64_t P, const int32_t *sel, const int32_t *row0, const int32_t *row1,
                        const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper, const FilterGradBlock *blocks,
                        int64_t num_blocks, const float *hs, const float *zs, const float *zmax, float *partial, int32_t *status, cudaStream_t st);
int filter_wgrad_parts(int64_t P, int64_t num_blocks);      // partial sums per block

// small_route.cu: see there.  All widths 128 but the output network's.
// 148 SMs x 16 rows: two passes of eight rows per SM.  Chains of 100 beads, three blocks, 12 A, us, this route : the tensor-core
// kernels, an evaluation and the kernels of a force-matching step,
//   beads       1200       2000       2400       3200       4000
//   evaluation  146 : 198  164 : 209  217 : 224  258 : 250  322 : 258
//   step        407 : 525  493 : 566  570 : 590  660 : 647  803 : 696
// The line lies where a third pass begins; the routes meet at about 2800 beads.
constexpr int64_t kSmallNodes = 2368;
// The chain of small_route.cu takes a batch (of a network whose widths are 128).  It brings its matrices in pieces of 16 bytes, so they have to lie on
// such boundaries; weights that do not (parts of a larger buffer, say) take the kernels of larger batches, which convert them value by value.
inline bool small_route(int64_t N, const mlcgb_schnet_weights *w) {
    if (N > kSmallNodes || w->num_blocks < 1 || w->num_blocks > kMaxBlocks || !w->blocks) return false;
    uintptr_t at = (uintptr_t)w->head_W;
    for (int64_t l = 0; l < w->num_blocks; l++) at |= (uintptr_t)w->blocks[l].lin1_w | (uintptr_t)w->blocks[l].lin2_w | (uintptr_t)w->blocks[l].lin_w;
    return (at & 15) == 0;
}
struct SmallForward {                      // per node unless said otherwise; NULL: not wanted
    const float *pos;
    const int64_t *types;
    const int32_t *row0, *row1, *pair_of;
    const int64_t *ptr;
    int64_t N, E, B;
    const mlcgb_schnet_weights *w;
    float *d;                              // [E]
    float *W, *Wd;                         // [L][padded P][128]
    int64_t wstride;                       // floats per block
    float *x[kMaxBlocks + 1], *xl[kMaxBlocks], *agg[kMaxBlocks], *a[kMaxBlocks], *gu[kMaxBlocks], *gagg[kMaxBlocks], *gxl[kMaxBlocks], *g[kMaxBlocks];
    float *ah, *en, *s;                    // s: [E] force-pass dot products
    int want_grad;
    int32_t *status;
};
// The radius graph and pair plan of up to kMaskNodes beads into lists of `capacity` edges, made in front of an evaluation without the
// host: more edges, an odd number of them or a list cut short leave a graph without edges, which is reported.
struct SmallGraph {
    const int64_t *sizes;                  // [B], or NULL: ptr is read
    int64_t *ptr;
    double r;
    int64_t max_nn, capacity;
    uint2 *masks;                          // [N][(N + 31) / 32]
    int32_t *deg, *upper;                  // [N]
    int32_t *row1, *twin, *pair_of;        // [capacity]
    float *pair_d;                         // [capacity / 2]: distances of the pairs, which the filters read in order
    int64_t *offsets, *counts;             // [N + 1]; {edges, pairs}
    Publish pub;                           // host NULL: reported in the evaluation's status word
};
inline size_t small_graph_scratch(int64_t N) { return (size_t)N * ((N + 31) / 32) * 8 + (size_t)N * 8 + 256; }
inline bool small_graph_ok(int64_t N, int64_t B, const mlcgb_schnet_weights *w) {
    return N > 0 && B > 0 && N <= kMaskNodes && B <= kMaskStructs && w->hidden == 128 && w->filters == 128 && w->conv_out == 128 && small_route(N, w);
}
int small_graph_start(const SmallForward &f, const SmallGraph &g, cudaStream_t st);    // graph, distances, embedding, lin1 of the first block
// interaction.cu: mlcgb_schnet_energy_forces / _eval_counted (grad_sign -1 / 1) behind it
int schnet_eval_small(const void *pos, const int64_t *types, int64_t N, int64_t B, const SmallGraph &g, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind,
                      double conv_lower, double conv_upper, const mlcgb_schnet_weights *w, int precision, void *workspace, size_t workspace_bytes,
                      void *energy, void *grad_pos, float grad_sign, int32_t *status, cudaStream_t st);
int small_start(const SmallForward &f, cudaStream_t st);    // distances, embedding, lin1 of the first block
int small_forward(const SmallForward &f, cudaStream_t st);  // the blocks, the output network and, if wanted, the force pass down to s of block 1
int small_finish(const SmallForward &f, const int32_t *twin, const int64_t *struct_ptr, float *energy, float *grad, float sign, cudaStream_t st);

struct SmallBackward {
    const float *dd, *gE;
    const int64_t *struct_ptr;
    float *xt[kMaxBlocks], *xlt[kMaxBlocks], *aggt[kMaxBlocks], *at[kMaxBlocks], *q[kMaxBlocks], *ub[kMaxBlocks], *agb[kMaxBlocks], *xlb[kMaxBlocks],
        *xb[kMaxBlocks + 1];               // xt[l], xb[l + 1]: of block l's output
    float *yb, *gy, *r;
};
int small_backward(const SmallForward &f, const SmallBackward &b, cudaStream_t st);

// The whole-model sequences on lists whose distances already lie in the workspace, at its start / at train_distances_at() bytes of it
// (mlcgb_schnet_energy_forces / _eval_counted with grad_sign -1 / 1, mlcgb_schnet_train_forward)
int schnet_eval_distances(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0, const int32_t *row1,
                          const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin, int64_t E, const mlcgb_rbf_spec *rbf,
                          int conv_cutoff_kind, double conv_lower, double conv_upper, const mlcgb_schnet_weights *w, int precision, void *workspace,
                          size_t workspace_bytes, void *energy, void *grad_pos, float grad_sign, int32_t *status, void *stream);
size_t train_distances_at(int64_t N, int64_t E, int64_t head_width, int64_t num_blocks);
int schnet_train_forward(const void *pos, const int64_t *types, const int64_t *struct_ptr, int64_t N, int64_t B, const int32_t *row0, const int32_t *row1,
                         const int64_t *offsets, const int32_t *sel, const int32_t *pair_of, const int32_t *twin, int64_t E, int64_t P, const mlcgb_rbf_spec *rbf,
                         int conv_cutoff_kind, double conv_lower, double conv_upper, const mlcgb_schnet_weights *w, int negate, bool have_distances,
                         void *workspace, size_t workspace_bytes, void *energy, void *grad_pos, int32_t *status, void *stream);

// edge_vd.cu: the last dot products of a force pass, one per pair: sp[p] = sum_f (x[i] a[j] + x[j] a[i]) W'[p] + s[(i,j)] + s[(j,i)], the
// sums of the blocks before (NULL: none)
int seg_pair_dot(const float *a, const float *x, const float *Wd, const int64_t *ptr, const int32_t *nbr, const int32_t *pair_of, const int32_t *twin,
                 const float *s, int64_t N, float *sp, cudaStream_t st);
// edge_ops.cu: position gradients (times sign: -1 gives forces) from the energy's derivative with respect to each pair's distance, and
// energies, in one launch
int finish_launch(const float *pos, const float *pair_g, const float *d, const int32_t *row1, const int64_t *ptr, const int32_t *pair_of, int64_t N, float *gpos,
                  float sign, const float *en, const int64_t *struct_ptr, int64_t B, float *energy, cudaStream_t st);

}  // namespace mlcgb

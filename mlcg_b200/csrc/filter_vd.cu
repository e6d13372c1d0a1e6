// Filter rows together with their distance derivative, one launch per interaction block:
//
//   W [p,:] = (h A2^T) C(d_p)                              h  = tanh(phi(d_p) A1^T + b1)      src/mlcg/nn/schnet.py:340-341
//   W'[p,:] = (C (1 - h^2) z' + C' h) A2^T                 z' = phi'(d_p) A1^T                  (dW/dd)
//
// A filter depends on the pair's distance alone, so with W' at hand the force pass is a dot product per edge inside the
// aggregation (edge_vd.cu), and a tangent of the filters along a change of the distances is W' times that change: neither runs
// the filter network again.  Same machinery as the forward in filter_tc.cu: persistent CTA per SM, 128-pair tiles, 16 compute
// warps (thread = one row x 32 columns) and a warp that only issues the tensor-core instructions.  A tile makes two passes through
// the two GEMMs, values and derivatives, interleaved so that each GEMM runs under element-wise work that does not wait for it:
//   warps   tanh(j)  store W'(j-1)  phi'(j)  store W(j)  phi(j+1)  derivative operand(j)
//   MMA     2d(j-1)  2v(j) ------------------  1d(j) ------------  1v(j+1) ------------
// Tensor memory holds four blocks of 128 columns; three of them change roles from tile to tile:
//   V  phi, then h, then C (1 - h^2) z' + C' h (in place: a thread rewrites its own columns)   -> next tile's Q
//   A  z, then W/C                                                                             -> next tile's V
//   Q  phi'                                                                                    -> next tile's A
//   R  z', then W'
// h for the derivative's second operand is read back from V (fp16 pairs: 22 bits of a value below one; the bf16 mode keeps it as
// fp32 in shared memory).
// Bound by instruction issue and latency at one CTA per SM.  With the four GEMMs of a tile in turn on two accumulators every pass
// waited for the one before: three launches over 553 k pairs took 757 us, like this 684, and with the arithmetic between the GEMMs
// in pairs (two operations an instruction) 662 (bf16: 470, 441), without the part of the basis that is zero and with the per-row values
// made where a product is waited for 624 (bf16: 410).  A tile takes 12 100 cycles: tanh 2100, the two stores 1700, phi' 1300 and phi
// 1450, the derivative operand 2000, waiting for products and other warps 2800; the products themselves 4600.
// Replaces the backward GEMM kernel in the force pass (filter_tc.cu): per block, forward + backward took 0.16 + 0.25 ms.
#include "filter_common.cuh"
#include "schnet_internal.cuh"

namespace mlcgb {

struct FilterVdBlock {
    const float *A1, *b1, *A2;
};
struct FilterVdParams {
    FilterFwdParams f;   // f.W: values; f.H: hidden rows kept for the weight gradients, or NULL
    FilterVdBlock blk[kMaxBlocks];       // weights of interaction block blockIdx.y (the filters of all blocks depend on the distances alone)
    int64_t block_rows, block_hidden;    // rows / kept floats between the blocks' results
    float *Wd;           // [E][kF] derivatives
    float *Zd;           // z' kept for the weight gradients in hidden_offset() order, or NULL
    const uint8_t *images;               // of the blocks' weights, two each (schnet_internal.cuh), or NULL
    float *zmax;         // with Zd: largest |z'| (to be zero before; non-negative floats order like their bits)
};

// per-row values of six tiles behind the shared layout of the filter kernels
constexpr int kRowSlots = 6, kRowBytes = kRowSlots * 4096;
template <bool SPLIT> constexpr int kVdSmem = FilterSmem<SPLIT>::kExtra + kRowBytes + (SPLIT ? 0 : 32768) + 1024;

template <bool SPLIT, bool APART>
__global__ void __launch_bounds__(kTcThreads + 32, 1)
filter_vd_kernel(FilterVdParams q, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap dmap) {
    using namespace tc;
    using L = FilterSmem<SPLIT>;
    FilterFwdParams p = q.f;
    p.A1 = q.blk[blockIdx.y].A1;
    p.b1 = q.blk[blockIdx.y].b1;
    p.A2 = q.blk[blockIdx.y].A2;
    // APART: a launch with few tiles gives each to two CTAs (blockIdx.z), one for the values and one for the derivatives, the first steps
    // done in both: a chain of two GEMMs each instead of four in turn.
    const bool values = !APART || blockIdx.z == 0, derivatives = !APART || blockIdx.z == 1;
    float4 *const h_keep = p.H && values ? reinterpret_cast<float4 *>(p.H + blockIdx.y * q.block_hidden) : nullptr;
    float4 *const z_keep = q.Zd && derivatives ? reinterpret_cast<float4 *>(q.Zd + blockIdx.y * q.block_hidden) : nullptr;
    const int row_base = (int)(blockIdx.y * q.block_rows);
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *stage = SPLIT ? smem + L::kA : smem + L::kStage;
    const float *s_b1 = reinterpret_cast<const float *>(smem + L::kMisc + L::kBias);
    const float2 *s_tab = reinterpret_cast<const float2 *>(smem + L::kMisc + L::kTable);
    float *s_red = reinterpret_cast<float *>(smem + L::kMisc + L::kRed);
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(smem + L::kMisc + L::kBar);
    // GEMM 1 / 2 of the values / derivatives: operand ready (one arrival per compute warp), GEMM complete
    const uint32_t bars = smem_u32(smem + L::kMisc + L::kBar + 64);
    const uint32_t r1v = bars, r2v = bars + 8, r1d = bars + 16, r2d = bars + 24, c1v = bars + 32, c2v = bars + 40, c1d = bars + 48, c2d = bars + 56;
    int *s_err = reinterpret_cast<int *>(reinterpret_cast<uint32_t *>(s_bar + 1) + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & 127, qt = (tid >> 7) & 3, col0 = qt * 32;
    const int R = p.rbf.R;
    const int Kpad1 = R <= 64 ? 64 : 128;
    const float wscale = SPLIT ? kWScale : 1.f;
    const float unscale = 1.f / wscale;

    uint8_t *s_live = smem + L::kMisc + L::kRed2;      // [tile & 1][16 warps]: the warp's part of the tile's phi is not all zero

    const uint32_t wbar = bars + 64;                   // both weights' images have arrived
    const bool images = SPLIT && q.images;
    if (images && tid == 0) {
        mbar_init(wbar, 2);
        const uint8_t *image = q.images + blockIdx.y * 2 * kWeightImage;
        fetch_image(smem_u32(smem + L::kB1), image, wbar);
        fetch_image(smem_u32(smem + L::kB2), image + kWeightImage, wbar);
    }
    const uint32_t tmem = filter_setup<SPLIT>(p, smem, Kpad1, 512, images);
    if (tid == 0) {
        for (int i = 0; i < 4; i++) {
            mbar_init(bars + 8 * i, kTcThreads / 32);
            mbar_init(bars + 32 + 8 * i, 1);
        }
    }
    // steepest basis function: |d g_k / dt| <= sqrt(2 ln2 w_k / e) where g_k = 2^(-w_k (t - c_k)^2).  (A lane looks at its share of the
    // table here and below: every thread going through all of it took 4 of the 8-10 us of a CTA's set-up.)
    const float slope = 0.7142f * sqrtf(table_max_width(s_tab, R, lane));
    // Where this quarter's functions are not zero as operands.  At w (t - c)^2 > 36 a function is below 2^-36: zero as a pair of fp16 (below
    // 2^-25), and so is its derivative on the scale of its row (below 16 (z / 0.6065 + 1) 2^-36 < 2^-28 at z = 7.1 widths).  Exp-normal
    // functions crowd the short distances that no bead comes to: of 128 over 15 A those beyond the 45th are zero at 4 A and more,
    // over 10 A those beyond the 29th.  A warp whose 32 rows are all outside stores zeros, and the first GEMMs leave a quarter of K out that
    // is zero in the whole tile: the same sums, bit by bit, in the mode of fp16 pairs.  The operands of the bf16 mode
    // reach further down: there the values left out are below 2^-36 where its rounding of the others is 2^-9 of them.  A weight that is not a
    // number is so in its whole row (spread_nan) and reaches the sums through the quarter that is always there.
    float near_lo = INFINITY, near_hi = -INFINITY;
    if (col0 + lane < R) {
        const float2 cw = s_tab[col0 + lane];
        const float reach = cw.y > 0.f ? sqrtf(36.f / cw.y) : INFINITY;
        near_lo = fminf(near_lo, cw.x - reach);
        near_hi = fmaxf(near_hi, cw.x + reach);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        near_lo = fminf(near_lo, __shfl_xor_sync(0xffffffffu, near_lo, o));
        near_hi = fmaxf(near_hi, __shfl_xor_sync(0xffffffffu, near_hi, o));
    }
    __syncthreads();
    pdl_wait();                      // set-up done (weights only); from here on the distances of the previous kernels are read
    pdl_launch_dependents();
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t t_lane = tmem + lane_off;
    const uint32_t b1_hi = smem_u32(smem + L::kB1), b1_lo = b1_hi + 32768, b2_hi = smem_u32(smem + L::kB2), b2_lo = b2_hi + 32768;
    bool failed = false;

    const int64_t nE = live_rows(p);
    const int64_t ntiles = (nE + kRows - 1) / kRows;
    const int64_t first = blockIdx.x, step = gridDim.x;
    const int64_t n_local = first < ntiles ? (ntiles - first + step - 1) / step : 0;
    // a wait that has run out is not repeated: the block runs on, so that every barrier of the schedule is still reached by
    // everybody, and reports the failure at the end
    auto await = [&](uint32_t bar, uint32_t parity) {
        if (!failed && !mbar_wait(bar, parity)) failed = true;
        tc_fence_after();
    };
    if (warp == kTcThreads / 32) {
        const bool elected = elect_one();
        // ---- the issuing warp
        const auto gemm = [&](uint32_t ready, uint32_t par, uint32_t d, uint32_t ta, uint32_t b_hi, uint32_t b_lo, int ksteps, uint32_t done) {
            await(ready, par);
            if (elected) {
                issue_gemm_ts<SPLIT>(d, ta, b_hi, b_lo, ksteps, 0, 128);
                mma_commit(done);
            }
            __syncwarp();
        };
        const auto gemm1 = [&](uint32_t d, uint32_t ta, uint32_t quarters, uint32_t done) {
            if (elected) {
                issue_gemm_ts_quarters<SPLIT>(d, ta, b1_hi, b1_lo, quarters ? quarters : 1u);
                mma_commit(done);
            }
            __syncwarp();
        };
        const auto live_quarters = [&](uint32_t parity) {      // of the tile whose phi has been signalled
            const unsigned w = __ballot_sync(0xffffffffu, lane < 16 && *reinterpret_cast<volatile uint8_t *>(s_live + parity * 16 + lane));
            return (w & 0xfu ? 1u : 0u) | (w & 0xf0u ? 2u : 0u) | (w & 0xf00u ? 4u : 0u) | (w & 0xf000u ? 8u : 0u);
        };
        uint32_t tV = tmem, tA = tmem + 128, tQ = tmem + 256;
        const uint32_t tR = tmem + 384;
        uint32_t quarters = 0, next = 0;
        if (images) await(wbar, 0);                    // (whether or not there is a tile: the block outlives its copies)
        if (n_local > 0) {
            await(r1v, 0);
            next = live_quarters(0);
            gemm1(tA, tV, next, c1v);
        }
        for (int64_t j = 0; j < n_local; j++) {
            const uint32_t par = (uint32_t)(j & 1);
            quarters = next;
            if (values) gemm(r2v, par, tA, tV, b2_hi, b2_lo, kF / 16, c2v);
            if (!derivatives) break;                   // (a tile of its own)
            await(r1d, par);
            gemm1(tR, tQ, quarters, c1d);
            if (j + 1 < n_local) {
                await(c1d, par);                       // phi' has been read: its block takes the next tile's values
                await(r1v, par ^ 1);
                next = live_quarters(par ^ 1);
                gemm1(tQ, tA, next, c1v);
            }
            gemm(r2d, par, tR, tV, b2_hi, b2_lo, kF / 16, c2d);
            const uint32_t old = tV;
            tV = tA;
            tA = tQ;
            tQ = old;
        }
    } else {
        uint32_t tV = t_lane, tA = t_lane + 128, tQ = t_lane + 256;
        const uint32_t tR = t_lane + 384;
        // fp32 hidden values of the bf16 mode (thread-private): chunks 0..3 in the operand region that it leaves free, 4..7 behind the rows
        float4 *const h_lo = reinterpret_cast<float4 *>(smem + L::kA) + tid, *const h_hi = reinterpret_cast<float4 *>(smem + L::kExtra + kRowBytes) + tid;
        const bool same_env = p.conv.cutoff_kind == p.rbf.cutoff_kind && p.conv.lower == p.rbf.lower && p.conv.upper == p.rbf.upper;
        // per-row values of a tile.  The four threads of a row (one per quarter) each work them out for one of the next four tiles and
        // share them: every thread for every tile took a fifth of the kernel's instructions.  That is done in the third of four tiles, where
        // the second value GEMM would be waited for, into slots that nobody reads any more by then (six, and the barrier before the
        // tile's next operand in between); the edge and its distance are fetched two tiles ahead of their use each.
        struct Scalars { float t, dt, e0, e1, c0, c1, s1, l2e; };
        auto scalars = [&](float de) {
            Scalars s;
            edge_arg(de, p.rbf, s.t, s.dt);
            const Jet<float, 1> env = envelope_jet<float, 1>(de, p.rbf);
            s.e0 = env.c[0];
            s.e1 = env.c[1];
            s.c0 = s.e0;
            s.c1 = s.e1;
            if (!same_env) {
                const Jet<float, 1> cj = envelope_jet<float, 1>(de, p.conv);
                s.c0 = cj.c[0];
                s.c1 = cj.c[1];
            }
            // power of two for the phi' operand, from a bound on the row's largest entry
            s.s1 = SPLIT ? row_scale(fmaf(s.e0 * fabsf(s.dt), slope, fabsf(s.e1))) : 1.f;
            s.l2e = log2f(s.e0);
            return s;
        };
        float4 *const s_rows = reinterpret_cast<float4 *>(smem + L::kExtra);       // [6 tiles][2][128]
        auto row_group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(2 + (warp & 3)) : "memory"); };
        // of the tile that this thread prepares next: its edge (-1: no row), then the edge's distance
        auto fetch_edge = [&](int64_t n) {
            const int64_t k = (first + (n + qt) * step) * kRows + r;
            return k < nE ? (p.sel ? __ldg(p.sel + k) : (int32_t)k) : -1;       // (lists have fewer than 2^31 edges)
        };
        auto fetch_d = [&](int32_t edge) { return edge < 0 ? 1.f : __ldg(p.d + edge); };
        auto prepare = [&](int64_t n, float d) {                     // tile n + qt of this block
            const Scalars s = scalars(d);
            float4 *row = s_rows + (int)((uint32_t)(n + qt) % (uint32_t)kRowSlots) * 256 + r;
            row[0] = make_float4(s.t, s.dt, s.e0, s.e1);
            row[128] = make_float4(s.c0, s.c1, s.s1, s.l2e);
        };
        auto read_scalars = [&](int64_t n) {
            const float4 *row = s_rows + (int)((uint32_t)n % (uint32_t)kRowSlots) * 256 + r;
            const float4 a = row[0], b = row[128];
            return Scalars{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        };
        auto signal = [&](uint32_t bar) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        auto store_zeros = [&](uint32_t ta) {
            tmem_zero16(ta + (col0 >> 1));
            if (SPLIT) tmem_zero16(ta + 64 + (col0 >> 1));
        };
        // (rows past the end count as far away; a distance that is not a number does not)
        auto basis = [&](const Scalars &s, uint32_t ta, int64_t n, int64_t tile) {
            const bool live = __any_sync(0xffffffffu, !(s.t <= near_lo) && !(s.t >= near_hi) && tile * kRows + r < nE);
            if (lane == 0) s_live[(n & 1) * 16 + warp] = live;
            if (!live) {
                if (col0 < Kpad1) store_zeros(ta);
            } else if (col0 < Kpad1) {
                const float l2a = s.l2e;
                float x[32];
                const float4 *tab4 = reinterpret_cast<const float4 *>(s_tab + col0);   // two (centre, width) pairs per 128-bit read
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float4 cw = tab4[j];
                    const float2 u = sub2(both(s.t), make_float2(cw.x, cw.z)), e = fma2(mul2(make_float2(-cw.y, -cw.w), u), u, both(l2a));
                    x[2 * j] = ex2_fast(e.x);
                    x[2 * j + 1] = ex2_fast(e.y);
                }
                store_a_tmem<SPLIT, kPackAsIs>(ta, col0, x, 1.f);
            }
            tmem_wait_st();
            return live;
        };
        // phi'_k = g_k (env' - env 2 ln2 w_k (t - c_k) t'); columns at or beyond R: exactly 0
        auto basis_derivative = [&](const Scalars &s, bool live) {
            if (!live) {
                if (col0 < Kpad1) store_zeros(tQ);
            } else if (col0 < Kpad1) {
                const float m2 = -2.f * kLn2 * s.dt * s.e0;
                float x[32];
                const float4 *tab4 = reinterpret_cast<const float4 *>(s_tab + col0);
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float4 cw = tab4[j];
                    // (the table's widths are taken with their sign turned: w' = -w)
                    const float2 u = sub2(both(s.t), make_float2(cw.x, cw.z)), wu = mul2(make_float2(-cw.y, -cw.w), u), e = mul2(wu, u);
                    const float2 f = mul2(make_float2(ex2_fast(e.x), ex2_fast(e.y)), fma2(both(-m2), wu, both(s.e1)));
                    x[2 * j] = f.x;
                    x[2 * j + 1] = f.y;
                }
                store_a_tmem<SPLIT, kPackPairs>(tQ, col0, x, s.s1);
            }
            tmem_wait_st();
        };
        // accumulator x (this row's factor) -> stage -> rows of the mapped matrix, by the copy engine.  A warp stages and stores its own box of
        // 32 rows x 32 columns: no warp waits for another one here (one box of 128 rows for the block took two block-wide barriers)
        // (a tile of its own: by the lanes of the warp, which need not stay until the copy engine is done, nor the host describe the matrix)
        auto store_rows = [&](const CUtensorMap *map, float *plain, int64_t tile, uint32_t acc, float f) {
            float v[32];
            tmem_ld32(acc + col0, v);
            if (lane == 0) bulk_wait_read<0>();                     // the copy before has read the stage
            __syncwarp();
#pragma unroll
            for (int w = 0; w < 8; w++) {
                const float2 lo = mul2(make_float2(v[4 * w], v[4 * w + 1]), both(f)), hi = mul2(make_float2(v[4 * w + 2], v[4 * w + 3]), both(f));
                *box_chunk(stage, qt, r, w) = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
            const int64_t row = tile * kRows + 32 * (warp & 3);
            if (APART) {
                __syncwarp();
                float4 *const to = reinterpret_cast<float4 *>(plain + (row_base + row) * kF + col0) + (lane & 7);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int k = 4 * i + (lane >> 3);
                    if (row + k < nE) to[k * (kF / 4)] = *box_chunk(stage, qt, 32 * (warp & 3) + k, lane & 7);
                }
                return;
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0 && row < nE) {
                tensor_store_box(map, col0, row_base + (int)row, stage + qt * 16384 + (warp & 3) * 4096);
                bulk_commit();
            }
        };

        float zmax = 0.f;
        int32_t edge_ahead = -1;
        float d_ahead = 1.f;
        bool live = false, live_next = false;                       // this warp's part of phi, this tile and the next
        float f_prev = 0.f;                                         // factor of the derivative rows whose GEMM is in flight
        if (n_local > 0) {
            prepare(0, fetch_d(fetch_edge(0)));
            edge_ahead = fetch_edge(4);
            row_group_sync();
            live_next = basis(read_scalars(0), tV, 0, first);
            signal(r1v);
            if (APART && derivatives) {
                basis_derivative(read_scalars(0), live_next);
                signal(r1d);
            }
        }
        int64_t tile = first;
        for (int64_t n = 0; n < n_local; n++, tile += step) {
            const uint32_t par = (uint32_t)(n & 1);
            live = live_next;
            if ((n & 3) == 0) d_ahead = fetch_d(edge_ahead);
            // ---- hidden layer
            await(c1v, par);
            {
                float v[32];
                tmem_ld32(tA + col0, v);
                tanh_row32<SPLIT>(v, s_b1 + kF, col0, unscale * (2.f * kLog2e));
                store_a_tmem<SPLIT, kPackAsIs>(tV, col0, v, 1.f);
                if (!SPLIT) {
#pragma unroll
                    for (int j = 0; j < 8; j++) (j < 4 ? h_lo : h_hi)[(j & 3) * kTcThreads] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
                if (h_keep) {                                        // (rows past the end hold finite filler)
#pragma unroll
                    for (int j = 0; j < 8; j++) __stcs(h_keep + hidden_offset(tile, qt, j, r), make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
                }
                tmem_wait_st();
            }
            if (values) signal(r2v);
            if (n > 0) {
                await(c2d, par ^ 1);
                store_rows(&dmap, q.Wd, tile - step, tR, f_prev);
            }
            const Scalars sc = read_scalars(n);
            if (!APART) {
                basis_derivative(sc, live);
                signal(r1d);
            }
            if ((n & 3) == 2 && n + 2 < n_local) {
                prepare(n + 2, d_ahead);
                edge_ahead = fetch_edge(n + 6);
            }
            if (values) {
                await(c2v, par);
                store_rows(&wmap, p.W, tile, tA, sc.c0 * unscale);
                if (!derivatives) break;
            }
            if (n + 1 < n_local) {
                // (the next tile's operand overwrites the accumulator just read: by all four quarters of the row)
                tc_fence_before();
                row_group_sync();
                tc_fence_after();
                live_next = basis(read_scalars(n + 1), tA, n + 1, tile + step);
                signal(r1v);
            }
            // ---- second operand of the derivatives, in place of h
            await(c1d, par);
            {
                float v[32];
                float rmax = 0.f;
                const float u1 = unscale / sc.s1;
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    float z[16], h[16];
                    tmem_ld16(tR + col0 + half * 16, z);
                    if (SPLIT) {
                        float hi[8], lo[8];
                        tmem_ld8(tV + (col0 >> 1) + half * 8, hi);
                        tmem_ld8(tV + 64 + (col0 >> 1) + half * 8, lo);
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const uint32_t a = __float_as_uint(hi[i]), b = __float_as_uint(lo[i]);
                            const float2 fa = __half22float2(*reinterpret_cast<const __half2 *>(&a)), fb = __half22float2(*reinterpret_cast<const __half2 *>(&b));
                            const float2 hh = add2(fa, fb);
                            h[2 * i] = hh.x;
                            h[2 * i + 1] = hh.y;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float4 x = (half ? h_hi : h_lo)[i * kTcThreads];
                            h[4 * i] = x.x; h[4 * i + 1] = x.y; h[4 * i + 2] = x.z; h[4 * i + 3] = x.w;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float2 z2 = mul2(make_float2(z[i], z[i + 1]), both(u1)), h2 = make_float2(h[i], h[i + 1]);
                        z[i] = z2.x;
                        z[i + 1] = z2.y;
                        const float2 x = fma2(mul2(both(sc.c0), z2), fma2(make_float2(-h2.x, -h2.y), h2, both(1.f)), mul2(both(sc.c1), h2));
                        v[half * 16 + i] = x.x;
                        v[half * 16 + i + 1] = x.y;
                        rmax = fmaxf(rmax, fmaxf(fabsf(x.x), fabsf(x.y)));
                    }
                    if (z_keep) {
#pragma unroll
                        for (int i = 0; i < 16; i++) zmax = fmaxf(zmax, fabsf(z[i]));
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            __stcs(z_keep + hidden_offset(tile, qt, half * 4 + j, r), make_float4(z[4 * j], z[4 * j + 1], z[4 * j + 2], z[4 * j + 3]));
                    }
                }
                float s2 = 1.f;
                if (SPLIT) {                                         // the row's four quarters: warps w, w+4, w+8, w+12
                    s_red[qt * 128 + r] = rmax;
                    row_group_sync();
                    s2 = row_scale(fmaxf(fmaxf(s_red[r], s_red[128 + r]), fmaxf(s_red[256 + r], s_red[384 + r])));
                }
                store_a_tmem<SPLIT, kPackPairs>(tV, col0, v, s2);
                tmem_wait_st();
                f_prev = unscale / s2;
            }
            signal(r2d);
            const uint32_t old = tV;
            tV = tA;
            tA = tQ;
            tQ = old;
        }
        if (n_local > 0 && derivatives) {
            await(c2d, (uint32_t)((n_local - 1) & 1));
            store_rows(&dmap, q.Wd, tile - step, tR, f_prev);
        }
        if (z_keep) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
            if (lane == 0) atomicMax(reinterpret_cast<int *>(q.zmax + blockIdx.y), __float_as_int(zmax));
        }
    }

    if (failed) s_err[0] = 1;
    bulk_wait_all();
    tc_fence_before();
    __syncthreads();
    if (s_err[0] && tid == 0) atomicOr(p.status, 8);
    if (warp == 0) tmem_free(tmem, 512);
}

template <bool SPLIT, bool APART>
static int filter_vd_launch(const FilterVdParams &q, int64_t ntiles, int64_t num_blocks, cudaStream_t st) {
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        if (cudaFuncSetAttribute(filter_vd_kernel<SPLIT, APART>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVdSmem<SPLIT>) != cudaSuccess) return check_launch();
        configured[dev] = true;
    }
    CUtensorMap wmap = {}, dmap = {};
    const int64_t rows = (num_blocks - 1) * q.block_rows + q.f.E;
    if (APART) {
        if (((uintptr_t)q.f.W | (uintptr_t)q.Wd) % 16) return MLCGB_E_LIMIT;
    } else if (!make_rows_map(&wmap, q.f.W, rows, kF, 32) || !make_rows_map(&dmap, q.Wd, rows, kF, 32)) {
        return MLCGB_E_LIMIT;
    }
    const int64_t per_block = num_blocks < kNumSM ? kNumSM / num_blocks : 1;
    const int grid = (int)(ntiles < per_block ? ntiles : per_block);
    launch_with_weights(filter_vd_kernel<SPLIT, APART>, dim3(grid, (unsigned)num_blocks, APART ? 2 : 1), dim3(kTcThreads + 32), kVdSmem<SPLIT>, st, q, wmap, dmap);
    return check_launch();
}

int filter_vd_blocks(const float *d, int64_t P, const int64_t *rows_dev, const int32_t *sel, const mlcgb_rbf_spec *rbf, int conv_cutoff_kind,
                     double conv_lower, double conv_upper, const mlcgb_schnet_block *blocks, int64_t num_blocks, int precision, float *W, float *Wd,
                     float *hs, float *zs, float *zmax, const uint8_t *images, int32_t *status, cudaStream_t st) {
    TimelineScope timeline_scope("filter_value_derivative", st);
    if (int rc = check_spec(rbf, 1)) return rc;
    if (P < 0 || !status || (precision != 0 && precision != 1) || (conv_cutoff_kind != 0 && conv_cutoff_kind != 1)) return MLCGB_E_ARG;
    if (rbf->num_rbf > 128 || num_blocks < 1 || num_blocks > kMaxBlocks) return MLCGB_E_LIMIT;
    if (P == 0) return MLCGB_OK;
    if (!d || !W || !Wd || (zs && !zmax)) return MLCGB_E_ARG;
    FilterVdParams q;
    for (int64_t l = 0; l < num_blocks; l++) {
        q.blk[l] = {(const float *)blocks[l].filter_w1, (const float *)blocks[l].filter_b1, (const float *)blocks[l].filter_w2};
        if (!q.blk[l].A1 || !q.blk[l].b1 || !q.blk[l].A2) return MLCGB_E_ARG;
    }
    q.f.d = d;
    q.f.E = P;
    q.f.rows_dev = rows_dev;
    q.f.sel = sel;
    q.f.twin = nullptr;
    q.f.rbf = to_dev<float>(rbf);
    q.f.conv = q.f.rbf;
    q.f.conv.cutoff_kind = conv_cutoff_kind;
    q.f.conv.lower = (float)conv_lower;
    q.f.conv.upper = (float)conv_upper;
    q.f.A1 = q.f.b1 = q.f.A2 = nullptr;
    q.f.W = W;
    q.f.H = hs;
    q.f.status = status;
    q.block_rows = padded_rows(P);
    q.block_hidden = (int64_t)(mlcgb_filter_hidden_bytes(P) / sizeof(float));
    q.Wd = Wd;
    q.Zd = zs;
    q.zmax = zmax;
    q.images = images;
    // two CTAs a tile while the chip holds them all (64 x 10 beads, two blocks: 51.9 -> 50.5 us an evaluation, 52.3 -> 50.3 replayed)
    const int64_t ntiles = (P + tc::kRows - 1) / tc::kRows;
    if (2 * ntiles * num_blocks <= kNumSM)
        return precision == 0 ? filter_vd_launch<true, true>(q, ntiles, num_blocks, st) : filter_vd_launch<false, true>(q, ntiles, num_blocks, st);
    return precision == 0 ? filter_vd_launch<true, false>(q, ntiles, num_blocks, st) : filter_vd_launch<false, false>(q, ntiles, num_blocks, st);
}

}  // namespace mlcgb

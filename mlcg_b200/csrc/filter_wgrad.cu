// Weight gradients of the filter network for one interaction block of a force-matching step.
//
// With S = sum_b gE_b E_b + (tangent of the energy along a displacement v of the positions), dL/dtheta = dS/dtheta.  Per pair p the
// block's aggregation sees the filter W and its tangent dd W' (dd: change of the distance along v), and hands back
//   w1 = d S/d(dd W') = gagg_i xl_j + gagg_j xl_i        w0 = dS/dW = agb_i xl_j + agb_j xl_i + gagg_i xt_j + gagg_j xt_i
// (xl, xt: lin1 features and their tangent; agb, gagg: gradients of the aggregate and of its tangent).  Through
//   W = C (h A2^T),  W' = (C h' + C' h) A2^T,  h = tanh(phi A1^T + b1),  h' = (1 - h^2) z',  z' = phi' A1^T
// with  o = C w0 + C' dd w1  and  od = dd C w1:
//   dA2 = o^T h + od^T h'          hb = o A2,  hd = od A2
//   zb = (1 - h^2) (hb - 2 h z' hd),  zd = (1 - h^2) hd
//   dA1 = zb^T phi + zd^T phi'     db1 = sum zb
// One persistent CTA per SM walks 128-pair tiles.  The four left operands of a tile pass through one shared-memory tile X and the
// right ones through Y (fp16 hi/lo pairs, 128-byte swizzle); X serves both as the K-major operand of hb / hd and, the same
// bytes read MN-major, as the transposed operand of the weight products, so nothing is transposed by hand.  The two weight
// gradients stay in tensor memory over all tiles of the CTA: left operands share one power-of-two scale per gradient, chosen from
// the first tile with room to grow (hi/lo keeps 2^-25 absolute, so 22 bits of every entry down to 2^-13 of the largest); when a
// tile outgrows it the sums so far are added to the CTA's partial and the scale is set anew.
// Bound by the conversions and the gathers of eight node rows per pair; before, every operand of these products went through
// HBM, each step an operator of its own.
#include "filter_common.cuh"
#include "schnet_internal.cuh"

namespace mlcgb {

struct FilterGradParams {
    const float *d, *dd;           // [E] distances and their tangents
    int64_t P;
    const int32_t *sel, *row0, *row1;
    RbfDev<float> rbf, conv;
    FilterGradBlock blk[kMaxBlocks];   // of interaction block blockIdx.y; xt NULL: zero
    const float *H, *Zd;           // hidden rows and z' in hidden_offset() order
    const float *zmax;             // largest |z'| (one value, as filter_vd leaves it)
    float *partial;                // per block and CTA [kF][kF] dA2 | [kF][R] dA1 | [kF] db1
    int64_t stride;                // floats per CTA
    int64_t block_hidden;          // kept floats per block
    int32_t *status;
};

struct FilterGradSmem {
    static constexpr int kA2 = 0, kX = 65536, kY = 131072, kMisc = 196608;
    static constexpr int kTotal = kMisc + 4096 + 1024;
};

// instruction descriptor with both operands read MN-major (A transposed)
__device__ __forceinline__ uint32_t instr_desc_tt(int n) { return tc::instr_desc(0, 1, n) | (1u << 15); }

__global__ void __launch_bounds__(kTcThreads, 1) filter_wgrad_kernel(const __grid_constant__ FilterGradParams q) {
    using namespace tc;
    using L = FilterGradSmem;
    const FilterGradBlock &nb = q.blk[blockIdx.y];
    const float *xl = nb.xl, *xt = nb.xt, *gagg = nb.gagg, *agb = nb.agb;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t *X = smem + L::kX, *Y = smem + L::kY;
    float2 *s_tab = reinterpret_cast<float2 *>(smem + L::kMisc);
    float *s_red = reinterpret_cast<float *>(smem + L::kMisc + 1024);         // [512]
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(smem + L::kMisc + 3072);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 1);
    int *s_err = reinterpret_cast<int *>(s_tmem + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & 127, qt = tid >> 7, col0 = qt * 32;
    const int R = q.rbf.R;
    const int Kpad1 = R <= 64 ? 64 : 128;
    if (load_weight_tile<true>(smem + L::kA2, smem + L::kA2 + 32768, nb.A2, kF, kF, kF, kWScale) && blockIdx.x == 0) atomicOr(q.status, (int)kWeightRange);
    if (tid < kF) {
        float c = 1e4f, w = 1.f;                       // beyond R: 2^(-(t - 1e4)^2) = 0
        if (tid < R) {
            c = q.rbf.p0[tid];
            w = (q.rbf.kind == 0 ? -q.rbf.p1[0] : q.rbf.p1[tid]) * kLog2e;
        }
        s_tab[tid] = make_float2(c, w);
    }
    const uint32_t bar = smem_u32(s_bar);
    if (tid == 0) {
        mbar_init(bar, 1);
        *s_err = 0;
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_u32(s_tmem), 512);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t tmem = *s_tmem;                     // dA2 [0,128) | dA1 [128,256) | hb [256,384) | hd [384,512)
    const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t a2_hi = smem_u32(smem + L::kA2), a2_lo = a2_hi + 32768, x_hi = smem_u32(X), x_lo = x_hi + 32768, y_hi = smem_u32(Y), y_lo = y_hi + 32768;

    const float slope = table_max_width(s_tab, R, lane);
    // right operands: |h|, |phi| <= 1, |h'| <= |z'|, and a bound on |phi'|
    const float env1 = q.rbf.cutoff_kind == 0 ? 0.f : 3.1416f / (q.rbf.lower > 0.f ? q.rbf.upper - q.rbf.lower : 2.f * q.rbf.upper);
    const float phi1 = 0.7142f * sqrtf(slope) * (q.rbf.kind == 0 ? 1.f : fabsf(q.rbf.alpha) * expf(fmaxf(q.rbf.alpha * q.rbf.lower, 0.f))) + fabsf(env1);
    const float sR2 = 32.f * row_scale(fmaxf(1.f, q.zmax[blockIdx.y])), sR1 = 32.f * row_scale(fmaxf(1.f, phi1));
    float sL2 = 0.f, sL1 = 0.f;                        // scales of the left operands (0: nothing accumulated yet)
    uint32_t acc2 = 0, acc1 = 0;                       // whether the next product adds to what tensor memory holds
    bool stored2 = false, stored1 = false;             // whether the CTA's partial already holds sums
    float *part2 = q.partial + ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * q.stride, *part1 = part2 + kF * kF, *partb = part1 + (int64_t)kF * R;
    float bsum = 0.f;                                  // db1 of column col0 + lane over this warp's rows
    const bool same_env = q.conv.cutoff_kind == q.rbf.cutoff_kind && q.conv.lower == q.rbf.lower && q.conv.upper == q.rbf.upper;
    uint32_t phase = 0;
    bool failed = false, pending = false;

    auto settle = [&]() {                              // all products issued so far are done: X, Y and the accumulators are free
        if (pending) {
            if (!failed && !mbar_wait(bar, phase)) failed = true;
            phase ^= 1;
            pending = false;
        }
        tc_fence_after();
    };
    auto block_max = [&](float v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        __syncthreads();
        if (lane == 0) s_red[warp] = v;
        __syncthreads();
        float m = s_red[0];
#pragma unroll
        for (int i = 1; i < 16; i++) m = fmaxf(m, s_red[i]);
        return m;
    };
    // sums held in tensor memory -> this CTA's partial (rows of `cols` floats)
    auto flush = [&](uint32_t col, float *part, int cols, float inv, bool add) {
        float *row = part + (int64_t)r * cols + col0;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            float v[16];
            tmem_ld16(t_lane + col + col0 + half * 16, v);
            if (((cols | (int)((uintptr_t)part >> 2)) & 3) == 0) {      // (a lane is a row: each store of a warp touches 32 lines, so as few as possible)
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    if (col0 + half * 16 + j < cols) {
                        float4 *at = reinterpret_cast<float4 *>(row + half * 16 + j);
                        const float4 old = add ? *at : make_float4(0.f, 0.f, 0.f, 0.f);
                        *at = make_float4(fmaf(v[j], inv, old.x), fmaf(v[j + 1], inv, old.y), fmaf(v[j + 2], inv, old.z), fmaf(v[j + 3], inv, old.w));
                    }
                continue;
            }
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (col0 + half * 16 + j < cols) row[half * 16 + j] = add ? fmaf(v[j], inv, row[half * 16 + j]) : v[j] * inv;
        }
        tc_fence_before();
    };
    // 32 values of row r, columns col0.. -> operand tile
    auto put_row = [&](uint8_t *tile, const float (&x)[32], float scale) {
        uint32_t hi[16], lo[16];
        pack32<true>(x, scale, hi, lo);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint32_t off = chunk_offset(r, col0 + 8 * c);
            *reinterpret_cast<uint4 *>(tile + off) = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
            *reinterpret_cast<uint4 *>(tile + 32768 + off) = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
        }
    };
    auto put4 = [&](uint8_t *tile, int row, int col, float4 v, float scale) {
        const float4 w = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
        const uint32_t off = elem_offset(row, col);
        const __half2 a0 = __floats2half2_rn(w.x, w.y), a1 = __floats2half2_rn(w.z, w.w);
        const float2 f0 = __half22float2(a0), f1 = __half22float2(a1);
        const __half2 c0 = __floats2half2_rn(w.x - f0.x, w.y - f0.y), c1 = __floats2half2_rn(w.z - f1.x, w.w - f1.y);
        *reinterpret_cast<uint2 *>(tile + off) = make_uint2(*reinterpret_cast<const uint32_t *>(&a0), *reinterpret_cast<const uint32_t *>(&a1));
        *reinterpret_cast<uint2 *>(tile + 32768 + off) = make_uint2(*reinterpret_cast<const uint32_t *>(&c0), *reinterpret_cast<const uint32_t *>(&c1));
    };
    // X^T Y into columns [col, col + n) (over the tile's 128 pairs); X A2 into columns [dst, dst + 128) where wanted
    auto issue = [&](uint32_t col, int n, uint32_t acc, int dst) {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after();
            if (dst >= 0) {
                const uint32_t id = instr_desc(0, 1, 128);
                const uint64_t dxh = desc_kmajor(x_hi), dxl = desc_kmajor(x_lo), bh = desc_mnmajor(a2_hi), bl = desc_mnmajor(a2_lo);
#pragma unroll
                for (int ks = 0; ks < 8; ks++) {      // (small products first: see issue_gemm_ts)
                    mma_f16_ss(tmem + dst, kstep_kmajor(dxh, ks), kstep_mnmajor(bl, ks), id, ks > 0 ? 1u : 0u);
                    mma_f16_ss(tmem + dst, kstep_kmajor(dxl, ks), kstep_mnmajor(bh, ks), id, 1u);
                }
#pragma unroll
                for (int ks = 0; ks < 8; ks++) mma_f16_ss(tmem + dst, kstep_kmajor(dxh, ks), kstep_mnmajor(bh, ks), id, 1u);
            }
            const uint32_t id = instr_desc_tt(n);
            const uint64_t dxh = desc_mnmajor(x_hi), dxl = desc_mnmajor(x_lo), yh = desc_mnmajor(y_hi), yl = desc_mnmajor(y_lo);
#pragma unroll
            for (int ks = 0; ks < 8; ks++) {
                mma_f16_ss(tmem + col, kstep_mnmajor(dxh, ks), kstep_mnmajor(yh, ks), id, ks > 0 ? 1u : acc);
                mma_f16_ss(tmem + col, kstep_mnmajor(dxh, ks), kstep_mnmajor(yl, ks), id, 1u);
                mma_f16_ss(tmem + col, kstep_mnmajor(dxl, ks), kstep_mnmajor(yh, ks), id, 1u);
            }
            mma_commit(bar);
        }
        pending = true;
    };

    const int64_t ntiles = (q.P + kRows - 1) / kRows;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        // ---- this lane's row: nodes, distance, envelopes (rows past the end: every left operand zero)
        const int64_t k = tile * kRows + r;
        const bool live = k < q.P;
        const int32_t e = live ? q.sel[k] : 0;
        const int32_t ni = live ? q.row0[e] : 0, nj = live ? q.row1[e] : 0;
        const float de = live ? q.d[e] : 1.f, dde = live ? q.dd[e] : 0.f;
        float t, dt;
        edge_arg(de, q.rbf, t, dt);
        const Jet<float, 1> env = envelope_jet<float, 1>(de, q.rbf);
        float c0 = env.c[0], c1 = env.c[1];
        if (!same_env) {
            const Jet<float, 1> cj = envelope_jet<float, 1>(de, q.conv);
            c0 = cj.c[0];
            c1 = cj.c[1];
        }
        const float fo = live ? c0 : 0.f, fo1 = live ? c1 * dde : 0.f, fd = live ? c0 * dde : 0.f;
        // ---- o, od: four rows per load instruction, four columns per lane
        const int sub = lane >> 3, cc = (col0 >> 2) + (lane & 7);
        float4 o[8], od[8];
        float m = 0.f;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int rl = u * 4 + sub;
            const int64_t i = __shfl_sync(0xffffffffu, ni, rl), j = __shfl_sync(0xffffffffu, nj, rl);
            const float go = __shfl_sync(0xffffffffu, fo, rl), go1 = __shfl_sync(0xffffffffu, fo1, rl), gd = __shfl_sync(0xffffffffu, fd, rl);
            const float4 xi = __ldg(reinterpret_cast<const float4 *>(xl + i * kF) + cc), xj = __ldg(reinterpret_cast<const float4 *>(xl + j * kF) + cc);
            const float4 gi = __ldg(reinterpret_cast<const float4 *>(gagg + i * kF) + cc), gj = __ldg(reinterpret_cast<const float4 *>(gagg + j * kF) + cc);
            const float4 bi = __ldg(reinterpret_cast<const float4 *>(agb + i * kF) + cc), bj = __ldg(reinterpret_cast<const float4 *>(agb + j * kF) + cc);
            float4 ti = make_float4(0.f, 0.f, 0.f, 0.f), tj = ti;
            if (xt) {
                ti = __ldg(reinterpret_cast<const float4 *>(xt + i * kF) + cc);
                tj = __ldg(reinterpret_cast<const float4 *>(xt + j * kF) + cc);
            }
            auto both = [&](float vxi, float vxj, float vgi, float vgj, float vbi, float vbj, float vti, float vtj, float &ro, float &rd) {
                const float w1 = fmaf(vgi, vxj, vgj * vxi);
                const float w0 = fmaf(vbi, vxj, vbj * vxi) + fmaf(vgi, vtj, vgj * vti);
                ro = fmaf(go, w0, go1 * w1);
                rd = gd * w1;
                m = fmaxf(m, fmaxf(fabsf(ro), fabsf(rd)));
            };
            both(xi.x, xj.x, gi.x, gj.x, bi.x, bj.x, ti.x, tj.x, o[u].x, od[u].x);
            both(xi.y, xj.y, gi.y, gj.y, bi.y, bj.y, ti.y, tj.y, o[u].y, od[u].y);
            both(xi.z, xj.z, gi.z, gj.z, bi.z, bj.z, ti.z, tj.z, o[u].z, od[u].z);
            both(xi.w, xj.w, gi.w, gj.w, bi.w, bj.w, ti.w, tj.w, o[u].w, od[u].w);
        }
        m = block_max(m);
        settle();                                      // (the last product of the tile before)
        if (sL2 == 0.f || m * sL2 > 32768.f) {         // (the same in every thread)
            if (acc2 && sL2 > 0.f) {
                flush(0, part2, kF, 1.f / (sL2 * sR2), stored2);
                stored2 = true;
                __syncthreads();
            }
            acc2 = 0;
            sL2 = m > 0.f ? 128.f * row_scale(m) : 0.f;        // largest entry to [2^10, 2^11); nothing but zeros: as good as unset
        }
        const float s2 = sL2 > 0.f ? sL2 : 1.f;
        const float4 *hb4 = reinterpret_cast<const float4 *>(q.H + blockIdx.y * q.block_hidden);
        const float4 *zb4 = reinterpret_cast<const float4 *>(q.Zd + blockIdx.y * q.block_hidden);
        const int row_base = (warp & 3) * 32;
        // ---- A: X = o, Y = h
#pragma unroll
        for (int u = 0; u < 8; u++) put4(X, row_base + u * 4 + sub, cc * 4, o[u], s2);
        {
            float x[32];
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float4 h = hb4[hidden_offset(tile, qt, c, r)];
                x[4 * c] = h.x; x[4 * c + 1] = h.y; x[4 * c + 2] = h.z; x[4 * c + 3] = h.w;
            }
            put_row(Y, x, sR2);
        }
        issue(0, kF, acc2, 256);
        acc2 = 1;
        // ---- B: X = od, Y = h'
        {
            float x[32];
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float4 h = hb4[hidden_offset(tile, qt, c, r)], z = zb4[hidden_offset(tile, qt, c, r)];
                x[4 * c] = fmaf(-h.x, h.x, 1.f) * z.x; x[4 * c + 1] = fmaf(-h.y, h.y, 1.f) * z.y;
                x[4 * c + 2] = fmaf(-h.z, h.z, 1.f) * z.z; x[4 * c + 3] = fmaf(-h.w, h.w, 1.f) * z.w;
            }
            settle();
            put_row(Y, x, sR2);
        }
#pragma unroll
        for (int u = 0; u < 8; u++) put4(X, row_base + u * 4 + sub, cc * 4, od[u], s2);
        issue(0, kF, 1u, 384);
        // ---- C: X = zb, Y = phi
        float zb[32], zd[32];
        settle();
        {
            const float inv = 1.f / (s2 * kWScale);
            m = 0.f;
#pragma unroll
            for (int half = 0; half < 2; half++) {
                float vb[16], vd[16];
                tmem_ld16(t_lane + 256 + col0 + half * 16, vb);
                tmem_ld16(t_lane + 384 + col0 + half * 16, vd);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float4 h4 = hb4[hidden_offset(tile, qt, half * 4 + c, r)], z4 = zb4[hidden_offset(tile, qt, half * 4 + c, r)];
                    const float hh[4] = {h4.x, h4.y, h4.z, h4.w}, zz[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int n = half * 16 + 4 * c + i;
                        const float s = fmaf(-hh[i], hh[i], 1.f), hd = vd[4 * c + i] * inv;
                        zd[n] = s * hd;
                        zb[n] = s * fmaf(-2.f * hh[i] * zz[i], hd, vb[4 * c + i] * inv);
                        m = fmaxf(m, fmaxf(fabsf(zb[n]), fabsf(zd[n])));
                    }
                }
            }
            tc_fence_before();
        }
        m = block_max(m);
        if (sL1 == 0.f || m * sL1 > 32768.f) {
            if (acc1 && sL1 > 0.f) {
                flush(128, part1, R, 1.f / (sL1 * sR1), stored1);
                stored1 = true;
                __syncthreads();
            }
            acc1 = 0;
            sL1 = m > 0.f ? 128.f * row_scale(m) : 0.f;
        }
        const float s1 = sL1 > 0.f ? sL1 : 1.f;
        put_row(X, zb, s1);
        {   // column sums of zb over the warp's 32 rows: after five exchanges lane l is left with column col0 + l
            float v[16];
#pragma unroll
            for (int c = 0; c < 16; c++) {
                const bool up = lane & 16;
                v[c] = (up ? zb[c + 16] : zb[c]) + __shfl_xor_sync(0xffffffffu, up ? zb[c] : zb[c + 16], 16);
            }
#pragma unroll
            for (int o2 = 8; o2 > 0; o2 >>= 1)
#pragma unroll
                for (int c = 0; c < o2; c++) {
                    const bool up = lane & o2;
                    v[c] = (up ? v[c + o2] : v[c]) + __shfl_xor_sync(0xffffffffu, up ? v[c] : v[c + o2], o2);
                }
            bsum += v[0];
        }
        const float4 *tab4 = reinterpret_cast<const float4 *>(s_tab + col0);
        if (col0 < Kpad1) {
            float x[32];
            const float l2a = log2f(env.c[0]);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float4 cw = tab4[j];
                const float u0 = t - cw.x, u1 = t - cw.z;
                x[2 * j] = ex2_fast(fmaf(-cw.y * u0, u0, l2a));
                x[2 * j + 1] = ex2_fast(fmaf(-cw.w * u1, u1, l2a));
            }
            put_row(Y, x, sR1);
        }
        issue(128, Kpad1, acc1, -1);
        acc1 = 1;
        // ---- D: X = zd, Y = phi'
        {
            float x[32];
            if (col0 < Kpad1) {
                const float m2 = -2.f * kLn2 * dt * env.c[0];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float4 cw = tab4[j];
                    const float u0 = t - cw.x, wu0 = cw.y * u0, u1 = t - cw.z, wu1 = cw.w * u1;
                    x[2 * j] = ex2_fast(-wu0 * u0) * fmaf(m2, wu0, env.c[1]);
                    x[2 * j + 1] = ex2_fast(-wu1 * u1) * fmaf(m2, wu1, env.c[1]);
                }
            }
            settle();
            put_row(X, zd, s1);
            if (col0 < Kpad1) put_row(Y, x, sR1);
        }
        issue(128, Kpad1, 1u, -1);
    }
    settle();
    __syncthreads();
    flush(0, part2, kF, sL2 > 0.f ? 1.f / (sL2 * sR2) : 0.f, stored2);
    flush(128, part1, R, sL1 > 0.f ? 1.f / (sL1 * sR1) : 0.f, stored1);
    s_red[(warp & 3) * 128 + col0 + lane] = bsum;
    if (failed) *s_err = 1;
    tc_fence_before();
    __syncthreads();
    if (tid < kF) partb[tid] = (s_red[tid] + s_red[128 + tid]) + (s_red[256 + tid] + s_red[384 + tid]);
    if (*s_err && tid == 0) atomicOr(q.status, 8);
    if (warp == 0) tmem_free(tmem, 512);
}

int filter_wgrad_parts(int64_t P, int64_t num_blocks) {
    const int64_t ntiles = (P + tc::kRows - 1) / tc::kRows, per_block = num_blocks < kNumSM ? kNumSM / num_blocks : 1;
    return (int)(ntiles < per_block ? ntiles : per_block);
}

int filter_wgrad_blocks(const float *d, const float *dd, int64_t P, const int32_t *sel, const int32_t *row0, const int32_t *row1,
                        const mlcgb_rbf_spec *rbf, int conv_cutoff_kind, double conv_lower, double conv_upper, const FilterGradBlock *blocks,
                        int64_t num_blocks, const float *hs, const float *zs, const float *zmax, float *partial, int32_t *status, cudaStream_t st) {
    TimelineScope timeline_scope("filter_weight_grad", st);
    if (int rc = check_spec(rbf, 1)) return rc;
    if (P < 0 || !status || (conv_cutoff_kind != 0 && conv_cutoff_kind != 1)) return MLCGB_E_ARG;
    if (rbf->num_rbf > 128 || num_blocks < 1 || num_blocks > kMaxBlocks) return MLCGB_E_LIMIT;
    if (P == 0) return MLCGB_OK;
    if (!d || !dd || !sel || !row0 || !row1 || !hs || !zs || !zmax || !partial) return MLCGB_E_ARG;
    FilterGradParams q;
    for (int64_t l = 0; l < num_blocks; l++) {
        q.blk[l] = blocks[l];
        if (!q.blk[l].A2 || !q.blk[l].xl || !q.blk[l].gagg || !q.blk[l].agb) return MLCGB_E_ARG;
    }
    q.d = d;
    q.dd = dd;
    q.P = P;
    q.sel = sel;
    q.row0 = row0;
    q.row1 = row1;
    q.rbf = to_dev<float>(rbf);
    q.conv = q.rbf;
    q.conv.cutoff_kind = conv_cutoff_kind;
    q.conv.lower = (float)conv_lower;
    q.conv.upper = (float)conv_upper;
    q.H = hs;
    q.Zd = zs;
    q.zmax = zmax;
    q.partial = partial;
    q.stride = (int64_t)kF * kF + (int64_t)kF * rbf->num_rbf + kF;
    q.block_hidden = (int64_t)(mlcgb_filter_hidden_bytes(P) / sizeof(float));
    q.status = status;
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        if (cudaFuncSetAttribute(filter_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FilterGradSmem::kTotal) != cudaSuccess) return check_launch();
        done[dev] = true;
    }
    launch_with_weights(filter_wgrad_kernel, dim3(filter_wgrad_parts(P, num_blocks), (unsigned)num_blocks), dim3(kTcThreads), FilterGradSmem::kTotal, st, q);
    return check_launch();
}

}  // namespace mlcgb

// Set-up and element-wise pieces shared by the fused filter-network kernels: parameters, shared-memory layout, weight tiles, basis
// table, tanh through the special-function unit, the order in which hidden rows are kept.
#pragma once
#include <type_traits>

#include "rbf_device.cuh"
#include "tc_common.cuh"
#include "tensor_map.cuh"

namespace mlcgb {

// Phase timing of the saved-hidden-layer backward (development builds only, -DMLCGB_PHASE_TIMING): thread 0 of every block adds
// the cycles between consecutive marks to per-phase totals that mlcgb_debug_phase_cycles reads back.
#ifdef MLCGB_PHASE_TIMING
__device__ unsigned long long g_phase_cycles[16];
#define PHASE_DECL long long ph_last = clock64();
#define PHASE(k)                                                          \
    if (tid == 0) {                                                       \
        const long long ph_now = clock64();                               \
        atomicAdd(&g_phase_cycles[k], (unsigned long long)(ph_now - ph_last)); \
        ph_last = clock64();                                              \
    }
#else
#define PHASE_DECL
#define PHASE(k)
#endif

constexpr int kF = 128;                 // filters / hidden width of the filter network
constexpr int kTcThreads = 512;         // thread t: row t % 128 of the tile, 32-column quarter t / 128
constexpr float kWScale = 64.f;         // power-of-two weight scaling keeps the fp16 "low" parts of the weights normal
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

struct FilterFwdParams {
    const float *d;      // [E]
    int64_t E;           // rows to process: all edges, or one edge per unordered pair when `sel` is given
    const int64_t *rows_dev;  // NULL, or the row count in device memory (written by an earlier kernel on the stream): the
                              // kernel then processes min(E, *rows_dev) rows and E only sizes the grid and the buffers
    const int32_t *sel;  // [E] edge handled by row k (NULL: k itself)
    const int32_t *twin; // reverse edge of each edge (NULL: none); with `sel`, results go to both edges of a pair
                         // (forward with `sel` alone: W has E rows, row k is the filter of edge sel[k])
    RbfDev<float> rbf;   // basis and its envelope
    RbfDev<float> conv;  // only cutoff_kind / lower / upper are used: the CFConv cutoff C(d)
    const float *A1;     // [kF][R]
    const float *b1;     // [kF]
    const float *A2;     // [kF][kF]
    float *W;            // [E][kF]
    float *H;            // NULL, or where the forward keeps h = tanh(phi A1^T + b1) for the backward (hidden_offset() order)
    int32_t *status;
};

// The hidden layer of a tile is kept in the order the threads hold it: thread (row r, 32-column quarter q) owns eight 16-byte
// chunks j; chunk (q, j) of all 128 rows is contiguous, so both kernels move it with fully coalesced 128-bit accesses and
// no staging.  Offset, in float4 units, of chunk j of quarter q of row r of tile t; a tile takes 16384 floats.
__device__ __forceinline__ int64_t hidden_offset(int64_t tile, int q, int j, int r) { return ((tile * 4 + q) * 8 + j) * 128 + r; }

// rows the kernel works on; read after the wait on the preceding kernels
__device__ __forceinline__ int64_t live_rows(const FilterFwdParams &p) {
    if (!p.rows_dev) return p.E;
    const int64_t n = *reinterpret_cast<const volatile int64_t *>(p.rows_dev);
    return n < 0 ? 0 : (n < p.E ? n : p.E);
}

template <bool SPLIT>
struct FilterSmem {
    static constexpr int kTile = SPLIT ? 2 * 32768 : 32768;   // one 128x128 operand tile (hi [+ lo])
    static constexpr int kStageBytes = 65536;                 // fp32 staging tile: 128 rows of 512 B
    static constexpr int kASize = SPLIT ? kStageBytes : kTile;
    static constexpr int kA = 0, kB1 = kASize, kB2 = kASize + kTile, kMisc = kASize + 2 * kTile;
    // misc: bias, scaled bias [2][128] f32 | basis table [128] float2 | exchange [4][128] f32 x2 | barrier, TMEM slot, error flag
    static constexpr int kBias = 0, kTable = 1024, kRed = 2048, kRed2 = 4096, kBar = 6144;
    // fp32 staging tile for coalesced global traffic: in the A region (free when the A operands live in TMEM) or its own
    static constexpr int kStage = SPLIT ? kA : kMisc + 7168;
    static constexpr int kTotal = kMisc + 7168 + (SPLIT ? 0 : kStageBytes) + 1024;   // + alignment slack
    // the backward that reads the saved hidden layer: two more [4][128] f32 exchange arrays behind everything else
    static constexpr int kExtra = kMisc + 7168 + (SPLIT ? 0 : kStageBytes);
    static constexpr int kTotalExtra = kExtra + 4096 + 1024;
};

__device__ __forceinline__ float tanh_fast(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_fast(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ex2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float min_nan(float x, float y) {      // (fminf gives the number where one of the two is none)
    float m;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(x), "f"(y));
    return m;
}
// Per-edge part of the basis: value t(d) the basis functions are centred on and its derivative.
//   Gaussian:   g_k = exp(coeff (d - offset_k)^2)                 t = d,                 t' = 1
//   exp-normal: g_k = exp(-beta_k (u - mean_k)^2), u = exp(alpha (lower - d)):  t = u,   t' = -alpha u
// The table holds (c_k, w_k) with g_k = 2^(-w_k (t - c_k)^2), w_k = width_k log2(e)
// (widths are positive: -coeff for the Gaussian, beta_k for the exp-normal basis).
__device__ __forceinline__ void edge_arg(float d, const RbfDev<float> &s, float &t, float &dt) {
    if (s.kind == 0) {
        t = d;
        dt = 1.f;
    } else {
        t = expf(s.alpha * (-d + s.lower));
        dt = -s.alpha * t;
    }
}

// Shared set-up of both kernels: weight tiles, bias, basis table, barrier, tensor memory.
template <bool SPLIT>
__device__ __forceinline__ uint32_t filter_setup(const FilterFwdParams &p, uint8_t *smem, int Kpad1, uint32_t tmem_cols, bool have_weights = false) {
    using namespace tc;
    using L = FilterSmem<SPLIT>;
    const int tid = threadIdx.x, warp = tid >> 5;
    const float wscale = SPLIT ? kWScale : 1.f;
    if (!have_weights) {
        const bool over1 = load_weight_tile<SPLIT>(smem + L::kB1, smem + L::kB1 + 32768, p.A1, kF, p.rbf.R, Kpad1, wscale, true);
        const bool over2 = load_weight_tile<SPLIT>(smem + L::kB2, smem + L::kB2 + 32768, p.A2, kF, kF, kF, wscale);
        if ((over1 || over2) && blockIdx.x == 0) atomicOr(p.status, (int)kWeightRange);
    }
    float *s_b1 = reinterpret_cast<float *>(smem + L::kMisc + L::kBias);
    float2 *s_tab = reinterpret_cast<float2 *>(smem + L::kMisc + L::kTable);
    if (tid < kF) {
        s_b1[tid] = p.b1[tid];
        float c = 1e4f, w = 1.f;                       // beyond R: 2^(-(t - 1e4)^2) = 0
        if (tid < p.rbf.R) {
            c = p.rbf.p0[tid];
            w = (p.rbf.kind == 0 ? -p.rbf.p1[0] : p.rbf.p1[tid]) * kLog2e;
        }
        s_tab[tid] = make_float2(c, w);
        s_b1[kF + tid] = p.b1[tid] * (2.f * kLog2e);    // bias pre-multiplied for the exp2-based tanh
    }
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(smem + L::kMisc + L::kBar);
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(s_bar + 1);
    int *s_err = reinterpret_cast<int *>(s_tmem + 1);
    if (tid == 0) {
        mbar_init(smem_u32(s_bar), 1);
        *s_err = 0;
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_u32(s_tmem), tmem_cols);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return *s_tmem;
}

// Largest |w_k| of the basis table, by all lanes of a warp
__device__ __forceinline__ float table_max_width(const float2 *s_tab, int R, int lane) {
    float w = 0.f;
    for (int k = lane; k < R; k += 32) w = fmaxf(w, fabsf(s_tab[k].y));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w = fmaxf(w, __shfl_xor_sync(0xffffffffu, w, o));
    return w;
}

// h = tanh(z) for this thread's accumulator values, z = v * unscale + b1, through exp2: tanh z = sign(z) (1 - 2/(2^{|zz|} + 1)),
// zz = 2 log2(e) z.  |zz| is clamped at 30, where the result has long rounded to 1, so that four denominators can share one
// reciprocal (1/A = B C D / (A B C D), ...): five special-function operations per four values instead of eight — this phase
// runs at the special-function unit's rate — for nine extra multiplies.
template <bool SPLIT, int NC = 32>
__device__ __forceinline__ void tanh_row32(float (&v)[NC], const float *s_b1s, int col0, float unscale2) {
    const float4 *b4 = reinterpret_cast<const float4 *>(s_b1s + col0);
#pragma unroll
    for (int q = 0; q < NC / 4; q++) {
        const float4 bq = b4[q];
        const float bb[4] = {bq.x, bq.y, bq.z, bq.w};
        if (SPLIT) {
            using tc::both;
            float2 zz[2], den[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                zz[i] = tc::fma2(make_float2(v[4 * q + 2 * i], v[4 * q + 2 * i + 1]), both(unscale2), make_float2(bb[2 * i], bb[2 * i + 1]));
                den[i] = tc::add2(make_float2(ex2_fast(min_nan(fabsf(zz[i].x), 30.f)), ex2_fast(min_nan(fabsf(zz[i].y), 30.f))), both(1.f));
            }
            // (products of the first and of the second of each pair, so that the pairs stay pairs)
            const float2 p = tc::mul2(den[0], den[1]);
            const float r = rcp_fast(p.x * p.y);
            const float2 ri = tc::mul2(both(r), make_float2(p.y, p.x));      // 1 / p
            const float2 inv[2] = {tc::mul2(ri, den[1]), tc::mul2(ri, den[0])};
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float2 m = tc::fma2(both(-2.f), inv[i], both(1.f));
                v[4 * q + 2 * i] = copysignf(m.x, zz[i].x);
                v[4 * q + 2 * i + 1] = copysignf(m.y, zz[i].y);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) v[4 * q + i] = tanh_fast(fmaf(v[4 * q + i], unscale2, bb[i]) * (0.5f * kLn2));
        }
    }
}

// fp32 staging tile [128 rows][32 chunks of 16 B], chunk index XOR-ed with (row & 7): a thread writing its own
// row and a warp reading one whole row are both free of bank conflicts
__device__ __forceinline__ float4 *stage_chunk(uint8_t *stage, int row, int chunk) {
    return reinterpret_cast<float4 *>(stage + row * 512 + ((chunk ^ (row & 7)) << 4));
}

}  // namespace mlcgb

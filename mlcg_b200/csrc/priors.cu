// Classical prior terms (bonds, angles, dihedrals, repulsion): energy per structure and dE/dpos in
// one pass over the static index lists.  One thread per term; the term's energy is reduced inside
// the warp when all 32 terms belong to the same structure (the common case, lists are ordered by
// structure), gradients go out as floating-point atomics.
#include "common.cuh"
#include "small_graph.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <type_traits>

namespace mlcgb {

template <typename T> struct V3 { T x, y, z; };
template <typename T> __device__ __forceinline__ V3<T> ld3(const T *p, int64_t i) { return V3<T>{p[i * 3], p[i * 3 + 1], p[i * 3 + 2]}; }
template <typename T> __device__ __forceinline__ V3<T> sub(const V3<T> &a, const V3<T> &b) { return V3<T>{a.x - b.x, a.y - b.y, a.z - b.z}; }
template <typename T> __device__ __forceinline__ T dot(const V3<T> &a, const V3<T> &b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <typename T> __device__ __forceinline__ V3<T> cross(const V3<T> &a, const V3<T> &b) {
    return V3<T>{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <typename T> __device__ __forceinline__ V3<T> scale(const V3<T> &a, T s) { return V3<T>{a.x * s, a.y * s, a.z * s}; }
template <typename T> __device__ __forceinline__ V3<T> axpy(T s, const V3<T> &a, const V3<T> &b) { return V3<T>{s * a.x + b.x, s * a.y + b.y, s * a.z + b.z}; }
template <typename T> __device__ __forceinline__ void atomic_add3(T *g, int64_t i, const V3<T> &v) {
    atomicAdd(g + i * 3, v.x);
    atomicAdd(g + i * 3 + 1, v.y);
    atomicAdd(g + i * 3 + 2, v.z);
}

// Bonds, angles and dihedrals are evaluated in double precision whatever the storage type: their lists are short (one term
// per bead, where a repulsion list has hundreds), and in float32 a harmonic bond loses most of its digits in d - x0 and a
// torsion gradient in the cross products of nearly collinear bonds.  Positions and parameters are read as stored; energy and
// gradient are rounded to the storage type once, at the end.
template <typename T> __device__ __forceinline__ V3<double> ld3d(const T *p, int64_t i) {
    return V3<double>{(double)p[i * 3], (double)p[i * 3 + 1], (double)p[i * 3 + 2]};
}
template <typename T> __device__ __forceinline__ V3<T> narrow(const V3<double> &a) { return V3<T>{(T)a.x, (T)a.y, (T)a.z}; }

// harmonic bond k (d - x0)^2: energy; g1 = dE/dpos[i1] (dE/dpos[i0] = -g1)
__device__ __forceinline__ double bond_term(const V3<double> &p0, const V3<double> &p1, double x0, double k, V3<double> &g1) {
    const V3<double> dr = sub(p1, p0);
    const double d = sqrt(dot(dr, dr));
    g1 = scale(dr, 2.0 * k * (d - x0) / d);
    return k * (d - x0) * (d - x0);
}

// harmonic angle in the cosine, k (cos - x0)^2: ga = dE/dpos[i0], gb = dE/dpos[i2] (dE/dpos[i1] = -ga - gb)
__device__ __forceinline__ double angle_term(const V3<double> &p0, const V3<double> &p1, const V3<double> &p2, double x0, double k,
                                             V3<double> &ga, V3<double> &gb) {
    const V3<double> a = sub(p0, p1), b = sub(p2, p1);
    const double ia = rsqrt(dot(a, a)), ib = rsqrt(dot(b, b)), inv = ia * ib;
    const double c = dot(a, b) * inv;
    const double dEdc = 2.0 * k * (c - x0);
    ga = scale(axpy(-c * (ia * ia), a, scale(b, inv)), dEdc);
    gb = scale(axpy(-c * (ib * ib), b, scale(a, inv)), dEdc);
    return k * (c - x0) * (c - x0);
}

// Fourier series in the torsion angle of compute_torsions (unit bond vectors, atan2(-m.n2, n1.n2)).  Only sines and cosines of
// its multiples enter: (cos, sin) is the normalised pair (n1.n2, -m.n2), and the multiples follow from the angle sum formulas, so
// that no inverse or direct trigonometric function is called (16 double-precision calls per six-term series before).
// params rows v0, k1_1..k1_n, k2_1..k2_n with stride M; g[0..3] = dE/dpos of the four beads
template <typename T>
__device__ __forceinline__ double torsion_term(const V3<double> &p0, const V3<double> &p1, const V3<double> &p2, const V3<double> &p3,
                                               const T *params, int64_t M, int64_t t, int n_degs, V3<double> (&g)[4]) {
    const V3<double> b1 = sub(p1, p0), b2 = sub(p2, p1), b3 = sub(p3, p2);
    const double G2 = dot(b2, b2), iG = rsqrt(G2), Gn = G2 * iG;
    const V3<double> u1 = scale(b1, rsqrt(dot(b1, b1)));
    const V3<double> u2 = scale(b2, iG);
    const V3<double> u3 = scale(b3, rsqrt(dot(b3, b3)));
    const V3<double> n1 = cross(u1, u2), n2 = cross(u2, u3), m1 = cross(n1, u2);
    const double x = dot(n1, n2), y = -dot(m1, n2), r2 = x * x + y * y;
    const double ir = rsqrt(r2);
    const double c1 = r2 > 0.0 ? x * ir : 1.0, s1 = r2 > 0.0 ? y * ir : 0.0;        // (atan2(0, 0) = 0)
    double cs = c1, sn = s1;
    double e = (double)params[t], dEdth = 0.0;
    for (int n = 1; n <= n_degs; n++) {
        const double k1 = (double)params[(int64_t)n * M + t], k2 = (double)params[(int64_t)(n_degs + n) * M + t];
        e += k1 * sn + k2 * cs;
        dEdth += (double)n * (k1 * cs - k2 * sn);
        const double cn = cs * c1 - sn * s1;
        sn = sn * c1 + cs * s1;
        cs = cn;
    }
    // d(theta)/d(positions): F = p0-p1 = -b1, G = p1-p2 = -b2, H = p3-p2 = b3, A = F x G, B = H x G
    const V3<double> A = cross(b1, b2), Bv = cross(b2, b3);
    const double iA2 = 1.0 / dot(A, A), iB2 = 1.0 / dot(Bv, Bv);
    const double fg = dot(b1, b2) * (iA2 * iG), hg = -dot(b3, b2) * (iB2 * iG), ga = Gn * iA2, gb = Gn * iB2;
    g[0] = scale(A, -ga * dEdth);
    g[3] = scale(Bv, gb * dEdth);
    g[1] = scale(axpy(-hg, Bv, scale(A, ga + fg)), dEdth);
    g[2] = scale(axpy(hg - gb, Bv, scale(A, -fg)), dEdth);
    return e;
}

// Adds v into g[i] with one atomic per run of consecutive lanes that share the same index i (pair lists are
// usually grouped by their first index, so a warp holds one or two runs).  Every lane of the warp must call this;
// lanes without a contribution pass i = -1.
template <typename T>
__device__ __forceinline__ void run_add3(T *g, int64_t i, V3<T> v, int lane) {
    const int64_t prev = __shfl_up_sync(0xffffffffu, i, 1);
    const bool head = lane == 0 || prev != i;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    // end of this lane's run = position of the next head above it
    const unsigned above = lane == 31 ? 0u : (heads >> (lane + 1));
    const int run_end = above ? lane + __ffs(above) : 32;   // exclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T x = __shfl_down_sync(0xffffffffu, v.x, o), y = __shfl_down_sync(0xffffffffu, v.y, o), z = __shfl_down_sync(0xffffffffu, v.z, o);
        if (lane + o < run_end) { v.x += x; v.y += y; v.z += z; }
    }
    if (head && i >= 0) atomic_add3(g, i, v);
}

template <typename T, int KIND>
__global__ void __launch_bounds__(256)
prior_kernel(const T *__restrict__ pos, const int64_t *__restrict__ mapping, const int64_t *__restrict__ mapping_batch,
             const T *__restrict__ params, int n_params, int64_t M, int64_t N, int64_t B, T *__restrict__ energy,
             T *__restrict__ grad, int32_t *__restrict__ status) {
    constexpr int ORDER = KIND == 0 || KIND == 3 ? 2 : (KIND == 1 ? 3 : 4);
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane;  // warp-uniform base
    for (int64_t base = first; base < M; base += stride) {
        const int64_t t = base + lane;
        bool valid = t < M;
        int64_t idx[ORDER];
        int64_t mb = 0;
        if (valid) {
#pragma unroll
            for (int o = 0; o < ORDER; o++) {
                idx[o] = mapping[(int64_t)o * M + t];
                if (idx[o] < 0 || idx[o] >= N) valid = false;
            }
            mb = mapping_batch[t];
            if (mb < 0 || mb >= B) valid = false;
            if (!valid) atomicOr(status, (int)kBadIndex);
        }
        T e = T(0);
        V3<T> g0{T(0), T(0), T(0)};   // pair terms: gradient on the first index, reduced over runs below
        if (valid) {
            if (KIND == 0) {
                V3<double> g1;
                e = (T)bond_term(ld3d(pos, idx[0]), ld3d(pos, idx[1]), (double)params[t], (double)params[M + t], g1);
                if (grad) {
                    atomic_add3(grad, idx[1], narrow<T>(g1));
                    g0 = narrow<T>(scale(g1, -1.0));
                }
            } else if (KIND == 3) {
                const V3<T> dr = sub(ld3(pos, idx[1]), ld3(pos, idx[0]));
                const T d = sqrt(dot(dr, dr));
                const T q = params[t] / d;
                const T rr = q * q;
                e = rr * rr * rr;
                if (grad) {
                    const V3<T> g1 = scale(dr, T(-6) * e / d / d);
                    atomic_add3(grad, idx[1], g1);
                    g0 = scale(g1, T(-1));
                }
            } else if (KIND == 1) {
                V3<double> ga, gb;
                e = (T)angle_term(ld3d(pos, idx[0]), ld3d(pos, idx[1]), ld3d(pos, idx[2]), (double)params[t], (double)params[M + t], ga, gb);
                if (grad) {
                    atomic_add3(grad, idx[0], narrow<T>(ga));
                    atomic_add3(grad, idx[2], narrow<T>(gb));
                    atomic_add3(grad, idx[1], narrow<T>(V3<double>{-ga.x - gb.x, -ga.y - gb.y, -ga.z - gb.z}));
                }
            } else {
                V3<double> g[4];
                e = (T)torsion_term(ld3d(pos, idx[0]), ld3d(pos, idx[1]), ld3d(pos, idx[2]), ld3d(pos, idx[3]), params, M, t, (n_params - 1) / 2, g);
                if (grad) {
#pragma unroll
                    for (int o = 0; o < 4; o++) atomic_add3(grad, idx[o], narrow<T>(g[o]));
                }
            }
        }
        if ((KIND == 0 || KIND == 3) && grad) run_add3(grad, valid ? idx[0] : (int64_t)-1, g0, lane);
        // energy: one atomic per warp when the whole warp sits in one structure
        const int64_t mb0 = __shfl_sync(0xffffffffu, mb, 0);
        const bool same = __all_sync(0xffffffffu, !valid || mb == mb0);
        const bool lane0_valid = __shfl_sync(0xffffffffu, (int)valid, 0) != 0;
        if (same && lane0_valid) {
            const T s = warp_sum(e);
            if (lane == 0) atomicAdd(energy + mb0, s);
        } else if (valid) {
            atomicAdd(energy + mb, e);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// All prior classes of a model together, in three launches (four where single terms are the larger part beside slices): a first one that widens the positions to one 16-byte (32-byte) record per
// bead with its structure and clears the sums, one for the slices of pair lists and all other terms, a last one that turns the
// sums into energies and gradients (or forces) and adds up the lists.  Up to MLCGB_MAX_PRIOR_SEGMENTS lists; every list has its own
// energy row and gradient block, so the caller still gets one energy / force set per prior, and the totals that SumOut forms
// (src/mlcg/nn/gradients.py:111-117).  Indices are 32-bit; the structure of a term is that of its first bead.
//   pair lists that hold both (i, j) and (j, i) ("symmetric"): the gradient on bead i is twice the sum over i's own terms,
//   so only the first bead of a term is written: no scatter.
//   FIXED: energies and gradients are accumulated as 64-bit fixed-point integers (integer addition is associative: the
//   result does not depend on the order in which the threads arrive) and converted afterwards.
// ------------------------------------------------------------------------------------------------
constexpr int kSliceWarps = 4, kSliceBlocks = 6;         // of prior_all_kernel; blocks each SM, float (5: 144.7 us instead of 133.5 for 1024 chains of 268 beads, 7: 141.6 with spills)
template <typename T> constexpr int kSliceStage = sizeof(T) == 4 ? 3072 : 2560;    // bytes of half the steps on their way, each warp: four, in float64 two, of a repulsion (1536: 143.8 us instead of 133.5; float64 2304, one: 306 instead of 260)
constexpr int kFixedShift = 36;          // fixed point: 2^-36 resolution, +-1.3e8 range

struct PriorSegments {
    int n;
    int kind[MLCGB_MAX_PRIOR_SEGMENTS], n_params[MLCGB_MAX_PRIOR_SEGMENTS], symmetric[MLCGB_MAX_PRIOR_SEGMENTS];
    int64_t M[MLCGB_MAX_PRIOR_SEGMENTS];                                           // terms
    int64_t vstart[MLCGB_MAX_PRIOR_SEGMENTS + 1];     // per-term lists: first thread of the list (a multiple of 32)
    int64_t steps[MLCGB_MAX_PRIOR_SEGMENTS];                                       // of all slices
    int n_slices[MLCGB_MAX_PRIOR_SEGMENTS];                                        // pair lists in slices (else 0)
    const int32_t *idx[MLCGB_MAX_PRIOR_SEGMENTS];                                  // [order, M]
    const void *params[MLCGB_MAX_PRIOR_SEGMENTS];                                  // [n_params, M]
    const int4 *slices[MLCGB_MAX_PRIOR_SEGMENTS];                                  // [n_slices]
    const int32_t *slice_beads[MLCGB_MAX_PRIOR_SEGMENTS];                          // [n_slices][32]
    const void *offsets[MLCGB_MAX_PRIOR_SEGMENTS], *slice_params[MLCGB_MAX_PRIOR_SEGMENTS];   // [steps][32][4], [n_params][steps][32][4]
};

template <typename T> __device__ __forceinline__ long long to_fixed(T v) { return __double2ll_rn((double)v * (double)(1ll << kFixedShift)); }

template <typename T, bool FIXED> struct Accum;
template <typename T> struct Accum<T, false> {
    using type = T;
    T *e, *g;
    __device__ __forceinline__ void energy(int64_t at, T v) const { atomicAdd(e + at, v); }
    __device__ __forceinline__ void grad3(int64_t at, const V3<T> &v) const { atomic_add3(g, at, v); }
};
template <typename T> struct Accum<T, true> {
    using type = unsigned long long;
    unsigned long long *e, *g;
    __device__ __forceinline__ void energy(int64_t at, T v) const { atomicAdd(e + at, (unsigned long long)to_fixed(v)); }
    __device__ __forceinline__ void grad3(int64_t at, const V3<T> &v) const {
        atomicAdd(g + at * 3, (unsigned long long)to_fixed(v.x));
        atomicAdd(g + at * 3 + 1, (unsigned long long)to_fixed(v.y));
        atomicAdd(g + at * 3 + 2, (unsigned long long)to_fixed(v.z));
    }
};

// a bead: position, and its structure in w (as an integer for float, as a number for double)
__device__ __forceinline__ int structure_of(const float4 &b) { return __float_as_int(b.w); }
__device__ __forceinline__ int structure_of(const double4 &b) { return (int)b.w; }
__device__ __forceinline__ void set_structure(float4 &b, int s) { b.w = __int_as_float(s); }
__device__ __forceinline__ void set_structure(double4 &b, int s) { b.w = (double)s; }
template <typename T, typename P> __device__ __forceinline__ V3<T> xyz(const P &b) { return V3<T>{(T)b.x, (T)b.y, (T)b.z}; }

template <typename T, typename A>
__global__ void __launch_bounds__(256)
prior_begin_kernel(const T *__restrict__ pos, const int64_t *__restrict__ batch, int64_t N, int64_t B, typename Vec4<T>::type *__restrict__ beads,
                   A *__restrict__ sums, int64_t n_sums) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = t; i < N; i += stride) {
        typename Vec4<T>::type b;
        b.x = pos[i * 3]; b.y = pos[i * 3 + 1]; b.z = pos[i * 3 + 2];
        const int64_t s = batch ? batch[i] : 0;
        set_structure(b, s >= 0 && s < B ? (int)s : -1);
        beads[i] = b;
    }
    for (int64_t i = t; i < n_sums; i += stride) sums[i] = A(0);
}

// v summed over runs of consecutive lanes with equal index i, added once per run (every lane calls; i = -1: nothing)
template <typename T, typename A>
__device__ __forceinline__ void run_accumulate(const A &acc, int64_t block0, int32_t i, V3<T> v, int lane) {
    const int32_t prev = __shfl_up_sync(0xffffffffu, i, 1);
    const bool head = lane == 0 || prev != i;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const unsigned above = lane == 31 ? 0u : (heads >> (lane + 1));
    const int run_end = above ? lane + __ffs(above) : 32;   // exclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T x = __shfl_down_sync(0xffffffffu, v.x, o), y = __shfl_down_sync(0xffffffffu, v.y, o), z = __shfl_down_sync(0xffffffffu, v.z, o);
        if (lane + o < run_end) { v.x += x; v.y += y; v.z += z; }
    }
    if (head && i >= 0) acc.grad3(block0 + i, v);
}

// Symmetric pair lists in slices of 32 runs of equal first bead: a lane per bead, four terms of each lane and step.  The terms of a
// slice are stored step by step, [step][lane][4], padded to the longest of its runs with terms of parameter 0 (at a distance that is
// not), so that every load is a full vector and no lane has a bound to check.  The second bead of a term is the slice's base plus a
// 16-bit offset.  Energy and gradient stay in registers: one addition per bead and component, no scatter and no reduction across
// lanes (the reverse terms of the list carry the other half of every pair's gradient).  In the lists of a topology the lanes of a
// slice meet the same second bead at nearly the same step: a gather of positions is one or two cache lines.
// Bound by the stream of terms, 6 bytes each at half of the memory's rate, and by what its warps do meanwhile (29 instructions a term and warp, 60 %
// of the issue slots): of 133.5 us for 72 M terms and three lists of single terms the first and the last launch take 12, the stream alone
// 81, with its arithmetic 94, the single terms 27 more.  With loads two steps ahead in registers 155 (then); with a warp per run in one kernel for all lists (32-bit indices, three 4-byte loads a position, a
// reduction a run) the pair terms alone took 390.
__device__ __forceinline__ float inv_sqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ double inv_sqrt(double x) { return rsqrt(x); }

// A warp's steps on their way from memory: two stages of a few steps each, filled by the copy engine (steps lie one behind the other, so
// a stage is one copy of offsets and one of each parameter), which takes neither issue slots nor the registers that loads ahead did.
template <int KIND, typename T> struct PairStages {
    using V = typename Vec4<T>::type;
    static constexpr int kParams = KIND == 0 ? 2 : 1, kPar = 32 * (int)sizeof(V), kStep = 256 + kParams * kPar;
    static constexpr int kSteps = kSliceStage<T> / kStep >= 4 ? 4 : kSliceStage<T> / kStep >= 2 ? 2 : 1, kBytes = kSteps * kStep;
    static_assert(kBytes <= kSliceStage<T>, "half of a warp's part of the shared memory");
};

// b - a; the first two components in one instruction (142.1 -> 133.5 us for 72 M terms)
__device__ __forceinline__ V3<float> difference(const float4 &b, const float4 &a) {
    const float2 xy = tc::sub2(make_float2(b.x, b.y), make_float2(a.x, a.y));
    return V3<float>{xy.x, xy.y, b.z - a.z};
}
__device__ __forceinline__ V3<double> difference(const double4 &b, const double4 &a) { return V3<double>{b.x - a.x, b.y - a.y, b.z - a.z}; }

template <int KIND, typename T, typename A, typename Bead>
__device__ __forceinline__ void prior_slices(const A &acc, const PriorSegments &seg, int s, int parts, const Bead *__restrict__ beads, int64_t N,
                                             int64_t B, int32_t *status, int block, int blocks, char *ring, uint32_t bars, int &turn, bool &failed) {
    const int lane = threadIdx.x & 31;
    const int64_t units = (int64_t)seg.n_slices[s] * parts;
    const int64_t steps = seg.steps[s], stride = steps * 128;
    const auto *off = (const uint2 *)seg.offsets[s];
    const T *pa = (const T *)seg.slice_params[s];
    for (int64_t w = (int64_t)block * kSliceWarps + (threadIdx.x >> 5); w < units; w += (int64_t)blocks * kSliceWarps) {
        const int slice = (int)(w / parts), part = (int)(w % parts);
        const int4 h = __ldg(seg.slices[s] + slice);             // {first step, steps, base, span}
        const int first = __ldg(seg.slice_beads[s] + (int64_t)slice * 32 + lane), c0 = first < 0 ? ~first : first;    // (~bead: an idle lane)
        const bool bad = h.x < 0 || h.y < 0 || (int64_t)h.x + h.y > steps || h.z < 0 || h.w < 0 || (int64_t)h.z + h.w >= N || c0 >= N;
        if (__any_sync(0xffffffffu, bad)) {
            if (lane == 0) atomicOr(status, (int)kBadIndex);
            continue;
        }
        const Bead b0 = beads[c0];
        const Bead *other = beads + h.z;
        using S = PairStages<KIND, T>;
        using V = typename S::V;
        // (a unit takes every `parts`-th stage: neighbouring warps read neighbouring memory)
        const int all = (h.y + S::kSteps - 1) / S::kSteps, stages = (all - part + parts - 1) / parts;
        if (part >= all) continue;
        T es = T(0);
        float2 es2 = make_float2(0.f, 0.f);
        V3<T> gs{T(0), T(0), T(0)};
        const auto step = [&](const uint2 j, const auto &a, const auto &b) {
            const Bead bj[4] = {other[j.x & 0xffffu], other[j.x >> 16], other[j.y & 0xffffu], other[j.y >> 16]};
            const T pa4[4] = {a.x, a.y, a.z, a.w}, pb4[4] = {b.x, b.y, b.z, b.w};
            V3<T> dr[4];
            T inv_d[4], d2[4], f[4];                              // f: dE/dd / d; of a repulsion without its factor -6
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                dr[u] = difference(bj[u], b0);
                d2[u] = dot(dr[u], dr[u]);
                inv_d[u] = inv_sqrt(d2[u]);
            }
            if constexpr (KIND == 3 && sizeof(T) == 4) {          // two terms an instruction
#pragma unroll
                for (int u = 0; u < 4; u += 2) {
                    const float2 inv = make_float2(inv_d[u], inv_d[u + 1]), q = tc::mul2(make_float2(pa4[u], pa4[u + 1]), inv), rr = tc::mul2(q, q),
                                 ee = tc::mul2(tc::mul2(rr, rr), rr), ff = tc::mul2(tc::mul2(ee, inv), inv);
                    es2 = tc::add2(es2, ee);
                    f[u] = ff.x;
                    f[u + 1] = ff.y;
                }
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if constexpr (KIND == 0) {
                        const T k = pb4[u], x = d2[u] * inv_d[u] - pa4[u];
                        es += k * x * x;
                        f[u] = T(2) * k * x * inv_d[u];
                    } else {
                        const T q = pa4[u] * inv_d[u], rr = q * q, ee = rr * rr * rr;
                        es += ee;
                        f[u] = ee * inv_d[u] * inv_d[u];
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) { gs.x += dr[u].x * f[u]; gs.y += dr[u].y * f[u]; gs.z += dr[u].z * f[u]; }
        };
        const auto fetch = [&](int k) {                          // stage k of this unit, into half (turn + k) & 1
            if (lane != 0 || k >= stages) return;
            const int half = (turn + k) & 1, first_step = (part + k * parts) * S::kSteps, m = h.y - first_step < S::kSteps ? h.y - first_step : S::kSteps;
            const uint32_t to = tc::smem_u32(ring + half * kSliceStage<T>), bar = bars + 8 * half;
            const int64_t from = ((int64_t)h.x + first_step) * 32;
            tc::mbar_expect_bytes(bar, (uint32_t)(m * S::kStep));
            tc::bulk_load(to, off + from, (uint32_t)(m * 256), bar);
#pragma unroll
            for (int q = 0; q < S::kParams; q++)
                tc::bulk_load(to + S::kSteps * (256 + q * S::kPar), (const V *)(pa + q * stride) + from, (uint32_t)(m * S::kPar), bar);
        };
        fetch(0);
        fetch(1);
        for (int k = 0; k < stages; k++) {
            const int half = (turn + k) & 1, m = h.y - (part + k * parts) * S::kSteps;
            // (a copy that does not arrive: what lies there are no offsets.  The other half's is waited for too, so that none is on its way when the block leaves)
            if (!__all_sync(0xffffffffu, tc::mbar_wait(bars + 8 * half, (uint32_t)(turn + k) >> 1 & 1u))) {
                failed = true;
                if (k + 1 < stages) tc::mbar_wait(bars + 8 * (half ^ 1), (uint32_t)(turn + k + 1) >> 1 & 1u);
                return;
            }
            const char *in = ring + half * kSliceStage<T>;
            const auto steps = [&](int u) {
                const V *par = reinterpret_cast<const V *>(in + S::kSteps * 256) + u * 32 + lane;
                step(reinterpret_cast<const uint2 *>(in)[u * 32 + lane], par[0], par[KIND == 0 ? S::kSteps * 32 : 0]);
            };
            if (m >= S::kSteps) {
#pragma unroll
                for (int u = 0; u < S::kSteps; u++) steps(u);
            } else {
                for (int u = 0; u < m; u++) steps(u);
            }
            tc::fence_async_smem();                              // the next copy into this half stays behind the reads of it
            __syncwarp();
            fetch(k + 2);
        }
        turn += stages;
        if constexpr (KIND == 3 && sizeof(T) == 4) es = es2.x + es2.y;
        const int mb = structure_of(b0);
        const bool mine = first >= 0 && mb >= 0;
        if (first >= 0 && mb < 0) atomicOr(status, (int)kBadIndex);
        if (mine) acc.grad3((int64_t)s * N + c0, scale(gs, KIND == 0 ? T(-2) : T(12)));
        const int mb0 = __shfl_sync(0xffffffffu, mb, 0);
        if (__all_sync(0xffffffffu, mb == mb0 && mb >= 0)) {
            es = warp_sum(mine ? es : T(0));
            if (lane == 0) acc.energy((int64_t)s * B + mb0, es);
        } else if (mine) {
            acc.energy((int64_t)s * B + mb, es);
        }
    }
}

// ---- what is made of a list on its first evaluation: 32-bit indices, the parameters of its terms from the tables of bead types, whether
//      a pair list holds the reverse of every term, where its runs of equal first bead begin, and its slices.  A pass over the list
//      for each of gather, starts and slices (two): bound by the memory it streams.  Gathered and sorted by library calls (two sorts
//      of all keys for the reverses) the lists of 1024 chains of 268 beads, 73 M terms, took 17 ms, like this 1.8 with the evaluation.
constexpr int kGatherThreads = 256, kGatherTerms = 8, kChunk = kGatherThreads * kGatherTerms;
struct PriorTables { const void *p[MLCGB_MAX_PRIOR_TABLES]; };

// finaliser of MurmurHash3 (Austin Appleby, public domain): every bit of the input moves every bit of the output
__device__ __forceinline__ uint64_t mix64(uint64_t k) {
    k ^= k >> 33; k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33; k *= 0xc4ceb9fe1a85ec53ull;
    return k ^ k >> 33;
}
__device__ __forceinline__ uint64_t value_bits(float v) { return __float_as_uint(v + 0.f); }           // (-0 and 0 are the same parameter)
__device__ __forceinline__ uint64_t value_bits(double v) { return (uint64_t)__double_as_longlong(v + 0.0); }

// PAIR: `difference` gains the sum over the terms of hash(i, j, parameters) - hash(j, i, parameters), modulo 2^64: zero where the list is
// the same set of terms reversed, and not zero otherwise but for one chance in 2^64; counts[chunk] = runs that begin in it
template <typename T, int ORDER, bool PAIR>
__global__ void __launch_bounds__(kGatherThreads)
prior_gather_kernel(const int64_t *__restrict__ mapping, int64_t M, const int64_t *__restrict__ types, int64_t N, int64_t num_types, int n_params,
                    const __grid_constant__ PriorTables tables, const T *__restrict__ given, int32_t *__restrict__ idx, T *__restrict__ params,
                    unsigned long long *__restrict__ difference, int32_t *__restrict__ counts, int32_t *__restrict__ status) {
    int runs = 0;
    uint64_t diff = 0;
    bool some_bad = false, no_type = false;
    const int64_t t0 = (int64_t)blockIdx.x * kChunk + threadIdx.x;
#pragma unroll 2        // (32 registers, an SM full of warps: four at a time take 47, 72 M terms 545 us instead of 502)
    for (int u = 0; u < kGatherTerms; u++) {
        const int64_t t = t0 + u * kGatherThreads;
        if (t >= M) break;
        int64_t at[ORDER], entry = 0;
#pragma unroll
        for (int o = 0; o < ORDER; o++) at[o] = mapping[(int64_t)o * M + t];
        if (PAIR) runs += t == 0 || mapping[t - 1] != at[0];
#pragma unroll
        for (int o = 0; o < ORDER; o++) {
            const bool there = (uint64_t)at[o] < (uint64_t)N;
            some_bad |= !there;
            if (!there) at[o] = -1;
            idx[(int64_t)o * M + t] = (int32_t)at[o];
        }
        if (!given) {
#pragma unroll
            for (int o = 0; o < ORDER; o++) {
                int64_t ty = at[o] < 0 ? 0 : __ldg(types + at[o]);
                if (ty < 0) ty += num_types;                 // (as indexing a table does)
                const bool there = (uint64_t)ty < (uint64_t)num_types;
                no_type |= !there;
                if (!there) ty = 0;
                entry = entry * num_types + ty;
            }
        }
        uint64_t h = 0;
        for (int q = 0; q < n_params; q++) {
            const T v = given ? given[(int64_t)q * M + t] : __ldg((const T *)tables.p[q] + entry);
            if (!given) params[(int64_t)q * M + t] = v;
            if (PAIR) h = mix64(h + value_bits(v) + 1);
        }
        if (PAIR) {
            const uint64_t i = (uint32_t)at[0], j = (uint32_t)at[1];
            diff += mix64(h ^ (i << 32 | j)) - mix64(h ^ (j << 32 | i));
        }
    }
    if (no_type) atomicOr(status, (int)kBadIndex | (int)kNotThere);
    if (some_bad) {                                          // (reported, and again by the evaluation, which leaves the terms out)
        int word = kBadIndex;
        for (int u = 0; u < kGatherTerms; u++) {
            const int64_t t = t0 + u * kGatherThreads;
            for (int o = 0; t < M && o < ORDER; o++) {
                const int64_t at = mapping[(int64_t)o * M + t];
                if (at >= N || at < -N) word |= kNotThere;
                // (runs of what is written, as run_starts_kernel finds them: none begins between two beads that do not exist)
                if (PAIR && o == 0 && t > 0 && (at < 0 || at >= N)) {
                    const int64_t before = mapping[t - 1];
                    runs -= before != at && (before < 0 || before >= N);
                }
            }
        }
        atomicOr(status, word);
    }
    if constexpr (PAIR) {
        __shared__ int s_runs[kGatherThreads / 32];
        __shared__ uint64_t s_diff[kGatherThreads / 32];
        runs = warp_sum(runs);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) diff += __shfl_xor_sync(0xffffffffu, diff, o);
        if ((threadIdx.x & 31) == 0) { s_runs[threadIdx.x >> 5] = runs; s_diff[threadIdx.x >> 5] = diff; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < kGatherThreads / 32; w++) { runs += s_runs[w]; diff += s_diff[w]; }
            counts[blockIdx.x] = runs;
            if (diff) atomicAdd(difference, (unsigned long long)diff);
        }
    }
}

// exclusive sums of n values by one block of 1024 threads, thread t holding `per` consecutive ones of each round: f(k) the value, g(k, sum before)
template <typename F, typename G>
__device__ __forceinline__ int64_t block_sums_before(int64_t n, F &&f, G &&g) {
    __shared__ int64_t s_warp[32], s_total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t carry = 0;
    for (int64_t k0 = 0; k0 < n; k0 += 1024) {
        const int64_t k = k0 + threadIdx.x;
        const int64_t v = k < n ? f(k) : 0;
        int64_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const int64_t w = s_warp[lane];
            int64_t wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += t;
            }
            s_warp[lane] = wi - w;
            if (lane == 31) s_total = wi;
        }
        __syncthreads();
        if (k < n) g(k, carry + s_warp[warp] + inc - v);
        carry += s_total;
        __syncthreads();
    }
    return carry;
}

__global__ void __launch_bounds__(1024) run_offsets_kernel(const int32_t *__restrict__ counts, int64_t n, const unsigned long long *__restrict__ difference,
                                                           int64_t *__restrict__ before, Publish pub) {
    const int64_t runs = block_sums_before(n, [&](int64_t k) { return (int64_t)counts[k]; }, [&](int64_t k, int64_t v) { before[k] = v; });
    if (threadIdx.x == 0) publish(pub, runs, *difference != 0);
}

// starts[r] = first term of run r (chunks and counts as above)
__global__ void __launch_bounds__(kGatherThreads)
run_starts_kernel(const int32_t *__restrict__ first, int64_t M, const int64_t *__restrict__ before, int64_t *__restrict__ starts) {
    __shared__ int s_warp[kGatherThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t at = before[blockIdx.x];
    for (int u = 0; u < kGatherTerms; u++) {
        const int64_t t = (int64_t)blockIdx.x * kChunk + u * kGatherThreads + threadIdx.x;
        const bool head = t < M && (t == 0 || first[t - 1] != first[t]);
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        if (lane == 0) s_warp[warp] = __popc(heads);
        __syncthreads();
        int mine = __popc(heads & lanemask_lt()), all = 0;
        for (int w = 0; w < kGatherThreads / 32; w++) {
            mine += w < warp ? s_warp[w] : 0;
            all += s_warp[w];
        }
        if (head) starts[at + mine] = t;
        at += all;
        __syncthreads();
    }
}

// The slices of a list (mlcgb_pair_slices), a warp each.  First {longest run, -, least, largest second bead} of every slice: its terms are
// consecutive, whatever their runs.
__global__ void __launch_bounds__(256)
pair_slices_kernel(const int32_t *__restrict__ idx, int64_t M, const int64_t *__restrict__ starts, int64_t n_runs, int64_t n_slices, int4 *__restrict__ slices) {
    const int lane = threadIdx.x & 31;
    for (int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n_slices; w += (int64_t)gridDim.x * (blockDim.x >> 5)) {
        const int64_t run = w * 32 + lane, end = (w + 1) * 32 < n_runs ? starts[(w + 1) * 32] : M;
        const int64_t k0 = run < n_runs ? starts[run] : end, k1 = __shfl_down_sync(0xffffffffu, k0, 1);
        int longest = (int)((lane == 31 ? end : k1) - k0), lo = 0x7fffffff, hi = -0x7fffffff - 1;
        for (int64_t k = __shfl_sync(0xffffffffu, k0, 0) + lane; k < end; k += 32) {
            const int j = idx[M + k];
            lo = min(lo, j);
            hi = max(hi, j);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
        }
        if (lane == 0) slices[w] = make_int4(longest, 0, lo, hi);
    }
}

// first step of every slice; to the host: all steps, lanes without a run times the last slice's steps, least second bead, largest span
__global__ void __launch_bounds__(1024) slices_plan_kernel(const int4 *__restrict__ slices, int64_t n_slices, int64_t n_runs, int64_t *__restrict__ step0, Publish pub) {
    __shared__ int s_low, s_span;
    if (threadIdx.x == 0) { s_low = 0x7fffffff; s_span = 0; }
    int low = 0x7fffffff;
    unsigned span = 0;
    const int64_t total = block_sums_before(
        n_slices,
        [&](int64_t k) {
            const int4 h = slices[k];
            low = min(low, h.z);
            span = max(span, (unsigned)min((int64_t)h.w - h.z, (int64_t)0x7fffffff));
            return (int64_t)((h.x + 3) / 4);
        },
        [&](int64_t k, int64_t v) { step0[k] = v; });
    atomicMin(&s_low, low);
    atomicMax(&s_span, (int)span);
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile int64_t *h = pub.host;
        h[1] = total;
        h[2] = (slices[n_slices - 1].x + 3) / 4 * (32 * n_slices - n_runs);
        h[3] = s_low;
        h[4] = s_span;
        __threadfence_system();
        h[0] = pub.seq;
    }
}

// The steps of a slice: the terms of 32 runs, read run by run in rows of 32 and turned over in shared memory.
template <typename T> constexpr int kPackWarps = sizeof(T) == 4 ? 8 : 4;
template <typename T> constexpr int kPackPitch = sizeof(T) == 4 ? 36 : 34;      // (128-bit reads along a row by eight lanes meet no bank twice)
template <typename T>
__global__ void __launch_bounds__(kPackWarps<T> * 32)
pair_slices_pack_kernel(const int32_t *__restrict__ idx, const T *__restrict__ params, int n_params, int64_t M, const int64_t *__restrict__ starts,
                        int64_t n_runs, int64_t n_slices, int64_t steps, const int64_t *__restrict__ step0, int4 *__restrict__ slices,
                        int32_t *__restrict__ beads, uint2 *__restrict__ offsets, typename Vec4<T>::type *__restrict__ out) {
    using V = typename Vec4<T>::type;
    __shared__ __align__(32) T s_tile[kPackWarps<T>][32][kPackPitch<T>];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto tile = s_tile[warp];
    for (int64_t w = (int64_t)blockIdx.x * kPackWarps<T> + warp; w < n_slices; w += (int64_t)gridDim.x * kPackWarps<T>) {
        const int64_t run = w * 32 + lane, end = (w + 1) * 32 < n_runs ? starts[(w + 1) * 32] : M;
        const bool mine = run < n_runs;
        const int64_t begin = starts[w * 32];
        const int at = (int)((mine ? starts[run] : end) - begin);                  // of this lane's run, from the slice's first term
        const int next = __shfl_down_sync(0xffffffffu, at, 1), len = (lane == 31 ? (int)(end - begin) : next) - at;
        const int4 h = slices[w];
        const int n = (h.x + 3) >> 2, base = h.z;
        const int filler = (mine ? idx[M + begin + at] : idx[M + begin]) - base;     // (no run: the slice's first second bead)
        const int64_t first = step0[w];
        for (int q = -1; q < n_params; q++) {                                    // the second beads, then the parameters
            for (int g0 = 0; g0 < n; g0 += 8) {
                __syncwarp();
#pragma unroll 8
                for (int r = 0; r < 32; r++) {
                    const int a = __shfl_sync(0xffffffffu, at, r), l = __shfl_sync(0xffffffffu, len, r), c = 4 * g0 + lane;
                    const int fill = __shfl_sync(0xffffffffu, filler, r);
                    const int64_t k = begin + a + c;
                    if (q < 0) reinterpret_cast<int *>(&tile[r][0])[lane] = c < l ? idx[M + k] - base : fill;
                    else tile[r][lane] = c < l ? params[(int64_t)q * M + k] : T(0);
                }
                __syncwarp();
                for (int g = g0; g < n && g < g0 + 8; g++) {
                    const int64_t to = (first + g) * 32 + lane;
                    if (q < 0) {
                        const int4 j = reinterpret_cast<const int4 *>(&tile[lane][0])[g - g0];
                        offsets[to] = make_uint2((uint32_t)j.x | (uint32_t)j.y << 16, (uint32_t)j.z | (uint32_t)j.w << 16);
                    } else {
                        out[(int64_t)q * steps * 32 + to] = reinterpret_cast<const V *>(&tile[lane][0])[g - g0];
                    }
                }
            }
        }
        beads[run] = mine ? idx[begin + at] : ~idx[begin];
        __syncwarp();
        if (lane == 0) slices[w] = make_int4((int)first, n, base, h.w - base);
    }
}

// All other terms, one per thread; a warp never mixes lists.  Short lists (about one term of a kind per bead): bound by the latency
// of their double-precision chains and by the scattered additions.  Terms of a chain that follow one another in the list share beads
// with their neighbours: a lane hands what it has for the beads that the next lane's term starts with over to that lane, so that a
// torsion adds to one bead instead of four (47 -> 33 us for the three lists of 1024 chains of 268 beads, the shorter torsion included).
template <typename T, typename A>
__device__ __forceinline__ void prior_terms(const A &acc, const PriorSegments &seg, const typename Vec4<T>::type *__restrict__ beads, int64_t N, int64_t B,
                                            int32_t *status, int block, int blocks) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)blocks * blockDim.x;
    const int64_t vtotal = seg.vstart[seg.n];
    for (int64_t vbase = (int64_t)block * blockDim.x + threadIdx.x - lane; vbase < vtotal; vbase += stride) {
        int s = 0;
        while (s + 1 < seg.n && vbase >= seg.vstart[s + 1]) s++;               // warp-uniform: lists start on warp boundaries
        const int kind = seg.kind[s];
        const int64_t M = seg.M[s], t = vbase - seg.vstart[s] + lane;
        const int32_t *idx = seg.idx[s];
        const T *params = (const T *)seg.params[s];
        const int64_t e_row = (int64_t)s * B, g_block = (int64_t)s * N;
        bool valid = t < M;
        int32_t i0 = 0, i1 = 0, i2 = 0, i3 = 0;
        if (valid) {
            i0 = idx[t];
            i1 = idx[M + t];
            if (kind == 1 || kind == 2) i2 = idx[2 * M + t];
            if (kind == 2) i3 = idx[3 * M + t];
            if (i0 < 0 || i0 >= N || i1 < 0 || i1 >= N || i2 < 0 || i2 >= N || i3 < 0 || i3 >= N) {
                valid = false;
                atomicOr(status, (int)kBadIndex);
            }
        }
        int32_t mb = 0;
        T e = T(0);
        V3<T> g0{T(0), T(0), T(0)};
        V3<double> g[4] = {};
        const bool listed = valid;
        if (valid) {
            const auto b0 = beads[i0], b1 = beads[i1];
            mb = structure_of(b0);
            if (mb < 0) {
                valid = false;
                mb = 0;
                atomicOr(status, (int)kBadIndex);
            } else if (kind == 0) {
                e = (T)bond_term(xyz<double>(b0), xyz<double>(b1), (double)params[t], (double)params[M + t], g[1]);
                g[0] = scale(g[1], -1.0);
            } else if (kind == 3) {
                const V3<T> dr = sub(xyz<T>(b1), xyz<T>(b0));
                const T d = sqrt(dot(dr, dr));
                const T q = params[t] / d;
                const T rr = q * q;
                e = rr * rr * rr;
                const V3<T> g1 = scale(dr, T(-6) * e / d / d);
                if (seg.symmetric[s]) {
                    g0 = scale(g1, T(-2));                       // the reverse term of the list adds the same again
                } else {
                    acc.grad3(g_block + i1, g1);
                    g0 = scale(g1, T(-1));
                }
            } else if (kind == 1) {
                e = (T)angle_term(xyz<double>(b0), xyz<double>(b1), xyz<double>(beads[i2]), (double)params[t], (double)params[M + t], g[0], g[2]);
                g[1] = V3<double>{-g[0].x - g[2].x, -g[0].y - g[2].y, -g[0].z - g[2].z};
            } else {
                e = (T)torsion_term(xyz<double>(b0), xyz<double>(b1), xyz<double>(beads[i2]), xyz<double>(beads[i3]), params, M, t,
                                    (seg.n_params[s] - 1) / 2, g);
            }
        }
        if (kind == 3) {
            run_accumulate<T>(acc, g_block, valid ? i0 : -1, g0, lane);
        } else {
            const bool chain = listed && i1 == i0 + 1 && (kind == 0 || i2 == i0 + 2) && (kind != 2 || i3 == i0 + 3);
            const unsigned chains = __ballot_sync(0xffffffffu, chain);
            const int32_t before = __shfl_up_sync(0xffffffffu, i0, 1);
            const bool link = lane > 0 && chain && ((chains >> (lane - 1)) & 1) && before + 1 == i0;
            const unsigned links = __ballot_sync(0xffffffffu, link);
            const bool last = lane == 31 || !((links >> (lane + 1)) & 1);
            const auto hand_over = [&](const V3<double> &from, V3<double> &to) {
                const double x = __shfl_up_sync(0xffffffffu, from.x, 1), y = __shfl_up_sync(0xffffffffu, from.y, 1), z = __shfl_up_sync(0xffffffffu, from.z, 1);
                if (link) { to.x += x; to.y += y; to.z += z; }
            };
            if (kind == 2) hand_over(g[3], g[2]);
            if (kind != 0) hand_over(g[2], g[1]);
            hand_over(g[1], g[0]);
            if (listed) {
                acc.grad3(g_block + i0, narrow<T>(g[0]));
                if (last) {
                    acc.grad3(g_block + i1, narrow<T>(g[1]));
                    if (kind != 0) acc.grad3(g_block + i2, narrow<T>(g[2]));
                    if (kind == 2) acc.grad3(g_block + i3, narrow<T>(g[3]));
                }
            }
        }
        // energy: one addition per warp when the whole warp sits in one structure
        const int64_t mb0 = __shfl_sync(0xffffffffu, mb, 0);
        const bool same = __all_sync(0xffffffffu, !valid || mb == mb0);
        const bool lane0_valid = __shfl_sync(0xffffffffu, (int)valid, 0) != 0;
        if (same && lane0_valid) {
            const T sum = warp_sum(e);
            if (lane == 0) acc.energy(e_row + mb0, sum);
        } else if (valid) {
            acc.energy(e_row + mb, e);
        }
    }
}

// Single terms in a launch of their own, where they are the larger part or the only one: without the stages' shared memory, which is taken from
// the cache that their beads come through.  256 chains of 268 beads, us, in prior_all_kernel's blocks : like this: every pair one way (9 M terms, not
// sliced) float32 331 : 278, float64 421 : 289; bonds, angles and dihedrals alone, 1024 chains, 40.6 : 39.0 and 55.4 : 45.1.
template <typename T, bool FIXED>
__global__ void __launch_bounds__(256)
prior_terms_kernel(const __grid_constant__ PriorSegments seg, const typename Vec4<T>::type *__restrict__ beads, int64_t N, int64_t B,
                   typename Accum<T, FIXED>::type *__restrict__ energy, typename Accum<T, FIXED>::type *__restrict__ grad, int32_t *__restrict__ status) {
    const Accum<T, FIXED> acc{energy, grad};
    pdl_wait();
    pdl_launch_dependents();
    prior_terms<T>(acc, seg, beads, N, B, status, (int)blockIdx.x, (int)gridDim.x);
}

// All terms: blocks of slices and blocks of single terms, dealt evenly, so that every SM holds both: the slices use the issue slots that the
// chains of double-precision operations leave.  In launches of their own the two hardly met (a launch starts when the last block of the
// one before has, whatever the former allows): 143.5 -> 141 us for the lists of 1024 chains of 268 beads when the launches were made one.
template <typename T, bool FIXED>
__global__ void __launch_bounds__(kSliceWarps * 32, sizeof(T) == 4 ? kSliceBlocks : 4)
prior_all_kernel(const __grid_constant__ PriorSegments seg, int parts, int term_blocks, const typename Vec4<T>::type *__restrict__ beads, int64_t N, int64_t B,
                 typename Accum<T, FIXED>::type *__restrict__ energy, typename Accum<T, FIXED>::type *__restrict__ grad, int32_t *__restrict__ status) {
    __shared__ __align__(128) char s_ring[kSliceWarps][2 * kSliceStage<T>];
    __shared__ uint64_t s_bar[kSliceWarps][2];
    const Accum<T, FIXED> acc{energy, grad};
    // term blocks before this one, and whether this is one
    const int before = (int)((int64_t)blockIdx.x * term_blocks / gridDim.x), upto = (int)(((int64_t)blockIdx.x + 1) * term_blocks / gridDim.x);
    if (upto > before) {
        pdl_wait();
        prior_terms<T>(acc, seg, beads, N, B, status, before, term_blocks);
        return;
    }
    char *const ring = s_ring[threadIdx.x >> 5];
    const uint32_t bars = tc::smem_u32(s_bar[threadIdx.x >> 5]);      // this warp's stages have arrived
    if ((threadIdx.x & 31) == 0) {
        tc::mbar_init(bars, 1);
        tc::mbar_init(bars + 8, 1);
        tc::fence_async_smem();
    }
    __syncwarp();
    int turn = 0;                                                     // stages this warp has used
    bool failed = false;
    pdl_wait();
    const int block = (int)blockIdx.x - before, blocks = (int)gridDim.x - term_blocks;
    for (int s = 0; s < seg.n; s++) {
        if (seg.n_slices[s] == 0 || failed) continue;
        if (seg.kind[s] == 0) prior_slices<0, T>(acc, seg, s, parts, beads, N, B, status, block, blocks, ring, bars, turn, failed);
        else prior_slices<3, T>(acc, seg, s, parts, beads, N, B, status, block, blocks, ring, bars, turn, failed);
    }
    if (failed) atomicOr(status, (int)kTensorWait);
}

template <typename T, typename A> __device__ __forceinline__ T sum_value(A v) {
    if constexpr (std::is_same<A, unsigned long long>::value) return (T)((double)(long long)v * (1.0 / (double)(1ll << kFixedShift)));
    else return (T)v;
}

// sums -> energies, gradients (sign +1) or forces (sign -1) of each list, and their totals where they are asked for
template <typename T, typename A>
__global__ void __launch_bounds__(256)
prior_finish_kernel(const A *__restrict__ sums, int n, int64_t N, int64_t B, T sign, T *__restrict__ energy, T *__restrict__ grad,
                    T *__restrict__ total_energy, T *__restrict__ total_grad) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, nB = (int64_t)n * B;
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < B + 3 * N; i += stride) {
        const bool e = i < B;
        const int64_t at = e ? i : i - B, step = e ? B : 3 * N;
        const A *in = e ? sums : sums + nB;
        T *out = e ? energy : grad, *tot = e ? total_energy : total_grad;
        T sum = T(0);
        for (int s = 0; s < n; s++) {
            T v = sum_value<T>(in[s * step + at]);
            if (!e) v *= sign;
            out[s * step + at] = v;
            sum += v;
        }
        if (tot) tot[at] = sum;
    }
}

template <typename T>
static int prior_launch(int kind, const void *pos, const int64_t *mapping, const int64_t *mapping_batch, const void *params,
                        int n_params, int64_t M, int64_t N, int64_t B, void *energy, void *grad, int32_t *status,
                        cudaStream_t st) {
    const int grid = grid_for(M, 256, 16);
#define GO(K) prior_kernel<T, K><<<grid, 256, 0, st>>>((const T *)pos, mapping, mapping_batch, (const T *)params, n_params, M, N, B, (T *)energy, (T *)grad, status)
    switch (kind) {
        case 0: GO(0); break;
        case 1: GO(1); break;
        case 2: GO(2); break;
        default: GO(3); break;
    }
#undef GO
    return check_launch();
}

}  // namespace mlcgb

using namespace mlcgb;

extern "C" int mlcgb_prior_terms(int kind, const void *pos, int dtype, const int64_t *mapping, const int64_t *mapping_batch,
                                 const void *params, int n_params, int64_t M, int64_t N, int64_t B, void *energy, void *grad,
                                 int32_t *status, void *stream) {
    TimelineScope timeline_scope("prior_terms", stream);
    if (kind < 0 || kind > 3 || M < 0 || N < 0 || B < 0 || !status) return MLCGB_E_ARG;
    if (M == 0) return MLCGB_OK;
    if (!pos || !mapping || !mapping_batch || !params || !energy) return MLCGB_E_ARG;
    const int need = kind == 3 ? 1 : (kind == 2 ? 3 : 2);
    if (n_params < need || (kind == 2 && (n_params - 1) % 2 != 0)) return MLCGB_E_ARG;
    return MLCGB_DISPATCH_DTYPE(dtype, [&] {
        return prior_launch<scalar_t>(kind, pos, mapping, mapping_batch, params, n_params, M, N, B, energy, grad, status,
                                      (cudaStream_t)stream);
    });
}

static inline size_t prior_bead_bytes(int64_t N, int dtype) { return ((size_t)N * (dtype == MLCGB_F32 ? 16 : 32) + 255) / 256 * 256; }

extern "C" size_t mlcgb_prior_list_workspace_bytes(int64_t M) {
    if (M < 0) return 0;
    return 256 + (size_t)((M + kChunk - 1) / kChunk) * 16;
}

extern "C" int mlcgb_prior_list_make(const int64_t *mapping, int order, int64_t M, const int64_t *types, int64_t N, int64_t num_types, int n_params,
                                     const void *const *tables, int dtype, const void *given, int32_t *idx, void *params, void *workspace,
                                     size_t workspace_bytes, int64_t *host_out, int32_t *status, void *stream) {
    TimelineScope timeline_scope("prior_list", stream);
    if (order < 2 || order > 4 || M < 0 || N < 0 || n_params < 0 || !status || (host_out && order != 2)) return MLCGB_E_ARG;
    if (n_params > MLCGB_MAX_PRIOR_TABLES && tables) return MLCGB_E_LIMIT;
    if (host_out) host_out[0] = host_out[1] = host_out[2] = 0;
    if (M == 0) return MLCGB_OK;
    if (!mapping || !idx || (!tables && n_params && !given) || (tables && (!types || !params || num_types < 1))) return MLCGB_E_ARG;
    if (host_out && (!workspace || workspace_bytes < mlcgb_prior_list_workspace_bytes(M) || ((uintptr_t)workspace & 7))) return MLCGB_E_WORKSPACE;
    PriorTables t = {};
    for (int q = 0; tables && q < n_params; q++)
        if (!(t.p[q] = tables[q])) return MLCGB_E_ARG;
    auto st = (cudaStream_t)stream;
    const int64_t chunks = (M + kChunk - 1) / kChunk;
    if (chunks >= (int64_t)1 << 31) return MLCGB_E_LIMIT;
    auto *difference = (unsigned long long *)workspace;
    auto *before = (int64_t *)((char *)workspace + 256);
    auto *counts = (int32_t *)(before + chunks);
    Publish pub;
    if (host_out) {
        if (int rc = publish_begin(&pub)) return rc;
        pub.pending = status;
        cudaMemsetAsync(difference, 0, 8, st);
    }
    int rc = MLCGB_DISPATCH_DTYPE(dtype, [&] {
        const auto *in = tables ? nullptr : (const scalar_t *)given;
        const bool rows = tables || given;
        auto go = [&](auto kern) {
            kern<<<(unsigned)chunks, kGatherThreads, 0, st>>>(mapping, M, types, N, num_types, rows ? n_params : 0, t, in, idx, (scalar_t *)params, difference, counts, status);
        };
        if (order == 2 && host_out) go(prior_gather_kernel<scalar_t, 2, true>);
        else if (order == 2) go(prior_gather_kernel<scalar_t, 2, false>);
        else if (order == 3) go(prior_gather_kernel<scalar_t, 3, false>);
        else go(prior_gather_kernel<scalar_t, 4, false>);
        return check_launch();
    });
    if (rc || !host_out) return rc;
    run_offsets_kernel<<<1, 1024, 0, st>>>(counts, chunks, difference, before, pub);
    if ((rc = check_launch()) || (rc = publish_wait(pub, st))) return rc;
    host_out[0] = pub.host[1];
    host_out[1] = pub.host[2] == 0;
    host_out[2] = pub.host[3];
    return MLCGB_OK;
}

extern "C" int mlcgb_prior_list_starts(const int32_t *first, int64_t M, const void *workspace, size_t workspace_bytes, int64_t *starts, void *stream) {
    if (M < 0) return MLCGB_E_ARG;
    if (M == 0) return MLCGB_OK;
    if (!first || !workspace || !starts) return MLCGB_E_ARG;
    if (workspace_bytes < mlcgb_prior_list_workspace_bytes(M)) return MLCGB_E_WORKSPACE;
    run_starts_kernel<<<(unsigned)((M + kChunk - 1) / kChunk), kGatherThreads, 0, (cudaStream_t)stream>>>(first, M, (const int64_t *)((const char *)workspace + 256), starts);
    return check_launch();
}

extern "C" int mlcgb_pair_slices(const int32_t *idx, const void *params, int dtype, int n_params, int64_t M, const int64_t *starts, int64_t n_runs,
                                 int64_t steps, const int64_t *step0, int32_t *slices, int32_t *beads, uint16_t *offsets, void *slice_params,
                                 void *stream) {
    if (!idx || !starts || !slices || M <= 0 || n_runs <= 0 || M >= (int64_t)1 << 31) return MLCGB_E_ARG;
    if (slice_params && (!params || n_params < 1 || !step0 || !beads || !offsets || steps <= 0)) return MLCGB_E_ARG;
    const int64_t n = (n_runs + 31) / 32;
    auto st = (cudaStream_t)stream;
    if (!slice_params) {
        pair_slices_kernel<<<grid_for(n, 8, 16), 256, 0, st>>>(idx, M, starts, n_runs, n, (int4 *)slices);
        return check_launch();
    }
    return MLCGB_DISPATCH_DTYPE(dtype, [&] {
        pair_slices_pack_kernel<scalar_t><<<grid_for(n, kPackWarps<scalar_t>, 16), kPackWarps<scalar_t> * 32, 0, st>>>(
            idx, (const scalar_t *)params, n_params, M, starts, n_runs, n, steps, step0, (int4 *)slices, beads, (uint2 *)offsets,
            (typename Vec4<scalar_t>::type *)slice_params);
        return check_launch();
    });
}

extern "C" int mlcgb_pair_slices_plan(const int32_t *slices, int64_t n_slices, int64_t n_runs, int64_t *step0, int64_t *host_out, void *stream) {
    if (!slices || !step0 || !host_out || n_slices <= 0 || n_runs <= 32 * (n_slices - 1) || n_runs > 32 * n_slices) return MLCGB_E_ARG;
    Publish pub;
    if (int rc = publish_begin(&pub)) return rc;
    slices_plan_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>((const int4 *)slices, n_slices, n_runs, step0, pub);
    if (int rc = check_launch()) return rc;
    if (int rc = publish_wait(pub, (cudaStream_t)stream)) return rc;
    for (int i = 0; i < 4; i++) host_out[i] = pub.host[1 + i];
    return MLCGB_OK;
}

extern "C" size_t mlcgb_prior_eval_workspace_bytes(int n_lists, int64_t N, int64_t B, int dtype) {
    if (n_lists <= 0 || N < 0 || B < 0) return 0;
    return prior_bead_bytes(N, dtype) + (size_t)n_lists * (size_t)(3 * N + B) * sizeof(unsigned long long);
}

extern "C" int mlcgb_prior_eval(int n_lists, const mlcgb_prior_list *lists, const void *pos, int dtype, const int64_t *batch, int64_t N,
                                int64_t B, void *energy, void *grad, int negate, void *total_energy, void *total_grad, int fixed_point,
                                void *workspace, size_t workspace_bytes, int32_t *status, void *stream) {
    TimelineScope timeline_scope("prior_eval", stream);
    if (n_lists < 0 || n_lists > MLCGB_MAX_PRIOR_SEGMENTS || N < 0 || B < 0 || !status) return MLCGB_E_ARG;
    if (n_lists == 0 || N + B == 0) return MLCGB_OK;
    if (!lists || !pos || !energy || !grad || !workspace || N >= ((int64_t)1 << 31) || B >= ((int64_t)1 << 31)) return MLCGB_E_ARG;
    if (workspace_bytes < mlcgb_prior_eval_workspace_bytes(n_lists, N, B, dtype)) return MLCGB_E_WORKSPACE;
    PriorSegments seg;
    seg.n = n_lists;
    int64_t v = 0, r = 0;
    for (int i = 0; i < n_lists; i++) {
        const mlcgb_prior_list &l = lists[i];
        const int need = l.kind == 3 ? 1 : (l.kind == 2 ? 3 : 2);
        if (l.kind < 0 || l.kind > 3 || l.M < 0 || l.n_params < need || (l.kind == 2 && (l.n_params - 1) % 2 != 0)) return MLCGB_E_ARG;
        seg.kind[i] = l.kind;
        seg.n_params[i] = l.n_params;
        seg.symmetric[i] = (l.kind == 0 || l.kind == 3) && l.symmetric ? 1 : 0;
        seg.M[i] = l.M;
        seg.idx[i] = l.idx;
        seg.params[i] = l.params;
        const bool sliced = seg.symmetric[i] && l.n_slices > 0;
        if (l.M > 0 && !sliced && (!l.idx || !l.params)) return MLCGB_E_ARG;
        if (sliced) {
            if (!l.slices || !l.slice_beads || !l.offsets || !l.slice_params || l.steps <= 0 || l.n_slices >= ((int64_t)1 << 31)) return MLCGB_E_ARG;
            if (((uintptr_t)l.slices | (uintptr_t)l.offsets | (uintptr_t)l.slice_params) & 31) return MLCGB_E_ARG;
        }
        seg.slices[i] = (const int4 *)l.slices;
        seg.slice_beads[i] = l.slice_beads;
        seg.offsets[i] = l.offsets;
        seg.slice_params[i] = l.slice_params;
        seg.steps[i] = l.steps;
        seg.n_slices[i] = sliced ? (int)l.n_slices : 0;
        seg.vstart[i] = v;
        if (seg.n_slices[i] > r) r = seg.n_slices[i];
        v += sliced ? 0 : (l.M + 31) / 32 * 32;
    }
    seg.vstart[n_lists] = v;
    auto st = (cudaStream_t)stream;
    const int64_t n_sums = (int64_t)n_lists * (3 * N + B);
    const auto go = [&](auto tag, auto fixed) {
        using T = decltype(tag);
        constexpr bool FIXED = decltype(fixed)::value;
        using A = typename Accum<T, FIXED>::type;
        auto *beads = (typename Vec4<T>::type *)workspace;
        auto *sums = (A *)((char *)workspace + prior_bead_bytes(N, dtype));
        A *se = sums, *sg = sums + (int64_t)n_lists * B;
        prior_begin_kernel<T, A><<<grid_for(N > n_sums / 4 ? N : n_sums / 4, 256, 8), 256, 0, st>>>((const T *)pos, batch, N, B, beads, sums, n_sums);
        // A slice is cut into parts until the chip holds a warp wherever it has room for one, into two at least (the last round of warps is shorter
        // then) and into no more than an average slice has stages of copies, or sixteen: a part without a stage looks up its beads for nothing.
        // us of device time, float32 / float64, aiming at 16, 24, 48 and 96 warps each SM:
        //   chains          32 x 268    64 x 268    96 x 268    200 x 268   400 x 268    1024 x 73   1024 x 268
        //   16              14.4, 20.6  17.9, 28.4  20.6, 38.7  35.8, 66.3  66.4, 126.6  25.1, 39.0  136.4, 269.4
        //   24              20.1, 22.5  20.5, 26.5  21.8, 34.4  34.9, 63.6  59.8, 113.3  25.1, 39.0  136.2, 269.6
        //   48              20.5, 23.0  26.2, 29.0  22.8, 36.9  36.2, 63.8  60.7, 111.1  32.6, 45.1  136.4, 269.5
        //   96              20.5, 23.2  28.3, 31.2  32.9, 44.9  42.7, 69.7  69.8, 116.9  39.8, 60.2  134.0, 260.1 (the only one with two parts here)
        const int64_t want = r ? (kSliceWarps * kSliceBlocks * (int64_t)kNumSM + r - 1) / r : 1;
        int64_t stages = 1, in_slices = 0;
        for (int i = 0; i < n_lists; i++) {
            const int64_t a_stage = seg.kind[i] == 0 ? PairStages<0, T>::kSteps : PairStages<3, T>::kSteps;
            if (!seg.n_slices[i]) continue;
            in_slices += 128 * seg.steps[i];
            stages = std::max(stages, (seg.steps[i] + seg.n_slices[i] * a_stage - 1) / (seg.n_slices[i] * a_stage));
        }
        const bool alone = v > in_slices;                // (prior_terms_kernel; beside a larger stream they cost least among its blocks)
        const int parts = (int)std::min(std::min(std::max(want, (int64_t)2), (int64_t)16), stages), slice_blocks = r ? grid_for(r * parts, kSliceWarps, 96) : 0,
                  term_blocks = v && !alone ? grid_for(v, kSliceWarps * 32, 96) : 0;
        if (v && alone) launch_pdl(prior_terms_kernel<T, FIXED>, dim3(grid_for(v, 256, 16)), dim3(256), 0, st, seg, beads, N, B, se, sg, status);
        if (slice_blocks + term_blocks)
            launch_pdl(prior_all_kernel<T, FIXED>, dim3(slice_blocks + term_blocks), dim3(kSliceWarps * 32), 0, st, seg, parts, term_blocks, beads, N, B, se, sg, status);
        launch_pdl(prior_finish_kernel<T, A>, dim3(grid_for(B + 3 * N, 256, 8)), dim3(256), 0, st, sums, n_lists, N, B, (T)(negate ? -1 : 1), (T *)energy,
                   (T *)grad, (T *)total_energy, (T *)total_grad);
        return check_launch();
    };
    return MLCGB_DISPATCH_DTYPE(dtype, [&] {
        return fixed_point ? go(scalar_t(0), std::true_type{}) : go(scalar_t(0), std::false_type{});
    });
}

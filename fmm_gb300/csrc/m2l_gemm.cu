// M2L as dense matrix products grouped by displacement (exact-coefficient
// modes; the reference's per-pair M2L is src/fmm.F90:826-882).
//
// Octree cells are cubes on a grid: the centre displacement of two cells is an
// integer multiple D of the smaller cell's half-width, and a pair's
// reduced-basis M2L operator depends only on D, the level difference and the
// pair's expansion order q.  The far pairs are sorted by that key; each group
// shares one operator G ((q+1)^2 x (q+1)^2, from the restricted tensor T of
// the group's displacement, computed once per group in FP64), and the group's
// pairs are the columns of one product C = G W.  FP32 products run on the
// tensor cores (tcgen05, kind::tf32 with operands split into two TF32 parts,
// three products per term, FP32 accumulators in tensor memory), FP64 products
// too, in fixed point (m2l_tc64.cuh), and either on request on the CUDA cores
// as register-tiled blocks.  Per-pair columns go to a buffer in target-sorted
// order and are summed per target with compensated sums.
//
// Where the reference's 32-bit tensor coefficients wrap (orders 2p > 10), its
// tensors are not harmonic: the FP64 product then runs over all Cartesian
// components (`full`), with the reference's closed form once per group.
//
// The basis functions are even or odd in x, y and z, so that displacements that
// differ in signs alone have the same operator up to the signs of its rows and
// columns.  Where the groups are small, those of the eight octants are taken
// together (`mirrored`): with up to eight times the pairs per operator the
// products' columns are filled and an eighth of the operators is built.
//
// Units: per-node weights w'_s = w^_s / h_j^|s|, per-target locals
// L'_f = h_i^(|f|+1) L_f, tensor T(D_c) at the displacement in units of the
// coarser cell's half-width h_c; then G_fs = a^(|f|+1) b^|s| T_{s+f}(D_c)
// with a = h_i/h_c, b = h_j/h_c (powers of two, at most 1), so all operands
// are O(1) and the FP32 products stay in range.
#include <algorithm>

#include <cub/cub.cuh>
#include <thrust/iterator/transform_iterator.h>

#include <cstdlib>
#include <cstring>

#include "internal.h"
#include "m2l_basis.cuh"
#include "m2l_size.h"
#include "m2l_tc64.cuh"
#include "umma.cuh"

namespace fmm {

namespace {

inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

constexpr int kFallback = 63;            // key code of pairs without a grid displacement
// Key layout (46 bits, so the radix sort needs 6 digit passes): level
// difference + 31 (6 bits) | order (4) | |Dx|, |Dy|, |Dz| (11 bits each) |
// octant (3): bit d set where D_d < 0.
constexpr int kKeyBits = 46;
constexpr int kKeyBitsImages = 56;       // with the target's depth and the source's image (5 bits each) above
constexpr int64_t kDMax = (1 << 11) - 1;
constexpr int kOctants = 8;
constexpr int kTaskCols = 512;           // pairs (columns) per product block
constexpr int kGemmThreads = 128;        // 16 row groups x 8 column groups
constexpr int kTcRows = 128;             // tensor-core MMA M: operator rows f per half
constexpr int kTcPairs = 256;            // tensor-core MMA N: pairs per task

// Operator halves of 128 rows f for order q (two above order 10).
__host__ __device__ __forceinline__ int tc_halves(int q) { return (q + 1) * (q + 1) > kTcRows ? 2 : 1; }

__global__ void k_far_targets(int M, const int32_t* __restrict__ off, int32_t* __restrict__ tgt) {
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= M) return;
    for (int q = off[i] + lane; q < off[i + 1]; q += 32) tgt[q] = i;
}

// w'_s = w^_s / h^|s| per node (h the node's half-width).
// (rows of ld >= nr entries, zero padded)
template <typename R>
__global__ void k_scale_weights(int M, int nr, int ld, const double* __restrict__ wred, const double* __restrict__ h,
                                R* __restrict__ wsc) {
    // warp per node: lane j holds ih^j (the same sequential product for every
    // component of order j), components across the lanes
    const int node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (node >= M) return;
    const double ih = 1.0 / h[node];
    double pw = 1.0;
    for (int u = 0; u < min(lane, 2 * kMaxP); ++u) pw *= ih;
    for (int s0 = 0; s0 < ld; s0 += 32) {
        const int s = s0 + lane;
        int k = 0;
        while ((k + 1) * (k + 1) <= s) ++k;  // order of reduced component s
        const double sc = __shfl_sync(0xffffffffu, pw, min(k, 31));
        if (s < ld) wsc[(size_t)node * ld + s] = s < nr ? (R)(wred[(size_t)node * nr + s] * sc) : (R)0;
    }
}

// Group key of every far pair: level difference, expansion order and integer
// displacement in units of the smaller half-width; pairs off the grid (or
// with out-of-range fields) get unique keys of their own (code 63 | index).
// With FP32 node data (chi: centre hi parts; clo: low parts, half-width in
// w) the displacement is formed from the double-float centres on the FP32
// pipe; its error (a few 1e-8 relative of the displacement, up to ~1e-4 cell
// units at the largest encodable displacement) stays far below the 1e-3
// tolerance of the integer test.  Without them, FP64 with a 1e-6 tolerance.
// Cell centres are rounded, so pairs of a group differ from its displacement by
// some 1e-16 of the coordinates (dev: the largest difference, in units of the
// smaller half-width, where FP64 pairs are asked for it).
// Sources in periodic images are displaced by their image's shift, the same in
// bohr but not in units of their cells: only pairs of one image and one level
// share an operator.
__global__ void k_m2l_keys(int64_t nfar, const TreeDev t, const int32_t* __restrict__ tgt, int p, int oclass,
                           const float4* __restrict__ chi, const float4* __restrict__ clo,
                           uint64_t* __restrict__ keys, int32_t* __restrict__ vals, int* __restrict__ dev) {
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const unsigned warp = __ballot_sync(0xffffffffu, q < nfar);  // whole warps are launched
    if (q >= nfar) return;
    const int i = tgt[q], j = src_node(t, t.far_src[q]);
    const int ord = t.far_ord ? min((int)t.far_ord[q], p) : p;
    // half-widths are the root's divided by powers of two: 1/h times an
    // integer multiple of h stays within rounding of that integer
    float rx, ry, rz, ex, ey, ez, tol;
    if (chi) {
        const float4 ci = chi[i], cj = chi[j], li = clo[i], lj = clo[j];
        const float ihf = 1.0f / fminf(li.w, lj.w);
        const float dx = ((ci.x - cj.x) + (li.x - lj.x)) * ihf, dy = ((ci.y - cj.y) + (li.y - lj.y)) * ihf,
                    dz = ((ci.z - cj.z) + (li.z - lj.z)) * ihf;
        rx = rintf(dx);
        ry = rintf(dy);
        rz = rintf(dz);
        ex = fabsf(dx - rx);
        ey = fabsf(dy - ry);
        ez = fabsf(dz - rz);
        tol = 1e-3f;
    } else {
        const double ihf = 1.0 / fmin(t.r[i], t.r[j]);
        const double dx = (t.cx[i] - t.cx[j]) * ihf, dy = (t.cy[i] - t.cy[j]) * ihf, dz = (t.cz[i] - t.cz[j]) * ihf;
        const double Rx = rint(dx), Ry = rint(dy), Rz = rint(dz);
        rx = (float)Rx;
        ry = (float)Ry;
        rz = (float)Rz;
        ex = (float)fabs(dx - Rx);
        ey = (float)fabs(dy - Ry);
        ez = (float)fabs(dz - Rz);
        tol = 1e-6f;
    }
    const int dl = t.depth[i] - t.depth[j];
    const int oc = (ord + oclass - 1) / oclass;  // order class: the group takes its pairs' highest order
    const float lim = (float)kDMax;
    const bool grid = ex < tol && ey < tol && ez < tol && fabsf(rx) <= lim && fabsf(ry) <= lim && fabsf(rz) <= lim &&
                      dl > -31 && dl < 31;
    uint64_t key;
    if (grid)
        key = ((uint64_t)(dl + 31) << 40) | ((uint64_t)oc << 36) | ((uint64_t)fabsf(rx) << 25) |
              ((uint64_t)fabsf(ry) << 14) | ((uint64_t)fabsf(rz) << 3) |
              (uint64_t)((rx < 0.0f ? 1 : 0) | (ry < 0.0f ? 2 : 0) | (rz < 0.0f ? 4 : 0)) |
              (t.nimg > 1 ? (uint64_t)(t.depth[i] | (src_image(t, t.far_src[q]) << 5)) << kKeyBits : 0);
    else
        key = ((uint64_t)kFallback << 40) | ((uint64_t)q << 3);
    keys[q] = key;
    vals[q] = (int32_t)q;
    if (dev) {  // largest deviation from the grid, as the bits of a float >= 0
        const int e = __reduce_max_sync(warp, grid ? __float_as_int(fmaxf(ex, fmaxf(ey, ez))) : 0);
        if ((threadIdx.x & 31) == 0 && e > *(volatile int*)dev) atomicMax(dev, e);
    }
}

// A group's order: the highest of its pairs' orders (gq starts at zero).  Warp
// per group and slice of its pairs (blockIdx.y), for large groups: the
// displacements of the deepest level have as many pairs as there are leaves, and
// a warp that reads them all keeps the tensors waiting (300,000 particles, 3,400
// pairs a group: a call 8.23 -> 8.14 ms, with sliced row offsets).  With few
// slices the extra launch costs more than it saves.
__global__ void k_group_orders(int ng, const int32_t* __restrict__ gstart, const int32_t* __restrict__ svals,
                               const TreeDev t, int p, int32_t* __restrict__ gq) {
    const int g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (g >= ng) return;
    int q = 0;
    for (int k = gstart[g] + 32 * blockIdx.y + lane; k < gstart[g + 1]; k += 32 * gridDim.y)
        q = max(q, t.far_ord ? min((int)t.far_ord[svals[k]], p) : p);
    q = __reduce_max_sync(0xffffffffu, q);
    if (lane == 0 && q > 0) atomicMax(&gq[g], q);
}

// Slices of the groups' pairs for the kernels with a warp per group: some eight
// steps of a warp each at the mean.
inline unsigned group_slices(int64_t nf, int ng) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(64, nf / ng / 256));
}

// One warp per group: restricted tensor T(D_c) of orders <= 2q in FP64 by the
// Hermite recursion (two level buffers in shared memory), stored as R, with
// the group's unit ratios a, b.  Mirrored groups: at the displacement
// of octant 0 (skeys: the pairs' keys in group order).
template <typename R, bool HAVE_Q>
__global__ void __launch_bounds__(128) k_group_tensor(int ngroups, bool mirrored, const uint64_t* __restrict__ skeys,
                                                      const int32_t* __restrict__ gstart,
                                                      const int32_t* __restrict__ svals,
                                                      const int32_t* __restrict__ tgt, const TreeDev t, int p,
                                                      int ldT, R* __restrict__ gT, int32_t* __restrict__ gq,
                                                      float2* __restrict__ gab) {
    extern __shared__ double smg[];
    const int N = 2 * p, nTr = rbase(N + 1);
    int2* rule = reinterpret_cast<int2*>(smg);
    // the rules' factors (as integers, their conversions took a quarter of the
    // FP64 pipe's time: 56,000 groups, orders to 12, 2.9 -> 2.2 ms)
    double* coef = smg + nTr;
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* TA = smg + 2 * nTr + wib * (2 * nTr + N + 1);
    double* TB = TA + nTr;
    double* gsh = TB + nTr;
    for (int e = threadIdx.x; e < nTr; e += blockDim.x) {
        const int2 ru = restricted_rule(e);
        rule[e] = ru;
        coef[e] = (double)(ru.y >> 16);
    }
    __syncthreads();
    const int g = blockIdx.x * (blockDim.x >> 5) + wib;
    if (g >= ngroups) return;
    const int oct = mirrored ? (int)(skeys[gstart[g]] & (kOctants - 1)) : 0;
    const int pos0 = svals[gstart[g]];
    const int i = tgt[pos0], j = t.far_src[pos0];
    int q = 0;
    if (HAVE_Q) {  // (k_group_orders)
        q = gq[g];
    } else {
        for (int k = gstart[g] + lane; k < gstart[g + 1]; k += 32)
            q = max(q, t.far_ord ? min((int)t.far_ord[svals[k]], p) : p);
        for (int off = 16; off > 0; off >>= 1) q = max(q, __shfl_xor_sync(0xffffffffu, q, off));
    }
    const double hi = t.r[i], hj = t.r[j], hc = fmax(hi, hj);
    const double X = ((oct & 1) ? -1.0 : 1.0) * (t.cx[i] - t.cx[j]) / hc,
                 Y = ((oct & 2) ? -1.0 : 1.0) * (t.cy[i] - t.cy[j]) / hc,
                 Z = ((oct & 4) ? -1.0 : 1.0) * (t.cz[i] - t.cz[j]) / hc;
    const int Nq = 2 * q;
    const double r2 = X * X + Y * Y + Z * Z;
    const double rinv = 1.0 / sqrt(r2), rinv2 = rinv * rinv;
    if (lane <= Nq) {
        double v = rinv, c = 1.0, k = -1.0;
        for (int jj = 1; jj <= lane; ++jj) {
            v *= rinv2;
            c *= k;  // -(2 jj - 1)
            k -= 2.0;
        }
        gsh[lane] = c * v;
    }
    __syncwarp();
    double* A = TA;
    double* B = TB;
    if (lane == 0) A[0] = gsh[Nq];
    __syncwarp();
    for (int lev = Nq - 1; lev >= 0; --lev) {
        const int lim = rbase(Nq - lev + 1);
        for (int e = lane; e < lim; e += 32) {
            double v;
            if (e == 0) {
                v = gsh[lev];
            } else {
                const int2 ru = rule[e];
                const int dir = ru.x >> 16, cnt = ru.y >> 16;
                const double crd = dir == 0 ? X : (dir == 1 ? Y : Z);
                v = crd * A[ru.x & 0xffff];
                if (cnt > 0) v += coef[e] * A[ru.y & 0xffff];
            }
            B[e] = v;
        }
        __syncwarp();
        double* tmp = A;
        A = B;
        B = tmp;
    }
    R* out = gT + (size_t)g * ldT;
    for (int e = lane; e < rbase(Nq + 1); e += 32) out[e] = (R)A[e];
    if (lane == 0) {
        if (!HAVE_Q) gq[g] = q;
        gab[g] = make_float2((float)(hi / hc), (float)(hj / hc));
    }
}

// Tasks of up to `cols` pairs of one group: counts, then (group, first
// column).  Tensor-core tasks (cols kTcTasks: kTcPairs pairs and one operator
// half each, (group, 2 x first column + half); kD64Tasks, kD64FullTasks: the
// FP64 products' kD64Pairs pairs and one part, (group, 4 x first column + part)).
constexpr int kTcTasks = -1, kD64Tasks = -2, kD64FullTasks = -3;

__device__ __forceinline__ int task_pairs(int cols) { return cols > 0 ? cols : (cols == kTcTasks ? kTcPairs : kD64Pairs); }
__device__ __forceinline__ int task_parts(int cols, int q) {
    return cols > 0 ? 1 : (cols == kTcTasks ? tc_halves(q) : d64_parts(q, cols == kD64FullTasks));
}

__global__ void k_task_counts(int ng, int cols, const int32_t* __restrict__ gq, const int32_t* __restrict__ gstart,
                              int32_t* __restrict__ tcnt) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g > ng) return;
    if (g == ng) {
        tcnt[g] = 0;
        return;
    }
    const int n = gstart[g + 1] - gstart[g], w = task_pairs(cols);
    tcnt[g] = (n + w - 1) / w * task_parts(cols, gq[g]);
}

__global__ void k_fill_tasks(int ng, int cols, const int32_t* __restrict__ gq, const int32_t* __restrict__ gstart,
                             const int32_t* __restrict__ toff, int2* __restrict__ tasks) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    const int n = toff[g + 1] - toff[g], w = task_pairs(cols), h = task_parts(cols, gq[g]);
    const int mul = cols > 0 ? 1 : (cols == kTcTasks ? 2 : 4);
    for (int k = 0; k < n; ++k) tasks[toff[g] + k] = make_int2(g, mul * w * (k / h) + k % h);
}

// Shared-memory plan of the product kernel (elements of R unless noted).
template <typename R, int CPT>
struct GemmSmem {
    static constexpr int TN = 8 * CPT;                // columns per tile
    static constexpr int VS = 16 / (int)sizeof(R);    // weights per 16-byte load
    int nrmax, rmmax, nTr;
    size_t off_dec, off_pow, off_T, off_col, off_G, bytes;
    __host__ __device__ GemmSmem(int p) {
        nrmax = (p + 1) * (p + 1);
        rmmax = 16 * ((nrmax + 15) / 16);
        nTr = rbase(2 * p + 1);
        size_t o = 0;
        off_dec = o;
        o += sizeof(int) * nrmax;
        o = (o + 15) & ~(size_t)15;
        off_pow = o;
        o += sizeof(R) * 32;
        off_T = o;
        o += sizeof(R) * nTr;
        o = (o + 15) & ~(size_t)15;
        off_col = o;  // the source nodes of the task's pairs
        o += sizeof(int) * kTaskCols;
        off_G = o;
        o += sizeof(R) * (size_t)((nrmax + VS - 1) / VS * VS) * rmmax;
        bytes = o;
    }
};

// Row stride of the per-node weights: (p+1)^2 rounded up to 16 bytes.
template <typename R>
__host__ __device__ constexpr int wsc_ld(int nr) {
    return (nr + 16 / (int)sizeof(R) - 1) / (16 / (int)sizeof(R)) * (16 / (int)sizeof(R));
}

template <typename R>
struct Vec;
template <>
struct Vec<float> {
    using T = float4;
    __device__ static __forceinline__ void get(const T& v, float* o) {
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
};
template <>
struct Vec<double> {
    using T = double2;
    __device__ static __forceinline__ void get(const T& v, double* o) {
        o[0] = v.x; o[1] = v.y;
    }
};

// RT consecutive operator rows as 16-byte loads where the alignment allows
// (row blocks of RT elements start at multiples of RT).
template <typename R, int RT>
__device__ __forceinline__ void load_rows(const R* p, R (&v)[RT]) {
    constexpr int VS = 16 / (int)sizeof(R);
    if constexpr (RT % VS == 0) {
        using V = typename Vec<R>::T;
#pragma unroll
        for (int k = 0; k < RT / VS; ++k) Vec<R>::get(reinterpret_cast<const V*>(p)[k], v + VS * k);
    } else if constexpr (sizeof(R) == 4 && RT % 2 == 0) {
#pragma unroll
        for (int k = 0; k < RT / 2; ++k) {
            const float2 x = reinterpret_cast<const float2*>(p)[k];
            v[2 * k] = x.x;
            v[2 * k + 1] = x.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < RT; ++k) v[k] = p[k];
    }
}

// Columns [c_begin, c_begin + kTaskCols) of one group: C = G W for tiles of
// TN pairs; thread (rg, cg) owns rows rg*RT + k (k < RT) and columns
// cg*CPT .. cg*CPT + CPT - 1 of each tile.  G^T sits in shared memory
// (s-major); each thread streams its columns' weights straight from global
// memory (L1/L2-resident), VS consecutive s per 16-byte load, so the tile loop
// needs no block barrier.
template <typename R, int RT, int CPT>
__device__ __forceinline__ void gemm_task(const GemmSmem<R, CPT>& L, char* sm, int c_begin, int tcols, int nrq,
                                          int cnt, int gs, const int32_t* __restrict__ psrc,
                                          const R* __restrict__ wsc, int ldw, R* __restrict__ gout, int ldo) {
    constexpr int TN = GemmSmem<R, CPT>::TN;
    constexpr int VS = GemmSmem<R, CPT>::VS;
    constexpr int RM = 16 * RT;
    using V = typename Vec<R>::T;
    const int tid = threadIdx.x;
    const int rg = tid & 15, cg = tid >> 4;
    const int* dec = reinterpret_cast<const int*>(sm + L.off_dec);
    const R* apow = reinterpret_cast<const R*>(sm + L.off_pow);
    const R* bpow = apow + 16;
    const R* Tsh = reinterpret_cast<const R*>(sm + L.off_T);
    R* G = reinterpret_cast<R*>(sm + L.off_G);
    int* csrc = reinterpret_cast<int*>(sm + L.off_col);
    const int nrv = (nrq + VS - 1) / VS * VS;
    const int c_end = min(cnt, c_begin + tcols);
    // the task's columns: source nodes (loaded once)
    for (int i = tid; i < c_end - c_begin; i += kGemmThreads) csrc[i] = psrc[gs + c_begin + i];
    // operator G^T (s-major, RM rows per s; rows f >= nrq and s >= nrq zero)
    for (int e = tid; e < nrv * RM; e += kGemmThreads) {
        const int s = e / RM, f = e - s * RM;
        R v = (R)0;
        if (f < nrq && s < nrq) {
            const int cs = dec[s], cf = dec[f];
            const int x = (cs & 0xff) + (cf & 0xff), y = ((cs >> 8) & 0xff) + ((cf >> 8) & 0xff),
                      z = ((cs >> 16) & 0xff) + ((cf >> 16) & 0xff);
            v = apow[(cf >> 24) + 1] * bpow[cs >> 24] * Tsh[ridx(x, y, z)];
        }
        G[e] = v;
    }
    __syncthreads();
    for (int cb = c_begin; cb < c_end; cb += TN) {
        int pos[CPT];
        const V* wp[CPT];
#pragma unroll
        for (int l = 0; l < CPT; ++l) {
            const int c = cb + cg * CPT + l;
            pos[l] = c < c_end ? c : -1;  // result row: the pair's place in its group
            wp[l] = pos[l] >= 0 ? reinterpret_cast<const V*>(wsc + (size_t)csrc[c - c_begin] * ldw) : nullptr;
        }
        R acc[RT][CPT];
#pragma unroll
        for (int k = 0; k < RT; ++k)
#pragma unroll
            for (int l = 0; l < CPT; ++l) acc[k][l] = (R)0;
        const R* Gp = G + rg * RT;  // this thread's RT consecutive rows
        for (int s0 = 0; s0 < nrv; s0 += VS) {
            R wv[CPT][VS];
#pragma unroll
            for (int l = 0; l < CPT; ++l) {
                if (wp[l]) {
                    Vec<R>::get(wp[l][s0 / VS], wv[l]);
                } else {
#pragma unroll
                    for (int u = 0; u < VS; ++u) wv[l][u] = (R)0;
                }
            }
#pragma unroll
            for (int u = 0; u < VS; ++u) {
                R gv[RT];
                load_rows<R, RT>(Gp + (s0 + u) * RM, gv);
#pragma unroll
                for (int k = 0; k < RT; ++k)
#pragma unroll
                    for (int l = 0; l < CPT; ++l) acc[k][l] = fma(gv[k], wv[l][u], acc[k][l]);
            }
        }
        // the group's rows are ldo = (q+1)^2 rounded up to kRowUnit entries
        // each (zeros above the pair's order)
#pragma unroll
        for (int l = 0; l < CPT; ++l) {
            if (pos[l] >= 0) {
                R* o = gout + (size_t)pos[l] * ldo;
#pragma unroll
                for (int k = 0; k < RT; ++k) {
                    const int f = rg * RT + k;
                    if (f < nrq)
                        o[f] = acc[k][l];
                    else if (f < ldo)
                        o[f] = (R)0;
                }
                for (int f = RM + rg; f < ldo; f += 16) o[f] = (R)0;
            }
        }
    }
}

// Result rows: group g's rows start at rowbase[g] x kRowUnit entries, one
// row of (q+1)^2 rounded up to kRowUnit entries per pair in group order.
__host__ __device__ __forceinline__ int row_len(int q, bool full = false) {
    return (d64_rows(q, full) + kRowUnit - 1) / kRowUnit * kRowUnit;
}

// tcols: pairs per task (at most kTaskCols); tasks of order < qmin are left
// to the tensor-core kernel.
template <typename R, int CPT>
__global__ void __launch_bounds__(kGemmThreads) k_m2l_gemm(const int2* __restrict__ tasks, int tcols, int qmin,
                                                           int p,
                                                           const int32_t* __restrict__ gstart,
                                                           const int32_t* __restrict__ gq,
                                                           const float2* __restrict__ gab, const R* __restrict__ gT,
                                                           int ldT, const int32_t* __restrict__ psrc,
                                                           const R* __restrict__ wsc, R* __restrict__ out,
                                                           const int64_t* __restrict__ rowbase) {
    extern __shared__ __align__(16) char sm_gemm[];
    const GemmSmem<R, CPT> L(p);
    const int nr = (p + 1) * (p + 1);
    const int2 task = tasks[blockIdx.x];
    const int g = task.x;
    const int q = gq[g], nrq = (q + 1) * (q + 1);
    if (q < qmin) return;
    const int gs = gstart[g], cnt = gstart[g + 1] - gs;
    int* dec = reinterpret_cast<int*>(sm_gemm + L.off_dec);
    R* apow = reinterpret_cast<R*>(sm_gemm + L.off_pow);
    R* bpow = apow + 16;
    R* Tsh = reinterpret_cast<R*>(sm_gemm + L.off_T);
    for (int e = threadIdx.x; e < nrq; e += kGemmThreads) dec[e] = qcomp(e);
    if (threadIdx.x < 16) {
        const float2 ab = gab[g];
        R a = (R)1, b = (R)1;
        for (int u = 0; u < (int)threadIdx.x; ++u) {
            a *= (R)ab.x;
            b *= (R)ab.y;
        }
        apow[threadIdx.x] = a;
        bpow[threadIdx.x] = b;
    }
    const int nTq = rbase(2 * q + 1);
    for (int e = threadIdx.x; e < nTq; e += kGemmThreads) Tsh[e] = gT[(size_t)g * ldT + e];
    __syncthreads();
    const int rt = (nrq + 15) / 16;
    switch (rt) {
#define FMM_GEMM_CASE(K)                                                                                     \
    case K:                                                                                                  \
        gemm_task<R, K, CPT>(L, sm_gemm, task.y, tcols, nrq, cnt, gs, psrc, wsc, wsc_ld<R>(nr),     \
                             out + (size_t)rowbase[g] * kRowUnit, row_len(q));                                      \
        break;
        FMM_GEMM_CASE(1)
        FMM_GEMM_CASE(2)
        FMM_GEMM_CASE(3)
        FMM_GEMM_CASE(4)
        FMM_GEMM_CASE(5)
        FMM_GEMM_CASE(6)
        FMM_GEMM_CASE(7)
        FMM_GEMM_CASE(8)
        FMM_GEMM_CASE(9)
        FMM_GEMM_CASE(10)
        FMM_GEMM_CASE(11)
#undef FMM_GEMM_CASE
        default:
            break;
    }
}

// ---------------------------------------------------------------------------
// Tensor-core product.  A task is up to 256 pairs of one group and one half
// of its operator: D = G W^T with G the operator half (f x s, M = 128 rows
// f), W the pairs' weights (pairs x s, N = the pairs rounded up to 16: small
// groups take a part of the tensor cores' time) and K = (q+1)^2
// in chunks of 8 (one MMA K step).  Both operands are split into TF32 parts,
// x = hi + lo, and D accumulates G_hi W_hi + G_hi W_lo + G_lo W_hi in FP32
// (the dropped G_lo W_lo and the rounding of the parts leave about 2^-22 of
// each term).  The parts are prepared once in global memory in the operand
// layout: per node the weights, per group the operator, chunk by chunk.
// Warp roles in a persistent block (one per SM):
//   warps 0-1  producers: per chunk, one bulk (TMA) copy of the operator
//              chunk and 16-byte cp.async gathers of the 256 pairs' weights
//              into a ring of shared-memory stages, completing on the
//              stage's full mbarrier; a stage is refilled once the MMAs that
//              read it have committed to its empty mbarrier;
//   warp 2     one thread issues the MMAs into one of two tensor-memory
//              accumulators (256 columns each) and commits the finished task;
//   warps 3+   epilogue (four per tensor-memory sub-partition, each a
//              quarter of the columns): each reads its 32 lanes (rows f),
//              32 columns (pairs) per wait, and writes, per pair, 32
//              consecutive entries of the pair's result row (one aligned
//              128-byte line), then frees the accumulator.
// The two accumulators let the epilogue of one task overlap the MMAs of the
// next.  Orders above 10 ((q+1)^2 > 128 rows f) have two operator halves,
// each a task of its own over the same pairs.
constexpr int kTcKC = 8;           // reduced components per chunk (one MMA K step)
constexpr int kTcStages = 8;
constexpr int kTcProducers = 64;   // warps 0-1
constexpr int kTcMmaWarp = 2;
constexpr int kTcEpiWarps = 16;    // warps 3 .. 2 + kTcEpiWarps
constexpr int kTcThreads = 32 * (3 + kTcEpiWarps);
constexpr int kTcEpiBatch = 2;     // tensor-memory loads (16 columns each) per wait
constexpr uint32_t kTcCols = 512;  // two accumulators of kTcPairs columns
constexpr long long kTcWaitCycles = 4000000000LL;  // about 2 s at 2 GHz

// Float offset of element (r, k) in a K-major, unswizzled chunk kTcKC wide:
// core matrices of 8 rows x 4 elements (128 bytes), K-adjacent ones 128 bytes
// apart (LBO), row groups kTcKC / 4 * 128 bytes apart (SBO).
__host__ __device__ constexpr int tc_off(int r, int k) {
    return (r >> 3) * (kTcKC * 8) + (k >> 2) * 32 + (r & 7) * 4 + (k & 3);
}
static_assert(tc_off(9, 6) == 64 + 32 + 4 + 2, "operand layout: row groups of 8, K groups of 4");

struct TcSmem {
    static constexpr int g_floats = kTcRows * kTcKC;   // one TF32 part of an operator chunk
    static constexpr int w_floats = kTcPairs * kTcKC;  // one TF32 part of a weight chunk
    static constexpr size_t stage_bytes = sizeof(float) * 2 * (g_floats + w_floats);
    static constexpr size_t off_bar = kTcStages * stage_bytes;
    // full[S], empty[S], acc_full[2], acc_empty[2]
    static constexpr size_t off_tmem = off_bar + sizeof(uint64_t) * (2 * kTcStages + 4);
    static constexpr size_t bytes = off_tmem + 16;
};

// Parities of component c (packed x, y, z): bit d set where the power is odd.
// The component changes sign between octant 0 and octant o where
// component_flips(c) & o has an odd number of bits.
__device__ __forceinline__ int component_flips(int c) {
    return (c & 1) | ((c >> 7) & 2) | ((c >> 14) & 4);
}

// Per-node weights as TF32 parts, chunk by chunk: [chunk][hi KC | lo KC].
// octants = 8 (mirrored groups): a copy for each octant, as its pairs' operator
// of octant 0 wants them.
__global__ void k_split_weights(int64_t total, int octants, int nr, int ldw, int ldk, const float* __restrict__ wsc,
                                float* __restrict__ wsp) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t node = e / ldk;
        const int s = (int)(e - node * ldk);
        const float v = s < nr ? wsc[node * ldw + s] : 0.0f;
        float h, l;
        umma::split_tf32(v, h, l);
        float* o = wsp + node * octants * 2 * ldk + (s / kTcKC) * 2 * kTcKC + (s % kTcKC);
        const int flips = octants > 1 && s < nr ? component_flips(qcomp(s)) : 0;
        for (int k = 0; k < octants; ++k, o += 2 * ldk) {
            const bool neg = __popc(flips & k) & 1;
            o[0] = neg ? -h : h;
            o[kTcKC] = neg ? -l : l;
        }
    }
}

// Rows of each group in units of kRowUnit entries (scanned into rowbase).
__global__ void k_row_sizes(int ng, bool full, const int32_t* __restrict__ gstart, const int32_t* __restrict__ gq,
                            int64_t* __restrict__ rsz) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g > ng) return;
    rsz[g] = g < ng ? (int64_t)(gstart[g + 1] - gstart[g]) * (row_len(gq[g], full) / kRowUnit) : 0;
}

// Row of every far pair, indexed in target order (svals maps group order to
// target order), in units of kRowUnit entries.  Warp per group and slice of its
// pairs (blockIdx.y).
__global__ void k_row_offsets(int ng, bool full, const int32_t* __restrict__ gstart, const int32_t* __restrict__ gq,
                              const int64_t* __restrict__ rowbase, const int32_t* __restrict__ svals,
                              int32_t* __restrict__ roff) {
    const int g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (g >= ng) return;
    const int lane = threadIdx.x & 31, u = row_len(gq[g], full) / kRowUnit;
    for (int k = gstart[g] + 32 * blockIdx.y + lane; k < gstart[g + 1]; k += 32 * gridDim.y)
        roff[svals[k]] = (int32_t)(rowbase[g] + (int64_t)(k - gstart[g]) * u);  // (m2l_rows_fit)
}

// Source node of every far pair in group order; mirrored groups: 8 x node +
// octant, the copy of the weights.
__global__ void k_pair_sources(int64_t nf, bool mirrored, const uint64_t* __restrict__ skeys,
                               const int32_t* __restrict__ svals, const TreeDev t, int32_t* __restrict__ psrc) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= nf) return;
    const int j = src_node(t, t.far_src[svals[k]]);
    psrc[k] = mirrored ? kOctants * j + (int)(skeys[k] & (kOctants - 1)) : j;
}

// Key of a mirrored group: the pair key without its octant.
struct MirroredKey {
    __host__ __device__ __forceinline__ uint64_t operator()(uint64_t key) const { return key >> 3; }
};

// Size in floats of a group's split operator (halves x chunks x (hi + lo) x
// 128 x KC).
__global__ void k_gop_sizes(int ng, const int32_t* __restrict__ gq, int64_t* __restrict__ sz) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g > ng) return;
    if (g == ng) {
        sz[g] = 0;
        return;
    }
    const int q = gq[g], nrq = (q + 1) * (q + 1), nch = (nrq + kTcKC - 1) / kTcKC;
    sz[g] = (int64_t)tc_halves(q) * nch * 2 * kTcRows * kTcKC;
}

// Block per group: G_fs = a^(|f|+1) b^|s| T_{f+s}(D_c) split into TF32 parts,
// written half by half and chunk by chunk in the operand layout:
// [half][chunk][hi 128 x KC][lo 128 x KC] (half h: rows f = 128 h ..).
__global__ void __launch_bounds__(256) k_group_operator(int ldT, const float* __restrict__ gT,
                                                        const int32_t* __restrict__ gq,
                                                        const float2* __restrict__ gab,
                                                        const int64_t* __restrict__ goff, int g0, int64_t gop_base,
                                                        float* __restrict__ gop) {
    __shared__ int dec[(kMaxP + 1) * (kMaxP + 1)];
    __shared__ float apow[32], bpow[32];
    __shared__ float Tsh[1 + 3 * (2 * kMaxP) * (2 * kMaxP + 1) / 2];
    const int g = g0 + blockIdx.x;
    const int q = gq[g];
    const int nrq = (q + 1) * (q + 1), nch = (nrq + kTcKC - 1) / kTcKC, nrow = tc_halves(q) * kTcRows;
    for (int e = threadIdx.x; e < nrq; e += blockDim.x) dec[e] = qcomp(e);
    if (threadIdx.x < 32) {
        const float2 ab = gab[g];
        float a = 1.0f, b = 1.0f;
        for (int u = 0; u < (int)threadIdx.x; ++u) {
            a *= ab.x;
            b *= ab.y;
        }
        apow[threadIdx.x] = a;
        bpow[threadIdx.x] = b;
    }
    const int nTq = rbase(2 * q + 1);
    for (int e = threadIdx.x; e < nTq; e += blockDim.x) Tsh[e] = gT[(size_t)g * ldT + e];
    __syncthreads();
    float* out = gop + (goff[g] - gop_base);
    // consecutive threads write consecutive floats of a (half, chunk) block:
    // pos inverts tc_off(r, k) = (r/8) 64 + (k/4) 32 + (r%8) 4 + k%4
    constexpr int BLK = kTcRows * kTcKC;
    const int nblk = (nrow / kTcRows) * nch;
    for (int e = threadIdx.x; e < nblk * BLK; e += blockDim.x) {
        const int blk = e / BLK, pos = e - blk * BLK;
        const int half = blk / nch, ch = blk - half * nch;
        const int n = half * kTcRows + (pos >> 6) * 8 + ((pos & 31) >> 2);
        const int s = ch * kTcKC + ((pos >> 5) & 1) * 4 + (pos & 3);
        float v = 0.0f;
        if (n < nrq && s < nrq) {
            const int cs = dec[s], cf = dec[n];
            const int x = (cs & 0xff) + (cf & 0xff), y = ((cs >> 8) & 0xff) + ((cf >> 8) & 0xff),
                      z = ((cs >> 16) & 0xff) + ((cf >> 16) & 0xff);
            v = apow[(cf >> 24) + 1] * bpow[cs >> 24] * Tsh[ridx(x, y, z)];
        }
        float h, l;
        umma::split_tf32(v, h, l);
        float* o = out + (size_t)blk * 2 * BLK + pos;
        o[0] = h;
        o[BLK] = l;
    }
}

// Columns of a task's MMAs: its pairs rounded up to the instruction's step.
__device__ __forceinline__ int tc_columns(int cnt) { return (cnt + 15) & ~15; }

// Sources of a producer thread's rows 8 (rg0 + k * producer warps) + rsub of
// task t (-1: none, a row of zeros).
template <int RG>
__device__ __forceinline__ void tc_load_rows(int t, const int2* __restrict__ tasks, const int32_t* __restrict__ gstart,
                                             const int32_t* __restrict__ psrc, int rg0, int rsub, int (&r)[RG]) {
    const int2 tk = tasks[t];
    const int gs = gstart[tk.x] + (tk.y >> 1), cnt = min(kTcPairs, gstart[tk.x + 1] - gs);
#pragma unroll
    for (int k = 0; k < RG; ++k) {
        const int pr = 8 * (rg0 + (kTcProducers / 32) * k) + rsub;
        r[k] = pr < cnt ? psrc[gs + pr] : -1;
    }
}

__global__ void __launch_bounds__(kTcThreads, 1) k_m2l_tc(const int2* __restrict__ tasks, int ntasks, bool mirrored,
                                                         const int32_t* __restrict__ gstart,
                                                         const int32_t* __restrict__ gq,
                                                         const int64_t* __restrict__ goff, int64_t gop_base,
                                                         const float* __restrict__ gop,
                                                         const int32_t* __restrict__ psrc,
                                                         const float* __restrict__ wsp, int ldk,
                                                         float* __restrict__ out,
                                                         const int64_t* __restrict__ rowbase,
                                                         int* __restrict__ err) {
    extern __shared__ __align__(1024) char sm_tc[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint64_t* full = reinterpret_cast<uint64_t*>(sm_tc + TcSmem::off_bar);
    uint64_t* empty = full + kTcStages;
    uint64_t* acc_full = empty + kTcStages;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm_tc + TcSmem::off_tmem);
    if (warp == 0) {
        umma::tmem_alloc(tslot, kTcCols);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        for (int st = 0; st < kTcStages; ++st) {
            umma::mbar_init(&full[st], kTcProducers + 1);  // producers' cp.async arrivals + the bulk copy's
            umma::mbar_init(&empty[st], 1);
        }
        for (int a = 0; a < 2; ++a) {
            umma::mbar_init(&acc_full[a], 1);
            umma::mbar_init(&acc_empty[a], kTcEpiWarps);  // one arrival per epilogue warp
        }
        umma::mbar_fence_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;
    bool ok = true;
    if (warp < kTcProducers / 32) {
        // ---- producers.  Each gather instruction covers one 8-row group x
        // (hi, lo) x two 16-byte pieces, which spreads its 512 bytes over all
        // shared-memory banks; a thread keeps its 16 rows' source nodes (-1:
        // no pair) in registers, loaded one task ahead.
        const int pt = tid, plane = tid & 31;
        const int part = plane >> 4, j = (plane >> 3) & 1, rsub = plane & 7;
        constexpr int RG = kTcPairs / 8 / (kTcProducers / 32);  // row groups per thread
        const int rg0 = pt >> 5;
        const uint64_t keep = umma::l2_evict_last();  // the weights stay in L2 beside the result stream
        uint32_t u = 0;
        int task = blockIdx.x;
        int rows[RG], nrows[RG];
        if (task < ntasks) tc_load_rows<RG>(task, tasks, gstart, psrc, rg0, rsub, rows);
        while (task < ntasks && ok) {
            const int g = tasks[task].x, q = gq[g];
            const int nch = ((q + 1) * (q + 1) + kTcKC - 1) / kTcKC;
            const int cols = tc_columns(min(kTcPairs, gstart[g + 1] - gstart[g] - (tasks[task].y >> 1)));
            const int next = task + gridDim.x;
            if (next < ntasks) tc_load_rows<RG>(next, tasks, gstart, psrc, rg0, rsub, nrows);  // in flight
            // the task's operator half
            const float* G = gop + (goff[g] - gop_base) + (size_t)(tasks[task].y & 1) * nch * 2 * TcSmem::g_floats;
            for (int ch = 0; ch < nch; ++ch, ++u) {
                const int st = (int)(u % kTcStages);
                if (u >= (uint32_t)kTcStages &&
                    !umma::mbar_wait(&empty[st], ((u / kTcStages) - 1) & 1, kTcWaitCycles)) {
                    ok = false;
                    break;
                }
                float* Gs = reinterpret_cast<float*>(sm_tc + (size_t)st * TcSmem::stage_bytes);
                float* Ws = Gs + 2 * TcSmem::g_floats;
                if (pt == 0) {
                    constexpr uint32_t gb = sizeof(float) * 2 * TcSmem::g_floats;
                    umma::mbar_arrive_expect_tx(&full[st], gb);
                    umma::bulk_g2s(Gs, G + (size_t)ch * 2 * TcSmem::g_floats, gb, &full[st]);
                }
                float* dst0 = Ws + part * TcSmem::w_floats + 4 * j * 8 + rsub * 4;  // tc_off(8 rg + rsub, 4 j)
                const int coff = ch * 2 * kTcKC + part * kTcKC + 4 * j;
                // four row groups at a time, as far as the MMAs read
                constexpr int KB = 4;
#pragma unroll
                for (int k0 = 0; k0 < RG; k0 += KB) {
                    if (8 * (kTcProducers / 32) * k0 >= cols) break;
#pragma unroll
                    for (int k = k0; k < k0 + KB; ++k) {
                        const int src = rows[k];
                        const float* gsrc = src >= 0 ? wsp + (size_t)src * 2 * ldk + coff : wsp;
                        umma::cp16_keep(dst0 + (rg0 + (kTcProducers / 32) * k) * kTcKC * 8, gsrc, src >= 0, keep);
                    }
                }
                umma::cp_async_mbar_arrive(&full[st]);
            }
#pragma unroll
            for (int k = 0; k < RG; ++k) rows[k] = nrows[k];
            task = next;
        }
    } else if (warp == kTcMmaWarp) {
        // ---- MMA issue (one thread)
        if (lane == 0) {
            uint32_t u = 0, tl = 0;
            constexpr uint32_t LBO = 128, SBO = kTcKC / 4 * 128;
            for (int task = blockIdx.x; task < ntasks && ok; task += gridDim.x) {
                const int g = tasks[task].x, q = gq[g];
                const int cnt = min(kTcPairs, gstart[g + 1] - gstart[g] - (tasks[task].y >> 1));
                const uint32_t idesc = umma::idesc_tf32(kTcRows, tc_columns(cnt));
                const int nch = ((q + 1) * (q + 1) + kTcKC - 1) / kTcKC;
                const int acc = (int)(tl & 1);
                if (tl >= 2 && !umma::mbar_wait(&acc_empty[acc], ((tl >> 1) - 1) & 1, kTcWaitCycles)) {
                    ok = false;
                    break;
                }
                umma::fence_after_sync();
                const uint32_t d = tmem + (uint32_t)(acc * kTcPairs);
                for (int ch = 0; ch < nch; ++ch, ++u) {
                    const int st = (int)(u % kTcStages);
                    if (!umma::mbar_wait(&full[st], (u / kTcStages) & 1, kTcWaitCycles)) {
                        ok = false;
                        break;
                    }
                    umma::fence_proxy_async();  // the cp.async data, for the tensor cores
                    umma::fence_after_sync();
                    const float* Gs = reinterpret_cast<const float*>(sm_tc + (size_t)st * TcSmem::stage_bytes);
                    const float* Ws = Gs + 2 * TcSmem::g_floats;
                    const uint64_t gh = umma::smem_desc(Gs, LBO, SBO);
                    const uint64_t gl = umma::smem_desc(Gs + TcSmem::g_floats, LBO, SBO);
                    const uint64_t wh = umma::smem_desc(Ws, LBO, SBO);
                    const uint64_t wl = umma::smem_desc(Ws + TcSmem::w_floats, LBO, SBO);
                    umma::mma_tf32(d, gh, wh, idesc, ch > 0 ? 1u : 0u);
                    umma::mma_tf32(d, gh, wl, idesc, 1u);
                    umma::mma_tf32(d, gl, wh, idesc, 1u);
                    umma::commit(&empty[st]);
                }
                if (!ok) break;
                umma::commit(&acc_full[acc]);
                ++tl;
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. + 31
        // (with more than four epilogue warps, each of a sub-partition's warps
        // takes its share of the columns), kTcEpiBatch loads per wait
        const int sp = warp & 3;
        const int f = 32 * sp + lane;
        constexpr int kShares = kTcEpiWarps / 4;
        const int share = (warp - 3) / 4;
        constexpr int CB = 16 * kTcEpiBatch;  // columns per wait
        static_assert(CB == 32, "a lane per column's octant");
        uint32_t tl = 0;
        for (int task = blockIdx.x; task < ntasks && ok; task += gridDim.x) {
            const int2 tk = tasks[task];
            const int g = tk.x, q = gq[g];
            const int f0 = kTcRows * (tk.y & 1), fr = f0 + f;  // the task's operator half; this lane's row
            const int gs = gstart[g] + (tk.y >> 1);
            const int cnt = min(kTcPairs, gstart[g + 1] - gs);
            const int acc = (int)(tl & 1);
            if (!umma::mbar_wait(&acc_full[acc], (tl >> 1) & 1, kTcWaitCycles)) {
                ok = false;
                break;
            }
            umma::fence_after_sync();
            const uint32_t base = tmem + ((uint32_t)(32 * sp) << 16) + (uint32_t)(acc * kTcPairs);
            // the group's rows: (q+1)^2 rounded up to kRowUnit entries, from
            // rowbase[g] x kRowUnit in group order
            const int rl = row_len(q);
            float* gout = out + ((size_t)rowbase[g] + (size_t)(tk.y >> 1) * (rl / kRowUnit)) * kRowUnit;
            const int flips = mirrored && fr < (q + 1) * (q + 1) ? component_flips(qcomp(fr)) : 0;
            // warps whose 32 rows f lie beyond the row length have nothing to write
#pragma unroll 1
            for (int c = share * CB; c < cnt && f0 + 32 * sp < rl; c += kShares * CB) {
                float v[CB];
                __syncwarp();
#pragma unroll
                for (int b = 0; b < kTcEpiBatch; ++b) umma::tmem_ld16(base + (uint32_t)(c + 16 * b), v + 16 * b);
                umma::tmem_ld_wait();
                umma::tmem_landed(v);
                if (mirrored) {
                    // columns (bits) in which this row changes sign
                    const int o = c + lane < cnt ? psrc[gs + c + lane] : 0;
                    const unsigned b0 = __ballot_sync(0xffffffffu, o & 1), b1 = __ballot_sync(0xffffffffu, o & 2),
                                   b2 = __ballot_sync(0xffffffffu, o & 4);
                    const unsigned neg = ((flips & 1) ? b0 : 0) ^ ((flips & 2) ? b1 : 0) ^ ((flips & 4) ? b2 : 0);
#pragma unroll
                    for (int jj = 0; jj < CB; ++jj)
                        v[jj] = __uint_as_float(__float_as_uint(v[jj]) ^ ((neg >> jj) << 31));
                }
                // the task's rows are consecutive; streaming stores of whole lines
                if (fr < rl) {
#pragma unroll
                    for (int jj = 0; jj < CB; ++jj)
                        if (c + jj < cnt) __stcs(gout + (size_t)(c + jj) * rl + fr, v[jj]);
                }
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&acc_empty[acc]);
            ++tl;
        }
    }
    if (!ok) atomicExch(err, 1);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, kTcCols);
}

// Running sum of one output: FP32 values as a double-float pair (TwoSum, on
// the FP32 pipe), FP64 values in FP64.
template <typename R>
struct Sum;
template <>
struct Sum<float> {
    float hi = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float v) {
        const float s = hi + v;
        const float bb = s - hi;
        lo += (hi - (s - bb)) + (v - bb);
        hi = s;
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};
template <>
struct Sum<double> {
    double v = 0.0;
    __device__ __forceinline__ void add(double x) { v += x; }
    __device__ __forceinline__ double value() const { return v; }
};

// Block per target, thread per component of the basis: compensated sum of the
// target's pair rows (stored in group order; roff gives each target-order
// pair's row in units of kRowUnit entries; a pair of order q contributes its
// first rows(q) entries; eight loads in flight), back to physical units, into
// the basis' components of the local expansion.
template <typename R, bool full>
__global__ void __launch_bounds__(256) k_m2l_sum(const TreeDev t, int p,
                                                 const R* __restrict__ out, const int32_t* __restrict__ roff,
                                                 double* __restrict__ loc) {
    const int i = blockIdx.x;
    const int nr = d64_rows(p, full);
    const int q0 = t.far_off[i], q1 = t.far_off[i + 1];
    const double ih = 1.0 / t.r[i];
    double* L = loc + (size_t)i * nT(p);
    for (int f = threadIdx.x; f < nr; f += blockDim.x) {
        constexpr int U = 8;
        Sum<R> acc;
        int q = q0;
        for (; q + U <= q1; q += U) {
            R v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int qq = t.far_ord ? min((int)t.far_ord[q + u], p) : p;
                v[u] = f < d64_rows(qq, full) ? out[(size_t)roff[q + u] * kRowUnit + f] : (R)0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) acc.add(v[u]);
        }
        for (; q < q1; ++q) {
            const int qq = t.far_ord ? min((int)t.far_ord[q], p) : p;
            if (f < d64_rows(qq, full)) acc.add(out[(size_t)roff[q] * kRowUnit + f]);
        }
        const int c = d64_comp(f, full);
        const int k = c >> 24;
        double s = ih;
        for (int e = 0; e < k; ++e) s *= ih;
        L[full ? f : pidx(c & 0xff, (c >> 8) & 0xff, (c >> 16) & 0xff)] = acc.value() * s;
    }
}

// Products on the CUDA cores instead of the tensor cores
// (FMM_GB300_M2L_PRODUCT=cuda; read at every call).
bool product_on_cuda_cores() {
    const char* e = std::getenv("FMM_GB300_M2L_PRODUCT");
    return e && std::strcmp(e, "cuda") == 0;
}

// Orders share a displacement group in classes of kOrderClass consecutive
// orders; the group takes its pairs' highest order (fewer operators for the
// learned selector's mixed orders).
constexpr int kOrderClass = 2;

// Mean far pairs per displacement group for the grouped products.  FP64: the
// tensor-core product of one group costs about what the per-pair kernel takes
// for one or two pairs (order 10: 33 ns against 44 ns a pair at the FP64 peak).
constexpr double kMinGroupPairs = 16.0, kMinGroupPairs64 = 2.0;
// Where the per-pair kernels are an alternative of the same kind, pairs may be
// off their group's displacement by this much (half-widths): they take each
// pair's own.  60,000 particles in a box of 98 with its corner at 0 are 7e-15 off,
// at 1,000 1.2e-13; 1,500 in a box of 3 6e-15 at 0, 6e-14 at 30 (their field 5e-14),
// 2e-12 at 1,000 (above 1e-12).
constexpr float kGroupDeviation = 1e-13f;
// Memory limit of the calls that need not take the grouped products
// (FMM_GB300_M2L_BYTES; read at every call).
double grouped_bytes() {
    const char* e = std::getenv("FMM_GB300_M2L_BYTES");
    return e ? std::atof(e) : kGroupedBytes;
}
// TF32 products with fewer pairs per group than this (a task's columns not
// filled by a group) take the groups of the eight octants together, where the
// weights' eight copies fit.  250,000 particles in clusters with learned orders
// (4.1e6 pairs): 157,000 groups of 26 pairs become 56,000 of 72, tensors and
// operators 18.7 -> 6.9 ms, products 12.2 -> 4.8 ms.  Where groups are large
// there is little to gain and the copies no longer stay in the L2 cache.
constexpr double kMirrorPairs = 256.0, kMirrorBytes = 8e9;

// Split operators of the groups of one batch.
int launch_operators(Workspace& ws, bool tc, bool full, int ldT, int ldr, const M2lBatch& b, int64_t base,
                     cudaStream_t st) {
    count_launches(1);
    if (tc) {
        k_group_operator<<<(unsigned)(b.g1 - b.g0), 256, 0, st>>>(ldT, ws.m2l_T.as<float>(), ws.m2l_gq.as<int32_t>(),
                                                                  ws.m2l_gab.as<float2>(), ws.m2l_gopoff.as<int64_t>(),
                                                                  b.g0, base, ws.m2l_gop.as<float>());
    } else {
        k_operator64<<<(unsigned)(b.g1 - b.g0), 256, sizeof(double) * ldT, st>>>(
            full, ldT, ws.m2l_T.as<double>(), ws.m2l_gq.as<int32_t>(), ws.m2l_gab.as<float2>(),
            ws.m2l_gopoff.as<int64_t>(), b.g0, base, ldr, ws.m2l_gop.as<uint4>(), ws.m2l_gexp.as<int>(),
            ws.m2l_gord.as<short>());
    }
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

// bounded: the memory is limited to grouped_bytes().  FMM_ENOTSUP: the pairs should
// go one by one.
template <typename R, int CPT>
int grouped(Workspace& ws, const TreeDev& t, int p, cudaStream_t st, bool full, bool bounded) {
    const int M = t.num_nodes, nr = d64_rows(p, full), N = 2 * p, nTr = full ? nT(N) : rbase(N + 1);
    const bool tc = sizeof(R) == 4 && !product_on_cuda_cores();
    const bool tc64 = sizeof(R) == 8 && (full || !product_on_cuda_cores());
    const int cols = tc ? kTcTasks : (tc64 ? (full ? kD64FullTasks : kD64Tasks) : kTaskCols);
    const int64_t nf = t.nfar;
    const int ldw = wsc_ld<R>(nr);
    const int ldk = (nr + 15) / 16 * 16;
    const int ldT = nTr;
    const int wchunks = d64_chunks(p, full);
    const int32_t* roff = nullptr;  // row of each far pair (target order), units of kRowUnit entries
    if (nf > 0 && !ws.reuse_structure) {
        // structure: displacement groups, their tensors and operators, tasks
        // and result rows (geometry only; kept for replays)
        M2lSize size{nf, 1, row_len(p, full), ldT, 0, (int)sizeof(R)};
        if (tc64) size.operator_bytes = (int64_t)d64_parts(p, full) * wchunks * D64Smem::g_bytes + sizeof(int) * (int64_t)nr;
        if (tc) size.operator_bytes = (int64_t)tc_halves(p) * ((nr + kTcKC - 1) / kTcKC) * kTcRows * kTcKC * 2 * sizeof(float);
        if (bounded && m2l_bytes(size) > grouped_bytes()) return FMM_ENOTSUP;
        FMM_TRY(ws.m2l_tgt.ensure(sizeof(int32_t) * nf));
        FMM_TRY(ws.m2l_keys.ensure(sizeof(uint64_t) * nf));
        FMM_TRY(ws.m2l_keys2.ensure(sizeof(uint64_t) * nf));
        FMM_TRY(ws.m2l_vals.ensure(sizeof(int32_t) * nf));
        FMM_TRY(ws.m2l_vals2.ensure(sizeof(int32_t) * nf));
        FMM_TRY(ws.m2l_ukeys.ensure(sizeof(uint64_t) * nf));
        FMM_TRY(ws.m2l_cnt.ensure(sizeof(int32_t) * (nf + 1)));
        FMM_TRY(ws.m2l_gstart.ensure(sizeof(int32_t) * (nf + 1)));
        if (!tc64) FMM_TRY(ws.m2l_wsc.ensure(sizeof(R) * (size_t)M * ldw));
        FMM_TRY(ws.counters.ensure(sizeof(unsigned long long) * 32));
        int32_t* tgt = ws.m2l_tgt.as<int32_t>();
        count_launches(1);
        k_far_targets<<<grid_for(M, 4), 128, 0, st>>>(M, t.far_off, tgt);
        count_launches(1);
        // FP32 node data where the mixed path prepared it
        const float4* chi = (sizeof(R) == 4 && ws.f32node_ok) ? ws.f32node.as<float4>() : nullptr;
        const int kbits = t.nimg > 1 ? kKeyBitsImages : kKeyBits;
        int* d_dev = sizeof(R) == 8 ? reinterpret_cast<int*>(ws.counters.as<unsigned long long>() + 10) : nullptr;
        if (d_dev) FMM_CUDA_TRY(cudaMemsetAsync(d_dev, 0, sizeof(int), st));
        k_m2l_keys<<<grid_for(nf, 256), 256, 0, st>>>(nf, t, tgt, p, kOrderClass, chi, chi ? chi + M : nullptr,
                                                       ws.m2l_keys.as<uint64_t>(), ws.m2l_vals.as<int32_t>(), d_dev);
        // sort by key, run-length encode into groups
        int* d_nruns = reinterpret_cast<int*>(ws.counters.as<unsigned long long>() + 14);
        size_t tb1 = 0, tb2 = 0, tb3 = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tb1, ws.m2l_keys.as<uint64_t>(), ws.m2l_keys2.as<uint64_t>(),
                                        ws.m2l_vals.as<int32_t>(), ws.m2l_vals2.as<int32_t>(), (int)nf, 0, kbits, st);
        cub::DeviceRunLengthEncode::Encode(nullptr, tb2, ws.m2l_keys2.as<uint64_t>(), ws.m2l_ukeys.as<uint64_t>(),
                                           ws.m2l_cnt.as<int32_t>(), d_nruns, (int)nf, st);
        cub::DeviceScan::ExclusiveSum(nullptr, tb3, ws.m2l_cnt.as<int32_t>(), ws.m2l_gstart.as<int32_t>(),
                                      (int)nf + 1, st);
        FMM_TRY(ws.cub_tmp.ensure(std::max(tb1, std::max(tb2, tb3))));
        FMM_CUDA_TRY(cub::DeviceRadixSort::SortPairs(ws.cub_tmp.p, tb1, ws.m2l_keys.as<uint64_t>(),
                                                     ws.m2l_keys2.as<uint64_t>(), ws.m2l_vals.as<int32_t>(),
                                                     ws.m2l_vals2.as<int32_t>(), (int)nf, 0, kbits, st));
        FMM_CUDA_TRY(cub::DeviceRunLengthEncode::Encode(ws.cub_tmp.p, tb2, ws.m2l_keys2.as<uint64_t>(),
                                                        ws.m2l_ukeys.as<uint64_t>(), ws.m2l_cnt.as<int32_t>(),
                                                        d_nruns, (int)nf, st));
        int ng = 0;
        float dev = 0.0f;
        FMM_CUDA_TRY(cudaMemcpyAsync(&ng, d_nruns, sizeof(int), cudaMemcpyDeviceToHost, st));
        if (d_dev) FMM_CUDA_TRY(cudaMemcpyAsync(&dev, d_dev, sizeof(float), cudaMemcpyDeviceToHost, st));
        FMM_CUDA_TRY(cudaStreamSynchronize(st));
        // displacement groups of a few pairs each (irregular trees, mixed orders)
        // leave the products' columns empty and multiply the per-group operators.
        // Counted before the octants are joined: what is below the line is summed in
        // FP64 (launch_m2l_grouped) or pair by pair, both more accurate than TF32
        // parts (3,001 clustered particles, 13 pairs a group, far field at order 12:
        // 2e-10 against 4.6e-9)
        const bool few = (double)nf < (tc64 ? kMinGroupPairs64 : kMinGroupPairs) * (double)ng;
        ws.m2l_mirrored = tc && t.nimg <= 1 && (double)nf < kMirrorPairs * (double)ng &&
                          sizeof(float) * 2.0 * kOctants * M * ldk <= kMirrorBytes;
        if (ws.m2l_mirrored) {
            auto mk = thrust::make_transform_iterator(ws.m2l_keys2.as<uint64_t>(), MirroredKey());
            size_t tbm = 0;
            cub::DeviceRunLengthEncode::Encode(nullptr, tbm, mk, ws.m2l_ukeys.as<uint64_t>(), ws.m2l_cnt.as<int32_t>(),
                                               d_nruns, (int)nf, st);
            FMM_TRY(ws.cub_tmp.ensure(tbm));
            FMM_CUDA_TRY(cub::DeviceRunLengthEncode::Encode(ws.cub_tmp.p, tbm, mk, ws.m2l_ukeys.as<uint64_t>(),
                                                            ws.m2l_cnt.as<int32_t>(), d_nruns, (int)nf, st));
            FMM_CUDA_TRY(cudaMemcpyAsync(&ng, d_nruns, sizeof(int), cudaMemcpyDeviceToHost, st));
            FMM_CUDA_TRY(cudaStreamSynchronize(st));
        }
        ws.m2l_groups = ng;
        if (few) return FMM_ENOTSUP;
        size.groups = ng;
        if ((bounded || (double)nf < kMinGroupPairs * (double)ng) &&
            (m2l_bytes(size) > grouped_bytes() || dev > kGroupDeviation))
            return FMM_ENOTSUP;
        FMM_CUDA_TRY(cudaMemsetAsync(ws.m2l_cnt.as<int32_t>() + ng, 0, sizeof(int32_t), st));
        size_t tb4 = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb4, ws.m2l_cnt.as<int32_t>(), ws.m2l_gstart.as<int32_t>(), ng + 1, st);
        FMM_TRY(ws.cub_tmp.ensure(tb4));
        FMM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(ws.cub_tmp.p, tb4, ws.m2l_cnt.as<int32_t>(),
                                                   ws.m2l_gstart.as<int32_t>(), ng + 1, st));
        // per-group tensors
        const unsigned slices = group_slices(nf, ng);
        FMM_TRY(ws.m2l_T.ensure(sizeof(R) * (size_t)ng * ldT));
        FMM_TRY(ws.m2l_gq.ensure(sizeof(int32_t) * ng));
        FMM_TRY(ws.m2l_gab.ensure(sizeof(float2) * ng));
        if (full) {
            FMM_TRY(launch_group_tensor_ref(ws, t, ng, tgt, p, ldT, st));
        } else {
            const int wpb = 4;
            const size_t sm = sizeof(double) * (2 * nTr + (size_t)wpb * (2 * nTr + N + 1));
            const bool have_q = slices > 4;
            auto kernel = have_q ? k_group_tensor<R, true> : k_group_tensor<R, false>;
            if (sm > 48 * 1024)
                FMM_CUDA_TRY(
                    cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
            if (have_q) {
                count_launches(1);
                FMM_CUDA_TRY(cudaMemsetAsync(ws.m2l_gq.p, 0, sizeof(int32_t) * ng, st));
                k_group_orders<<<dim3(grid_for(ng, 8), slices), 256, 0, st>>>(
                    ng, ws.m2l_gstart.as<int32_t>(), ws.m2l_vals2.as<int32_t>(), t, p, ws.m2l_gq.as<int32_t>());
            }
            count_launches(1);
            kernel<<<grid_for(ng, wpb), 32 * wpb, sm, st>>>(
                ng, ws.m2l_mirrored, ws.m2l_keys2.as<uint64_t>(), ws.m2l_gstart.as<int32_t>(),
                ws.m2l_vals2.as<int32_t>(), tgt, t, p, ldT, ws.m2l_T.as<R>(), ws.m2l_gq.as<int32_t>(),
                ws.m2l_gab.as<float2>());
        }
        // tasks: up to kTaskCols pairs of one group each (tensor cores: 256
        // pairs and one operator half)
        FMM_TRY(ws.m2l_tcnt.ensure(sizeof(int32_t) * (ng + 1)));
        FMM_TRY(ws.m2l_toff.ensure(sizeof(int32_t) * (ng + 1)));
        count_launches(1);
        k_task_counts<<<grid_for(ng + 1, 256), 256, 0, st>>>(ng, cols, ws.m2l_gq.as<int32_t>(),
                                                              ws.m2l_gstart.as<int32_t>(), ws.m2l_tcnt.as<int32_t>());
        size_t tb5 = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb5, ws.m2l_tcnt.as<int32_t>(), ws.m2l_toff.as<int32_t>(), ng + 1, st);
        FMM_TRY(ws.cub_tmp.ensure(tb5));
        FMM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(ws.cub_tmp.p, tb5, ws.m2l_tcnt.as<int32_t>(),
                                                   ws.m2l_toff.as<int32_t>(), ng + 1, st));
        // result rows in group order, (q+1)^2 rounded up to kRowUnit entries per
        // pair; the per-target sum finds them through roff (in the free
        // unsorted-keys buffer)
        FMM_TRY(ws.m2l_rowbase.ensure(sizeof(int64_t) * (ng + 1)));
        int64_t* rowbase = ws.m2l_rowbase.as<int64_t>();
        count_launches(1);
        k_row_sizes<<<grid_for(ng + 1, 256), 256, 0, st>>>(ng, full, ws.m2l_gstart.as<int32_t>(), ws.m2l_gq.as<int32_t>(),
                                                            rowbase);
        size_t tb7 = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb7, rowbase, rowbase, ng + 1, st);
        FMM_TRY(ws.cub_tmp.ensure(tb7));
        FMM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(ws.cub_tmp.p, tb7, rowbase, rowbase, ng + 1, st));
        int ntasks = 0;
        int64_t rows = 0;  // in units of kRowUnit entries
        FMM_CUDA_TRY(cudaMemcpyAsync(&ntasks, ws.m2l_toff.as<int32_t>() + ng, sizeof(int), cudaMemcpyDeviceToHost, st));
        FMM_CUDA_TRY(cudaMemcpyAsync(&rows, rowbase + ng, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        FMM_CUDA_TRY(cudaStreamSynchronize(st));
        if (!m2l_rows_fit(rows)) return FMM_ENOTSUP;
        count_launches(1);
        k_row_offsets<<<dim3(grid_for(ng, 8), slices), 256, 0, st>>>(
            ng, full, ws.m2l_gstart.as<int32_t>(), ws.m2l_gq.as<int32_t>(), rowbase, ws.m2l_vals2.as<int32_t>(),
            reinterpret_cast<int32_t*>(ws.m2l_keys.p));
        FMM_TRY(ws.m2l_out.ensure(sizeof(R) * kRowUnit * (size_t)std::max<int64_t>(1, rows)));
        FMM_TRY(ws.m2l_tasks.ensure(sizeof(int2) * std::max(1, ntasks)));
        count_launches(1);
        k_fill_tasks<<<grid_for(ng, 256), 256, 0, st>>>(ng, cols, ws.m2l_gq.as<int32_t>(), ws.m2l_gstart.as<int32_t>(),
                                                        ws.m2l_toff.as<int32_t>(), ws.m2l_tasks.as<int2>());
        // source node per sorted pair (into the free unsorted-values buffer)
        count_launches(1);
        k_pair_sources<<<grid_for(nf, 256), 256, 0, st>>>(nf, ws.m2l_mirrored, ws.m2l_keys2.as<uint64_t>(),
                                                          ws.m2l_vals2.as<int32_t>(), t, ws.m2l_vals.as<int32_t>());
        if (tc || tc64) {
            // tensor-core operands: per node the weights, per group the operator
            FMM_TRY(ws.m2l_wsplit.ensure(tc ? sizeof(float) * 2 * (size_t)M * ldk * (ws.m2l_mirrored ? kOctants : 1)
                                            : (size_t)M * (wchunks * kDig * kD64K * 2 + sizeof(int) + sizeof(short) * kD64Orders)));
            if (tc64) {
                FMM_TRY(ws.m2l_gexp.ensure(sizeof(int) * (size_t)ng * nr));
                FMM_TRY(ws.m2l_gord.ensure(sizeof(short) * kD64Orders * (size_t)ng));
            }
            FMM_TRY(ws.m2l_gopoff.ensure(sizeof(int64_t) * (ng + 1)));
            int64_t* goff = ws.m2l_gopoff.as<int64_t>();
            count_launches(1);
            if (tc)
                k_gop_sizes<<<grid_for(ng + 1, 256), 256, 0, st>>>(ng, ws.m2l_gq.as<int32_t>(), goff);
            else
                k_op64_sizes<<<grid_for(ng + 1, 256), 256, 0, st>>>(ng, full, ws.m2l_gq.as<int32_t>(), goff);
            size_t tb6 = 0;
            cub::DeviceScan::ExclusiveSum(nullptr, tb6, goff, goff, ng + 1, st);
            FMM_TRY(ws.cub_tmp.ensure(tb6));
            FMM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(ws.cub_tmp.p, tb6, goff, goff, ng + 1, st));
            // split operators (per group, at each group's order; offsets in
            // floats, FP64: in 16-byte units), in batches of consecutive groups of at most kOperatorBytes: one
            // batch is built here once; several are built, each before the
            // product over its tasks, at every evaluation
            std::vector<int64_t> hgoff((size_t)ng + 1);
            std::vector<int32_t> htoff((size_t)ng + 1);
            FMM_CUDA_TRY(cudaMemcpyAsync(hgoff.data(), goff, sizeof(int64_t) * (ng + 1), cudaMemcpyDeviceToHost, st));
            FMM_CUDA_TRY(cudaMemcpyAsync(htoff.data(), ws.m2l_toff.as<int32_t>(), sizeof(int32_t) * (ng + 1),
                                         cudaMemcpyDeviceToHost, st));
            FMM_CUDA_TRY(cudaStreamSynchronize(st));
            const size_t unit = tc ? sizeof(float) : sizeof(uint4);
            const int64_t cap = (int64_t)(kOperatorBytes / unit);
            ws.m2l_batches.clear();
            int64_t biggest = 0;
            for (int g0 = 0; g0 < ng;) {
                int g1 = g0 + 1;
                while (g1 < ng && hgoff[g1 + 1] - hgoff[g0] <= cap) ++g1;
                ws.m2l_batches.push_back({g0, g1, hgoff[g0], htoff[g0], htoff[g1]});
                biggest = std::max(biggest, hgoff[g1] - hgoff[g0]);
                g0 = g1;
            }
            FMM_TRY(ws.m2l_gop.ensure(unit * std::max<int64_t>(1, biggest)));
            if (ws.m2l_batches.size() == 1) FMM_TRY(launch_operators(ws, tc, full, ldT, nr, ws.m2l_batches[0], 0, st));
        }
        ws.m2l_ng = ng;
        ws.m2l_ntasks = ntasks;
    }
    if (nf > 0) {
        // numeric: scaled weights, the product, (below) the per-target sums
        const int ntasks = ws.m2l_ntasks;
        const int64_t* rowbase = ws.m2l_rowbase.as<int64_t>();
        roff = reinterpret_cast<const int32_t*>(ws.m2l_keys.p);
        if (!tc64) {
            count_launches(1);
            k_scale_weights<R><<<grid_for(M, 4), 128, 0, st>>>(M, nr, ldw, ws.wred.as<double>(), t.r,
                                                               ws.m2l_wsc.as<R>());
        }
        int* d_err = reinterpret_cast<int*>(ws.counters.as<unsigned long long>() + 13);
        if (tc || tc64) {
            // TF32 parts or digits of the weights (per node)
            int* wexp = nullptr;
            short* word = nullptr;
            count_launches(1);
            if (tc) {
                k_split_weights<<<grid_for((int64_t)M * ldk, 256), 256, 0, st>>>(
                    (int64_t)M * ldk, ws.m2l_mirrored ? kOctants : 1, nr, ldw, ldk, reinterpret_cast<const float*>(ws.m2l_wsc.p),
                    ws.m2l_wsplit.as<float>());
                FMM_CUDA_TRY(cudaFuncSetAttribute((const void*)k_m2l_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)TcSmem::bytes));
            } else {
                word = reinterpret_cast<short*>(ws.m2l_wsplit.as<uint4>() + (size_t)M * wchunks * kDig * 2);
                wexp = reinterpret_cast<int*>(word + (size_t)M * kD64Orders);
                k_weights64<<<grid_for(M, 4), 128, 0, st>>>(M, p, full, full ? ws.mom.as<double>() : ws.wred.as<double>(),
                                                            t.r, ws.m2l_wsplit.as<uint4>(), wexp, word);
                FMM_CUDA_TRY(cudaFuncSetAttribute((const void*)k_m2l_tc64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)D64Smem::bytes));
            }
            int dev = 0, sms = 0;
            FMM_CUDA_TRY(cudaGetDevice(&dev));
            FMM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            if (!ws.product_err) FMM_CUDA_TRY(cudaMemsetAsync(d_err, 0, sizeof(int), st));  // first product of the call
            if (ws.events_ready) {
                cudaEventRecord(ws.ev[8], st);
                ws.product_timed = true;
            }
            const bool many = ws.m2l_batches.size() > 1;
            for (const M2lBatch& b : ws.m2l_batches) {
                if (many) FMM_TRY(launch_operators(ws, tc, full, ldT, nr, b, b.gop_base, st));
                const int nt = b.t1 - b.t0;
                if (nt <= 0) continue;
                const int grid = std::max(1, std::min(nt, sms));  // one block per SM (all tensor memory)
                count_launches(1);
                if (tc)
                    k_m2l_tc<<<(unsigned)grid, kTcThreads, TcSmem::bytes, st>>>(
                        ws.m2l_tasks.as<int2>() + b.t0, nt, ws.m2l_mirrored, ws.m2l_gstart.as<int32_t>(),
                        ws.m2l_gq.as<int32_t>(), ws.m2l_gopoff.as<int64_t>(), many ? b.gop_base : 0, ws.m2l_gop.as<float>(),
                        ws.m2l_vals.as<int32_t>(), ws.m2l_wsplit.as<float>(), ldk,
                        reinterpret_cast<float*>(ws.m2l_out.p), rowbase, d_err);
                else
                    k_m2l_tc64<<<(unsigned)grid, kD64Threads, D64Smem::bytes, st>>>(
                        ws.m2l_tasks.as<int2>() + b.t0, nt, full, ws.m2l_gstart.as<int32_t>(),
                        ws.m2l_gq.as<int32_t>(), ws.m2l_gopoff.as<int64_t>(), many ? b.gop_base : 0,
                        ws.m2l_gop.as<uint4>(), nr, ws.m2l_gexp.as<int>(), ws.m2l_vals.as<int32_t>(),
                        ws.m2l_wsplit.as<uint4>(), wchunks, wexp, reinterpret_cast<double*>(ws.m2l_out.p), rowbase,
                        kRowUnit, d_err);
            }
            if (tc64 && ntasks > 0) {
                const size_t sm = sizeof(double) * ((size_t)ldT + 4 * nr);
                FMM_CUDA_TRY(cudaFuncSetAttribute((const void*)k_m2l_pairs64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)sm));
                count_launches(1);
                k_m2l_pairs64<<<(unsigned)std::min(ntasks, 8 * sms), 128, sm, st>>>(
                    ws.m2l_tasks.as<int2>(), ntasks, full, ws.m2l_gstart.as<int32_t>(), ws.m2l_gq.as<int32_t>(),
                    ws.m2l_gab.as<float2>(), ws.m2l_T.as<double>(), ldT, ws.m2l_gord.as<short>(),
                    ws.m2l_vals.as<int32_t>(), full ? ws.mom.as<double>() : ws.wred.as<double>(), nr, t.r, word, wexp,
                    reinterpret_cast<double*>(ws.m2l_out.p), rowbase, kRowUnit);
            }
            if (ws.product_timed) cudaEventRecord(ws.ev[9], st);
            // the product's error flag is read with the call's final copies
            ws.product_err = d_err;
        } else {
            const GemmSmem<R, CPT> L(p);
            FMM_CUDA_TRY(cudaFuncSetAttribute((const void*)k_m2l_gemm<R, CPT>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.bytes));
            if (ws.events_ready) {
                cudaEventRecord(ws.ev[8], st);
                ws.product_timed = true;
            }
            count_launches(1);
            k_m2l_gemm<R, CPT><<<(unsigned)ntasks, kGemmThreads, L.bytes, st>>>(
                ws.m2l_tasks.as<int2>(), cols, 0, p, ws.m2l_gstart.as<int32_t>(), ws.m2l_gq.as<int32_t>(),
                ws.m2l_gab.as<float2>(), ws.m2l_T.as<R>(), ldT, ws.m2l_vals.as<int32_t>(), ws.m2l_wsc.as<R>(), ws.m2l_out.as<R>(), rowbase);
            if (ws.product_timed) cudaEventRecord(ws.ev[9], st);
        }
    }
    count_launches(1);
    if (nf == 0) FMM_TRY(ws.m2l_out.ensure(sizeof(R) * kRowUnit));
    // one output per thread: the basis rounded up to whole warps (192 at p = 12)
    const unsigned sum_threads = (unsigned)std::min(256, (nr + 31) / 32 * 32);
    if (sizeof(R) == 8 && full)
        k_m2l_sum<double, true><<<(unsigned)M, sum_threads, 0, st>>>(t, p, ws.m2l_out.as<double>(), roff,
                                                                     ws.loc.as<double>());
    else
        k_m2l_sum<R, false><<<(unsigned)M, sum_threads, 0, st>>>(t, p, ws.m2l_out.as<R>(), roff,
                                                                 ws.loc.as<double>());
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

}  // namespace

// Grouped M2L into the local expansions ws.loc: the reduced components from the
// weights ws.wred (which must be current), in FP32 products for `fp32`, else
// FP64; or (full) all Cartesian components in FP64 with the reference's wrapped
// tensors.  Groups too small for the FP32 products take the FP64 ones where they
// hold two pairs or more (3,001 clustered particles, 13 pairs a group: the M2L at
// orders 4 / 8 / 12 0.7 / 1.1 / 2.7 ms, pair by pair 0.8 / 2.6 / 15.6).  Returns FMM_ENOTSUP where the pairs should be evaluated one by one,
// which replays keep (ws.m2l_pairwise): small groups, more rows than their
// 32-bit numbers reach, or memory that is not there (the per-pair kernels need
// none per pair) or, bounded, not for these products to take.
int launch_m2l_grouped(Workspace& ws, const TreeDev& t, int p, bool fp32, cudaStream_t st, bool full, bool bounded) {
    if (ws.reuse_structure && ws.m2l_pairwise) return FMM_ENOTSUP;
    int rc = FMM_ENOTSUP;
    if (!ws.reuse_structure) ws.m2l_fp64 = !fp32;
    if (!ws.m2l_fp64) {
        rc = grouped<float, 8>(ws, t, p, st, false, bounded);
        if (rc == FMM_ENOTSUP && !product_on_cuda_cores()) {
            const int64_t groups = ws.m2l_groups;  // (the octants' joined, as the statistics count them)
            ws.m2l_fp64 = true;
            rc = grouped<double, 4>(ws, t, p, st, false, true);
            ws.m2l_groups = groups;
        }
    } else if (full || !product_on_cuda_cores() || GemmSmem<double, 4>(p).bytes <= 227 * 1024)
        rc = grouped<double, 4>(ws, t, p, st, full, bounded);
    if (ws.reuse_structure) return rc;
    if (rc == FMM_ENOMEM) {
        ws.release_grouped();
        rc = FMM_ENOTSUP;
    }
    ws.m2l_pairwise = rc == FMM_ENOTSUP;
    return rc;
}

}  // namespace fmm

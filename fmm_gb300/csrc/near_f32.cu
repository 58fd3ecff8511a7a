// Mixed-precision near field (P2P): FP32 pair arithmetic with FP64 sums.
//
// Same pairs as particle_fields (src/fmm.F90:623-747).  Coordinates are held
// relative to the root cell's centre as double-float pairs (hi + lo, about 49
// bits of the box), so the displacement R = (x_t - x_s)_hi + (x_t - x_s)_lo of
// two near particles, whose hi parts subtract without rounding, carries about
// one FP32 rounding of its own size.  r^2 is compensated and 1/r
// Newton-refined.  Contributions are summed in compensated FP32 (TwoSum hi +
// lo) and added into FP64 at the end.  Excluded partners and the self pair are
// masked in the loop.
//
// Because positions need no leaf, the source leaves of a near list that follow
// one another in the sorted order (most do: the list is sorted) form runs,
// which a warp walks as one: lane groups are filled across leaf boundaries
// (leaves of about a dozen particles leave 40% of them idle otherwise).
//
// The packed kernel (field orders 0 and 1) evaluates
// each target against two sources at once in f32x2 arithmetic from a second
// record array with even leaf starts and interleaved slot pairs, and, with
// learned lists on AMOEBA, a second launch walks a damping-correction list:
// far leaf pairs inside the damping range, of which only the pairs
// with a r below the range's cutoff are evaluated, as the difference of the
// damped and undamped kernels (the M2L carries the undamped one).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>

#include <cub/cub.cuh>

#include "dispatch.cuh"
#include "internal.h"
#include "pair.cuh"
#include "pair_x2.cuh"

namespace fmm {

namespace {

inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

// Pairs (packed: blocks) between folds of the plain block sum into the
// compensated one.  A fold is 24 packed operations of about 140 a block; at
// four, water with Thole damping (60,000 sites) is 1.31e-6 off the FP64 near
// field, at three 1.27e-6, as with the folds at every leaf end before.
// Potentials alone (F = 0), of which every one is a sum of charges' and multipoles'
// large terms, fold at two: dipoles and quadrupoles with Thole damping 2.99e-7 off
// (700 points, box of 20), at three 3.27e-7; 1 to 3% of the kernel's time.
__host__ __device__ constexpr int fold_of(int f) { return f == 0 ? 2 : 3; }
// Exclusion entries held in registers per target; for the others a piece is
// checked by the range of their slots.  Eight cost the kernels 3 to 7%, so longer
// lists than four have kernels of their own (WIDE).  240,000 particles in
// molecules of eight, near field with four / eight: charges 2.0 / 1.4 ms, dipoles with
// field gradients 3.5 / 2.8.
__host__ __device__ constexpr int exw_regs(bool wide) { return wide ? 8 : 4; }

// Sub-chunks of a target leaf's last rem < 32 particles (index rem): the
// count that minimises the lane-steps of a piece of source blocks for leaves
// of about 30 particles (c sub-chunks of ceil(rem / c) targets run
// floor(32 / ceil(rem / c)) lane groups each).
__constant__ int kSubChunks[32] = {1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 2, 2, 1, 1, 1,
                                   1, 3, 3, 2, 2, 3, 3, 3, 3, 1, 1, 1, 1, 1, 1, 1};

// Per sorted particle, one record of float4s: (x, y, z, d), (x_lo, y_lo, z_lo,
// original index + 1 as int bits), then the FP32 scaled multipoles padded to
// a multiple of 4 (for quadrupoles the first pad slot holds the trace of the
// scaled second moments, used by the near-field contraction).  Positions are
// relative to the root centre (leaf: to the particle's own leaf centre, the
// records of the selector's kernels) as double-float pairs (hi = rounded value,
// lo = rounded remainder).  A source is then read with a handful of 16-byte
// loads from one base address.
__host__ __device__ constexpr int rec_vec(int dim) { return 2 + (dim + 3) / 4; }

__global__ void k_gather_f32(int64_t n, int dim, bool leaf, const TreeDev t, const double* __restrict__ sx,
                             const double* __restrict__ sy, const double* __restrict__ sz,
                             const double* __restrict__ sd, const double* __restrict__ smc,
                             float4* __restrict__ rec) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int nv = rec_vec(dim);
    const int l = leaf ? t.leaf_of[k] : 0;
    const double rx = sx[k] - (leaf ? t.cx[l] : t.root_c[0]), ry = sy[k] - (leaf ? t.cy[l] : t.root_c[1]),
                 rz = sz[k] - (leaf ? t.cz[l] : t.root_c[2]);
    const float hx = (float)rx, hy = (float)ry, hz = (float)rz;
    float4* r = rec + (size_t)k * nv;
    r[0] = make_float4(hx, hy, hz, (float)sd[k]);
    r[1] = make_float4((float)(rx - (double)hx), (float)(ry - (double)hy), (float)(rz - (double)hz),
                       __int_as_float((int32_t)t.perm[k] + 1));  // 1-based, as in the exclusion lists
    for (int v = 2; v < nv; ++v) {
        float m[4];
        for (int c = 0; c < 4; ++c) {
            const int s = 4 * (v - 2) + c;
            m[c] = s < dim ? (float)smc[(size_t)s * n + k] : 0.0f;
            if (dim == 10 && s == 10)
                m[c] = (float)(smc[(size_t)4 * n + k] + smc[(size_t)7 * n + k] + smc[(size_t)9 * n + k]);
        }
        r[v] = make_float4(m[0], m[1], m[2], m[3]);
    }
}

// Source records of the packed near field: the sorted particles of each leaf
// from an even slot ps[leaf] on, an odd leaf padded by one empty particle
// (zero multipoles, damping factor 1, outside the root cell by its width and
// 1000 bohr: no target is there, whose field would be 0 x infinity, and the pair
// terms are exactly zero); slots 2b and 2b + 1 form block b, stored
// element by element interleaved (float 2e + h of the block is element e of
// the record of slot 2b + h), so one 16-byte shared-memory load gives two
// elements of both particles as two packed pairs.
// With q1 (quadrupole sources, field order 1: contract_q1_x2) the
// off-diagonal second moments xy, xz, yz (record elements 13, 14, 16) are
// stored halved, an exact scaling.
__global__ void k_gather_x2(int64_t n, int nv, bool q1, const TreeDev t, const int32_t* __restrict__ ps,
                            const float4* __restrict__ rec, float* __restrict__ x2) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int leaf = t.leaf_of[k];
    const int within = (int)(k - t.start[leaf]), cnt = t.count[leaf];
    const int64_t slot = (int64_t)ps[leaf] + within;
    const float* s = reinterpret_cast<const float*>(rec + (size_t)k * nv);
    float* d = x2 + (size_t)(slot >> 1) * 8 * nv + (slot & 1);
    for (int e = 0; e < 4 * nv; ++e) d[2 * e] = s[e];
    if (q1) {
        d[2 * 13] = 0.5f * s[13];
        d[2 * 14] = 0.5f * s[14];
        d[2 * 16] = 0.5f * s[16];
    }
    if (within == cnt - 1 && (cnt & 1)) {
        float* dd = d + 1;  // slot + 1: the odd half of the same block
        for (int e = 0; e < 4 * nv; ++e) dd[2 * e] = 0.0f;
        // positions are relative to the root's or a leaf's centre, so a target is
        // within 2 root_r of the origin along each axis
        dd[0] = 4.0f * (float)t.root_r + 1000.0f;  // x
        dd[2 * 3] = 1.0f; // damping factor
    }
}

// Per leaf: the largest distance of its particles from its centre (from the
// FP32 records, plus a rounding margin) and its smallest damping factor;
// bounds for skipping whole damping-correction pieces.
__global__ void k_leaf_extent(int nv, const TreeDev t, const float4* __restrict__ rec, float2* __restrict__ ext) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= t.num_leaves) return;
    const int leaf = t.leaves[w];
    const int s0 = t.start[leaf], cnt = t.count[leaf];
    float r2 = 0.0f, dmin = 3.0e38f;
    for (int k = lane; k < cnt; k += 32) {
        const float4 a = rec[(size_t)(s0 + k) * nv];
        r2 = fmaxf(r2, a.x * a.x + a.y * a.y + a.z * a.z);
        dmin = fminf(dmin, a.w);
    }
    for (int o = 16; o > 0; o >>= 1) {
        r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
        dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
    }
    if (lane == 0) ext[leaf] = make_float2(sqrtf(r2) * 1.0001f + 1e-3f, dmin);
}

__global__ void k_leaf_odd(const TreeDev t, int32_t* __restrict__ odd) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w < t.num_leaves) odd[w] = t.count[t.leaves[w]] & 1;
}

// Leaves are in DFS order, i.e. by increasing start: the padded start of a
// leaf is its start plus the odd leaves before it.
__global__ void k_leaf_pstart(const TreeDev t, const int32_t* __restrict__ pre, int32_t* __restrict__ ps) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w < t.num_leaves) ps[t.leaves[w]] = t.start[t.leaves[w]] + pre[w];
}

// Node centres as double-float pairs (hi = rounded centre, lo = rounded
// remainder), so leaf-centre offsets are formed in FP32 without losing bits;
// the w components carry rmax (hi) and the half-width (lo) in FP32 for the
// learned list build.
__global__ void k_node_centres_f32(int M, const TreeDev t, float4* __restrict__ hi, float4* __restrict__ lo) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const float hx = (float)t.cx[k], hy = (float)t.cy[k], hz = (float)t.cz[k];
    hi[k] = make_float4(hx, hy, hz, (float)t.rmax[k]);
    lo[k] = make_float4((float)(t.cx[k] - (double)hx), (float)(t.cy[k] - (double)hy), (float)(t.cz[k] - (double)hz),
                        (float)t.r[k]);
}

// One target's position and the sorted positions (slots) that it passes over.
template <bool WIDE>
struct Target {
    float4 a, b;          // the record's first two float4s
    int slot;             // its own slot
    int ex[exw_regs(WIDE)];  // slots of the excluded partners listed first (-1: none)
    int lo, hi;           // range of the slots of the others
    int orig;             // original index
};

// First block of a piece that lane group grp of ngr takes: block b of the sorted
// slots is group b mod ngr's, so that sums do not depend on where pieces end.
__device__ __forceinline__ int first_block(int b0, int grp, int ngr) {
    const int d = grp - b0 % ngr;
    return d < 0 ? d + ngr : d;
}

// Sum over the sources src[0, cnt) of one staged piece (lane group grp of ngr)
// for the lane's target: compensated FP32 (TwoSum hi + lo), since the per-atom
// terms are much larger than their neutral total.  The contraction adds each
// pair into a plain FP32 block sum (blk, of nb pairs so far, kept from piece to
// piece) that is folded into (hi, lo) every fold_of(F) pairs: the block sum's
// rounding is of the order of a single pair's, and the TwoSum cost is paid once
// per fold.  k0 is the slot of src[0].  CHECK: the piece may hold the
// target itself or one of its excluded partners.
template <int M, int F, int DAMP, bool CHECK, bool WIDE>
__device__ __forceinline__ void p2p_piece(const float4* src, int cnt, int k0, int grp, int ngr, const Target<WIDE>& T,
                                          const int32_t* __restrict__ excl, int exw, int64_t n, float* hi, float* lo,
                                          float* blk, int& nb) {
    constexpr int NF = nT(F), NM = nT(M), NV = rec_vec(NM);
    for (int k = first_block(k0, grp, ngr); k < cnt; k += ngr) {
        const float4* r = src + k * NV;
        const float4 a = r[0], b = r[1];
        if (CHECK) {
            const int o = __float_as_int(b.w);
            bool skip = k0 + k == T.slot;
#pragma unroll
            for (int e = 0; e < exw_regs(WIDE); ++e) skip |= k0 + k == T.ex[e];
            for (int e = exw_regs(WIDE); e < exw; ++e) skip |= (excl[(size_t)e * n + T.orig] == o);
            if (skip) continue;
        }
        float mc[4 * (NV - 2)];
#pragma unroll
        for (int v = 0; v < NV - 2; ++v) {
            const float4 w = r[2 + v];
            mc[4 * v] = w.x;
            mc[4 * v + 1] = w.y;
            mc[4 * v + 2] = w.z;
            mc[4 * v + 3] = w.w;
        }
        const float dx = (T.a.x - a.x) + (T.b.x - b.x);
        const float dy = (T.a.y - a.y) + (T.b.y - b.y);
        const float dz = (T.a.z - a.z) + (T.b.z - b.z);
        pair_field_f32acc<M, F>(dx, dy, dz, T.a.w * a.w, DAMP, mc, blk);
        if (++nb == fold_of(F)) {
            nb = 0;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const float s = hi[f] + blk[f];
                const float bb = s - hi[f];
                lo[f] += (hi[f] - (s - bb)) + (blk[f] - bb);
                hi[f] = s;
                blk[f] = 0.0f;
            }
        }
    }
}

// p2p_piece on the packed records (k_gather_x2): blocks b = grp, grp + ngr,
// ... of the staged piece, each the lane's target against two sources in
// packed arithmetic.  Each half keeps its own compensated sum (H, L) over all
// pieces of the target chunk, fed from a plain block sum B (of nb blocks so far)
// folded every fold_of(F) blocks (as many pairs per fold and half as in the scalar
// loop).  k0 is the slot
// of the piece's first source.
// CORR (a piece of a far leaf inside the damping range): only the damping
// correction (damped minus undamped kernel) of the pairs with (a r)^2 below
// xcut2, beyond which the damped kernel equals the undamped one to the
// requested accuracy; a block is skipped when no lane has such a pair.  (A pair
// evaluated with another lane's loses its undamped potential too, which AMOEBA
// damping leaves undefined: which pairs those are is part of the result, so
// correction pieces are single leaves, their blocks counted from the leaf's
// start and their test made on leaf-relative positions, whatever the runs.)
template <int M, int F, int DAMP, bool CHECK, bool CORR, bool WIDE>
__device__ __forceinline__ void p2p_piece_x2(const float4* src, int nblk, int k0, int grp, int ngr, const Target<WIDE>& T,
                                             const int32_t* __restrict__ excl, int exw, int64_t n, f2* H, f2* L,
                                             f2* B, int& nb, float xcut2 = 0.0f, int* ncorr = nullptr) {
    constexpr int NF = nT(F), NM = nT(M), NV = rec_vec(NM), NE = 4 * (NV - 2);
    const f2 xt = bc2(T.a.x), yt = bc2(T.a.y), zt = bc2(T.a.z), dt = bc2(T.a.w);
    const f2 xl = bc2(T.b.x), yl = bc2(T.b.y), zl = bc2(T.b.z);
    for (int b = CORR ? grp : first_block(k0 >> 1, grp, ngr); b < nblk; b += ngr) {
        const ulonglong2* r = reinterpret_cast<const ulonglong2*>(src + (size_t)b * 2 * NV);
        // element pairs: (x, y), (z, d), (x_lo, y_lo), (z_lo, index), multipoles
        const ulonglong2 v0 = r[0], v1 = r[1];
        if constexpr (CORR) {
            const f2 cx = xt - f2{v0.x}, cy = yt - f2{v0.y}, cz = zt - f2{v1.x};
            const f2 aa = dt * f2{v1.y};
            const f2 tt = (aa * aa) * fma2(cx, cx, fma2(cy, cy, cz * cz));
            float t0, t1;
            sp2(tt, t0, t1);
            if (!__any_sync(__activemask(), t0 < xcut2 || t1 < xcut2)) continue;
            *ncorr += (t0 < xcut2 ? 1 : 0) + (t1 < xcut2 ? 1 : 0);  // pairs whose correction is needed
        }
        const ulonglong2 v2 = r[2], v3 = r[3];
        f2 mc[NE];
#pragma unroll
        for (int v = 0; v < NE / 2; ++v) {
            const ulonglong2 w = r[4 + v];
            mc[2 * v].v = w.x;
            mc[2 * v + 1].v = w.y;
        }
        f2 dx = (xt - f2{v0.x}) + (xl - f2{v2.x});
        const f2 dy = (yt - f2{v0.y}) + (yl - f2{v2.y});
        const f2 dz = (zt - f2{v1.x}) + (zl - f2{v3.x});
        const f2 a = dt * f2{v1.y};
        if (CHECK) {
            const int k = k0 + 2 * b;
            bool s0 = k == T.slot, s1 = k + 1 == T.slot;
#pragma unroll
            for (int e = 0; e < exw_regs(WIDE); ++e) {
                s0 |= k == T.ex[e];
                s1 |= k + 1 == T.ex[e];
            }
            if (exw > exw_regs(WIDE)) {
                float o0, o1;
                sp2(f2{v3.y}, o0, o1);
                for (int e = exw_regs(WIDE); e < exw; ++e) {
                    const int x = excl[(size_t)e * n + T.orig];
                    s0 |= x == __float_as_int(o0);
                    s1 |= x == __float_as_int(o1);
                }
            }
            if (s0 || s1) {
                // a skipped half gets zero multipoles at a finite distance
                const f2 keep = mk2(s0 ? 0.0f : 1.0f, s1 ? 0.0f : 1.0f);
#pragma unroll
                for (int e = 0; e < NE; ++e) mc[e] = mc[e] * keep;
                float d0, d1;
                sp2(dx, d0, d1);
                dx = mk2(s0 ? 1000.0f : d0, s1 ? 1000.0f : d1);
            }
        }
        pair_field_x2<M, F, CORR>(dx, dy, dz, a, DAMP, mc, B);
        if (++nb == fold_of(F)) {
            nb = 0;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const f2 s = H[f] + B[f];
                const f2 bb = s - H[f];
                L[f] += (H[f] - (s - bb)) + (B[f] - bb);
                H[f] = s;
                B[f] = bc2(0.0f);
            }
        }
    }
}

// Source records are staged per warp in shared memory, double-buffered:
// while one piece (a run of source leaves, or `stage` / NV of its particles when
// it is longer) is evaluated, the next is copied with cp.async.  The staging
// size (float4s per buffer) is a launch parameter (dynamic shared memory).
constexpr int kStage = 320;  // default float4s per staging buffer

__device__ __forceinline__ void cp_async16(float4* smem, const float4* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// a - b as an unevaluated pair s + e (Knuth's TwoSum with b negated).
__device__ __forceinline__ float two_diff(float a, float b, float& e) {
    const float s = a - b;
    const float bb = s - a;
    e = (a - (s - bb)) - (b + bb);
    return s;
}

// The damping-correction list's data: the targets in the selector's records
// (positions relative to the leaf centres, as the sources' packed ones) and what
// its leaves are passed over by.
struct CorrArgs {
    float xcut2;
    unsigned long long* count;
    float4 root;          // root centre; w: what rounding may take from a distance
    const float4 *chi, *clo;  // node centres (hi, lo)
    const float2* ext;    // leaf extents and smallest damping factors
    const float4* rec;
};

// A warp's walk over a target leaf's list: 32 entries are looked up at a time,
// one per lane, and near entries whose slots follow one another are merged into
// runs.  All members but a, e, j are the same in every lane.
struct RunWalk {
    int q, qend;            // next entry, the list's end
    int a, e, j;            // this lane's entry: first slot, end, leaf
    unsigned starts, keep;  // lanes that start a run, lanes with an entry
};

// One warp per item, a target leaf and a slice of its near list, the leaf's
// particles across the lanes (chunks of fewer than 32 particles run several
// lane groups, each taking every ngr-th block of a staged piece).
// Pieces that hold neither the target nor an excluded partner of any of the
// warp's targets run without the exclusion test.
// DAMP is the damping kind as a template parameter: one specialised kernel
// per kind keeps the pair loop free of kind dispatch and its code small.
// Work: with `next` null, warp w takes item w; otherwise the warps stay
// resident and take items in order from the counter `next`, the leaves by
// decreasing pair count (order), so the largest start first and the last wave
// is made of the smallest.  Slice s of leaf l goes to out[s][f][particle];
// systems of few leaves are split so that the items cover the GPU several
// times (30,000 particles, order-1 sources: 1.83 ms with an item per leaf).
// X2: sources from the packed records `srec` (k_gather_x2, padded leaf starts
// sstart) evaluated two at a time; otherwise srec = rec, sstart = t.start.
// CORR (packed kernel, AMOEBA): the damping-correction list (t.corr_off) in
// place of the near list, passing over the entries whose leaf bound (C.ext)
// rules out a pair inside xcut2 for every lane, the result added to out and the
// corrected pairs counted into C.count.  (A kernel of its own: walked after the
// near list in one kernel it cost that one registers, and spills.)
template <int M, int F, int DAMP, bool X2, bool CORR, bool WIDE>
__global__ void __launch_bounds__(256, 2) k_p2p_f32(const TreeDev t, const float4* __restrict__ rec,
                                                    const float4* __restrict__ srec,
                                                    const int32_t* __restrict__ sstart,
                                                    const int32_t* __restrict__ excl, int exw, int64_t n,
                                                    double* __restrict__ out, int stage, int slices,
                                                    const int32_t* __restrict__ order, unsigned* __restrict__ next,
                                                    const CorrArgs C) {
    constexpr int NF = nT(F), NM = nT(M), NV = rec_vec(NM);
    static_assert(!CORR || (X2 && DAMP == DAMP_AMOEBA), "corrections: packed kernel, AMOEBA");
    const int32_t* const list_off = CORR ? t.corr_off : t.near_off;
    const int32_t* const list_src = CORR ? t.corr_src : t.near_src;
    extern __shared__ __align__(16) float4 sbuf_p2p[];
    const int cap = X2 ? (stage / NV) & ~1 : stage / NV;  // particles (slots) per staged piece
    const int lane = threadIdx.x & 31;
    float4* const bufs = sbuf_p2p + (size_t)(threadIdx.x >> 5) * 2 * stage;
    const int w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int ncorr = 0;  // corrected pairs evaluated by this lane
    for (int round = 0;; ++round) {
        int item;
        if (next) {
            unsigned v = 0;
            if (lane == 0) v = atomicAdd(next, 1u);
            item = (int)__shfl_sync(0xffffffffu, v, 0);
        } else {
            if (round > 0) break;
            item = w0;
        }
        if (item >= t.num_leaves * slices) break;
        const int slice = item % slices;
        const int leaf = order ? order[item / slices] : t.leaves[item / slices];
        const int s0 = t.start[leaf], cnt = t.count[leaf];
        auto part = [&](int lo, int hi, int s) { return lo + (int)((int64_t)(hi - lo) * s / slices); };
        const int n0 = list_off[leaf], n1 = list_off[leaf + 1];
        const int q0 = part(n0, n1, slice), q1 = part(n0, n1, slice + 1);
        if (CORR && q0 == q1) continue;
        // chunks of 32 targets, then the remaining rem < 32 in cs sub-chunks of
        // gs targets; a chunk of g targets runs ngr = 32 / g lane groups of g
        // lanes (any g), each taking every ngr-th block of each staged piece
        const int full = cnt >> 5, rem = cnt & 31;
        const int cs = rem ? kSubChunks[rem] : 0, gs = rem ? (rem + cs - 1) / cs : 1;
        for (int ci = 0; ci < full + cs; ++ci) {
            const int chunk = ci < full ? 32 * ci : 32 * full + (ci - full) * gs;
            const int g = ci < full ? 32 : gs;
            const int nt = min(g, cnt - chunk);
            const int ngr = 32 / g;
            const int tl = lane % g, grp = lane / g;
            const bool valid = tl < nt && grp < ngr;
            const int tgt = s0 + chunk + (valid ? tl : 0);
            Target<WIDE> T;
            T.a = rec[(size_t)tgt * NV];
            T.b = rec[(size_t)tgt * NV + 1];
            T.orig = __float_as_int(T.b.w) - 1;
            T.slot = sstart[leaf] + (tgt - s0);
            auto slot_of = [&](int o) {  // -1: unused entry
                if (o <= 0) return -1;
                const int pos = t.pos_of[o - 1], l = t.leaf_of[pos];
                return sstart[l] + (pos - t.start[l]);
            };
#pragma unroll
            for (int e = 0; e < exw_regs(WIDE); ++e) T.ex[e] = e < exw ? slot_of(excl[(size_t)e * n + T.orig]) : -1;
            T.lo = INT_MAX;
            T.hi = -1;
            for (int e = exw_regs(WIDE); e < exw; ++e) {
                const int x = slot_of(excl[(size_t)e * n + T.orig]);
                if (x >= 0) T.lo = min(T.lo, x);
                T.hi = max(T.hi, x);
            }
            // per-target sums over all source leaves as double-float pairs (FP32
            // arithmetic; the FP64 pipe is the scarce one)
            float AH[NF], AL[NF], AB[NF];
            f2 XH[NF], XL[NF], XB[NF];  // packed kernel: one compensated sum per half
            int nb = 0;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                AH[f] = AL[f] = AB[f] = 0.0f;
                XH[f] = XL[f] = XB[f] = bc2(0.0f);
            }
            RunWalk W{q0, q1, 0, 0, 0, 0u, 0u};
            // looks up the next 32 entries; false at the end of the list
            auto load_window = [&]() -> bool {
                while (W.q < W.qend) {
                    const int q = W.q + lane;
                    const bool ok = q < W.qend;
                    W.a = W.e = W.j = 0;
                    if (ok) {
                        W.j = list_src[q];
                        int c = t.count[W.j];
                        if (X2) c += c & 1;  // padded to whole blocks
                        W.a = sstart[W.j];
                        W.e = W.a + c;
                    }
                    W.keep = __ballot_sync(0xffffffffu, ok);
                    if constexpr (CORR) {
                        // entries whose leaf cannot hold a pair that needs a
                        // correction for any of this chunk's targets: for target t
                        // and leaf B, a r >= d_t dmin_B (|x_t - c_B| - extent_B)
                        // (all lanes take part)
                        const int ne = __popc(W.keep);
                        unsigned keep = 0;
                        for (int l = 0; l < ne; ++l) {
                            const int Bn = __shfl_sync(0xffffffffu, W.j, l);
                            bool need = false;
                            if (valid) {
                                const float4 cb = C.chi[Bn];
                                const float2 eb = C.ext[Bn];
                                const float dx = (T.a.x + C.root.x) - cb.x, dy = (T.a.y + C.root.y) - cb.y,
                                            dz = (T.a.z + C.root.z) - cb.z;
                                const float rmin = fmaxf(sqrtf(dx * dx + dy * dy + dz * dz) - eb.x - C.root.w, 0.0f);
                                const float xm = T.a.w * eb.y * rmin;
                                need = xm * xm < C.xcut2;
                            }
                            if (__any_sync(0xffffffffu, need)) keep |= 1u << l;
                        }
                        W.keep = keep;
                    }
                    W.q += 32;
                    if (!W.keep) continue;
                    const int pe = __shfl_up_sync(0xffffffffu, W.e, 1);
                    const bool follows = !CORR && lane > 0 && ((W.keep >> (lane - 1)) & 1u) && pe == W.a;
                    W.starts = __ballot_sync(0xffffffffu, ((W.keep >> lane) & 1u) && !follows);
                    return true;
                }
                return false;
            };
            // next run of slots [rs, re) (CORR: of leaf rj); false at the end of the
            // list
            auto next_run = [&](int& rs, int& re, int& rj) -> bool {
                if (!W.starts && !load_window()) return false;
                const int sl = __ffs(W.starts) - 1;
                W.starts &= W.starts - 1;
                const unsigned stop = (W.starts | ~W.keep) & ~((2u << sl) - 1u);
                const int el = stop ? __ffs(stop) - 2 : 31;
                rs = __shfl_sync(0xffffffffu, W.a, sl);
                re = __shfl_sync(0xffffffffu, W.e, el);
                if (CORR) rj = __shfl_sync(0xffffffffu, W.j, sl);
                return true;
            };
            // current piece [ps, ps + pl) of run [.., re); the first one is staged
            // before the loop
            int ps = 0, re = 0, pl = 0, pj = 0;
            bool have = next_run(ps, re, pj);
            if (have) {
                pl = min(cap, re - ps);
                const float4* gsrc = srec + (size_t)ps * NV;
                for (int i = lane; i < pl * NV; i += 32) cp_async16(&bufs[i], gsrc + i);
            }
            cp_async_commit();
            int slot = 0;
            while (have) {
                // stage the next piece
                int nps = ps + pl, nre = re, npj = pj;
                bool more = nps < re;
                if (!more) more = next_run(nps, nre, npj);
                const int npl = more ? min(cap, nre - nps) : 0;
                if (more) {
                    const float4* gsrc = srec + (size_t)nps * NV;
                    float4* dst = bufs + (slot ^ 1) * stage;
                    for (int i = lane; i < npl * NV; i += 32) cp_async16(&dst[i], gsrc + i);
                }
                cp_async_commit();
                cp_async_wait_prev();
                __syncwarp();
                if (valid) {
                    bool need = (unsigned)(T.slot - ps) < (unsigned)pl || (T.hi >= ps && T.lo < ps + pl);
#pragma unroll
                    for (int e = 0; e < exw_regs(WIDE); ++e) need |= (unsigned)(T.ex[e] - ps) < (unsigned)pl;
                    const float4* cur = bufs + slot * stage;
                    const bool anyneed = __any_sync(__activemask(), need);
                    if constexpr (CORR) {
                        // the target relative to the source's leaf centre: the
                        // centres' offset hi + lo, its low part with the target's
                        const float4 ta = C.rec[(size_t)tgt * NV], tb = C.rec[(size_t)tgt * NV + 1];
                        const float4 ca = C.chi[leaf], cal = C.clo[leaf], cb = C.chi[pj], cbl = C.clo[pj];
                        float ex, ey, ez;
                        const float ox = two_diff(ca.x, cb.x, ex), oy = two_diff(ca.y, cb.y, ey),
                                    oz = two_diff(ca.z, cb.z, ez);
                        Target<WIDE> U = T;
                        U.a = make_float4(ta.x + ox, ta.y + oy, ta.z + oz, ta.w);
                        U.b = make_float4((ex + (cal.x - cbl.x)) + tb.x, (ey + (cal.y - cbl.y)) + tb.y,
                                          (ez + (cal.z - cbl.z)) + tb.z, 0.0f);
                        if (anyneed)
                            p2p_piece_x2<M, F, DAMP, true, true, WIDE>(cur, pl >> 1, ps, grp, ngr, U, excl, exw, n, XH, XL,
                                                                 XB, nb, C.xcut2, &ncorr);
                        else
                            p2p_piece_x2<M, F, DAMP, false, true, WIDE>(cur, pl >> 1, ps, grp, ngr, U, excl, exw, n, XH, XL,
                                                                  XB, nb, C.xcut2, &ncorr);
                    } else if constexpr (X2) {
                        if (anyneed)
                            p2p_piece_x2<M, F, DAMP, true, false, WIDE>(cur, pl >> 1, ps, grp, ngr, T, excl, exw, n, XH, XL, XB, nb);
                        else
                            p2p_piece_x2<M, F, DAMP, false, false, WIDE>(cur, pl >> 1, ps, grp, ngr, T, excl, exw, n, XH, XL, XB, nb);
                    } else {
                        if (anyneed)
                            p2p_piece<M, F, DAMP, true, WIDE>(cur, pl, ps, grp, ngr, T, excl, exw, n, AH, AL, AB, nb);
                        else
                            p2p_piece<M, F, DAMP, false, WIDE>(cur, pl, ps, grp, ngr, T, excl, exw, n, AH, AL, AB, nb);
                    }
                }
                __syncwarp();
                ps = nps;
                re = nre;
                pl = npl;
                pj = npj;
                have = more;
                slot ^= 1;
            }
            cp_async_wait_all();
            __syncwarp();
            double acc[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                if constexpr (X2) {
                    float h0, h1, l0, l1;
                    sp2(XH[f], h0, h1);
                    sp2(XL[f], l0, l1);
                    float b0, b1;
                    sp2(XB[f], b0, b1);
                    acc[f] = ((double)h0 + (double)h1) + (((double)l0 + (double)l1) + ((double)b0 + (double)b1));
                } else {
                    acc[f] = (double)AH[f] + ((double)AL[f] + (double)AB[f]);
                }
            }
            if ((g & (g - 1)) == 0) {
                for (int o = g; o < 32; o <<= 1) {
#pragma unroll
                    for (int f = 0; f < NF; ++f) acc[f] += __shfl_xor_sync(0xffffffffu, acc[f], o);
                }
            } else {
                // group 0 adds groups 1 .. ngr - 1 (lanes tl + k g)
                double part_f[NF];
#pragma unroll
                for (int f = 0; f < NF; ++f) part_f[f] = acc[f];
                for (int k = 1; k < ngr; ++k) {
#pragma unroll
                    for (int f = 0; f < NF; ++f) acc[f] += __shfl_sync(0xffffffffu, part_f[f], (tl + k * g) & 31);
                }
            }
            if (grp == 0 && valid) {
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    double* o = out + ((size_t)slice * NF + f) * n + tgt;
                    *o = CORR ? *o + acc[f] : acc[f];
                }
            }
        }
    }
    if (CORR) {
        // every lane of the warp is here (items are taken per warp)
        const int sc = __reduce_add_sync(0xffffffffu, ncorr);
        if ((threadIdx.x & 31) == 0 && sc) atomicAdd(C.count, (unsigned long long)sc);
    }
}

// Local field scale of each leaf for the learned selector's error budgets:
// the field (order-1 components, FP32, damped as the call) at up to
// kScaleSamples particles of the leaf from every particle of its smallest
// ancestor holding at least kScaleNeighbours particles (a subtree is one
// contiguous range of the sorted particles; at most kScaleWindow of them
// around the leaf), excluded partners and the
// particle itself skipped; the leaf's values are the mean and the minimum
// of log10 of the magnitudes found (-30 for a zero field), at scale[leaf]
// and scale[num_nodes + leaf].  The field at a particle is
// dominated by its nearest neighbours, which lie in that range except near
// the range's faces; the estimate sets how much absolute error each far pair
// may carry at the leaf.
constexpr int kScaleSamples = 4;
constexpr int kScaleNeighbours = 256;
constexpr int kScaleWindow = 1024;

template <int M>
__global__ void __launch_bounds__(128) k_leaf_field_scale(const TreeDev t, const float4* __restrict__ rec,
                                                          const float4* __restrict__ chi, int damp, int exw,
                                                          const int32_t* __restrict__ excl, int64_t n,
                                                          float* __restrict__ scale) {
    constexpr int NM = nT(M), NV = rec_vec(NM);
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= t.num_leaves) return;
    const int leaf = t.leaves[w];
    const int s0 = t.start[leaf], cnt = t.count[leaf];
    int anc = leaf;
    while (t.count[anc] < kScaleNeighbours && t.parent[anc] >= 0) anc = t.parent[anc];
    // at most kScaleWindow particles of that range, centred on the leaf's
    // (Morton order keeps them near it)
    int a0 = t.start[anc], a1 = a0 + t.count[anc];
    if (a1 - a0 > kScaleWindow) {
        a0 = max(a0, min(s0 + cnt / 2 - kScaleWindow / 2, a1 - kScaleWindow));
        a1 = a0 + kScaleWindow;
    }
    const int ns = min(kScaleSamples, cnt);
    float lsum = 0.0f, lmin = 30.0f;
    for (int sidx = 0; sidx < ns; ++sidx) {
        const int k = s0 + (int)((int64_t)sidx * cnt / ns);
        const float4 ta = rec[(size_t)k * NV], tb = rec[(size_t)k * NV + 1];
        const float4 ca = chi[leaf];
        const float tx = ta.x + ca.x, ty = ta.y + ca.y, tz = ta.z + ca.z;
        const int ot = __float_as_int(tb.w) - 1;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int q = a0 + lane; q < a1; q += 32) {
            if (q == k) continue;
            const float4* r = rec + (size_t)q * NV;
            const float4 sa = r[0], sb = r[1];
            const int o = __float_as_int(sb.w);
            bool ex = false;
            for (int e = 0; e < exw; ++e) ex |= (excl[(size_t)e * n + ot] == o);
            if (ex) continue;
            float mc[4 * (NV - 2)];
#pragma unroll
            for (int v = 0; v < NV - 2; ++v) {
                const float4 wv = r[2 + v];
                mc[4 * v] = wv.x;
                mc[4 * v + 1] = wv.y;
                mc[4 * v + 2] = wv.z;
                mc[4 * v + 3] = wv.w;
            }
            const float4 cb = chi[t.leaf_of[q]];
            const float dx = tx - (sa.x + cb.x), dy = ty - (sa.y + cb.y), dz = tz - (sa.z + cb.z);
            if constexpr (M == 2) {
                // quadrupole sources: the dot-product contraction (the record's
                // pad slot holds the trace of the second moments)
                float g[4];
                radial_g<3, float>(damp, dx * dx + dy * dy + dz * dz, ta.w * sa.w, g);
                contract_q1<float>(dx, dy, dz, g, mc, mc[10], damp, acc);
            } else {
                pair_field<M, 1, float>(dx, dy, dz, ta.w * sa.w, damp, mc, acc);
            }
        }
#pragma unroll
        for (int c = 1; c < 4; ++c)
            for (int off = 16; off > 0; off >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], off);
        const float l = log10f(fmaxf(sqrtf(acc[1] * acc[1] + acc[2] * acc[2] + acc[3] * acc[3]), 1e-30f));
        lsum += l;
        lmin = fminf(lmin, l);
    }
    if (lane == 0) {
        scale[leaf] = ns > 0 ? lsum / (float)ns : -30.0f;
        scale[t.num_nodes + leaf] = ns > 0 ? lmin : -30.0f;
    }
}

// Pair work of each target leaf (its particles times the particles of its
// near list) for the work queue's order.
__global__ void k_leaf_cost(const TreeDev t, uint32_t* __restrict__ cost, int32_t* __restrict__ ids) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= t.num_leaves) return;
    const int leaf = t.leaves[w];
    uint32_t s = 0;
    for (int q = t.near_off[leaf] + lane; q < t.near_off[leaf + 1]; q += 32) s += (uint32_t)t.count[t.near_src[q]];
    if (t.corr_off) {
        // damping-correction pieces: mostly the cheap range test, about a
        // quarter of a near pair each
        uint32_t c = 0;
        for (int q = t.corr_off[leaf] + lane; q < t.corr_off[leaf + 1]; q += 32) c += (uint32_t)t.count[t.corr_src[q]];
        s += c / 4;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        const uint64_t c = (uint64_t)t.count[leaf] * s;
        cost[w] = c > 0xffffffffull ? 0xffffffffu : (uint32_t)c;
        ids[w] = leaf;
    }
}

template <int M, int F, bool X2, bool WIDE>
void launch_p2p_kind(unsigned blocks, int threads, size_t smem, int stage, int slices, const int32_t* order,
                     unsigned* next, cudaStream_t st, const TreeDev& t, const float4* rec, const float4* srec,
                     const int32_t* sstart, const int32_t* excl, int exw, int64_t n, int damp, double* out,
                     const CorrArgs& C) {
    if constexpr (X2 && F > 1) {
        return;  // not instantiated: the packed kernel is used for field orders 0 and 1
    } else {
#define FMM_P2P_KIND(D)                                                                                              \
    k_p2p_f32<M, F, D, X2, false, WIDE><<<blocks, threads, smem, st>>>(t, rec, srec, sstart, excl, exw, n, out, stage,     \
                                                                 slices, order, next, C)
        switch (damp) {
            case DAMP_AMOEBA: FMM_P2P_KIND(DAMP_AMOEBA); break;
            case DAMP_THOLE: FMM_P2P_KIND(DAMP_THOLE); break;
            case DAMP_ERF: FMM_P2P_KIND(DAMP_ERF); break;
            default: FMM_P2P_KIND(DAMP_NONE); break;
        }
#undef FMM_P2P_KIND
    }
}

template <int M, int F>
void launch_p2p_corr(unsigned blocks, int threads, size_t smem, int stage, const int32_t* order, unsigned* next,
                     cudaStream_t st, const TreeDev& t, const float4* rec, const float4* srec, const int32_t* sstart,
                     const int32_t* excl, int exw, int64_t n, double* out, const CorrArgs& C) {
    if constexpr (F <= 1)
        k_p2p_f32<M, F, DAMP_AMOEBA, true, true, false><<<blocks, threads, smem, st>>>(t, rec, srec, sstart, excl, exw, n, out,
                                                                              stage, 1, order, next, C);
}

template <int M, int F, bool X2, bool WIDE>
const void* p2p_kernel(int damp) {
    if constexpr (X2 && F > 1) return nullptr;
    else
    return damp == DAMP_AMOEBA  ? (const void*)k_p2p_f32<M, F, DAMP_AMOEBA, X2, false, WIDE>
           : damp == DAMP_THOLE ? (const void*)k_p2p_f32<M, F, DAMP_THOLE, X2, false, WIDE>
           : damp == DAMP_ERF   ? (const void*)k_p2p_f32<M, F, DAMP_ERF, X2, false, WIDE>
                                : (const void*)k_p2p_f32<M, F, DAMP_NONE, X2, false, WIDE>;
}

template <int M, int F>
const void* p2p_kernel(int damp, bool x2, bool wide) {
    return x2 ? (wide ? p2p_kernel<M, F, true, true>(damp) : p2p_kernel<M, F, true, false>(damp))
              : (wide ? p2p_kernel<M, F, false, true>(damp) : p2p_kernel<M, F, false, false>(damp));
}

template <int M, int F>
int set_p2p_smem(int damp, bool x2, bool wide, size_t smem) {
    FMM_CUDA_TRY(cudaFuncSetAttribute(p2p_kernel<M, F>(damp, x2, wide), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    if constexpr (F <= 1)
        FMM_CUDA_TRY(cudaFuncSetAttribute((const void*)k_p2p_f32<M, F, DAMP_AMOEBA, true, true, false>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return FMM_OK;
}

template <int M, int F>
int p2p_blocks_per_sm(int damp, bool x2, bool wide, int threads, size_t smem) {
    int nb = 0;
    const void* fn = p2p_kernel<M, F>(damp, x2, wide);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return std::max(1, nb);
}

int num_sms_f32() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    return sms;
}

}  // namespace

int prepare_f32_records(Workspace& ws, const Particles& P, const TreeDev& t, bool near, bool selector,
                        cudaStream_t st) {
    const int64_t n = P.n;
    const int nv = rec_vec(P.dim);
    for (int leaf = near ? 0 : 1; leaf <= (selector ? 1 : 0); ++leaf) {
        DevBuf& b = leaf ? ws.f32sel : ws.f32buf;
        FMM_TRY(b.ensure(sizeof(float4) * (size_t)n * nv));
        count_launches(1);
        k_gather_f32<<<grid_for(n, 256), 256, 0, st>>>(n, P.dim, leaf != 0, t, ws.sx.as<double>(), ws.sy.as<double>(),
                                                        ws.sz.as<double>(), ws.sd.as<double>(), ws.smc.as<double>(),
                                                        b.as<float4>());
    }
    FMM_TRY(ws.f32node.ensure(sizeof(float4) * 2 * (size_t)t.num_nodes));
    float4* chi = ws.f32node.as<float4>();
    count_launches(1);
    k_node_centres_f32<<<grid_for(t.num_nodes, 256), 256, 0, st>>>(t.num_nodes, t, chi, chi + t.num_nodes);
    FMM_CUDA_TRY(cudaGetLastError());
    ws.f32node_ok = true;
    return FMM_OK;
}

int launch_leaf_extent(Workspace& ws, const Particles& P, const TreeDev& t, cudaStream_t st) {
    FMM_TRY(ws.leaf_ext.ensure(sizeof(float2) * (size_t)t.num_nodes));
    count_launches(1);
    k_leaf_extent<<<grid_for((int64_t)t.num_leaves * 32, 128), 128, 0, st>>>(rec_vec(P.dim), t, ws.f32sel.as<float4>(),
                                                                             ws.leaf_ext.as<float2>());
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int launch_leaf_field_scale(Workspace& ws, const Particles& P, const TreeDev& t, float* d_scale, cudaStream_t st) {
    const int m = dim_to_order(P.dim);
    const float4* rec = ws.f32sel.as<float4>();  // prepare_f32_records
    const float4* chi = ws.f32node.as<float4>();
    const unsigned blocks = grid_for((int64_t)t.num_leaves * 32, 128);
    switch (m) {
        case 0:
            k_leaf_field_scale<0><<<blocks, 128, 0, st>>>(t, rec, chi, P.damp_type, P.exw, P.excl, P.n, d_scale);
            break;
        case 1:
            k_leaf_field_scale<1><<<blocks, 128, 0, st>>>(t, rec, chi, P.damp_type, P.exw, P.excl, P.n, d_scale);
            break;
        case 2:
            k_leaf_field_scale<2><<<blocks, 128, 0, st>>>(t, rec, chi, P.damp_type, P.exw, P.excl, P.n, d_scale);
            break;
        default:
            return FMM_ENOTSUP;
    }
    count_launches(1);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

bool p2p_packed_enabled(const P2pShape& sh, int field_order) {
    const char* pe = std::getenv("FMM_GB300_P2P_PACKED");
    return sh.pack && !(pe && pe[0] == '0') && field_order <= 1;
}

bool P2pShape::valid() const {
    return (threads == 64 || threads == 128 || threads == 256) && stage >= 64 && stage <= 1024 && stage % 16 == 0 &&
           (queue == 0 || queue == 1) && (pack == 0 || pack == 1);
}

int launch_p2p_f32(Workspace& ws, const Particles& P, const TreeDev& t, int field_order, cudaStream_t st) {
    const int m = dim_to_order(P.dim);
    const int64_t n = P.n;
    const int nf = nT(field_order);
    const float4* rec = ws.f32buf.as<float4>();  // prepare_f32_records
    FMM_TRY(ws.fsorted.ensure(sizeof(double) * (size_t)n * nf));
    const P2pShape sh = ws.p2p_shape.valid() ? ws.p2p_shape : P2pShape{};
    const size_t smem = sizeof(float4) * 2 * (size_t)sh.stage * (sh.threads / 32);
    if (rec_vec(P.dim) > sh.stage) return FMM_EINVAL;
    // packed kernel: sources two at a time from the padded, interleaved
    // records, for field orders 0 and 1 (at order 2 the packed registers do
    // not fit); FMM_GB300_P2P_PACKED=0 selects the one-source kernel
    const bool x2 = p2p_packed_enabled(sh, field_order) && t.num_leaves > 0 &&
                    n + (int64_t)t.num_leaves < (int64_t)INT32_MAX;
    const bool wide = P.exw > exw_regs(false);
    // a damping-correction list is walked by the packed kernel only; the
    // pairs it corrects are counted in counter 9
    if (t.ncorr > 0 && !(x2 && P.damp_type == DAMP_AMOEBA)) return FMM_ENOTSUP;
    FMM_TRY(ws.counters.ensure(sizeof(unsigned long long) * 32));
    unsigned long long* corr_count = ws.counters.as<unsigned long long>() + 9;
    FMM_CUDA_TRY(cudaMemsetAsync(corr_count, 0, sizeof(unsigned long long), st));
    // leaf extents: computed with the lists (launch_leaf_extent)
    const double big = std::max({std::fabs(t.root_c[0]), std::fabs(t.root_c[1]), std::fabs(t.root_c[2])}) + t.root_r;
    CorrArgs C{ws.corr_xcut2, corr_count,
               make_float4((float)t.root_c[0], (float)t.root_c[1], (float)t.root_c[2], (float)(1e-2 + 1e-6 * big)),
               ws.f32node.as<float4>(), ws.f32node.as<float4>() + t.num_nodes,
               ws.leaf_ext.as<float2>(), ws.f32sel.as<float4>()};
    // slices of the source lists: at least four items per resident warp (about
    // 16 an SM), while a slice keeps eight list entries
    int64_t slices = 1;
    if (t.num_leaves > 0) {
        slices = (4LL * 16 * num_sms_f32() + t.num_leaves - 1) / t.num_leaves;
        slices = std::max<int64_t>(1, std::min<int64_t>({slices, t.nnear / (8LL * t.num_leaves), 16}));
    }
    double* out = ws.fsorted.as<double>();
    if (slices > 1) {
        FMM_TRY(ws.near_part.ensure(sizeof(double) * (size_t)slices * nf * n));
        out = ws.near_part.as<double>();
    }
    if (x2) {
        const int nv = rec_vec(P.dim);
        const int L = t.num_leaves;
        FMM_TRY(ws.f32x2.ensure(sizeof(float4) * (size_t)(n + L + 1) * nv));
        if (!ws.reuse_structure) {
            // padded leaf starts (structure: kept for replays)
            FMM_TRY(ws.p2p_pad.ensure(sizeof(int32_t) * ((size_t)t.num_nodes + 2 * (size_t)L)));
            int32_t* ps = ws.p2p_pad.as<int32_t>();
            int32_t* odd = ps + t.num_nodes;
            int32_t* pre = odd + L;
            count_launches(1);
            k_leaf_odd<<<grid_for(L, 256), 256, 0, st>>>(t, odd);
            size_t tb = 0;
            cub::DeviceScan::ExclusiveSum(nullptr, tb, odd, pre, L, st);
            FMM_TRY(ws.cub_tmp.ensure(tb));
            FMM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(ws.cub_tmp.p, tb, odd, pre, L, st));
            count_launches(1);
            k_leaf_pstart<<<grid_for(L, 256), 256, 0, st>>>(t, pre, ps);
        }
        // (with a damping-correction list, a second set from the selector's records)
        if (t.ncorr > 0) FMM_TRY(ws.f32x2c.ensure(sizeof(float4) * (size_t)(n + L + 1) * nv));
        for (int c = 0; c < (t.ncorr > 0 ? 2 : 1); ++c) {
            count_launches(1);
            k_gather_x2<<<grid_for(n, 256), 256, 0, st>>>(n, nv, P.dim == 10 && field_order == 1, t,
                                                           ws.p2p_pad.as<int32_t>(), c ? ws.f32sel.as<float4>() : rec,
                                                           (c ? ws.f32x2c : ws.f32x2).as<float>());
        }
    }
    const int32_t* order = nullptr;
    unsigned* next = nullptr;
    unsigned blocks = grid_for((int64_t)t.num_leaves * slices * 32, sh.threads);
    if (sh.queue && t.num_leaves > 0) {
        // target leaves by decreasing pair work (structure: kept for replays)
        FMM_TRY(ws.counters.ensure(sizeof(unsigned long long) * 32));
        next = reinterpret_cast<unsigned*>(ws.counters.as<unsigned long long>() + 11);
        if (!ws.reuse_structure) {
            const int L = t.num_leaves;
            FMM_TRY(ws.p2p_order.ensure(sizeof(int32_t) * 2 * (size_t)L + sizeof(uint32_t) * 2 * (size_t)L));
            int32_t* ids = ws.p2p_order.as<int32_t>() + L;
            uint32_t* cost = reinterpret_cast<uint32_t*>(ws.p2p_order.as<int32_t>() + 2 * (size_t)L);
            uint32_t* cost2 = cost + L;
            count_launches(1);
            k_leaf_cost<<<grid_for((int64_t)L * 32, 128), 128, 0, st>>>(t, cost, ids);
            size_t tb = 0;
            cub::DeviceRadixSort::SortPairsDescending(nullptr, tb, cost, cost2, ids, ws.p2p_order.as<int32_t>(), L, 0,
                                                      32, st);
            FMM_TRY(ws.cub_tmp.ensure(tb));
            FMM_CUDA_TRY(cub::DeviceRadixSort::SortPairsDescending(ws.cub_tmp.p, tb, cost, cost2, ids,
                                                                   ws.p2p_order.as<int32_t>(), L, 0, 32, st));
        }
        order = ws.p2p_order.as<int32_t>();
        FMM_CUDA_TRY(cudaMemsetAsync(next, 0, sizeof(unsigned), st));
        int bps = 1;
        FMM_MF_SWITCH(m, field_order, (bps = p2p_blocks_per_sm<MM, FF>(P.damp_type, x2, wide, sh.threads, smem)));
        blocks = (unsigned)std::min<int64_t>(blocks, (int64_t)bps * num_sms_f32());
    }
    if (smem > 48 * 1024) {
        FMM_MF_SWITCH(m, field_order, FMM_TRY((set_p2p_smem<MM, FF>(P.damp_type, x2, wide, smem))));
    }
#define FMM_P2P_LAUNCH(X2, WIDE, SREC, SSTART)                                                                       \
    FMM_MF_SWITCH(m, field_order,                                                                                    \
                  (launch_p2p_kind<MM, FF, X2, WIDE>(blocks, sh.threads, smem, sh.stage, (int)slices, order, next, st, \
                                                     t, rec, SREC, SSTART, P.excl, P.exw, n, P.damp_type, out, C)))
    if (x2 && wide) {
        FMM_P2P_LAUNCH(true, true, ws.f32x2.as<float4>(), ws.p2p_pad.as<int32_t>());
    } else if (x2) {
        FMM_P2P_LAUNCH(true, false, ws.f32x2.as<float4>(), ws.p2p_pad.as<int32_t>());
    } else if (wide) {
        FMM_P2P_LAUNCH(false, true, rec, t.start);
    } else {
        FMM_P2P_LAUNCH(false, false, rec, t.start);
    }
#undef FMM_P2P_LAUNCH
    if (slices > 1) FMM_TRY(sum_slices(n * nf, (int)slices, out, ws.fsorted.as<double>(), st));
    if (t.ncorr > 0) {
        if (next) FMM_CUDA_TRY(cudaMemsetAsync(next, 0, sizeof(unsigned), st));
        const unsigned cblocks = std::min(blocks, grid_for((int64_t)t.num_leaves * 32, sh.threads));
        FMM_MF_SWITCH(m, field_order,
                      (launch_p2p_corr<MM, FF>(next ? cblocks : grid_for((int64_t)t.num_leaves * 32, sh.threads),
                                               sh.threads, smem, sh.stage, order, next, st, t, rec,
                                               ws.f32x2c.as<float4>(), ws.p2p_pad.as<int32_t>(), P.excl, P.exw, n,
                                               ws.fsorted.as<double>(), C)));
    }
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

}  // namespace fmm

// Near field (P2P), direct sum and the exclusion corrections, FP64.
//
// Reference: particle_fields (src/fmm.F90:623-747) and particle_fields_direct
// (src/fmm.F90:749-824).  Both loop over target particles and call
// multipole_field on a vector of sources, moving excluded sources to
// R = (1e10, 1e10, 1e10).  The kernels here do the same pair by pair: a warp
// holds one target, its lanes take consecutive sources, and a source that the
// target excludes (itself included, where it lists itself) is evaluated at
// R = (1e10, 1e10, 1e10) in reference mode (a small potential term,
// src/fmm.F90:714-720) and passed over in mask mode.
//
// The pairs are bound by FP64 issue (pair_f64.cuh): a warp instruction takes a
// scheduler's FP64 pipe 64 cycles, so index arithmetic, exclusion tests and
// loads (14 doubles per pair, about 1 TB/s from L1 and L2) are hidden behind
// it.  What the layout has to give is full lanes and an even spread over the
// 4 x 152 schedulers: with the sources across the lanes no leaf or system size
// leaves lanes idle beyond a target's last step, and a warp per target (and
// source slice, where there are few targets) makes thousands of equal items.
#include <algorithm>

#include "internal.h"
#include "pair_f64.cuh"
#include "dispatch.cuh"

namespace fmm {

namespace {

inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

int num_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    return sms;
}

// Contraction coefficients c_s of the multipole components (order <= 3),
// folded at compile time (no FP64 division per element).
__constant__ double cSrcCoef[20] = {src_coef(0),  src_coef(1),  src_coef(2),  src_coef(3),  src_coef(4),
                                    src_coef(5),  src_coef(6),  src_coef(7),  src_coef(8),  src_coef(9),
                                    src_coef(10), src_coef(11), src_coef(12), src_coef(13), src_coef(14),
                                    src_coef(15), src_coef(16), src_coef(17), src_coef(18), src_coef(19)};

// Multipoles times the contraction coefficient c_s, original particle order.
__global__ void k_scale_mp(int64_t n, int dim, const double* __restrict__ mp, double* __restrict__ out) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    for (int c = 0; c < dim; ++c) out[(size_t)c * n + k] = cSrcCoef[c] * mp[(size_t)c * n + k];
}

// Near rows (pair_f64.cuh) of quadrupole sources: the contraction coefficients
// (scaled: already folded in), off-diagonal second moments halved, and the
// trace of the second moments as row 10.
__global__ void k_near_rows(int64_t n, bool scaled, const double* __restrict__ mp, double* __restrict__ out) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    double tr = 0.0;
#pragma unroll
    for (int c = 0; c < 10; ++c) {
        double v = mp[(size_t)c * n + k];
        if (!scaled) v *= cSrcCoef[c];
        if (c == 4 || c == 7 || c == 9) tr += v;
        if (c == 5 || c == 6 || c == 8) v *= 0.5;
        out[(size_t)c * n + k] = v;
    }
    out[(size_t)10 * n + k] = tr;
}

// Particle data in key-sorted order (coordinates, damping, scaled multipoles).
__global__ void k_gather(int64_t n, int dim, const uint32_t* __restrict__ perm, const double* __restrict__ X,
                         const double* __restrict__ mp, const double* __restrict__ damp, double* __restrict__ sx,
                         double* __restrict__ sy, double* __restrict__ sz, double* __restrict__ sd,
                         double* __restrict__ smc) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t o = perm[k];
    sx[k] = X[o];
    sy[k] = X[n + o];
    sz[k] = X[2 * n + o];
    sd[k] = damp ? damp[o] : 0.0;
    for (int c = 0; c < dim; ++c) smc[(size_t)c * n + k] = cSrcCoef[c] * mp[(size_t)c * n + o];
}

// The target's exclusion list: its first kExRegs entries in registers (0:
// unused slot, which no 1-based index equals), the rest read where needed.
constexpr int kExRegs = 4;
struct ExList {
    int e[kExRegs];
    const int32_t* more;
    int64_t n;
    int exw;
    __device__ __forceinline__ ExList(const int32_t* __restrict__ excl, int exw_, int64_t n_, int64_t i)
        : more(excl + i), n(n_), exw(exw_) {
#pragma unroll
        for (int w = 0; w < kExRegs; ++w) e[w] = w < exw ? excl[(size_t)w * n + i] : 0;
    }
    __device__ __forceinline__ bool has(int j1) const {
        bool x = false;
#pragma unroll
        for (int w = 0; w < kExRegs; ++w) x |= e[w] == j1;
        for (int w = kExRegs; w < exw; ++w) x |= more[(size_t)w * n] == j1;
        return x;
    }
};

// P2P: a warp per target particle and source slice (blockIdx.y of gridDim.y),
// its lanes over the concatenated particles of the target leaf's near list
// (each lane walks the list on its own).  Totals go to out[slice][f][particle].
// IMG: the sources are cells of the periodic images: their particles sit at
// x_j + the image's shift, and the self pair and the exclusions count only in
// the central image (src/fmm.F90:704-736).
// 66,666 water molecules, Thole, f = 2 (4.6e8 pairs): 294 ms with a warp per
// target leaf (targets across the lanes) and the tensor contraction.
template <int M, int F, bool IMG>
__global__ void __launch_bounds__(128) k_p2p_f64(const TreeDev t, const double* __restrict__ sx,
                                                 const double* __restrict__ sy, const double* __restrict__ sz,
                                                 const double* __restrict__ sd, const double* __restrict__ rows,
                                                 int64_t n, int damp, int excl_mode, int exw,
                                                 const int32_t* __restrict__ excl, double* __restrict__ out) {
    constexpr int NF = nT(F), NA = acc_count(M, F), NR = near_row_count(M, F);
    const int64_t tgt = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (tgt >= n) return;
    const int leaf = t.leaf_of[tgt];
    const double xt = sx[tgt], yt = sy[tgt], zt = sz[tgt], dt = sd[tgt];
    const ExList ex(excl, exw, n, (int64_t)t.perm[tgt]);
    double acc[NA];
#pragma unroll
    for (int f = 0; f < NA; ++f) acc[f] = 0.0;
    const int q1 = t.near_off[leaf + 1], step = 32 * (int)gridDim.y;
    int q = t.near_off[leaf] - 1, js = 0, jc = 0, img = 0;
    for (int off = lane + 32 * (int)blockIdx.y;; off += step) {
        while (off >= jc) {
            off -= jc;
            if (++q >= q1) break;
            const int j = t.near_src[q];
            js = t.start[j];
            jc = t.count[j];
            if (IMG) img = src_image(t, j);
        }
        if (q >= q1) break;
        const int k = js + off;
        double dx, dy, dz;
        if (IMG) {
            const double* sh = t.img_shift + 3 * img;
            dx = xt - (sx[k] + sh[0]);
            dy = yt - (sy[k] + sh[1]);
            dz = zt - (sz[k] + sh[2]);
        } else {
            dx = xt - sx[k];
            dy = yt - sy[k];
            dz = zt - sz[k];
        }
        if (!IMG || img == 0) {
            const bool out_of = ex.has((int)t.perm[k] + 1);
            if (excl_mode == 0) {
                if (out_of) dx = dy = dz = 1e10;
            } else if (out_of || k == tgt) {
                continue;
            }
        }
        double mc[NR];
#pragma unroll
        for (int s = 0; s < NR; ++s) mc[s] = rows[(size_t)s * n + k];
        pair_field_f64<M, F>(dx, dy, dz, dt * sd[k], damp, mc, acc);
    }
    int f;
    double fld[NF];
    finish_f64<M, F>(acc, fld);
    if (warp_totals<NF>(fld, lane, &f)) out[((size_t)blockIdx.y * NF + f) * n + tgt] = fld[0];
}

// out[e] = sum over the slices of part[slice][e].
__global__ void k_sum_slices(int64_t total, int slices, const double* __restrict__ part, double* __restrict__ fs) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= total) return;
    double s = 0.0;
    for (int k = 0; k < slices; ++k) s += part[(size_t)k * total + e];
    fs[e] = s;
}

// Direct sum: a warp per target and slice of `chunk` sources (blockIdx.y), the
// sources across the lanes; totals go to out[slice][f][target].
template <int M, int F>
__global__ void __launch_bounds__(128) k_direct_f64(int64_t n, const int64_t* __restrict__ targets, int64_t ntgt,
                                                    const double* __restrict__ X, const double* __restrict__ rows,
                                                    const double* __restrict__ damp, int damp_type, int excl_mode,
                                                    int exw, const int32_t* __restrict__ excl, int64_t chunk,
                                                    double* __restrict__ out) {
    constexpr int NF = nT(F), NA = acc_count(M, F), NR = near_row_count(M, F);
    const int64_t ti = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (ti >= ntgt) return;
    const int64_t i = targets ? targets[ti] : ti;
    const double xi = X[i], yi = X[n + i], zi = X[2 * n + i];
    const double di = damp ? damp[i] : 0.0;
    const ExList ex(excl, exw, n, i);
    double acc[NA];
#pragma unroll
    for (int f = 0; f < NA; ++f) acc[f] = 0.0;
    const int64_t j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
    for (int64_t j = j0 + lane; j < j1; j += 32) {
        double dx = xi - X[j], dy = yi - X[n + j], dz = zi - X[2 * n + j];
        const bool out_of = ex.has((int)j + 1);
        if (excl_mode == 0) {
            if (out_of) dx = dy = dz = 1e10;
        } else if (out_of || j == i) {
            continue;
        }
        double mc[NR];
#pragma unroll
        for (int s = 0; s < NR; ++s) mc[s] = rows[(size_t)s * n + j];
        pair_field_f64<M, F>(dx, dy, dz, di * (damp ? damp[j] : 0.0), damp_type, mc, acc);
    }
    int f;
    double fld[NF];
    finish_f64<M, F>(acc, fld);
    if (warp_totals<NF>(fld, lane, &f)) out[((size_t)blockIdx.y * NF + f) * ntgt + ti] = fld[0];
}

__device__ __forceinline__ bool is_near_leaf(const int32_t* near_off, const int32_t* near_src, int li, int lj) {
    int a = near_off[li], h = near_off[li + 1];
    while (a < h) {
        const int mid = (a + h) >> 1;
        if (near_src[mid] < lj)
            a = mid + 1;
        else
            h = mid;
    }
    return a < near_off[li + 1] && near_src[a] == lj;
}

// Mask mode: the far field holds the undamped contribution of excluded
// partners whose leaf is not in the near list of the target's leaf (the
// near-field kernels pass over the others); this takes it out again.  One
// thread per particle (original index i, field in sorted order).
template <int M, int F>
__global__ void k_excl_fix(int64_t n, const double* __restrict__ X, const double* __restrict__ mc, int exw,
                           const int32_t* __restrict__ excl, const int32_t* __restrict__ pos_of,
                           const int32_t* __restrict__ leaf_of, const int32_t* __restrict__ near_off,
                           const int32_t* __restrict__ near_src, double* __restrict__ field) {
    constexpr int NF = nT(F), NM = nT(M);
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t ki = pos_of[i];
    double sub[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) sub[f] = 0.0;
    bool any = false;
    for (int w = 0; w < exw; ++w) {
        const int e = excl[(size_t)w * n + i];
        if (e == 0) continue;
        bool dup = false;
        for (int w2 = 0; w2 < w; ++w2)
            if (excl[(size_t)w2 * n + i] == e) dup = true;
        if (dup) continue;
        const int64_t j = e - 1;
        if (j == i || is_near_leaf(near_off, near_src, leaf_of[ki], leaf_of[pos_of[j]])) continue;
        double m[NM];
#pragma unroll
        for (int s = 0; s < NM; ++s) m[s] = mc[(size_t)s * n + j];
        pair_field_cold<M, F, double>(X[i] - X[j], X[n + i] - X[n + j], X[2 * n + i] - X[2 * n + j], 0.0, DAMP_NONE, m,
                                      sub);
        any = true;
    }
    if (!any) return;
#pragma unroll
    for (int f = 0; f < NF; ++f) field[(size_t)f * n + ki] -= sub[f];
}

__global__ void k_scatter(int64_t n, int nf, const uint32_t* __restrict__ perm, const double* __restrict__ fs,
                          double* __restrict__ field) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t o = perm[k];
    for (int f = 0; f < nf; ++f) field[(size_t)f * n + o] = fs[(size_t)f * n + k];
}

}  // namespace

bool near_orders_supported(int m, int f) { return m >= 0 && m <= 3 && f >= 0 && f <= 3; }

int sum_slices(int64_t total, int slices, const double* part, double* out, cudaStream_t st) {
    count_launches(1);
    k_sum_slices<<<grid_for(total, 128), 128, 0, st>>>(total, slices, part, out);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int launch_direct_f64(Workspace& ws, const Particles& P, int field_order, const Modes& md, double* d_field,
                      cudaStream_t st, int64_t ntgt, const int64_t* d_targets, int split_cap) {
    const int m = dim_to_order(P.dim);
    if (!near_orders_supported(m, field_order)) return FMM_ENOTSUP;
    const int64_t n = P.n;
    if (!d_targets) ntgt = n;
    const int nf = nT(field_order);
    // own buffer: may overlap the FMM phases
    FMM_TRY(ws.dsmc.ensure(sizeof(double) * (size_t)n * near_row_count(m, field_order)));
    double* rows = ws.dsmc.as<double>();
    count_launches(1);
    if (near_row_count(m, field_order) > P.dim)
        k_near_rows<<<grid_for(n, 128), 128, 0, st>>>(n, false, P.mp, rows);
    else
        k_scale_mp<<<grid_for(n, 128), 128, 0, st>>>(n, P.dim, P.mp, rows);
    // Slices: 16 items per scheduler where the sum is long enough, at least
    // one step of 32 sources each (300 targets: 10 slices of one step; 4096: 2
    // of 64 steps; from 10,000 on one slice, written straight to the field)
    const int64_t steps = (n + 31) / 32;
    const int64_t per = std::max<int64_t>(1, ntgt * steps / (16LL * 4 * num_sms()));
    int64_t ks = (steps + per - 1) / per;
    if (split_cap > 0) ks = std::min<int64_t>(ks, 4LL * split_cap);
    ks = std::min<int64_t>(ks, 65535);
    const int64_t chunk = (steps + ks - 1) / ks * 32;
    ks = (n + chunk - 1) / chunk;
    double* out = d_field;
    if (ks > 1) {
        FMM_TRY(ws.partial.ensure(sizeof(double) * (size_t)ks * nf * ntgt));
        out = ws.partial.as<double>();
    }
    const dim3 grid(grid_for(ntgt, 4), (unsigned)ks);
    FMM_MF_SWITCH_F64(m, field_order,
                      (k_direct_f64<MM, FF><<<grid, 128, 0, st>>>(n, d_targets, ntgt, P.x, rows, P.damp, P.damp_type,
                                                                  md.excl_mode, P.exw, P.excl, chunk, out)));
    if (ks > 1) FMM_TRY(sum_slices(ntgt * nf, (int)ks, out, d_field, st));
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int gather_sorted(Workspace& ws, const Particles& P, const TreeDev& t, cudaStream_t st) {
    const int64_t n = P.n;
    FMM_TRY(ws.sx.ensure(sizeof(double) * n));
    FMM_TRY(ws.sy.ensure(sizeof(double) * n));
    FMM_TRY(ws.sz.ensure(sizeof(double) * n));
    FMM_TRY(ws.sd.ensure(sizeof(double) * n));
    FMM_TRY(ws.smc.ensure(sizeof(double) * (size_t)n * P.dim * 2));
    count_launches(1);
    k_gather<<<grid_for(n, 256), 256, 0, st>>>(n, P.dim, t.perm, P.x, P.mp, P.damp, ws.sx.as<double>(),
                                                ws.sy.as<double>(), ws.sz.as<double>(), ws.sd.as<double>(),
                                                ws.smc.as<double>());
    // original-order scaled multipoles for the exclusion pass
    count_launches(1);
    k_scale_mp<<<grid_for(n, 256), 256, 0, st>>>(n, P.dim, P.mp, ws.smc.as<double>() + (size_t)n * P.dim);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int launch_p2p_f64(Workspace& ws, const Particles& P, const TreeDev& t, int field_order, const Modes& md,
                   cudaStream_t st) {
    const int m = dim_to_order(P.dim);
    if (!near_orders_supported(m, field_order)) return FMM_ENOTSUP;
    const int64_t n = P.n;
    const int nf = nT(field_order);
    FMM_TRY(ws.fsorted.ensure(sizeof(double) * (size_t)n * nf));
    const double* rows = ws.smc.as<double>();
    if (near_row_count(m, field_order) > P.dim) {
        FMM_TRY(ws.near_rows.ensure(sizeof(double) * (size_t)n * near_row_count(m, field_order)));
        count_launches(1);
        k_near_rows<<<grid_for(n, 128), 128, 0, st>>>(n, true, ws.smc.as<double>(), ws.near_rows.as<double>());
        rows = ws.near_rows.as<double>();
    }
    // slices of the near lists while there are fewer than 16 targets per
    // scheduler (a near list holds many steps of 32 sources)
    const int ks = (int)std::max<int64_t>(1, std::min<int64_t>(8, 16LL * 4 * num_sms() / n));
    double* out = ws.fsorted.as<double>();
    if (ks > 1) {
        FMM_TRY(ws.near_part.ensure(sizeof(double) * (size_t)ks * nf * n));
        out = ws.near_part.as<double>();
    }
    const dim3 grid(grid_for(n, 4), (unsigned)ks);
    if (t.nimg > 1) {
        FMM_MF_SWITCH_F64(m, field_order,
                      (k_p2p_f64<MM, FF, true><<<grid, 128, 0, st>>>(
                          t, ws.sx.as<double>(), ws.sy.as<double>(), ws.sz.as<double>(), ws.sd.as<double>(), rows, n,
                          P.damp_type, md.excl_mode, P.exw, P.excl, out)));
    } else {
        FMM_MF_SWITCH_F64(m, field_order,
                      (k_p2p_f64<MM, FF, false><<<grid, 128, 0, st>>>(
                          t, ws.sx.as<double>(), ws.sy.as<double>(), ws.sz.as<double>(), ws.sd.as<double>(), rows, n,
                          P.damp_type, md.excl_mode, P.exw, P.excl, out)));
    }
    if (ks > 1) FMM_TRY(sum_slices(n * nf, ks, out, ws.fsorted.as<double>(), st));
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int launch_excl_correction(Workspace& ws, const Particles& P, const TreeDev* t, int field_order, const Modes& md,
                           double* d_field, cudaStream_t st) {
    if (md.excl_mode == 0 || P.exw == 0) return FMM_OK;  // reference mode leaves far partners in
    const int m = dim_to_order(P.dim);
    const int64_t n = P.n;
    const double* mc_orig = ws.smc.as<double>() + (size_t)n * P.dim;
    FMM_MF_SWITCH_F64(m, field_order,
                  (k_excl_fix<MM, FF><<<grid_for(n, 128), 128, 0, st>>>(
                      n, P.x, mc_orig, P.exw, P.excl, t->pos_of, t->leaf_of, t->near_off, t->near_src, d_field)));
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

int scatter_field(Workspace& ws, const TreeDev& t, int64_t n, int nf, double* d_field, cudaStream_t st) {
    count_launches(1);
    k_scatter<<<grid_for(n, 256), 256, 0, st>>>(n, nf, t.perm, ws.fsorted.as<double>(), d_field);
    FMM_CUDA_TRY(cudaGetLastError());
    return FMM_OK;
}

}  // namespace fmm

// FP64 grouped M2L products on the tensor cores (included by m2l_gemm.cu).
//
// The FP64 pipe gives 1.06 TFLOP/s; the tensor cores multiply 16-bit floats
// exactly and add the products in FP32.  A product C = G W of FP64 matrices is
// therefore evaluated in fixed point (the Ozaki splitting: Ozaki, Ogita,
// Oishi, Rump, Numer. Algorithms 59, 2012): every row of G and every column of
// W gets a power-of-two scale, its entries become 62-bit integers, and those
// eight signed base-256 digits each, which FP16 holds exactly.  Digit products
// of equal weight 256^-d, d = i + j, are accumulated by the tensor cores in one
// FP32 accumulator per weight, and the eight sums are put together in 64-bit
// integers and rounded once to FP64.  The leading digits being at most 64, an
// accumulator holds at most max(d, 1/4) K 2^14, and sums to 2^24 are exact: K is
// taken in segments of kD64Segment chunks (176 components), each of which ends
// in the rounded sum, so that every weight to 256^-5 is exact whatever the digits.
// (256^-6 and 256^-7 could reach 1.03 and 1.2 times 2^24 if all digits were
// extreme and of one sign; 37 and 238 additions would then round by a unit at
// most, which is below an eighth of what the products left out can be.)  Digit
// products below 256^-7 are left out: 36 of 64 remain.  The result is within 2^-60 K of the row scale
// times the column scale, where an FP64 sum rounds K times at 2^-53 of its
// partial sums.  So that a scale fits all the entries it covers, component s is
// weighted by 2^sigma(|s|) ~ |s|! / 3^(|s|/2) in W and the inverse in G: tensors
// of order k grow like k!, and the scaled moments of a particle at its cell's
// corner, sqrt(3) half-widths out, fall like 3^(k/2) / k!.  (With sigma = log2 k!
// a corner's high orders would take 8 bits from the column of order 10.)
// Measured against long-double sums, relative to the sum of the terms'
// magnitudes, at corner moments and D = 8: within 9e-16 at order 10, the FP64
// sum 1.0e-15.
//
// 60,003 particles, order 10, 2.07e6 pairs: the products take 4.7 ms, on the
// FP64 pipe 60.3 ms (80% of its rate).
//
// A task is up to 64 pairs of one group and 128 operator rows: eight
// accumulators of 64 columns fill tensor memory.  Operator chunks (16
// components, eight digits, 32 KB) come by one bulk copy each, the pairs'
// digits by 16-byte gathers, in a ring of four 48 KB stages; per stage 36 MMAs
// of 128 x 64 x 16.
#pragma once

#include <cuda_fp16.h>

#include "internal.h"
#include "m2l_basis.cuh"
#include "umma.cuh"

namespace fmm {

namespace {

constexpr int kDig = 8;            // base-256 digits of an operand entry
constexpr int kD64Rows = 128;      // operator rows per part (MMA M)
constexpr int kD64Pairs = 64;      // pairs per task (MMA N)
constexpr int kD64K = 16;          // components per chunk (MMA K)
constexpr int kD64Stages = 4;
constexpr int kD64Segment = 11;    // chunks per accumulation (reduced basis: all, to order 12)
constexpr int kD64Producers = 64;  // warps 0-1
constexpr int kD64MmaWarp = 2;
constexpr int kD64EpiWarps = 16;
constexpr int kD64Threads = 32 * (3 + kD64EpiWarps);
constexpr int kD64BadExp = 1 << 20;  // column exponent of non-finite weights: their products are NaN
constexpr long long kD64WaitCycles = 4000000000LL;
// Exponents per order of a node's weights and of a group's first row, and (the
// last) the group's scale: 32 bytes each.
constexpr int kD64Orders = 16;
constexpr int kD64NoExp = -32000;  // no such entry
// Bits by which a pair's scales may exceed its largest term (k_m2l_pairs64).
constexpr int kD64Loss = 6;

// Operator rows (and columns) of order q: the reduced basis, or all Cartesian
// components (full).
__host__ __device__ __forceinline__ int d64_rows(int q, bool full) { return full ? nT(q) : (q + 1) * (q + 1); }
__host__ __device__ __forceinline__ int d64_parts(int q, bool full) {
    return (d64_rows(q, full) + kD64Rows - 1) / kD64Rows;
}
__host__ __device__ __forceinline__ int d64_chunks(int q, bool full) {
    return (d64_rows(q, full) + kD64K - 1) / kD64K;
}
constexpr int kD64MaxRows = (nT(kMaxP) + kD64Rows - 1) / kD64Rows * kD64Rows;

// floor(log2(k! / 3^(k/2)))
__device__ __forceinline__ int d64_sigma(int k) {
    constexpr int t[kMaxP + 1] = {0, -1, -1, 0, 1, 2, 4, 6, 8, 11, 13, 16, 19};
    int v = 0;
#pragma unroll
    for (int i = 0; i <= kMaxP; ++i) v = k == i ? t[i] : v;
    return v;
}

// Packed (x, y, z, order) of component s of the basis.
__device__ __forceinline__ int d64_comp(int s, bool full) {
    if (!full) return qcomp(s);
    return comp_x(s) | (comp_y(s) << 8) | (comp_z(s) << 16) | (order_of(s) << 24);
}

// Exponent E of v 2^x (|v 2^x| in [2^E, 2^(E+1))); very small for zero and
// subnormal v.
__device__ __forceinline__ int d64_exp(double v, int x) {
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    return e == 0 ? -100000 : e - 1023 + x;
}
// v 2^(x + 62 - e) rounded to an integer, for |v 2^x| < 2^e.
__device__ __forceinline__ long long d64_fix(double v, int x, int e) {
    const long long b = __double_as_longlong(v);
    const int ex = (int)(b >> 52) & 0x7ff;
    if (ex == 0) return 0;
    const long long m = (b & 0xfffffffffffffll) | 0x10000000000000ll;
    const int sh = ex - 1023 + x - e + 10;
    long long q;
    if (sh >= 0)
        q = m << sh;
    else
        q = sh < -54 ? 0 : (m + (1ll << (-sh - 1))) >> -sh;
    return b < 0 ? -q : q;
}
// Eight entries' digits as FP16, digit i of all eight in out[i] (16 bytes).
__device__ __forceinline__ void d64_digits(const long long (&q)[8], uint4 (&out)[kDig]) {
    long long r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = q[k];
#pragma unroll
    for (int i = kDig - 1; i >= 0; --i) {
        unsigned w[4];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            int d = i == 0 ? (int)r[k] : (int)(signed char)(r[k] & 255);
            r[k] = (r[k] - d) >> 8;
            const unsigned h = __half_as_ushort(__int2half_rn(d));
            w[k >> 1] = (k & 1) ? (w[k >> 1] | (h << 16)) : h;
        }
        out[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
// v 2^e rounded to nearest even; underflow to zero, overflow to infinity.
__device__ __forceinline__ double d64_round(long long v, int e) {
    if (v == 0) return 0.0;
    unsigned long long m = v < 0 ? (unsigned long long)(-v) : (unsigned long long)v;
    const int z = __clzll((long long)m);
    m <<= z;
    const unsigned r = (unsigned)m & 0x7ffu;
    m >>= 11;
    if (r > 0x400u || (r == 0x400u && (m & 1))) ++m;
    const int be = 1023 + 52 + 11 - z + e;  // biased exponent of the leading bit
    unsigned long long b;
    if (be <= 0)
        b = 0;
    else if (be >= 2046)
        b = 0x7ff0000000000000ull;
    else
        b = ((unsigned long long)(be - 1) << 52) + m;
    return __longlong_as_double((long long)(v < 0 ? b | 0x8000000000000000ull : b));
}

// Digits of every node's weights w'_s = w_s / h^|s|, node by node and chunk by
// chunk ([chunk][digit][16]), the node's exponent and those of its orders.  w is
// the reduced weights, or (full) (-1)^(|s|+1) M'_s of the moments.  Warp per node.
__global__ void __launch_bounds__(128) k_weights64(int M, int p, bool full, const double* __restrict__ w,
                                                   const double* __restrict__ h, uint4* __restrict__ dig,
                                                   int* __restrict__ wexp, short* __restrict__ word) {
    __shared__ int eord[4][kD64Orders];
    const int node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (node >= M) return;
    int* eo = eord[threadIdx.x >> 5];
    if (lane < kD64Orders) eo[lane] = kD64NoExp;
    __syncwarp();
    const int K = d64_rows(p, full), pieces = 2 * d64_chunks(p, full);
    const double ih = 1.0 / h[node];
    double pw = 1.0;  // lane j: ih^j
    for (int u = 0; u < min(lane, kMaxP); ++u) pw *= ih;
    const double* wn = w + (size_t)node * K;
    int emax = -100000;
    for (int pass = 0; pass < 2; ++pass) {
        for (int p0 = 0; p0 < pieces; p0 += 32) {
            const int pc = p0 + lane;
            long long q[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int s = 8 * pc + k;
                int o = 0;
                if (s < K) {
                    if (full) o = order_of(s);
                    else while ((o + 1) * (o + 1) <= s) ++o;
                }
                const double sc = __shfl_sync(0xffffffffu, pw, o);
                double v = s < K ? wn[s] * sc : 0.0;
                if (full && (o & 1) == 0) v = -v;
                const int x = d64_sigma(o);
                if (pass == 0) {
                    const bool bad = ((__double2hiint(v) >> 20) & 0x7ff) == 0x7ff;
                    const int e = d64_exp(v, x);
                    emax = max(emax, bad ? kD64BadExp : e);
                    if (s < K && e > kD64NoExp) atomicMax(&eo[o], e);
                } else {
                    q[k] = emax >= kD64BadExp ? 0 : d64_fix(v, x, emax + 1);
                }
            }
            if (pass == 1 && pc < pieces) {
                uint4 d[kDig];
                d64_digits(q, d);
                // uint4 = 8 halves; a digit's 16 components are two of them
                uint4* o = dig + ((size_t)node * (pieces / 2) + (pc >> 1)) * (2 * kDig) + (pc & 1);
#pragma unroll
                for (int i = 0; i < kDig; ++i) o[2 * i] = d[i];
            }
        }
        if (pass == 0)
            for (int off = 16; off > 0; off >>= 1) emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, off));
    }
    if (lane == 0) wexp[node] = emax >= kD64BadExp ? kD64BadExp : emax + 1;
    if (lane < kD64Orders) word[(size_t)node * kD64Orders + lane] = (short)eo[lane];
}

// Bytes / 16 of a group's operator digits.
__global__ void k_op64_sizes(int ng, bool full, const int32_t* __restrict__ gq, int64_t* __restrict__ sz) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g > ng) return;
    sz[g] = g < ng ? (int64_t)d64_parts(gq[g], full) * d64_chunks(gq[g], full) * kDig * kD64Rows * 2 : 0;
}

// Block per group: the digits of G_fs = a^(|f|+1) b^|s| T_{f+s}(D_c)
// 2^-sigma(|s|), part by part and chunk by chunk ([digit][128 x 16] in the
// operand layout), the exponent of every row f, and (gord) those of the first
// row's orders and the largest of 2^-sigma(|f|) G_f, which is what row f weighs in
// the target's potential.  a and b are powers of two and only move exponents.
__global__ void __launch_bounds__(256) k_operator64(bool full, int ldT, const double* __restrict__ gT,
                                                    const int32_t* __restrict__ gq, const float2* __restrict__ gab,
                                                    const int64_t* __restrict__ goff, int g0, int64_t gop_base, int ldr,
                                                    uint4* __restrict__ gop, int* __restrict__ gexp,
                                                    short* __restrict__ gord) {
    __shared__ int dec[nT(kMaxP)], rexp[kD64MaxRows], eord[kD64Orders];
    extern __shared__ double Tsh[];
    const int g = g0 + blockIdx.x, q = gq[g];
    const int K = d64_rows(q, full), nch = d64_chunks(q, full), nrow = d64_parts(q, full) * kD64Rows;
    const int nTq = full ? nT(2 * q) : rbase(2 * q + 1);
    for (int e = threadIdx.x; e < K; e += blockDim.x) dec[e] = d64_comp(e, full);
    for (int e = threadIdx.x; e < nTq; e += blockDim.x) Tsh[e] = gT[(size_t)g * ldT + e];
    const float2 ab = gab[g];
    const int ea = ((__float_as_int(ab.x) >> 23) & 255) - 127, eb = ((__float_as_int(ab.y) >> 23) & 255) - 127;
    if (threadIdx.x < kD64Orders) eord[threadIdx.x] = kD64NoExp;
    __syncthreads();
    auto entry = [&](int cf, int cs, int* x) {
        const int tx = (cs & 0xff) + (cf & 0xff), ty = ((cs >> 8) & 0xff) + ((cf >> 8) & 0xff),
                  tz = ((cs >> 16) & 0xff) + ((cf >> 16) & 0xff);
        *x = ea * ((cf >> 24) + 1) + eb * (cs >> 24) - d64_sigma(cs >> 24);
        return Tsh[full ? pidx(tx, ty, tz) : ridx(tx, ty, tz)];
    };
    const int lane = threadIdx.x & 31;
    for (int f = threadIdx.x >> 5; f < nrow; f += blockDim.x >> 5) {
        int emax = -100000;
        if (f < K)
            for (int s = lane; s < K; s += 32) {
                int x;
                const double v = entry(dec[f], dec[s], &x);
                const int e = d64_exp(v, x);
                emax = max(emax, e);
                if (f == 0 && e > kD64NoExp) atomicMax(&eord[dec[s] >> 24], e);
            }
        for (int off = 16; off > 0; off >>= 1) emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, off));
        if (lane == 0) {
            rexp[f] = emax + 1;
            if (f < ldr) gexp[(size_t)g * ldr + f] = emax + 1;
            if (f < K) atomicMax(&eord[kD64Orders - 1], emax - d64_sigma(dec[f] >> 24));
        }
    }
    __syncthreads();
    if (threadIdx.x < kD64Orders) gord[(size_t)g * kD64Orders + threadIdx.x] = (short)eord[threadIdx.x];
    uint4* out = gop + (goff[g] - gop_base);
    for (int it = threadIdx.x; it < nrow * nch * 2; it += blockDim.x) {
        // consecutive threads: consecutive rows of one (part, chunk, half of K)
        const int r = it % kD64Rows, b = it / kD64Rows;
        const int kh = b & 1, ch = (b >> 1) % nch, part = (b >> 1) / nch;
        const int f = part * kD64Rows + r;
        long long qv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int s = ch * kD64K + kh * 8 + k;
            qv[k] = 0;
            if (f < K && s < K) {
                int x;
                const double v = entry(dec[f], dec[s], &x);
                qv[k] = d64_fix(v, x, rexp[f]);
            }
        }
        uint4 d[kDig];
        d64_digits(qv, d);
        // core matrices of 8 rows x 8 halves (8 uint4), the two of a row group adjacent
        uint4* o = out + (size_t)(part * nch + ch) * kDig * kD64Rows * 2 + (r >> 3) * 16 + kh * 8 + (r & 7);
#pragma unroll
        for (int i = 0; i < kDig; ++i) o[(size_t)i * kD64Rows * 2] = d[i];
    }
}

struct D64Smem {
    static constexpr uint32_t g_bytes = kDig * kD64Rows * kD64K * 2;   // operator chunk, all digits
    static constexpr uint32_t w_bytes = kDig * kD64Pairs * kD64K * 2;  // weight chunk, all digits
    static constexpr size_t stage_bytes = g_bytes + w_bytes;
    static constexpr size_t off_bar = kD64Stages * stage_bytes;
    // full[S], empty[S], acc_full, acc_empty
    static constexpr size_t off_tmem = off_bar + sizeof(uint64_t) * (2 * kD64Stages + 2);
    static constexpr size_t bytes = off_tmem + 16;
};
static_assert(D64Smem::bytes <= 227 * 1024, "shared memory of one SM");

// Source nodes of a producer thread's pairs 8 k + rsub (k < 8) of a task.
__device__ __forceinline__ void d64_load_rows(int2 tk, const int32_t* __restrict__ gstart,
                                              const int32_t* __restrict__ psrc, int rsub, int (&r)[kD64Pairs / 8]) {
    const int gs = gstart[tk.x] + (tk.y >> 2), cnt = min(kD64Pairs, gstart[tk.x + 1] - gs);
#pragma unroll
    for (int k = 0; k < kD64Pairs / 8; ++k) {
        const int pr = 8 * k + rsub;
        r[k] = pr < cnt ? psrc[gs + pr] : -1;
    }
}

// Tasks (group, 4 x first pair + part).  Result rows of rl(q) entries per pair
// in group order, from rowbase[g] x row_unit entries of out.
__global__ void __launch_bounds__(kD64Threads, 1) k_m2l_tc64(const int2* __restrict__ tasks, int ntasks, bool full,
                                                            const int32_t* __restrict__ gstart,
                                                            const int32_t* __restrict__ gq,
                                                            const int64_t* __restrict__ goff, int64_t gop_base,
                                                            const uint4* __restrict__ gop, int ldr,
                                                            const int* __restrict__ gexp,
                                                            const int32_t* __restrict__ psrc,
                                                            const uint4* __restrict__ wdig, int wchunks,
                                                            const int* __restrict__ wexp, double* __restrict__ out,
                                                            const int64_t* __restrict__ rowbase, int row_unit,
                                                            int* __restrict__ err) {
    extern __shared__ __align__(1024) char sm_d64[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint64_t* fullb = reinterpret_cast<uint64_t*>(sm_d64 + D64Smem::off_bar);
    uint64_t* empty = fullb + kD64Stages;
    uint64_t* acc_full = empty + kD64Stages;
    uint64_t* acc_empty = acc_full + 1;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm_d64 + D64Smem::off_tmem);
    if (warp == 0) {
        umma::tmem_alloc(tslot, kDig * kD64Pairs);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        for (int st = 0; st < kD64Stages; ++st) {
            umma::mbar_init(&fullb[st], kD64Producers + 1);  // producers' cp.async arrivals + the bulk copy's
            umma::mbar_init(&empty[st], 1);
        }
        umma::mbar_init(acc_full, 1);
        umma::mbar_init(acc_empty, kD64EpiWarps);
        umma::mbar_fence_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;
    bool ok = true;
    if (warp < kD64Producers / 32) {
        // ---- producers: per instruction 8 pairs x two 16-byte pieces x two
        // digits (512 bytes over all shared-memory banks)
        const int rsub = lane & 7, j = (lane >> 3) & 1, dsub = lane >> 4;
        const uint64_t keep = umma::l2_evict_last();
        uint32_t u = 0;
        int rows[kD64Pairs / 8];
        for (int task = blockIdx.x; task < ntasks && ok; task += gridDim.x) {
            const int2 tk = tasks[task];
            const int nch = d64_chunks(gq[tk.x], full);
            d64_load_rows(tk, gstart, psrc, rsub, rows);
            const uint4* G = gop + (goff[tk.x] - gop_base) + (size_t)(tk.y & 3) * nch * (D64Smem::g_bytes / 16);
            for (int ch = 0; ch < nch; ++ch, ++u) {
                const int st = (int)(u % kD64Stages);
                if (u >= (uint32_t)kD64Stages &&
                    !umma::mbar_wait(&empty[st], ((u / kD64Stages) - 1) & 1, kD64WaitCycles)) {
                    ok = false;
                    break;
                }
                char* Gs = sm_d64 + (size_t)st * D64Smem::stage_bytes;
                char* Ws = Gs + D64Smem::g_bytes;
                if (tid == 0) {
                    umma::mbar_arrive_expect_tx(&fullb[st], D64Smem::g_bytes);
                    umma::bulk_g2s(Gs, G + (size_t)ch * (D64Smem::g_bytes / 16), D64Smem::g_bytes, &fullb[st]);
                }
#pragma unroll
                for (int dp = 0; dp < kDig / 4; ++dp) {
                    // this warp's digits: 2 (2 dp + warp) + dsub
                    const int dg = 2 * (2 * dp + warp) + dsub;
#pragma unroll
                    for (int k = 0; k < kD64Pairs / 8; ++k) {
                        const int src = rows[k];
                        const uint4* gsrc =
                            src >= 0 ? wdig + ((size_t)src * wchunks + ch) * (2 * kDig) + 2 * dg + j : wdig;
                        umma::cp16_keep(Ws + dg * (kD64Pairs * kD64K * 2) + k * 256 + j * 128 + rsub * 16, gsrc,
                                        src >= 0, keep);
                    }
                }
                umma::cp_async_mbar_arrive(&fullb[st]);
            }
        }
    } else if (warp == kD64MmaWarp) {
        // ---- MMA issue (one thread)
        if (lane == 0) {
            uint32_t u = 0, tl = 0;
            const uint32_t idesc = umma::idesc_f16(kD64Rows, kD64Pairs);
            constexpr uint32_t LBO = 128, SBO = 256;
            for (int task = blockIdx.x; task < ntasks && ok; task += gridDim.x) {
                const int nch = d64_chunks(gq[tasks[task].x], full);
                for (int c0 = 0; c0 < nch && ok; c0 += kD64Segment) {
                    if (tl >= 1 && !umma::mbar_wait(acc_empty, (tl - 1) & 1, kD64WaitCycles)) {
                        ok = false;
                        break;
                    }
                    umma::fence_after_sync();
                    for (int ch = c0; ch < min(nch, c0 + kD64Segment); ++ch, ++u) {
                        const int st = (int)(u % kD64Stages);
                        if (!umma::mbar_wait(&fullb[st], (u / kD64Stages) & 1, kD64WaitCycles)) {
                            ok = false;
                            break;
                        }
                        umma::fence_proxy_async();
                        umma::fence_after_sync();
                        const char* Gs = sm_d64 + (size_t)st * D64Smem::stage_bytes;
                        const char* Ws = Gs + D64Smem::g_bytes;
#pragma unroll 1
                        for (int i = 0; i < kDig; ++i) {
                            const uint64_t a = umma::smem_desc(Gs + i * (kD64Rows * kD64K * 2), LBO, SBO);
#pragma unroll 1
                            for (int k = 0; k < kDig - i; ++k)
                                umma::mma_f16(tmem + (uint32_t)((i + k) * kD64Pairs), a,
                                              umma::smem_desc(Ws + k * (kD64Pairs * kD64K * 2), LBO, SBO), idesc,
                                              (ch > c0 || i > 0) ? 1u : 0u);
                        }
                        umma::commit(&empty[st]);
                    }
                    if (!ok) break;
                    umma::commit(acc_full);
                    ++tl;
                }
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. + 31,
        // eight pairs at a time, each of the sub-partition's warps a quarter
        // of the pairs
        const int sp = warp & 3, share = (warp - 3) / 4;
        constexpr int kShares = kD64EpiWarps / 4, CB = 8;
        uint32_t tl = 0;
        for (int task = blockIdx.x; task < ntasks && ok; task += gridDim.x) {
            const int2 tk = tasks[task];
            const int g = tk.x, q = gq[g];
            const int f0 = kD64Rows * (tk.y & 3), f = f0 + 32 * sp + lane;
            const int first = tk.y >> 2, gs = gstart[g] + first, cnt = min(kD64Pairs, gstart[g + 1] - gs);
            const int K = d64_rows(q, full), rl = (K + row_unit - 1) / row_unit * row_unit;
            const int ef = f < K ? gexp[(size_t)g * ldr + f] : 0;
            double* gout = out + (size_t)rowbase[g] * row_unit + (size_t)first * rl;
            const int nch = d64_chunks(q, full);
            const uint32_t base = tmem + ((uint32_t)(32 * sp) << 16);
            for (int c0 = 0; c0 < nch; c0 += kD64Segment, ++tl) {
                if (!umma::mbar_wait(acc_full, tl & 1, kD64WaitCycles)) {
                    ok = false;
                    break;
                }
                umma::fence_after_sync();
#pragma unroll 1
                for (int c = share * CB; c < cnt && f0 + 32 * sp < rl; c += kShares * CB) {
                    float v[kDig][CB];
                    __syncwarp();
#pragma unroll
                    for (int d = 0; d < kDig; ++d) umma::tmem_ld8(base + (uint32_t)(d * kD64Pairs + c), v[d]);
                    umma::tmem_ld_wait();
#pragma unroll
                    for (int d = 0; d < kDig; ++d) umma::tmem_landed(v[d]);
#pragma unroll
                    for (int jj = 0; jj < CB; ++jj) {
                        if (c + jj < cnt) {
                            // sum of the accumulators 256^-d: (hi 2^32 + lo) units of
                            // 2^(ef + ew - 68)
                            const int ew = wexp[psrc[gs + c + jj]];
                            long long hi = 0, lo = 0;
#pragma unroll
                            for (int d = 0; d < 4; ++d) hi = (hi << 8) + (long long)__float2int_rn(v[d][jj]);
#pragma unroll
                            for (int d = 4; d < 8; ++d) lo = (lo << 8) + (long long)__float2int_rn(v[d][jj]);
                            // as many bits of lo as hi leaves room for (|hi| < 2^46)
                            const int up = min(32, __clzll(hi < 0 ? ~hi : hi) - 2);
                            double r = d64_round((hi << up) + (lo >> (32 - up)), ef + ew - 36 - up);
                            if (ew >= kD64BadExp) r = __longlong_as_double(0x7ff8000000000000ll);
                            double* o = gout + (size_t)(c + jj) * rl + f;
                            if (c0 == 0) {
                                if (f < rl) __stcs(o, f < K ? r : 0.0);
                            } else if (f < K) {
                                *o += r;  // (this thread's, of the segments before)
                            }
                        }
                    }
                }
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) umma::mbar_arrive(acc_empty);
            }
        }
    }
    if (!ok) atomicExch(err, 1);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, kDig * kD64Pairs);
}

// Pairs whose scales exceed their terms: FP64 sums in place of the products.  The
// products' error follows the row's scale times the column's, which can lie far
// above the largest term: quadrupoles without charges in a fine cell meet the
// row's third order, (h_j / D)^2 below its first.  With the exponents e_k of the
// node's orders, r_k of the group's first row (which is of the potential's size)
// and S of all rows, S + max e - max (r_k + e_k) bits are lost.  Emulated against
// long double at orders 5 to 12, D from 1.3 to 20 half-widths, level differences
// to 4, charges, dipoles, quadrupoles and all of them, the products' error is 0.1 to
// 0.65 of an FP64 sum's to 6 bits, as large at 7, and then doubles with each.
// A thread checks a pair, a warp sums one (a task's first part does the whole row).
__global__ void __launch_bounds__(128) k_m2l_pairs64(const int2* __restrict__ tasks, int ntasks, bool full,
                                                     const int32_t* __restrict__ gstart,
                                                     const int32_t* __restrict__ gq, const float2* __restrict__ gab,
                                                     const double* __restrict__ gT, int ldT,
                                                     const short* __restrict__ gord, const int32_t* __restrict__ psrc,
                                                     const double* __restrict__ w, int ldw,
                                                     const double* __restrict__ h, const short* __restrict__ word,
                                                     const int* __restrict__ wexp, double* __restrict__ out,
                                                     const int64_t* __restrict__ rowbase, int row_unit) {
    extern __shared__ double sm_pairs64[];
    __shared__ int list[kD64Pairs], count, dec[nT(kMaxP)];
    static_assert(kD64Pairs <= 128, "a thread per pair");
    double* T = sm_pairs64;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double* ws = T + ldT + warp * ldw;
    if (tid == 0) count = 0;
    __syncthreads();
    for (int task = blockIdx.x; task < ntasks; task += gridDim.x) {
        const int2 tk = tasks[task];
        if ((tk.y & 3) != 0) continue;
        const int g = tk.x, first = tk.y >> 2, gs = gstart[g] + first, cnt = min(kD64Pairs, gstart[g + 1] - gs);
        bool lossy = false;
        if (tid < cnt) {
            const int src = psrc[gs + tid];
            const uint4* ep = reinterpret_cast<const uint4*>(word) + 2 * (size_t)src;
            const uint4* rp = reinterpret_cast<const uint4*>(gord) + 2 * (size_t)g;
            const uint4 e0 = ep[0], e1 = ep[1], r0 = rp[0], r1 = rp[1];
            const unsigned ev[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
            const unsigned rv[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
            auto at = [](const unsigned (&v)[8], int k) { return (int)(short)(v[k >> 1] >> (16 * (k & 1))); };
            int emax = kD64NoExp, term = 2 * kD64NoExp;
#pragma unroll
            for (int k = 0; k <= kMaxP; ++k) {
                emax = max(emax, at(ev, k));
                term = max(term, at(ev, k) + at(rv, k));
            }
            lossy = emax > kD64NoExp && at(rv, kD64Orders - 1) + emax - term > kD64Loss && wexp[src] < kD64BadExp;
            if (lossy) list[atomicAdd(&count, 1)] = tid;
        }
        const int n = __syncthreads_count(lossy);
        if (n == 0) continue;
        const int q = gq[g], K = d64_rows(q, full), rl = (K + row_unit - 1) / row_unit * row_unit;
        for (int e = tid; e < (full ? nT(2 * q) : rbase(2 * q + 1)); e += blockDim.x) T[e] = gT[(size_t)g * ldT + e];
        for (int e = tid; e < K; e += blockDim.x) dec[e] = d64_comp(e, full);
        __syncthreads();
        const double a = gab[g].x, b = gab[g].y;
        for (int l = warp; l < n; l += 4) {
            const int pr = list[l], src = psrc[gs + pr];
            const double bh = b / h[src];
            for (int s = lane; s < K; s += 32) {
                const int o = dec[s] >> 24;
                double v = w[(size_t)src * ldw + s];
                for (int k = 0; k < o; ++k) v *= bh;
                ws[s] = full && (o & 1) == 0 ? -v : v;
            }
            __syncwarp();
            double* row = out + (size_t)rowbase[g] * row_unit + (size_t)(first + pr) * rl;
            for (int f = lane; f < rl; f += 32) {
                double v = 0.0;
                if (f < K) {
                    const int cf = dec[f];
                    for (int s = 0; s < K; ++s) {
                        const int c = cf + dec[s], x = c & 0xff, y = (c >> 8) & 0xff, z = (c >> 16) & 0xff;
                        v = fma(T[full ? pidx(x, y, z) : ridx(x, y, z)], ws[s], v);
                    }
                    for (int k = 0; k <= (cf >> 24); ++k) v *= a;
                }
                row[f] = v;
            }
            __syncwarp();
        }
        __syncthreads();
        if (tid == 0) count = 0;
        __syncthreads();
    }
}

}  // namespace

}  // namespace fmm

// PNAMP kernels for GB300 (sm_103a): the per-point algebra in FP64 (zc) or double-float
// (zd, float pairs on the FP32 pipes), one template.
//
// Work decomposition (one CUDA launch per stage, batched over pairs):
//   setup_kernel   four CTAs per (q,q') pair: W = V1 U1^-1, Z0 = V0 U0^-1, the
//                  bare-vacuum overlaps det(1 + Z^T Z)^(-1/4) (zbareover,
//                  Codes/PNAMP/PNAMP_Proj.f90:6-79), the once-per-pair pieces of the
//                  Pfaffians and what kind of points the pair has (pair_kind).
//   point_kernel   persistent; per Euler point the block-diagonal Wigner-D rotation R
//                  (ROTATION_MAT, PNAMP_Proj.f90:83-136) and what of it does not depend on
//                  the gauge angles, then per gauge point the norm (Pfaf_Over + ZPfaffianF +
//                  ZExch, PNAMP_Proj.f90:142-392), rho, kappa10, kappa01 (ROKAPPAphiomega,
//                  :459-551) and the observables of Kernel3D.f90:296-358 (ZN_0, the energy of
//                  PNAMP_Energy_OpenMP.f90:31-90 or the split-bf16 rows for the tensor-core
//                  contraction in contract_tc.cu, ZJ2_0, ZQ2/ZQ2t), summed into ZRES(iang, io)
//                  (Kernel3D.f90:385-387). Three bodies by the kind of pair:
//     split_items    (point_reduced.cuh) no proton-neutron blocks: 2 NFOM problems of order n/2 per
//                    Euler point, one per species and angle, by one skew inverse where U0 and
//                    V1 are well conditioned, by T22 where only V0 is;
//     reduced_item   (point_reduced.cuh) U0 and V1 well conditioned: NFOM^2 problems of order n;
//     full_item      the rest (nearly empty or nearly full levels): Pfaffian of the n x n
//                    Schur complement or the 2n x 2n matrix, Gauss-Jordan solve Y T22^-1.
//   project_kernel J/K projection of ZRES (Kernel3D.f90:415-751, plain form of
//                  PNAMP_Kernel3D_v2.f90:477-498).
//
// Algebra of full_item instead of the reference's per-point LU inverses (exact in exact
// arithmetic): with A = D_phi R, D_phi = diag(e^{i phi_p}, e^{i phi_n}),
//   conj(Vbar1) conj(Ubar1)^-1 = A V1 U1^-1 A^T = D (R W R^T) D,
//   T22 = V0^T A V1 + U0^T A* U1 = sum_s e^{+-i phi_s} (species partials),
//   rho = D (R V1 T22^-1) V0^T, kappa10 = D (R V1 T22^-1) U0^T,
//   kappa01 = -D* (R* U1 T22^-1) V0^T.
// Measured on GB300, pf shell (n = 40), Euler 10 x 20 x 10, gauge 9 x 9, one pair: charge-conserving
// FP64 195.3 -> 9.1 ms and double-float 74.7 -> 4.2 ms, proton-neutron mixing with the BF16x6
// contraction 193.3 -> 66.5 ms, against full_item's algebra for every pair (two points in flight
// for charge-conserving ones).
#pragma once
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "pnamp_df64.cuh"
#include "../../include/pnamp_gpu.h"
#include "pnamp_internal.h"

namespace pnamp {

// A value as S = 2 or 3 bf16 terms t0 + t1 (+ t2), each the bf16 rounding of what the
// previous terms leave (8 significant bits each: ~2^-17 relative left for S = 2, ~2^-25 for
// S = 3). v - t0 is exact in FP32 (t0 is v rounded to 8 bits); the double-float low word
// enters the first remainder.
__device__ __forceinline__ void bf16_terms(dd v, int S, unsigned short (&t)[3]) {
    const __nv_bfloat16 b0 = __float2bfloat16_rn(v.hi);
    const float r1 = __fadd_rn(__fsub_rn(v.hi, __bfloat162float(b0)), v.lo);
    const __nv_bfloat16 b1 = __float2bfloat16_rn(r1);
    const float r2 = __fsub_rn(r1, __bfloat162float(b1));
    t[0] = __bfloat16_as_ushort(b0);
    t[1] = __bfloat16_as_ushort(b1);
    t[2] = S > 2 ? __bfloat16_as_ushort(__float2bfloat16_rn(r2)) : (unsigned short)0;
}
__device__ __forceinline__ dd as_dd(double v) { return dd_from(v); }
__device__ __forceinline__ dd as_dd(dd v) { return v; }

// ------------------------------------------------------------------ scalars
__device__ __forceinline__ double sabs1(double a) { return fabs(a); }
__device__ __forceinline__ double sabs1(zc a) { return fabs(a.x) + fabs(a.y); }
__device__ __forceinline__ double srecip(double a) { return 1.0 / a; }
__device__ __forceinline__ zc srecip(zc a) { return zrecip(a); }
__device__ __forceinline__ double smul(double a, double b) { return a * b; }
__device__ __forceinline__ zc smul(zc a, zc b) { return a * b; }
__device__ __forceinline__ double sfms(double a, double b, double c) { return fma(-a, b, c); }
__device__ __forceinline__ zc sfms(zc a, zc b, zc c) { return zfms(a, b, c); }
template <typename T> __device__ __forceinline__ T szero();
template <> __device__ __forceinline__ double szero<double>() { return 0.0; }
template <> __device__ __forceinline__ zc szero<zc>() { return mk(0.0, 0.0); }
// pivot magnitude of a double-float value: the float sum of the high words, compared as a
// float (the FP64 pipe is narrow on this part, and a float compares the same as its double)
__device__ __forceinline__ float sabs1(zd a) { return fabsf(f2_a(a.hi)) + fabsf(f2_b(a.hi)); }
__device__ __forceinline__ zd srecip(zd a) { return zrecip(a); }
__device__ __forceinline__ zd smul(zd a, zd b) { return a * b; }
__device__ __forceinline__ zd sfms(zd a, zd b, zd c) { return zfms(a, b, c); }
template <> __device__ __forceinline__ zd szero<zd>() { return mkd(dd_make(0.0f, 0.0f), dd_make(0.0f, 0.0f)); }

// Arithmetic traits of the per-point algebra: zc = FP64 complex (plain form),
// zd = double-float complex (df64 form). R is the matching real type.
template <class Z> struct Ar;
template <> struct Ar<zc> {
    using R = double;
    static __device__ __forceinline__ zc from(zc a) { return a; }
    static __device__ __forceinline__ zc to(zc a) { return a; }
    static __device__ __forceinline__ R real(double v) { return v; }
    static __device__ __forceinline__ R rmul(R a, R b) { return a * b; }
    static __device__ __forceinline__ bool nz(R a) { return a != 0.0; }
    static __device__ __forceinline__ R pick(const double *d, const dd *, long long i) { return d[i]; }
    static __device__ __forceinline__ R rzero() { return 0.0; }
    static __device__ __forceinline__ zc neg_real(R a) { return mk(-a, 0.0); }
    static __device__ __forceinline__ R rneg(R a) { return -a; }
    static __device__ __forceinline__ R rconst(float v) { return (double)v; }   // exact
    static __device__ __forceinline__ R radd(R a, R b) { return a + b; }
    static __device__ __forceinline__ R rfma(R a, R b, R c) { return fma(a, b, c); }
    static __device__ __forceinline__ double dbl(R a) { return a; }
    static __device__ __forceinline__ R wsum(R v) {   // butterfly: the sum in every lane
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
    // pivot key: max(|re|, |im|) as the bit pattern of a non-negative double
    static __device__ __forceinline__ unsigned long long key(zc z) {
        const unsigned long long kx = (unsigned long long)__double_as_longlong(z.x) & 0x7fffffffffffffffull;
        const unsigned long long ky = (unsigned long long)__double_as_longlong(z.y) & 0x7fffffffffffffffull;
        return kx > ky ? kx : ky;
    }
};
template <> struct Ar<zd> {
    using R = dd;
    static __device__ __forceinline__ zd from(zc a) { return zd_from(a); }
    static __device__ __forceinline__ zc to(zd a) { return zd_to(a); }
    static __device__ __forceinline__ R real(double v) { return dd_from(v); }
    static __device__ __forceinline__ R rmul(R a, R b) { return dd_mul(a, b); }
    static __device__ __forceinline__ bool nz(R a) { return a.hi != 0.0f; }
    static __device__ __forceinline__ R pick(const double *, const dd *f, long long i) { return f[i]; }
    static __device__ __forceinline__ R rzero() { return dd_make(0.0f, 0.0f); }
    static __device__ __forceinline__ zd neg_real(R a) { return mkd(dd_neg(a), dd_make(0.0f, 0.0f)); }
    static __device__ __forceinline__ R rneg(R a) { return dd_neg(a); }
    static __device__ __forceinline__ R rconst(float v) { return dd_make(v, 0.0f); }   // exact
    static __device__ __forceinline__ R radd(R a, R b) { return dd_add(a, b); }
    static __device__ __forceinline__ R rfma(R a, R b, R c) { return dd_fma(a, b, c); }
    static __device__ __forceinline__ double dbl(R a) { return dd_to(a); }
    static __device__ __forceinline__ R wsum(R v) {   // in double-float on the FP32 pipes
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v = dd_add(v, dd_make(__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)));
        return v;
    }
    static __device__ __forceinline__ unsigned long long key(zd z) {
        const unsigned int kx = __float_as_uint(f2_a(z.hi)) & 0x7fffffffu;
        const unsigned int ky = __float_as_uint(f2_b(z.hi)) & 0x7fffffffu;
        return kx > ky ? kx : ky;
    }
};


// Pivot row for column k (largest |re|+|im|, first on ties, as IZAMAX): warp 0
// searches, the result is broadcast through sh[0] (row) and sh[1] (zero column).
template <typename T>
__device__ __forceinline__ int pivot_search(const T *A, int lda, int k, int n, int *sh, T *invd, bool &zero) {
    using Mag = decltype(sabs1(A[0]));
    if (threadIdx.x < 32) {
        Mag v = -1;
        int idx = 0x7fffffff;
        for (int i = k + (int)threadIdx.x; i < n; i += 32) {
            const Mag a = sabs1(A[i * lda + k]);
            if (a > v) {
                v = a;
                idx = i;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const Mag ov = __shfl_down_sync(0xffffffffu, v, o);
            const int oi = __shfl_down_sync(0xffffffffu, idx, o);
            if (ov > v || (ov == v && oi < idx)) {
                v = ov;
                idx = oi;
            }
        }
        if (threadIdx.x == 0) {
            // no comparable entry (all NaN): report a zero column, keep row k
            const bool none = (idx == 0x7fffffff);
            const bool z = none || v == Mag(0);
            sh[0] = none ? k : idx;
            sh[1] = z ? 1 : 0;
            invd[k] = z ? szero<T>() : srecip(A[(none ? k : idx) * lda + k]);
        }
    }
    __syncthreads();
    zero = sh[1] != 0;
    return sh[0];
}

// In-place LU with partial pivoting, P A = L U (L unit lower). perm[k] is the
// row exchanged with row k at step k (LAPACK ipiv, 0-based); invd[k] = 1/U_kk.
// Returns true if an exactly zero pivot column was met.
template <typename T>
__device__ bool lu_factor(T *A, int n, int lda, int *perm, T *invd, int *sh) {
    bool sing = false;
    for (int k = 0; k < n; ++k) {
        bool zero;
        const int p = pivot_search(A, lda, k, n, sh, invd, zero);
        if (p != k)
            for (int j = threadIdx.x; j < n; j += blockDim.x) {
                const T t = A[k * lda + j];
                A[k * lda + j] = A[p * lda + j];
                A[p * lda + j] = t;
            }
        if (threadIdx.x == 0) perm[k] = p;
        __syncthreads();
        if (zero) {
            sing = true;
            continue;
        }
        const T inv = invd[k];
        for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) A[i * lda + k] = smul(A[i * lda + k], inv);
        __syncthreads();
        const int m = n - k - 1;
        if (m > 0) {
            const int dq = blockDim.x / m, dr = blockDim.x % m;
            int i = k + 1 + threadIdx.x / m, j = k + 1 + threadIdx.x % m;
            for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
                A[i * lda + j] = sfms(A[i * lda + k], A[k * lda + j], A[i * lda + j]);
                i += dq;
                j += dr;
                if (j >= k + 1 + m) {
                    j -= m;
                    ++i;
                }
            }
        }
        __syncthreads();
    }
    return sing;
}

// Warp argmax by one integer max-reduction (redux.sync): the key of candidate j (offset
// jrel = j - j0 < 64) is the magnitude's bit pattern (a non-negative float compares like its
// bits) with the low 6 bits replaced by 63 - jrel, so the largest magnitude wins and ties go
// to the first column, magnitudes being compared to 2^-17 relative. Lanes pass their best key
// (0 for no candidate). Returns the winning offset in bits 0..5 of the reduced key; the key's
// magnitude part is 0 when every candidate was zero (or not a number, which counts as zero).
__device__ __forceinline__ unsigned pack_key(float mag, int jrel) {
    return (mag >= 0.0f ? (__float_as_uint(mag) & ~63u) : 0u) | (unsigned)(63 - jrel);
}
static_assert(PNAMP_MAX_NLEV <= 64, "pivot offsets are packed into 6 bits (7 for the 2n x 2n Pfaffian)");

// A warp-aligned group of the CTA's threads that owns one problem, with its named barrier
// (bar.sync id, count); a one-warp group needs only __syncwarp.
struct Grp {
    int tid, nthr, bar;
};
__device__ __forceinline__ void gsync(const Grp &g) {
    if (g.nthr == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(g.bar), "r"(g.nthr) : "memory");
}

// Y <- Y A^-1 (Y: ny x n, A: n x n, both row-major with leading dimension n) by
// column-oriented Gauss-Jordan elimination: column operations E reduce A to the
// identity (A E = I, so E = A^-1), and the same operations applied to the rows of Y
// give Y A^-1. Step k takes the pivot in row k (largest |A_kc|, c >= k; partial
// pivoting on A^T), moves column c to k, scales it and removes row k from every other
// column. Rows < k of A are unit rows by then and are not touched again. Two barriers
// per step and (n - k - 1 + ny)(n - 1) independent updates per step, against the
// 2n + n sequential steps of an LU followed by two triangular column sweeps: the
// elimination is latency-bound at these sizes, so fewer, fuller steps win although
// the flop count is higher. A holds garbage on return; prow (n) and pinv (1) are
// shared scratch. Returns true if an exactly zero pivot row was met.
template <typename T>
__device__ bool gj_right_solve(T *A, int n, T *Y, int ny, T *prow, T *pinv, int *sh) {
    const int lane = threadIdx.x & 31;
    auto search = [&](int k) {  // warp 0: pivot column of row k -> sh[0], zero flag sh[1], pinv[0]
        if constexpr (std::is_same<T, zd>::value) {   // one redux.sync
            unsigned key = 0u;
            for (int j = k + lane; j < n; j += 32) {
                const unsigned kk = pack_key(sabs1(A[k * n + j]), j - k);
                key = key > kk ? key : kk;
            }
            const unsigned m = __reduce_max_sync(0xffffffffu, key);
            if (lane == 0) {
                const int idx = k + 63 - (int)(m & 63u);
                const bool z = (m >> 6) == 0u;
                sh[0] = idx;
                sh[1] = z ? 1 : 0;
                pinv[0] = z ? szero<T>() : srecip(A[k * n + idx]);
            }
        } else {
            using Mag = decltype(sabs1(A[0]));
            Mag v = -1;
            int idx = 0x7fffffff;
            for (int j = k + lane; j < n; j += 32) {
                const Mag a = sabs1(A[k * n + j]);
                if (a > v) {
                    v = a;
                    idx = j;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const Mag ov = __shfl_down_sync(0xffffffffu, v, o);
                const int oi = __shfl_down_sync(0xffffffffu, idx, o);
                if (ov > v || (ov == v && oi < idx)) {
                    v = ov;
                    idx = oi;
                }
            }
            if (lane == 0) {
                const bool none = (idx == 0x7fffffff);  // all NaN: keep column k, report zero
                const bool z = none || v == Mag(0);
                sh[0] = none ? k : idx;
                sh[1] = z ? 1 : 0;
                pinv[0] = z ? szero<T>() : srecip(A[k * n + (none ? k : idx)]);
            }
        }
    };
    bool sing = false;
    if (threadIdx.x < 32) search(0);
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        const int c = sh[0];
        if (sh[1]) sing = true;
        const T pv = pinv[0];
        // phase 1: each remaining row r gets m_r = M[r][c] / A[k][c] in column k and its old
        // column k in column c; the pivot row (columns k and c exchanged) goes to prow
        const int nrT = n - k - 1, nrows = nrT + ny;
        for (int t = threadIdx.x; t < nrows + n; t += blockDim.x) {
            if (t < nrows) {
                T *row = t < nrT ? A + (long long)(k + 1 + t) * n : Y + (long long)(t - nrT) * n;
                const T a = row[c], b = row[k];
                row[k] = smul(a, pv);
                if (c != k) row[c] = b;
            } else {
                const int j = t - nrows;
                prow[j] = (j == c) ? A[k * n + k] : A[k * n + j];
            }
        }
        __syncthreads();
        // phase 2: M[r][j] -= m_r prow[j] for j != k. Warp 0 takes row k + 1 of A and then
        // searches its pivot, so the next step needs no extra barrier.
        if (threadIdx.x < 32) {
            if (k + 1 < n) {
                T *row = A + (long long)(k + 1) * n;
                const T m = row[k];
                for (int j = lane; j < n; j += 32)
                    if (j != k) row[j] = sfms(m, prow[j], row[j]);
                __syncwarp();
                search(k + 1);
            }
        } else {
            const int nrA = n - k - 2 > 0 ? n - k - 2 : 0;
            const int total = (nrA + ny) * n, stride = blockDim.x - 32;
            const int dq = stride / n, dr = stride % n;
            int rr = (threadIdx.x - 32) / n, j = (threadIdx.x - 32) % n;
            for (int t = threadIdx.x - 32; t < total; t += stride) {
                if (j != k) {
                    T *row = rr < nrA ? A + (long long)(k + 2 + rr) * n : Y + (long long)(rr - nrA) * n;
                    row[j] = sfms(row[k], prow[j], row[j]);
                }
                rr += dq;
                j += dr;
                if (j >= n) {
                    j -= n;
                    ++rr;
                }
            }
        }
        __syncthreads();
    }
    return sing;
}

// gj_right_solve by the thread group g (its first warp searches the pivots): prow holds n
// scratch values, pinv 1, sh 2 ints. Runs beside the Pfaffian elimination of the same point
// on other warps.
template <typename T>
__device__ bool gj_right_solve_g(const Grp &g, T *A, int n, T *Y, int ny, T *prow, T *pinv, int *sh) {
    const int lane = g.tid & 31, wid = g.tid >> 5;
    // The search of step k + 1 runs beside each step's updates, on its critical path, so in
    // the double-float form it is one redux.sync; the FP64 form keeps the shuffle search.
    constexpr bool kDF = std::is_same<T, zd>::value;
    auto search = [&](int k) {  // pivot column of row k
        if constexpr (kDF) {
            unsigned key = 0u;
            for (int j = k + lane; j < n; j += 32) {
                const unsigned kk = pack_key(sabs1(A[k * n + j]), j - k);
                key = key > kk ? key : kk;
            }
            const unsigned m = __reduce_max_sync(0xffffffffu, key);
            if (lane == 0) {
                const int idx = k + 63 - (int)(m & 63u);
                const bool z = (m >> 6) == 0u;
                sh[0] = idx;
                sh[1] = z ? 1 : 0;
                pinv[0] = z ? szero<T>() : srecip(A[k * n + idx]);
            }
        } else {
            using Mag = decltype(sabs1(A[0]));
            Mag v = -1;
            int idx = 0x7fffffff;
            for (int j = k + lane; j < n; j += 32) {
                const Mag a = sabs1(A[k * n + j]);
                if (a > v) {
                    v = a;
                    idx = j;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const Mag ov = __shfl_down_sync(0xffffffffu, v, o);
                const int oi = __shfl_down_sync(0xffffffffu, idx, o);
                if (ov > v || (ov == v && oi < idx)) {
                    v = ov;
                    idx = oi;
                }
            }
            if (lane == 0) {
                const bool none = (idx == 0x7fffffff);
                const bool z = none || v == Mag(0);
                sh[0] = none ? k : idx;
                sh[1] = z ? 1 : 0;
                pinv[0] = z ? szero<T>() : srecip(A[k * n + (none ? k : idx)]);
            }
        }
    };
    bool sing = false;
    // phase-2 layout of the other warps: rpi rows at a time, one column per thread
    const int rpi = (g.nthr - 32) / n, jc = (g.tid - 32) % n, r0 = (g.tid - 32) / n;
    if (wid == 0) search(0);
    gsync(g);
    for (int k = 0; k < n; ++k) {
        const int c = sh[0];
        if (sh[1]) sing = true;
        // phase 1: m_r = M[r][c] / A[k][c] into column k, old column k into column c, the
        // exchanged pivot row into prow
        const int nrT = n - k - 1, nrows = nrT + ny;
        for (int t = g.tid; t < nrows + n; t += g.nthr) {
            if (t < nrows) {
                T *row = t < nrT ? A + (k + 1 + t) * n : Y + (t - nrT) * n;
                const T a = row[c], bb = row[k];
                row[k] = smul(a, pinv[0]);
                if (c != k) row[c] = bb;
            } else {
                const int j = t - nrows;
                prow[j] = (j == c) ? A[k * n + k] : A[k * n + j];
            }
        }
        gsync(g);
        // phase 2: M[r][j] -= m_r prow[j] for j != k; warp 0 takes row k + 1 of A, then its pivot
        if (wid == 0) {
            if (k + 1 < n) {
                T *row = A + (k + 1) * n;
                const T m = row[k];
                for (int j = lane; j < n; j += 32)
                    if (j != k) row[j] = sfms(m, prow[j], row[j]);
                __syncwarp();
                search(k + 1);
            }
        } else if (r0 < rpi && jc != k) {
            const int nrA = n - k - 2 > 0 ? n - k - 2 : 0;
            const T pj = prow[jc];
            for (int R = r0; R < nrA + ny; R += rpi) {
                T *row = R < nrA ? A + (k + 2 + R) * n : Y + (R - nrA) * n;
                row[jc] = sfms(row[k], pj, row[jc]);
            }
        }
        gsync(g);
    }
    return sing;
}

// Y <- Y A^-1 for nr rows of Y (leading dimension ldy), A = P^T L U from lu_factor.
template <typename T>
__device__ void row_solve(T *Y, int nr, int ldy, const T *A, int n, int lda, const int *perm,
                          const T *invd) {
    for (int j = 0; j < n; ++j) {  // Z U = B, column by column
        const T inv = invd[j];
        for (int r = threadIdx.x; r < nr; r += blockDim.x) Y[r * ldy + j] = smul(Y[r * ldy + j], inv);
        __syncthreads();
        const int m = n - j - 1;
        if (m > 0) {
            const int dq = blockDim.x / m, dr = blockDim.x % m;
            int r = threadIdx.x / m, c = j + 1 + threadIdx.x % m;
            for (int t = threadIdx.x; t < nr * m; t += blockDim.x) {
                Y[r * ldy + c] = sfms(Y[r * ldy + j], A[j * lda + c], Y[r * ldy + c]);
                r += dq;
                c += dr;
                if (c >= n) {
                    c -= m;
                    ++r;
                }
            }
            __syncthreads();
        }
    }
    for (int j = n - 1; j > 0; --j) {  // Y2 L = Z, last column first
        const int dq = blockDim.x / j, dr = blockDim.x % j;
        int r = threadIdx.x / j, c = threadIdx.x % j;
        for (int t = threadIdx.x; t < nr * j; t += blockDim.x) {
            Y[r * ldy + c] = sfms(Y[r * ldy + j], A[j * lda + c], Y[r * ldy + c]);
            r += dq;
            c += dr;
            if (c >= j) {
                c -= j;
                ++r;
            }
        }
        __syncthreads();
    }
    for (int r = threadIdx.x; r < nr; r += blockDim.x)  // Y = Y2 P: column swaps in reverse
        for (int k = n - 1; k >= 0; --k) {
            const int p = perm[k];
            if (p != k) {
                const T t = Y[r * ldy + k];
                Y[r * ldy + k] = Y[r * ldy + p];
                Y[r * ldy + p] = t;
            }
        }
    __syncthreads();
}

// ------------------------------------------------------------------ Pfaffian
// Exchange of indices p < q of a skew matrix held in its upper triangle, rows
// >= r only (ZExch, PNAMP_Proj.f90:356-392). Every thread touches distinct entries.
template <class Z>
__device__ __forceinline__ void exch_upper(Z *S, int N, int r, int p, int q) {
    for (int i = r + threadIdx.x; i < N; i += blockDim.x) {
        if (i < p) {
            const Z t = S[i * N + p];
            S[i * N + p] = S[i * N + q];
            S[i * N + q] = t;
        } else if (i > q) {
            const Z t = S[p * N + i];
            S[p * N + i] = S[q * N + i];
            S[q * N + i] = t;
        } else if (i > p && i < q) {
            const Z t = S[p * N + i];
            S[p * N + i] = -S[i * N + q];
            S[i * N + q] = -t;
        } else if (i == p) {
            S[p * N + q] = -S[p * N + q];
        }
    }
    __syncthreads();
}

// Running product of the Pfaffian's pivots. FP64 form: a complex double. Double-float
// form: a double-float mantissa renormalised to [1/2, 1) in its largest part after every
// factor, with the power of two kept as an integer, so that a product of many small or
// large pivots neither leaves the float range nor needs the (narrow) FP64 pipe; one
// conversion at the end.
template <class Z> struct PfProd;
template <> struct PfProd<zc> {
    zc v = {1.0, 0.0};
    __device__ __forceinline__ void mul(zc f, bool neg) { v = (neg ? -1.0 : 1.0) * (v * f); }
    // times the product of the lane o away
    __device__ __forceinline__ void join(int o) {
        v = v * mk(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
    }
    __device__ __forceinline__ zc get() const { return v; }
};
template <> struct PfProd<zd> {
    zd m = {f2_make(1.0f, 0.0f), f2_make(0.0f, 0.0f)};
    int e = 0;
    __device__ __forceinline__ void join(int o) {
        zd f;
        f.hi.u = __shfl_xor_sync(0xffffffffu, m.hi.u, o);
        f.lo.u = __shfl_xor_sync(0xffffffffu, m.lo.u, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
        mul(f, false);
    }
    __device__ __forceinline__ void mul(zd f, bool neg) {
        m = m * f;
        if (neg) m = -m;
        const float a = fmaxf(fabsf(f2_a(m.hi)), fabsf(f2_b(m.hi)));
        if (a > 0.0f && a <= 3.0e38f) {
            int ex;
            frexpf(a, &ex);
            m.hi = f2_make(ldexpf(f2_a(m.hi), -ex), ldexpf(f2_b(m.hi), -ex));
            m.lo = f2_make(ldexpf(f2_a(m.lo), -ex), ldexpf(f2_b(m.lo), -ex));
            e += ex;
        }
    }
    __device__ __forceinline__ zc get() const {
        const zc z = zd_to(m);
        return mk(ldexp(z.x, e), ldexp(z.y, e));
    }
};
// Pivot test of the Pfaffians: 0 fine, 1 |pivot| <= 1e-13 (the reference's exit), 2 not finite.
__device__ __forceinline__ int pivot_flag(zc ss) { return !zfinite(ss) ? 2 : (!(abs2(ss) > 1.0e-26) ? 1 : 0); }
__device__ __forceinline__ int pivot_flag(zd ss) {
    if (!zfinite(ss)) return 2;
    const float a = fabsf(f2_a(ss.hi)), b = fabsf(f2_b(ss.hi));
    // |ss|^2 > 1e-26 in float (the sum of squares underflows only far below the threshold)
    return (a > 1.0e-13f || b > 1.0e-13f || a * a + b * b > 1.0e-26f) ? 0 : 1;
}

// Pfaffian of the N x N skew matrix in the upper triangle of S (row-major), the
// 2x2-block elimination of ZPfaffianF (PNAMP_Proj.f90:218-350) with partial instead of
// global pivoting: at each step the largest entry of row r right of the diagonal (first
// maximum; magnitude max(|re|,|im|)) is moved to (r, r+1), the sign flips once per
// exchange, Pf = 0 when |pivot| <= 1e-13, and the Schur complement is updated in place.
// The running product is a PfProd. `vec` holds N scratch values; `flag` 2 ints.
template <class Z>
__device__ zc pfaffian_upper(Z *S, int N, Z *vec, double *red, int *flag, int &underflow) {
    // Parlett-Reid elimination with partial pivoting: step k takes the largest entry of
    // row r = 2k right of the diagonal as the 2x2 pivot (swapping its column with c = r + 1),
    // a one-warp search. (The reference's ZPfaffianF searches the whole remaining upper
    // triangle, PNAMP_Proj.f90:258-268; both are stable, results agree to rounding.)
    using A = Ar<Z>;
    PfProd<Z> pf;  // running product, meaningful in thread 0
    underflow = 0;
    const int NB = N / 2;
    for (int k = 0; k < NB - 1; ++k) {
        const int r = 2 * k, c = r + 1;
        if (std::is_same<Z, zd>::value && threadIdx.x < 32) {
            // one redux.sync over keys with 7 offset bits (N = 2n <= 128 candidates; the
            // high bits of the 31-bit magnitude key first, ties to the first column)
            unsigned key = 0u;
            for (int j = c + (int)threadIdx.x; j < N; j += 32) {
                const unsigned kk = ((unsigned)A::key(S[r * N + j]) & ~127u) | (unsigned)(127 - (j - c));
                key = key > kk ? key : kk;
            }
            const unsigned m = __reduce_max_sync(0xffffffffu, key);
            if (threadIdx.x == 0) flag[1] = c + 127 - (int)(m & 127u);
        } else if (threadIdx.x < 32) {
            unsigned long long best = 0ull;
            int bidx = 0x7fffffff;
            for (int j = c + (int)threadIdx.x; j < N; j += 32) {
                const unsigned long long key = A::key(S[r * N + j]);
                if (key > best || bidx == 0x7fffffff) {
                    best = key;
                    bidx = j;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ob = __shfl_down_sync(0xffffffffu, best, o);
                const int oi = __shfl_down_sync(0xffffffffu, bidx, o);
                if (oi != 0x7fffffff && (bidx == 0x7fffffff || ob > best || (ob == best && oi < bidx))) {
                    best = ob;
                    bidx = oi;
                }
            }
            if (threadIdx.x == 0) flag[1] = bidx;
        }
        __syncthreads();
        const int i2 = flag[1];
        if (i2 == 0x7fffffff) {  // no candidate: cannot happen for N - c >= 1
            underflow = 2;
            return mk(0.0, 0.0);
        }
        // the global-pivot sign rule with i1 = r (PNAMP_Proj.f90:273-275): -1, +1 without exchange
        const bool neg = (i2 != c);
        if (i2 != c) exch_upper(S, N, r, c, i2);
        if (threadIdx.x == 0) {  // pivot test, reciprocal and running product by one thread
            const Z ssz = S[r * N + c];
            const int f = pivot_flag(ssz);
            flag[0] = f;
            if (f == 0) {
                vec[c] = zrecip(ssz);
                pf.mul(ssz, neg);
            }
        }
        __syncthreads();
        if (flag[0]) {
            underflow = flag[0];
            __syncthreads();
            return mk(0.0, 0.0);
        }
    const Z inv = vec[c];
        for (int i = c + 1 + threadIdx.x; i < N; i += blockDim.x) vec[i] = S[c * N + i] * inv;
        __syncthreads();
        const int mm = N - c - 1, TT = mm * (mm - 1) / 2;
        for (int t = threadIdx.x; t < TT; t += blockDim.x) {
            int i, j;
            tri_index(t, mm, i, j);
            i += c + 1;
            j += c + 1;
            Z s = S[i * N + j];
            s = zfma(vec[i], S[r * N + j], s);
            s = zfms(S[r * N + i], vec[j], s);
            S[i * N + j] = s;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) pf.mul(S[(N - 2) * N + N - 1], false);
    __syncthreads();
    return threadIdx.x == 0 ? pf.get() : mk(0.0, 0.0);
}

// Pfaffian of the skew n x n matrix in the upper triangle of S (row-major) by the thread group
// g, row pivoting as in pfaffian_upper. Two group barriers per step: (a) the exchange of
// column c with the pivot column and the scaled pivot row v = S[c][.] / S[r][c] in one pass,
// (b) the rank-2 update, in which the first warp updates the next pivot row and searches it
// (pivot index, value and reciprocal for the next step), then joins the rest. A small pivot
// (|S[r][c]|^2 <= 1e-26, PNAMP_Proj.f90:290,333) or a non-finite one is recorded and the
// elimination runs on (its values are discarded): the result is 0 with `underflow` set.
// Returns the Pfaffian and `underflow` in the group's thread 0. `vec` holds n scratch values,
// `pv` 2 (pivot and reciprocal), `flag` 2 ints.
template <class Z>
__device__ zc pfaffian_upper_g(const Grp &g, Z *S, int n, Z *vec, Z *pv, int *flag, int &underflow) {
    using A = Ar<Z>;
    const int lane = g.tid & 31, wid = g.tid >> 5;
    const int nstep = n / 2 - 1;
    PfProd<Z> pf;
    int uf = 0;
    auto search = [&](int r) {   // pivot of row r -> flag[0] index, flag[1] its test, pv
        int q;
        bool none = false;
        if constexpr (std::is_same<Z, zd>::value) {   // one redux.sync; candidates r + 1 .. n - 1 exist
            unsigned key = 0u;
            for (int j = r + 1 + lane; j < n; j += 32) {
                const unsigned kk = ((unsigned)A::key(S[r * n + j]) & ~63u) | (unsigned)(63 - (j - r - 1));
                key = key > kk ? key : kk;
            }
            q = r + 1 + 63 - (int)(__reduce_max_sync(0xffffffffu, key) & 63u);
        } else {
            unsigned long long best = 0ull;
            int bidx = 0x7fffffff;
            for (int j = r + 1 + lane; j < n; j += 32) {
                const unsigned long long key = A::key(S[r * n + j]);
                if (key > best || bidx == 0x7fffffff) {
                    best = key;
                    bidx = j;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ob = __shfl_down_sync(0xffffffffu, best, o);
                const int oi = __shfl_down_sync(0xffffffffu, bidx, o);
                if (oi != 0x7fffffff && (bidx == 0x7fffffff || ob > best || (ob == best && oi < bidx))) {
                    best = ob;
                    bidx = oi;
                }
            }
            none = bidx == 0x7fffffff;
            q = none ? r + 1 : bidx;
        }
        if (lane == 0) {
            const Z ssz = S[r * n + q];
            const int f = none ? 2 : pivot_flag(ssz);
            flag[0] = q;
            flag[1] = f;
            pv[0] = ssz;
            pv[1] = f ? ssz : zrecip(ssz);
        }
    };
    if (wid == 0 && nstep > 0) search(0);
    gsync(g);
    for (int k = 0; k < nstep; ++k) {
        const int r = 2 * k, c = r + 1;
        const int q = flag[0];
        if (g.tid == 0) {
            if (uf == 0) uf = flag[1];  // the first failing step decides, as an early return would
            pf.mul(pv[0], q != c);
        }
        // (a) exchange c <-> q (exch_upper) and v_i = S'[c][i] / S'[r][c], i > c
        for (int i = r + g.tid; i < n; i += g.nthr) {
            const Z inv = pv[1];
            if (q == c) {
                if (i > c) vec[i] = S[c * n + i] * inv;
                continue;
            }
            if (i < c) {  // i == r: the pivot moves to column c
                const Z x = S[i * n + c];
                S[i * n + c] = S[i * n + q];
                S[i * n + q] = x;
            } else if (i > q) {
                const Z x = S[c * n + i];
                const Z y = S[q * n + i];
                S[c * n + i] = y;
                S[q * n + i] = x;
                vec[i] = y * inv;
            } else if (i > c && i < q) {
                const Z x = S[c * n + i];
                const Z y = -S[i * n + q];
                S[c * n + i] = y;
                S[i * n + q] = -x;
                vec[i] = y * inv;
            } else if (i == c) {  // S'[c][q] = -S[c][q]; its thread also sets v_q
                const Z y = -S[c * n + q];
                S[c * n + q] = y;
                vec[q] = y * inv;
            }
        }
        gsync(g);
        // (b) S_ij += v_i S_rj - S_ri v_j for c < i < j; row c + 1 (the next pivot row) first
        if (wid == 0) {
            const int i = c + 1;
            const Z vi = vec[i], sri = S[r * n + i];
            for (int j = i + 1 + lane; j < n; j += 32) {
                Z sv = S[i * n + j];
                sv = zfma(vi, S[r * n + j], sv);
                sv = zfms(sri, vec[j], sv);
                S[i * n + j] = sv;
            }
            __syncwarp();
            if (k + 1 < nstep) search(c + 1);
        }
        const int mm = n - c - 2, TT = mm * (mm - 1) / 2;
        for (int t = g.tid; t < TT; t += g.nthr) {
            int i, j;
            tri_index(t, mm, i, j);
            i += c + 2;
            j += c + 2;
            Z sv = S[i * n + j];
            sv = zfma(vec[i], S[r * n + j], sv);
            sv = zfms(S[r * n + i], vec[j], sv);
            S[i * n + j] = sv;
        }
        gsync(g);
    }
    zc out = mk(0.0, 0.0);
    if (g.tid == 0) {
        pf.mul(S[(n - 2) * n + n - 1], false);
        if (!uf) out = pf.get();
    }
    underflow = uf;
    return out;
}

// ------------------------------------------------------------------ points
static_assert(sizeof(dd) == sizeof(double), "per-warp double-float partials share the double slots of red");
constexpr int kNSlot = 36;  // observable sums: slots 0..37 final values, then per-warp partials
constexpr int kR1BSlot = 128;  // one-body density block sums: red[kR1BSlot + 2b], re and im
constexpr int kPfScratch = 608;  // point-arithmetic values: the grouped Pfaffian's pivot and reciprocal
constexpr int kR2Norm = 260;   // the gauge point's norm, re and im, for the two-body density pass
static_assert(kThreads >= 32 * (kNTrace + 1), "one warp per Q trace plus warp 0");

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace pnamp
#include "point_reduced.cuh"
namespace pnamp {

// One Euler point of a pair that no other body takes: the Pfaffian of the n x n Schur complement (V0
// well conditioned) or of the 2n x 2n matrix or, for NFOM = 1, the Onishi norm, and an n x n
// solve, by the whole CTA.
// `reload` is set when the previous item of this CTA belonged to another pair (or context):
// V0^T, U0^T and the phase tables are then (re)loaded.
template <class Z>
__device__ __noinline__ void full_item(const Params &p, const double *__restrict__ pairbuf, zc *slot,
                                           int pair, int ie, bool reload, double *__restrict__ zres,
                                           int *__restrict__ status, double *__restrict__ gout = nullptr,
                                           double *__restrict__ r1out = nullptr,
                                           double *__restrict__ r2out = nullptr, long long pt0 = 0) {
    using A = Ar<Z>;
    using R = typename A::R;
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = p.n, h = p.h, N = p.N2;
    const int nn = n * n;
    const int ld = n + 1;  // density row stride: transposed reads stay bank-conflict free
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const Placement &pl = p.place;
    Z *X = reinterpret_cast<Z *>(slot + pl.g_x);    // R W R^T
    Z *B = reinterpret_cast<Z *>(slot + pl.g_b);    // rows 0..n-1: R V1, rows n..2n-1: conj(R) U1
    zc *Bz = slot + pl.g_b;                         // the same storage while it holds FP64 values
    Z *P = reinterpret_cast<Z *>(slot + pl.g_p);    // T22 partials: V0p, V0n, U0p, U0n
    zc *RW = slot + pl.g_rw;                        // R W
    // -Cscale Z0 (or -Cscale Z0^-1): the constant block of the Pfaffian matrix, converted once
    // per pair so that building S takes no FP64 work per gauge point
    Z *CZ = reinterpret_cast<Z *>(slot + pl.g_zr);
    Z *S = reinterpret_cast<Z *>(pl.s_smem ? (void *)(smem + pl.off_s) : (void *)(slot + pl.g_s));
    Z *T = reinterpret_cast<Z *>(pl.t_smem ? (void *)(smem + pl.off_t) : (void *)(slot + pl.g_t));
    Z *Y = reinterpret_cast<Z *>(pl.y_smem ? (void *)(smem + pl.off_y) : (void *)(slot + pl.g_y));
    // V0^T and U0^T: V0t[k n + j] = V0(j, k)
    R *V0t = reinterpret_cast<R *>(pl.uv_smem ? (void *)(smem + pl.off_uv) : (void *)(slot + pl.g_uv));
    R *U0t = V0t + nn;
    int *perm = reinterpret_cast<int *>(smem + pl.off_piv);
    int *sh = perm + n;
    Z *invd = reinterpret_cast<Z *>(smem + pl.off_inv);
    double *red = reinterpret_cast<double *>(smem + pl.off_red);
    zc *rot = reinterpret_cast<zc *>(smem + pl.off_rot);
    Z *vec = reinterpret_cast<Z *>(smem + pl.off_vec);
    zc *acc = reinterpret_cast<zc *>(vec + N);      // kNobs accumulators (thread 0)
    zc *eph = acc + kNobs;                          // e^{i phi_l}, l < NFOM
    Z *ephz = reinterpret_cast<Z *>(eph + p.nfom);  // the same in the point arithmetic
    zc *acc_r1b = reinterpret_cast<zc *>(ephz + p.nfom);  // one-body density blocks (thread 0)
    Z *rho = S, *k10 = S + n * ld, *k01 = S + 2 * n * ld;
    Z *Kc = S + 3 * n * ld;  // antisymmetrised pairing tensors

    const double twopi = 6.283185307179586476925287;
    {
        const double *pr = pairbuf + (long long)pair * p.pl.stride;
        const double *gU1 = pr + p.pl.u1, *gV1 = pr + p.pl.v1, *gU0 = pr + p.pl.u0, *gV0 = pr + p.pl.v0;
        const double *gW = pr + p.pl.w;
        const double det0 = pr[p.pl.dets], det1 = pr[p.pl.dets + 1];
        // V0 well conditioned: the n x n Schur complement c (D X D - Z0^-1), times Pf(-c Z0), instead
        // of the 2n x 2n matrix
        const bool schur = pr[p.pl.dets + 3] != 0.0;
        const double *gZc = pr + (schur ? p.pl.zi : p.pl.z0);
        const zc pfz = mk(pr[p.pl.pfz], pr[p.pl.pfz + 1]);
        const int NP = N;  // order of the skew matrix the whole CTA eliminates
        double *zout = zres + 2LL * (long long)pair * kNobs * p.n_euler;
        if (reload) {
            __syncthreads();
            for (int t = threadIdx.x; t < nn; t += blockDim.x) {
                const int k = t / n, j = t % n;
                V0t[t] = A::real(gV0[j * n + k]);
                U0t[t] = A::real(gU0[j * n + k]);
                CZ[t] = A::from(mk(-p.cscale * gZc[t], 0.0));
            }
            for (int l = threadIdx.x; l < p.nfom; l += blockDim.x) {
                const zc e = expi(p.nfom == 1 ? 0.0 : twopi * l / p.nfom);
                eph[l] = e;
                ephz[l] = A::from(e);
            }
        }
        rotation_blocks(p, ie, threadIdx.x, blockDim.x, rot);
        if (threadIdx.x == 0) {
            for (int io = 0; io < kNobs; ++io) acc[io] = mk(0.0, 0.0);
            for (int b = 0; b < (r1out ? p.obs.n_r1b : 0); ++b) acc_r1b[b] = mk(0.0, 0.0);
        }
        // two-body density sums of this Euler point: thread t owns quadruples t, t + blockDim, ...
        // (zeroed, accumulated and flushed by the same thread, so no barrier between the steps)
        double *r2acc = r2out ? p.r2acc + p.r2_stride * blockIdx.x : nullptr;
        for (int q = threadIdx.x; q < (r2out ? p.n_r2q : 0); q += blockDim.x) {
            r2acc[2 * q] = 0.0;
            r2acc[2 * q + 1] = 0.0;
        }
        __syncthreads();
        // ---- R W (or, for the Onishi norm, R U1 and conj(R) V1), R V1, conj(R) U1 (FP64)
        const bool onishi = (p.nfom == 1);
        zc *Xz = reinterpret_cast<zc *>(X);
        for (int t = threadIdx.x; t < nn; t += blockDim.x) {
            const int a = t / n, j = t % n;
            const int b = p.row_blk[a], s0 = p.blk_start[b], d = p.blk_size[b];
            const zc *Rr = rot + p.blk_roff[b] + (a - s0) * d;
            zc rw = mk(0, 0), b1 = mk(0, 0), b2 = mk(0, 0), cv = mk(0, 0);
            for (int k = 0; k < d; ++k) {
                const zc r = Rr[k];
                rw = rfma(onishi ? gU1[(s0 + k) * n + j] : gW[(s0 + k) * n + j], r, rw);
                b1 = rfma(gV1[(s0 + k) * n + j], r, b1);
                b2 = rfma(gU1[(s0 + k) * n + j], zconj(r), b2);
                cv = rfma(gV1[(s0 + k) * n + j], zconj(r), cv);
            }
            RW[t] = rw;
            Bz[t] = b1;
            Bz[nn + t] = b2;
            if (onishi) Xz[t] = cv;
        }
        __syncthreads();
        // ---- X = (R W) R^T and the T22 partials (FP64), stored in the point arithmetic
        for (int t = threadIdx.x; t < (onishi ? 0 : nn); t += blockDim.x) {
            const int a = t / n, c = t % n;
            const int b = p.row_blk[c], s0 = p.blk_start[b], d = p.blk_size[b];
            const zc *Rr = rot + p.blk_roff[b] + (c - s0) * d;
            zc x = mk(0, 0);
            for (int k = 0; k < d; ++k) x = zfma(RW[a * n + s0 + k], Rr[k], x);
            X[t] = A::from(x);
        }
        for (int t = threadIdx.x; t < (p.norm_only ? 0 : 4 * nn); t += blockDim.x) {
            const int q = t / nn, e = t % nn, i = e / n, j = e % n;
            const double *M = (q < 2) ? gV0 : gU0;
            const zc *Bq = (q < 2) ? Bz : Bz + nn;
            const int k0 = (q & 1) ? h : 0;
            zc s = mk(0, 0);
            for (int k = k0; k < k0 + h; ++k) s = rfma(M[k * n + i], Bq[k * n + j], s);
            P[t] = A::from(s);
        }
        __syncthreads();
        for (int t = threadIdx.x; t < (p.norm_only ? 0 : 2 * nn); t += blockDim.x) {  // in place
            const zc v = Bz[t];
            B[t] = A::from(v);
        }
        __syncthreads();

        int flags = 0;
        const Z zero = A::from(mk(0.0, 0.0));
        const Z csz = A::from(mk(p.cscale, 0.0)), mcs = A::from(mk(-p.cscale, 0.0));
        for (int lp = 0; lp < p.nfom; ++lp) {
            const Z zep = ephz[lp], zepc = zconj(zep);
            for (int ln = 0; ln < p.nfom; ++ln) {
                const Z zen = ephz[ln], zenc = zconj(zen);
                // ---- S = Cscale [[D X D, -I], [I, -Z0]] (upper triangle)
                const Z dpp = csz * (zep * zep), dpn = csz * (zep * zen), dnn = csz * (zen * zen);
                int under = 0;
                zc pf = mk(0.0, 0.0);
                bool sing = false;
                // the Schur complement's elimination (warps 0 .. kPfWarpsG-1, named barrier 1) beside
                // the Gauss-Jordan solve on the other warps (named barrier 2)
                const bool concg = schur && !onishi;
                if (concg) {
                    constexpr int kPfWarpsG = 3;
                    if (wid < kPfWarpsG) {
                        const Grp g{(int)threadIdx.x, kPfWarpsG * 32, 1};
                        for (int t = g.tid; t < n * (n - 1) / 2; t += g.nthr) {
                            int i, j;
                            tri_index(t, n, i, j);
                            const Z dd_ = (j < h) ? dpp : ((i < h) ? dpn : dnn);
                            S[i * n + j] = X[i * n + j] * dd_ + CZ[i * n + j];
                        }
                        gsync(g);
                        pf = pfaffian_upper_g<Z>(g, S, n, vec, reinterpret_cast<Z *>(red + kPfScratch), sh, under);
                        pf = pf * pfz;  // meaningful in thread 0
                    } else if (!p.norm_only) {
                        const Grp g{(int)threadIdx.x - kPfWarpsG * 32, (int)blockDim.x - kPfWarpsG * 32, 2};
                        for (int t = g.tid; t < nn; t += g.nthr) {
                            Z sv = zep * P[t];
                            sv = zfma(zen, P[nn + t], sv);
                            sv = zfma(zepc, P[2 * nn + t], sv);
                            sv = zfma(zenc, P[3 * nn + t], sv);
                            T[t] = sv;
                        }
                        for (int t = g.tid; t < 2 * nn; t += g.nthr) Y[t] = B[t];
                        gsync(g);
                        const bool sg = gj_right_solve_g<Z>(g, T, n, Y, 2 * n, invd, vec + n, sh + 4);
                        if (g.tid == 0) sh[4] = sg ? 1 : 0;
                    }
                    __syncthreads();
                    if (!p.norm_only) sing = sh[4] != 0;
                }
                for (int t = threadIdx.x; t < (onishi || concg ? 0 : NP * (NP - 1) / 2); t += blockDim.x) {
                    int i, j;
                    tri_index(t, NP, i, j);
                    Z v;
                    if (j < n) {
                        const Z dd_ = (j < h) ? dpp : ((i < h) ? dpn : dnn);
                        v = X[i * n + j] * dd_;
                    } else if (i < n) {
                        v = (j - n == i) ? mcs : zero;
                    } else {
                        v = CZ[(i - n) * n + (j - n)];
                    }
                    S[i * NP + j] = v;
                }
                if (!concg) __syncthreads();
                if (concg) {
                } else if (onishi) {
                    // Onishi (PNAMP_Onishi.f90:21-37): sqrt(det(Ubar^T U0 + Vbar^T V0)),
                    // Ubar = R U1, Vbar = conj(R) V1 at phi = 0; LU determinant, principal root
                    zc *Bm = reinterpret_cast<zc *>(S);
                    for (int t = threadIdx.x; t < nn; t += blockDim.x) {
                        const int i = t / n, j = t % n;
                        zc acc2 = mk(0, 0);
                        for (int k = 0; k < n; ++k) {
                            acc2 = rfma(gU0[k * n + j], RW[k * n + i], acc2);
                            acc2 = rfma(gV0[k * n + j], Xz[k * n + i], acc2);
                        }
                        Bm[t] = acc2;
                    }
                    __syncthreads();
                    zc *invz = reinterpret_cast<zc *>(invd);
                    const bool bsing = lu_factor<zc>(Bm, n, n, perm, invz, sh);
                    if (threadIdx.x == 0) {
                        zc det = mk(1.0, 0.0);
                        for (int k = 0; k < n; ++k) {
                            det = det * Bm[k * n + k];
                            if (perm[k] != k) det = -det;
                        }
                        if (bsing) det = mk(0.0, 0.0);
                        const double r = sqrt(det.x * det.x + det.y * det.y);
                        const double re = sqrt(0.5 * (r + det.x)), im = copysign(sqrt(0.5 * fmax(r - det.x, 0.0)), det.y);
                        acc[kNobs - 1] = mk(re, im);  // scratch slot: observable 19 is never set
                    }
                    __syncthreads();
                    pf = acc[kNobs - 1];
                    __syncthreads();
                } else {
                    pf = pfaffian_upper<Z>(S, NP, vec, red, sh + 2, under);
                }
                // fin: final sums (double); pwR: per-warp energy and <J^2> partials in R (8 bytes,
                // like a double, in both forms)
                double *fin = red;
                R *pwR = reinterpret_cast<R *>(red + kNSlot + 2);
                if (!p.norm_only) {  // uniform over the block: norm-only launches skip the densities
                // ---- T22(phi) and right-hand sides
                if (!concg) {  // (2n x 2n Pfaffian or Onishi norm) the whole CTA solves after the norm
                    for (int t = threadIdx.x; t < nn; t += blockDim.x) {
                        Z s = zep * P[t];
                        s = zfma(zen, P[nn + t], s);
                        s = zfma(zepc, P[2 * nn + t], s);
                        s = zfma(zenc, P[3 * nn + t], s);
                        T[t] = s;
                    }
                    for (int t = threadIdx.x; t < 2 * nn; t += blockDim.x) Y[t] = B[t];
                    __syncthreads();
                    sing = gj_right_solve<Z>(T, n, Y, 2 * n, invd, vec, sh);
                }
                // ---- densities into the Pfaffian's storage, row stride ld
                {
                    const int dq = blockDim.x / n, dr = blockDim.x % n;
                    for (int q = 0; q < 3; ++q) {
                        const R *Mq = (q == 1) ? U0t : V0t;
                        const Z *Yq = (q == 2) ? Y + nn : Y;
                        Z *Sq = S + q * n * ld;
                        int i = threadIdx.x / n, j = threadIdx.x % n;
                        for (int t = threadIdx.x; t < nn; t += blockDim.x) {
                            const Z *Yr = Yq + i * n;
                            const R *M = Mq + j;
                            Z s = zero;
                            for (int k = 0; k < n; ++k) s = rfma(M[k * n], Yr[k], s);
                            const Z di = (i < h) ? zep : zen;
                            Sq[i * ld + j] = (q == 2) ? -(zconj(di) * s) : di * s;
                            i += dq;
                            j += dr;
                            if (j >= n) {
                                j -= n;
                                ++i;
                            }
                        }
                    }
                }
                __syncthreads();
                // K01_ij (i < j) at Kc[i ld + j], K10_ij at Kc[j ld + i]
                for (int t = threadIdx.x; t < n * (n - 1) / 2; t += blockDim.x) {
                    int i, j;
                    tri_index(t, n, i, j);
                    Kc[i * ld + j] = k01[i * ld + j] - k01[j * ld + i];
                    Kc[j * ld + i] = k10[i * ld + j] - k10[j * ld + i];
                }
                __syncthreads();
                // ---- observables. Final sums land in red[0..kNSlot); the energy and <J^2>
                // sums, spread over all warps, leave per-warp partials in red[kNSlot + ..].
                // traces of rho, spread over warps 0 (species traces, sum j(j+1) rho_aa), 11 (J+, J-,
                // Jz) and 12 (one-body energy) so that no warp starts the energy loop much later
                // The sums run in the point arithmetic's real type R (double-float on the FP32
                // pipes in that form) and leave it once per warp, in lane 0.
                if (wid == 0 || wid == kNTrace + 1 || wid == kNTrace + 2) {
                    R v0 = A::rzero(), v1 = v0, v2 = v0, v3 = v0, v4 = v0, v5 = v0;
                    if (wid == 0) {
                        for (int a = lane; a < n; a += 32) {
                            const Z d = rho[a * ld + a];
                            if (a < h) { v0 = A::radd(v0, re(d)); v1 = A::radd(v1, im(d)); }
                            else { v2 = A::radd(v2, re(d)); v3 = A::radd(v3, im(d)); }
                            const R jj = A::pick(p.obs.jj1, p.obs.jj1_d, a);
                            v4 = A::rfma(jj, re(d), v4);
                            v5 = A::rfma(jj, im(d), v5);
                        }
                    } else if (wid == kNTrace + 1) {
                        for (int a = lane; a < n; a += 32) {
                            const R jpa = A::pick(p.obs.jp, p.obs.jp_d, a), jma = A::pick(p.obs.jm, p.obs.jm_d, a);
                            const R mza = A::pick(p.obs.mz, p.obs.mz_d, a);
                            if (A::nz(jpa)) {
                                const Z r = rho[(a + 1) * ld + a];
                                v0 = A::rfma(jpa, re(r), v0);
                                v1 = A::rfma(jpa, im(r), v1);
                            }
                            if (A::nz(jma)) {
                                const Z r = rho[(a - 1) * ld + a];
                                v2 = A::rfma(jma, re(r), v2);
                                v3 = A::rfma(jma, im(r), v3);
                            }
                            const Z d = rho[a * ld + a];
                            v4 = A::rfma(mza, re(d), v4);
                            v5 = A::rfma(mza, im(d), v5);
                        }
                    } else {
                        for (int e = lane; e < p.obs.n_t1b; e += 32) {
                            const int ix = p.obs.t1b_idx[e];
                            const Z r = rho[(ix >> 8) * ld + (ix & 255)];
                            const R tv = A::pick(p.obs.t1b_val, p.obs.t1b_val_d, e);
                            v0 = A::rfma(tv, re(r), v0);
                            v1 = A::rfma(tv, im(r), v1);
                        }
                    }
                    // result slots: z 0,1  n 2,3  t1b 4,5  J+ 10,11  J- 12,13  Jz 14,15  j(j+1) 16,17
                    const int s0 = wid == 0 ? 0 : (wid == kNTrace + 1 ? 10 : 4);
                    const int cnt = wid == kNTrace + 2 ? 2 : 6;
                    const R vals[6] = {v0, v1, v2, v3, v4, v5};
#pragma unroll
                    for (int q = 0; q < 6; ++q) {
                        if (q >= cnt) break;
                        const R v = A::wsum(vals[q]);
                        const int slot = (wid == 0 && q >= 4) ? 12 + q : s0 + q;
                        if (lane == 0) fin[slot] = A::dbl(v);
                    }
                } else if (p.iE2 && wid <= kNTrace) {  // Q_{2mu} traces: one warp per trace
                    const int q = wid - 1;
                    R sr = A::rzero(), si = A::rzero();
                    for (int e = p.obs.q_off[q] + lane; e < p.obs.q_off[q + 1]; e += 32) {
                        const int ix = p.obs.q_idx[e];
                        const Z r = rho[(ix >> 8) * ld + (ix & 255)];
                        const R qv = A::pick(p.obs.q_val, p.obs.q_val_d, e);
                        sr = A::rfma(qv, re(r), sr);
                        si = A::rfma(qv, im(r), si);
                    }
                    sr = A::wsum(sr);
                    si = A::wsum(si);
                    if (lane == 0) {
                        fin[18 + 2 * q] = A::dbl(sr);
                        fin[19 + 2 * q] = A::dbl(si);
                    }
                }
                if (r1out && wid > kNTrace) {  // one-body density blocks (ZRho1B_Angles): the idle warps
                    for (int b = wid - kNTrace - 1; b < p.obs.n_r1b; b += nw - kNTrace - 1) {
                        R sr = A::rzero(), si = A::rzero();
                        for (int e = p.obs.r1b_off[b] + lane; e < p.obs.r1b_off[b + 1]; e += 32) {
                            const int ix = p.obs.r1b_idx[e];
                            const Z r = rho[(ix >> 8) * ld + (ix & 255)];
                            const R bv = A::pick(p.obs.r1b_val, p.obs.r1b_val_d, e);
                            sr = A::rfma(bv, re(r), sr);
                            si = A::rfma(bv, im(r), si);
                        }
                        sr = A::wsum(sr);
                        si = A::wsum(si);
                        if (lane == 0) {
                            red[kR1BSlot + 2 * b] = A::dbl(sr);
                            red[kR1BSlot + 2 * b + 1] = A::dbl(si);
                        }
                    }
                }
                auto put = [&](int slot, R v) {  // slot 0..3: energy re/im, <J^2> re/im
                    v = A::wsum(v);
                    if (lane == 0) pwR[slot * nw + wid] = v;
                };
                if (p.tc_splits) {
                    // tensor-core contraction: this gauge point's operand rows X[2 pt + ri] (rho
                    // entries, then K10 pairs) and epilogue rows Y[2 pt + ri] (K01 pairs) as bf16
                    // terms; contract_tc.cu forms the two bilinear forms for the whole launch
                    const long long pt = pt0 + lp * p.nfom + ln;
                    const int S = p.tc_splits, nk = p.tc_nk, npp = p.tc_nk - p.tc_nph;
                    for (int e = threadIdx.x; e < nk; e += blockDim.x) {
                        const int src = p.tc_src[e];
                        Z v = zero, y = zero;
                        if (src >= 0) {
                            const int r = src >> 8, c = src & 255;
                            if (e < p.tc_nph) {
                                v = rho[r * ld + c];
                            } else {
                                v = Kc[c * ld + r];   // K10_rc, r < c
                                y = Kc[r * ld + c];   // K01_rc
                            }
                        }
                        unsigned short tr[3], ti[3];
                        bf16_terms(as_dd(re(v)), S, tr);
                        bf16_terms(as_dd(im(v)), S, ti);
                        for (int sp = 0; sp < S; ++sp) {
                            p.tc_x[sp][(2 * pt) * nk + e] = tr[sp];
                            p.tc_x[sp][(2 * pt + 1) * nk + e] = ti[sp];
                        }
                        if (e >= p.tc_nph) {
                            bf16_terms(as_dd(re(y)), S, tr);
                            bf16_terms(as_dd(im(y)), S, ti);
                            const int ey = e - p.tc_nph;
                            for (int sp = 0; sp < S; ++sp) {
                                p.tc_y[sp][(2 * pt) * npp + ey] = tr[sp];
                                p.tc_y[sp][(2 * pt + 1) * npp + ey] = ti[sp];
                            }
                        }
                    }
                    if (lane == 0) {   // no energy sum in this form
                        pwR[wid] = A::rzero();
                        pwR[nw + wid] = A::rzero();
                    }
                } else {   // two-body energy, exact regrouping of the 8-term sum of
                    // PNAMP_Energy_OpenMP.f90:40-78:
                    // V[rho_ki rho_lj - rho_li rho_kj + d(rho_ik rho_jl - rho_jk rho_il)]
                    // + V/4 [K01_ij K10_kl + d K01_kl K10_ij],  K_xy = kappa_xy - kappa_yx
                    const R quarter = A::rconst(0.25f);
                    Z e2 = zero;
                    auto rec = [&](uint32_t pk, R v) {
                        const int i = pk & 0xff, j = (pk >> 8) & 0xff, k = (pk >> 16) & 0xff, l = pk >> 24;
                        Z t = rho[k * ld + i] * rho[l * ld + j];
                        t = zfms(rho[l * ld + i], rho[k * ld + j], t);
                        Z u = Kc[i * ld + j] * Kc[l * ld + k];
                        if (i + j != k + l) {
                            t = zfma(rho[i * ld + k], rho[j * ld + l], t);
                            t = zfms(rho[j * ld + k], rho[i * ld + l], t);
                            u = zfma(Kc[k * ld + l], Kc[j * ld + i], u);
                        }
                        t = rfma(quarter, u, t);
                        e2 = rfma(v, t, e2);
                    };
                    const int stride = blockDim.x;
                    for (int e = threadIdx.x; e < p.nrec; e += 2 * stride) {
                        const int e1 = e + stride;
                        const uint32_t pk0 = p.rec_idx[e];
                        const R v0 = A::pick(p.rec_v, p.rec_vd, e);
                        const bool two = e1 < p.nrec;
                        const uint32_t pk1 = two ? p.rec_idx[e1] : 0u;
                        const R v1 = two ? A::pick(p.rec_v, p.rec_vd, e1) : A::rzero();
                        rec(pk0, v0);
                        if (two) rec(pk1, v1);
                    }
                    put(0, re(e2));
                    put(1, im(e2));
                }
                {   // <J^2> (ZJ2_0, PNAMP_ME2B.f90:45-147) summed over x, y, z with
                    // Jx, Jy = (J+ +- J-)/(2, 2i):  sum_a j(j+1) rho_aa [above]
                    // + Tr(J+ rho) Tr(J- rho) + Tr(Jz rho)^2 - Tr(J+ rho J- rho) - Tr(Jz rho Jz rho)
                    // + [Tr(J+ k10 J+ k01^T) + Tr(J- k10 J- k01^T)]/2 + Tr(Jz k10 Jz k01^T)
                    const R half = A::rconst(0.5f);
                    Z rest = zero;
                    for (int t = threadIdx.x; t < nn; t += blockDim.x) {
                        const int a = t / n, c = t % n;
                        const R jpa = A::pick(p.obs.jp, p.obs.jp_d, a), jma = A::pick(p.obs.jm, p.obs.jm_d, a);
                        const R jpc = A::pick(p.obs.jp, p.obs.jp_d, c), jmc = A::pick(p.obs.jm, p.obs.jm_d, c);
                        const R mzz = A::rmul(A::pick(p.obs.mz, p.obs.mz_d, a), A::pick(p.obs.mz, p.obs.mz_d, c));
                        const int ac = a * ld + c;
                        Z q = mzz * (k10[ac] * k01[ac]);
                        q = zfms(mzz * rho[ac], rho[c * ld + a], q);
                        if (A::nz(jpa) && A::nz(jmc))
                            q = zfms(A::rmul(jpa, jmc) * rho[ac + ld], rho[(c - 1) * ld + a], q);
                        if (A::nz(jpa) && A::nz(jpc))
                            q = zfma(A::rmul(half, A::rmul(jpa, jpc)) * k10[ac + ld], k01[ac + 1], q);
                        if (A::nz(jma) && A::nz(jmc))
                            q = zfma(A::rmul(half, A::rmul(jma, jmc)) * k10[ac - ld], k01[ac - 1], q);
                        rest = rest + q;
                    }
                    put(2, re(rest));
                    put(3, im(rest));
                }
                }  // !norm_only
                __syncthreads();
                if (wid == 0) {  // accumulation over the gauge points: warp 0, one observable per lane
                    // The FP64 pipe is narrow on this part and its cost grows with the active lanes,
                    // so each FP64 value is formed by the one lane that needs it: the norm by lane
                    // 0 (then broadcast), H/N by lane 6 (and 0 for the per-gauge output), <J^2> by
                    // lane 7; the per-warp energy and <J^2> partials are summed in the point
                    // arithmetic first.
                    const unsigned full = 0xffffffffu;
                    R ws[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) ws[q] = A::wsum(lane < nw ? pwR[q * nw + lane] : A::rzero());
                    const bool eval = !p.norm_only && !sing;
                    zc norm = mk(0.0, 0.0);
                    if (lane == 0) {
                        const zc zph = mk(p.gphase[2 * (lp * p.nfom + ln)], p.gphase[2 * (lp * p.nfom + ln) + 1]);
                        norm = onishi ? pf : (p.vacfac * det0 * det1) * (pf * zph);
                    }
                    norm.x = __shfl_sync(full, norm.x, 0);
                    norm.y = __shfl_sync(full, norm.y, 0);
                    zc o = mk(0.0, 0.0), hg = mk(0.0, 0.0);   // hg: H/N at this gauge point (0 if not computed)
                    bool use = eval;
                    if ((lane == 6 || (lane == 0 && gout)) && eval)
                        hg = mk(fin[4] + A::dbl(ws[0]) + p.e0, fin[5] + A::dbl(ws[1]));
                    if (lane == 1) o = mk(fin[0], fin[1]);
                    else if (lane == 2) o = mk(fin[2], fin[3]);
                    else if (lane == 3) o = mk(fin[4], fin[5]);      // one-body energy
                    else if (lane == 6) o = hg;
                    else if (lane == 7) {
                        const zc trp = mk(fin[10], fin[11]), trm = mk(fin[12], fin[13]), trz = mk(fin[14], fin[15]);
                        o = mk(fin[16] + A::dbl(ws[2]), fin[17] + A::dbl(ws[3])) + trp * trm + trz * trz;
                    } else if (lane >= 8 && lane < 18 && p.iE2) o = mk(fin[2 * lane + 2], fin[2 * lane + 3]);  // Q slots 18..37
                    else use = false;
                    if (p.tc_splits && lane == 0) {   // w = N / NFOM^2 of this gauge point, 0 if not evaluated
                        const long long pt = pt0 + lp * p.nfom + ln;
                        const double inv = 1.0 / ((double)p.nfom * p.nfom);
                        p.tc_w[2 * pt] = eval ? inv * norm.x : 0.0;
                        p.tc_w[2 * pt + 1] = eval ? inv * norm.y : 0.0;
                    }
                    if (lane == 0) {
                        acc[0] = acc[0] + norm;
                        if (r2out) {
                            red[kR2Norm] = norm.x;
                            red[kR2Norm + 1] = norm.y;
                        }
                        if (gout) {  // per gauge point: N (with the gauge phase) and H/N
                            double *g = gout + 4LL * (((long long)pair * p.n_euler + ie) * p.n_gauge + lp * p.nfom + ln);
                            g[0] = norm.x;
                            g[1] = norm.y;
                            g[2] = hg.x;
                            g[3] = hg.y;
                        }
                        int f = (under == 1) ? 1 : (under == 2 ? 4 : 0);
                        if (!p.norm_only && sing) f |= 2;
                        flags |= f;
                    }
                    if (use) acc[lane] = zfma(norm, o, acc[lane]);
                    if (eval)
                        for (int b = lane; b < (r1out ? p.obs.n_r1b : 0); b += 32)
                            acc_r1b[b] = zfma(norm, mk(red[kR1BSlot + 2 * b], red[kR1BSlot + 2 * b + 1]), acc_r1b[b]);
                    __syncwarp();   // thread 0 reads every lane's accumulator after the last gauge point
                }
                // No CTA barrier here: the other warps go on to the next gauge point while warp 0
                // accumulates this one. What warp 0 reads (the sums in red, pf, sing) is written
                // again only after the next point's first CTA-wide barrier, which waits for warp 0;
                // the two-body density pass reads the densities, so it keeps the barrier.
                if (r2out) __syncthreads();
                if (r2out && !p.norm_only && !sing) {
                    // ZRho2B_Angles (PNAMP_Rho2B.f90:105-112) before its Clebsch-Gordan sums:
                    // N [ZRO(k,i) ZRO(l,j) - ZRO(l,i) ZRO(k,j) + ZKAPA01(i,j) ZKAPA10(k,l)] per quadruple,
                    // summed over the gauge points in FP64; the densities are still in S here
                    const zc nrm = mk(red[kR2Norm], red[kR2Norm + 1]);
                    for (int q = threadIdx.x; q < p.n_r2q; q += blockDim.x) {
                        const uint32_t pk = p.r2q[q];
                        const int i = pk & 0xff, j = (pk >> 8) & 0xff, k = (pk >> 16) & 0xff, l = pk >> 24;
                        Z t = rho[k * ld + i] * rho[l * ld + j];
                        t = zfms(rho[l * ld + i], rho[k * ld + j], t);
                        t = zfma(k01[i * ld + j], k10[k * ld + l], t);
                        const zc a = zfma(nrm, A::to(t), mk(r2acc[2 * q], r2acc[2 * q + 1]));
                        r2acc[2 * q] = a.x;
                        r2acc[2 * q + 1] = a.y;
                    }
                    __syncthreads();  // the next gauge point overwrites the densities
                }
            }
        }
        if (threadIdx.x == 0) {
            const double inv = 1.0 / ((double)p.nfom * p.nfom);
            int f = flags;
            acc[kNobs - 1] = mk(0.0, 0.0);
            for (int io = 0; io < kNobs; ++io) {
                const zc v = inv * acc[io];
                if (!zfinite(v)) f |= 4;
                zout[2LL * (io * p.n_euler + ie)] = re(v);
                zout[2LL * (io * p.n_euler + ie) + 1] = im(v);
            }
            status[(long long)pair * p.n_euler + ie] = f;
            for (int b = 0; b < (r1out ? p.obs.n_r1b : 0); ++b) {
                const zc v = inv * acc_r1b[b];
                r1out[2LL * (((long long)pair * p.obs.n_r1b + b) * p.n_euler + ie)] = re(v);
                r1out[2LL * (((long long)pair * p.obs.n_r1b + b) * p.n_euler + ie) + 1] = im(v);
            }
        }
        if (r2out) {  // Euler weight x gauge mean, added into the pair's sums (ZRho2B_Integral at J = 0)
            const double wgt = p.euler[4 * ie + 3] / ((double)p.nfom * p.nfom);
            double *o = r2out + 2LL * p.n_r2q * pair;
            for (int q = threadIdx.x; q < p.n_r2q; q += blockDim.x) {
                atomicAdd(o + 2 * q, wgt * r2acc[2 * q]);
                atomicAdd(o + 2 * q + 1, wgt * r2acc[2 * q + 1]);
            }
        }
        __syncthreads();
    }
}

// What a pair's set-up record says about its points.
enum { kPairBad = 0, kPairFull = 1, kPairReduced = 2, kPairSplit = 3, kPairSplitSolve = 4 };
__device__ __forceinline__ int pair_kind(const Params &p, const double *pr) {
    if (pr[p.pl.dets + 2] != 0.0) return kPairBad;
    const bool conserving = pr[p.pl.dets + 6] != 0.0;
    if (pr[p.pl.dets + 7] == 0.0) return conserving && pr[p.pl.dets + 3] != 0.0 ? kPairSplitSolve : kPairFull;
    return conserving ? kPairSplit : kPairReduced;
}
// Charge-conserving pairs factorise by species (split_items); H/N of every gauge point needs room
// for the neutrons' part in the CTA's slot (NFOM up to 18, more at n = 64).
__device__ __forceinline__ bool split_path(const Params &p, bool gout, bool r2out) {
    return p.nfom > 1 && p.split_ok && (!p.tc_splits || p.tc_sp) && (!r2out || p.r2_ss >= 0) &&
           (!gout || p.norm_only || (gauge_chunks(p, false) > 0 && gauge_chunks(p, true) > 0));
}

// One Euler point of a pair that does not take split_items.
template <class Z>
__device__ __forceinline__ void point_item(const Params &p, const double *__restrict__ pairbuf, zc *slot, int pair,
                                           int ie, int kind, bool reload, double *__restrict__ zres,
                                           int *__restrict__ status, double *__restrict__ gout,
                                           double *__restrict__ r1out, double *__restrict__ r2out, long long pt0) {
    double *zout = zres + 2LL * (long long)pair * kNobs * p.n_euler;
    if (kind == kPairBad) {
        for (int io = threadIdx.x; io < kNobs; io += blockDim.x) {
            zout[2LL * (io * p.n_euler + ie)] = 0.0;
            zout[2LL * (io * p.n_euler + ie) + 1] = 0.0;
        }
        if (threadIdx.x == 0) status[(long long)pair * p.n_euler + ie] = 8;
        for (int g = threadIdx.x; g < (p.tc_splits ? p.n_gauge : 0); g += blockDim.x) {
            p.tc_w[2 * (pt0 + g)] = 0.0;
            p.tc_w[2 * (pt0 + g) + 1] = 0.0;
        }
    } else if (kind == kPairFull || kind == kPairSplitSolve) {
        full_item<Z>(p, pairbuf, slot, pair, ie, reload, zres, status, gout, r1out, r2out, pt0);
    } else {
        reduced_item<Z>(p, pairbuf + (long long)pair * p.pl.stride, slot, pair, ie, reload, zout, status, gout, r1out,
                        r2out, pt0);
    }
}

// Gauge: launches that want H/N of every gauge point, a kernel of their own because the other
// launches' code is 1 to 2 % slower beside that body (registers of the functions they share).
template <class Z, bool Gauge>
__global__ void __launch_bounds__(kThreads, 1)
point_kernel(const __grid_constant__ Params p, int npairs, const double *__restrict__ pairbuf, zc *scratch,
             double *__restrict__ zres, int *__restrict__ status, const int2 *__restrict__ items,
             long long nitems, double *__restrict__ gout, double *__restrict__ r1out,
             double *__restrict__ r2out, int batch) {
    // items == nullptr: every (pair, Euler point) of the batch; else the listed (pair, ie)
    zc *slot = scratch + (long long)blockIdx.x * p.place.slot_elems;
    int cur_pair = -1, cur_kind = -1;
    if (split_path(p, gout != nullptr, r2out != nullptr)) {
        // species-split pairs: `batch` Euler points at a time, runs of one pair
        const long long per = items ? nitems : p.n_euler, nb = (per + batch - 1) / batch;
        const long long total = items ? nb : nb * npairs;
        for (long long b = blockIdx.x; b < total; b += gridDim.x) {
            const int pair0 = items ? 0 : (int)(b / nb);
            const long long i0 = (b % nb) * batch;
            const int cnt = (int)min((long long)batch, per - i0);
            for (int k = 0; k < cnt;) {
                int pair = pair0, m = cnt - k;
                if (items) {
                    const int2 it = items[i0 + k];
                    pair = it.x;
                    if (pair < 0 || pair >= npairs || it.y < 0 || it.y >= p.n_euler) {   // out of range: skipped
                        ++k;
                        continue;
                    }
                    m = 1;
                    while (k + m < cnt && items[i0 + k + m].x == pair && items[i0 + k + m].y >= 0 &&
                           items[i0 + k + m].y < p.n_euler)
                        ++m;
                }
                const double *pr = pairbuf + (long long)pair * p.pl.stride;
                const int kind = pair_kind(p, pr);
                if (kind >= kPairSplit) {
                    const bool solve = kind == kPairSplitSolve;
                    if (Gauge) m = 1;
                    else if (solve) m = min(m, p.place.sol.items);
                    double *zout = zres + 2LL * (long long)pair * kNobs * p.n_euler;
                    const int2 *list = items ? items + i0 + k : nullptr;
                    const int ie0 = (int)(i0 + k);
                    const long long pt0 = ((long long)pair0 * p.n_euler + i0 + k) * p.n_gauge;
                    if (solve)
                        split_items<Z, true, Gauge>(p, pr, slot, pair, list, ie0, m, pair != cur_pair, zout, status, gout,
                                                    r1out, r2out, pt0);
                    else
                        split_items<Z, false, Gauge>(p, pr, slot, pair, list, ie0, m, pair != cur_pair, zout, status, gout,
                                                     r1out, r2out, pt0);
                    cur_pair = pair;
                }
                k += m;
            }
        }
        cur_pair = -1;
        cur_kind = kPairSplit;
    }
    const bool skip = cur_kind == kPairSplit;
    const long long total = items ? nitems : (long long)npairs * p.n_euler;
    for (long long item = blockIdx.x; item < total; item += gridDim.x) {
        int pair, ie;
        if (items) {
            const int2 it = items[item];
            pair = it.x;
            ie = it.y;
            if (pair < 0 || pair >= npairs || ie < 0 || ie >= p.n_euler) continue;  // out of range: skipped
        } else {
            pair = (int)(item / p.n_euler);
            ie = (int)(item % p.n_euler);
        }
        const int kind = pair_kind(p, pairbuf + (long long)pair * p.pl.stride);
        if (skip && kind >= kPairSplit) continue;
        point_item<Z>(p, pairbuf, slot, pair, ie, kind, pair != cur_pair, zres, status, gout, r1out, r2out,
                      item * p.n_gauge);
        cur_pair = pair;
    }
}

// Persistent kernel over an uneven batch: work items (context, pair, Euler point) of up to
// kMultiCtx contexts (model spaces, meshes, placements), taken `grab` at a time from a global
// counter in the order of `items` (set by the schedule). Every context's parameters travel by
// value in the launch's parameter space. Runs of Euler points of one species-split pair within
// a grab go through split_items together.
template <class Z>
__device__ __forceinline__ void multi_items(const MultiArgs &a, const int4 *items, int cnt, zc *slot, bool reload) {
    const int4 m = items[0];
    const Params &p = a.p[m.x];
    const double *pr = a.pairbuf[m.x] + (long long)m.y * p.pl.stride;
    const int kind = pair_kind(p, pr);
    if (kind >= kPairSplit && split_path(p, false, false)) {
        double *zout = a.zres[m.x] + 2LL * (long long)m.y * kNobs * p.n_euler;
        if (kind == kPairSplit)
            split_items<Z, false, false>(p, pr, slot, m.y, nullptr, m.z, cnt, reload, zout, a.status[m.x], nullptr, nullptr,
                                         nullptr, 0);
        else
            for (int k = 0; k < cnt; k += p.place.sol.items)
                split_items<Z, true, false>(p, pr, slot, m.y, nullptr, m.z + k, min(p.place.sol.items, cnt - k),
                                            reload && k == 0, zout, a.status[m.x], nullptr, nullptr, nullptr, 0);
    } else
        for (int k = 0; k < cnt; ++k)
            point_item<Z>(p, a.pairbuf[m.x], slot, m.y, m.z + k, kind, reload && k == 0, a.zres[m.x], a.status[m.x],
                          nullptr, nullptr, nullptr, 0);
}

template <class Z>
__global__ void __launch_bounds__(kThreads, 1)
multi_point_kernel(const __grid_constant__ MultiArgs a, const int4 *__restrict__ items, int nitems, int grab,
                   zc *scratch, int *counter, int smem_tail) {
    // the work counter's broadcast lives past every context's placement (no static
    // shared memory, so the dynamic limit can be the device maximum)
    extern __shared__ __align__(16) unsigned char smem_all[];
    int &s_next = *reinterpret_cast<int *>(smem_all + smem_tail);
    zc *slot = scratch + (long long)blockIdx.x * a.slot_stride;
    int cur_ctx = -1, cur_pair = -1;
    for (;;) {
        if (threadIdx.x == 0) s_next = atomicAdd(counter, grab);
        __syncthreads();
        const int base = s_next;
        __syncthreads();
        if (base >= nitems) break;
        const int end = min(base + grab, nitems);
        for (int it = base; it < end;) {
            const int4 m = items[it];  // (context, pair, first Euler point, unused)
            int cnt = 1;
            while (it + cnt < end && cnt < a.p[m.x].place.spl.items && items[it + cnt].x == m.x &&
                   items[it + cnt].y == m.y && items[it + cnt].z == m.z + cnt)
                ++cnt;
            multi_items<Z>(a, items + it, cnt, slot, m.x != cur_ctx || m.y != cur_pair);
            cur_ctx = m.x;
            cur_pair = m.y;
            it += cnt;
        }
    }
}

// Launches of one arithmetic form, instantiated in a translation unit of its own.
template <class Z, bool Gauge>
cudaError_t launch_points_z(const Params &p, int npairs, const double *pairbuf, zc *scratch, int grid, double *zres,
                            int *status, cudaStream_t st, const int2 *items, long long nitems, double *gout,
                            double *r1out, double *r2out, int batch) {
    point_kernel<Z, Gauge><<<grid, kThreads, p.place.smem_bytes, st>>>(p, npairs, pairbuf, scratch, zres, status, items,
                                                                      nitems, gout, r1out, r2out, batch);
    return cudaGetLastError();
}
template <class Z>
cudaError_t launch_multi_z(const MultiArgs &a, const int4 *items, int nitems, int grab, int *counter, zc *scratch,
                           int grid, int smem, cudaStream_t st) {
    multi_point_kernel<Z><<<grid, kThreads, smem, st>>>(a, items, nitems, grab, scratch, counter, smem - kMultiSmemTail);
    return cudaGetLastError();
}
template <class Z, bool Gauge> const void *point_fn() { return reinterpret_cast<const void *>(point_kernel<Z, Gauge>); }
template <class Z> const void *multi_fn() { return reinterpret_cast<const void *>(multi_point_kernel<Z>); }

}  // namespace pnamp

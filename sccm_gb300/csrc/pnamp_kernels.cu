// Set-up of the pairs, projection onto J and K, and the launchers of the point kernels
// (point_kernels.cuh, one translation unit per arithmetic form).
#include <cooperative_groups.h>

#include <algorithm>

#include "point_kernels.cuh"

namespace pnamp {

// ------------------------------------------------------------------ setup
// min |U_kk| >= ratio x max |U_kk| over the pivots of a factored matrix, and max > 0.
__device__ __forceinline__ bool pivots_within(const double *A, int n, double ratio) {
    double mx = 0.0, mn = 1e300;
    for (int k = 0; k < n; ++k) {
        const double d = fabs(A[k * n + k]);
        mx = fmax(mx, d);
        mn = fmin(mn, d);
    }
    return mx > 0.0 && mn >= ratio * mx;
}

// One pair per cluster of four CTAs, bra and ket side by side and within each the two independent
// chains: (0, 1) U = LU, Z = V U^-1 (W or Z0), log|det U| and the Pfaffian of Z; (2, 3) log det of
// U^T U + V^T V, V = LU and U V^-1. The elimination steps follow one another at the FP64 pipe's
// latency, so the chains' length is the time: 460 steps in one CTA took 596 us for n = 40,
// 140 to 160 here.
//   det(1 + Z^T Z) = det(U^T U + V^T V) / det(U)^2, whose -1/4 power is the vacuum's overlap
// (the eigenvalue product of zbareover).
__global__ void __cluster_dims__(kSetupCluster, 1, 1) __launch_bounds__(kSetupThreads)
setup_kernel(Params p, const double *__restrict__ uv, double *__restrict__ pairbuf) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double xchg[4];   // this chain's logarithm of a determinant, its flags
    const int n = p.n, part = (int)cl.block_rank(), ket = (part & 1) == 0, tail = part >= 2;
    const long long nn = (long long)n * n, pair = blockIdx.x / kSetupCluster;
    const double *in = uv + pair * 4 * nn;
    double *out = pairbuf + pair * p.pl.stride;
    double *A = reinterpret_cast<double *>(smem_raw);
    double *Yb = A + nn;
    double *invd = Yb + nn;
    double *red = invd + n;
    zc *vecz = reinterpret_cast<zc *>(red + 64);    // n complex: the Pfaffian's pivot row
    int *perm = reinterpret_cast<int *>(vecz + n);
    int *sh = perm + n;
    const double *inU = in + (ket ? 2 : 0) * nn, *inV = inU + nn;   // column-major
    // row-major U0, V0, U1, V1 of the pair record: chain (bra, ket) x (U, V)
    for (long long t = threadIdx.x; t < nn; t += blockDim.x) {
        const int i = (int)(t / n), j = (int)(t % n);
        const double u = inU[i + (long long)j * n], v = inV[i + (long long)j * n];
        A[t] = tail ? v : u;
        Yb[t] = tail ? u : v;
        out[(tail ? (ket ? p.pl.v1 : p.pl.v0) : (ket ? p.pl.u1 : p.pl.u0)) + t] = A[t];
    }
    __syncthreads();
    int st = 0;
    double logdet = 0.0;
    if (tail) {   // U^T U + V^T V: both matrices are needed again, so the sum goes through registers
        constexpr int kMost = (kMaxN * kMaxN + kSetupThreads - 1) / kSetupThreads;
        double g[kMost];
#pragma unroll
        for (int e = 0; e < kMost; ++e) {
            const int t = threadIdx.x + e * kSetupThreads, i = t / n, j = t % n;
            double s = 0.0;
            if (t < n * n)
                for (int k = 0; k < n; ++k) {
                    s = fma(A[k * n + i], A[k * n + j], s);
                    s = fma(Yb[k * n + i], Yb[k * n + j], s);
                }
            g[e] = s;
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < kMost; ++e)
            if (threadIdx.x + e * kSetupThreads < n * n) A[threadIdx.x + e * kSetupThreads] = g[e];
        __syncthreads();
        if (lu_factor<double>(A, n, n, perm, invd, sh)) st = 1;
    }
    bool ok = false;
    for (int pass = tail ? 0 : 1; pass < 2; ++pass) {
        if (pass == 1) {
            if (tail) {
                for (long long t = threadIdx.x; t < nn; t += blockDim.x)
                    A[t] = inV[t / n + (t % n) * n];
                __syncthreads();
            }
            const bool sing = lu_factor<double>(A, n, n, perm, invd, sh);
            if (sing && !tail) st = 1;
            ok = !sing && pivots_within(A, n, kReducedPivotRatio);
        }
        if (pass == 0 || !tail) {
            double v[1] = {0.0};
            for (int k = threadIdx.x; k < n; k += blockDim.x) v[0] += log(fabs(A[k * n + k]));
            block_sum<1>(v, red);
            logdet = v[0];
        }
        __syncthreads();
    }
    if (!tail || ok) row_solve<double>(Yb, n, n, A, n, n, perm, invd);  // V U^-1, or U V^-1
    // entries of W^-1 and, where two-body densities are wanted, of Z0 (parts 2 and 1)
    const bool bounded = part == 2 || (part == 1 && p.n_r2q > 0);
    const double most = part == 2 ? kReducedMaxEntry : kReducedMaxZ0Rho2B;
    int big = 0;
    for (long long t = threadIdx.x; t < nn; t += blockDim.x) {
        if (!tail) out[(ket ? p.pl.w : p.pl.z0) + t] = Yb[t];
        if (!(fabs(Yb[t]) <= most)) big = 1;
    }
    big = __syncthreads_or(big);
    int cross = 0;   // proton-neutron blocks of this chain's matrix
    for (long long t = threadIdx.x; t < nn; t += blockDim.x) {
        const int i = (int)(t / n), j = (int)(t % n);
        if ((i < p.h) != (j < p.h) && (tail ? inV : inU)[i + (long long)j * n] != 0.0) cross = 1;
    }
    cross = __syncthreads_or(cross);
    if (threadIdx.x == 0) {
        xchg[0] = logdet;
        xchg[1] = (double)st;
        xchg[2] = ok && !(bounded && big) ? 1.0 : 0.0;
        xchg[3] = (double)cross;
    }
    cl.sync();
    double x[4][4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int q = 0; q < 4; ++q) x[k][q] = *cl.map_shared_rank(&xchg[q], k);
    cl.sync();   // read before any CTA exits
    // Once-per-pair pieces of the Pfaffians. Reduced pairs (V1 and U0 well conditioned): W^-1 and
    // Pf(c W) for point_reduced.cuh. Others with a well conditioned V0: block elimination of the
    // lower-right block of S = c [[D X D, -I], [I, -Z0]] gives Pf(S) = Pf(c (D X D - Z0^-1))
    // Pf(-c Z0). Otherwise both flags stay 0 and the 2n x 2n form is used. (A Pfaffian that
    // underflows is kept as the 2n x 2n form too.)
    const bool reduced = x[1][2] != 0.0 && x[2][2] != 0.0, schur = !reduced && x[3][2] != 0.0;
    // (the skew parts of W, W^-1 and Z0 for the reduced pairs, see point_reduced.cuh)
    if (reduced && (part == 1 || part == 2))
        for (int t = threadIdx.x; t < n * n; t += blockDim.x)
            out[(part == 1 ? p.pl.z0 : p.pl.zi) + t] = 0.5 * (Yb[t] - Yb[(t % n) * n + t / n]);
    if (schur && part == 3)
        for (long long t = threadIdx.x; t < nn; t += blockDim.x) out[p.pl.zi + t] = Yb[t];
    const int pfpart = schur ? 1 : 0;
    if (part != pfpart) return;
    int under = 0;
    zc pf = mk(0.0, 0.0);
    if (reduced || schur) {
        const double f = reduced ? p.cscale : -p.cscale;
        const double *Z = out + (reduced ? p.pl.w : p.pl.z0);   // this CTA's own result
        zc *Sz = reinterpret_cast<zc *>(A);  // n^2 complex over A and Yb
        for (long long t = threadIdx.x; t < nn; t += blockDim.x) {
            const int i = (int)(t / n), j = (int)(t % n);
            Sz[t] = mk(i < j ? f * (reduced ? 0.5 * (Z[t] - Z[j * n + i]) : Z[t]) : 0.0, 0.0);
        }
        __syncthreads();
        pf = pfaffian_upper<zc>(Sz, n, vecz, red, sh, under);   // in thread 0
    }
    if (threadIdx.x == 0) {
        const bool fine = under == 0 && zfinite(pf);
        out[p.pl.dets] = exp(-0.25 * (x[3][0] - 2.0 * x[1][0]));
        out[p.pl.dets + 1] = exp(-0.25 * (x[2][0] - 2.0 * x[0][0]));
        out[p.pl.dets + 2] = x[0][1] + x[1][1] + x[2][1] + x[3][1] != 0.0 ? 1.0 : 0.0;
        out[p.pl.dets + 3] = schur && fine ? 1.0 : 0.0;
        out[p.pl.pfz] = pf.x;
        out[p.pl.pfz + 1] = pf.y;
        // species split: U0, V0, U1, V1 without proton-neutron blocks (charge-conserving vacua)
        // make every per-point matrix block-diagonal by species (protons first, h = n/2 each)
        out[p.pl.dets + 6] = x[0][3] + x[1][3] + x[2][3] + x[3][3] != 0.0 ? 0.0 : 1.0;
        out[p.pl.dets + 7] = reduced && fine ? 1.0 : 0.0;
    }
}

int setup_smem_bytes(int n) { return (2 * n * n + n + 64 + 2 * n) * 8 + (n + 8) * 4; }

// The dynamic shared-memory limit of a kernel is a property of the function,
// shared by every context on the device: it is raised to the device maximum
// (never lowered to one context's need), so a context created later cannot
// invalidate the launches of an earlier one with a larger placement.
static cudaError_t raise_smem_limit(const void *f) {
    int dev = 0, optin = 0;
    cudaFuncAttributes fa;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, f);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    return e;
}

cudaError_t prepare_setup(int n) {
    if (setup_smem_bytes(n) <= 48 * 1024) return cudaSuccess;
    return raise_smem_limit((const void *)setup_kernel);
}

// Enqueues only (no attribute calls): usable under stream capture once
// prepare_setup(n) ran at context creation.
cudaError_t launch_setup(const Params &p, int npairs, const double *uv, double *pairbuf, cudaStream_t st) {
    setup_kernel<<<npairs * kSetupCluster, kSetupThreads, setup_smem_bytes(p.n), st>>>(p, uv, pairbuf);
    return cudaGetLastError();
}

// instantiated in point_fp64.cu and point_df64.cu, with the gauge points' values in point_gauge_*.cu
#define POINT_FORM(Z, Gauge)                                                                                           \
    extern template cudaError_t launch_points_z<Z, Gauge>(const Params &, int, const double *, zc *, int, double *,    \
                                                          int *, cudaStream_t, const int2 *, long long, double *,      \
                                                          double *, double *, int);                                    \
    extern template const void *point_fn<Z, Gauge>();
#define MULTI_FORM(Z)                                                                                                  \
    extern template cudaError_t launch_multi_z<Z>(const MultiArgs &, const int4 *, int, int, int *, zc *, int, int,    \
                                                  cudaStream_t);                                                       \
    extern template const void *multi_fn<Z>();
POINT_FORM(zc, false)
POINT_FORM(zc, true)
POINT_FORM(zd, false)
POINT_FORM(zd, true)
MULTI_FORM(zc)
MULTI_FORM(zd)
#undef POINT_FORM
#undef MULTI_FORM

cudaError_t multi_blocks_per_sm(int form, int smem_bytes, int *per_sm) {
    const void *f = form == 1 ? multi_fn<zd>() : multi_fn<zc>();
    cudaError_t e = raise_smem_limit(f);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, f, kThreads, smem_bytes);
}

cudaError_t launch_multi(int form, const MultiArgs &a, const int4 *items, int nitems, int grab, int *counter,
                         zc *scratch, int grid, int smem, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    return form == 1 ? launch_multi_z<zd>(a, items, nitems, grab, counter, scratch, grid, smem, st)
                     : launch_multi_z<zc>(a, items, nitems, grab, counter, scratch, grid, smem, st);
}

cudaError_t point_blocks_per_sm(int form, int smem_bytes, int *per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        per_sm, form == 1 ? point_fn<zd, false>() : point_fn<zc, false>(), kThreads, smem_bytes);
}

cudaError_t set_point_smem(int form, int bytes) {
    (void)bytes;  // checked against the device maximum by the placement planner
    const cudaError_t e = raise_smem_limit(form == 1 ? point_fn<zd, false>() : point_fn<zc, false>());
    return e != cudaSuccess ? e : raise_smem_limit(form == 1 ? point_fn<zd, true>() : point_fn<zc, true>());
}

// Euler points per split_items call: the choice with the fewest rounds of problems, where a
// batch of m points runs ceil(NFOM / chunks) rounds of one problem per thread group and the
// launch ceil(batches / grid) batches one after the other.
static int split_batch(const Params &p, long long nitems, long long per, int grid) {
    const RedPlan &L = p.place.spl;
    int best = 1;
    long long cost = -1;
    for (int m = 1; m <= L.items; m *= 2) {
        const int nc = std::max(1, std::min(L.ng / (2 * m), p.nfom));
        const long long units = 2LL * m * nc, rounds = ((units + L.ng - 1) / L.ng) * ((p.nfom + nc - 1) / nc);
        const long long batches = per > 0 ? (nitems / per) * ((per + m - 1) / m) : (nitems + m - 1) / m;
        const long long c = ((batches + grid - 1) / grid) * rounds;
        if (cost < 0 || c < cost) {
            cost = c;
            best = m;
        }
    }
    return best;
}

cudaError_t launch_points(const Params &p, int npairs, const double *pairbuf, zc *scratch, int grid,
                          double *zres, int *status, cudaStream_t st, const int2 *items, long long nitems,
                          double *gout, double *r1out, double *r2out) {
    if (r2out && (p.n_r2q <= 0 || !p.r2q || !p.r2acc)) return cudaErrorInvalidValue;
    const bool gauge = gout && !p.norm_only;   // H/N of every gauge point: one Euler point at a time
    const int batch = gauge ? 1 : split_batch(p, items ? nitems : (long long)npairs * p.n_euler, items ? 0 : p.n_euler, grid);
    const auto launch = p.form == 1 ? (gauge ? launch_points_z<zd, true> : launch_points_z<zd, false>)
                                    : (gauge ? launch_points_z<zc, true> : launch_points_z<zc, false>);
    return launch(p, npairs, pairbuf, scratch, grid, zres, status, st, items, nitems, gout, r1out, r2out, batch);
}

// ------------------------------------------------------------------ projection
// Weights W[ie][jkk] = wJ * w_ie * e^{i K1 alp} d^J_{K1K2}(bet) e^{i K2 gam}, jkk over
// (J = 0,2,4,6; K1 = -J..J; K2 = -J..J), wJ = (2J+1)/(8 pi^2) or (2J+1)/2 for an
// N_alp N_gam = 1 mesh (Kernel3D.f90:78-81).
__global__ void proj_weights_kernel(Params p, int axial, zc *w) {
    const int ie = blockIdx.x;
    const double alp = p.euler[4 * ie], bet = p.euler[4 * ie + 1], gam = p.euler[4 * ie + 2],
                 wt = p.euler[4 * ie + 3];
    double cb, sb;
    sincos(0.5 * bet, &sb, &cb);
    for (int jkk = threadIdx.x; jkk < kNJKK; jkk += blockDim.x) {
        int J = 0, rem = jkk;
        while (rem >= (2 * J + 1) * (2 * J + 1)) {
            rem -= (2 * J + 1) * (2 * J + 1);
            J += 2;
        }
        const int K1 = rem / (2 * J + 1) - J, K2 = rem % (2 * J + 1) - J;
        const double wj = axial ? (2.0 * J + 1.0) / 2.0 : (2.0 * J + 1.0) / (8.0 * M_PI * M_PI);
        const double d = wigner_d(2 * J, 2 * K1, 2 * K2, cb, sb, p.fact);
        w[(long long)ie * kNJKK + jkk] = (wj * wt * d) * expi(K1 * alp + K2 * gam);
    }
}

// One (pair, tile of 16 (J, K1, K2)) per cluster of 8 CTAs: the CTAs share the Euler points, a CTA's
// 256 threads are 16 weights x 16 points, partial sums meet in shared memory and then in the
// cluster's first CTA, in a fixed order. The sums are FP64 multiply-adds (8 complex ones per
// Euler point and weight) and a lone pair must reach every SM's narrow FP64 pipe: 144 CTAs per
// pair. One thread per weight over all Euler points took 2.35 ms for a pf pair's 2000 points.
constexpr int kProjTile = 16, kProjLanes = 16, kProjCluster = 8;
constexpr int kProjTiles = (kNJKK + kProjTile - 1) / kProjTile;
__global__ void __cluster_dims__(kProjCluster, 1, 1) __launch_bounds__(kProjTile * kProjLanes)
project_kernel(Params p, const zc *__restrict__ w, const double *__restrict__ zres, int core_prot, int core_neut,
               int chop, double *__restrict__ out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ zc part[8][kProjLanes][kProjTile];
    __shared__ zc sum[8][kProjTile];
    const int rank = (int)cl.block_rank();
    const int unit = (int)(blockIdx.x / kProjCluster);
    const int pair = unit / kProjTiles, j = threadIdx.x % kProjTile, ln = threadIdx.x / kProjTile;
    const int jkk = (unit % kProjTiles) * kProjTile + j;
    const double *z = zres + 2LL * pair * kNobs * p.n_euler;
    zc s[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = mk(0, 0);
    for (int ie = rank * kProjLanes + ln; ie < p.n_euler && jkk < kNJKK; ie += kProjCluster * kProjLanes) {
        const zc wv = w[(long long)ie * kNJKK + jkk];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q > 2 && q < 6) continue;   // not projected
            s[q] = zfma(wv, mk(z[2LL * (q * p.n_euler + ie)], z[2LL * (q * p.n_euler + ie) + 1]), s[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) part[q][ln][j] = s[q];
    __syncthreads();
    if (threadIdx.x < 8 * kProjTile) {
        const int q = threadIdx.x / kProjTile;
        zc v = part[q][0][j];
        for (int k = 1; k < kProjLanes; ++k) v = v + part[q][k][j];
        sum[q][j] = v;
    }
    cl.sync();
    if (rank == 0 && threadIdx.x < 8 * kProjTile) {
        const int q = threadIdx.x / kProjTile;
        zc v = sum[q][j];
        for (int k = 1; k < kProjCluster; ++k) v = v + *cl.map_shared_rank(&sum[q][j], k);
        part[q][0][j] = v;
    }
    cl.sync();   // the other CTAs' sums are read before they exit
    if (rank != 0 || threadIdx.x >= kProjTile || jkk >= kNJKK) return;
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] = part[q][0][j];
    int J = 0, rem = jkk;
    while (rem >= (2 * J + 1) * (2 * J + 1)) {
        rem -= (2 * J + 1) * (2 * J + 1);
        J += 2;
    }
    const int K1 = rem / (2 * J + 1) - J, K2 = rem % (2 * J + 1) - J;
    const long long fs = (long long)(kJJMax + 1) * kNK * kNK;
    const long long o = ((long long)J * kNK + (K1 + kJJMax)) * kNK + (K2 + kJJMax);
    double *op = out + 2LL * pair * kProjFields * fs;
    if (chop && !(sqrt(abs2(s[0])) >= 1.0e-8)) return;  // fields stay 0 (Kernel3D.f90:732)
    const zc inv0 = zrecip(s[0]);
    const zc f[kProjFields] = {s[0], s[6], s[2] * inv0 + mk(core_neut, 0), s[1] * inv0 + mk(core_prot, 0),
                               s[7] * inv0};
#pragma unroll
    for (int q = 0; q < kProjFields; ++q) {
        op[2 * (q * fs + o)] = f[q].x;
        op[2 * (q * fs + o) + 1] = f[q].y;
    }
}

cudaError_t launch_project(const Params &p, int npairs, const zc *w, const double *zres, int core_prot,
                           int core_neut, int chop, double *out, cudaStream_t st) {
    const int step = 0x7fffffff / (kProjTiles * kProjCluster);
    const long long fs = 2LL * kProjFields * (kJJMax + 1) * kNK * kNK;
    for (int p0 = 0; p0 < npairs; p0 += step) {
        const int np = std::min(step, npairs - p0);
        project_kernel<<<np * kProjTiles * kProjCluster, kProjTile * kProjLanes, 0, st>>>(
            p, w, zres + 2LL * p0 * kNobs * p.n_euler, core_prot, core_neut, chop, out + p0 * fs);
    }
    return cudaGetLastError();
}

// Quadrupole reduced elements <J1 K1||Q2||J2 K2>, J1 = J2 + dJ, dJ = 0, 1, 2
// (PNAMP_Kernel3D_v2.f90:515-600): one thread per (J2, dJ, K1, K2) output,
// direct and, when `exchange`, the q1 <-> q2 exchanged element from the Q^dagger
// traces. `tj` holds the 3j symbols (J1 2 J2; -K1 mu K2p) per output and mu.
// Output [pair][2][7][3][17][13] complex (direct, exchanged), zeroed beforehand.
__global__ void project_q_kernel(Params p, int axial, const double *__restrict__ zres, const double *__restrict__ tj,
                                 int exchange, double *__restrict__ out) {
    const int pair = blockIdx.x;
    const int o = blockIdx.y * blockDim.x + threadIdx.x;  // index into the (J2, dJ, K1, K2) list
    int J2 = 0, dJ = 0, rem = o, found = 0;
    for (J2 = 0; J2 <= kJJMax && !found; J2 += 2)
        for (dJ = 0; dJ < 3; ++dJ) {
            const int cnt = (2 * (J2 + dJ) + 1) * (2 * J2 + 1);
            if (rem < cnt) {
                found = 1;
                break;
            }
            rem -= cnt;
        }
    if (!found) return;
    J2 -= 2;  // undo the outer loop's final increment
    const int J1 = J2 + dJ;
    const int K1 = rem / (2 * J2 + 1) - J1, K2 = rem % (2 * J2 + 1) - J2;
    const double *z = zres + 2LL * pair * kNobs * p.n_euler;
    zc sd = mk(0, 0), sx = mk(0, 0);
    for (int ie = 0; ie < p.n_euler; ++ie) {
        const double alp = p.euler[4 * ie], bet = p.euler[4 * ie + 1], gam = p.euler[4 * ie + 2],
                     w = p.euler[4 * ie + 3];
        double cb, sb;
        sincos(0.5 * bet, &sb, &cb);
        for (int mu = -2; mu <= 2; ++mu) {
            const int K2p = K1 - mu;
            const double t3 = tj[5 * o + mu + 2];
            if (K2p > J2 || -K2p > J2 || t3 == 0.0) continue;
            const double ph = ((J1 - K1) & 1) ? -1.0 : 1.0;
            const zc zq = mk(z[2LL * ((10 + mu) * p.n_euler + ie)], z[2LL * ((10 + mu) * p.n_euler + ie) + 1]);
            const double d1 = wigner_d(2 * J2, 2 * K2p, 2 * K2, cb, sb, p.fact);
            sd = zfma((w * ph * t3 * d1) * expi(K2p * alp + K2 * gam), zq, sd);
            if (exchange) {
                const double d2 = wigner_d(2 * J2, 2 * K2, 2 * K2p, cb, sb, p.fact);
                const zc e2 = expi(-(K2 * alp + K2p * gam));
                for (int nu = -2; nu <= 2; ++nu) {
                    const int ix = 15 + nu;
                    const zc zt = mk(z[2LL * (ix * p.n_euler + ie)], -z[2LL * (ix * p.n_euler + ie) + 1]);
                    const double sg = ((mu - nu) & 1) ? -1.0 : 1.0;
                    const double dq = wigner_d(4, -2 * nu, -2 * mu, cb, sb, p.fact);
                    sx = zfma((w * ph * sg * dq * t3 * d2) * (expi(-(nu * alp + mu * gam)) * e2), zt, sx);
                }
            }
        }
    }
    const double wj = axial ? (2.0 * J2 + 1.0) / 2.0 : (2.0 * J2 + 1.0) / (8.0 * M_PI * M_PI);
    const double f = wj * (2 * J1 + 1);
    const long long blk = 7LL * 3 * 17 * 13;
    const long long idx = (((long long)J2 * 3 + dJ) * 17 + (K1 + 8)) * 13 + (K2 + 6);
    double *op = out + 2LL * pair * 2 * blk;
    op[2 * idx] = f * sd.x;
    op[2 * idx + 1] = f * sd.y;
    op[2 * (blk + idx)] = f * sx.x;
    op[2 * (blk + idx) + 1] = f * sx.y;
}

int n_q_outputs() {
    int c = 0;
    for (int J2 = 0; J2 <= kJJMax; J2 += 2)
        for (int dJ = 0; dJ < 3; ++dJ) c += (2 * (J2 + dJ) + 1) * (2 * J2 + 1);
    return c;
}

cudaError_t launch_project_q(const Params &p, int axial, int npairs, const double *zres, const double *tj,
                             int exchange, double *out, cudaStream_t st) {
    dim3 grid(npairs, (n_q_outputs() + 127) / 128);
    project_q_kernel<<<grid, 128, 0, st>>>(p, axial, zres, tj, exchange, out);
    return cudaGetLastError();
}

cudaError_t launch_proj_weights(const Params &p, int axial, zc *w, cudaStream_t st) {
    proj_weights_kernel<<<p.n_euler, 128, 0, st>>>(p, axial, w);
    return cudaGetLastError();
}

}  // namespace pnamp

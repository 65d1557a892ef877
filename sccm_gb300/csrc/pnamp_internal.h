// Internal interface between the C ABI (pnamp_capi.cu) and the kernels
// (pnamp_kernels.cu). Not part of the public header.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pnamp_df64.cuh"

namespace pnamp {

constexpr int kNobs = 19;
constexpr int kJJMax = 6;
constexpr int kNK = 2 * kJJMax + 1;
constexpr int kMaxN = 64;
constexpr int kMaxBlocks = 64;           // rotation blocks (t, n, l, j) of a model space
constexpr int kThreads = 512;            // threads per CTA of the point kernel (<= 128 registers)
constexpr int kNTrace = 10;              // proton traces of Q_{2mu} rho and Q_{2mu}^dagger rho
constexpr int kNJKK = 1 + 25 + 81 + 169; // (J, K1, K2) with even J <= 6
constexpr int kProjFields = 5;           // njkk, hjkk, nn, zz, j2
constexpr int kSetupThreads = 256;
constexpr int kSetupCluster = 4;          // CTAs that share one pair's set-up
constexpr int kMultiSmemTail = 16;       // dynamic shared bytes after the placement: multi kernel's counter

// One pair record (doubles), all matrices row-major n x n:
// U0 V0 U1 V1 W Z0 ZI then [det0, det1, status-as-double, Schur flag, Pf re, im, no
// proton-neutron blocks, reduced flag]. Reduced pairs (point_reduced.cuh): ZI = W^-1 = U1 V1^-1
// and Pf = Pf(c W). Others with the Schur flag: ZI = Z0^-1 = U0 V0^-1, Pf = Pf(-c Z0), and the
// point kernel eliminates the n x n matrix c (D X D - ZI) instead of the 2n x 2n one.
struct PairLayout {
    long long u0, v0, u1, v1, w, z0, zi, dets, pfz, stride;
    __host__ __device__ void make(int n) {
        long long nn = (long long)n * n;
        u0 = 0; v0 = nn; u1 = 2 * nn; v1 = 3 * nn; w = 4 * nn; z0 = 5 * nn; zi = 6 * nn; dets = 7 * nn;
        pfz = dets + 4;
        stride = 7 * nn + 8;
    }
};
// min/max |LU pivot| of V0 for the Schur complement's Pfaffian. A bra with nearly empty levels (small
// singular values of V0) makes Z0^-1 dominate the Schur complement c (D X D - Z0^-1), whose
// Pfaffian then carries the point's dependence in its low-order bits: on the shipped Ti48
// vacua a ratio of 2e-6 cost 2e-9 relative and 8e-5 cost 3e-7, while every bra at >= 3e-2
// stayed within 6e-13 of the 2n x 2n elimination. Below the bound the pair keeps the
// 2n x 2n form.
constexpr double kReducedPivotRatio = 1e-2;
// The reduced pairs of point_reduced.cuh: pivot ratios of U0 and V1 within the same bound and
// no entry of W^-1 = U1 V1^-1 above this. Its entries enter K = M^-1 - Z0 with their rounding in
// the point arithmetic. Double-float errors against FP64 over those of T22, geometric means over 250 sd and
// pf pairs of 4 to 32 nucleons and gaps of 0.35 to 1.5 MeV: norm, energy, <J^2> and one-body
// traces 0.7 to 1.2 up to 25, 1.0 to 2.0 between 25 and 40 (Ti48 pairs, at 18 to 36: 1.2); in a
// simulation with 24-bit words the densities are 10 to 20 times less exact at 76 (Ti48's beta2 = 0.3
// as the ket).
constexpr double kReducedMaxEntry = 40.0;
// kappa01 = Z0 + Z0 kappa10 Z0 cancels when Z0 is large (nearly full levels in the bra): its largest
// error, relative to its largest entry, is about Z0 times that of T22. The energy and <J^2>, where it
// meets kappa10 and the norm's error, do not show it: 0.8 to 1.1 of T22's error for entries of
// Z0 from 8 to 25, 0.3 to 0.7 from 30 to 130 (nearly full sd and pf shells). The two-body
// densities do, 1.1 to 1.6 times T22's error from 10 to 25 in the mean and 8 times in single pairs
// (1.0 below 8), so launches that form them hold Z0 below this.
constexpr double kReducedMaxZ0Rho2B = 8.0;

// Thread groups and shared memory (byte offsets) of the reduced pairs' problems, order N: ng
// groups of w warps, each with the inverse (then kappa10 above and kappa01 below the diagonal) and rho (N x ld complex each), the
// factorisation's scratch from off_scr in a region of grp_bytes. tile: the register tiles of
// the density products (rho in bits 0..3, kappa01 above). items: Euler points per batch of
// the species-split path. off_y: the right-hand sides of a group that goes by T22.
struct RedPlan {
    int ng, w, ld, items, tile;
    int off_eph, off_acc, off_z0, off_grp, off_scr, off_y, grp_bytes, smem_bytes;
};

// Where the per-point work arrays live: shared memory or the CTA's global slot.
// Offsets are in bytes (shared) or complex elements (global slot).
struct Placement {
    int s_smem, t_smem, y_smem, uv_smem;
    int off_s, off_t, off_y, off_uv;     // shared byte offsets (when *_smem)
    int off_piv, off_inv, off_red, off_rot, off_vec;
    RedPlan gen, spl;                    // reduced pairs: n x n problems, species-split h x h problems
    RedPlan sol;                         // other charge-conserving pairs: h x h problems by T22
    int smem_bytes;
    long long g_x, g_b, g_p, g_rw, g_zr, g_s, g_t, g_y, g_uv;
    long long slot_elems;
};

// Sparse one-body data used by the observables, built on the host once.
struct ObsTables {
    int n_t1b;                 // entries of the single-particle matrix
    const int *t1b_idx;        // index into rho (c*n + a) for t(a,c) rho(c,a)
    const double *t1b_val;
    int q_off[kNTrace + 1];    // entry ranges per trace
    const int *q_idx;          // index into rho
    const double *q_val;
    const double *jp;          // [n] J+_{a,a+1} (0 at the last state of a block)
    const double *jm;          // [n] J-_{a,a-1} (0 at the first state of a block)
    const double *mz;          // [n] m_a
    const double *jj1;         // [n] j(j+1)
    const dd *jp_d, *jm_d, *mz_d;   // the same coefficients as double-float
    const dd *jj1_d, *t1b_val_d, *q_val_d;
    // one-body density blocks (t, lj, n1, n2) of ZRho1B_Angles: block b sums
    // r1b_val[e] rho(row, col) over e in [r1b_off[b], r1b_off[b + 1]), packed row*256+col
    int n_r1b;
    const int *r1b_off, *r1b_idx;
    const double *r1b_val;
    const dd *r1b_val_d;
};
constexpr int kMaxR1B = 64;               // one-body density blocks per model space

// A bilinear form sum_r y_r sum_k V_rk s_rk over densities in shared memory, as slices of 32 rows
// (one per lane, longest rows first, padded with V = 0 to the slice's longest): slice q's steps are
// [start[q], start[q + 1]), entry (step, lane) has the element offset off of s and the value v;
// yoff[q * 32 + lane] is the row's y. The order of a row's entries spreads the 8 lanes that read
// shared memory together over the 8 16-byte bank groups.
struct EnergyTab {
    int nslice;
    const int *start;
    const unsigned short *yoff, *off;
    const double *v;
    const dd *vd;
};
enum { kTabGeneral = 0, kTabProton = 1, kTabNeutron = 2, kTabMixed = 3, kTabs = 4 };

struct Params {
    int n, h, N2;              // n, n/2, 2n
    int nprot, nneut;
    int n_euler, nfom, n_gauge;
    double cscale;
    double e0;                 // H%E0, added to every energy (Kernel3D.f90:324)
    double vacfac;             // (-1)^{n(n+1)/2} * 10^(-2*(n*iscale/2))
    int iE2;
    int form;                  // 0: FP64 (plain), 1: double-float per-point algebra
    int norm_only;             // 1: only the norm kernel N(Omega) (observable 0); the others are 0
    // rotation blocks
    int nblk, rot_elems;
    const int *blk_start, *blk_size, *blk_tj, *blk_roff, *row_blk, *twom;
    const double *euler;       // [n_euler][4] alpha, beta, gamma, weight
    int n_alpgam;              // Euler points per beta node (beta is the outermost loop)
    const double *wigner;      // [beta nodes][rot_elems] d^j_{m_i m_k}(beta) in the order of the blocks
    const unsigned short *rot_m;   // [rot_elems] 2 m_i + 64 | (2 m_k + 64) << 8
    const double *gphase;      // [nfom][nfom] complex e^{-i (phi_lp Z + phi_ln N)}, the projection phase
    const double *fact;        // k!, k = 0..23
    // Hamiltonian two-body list
    int nrec;
    int split_ok;              // every record: four protons, four neutrons, or a, c protons and b, d neutrons
    const uint32_t *rec_idx;   // packed 8-bit a,b,c,d (0-based)
    const double *rec_v;
    const dd *rec_vd;          // rec_v as double-float (df64 form)
    // the same interaction for the reduced points: over (A, Rh) of the n x n problem, of one
    // species' h x h problem, and the proton-neutron part over two h x h densities
    EnergyTab tab[kTabs];
    // slices dealt to the CTA's warps, general and (proton, neutron): [2 warps + 1] offsets by (warp,
    // species), then the slice numbers
    const int *sched[2];
    ObsTables obs;
    PairLayout pl;
    Placement place;
    // two-body density quadruples (ZRho2B_Angles): packed 8-bit k_i, k_j, k_k, k_l, and the
    // per-CTA FP64 accumulators [grid][r2_stride]; n_r2q = 0 outside Rho2B launches
    int n_r2q;
    const uint32_t *r2q;
    // the same quadruples with their index, [r2_off[0], r2_off[1]) four protons, [.., r2_off[2]) four
    // neutrons, the rest proton-neutron; r2_ss the longer same-species list, -1 when a quadruple
    // is of another kind
    const uint2 *r2s;
    int r2_off[3], r2_ss;
    double *r2acc;
    long long r2_stride;       // doubles of one CTA's sums, the same for pairs of every kind
    // tensor-core contraction (contract_tc.cu): tc_splits = 0 runs the record loop here;
    // 2 or 3 makes the point kernel write each gauge point's density rows as that many bf16
    // terms instead (X: tc_nk entries, ph part first, pp part from tc_nph; Y: the pp
    // epilogue vector, tc_nk - tc_nph entries) and its weight N / NFOM^2 (0 when T22 was
    // singular); point p of a launch is item * n_gauge + gauge index
    int tc_splits, tc_nk, tc_nph;
    const int *tc_src;         // [tc_nk]: r << 8 | c (ph entries), i << 8 | j (pp, i < j), -1 padding
    unsigned short *tc_x[3], *tc_y[3];
    double *tc_w;
    // species-split pairs: per CTA the rows of each species' problems [items][2][NFOM][3 terms][2]
    // of 2 tc_nk - tc_nph entries, zero outside the 16-byte chunks tc_chunks[tc_choff[s] ..) of
    // species s
    unsigned short *tc_sp;
    const int *tc_chunks;
    int tc_choff[3];
};

// Rows of the proton-neutron table per gauge angle, and the chunks of each species' gauge points
// for which the CTA's slot has room when H/N of every gauge point is wanted (split_items).
__host__ __device__ inline int gauge_rows(int h) { return (h * h + 31) / 32 * 32; }
__host__ __device__ inline int gauge_chunks(const Params &p, bool solve) {
    const long long hh = (long long)p.h * p.h;
    const long long room = p.place.slot_elems - (solve ? 13 : 2) * hh - (long long)p.nfom * (2 + gauge_rows(p.h));
    return room > 0 ? (int)(room / (2 * hh)) : 0;
}

// One group of the contraction: a contiguous range [off, off + dpad) of the X row (and, for
// a pp group, [yoff, yoff + dpad) of the Y row), whose square matrix occupies rows
// [rowbase, rowbase + dpad) of the stacked bf16 matrices (columns 0..dpad-1).
struct TcGroup {
    int kind;      // 0 particle-hole (epilogue vector = X), 1 particle-particle (epilogue vector = Y)
    int off, dpad, rowbase, yoff;
};
struct TcArgs {
    int splits;
    int ngroups;
    long long npts;
    int nk, npp;
    const TcGroup *groups;
    const unsigned short *x[3], *y[3];
    double *e2;        // [npts][2]
    int *err;
};

// Contexts of one multi-context launch, passed by value (kernel parameter space).
constexpr int kMultiCtx = 4;
struct MultiArgs {
    Params p[kMultiCtx];
    const double *pairbuf[kMultiCtx];
    double *zres[kMultiCtx];
    int *status[kMultiCtx];
    long long slot_stride;     // complex elements of one CTA's global slot
};

// launchers (pnamp_kernels.cu)
cudaError_t launch_setup(const Params &p, int npairs, const double *uv, double *pairbuf,
                         cudaStream_t st);
cudaError_t launch_points(const Params &p, int npairs, const double *pairbuf, zc *scratch,
                          int grid, double *zres, int *status, cudaStream_t st,
                          const int2 *items = nullptr, long long nitems = 0, double *gout = nullptr,
                          double *r1out = nullptr, double *r2out = nullptr);
cudaError_t launch_proj_weights(const Params &p, int axial, zc *w, cudaStream_t st);
cudaError_t launch_project(const Params &p, int npairs, const zc *w, const double *zres,
                           int core_prot, int core_neut, int chop, double *out, cudaStream_t st);
cudaError_t launch_project_q(const Params &p, int axial, int npairs, const double *zres, const double *tj,
                             int exchange, double *out, cudaStream_t st);
int n_q_outputs();
cudaError_t multi_blocks_per_sm(int form, int smem_bytes, int *per_sm);
cudaError_t launch_multi(int form, const MultiArgs &a, const int4 *items, int nitems, int grab, int *counter,
                         zc *scratch, int grid, int smem, cudaStream_t st);
cudaError_t set_point_smem(int form, int bytes);
cudaError_t point_blocks_per_sm(int form, int smem_bytes, int *per_sm);
int setup_smem_bytes(int n);
cudaError_t prepare_setup(int n);
// tensor-core contraction (contract_tc.cu)
cudaError_t prepare_contract();
int tc_smem_bytes(int splits);
int tc_chunk_rows(int splits);
cudaError_t launch_contract(const TcArgs &a, const void *const *mat, long long mat_rows, int kmax, int grid,
                            cudaStream_t st);
cudaError_t launch_contract_finish(int npairs, int n_euler, int n_gauge, long long nitems, const int2 *items,
                                   const double *w, const double *e2, double *zres, int *status, const int *err,
                                   cudaStream_t st);

}  // namespace pnamp

// Points of pairs with a well conditioned U0 (bra) and V1 (ket), the "reduced" pairs of
// setup_kernel: one skew-symmetric inverse per gauge point instead of a Pfaffian elimination,
// an n x n solve and three density products.
//
// With M = D X D (X = R W R^T, W = V1 U1^-1, D = diag(e^{i phi})), M^-1 = D* Y D* (Y = R* Wi R^+,
// Wi = W^-1 = U1 V1^-1, real and skew, one per pair) and Z0 = V0 U0^-1 (the same), the
// transition densities are functions of K = Y - D Z0 D alone:
//     kappa10 = D K^-1 D,   rho = -kappa10 Z0,   kappa01 = Z0 + Z0 kappa10 Z0,
// which follows from T22 = U0^T (1 - Z0 M) (D* R* U1): insert D R V1 = M D* R* U1 and rho =
// -M (1 - Z0 M)^-1 Z0 etc. K is also a Schur complement of the norm's matrix,
// Pf(c [[M, -1], [1, -Z0]]) = Pf(c M) Pf(c (M^-1 - Z0)) = Pf(c W) Pf(c K) (det R = 1, and the det D of
// the two factors cancel), so one factorisation by 2 x 2 pivots yields both: N/2 steps each way and N^3/2 complex
// multiply-adds for the inverse and the Pfaffian, 1.5 N^3 complex x real ones for rho and the
// upper triangle of kappa01 (skew), where the separate Pfaffian, Gauss-Jordan solve and
// density products took 4.3 N^3 complex-equivalents and N + N/2 steps. Nothing else of the
// ket enters, so T22, R V1 and R* U1 are not formed. (The other complement, M - Z0^-1, has the
// same form with Z0^-1 as the multiplier; its entries are 15 to 80 where those of Z0 are 2 to 20,
// and its kappa10 loses that factor. The phases stand with Z0 and not with the larger Y for
// the same reason.)
//
// W, W^-1 and Z0 are skew up to the rounding of the vacua times the condition of U or V. Their skew parts
// are taken: a symmetric error of Z0 or W then drops out of the norm to first order, where the upper
// triangles carried it in full. Against extended precision the norm of the Ti48 pairs (4, 5) and (5, 5) is
// exact to 2.4e-15 and 4.4e-15 instead of 2.4e-14 and 2.3e-14, of pf pairs at gap 0.4 MeV to 2.5e-14
// instead of 4.2e-14.
#pragma once

namespace pnamp {

// ------------------------------------------------------------------ accumulating arithmetic
// Sums of products with the factors prepared outside the loop (broadcast and negated words for
// the packed form). FP64: plain complex FMAs. Double-float: dd2_fma, renormalised after every
// product; joining the low words only at the end of the sum is 12 operations per product
// instead of 15, but its error is 3 times larger after 20 terms and 4 times after 40.
template <class Z> struct Op;
template <> struct Op<zc> {
    struct Mul { double x, y; };
    struct RMul { double r; };
    struct Rot {};
    using Acc = zc;
    static __device__ __forceinline__ Mul mul(zc a) { return {a.x, a.y}; }
    static __device__ __forceinline__ Mul mul_neg(zc a) { return {-a.x, -a.y}; }
    static __device__ __forceinline__ RMul rmul(double r) { return {r}; }
    static __device__ __forceinline__ Rot rot(zc) { return {}; }
    static __device__ __forceinline__ Acc acc(zc a) { return a; }
    static __device__ __forceinline__ void cadd(Acc &s, const Mul &a, zc b, Rot) {
        s.x = fma(a.x, b.x, fma(-a.y, b.y, s.x));
        s.y = fma(a.x, b.y, fma(a.y, b.x, s.y));
    }
    static __device__ __forceinline__ void radd(Acc &s, const RMul &r, zc b) {
        s.x = fma(r.r, b.x, s.x);
        s.y = fma(r.r, b.y, s.y);
    }
    static __device__ __forceinline__ zc done(const Acc &s) { return s; }
};
template <> struct Op<zd> {
    struct Mul { dd2 x; f2 nx; dd2 y; f2 ny; };
    struct RMul { dd2 r; f2 nr; };
    struct Rot { dd2 b; };
    struct Acc { f2 hi, lo; };
    static __device__ __forceinline__ Mul mul(zd a) {
        const dd x = re(a), y = im(a);
        return {dup(x), f2_dup(-x.hi), dup(y), f2_dup(-y.hi)};
    }
    static __device__ __forceinline__ Mul mul_neg(zd a) {
        const dd x = re(a), y = im(a);
        return {dup(dd_neg(x)), f2_dup(x.hi), dup(dd_neg(y)), f2_dup(y.hi)};
    }
    static __device__ __forceinline__ RMul rmul(dd r) { return {dup(r), f2_dup(-r.hi)}; }
    // i b = (-im, re)
    static __device__ __forceinline__ Rot rot(zd b) {
        return {{f2_make(-f2_b(b.hi), f2_a(b.hi)), f2_make(-f2_b(b.lo), f2_a(b.lo))}};
    }
    static __device__ __forceinline__ Acc acc(zd a) { return {a.hi, a.lo}; }
    // s += a b (both lanes), na = -a.hi
    static __device__ __forceinline__ void padd(Acc &s, dd2 a, f2 na, f2 bh, f2 bl) {
        const f2 p = f2_mul(na, bh);              // -(a b) rounded
        f2 e = f2_fma(a.hi, bh, p);               // its error
        e = f2_fma(a.hi, bl, e);
        e = f2_fma(a.lo, bh, e);
        const f2 t = f2_sub(s.hi, p);             // two_sum(s.hi, -p)
        const f2 v = f2_sub(t, s.hi);
        const f2 d = f2_sub(f2_sub(s.hi, f2_sub(t, v)), f2_add(p, v));
        const dd2 r = quick_two_sum(t, f2_add(d, f2_add(e, s.lo)));
        s.hi = r.hi;
        s.lo = r.lo;
    }
    static __device__ __forceinline__ void cadd(Acc &s, const Mul &a, zd b, const Rot &ib) {
        padd(s, a.x, a.nx, b.hi, b.lo);
        padd(s, a.y, a.ny, ib.b.hi, ib.b.lo);
    }
    static __device__ __forceinline__ void radd(Acc &s, const RMul &r, zd b) { padd(s, r.r, r.nr, b.hi, b.lo); }
    static __device__ __forceinline__ zd done(const Acc &s) { return {s.hi, s.lo}; }
};

// Magnitude key of a pivot candidate in 26 bits above the 6 index bits.
__device__ __forceinline__ unsigned sweep_key(zd a, int m) {
    return (fmaxf(fabsf(f2_a(a.hi)), fabsf(f2_b(a.hi))) >= 0.0f
                ? (__float_as_uint(fmaxf(fabsf(f2_a(a.hi)), fabsf(f2_b(a.hi)))) & ~63u) : 0u) | (unsigned)(63 - m);
}
__device__ __forceinline__ unsigned sweep_key(zc a, int m) {
    const unsigned x = (unsigned)__double2hiint(a.x) & 0x7fffffffu, y = (unsigned)__double2hiint(a.y) & 0x7fffffffu;
    const unsigned k = x > y ? x : y;
    return (k < 0x7ff00000u ? (k & ~63u) : 0u) | (unsigned)(63 - m);
}

__device__ __forceinline__ zc shfl_xor(zc a, int o) {
    return mk(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
}
__device__ __forceinline__ zd shfl_xor(zd a, int o) {
    zd r;
    r.hi.u = __shfl_xor_sync(0xffffffffu, a.hi.u, o);
    r.lo.u = __shfl_xor_sync(0xffffffffu, a.lo.u, o);
    return r;
}
template <class Z>
__device__ __forceinline__ Z warp_sum_z(Z v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = v + shfl_xor(v, o);
    return v;
}
// Scratch of one problem's factorisation: the pivots and their values, then byte lists of the
// remaining indices (two, alternating) and of the pivot order, last step first.
template <class Z> struct SkewScratch {
    Z piv[32], s[32], red[16];
    unsigned char list[2][64], ord[64];
};

// Entry t = b (b - 1) / 2 + a of an upper triangle, a < b.
__device__ __forceinline__ void skew_entry(int t, int &a, int &b) {
    b = (int)((sqrtf(8.0f * (float)t + 1.0f) + 1.0f) * 0.5f);
    if (b * (b - 1) / 2 > t) --b;
    if (b * (b + 1) / 2 <= t) ++b;
    a = t - b * (b - 1) / 2;
}

// Pfaffian factorisation of the skew matrix in the upper triangle of A (order N <= 64, even,
// row stride ld) by a thread group, and (`inverse`) its inverse over all of A.
//
// Forward: N/2 steps, each takes the first remaining row r, its largest remaining entry as pivot
// s = K_rq, and updates the remaining entries K_ij += v_i K_rj - K_ri v_j, v = K_q. / s. Rows
// move nowhere, the list of remaining indices shrinks instead; the sign of the pivot order goes
// into the pivots, so Pf(K) = prod piv. Entry t of the remaining triangle is (list[a], list[b])
// with t = b(b-1)/2 + a, so a thread's (a, b) are the same in every step (ab: a << 8 | b).
//
// Backward: with G = [[-v], [K_r. / s]] of a step and Y the inverse over the indices that remain
// after it, the step's two rows of the inverse are -G Y and its pivot entry is
// -1/s + (G Y G^T)_rq. Every intermediate is part of the inverse itself. (A sweep that carries
// the inverse forward, K_rj -> v_j and so on, has the same operation count in one pass over
// registers but passes through inverses of leading blocks, which can be large: its errors were
// 4 to 50 times larger.) v is kept at A[.][r], K_r. / s at A[q][.] in between.
// Returns true if a row had no usable entry (exactly singular or not finite).
template <class Z, int E>
__device__ __forceinline__ bool skew_factor(const Grp &g, int N, int ld, const int (&ab)[E], Z *A, Z *buf, int nbuf,
                                            SkewScratch<Z> &w, bool inverse) {
    using O = Op<Z>;
    const int lane = g.tid & 31;
    Z *Wb = buf, *Vb = buf + N;
    bool sing = false;
    for (int t = g.tid; t < N; t += g.nthr) w.list[0][t] = (unsigned char)t;
    gsync(g);
    for (int k = 0; k < N / 2; ++k) {
        const int m = N - 2 * k;
        const unsigned char *L = w.list[k & 1];
        unsigned char *Ln = w.list[(k + 1) & 1];
        const int r = L[0];
        unsigned key = 0u;
        for (int t = 1 + lane; t < m; t += 32) {
            const unsigned kk = sweep_key(A[r * ld + L[t]], t);
            key = key > kk ? key : kk;
        }
        key = __reduce_max_sync(0xffffffffu, key);
        const bool none = (key >> 6) == 0u;
        const int pos = none ? 1 : 63 - (int)(key & 63u);
        sing = sing || none;
        const int q = L[pos];
        const Z s = A[r * ld + q];
        if (g.tid == 0) {
            w.piv[k] = (pos & 1) ? s : -s;   // pos - 1 remaining indices lie between r and q
            w.s[k] = s;
            w.ord[m - 2] = (unsigned char)r;
            w.ord[m - 1] = (unsigned char)q;
        }
        if (m == 2) break;
        if (1 + g.tid < m) {
            const Z inv = zrecip(s);
            for (int t = 1 + g.tid; t < m; t += g.nthr) {
                if (t == pos) continue;
                const int c = t - 1 - (t > pos), i = L[t];
                const Z wi = A[r * ld + i], qi = i > q ? A[q * ld + i] : -A[i * ld + q];
                const Z vi = qi * inv;
                Wb[c] = wi;
                Vb[c] = vi;
                Ln[c] = (unsigned char)i;
                if (inverse) {
                    A[i * ld + r] = vi;
                    A[q * ld + i] = wi * inv;
                }
            }
        }
        gsync(g);
        const int T = (m - 2) * (m - 3) / 2;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if (g.tid + e * g.nthr >= T) break;
            const int a = ab[e] >> 8, b = ab[e] & 255;
            Z *x = A + (int)Ln[a] * ld + (int)Ln[b];
            const Z wb = Wb[b], vb = Vb[b];
            typename O::Acc c = O::acc(*x);
            O::cadd(c, O::mul(Vb[a]), wb, O::rot(wb));
            O::cadd(c, O::mul_neg(Wb[a]), vb, O::rot(vb));
            *x = O::done(c);
        }
        gsync(g);
    }
    if (!inverse) {
        gsync(g);
        return sing;
    }
    gsync(g);
    // (G Y G^T)_rq as one sum over all threads' pieces in double-float, where the one warp that
    // finished a step alone held the others up (pf mixing: 10.8 -> 9.0 of 44 Mcycles); in FP64 by
    // one warp over finished columns, since the extra products cost the narrow pipe more (sd
    // mixing: 7.0 against 7.8 of 34 Mcycles).
    constexpr bool kSpread = std::is_same<Z, zd>::value;
    const int wid = g.tid >> 5, nw = g.nthr >> 5;
    for (int k = N / 2 - 1; k >= 0; --k) {
        const int m = N - 2 - 2 * k, r = w.ord[m], q = w.ord[m + 1];
        // column b of -G Y in `parts` pieces, and this thread's piece of (G Y G^T)_rq
        const int parts = m > 0 ? min(min(g.nthr / m, m), nbuf / (2 * m)) : 0;
        const int b = m > 0 ? g.tid % m : 0, part = m > 0 ? g.tid / m : 0;
        Z x = szero<Z>();
        if (part < parts) {
            const int jb = w.ord[b];
            typename O::Acc xp = O::acc(szero<Z>()), xq = xp;
            for (int a = part; a < m; a += parts) {
                const int ia = w.ord[a];
                const Z y = A[ia * ld + jb];
                const typename O::Rot yr = O::rot(y);
                O::cadd(xp, O::mul(A[ia * ld + r]), y, yr);
                O::cadd(xq, O::mul_neg(A[q * ld + ia]), y, yr);
            }
            const Z yp = O::done(xp);
            buf[(2 * part) * m + b] = yp;
            buf[(2 * part + 1) * m + b] = O::done(xq);
            if constexpr (kSpread) x = A[q * ld + jb] * yp;
        }
        if constexpr (kSpread) {
            x = warp_sum_z(x);
            if (lane == 0) w.red[wid] = x;
        }
        gsync(g);
        if constexpr (kSpread) {
            for (int t = g.tid; t < 2 * m; t += g.nthr) {
                const int row = t < m ? 0 : 1, c = t - row * m, i = row ? q : r, j = w.ord[c];
                Z y = buf[row * m + c];
                for (int piece = 1; piece < parts; ++piece) y = y + buf[(2 * piece + row) * m + c];
                A[i * ld + j] = y;
                A[j * ld + i] = -y;
            }
        } else if (wid == 0) {
            typename O::Acc xs = O::acc(szero<Z>());
            for (int c = lane; c < m; c += 32) {
                Z yr = buf[c], yq = buf[m + c];
                for (int piece = 1; piece < parts; ++piece) {
                    yr = yr + buf[(2 * piece) * m + c];
                    yq = yq + buf[(2 * piece + 1) * m + c];
                }
                const int j = w.ord[c];
                O::cadd(xs, O::mul(A[q * ld + j]), yr, O::rot(yr));
                A[r * ld + j] = yr;
                A[j * ld + r] = -yr;
                A[q * ld + j] = yq;
                A[j * ld + q] = -yq;
            }
            x = warp_sum_z(O::done(xs));
        }
        if (g.tid == (kSpread ? g.nthr - 1 : 0)) {   // the spread form's last thread has no column
            if (kSpread) {
                x = w.red[0];
                for (int c = 1; c < nw; ++c) x = x + w.red[c];
            }
            const Z y = -(zrecip(w.s[k]) + x);
            A[r * ld + q] = y;
            A[q * ld + r] = -y;
            A[r * ld + r] = szero<Z>();
            A[q * ld + q] = szero<Z>();
        }
        gsync(g);
    }
    return sing;
}

// Pf = prod piv[k] (c times each, k < N/2 <= 32) by the lanes of one warp; the reference's
// pivot test |c piv| <= 1e-13 (or a non-finite pivot) sets `under` to 1 (2). Every lane
// gets the product.
template <class Z>
__device__ __forceinline__ zc pivot_product(const Z *piv, int np, double c, int &under) {
    const int lane = threadIdx.x & 31;
    int f = 0;
    Z v = Ar<Z>::from(mk(1.0, 0.0));
    if (lane < np) {
        v = Ar<Z>::from(mk(c, 0.0)) * piv[lane];
        f = pivot_flag(v);
    }
    const unsigned bad = __ballot_sync(0xffffffffu, f != 0);
    const int first = __shfl_sync(0xffffffffu, f, bad ? __ffs((int)bad) - 1 : 0);
    PfProd<Z> pf;
    pf.mul(v, false);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) pf.join(o);
    under = bad ? first : 0;
    return under ? mk(0.0, 0.0) : pf.get();
}

// rho^T = -Z0 K^-1 (A holds K^-1 in full), stored transposed, TI x TJ register tiles over the
// group. Z: Z0, skew, row stride N.
template <class Z, int TI, int TJ>
__device__ __forceinline__ void rho_tiles(const Grp &g, int N, int ld, const typename Ar<Z>::R *Z0, const Z *A, Z *Rh) {
    using O = Op<Z>;
    const int nj = (N + TJ - 1) / TJ, nt = ((N + TI - 1) / TI) * nj;
    for (int t = g.tid; t < nt; t += g.nthr) {
        const int i0 = (t / nj) * TI, j0 = (t % nj) * TJ;
        typename O::Acc acc[TI][TJ];
#pragma unroll
        for (int a = 0; a < TI; ++a)
#pragma unroll
            for (int b = 0; b < TJ; ++b) acc[a][b] = O::acc(szero<Z>());
        for (int k = 0; k < N; ++k) {
            Z bv[TJ];
#pragma unroll
            for (int b = 0; b < TJ; ++b) bv[b] = A[k * ld + min(j0 + b, N - 1)];
#pragma unroll
            for (int a = 0; a < TI; ++a) {   // -Z0_ik = Z0_ki
                const typename O::RMul m = O::rmul(Z0[k * N + min(i0 + a, N - 1)]);
#pragma unroll
                for (int b = 0; b < TJ; ++b) O::radd(acc[a][b], m, bv[b]);
            }
        }
#pragma unroll
        for (int a = 0; a < TI; ++a)
#pragma unroll
            for (int b = 0; b < TJ; ++b)
                if (i0 + a < N && j0 + b < N) Rh[(j0 + b) * ld + i0 + a] = O::done(acc[a][b]);
    }
}

// kappa01_ij = Z0_ij - sum_k rho_ki Z0_kj for i < j, stored at A[j][i]: the TI x TJ tiles that
// reach above the diagonal, in row order.
template <class Z, int TI, int TJ>
__device__ __forceinline__ void k01_tiles(const Grp &g, int N, int ld, const typename Ar<Z>::R *Z0, const Z *Rh, Z *A) {
    using O = Op<Z>;
    const int ni = (N + TI - 1) / TI, nj = (N + TJ - 1) / TJ;
    int t = g.tid, row = 0;
    for (;;) {
        // tiles of a row start at the first column tile that reaches above its first row
        int first = (row * TI + 1) / TJ;
        while (row < ni && t >= nj - first) {
            t -= max(nj - first, 0);
            ++row;
            first = (row * TI + 1) / TJ;
        }
        if (row >= ni) break;
        const int i0 = row * TI, j0 = (first + t) * TJ;
        typename O::Acc acc[TI][TJ];
#pragma unroll
        for (int a = 0; a < TI; ++a)
#pragma unroll
            for (int b = 0; b < TJ; ++b)   // Z0_ij = -Z0_ji
                acc[a][b] = O::acc(Ar<Z>::neg_real(Z0[min(j0 + b, N - 1) * N + min(i0 + a, N - 1)]));
        for (int k = 0; k < N; ++k) {
            Z av[TI];
#pragma unroll
            for (int a = 0; a < TI; ++a) av[a] = Rh[k * ld + min(i0 + a, N - 1)];
#pragma unroll
            for (int b = 0; b < TJ; ++b) {   // -Z0_kj = Z0_jk
                const typename O::RMul m = O::rmul(Z0[min(j0 + b, N - 1) * N + k]);
#pragma unroll
                for (int a = 0; a < TI; ++a) O::radd(acc[a][b], m, av[a]);
            }
        }
#pragma unroll
        for (int a = 0; a < TI; ++a)
#pragma unroll
            for (int b = 0; b < TJ; ++b)
                if (i0 + a < j0 + b && j0 + b < N) A[(j0 + b) * ld + i0 + a] = O::done(acc[a][b]);
        t += g.nthr;
    }
}

// One gauge point's skew matrix K = Y - d Z0 (order N, Y with row stride ldx, phase factors by
// the species of the row and column: d0 both below h0, d1 mixed, d2 both above), its Pfaffian
// factors into w and (`inverse`) rho into Rh and (kappa10, kappa01) into A: kappa10_ij =
// A[i][j] and kappa01_ij = A[j][i] for i < j.
template <class Z, int E>
__device__ __forceinline__ bool skew_problem_e(const Grp &g, int N, int ld, int h0, Z d0, Z d1, Z d2, const Z *Y, int ldx,
                                               const typename Ar<Z>::R *Z0, Z *A, Z *Rh, SkewScratch<Z> &w, bool inverse) {
    int ab[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int t = g.tid + e * g.nthr;
        int a, b;
        skew_entry(t, a, b);
        ab[e] = (a << 8) | b;
        if (t < N * (N - 1) / 2) {
            const Z d = b < h0 ? d0 : (a < h0 ? d1 : d2);
            A[a * ld + b] = rfma(Ar<Z>::rneg(Z0[a * N + b]), d, Y[a * ldx + b]);
        }
    }
    const bool sing = skew_factor<Z, E>(g, N, ld, ab, A, Rh, N * max(ld, 5), w, inverse);
    if (inverse) {   // kappa10 = D K^-1 D
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if (g.tid + e * g.nthr >= N * (N - 1) / 2) break;
            const int a = ab[e] >> 8, b = ab[e] & 255;
            const Z v = A[a * ld + b] * (b < h0 ? d0 : (a < h0 ? d1 : d2));
            A[a * ld + b] = v;
            A[b * ld + a] = -v;
        }
        gsync(g);
    }
    return sing;
}

template <class Z>
__device__ __noinline__ bool skew_problem(const Grp g, int N, int ld, int h0, Z d0, Z d1, Z d2, const Z *Y, int ldx,
                                          const typename Ar<Z>::R *Z0, Z *A, Z *Rh, SkewScratch<Z> &w, bool inverse,
                                          int tile) {
    bool sing = false;
    switch ((N * (N - 1) / 2 + g.nthr - 1) / g.nthr) {
#define CASE(E) \
    case E: sing = skew_problem_e<Z, E>(g, N, ld, h0, d0, d1, d2, Y, ldx, Z0, A, Rh, w, inverse); break;
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8)
#undef CASE
    }
    if (!inverse) return sing;
    switch (tile & 15) {
        case 0: rho_tiles<Z, 3, 2>(g, N, ld, Z0, A, Rh); break;
        case 1: rho_tiles<Z, 3, 3>(g, N, ld, Z0, A, Rh); break;
        case 2: rho_tiles<Z, 4, 2>(g, N, ld, Z0, A, Rh); break;
        case 3: rho_tiles<Z, 5, 3>(g, N, ld, Z0, A, Rh); break;
        default: rho_tiles<Z, 4, 4>(g, N, ld, Z0, A, Rh); break;
    }
    gsync(g);
    switch (tile >> 4) {
        case 0: k01_tiles<Z, 2, 2>(g, N, ld, Z0, Rh, A); break;
        case 1: k01_tiles<Z, 2, 4>(g, N, ld, Z0, Rh, A); break;
        case 2: k01_tiles<Z, 3, 3>(g, N, ld, Z0, Rh, A); break;
        default: k01_tiles<Z, 4, 4>(g, N, ld, Z0, Rh, A); break;
    }
    gsync(g);
    return sing;
}

// ------------------------------------------------------------------ problems by T22
// Charge-conserving pairs outside the reduced class (nearly empty or nearly full levels, so that Z0
// or W^-1 is large) whose V0 is well conditioned: one species' densities at one gauge angle from
// T22 = V0^T (d R V1) + U0^T (d* R* U1), d = e^{i phi}, whose entries are bounded whatever the levels,
//     rho = d R V1 T22^-1 V0^T,  kappa10 = d R V1 T22^-1 U0^T,  kappa01 = -d* R* U1 T22^-1 V0^T,
// and the norm from Pf(c (d^2 X - Z0^-1)) Pf(-c Z0), X = R W R^T: the algebra of full_item on a species'
// h x h block, which depends on its own gauge angle only. A solve with 2 h right-hand
// sides and three products: 1.8 times the time of the skew inverse. One pf pair, 4 + 4 nucleons, gap
// 0.2 MeV, 432 Euler x 81 gauge points: FP64 4.3 ms, double-float 2.4 ms; the same pair as n x n points
// (full_item) 116 and 46.6 ms, species blocks point by point 41.9 and 17.3 ms.
//
// One pair's constants and one (Euler point, species)'s matrices, in the CTA's global slot.
template <class Z> struct SolveData {
    const typename Ar<Z>::R *V0t, *U0t, *Zi;   // [h][h]: V0(j, k) at k h + j, U0 likewise; Z0^-1
    const Z *X, *B, *P;                        // [h][h]; [2][h][h] R V1, R* U1; [2][h][h] V0^T R V1, U0^T R* U1
};

// Y <- Y T^-1 (Y: ny x N, row stride N; T: N x N, row stride ld, destroyed) by column-oriented
// Gauss-Jordan elimination as gj_right_solve, for a thread group of any size: every warp searches the
// pivot of row k itself, so a step is two group barriers and all warps share its updates. Row k of
// T stays as it is in step k, and the columns k and c are exchanged in the rows below and in Y.
template <class Z>
__device__ __forceinline__ bool col_solve(const Grp &g, int N, int ld, Z *T, Z *Y, int ny) {
    using O = Op<Z>;
    const int lane = g.tid & 31, dq = g.nthr / N, dr = g.nthr % N, t0 = g.tid / N, j0 = g.tid % N;
    bool sing = false;
    for (int k = 0; k < N; ++k) {
        const Z *row = T + k * ld;
        unsigned key = 0u;
        for (int j = k + lane; j < N; j += 32) {
            const unsigned kk = sweep_key(row[j], j - k);
            key = key > kk ? key : kk;
        }
        key = __reduce_max_sync(0xffffffffu, key);
        const bool none = (key >> 6) == 0u;
        const int c = none ? k : k + 63 - (int)(key & 63u), nrT = N - k - 1, rows = nrT + ny;
        sing = sing || none;
        if (g.tid < rows) {
            const Z inv = none ? szero<Z>() : zrecip(row[c]);
            for (int t = g.tid; t < rows; t += g.nthr) {
                Z *r = t < nrT ? T + (k + 1 + t) * ld : Y + (t - nrT) * N;
                const Z a = r[c], b = r[k];
                r[k] = a * inv;
                if (c != k) r[c] = b;
            }
        }
        gsync(g);
        int j = j0;
        for (int t = t0; t < rows;) {
            if (j != k) {
                Z *r = t < nrT ? T + (k + 1 + t) * ld : Y + (t - nrT) * N;
                const Z p = row[j == c ? k : j];
                typename O::Acc x = O::acc(r[j]);
                O::cadd(x, O::mul_neg(r[k]), p, O::rot(p));
                r[j] = O::done(x);
            }
            t += dq;
            j += dr;
            if (j >= N) {
                j -= N;
                ++t;
            }
        }
        gsync(g);
    }
    return sing;
}

// The pivots of d^2 X - Z0^-1 into w and (`inverse`) the densities of the N
// levels at A and Rh (row stride ld) as skew_problem leaves them, kappa as the skew part. Y: 2 N x N.
template <class Z>
__device__ __noinline__ bool solve_problem(const Grp g, int N, int ld, Z d, const SolveData<Z> &S, Z *A, Z *Rh, Z *Y,
                                           SkewScratch<Z> &w, bool inverse) {
    using O = Op<Z>;
    const Z dc = zconj(d), d2 = d * d;
    {   // The phase stands with X, whose entries are smaller than those of Z0^-1 (the norm's error in
        // double-float is 1.2 to 1.8 times larger the other way). Y serves as the factorisation's scratch.
        // One form for up to 8 entries per thread, and not a call of skew_problem: a second caller of
        // that costs it registers (pf double-float 8.49 -> 8.56 ms).
        int ab[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            int a = 0, b = 1;
            const int t = g.tid + e * g.nthr;
            if (t < N * (N - 1) / 2) {
                skew_entry(t, a, b);
                A[a * ld + b] = zfma(d2, S.X[a * N + b], Ar<Z>::neg_real(S.Zi[a * N + b]));
            }
            ab[e] = (a << 8) | b;
        }
        skew_factor<Z, 8>(g, N, ld, ab, A, Y, 2 * N * N, w, false);
    }
    if (!inverse) return false;
    for (int t = g.tid; t < N * N; t += g.nthr) Rh[(t / N) * ld + t % N] = zfma(d, S.P[t], dc * S.P[N * N + t]);
    for (int t = g.tid; t < 2 * N * N; t += g.nthr) Y[t] = S.B[t];
    gsync(g);
    const bool sing = col_solve<Z>(g, N, ld, Rh, Y, 2 * N);
    const Z *Yu = Y + N * N;
    const typename Ar<Z>::R half = Ar<Z>::rconst(0.5f);
    for (int t = g.tid; t < N * N; t += g.nthr) {
        const int i = t / N, j = t % N;
        typename O::Acc x = O::acc(szero<Z>());
        for (int k = 0; k < N; ++k) O::radd(x, O::rmul(S.V0t[k * N + j]), Y[i * N + k]);
        Rh[i * ld + j] = d * O::done(x);
        if (i < j) {
            typename O::Acc a = O::acc(szero<Z>()), b = a;
            for (int k = 0; k < N; ++k) {
                O::radd(a, O::rmul(S.U0t[k * N + j]), Y[i * N + k]);
                O::radd(a, O::rmul(Ar<Z>::rneg(S.U0t[k * N + i])), Y[j * N + k]);
                O::radd(b, O::rmul(Ar<Z>::rneg(S.V0t[k * N + j])), Yu[i * N + k]);
                O::radd(b, O::rmul(S.V0t[k * N + i]), Yu[j * N + k]);
            }
            A[i * ld + j] = half * (d * O::done(a));
            A[j * ld + i] = half * (dc * O::done(b));
        } else if (i == j) {
            A[i * ld + i] = szero<Z>();
        }
    }
    gsync(g);
    return sing;
}

// One pair's constants of SolveData, both species: V0t, U0t, Zi [2][h][h] each from `c` on.
template <class Z>
__device__ __noinline__ void solve_constants(const Params &p, const double *__restrict__ pr, typename Ar<Z>::R *c) {
    const int h = p.h, hh = h * h, n = p.n;
    for (int t = threadIdx.x; t < 2 * hh; t += blockDim.x) {
        const int s = t / hh, k = (t % hh) / h, j = t % h, o = (s * h + j) * n + s * h + k;
        c[t] = Ar<Z>::real(pr[p.pl.v0 + o]);
        c[2 * hh + t] = Ar<Z>::real(pr[p.pl.u0 + o]);
        c[4 * hh + t] = Ar<Z>::real(pr[p.pl.zi + (s * h + k) * n + s * h + j]);
    }
}

// B and P of SolveData for m Euler points, both species: B[m][2][2][h][h] holds the FP64 values until the
// products are formed; rot: the Euler points' rotation blocks.
template <class Z>
__device__ __noinline__ void solve_setup(const Params &p, const double *__restrict__ pr, int m, const zc *rot, Z *B, Z *P) {
    const int h = p.h, hh = h * h, n = p.n;
    const double *gU0 = pr + p.pl.u0, *gV0 = pr + p.pl.v0, *gU1 = pr + p.pl.u1, *gV1 = pr + p.pl.v1;
    zc *Bz = reinterpret_cast<zc *>(B);
    __syncthreads();
    for (int t = threadIdx.x; t < 2 * hh * m; t += blockDim.x) {
        const int is = t / hh, e = t % hh, s = is & 1, a = s * h + e / h, j = s * h + e % h;
        const int b = p.row_blk[a], s0 = p.blk_start[b], d = p.blk_size[b];
        const zc *Rr = rot + (long long)(is >> 1) * p.rot_elems + p.blk_roff[b] + (a - s0) * d;
        zc v = mk(0, 0), u = mk(0, 0);
        for (int k = 0; k < d; ++k) {
            v = rfma(gV1[(s0 + k) * n + j], Rr[k], v);
            u = rfma(gU1[(s0 + k) * n + j], zconj(Rr[k]), u);
        }
        Bz[2 * is * hh + e] = v;
        Bz[(2 * is + 1) * hh + e] = u;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 4 * hh * m; t += blockDim.x) {
        const int q = t / hh, e = t % hh, i = e / h, j = e % h, o = ((q >> 1) & 1) * h;
        const double *M = (q & 1 ? gU0 : gV0) + o * n + o + i;
        zc s = mk(0, 0);
        for (int k = 0; k < h; ++k) s = rfma(M[k * n], Bz[q * hh + k * h + j], s);
        P[t] = Ar<Z>::from(s);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 4 * hh * m; t += blockDim.x) {   // in place
        const zc v = Bz[t];
        B[t] = Ar<Z>::from(v);
    }
    __syncthreads();
}

// ------------------------------------------------------------------ observables of one point
template <class Z> struct PointSums {
    Z e2, t1, j2, tp, tm, tz;   // two- and one-body energy, <J^2> without its traces, Tr J+, J-, Jz rho
};
// Sum over the group, valid in its first warp. red: 16 values.
template <class Z>
__device__ __forceinline__ Z group_sum(const Grp &g, Z v, Z *red) {
    v = warp_sum_z(v);
    if (g.nthr == 32) return v;
    const int lane = g.tid & 31, wid = g.tid >> 5, nw = g.nthr >> 5;
    if (lane == 0) red[wid] = v;
    gsync(g);
    if (wid == 0) v = warp_sum_z(lane < nw ? red[lane] : szero<Z>());
    gsync(g);
    return v;
}

// Slices [first, ..) in steps of `stride` of a bilinear form over the densities at M, added to e2:
// one row per lane, the row's factor applied at its end.
template <class Z>
__device__ __forceinline__ void energy_slices(const EnergyTab &t, int first, int stride, int lane, const Z *M,
                                              typename Op<Z>::Acc &e2) {
    using O = Op<Z>;
    using Ra = Ar<Z>;
    for (int q = first; q < t.nslice; q += stride) {
        const int e0 = t.start[q] * 32 + lane, e1 = t.start[q + 1] * 32;
        typename O::Acc s = O::acc(szero<Z>());
#pragma unroll 4
        for (int e = e0; e < e1; e += 32) O::radd(s, O::rmul(Ra::pick(t.v, t.vd, e)), M[t.off[e]]);
        const Z y = O::done(s);
        O::cadd(e2, O::mul(M[t.yoff[q * 32 + lane]]), y, O::rot(y));
    }
}

// The double-float energies of `cnt` problems at once by the whole CTA: each warp takes the slices
// that `sched` deals it and applies every table entry to all problems, whose (A, Rh) start at
// smem + off[k]; its sum for problem k goes to its reduction slot in that problem's scratch. The
// table (10 bytes per entry, 0.12 MB for a pf species, 0.8 MB for n = 40) comes from L2: read by
// every problem for itself its latency bound the loop (FP64 and double-float took the same
// time), shared by the CTA's problems it is read 4 times less often (pf, split and mixing; 7 or 8
// times for split sd). The slices are dealt longest first to the least loaded warp over both species. FP64 is
// bound by its pipe either way and keeps the groups independent (energy_slices).
template <class Z, int C>
__device__ __forceinline__ void energy_round_c(const EnergyTab &t, const int *task, int ntask, unsigned char *smem,
                                               const int (&off)[8], int scr) {
    using O = Op<Z>;
    using Ra = Ar<Z>;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    typename O::Acc sum[C];
#pragma unroll
    for (int k = 0; k < C; ++k) sum[k] = O::acc(szero<Z>());
    for (int i = 0; i < ntask; ++i) {
        const int q = task[i];
        const int e0 = t.start[q] * 32 + lane, e1 = t.start[q + 1] * 32;
        typename O::Acc a[C];
#pragma unroll
        for (int k = 0; k < C; ++k) a[k] = O::acc(szero<Z>());
#pragma unroll 2
        for (int e = e0; e < e1; e += 32) {
            const typename O::RMul v = O::rmul(Ra::pick(t.v, t.vd, e));
            const int o = t.off[e];
#pragma unroll
            for (int k = 0; k < C; ++k) O::radd(a[k], v, reinterpret_cast<const Z *>(smem + off[k])[o]);
        }
        const int y = t.yoff[q * 32 + lane];
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const Z x = O::done(a[k]);
            O::cadd(sum[k], O::mul(reinterpret_cast<const Z *>(smem + off[k])[y]), x, O::rot(x));
        }
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const Z v = warp_sum_z(O::done(sum[k]));
        if (lane == 0) reinterpret_cast<SkewScratch<Z> *>(smem + off[k] + scr)->red[wid] = v;
    }
}
template <class Z>
__device__ __noinline__ void energy_round(const EnergyTab &t, const int *sched, int sp, unsigned char *smem, int cnt,
                                          const int *list, int grp, int grp_bytes, int scr) {
    const int b = 2 * ((int)threadIdx.x >> 5) + sp, *task = sched + 2 * (kThreads / 32) + 1 + sched[b];
    const int nt = sched[b + 1] - sched[b];
    for (int k0 = 0; k0 < cnt; k0 += 8) {
        int off[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) off[k] = grp + list[min(k0 + k, cnt - 1)] * grp_bytes;
        switch (min(cnt - k0, 8)) {   // a count without a case of its own repeats its last problem
            case 1: energy_round_c<Z, 1>(t, task, nt, smem, off, scr); break;
            case 2: energy_round_c<Z, 2>(t, task, nt, smem, off, scr); break;
            case 3:
            case 4: energy_round_c<Z, 4>(t, task, nt, smem, off, scr); break;
            default: energy_round_c<Z, 8>(t, task, nt, smem, off, scr); break;
            case 5:
            case 6:
            case 7: energy_round_c<Z, 7>(t, task, nt, smem, off, scr); break;
        }
    }
}
template <class Z> struct Shared { static constexpr bool energies = std::is_same<Z, zd>::value; };

// Observables of the densities of skew_problem over the levels [lev0, lev0 + N): the two-body
// energy by tab (null: left out; double-float: from energy_round's sums in red), the one-body
// energy, and <J^2> (ZJ2_0, PNAMP_ME2B.f90:45-147;
// Jx, Jy = (J+ +- J-)/(2, 2i), J-_{a+1,a} = J+_{a,a+1}) without sum_a j(j+1) rho_aa, which is
// linear in rho, and without the products of traces. Sums are valid in the group's first warp.
template <class Z>
__device__ __noinline__ PointSums<Z> point_sums(const Grp g, const Params &p, int N, int ld, int lev0,
                                                const EnergyTab *tab, const Z *A, const Z *Rh, Z *red) {
    using O = Op<Z>;
    using Ra = Ar<Z>;
    using R = typename Ra::R;
    PointSums<Z> out;
    typename O::Acc t1 = O::acc(szero<Z>()), j2 = t1, tp = t1, tm = t1, tz = t1;
    out.e2 = szero<Z>();
    if (tab) {
        if constexpr (Shared<Z>::energies) {
            if (g.tid < 32) out.e2 = warp_sum_z(g.tid < kThreads / 32 ? red[g.tid] : szero<Z>());
            gsync(g);
        } else {
            typename O::Acc e2 = O::acc(szero<Z>());
            energy_slices<Z>(*tab, g.tid >> 5, g.nthr >> 5, g.tid & 31, A, e2);   // Rh follows A
            out.e2 = group_sum(g, O::done(e2), red);
        }
    }
    for (int e = g.tid; e < p.obs.n_t1b; e += g.nthr) {
        const int ix = p.obs.t1b_idx[e], r = (ix >> 8) - lev0, c = (ix & 255) - lev0;
        if ((unsigned)r < (unsigned)N && (unsigned)c < (unsigned)N)
            O::radd(t1, O::rmul(Ra::pick(p.obs.t1b_val, p.obs.t1b_val_d, e)), Rh[r * ld + c]);
    }
    for (int t = g.tid; t < N * N; t += g.nthr) {
        const int a = t / N, c = t % N;
        const R jpa = Ra::pick(p.obs.jp, p.obs.jp_d, lev0 + a), jpc = Ra::pick(p.obs.jp, p.obs.jp_d, lev0 + c);
        const R mza = Ra::pick(p.obs.mz, p.obs.mz_d, lev0 + a), mzc = Ra::pick(p.obs.mz, p.obs.mz_d, lev0 + c);
        if (a <= c) {
            const Z rac = Rh[a * ld + c], rca = Rh[c * ld + a];
            typename O::Acc x = O::acc(szero<Z>());
            O::cadd(x, O::mul_neg(rac), rca, O::rot(rca));
            R f = Ra::rmul(mza, mzc);
            if (a < c) {
                const Z kk = A[c * ld + a];
                O::cadd(x, O::mul(A[a * ld + c]), kk, O::rot(kk));
                f = Ra::radd(f, f);
            }
            O::radd(j2, O::rmul(f), O::done(x));
        }
        if (Ra::nz(jpa) && Ra::nz(jpc)) {
            const Z rc = Rh[c * ld + a];
            typename O::Acc x = O::acc(szero<Z>());
            O::cadd(x, O::mul_neg(Rh[(a + 1) * ld + c + 1]), rc, O::rot(rc));
            // kappa10_{a+1,c} kappa01_{a,c+1}
            if (c > a + 1) {
                const Z k2 = A[(c + 1) * ld + a];
                O::cadd(x, O::mul(A[(a + 1) * ld + c]), k2, O::rot(k2));
            } else if (c < a - 1) {
                const Z k2 = A[a * ld + c + 1];
                O::cadd(x, O::mul(A[c * ld + a + 1]), k2, O::rot(k2));
            } else if (c == a) {
                const Z k2 = A[(a + 1) * ld + a];
                O::cadd(x, O::mul_neg(A[a * ld + a + 1]), k2, O::rot(k2));
            }
            O::radd(j2, O::rmul(Ra::rmul(jpa, jpc)), O::done(x));
        }
        if (a == c) {
            O::radd(tz, O::rmul(mza), Rh[a * ld + a]);
            if (Ra::nz(jpa)) {
                O::radd(tp, O::rmul(jpa), Rh[(a + 1) * ld + a]);
                O::radd(tm, O::rmul(jpa), Rh[a * ld + a + 1]);
            }
        }
    }
    out.t1 = group_sum(g, O::done(t1), red);
    out.j2 = group_sum(g, O::done(j2), red);
    out.tp = group_sum(g, O::done(tp), red);
    out.tm = group_sum(g, O::done(tm), red);
    out.tz = group_sum(g, O::done(tz), red);
    return out;
}

// ZRho2B_Angles (PNAMP_Rho2B.f90:105-112) before its Clebsch-Gordan sums, for the levels (i, j, k, l)
// of a packed quadruple less lev0: rho_ki rho_lj - rho_li rho_kj + kappa01_ij kappa10_kl.
template <class Z>
__device__ __forceinline__ Z quad_product(uint32_t pk, int lev0, int ld, const Z *A, const Z *Rh) {
    const int i = (int)(pk & 0xff) - lev0, j = (int)((pk >> 8) & 0xff) - lev0, k = (int)((pk >> 16) & 0xff) - lev0,
              l = (int)(pk >> 24) - lev0;
    Z t = Rh[k * ld + i] * Rh[l * ld + j];
    t = zfms(Rh[l * ld + i], Rh[k * ld + j], t);
    if (i != j && k != l) {
        const Z u = A[max(i, j) * ld + min(i, j)], v = A[min(k, l) * ld + max(k, l)];
        t = (i < j) == (k < l) ? zfma(u, v, t) : zfms(u, v, t);
    }
    return t;
}

// The group's part of the tensor-core operand rows of point pt (X: rho entries, then K10 pairs;
// Y: K01 pairs) as split-bf16 terms; K_xy = kappa_xy - kappa_yx = 2 kappa_xy.
template <class Z>
__device__ __noinline__ void tc_rows(const Grp g, const Params &p, int ld, const Z *A, const Z *Rh, long long pt) {
    const int S = p.tc_splits, nk = p.tc_nk, npp = p.tc_nk - p.tc_nph;
    for (int e = g.tid; e < nk; e += g.nthr) {
        const int src = p.tc_src[e];
        Z v = szero<Z>(), y = v;
        if (src >= 0) {
            const int r = src >> 8, c = src & 255;
            if (e < p.tc_nph) {
                v = Rh[r * ld + c];
            } else {
                v = A[r * ld + c];
                y = A[c * ld + r];
                v = v + v;
                y = y + y;
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
}

// The same of one species' problem (levels [lev0, lev0 + N)): a row of the full width, X entries
// then Y entries, [term][re, im], in which only the 16-byte chunks with entries of that species
// are written (`chunks`; the rest of the buffer stays zero). A gauge point's operand rows are
// the bitwise union of its two species' rows (join_rows).
template <class Z>
__device__ __noinline__ void species_rows(const Grp g, const Params &p, int s, int N, int ld, const Z *A, const Z *Rh,
                                          unsigned short *row) {
    const int S = p.tc_splits, nk = p.tc_nk, W = 2 * nk - p.tc_nph, lev0 = s * N;
    for (int ci = p.tc_choff[s] + g.tid; ci < p.tc_choff[s + 1]; ci += g.nthr) {
        const int e0 = 8 * p.tc_chunks[ci];
        uint32_t o[3][2][4];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int e = e0 + q, src = p.tc_src[e < nk ? e : e - nk + p.tc_nph];
            const int r = (src >> 8) - lev0, c = (src & 255) - lev0;
            Z v = szero<Z>();
            if (src >= 0 && (unsigned)r < (unsigned)N && (unsigned)c < (unsigned)N) {
                v = e < p.tc_nph ? Rh[r * ld + c] : (e < nk ? A[r * ld + c] : A[c * ld + r]);
                if (e >= p.tc_nph) v = v + v;   // K_xy = 2 kappa_xy
            }
            unsigned short tr[3], ti[3];
            bf16_terms(as_dd(re(v)), S, tr);
            bf16_terms(as_dd(im(v)), S, ti);
#pragma unroll
            for (int sp = 0; sp < 3; ++sp) {
                if (q & 1) {
                    o[sp][0][q >> 1] |= (uint32_t)tr[sp] << 16;
                    o[sp][1][q >> 1] |= (uint32_t)ti[sp] << 16;
                } else {
                    o[sp][0][q >> 1] = tr[sp];
                    o[sp][1][q >> 1] = ti[sp];
                }
            }
        }
#pragma unroll
        for (int sp = 0; sp < 3; ++sp)
            if (sp < S)
#pragma unroll
                for (int ri = 0; ri < 2; ++ri)
                    *reinterpret_cast<uint4 *>(row + (long long)(2 * sp + ri) * W + e0) =
                        make_uint4(o[sp][ri][0], o[sp][ri][1], o[sp][ri][2], o[sp][ri][3]);
    }
}

// Operand rows of the NFOM^2 gauge points of m Euler points from their species' rows, by the
// whole CTA: a thread holds one 16-byte chunk of eight neutron rows and joins every proton row
// to them. Bound by the stores (40 KB per point for three terms and the pf shell, 2.5 TB/s
// reached), which leave as streaming writes; 31.2 -> 30.7 ms for four pf pairs against loading a
// neutron chunk per store.
static __device__ __noinline__ void join_rows(const Params &p, int m, const unsigned short *rows, long long pt0) {
    constexpr int kHold = 8;
    const int S = p.tc_splits, nk = p.tc_nk, npp = nk - p.tc_nph, W = nk + npp, nf = p.nfom, nch = W / 8;
    const int total = m * S * 2 * nch;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int c = t % nch, u = t / nch, ri = u & 1, sp = (u >> 1) % S, it = (u >> 1) / S;
        const unsigned short *r0 = rows + (long long)it * 2 * nf * 6 * W + (2 * sp + ri) * W + 8 * c;
        const bool x = 8 * c < nk;
        const long long width = x ? nk : npp, pt = 2 * (pt0 + (long long)it * p.n_gauge) + ri;
        unsigned short *dst = (x ? p.tc_x[sp] + 8 * c : p.tc_y[sp] + (8 * c - nk)) + pt * width;
        for (int l0 = 0; l0 < nf; l0 += kHold) {
            uint4 b[kHold];
#pragma unroll
            for (int k = 0; k < kHold; ++k)
                if (l0 + k < nf) b[k] = *reinterpret_cast<const uint4 *>(r0 + (long long)(nf + l0 + k) * 6 * W);
#pragma unroll 3
            for (int lp = 0; lp < nf; ++lp) {
                const uint4 a = *reinterpret_cast<const uint4 *>(r0 + (long long)lp * 6 * W);
                unsigned short *o = dst + 2LL * width * (lp * nf + l0);
#pragma unroll
                for (int k = 0; k < kHold; ++k)
                    if (l0 + k < nf)
                        __stcs(reinterpret_cast<uint4 *>(o + 2LL * width * k),
                               make_uint4(a.x | b[k].x, a.y | b[k].y, a.z | b[k].z, a.w | b[k].w));
            }
        }
    }
}

// Rotation blocks R_b(i,k) = e^{-i alp m_i} d^j_{m_i m_k}(bet) e^{-i gam m_k} of one Euler point
// (ROTATION_MAT, PNAMP_Proj.f90:83-136), entries t = tid, tid + nthr, ... of rot.
// d^j comes from the context's table, made once per mesh: Wigner's sum at every point was half of
// a norm-only pass (2.07 -> 1.45 ms for 2 x 1024 Euler points of pf).
__device__ __forceinline__ void rotation_blocks(const Params &p, int ie, int tid, int nthr, zc *rot) {
    const double alp = p.euler[4 * ie], gam = p.euler[4 * ie + 2];
    const double *d = p.wigner + (long long)(ie / p.n_alpgam) * p.rot_elems;
    for (int e = tid; e < p.rot_elems; e += nthr) {
        const int mm = p.rot_m[e];   // 2 m_i + 64 | (2 m_k + 64) << 8
        rot[e] = d[e] * expi(-0.5 * (alp * ((mm & 255) - 64) + gam * ((mm >> 8) - 64)));
    }
}

// One-body sums over the weighted density (FP64, rows and columns of the levels
// [lev0, lev0 + N), stored at Sb[(r - lev0) lds + c - lev0]) of one (item, species) or item:
// slots 0 Tr over protons, 1 over neutrons, 2 one-body energy, 3 sum j(j+1) rho_aa,
// 4..6 Tr J+, J-, Jz, 7..16 the Q_{2mu} traces (proton rows).
constexpr int kOneBody = 17;
__device__ __forceinline__ zc one_body(const Params &p, int q, int lane, int lev0, int N, const zc *Sb, int lds) {
    zc s = mk(0.0, 0.0);
    if (q == 0 || q == 1 || q == 3 || q == 6) {
        for (int a = lane; a < N; a += 32) {
            const int g = lev0 + a;
            double f = 1.0;
            if (q == 0) f = g < p.h ? 1.0 : 0.0;
            else if (q == 1) f = g < p.h ? 0.0 : 1.0;
            else if (q == 3) f = p.obs.jj1[g];
            else f = p.obs.mz[g];
            if (f != 0.0) s = rfma(f, Sb[a * lds + a], s);
        }
    } else if (q == 4 || q == 5) {
        for (int a = lane; a < N; a += 32) {
            const double f = p.obs.jp[lev0 + a];
            if (f != 0.0) s = rfma(f, q == 4 ? Sb[(a + 1) * lds + a] : Sb[a * lds + a + 1], s);
        }
    } else {
        const int e0 = q == 2 ? 0 : p.obs.q_off[q - 7], e1 = q == 2 ? p.obs.n_t1b : p.obs.q_off[q - 6];
        const int *idx = q == 2 ? p.obs.t1b_idx : p.obs.q_idx;
        const double *val = q == 2 ? p.obs.t1b_val : p.obs.q_val;
        for (int e = e0 + lane; e < e1; e += 32) {
            const int ix = idx[e], r = (ix >> 8) - lev0, c = (ix & 255) - lev0;
            if ((unsigned)r < (unsigned)N && (unsigned)c < (unsigned)N) s = rfma(val[e], Sb[r * lds + c], s);
        }
    }
    s.x = warp_sum(s.x);
    s.y = warp_sum(s.y);
    return s;
}

// sb (+)= w rho: the sum over gauge points stays FP64.
template <class Z>
__device__ __noinline__ void add_weighted(const Grp g, int N, int ld, zc w, const Z *Rh, zc *sb, bool first) {
    for (int t = g.tid; t < N * N; t += g.nthr) {
        const zc rv = Ar<Z>::to(Rh[(t / N) * ld + t % N]);
        sb[t] = first ? w * rv : zfma(w, rv, sb[t]);
    }
}

// ------------------------------------------------------------------ general reduced points
// One Euler point of a reduced pair: its NFOM^2 gauge points dealt to the plan's thread
// groups, which run them independently (n x n problems, named barriers per group). Observables
// linear in rho are taken once per Euler point from the norm-weighted sum of rho.
template <class Z>
__device__ __noinline__ void reduced_item(const Params &p, const double *__restrict__ pr, zc *slot, int pair, int ie,
                                          bool reload, double *__restrict__ zout, int *__restrict__ status,
                                          double *__restrict__ gout, double *__restrict__ r1out,
                                          double *__restrict__ r2out, long long pt0) {
    using Ra = Ar<Z>;
    using R = typename Ra::R;
    extern __shared__ __align__(16) unsigned char smem[];
    const RedPlan &L = p.place.gen;
    const int n = p.n, h = p.h, nn = n * n, ld = L.ld;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ng = L.ng, gthr = 32 * L.w, gid = (int)threadIdx.x / gthr;
    const bool onishi = p.nfom == 1, inverse = !p.norm_only;
    Z *ephz = reinterpret_cast<Z *>(smem + L.off_eph);
    zc *gacc = reinterpret_cast<zc *>(smem + L.off_acc);    // [ng][4]: N, N E2, N J2, N (unused)
    int *gflag = reinterpret_cast<int *>(gacc + 4 * ng);
    R *Z0 = reinterpret_cast<R *>(smem + L.off_z0);
    Z *Y = reinterpret_cast<Z *>(slot);                     // R* Wi R^+
    zc *RW = slot + nn;                                     // R* Wi
    zc *Sb = slot + nn;                                     // [ng][n n], after RW is used
    const double *gU1 = pr + p.pl.u1, *gV1 = pr + p.pl.v1, *gWi = pr + p.pl.zi, *gZ0 = pr + p.pl.z0;
    const zc pfw = mk(pr[p.pl.pfz], pr[p.pl.pfz + 1]);
    const double pre = p.vacfac * pr[p.pl.dets] * pr[p.pl.dets + 1];
    if (reload) {
        __syncthreads();
        for (int t = threadIdx.x; t < nn; t += blockDim.x) Z0[t] = Ra::real(gZ0[t]);
        const double twopi = 6.283185307179586476925287;
        for (int l = threadIdx.x; l < p.nfom; l += blockDim.x)
            ephz[l] = Ra::from(expi(onishi ? 0.0 : twopi * l / p.nfom));
    }
    zc *rot = reinterpret_cast<zc *>(smem + L.off_grp);     // before the groups use their storage
    __syncthreads();
    rotation_blocks(p, ie, threadIdx.x, blockDim.x, rot);
    __syncthreads();
    for (int t = threadIdx.x; t < nn; t += blockDim.x) {
        const int a = t / n, j = t % n;
        const int b = p.row_blk[a], s0 = p.blk_start[b], d = p.blk_size[b];
        const zc *Rr = rot + p.blk_roff[b] + (a - s0) * d;
        zc rw = mk(0, 0);
        for (int k = 0; k < d; ++k) rw = rfma(gWi[(s0 + k) * n + j], zconj(Rr[k]), rw);
        RW[t] = rw;
    }
    __syncthreads();
    // Y = (R* Wi) R^+, upper triangle (Y is skew)
    for (int t = threadIdx.x; t < n * (n - 1) / 2; t += blockDim.x) {
        int a, c;
        tri_index(t, n, a, c);
        const int b = p.row_blk[c], s0 = p.blk_start[b], d = p.blk_size[b];
        const zc *Rr = rot + p.blk_roff[b] + (c - s0) * d;
        zc x = mk(0, 0);
        for (int k = 0; k < d; ++k) x = zfma(RW[a * n + s0 + k], zconj(Rr[k]), x);
        Y[a * n + c] = Ra::from(x);
    }
    zc nrm1 = mk(0.0, 0.0);
    if (onishi) {
        // Onishi (PNAMP_Onishi.f90:21-37): sqrt(det(Ubar^T U0 + Vbar^T V0)), Ubar = R U1,
        // Vbar = conj(R) V1 at phi = 0; LU determinant, principal root
        const double *gU0 = pr + p.pl.u0, *gV0 = pr + p.pl.v0;
        zc *RU = slot + 2 * nn, *RV = slot + 3 * nn;
        for (int t = threadIdx.x; t < nn; t += blockDim.x) {
            const int a = t / n, j = t % n;
            const int b = p.row_blk[a], s0 = p.blk_start[b], d = p.blk_size[b];
            const zc *Rr = rot + p.blk_roff[b] + (a - s0) * d;
            zc ru = mk(0, 0), rv = mk(0, 0);
            for (int k = 0; k < d; ++k) {
                ru = rfma(gU1[(s0 + k) * n + j], Rr[k], ru);
                rv = rfma(gV1[(s0 + k) * n + j], zconj(Rr[k]), rv);
            }
            RU[t] = ru;
            RV[t] = rv;
        }
        __syncthreads();
        zc *Bm = reinterpret_cast<zc *>(smem + L.off_grp);   // n x n, one group's A and Rh hold it
        zc *invz = Bm + nn;
        int *perm = reinterpret_cast<int *>(invz + n);
        for (int t = threadIdx.x; t < nn; t += blockDim.x) {
            const int i = t / n, j = t % n;
            zc s = mk(0, 0);
            for (int k = 0; k < n; ++k) {
                s = rfma(gU0[k * n + j], RU[k * n + i], s);
                s = rfma(gV0[k * n + j], RV[k * n + i], s);
            }
            Bm[t] = s;
        }
        __syncthreads();
        const bool bsing = lu_factor<zc>(Bm, n, n, perm, invz, perm + n);
        if (threadIdx.x == 0) {
            zc det = mk(1.0, 0.0);
            for (int k = 0; k < n; ++k) {
                det = det * Bm[k * n + k];
                if (perm[k] != k) det = -det;
            }
            if (bsing) det = mk(0.0, 0.0);
            const double r = sqrt(det.x * det.x + det.y * det.y);
            nrm1 = mk(sqrt(0.5 * (r + det.x)), copysign(sqrt(0.5 * fmax(r - det.x, 0.0)), det.y));
        }
        __syncthreads();
    }
    __syncthreads();
    const Grp g{(int)threadIdx.x - gid * gthr, gthr, 1 + gid};
    const bool mine = gid < ng, energies = inverse && !p.tc_splits;
    const bool rounds = energies && Shared<Z>::energies;   // spare warps only join energy_round
    unsigned char *gb = smem + L.off_grp + (mine ? gid : 0) * L.grp_bytes;
    Z *A = reinterpret_cast<Z *>(gb), *Rh = A + n * ld;
    SkewScratch<Z> &w = *reinterpret_cast<SkewScratch<Z> *>(gb + L.off_scr);
    zc *nsh = reinterpret_cast<zc *>(gb + L.off_scr + sizeof(SkewScratch<Z>));   // the point's norm
    zc *sb = Sb + (long long)gid * nn;
    double *r2acc = r2out && mine ? p.r2acc + p.r2_stride * blockIdx.x + 2LL * p.n_r2q * gid : nullptr;
    for (int q = g.tid; q < (r2acc ? p.n_r2q : 0); q += g.nthr) {
        r2acc[2 * q] = 0.0;
        r2acc[2 * q + 1] = 0.0;
    }
    zc aN = mk(0, 0), aE = mk(0, 0), aJ = mk(0, 0);      // the group's thread 0
    int flags = 0, list[8];
    for (int k = 0; k < 8; ++k) list[k] = k;
    bool first = true;
    for (int g0 = 0; g0 < p.n_gauge; g0 += ng) {
        const int gi = g0 + gid;
        const bool act = mine && gi < p.n_gauge;
        bool sing = false;
        zc norm = mk(0, 0);
        if (act) {
            const int lp = gi / p.nfom, ln = gi % p.nfom;
            const Z zep = ephz[lp], zen = ephz[ln];
            sing = skew_problem<Z>(g, n, ld, h, zep * zep, zep * zen, zen * zen, Y, n, Z0, A, Rh, w, inverse, L.tile);
            if (g.tid < 32) {
                int under;
                const zc pf = pivot_product<Z>(w.piv, n / 2, p.cscale, under);
                if (lane == 0) {
                    const zc zph = mk(p.gphase[2 * gi], p.gphase[2 * gi + 1]);
                    norm = onishi ? nrm1 : pre * ((pf * pfw) * zph);
                    flags |= (onishi ? 0 : (under == 1 ? 1 : (under == 2 ? 4 : 0))) | (inverse && sing ? 2 : 0);
                    aN = aN + norm;
                    nsh[0] = norm;
                }
            }
        }
        if (rounds) {
            __syncthreads();
            energy_round<Z>(p.tab[kTabGeneral], p.sched[0], 0, smem, min(ng, p.n_gauge - g0), list, L.off_grp, L.grp_bytes, L.off_scr);
            __syncthreads();
        }
        if (!act) continue;
        const bool eval = inverse && !sing;
        PointSums<Z> s;
        if (eval) {
            s = point_sums<Z>(g, p, n, ld, 0, energies ? &p.tab[kTabGeneral] : nullptr, A, Rh, w.red);
            if (p.tc_splits) tc_rows<Z>(g, p, ld, A, Rh, pt0 + gi);
        }
        if (g.tid == 0) {
            zc hg = mk(0, 0);
            if (eval) {
                const zc e = Ra::to(s.e2), t = Ra::to(s.t1);
                hg = mk(e.x + t.x + p.e0, e.y + t.y);
                aE = zfma(norm, hg, aE);
                const zc a = Ra::to(s.tp), b = Ra::to(s.tm), c = Ra::to(s.tz);
                aJ = zfma(norm, Ra::to(s.j2) + a * b + c * c, aJ);
            }
            if (gout) {
                double *o = gout + 4LL * (((long long)pair * p.n_euler + ie) * p.n_gauge + gi);
                o[0] = norm.x;
                o[1] = norm.y;
                o[2] = hg.x;
                o[3] = hg.y;
            }
            if (p.tc_splits) {
                const double inv = 1.0 / ((double)p.nfom * p.nfom);
                p.tc_w[2 * (pt0 + gi)] = eval ? inv * norm.x : 0.0;
                p.tc_w[2 * (pt0 + gi) + 1] = eval ? inv * norm.y : 0.0;
            }
        }
        gsync(g);   // nsh
        if (eval) {
            const zc nv = nsh[0];
            add_weighted<Z>(g, n, ld, nv, Rh, sb, first);
            first = false;
            for (int q = g.tid; q < (r2acc ? p.n_r2q : 0); q += g.nthr) {
                const zc a = zfma(nv, Ra::to(quad_product<Z>(p.r2q[q], 0, ld, A, Rh)),
                                  mk(r2acc[2 * q], r2acc[2 * q + 1]));
                r2acc[2 * q] = a.x;
                r2acc[2 * q + 1] = a.y;
            }
        }
        gsync(g);   // the next point overwrites the densities
    }
    if (first && inverse && mine)
        for (int t = g.tid; t < nn; t += g.nthr) sb[t] = mk(0.0, 0.0);
    if (g.tid == 0 && mine) {
        gacc[4 * gid] = aN;
        gacc[4 * gid + 1] = aE;
        gacc[4 * gid + 2] = aJ;
        gflag[gid] = flags;
    }
    __syncthreads();
    // ---- the groups' sums: weighted density into the first group's storage, one-body traces
    zc *St = reinterpret_cast<zc *>(smem + L.off_grp), *ob = St + nn;
    if (inverse) {
        for (int t = threadIdx.x; t < nn; t += blockDim.x) {
            zc s = Sb[t];
            for (int q = 1; q < ng; ++q) s = s + Sb[(long long)q * nn + t];
            St[t] = s;
        }
        __syncthreads();
        for (int q = wid; q < kOneBody; q += kThreads / 32) {
            const zc v = q >= 7 && !p.iE2 ? mk(0, 0) : one_body(p, q, lane, 0, n, St, n);
            if (lane == 0) ob[q] = v;
        }
        if (r1out) {
            const double inv = 1.0 / ((double)p.nfom * p.nfom);
            for (int b = wid; b < p.obs.n_r1b; b += kThreads / 32) {
                zc s = mk(0, 0);
                for (int e = p.obs.r1b_off[b] + lane; e < p.obs.r1b_off[b + 1]; e += 32) {
                    const int ix = p.obs.r1b_idx[e];
                    s = rfma(p.obs.r1b_val[e], St[(ix >> 8) * n + (ix & 255)], s);
                }
                s.x = warp_sum(s.x);
                s.y = warp_sum(s.y);
                if (lane == 0) {
                    r1out[2LL * (((long long)pair * p.obs.n_r1b + b) * p.n_euler + ie)] = inv * s.x;
                    r1out[2LL * (((long long)pair * p.obs.n_r1b + b) * p.n_euler + ie) + 1] = inv * s.y;
                }
            }
        }
        if (r2out) {   // Euler weight x gauge mean, added into the pair's sums (ZRho2B_Integral at J = 0)
            const double wgt = p.euler[4 * ie + 3] / ((double)p.nfom * p.nfom);
            double *o = r2out + 2LL * p.n_r2q * pair;
            const double *a = p.r2acc + p.r2_stride * blockIdx.x;
            for (int q = threadIdx.x; q < 2 * p.n_r2q; q += blockDim.x) {
                double s = 0.0;
                for (int k = 0; k < ng; ++k) s += a[2LL * p.n_r2q * k + q];
                atomicAdd(o + q, wgt * s);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < kNobs) {
        const int io = threadIdx.x;
        const double inv = 1.0 / ((double)p.nfom * p.nfom);
        zc v = mk(0, 0);
        int f = 0;
        for (int q = 0; q < ng; ++q) {
            f |= gflag[q];
            if (io == 0) v = v + gacc[4 * q];
            else if (io == 6) v = v + gacc[4 * q + 1];
            else if (io == 7) v = v + gacc[4 * q + 2];
        }
        if (inverse) {
            if (io >= 1 && io <= 3) v = ob[io - 1];
            else if (io == 7) v = v + ob[3];
            else if (io >= 8 && io < 18) v = ob[io - 1];
        }
        v = inv * v;
        const unsigned bad = __ballot_sync((1u << kNobs) - 1u, !zfinite(v));
        zout[2LL * (io * p.n_euler + ie)] = v.x;
        zout[2LL * (io * p.n_euler + ie) + 1] = v.y;
        if (io == 0) status[(long long)pair * p.n_euler + ie] = f | (bad ? 4 : 0);
    }
    __syncthreads();
}

// ------------------------------------------------------------------ species-split pairs
// A pair without proton-neutron blocks: K is block-diagonal by species and the proton block
// depends on phi_p only, the neutron block on phi_n only (K_s = Y_s - e^{2 i phi_s} Z0_s). So an
// Euler point needs 2 NFOM problems of order h = n / 2, not NFOM^2 of order n. With the species'
// weights a_s(phi) = Pf(c K_s) e^{-i phi N_s}, the norm is the product of the two sums of a_s,
// observables of one species are its weighted sum times the other's norm sum, and the
// proton-neutron energy and the cross terms of <J^2> are bilinear in the two weighted densities
// sum_phi a_s rho_s, one contraction per Euler point.
//
// H/N of one species' problem at angle l with the other species' angles: the neutrons leave their
// energy `e` (two- and one-body, in the group's first warp) in En and F in F; the protons, when all
// neutrons are through, write E_p + E_n + E_pn + e0 for every phi_n whose neutron problem was
// regular. A is free: the density goes there without its padding.
template <class Z>
__device__ __noinline__ void gauge_values(const Grp g, const Params &p, int h, int ld, int s, int l, zc e, Z *A,
                                          const Z *Rh, zc *En, Z *F, double *gp) {
    using O = Op<Z>;
    using Ra = Ar<Z>;
    const EnergyTab &t = p.tab[kTabMixed];
    const int lane = g.tid & 31, wid = g.tid >> 5, nw = g.nthr >> 5, hh = h * h, nf = p.nfom, rows = gauge_rows(h);
    gsync(g);
    for (int k = g.tid; k < hh; k += g.nthr) A[k] = Rh[(k / h) * ld + k % h];
    gsync(g);
    if (s) {
        for (int q = wid; q < t.nslice; q += nw) {
            typename O::Acc x = O::acc(szero<Z>());
            for (int k = t.start[q] * 32 + lane; k < t.start[q + 1] * 32; k += 32)
                O::radd(x, O::rmul(Ra::pick(t.v, t.vd, k)), A[t.v[k] != 0.0 ? t.off[k] - hh : 0]);
            F[(long long)l * rows + q * 32 + lane] = O::done(x);
        }
        if (g.tid == 0) {
            En[2 * l] = e;
            En[2 * l + 1] = mk(1.0, 0.0);
        }
        return;
    }
    for (int ln = wid; ln < nf; ln += nw) {
        typename O::Acc x = O::acc(szero<Z>());
        for (int q = 0; q < t.nslice; ++q) {
            const Z y = A[t.yoff[q * 32 + lane]];
            O::cadd(x, O::mul(F[(long long)ln * rows + q * 32 + lane]), y, O::rot(y));
        }
        const Z v = warp_sum_z(O::done(x));
        if (lane == 0 && En[2 * ln + 1].x != 0.0) {
            const zc r = Ra::to(v) + En[2 * ln];
            gp[4 * (l * nf + ln) + 2] = r.x;
            gp[4 * (l * nf + ln) + 3] = r.y;
        }
    }
    gsync(g);
    if (wid == 0)
        for (int ln = lane; ln < nf; ln += 32)
            if (En[2 * ln + 1].x != 0.0) {
                gp[4 * (l * nf + ln) + 2] += e.x + p.e0;
                gp[4 * (l * nf + ln) + 3] += e.y;
            }
}

// Rotation blocks of m Euler points (listed, or from ie0 on) and the species blocks of
// Y = (R* Wi) R^+ or (Solve, gWi = W) X = (R W) R^T, upper triangles. Like add_weighted a function of its
// own: inlined in split_items they cost it registers (four pf pairs in BF16x6 30.77 ms, 30.54 ms so).
template <class Z, bool Solve>
__device__ __noinline__ void split_setup(const Params &p, const double *__restrict__ gWi, const int2 *__restrict__ items,
                                         int ie0, int m, zc *rot, zc *RW, Z *Y) {
    using Ra = Ar<Z>;
    const int h = p.h, n = p.n, hh = h * h, wid = threadIdx.x >> 5;
    auto euler = [&](int k) { return items ? items[k].y : ie0 + k; };
    {
        // warps share the Euler points evenly
        const int wpi = max(1, (kThreads / 32) / m), item = wid / wpi;
        if (item < m)
            rotation_blocks(p, euler(item), (int)threadIdx.x - item * wpi * 32, wpi * 32, rot + (long long)item * p.rot_elems);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 2 * hh * m; t += blockDim.x) {
        const int it = t / (2 * hh), e = t % (2 * hh), s = e / hh, a = s * h + (e % hh) / h, j = s * h + e % h;
        const int b = p.row_blk[a], s0 = p.blk_start[b], d = p.blk_size[b];
        const zc *Rr = rot + (long long)it * p.rot_elems + p.blk_roff[b] + (a - s0) * d;
        zc rw = mk(0, 0);
        for (int k = 0; k < d; ++k) rw = rfma(gWi[(s0 + k) * n + j], Solve ? Rr[k] : zconj(Rr[k]), rw);
        RW[t] = rw;
    }
    __syncthreads();
    const int Th = h * (h - 1) / 2;
    for (int t = threadIdx.x; t < 2 * Th * m; t += blockDim.x) {
        const int it = t / (2 * Th), e = t % (2 * Th), s = e / Th;
        int a, c;
        tri_index(e % Th, h, a, c);
        const int b = p.row_blk[s * h + c], s0 = p.blk_start[b], d = p.blk_size[b];
        const zc *Rr = rot + (long long)it * p.rot_elems + p.blk_roff[b] + (s * h + c - s0) * d;
        const zc *rw = RW + (long long)(2 * it + s) * hh + a * h + s0 - s * h;
        zc x = mk(0, 0);
        for (int k = 0; k < d; ++k) x = zfma(rw[k], Solve ? Rr[k] : zconj(Rr[k]), x);
        Y[(long long)(2 * it + s) * hh + a * h + c] = Ra::from(x);
    }
}

// Up to ng / 2 Euler points at a time: a unit (Euler point, species, chunk of the gauge
// points) per thread group, so that a launch with few Euler points still fills the groups.
//
// Solve: the pair's problems go by T22 (solve_problem) instead of the skew inverse. Gauge: H/N of
// every gauge point goes to gout, for one Euler point at a time and the neutrons' problems first.
// H/N at (phi_p, phi_n) is E_p + E_n + sum_r rho_p,r F_r(phi_n), F_r = sum_k V_rk rho_n,k over the table
// of the proton-neutron energy: the table is read NFOM times, not NFOM^2 (the pair above with H/N
// of every gauge point: FP64 6.1 ms, double-float 4.1 ms).
// Both are compile-time choices: as arguments of one function they cost the plain form 4 to 7 %
// (spills; pf double-float 8.43 -> 8.84 ms, norm pass 1.46 -> 1.56 ms).
template <class Z, bool Solve, bool Gauge>
__device__ __noinline__ void split_items(const Params &p, const double *__restrict__ pr, zc *slot, int pair,
                                         const int2 *__restrict__ items, int ie0, int m, bool reload,
                                         double *__restrict__ zout, int *__restrict__ status,
                                         double *__restrict__ gout, double *__restrict__ r1out,
                                         double *__restrict__ r2out, long long pt0) {
    using Ra = Ar<Z>;
    using R = typename Ra::R;
    extern __shared__ __align__(16) unsigned char smem[];
    const RedPlan &L = Solve ? p.place.sol : p.place.spl;
    const int h = p.h, n = p.n, hh = h * h, ld = L.ld, nf = p.nfom;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ng = L.ng, gthr = 32 * L.w, gid = (int)threadIdx.x / gthr;
    const bool inverse = !p.norm_only;
    int nc = max(1, min(ng / (2 * m), nf));                          // chunks per species
    if (Gauge) nc = min(nc, gauge_chunks(p, Solve));
    const int nu = 2 * m * nc;                                       // units
    const int tcw = 2 * p.tc_nk - p.tc_nph;                          // width of a species row
    unsigned short *rows =
        p.tc_splits ? p.tc_sp + (long long)blockIdx.x * p.place.spl.items * 2 * nf * 6 * tcw : nullptr;
    Z *ephz = reinterpret_cast<Z *>(smem + L.off_eph);
    zc *asum = reinterpret_cast<zc *>(smem + L.off_acc);     // [m][2][nf]: a_s(phi)
    zc *uacc = asum + 2 * L.items * nf;                      // [unit][2]: sum a E_ss, sum a J2_ss
    int *uflag = reinterpret_cast<int *>(uacc + 2 * max(ng, 2 * L.items));
    R *Z0 = reinterpret_cast<R *>(smem + L.off_z0);          // [2][h][h]
    // per unit: weighted density; per item: the species blocks of Y. R* Wi takes the densities' place
    Z *Y = reinterpret_cast<Z *>(slot);                      // [m][2][h h]
    const int I = Gauge ? 1 : L.items;
    zc *Sb = slot + 2LL * I * hh;
    zc *RW = slot + 2LL * I * hh;                            // [m][2][h h]
    // by T22: Y is X = R W R^T; SolveData's matrices follow the densities
    Z *SB = reinterpret_cast<Z *>(Sb + (long long)(Gauge ? nu : max(ng, 2 * I)) * hh), *SP = SB + 4LL * I * hh;
    R *Sc = reinterpret_cast<R *>(SP + 4LL * I * hh);
    // Gauge: [nf] (neutron energy; 1 once it is there), [nf][rows] F
    zc *En = reinterpret_cast<zc *>(SB + (Solve ? 11LL * hh : 0));
    Z *F = reinterpret_cast<Z *>(En + 2 * nf);
    const double *gWi = pr + (Solve ? p.pl.w : p.pl.zi), *gZ0 = pr + p.pl.z0;
    auto euler = [&](int k) { return items ? items[k].y : ie0 + k; };
    if (reload) {
        __syncthreads();
        if (Solve) solve_constants<Z>(p, pr, Sc);
        for (int t = threadIdx.x; t < (Solve ? 0 : 2 * hh); t += blockDim.x) {
            const int b = t / hh, i = (t % hh) / h, j = t % h;
            Z0[t] = Ra::real(gZ0[(b * h + i) * n + b * h + j]);
        }
        const double twopi = 6.283185307179586476925287;
        for (int l = threadIdx.x; l < nf; l += blockDim.x) {
            const zc e = expi(twopi * l / nf);
            ephz[l] = Ra::from(e);
        }
    }
    zc *rot = reinterpret_cast<zc *>(smem + L.off_grp);      // [m][rot_elems], before the groups run
    __syncthreads();
    split_setup<Z, Solve>(p, gWi, items, ie0, m, rot, RW, Y);
    if (Solve && inverse) solve_setup<Z>(p, pr, m, rot, SB, SP);
    double *gp = Gauge ? gout + 4LL * ((long long)pair * p.n_euler + euler(0)) * p.n_gauge : nullptr;
    if (Gauge) {
        for (int l = threadIdx.x; l < nf; l += blockDim.x) En[2 * l + 1] = mk(0.0, 0.0);
        for (int t = threadIdx.x; t < p.n_gauge; t += blockDim.x) gp[4 * t + 2] = gp[4 * t + 3] = 0.0;
    }
    __syncthreads();
    // ---- the problems
    const Grp g{(int)threadIdx.x - gid * gthr, gthr, 1 + gid};
    const bool energies = inverse && !p.tc_splits;
    const bool rounds = energies && Shared<Z>::energies;   // spare warps only join energy_round
    const int step = Gauge ? nc : ng;
    for (int u0 = 0; u0 < nu; u0 += step) {
        if (Gauge) __syncthreads();   // the protons' problems read the neutrons' F
        const int ub = Gauge ? nc - u0 : u0, cnt_u = min(step, nu - u0);   // this round's first unit, units
        const int u = ub + gid;
        const bool mine = gid < cnt_u;
        const int it = mine ? u / (2 * nc) : 0, s = mine ? (u / nc) & 1 : 0, chunk = mine ? u % nc : 0;
        unsigned char *gb = smem + L.off_grp + (mine ? gid : 0) * L.grp_bytes;
        Z *A = reinterpret_cast<Z *>(gb), *Rh = A + h * ld;
        SkewScratch<Z> &w = *reinterpret_cast<SkewScratch<Z> *>(gb + L.off_scr);
        zc *ash = reinterpret_cast<zc *>(gb + L.off_scr + sizeof(SkewScratch<Z>));
        zc *sb = Sb + (long long)u * hh;
        // two-body density: same-species quadruples, sum over phi of a_s times their products
        const int q0 = p.r2_off[s], nq = r2out && mine ? p.r2_off[s + 1] - q0 : 0;
        double *r2acc = nq ? p.r2acc + p.r2_stride * blockIdx.x + 2LL * p.r2_ss * u : nullptr;
        zc aE = mk(0, 0), aJ = mk(0, 0);   // the group's thread 0
        int flags = 0;
        bool first = true;
        for (int l0 = 0; l0 < nf; l0 += nc) {
            const int l = l0 + chunk;
            const bool act = mine && l < nf;
            bool sing = false;
            if (act) {
                const long long is = 2 * it + s;
                if constexpr (Solve) {
                    const SolveData<Z> D{Sc + s * hh, Sc + (2 + s) * hh, Sc + (4 + s) * hh, Y + is * hh, SB + 2 * is * hh,
                                         SP + 2 * is * hh};
                    sing = solve_problem<Z>(g, h, ld, ephz[l], D, A, Rh, reinterpret_cast<Z *>(gb + L.off_y), w, inverse);
                } else {
                    const Z d = ephz[l] * ephz[l];
                    sing = skew_problem<Z>(g, h, ld, h, d, d, d, Y + is * hh, h, Z0 + s * hh, A, Rh, w, inverse, L.tile);
                }
                if (g.tid < 32) {
                    int under;
                    const zc pf = pivot_product<Z>(w.piv, h / 2, p.cscale, under);
                    if (lane == 0) {
                        const int o = s ? l : l * nf;   // e^{-i phi N_s}: the other species' angle is 0
                        const zc a = pf * mk(p.gphase[2 * o], p.gphase[2 * o + 1]);
                        asum[(2 * it + s) * nf + l] = a;
                        ash[0] = a;
                        flags |= (under == 1 ? 1 : (under == 2 ? 4 : 0)) | (inverse && sing ? 2 : 0);
                    }
                }
            }
            if (rounds) {
                __syncthreads();
                for (int sp = 0; sp < 2; ++sp) {   // the groups whose problem of this round is of species sp
                    int list[16], cnt = 0;
                    for (int k = 0; k < cnt_u; ++k)
                        if ((((ub + k) / nc) & 1) == sp && l0 + (ub + k) % nc < nf) list[cnt++] = k;
                    energy_round<Z>(p.tab[kTabProton + sp], p.sched[1], sp, smem, cnt, list, L.off_grp, L.grp_bytes, L.off_scr);
                }
                __syncthreads();
            }
            if (!act || !inverse || sing) continue;   // uniform over the group
            const PointSums<Z> q = point_sums<Z>(g, p, h, ld, s * h, energies ? &p.tab[kTabProton + s] : nullptr, A, Rh,
                                                 w.red);
            if (p.tc_splits) species_rows<Z>(g, p, s, h, ld, A, Rh, rows + ((long long)(2 * it + s) * nf + l) * 6 * tcw);
            if (g.tid == 0) {
                const zc a = ash[0];
                aE = zfma(a, Ra::to(q.e2), aE);
                const zc tp = Ra::to(q.tp), tm = Ra::to(q.tm), tz = Ra::to(q.tz);
                aJ = zfma(a, Ra::to(q.j2) + tp * tm + tz * tz, aJ);
            }
            if constexpr (Gauge) gauge_values<Z>(g, p, h, ld, s, l, Ra::to(q.e2) + Ra::to(q.t1), A, Rh, En, F, gp);
            gsync(g);
            add_weighted<Z>(g, h, ld, ash[0], Rh, sb, first);
            for (int q = g.tid; q < nq; q += g.nthr) {
                const zc x = Ra::to(quad_product<Z>(p.r2s[q0 + q].x, s * h, ld, A, Rh));
                const zc v = first ? ash[0] * x : zfma(ash[0], x, mk(r2acc[2 * q], r2acc[2 * q + 1]));
                r2acc[2 * q] = v.x;
                r2acc[2 * q + 1] = v.y;
            }
            first = false;
            gsync(g);   // the next problem overwrites the densities
        }
        if (first && inverse && mine) {
            for (int t = g.tid; t < hh; t += g.nthr) sb[t] = mk(0.0, 0.0);
            for (int q = g.tid; q < 2 * nq; q += g.nthr) r2acc[q] = 0.0;
        }
        if (g.tid == 0 && mine) {
            uacc[2 * u] = aE;
            uacc[2 * u + 1] = aJ;
            uflag[u] = flags;
        }
    }
    __syncthreads();
    // ---- per Euler point: weighted densities of both species side by side, then the sums
    const double inv = 1.0 / ((double)nf * nf);
    const zc pre = (p.vacfac * pr[p.pl.dets] * pr[p.pl.dets + 1]) * mk(pr[p.pl.pfz], pr[p.pl.pfz + 1]);
    zc *St = reinterpret_cast<zc *>(smem + L.off_grp);                    // [m][2][h h]
    Z *Se = reinterpret_cast<Z *>(St + 2 * hh * m);                       // the same in the point arithmetic
    zc *ob = reinterpret_cast<zc *>(Se + 2 * hh * m);                     // [m][2][kOneBody]
    zc *epn = ob + 2 * kOneBody * m;                                      // [m]
    zc *asm2 = epn + m;                                                   // [m][2] sums of a_s
    zc *part = asm2 + 2 * m;                                              // [warps] proton-neutron energies
    int *sexp = reinterpret_cast<int *>(part + kThreads / 32);            // [m][2] exponents taken from St in Se
    if (inverse) {
        for (int t = threadIdx.x; t < 2 * hh * m; t += blockDim.x) {
            const int is = t / hh, e = t % hh;
            zc v = Sb[(long long)is * nc * hh + e];
            for (int q = 1; q < nc; ++q) v = v + Sb[((long long)is * nc + q) * hh + e];
            St[t] = v;
            if (!Shared<Z>::energies) Se[t] = Ra::from(v);
        }
        __syncthreads();
        if constexpr (Shared<Z>::energies) {
            // The weighted densities carry the Pfaffians as they come, sum_phi Pf(c K_s) rho_s: 1e20 for
            // each species of an sd+pf pair, and c^(h/2) more for another Pfaffian scale c. Two FP32
            // words hold neither that nor the product of the two species, so each density is
            // divided by the power of two of its largest entry, which goes back on the energy in FP64.
            for (int is = wid; is < (energies ? 2 * m : 0); is += kThreads / 32) {
                unsigned x = 0u;
                for (int e = lane; e < hh; e += 32) {
                    const zc v = St[is * hh + e];
                    x = max(x, max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu));
                }
                const int ex = (int)(__reduce_max_sync(0xffffffffu, x) >> 20);
                // all zero: any power will do; Inf or NaN: stays so under the largest
                if (lane == 0) sexp[is] = ex == 0 ? 1023 : min(ex, 2045);
            }
        }
        for (int t = wid; t < 2 * kOneBody * m; t += kThreads / 32) {
            const int is = t / kOneBody, q = t % kOneBody, s = is & 1;
            const bool none = (q == 0 && s) || (q == 1 && !s) || (q >= 7 && (s || !p.iE2));
            const zc v = none ? mk(0, 0) : one_body(p, q, lane, s * h, h, St + (long long)is * hh, h);
            if (lane == 0) ob[t] = v;
        }
        if constexpr (Shared<Z>::energies) {
            __syncthreads();
            for (int t = threadIdx.x; t < (energies ? 2 * hh * m : 0); t += blockDim.x)
                Se[t] = Ra::from(__hiloint2double((2046 - sexp[t / hh]) << 20, 0) * St[t]);
            __syncthreads();
        }
        // the proton-neutron energy, bilinear in the two weighted densities
        const int wpi = max(1, (kThreads / 32) / m);
        if (wid / wpi < m) {
            using O = Op<Z>;
            typename O::Acc e2 = O::acc(szero<Z>());
            if (!p.tc_splits)
                energy_slices<Z>(p.tab[kTabMixed], wid % wpi, wpi, lane, Se + (long long)(wid / wpi) * 2 * hh, e2);
            const Z v = warp_sum_z(O::done(e2));
            if (lane == 0) part[wid] = Ra::to(v);
        }
        __syncthreads();
        if (threadIdx.x < m) {
            zc v = mk(0, 0);
            for (int q = 0; q < wpi; ++q) v = v + part[threadIdx.x * wpi + q];
            if (rounds) {
                const int ex = sexp[2 * threadIdx.x] + sexp[2 * threadIdx.x + 1] - 2046;
                v = mk(scalbn(v.x, ex), scalbn(v.y, ex));
            }
            epn[threadIdx.x] = v;
        }
    }
    if (threadIdx.x >= 64 && threadIdx.x - 64 < 2 * m) {
        const int is = threadIdx.x - 64;
        zc v = mk(0, 0);
        for (int l = 0; l < nf; ++l) v = v + asum[is * nf + l];
        asm2[is] = v;
    }
    __syncthreads();
    if (p.tc_splits) {
        join_rows(p, m, rows, pt0);
        for (int t = threadIdx.x; t < m * p.n_gauge; t += blockDim.x) {   // w = N / NFOM^2
            const int it = t / p.n_gauge, gi = t % p.n_gauge;
            const zc v = inv * (pre * (asum[2 * it * nf + gi / nf] * asum[(2 * it + 1) * nf + gi % nf]));
            p.tc_w[2 * (pt0 + t)] = v.x;
            p.tc_w[2 * (pt0 + t) + 1] = v.y;
        }
    }
    if (r2out) {   // Euler weight x gauge mean over the batch, added into the pair's sums
        double *o = r2out + 2LL * p.n_r2q * pair;
        const long long us = 2LL * p.r2_ss;
        const double *acc = p.r2acc + p.r2_stride * blockIdx.x;
        for (int t = threadIdx.x; t < p.n_r2q; t += blockDim.x) {
            const int s = t < p.r2_off[1] ? 0 : (t < p.r2_off[2] ? 1 : 2);
            const uint2 qd = p.r2s[t];
            zc v = mk(0, 0);
            for (int it = 0; it < m; ++it) {
                const double wgt = inv * p.euler[4 * euler(it) + 3];
                zc x = mk(0, 0);
                if (s < 2) {
                    for (int q = 0; q < nc; ++q) {
                        const double *a = acc + us * ((2 * it + s) * nc + q) + 2 * (t - p.r2_off[s]);
                        x = x + mk(a[0], a[1]);
                    }
                    x = asm2[2 * it + 1 - s] * x;
                } else {   // one proton and one neutron density, rho_ki rho_lj
                    const int i = qd.x & 0xff, j = (qd.x >> 8) & 0xff, k = (qd.x >> 16) & 0xff, l = qd.x >> 24;
                    const int si = i >= h ? 1 : 0, sj = 1 - si;
                    const zc *Sa = St + (long long)(2 * it + si) * hh, *Sc = St + (long long)(2 * it + sj) * hh;
                    x = Sa[(k - si * h) * h + i - si * h] * Sc[(l - sj * h) * h + j - sj * h];
                }
                v = v + wgt * x;
            }
            v = pre * v;
            atomicAdd(o + 2 * qd.y, v.x);
            atomicAdd(o + 2 * qd.y + 1, v.y);
        }
    }
    for (int it = wid; it < m; it += kThreads / 32) {
        const int ie = euler(it);
        const zc ap = asm2[2 * it], an = asm2[2 * it + 1];
        zc v = mk(0, 0);
        int f = 0;
        if (lane < 2 * nc) f = uflag[2 * it * nc + lane];
        for (int k = 32 + lane; k < 2 * nc; k += 32) f |= uflag[2 * it * nc + k];
        f = (int)__reduce_or_sync(0xffffffffu, (unsigned)f);
        if (lane == 0) v = pre * (ap * an);
        if (inverse && lane > 0 && lane < 18) {
            const zc *op = ob + 2 * it * kOneBody, *on = op + kOneBody;
            if (lane == 1) v = an * op[0];
            else if (lane == 2) v = ap * on[1];
            else if (lane == 3) v = an * op[2] + ap * on[2];
            else if (lane == 6 || lane == 7) {
                zc sp = mk(0, 0), sn = mk(0, 0);
                for (int q = 0; q < nc; ++q) {
                    sp = sp + uacc[2 * (2 * it * nc + q) + lane - 6];
                    sn = sn + uacc[2 * ((2 * it + 1) * nc + q) + lane - 6];
                }
                if (lane == 6) {   // two-body + one-body energy + e0 N
                    v = an * (sp + op[2]) + ap * (sn + on[2]) + epn[it] + p.e0 * (ap * an);
                } else {
                    v = an * (sp + op[3]) + ap * (sn + on[3]) + op[4] * on[5] + on[4] * op[5] +
                        2.0 * (op[6] * on[6]);
                }
            } else if (lane >= 8) v = an * op[lane - 1];
            v = pre * v;
        }
        v = inv * v;
        const unsigned bad = __ballot_sync(0xffffffffu, !zfinite(v));
        if (lane < kNobs) {
            zout[2LL * (lane * p.n_euler + ie)] = v.x;
            zout[2LL * (lane * p.n_euler + ie) + 1] = v.y;
        }
        if (lane == 0) status[(long long)pair * p.n_euler + ie] = f | (bad ? 4 : 0);
        if (r1out) {
            for (int b = 0; b < p.obs.n_r1b; ++b) {
                zc s = mk(0, 0);
                int sp = 0;
                for (int e = p.obs.r1b_off[b] + lane; e < p.obs.r1b_off[b + 1]; e += 32) {
                    const int ix = p.obs.r1b_idx[e], r = ix >> 8, c = ix & 255;
                    sp = r >= h ? 1 : 0;
                    s = rfma(p.obs.r1b_val[e], St[(long long)(2 * it + sp) * hh + (r - sp * h) * h + c - sp * h], s);
                }
                s.x = warp_sum(s.x);
                s.y = warp_sum(s.y);
                if (lane == 0) {   // a block is one species: lane 0 holds its first entry
                    const zc o = inv * (pre * ((sp ? ap : an) * s));
                    r1out[2LL * (((long long)pair * p.obs.n_r1b + b) * p.n_euler + ie)] = o.x;
                    r1out[2LL * (((long long)pair * p.obs.n_r1b + b) * p.n_euler + ie) + 1] = o.y;
                }
            }
        }
        if (gout)   // N at every gauge point
            for (int gi = lane; gi < p.n_gauge; gi += 32) {
                const zc w = pre * (asum[2 * it * nf + gi / nf] * asum[(2 * it + 1) * nf + gi % nf]);
                double *o = gout + 4LL * (((long long)pair * p.n_euler + ie) * p.n_gauge + gi);
                o[0] = w.x;
                o[1] = w.y;
                if (!Gauge) o[2] = o[3] = 0.0;
            }
    }
    __syncthreads();
}

}  // namespace pnamp

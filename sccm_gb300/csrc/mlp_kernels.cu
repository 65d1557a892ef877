// Hand-written FP32 kernels of the learned mode's network: dense layers
// (forward with fused bias + tanh, backward with deterministic split-K weight
// gradients), the heteroscedastic Gaussian loss and the Adam update.
//
// The network predicts the normalised energy kernel H/N at fine-mesh points
// from cheap inputs; it has no counterpart in the reference, which evaluates
// every mesh point exactly. All layers are small (width 256) and the batch is
// large (10^4 - 10^6 rows), so a register-tiled SIMT GEMM on the FP32 pipes is
// used for every product; the weight gradient (K = rows) is split over row
// chunks into a workspace and summed in chunk order, so results do not depend
// on scheduling.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pnamp_mlp.h"
#include "pnamp_df64.cuh"

namespace {
using pnamp::f2;
using pnamp::f2_dup;
using pnamp::f2_fma;

// 128 x 64 tile, 128 threads of 8 x 8 outputs each, K in double-buffered steps of 16. Every output
// is one chain of FP32 fused multiply-adds over K, two neighbouring columns per packed
// instruction: 64 lane operations for 4 shared-memory loads per thread and k (the 64 x 64 tile of
// 4 x 4 outputs before it was bound by its loads, 8 for 16), and the next step's tile is on its
// way from memory meanwhile. Smaller than 128 x 128, so that 16384 x 256 outputs give 512 tiles
// for 152 SMs. A training step of 16384 rows, width 256, depth 4, all
// kernels of this file: 1175 us with the 64 x 64 tile, 815 us.
constexpr int BM = 128, BN = 64, BK = 16, TH = 128;
constexpr int LDA = BM + 4, LDB = BN + 4;

// One BR x BK tile of an operand into registers and from there to shared memory as [k][r].
// KC: contiguous along k (P[r * ld + k]), else along r (P[k * ld + r]); vec: 16-byte loads
// (leading dimension and base multiples of 4 floats).
template <int BR, bool KC>
struct Stage {
    static constexpr int Q = BR * BK / 4 / TH;   // float4 per thread
    float4 v[Q];
    __device__ __forceinline__ void load(const float *__restrict__ P, int ld, int r0, int R, int k0, int k1, bool vec) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int e = threadIdx.x + q * TH;
            const int r = r0 + (KC ? e / (BK / 4) : 4 * (e % (BR / 4)));
            const int k = k0 + (KC ? 4 * (e % (BK / 4)) : e / (BR / 4));
            float x[4] = {0.f, 0.f, 0.f, 0.f};
            if (vec && (KC ? (r < R && k + 3 < k1) : (k < k1 && r + 3 < R))) {
                const float4 t = *reinterpret_cast<const float4 *>(KC ? P + (long long)r * ld + k : P + (long long)k * ld + r);
                x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int rr = KC ? r : r + i, kk = KC ? k + i : k;
                    if (rr < R && kk < k1) x[i] = KC ? P[(long long)rr * ld + kk] : P[(long long)kk * ld + rr];
                }
            }
            v[q] = make_float4(x[0], x[1], x[2], x[3]);
        }
    }
    __device__ __forceinline__ void store(float *S, int lds) const {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int e = threadIdx.x + q * TH;
            if (KC) {
                const int r = e / (BK / 4), k = 4 * (e % (BK / 4));
                S[k * lds + r] = v[q].x;
                S[(k + 1) * lds + r] = v[q].y;
                S[(k + 2) * lds + r] = v[q].z;
                S[(k + 3) * lds + r] = v[q].w;
            } else {
                *reinterpret_cast<float4 *>(S + (e / (BR / 4)) * lds + 4 * (e % (BR / 4))) = v[q];
            }
        }
    }
};

// C[m][n] = sum_k A(m, k) B(k, n) over k in [k0, k1) of this split
//   A(m, k) = TA ? A[k * lda + m] : A[m * lda + k]
//   B(k, n) = TB ? B[n * ldb + k] : B[k * ldb + n]
// Epilogue: + bias[n] (if bias), tanh (if act == 1). Split z writes C + z * c_split_stride.
template <bool TA, bool TB>
__global__ void __launch_bounds__(TH, 4) gemm_kernel(const float *__restrict__ A, int lda, const float *__restrict__ B,
                                                  int ldb, float *__restrict__ C, int ldc, int M, int N, int K,
                                                  int kchunk, long long c_split_stride, const float *__restrict__ bias,
                                                  int act, int veca, int vecb) {
    __shared__ __align__(16) float As[2][BK * LDA];
    __shared__ __align__(16) float Bs[2][BK * LDB];
    const int tx = threadIdx.x % 8, ty = threadIdx.x / 8;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int k0 = blockIdx.z * kchunk, k1 = min(K, k0 + kchunk);
    f2 acc[8][4];   // rows 4 ty + i, 64 + 4 ty + i; columns 4 tx + 2 j, 32 + 4 tx + 2 j
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = f2_dup(0.f);
    Stage<BM, !TA> sa;
    Stage<BN, TB> sb;
    sa.load(A, lda, m0, M, k0, k1, veca);
    sb.load(B, ldb, n0, N, k0, k1, vecb);
    sa.store(As[0], LDA);
    sb.store(Bs[0], LDB);
    __syncthreads();
    int cur = 0;
    for (int kt = k0; kt < k1; kt += BK, cur ^= 1) {
        const bool more = kt + BK < k1;
        if (more) {
            sa.load(A, lda, m0, M, kt + BK, k1, veca);
            sb.load(B, ldb, n0, N, kt + BK, k1, vecb);
        }
        const float *Ac = As[cur], *Bc = Bs[cur];
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 a0 = *reinterpret_cast<const float4 *>(Ac + kk * LDA + 4 * ty);
            const float4 a1 = *reinterpret_cast<const float4 *>(Ac + kk * LDA + 64 + 4 * ty);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(Bc + kk * LDB + 4 * tx);
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2 *>(Bc + kk * LDB + 32 + 4 * tx);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const f2 bv[4] = {{b0.x}, {b0.y}, {b1.x}, {b1.y}};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const f2 ad = f2_dup(av[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = f2_fma(ad, bv[j], acc[i][j]);
            }
        }
        if (more) {   // the other buffer was last read before the previous barrier
            sa.store(As[cur ^ 1], LDA);
            sb.store(Bs[cur ^ 1], LDB);
        }
        __syncthreads();
    }
    float *Cs = C + blockIdx.z * c_split_stride;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gm = m0 + (i < 4 ? 4 * ty + i : 60 + 4 * ty + i);
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int gn = n0 + (j < 4 ? 4 * tx + j : 28 + 4 * tx + j);
            if (gn >= N) continue;
            float v = j & 1 ? pnamp::f2_b(acc[i][j >> 1]) : pnamp::f2_a(acc[i][j >> 1]);
            if (bias) v += bias[gn];
            if (act == 1) v = tanhf(v);
            Cs[(long long)gm * ldc + gn] = v;
        }
    }
}

int vec_ok(const float *p, int ld) { return ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// out[i] = sum_s part[s * n + i], s in order
__global__ void sum_splits(const float *__restrict__ part, int splits, long long n, float *__restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float s = 0.f;
        for (int k = 0; k < splits; ++k) s += part[k * n + i];
        out[i] = s;
    }
}

// dZ = dY * (1 - Y^2) (tanh; y null: dZ = dY) in place, and its column sums over row chunks,
// part[s][o]: one pass over dY for both. 64 columns x 8 row groups per block, so that a chunk's
// rows are not one serial chain.
constexpr int kColLanes = 64, kRowLanes = 8;
__global__ void __launch_bounds__(kColLanes * kRowLanes)
grad_colsum(float *__restrict__ dy, const float *__restrict__ y, int rows, int out, int chunk,
            float *__restrict__ part) {
    __shared__ float red[kRowLanes][kColLanes];
    const int s = blockIdx.x, c = threadIdx.x % kColLanes, g = threadIdx.x / kColLanes;
    const int o = blockIdx.y * kColLanes + c;
    const int r1 = min(rows, (s + 1) * chunk);
    float acc = 0.f;
    for (int r = s * chunk + g; r < r1 && o < out; r += 8 * kRowLanes) {
        float d[8], v[8];   // 16 loads in flight before the first store
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const long long i = (long long)(r + k * kRowLanes) * out + o;
            d[k] = r + k * kRowLanes < r1 ? dy[i] : 0.f;
            v[k] = y && r + k * kRowLanes < r1 ? y[i] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (y && r + k * kRowLanes < r1) {
                d[k] *= 1.f - v[k] * v[k];
                dy[(long long)(r + k * kRowLanes) * out + o] = d[k];
            }
            acc += d[k];
        }
    }
    red[g][c] = acc;
    __syncthreads();
    if (g == 0 && o < out) {
        for (int k = 1; k < kRowLanes; ++k) acc += red[k][c];
        part[(long long)s * out + o] = acc;
    }
}

// mode 0: loss_r = w_r [ |y - mu|^2 e^{-2s} / 2 + 2 s ],  s = clamp(out[2], -12, 6)
//         dout = w_r / rows * [ -(y - mu) e^{-2s},  -|y - mu|^2 e^{-2s} + 2 ]
// mode 1: the same with s = 0 and no gradient to s (weighted least squares on mu)
// mode 2: the same with no gradient to mu (fits s to the current errors)
__global__ void gauss_loss(const float *__restrict__ out, const float *__restrict__ y, const float *__restrict__ w,
                           int rows, int mode, float *__restrict__ dout, float *__restrict__ loss_part) {
    __shared__ float red[256];
    float acc = 0.f;
    const float inv_rows = 1.f / (float)rows;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const float mr = out[3 * r], mi = out[3 * r + 1], s_raw = out[3 * r + 2];
        const float s = mode == 1 ? 0.f : fminf(fmaxf(s_raw, -12.f), 6.f);
        const float er = y[2 * r] - mr, ei = y[2 * r + 1] - mi;
        const float iv = expf(-2.f * s);
        const float e2 = er * er + ei * ei;
        const float wr = w ? w[r] : 1.f;
        acc += wr * (0.5f * e2 * iv + 2.f * s);
        const float g = wr * inv_rows;
        dout[3 * r] = mode == 2 ? 0.f : -g * er * iv;
        dout[3 * r + 1] = mode == 2 ? 0.f : -g * ei * iv;
        dout[3 * r + 2] = (mode != 1 && s_raw > -12.f && s_raw < 6.f) ? g * (2.f - e2 * iv) : 0.f;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss_part[blockIdx.x] = red[0] * inv_rows;
}

__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, long long n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    }
}

int grid_1d(long long n) { return (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096); }

constexpr int kSplitRows = 512;  // rows per weight-gradient chunk
constexpr int kMaxSplits = 128;

}  // namespace

extern "C" {

long long pnamp_mlp_work_floats(int rows, int in, int out) {
    const int splits = rows <= 0 ? 1 : (rows + kSplitRows - 1) / kSplitRows;
    const int s = splits < kMaxSplits ? splits : kMaxSplits;
    return (long long)s * in * out + (long long)s * out;
}

int pnamp_mlp_linear_forward(const float *X, const float *W, const float *b, float *Y, int rows, int in, int out,
                             int act, void *stream) {
    if (!X || !W || !Y || rows < 0 || in < 1 || out < 1 || (act != 0 && act != 1)) return 1;
    if (rows == 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    dim3 grid((out + BN - 1) / BN, (rows + BM - 1) / BM, 1);
    gemm_kernel<false, true><<<grid, TH, 0, st>>>(X, in, W, in, Y, out, rows, out, in, in, 0, b, act, vec_ok(X, in),
                                                  vec_ok(W, in));
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pnamp_mlp_linear_backward(const float *X, const float *W, const float *Y, float *dY, float *dW, float *db,
                              float *dX, int rows, int in, int out, int act, float *work, void *stream) {
    if (!X || !W || !dY || !dW || !db || !work || rows < 1 || in < 1 || out < 1 || (act != 0 && act != 1) ||
        (act == 1 && !Y))
        return 1;
    cudaStream_t st = (cudaStream_t)stream;
    // split-K over row chunks: chunk a multiple of BK, at most kMaxSplits chunks
    int splits = (rows + kSplitRows - 1) / kSplitRows;
    if (splits > kMaxSplits) splits = kMaxSplits;
    int chunk = (rows + splits - 1) / splits;
    chunk = (chunk + BK - 1) / BK * BK;
    splits = (rows + chunk - 1) / chunk;
    float *partW = work, *partB = work + (long long)splits * in * out;
    grad_colsum<<<dim3(splits, (out + kColLanes - 1) / kColLanes), kColLanes * kRowLanes, 0, st>>>(dY, act == 1 ? Y : nullptr, rows, out, chunk, partB);
    // dW[o][i] = sum_r dZ[r][o] X[r][i]: A = dZ^T (TA, lda = out), B = X (ldb = in)
    dim3 gw((in + BN - 1) / BN, (out + BM - 1) / BM, splits);
    gemm_kernel<true, false><<<gw, TH, 0, st>>>(dY, out, X, in, partW, in, out, in, rows, chunk,
                                                (long long)out * in, nullptr, 0, vec_ok(dY, out), vec_ok(X, in));
    sum_splits<<<grid_1d((long long)out * in), 256, 0, st>>>(partW, splits, (long long)out * in, dW);
    sum_splits<<<grid_1d(out), 256, 0, st>>>(partB, splits, out, db);
    if (dX) {  // dX[r][i] = sum_o dZ[r][o] W[o][i]
        dim3 gx((in + BN - 1) / BN, (rows + BM - 1) / BM, 1);
        gemm_kernel<false, false><<<gx, TH, 0, st>>>(dY, out, W, in, dX, in, rows, in, out, out, 0, nullptr, 0,
                                                     vec_ok(dY, out), vec_ok(W, in));
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pnamp_mlp_loss_blocks(int rows) { return rows < 1 ? 1 : (grid_1d(rows) < 1024 ? grid_1d(rows) : 1024); }

int pnamp_mlp_gauss_loss(const float *out, const float *y, const float *w, int rows, int mode, float *dout,
                         float *loss_part, void *stream) {
    if (!out || !y || !dout || !loss_part || rows < 1 || mode < 0 || mode > 2) return 1;
    gauss_loss<<<pnamp_mlp_loss_blocks(rows), 256, 0, (cudaStream_t)stream>>>(out, y, w, rows, mode, dout,
                                                                             loss_part);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pnamp_mlp_adam(float *p, const float *g, float *m, float *v, long long n, float lr, float beta1, float beta2,
                   float eps, int step, void *stream) {
    if (!p || !g || !m || !v || n < 0 || step < 1) return 1;
    if (n == 0) return 0;
    const float c1 = 1.f / (1.f - powf(beta1, (float)step)), c2 = 1.f / (1.f - powf(beta2, (float)step));
    adam_kernel<<<grid_1d(n), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, lr, beta1, beta2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // extern "C"

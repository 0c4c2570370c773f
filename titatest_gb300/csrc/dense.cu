// Dense FP64 kernels for the model uncertainty and resolution of
// src/bmcm_mod.f90 (bata, bmcm, bres, bmcm2): a tiled matrix product, and the
// blocked Cholesky factor, triangular inverse and inverse product that
// replace DPOTRF / DPOTRI.  All matrices are column-major with leading
// dimension ld; blocks of the factorisation are kNB = 64 wide.
//
// On GB300 these run on the FP64 pipe (a small fraction of the FP32 rate):
// each thread of a 256-thread block accumulates its entries of an output tile
// in registers from 16-deep slices of the operands staged in shared memory,
// which is far more data reuse than the FP64 pipe needs.
#include <algorithm>
#include <mutex>

#include "kernels.h"

namespace crgpu {

namespace {

constexpr int kNB = 64;   // block size of the tiles and of the blocked factorisations
constexpr int kBK = 16;   // depth of a staged operand slice
constexpr int kGT = 256;  // threads of a product block

// Operand access: element (row i of the product, depth k).  kmaj: the depth
// index is contiguous (A^T of a column-major matrix, stored A(k, i) at
// i*ld + k); otherwise the row index is (A(i, k) at k*ld + i).
template <bool KMAJ>
__device__ __forceinline__ double opnd(const double *__restrict__ A, int ld, int i, int k) {
    return KMAJ ? A[(size_t)i * ld + k] : A[(size_t)k * ld + i];
}

// C(i, j) = alpha * sum_k A(i, k) B(j, k) + beta * C(i, j) for the TS x TS
// output tile (blockIdx.x, blockIdx.y) of an M x N product, depth K.
// lower: only blocks on or below the diagonal.  depth: kDepthLower starts at
// the block's first index (operands lower triangular in k, as Y^T Y with Y
// lower), kDepthFromCol at the block column's (B(j, k) is 0 for k < j),
// kDepthToCol ends with it (0 for k > j).  sq: instead of storing C, store the
// sums over each tile's rows of the squared entries and of the entries times
// D(i, j) (leading dimension ldc), sq[(2 bi) * N + j] and sq[(2 bi + 1) * N + j] (the diagonals of G^T G
// and G^T D).
enum { kDepthAll = 0, kDepthLower, kDepthFromCol, kDepthToCol };

template <bool AK, bool BK, int TS>
__global__ __launch_bounds__(kGT) void k_gemm(int M, int N, int K, double alpha, const double *__restrict__ A, int lda,
                                              const double *__restrict__ B, int ldb, double beta, double *C, int ldc,
                                              int lower, int depth, const double *__restrict__ D, double *sq) {
    // the deepest block columns first
    const int bi = blockIdx.x, bj = depth == kDepthToCol ? gridDim.y - 1 - blockIdx.y : blockIdx.y;
    if (lower && bi < bj) return;
    constexpr int R = TS / 16;  // a thread's R x R entries
    __shared__ double As[kBK][TS + 1], Bs[kBK][TS + 1];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int i0 = bi * TS, j0 = bj * TS;
    double acc[R][R];
#pragma unroll
    for (int a = 0; a < R; a++)
#pragma unroll
        for (int b = 0; b < R; b++) acc[a][b] = 0.0;
    const int kbeg = depth == kDepthLower ? max(i0, j0) : depth == kDepthFromCol ? j0 : 0;
    if (depth == kDepthToCol) K = min(K, j0 + TS);
    for (int k0 = kbeg; k0 < K; k0 += kBK) {
        // stage the TS x 16 slices, R values of each operand a thread
#pragma unroll
        for (int q = 0; q < R; q++) {
            const int e = tid + q * kGT;
            // depth-contiguous operands load along k, the others along the row index
            const int r = AK ? e >> 4 : e % TS, kk = AK ? e & 15 : e / TS;
            const int gi = i0 + r, gk = k0 + kk;
            As[kk][r] = (gi < M && gk < K) ? opnd<AK>(A, lda, gi, gk) : 0.0;
            const int r2 = BK ? e >> 4 : e % TS, kk2 = BK ? e & 15 : e / TS;
            const int gj = j0 + r2, gk2 = k0 + kk2;
            Bs[kk2][r2] = (gj < N && gk2 < K) ? opnd<BK>(B, ldb, gj, gk2) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kBK; kk++) {
            double av[R], bv[R];
#pragma unroll
            for (int a = 0; a < R; a++) av[a] = As[kk][ty + 16 * a];
#pragma unroll
            for (int b = 0; b < R; b++) bv[b] = Bs[kk][tx + 16 * b];
#pragma unroll
            for (int a = 0; a < R; a++)
#pragma unroll
                for (int b = 0; b < R; b++) acc[a][b] = fma(av[a], bv[b], acc[a][b]);
        }
        __syncthreads();
    }
    if (sq) {  // column sums of this row block, in a fixed order
        __shared__ double red[2][16][TS];
#pragma unroll
        for (int b = 0; b < R; b++) {
            const int j = j0 + tx + 16 * b;
            double s = 0.0, t = 0.0;
#pragma unroll
            for (int a = 0; a < R; a++) {
                const int i = i0 + ty + 16 * a;
                if (i >= M) continue;
                s = fma(acc[a][b], acc[a][b], s);
                if (D && j < N) t = fma(acc[a][b], D[(size_t)j * ldc + i], t);
            }
            red[0][ty][tx + 16 * b] = s;
            red[1][ty][tx + 16 * b] = t;
        }
        __syncthreads();
        if (tid < 2 * TS && j0 + tid % TS < N) {
            const int w = tid / TS, c = tid % TS;
            double s = 0.0;
            for (int q = 0; q < 16; q++) s += red[w][q][c];
            sq[(size_t)(2 * bi + w) * N + j0 + c] = s;
        }
        return;
    }
#pragma unroll
    for (int a = 0; a < R; a++) {
        const int i = i0 + ty + 16 * a;
        if (i >= M) continue;
#pragma unroll
        for (int b = 0; b < R; b++) {
            const int j = j0 + tx + 16 * b;
            if (j >= N || (lower && i < j)) continue;
            double *c = C + (size_t)j * ldc + i;
            *c = alpha * acc[a][b] + (beta == 0.0 ? 0.0 : beta * *c);
        }
    }
}

// 1/sqrt(v) for a pivot without FP64 division and root (each costs its warp tens
// of FP64 instructions of 16 cycles): an FP32 estimate and two Newton steps
__device__ __forceinline__ double rsqrt_newton(double v) {
    if (!(v > 1e-30 && v < 1e30)) return 1.0 / sqrt(v);
    double y = (double)rsqrtf((float)v);
#pragma unroll
    for (int it = 0; it < 2; it++) y = y * (1.5 - 0.5 * v * y * y);
    return y;
}

// Cholesky factor of the diagonal block at (c0, c0), nb x nb (nb <= 64), and its
// inverse, one block: L into A, L^-1 (zero above the diagonal) into Y at the
// same place.  Two halves of 32: each is factored and inverted together, lane =
// row, warp w the columns w, w + 8, ..., one barrier a column; the coupling
// block, the second half's update and the inverse's lower left block are
// products.  info: first column (1-based) whose pivot is not positive.  Bound
// by the pivot chain and this one SM's FP64 pipe (108 us column by column with
// three barriers, without the inverse).
__global__ __launch_bounds__(256) void k_potf2_inv(int n, double *A, double *Y, int lda, int c0, int *info) {
    constexpr int H = 32;
    extern __shared__ double dsm[];
    double(*S)[kNB + 1] = reinterpret_cast<double(*)[kNB + 1]>(dsm);
    double(*V)[kNB + 1] = S + kNB;
    __shared__ double col[2][H], inv[2];
    const int nb = min(kNB, n - c0), tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int e = tid; e < kNB * kNB; e += 256) {
        const int r = e % kNB, c = e / kNB;
        S[r][c] = r < nb && c <= r ? A[(size_t)(c0 + c) * lda + c0 + r] : (r == c ? 1.0 : 0.0);
        V[r][c] = 0.0;
    }
    __syncthreads();
    for (int o = 0; o < kNB; o += H) {
        double a[4], x[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            a[q] = S[o + lane][o + 8 * q + wid];
            x[q] = lane == 8 * q + wid ? 1.0 : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int w = 0; w < 8; w++) {
                const int p = 8 * q + w, b = p & 1;
                if (wid == w) {
                    double d = __shfl_sync(0xffffffffu, a[q], p);
                    if (!(d > 0.0)) {
                        if (lane == 0 && o + p < nb && *info == 0) *info = c0 + o + p + 1;
                        d = 1.0;
                    }
                    const double iv = rsqrt_newton(d);
                    a[q] = lane > p ? a[q] * iv : lane == p ? d * iv : 0.0;
                    col[b][lane] = lane > p ? a[q] : 0.0;
                    if (lane == 0) inv[b] = iv;
                }
                __syncthreads();
                const double l = col[b][lane], iv = inv[b];
#pragma unroll
                for (int z = 0; z < 4; z++) {
                    const int c = 8 * z + wid;
                    if (z >= q && c > p) a[z] = fma(-l, col[b][c], a[z]);
                    if (z <= q) {
                        const double xp = __shfl_sync(0xffffffffu, x[z], p) * iv;
                        x[z] = lane == p ? xp : fma(-l, xp, x[z]);  // l is 0 above the pivot
                    }
                }
            }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = 8 * q + wid;
            S[o + lane][o + c] = a[q];
            V[o + lane][o + c] = lane >= c ? x[q] : 0.0;
        }
        __syncthreads();
        if (o) break;
        // L21 = A21 L11^-T, then A22 -= L21 L21^T: lane = row, four columns a warp
        double t[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = 8 * q + wid;
            t[q] = 0.0;
            for (int p = 0; p <= c; p++) t[q] = fma(S[H + lane][p], V[c][p], t[q]);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) S[H + lane][8 * q + wid] = t[q];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = 8 * q + wid;
            double s = S[H + lane][H + c];
            for (int p = 0; p < H; p++) s = fma(-S[H + lane][p], S[H + c][p], s);
            S[H + lane][H + c] = s;
        }
        __syncthreads();
    }
    // V21 = -V22 (L21 V11)
    double t[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = 8 * q + wid;
        t[q] = 0.0;
        for (int p = c; p < H; p++) t[q] = fma(S[H + lane][p], V[p][c], t[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) V[lane][H + 8 * q + wid] = t[q];  // the upper right block, not part of the result
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = 8 * q + wid;
        double s = 0.0;
        for (int p = 0; p < H; p++) s = fma(-V[H + lane][H + p], V[p][H + c], s);
        V[H + lane][c] = s;
    }
    __syncthreads();
    for (int e = tid; e < kNB * kNB; e += 256) {
        const int r = e % kNB, c = e / kNB;
        if (r >= nb || c >= nb) continue;
        const size_t at = (size_t)(c0 + c) * lda + c0 + r;
        if (r >= c) A[at] = S[r][c];
        Y[at] = r >= c ? V[r][c] : 0.0;
    }
}

// X = T L11^-T or X = -L11^-1 T with the inverse block Yd (64 x 64, column
// stride ldy, zero above the diagonal): the panel below a diagonal block
// (ROWS: 16 rows r of T(r, .) a block, X(r, c) = sum_{p <= c} T(r, p) Yd(c, p))
// or block row i of the triangular inverse (16 columns a block, X(c, r) =
// -sum_{p <= c} Yd(c, p) T(p, r)).  T is overwritten.  16 at a time because 64
// leave most SMs idle, each bound by its FP64 pipe.
template <bool PANEL>
__global__ __launch_bounds__(256) void k_times_inverse(int nb, const double *__restrict__ Yd, int ldy, double *T,
                                                       int ldt, int len) {
    __shared__ double Yi[kNB][kNB + 1], X[kNB][17];
    const int tid = threadIdx.x, r0 = blockIdx.x * 16, nr = min(16, len - r0);
    for (int e = tid; e < kNB * kNB; e += 256) {
        const int c = e % kNB, p = e / kNB;
        Yi[p][c] = c < nb && p <= c ? Yd[(size_t)p * ldy + c] : 0.0;
    }
    for (int e = tid; e < kNB * 16; e += 256) {
        const int r = PANEL ? e % 16 : e / kNB, p = PANEL ? e / 16 : e % kNB;
        const size_t at = PANEL ? (size_t)p * ldt + r0 + r : (size_t)(r0 + r) * ldt + p;
        X[p][r] = r < nr && p < nb ? T[at] : 0.0;
    }
    __syncthreads();
    // each warp one column c at a time for two halves of 16: warp w takes c = w, w + 8, ...
    const int r = tid & 15, h = tid >> 4;
    double out[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = h + 16 * q;
        double s = 0.0;
        for (int p = 0; p <= c; p++) s = fma(X[p][r], Yi[p][c], s);
        out[q] = s;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = h + 16 * q;
        if (r >= nr || c >= nb) continue;
        if (PANEL) T[(size_t)c * ldt + r0 + r] = out[q];
        else T[(size_t)(r0 + r) * ldt + c] = -out[q];
    }
}

// d_j = sum_i M(i, j)^2 over the rows i >= j of a lower triangular n x n matrix
__global__ __launch_bounds__(256) void k_lower_col_sq(int n, const double *__restrict__ M, double *__restrict__ d) {
    const int j = blockIdx.x;
    double s = 0.0;
    for (int i = j + threadIdx.x; i < n; i += 256) {
        const double v = M[(size_t)j * n + i];
        s = fma(v, v, s);
    }
    __shared__ double red[8];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int q = 0; q < 8; q++) t += red[q];
        d[j] = t;
    }
}

// d2 and dd += the sums over the row blocks of sq (nblk x 2 x n), in block order
__global__ void k_sum_blocks(int nblk, int n, const double *__restrict__ sq, double *__restrict__ d2,
                             double *__restrict__ dd) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double s = d2[j], t = dd[j];
    for (int b = 0; b < nblk; b++) {
        s += sq[(size_t)(2 * b) * n + j];
        t += sq[(size_t)(2 * b + 1) * n + j];
    }
    d2[j] = s;
    dd[j] = t;
}

inline int nblk(int n) { return (n + kNB - 1) / kNB; }

// Tiles of 32: a 64 x 64 tile of depth 64 takes its SM's FP64 pipe 63 us, and the
// factor's updates have few of them (the last round of SMs nearly empty): the
// covariance diagonals of 2400 cells x 600 data 43 -> 32.5 ms.
constexpr int kTS = 32;

inline int ntile(int n) { return (n + kTS - 1) / kTS; }

template <bool AK, bool BK>
void gemm(int M, int N, int K, double alpha, const double *A, int lda, const double *B, int ldb, double beta,
          double *C, int ldc, int lower, int depth, const double *D, double *sq, cudaStream_t st) {
    if (M <= 0 || N <= 0) return;
    dim3 grid(ntile(M), ntile(N));
    k_gemm<AK, BK, kTS><<<grid, kGT, 0, st>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, lower, depth, D, sq);
}

}  // namespace

void dense_syrk_t(int n, int k, const double *S, int lds, double *C, cudaStream_t st) {
    // C (lower) = S^T S, S k x n column-major: both operands depth-contiguous
    gemm<true, true>(n, n, k, 1.0, S, lds, S, lds, 0.0, C, n, 1, kDepthAll, nullptr, nullptr, st);
}

// The factor's chain (a diagonal block on one SM, its panel, the trailing update)
// runs on hi, and a block row of the inverse follows on st as soon as its panel is
// there: the inverse's products fill the chip while a diagonal block (0.11 ms, 13 %
// of the time at n = 2400) or a small trailing update leaves it empty.  Covariance
// diagonals of 2400 cells x 600 data 32.5 -> 29.3 ms.
void dense_potrf_inverse(int n, double *A, double *Y, int *info_dev, cudaStream_t st, cudaStream_t hi, cudaEvent_t ev) {
    constexpr int smem = (int)sizeof(double) * 2 * kNB * (kNB + 1);
    static std::once_flag once;
    std::call_once(once, [] { cudaFuncSetAttribute(k_potf2_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
    const int nb = nblk(n);
    cudaEventRecord(ev, st);
    cudaStreamWaitEvent(hi, ev, 0);
    for (int b = 0; b < nb; b++) {
        const int c0 = b * kNB, w = std::min(kNB, n - c0), r0 = c0 + w, rest = n - r0;
        double *Yd = Y + (size_t)c0 * n + c0, *X = A + (size_t)c0 * n + r0;
        k_potf2_inv<<<1, 256, smem, hi>>>(n, A, Y, n, c0, info_dev);
        if (rest > 0) k_times_inverse<true><<<(rest + 15) / 16, 256, 0, hi>>>(w, Yd, n, X, n, rest);
        cudaEventRecord(ev, hi);
        // trailing update A22 -= X X^T, X = the panel (row-index contiguous)
        if (rest > 0)
            gemm<false, false>(rest, rest, w, -1.0, X, n, X, n, 1.0, A + (size_t)r0 * n + r0, n, 1, kDepthAll, nullptr,
                               nullptr, hi);
        // Y = L^-1 (lower), block row by block row; its diagonal blocks are there.
        // Y_(b, j) = -Y_bb acc_(b, j), j < b
        cudaStreamWaitEvent(st, ev, 0);
        if (b > 0) k_times_inverse<false><<<(c0 + 15) / 16, 256, 0, st>>>(w, Yd, n, Y + c0, n, c0);
        if (rest <= 0) break;
        // acc_(i, j) (+)= L_(i, b) Y_(b, j) for the block rows below, j <= b; block
        // column b begins here
        if (b > 0)
            gemm<false, true>(rest, c0, w, 1.0, X, n, Y + c0, n, 1.0, Y + r0, n, 0, kDepthAll, nullptr, nullptr, st);
        gemm<false, true>(rest, w, w, 1.0, X, n, Yd, n, 0.0, Y + (size_t)c0 * n + r0, n, 0, kDepthAll, nullptr, nullptr,
                          st);
    }
}

void dense_lauum_t(int n, const double *Y, double *C, cudaStream_t st) {
    // C (lower) = Y^T Y with the depth starting at each block row (Y lower)
    gemm<true, true>(n, n, n, 1.0, Y, n, Y, n, 0.0, C, n, 1, kDepthLower, nullptr, nullptr, st);
}

void dense_lower_col_sq(int n, const double *Y, double *d, cudaStream_t st) {
    if (n > 0) k_lower_col_sq<<<n, 256, 0, st>>>(n, Y, d);
}

int dense_product_rows(int m, int n) {
    // whole where T takes 32 MB at most or no more than a matrix of n x n; at least a tile
    const int rows = std::max(n, (4 << 20) / std::max(n, 1));
    return std::min(m, std::max(kTS, rows / kTS * kTS));
}

size_t dense_product_work(int rows, int n) { return (size_t)ntile(rows) * 2 * n; }

void dense_product_sums(int m, int n, const double *S, const double *Y, double *T, double *work, double *d2, double *dd,
                        cudaStream_t st) {
    // By chunks of rows: T = S Y^T: T(l, j) = sum_{p <= j} S(l, p) Y(j, p), then G = T Y: G(l, j) =
    // sum_{p >= j} T(l, p) Y(p, j), kept as per-row-block partial sums in work
    const int rows = dense_product_rows(m, n);
    cudaMemsetAsync(d2, 0, sizeof(double) * n, st);
    cudaMemsetAsync(dd, 0, sizeof(double) * n, st);
    for (int r0 = 0; r0 < m; r0 += rows) {
        const int r = std::min(rows, m - r0);
        gemm<false, false>(r, n, n, 1.0, S + r0, m, Y, n, 0.0, T, r, 0, kDepthToCol, nullptr, nullptr, st);
        gemm<false, true>(r, n, n, 1.0, T, r, Y, n, 0.0, nullptr, m, 0, kDepthFromCol, S + r0, work, st);
        k_sum_blocks<<<(n + 255) / 256, 256, 0, st>>>(ntile(r), n, work, d2, dd);
    }
}

}  // namespace crgpu

// Model update of the Gauss-Newton step: src/update.f90:27-353 with the
// complex preconditioned CG of src/cg_mod.f90:426-726 (cjggra, bap, bp,
// bptri, bb), or in the final phase improvement (lfpi) the real CG of
// src/cg_mod.f90:136-400 (cjggdc, bapdc, bpdc, bpdctri, bbdc) on Re(J) and the
// phases.  The Jacobian is column-major (nanz, manz): column j is
// contiguous, so the column reductions (preconditioner, right-hand side,
// J^H W (J p)) read coalesced columns, and J p is formed from column chunks
// with fixed-order partial sums (deterministic, no atomics).
#include <algorithm>

#include "crgpu_internal.h"
#include "kernels.h"

namespace crgpu {

namespace {

constexpr int kRowTile = 256;   // rows of J per block in J p
constexpr int kColChunk = 64;   // columns of J per block in J p
constexpr int kRedThreads = 256;
constexpr int kRedBlocks = 512;  // most blocks of the vector kernels

// R v (optionally R (w o v)) at cell i: structured 5-point stencil (ltri 0,
// src/cg_mod.f90:547-577 / src/update.f90:63-91) or the neighbour stencil
// (ltri 1, 2: src/cg_mod.f90:579-613 / src/update.f90:99-120)
__device__ __forceinline__ double2 smooth_at(const CGArgs &a, const double2 *__restrict__ v,
                                             const double *__restrict__ w, int i) {
    const int manz = a.manz;
    auto wv = [&](int j) { return w ? cscale(v[j], w[j]) : v[j]; };
    double2 c = cz(0.0, 0.0);
    if (a.ltri == 0) {
        const double *sm1 = a.smatm, *sm2 = a.smatm + manz, *sm3 = a.smatm + 2 * (size_t)manz;
        const int nx = a.nx;
        if (i > 0) c = cscale(wv(i - 1), sm2[i - 1]);
        if (i < manz - 1) c = cadd(c, cscale(wv(i + 1), sm2[i]));
        if (i >= nx) c = cadd(c, cscale(wv(i - nx), sm3[i - nx]));
        if (i < manz - nx) c = cadd(c, cscale(wv(i + nx), sm3[i]));
        return cadd(c, cscale(wv(i), sm1[i]));
    }
    for (int q = 0; q < a.maxnk; q++) {
        const int nb = a.nachbar[(size_t)q * manz + i];
        if (nb != 0) c = cadd(c, cscale(wv(nb - 1), a.smatm[(size_t)q * manz + i]));
    }
    return cadd(c, cscale(wv(i), a.smatm[(size_t)a.maxnk * manz + i]));
}

__global__ void k_rmul(CGArgs a, const double2 *__restrict__ v, double2 *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.manz) out[i] = smooth_at(a, v, nullptr, i);
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One block per column j: |g_j|, g_j = sum_i conj(s_ij) w_i vec_i (w_i = wmatd_i wdfak_i)
__global__ __launch_bounds__(kRedThreads) void k_colred_abs(CGArgs a, const double2 *__restrict__ vec, double *out) {
    const int j = blockIdx.x;
    const double2 *col = a.sens + (size_t)j * a.nanz;
    double gr = 0.0, gi = 0.0;
    for (int i = threadIdx.x; i < a.nanz; i += kRedThreads) {
        double2 s = col[i];
        if (a.part) s.y = 0.0;  // DBLE(sens)
        const double2 v = vec[i];  // weighted
        gr = fma(s.x, v.x, gr);
        gr = fma(s.y, v.y, gr);
        gi = fma(s.x, v.y, gi);
        gi = fma(-s.y, v.x, gi);
    }
    __shared__ double red[2][kRedThreads / 32];
    gr = warp_sum(gr);
    gi = warp_sum(gi);
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    if (lane == 0) {
        red[0][wl] = gr;
        red[1][wl] = gi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        gr = gi = 0.0;
        for (int q = 0; q < kRedThreads / 32; q++) {
            gr += red[0][q];
            gi += red[1][q];
        }
        out[j] = hypot(gr, gi);
    }
}

// State of the CG on the device: the steps run without the host, which only
// looks every kCgPoll steps whether they have stopped (a step after that
// returns at once).  dr of step k is in dr[k & 1].
struct CGState {
    double dr[2], dr0;
    int stop;  // step at which the residual test held; > ncgmax: not yet
};
constexpr int kCgPoll = 8;

// sum of n partial sums, in a fixed order, the same in every block
__device__ __forceinline__ double sum_parts(const double *__restrict__ part, int n) {
    __shared__ double red[kRedThreads / 32];
    double s = 0.0;
    for (int q = threadIdx.x; q < n; q += kRedThreads) s += part[q];
    s = warp_sum(s);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    s = 0.0;
#pragma unroll
    for (int q = 0; q < kRedThreads / 32; q++) s += red[q];
    return s;
}

// this block's sum of v over its threads, to part[blockIdx.x]
__device__ __forceinline__ void store_part(double v, double *part) {
    __shared__ double red[kRedThreads / 32];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int q = 0; q < kRedThreads / 32; q++) t += red[q];
        part[blockIdx.x] = t;
    }
}

// r = b (its imaginary or real part for the real CG, src/cg_mod.f90:160-164),
// p = x = 0, partial sums of |r|^2
__global__ __launch_bounds__(kRedThreads) void k_cg_init(CGArgs a, const double2 *__restrict__ b, double2 *r,
                                                         double2 *p, double *rr, CGState *st) {
    double s = 0.0;
    for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < a.manz; i += gridDim.x * kRedThreads) {
        double2 v = b[i];
        if (a.part) v = cz(a.part == 1 ? v.y : v.x, 0.0);
        r[i] = v;
        p[i] = a.dpar[i] = cz(0.0, 0.0);
        s = fma(v.x, v.x, s);
        s = fma(v.y, v.y, s);
    }
    store_part(s, rr);
    if (blockIdx.x == 0 && threadIdx.x == 0) st->stop = a.ncgmax + 1;
}

// step k: dr = |r|^2, the residual test, p = r + (dr / dr_before) p
__global__ __launch_bounds__(kRedThreads) void k_cg_direction(CGArgs a, int k, int nrr, const double *__restrict__ rr,
                                                              const double2 *__restrict__ r, double2 *p, CGState *st) {
    if (st->stop < k) return;
    const double dr = sum_parts(rr, nrr), dr0 = k == 1 ? dr * a.eps : st->dr0;
    const double beta = k == 1 ? 0.0 : dr / st->dr[(k - 1) & 1];
    // cjggdc tests the first step too
    const bool stop = (k > 1 || a.part) && dr <= dr0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->dr[k & 1] = dr;
        if (k == 1) st->dr0 = dr0;
        if (stop) st->stop = k;
    }
    if (stop) return;
    for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < a.manz; i += gridDim.x * kRedThreads) {
        const double2 u = r[i], v = p[i];
        p[i] = cz(u.x + beta * v.x, u.y + beta * v.y);
    }
}

// b_j = (sum_i conj(s_ij) wv_i + lam (R (cgfac o p))_j) cgfac_j (src/cg_mod.f90
// bb) and partial sums of Re(conj(p) b).  One warp per column: four FP64
// multiply-adds an element of J, the FP64 pipe's minimum for a complex
// product; with a block per column the block's sums took a third as many
// operations again (172 -> 118 us at 2000 x 8000).
__global__ __launch_bounds__(kRedThreads) void k_cg_back(CGArgs a, int k, const double2 *__restrict__ wv,
                                                         const double2 *__restrict__ p, double2 *__restrict__ b,
                                                         double *pb, const CGState *st) {
    if (st->stop <= k) return;
    const int lane = threadIdx.x & 31, j = blockIdx.x * (kRedThreads / 32) + (threadIdx.x >> 5);
    double dot = 0.0;
    if (j < a.manz) {
        const double2 *col = a.sens + (size_t)j * a.nanz;
        double gr = 0.0, gi = 0.0;
        for (int i0 = lane; i0 < a.nanz; i0 += 128) {
            double2 s[4], v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const bool in = i0 + 32 * q < a.nanz;
                s[q] = in ? col[i0 + 32 * q] : cz(0.0, 0.0);
                v[q] = in ? wv[i0 + 32 * q] : cz(0.0, 0.0);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (a.part) s[q].y = 0.0;
                gr = fma(s[q].x, v[q].x, gr);
                gr = fma(s[q].y, v[q].y, gr);
                gi = fma(s[q].x, v[q].y, gi);
                gi = fma(-s[q].y, v[q].x, gi);
            }
        }
        gr = warp_sum(gr);
        gi = warp_sum(gi);
        if (lane == 0) {
            const double2 rm = smooth_at(a, p, a.cgfac, j), pj = p[j];
            const double cf = a.cgfac[j];
            const double2 o = cz((gr + a.lam * rm.x) * cf, (gi + a.lam * rm.y) * cf);
            b[j] = o;
            dot = pj.x * o.x + pj.y * o.y;
        }
    }
    __shared__ double red[kRedThreads / 32];
    if (lane == 0) red[threadIdx.x >> 5] = dot;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int q = 0; q < kRedThreads / 32; q++) t += red[q];
        pb[blockIdx.x] = t;
    }
}

// alpha = dr / (p, b); x += alpha p, r -= alpha b, partial sums of |r|^2
__global__ __launch_bounds__(kRedThreads) void k_cg_advance(CGArgs a, int k, int npb, const double *__restrict__ pb,
                                                            const double2 *__restrict__ p,
                                                            const double2 *__restrict__ b, double2 *r, double *rr,
                                                            float *res, const CGState *st) {
    if (st->stop <= k) return;
    const double dr = st->dr[k & 1], alpha = dr / sum_parts(pb, npb);
    double s = 0.0;
    for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < a.manz; i += gridDim.x * kRedThreads) {
        const double2 u = p[i], v = b[i], x = a.dpar[i];
        double2 w = r[i];
        a.dpar[i] = cz(x.x + alpha * u.x, x.y + alpha * u.y);
        w = cz(w.x - alpha * v.x, w.y - alpha * v.y);
        r[i] = w;
        s = fma(w.x, w.x, s);
        s = fma(w.y, w.y, s);
    }
    store_part(s, rr);
    if (blockIdx.x == 0 && threadIdx.x == 0) res[k] = (float)(a.eps * dr / st->dr0);
}

// partial[chunk][i] = sum_{j in chunk} s_ij (cgfac_j p_j)   (src/cg_mod.f90:520-545)
__global__ __launch_bounds__(kRowTile) void k_jp_partial(CGArgs a, const double2 *__restrict__ p,
                                                         double2 *__restrict__ partial, int k, const CGState *st) {
    __shared__ double2 q[kColChunk];
    if (st && st->stop <= k) return;
    const int i = blockIdx.x * kRowTile + threadIdx.x;
    const int j0 = blockIdx.y * kColChunk;
    const int j1 = min(j0 + kColChunk, a.manz);
    for (int t = threadIdx.x; t < j1 - j0; t += kRowTile) {
        double2 v = p[j0 + t];
        double f = a.cgfac[j0 + t];
        q[t] = cz(v.x * f, v.y * f);
    }
    __syncthreads();
    if (i >= a.nanz) return;
    double ar = 0.0, ai = 0.0;
    for (int j = j0; j < j1; j++) {
        double2 s = a.sens[(size_t)j * a.nanz + i];
        if (a.part) s.y = 0.0;  // bapdc, src/cg_mod.f90:222-230
        const double2 v = q[j - j0];
        ar = fma(s.x, v.x, ar);
        ar = fma(-s.y, v.y, ar);
        ai = fma(s.x, v.y, ai);
        ai = fma(s.y, v.x, ai);
    }
    partial[(size_t)blockIdx.y * a.nanz + i] = cz(ar, ai);
}

// ap_i = w_i times the sum of the chunks (w_i = wmatd_i wdfak_i): 32 rows x 8
// groups of chunks a block, the groups added in order
__global__ __launch_bounds__(256) void k_jp_reduce(CGArgs a, int nchunk, const double2 *__restrict__ partial,
                                                   double2 *__restrict__ ap, int k, const CGState *st) {
    if (st && st->stop <= k) return;
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    const int c0 = nchunk * g / 8, c1 = nchunk * (g + 1) / 8;
    double2 s = cz(0.0, 0.0);
    if (i < a.nanz)
        for (int c = c0; c < c1; c++) s = cadd(s, partial[(size_t)c * a.nanz + i]);
    __shared__ double2 red[8][32];
    red[g][lane] = s;
    __syncthreads();
    if (g || i >= a.nanz) return;
    for (int q = 1; q < 8; q++) s = cadd(s, red[q][lane]);
    const double w = a.wmatd[i] * (double)a.wdfak[i];
    ap[i] = cz(w * s.x, w * s.y);
}

// wv = w (dat - f), w: the data weights of the right-hand side
__global__ void k_cg_data(CGArgs a, double2 *__restrict__ wv, double *__restrict__ w) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nanz) return;
    const double f = a.wmatd[i] * (double)a.wdfak[i];
    const double2 d = csub(a.dat[i], a.sigmaa[i]);
    w[i] = f;
    wv[i] = cz(f * d.x, f * d.y);
}

// preconditioner and right-hand side (src/update.f90:182-192, 236-293), one
// warp per column: cgfac_j = 1/sqrt(sum_i |s_ij|^2 w_i + lam R_jj), b_j =
// (sum_i conj(s_ij) wv_i - lam rm_j) cgfac_j, where b holds rm = R m
__global__ __launch_bounds__(kRedThreads) void k_cg_rhs(CGArgs a, const double2 *__restrict__ wv,
                                                        const double *__restrict__ w, double2 *b) {
    const int lane = threadIdx.x & 31, j = blockIdx.x * (kRedThreads / 32) + (threadIdx.x >> 5);
    if (j >= a.manz) return;
    const double2 *col = a.sens + (size_t)j * a.nanz;
    double gr = 0.0, gi = 0.0, dg = 0.0;
#pragma unroll 4
    for (int i = lane; i < a.nanz; i += 32) {
        double2 s = col[i];
        if (a.part) s.y = 0.0;
        const double2 v = wv[i];
        dg = fma(fma(s.x, s.x, s.y * s.y), w[i], dg);
        gr = fma(s.x, v.x, gr);
        gr = fma(s.y, v.y, gr);
        gi = fma(s.x, v.y, gi);
        gi = fma(-s.y, v.x, gi);
    }
    gr = warp_sum(gr);
    gi = warp_sum(gi);
    dg = warp_sum(dg);
    if (lane) return;
    const double diagR = a.ltri == 0 ? a.smatm[j] : a.smatm[(size_t)a.maxnk * a.manz + j];
    const double cf = 1.0 / sqrt(dg + a.lam * diagR);
    const double2 rm = b[j];
    a.cgfac[j] = cf;
    b[j] = cz((gr - a.lam * rm.x) * cf, (gi - a.lam * rm.y) * cf);
}

// dpar = cgfac o dpar (part 1: i Re(dpar), src/update.f90:299-302; part 2:
// Re(dpar)), par += step dpar
__global__ void k_final(int n, double2 *dpar, const double *__restrict__ cgfac, double step, double2 *par,
                        int part) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double2 d = dpar[i];
    double f = cgfac[i];
    d = part == 1 ? cz(0.0, d.x * f) : part == 2 ? cz(d.x * f, 0.0) : cz(d.x * f, d.y * f);
    dpar[i] = d;
    double2 p = par[i];
    par[i] = cz(p.x + step * d.x, p.y + step * d.y);
}

inline unsigned nblk(int n, int t) { return (unsigned)((n + t - 1) / t); }

__global__ void k_fill_one(int n, double2 *v, double *f) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    v[i] = cz(1.0, 0.0);
    f[i] = 1.0;
}

}  // namespace

// work layout (double2 units): bvec, rvec, pvec (manz) | ap, dmf (nanz) |
// partial (nchunk * nanz) | state, partial sums of |r|^2 and (p, b), record
size_t update_work_bytes(int nanz, int manz, int ncgmax) {
    int nchunk = (manz + kColChunk - 1) / kColChunk;
    return sizeof(double2) * ((size_t)3 * manz + 2 * (size_t)nanz + (size_t)nchunk * nanz) + sizeof(CGState) + 64 +
           sizeof(double) * (kRedBlocks + manz / 8 + 8) + sizeof(float) * ((size_t)ncgmax + 2);
}

int run_update(const CGArgs &a, cudaStream_t st, int *ncg_out, float *cgres_host) {
    const int manz = a.manz, nanz = a.nanz;
    const int nchunk = (manz + kColChunk - 1) / kColChunk;
    double2 *bvec = a.work, *rvec = bvec + manz, *pvec = rvec + manz;
    double2 *ap = pvec + manz, *dmf = ap + nanz, *partial = dmf + nanz;
    CGState *state = (CGState *)(partial + (size_t)nchunk * nanz);
    double *rr = (double *)(state + 1), *pb = rr + kRedBlocks;
    const int T = 256, npb = (manz + 7) / 8, nrr = std::min(kRedBlocks, (int)nblk(manz, kRedThreads));
    float *res = (float *)(pb + npb);
    // bvec = R m ; right-hand side and preconditioner
    k_rmul<<<nblk(manz, T), T, 0, st>>>(a, a.par, bvec);
    k_cg_data<<<nblk(nanz, T), T, 0, st>>>(a, ap, (double *)dmf);
    k_cg_rhs<<<npb, kRedThreads, 0, st>>>(a, ap, (const double *)dmf, bvec);
    // cjggra (complex) or cjggdc (parts 1, 2: the same recursion on real vectors)
    cudaMemsetAsync(res, 0, sizeof(float) * (a.ncgmax + 2), st);
    k_cg_init<<<nrr, kRedThreads, 0, st>>>(a, bvec, rvec, pvec, rr, state);
    int stop = a.ncgmax + 1;
    const dim3 g1(nblk(nanz, kRowTile), nchunk);
    for (int k = 1; k <= a.ncgmax && stop > a.ncgmax; k++) {
        k_cg_direction<<<nrr, kRedThreads, 0, st>>>(a, k, nrr, rr, rvec, pvec, state);
        k_jp_partial<<<g1, kRowTile, 0, st>>>(a, pvec, partial, k, state);
        k_jp_reduce<<<nblk(nanz, 32), 256, 0, st>>>(a, nchunk, partial, dmf, k, state);
        k_cg_back<<<npb, kRedThreads, 0, st>>>(a, k, dmf, pvec, bvec, pb, state);
        k_cg_advance<<<nrr, kRedThreads, 0, st>>>(a, k, npb, pb, pvec, bvec, rvec, rr, res, state);
        if (k % kCgPoll == 0 || k == a.ncgmax) {
            cudaMemcpyAsync(&stop, &state->stop, sizeof(int), cudaMemcpyDeviceToHost, st);
            cudaError_t e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return ERR_CUDA;
        }
    }
    const int ncg = std::min(stop - 1, a.ncgmax);
    k_final<<<nblk(manz, T), T, 0, st>>>(manz, a.dpar, a.cgfac, a.step, a.par, a.part);
    cudaMemcpyAsync(cgres_host, res, sizeof(float) * (a.ncgmax + 2), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    cgres_host[0] = (float)ncg;
    *ncg_out = ncg;
    return e == cudaSuccess ? 0 : ERR_CUDA;
}

// |(J^H W J 1)_j| of src/blam0.f90:60-130 (phase only: Re(J)): the double
// sum over data and model cells as two products with J.  Reads a.sens,
// a.wmatd, a.wdfak and the work space; a.smatm, a.nachbar, a.par, a.dpar,
// a.dat and a.sigmaa are not used.
int run_jhwj1(CGArgs a, cudaStream_t st, double *jtj_host) {
    const int manz = a.manz, nanz = a.nanz;
    const int nchunk = (manz + kColChunk - 1) / kColChunk;
    double2 *bvec = a.work, *ones = bvec + manz;
    double2 *ap = ones + 2 * (size_t)manz, *partial = ap + 2 * (size_t)nanz;
    const int T = 256;
    k_fill_one<<<nblk(manz, T), T, 0, st>>>(manz, ones, a.cgfac);
    dim3 g1(nblk(nanz, kRowTile), nchunk);
    k_jp_partial<<<g1, kRowTile, 0, st>>>(a, ones, partial, 0, nullptr);
    k_jp_reduce<<<nblk(nanz, 32), 256, 0, st>>>(a, nchunk, partial, ap, 0, nullptr);
    k_colred_abs<<<manz, kRedThreads, 0, st>>>(a, ap, (double *)bvec);
    cudaMemcpyAsync(jtj_host, bvec, sizeof(double) * manz, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? 0 : ERR_CUDA;
}

}  // namespace crgpu

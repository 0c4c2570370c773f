// Substructured solver of the (wavenumber, electrode) systems of src/fem.f90:
// 355-397 (src/kompab.f90, src/chol.f90, src/vre.f90).
//
// Of a wavenumber's matrix only the entries among the nodes of the mixed
// boundary depend on the electrode (src/beta.f90).  Every other node is
// eliminated once per wavenumber, by nested dissection (sub_plan.cpp): a
// front's pivot block is inverted, G = F11^-1 F12, and S = F22 - F12^T G goes
// to its parent.  What remains is one dense complex symmetric matrix per
// system over the m boundary nodes, the wavenumber's Schur complement plus the
// electrode's boundary terms, which is factored C C^T as src/chol.f90 does.  A
// solve runs up the tree (all electrodes as columns of dense products),
// through the root, and down again.
//
// Config 2 (12261 nodes, 13 wavenumbers x 96 electrodes, m = 321): 3.9e7
// complex multiply-adds a wavenumber for the shared part and 5.5e6 a system
// for the root, against 2.4e7 a system for the band of 62 and 9.0e7 for the
// grid's band of 121; and a triangle of 0.4 MB a system for the root instead of
// 6.2 MB (12).
#include <algorithm>
#include <mutex>

#include "async.cuh"
#include "convert.cuh"
#include "kernels.h"
#include "mixed_common.cuh"
#include "substruct.h"

namespace crgpu {

namespace {

// ---------------------------------------------------------------- arithmetic
__device__ __forceinline__ void fma_(float2 &s, float2 a, float2 b) {
    s.x = fmaf(a.x, b.x, s.x);
    s.x = fmaf(-a.y, b.y, s.x);
    s.y = fmaf(a.x, b.y, s.y);
    s.y = fmaf(a.y, b.x, s.y);
}
__device__ __forceinline__ void fma_(double2 &s, double2 a, double2 b) {
    s.x = fma(a.x, b.x, s.x);
    s.x = fma(-a.y, b.y, s.x);
    s.y = fma(a.x, b.y, s.y);
    s.y = fma(a.y, b.x, s.y);
}
__device__ __forceinline__ void fms_(float2 &s, float2 a, float2 b) { s = cfmsf(s, a, b); }
__device__ __forceinline__ void fms_(double2 &s, double2 a, double2 b) { s = cfms(s, a, b); }
__device__ __forceinline__ float2 mul_(float2 a, float2 b) { return cmulf(a, b); }
__device__ __forceinline__ double2 mul_(double2 a, double2 b) { return cmul(a, b); }
// reciprocals and inverse roots of pivots.  complex128 without FP64 divisions
// and roots (about 100 FP64 operations a lane): an FP32 estimate and two Newton
// steps, which square its error.
__device__ __forceinline__ float2 rcp_(float2 a) { return crecip_fast(a); }
__device__ __forceinline__ double2 rcp_(double2 a) {
    const double m = a.x * a.x + a.y * a.y;
    if (!(m > 1e-30 && m < 1e30)) return crecip(a);
    double q = (double)__frcp_rn((float)m);
#pragma unroll
    for (int it = 0; it < 2; it++) q = q * (2.0 - m * q);
    return cz(a.x * q, -a.y * q);
}
// 1 / (principal square root); w <- w (3 - d w^2) / 2
__device__ __forceinline__ float2 rsqrt_(float2 a) { return crecip_fast(csqrt_fast(a)); }
__device__ __forceinline__ double2 rsqrt_(double2 d) {
    const float2 f = to_f(d);
    const float m = fmaxf(fabsf(f.x), fabsf(f.y));
    if (!(m > 1e-15f && m < 1e15f)) return crecip(csqrtd(d));
    double2 w = to_d(crecipf(csqrtf_(f)));
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const double2 h = cmul(d, cmul(w, w));
        w = cmul(w, cz(1.5 - 0.5 * h.x, -0.5 * h.y));
    }
    return w;
}
__device__ __forceinline__ float2 neg_(float2 a) { return cf(-a.x, -a.y); }
__device__ __forceinline__ double2 neg_(double2 a) { return cz(-a.x, -a.y); }
// bit pattern of |v|: the patterns of non-negative doubles order like the values
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

template <typename T>
__device__ __forceinline__ T from_(double2 v);
template <>
__device__ __forceinline__ float2 from_<float2>(double2 v) {
    return to_f(v);
}
template <>
__device__ __forceinline__ double2 from_<double2>(double2 v) {
    return v;
}
template <typename T>
__device__ __forceinline__ T shfl_(T v, int src) {
    v.x = __shfl_sync(0xffffffffu, v.x, src);
    v.y = __shfl_sync(0xffffffffu, v.y, src);
    return v;
}
template <typename T>
__device__ __forceinline__ T warp_sum_(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}
template <typename T>
__device__ __forceinline__ T zero_() {
    T z;
    z.x = 0;
    z.y = 0;
    return z;
}
__device__ __forceinline__ bool is_bad(float2 v) { return !(isfinite(v.x) && isfinite(v.y)) || (v.x == 0.f && v.y == 0.f); }
__device__ __forceinline__ bool is_bad(double2 v) { return !(isfinite(v.x) && isfinite(v.y)) || (v.x == 0.0 && v.y == 0.0); }

// two consecutive entries at a 16-byte boundary of shared memory
__device__ __forceinline__ void load2(const float2 *p, float2 (&v)[2]) {
    const float4 a = *(const float4 *)p;
    v[0] = cf(a.x, a.y);
    v[1] = cf(a.z, a.w);
}
__device__ __forceinline__ void load2(const double2 *p, double2 (&v)[2]) {
    v[0] = p[0];
    v[1] = p[1];
}

// Programmatic dependent launch: a forward is a chain of up to 250 short
// kernels, and the start of each (launch, tables, index loads) overlaps the end
// of the one before.  A kernel waits for its predecessor before it reads or writes
// anything but the plan's tables and what is older than that predecessor.  A block
// may return without the wait, but of every grid at least one block waits, so a
// grid ends only after all earlier ones and its successor's wait covers them.  GB300:
// 60x20 quads mixed with Jacobian 2.11 -> 1.82 ms, triangle gradient 14.7 -> 13.8
// ms.  Letting the successor's blocks in before this kernel ends
// (launch_dependents) cost complex128 3 %: they take the places of its last
// wave.  In a recorded graph plain edges are the faster ones (9.7 against 10.0
// ms).
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
void chain_launch(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cap);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = cap == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

constexpr int kKT = 32;  // depth of a chunk of the dense products

// Tile edge of the dense kernels and results a thread: 256 threads own a 32 x
// 32 tile with 2 x 2 results each in complex64.  In complex128 a tile is bound
// by its SM's FP64 pipe (32 x 32 x 32 takes 32 us) and the topmost fronts have
// few tiles, so there it is 16 x 16, one result a thread; and fronts of at most
// 32 nodes leave more of the elimination to the tiles.  Leaves of 16 / 24 / 32 /
// 48 nodes: config-2 mixed forward 13.2 / 12.8 / 12.6 / 12.6 ms.
template <typename T>
struct Tile;
template <>
struct Tile<float2> {
    static constexpr int E = 32, M = 2, P = 34, leaf = 32, emax = 64;
};
template <>
struct Tile<double2> {
    static constexpr int E = 16, M = 1, P = 17, leaf = 24, emax = 32;
};

// ------------------------------------------------------- values and scaling
// fk: 1/sqrt|diagonal of the area part| (1 on Dirichlet rows); a zero
// diagonal is error 27 (src/scalab.f90:57-61).  A boundary node whose area
// part alone is zero while its boundary terms are not keeps scale 1.
__global__ void k_sub_scale(DevProblem P, DevSub D, const double2 *__restrict__ sigma,
                            const double *__restrict__ fak_area) {
    const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= (size_t)P.K * P.n) return;
    const int k = (int)(g / P.n), i = (int)(g % P.n);
    double f = fak_area[g];
    if (P.dirichlet[i]) {
        f = 1.0;
    } else if (!(f > 0.0)) {
        f = 1.0;
        bool some = false;
        for (int p = P.rowptr[i]; p < P.rowptr[i + 1]; p++)
            if (P.col[p] == i)
                for (int q = P.bnd_ptr[p]; q < P.bnd_ptr[p + 1]; q++) {
                    const double2 s = sigma[P.brnr[P.bnd_list[q] >> 4]];
                    some = some || s.x != 0.0 || s.y != 0.0;
                }
        if (!some) atomicCAS(&D.kbad[k], 0, 27);
    }
    D.fk[g] = f;
}

__global__ void k_sub_values(DevProblem P, DevSub D, const double2 *__restrict__ adom) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (p >= P.nnz) return;
    const int c = P.col[p];
    double2 v = cz(0.0, 0.0);
    if (c >= 0) {
        const int i = P.row[p];
        if (P.dirichlet[i] || P.dirichlet[c]) {
            v = i == c ? cz(1.0, 0.0) : cz(0.0, 0.0);
        } else {
            const double f = D.fk[(size_t)k * P.n + i] * D.fk[(size_t)k * P.n + c];
            const double2 a = adom[(size_t)k * P.nnz + p];
            v = cz(a.x * f, a.y * f);
        }
    }
    D.As[(size_t)k * P.nnz + p] = v;
}

// ------------------------------------------------------------ shared factor
// A front's F11 (into D.F) and F12 (into D.H) from its children's Schur
// complements, one block per 32 x 32 tile of the e x (e + r) rows.  (Gathered
// by the pivot kernel's one block per front, the indices and the dependent
// loads took longer than the elimination: 166 -> 60 us at e = 61, r = 321.)
template <typename T>
__global__ __launch_bounds__(256) void k_sub_gather(DevSub D, int t0) {
    constexpr int E = Tile<T>::E, NZ = E * E / 256, RS = 256 / E;
    __shared__ int si[kSubCh][E], sj[kSubCh][E];
    const SubTile tl = D.tA[t0 + blockIdx.x];
    const SubFront &t = D.fr[tl.front];
    const int k = blockIdx.y, e = t.e, r = t.r, nch = t.nch, i0 = tl.ti * E, j0 = tl.tj * E;
    const int col = threadIdx.x % E, row = threadIdx.x / E;
    for (int q = threadIdx.x; q < 2 * nch * E; q += 256) {
        const int c = q / (2 * E), b = q / E & 1, o = q % E, at = (b ? j0 : i0) + o;
        (b ? sj : si)[c][o] = at < (b ? e + r : e) ? D.inv[t.inv[c] + at] : -1;
    }
    chain_wait();
    __syncthreads();
    const T *Sk = (const T *)D.S + (size_t)k * D.szS;
    T *F = (T *)D.F + (size_t)k * D.szF + t.oF, *H = (T *)D.H + (size_t)k * D.szG + t.oG;
    T v[NZ];
#pragma unroll
    for (int z = 0; z < NZ; z++) v[z] = zero_<T>();
    for (int c = 0; c < nch; c++) {
        const T *S = Sk + t.cS[c];
        const int cr = t.cr[c], y = sj[c][col];
        T g[NZ];
#pragma unroll
        for (int z = 0; z < NZ; z++) {
            const int x = si[c][row + RS * z];
            g[z] = x >= 0 && y >= 0 ? S[(size_t)x * cr + y] : zero_<T>();
        }
#pragma unroll
        for (int z = 0; z < NZ; z++) {
            v[z].x += g[z].x;
            v[z].y += g[z].y;
        }
    }
#pragma unroll
    for (int z = 0; z < NZ; z++) {
        const int i = i0 + row + RS * z, j = j0 + col;
        if (i >= e || j >= e + r) continue;
        if (j < e) F[(size_t)i * e + j] = v[z];
        else H[(size_t)i * r + j - e] = v[z];
    }
}

// In-place inverse of the symmetric h x h matrix M (h <= 32, row stride ld) in
// shared memory by Gauss-Jordan sweeps: lane = row, warp w the columns w, w + 8,
// ..., in registers.  Per sweep the pivot's warp publishes its column and the
// pivot row over the pivot, which is the column again up to the sign between
// swept and unswept rows; one barrier, and one complex multiply-add an entry.
// Ends with a barrier.  False where a pivot is zero or not finite.
template <typename T>
struct Sweep {
    T col[2][32], row[2][32];
};

template <typename T>
__device__ __forceinline__ bool invert_block(T *M, int ld, int h, Sweep<T> &sw) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T a[4];
#pragma unroll
    for (int q = 0; q < 4; q++) a[q] = lane < h && 8 * q + w < h ? M[lane * ld + 8 * q + w] : zero_<T>();
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int ww = 0; ww < 8; ww++) {
            const int p = 8 * q + ww, b = p & 1;
            if (p >= h) continue;  // the same for all threads
            if (w == ww) {
                const T d = shfl_(a[q], p);
                if (is_bad(d)) ok = false;
                const T iv = rcp_(d);
                sw.col[b][lane] = a[q];
                sw.row[b][lane] = lane == p ? iv : mul_(lane < p ? neg_(a[q]) : a[q], iv);
                a[q] = zero_<T>();
            }
            __syncthreads();
            const T c = sw.col[b][lane];
#pragma unroll
            for (int z = 0; z < 4; z++) {
                const T t = sw.row[b][8 * z + w];
                fms_(a[z], c, t);
                if (lane == p) a[z] = t;
            }
        }
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (lane < h && 8 * q + w < h) M[lane * ld + 8 * q + w] = a[q];
    __syncthreads();
    return ok;
}

// Adds a front's matrix entries to F11 and F12 and inverts F11, one block of
// 256 threads.  Beyond 32 nodes by blocks, F11 = [A B; B^T D]: G = A^-1 B, the
// complement D - B^T G inverted, [A^-1 + K G^T, -K; -K^T, Si] with K = G Si.  (Swept
// as a whole, lower triangle only, a front of 61 nodes took 114 us: a chain of
// two barriers and divergent updates a node.)
template <typename T>
__global__ __launch_bounds__(256) void k_sub_pivot(DevSub D, int f0, int nnz) {
    extern __shared__ __align__(16) unsigned char sm[];
    constexpr int H = 32, PH = H + 1;
    T *Fm = (T *)sm;  // [e][e | 1], then G and K, [32][33] each, beyond 32 nodes
    __shared__ Sweep<T> sw;
    const SubFront &t = D.fr[f0 + blockIdx.x];
    const int k = blockIdx.y, e = t.e, r = t.r, ld = e | 1, tid = threadIdx.x, nent = t.nent, ent0 = t.ent0;
    const bool leaf = t.nch == 0;
    const double2 *As = D.As + (size_t)k * nnz;
    T *F = (T *)D.F + (size_t)k * D.szF + t.oF, *Hm = (T *)D.H + (size_t)k * D.szG + t.oG;
    chain_wait();
    for (int q = tid; q < e * e; q += 256) Fm[(q / e) * ld + q % e] = leaf ? zero_<T>() : F[q];
    if (leaf)
        for (int q = tid; q < e * r; q += 256) Hm[q] = zero_<T>();
    __syncthreads();
    for (int q = tid; q < nent; q += 256) {
        const SubEnt en = D.ent[ent0 + q];
        const T v = from_<T>(As[en.p]);
        if (en.lc < e) {
            T &d = Fm[en.lr * ld + en.lc];
            d.x += v.x;
            d.y += v.y;
            if (en.lr != en.lc) {
                T &u = Fm[en.lc * ld + en.lr];
                u.x += v.x;
                u.y += v.y;
            }
        } else {
            T &d = Hm[(size_t)en.lr * r + en.lc - e];
            d.x += v.x;
            d.y += v.y;
        }
    }
    __syncthreads();
    bool ok = invert_block(Fm, ld, min(e, H), sw);
    if (Tile<T>::emax > H && e > H) {
        const int h = e - H, lane = tid & 31, w = tid >> 5;
        T *G = Fm + e * ld, *K = G + H * PH;
        // G = A^-1 B: row = lane, columns w, w + 8, ...
        for (int c = w; c < h; c += 8) {
            T s = zero_<T>();
#pragma unroll 8
            for (int p = 0; p < H; p++) fma_(s, Fm[lane * ld + p], Fm[p * ld + H + c]);
            G[lane * PH + c] = s;
        }
        __syncthreads();
        if (lane < h)
            for (int c = w; c < h; c += 8) {
                T s = Fm[(H + lane) * ld + H + c];
#pragma unroll 8
                for (int p = 0; p < H; p++) fms_(s, Fm[(H + lane) * ld + p], G[p * PH + c]);
                Fm[(H + lane) * ld + H + c] = s;
            }
        __syncthreads();
        if (!invert_block(Fm + H * ld + H, ld, h, sw)) ok = false;
        for (int c = w; c < h; c += 8) {
            T s = zero_<T>();
            for (int p = 0; p < h; p++) fma_(s, G[lane * PH + p], Fm[(H + p) * ld + H + c]);
            K[lane * PH + c] = s;
            Fm[lane * ld + H + c] = neg_(s);
            Fm[(H + c) * ld + lane] = neg_(s);
        }
        __syncthreads();
        for (int c = w; c < H; c += 8) {
            T s = Fm[lane * ld + c];
            for (int p = 0; p < h; p++) fma_(s, K[lane * PH + p], G[c * PH + p]);
            Fm[lane * ld + c] = s;
        }
        __syncthreads();
    }
    for (int q = tid; q < e * e; q += 256) F[q] = Fm[(q / e) * ld + q % e];
    if (!ok) atomicCAS(&D.kbad[k], 0, 28);
}

// A thread's entries of a kKT x E operand tile (k-major) in registers: the
// loads of the next chunk are in flight while the present one is multiplied.
template <typename T>
struct Operand {
    static constexpr int E = Tile<T>::E, P = Tile<T>::P, N = kKT * E / 256;
    T v[N];
    // along a row of the tile: column threadIdx % E, rows row(0), row(1), ...
    __device__ __forceinline__ static int col() { return threadIdx.x % E; }
    __device__ __forceinline__ static int row(int z) { return threadIdx.x / E + (256 / E) * z; }
    __device__ __forceinline__ void load(const T *src, size_t ls, int nr, int nc) {
#pragma unroll
        for (int z = 0; z < N; z++) v[z] = row(z) < nr && col() < nc ? src[(size_t)row(z) * ls + col()] : zero_<T>();
    }
    __device__ __forceinline__ void store(T *dst) const {
#pragma unroll
        for (int z = 0; z < N; z++) dst[row(z) * P + col()] = v[z];
    }
    // from the transposed source, E rows of kKT: one warp a row
    __device__ __forceinline__ void load_t(const T *src, size_t ls, int nr, int nc) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
        for (int z = 0; z < N; z++)
            v[z] = w + 8 * z < nr && lane < nc ? src[(size_t)(w + 8 * z) * ls + lane] : zero_<T>();
    }
    __device__ __forceinline__ void store_t(T *dst) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
        for (int z = 0; z < N; z++) dst[lane * P + w + 8 * z] = v[z];
    }
};

// a thread's M x M results of a tile: rows tr.., columns tc..
template <typename T>
struct Result {
    static constexpr int M = Tile<T>::M, E = Tile<T>::E, P = Tile<T>::P;
    T v[M][M];
    __device__ __forceinline__ static int tr() { return threadIdx.x / (E / M) * M; }
    __device__ __forceinline__ static int tc() { return threadIdx.x % (E / M) * M; }
    // first row of the warp's results
    __device__ __forceinline__ static int warp_row() { return (threadIdx.x & ~31) / (E / M) * M; }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < M; i++)
#pragma unroll
            for (int j = 0; j < M; j++) v[i][j] = zero_<T>();
    }
    __device__ __forceinline__ void multiply(const T *A, const T *Bm, int kk) {
        const int r = tr(), c = tc();
#pragma unroll 8
        for (int q = 0; q < kk; q++) {
            if constexpr (M == 2) {
                T a[2], b[2];
                load2(A + q * P + r, a);
                load2(Bm + q * P + c, b);
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 2; j++) fma_(v[i][j], a[i], b[j]);
            } else {
                fma_(v[0][0], A[q * P + r], Bm[q * P + c]);
            }
        }
    }
};

// G = F11^-1 F12
template <typename T>
__global__ __launch_bounds__(256) void k_sub_g(DevSub D, int t0) {
    constexpr int E = Tile<T>::E, M = Tile<T>::M, P = Tile<T>::P;
    __shared__ __align__(16) T A[kKT * P], Bm[kKT * P];
    const SubTile tl = D.tG[t0 + blockIdx.x];
    const SubFront &t = D.fr[tl.front];
    const int k = blockIdx.y, e = t.e, r = t.r, i0 = tl.ti * E, j0 = tl.tj * E;
    const T *F = (const T *)D.F + (size_t)k * D.szF + t.oF, *H = (const T *)D.H + (size_t)k * D.szG + t.oG;
    T *G = (T *)D.G + (size_t)k * D.szG + t.oG;
    Result<T> acc;
    acc.clear();
    const bool work = i0 + acc.warp_row() < e;
    Operand<T> a, b;
    chain_wait();
    a.load(F + i0, e, e, e - i0);  // symmetric: F[p][i]
    b.load(H + j0, r, e, r - j0);
    for (int p = 0; p < e; p += kKT) {
        a.store(A);
        b.store(Bm);
        __syncthreads();
        if (p + kKT < e) {
            a.load(F + (size_t)(p + kKT) * e + i0, e, e - p - kKT, e - i0);
            b.load(H + (size_t)(p + kKT) * r + j0, r, e - p - kKT, r - j0);
        }
        if (work) acc.multiply(A, Bm, min(kKT, e - p));
        __syncthreads();
    }
#pragma unroll
    for (int ii = 0; ii < M; ii++)
#pragma unroll
        for (int jj = 0; jj < M; jj++) {
            const int i = i0 + acc.tr() + ii, j = j0 + acc.tc() + jj;
            if (i < e && j < r) G[(size_t)i * r + j] = acc.v[ii][jj];
        }
}

// S = (children's complements) - F12^T G, lower tiles, mirrored
template <typename T>
__global__ __launch_bounds__(256) void k_sub_s(DevSub D, int t0) {
    constexpr int E = Tile<T>::E, M = Tile<T>::M, P = Tile<T>::P;
    __shared__ __align__(16) T A[kKT * P], Bm[kKT * P];
    __shared__ int si[kSubCh][E], sj[kSubCh][E];
    const SubTile tl = D.tS[t0 + blockIdx.x];
    const SubFront &t = D.fr[tl.front];
    const int k = blockIdx.y, e = t.e, r = t.r, nch = t.nch, i0 = tl.ti * E, j0 = tl.tj * E;
    const T *H = (const T *)D.H + (size_t)k * D.szG + t.oG, *G = (const T *)D.G + (size_t)k * D.szG + t.oG;
    T *Sk = (T *)D.S + (size_t)k * D.szS, *S = Sk + t.oS;
    Operand<T> a, b;
    for (int q = threadIdx.x; q < 2 * nch * E; q += 256) {
        const int c = q / (2 * E), bb = q / E & 1, o = q % E, at = (bb ? j0 : i0) + o;
        (bb ? sj : si)[c][o] = at < r ? D.inv[t.inv[c] + e + at] : -1;
    }
    chain_wait();
    a.load(H + i0, r, e, r - i0);
    b.load(G + j0, r, e, r - j0);
    __syncthreads();
    Result<T> acc, sum;
    acc.clear();
    sum.clear();
    const int tr = acc.tr(), tc = acc.tc();
    const bool work = i0 + acc.warp_row() < r;
    for (int c = 0; c < nch; c++) {
        const T *Sc = Sk + t.cS[c];
        const int cr = t.cr[c];
#pragma unroll
        for (int i = 0; i < M; i++)
#pragma unroll
            for (int j = 0; j < M; j++) {
                const int x = si[c][tr + i], y = sj[c][tc + j];
                if (x >= 0 && y >= 0) {
                    const T v = Sc[(size_t)x * cr + y];
                    sum.v[i][j].x += v.x;
                    sum.v[i][j].y += v.y;
                }
            }
    }
    for (int p = 0; p < e; p += kKT) {
        a.store(A);
        b.store(Bm);
        __syncthreads();
        if (p + kKT < e) {
            a.load(H + (size_t)(p + kKT) * r + i0, r, e - p - kKT, r - i0);
            b.load(G + (size_t)(p + kKT) * r + j0, r, e - p - kKT, r - j0);
        }
        if (work) acc.multiply(A, Bm, min(kKT, e - p));
        __syncthreads();
    }
#pragma unroll
    for (int ii = 0; ii < M; ii++)
#pragma unroll
        for (int jj = 0; jj < M; jj++) {
            const int i = i0 + tr + ii, j = j0 + tc + jj;
            if (i >= r || j > i) continue;
            T v = sum.v[ii][jj];
            v.x -= acc.v[ii][jj].x;
            v.y -= acc.v[ii][jj].y;
            S[(size_t)i * r + j] = v;
            S[(size_t)j * r + i] = v;
        }
}

// the root's shared part, column-major lower, padded by a unit diagonal:
// the last front's complement, then the area entries among root nodes
template <typename T>
__global__ void k_sub_root_base(DevSub D) {
    const int c = blockIdx.x, k = blockIdx.y;
    const T *S = (const T *)D.S + (size_t)k * D.szS + D.root_oS;
    T *R = (T *)D.R + ((size_t)k * D.mp + c) * D.ldc;
    const int y = c < D.m ? D.root_inv[c] : -1;
    for (int i = threadIdx.x; i < D.ldc; i += blockDim.x) {
        T v = zero_<T>();
        if (i < D.m && y >= 0) {
            const int x = D.root_inv[i];
            if (x >= 0) v = S[(size_t)x * D.root_r + y];
        }
        if (i == c && c >= D.m) v.x = 1;
        R[i] = v;
    }
}

template <typename T>
__global__ void k_sub_root_ent(DevSub D, int nnz) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (q >= D.n_root_ent) return;
    const SubEnt en = D.ent[D.root_ent0 + q];
    const T v = from_<T>(D.As[(size_t)k * nnz + en.p]);
    T &d = ((T *)D.R)[((size_t)k * D.mp + en.lc) * D.ldc + en.lr];
    d.x += v.x;
    d.y += v.y;
}

// ------------------------------------------------------------- root factor
// The electrodes' boundary terms, summed per root entry in FP64, the
// electrode fastest: [Kb][n_be][Lb]
__global__ void k_sub_bval(DevProblem P, DevSub D, SubBatch B, const double2 *__restrict__ sigma) {
    const int l = blockIdx.y * 32 + (threadIdx.x & 31), q = blockIdx.x * 8 + (threadIdx.x >> 5), kk = blockIdx.z;
    if (l >= B.Lb || q >= D.n_be) return;
    const int p = D.be[q].p, i = P.row[p], c = P.col[p], k = B.k0 + kk;
    double2 v = cz(0.0, 0.0);
    if (!P.dirichlet[i] && !P.dirichlet[c]) {
        const double *kgl = P.kg + ((size_t)k * P.eanz + B.l0 + l) * P.relanz, *fk = D.fk + (size_t)k * P.n;
        const double f = fk[i] * fk[c];
        for (int z = P.bnd_ptr[p]; z < P.bnd_ptr[p + 1]; z++) {
            const int rb = P.bnd_list[z] >> 4;
            const double g = P.relbg[rb * 3 + (P.bnd_list[z] & 15)] * kgl[rb];
            const double2 sg = sigma[P.brnr[rb]];
            v = cz(v.x + g * sg.x, v.y + g * sg.y);
        }
        v = cz(v.x * f, v.y * f);
    }
    B.bval[((size_t)kk * D.n_be + q) * B.Lb + l] = v;
}

// C C^T of one system's root, column-major lower with leading dimension ldc,
// one block of 128 threads per system, left-looking in NB columns.  A block's
// rows are worked in tiles of 64, a warp on 16 of them: W = M - C C_j^T from
// the finished columns (cp.async, S chunks of KC columns in flight, one
// barrier a chunk), then W C_jj^-T.  The diagonal block is factored and
// inverted together, one barrier a column; its inverse is stored in its place,
// which is all that the later solves need.  Bound by the FP64 pipe in
// complex128, so NB is 16 there: the panel's products with the full inverse
// and the upper halves of the diagonal blocks cost m^2 NB / 2 and m^2 NB / 4
// beside m^3 / 6.  In complex64 the operand traffic counts too and NB is 32.
// Five blocks an SM (96 registers): the phases between the products are chains
// of loads and barriers, which only other blocks fill (at 4 / 5 / 6 the factor
// of config 2 takes 4.07 / 3.98 / 4.02 ms; tiles of 128 rows with 8 x 4 results a
// thread were slower).  Warps whose rows lie beyond the matrix skip the
// products.
constexpr int kRT = 128;  // threads

template <typename T>
struct RootShape {
    static constexpr bool F = sizeof(T) == 8;
    static constexpr int NB = F ? 32 : 16;
    static constexpr int TR = F ? 4 : 2;            // rows of a thread; it has 4 columns
    static constexpr int ROWS = kRT / (NB / 4) * TR;  // rows of a tile
    static constexpr int WR = ROWS / 4;             // rows of a warp
    static constexpr int KC = F ? 16 : 8;           // columns of a chunk
    static constexpr int S = 3;                     // chunks in flight
    static constexpr int AT = S * KC * ROWS, BT = S * KC * NB;  // operand buffers; also W and the block inverse
    static_assert(AT >= NB * ROWS && BT >= NB * NB, "buffers are used twice");
};

template <typename T, int TR>
__device__ __forceinline__ void load_rows(const T *p, T (&v)[TR]) {
    if constexpr (sizeof(T) == 8) {
#pragma unroll
        for (int i = 0; i < TR; i += 2) {
            const float4 a = *(const float4 *)(p + i);
            v[i].x = a.x, v[i].y = a.y, v[i + 1].x = a.z, v[i + 1].y = a.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < TR; i++) v[i] = p[i];
    }
}
template <typename T, int TR>
__device__ __forceinline__ void store_rows(T *p, const T (&v)[TR]) {
    if constexpr (sizeof(T) == 8) {
#pragma unroll
        for (int i = 0; i < TR; i += 2) *(float4 *)(p + i) = make_float4(v[i].x, v[i].y, v[i + 1].x, v[i + 1].y);
    } else {
#pragma unroll
        for (int i = 0; i < TR; i++) p[i] = v[i];
    }
}

// column of a thread's four: two pairs 16 apart in complex64, so that the
// warp's 16-byte loads of a pair lie side by side; four in a row in complex128
template <typename T>
__device__ __forceinline__ int root_col(int g, int b) {
    return sizeof(T) == 8 ? 2 * g + (b & 1) + 16 * (b >> 1) : 4 * g + b;
}

// acc[column][row] += A[q][row] B[q][column]
template <typename T, int TR>
__device__ __forceinline__ void root_fma(const T *A, const T *Bm, int kk, int tr, int g, T (&acc)[4][TR]) {
    constexpr int NB = RootShape<T>::NB;
#pragma unroll 4
    for (int q = 0; q < kk; q++) {
        T a[TR], b[4];
        load_rows<T, TR>(A + q * RootShape<T>::ROWS + tr, a);
        if constexpr (sizeof(T) == 8) {
            const float4 u = *(const float4 *)(Bm + q * NB + 2 * g), v = *(const float4 *)(Bm + q * NB + 16 + 2 * g);
            b[0].x = u.x, b[0].y = u.y, b[1].x = u.z, b[1].y = u.w;
            b[2].x = v.x, b[2].y = v.y, b[3].x = v.z, b[3].y = v.w;
        } else {
#pragma unroll
            for (int z = 0; z < 4; z++) b[z] = Bm[q * NB + 4 * g + z];
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < TR; i++) fma_(acc[j][i], a[i], b[j]);
    }
}

template <typename T>
__global__ __launch_bounds__(kRT, 5) void k_sub_root(DevSub D, SubBatch B) {
    extern __shared__ __align__(16) unsigned char sm[];
    using Q = RootShape<T>;
    constexpr int kRows = Q::ROWS, WR = Q::WR, NB = Q::NB, TR = Q::TR, KC = Q::KC, S = Q::S;
    constexpr int NQ = NB / 4, CT = NB / 4, per = 16 / sizeof(T);
    T *As = (T *)sm;       // [S][KC][ROWS]; also W of a tile, [NB][ROWS]
    T *Bs = As + Q::AT;    // [S][KC][NB]; also the inverse block, Bs[a][b] = inverse(b, a)
    __shared__ T col[2][32], mul[2][32], piv[32];
    const int s = blockIdx.x, kk_ = s / B.Lb, k = B.k0 + kk_, l = s % B.Lb;
    const int mp = D.mp, ldc = D.ldc, m = D.m, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    T *C = (T *)B.C + (size_t)s * mp * ldc;
    const T *R = (const T *)D.R + (size_t)k * mp * ldc;
    const double2 *bval = B.bval + (size_t)kk_ * D.n_be * B.Lb + l;
    const int tr = tid / CT * TR, g = tid % CT;
    bool bad = false;
    for (int j = 0; j < mp; j += NB) {
        // the electrode's terms of these columns: one a thread ahead of the products, the rest when they are added
        const int be0 = D.be_ptr[min(j, m)], be1 = D.be_ptr[min(j + NB, m)];
        SubEnt en0{0, -1, 0};
        double2 bv0 = cz(0.0, 0.0);
        if (be0 + tid < be1) {
            en0 = D.be[be0 + tid];
            bv0 = bval[(size_t)(be0 + tid) * B.Lb];
        }
        for (int r0 = j; r0 < mp; r0 += kRows) {
            const bool work = r0 + WR * wid < m;
            // acc = sum - M, M the wavenumber's part
            T acc[4][TR];
#pragma unroll
            for (int b = 0; b < 4; b++) {
                load_rows<T, TR>(R + (size_t)(j + root_col<T>(g, b)) * ldc + r0 + tr, acc[b]);
#pragma unroll
                for (int a = 0; a < TR; a++) acc[b][a] = neg_(acc[b][a]);
            }
            const int nch = j / KC;
            auto fetch = [&](int ch) {
                if (ch < nch) {
                    T *a = As + (ch % S) * KC * kRows, *b = Bs + (ch % S) * KC * NB;
                    const T *src = C + (size_t)ch * KC * ldc;
                    // rows beyond the matrix are read (ldc covers them) and not stored
                    for (int q = tid; q < KC * kRows / per; q += kRT) {
                        const int c = q / (kRows / per), o = (q % (kRows / per)) * per;
                        cp_async16(a + c * kRows + o, src + (size_t)c * ldc + r0 + o);
                    }
                    for (int q = tid; q < KC * NB / per; q += kRT) {
                        const int c = q / (NB / per), o = (q % (NB / per)) * per;
                        cp_async16(b + c * NB + o, src + (size_t)c * ldc + j + o);
                    }
                }
                cp_commit();
            };
#pragma unroll
            for (int q = 0; q < S - 1; q++) fetch(q);
            for (int ch = 0; ch < nch; ch++) {
                cp_wait<S - 2>();
                __syncthreads();
                fetch(ch + S - 1);  // into the buffer that every warp left before this barrier
                if (work) root_fma<T, TR>(As + (ch % S) * KC * kRows, Bs + (ch % S) * KC * NB, KC, tr, g, acc);
            }
            cp_wait<0>();
            __syncthreads();
            if (r0 != j) {  // the inverse of the diagonal block, for the panel
                for (int q = tid; q < NB * NB / per; q += kRT) {
                    const int c = q / (NB / per), o = (q % (NB / per)) * per;
                    cp_async16(Bs + c * NB + o, C + (size_t)(j + c) * ldc + j + o);
                }
                cp_commit();
            }
            // W = M - sum, then the electrode's terms
#pragma unroll
            for (int b = 0; b < 4; b++) {
#pragma unroll
                for (int a = 0; a < TR; a++) acc[b][a] = neg_(acc[b][a]);
                store_rows<T, TR>(As + root_col<T>(g, b) * kRows + tr, acc[b]);
            }
            __syncthreads();
            auto add_term = [&](const SubEnt &en, double2 v) {
                if (en.lr < r0 || en.lr >= r0 + kRows) return;
                T &d = As[(en.lc - j) * kRows + en.lr - r0];
                d = from_<T>(cz((double)d.x + v.x, (double)d.y + v.y));
            };
            add_term(en0, bv0);
            for (int q = be0 + kRT + tid; q < be1; q += kRT) add_term(D.be[q], bval[(size_t)q * B.Lb]);
            cp_wait<0>();
            __syncthreads();
            if (r0 == j) {
                // Diagonal block, L D L^T with the inverse of L beside it: per column the
                // multipliers a_ip / d update both, one barrier; the rows of the inverse
                // are scaled by 1 / sqrt(d) at the end, all at once.  Warp w has the
                // columns w, w + 4, ...; lane = row, in complex128 the lower half of the
                // warp on the block, the upper on the inverse.
                constexpr bool split = NB == 16;
                const int row = lane & (NB - 1), half = split ? lane >> 4 : 0;
                T a[NQ], x[split ? 1 : NQ];
#pragma unroll
                for (int q = 0; q < NQ; q++) {
                    T one = zero_<T>();
                    if (row == 4 * q + wid) one.x = 1;
                    a[q] = half ? one : As[(4 * q + wid) * kRows + row];
                    if constexpr (!split) x[q] = one;
                }
#pragma unroll
                for (int q = 0; q < NQ; q++)
#pragma unroll
                    for (int ww = 0; ww < 4; ww++) {
                        const int p = 4 * q + ww, buf = p & 1;
                        if (wid == ww) {
                            const T d = shfl_(a[q], p), raw = split ? shfl_(a[q], row) : a[q];
                            if (is_bad(d)) bad = true;
                            const T m1 = mul_(raw, rcp_(d));
                            if (!half) {
                                col[buf][row] = raw;
                                mul[buf][row] = row > p ? m1 : zero_<T>();
                                if (row == p) piv[p] = d;
                            }
                        }
                        __syncthreads();
                        const T mi = mul[buf][row];
#pragma unroll
                        for (int z = 0; z < NQ; z++) {
                            const int c = 4 * z + wid;
                            if constexpr (split) {
                                const T xp = shfl_(a[z], 16 + p);
                                T f = c > p ? col[buf][c] : zero_<T>();
                                if (half) f = xp;
                                fms_(a[z], mi, f);
                            } else {
                                if (z >= q && c > p) fms_(a[z], mi, col[buf][c]);
                                if (z <= q) fms_(x[z], mi, shfl_(x[z], p));
                            }
                        }
                    }
                const T iv = rsqrt_(piv[row]);
                if (!split || half) {
#pragma unroll
                    for (int q = 0; q < NQ; q++) {
                        const int c = 4 * q + wid;
                        const T v = row >= c ? mul_(split ? a[q] : x[split ? 0 : q], iv) : zero_<T>();
                        Bs[c * NB + row] = v;
                        C[(size_t)(j + c) * ldc + j + row] = v;
                    }
                }
                __syncthreads();
            }
            // C_ij = W C_jj^-T
            if (r0 + WR * (wid + 1) > j + NB && r0 + WR * wid < mp) {
#pragma unroll
                for (int b = 0; b < 4; b++)
#pragma unroll
                    for (int a = 0; a < TR; a++) acc[b][a] = zero_<T>();
                if (work) root_fma<T, TR>(As, Bs, NB, tr, g, acc);
                if (r0 + tr >= j + NB && r0 + tr < mp) {
#pragma unroll
                    for (int b = 0; b < 4; b++)
                        store_rows<T, TR>(C + (size_t)(j + root_col<T>(g, b)) * ldc + r0 + tr, acc[b]);
                }
            }
            __syncthreads();
        }
    }
    if (D.kbad[k]) {
        if (tid == 0) atomicCAS(&B.status[s], 0, D.kbad[k]);
    } else if (bad) {
        atomicCAS(&B.status[s], 0, 28);
    }
}

// ------------------------------------------------------------------- solves
// x = (C C^T)^-1 u of one system's root, one block per system.  The vector stays in
// shared memory, which limits the root (root_max): larger ones keep the band.
constexpr int kST = 256;

template <typename T>
constexpr int root_max() {  // beside t and part, of the 48 KB that a launch gets without asking
    return 48 * 1024 / (int)sizeof(T) - RootShape<T>::NB - 8 * 33;
}

template <typename T>
__global__ __launch_bounds__(kST) void k_sub_root_solve(DevSub D, SubBatch B, int unit, const int *nprev) {
    extern __shared__ __align__(16) unsigned char sm[];
    constexpr int NB = RootShape<T>::NB, CW = NB / 8;  // columns of a warp
    T *v = (T *)sm;  // [mp]
    __shared__ T t[NB], part[8][33];
    chain_wait();
    if (nprev && *nprev == 0) return;
    const int s = blockIdx.x, kk = s / B.Lb, l = s % B.Lb;
    if (B.kact && !B.kact[kk]) return;
    const int mp = D.mp, ldc = D.ldc, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const T *C = (const T *)B.C + (size_t)s * mp * ldc;
    const T *Y = (const T *)B.Y + ((size_t)kk * D.n + D.nI) * B.Lb + l;
    const T *U = (const T *)B.U + ((size_t)kk * D.szU + D.root_u0) * B.Lb + l;
    T *Z = (T *)B.Z + ((size_t)kk * D.n + D.nI) * B.Lb + l;
    for (int i = tid; i < mp; i += kST) {
        T u = zero_<T>();
        if (i < D.m) {
            u = Y[(size_t)i * B.Lb];
            const int x = D.root_inv[i];
            if (x >= 0 && (!unit || D.root_live)) {
                const T w = U[(size_t)x * B.Lb];
                u.x += w.x;
                u.y += w.y;
            }
        }
        v[i] = u;
    }
    __syncthreads();
    for (int j = 0; j < mp; j += NB) {
        // y_j = C_jj^-1 v_j: warp w takes CW columns of the inverse, lane = row
        T p = zero_<T>();
#pragma unroll
        for (int q = 0; q < CW; q++) {
            const int c = wid * CW + q;
            if (lane >= c && lane < NB) fma_(p, C[(size_t)(j + c) * ldc + j + lane], v[j + c]);
        }
        part[wid][lane] = p;
        __syncthreads();
        if (tid < NB) {
            T y = zero_<T>();
#pragma unroll
            for (int q = 0; q < 8; q++) {
                y.x += part[q][lane].x;
                y.y += part[q][lane].y;
            }
            v[j + lane] = y;
            t[lane] = y;
        }
        __syncthreads();
        for (int i = j + NB + tid; i < mp; i += kST) {
            T a = v[i];
#pragma unroll 8
            for (int c = 0; c < NB; c++) fms_(a, C[(size_t)(j + c) * ldc + i], t[c]);
            v[i] = a;
        }
        __syncthreads();
    }
    for (int j = mp - NB; j >= 0; j -= NB) {
        // t_c = y_c - sum_i C(i, c) x_i: CW columns a warp
#pragma unroll
        for (int q = 0; q < CW; q++) {
            const int c = wid * CW + q;
            T a = zero_<T>();
            for (int i = j + NB + lane; i < mp; i += 32) fma_(a, C[(size_t)(j + c) * ldc + i], v[i]);
            a = warp_sum_(a);
            if (lane == 0) {
                t[c].x = v[j + c].x - a.x;
                t[c].y = v[j + c].y - a.y;
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < CW; q++) {
            const int c = wid * CW + q;
            T a = zero_<T>();
            if (lane >= c && lane < NB) fma_(a, C[(size_t)(j + c) * ldc + j + lane], t[lane]);
            a = warp_sum_(a);
            if (lane == 0) v[j + c] = a;
        }
        __syncthreads();
    }
    for (int i = tid; i < D.m; i += kST) Z[(size_t)i * B.Lb] = v[i];
}

// Up the tree: b_E (own right-hand sides and the children's updates) goes to
// W, the update rows U = (children's updates) - G^T b_E to the parent.  One
// block per tile of update rows x electrodes.  unit: kompab's right-hand sides,
// zero but at the electrodes, so only the fronts above an electrode take part and
// the others' rows of W and U are not read.
template <typename T>
__global__ __launch_bounds__(256) void k_sub_up(DevSub D, SubBatch B, int t0, int unit, const int *nprev) {
    constexpr int E = Tile<T>::E, M = Tile<T>::M, P = Tile<T>::P;
    __shared__ __align__(16) T A[kKT * P], Bm[kKT * P];
    __shared__ int se[kSubCh][kSubEMax], sr[kSubCh][E];
    const int kk = blockIdx.z, k = B.k0 + kk;
    const SubTile tl = (unit ? D.tV : D.tU)[t0 + blockIdx.x];
    const SubFront &t = D.fr[tl.front];
    const int e = t.e, r = t.r, nch = t.nch, from = unit ? t.live : -1, i0 = tl.ti * E, l0 = blockIdx.y * E, L = B.Lb, nl = min(E, L - l0);
    const T *G = (const T *)D.G + (size_t)k * D.szG + t.oG;
    const T *__restrict__ Y = (const T *)B.Y + ((size_t)kk * D.n + t.nd0) * L + l0;
    T *__restrict__ W = (T *)B.W + ((size_t)kk * D.n + t.nd0) * L + l0;
    T *Uk = (T *)B.U + (size_t)kk * D.szU * L + l0;
    for (int q = threadIdx.x; q < nch * kSubEMax; q += 256) {
        const int c = q / kSubEMax, o = q % kSubEMax;
        if (o < e) se[c][o] = D.inv[t.inv[c] + o];
    }
    for (int q = threadIdx.x; q < nch * E; q += 256) {
        const int c = q / E, o = q % E;
        sr[c][o] = i0 + o < r ? D.inv[t.inv[c] + e + i0 + o] : -1;
    }
    chain_wait();
    if (nprev && *nprev == 0) return;
    if (B.kact && !B.kact[kk]) return;
    __syncthreads();
    Operand<T> a, b;
    const int col = b.col();
    auto load_b = [&](int p) {
        b.load(Y + (size_t)p * L, L, e - p, nl);
        for (int c = 0; c < nch; c++) {
            if (!(from >> c & 1)) continue;
            const T *U = Uk + (size_t)t.cu[c] * L + col;
            T g[Operand<T>::N];
#pragma unroll
            for (int z = 0; z < Operand<T>::N; z++) {
                const int q = p + b.row(z), x = q < e && col < nl ? se[c][q] : -1;
                g[z] = x >= 0 ? U[(size_t)x * L] : zero_<T>();
            }
#pragma unroll
            for (int z = 0; z < Operand<T>::N; z++) {
                b.v[z].x += g[z].x;
                b.v[z].y += g[z].y;
            }
        }
    };
    a.load(G + i0, r, e, r - i0);
    load_b(0);
    // the children's updates of this thread's results
    Result<T> acc, sum;
    acc.clear();
    sum.clear();
    const int tr = acc.tr(), tc = acc.tc();
    const bool work = i0 + acc.warp_row() < r;
    for (int c = 0; c < nch; c++) {
        if (!(from >> c & 1)) continue;
        const T *U = Uk + (size_t)t.cu[c] * L;
#pragma unroll
        for (int i = 0; i < M; i++) {
            const int x = sr[c][tr + i];
#pragma unroll
            for (int j = 0; j < M; j++)
                if (x >= 0 && tc + j < nl) {
                    const T v = U[(size_t)x * L + tc + j];
                    sum.v[i][j].x += v.x;
                    sum.v[i][j].y += v.y;
                }
        }
    }
    for (int p = 0; p < e; p += kKT) {
        a.store(A);
        b.store(Bm);
        if (tl.ti == 0) {
#pragma unroll
            for (int z = 0; z < Operand<T>::N; z++)
                if (p + b.row(z) < e && col < nl) W[(size_t)(p + b.row(z)) * L + col] = b.v[z];
        }
        __syncthreads();
        if (p + kKT < e) {
            a.load(G + (size_t)(p + kKT) * r + i0, r, e - p - kKT, r - i0);
            load_b(p + kKT);
        }
        if (work) acc.multiply(A, Bm, min(kKT, e - p));
        __syncthreads();
    }
    T *U = Uk + (size_t)t.u0 * L;
#pragma unroll
    for (int i = 0; i < M; i++)
#pragma unroll
        for (int j = 0; j < M; j++)
            if (i0 + tr + i < r && tc + j < nl) {
                T v = sum.v[i][j];
                v.x -= acc.v[i][j].x;
                v.y -= acc.v[i][j].y;
                U[(size_t)(i0 + tr + i) * L + tc + j] = v;
            }
}

// Down the tree: x_E = F11^-1 b_E - G x_R, one block per tile of rows x
// electrodes
template <typename T>
__global__ __launch_bounds__(256) void k_sub_down(DevSub D, SubBatch B, int t0, int unit, const int *nprev) {
    constexpr int E = Tile<T>::E, M = Tile<T>::M, P = Tile<T>::P, kIdx = 512;
    __shared__ __align__(16) T A[kKT * P], Bm[kKT * P];
    __shared__ int sidx[kIdx];
    const int kk = blockIdx.z, k = B.k0 + kk;
    const SubTile tl = D.tD[t0 + blockIdx.x];
    const SubFront &t = D.fr[tl.front];
    const int e = t.e, r = t.r, i0 = tl.ti * E, l0 = blockIdx.y * E, L = B.Lb, nl = min(E, L - l0);
    const T *F = (const T *)D.F + (size_t)k * D.szF + t.oF, *G = (const T *)D.G + (size_t)k * D.szG + t.oG;
    const T *W = (const T *)B.W + ((size_t)kk * D.n + t.nd0) * L + l0;
    T *Zk = (T *)B.Z + (size_t)kk * D.n * L + l0;
    const int32_t *rows = D.rows + t.rows0;
    for (int q = threadIdx.x; q < min(r, kIdx); q += 256) sidx[q] = rows[q];
    chain_wait();
    if (nprev && *nprev == 0) return;
    if (B.kact && !B.kact[kk]) return;
    __syncthreads();
    Operand<T> a, b;
    Result<T> acc;
    acc.clear();
    const int tr = acc.tr(), tc = acc.tc();
    const bool work = i0 + acc.warp_row() < e;
    // chunks: first the columns of G, then those of F11^-1
    const int nr = (r + kKT - 1) / kKT, nc = nr + (unit && !t.live ? 0 : (e + kKT - 1) / kKT);
    auto load = [&](int ch) {
        if (ch < nr) {
            const int p = ch * kKT;
            a.load_t(G + (size_t)i0 * r + p, r, e - i0, r - p);
#pragma unroll
            for (int z = 0; z < Operand<T>::N; z++) {
                const int q = p + b.row(z);
                b.v[z] = zero_<T>();
                if (q < r && b.col() < nl) b.v[z] = Zk[(size_t)(q < kIdx ? sidx[q] : rows[q]) * L + b.col()];
            }
        } else {
            const int p = (ch - nr) * kKT;
            a.load(F + (size_t)p * e + i0, e, e - p, e - i0);
            b.load(W + (size_t)p * L, L, e - p, nl);
        }
    };
    if (nc > 0) load(0);
    for (int ch = 0; ch < nc; ch++) {
        if (ch < nr) a.store_t(A);
        else a.store(A);
        b.store(Bm);
        __syncthreads();
        if (ch + 1 < nc) load(ch + 1);
        if (ch == nr) {
#pragma unroll
            for (int i = 0; i < M; i++)
#pragma unroll
                for (int j = 0; j < M; j++) acc.v[i][j] = neg_(acc.v[i][j]);
        }
        if (work) acc.multiply(A, Bm, ch < nr ? min(kKT, r - ch * kKT) : min(kKT, e - (ch - nr) * kKT));
        __syncthreads();
    }
    T *Z = Zk + (size_t)t.nd0 * L;
#pragma unroll
    for (int i = 0; i < M; i++)
#pragma unroll
        for (int j = 0; j < M; j++)
            if (i0 + tr + i < e && tc + j < nl)
                Z[(size_t)(i0 + tr + i) * L + tc + j] = nc > nr ? acc.v[i][j] : neg_(acc.v[i][j]);
}

// The same two sweeps for the upper levels, whose fronts are too few to fill the
// chip with tiles: a block has kFewR rows x 32 electrodes, its eight warps take
// every eighth step of the depth and add up at the end.  No staging of the
// vectors (a warp reads a row of 32 electrodes once), one barrier before and one
// after the products, and the factor's rows are read before the chain's wait (they
// are older than its predecessor).  A tile of 32 x 32 takes ten chunks of the
// depth one after the other, 2 us each, at the top of config 2's tree (36 tiles).
constexpr int kFewR = 8, kFewSplit = Tile<float2>::E / kFewR;  // rows, blocks of a tile
struct Few {
    static constexpr int D = 128;                    // depth of a piece of the factor's rows in shared memory
    static constexpr int P = kFewR + 2;              // its pitch
    float2 a[D * P], red[8][kFewR][32];
    __device__ __forceinline__ void put(int q, int ri, float2 v) { a[q * P + ri] = v; }
    // s += (row q of the piece)^T b
    __device__ __forceinline__ void add(float2 (&s)[kFewR], int q, float2 b) const {
#pragma unroll
        for (int ri = 0; ri < kFewR; ri += 2) {
            float2 v[2];
            load2(a + q * P + ri, v);
            fma_(s[ri], v[0], b);
            fma_(s[ri + 1], v[1], b);
        }
    }
    // the block's sum in row threadIdx / 32
    __device__ __forceinline__ float2 sum(const float2 (&s)[kFewR]) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
        for (int ri = 0; ri < kFewR; ri++) red[w][ri][lane] = s[ri];
        __syncthreads();
        float2 v = red[0][w][lane];
#pragma unroll
        for (int z = 1; z < 8; z++) {
            v.x += red[z][w][lane].x;
            v.y += red[z][w][lane].y;
        }
        return v;
    }
};

__global__ __launch_bounds__(256) void k_sub_up_few(DevSub D, SubBatch B, int t0, int unit, const int *nprev) {
    constexpr int E = Tile<float2>::E;
    __shared__ __align__(16) Few sh;
    __shared__ int se[kSubCh][kSubEMax];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int kk = blockIdx.z, k = B.k0 + kk, L = B.Lb, col = blockIdx.y * 32 + lane;
    const SubTile tl = (unit ? D.tV : D.tU)[t0 + blockIdx.x / kFewSplit];
    const SubFront &t = D.fr[tl.front];
    const int e = t.e, r = t.r, nch = t.nch, from = unit ? t.live : -1;
    const int i0 = tl.ti * E + blockIdx.x % kFewSplit * kFewR;
    if (i0 > 0 && i0 >= r) return;
    const float2 *G = (const float2 *)D.G + (size_t)k * D.szG + t.oG;
    for (int q = threadIdx.x; q < nch * kSubEMax; q += 256) {
        const int c = q / kSubEMax, o = q % kSubEMax;
        if (o < e) se[c][o] = D.inv[t.inv[c] + o];
    }
    int x[kSubCh];  // the children's rows of this thread's result
#pragma unroll
    for (int c = 0; c < kSubCh; c++) x[c] = c < nch && i0 + w < r && (from >> c & 1) ? D.inv[t.inv[c] + e + i0 + w] : -1;
    for (int q = threadIdx.x / kFewR; q < e; q += 256 / kFewR) {  // e <= kSubEMax <= Few::D
        const int ri = threadIdx.x % kFewR;
        sh.put(q, ri, i0 + ri < r ? G[(size_t)q * r + i0 + ri] : zero_<float2>());
    }
    chain_wait();
    if (nprev && *nprev == 0) return;
    if (B.kact && !B.kact[kk]) return;
    __syncthreads();
    const float2 *Y = (const float2 *)B.Y + ((size_t)kk * D.n + t.nd0) * L + col;
    float2 *W = (float2 *)B.W + ((size_t)kk * D.n + t.nd0) * L + col;
    float2 *U = (float2 *)B.U + (size_t)kk * D.szU * L + col;
    float2 s[kFewR], own = zero_<float2>();
#pragma unroll
    for (int ri = 0; ri < kFewR; ri++) s[ri] = zero_<float2>();
    if (col < L) {
        constexpr int N = kSubEMax / 8;
        float2 b[N];
#pragma unroll
        for (int z = 0; z < N; z++) b[z] = w + 8 * z < e ? Y[(size_t)(w + 8 * z) * L] : zero_<float2>();
#pragma unroll
        for (int c = 0; c < kSubCh; c++) {
            if (c >= nch || !(from >> c & 1)) continue;
            const float2 *Uc = U + (size_t)t.cu[c] * L;
            float2 g[N];
#pragma unroll
            for (int z = 0; z < N; z++) {
                const int y = w + 8 * z < e ? se[c][w + 8 * z] : -1;
                g[z] = y >= 0 ? Uc[(size_t)y * L] : zero_<float2>();
            }
            if (x[c] >= 0) {
                const float2 v = Uc[(size_t)x[c] * L];
                own.x += v.x;
                own.y += v.y;
            }
#pragma unroll
            for (int z = 0; z < N; z++) {
                b[z].x += g[z].x;
                b[z].y += g[z].y;
            }
        }
#pragma unroll
        for (int z = 0; z < N; z++)
            if (w + 8 * z < e) {
                if (i0 == 0) W[(size_t)(w + 8 * z) * L] = b[z];
                sh.add(s, w + 8 * z, b[z]);
            }
    }
    const float2 v = sh.sum(s);
    if (i0 + w < r && col < L) {
        own.x -= v.x;
        own.y -= v.y;
        U[(size_t)(t.u0 + i0 + w) * L] = own;
    }
}

__global__ __launch_bounds__(256) void k_sub_down_few(DevSub D, SubBatch B, int t0, int unit, const int *nprev) {
    constexpr int E = Tile<float2>::E, N = Few::D / 8;
    __shared__ __align__(16) Few sh;
    __shared__ int at[Few::D];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int kk = blockIdx.z, k = B.k0 + kk, L = B.Lb, col = blockIdx.y * 32 + lane;
    const SubTile tl = D.tD[t0 + blockIdx.x / kFewSplit];
    const SubFront &t = D.fr[tl.front];
    const int e = t.e, r = t.r, i0 = tl.ti * E + blockIdx.x % kFewSplit * kFewR;
    if (i0 >= e) return;
    const float2 *F = (const float2 *)D.F + (size_t)k * D.szF + t.oF, *G = (const float2 *)D.G + (size_t)k * D.szG + t.oG;
    const float2 *W = (const float2 *)B.W + ((size_t)kk * D.n + t.nd0) * L + col;
    float2 *Z = (float2 *)B.Z + (size_t)kk * D.n * L + col;
    const int32_t *rows = D.rows + t.rows0;
    const int depth = r + (unit && !t.live ? 0 : e);
    float2 s[kFewR];
#pragma unroll
    for (int ri = 0; ri < kFewR; ri++) s[ri] = zero_<float2>();
    for (int p = 0; p < depth; p += Few::D) {  // G's columns (negative), then F11^-1's
        const int n = min(Few::D, depth - p);
        if (p) __syncthreads();
        for (int q = lane; q < n; q += 32) {  // one row a warp
            float2 v = zero_<float2>();
            if (i0 + w < e) v = p + q < r ? neg_(G[(size_t)(i0 + w) * r + p + q]) : F[(size_t)(i0 + w) * e + p + q - r];
            sh.put(q, w, v);
        }
        for (int q = threadIdx.x; q < n; q += 256)
            if (p + q < r) at[q] = rows[p + q];
        if (!p) {
            chain_wait();
            if (nprev && *nprev == 0) return;
            if (B.kact && !B.kact[kk]) return;
        }
        __syncthreads();
        float2 b[N];
#pragma unroll
        for (int z = 0; z < N; z++) {
            const int q = w + 8 * z;
            b[z] = zero_<float2>();
            if (q < n && col < L) b[z] = p + q < r ? Z[(size_t)at[q] * L] : W[(size_t)(p + q - r) * L];
        }
#pragma unroll
        for (int z = 0; z < N; z++)
            if (w + 8 * z < n) sh.add(s, w + 8 * z, b[z]);
    }
    const float2 v = sh.sum(s);
    if (i0 + w < e && col < L) Z[(size_t)(t.nd0 + i0 + w) * L] = v;
}

// -------------------------------------------------- vectors of a rectangle
// Right-hand sides from the rows of src ([eanz][n]), scaled by fk
template <typename T>
__global__ void k_sub_rhs(DevProblem P, DevSub D, SubBatch B, const double2 *__restrict__ src, int keep) {
    const int l = blockIdx.y * 32 + (threadIdx.x & 31), p = blockIdx.x * 8 + (threadIdx.x >> 5), kk = blockIdx.z;
    if (l >= B.Lb || p >= D.n) return;
    const int i = D.node[p];
    double2 v = P.dirichlet[i] ? cz(0.0, 0.0) : src[(size_t)(B.l0 + l) * P.n + i];
    const size_t at = ((size_t)kk * D.n + p) * B.Lb + l;
    if (v.x != 0.0 || v.y != 0.0) {  // the adjoint sources are zero but at the electrodes
        const double f = D.fk[(size_t)(B.k0 + kk) * P.n + i];
        v = cz(v.x * f, v.y * f);
    }
    if (keep) B.Bt[at] = v;
    ((T *)B.Y)[at] = from_<T>(v);
}

// kompab's right-hand side of electrode l at node i (src/kompab.f90:180-190):
// the unit sink at the electrode, the fictitious sink, zero on Dirichlet nodes
__device__ __forceinline__ double unit_rhs(const DevProblem &P, int el, int i, int lsink, int nsink) {
    if (P.dirichlet[i]) return 0.0;
    if (lsink && i == nsink) return 1.0;
    return i == P.enr0[el] ? -1.0 : 0.0;
}

// ... scaled by fk, into a zeroed Y: one thread per system
template <typename T>
__global__ void k_sub_unit_rhs(DevProblem P, DevSub D, SubBatch B, int lsink, int nsink) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= B.Kb * B.Lb) return;
    const int kk = s / B.Lb, l = s % B.Lb, el = B.l0 + l;
    const int nodes[2] = {P.enr0[el], lsink ? nsink : -1};
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int i = nodes[q];
        if (i < 0 || i >= P.n) continue;
        const double v = unit_rhs(P, el, i, lsink, nsink) * D.fk[(size_t)(B.k0 + kk) * P.n + i];
        ((T *)B.Y)[((size_t)kk * D.n + D.pos[i]) * B.Lb + l] = from_<T>(cz(v, 0.0));
    }
}

// Y = b - A x in FP64 (rounded to complex64 at the end): one warp per row, the
// electrodes across its lanes, so the matrix entries are one broadcast load.
// Bound by the FP64 pipe: 36 fused multiply-adds a node and system.  unit: b
// is kompab's, else B.Bt.
__global__ __launch_bounds__(256) void k_sub_residual(DevProblem P, DevSub D, SubBatch B, int unit, int lsink,
                                                      int nsink, const int *nprev) {
    chain_wait();
    if (nprev && *nprev == 0) return;
    const int kk = blockIdx.z, k = B.k0 + kk, L = B.Lb;
    if (!B.kact[kk]) return;
    const int l = blockIdx.y * 32 + (threadIdx.x & 31), p = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (l >= L || p >= D.n) return;
    const int i = D.node[p];
    const double2 *As = D.As + (size_t)k * P.nnz;
    const double2 *X = B.X + (size_t)kk * D.n * L + l;
    double2 acc = cz(0.0, 0.0);
    for (int q = P.fptr[i]; q < P.fptr[i + 1]; q++) fma_(acc, As[P.fidx[q]], X[(size_t)D.fcolpos[q] * L]);
    if (p >= D.nI) {
        const double2 *bv = B.bval + (size_t)kk * D.n_be * L + l;
        for (int q = D.rb_ptr[p - D.nI]; q < D.rb_ptr[p - D.nI + 1]; q++)
            fma_(acc, bv[(size_t)D.rb_ent[q] * L], X[(size_t)D.rb_pos[q] * L]);
    }
    const size_t at = ((size_t)kk * D.n + p) * L + l;
    double2 b = cz(0.0, 0.0);
    if (!unit) {
        b = B.Bt[at];
    } else {
        const double v = unit_rhs(P, B.l0 + l, i, lsink, nsink);
        if (v != 0.0) b.x = v * D.fk[(size_t)k * P.n + i];
    }
    ((float2 *)B.Y)[at] = narrow(cz(b.x - acc.x, b.y - acc.y));
}

constexpr int kAccRows = 128;

// X (+)= Z with the largest entries of both per system (as bit patterns)
__global__ __launch_bounds__(256) void k_sub_accumulate(DevSub D, SubBatch B, int first, const int *nprev) {
    chain_wait();
    if (nprev && *nprev == 0) return;
    const int kk = blockIdx.z, L = B.Lb;
    if (!first && !B.kact[kk]) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, l = blockIdx.y * 32 + lane;
    const bool on = l < L && (first || B.active[kk * L + l]);
    float mz = 0.f;
    bool nan = false;
    unsigned long long mx = 0ull;
    if (on) {
        const float2 *__restrict__ Z = (const float2 *)B.Z + (size_t)kk * D.n * L + l;
        double2 *__restrict__ X = B.X + (size_t)kk * D.n * L + l;
        const int p0 = blockIdx.x * kAccRows + w, p1 = min(D.n, (int)(blockIdx.x + 1) * kAccRows);
        for (int p = p0; p < p1; p += 32) {
            float2 z[4];
            double2 x[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (p + 8 * q < p1) {
                    z[q] = Z[(size_t)(p + 8 * q) * L];
                    if (!first) x[q] = X[(size_t)(p + 8 * q) * L];
                }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (p + 8 * q < p1) {
                    const double2 zd = widen(z[q]), v = first ? zd : cz(x[q].x + zd.x, x[q].y + zd.y);
                    X[(size_t)(p + 8 * q) * L] = v;
                    mz = fmaxf(mz, fmaxf(fabsf(z[q].x), fabsf(z[q].y)));
                    nan = nan || z[q].x != z[q].x || z[q].y != z[q].y;  // fmaxf drops them
                    mx = max(mx, max(abs_bits(v.x), abs_bits(v.y)));
                }
        }
    }
    __shared__ float sz[8][32];
    __shared__ unsigned long long sx[8][32];
    sz[w][lane] = nan ? INFINITY : mz;
    sx[w][lane] = mx;
    __syncthreads();
    if (w == 0 && on) {
        mz = sz[0][lane];
        for (int q = 1; q < 8; q++) {
            mz = fmaxf(mz, sz[q][lane]);
            mx = max(mx, sx[q][lane]);
        }
        atomicMax(&B.mz[kk * L + l], abs_bits(widen(mz)));
        atomicMax(&B.mx[kk * L + l], mx);
    }
}

// A system stops once its correction is at most tol times its solution; one
// block per wavenumber counts those that go on, the last block passes the sum on
// (SubStop).
__global__ __launch_bounds__(256) void k_sub_stop(SubBatch B, int first, double tol, const int *nprev, SubStop stop) {
    chain_wait();
    if (nprev && *nprev == 0) return;
    const int kk = blockIdx.x, L = B.Lb;
    const int it = stop.steps ? stop.cnt[kRefineCap].n : 0;
    RefineCount *cnt = stop.cnt ? stop.cnt + it : nullptr;
    int count = 0;
    if (first || B.kact[kk]) {
        for (int l = threadIdx.x; l < L; l += blockDim.x) {
            const int s = kk * L + l;
            const double mz = __longlong_as_double((long long)B.mz[s]), mx = __longlong_as_double((long long)B.mx[s]);
            B.mz[s] = 0ull;
            B.mx[s] = 0ull;
            int act = first ? 1 : B.active[s];
            if (!act) continue;
            if (!first && !(mz > tol * mx)) act = 0;
            if (cnt && mx > 0.0)
                atomicMax((unsigned long long *)&cnt->z, (unsigned long long)__double_as_longlong(mz / mx));
            if (!isfinite(mz) || !isfinite(mx)) {
                atomicCAS(&B.status[s], 0, 28);
                act = 0;
            }
            B.active[s] = act;
            count += act;
        }
    }
    __shared__ int tot;
    if (threadIdx.x == 0) tot = 0;
    __syncthreads();
    if (count) atomicAdd(&tot, count);
    __syncthreads();
    if (threadIdx.x != 0) return;
    B.kact[kk] = tot;
    if (!cnt) return;
    if (tot) atomicAdd(&cnt->n, tot);
    __threadfence();
    if (atomicAdd(&cnt->ticket, 1) != (int)gridDim.x - 1) return;
    const int n = atomicAdd(&cnt->n, 0);
    if (stop.left) {
        *(volatile int *)stop.left = n;
        __threadfence_system();
    }
    if (stop.steps) {
        stop.cnt[kRefineCap].n = it + 1;
        cudaGraphSetConditional(stop.loop, n > 0 && it + 1 < stop.steps ? 1 : 0);
    }
}

// out[k][l][node] = sign fk x (src/fem.f90:388-389), through shared memory:
// 32 nodes x 32 electrodes a block; out32 the complex64 hi and lo planes
__global__ __launch_bounds__(256) void k_sub_unpack(DevProblem P, DevSub D, SubBatch B, double sign, double2 *out,
                                                    float2 *out32) {
    __shared__ double2 tile[32][33];
    const int kk = blockIdx.z, k = B.k0 + kk, n0 = blockIdx.x * 32, l0 = blockIdx.y * 32;
    const int a = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int q = w; q < 32; q += 8)
        if (n0 + q < D.n && l0 + a < B.Lb)
            tile[q][a] = B.X[((size_t)kk * D.n + D.pos[n0 + q]) * B.Lb + l0 + a];
    __syncthreads();
    if (n0 + a >= D.n) return;
    const double f = sign * D.fk[(size_t)k * P.n + n0 + a];
    for (int q = w; q < 32; q += 8) {
        if (l0 + q >= B.Lb) continue;
        const double2 x = tile[a][q], v = cz(x.x * f, x.y * f);
        const size_t at = ((size_t)k * P.eanz + B.l0 + l0 + q) * P.n + n0 + a;
        out[at] = v;
        if (out32) {
            const float2 hi = narrow(v);
            const double2 h = widen(hi);
            out32[at] = hi;
            out32[at + (size_t)P.K * P.eanz * P.n] = narrow(cz(v.x - h.x, v.y - h.y));
        }
    }
}

inline unsigned nb(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

template <typename T>
int factor_t(const DevProblem &P, const DevSub &D, const SubPlan &sp, int K, cudaStream_t st) {
    auto bytes = [](int e) { return sizeof(T) * (e * (e | 1) + (e > 32 ? 2 * 32 * 33 : 0)); };
    static std::once_flag once;
    std::call_once(once, [&] {
        cudaFuncSetAttribute(k_sub_pivot<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(Tile<T>::emax));
    });
    int launches = 0;
    for (int lv = 0; lv < sp.nlevel; lv++) {
        const int f0 = sp.level[lv], nf = sp.level[lv + 1] - f0;
        int emax = 1;
        for (int q = f0; q < f0 + nf; q++) emax = std::max(emax, sp.fronts[q].e);
        const int na = sp.lA[lv + 1] - sp.lA[lv], ng = sp.lG[lv + 1] - sp.lG[lv], ns = sp.lS[lv + 1] - sp.lS[lv];
        if (na) chain_launch(k_sub_gather<T>, dim3(na, K), 256, 0, st, D, sp.lA[lv]);
        chain_launch(k_sub_pivot<T>, dim3(nf, K), 256, bytes(emax), st, D, f0, P.nnz);
        if (ng) chain_launch(k_sub_g<T>, dim3(ng, K), 256, 0, st, D, sp.lG[lv]);
        if (ns) chain_launch(k_sub_s<T>, dim3(ns, K), 256, 0, st, D, sp.lS[lv]);
        launches += 1 + (na > 0) + (ng > 0) + (ns > 0);
    }
    k_sub_root_base<T><<<dim3(D.mp, K), 128, 0, st>>>(D);
    if (D.n_root_ent) k_sub_root_ent<T><<<dim3(nb(D.n_root_ent, 128), K), 128, 0, st>>>(D, P.nnz);
    return launches + 2;
}

template <typename T>
size_t root_smem() {
    return sizeof(T) * (RootShape<T>::AT + RootShape<T>::BT);
}

template <typename T>
void root_t(const DevProblem &P, const DevSub &D, const SubBatch &B, const double2 *sigma, cudaStream_t st) {
    static std::once_flag once;
    std::call_once(once, [] {
        cudaFuncSetAttribute(k_sub_root<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)root_smem<T>());
    });
    if (D.n_be) k_sub_bval<<<dim3(nb(D.n_be, 8), nb(B.Lb, 32), B.Kb), 256, 0, st>>>(P, D, B, sigma);
    k_sub_root<T><<<B.Kb * B.Lb, kRT, root_smem<T>(), st>>>(D, B);
}

// Levels with tiles for at most 48 blocks (a third of the 152 SMs) take the kernels
// for few fronts.  Blocks at most against forwards in ms (60x20 line with
// Jacobian / 200x60 / triangle gradient / 300x80 / eight contexts at once): none
// 1.31 9.53 12.23 26.1 16.9, 30 1.28 9.54 12.0 26.1 16.9, 48 1.27 9.40 11.84 25.9
// 16.9, 76 1.25 9.35 11.82 25.9 17.2, 152 1.24 9.35 11.75 25.7 17.2, 608 1.25 9.59
// 12.07 25.7 18.4: they read the vectors four times as often as the tiles do,
// which costs where other work could use the chip.  In complex128 every block is
// FP64-bound and they give nothing (160x50 32.6 -> 32.8), so there the tiles stay.
constexpr int kFewBlocks = 48;

template <typename T>
int apply_t(const DevSub &D, const SubPlan &sp, const SubBatch &B, bool unit, const int *nprev, cudaStream_t st) {
    const bool few = std::is_same<T, float2>::value;
    const int lt = nb(B.Lb, Tile<T>::E);
    const std::vector<int32_t> &up = unit ? sp.lV : sp.lU;
    int launches = 1;
    for (int lv = 0; lv < sp.nlevel; lv++) {
        const int nu = up[lv + 1] - up[lv];
        if (!nu) continue;
        if (few && nu * lt * B.Kb <= kFewBlocks)
            chain_launch(k_sub_up_few, dim3(nu * kFewSplit, lt, B.Kb), 256, 0, st, D, B, up[lv], unit ? 1 : 0,
                         nprev);
        else
            chain_launch(k_sub_up<T>, dim3(nu, lt, B.Kb), 256, 0, st, D, B, up[lv], unit ? 1 : 0, nprev);
        launches++;
    }
    chain_launch(k_sub_root_solve<T>, dim3(B.Kb * B.Lb), kST, sizeof(T) * D.mp, st, D, B, unit ? 1 : 0, nprev);
    for (int lv = sp.nlevel - 1; lv >= 0; lv--) {
        const int nd = sp.lD[lv + 1] - sp.lD[lv];
        if (!nd) continue;
        if (few && nd * lt * B.Kb <= kFewBlocks)
            chain_launch(k_sub_down_few, dim3(nd * kFewSplit, lt, B.Kb), 256, 0, st, D, B, sp.lD[lv],
                         unit ? 1 : 0, nprev);
        else
            chain_launch(k_sub_down<T>, dim3(nd, lt, B.Kb), 256, 0, st, D, B, sp.lD[lv], unit ? 1 : 0, nprev);
        launches++;
    }
    return launches;
}

}  // namespace

void sub_launch_values(const DevProblem &P, const DevSub &D, const double2 *sigma, const double2 *adom,
                       cudaStream_t st) {
    cudaMemsetAsync(D.kbad, 0, sizeof(int) * P.K, st);
    const double *fak_area = (const double *)(adom + (size_t)P.K * P.nnz);
    k_sub_scale<<<nb((size_t)P.K * P.n, 256), 256, 0, st>>>(P, D, sigma, fak_area);
    k_sub_values<<<dim3(nb(P.nnz, 256), P.K), 256, 0, st>>>(P, D, adom);
}

SubShape sub_shape(bool mixed) {
    if (mixed) return {Tile<float2>::leaf, Tile<float2>::emax, Tile<float2>::E};
    return {Tile<double2>::leaf, Tile<double2>::emax, Tile<double2>::E};
}

int sub_root_block(bool mixed) { return mixed ? RootShape<float2>::NB : RootShape<double2>::NB; }
int sub_root_rows(bool mixed) { return mixed ? RootShape<float2>::ROWS : RootShape<double2>::ROWS; }

int sub_root_max(bool mixed) { return mixed ? root_max<float2>() : root_max<double2>(); }

int sub_launch_factor(const DevProblem &P, const DevSub &D, const SubPlan &sp, int K, bool mixed, cudaStream_t st) {
    return mixed ? factor_t<float2>(P, D, sp, K, st) : factor_t<double2>(P, D, sp, K, st);
}

void sub_launch_root(const DevProblem &P, const DevSub &D, const SubBatch &B, const double2 *sigma, bool mixed,
                     cudaStream_t st) {
    mixed ? root_t<float2>(P, D, B, sigma, st) : root_t<double2>(P, D, B, sigma, st);
}

int sub_launch_apply(const DevSub &D, const SubPlan &sp, const SubBatch &B, bool mixed, bool unit, const int *nprev,
                     cudaStream_t st) {
    return mixed ? apply_t<float2>(D, sp, B, unit, nprev, st) : apply_t<double2>(D, sp, B, unit, nprev, st);
}

void sub_launch_rhs(const DevProblem &P, const DevSub &D, const SubBatch &B, bool mixed, int lsink, int nsink,
                    const double2 *src, cudaStream_t st) {
    if (!src) {
        const int ns = B.Kb * B.Lb;
        cudaMemsetAsync(B.Y, 0, (mixed ? sizeof(float2) : sizeof(double2)) * (size_t)ns * D.n, st);
        if (mixed) k_sub_unit_rhs<float2><<<nb(ns, 128), 128, 0, st>>>(P, D, B, lsink, nsink);
        else k_sub_unit_rhs<double2><<<nb(ns, 128), 128, 0, st>>>(P, D, B, lsink, nsink);
        return;
    }
    const dim3 g(nb(D.n, 8), nb(B.Lb, 32), B.Kb);
    if (mixed) k_sub_rhs<float2><<<g, 256, 0, st>>>(P, D, B, src, 1);
    else k_sub_rhs<double2><<<g, 256, 0, st>>>(P, D, B, src, 0);
}

void sub_launch_residual(const DevProblem &P, const DevSub &D, const SubBatch &B, bool unit, int lsink, int nsink,
                         const int *nprev, cudaStream_t st) {
    chain_launch(k_sub_residual, dim3(nb(D.n, 8), nb(B.Lb, 32), B.Kb), 256, 0, st, P, D, B, unit ? 1 : 0, lsink, nsink,
                 nprev);
}

void sub_launch_accumulate(const DevSub &D, const SubBatch &B, bool first, double tol, const int *nprev,
                           const SubStop &stop, cudaStream_t st) {
    chain_launch(k_sub_accumulate, dim3(nb(D.n, kAccRows), nb(B.Lb, 32), B.Kb), 256, 0, st, D, B, first ? 1 : 0, nprev);
    chain_launch(k_sub_stop, dim3(B.Kb), 256, 0, st, B, first ? 1 : 0, tol, nprev, stop);
}

void sub_launch_unpack(const DevProblem &P, const DevSub &D, const SubBatch &B, double sign, double2 *out,
                       float2 *out32, cudaStream_t st) {
    k_sub_unpack<<<dim3(nb(D.n, 32), nb(B.Lb, 32), B.Kb), 256, 0, st>>>(P, D, B, sign, out, out32);
}

}  // namespace crgpu

// Adjoint of the forward block: the exact derivative of a linear functional
// of the voltages, L = sum_i g_i V_i, with respect to the conductivities.
// No single reference routine does this: CRTomo forms the Jacobian with
// src/bsensi.f90 (reciprocity, without the mixed-boundary term) and applies
// J^H in src/update.f90.  Here, with kpot_(k,l) = A_(k,l)^{-1} e_l and
//   V_i = sum_k w_k/pi [(kpot_(k,e2) - kpot_(k,e1))(P4) - (...)(P3)]
// (src/bvolt.f90, src/rtrafo.f90):
//   dL/dsigma_e = -sum_(k,l) w_k/pi lambda_(k,l)^T (dA_(k,l)/dsigma_e) kpot_(k,l),
//   lambda_(k,l) = A_(k,l)^{-1} c_l,  c_l = sum_(i: e2=l) g_i (e_P4 - e_P3)
//                                        - sum_(i: e1=l) g_i (e_P4 - e_P3).
// dA/dsigma_e is the element matrix of src/precal.f90 plus, for elements
// carrying a mixed boundary (src/kompab.f90:112-139), the boundary matrix
// relbg * beta(k, l).
#include "device.cuh"
#include "kernels.h"

namespace crgpu {

static constexpr double kPiA = 3.14159265358979323846264338327950288;

__device__ __forceinline__ void atomic_add_c(double2 *p, double2 v) {
    atomicAdd(&p->x, v.x);
    atomicAdd(&p->y, v.y);
}

// c_l for every electrode l: [eanz][n]
__global__ void k_adj_sources(DevProblem P, const double2 *__restrict__ g, double2 *src) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.nanz) return;
    const int e1 = P.meas[i * 4], e2 = P.meas[i * 4 + 1], e3 = P.meas[i * 4 + 2], e4 = P.meas[i * 4 + 3];
    const double2 gi = g[i];
    const double2 mg = cz(-gi.x, -gi.y);
    const int p3 = e3 >= 0 ? P.enr0[e3] : -1, p4 = e4 >= 0 ? P.enr0[e4] : -1;
    if (e2 >= 0) {
        if (p4 >= 0) atomic_add_c(&src[(size_t)e2 * P.n + p4], gi);
        if (p3 >= 0) atomic_add_c(&src[(size_t)e2 * P.n + p3], mg);
    }
    if (e1 >= 0) {
        if (p4 >= 0) atomic_add_c(&src[(size_t)e1 * P.n + p4], mg);
        if (p3 >= 0) atomic_add_c(&src[(size_t)e1 * P.n + p3], gi);
    }
}

void launch_adjoint_sources(const DevProblem &P, const double2 *g, double2 *src, int lsink, int nsink,
                            cudaStream_t st) {
    (void)lsink;
    (void)nsink;  // the sink enters b, not the measured functional
    cudaMemsetAsync(src, 0, sizeof(double2) * (size_t)P.eanz * P.n, st);
    const int nt = 128;
    if (P.nanz > 0) k_adj_sources<<<(P.nanz + nt - 1) / nt, nt, 0, st>>>(P, g, src);
}

// scaled right-hand side D c_l of item (s, r) (src/scalab.f90 scaling);
// Dirichlet rows keep b = 0 (src/randb.f90)
__global__ void k_adj_rhs(DevProblem P, DevBatch B, int nrhs, const double2 *__restrict__ src) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, item = blockIdx.y;
    if (i >= P.n) return;
    const int s = item / nrhs, r = item % nrhs;
    const int l = (nrhs == 1) ? B.ls[s] : r;
    const double f = B.fak[(size_t)s * P.n + i];
    const double2 v = P.dirichlet[i] ? cz(0.0, 0.0) : src[(size_t)l * P.n + i];
    B.b[(size_t)item * P.n + i] = cz(v.x * f, v.y * f);
}

void launch_adjoint_rhs(const DevProblem &P, const DevBatch &B, int nrhs, const double2 *src, cudaStream_t st) {
    const int nt = 128;
    k_adj_rhs<<<dim3((P.n + nt - 1) / nt, B.nsys * nrhs), nt, 0, st>>>(P, B, nrhs, src);
}

// lambda_(k,l) = D x in the layout of kpot, [K][eanz][n]
__global__ void k_adj_lambda(DevProblem P, DevBatch B, int nrhs, double2 *lambda) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, item = blockIdx.y;
    if (i >= P.n) return;
    const int s = item / nrhs, r = item % nrhs;
    const int k = B.ks[s], l = (nrhs == 1) ? B.ls[s] : r;
    const double f = B.fak[(size_t)s * P.n + i];
    const double2 x = B.x[(size_t)item * P.n + i];
    lambda[((size_t)k * P.eanz + l) * P.n + i] = cz(x.x * f, x.y * f);
}

void launch_adjoint_lambda(const DevProblem &P, const DevBatch &B, int nrhs, double2 *lambda, cudaStream_t st) {
    const int nt = 128;
    k_adj_lambda<<<dim3((P.n + nt - 1) / nt, B.nsys * nrhs), nt, 0, st>>>(P, B, nrhs, lambda);
}

// The gradient's contraction: lanes run over neighbouring elements, whose nodes
// lie side by side in kpot and lambda, the block's warps over the (k, l) pairs;
// an element's matrix stays in registers for a wavenumber, and triangles take 9
// products instead of 16.  FP64 bound: 18 + 12 operations a pair on triangles.
// GB300, 18000 triangles x 832 pairs: 1.78 -> 0.85 ms (one block per element with
// its threads over the pairs read a 32-byte sector for every 16 bytes used).
constexpr int kAdjWarps = 8;

// sum over this warp's pairs of w_k lambda^T K kpot for an element of at most NK nodes
template <int NK>
__device__ __forceinline__ double2 adj_element(const DevProblem &P, const double2 *__restrict__ kpot,
                                               const double2 *__restrict__ lambda, int e, int nk) {
    int nodes[NK];
    bool dir[NK];
#pragma unroll
    for (int q = 0; q < NK; q++) {
        nodes[q] = q < nk ? P.enodes[e * 4 + q] : 0;
        // a Dirichlet node keeps its potential (its value enters the other rows
        // through the moved column, src/randb2.f90); lambda is 0 there
        dir[q] = q >= nk || P.dirichlet[nodes[q]] != 0;
    }
    double2 acc = cz(0.0, 0.0);
    for (int k = 0; k < P.K; k++) {
        const double *Ke = P.elbg + ((size_t)k * P.elanz + e) * 10;
        double K[NK * (NK + 1) / 2];
#pragma unroll
        for (int m = 0; m < NK; m++)
#pragma unroll
            for (int q = 0; q <= m; q++) K[m * (m + 1) / 2 + q] = m < nk ? Ke[m * (m + 1) / 2 + q] : 0.0;
        double2 s = cz(0.0, 0.0);
        const int t0 = k * P.eanz, w = threadIdx.x >> 5;
#pragma unroll 2
        for (int l = (w + kAdjWarps - t0 % kAdjWarps) % kAdjWarps; l < P.eanz; l += kAdjWarps) {
            const size_t base = (size_t)(t0 + l) * P.n;
            double2 kv[NK], lv[NK];
#pragma unroll
            for (int q = 0; q < NK; q++) {
                kv[q] = q < nk ? kpot[base + nodes[q]] : cz(0.0, 0.0);
                lv[q] = dir[q] ? cz(0.0, 0.0) : lambda[base + nodes[q]];
            }
#pragma unroll
            for (int m = 0; m < NK; m++) {
                double2 u = cz(0.0, 0.0);
#pragma unroll
                for (int q = 0; q < NK; q++) {
                    const double a = K[m > q ? m * (m + 1) / 2 + q : q * (q + 1) / 2 + m];
                    u.x = fma(a, kv[q].x, u.x);
                    u.y = fma(a, kv[q].y, u.y);
                }
                s.x = fma(lv[m].x, u.x, s.x);
                s.x = fma(-lv[m].y, u.y, s.x);
                s.y = fma(lv[m].x, u.y, s.y);
                s.y = fma(lv[m].y, u.x, s.y);
            }
        }
        const double w0 = P.swrtr ? P.kwnwi[k] / kPiA : 1.0;
        acc.x = fma(w0, s.x, acc.x);
        acc.y = fma(w0, s.y, acc.y);
    }
    return acc;
}

__global__ __launch_bounds__(32 * kAdjWarps) void k_adj_grad(DevProblem P, const double2 *__restrict__ kpot,
                                                             const double2 *__restrict__ lambda, double2 *grad) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
    const bool in = e < P.elanz;
    const int ee = in ? e : P.elanz - 1, nk = P.etype[ee] == 3 ? 3 : 4;
    double2 acc = __all_sync(0xffffffffu, nk == 3) ? adj_element<3>(P, kpot, lambda, ee, nk)
                                                   : adj_element<4>(P, kpot, lambda, ee, nk);
    __shared__ double2 red[kAdjWarps][32];
    red[w][lane] = acc;
    __syncthreads();
    if (w || !in) return;
    for (int q = 1; q < kAdjWarps; q++) acc = cadd(acc, red[q][lane]);
    grad[e] = cz(-acc.x, -acc.y);
}

// The mixed boundaries that an element carries, added to its entry: one block per
// element, its threads over the pairs (few elements have any; inside k_adj_grad
// the 32 of a side that share a block took 0.2 ms one after the other).
__global__ __launch_bounds__(128) void k_adj_boundary(DevProblem P, const double2 *__restrict__ kpot,
                                                      const double2 *__restrict__ lambda,
                                                      const int32_t *__restrict__ ebnd_ptr,
                                                      const int32_t *__restrict__ ebnd_list, double2 *grad) {
    const int e = blockIdx.x, q0 = ebnd_ptr[e], q1 = ebnd_ptr[e + 1], lane = threadIdx.x & 31;
    if (q0 == q1) return;
    double2 acc = cz(0.0, 0.0);
    for (int q = q0; q < q1; q++) {
        const int rb = ebnd_list[q], n0 = P.bnodes[rb * 2], n1 = P.bnodes[rb * 2 + 1];
        const double b0 = P.relbg[rb * 3], b1 = P.relbg[rb * 3 + 1], b2 = P.relbg[rb * 3 + 2];
        const bool d0 = P.dirichlet[n0] != 0, d1 = P.dirichlet[n1] != 0;
        for (int t = threadIdx.x; t < P.K * P.eanz; t += 128) {
            const size_t base = (size_t)t * P.n;
            const double beta = P.kg[(size_t)t * P.relanz + rb] * (P.swrtr ? P.kwnwi[t / P.eanz] / kPiA : 1.0);
            const double r0 = b0 * beta, r1 = b1 * beta, r2 = b2 * beta;
            const double2 k0 = kpot[base + n0], k1 = kpot[base + n1];
            const double2 l0 = d0 ? cz(0.0, 0.0) : lambda[base + n0], l1 = d1 ? cz(0.0, 0.0) : lambda[base + n1];
            const double2 u0 = cz(r0 * k0.x + r1 * k1.x, r0 * k0.y + r1 * k1.y);
            const double2 u1 = cz(r1 * k0.x + r2 * k1.x, r1 * k0.y + r2 * k1.y);
            acc = cadd(acc, cadd(cmul(l0, u0), cmul(l1, u1)));
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    __shared__ double2 red[4];
    if (lane == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x) return;
    for (int q = 1; q < 4; q++) acc = cadd(acc, red[q]);
    grad[e] = cz(grad[e].x - acc.x, grad[e].y - acc.y);
}

void launch_adjoint_grad(const DevProblem &P, const double2 *kpot, const double2 *lambda, const int32_t *ebnd_ptr,
                         const int32_t *ebnd_list, double2 *grad, cudaStream_t st) {
    if (P.elanz <= 0) return;
    k_adj_grad<<<(P.elanz + 31) / 32, 32 * kAdjWarps, 0, st>>>(P, kpot, lambda, grad);
    k_adj_boundary<<<P.elanz, 128, 0, st>>>(P, kpot, lambda, ebnd_ptr, ebnd_list, grad);
}

}  // namespace crgpu

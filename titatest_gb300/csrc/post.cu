// Wavenumber back-transform, voltages and sensitivities:
// src/rtrafo.f90:13-92, src/bvolt.f90:7-89, src/bvolti.f90:8-100,
// src/bsens.f90:23-197, src/bsensi.f90:23-194.
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "async.cuh"
#include "convert.cuh"
#include "device.cuh"
#include "kernels.h"

namespace crgpu {

static constexpr double kPi = 3.14159265358979323846264338327950288;

// hpot(j, l) = sum_k kpot(j, l, k) * kwnwi(k) / pi  (2D: kpot(j, l, 1))
__global__ void k_rtrafo(DevProblem P, const double2 *__restrict__ kpot, double2 *__restrict__ hpot) {
    size_t gid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t tot = (size_t)P.eanz * P.n;
    if (gid >= tot) return;
    if (P.swrtr == 0) {
        hpot[gid] = kpot[gid];
        return;
    }
    double2 s = cz(0.0, 0.0);
    for (int k = 0; k < P.K; k++) {
        double2 v = kpot[(size_t)k * tot + gid];
        double w = P.kwnwi[k];
        s = cadd(s, cz(v.x * w, v.y * w));
    }
    hpot[gid] = cz(s.x / kPi, s.y / kPi);
}

void launch_rtrafo(const DevProblem &P, const double2 *kpot, double2 *hpot, cudaStream_t st) {
    size_t tot = (size_t)P.eanz * P.n;
    int nt = 256;
    k_rtrafo<<<(unsigned)((tot + nt - 1) / nt), nt, 0, st>>>(P, kpot, hpot);
}

// V_i = (phi_e2(P_e4) - phi_e1(P_e4)) - (phi_e2(P_e3) - phi_e1(P_e3))
__global__ void k_bvolt(DevProblem P, const double2 *__restrict__ hpot, int mode,
                        const double *__restrict__ kfak, double2 *volt, double2 *sigmaa) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.nanz) return;
    int e1 = P.meas[i * 4], e2 = P.meas[i * 4 + 1], e3 = P.meas[i * 4 + 2], e4 = P.meas[i * 4 + 3];
    auto hp = [&](int node_e, int src_e) -> double2 {
        if (node_e < 0 || src_e < 0) return cz(0.0, 0.0);
        return hpot[(size_t)src_e * P.n + P.enr0[node_e]];
    };
    double2 d1 = hp(e4, e2), d2 = hp(e4, e1), d3 = hp(e3, e2), d4 = hp(e3, e1);
    double2 v = csub(csub(d1, d2), csub(d3, d4));
    if (P.ldc) v.y = 0.0;  // dcmplx of the real DC voltage (src/bvolti.f90:56-62): -log(V < 0) = -ln|V| - i pi
    if (volt) volt[i] = v;
    if (mode == 0) {
        double kf = kfak ? kfak[i] : 1.0;
        if (sigmaa) sigmaa[i] = cz(kf * v.x, kf * v.y);
    } else {
        double a = cabsd(v);
        if (!(a > 0.0)) {  // src/bvolti.f90:80-85
            atomicCAS(P.err, 0, 82);
            if (sigmaa) sigmaa[i] = cz(0.0, 0.0);
            return;
        }
        if (sigmaa) sigmaa[i] = cz(-log(a), -atan2(v.y, v.x));
    }
}

__global__ void k_real_part(double2 *v, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i].y = 0.0;
}

void launch_real_part(double2 *v, int n, cudaStream_t st) {
    if (n > 0) k_real_part<<<(n + 127) / 128, 128, 0, st>>>(v, n);
}

void launch_bvolt(const DevProblem &P, const double2 *hpot, int mode, const double *kfak, double2 *volt,
                  double2 *sigmaa, cudaStream_t st) {
    int nt = 128;
    k_bvolt<<<(P.nanz + nt - 1) / nt, nt, 0, st>>>(P, hpot, mode, kfak, volt, sigmaa);
}

// ---------------------------------------------------------------------------
// Sensitivities by reciprocity.  For element e, wavenumber k and measurement
// i with current electrodes (e1, e2) and voltage electrodes (e3, e4):
//   hsens_k = sum_{m,n} K_k[m][n] (kpot(node_m,e4) - kpot(node_m,e3))
//                                 (kpot(node_n,e2) - kpot(node_n,e1))
// with K_k the element matrix elbg; then the quadrature over k.
//
// One block per element.  Per wavenumber the element's potentials of all
// electrodes are staged in shared memory (cp.async, one wavenumber ahead), the
// product w_k K_k d is formed once for every distinct dipole d of the side
// (current or voltage) that has fewer of them, and a measurement is then the
// other side's difference (from a second table where the pass uses it again) and
// one dot product; threads run over measurements and keep their k-sums in
// registers.  K is symmetric, so either side may take it.  A survey repeats its dipoles: config 2's 4000 measurements have 374
// voltage dipoles.  Per measurement and wavenumber that leaves 24 operations
// instead of 66, and the scaling by strom / pi or sigma / (pi V) is a product
// with a factor formed once per measurement: its six FP64 divisions an entry of
// J took longer than the whole complex64 contraction.  GB300: bsensi of 4800
// cells x 2000 in complex128 15.2 -> 5.8 ms (the FP64 pipe bounds it; 0.7 more without
// the second table, whose differences are additions on that pipe), 12000 x 4000 in
// complex64 12.8 -> 5.0 ms (shared-memory reads; 6.7 without the second table,
// which leaves 6 of the 9 reads of a measurement and wavenumber).  Blocks an
// SM: complex64 spends its time waiting on shared memory, and four at 64 registers
// (100 bytes spilled) do better than the two of 104 registers, 6.4 -> 5.0 ms;
// complex128 gains nothing beyond two (6.09 and 6.10 ms).
// ---------------------------------------------------------------------------
constexpr int kSensThreads = 256;
constexpr int kSensMPT = 16;    // measurements per thread per pass (4096 per pass)
constexpr int kSensGroup = 2;   // of them taken together (4: 6.5 and 6.0 ms in complex128 and 64, registers)
constexpr int kSensK = 160;     // bytes of two element matrices in complex128
constexpr int kSensDip = 1024;  // dipoles of a pass's first table (64 KB in complex128)
constexpr int kSensDip2 = 512;  // ... of its second table (256: 5.15 ms in complex64, 512 and 1024: 5.0)

// The measurements in passes of at most kSensThreads * kSensMPT with at most
// kSensDip distinct dipoles on the side that has the first table, whichever side
// makes the longer pass (the fewer dipoles).  The other side's dipoles that the
// pass uses at least twice go into a second table (their differences alone);
// measurements with one of those come first.  meas: e1..e4 per measurement (-1:
// none, which becomes the zero entry eanz).
//
// Without tables where the survey hardly repeats its dipoles: a table then has an
// entry nearly for every measurement, and its capacity cuts the pass, which
// stages the same potentials again.  Random four-electrode surveys of 4000
// measurements, bsensi in ms, tables -> none (measurements a dipole of a full
// table): complex64, 3000 cells, 40 electrodes 2.64 -> 2.72 (1.6), 50 2.98 -> 2.81 (1.3),
// 64 3.33 -> 3.08 (1.15); 5400 cells, 150 electrodes 12.0 -> 6.6 (1.02), and a pass that is
// not cut 2.82 -> 2.01 (1000 measurements).  complex128 is bound by its operations,
// which tables save from the first repetition on: 64 electrodes 20.0 -> 21.4, 110 46.4
// -> 42.6, 150 47.2 -> 42.9, not cut 10.4 -> 11.8.
void host_sens_passes(const std::vector<int32_t> &meas, int nanz, int eanz, bool single, SensPlan &sp) {
    auto el = [&](int i, int q) { return meas[(size_t)i * 4 + q] < 0 ? eanz : meas[(size_t)i * 4 + q]; };
    sp.slot.resize(nanz);
    for (int i0 = 0; i0 < nanz;) {
        int end[2];
        std::vector<int2> list[2];
        std::vector<int> at[2];
        for (int side = 0; side < 2; side++) {
            std::unordered_map<int64_t, int> seen;
            int i = i0;
            for (; i < nanz && i < i0 + kSensThreads * kSensMPT; i++) {
                const int a = el(i, 2 * side), b = el(i, 2 * side + 1);
                const int64_t key = (int64_t)a * (eanz + 1) + b;
                auto it = seen.find(key);
                if (it == seen.end()) {
                    if ((int)list[side].size() == kSensDip) break;
                    it = seen.emplace(key, (int)list[side].size()).first;
                    list[side].push_back(make_int2(a, b));
                }
                at[side].push_back(it->second);
            }
            end[side] = i;
        }
        const int t = end[1] > end[0] || (end[1] == end[0] && list[1].size() <= list[0].size()) ? 1 : 0, o = 1 - t;
        const int n = end[t] - i0;
        const bool cut = end[t] < nanz && n < kSensThreads * kSensMPT;
        const double repeat = single ? 1.5 : cut ? 1.12 : 0.0;
        if (n < repeat * (double)list[t].size()) {  // without tables, in the survey's order
            for (int i = i0; i < end[t]; i++) sp.slot[i] = make_int4(el(i, 0), el(i, 1), el(i, 2), el(i, 3));
            SensPass *last = sp.direct.empty() ? nullptr : &sp.direct.back();
            if (last && last->i1 == i0 && end[t] - last->i0 <= kSensThreads * kSensMPT) last->i1 = end[t];
            else sp.direct.push_back({i0, i0, end[t], 0, 0, 0});
            i0 = end[t];
            continue;
        }
        // the other side: uses of a dipole, then the second table
        std::unordered_map<int64_t, int> uses;
        auto key = [&](int i) { return (int64_t)el(i, 2 * o) * (eanz + 1) + el(i, 2 * o + 1); };
        for (int i = i0; i < end[t]; i++) uses[key(i)]++;
        std::unordered_map<int64_t, int> second;
        std::vector<int2> list2;
        std::vector<int> order[2];
        // whole groups of slots (a thread's kSensGroup at a time take the same way)
        int often = 0, kinds = 0;
        for (const auto &u : uses)
            if (u.second > 1 && kinds < kSensDip2) kinds++, often += u.second;
        for (int i = i0, left = often / (kSensThreads * kSensGroup) * (kSensThreads * kSensGroup); i < end[t]; i++) {
            const int64_t q = key(i);
            auto it = second.find(q);
            if (it == second.end() && left > 0 && uses[q] > 1 && (int)list2.size() < kSensDip2) {
                it = second.emplace(q, (int)list2.size()).first;
                list2.push_back(make_int2(el(i, 2 * o), el(i, 2 * o + 1)));
            }
            const bool in = it != second.end() && left > 0;
            order[!in].push_back(i);
            left -= in;
        }
        if (order[0].size() % (kSensThreads * kSensGroup)) {  // fewer uses than counted: none
            order[1].insert(order[1].end(), order[0].begin(), order[0].end());
            std::sort(order[1].begin(), order[1].end());
            order[0].clear();
            list2.clear();
        }
        // Threads in an order in which eight neighbours (one shared-memory phase
        // of 16-byte loads) differ in their places modulo 8, as far as the next 64
        // measurements allow: fewer bank conflicts
        int slot = i0;
        for (int kind = 0; kind < 2; kind++) {
            std::vector<int4> wait;
            size_t next = 0;
            int used[3] = {0, 0, 0}, filled = 0;
            while (filled < (int)order[kind].size()) {
                if (filled % 8 == 0) used[0] = used[1] = used[2] = 0;
                while (next < order[kind].size() && wait.size() < 64) {
                    const int i = order[kind][next++];
                    wait.push_back(kind == 0 ? make_int4(second[key(i)], 0, at[t][i - i0], i)
                                             : make_int4(el(i, 2 * o), el(i, 2 * o + 1), at[t][i - i0], i));
                }
                size_t best = 0;
                int cost = 100;
                for (size_t w = 0; w < wait.size() && cost; w++) {
                    const int4 v = wait[w];
                    const int cw = 2 * (used[0] >> (v.x & 7) & 1) + (kind ? 2 * (used[1] >> (v.y & 7) & 1) : 0) +
                                   (used[2] >> (v.z & 7) & 1);
                    if (cw < cost) {
                        cost = cw;
                        best = w;
                    }
                }
                const int4 v = wait[best];
                wait.erase(wait.begin() + best);
                sp.slot[slot++] = v;
                used[0] |= 1 << (v.x & 7);
                used[1] |= 1 << (v.y & 7);
                used[2] |= 1 << (v.z & 7);
                filled++;
            }
        }
        SensPass p;
        p.i0 = i0;
        p.split = i0 + (int)order[0].size();
        p.i1 = i0 + n;
        p.d0 = (int)sp.dip.size();
        p.nd = (int)list[t].size();
        p.nd2 = (int)list2.size();
        sp.pass.push_back(p);
        sp.dip.insert(sp.dip.end(), list[t].begin(), list[t].end());
        sp.dip.insert(sp.dip.end(), list2.begin(), list2.end());
        sp.most = std::max(sp.most, p.nd + p.nd2);
        i0 = end[t];
    }
}

// scaling of row i of J: -strom / pi (mode 0), 1 / (pi V_i) (mode 1; sigma_e is
// the element's)
__global__ void k_sens_factor(DevProblem P, const double2 *__restrict__ volt, int mode) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.nanz) return;
    if (mode == 0) {
        P.sfac[i] = cz(-(P.swrtr ? P.strom[i] / kPi : P.strom[i]), 0.0);
    } else {
        double2 v = volt[i];
        if (P.swrtr) v = cz(kPi * v.x, kPi * v.y);
        P.sfac[i] = cdiv(cz(1.0, 0.0), v);
    }
}

// potentials of one electrode at one node: complex128, or complex64 hi and lo
template <typename R>
struct SensT;
template <>
struct SensT<double> {
    using C = double2;
    using S = double2;
    __device__ static C mk(double a, double b) { return cz(a, b); }
    __device__ static C diff(S a, S b) { return cz(b.x - a.x, b.y - a.y); }
    __device__ static S none() { return cz(0.0, 0.0); }
};
template <>
struct SensT<float> {
    using C = float2;
    using S = float4;  // the differences to ~complex64 accuracy of the difference
    __device__ static C mk(float a, float b) { return cf(a, b); }
    __device__ static C diff(S a, S b) { return cf((b.x - a.x) + (b.z - a.z), (b.y - a.y) + (b.w - a.w)); }
    __device__ static S none() { return make_float4(0.f, 0.f, 0.f, 0.f); }
};

__device__ __forceinline__ double2 to_double(double2 v) { return v; }
__device__ __forceinline__ double2 to_double(float2 v) { return widen(v); }

// the potentials of wavenumber k at an element's nodes, all electrodes, to dst [NK][eanz + 1]
template <typename R, int NK>
__device__ __forceinline__ void sens_stage(const DevProblem &P, const typename SensT<R>::C *__restrict__ kpot,
                                           const int (&nodes)[NK], int k, typename SensT<R>::S *dst) {
    const size_t plane = (size_t)P.K * P.eanz * P.n;
    for (int t = threadIdx.x; t < NK * P.eanz; t += kSensThreads) {
        const int q = t / P.eanz, l = t - q * P.eanz;
        const auto *src = kpot + ((size_t)k * P.eanz + l) * P.n + nodes[q];
        char *to = (char *)(dst + q * (P.eanz + 1) + l);
        if constexpr (sizeof(R) == 8) {
            cp_async16(to, src);
        } else {
            cp_async8(to, src);
            cp_async8(to + 8, src + plane);
        }
    }
    cp_commit();
}

// MODE 0: src/bsens.f90, MODE 1: src/bsensi.f90.  R: arithmetic type of the
// element contraction (double: the reference arithmetic, from kpot; float: the
// mixed mode, from its complex64 planes, with FP64 output).
template <int MODE, typename R, int NK>
__device__ __forceinline__ void sens_element(const DevProblem &P, const typename SensT<R>::C *__restrict__ kpot,
                                             const double2 *__restrict__ sigma, double2 *__restrict__ sens, int e,
                                             unsigned char *smem) {
    using T = SensT<R>;
    using C = typename T::C;
    using S = typename T::S;
    // complex64: a wavenumber's sum over the nodes, whose terms nearly cancel, on its
    // own and the weight afterwards; inside the running sum the rounding of its
    // terms made J's error 4.9e-6 instead of 3.4e-6 (12000 x 4000)
    constexpr bool kOwnSum = sizeof(R) == 4;
    const int eanz = P.eanz, E1 = eanz + 1, tid = threadIdx.x;
    constexpr int NM = NK * (NK + 1) / 2;
    R *ks = (R *)smem;                           // [2][NM], complex128
    S *kp = (S *)(smem + (kOwnSum ? 0 : kSensK));  // [2][NK][E1], the last entry of a row an absent electrode's zero
    C *tab = (C *)(kp + 2 * NK * E1);  // [NK][dipoles of the pass], then [NK][those of its second table]
    int nodes[NK];
#pragma unroll
    for (int q = 0; q < NK; q++) nodes[q] = P.enodes[e * 4 + q];
    if (tid < 2 * NK) kp[tid * E1 + eanz] = T::none();
    auto fetch = [&](int k, int buf) {
        sens_stage<R, NK>(P, kpot, nodes, k, kp + buf * NK * E1);
        if (!kOwnSum && tid < NM)  // w_k K_k by one warp: 6.10 -> 5.81 ms against every thread forming it
            ks[buf * NM + tid] = (R)P.elbg[((size_t)k * P.elanz + e) * 10 + tid] * (P.swrtr ? (R)P.kwnwi[k] : (R)1);
    };
    const double2 sg = sigma[e];
    for (int ps = 0; ps < P.nspass; ps++) {
        const SensPass pass = P.spass[ps];
        const int i0 = pass.i0, i1 = pass.i1, split = pass.split, nd = pass.nd, nd2 = pass.nd2;
        const int2 *dip = P.dip + pass.d0;
        C *tab2 = tab + NK * nd;
        C acc[kSensMPT];
#pragma unroll
        for (int m = 0; m < kSensMPT; m++) acc[m] = T::mk(0, 0);
        __syncthreads();
        fetch(0, 0);
        for (int k = 0; k < P.K; k++) {
            const S *u = kp + (k & 1) * NK * E1;
            R kel[NM];
            const R w = P.swrtr ? (R)P.kwnwi[k] : (R)1;
            if (kOwnSum)
#pragma unroll
                for (int q = 0; q < NM; q++) kel[q] = (R)P.elbg[((size_t)k * P.elanz + e) * 10 + q];
            cp_wait<0>();
            __syncthreads();
            if (!kOwnSum)
#pragma unroll
                for (int q = 0; q < NM; q++) kel[q] = ks[(k & 1) * NM + q];
            if (k + 1 < P.K) fetch(k + 1, (k + 1) & 1);
            for (int d = tid; d < nd + nd2; d += kSensThreads) {
                const int2 p = dip[d];
                C v[NK];
#pragma unroll
                for (int q = 0; q < NK; q++) v[q] = T::diff(u[q * E1 + p.x], u[q * E1 + p.y]);
                if (d >= nd) {
#pragma unroll
                    for (int q = 0; q < NK; q++) tab2[q * nd2 + d - nd] = v[q];
                    continue;
                }
#pragma unroll
                for (int mi = 0; mi < NK; mi++) {
                    C s = T::mk(0, 0);
#pragma unroll
                    for (int mj = 0; mj < NK; mj++) {
                        const int hi = mi > mj ? mi : mj, lo = mi < mj ? mi : mj;
                        const R kk = kel[hi * (hi + 1) / 2 + lo];
                        s.x = fma(kk, v[mj].x, s.x);
                        s.y = fma(kk, v[mj].y, s.y);
                    }
                    tab[mi * nd + d] = s;
                }
            }
            __syncthreads();
#pragma unroll
            for (int m0 = 0; m0 < kSensMPT; m0 += kSensGroup) {
                const int f = i0 + m0 * kSensThreads;  // the group's first slot
                if (f + (kOwnSum ? 0 : tid & ~31) >= i1) break;  // complex128 (FP64 pipe): warp by warp
                int4 md[kSensGroup];
#pragma unroll
                for (int h = 0; h < kSensGroup; h++) {
                    const int i = f + h * kSensThreads + tid;
                    md[h] = P.mdip[i < i1 ? i : i1 - 1];  // L1-resident
                }
                C a[kSensGroup][NK];
                if (f < split) {
#pragma unroll
                    for (int h = 0; h < kSensGroup; h++)
#pragma unroll
                        for (int q = 0; q < NK; q++) a[h][q] = tab2[q * nd2 + md[h].x];
                } else {
#pragma unroll
                    for (int h = 0; h < kSensGroup; h++)
#pragma unroll
                        for (int q = 0; q < NK; q++)
                            a[h][q] = T::diff(u[q * E1 + md[h].x], u[q * E1 + md[h].y]);
                }
#pragma unroll
                for (int h = 0; h < kSensGroup; h++) {
                    C own = T::mk(0, 0), &s = kOwnSum ? own : acc[m0 + h];
#pragma unroll
                    for (int q = 0; q < NK; q++) {
                        const C b = tab[q * nd + md[h].z];
                        s.x = fma(a[h][q].x, b.x, s.x);
                        s.x = fma(-a[h][q].y, b.y, s.x);
                        s.y = fma(a[h][q].x, b.y, s.y);
                        s.y = fma(a[h][q].y, b.x, s.y);
                    }
                    if (kOwnSum) {
                        acc[m0 + h].x = fma(w, own.x, acc[m0 + h].x);
                        acc[m0 + h].y = fma(w, own.y, acc[m0 + h].y);
                    }
                }
            }
        }
#pragma unroll
        for (int m = 0; m < kSensMPT; m++) {
            if (i0 + m * kSensThreads + tid >= i1) continue;
            const int i = P.mdip[i0 + m * kSensThreads + tid].w;
            const double2 d = to_double(acc[m]), f = P.sfac[i];
            sens[(size_t)e * P.nanz + i] = MODE == 0 ? cz(d.x * f.x, d.y * f.x) : cmul(d, cmul(sg, f));
        }
    }
}

// The passes without tables: both differences and the product with K of every
// measurement on its own, rows of J in the survey's order.
template <int MODE, typename R, int NK>
__device__ __forceinline__ void sens_direct(const DevProblem &P, const typename SensT<R>::C *__restrict__ kpot,
                                            const double2 *__restrict__ sigma, double2 *__restrict__ sens, int e,
                                            unsigned char *smem) {
    using T = SensT<R>;
    using C = typename T::C;
    using S = typename T::S;
    constexpr bool kOwnSum = sizeof(R) == 4;  // as in sens_element
    constexpr int NM = NK * (NK + 1) / 2;
    const int E1 = P.eanz + 1, tid = threadIdx.x;
    R *ks = (R *)smem;                             // [2][NM], complex128: w_k K_k
    S *kp = (S *)(smem + (kOwnSum ? 0 : kSensK));  // [2][NK][E1]
    int nodes[NK];
#pragma unroll
    for (int q = 0; q < NK; q++) nodes[q] = P.enodes[e * 4 + q];
    if (tid < 2 * NK) kp[tid * E1 + P.eanz] = T::none();
    auto fetch = [&](int k, int buf) {
        sens_stage<R, NK>(P, kpot, nodes, k, kp + buf * NK * E1);
        if (!kOwnSum && tid < NM)
            ks[buf * NM + tid] = (R)P.elbg[((size_t)k * P.elanz + e) * 10 + tid] * (P.swrtr ? (R)P.kwnwi[k] : (R)1);
    };
    const double2 sg = sigma[e];
    for (int ps = P.nspass; ps < P.nspass + P.nsdirect; ps++) {
        const int i0 = P.spass[ps].i0, i1 = P.spass[ps].i1;
        C acc[kSensMPT];
#pragma unroll
        for (int m = 0; m < kSensMPT; m++) acc[m] = T::mk(0, 0);
        __syncthreads();
        fetch(0, 0);
        for (int k = 0; k < P.K; k++) {
            const S *u = kp + (k & 1) * NK * E1;
            R kel[NM];
            const R w = P.swrtr ? (R)P.kwnwi[k] : (R)1;
            if (kOwnSum)
#pragma unroll
                for (int q = 0; q < NM; q++) kel[q] = (R)P.elbg[((size_t)k * P.elanz + e) * 10 + q];
            cp_wait<0>();
            __syncthreads();
            if (!kOwnSum)
#pragma unroll
                for (int q = 0; q < NM; q++) kel[q] = ks[(k & 1) * NM + q];
            if (k + 1 < P.K) fetch(k + 1, (k + 1) & 1);
#pragma unroll
            for (int m = 0; m < kSensMPT; m++) {
                const int f = i0 + m * kSensThreads;
                if (f + (tid & ~31) >= i1) break;  // the warp has no more
                const int4 el = P.mdip[min(f + tid, i1 - 1)];
                C a[NK], own = T::mk(0, 0), &s = kOwnSum ? own : acc[m];
#pragma unroll
                for (int q = 0; q < NK; q++) a[q] = T::diff(u[q * E1 + el.x], u[q * E1 + el.y]);
#pragma unroll
                for (int mi = 0; mi < NK; mi++) {
                    C b = T::mk(0, 0);
#pragma unroll
                    for (int mj = 0; mj < NK; mj++) {
                        const int hi = mi > mj ? mi : mj, lo = mi < mj ? mi : mj;
                        const R kk = kel[hi * (hi + 1) / 2 + lo];
                        b.x = fma(kk, a[mj].x, b.x);
                        b.y = fma(kk, a[mj].y, b.y);
                    }
                    const C v = T::diff(u[mi * E1 + el.z], u[mi * E1 + el.w]);
                    s.x = fma(v.x, b.x, s.x);
                    s.x = fma(-v.y, b.y, s.x);
                    s.y = fma(v.x, b.y, s.y);
                    s.y = fma(v.y, b.x, s.y);
                }
                if (kOwnSum) {
                    acc[m].x = fma(w, own.x, acc[m].x);
                    acc[m].y = fma(w, own.y, acc[m].y);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < kSensMPT; m++) {
            const int i = i0 + m * kSensThreads + tid;
            if (i >= i1) continue;
            const double2 d = to_double(acc[m]), f = P.sfac[i];
            sens[(size_t)e * P.nanz + i] = MODE == 0 ? cz(d.x * f.x, d.y * f.x) : cmul(d, cmul(sg, f));
        }
    }
}

template <int MODE, typename R>
__global__ __launch_bounds__(kSensThreads, sizeof(R) == 4 ? 4 : 1) void k_bsens_direct(
    DevProblem P, const typename SensT<R>::C *__restrict__ kpot, const double2 *__restrict__ sigma,
    double2 *__restrict__ sens, int e_first) {
    extern __shared__ __align__(16) unsigned char kp_raw[];
    const int e = e_first + blockIdx.x;
    if (P.etype[e] == 3) sens_direct<MODE, R, 3>(P, kpot, sigma, sens, e, kp_raw);
    else sens_direct<MODE, R, 4>(P, kpot, sigma, sens, e, kp_raw);
}

template <int MODE, typename R>
__global__ __launch_bounds__(kSensThreads, sizeof(R) == 4 ? 4 : 2) void k_bsens(DevProblem P,
                                                        const typename SensT<R>::C *__restrict__ kpot,
                                                        const double2 *__restrict__ sigma,
                                                        double2 *__restrict__ sens, int e_first) {
    extern __shared__ __align__(16) unsigned char kp_raw[];
    const int e = e_first + blockIdx.x;
    if (P.etype[e] == 3) sens_element<MODE, R, 3>(P, kpot, sigma, sens, e, kp_raw);
    else sens_element<MODE, R, 4>(P, kpot, sigma, sens, e, kp_raw);
}

// the block's shared memory (both element types) with tables of dips dipoles
static size_t sens_smem(const DevProblem &P, bool single, int dips) {
    const size_t c = single ? sizeof(float2) : sizeof(double2);
    return (single ? 0 : kSensK) + 2 * 4 * (size_t)(P.eanz + 1) * 16 + 4 * (size_t)dips * c;
}

void launch_bsens(const DevProblem &P, const double2 *kpot, const float2 *kpot32, const double2 *sigma,
                  const double2 *volt, int mode, bool single, double2 *sens, cudaStream_t st, int e_first,
                  int e_count) {
    if (e_count < 0) e_count = P.elanz - e_first;
    if (e_count <= 0) return;
    if (single && sens_tc_supported(P, mode) && P.tune_sens != 2) {
        launch_sens_tc(P, kpot32, sens, st, e_first, e_count);
        return;
    }
    static std::once_flag once;
    std::call_once(once, [] {
        int dev = 0, optin = 48 * 1024;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        for (const void *f : {(const void *)k_bsens<0, float>, (const void *)k_bsens<1, float>,
                              (const void *)k_bsens<0, double>, (const void *)k_bsens<1, double>,
                              (const void *)k_bsens_direct<0, float>, (const void *)k_bsens_direct<1, float>,
                              (const void *)k_bsens_direct<0, double>, (const void *)k_bsens_direct<1, double>})
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    });
    if (P.nanz > 0) k_sens_factor<<<(P.nanz + 127) / 128, 128, 0, st>>>(P, volt, mode);
    const size_t smem = sens_smem(P, single, P.sens_dips), direct_smem = sens_smem(P, single, 0);
    auto run = [&](auto table, auto direct, const auto *pot) {
        if (P.nspass) table<<<e_count, kSensThreads, smem, st>>>(P, pot, sigma, sens, e_first);
        if (P.nsdirect) direct<<<e_count, kSensThreads, direct_smem, st>>>(P, pot, sigma, sens, e_first);
    };
    if (single) {
        if (mode == 0) run(k_bsens<0, float>, k_bsens_direct<0, float>, kpot32);
        else run(k_bsens<1, float>, k_bsens_direct<1, float>, kpot32);
    } else {
        if (mode == 0) run(k_bsens<0, double>, k_bsens_direct<0, double>, kpot);
        else run(k_bsens<1, double>, k_bsens_direct<1, double>, kpot);
    }
}

}  // namespace crgpu

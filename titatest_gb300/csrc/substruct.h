// Device side of the substructured solver (substruct.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "device.cuh"
#include "sub_plan.h"

namespace crgpu {

// Shared by all electrodes of a wavenumber; T is float2 (mixed) or double2.
struct DevSub {
    int n, m, nI, mp, ldc, szU;
    int64_t szF, szG, szS;
    const SubFront *fr;
    const SubEnt *ent, *be;
    const SubTile *tA, *tG, *tS, *tU, *tV, *tD;
    const int32_t *pos, *node, *rows, *inv, *root_inv, *fcolpos;
    const int32_t *be_ptr, *rb_ptr, *rb_ent, *rb_pos;
    int root_ent0, n_root_ent, n_be, root_u0, root_r, root_live;
    int64_t root_oS;
    double2 *As;     // [K][nnz] area parts, scaled by fk on both sides
    double *fk;      // [K][n]   scaling of the area parts' diagonal, by node
    int *kbad;       // [K]      error of the wavenumber's elimination
    void *F, *G, *H, *S, *R;  // [K][szF], [K][szG] (G and its right factor), [K][szS], [K][mp * ldc]
};

// A rectangle of systems, wavenumbers k0 .. k0+Kb-1 x electrodes l0 .. l0+Lb-1.
// Vectors are [Kb][positions][Lb]: the electrode runs fastest.
struct SubBatch {
    int k0, Kb, l0, Lb;
    void *C;                        // [Kb * Lb][mp * ldc] root factors
    double2 *bval;                  // [Kb][n_be][Lb] boundary terms of the root entries
    double2 *X, *Bt;                // solution; right-hand side of the adjoint (scaled by fk)
    void *Y, *W, *Z, *U;            // input, assembled input, output, update rows
    int *status, *active, *kact;    // per system, per system, per wavenumber (null: all)
    unsigned long long *mz, *mx;    // per system: bit patterns of the largest correction and solution
};

// counters of one refinement step
struct RefineCount {
    int n;       // systems (band: items) still refining after the step
    int ticket;  // blocks of k_sub_stop that have counted
    double z;    // largest relative correction of the step
};
constexpr int kRefineCap = 64;  // refinement steps at most (crgpu_set_refinement)

// Where a step counts, and who learns whether systems are left: the host (a word
// of mapped memory), or the loop node of a graph, whose one recorded step numbers
// itself (cnt[kRefineCap].n).
struct SubStop {
    RefineCount *cnt = nullptr;  // of this step; of step 0 in a loop; null: the first solve
    int *left = nullptr;
    cudaGraphConditionalHandle loop = 0;
    int steps = 0;  // of a loop at most; 0: no loop
};

SubShape sub_shape(bool mixed);
int sub_root_block(bool mixed);  // columns of a block of the root factor
int sub_root_rows(bool mixed);   // rows of one of its tiles
int sub_root_max(bool mixed);    // most padded nodes of a root
void sub_launch_values(const DevProblem &P, const DevSub &D, const double2 *sigma, const double2 *adom, cudaStream_t st);
// the first K wavenumbers of D's arrays
int sub_launch_factor(const DevProblem &P, const DevSub &D, const SubPlan &sp, int K, bool mixed, cudaStream_t st);
void sub_launch_root(const DevProblem &P, const DevSub &D, const SubBatch &B, const double2 *sigma, bool mixed,
                     cudaStream_t st);
// unit: the right-hand sides are kompab's, zero but at the sources of the plan
int sub_launch_apply(const DevSub &D, const SubPlan &sp, const SubBatch &B, bool mixed, bool unit, const int *nprev,
                     cudaStream_t st);
void sub_launch_rhs(const DevProblem &P, const DevSub &D, const SubBatch &B, bool mixed, int lsink, int nsink,
                    const double2 *src, cudaStream_t st);
void sub_launch_residual(const DevProblem &P, const DevSub &D, const SubBatch &B, bool unit, int lsink, int nsink,
                         const int *nprev, cudaStream_t st);
void sub_launch_accumulate(const DevSub &D, const SubBatch &B, bool first, double tol, const int *nprev,
                           const SubStop &stop, cudaStream_t st);
void sub_launch_unpack(const DevProblem &P, const DevSub &D, const SubBatch &B, double sign, double2 *out,
                       float2 *out32, cudaStream_t st);

}  // namespace crgpu

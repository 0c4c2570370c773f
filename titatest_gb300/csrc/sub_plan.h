// Elimination plan of the substructured solver (substruct.cu): which nodes
// are eliminated once per wavenumber for all current electrodes, in which
// order, and where every piece lives.
#pragma once

#include <cstdint>
#include <vector>

#include "crgpu_internal.h"

namespace crgpu {

constexpr int kSubEMax = 64;   // most nodes one front may eliminate
constexpr int kSubCh = 4;      // most children of a front

// What suits a precision (substruct.cu): nodes that are not cut further, most
// nodes a front eliminates, and the edge of the dense kernels' tiles.
struct SubShape {
    int leaf, emax, tile;
};

// One front: e nodes eliminated here, r nodes it is coupled to (eliminated
// later, or root nodes).  Local rows 0..e-1 are positions nd0..nd0+e-1, rows
// e..e+r-1 the positions rows[rows0 .. rows0+r-1].
struct SubFront {
    int32_t e, r, nd0, nch;
    int32_t live;         // bit kSubCh: a source node is eliminated here or below; bit c: ... below child c
    int32_t ent0, nent;   // matrix entries assembled here
    int32_t rows0;        // into SubPlan::rows
    int32_t u0;           // first row of this front's update vectors
    int64_t oF, oG, oS;   // inverse pivot block (e x e), G (e x r), Schur complement (r x r)
    // children: their r, first update row and Schur complement, and
    // (in SubPlan::inv) the row among a child's r rows of every local row, or -1
    int32_t cr[kSubCh], cu[kSubCh], inv[kSubCh];
    int64_t cS[kSubCh];
};

struct SubEnt {
    int32_t p, lr, lc;    // lower-pattern entry and its local row (eliminated) and column
};

struct SubTile {
    int32_t front, ti, tj;
};

struct SubPlan {
    int n = 0, m = 0, nI = 0, nfront = 0, nlevel = 0;
    std::vector<int32_t> pos, node;            // node -> position, position -> node
    std::vector<SubFront> fronts;              // by level
    std::vector<int32_t> level;                // nlevel + 1: first front of a level
    std::vector<int32_t> rows, inv;
    std::vector<SubEnt> ent;                   // of the fronts, then (from root_ent0) of the root
    int root_ent0 = 0;
    std::vector<int32_t> root_inv;             // root row -> row of the last front's r rows, or -1
    std::vector<SubEnt> be;                    // root entries with mixed-boundary terms, by column (row >= column)
    std::vector<int32_t> be_ptr;               // m + 1: first of a column
    std::vector<int32_t> rb_ptr, rb_ent, rb_pos;  // by root row: its entries in be and the other node's position
    // tiles of a front's gather (e x (e + r)), of G (e x r), of S (r x r, lower)
    // and row tiles of the solves (r up, e down), by level
    std::vector<SubTile> tA, tG, tS, tU, tD;
    std::vector<int32_t> lA, lG, lS, lU, lD;   // nlevel + 1 each
    std::vector<SubTile> tV;                   // those of tU whose front is live
    std::vector<int32_t> lV;
    int64_t szF = 0, szG = 0, szS = 0;         // entries per wavenumber
    int32_t szU = 0;                           // update rows per wavenumber
    double c_factor = 0, c_apply = 0;          // complex multiply-adds: factor per wavenumber, one solve
};

// The plan for the grid, or false where it has no root (no mixed boundary)
// or no interior.  sources: the nodes that kompab's right-hand sides have
// entries at (electrodes, the fictitious sink).
bool build_sub_plan(const HostGrid &hg, const Pattern &pat, const SubShape &shape,
                    const std::vector<int32_t> &sources, SubPlan &sp);

// A problem as the choice between the band and this solver sees it: nodes, band
// width, nodes of the root, the same padded and the most that k_sub_root_solve
// holds, electrodes, wavenumbers, the plan's complex multiply-adds.
struct SubCost {
    bool mixed;
    int n, mb, m, mp, root_max, eanz, K;
    double c_factor, c_apply;
};
// GB300 times of a forward in microseconds at the default refinement, as
// sub_fits compares them
double band_us(const SubCost &q);
double sub_us(const SubCost &q);
bool sub_fits(const SubCost &q);

}  // namespace crgpu

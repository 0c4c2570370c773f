// Nested dissection of the nodes that no mixed boundary touches.
//
// The systems of one wavenumber differ between current electrodes only in the
// mixed-boundary terms (src/beta.f90, src/kompab.f90:112-139), that is in the
// entries among the nodes of the type-11 lines.  Those nodes form the root;
// the others are cut recursively, across x or y, by the smaller vertex
// separator, and eliminated leaves first.
#include <algorithm>
#include <cmath>

#include "sub_plan.h"

namespace crgpu {

namespace {

struct Build {
    const HostGrid &hg;
    const Pattern &pat;
    const SubShape shape;
    struct F {
        std::vector<int32_t> E, R;
        std::vector<int> ch;
        int lev = 0;
        bool gone = false;  // taken into its parent
    };
    std::vector<F> f;
    std::vector<int32_t> owner;  // front of a node, -1: not eliminated (yet)
    std::vector<int32_t> mark, seen;
    std::vector<int32_t> rank[2], reach[2];  // places across x and across y, the neighbours' last place
    int stamp = 0;

    Build(const HostGrid &h, const Pattern &p, const SubShape &s)
        : hg(h), pat(p), shape(s), owner(h.n, -1), mark(h.n, 0), seen(h.n, 0) {}

    // the nodes across x (dir 0) or y, ties by the other coordinate, then by number
    std::vector<int32_t> sorted(std::vector<int32_t> nodes, int dir) {
        const std::vector<double> &c0 = dir ? hg.y : hg.x, &c1 = dir ? hg.x : hg.y;
        struct Key {
            double a, b;
            int32_t v;
            bool operator<(const Key &o) const { return a != o.a ? a < o.a : b != o.b ? b < o.b : v < o.v; }
        };
        std::vector<Key> key;
        key.reserve(nodes.size());
        for (int v : nodes) key.push_back({c0[v], c1[v], v});
        if (!std::is_sorted(key.begin(), key.end())) std::sort(key.begin(), key.end());
        rank[dir].assign(hg.n, -1);
        for (size_t q = 0; q < key.size(); q++) rank[dir][nodes[q] = key[q].v] = (int)q;
        reach[dir].assign(hg.n, -1);
        for (int v : nodes)
            for (int z = pat.fptr[v]; z < pat.fptr[v + 1]; z++)
                reach[dir][v] = std::max(reach[dir][v], rank[dir][pat.fcol[z]]);
        return nodes;
    }

    // Eliminates E after the fronts of ch; long lists as a chain.  A front that
    // has children itself is taken into its parent where the two fit one
    // front: fewer levels, and its update vectors are never stored.
    int add(std::vector<int32_t> E, std::vector<int> ch) {
        std::vector<int> up;
        size_t left = ch.size();
        for (int c : ch) {
            left--;
            F &s = f[c];
            if (!s.ch.empty() && E.size() + s.E.size() <= (size_t)shape.emax &&
                up.size() + s.ch.size() + left <= (size_t)kSubCh) {
                E.insert(E.begin(), s.E.begin(), s.E.end());
                up.insert(up.end(), s.ch.begin(), s.ch.end());
                s.gone = true;
            } else {
                up.push_back(c);
            }
        }
        const int s = (int)E.size(), parts = std::max(1, (s + shape.emax - 1) / shape.emax);
        for (int q = 0; q < parts; q++) {
            F t;
            t.E.assign(E.begin() + (size_t)s * q / parts, E.begin() + (size_t)s * (q + 1) / parts);
            t.ch = up;
            const int id = (int)f.size();
            for (int v : t.E) owner[v] = id;
            // the rest of a chain is not eliminated yet
            if (q == 0)
                for (size_t z = t.E.size(); z < E.size(); z++) owner[E[z]] = -1;
            const int st = ++stamp;
            auto take = [&](int v) {
                if (owner[v] < 0 && mark[v] != st) {
                    mark[v] = st;
                    t.R.push_back(v);
                }
            };
            for (int v : t.E)
                for (int z = pat.fptr[v]; z < pat.fptr[v + 1]; z++) take(pat.fcol[z]);
            for (int c : t.ch) {
                for (int v : f[c].R) take(v);
                t.lev = std::max(t.lev, f[c].lev + 1);
            }
            f.push_back(std::move(t));
            up.assign(1, id);
        }
        return (int)f.size() - 1;
    }

    // The smaller of the two vertex separators of the halves nodes[0..h) and
    // nodes[h..) of nodes marked st, ordered by rank: only the nodes with a
    // neighbour ranked beyond the cut are looked at closer.
    std::vector<int32_t> separator(const std::vector<int32_t> &nodes, int h, int dir, int st) {
        const std::vector<int32_t> &rk = rank[dir];
        const int last = rk[nodes[h - 1]], met = ++stamp;
        std::vector<int32_t> a, b;
        for (int q = 0; q < h; q++) {
            const int v = nodes[q];
            if (reach[dir][v] <= last) continue;
            bool cut = false;
            for (int z = pat.fptr[v]; z < pat.fptr[v + 1]; z++) {
                const int w = pat.fcol[z];
                if (mark[w] != st || rk[w] <= last) continue;
                cut = true;
                if (seen[w] == met) continue;
                seen[w] = met;
                b.push_back(w);
            }
            if (cut) a.push_back(v);
        }
        if (a.size() <= b.size()) return a;
        std::sort(b.begin(), b.end(), [&](int u, int v) { return rk[u] < rk[v]; });
        return b;
    }

    // by[0] and by[1]: the same nodes ordered across x and across y
    int cut(std::vector<int32_t> (&by)[2]) {
        const int n = (int)by[0].size();
        if (n <= shape.leaf) return add(std::move(by[1]), {});
        const int h = n / 2;
        const int st = ++stamp;
        for (int v : by[0]) mark[v] = st;
        std::vector<int32_t> best = separator(by[0], h, 0, st), other = separator(by[1], h, 1, st);
        const int dir = other.size() < best.size() ? 1 : 0;
        if (dir) best = std::move(other);
        if (best.size() * 2 >= (size_t)n) return add(std::move(by[dir]), {});
        const int half = ++stamp, sep = ++stamp;
        for (int q = 0; q < h; q++) mark[by[dir][q]] = half;
        for (int v : best) mark[v] = sep;
        std::vector<int32_t> part[2][2];
        for (int d = 0; d < 2; d++) {
            for (auto &p : part) p[d].reserve(n - h);
            for (int v : by[d])
                if (mark[v] != sep) part[mark[v] != half][d].push_back(v);
            by[d] = std::vector<int32_t>();
        }
        std::vector<int> ch;
        for (auto &p : part)
            if (!p[0].empty()) ch.push_back(cut(p));
        return add(std::move(best), std::move(ch));
    }
};

}  // namespace

bool build_sub_plan(const HostGrid &hg, const Pattern &pat, const SubShape &shape,
                    const std::vector<int32_t> &sources, SubPlan &sp) {
    sp = SubPlan();
    const int n = hg.n;
    std::vector<uint8_t> root(n, 0);
    for (int rb = 0; rb < hg.relanz; rb++)
        if (hg.btype[rb] == 11) root[hg.bnodes[(size_t)rb * 2]] = root[hg.bnodes[(size_t)rb * 2 + 1]] = 1;
    std::vector<int32_t> inner, outer;
    for (int i = 0; i < n; i++) (root[i] ? outer : inner).push_back(i);
    if (inner.empty() || outer.empty()) return false;
    Build b(hg, pat, shape);
    std::vector<int32_t> by[2] = {b.sorted(inner, 0), b.sorted(inner, 1)};
    b.cut(by);
    std::vector<int32_t> order;
    for (int q = 0; q < (int)b.f.size(); q++)
        if (!b.f[q].gone) order.push_back(q);
    const int nf = (int)order.size();
    sp.n = n;
    sp.m = (int)outer.size();
    sp.nI = (int)inner.size();
    sp.nfront = nf;
    // fronts by level
    std::vector<int32_t> at(b.f.size(), -1);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return b.f[x].lev < b.f[y].lev; });
    for (int q = 0; q < nf; q++) at[order[q]] = q;
    sp.nlevel = b.f[order[nf - 1]].lev + 1;
    sp.level.assign(sp.nlevel + 1, nf);
    for (int q = nf - 1; q >= 0; q--) sp.level[b.f[order[q]].lev] = q;
    // positions
    sp.pos.assign(n, -1);
    for (int q = 0, p = 0; q < nf; q++)
        for (int v : b.f[order[q]].E) {
            sp.pos[v] = p++;
            sp.node.push_back(v);
        }
    for (int v : outer) {
        sp.pos[v] = (int)sp.node.size();
        sp.node.push_back(v);
    }
    // fronts, their rows and the children's rows in them
    std::vector<int32_t> local(n, -1);
    std::vector<uint8_t> source(n, 0);
    for (int v : sources) source[v] = 1;
    sp.fronts.resize(nf);
    for (int q = 0; q < nf; q++) {
        Build::F &s = b.f[order[q]];
        std::sort(s.R.begin(), s.R.end(), [&](int x, int y) { return sp.pos[x] < sp.pos[y]; });
        SubFront &t = sp.fronts[q];
        t.e = (int)s.E.size();
        t.r = (int)s.R.size();
        t.nd0 = t.e ? sp.pos[s.E[0]] : 0;
        t.rows0 = (int)sp.rows.size();
        for (int v : s.R) sp.rows.push_back(sp.pos[v]);
        t.u0 = sp.szU;
        sp.szU += t.r;
        t.oF = sp.szF;
        t.oG = sp.szG;
        t.oS = sp.szS;
        sp.szF += (int64_t)t.e * t.e;
        sp.szG += (int64_t)t.e * t.r;
        sp.szS += (int64_t)t.r * t.r;
        sp.c_factor += (double)t.e * t.e * t.e + (double)t.e * t.e * t.r + 0.5 * t.e * t.r * (double)t.r;
        sp.c_apply += (double)t.e * (t.e + 2.0 * t.r);
        t.nch = (int)s.ch.size();
        t.live = 0;
        for (int v : s.E)
            if (source[v]) t.live = 1 << kSubCh;
        for (int z = 0; z < kSubCh; z++) {
            t.cr[z] = t.cu[z] = t.inv[z] = 0;
            t.cS[z] = 0;
            if (z >= t.nch) continue;
            const SubFront &u = sp.fronts[at[s.ch[z]]];
            t.cr[z] = u.r;
            t.cu[z] = u.u0;
            t.cS[z] = u.oS;
            if (u.live) t.live |= 1 << kSubCh | 1 << z;
            t.inv[z] = (int)sp.inv.size();
            const std::vector<int32_t> &cr = b.f[s.ch[z]].R;
            for (size_t y = 0; y < cr.size(); y++) local[cr[y]] = (int)y;
            for (int v : s.E) sp.inv.push_back(local[v]);
            for (int v : s.R) sp.inv.push_back(local[v]);
            for (int v : cr) local[v] = -1;
        }
    }
    // matrix entries, each in the front that eliminates its earlier node
    std::vector<int32_t> root_p, own(pat.nnz, -1), place(nf + 1, 0);
    for (int p = 0; p < pat.nnz; p++) {
        if (pat.col[p] < 0) continue;
        const int i = pat.row[p], c = pat.col[p];
        const int first = sp.pos[i] < sp.pos[c] ? i : c;
        if (b.owner[first] < 0) root_p.push_back(p);
        else place[(own[p] = at[b.owner[first]]) + 1]++;
    }
    for (int q = 0; q < nf; q++) place[q + 1] += place[q];
    std::vector<int32_t> list(place[nf]), next(place.begin(), place.end() - 1);
    for (int p = 0; p < pat.nnz; p++)
        if (own[p] >= 0) list[next[own[p]]++] = p;
    sp.ent.reserve(list.size() + root_p.size());
    for (int q = 0; q < nf; q++) {
        const Build::F &s = b.f[order[q]];
        for (size_t z = 0; z < s.E.size(); z++) local[s.E[z]] = (int)z;
        for (size_t z = 0; z < s.R.size(); z++) local[s.R[z]] = (int)(s.E.size() + z);
        SubFront &t = sp.fronts[q];
        t.ent0 = (int)sp.ent.size();
        t.nent = place[q + 1] - place[q];
        for (int z = place[q]; z < place[q + 1]; z++) {
            const int p = list[z], a = local[pat.row[p]], c = local[pat.col[p]];
            sp.ent.push_back({p, std::min(a, c), std::max(a, c)});
        }
        for (int v : s.E) local[v] = -1;
        for (int v : s.R) local[v] = -1;
    }
    // the root: its entries, the last front's rows in it, the boundary terms by column
    sp.root_ent0 = (int)sp.ent.size();
    for (int v : outer) local[v] = sp.pos[v] - sp.nI;
    std::vector<std::vector<SubEnt>> cols(sp.m);
    for (int p : root_p) {
        const int a = local[pat.row[p]], c = local[pat.col[p]], r = std::max(a, c), l = std::min(a, c);
        sp.ent.push_back({p, r, l});
        if (pat.bnd_ptr[p] < pat.bnd_ptr[p + 1]) cols[l].push_back({p, r, l});
    }
    std::vector<std::vector<std::pair<int32_t, int32_t>>> rowse(sp.m);
    sp.be_ptr.assign(1, 0);
    for (int c = 0; c < sp.m; c++) {
        std::sort(cols[c].begin(), cols[c].end(), [](const SubEnt &x, const SubEnt &y) { return x.lr < y.lr; });
        for (const SubEnt &en : cols[c]) {
            const int q = (int)sp.be.size();
            rowse[en.lr].push_back({q, sp.nI + c});
            if (en.lr != c) rowse[c].push_back({q, sp.nI + en.lr});
            sp.be.push_back(en);
        }
        sp.be_ptr.push_back((int)sp.be.size());
    }
    sp.rb_ptr.assign(1, 0);
    for (int i = 0; i < sp.m; i++) {
        for (const auto &x : rowse[i]) {
            sp.rb_ent.push_back(x.first);
            sp.rb_pos.push_back(x.second);
        }
        sp.rb_ptr.push_back((int)sp.rb_ent.size());
    }
    sp.root_inv.assign(sp.m, -1);
    const std::vector<int32_t> &tr = b.f[order[nf - 1]].R;
    for (size_t z = 0; z < tr.size(); z++) sp.root_inv[local[tr[z]]] = (int)z;
    // tiles
    auto tiles = [&](int v) { return (v + shape.tile - 1) / shape.tile; };
    sp.lG.assign(1, 0);
    sp.lA = sp.lS = sp.lU = sp.lD = sp.lV = sp.lG;
    for (int lv = 0; lv < sp.nlevel; lv++) {
        for (int q = sp.level[lv]; q < sp.level[lv + 1]; q++) {
            const SubFront &t = sp.fronts[q];
            const int te = tiles(t.e), tr2 = tiles(t.r);
            for (int i = 0; i < te; i++) {
                sp.tD.push_back({q, i, 0});
                for (int j = 0; j < tr2; j++) sp.tG.push_back({q, i, j});
                for (int j = 0; t.nch && j < tiles(t.e + t.r); j++) sp.tA.push_back({q, i, j});
            }
            for (int i = 0; i < tr2; i++) {
                for (int j = 0; j <= i; j++) sp.tS.push_back({q, i, j});
            }
            for (int i = 0; i < std::max(1, tr2); i++) {
                sp.tU.push_back({q, i, 0});
                if (t.live) sp.tV.push_back({q, i, 0});
            }
        }
        sp.lA.push_back((int)sp.tA.size());
        sp.lG.push_back((int)sp.tG.size());
        sp.lS.push_back((int)sp.tS.size());
        sp.lU.push_back((int)sp.tU.size());
        sp.lV.push_back((int)sp.tV.size());
        sp.lD.push_back((int)sp.tD.size());
    }
    return true;
}

// The band is eliminated node by node, in mixed precision about as fast for 32
// systems as for the 1248 that are resident at once (a latency of 1.6 us a node
// up to the warp kernels' width, 2.35 with all of them at work); in complex128 an
// SM takes one system at a time, beyond width 126 two.
double band_us(const SubCost &q) {
    const double n = q.n, mb = q.mb, systems = (double)q.K * q.eanz, base = 250.0;
    if (!q.mixed) {
        if (mb > 126) return base + n * std::max(1.0, systems / 304.0) * 1.4e-3 * mb * mb;
        return base + n * std::ceil(systems / 152.0) * (2.6 + 0.02 * mb + 3.8e-4 * mb * mb);
    }
    const double full = systems / 1248.0;
    if (mb <= 62) return base + n * std::max(1.0, full) * (1.6 + 0.75 * std::min(1.0, full));
    return base + n * (1.6 + 2.5e-3 * systems * (mb / 100.0) * (mb <= 124 ? 1.0 : mb / 100.0));
}

// A root is one block's work, at 215 (complex64) and 6.5 (complex128) GFLOP/s; up
// to five blocks share an SM, and more systems than SMs do not spread evenly:
// the second group's blocks come to where the first one's shared elimination has
// left room, the more so the longer a root takes.  The rest is the shared
// elimination, the sweeps and residuals, and the chains of the root's solves.
double sub_us(const SubCost &q) {
    const double m = q.m, systems = (double)q.K * q.eanz, x = systems / 152.0, flop = 4.0 / 3.0 * m * m * m;
    const double crowd = q.mixed ? std::min(2.9, std::max(1.3, m / 700.0)) : 1.7;
    const double load = x <= 1.0 ? 1.0 : std::max(x, std::min(5.0, crowd * x));
    const double shared = 8.0 * q.K * q.c_factor;
    if (!q.mixed)
        return 200.0 + flop / 6.5e3 * load + (shared + 8.0 * systems * q.c_apply) / 0.6e6 + 2e-3 * m * m;
    return 200.0 + flop / 215e3 * std::max(1.0, 0.82 * load) + shared / 8e6 + 4.5e-4 * q.n * systems + 2.3e-3 * m * m +
           1.5 * m;
}

// Long meshes have a narrow band and a large root.  By time, since the two run at
// very different rates (per counted operation the band is 60 times slower at width
// 12, 1.4 times at 62).  Forwards, band -> this solver in ms, columns x rows of
// cells: complex64, 1248 systems 300x10 8.4 -> 4.8, 500x6 8.9 -> 10.8, 500x20 25.7
// -> 13.9, 700x20 34.9 -> 28.2, 1000x20 50.0 -> 61.1, 2000x20 99 -> 369, 800x30 58.4
// -> 41.1, 1000x30 73.1 -> 70.1, 1500x30 110 -> 182, 500x60 78.7 -> 26.7, 1250x60
// 196 -> 139, 1500x60 235 -> 212, 2000x60 313 -> 448, 2000x100 1531 -> 516; 240
// systems 1000x20 33.8 -> 18.7, 2000x20 67 -> 203, 1500x60 165 -> 112, 2000x60 220
// -> 243, 2600x60 286 -> 486; 32 systems 2000x60 208 -> 77, 2000x20 63.3 -> 63.8;
// complex128, 96 systems 200x10 7.2 -> 4.7, 400x10 14.2 -> 21.1, 300x20 25.0 ->
// 13.2, 600x20 49.7 -> 63.9, 600x30 91 -> 69, 1000x30 151 -> 251, 1500x60 974 ->
// 845, 2000x60 1298 -> 1819; 384 systems 300x20 69 -> 30, 600x20 137 -> 261, 500x30
// 213 -> 182, 600x60 1145 -> 367.  Over these and 80 others the band is kept at most
// where it costs 11 % more, and never left where it is the faster one; above 5 ms
// the band's estimate is 0.63 to 1.22 of its time, this solver's 0.71 to 2.14, nine
// tenths of both 0.8 to 1.25.  Beyond the two operation counts the choice is not
// measured over the whole range: those problems keep the band, as do the smallest
// complex128 grids, all latency (8x4 cells 0.29 -> 0.35 ms, 16x6 0.52 -> 0.43).
bool sub_fits(const SubCost &q) {
    if (q.mp > q.root_max) return false;  // the root's vector stays in one block's shared memory
    const double n = q.n, mb = q.mb, m = q.m;
    const double band = 0.5 * n * mb * mb + 6.0 * n * mb;
    const double sub = m * m * m / 6.0 + 4.0 * q.c_apply + q.c_factor / q.eanz;
    if (sub > (q.mixed ? 30.0 : 5.0) * band || (!q.mixed && q.n < 100)) return false;
    return sub_us(q) <= band_us(q);
}

}  // namespace crgpu

// sub_fits by its numbers, for the tests (not part of the C ABI)
extern "C" int crgpu_sub_fits(int32_t mixed, int32_t n, int32_t mb, int32_t m, int32_t mp, int32_t root_max, int32_t eanz,
                              int32_t K, double c_factor, double c_apply) {
    return crgpu::sub_fits({mixed != 0, n, mb, m, mp, root_max, eanz, K, c_factor, c_apply});
}

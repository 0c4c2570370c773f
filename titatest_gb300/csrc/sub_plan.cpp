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

constexpr int kLeaf = 24;

struct Build {
    const HostGrid &hg;
    const Pattern &pat;
    struct F {
        std::vector<int32_t> E, R;
        int ch0 = -1, ch1 = -1, lev = 0;
    };
    std::vector<F> f;
    std::vector<int32_t> owner;  // front of a node, -1: not eliminated (yet)
    std::vector<int32_t> mark;
    int stamp = 0;

    Build(const HostGrid &h, const Pattern &p) : hg(h), pat(p), owner(h.n, -1), mark(h.n, 0) {}

    // eliminates E after the fronts a and b; long lists as a chain
    int add(const std::vector<int32_t> &E, int a, int b) {
        const int s = (int)E.size(), parts = std::max(1, (s + kSubEMax - 1) / kSubEMax);
        for (int q = 0; q < parts; q++) {
            F t;
            t.E.assign(E.begin() + (size_t)s * q / parts, E.begin() + (size_t)s * (q + 1) / parts);
            t.ch0 = a;
            t.ch1 = b;
            const int id = (int)f.size();
            for (int v : t.E) owner[v] = id;
            const int st = ++stamp;
            auto take = [&](int v) {
                if (owner[v] < 0 && mark[v] != st) {
                    mark[v] = st;
                    t.R.push_back(v);
                }
            };
            for (int v : t.E)
                for (int z = pat.fptr[v]; z < pat.fptr[v + 1]; z++) take(pat.fcol[z]);
            for (int c : {a, b})
                if (c >= 0) {
                    for (int v : f[c].R) take(v);
                    t.lev = std::max(t.lev, f[c].lev + 1);
                }
            f.push_back(std::move(t));
            a = id;
            b = -1;
        }
        return (int)f.size() - 1;
    }

    // the smaller of the two vertex separators of the halves nodes[0..h) and nodes[h..)
    std::vector<int32_t> separator(const std::vector<int32_t> &nodes, int h) {
        const int lo = ++stamp, hi = ++stamp;
        for (size_t q = 0; q < nodes.size(); q++) mark[nodes[q]] = (int)q < h ? lo : hi;
        std::vector<int32_t> a, b;
        for (size_t q = 0; q < nodes.size(); q++) {
            const int v = nodes[q], other = (int)q < h ? hi : lo;
            for (int z = pat.fptr[v]; z < pat.fptr[v + 1]; z++)
                if (mark[pat.fcol[z]] == other) {
                    ((int)q < h ? a : b).push_back(v);
                    break;
                }
        }
        return a.size() <= b.size() ? a : b;
    }

    int cut(std::vector<int32_t> nodes) {
        if ((int)nodes.size() <= kLeaf) return add(nodes, -1, -1);
        const int h = (int)nodes.size() / 2;
        std::vector<int32_t> best, best_nodes;
        for (int dir = 0; dir < 2; dir++) {
            const std::vector<double> &c0 = dir ? hg.y : hg.x, &c1 = dir ? hg.x : hg.y;
            std::nth_element(nodes.begin(), nodes.begin() + h, nodes.end(), [&](int a, int b) {
                if (c0[a] != c0[b]) return c0[a] < c0[b];
                if (c1[a] != c1[b]) return c1[a] < c1[b];
                return a < b;
            });
            std::vector<int32_t> s = separator(nodes, h);
            if (dir == 0 || s.size() < best.size()) {
                best = std::move(s);
                best_nodes = nodes;
            }
        }
        if (best.size() * 2 >= nodes.size()) return add(nodes, -1, -1);
        const int st = ++stamp;
        for (int v : best) mark[v] = st;
        std::vector<int32_t> part[2];
        for (size_t q = 0; q < best_nodes.size(); q++)
            if (mark[best_nodes[q]] != st) part[(int)q >= h].push_back(best_nodes[q]);
        int ch[2] = {-1, -1};
        for (int q = 0; q < 2; q++)
            if (!part[q].empty()) ch[q] = cut(std::move(part[q]));
        return add(best, ch[0], ch[1]);
    }
};

int tiles(int v) { return (v + kSubTile - 1) / kSubTile; }

}  // namespace

bool build_sub_plan(const HostGrid &hg, const Pattern &pat, SubPlan &sp) {
    sp = SubPlan();
    const int n = hg.n;
    std::vector<uint8_t> root(n, 0);
    for (int rb = 0; rb < hg.relanz; rb++)
        if (hg.btype[rb] == 11) root[hg.bnodes[(size_t)rb * 2]] = root[hg.bnodes[(size_t)rb * 2 + 1]] = 1;
    std::vector<int32_t> inner, outer;
    for (int i = 0; i < n; i++) (root[i] ? outer : inner).push_back(i);
    if (inner.empty() || outer.empty()) return false;
    Build b(hg, pat);
    b.cut(inner);
    const int nf = (int)b.f.size();
    sp.n = n;
    sp.m = (int)outer.size();
    sp.nI = (int)inner.size();
    sp.nfront = nf;
    // fronts by level
    std::vector<int32_t> order(nf), at(nf);
    for (int q = 0; q < nf; q++) order[q] = q;
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
    sp.fronts.resize(nf);
    for (int q = 0; q < nf; q++) {
        Build::F &s = b.f[order[q]];
        std::sort(s.R.begin(), s.R.end(), [&](int x, int y) { return sp.pos[x] < sp.pos[y]; });
        SubFront &t = sp.fronts[q];
        t.e = (int)s.E.size();
        t.r = (int)s.R.size();
        t.nd0 = t.e ? sp.pos[s.E[0]] : 0;
        t.ch0 = s.ch0 >= 0 ? at[s.ch0] : -1;
        t.ch1 = s.ch1 >= 0 ? at[s.ch1] : -1;
        t.pad = 0;
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
        auto inverse = [&](int ch) {
            const int o = (int)sp.inv.size();
            if (ch < 0) return 0;
            const std::vector<int32_t> &cr = b.f[order[ch]].R;
            for (size_t z = 0; z < cr.size(); z++) local[cr[z]] = (int)z;
            for (int v : s.E) sp.inv.push_back(local[v]);
            for (int v : s.R) sp.inv.push_back(local[v]);
            for (int v : cr) local[v] = -1;
            return o;
        };
        t.inv0 = inverse(t.ch0);
        t.inv1 = inverse(t.ch1);
    }
    // matrix entries, each in the front that eliminates its earlier node
    std::vector<std::vector<int32_t>> own(nf);
    std::vector<int32_t> root_p;
    for (int p = 0; p < pat.nnz; p++) {
        if (pat.col[p] < 0) continue;
        const int i = pat.row[p], c = pat.col[p];
        const int first = sp.pos[i] < sp.pos[c] ? i : c;
        if (b.owner[first] < 0) root_p.push_back(p);
        else own[at[b.owner[first]]].push_back(p);
    }
    for (int q = 0; q < nf; q++) {
        const Build::F &s = b.f[order[q]];
        for (size_t z = 0; z < s.E.size(); z++) local[s.E[z]] = (int)z;
        for (size_t z = 0; z < s.R.size(); z++) local[s.R[z]] = (int)(s.E.size() + z);
        SubFront &t = sp.fronts[q];
        t.ent0 = (int)sp.ent.size();
        t.nent = (int)own[q].size();
        for (int p : own[q]) {
            const int a = local[pat.row[p]], c = local[pat.col[p]];
            sp.ent.push_back({p, std::min(a, c), std::max(a, c)});
        }
        for (int v : s.E) local[v] = -1;
        for (int v : s.R) local[v] = -1;
    }
    // the root: its entries, the last front's rows in it, the boundary terms by column
    sp.root_ent0 = (int)sp.ent.size();
    sp.root_child = nf - 1;
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
    sp.lG.assign(1, 0);
    sp.lS = sp.lU = sp.lD = sp.lG;
    for (int lv = 0; lv < sp.nlevel; lv++) {
        for (int q = sp.level[lv]; q < sp.level[lv + 1]; q++) {
            const SubFront &t = sp.fronts[q];
            const int te = tiles(t.e), tr2 = tiles(t.r);
            for (int i = 0; i < te; i++) {
                sp.tD.push_back({q, i, 0});
                for (int j = 0; j < tr2; j++) sp.tG.push_back({q, i, j});
            }
            for (int i = 0; i < tr2; i++) {
                for (int j = 0; j <= i; j++) sp.tS.push_back({q, i, j});
            }
            for (int i = 0; i < std::max(1, tr2); i++) sp.tU.push_back({q, i, 0});
        }
        sp.lG.push_back((int)sp.tG.size());
        sp.lS.push_back((int)sp.tS.size());
        sp.lU.push_back((int)sp.tU.size());
        sp.lD.push_back((int)sp.tD.size());
    }
    return true;
}

}  // namespace crgpu

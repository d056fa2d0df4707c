// The frequency plan of the weight-anchored G2 sum (pgx_g2a.cu): which points a
// call evaluates, which z1' and z3' they hold, and the classes of points whose
// contractions are one product.  Host code only, so that it can be compiled and
// checked without a GPU.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <iterator>
#include <map>
#include <tuple>
#include <unordered_map>
#include <utility>
#include <vector>

#include "pgx_common.cuh"
#include "pgx_numbers.h"

namespace pgx {

// A contraction class (see pgx_g2a.cu): groups of a plan whose points carry the
// same frequency sums.
struct CClass {
    int term;          // index into the DTerm list
    int nrows, ncols;  // rows (groups) and columns (frequency sums) of the class
    const cd* s;       // ncols frequency sums
    const int* rows;   // nrows group indices
    const int* slots;  // nrows x ncols triple ids (row-major), -1 where absent
};
constexpr int CG_BN_MAX = 32;  // columns of a class; one with more is split into column chunks

// The values of z1, z2 and -z3 in a call, numbered per axis, those that occur
// first; for a real Hamiltonian their conjugates after them.
struct Values {
    std::vector<cd> val[3];
    std::vector<int> cj[3];  // value -> its conjugate
    std::vector<int> id[3];  // triple -> value
    int occur[3] = {0, 0, 0};
};

// The evaluation points of a call.  Values of z1, z2 and -z3 are numbered per
// axis (`val`), and a point is three numbers (`id`).  For a real Hamiltonian
// every matrix element and energy is real, so a part's sum at the conjugate
// triple is the conjugate of its sum (the resonant test |D| <= PoleResolution
// is the same at both).  Triples are therefore taken up to conjugation: class
// u has the points u (its triple) and ncls + u (the conjugate), each
// permutation evaluates the one of the two whose z1' has a positive imaginary
// part, and the class's value is out[u] + conj(out[ncls + u]).  On a grid that
// holds the conjugates of its frequencies this halves the z1' of every
// permutation, and with them the stacked products, the contractions and the
// workspace: Anderson 1+5, 16^3: 11.9 -> 7.3
// ms; the 8-site ring's largest chain, 16^3, split products: 288 -> 158 ms.  A
// complex Hamiltonian has the triples themselves as classes, in order, without
// conjugates.
struct Points {
    int ncls = 0, npts = 0;
    std::vector<cd> val[3];
    std::vector<int> cj[3];        // per axis: value -> its conjugate (real Hamiltonians only)
    std::vector<int> id[3];        // per axis: point -> value
    std::vector<int> cls;          // triple of the call -> class
    std::vector<char> flip;        // the triple is the conjugate of its class's
    cd at(int axis, int e) const { return val[axis][id[axis][e]]; }
};

inline void number_values(Values& v, int nfreq, const double* z, bool real) {
    for (int k = 0; k < 3; ++k) {
        CdMap seen;
        auto& val = v.val[k];
        auto& tid = v.id[k];
        auto& cj = v.cj[k];
        auto number = [&](cd x) {
            const auto it = seen.emplace(cd_key(x), (int)val.size());
            if (it.second) val.push_back(cd{x.x + 0.0, x.y + 0.0});
            return it.first->second;
        };
        const double s = k == 2 ? -1.0 : 1.0;
        tid.resize(nfreq);
        for (int t = 0; t < nfreq; ++t) {
            const double* p = z + 6 * (size_t)t + 2 * k;
            tid[t] = t > 0 && p[0] == p[-6] && p[1] == p[-5] ? tid[t - 1] : number(cd{s * p[0], s * p[1]});
        }
        v.occur[k] = (int)val.size();
        if (real)
            for (size_t i = 0; i < val.size(); ++i) {
                const int j = number(conj(val[i]));
                cj.resize(std::max(cj.size(), std::max(i, (size_t)j) + 1));
                cj[i] = j;
                cj[j] = (int)i;
            }
    }
}

inline void build_points(Points& pt, Values v, int nfreq, bool real) {
    std::vector<int>* tid = v.id;
    auto& cj = pt.cj;
    for (int k = 0; k < 3; ++k) {
        pt.val[k] = std::move(v.val[k]);
        pt.cj[k] = std::move(v.cj[k]);
    }
    pt.cls.resize(nfreq);
    pt.flip.assign(nfreq, 0);
    if (!real) {
        pt.ncls = pt.npts = nfreq;
        for (int k = 0; k < 3; ++k) pt.id[k] = std::move(tid[k]);
        for (int t = 0; t < nfreq; ++t) pt.cls[t] = t;
        return;
    }
    CdMap seen;
    seen.reserve(nfreq);
    std::vector<int> rep;  // class -> its first triple
    for (int t = 0; t < nfreq; ++t) {
        const CdKey key{(unsigned long long)tid[0][t] << 32 | (unsigned)tid[1][t], (unsigned long long)tid[2][t]};
        const CdKey ckey{(unsigned long long)cj[0][tid[0][t]] << 32 | (unsigned)cj[1][tid[1][t]],
                         (unsigned long long)cj[2][tid[2][t]]};
        auto it = seen.find(ckey);
        if (it != seen.end() && !(ckey == key)) {
            pt.cls[t] = it->second;
            pt.flip[t] = 1;
            continue;
        }
        const auto in = seen.emplace(key, (int)rep.size());
        if (in.second) rep.push_back(t);
        pt.cls[t] = in.first->second;
    }
    pt.ncls = (int)rep.size();
    pt.npts = 2 * pt.ncls;
    for (int k = 0; k < 3; ++k) {
        pt.id[k].resize(pt.npts);
        for (int u = 0; u < pt.ncls; ++u) {
            pt.id[k][u] = tid[k][rep[u]];
            pt.id[k][pt.ncls + u] = cj[k][tid[k][rep[u]]];
        }
    }
}
inline void build_points(Points& pt, int nfreq, const double* z, bool real) {
    Values v;
    number_values(v, nfreq, z, real);
    build_points(pt, std::move(v), nfreq, real);
}

// The points a permutation evaluates (one per class), their distinct z1' and
// z3' in order of first appearance, and each point's index into them.  Per
// point also the numbers of the four frequency sums the contractions use: z2',
// z1'+z2'+z3', z1'+z2', z2'+z3', where (z1', z2', z3') is the permuted (z1, z2,
// -z3), z1' dressing O1 and z3' dressing O3.  Sums equal up to rounding have one
// number; the values of z2' are the caller's and keep theirs.  Numbers ascend
// with order_values's order.
struct PermIndex {
    std::vector<int> pts;
    std::vector<cd> Z1, Z3;
    std::vector<int> j1, j3;
    std::vector<int> conj3;   // z3' -> index of its conjugate in Z3 (itself on the real axis), -1 where there is none
    std::vector<int> sid[4];  // sum k of point e (of pts): number sid[k][e]
    std::vector<cd> sval[4];  // its value
    std::vector<double> size[4];  // the largest part of what it was added up from
};
inline double largest_part(cd v) { return std::max(std::fabs(v.x), std::fabs(v.y)); }

// Numbers of x + y over the pairs (i, j) that occur: `val` receives a value
// per distinct pair, `id` each point's pair.  A pair is added once, so the
// cost per point is a table lookup.
inline void number_pairs(const std::vector<int>& pts, const std::vector<int>& xi, const std::vector<cd>& xv,
                  const std::vector<int>& yi, const std::vector<cd>& yv, const std::vector<double>* xs,
                  std::vector<int>& id, std::vector<cd>& val, std::vector<double>& size) {
    const size_t ny = yv.size(), cells = xv.size() * ny;
    std::vector<int> dense(cells <= (size_t(1) << 20) ? cells : 0, -1);
    std::unordered_map<size_t, int> sparse;
    for (int e : pts) {
        const size_t cell = (size_t)xi[e] * ny + yi[e];
        int& q = dense.empty() ? sparse.emplace(cell, -1).first->second : dense[cell];
        if (q < 0) {
            q = (int)val.size();
            val.push_back(xv[xi[e]] + yv[yi[e]]);
            size.push_back(std::max(xs ? (*xs)[xi[e]] : largest_part(xv[xi[e]]), largest_part(yv[yi[e]])));
        }
        id[e] = q;
    }
}

// Orders the numbers by value and merges those of sums equal up to rounding: of
// values no further apart than `ulps` units in the last place of what the
// larger-sized one was added up from, that one takes the number of the
// smaller-sized, which is the more accurate.  So no sum moves by more than its
// own rounding, whatever else the list holds.  Undefined and infinite values
// are merged with none.  The order is that of x + c y: two values close in both
// parts are close in it, and others seldom are (on the axis it is that of y).
inline void order_values(const std::vector<int>& pts, std::vector<int>& id, std::vector<cd>& val,
                         std::vector<double>& size, int ulps) {
    const int n = (int)val.size();
    std::vector<std::pair<double, int>> key;  // finite values in order
    std::vector<int> rep(n), to(n), run;
    double most = 0.0;
    for (int i = 0; i < n; ++i) {
        rep[i] = i;
        const double k = val[i].x + 0.6180339887498949 * val[i].y;
        if (!std::isfinite(k)) continue;
        key.emplace_back(k, i);
        most = std::max(most, size[i]);
    }
    std::sort(key.begin(), key.end());
    const double unit = ulps * std::ldexp(1.0, -52), reach = 2.0 * unit * most;
    for (size_t a = 0, b; ulps > 0 && a < key.size(); a = b) {
        for (b = a + 1; b < key.size() && key[b].first - key[b - 1].first <= reach; ++b) {}
        if (b - a < 2) continue;  // merges are within runs of such neighbours
        run.clear();
        for (size_t q = a; q < b; ++q) run.push_back((int)q);
        std::sort(run.begin(), run.end(),
                  [&](int p, int q) { return std::tie(size[key[p].second], p) < std::tie(size[key[q].second], q); });
        std::multimap<double, int> stand;  // values that keep their number
        for (int q : run) {
            const int i = key[q].second;
            const double tol = unit * size[i], at = key[q].first;
            auto it = stand.lower_bound(at - 2.0 * tol);
            for (; it != stand.end() && it->first <= at + 2.0 * tol; ++it) {
                const cd v = val[it->second];
                if (std::fabs(v.x - val[i].x) <= tol && std::fabs(v.y - val[i].y) <= tol) break;
            }
            if (it != stand.end() && it->first <= at + 2.0 * tol) rep[i] = it->second;
            else stand.emplace(at, i);
        }
    }
    std::vector<cd> out;
    std::vector<double> osize;
    auto keep = [&](int i) {
        to[i] = (int)out.size();
        out.push_back(val[i]);
        osize.push_back(size[i]);
    };
    for (const auto& k : key)
        if (rep[k.second] == k.second) keep(k.second);
    for (int i = 0; i < n; ++i) {
        if (!std::isfinite(val[i].x + 0.6180339887498949 * val[i].y)) keep(i);
        else to[i] = to[rep[i]];
    }
    for (int e : pts) id[e] = to[id[e]];
    val = std::move(out);
    size = std::move(osize);
}

inline void index_perm(PermIndex& ix, const int perm[3], const Points& pt) {
    ix.pts.resize(pt.ncls);
    for (int u = 0; u < pt.ncls; ++u) {
        int e = u;
        if (pt.npts > pt.ncls) {
            const double y1 = pt.at(perm[0], u).y, y3 = pt.at(perm[2], u).y;
            if (y1 < 0.0 || (y1 == 0.0 && y3 < 0.0)) e = pt.ncls + u;
        }
        ix.pts[u] = e;
    }
    auto order = [&](int axis, std::vector<cd>& Z, std::vector<int>& j) {
        std::vector<int> at(pt.val[axis].size(), -1);
        j.assign(pt.npts, -1);
        for (int e : ix.pts) {
            int& q = at[pt.id[axis][e]];
            if (q < 0) {
                q = (int)Z.size();
                Z.push_back(pt.at(axis, e));
            }
            j[e] = q;
        }
    };
    order(perm[0], ix.Z1, ix.j1);
    order(perm[2], ix.Z3, ix.j3);
    // conjugates by number, so that undefined values, which compare equal to
    // nothing, pair with their own bits only
    ix.conj3.assign(ix.Z3.size(), -1);
    if (!pt.cj[perm[2]].empty()) {
        std::vector<int> at(pt.val[perm[2]].size(), -1);
        for (int e : ix.pts) at[pt.id[perm[2]][e]] = ix.j3[e];
        for (int e : ix.pts) ix.conj3[ix.j3[e]] = at[pt.cj[perm[2]][pt.id[perm[2]][e]]];
    }
    order(perm[1], ix.sval[0], ix.sid[0]);
}

// The numbers of the sums (after index_perm).
inline void number_sums(PermIndex& ix) {
    const std::vector<int> j2 = ix.sid[0];
    const std::vector<cd> Z2 = ix.sval[0];
    for (auto& v : ix.sid) v.resize(j2.size());
    for (const cd& v : Z2) ix.size[0].push_back(largest_part(v));
    // An odd multiple of pi / beta, a product and a quotient, is off by up to one
    // unit, a sum of two by three, of three by five and a half.  Eight units apart
    // join all but the rarest of equal sums (apart they cost a column each).
    auto order = [&](int k) { order_values(ix.pts, ix.sid[k], ix.sval[k], ix.size[k], k == 0 ? 0 : 8); };
    order(0);
    number_pairs(ix.pts, ix.j1, ix.Z1, j2, Z2, nullptr, ix.sid[2], ix.sval[2], ix.size[2]);
    order(2);
    number_pairs(ix.pts, ix.sid[2], ix.sval[2], ix.j3, ix.Z3, &ix.size[2], ix.sid[1], ix.sval[1], ix.size[1]);
    order(1);
    number_pairs(ix.pts, j2, Z2, ix.j3, ix.Z3, nullptr, ix.sid[3], ix.sval[3], ix.size[3]);
    order(3);
}

// What the device needs of all plans of a call, gathered on the host and
// uploaded at once; until then pointers are offsets into it.
struct Blob {
    std::vector<char> h;
    template <typename T> T* put(const T* src, size_t n) {
        const size_t at = (h.size() + 15) & ~size_t(15);
        h.resize(at);
        h.insert(h.end(), reinterpret_cast<const char*>(src), reinterpret_cast<const char*>(src + n));
        return reinterpret_cast<T*>(at);
    }
    template <typename T> T* put(const std::vector<T>& v) { return put(v.data(), v.size()); }
};
template <typename T> void rebase(T*& p, char* base) {
    p = reinterpret_cast<T*>(base + reinterpret_cast<size_t>(p));
}

// The points of one tile of a permutation's (z1', z3') plane: z1' indices
// [o1, o1 + n1) and z3' indices [o3, o3 + n3) of its PermIndex, the points
// grouped by (z1', z3'), and the contraction classes per frequency sum (term
// unset).
struct APlan {
    std::vector<cd> Z1, Z3;
    std::vector<int> gt, goff, gi1, gi3;  // points grouped by (i1, i3)
    // For a real Hamiltonian the first n3p of Z3 lie above the real axis, the
    // next n3p are their conjugates in order, and the rest have none in Z3.
    int n3p = 0;
    cd *dZ1 = nullptr, *dZ3 = nullptr;
    int *dgi1 = nullptr, *dgi3 = nullptr;
    std::vector<CClass> cls[4];
};

// Contraction classes of one plan for frequency sum k: the (z1, z3) groups
// whose points carry the same sums form a class, columns ordered by sum, split
// into chunks of at most CG_BN_MAX columns.
inline void build_classes(APlan& pl, int k, const PermIndex& ix, Blob& blob) {
    const std::vector<int>& sid = ix.sid[k];
    struct HC {
        std::vector<int> s, rows, slots;  // sum numbers; groups; points, row by row
    };
    std::unordered_multimap<size_t, int> idx;  // hash of a list of sums -> class
    std::vector<HC> hc;
    const int ng = (int)pl.gi1.size();
    std::vector<std::pair<int, int>> el;
    std::vector<int> ids, pts;
    int ci = -1;
    for (int g = 0; g < ng; ++g) {
        const int* t = pl.gt.data() + pl.goff[g];
        const int n = pl.goff[g + 1] - pl.goff[g];
        ids.resize(n);
        bool ordered = true;
        for (int i = 0; i < n; ++i) {
            ids[i] = sid[t[i]];
            ordered = ordered && (i == 0 || ids[i - 1] <= ids[i]);
        }
        if (!ordered) {
            el.clear();
            for (int i = 0; i < n; ++i) el.emplace_back(ids[i], t[i]);
            std::sort(el.begin(), el.end());
            pts.resize(n);
            for (int i = 0; i < n; ++i) {
                ids[i] = el[i].first;
                pts[i] = el[i].second;
            }
            t = pts.data();
        }
        if (ci < 0 || hc[ci].s != ids) {  // most often the class of the group before
            size_t h = n;
            for (int x : ids) h = (h ^ (size_t)x) * 0x9E3779B97F4A7C15ull;
            ci = -1;
            for (auto r = idx.equal_range(h); r.first != r.second && ci < 0; ++r.first)
                if (hc[r.first->second].s == ids) ci = r.first->second;
            if (ci < 0) {
                ci = (int)hc.size();
                idx.emplace(h, ci);
                hc.emplace_back();
                hc.back().s = ids;
            }
        }
        hc[ci].rows.push_back(g);
        hc[ci].slots.insert(hc[ci].slots.end(), t, t + n);
    }
    std::sort(hc.begin(), hc.end(), [](const HC& x, const HC& y) { return x.s < y.s; });
    // Classes of few rows (such as the z1 + z3 classes of the T2 sub-terms
    // near the grid's corners) make 8- or 16-row tiles that leave the FP64 pipe
    // idle.  Consecutive ones, in the order of their sum lists, are merged while
    // the union of their sums stays within CG_BN_MAX columns and their rows
    // within 64; a merged row holds -1 in the columns that are not its own, so
    // its tile computes those products and drops them.
    std::vector<HC> merged;
    {
        std::vector<int> both;
        auto unite = [&](std::vector<int>& u, const std::vector<int>& v) {
            both.clear();
            std::set_union(u.begin(), u.end(), v.begin(), v.end(), std::back_inserter(both));
            return (int)both.size();
        };
        // groups of consecutive small classes under a row cap (sums within CG_BN_MAX)
        auto split_run = [&](const std::vector<int>& run, int cap) {
            std::vector<std::vector<int>> out;
            std::vector<int> uni;
            int rows = 0;
            for (int ci : run) {
                const int r = (int)hc[ci].rows.size();
                if (out.empty() || unite(uni, hc[ci].s) > CG_BN_MAX || rows + r > cap) {
                    out.emplace_back();
                    uni = hc[ci].s;
                    rows = 0;
                } else {
                    uni = both;
                }
                out.back().push_back(ci);
                rows += r;
            }
            return out;
        };
        auto emit = [&](const std::vector<int>& group) {
            if (group.size() == 1) {
                merged.push_back(std::move(hc[group[0]]));
                return;
            }
            HC m;
            for (int ci : group) {
                unite(m.s, hc[ci].s);
                m.s = both;
            }
            const int w = (int)m.s.size();
            for (int ci : group) {
                const HC& c = hc[ci];
                const int nc = (int)c.s.size();
                for (size_t r = 0; r < c.rows.size(); ++r) {
                    m.rows.push_back(c.rows[r]);
                    const size_t base = m.slots.size();
                    m.slots.resize(base + w, -1);
                    for (int j = 0, col = 0; j < nc; ++j) {
                        while (m.s[col] != c.s[j]) ++col;
                        m.slots[base + col] = c.slots[r * nc + j];
                    }
                }
            }
            merged.push_back(std::move(m));
        };
        // a run of consecutive small classes is cut into as few groups as 64
        // rows allow, then re-cut with the rows spread evenly over that many
        // groups, so that no group is left with a few rows
        auto flush_run = [&](std::vector<int>& run) {
            if (run.empty()) return;
            int total = 0, big = 0;
            for (int ci : run) {
                total += (int)hc[ci].rows.size();
                big = std::max(big, (int)hc[ci].rows.size());
            }
            const int ng2 = (int)split_run(run, 64).size();
            const int cap = std::max(big, (total + ng2 - 1) / ng2);
            for (const auto& g : split_run(run, cap)) emit(g);
            run.clear();
        };
        std::vector<int> run;
        for (int ci = 0; ci < (int)hc.size(); ++ci) {
            const HC& c = hc[ci];
            // large classes, and classes holding one sum twice (one column each
            // in a merged class would collide), stay as they are
            if (c.rows.size() > 16 || std::adjacent_find(c.s.begin(), c.s.end()) != c.s.end()) {
                flush_run(run);
                emit({ci});
                continue;
            }
            run.push_back(ci);
        }
        flush_run(run);
    }
    std::vector<cd> sums;
    std::vector<int> part;
    for (const HC& c : merged) {
        const int nc = (int)c.s.size(), nr = (int)c.rows.size();
        for (int j0 = 0; j0 < nc; j0 += CG_BN_MAX) {
            const int w = std::min(CG_BN_MAX, nc - j0);
            sums.clear();
            for (int j = 0; j < w; ++j) sums.push_back(ix.sval[k][c.s[j0 + j]]);
            if (w < nc) {
                part.clear();
                for (int r = 0; r < nr; ++r)
                    part.insert(part.end(), c.slots.begin() + (size_t)r * nc + j0, c.slots.begin() + (size_t)r * nc + j0 + w);
            }
            const std::vector<int>& slots = w < nc ? part : c.slots;
            CClass f{};
            f.term = -1;
            f.nrows = nr;
            f.ncols = w;
            f.s = blob.put(sums);
            f.rows = blob.put(c.rows);
            f.slots = blob.put(slots);
            pl.cls[k].push_back(f);
        }
    }
}

inline void build_aplan(APlan& pl, const std::vector<int>& pts, const PermIndex& ix, int o1, int n1, int o3, int n3,
                        Blob& blob) {
    pl.Z1.assign(ix.Z1.begin() + o1, ix.Z1.begin() + o1 + n1);
    pl.Z3.assign(ix.Z3.begin() + o3, ix.Z3.begin() + o3 + n3);
    const size_t nt = pts.size();
    // in the order of (j1, j3): by j3, then stably by j1
    pl.gt = pts;
    std::vector<int> start, to(nt);
    auto sort_by = [&](const std::vector<int>& j, int o, int n) {
        start.assign(n + 1, 0);
        for (int t : pl.gt) ++start[j[t] - o + 1];
        for (int i = 0; i < n; ++i) start[i + 1] += start[i];
        for (int t : pl.gt) to[start[j[t] - o]++] = t;
        pl.gt.swap(to);
    };
    sort_by(ix.j3, o3, n3);
    sort_by(ix.j1, o1, n1);
    for (size_t q = 0; q < nt; ++q) {
        const int t = pl.gt[q];
        if (q == 0 || ix.j1[t] != ix.j1[pl.gt[q - 1]] || ix.j3[t] != ix.j3[pl.gt[q - 1]]) {
            pl.goff.push_back((int)q);
            pl.gi1.push_back(ix.j1[t] - o1);
            pl.gi3.push_back(ix.j3[t] - o3);
        }
    }
    pl.goff.push_back((int)nt);
    std::vector<int> order, low, rest;
    for (int i = 0; i < n3; ++i) {
        const int c = ix.conj3[o3 + i] - o3;
        const double y = pl.Z3[i].y;
        if (c < 0 || c >= n3 || !(y > 0.0 || y < 0.0)) {
            rest.push_back(i);
        } else if (y > 0.0) {
            order.push_back(i);
            low.push_back(c);
        }
    }
    PGX_CHECK((int)(order.size() + low.size() + rest.size()) == n3, PGX_ERR_ARG, "G2 plan: unpaired frequencies");
    if (!order.empty()) {
        pl.n3p = (int)order.size();
        order.insert(order.end(), low.begin(), low.end());
        order.insert(order.end(), rest.begin(), rest.end());
        std::vector<int> pos(n3);
        std::vector<cd> Z3(n3);
        for (int i = 0; i < n3; ++i) {
            pos[order[i]] = i;
            Z3[i] = pl.Z3[order[i]];
        }
        pl.Z3 = std::move(Z3);
        for (int& i : pl.gi3) i = pos[i];
    }
    pl.dZ1 = blob.put(pl.Z1);
    pl.dZ3 = blob.put(pl.Z3);
    pl.dgi1 = blob.put(pl.gi1);
    pl.dgi3 = blob.put(pl.gi3);
}

}  // namespace pgx

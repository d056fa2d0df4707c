// The frequency plan of the anchored G2 sum on lists with undefined and
// infinite entries, tiled and untiled: every point in one group with its own z1'
// and z3', the first z3' in conjugate pairs, and every point once per frequency
// sum with that sum.  Built with the library's range checks on.
#include <cstdio>
#include <set>

#include "pgx_g2plan.h"

using namespace pgx;
static int bad = 0;
#define EXPECT(c)                                                \
    do {                                                         \
        if (!(c)) {                                              \
            if (++bad < 20) std::printf("line %d: %s\n", __LINE__, #c); \
        }                                                        \
    } while (0)

static bool same(cd a, cd b) {
    auto eq = [](double x, double y) { return x == y || (std::isnan(x) && std::isnan(y)); };
    return eq(a.x, b.x) && eq(a.y, b.y);
}
static bool finite(cd a) { return std::isfinite(a.x) && std::isfinite(a.y); }
template <typename T> static const T* in(const Blob& b, const T* p) {
    return reinterpret_cast<const T*>(b.h.data() + reinterpret_cast<size_t>(p));
}

static void check(const std::vector<double>& z, bool real, int tiles1, int tiles3) {
    static const int perms[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
    const int nfreq = (int)(z.size() / 6);
    Points pt;
    build_points(pt, nfreq, z.data(), real);
    for (int t = 0; t < nfreq; ++t)  // a triple's class holds its own value, or its conjugate's
        for (int k = 0; k < 3; ++k) {
            const double s = k == 2 ? -1.0 : 1.0;
            const cd v{s * z[6 * t + 2 * k], s * z[6 * t + 2 * k + 1]};
            EXPECT(same(pt.at(k, pt.flip[t] ? pt.ncls + pt.cls[t] : pt.cls[t]), v));
        }
    for (const auto& perm : perms) {
        PermIndex ix;
        index_perm(ix, perm, pt);
        number_sums(ix);
        const int N1 = (int)ix.Z1.size(), N3 = (int)ix.Z3.size();
        const int b1 = (N1 + tiles1 - 1) / tiles1, b3 = (N3 + tiles3 - 1) / tiles3;
        std::set<int> all;
        for (int o1 = 0; o1 < N1; o1 += b1)
            for (int o3 = 0; o3 < N3; o3 += b3) {
                const int n1 = std::min(b1, N1 - o1), n3 = std::min(b3, N3 - o3);
                std::vector<int> mine;
                for (int e : ix.pts)
                    if (ix.j1[e] / b1 == o1 / b1 && ix.j3[e] / b3 == o3 / b3) mine.push_back(e);
                if (mine.empty()) continue;
                APlan pl;
                Blob blob;
                build_aplan(pl, mine, ix, o1, n1, o3, n3, blob);
                EXPECT((int)pl.Z3.size() == n3 && 2 * pl.n3p <= n3);
                for (int i = 0; i < pl.n3p; ++i) EXPECT(same(pl.Z3[pl.n3p + i], conj(pl.Z3[i])));
                for (int i = 0; i < n3; ++i) {
                    int n = 0;
                    for (int j = 0; j < n3; ++j) n += same(pl.Z3[j], ix.Z3[o3 + i]);
                    EXPECT(n == 1);
                }
                for (size_t g = 0; g < pl.gi1.size(); ++g)
                    for (int u = pl.goff[g]; u < pl.goff[g + 1]; ++u) {
                        const int e = pl.gt[u];
                        EXPECT(all.insert(e).second);
                        EXPECT(same(pl.Z1.at(pl.gi1[g]), pt.at(perm[0], e)));
                        EXPECT(same(pl.Z3.at(pl.gi3[g]), pt.at(perm[2], e)));
                    }
                for (int k = 0; k < 4; ++k) {
                    build_classes(pl, k, ix, blob);
                    std::set<int> seen;
                    for (const CClass& c : pl.cls[k]) {
                        EXPECT(c.ncols >= 1 && c.ncols <= CG_BN_MAX);
                        for (int r = 0; r < c.nrows; ++r)
                            for (int j = 0; j < c.ncols; ++j) {
                                const int e = in(blob, c.slots)[r * c.ncols + j];
                                if (e < 0) continue;
                                EXPECT(seen.insert(e).second);
                                const int g = in(blob, c.rows)[r];
                                EXPECT(same(pl.Z1.at(pl.gi1[g]), pt.at(perm[0], e)));
                                EXPECT(same(pl.Z3.at(pl.gi3[g]), pt.at(perm[2], e)));
                                const cd a = pt.at(perm[0], e), b = pt.at(perm[1], e), d = pt.at(perm[2], e);
                                const cd sum = k == 0 ? b : k == 1 ? a + b + d : k == 2 ? a + b : b + d;
                                if (!finite(sum)) continue;
                                const cd s = in(blob, c.s)[j];
                                double size = std::max(std::fabs(b.x), std::fabs(b.y));
                                if (k == 1 || k == 2) size = std::max(size, std::max(std::fabs(a.x), std::fabs(a.y)));
                                if (k == 1 || k == 3) size = std::max(size, std::max(std::fabs(d.x), std::fabs(d.y)));
                                const double tol = k == 0 ? 0.0 : std::ldexp(size, -48);  // two merges of eight units
                                EXPECT(std::fabs(s.x - sum.x) <= tol && std::fabs(s.y - sum.y) <= tol);
                            }
                    }
                    EXPECT(seen.size() == mine.size());
                }
            }
        EXPECT((int)all.size() == pt.ncls);
    }
}

int main() {
    const double nan = std::nan(""), inf = INFINITY;
    const cd odd[] = {{nan, nan}, {nan, 1.0}, {0.0, nan}, {inf, 1.0}, {0.0, inf}, {0.0, -inf}, {-inf, nan}, {nan, -3.0}};
    for (int form = 0; form < 3; ++form) {  // all, some or none of its conjugates
        const int lo = form == 0 ? -2 : form == 1 ? -1 : 0, hi = form == 2 ? 4 : 2;
        std::vector<double> z;
        for (int a = lo; a < hi; ++a)
            for (int b = lo; b < hi; ++b)
                for (int c = lo; c < hi; ++c)
                    for (int n : {a, b, c}) {
                        z.push_back(0.0);
                        z.push_back(2 * n + 1);
                    }
        const int nfreq = (int)(z.size() / 6);
        for (int place = -1; place < 4; ++place)  // none; one frequency of a triple; all of them
            for (size_t q = 0; q < sizeof(odd) / sizeof(odd[0]); ++q)
                for (int every : {1000, 7}) {
                    std::vector<double> y = z;
                    for (int t = 3; t < nfreq && place >= 0; t += every)
                        for (int k = 0; k < 3; ++k)
                            if (place == 3 || place == k) {
                                const cd v = place == 3 ? odd[(q + t + k) % (sizeof(odd) / sizeof(odd[0]))] : odd[q];
                                y[6 * t + 2 * k] = v.x;
                                y[6 * t + 2 * k + 1] = v.y;
                            }
                    for (bool real : {true, false})
                        for (int tiles : {1, 3}) check(y, real, tiles, tiles == 1 ? 1 : 2);
                }
    }
    // neighbours of one frequency a few units apart; large opposite addends with
    // small sums; magnitudes far apart: no sum moves by more than its own rounding
    for (int form = 0; form < 4; ++form) {
        std::vector<double> z;
        auto value = [&](int k, int i) {
            if (form == 0) return cd{0.0, (2 * i + 1) * (1.0 + (k == 1 ? i * 3e-16 : 0.0)) * (k == 1 ? 1.0 : 3.0)};
            if (form == 1) return cd{0.25 * i, k == 0 ? 1e14 + i : k == 1 ? -1e14 + 3 * i : 1.0 + i};
            if (form == 2) return cd{0.0, (k == 2 ? 1e-3 : 1.0) * std::ldexp(2 * i + 1.0, 12 * (i % 4))};
            return cd{0.1 * i, 0.05};  // a line above the real axis
        };
        for (int a = 0; a < 6; ++a)
            for (int b = 0; b < 6; ++b)
                for (int c = 0; c < 6; ++c)
                    for (const cd& v : {value(0, a), value(1, b), value(2, c)}) {
                        z.push_back(v.x);
                        z.push_back(v.y);
                    }
        for (bool real : {true, false}) check(z, real, 1, 1);
    }
    // on Matsubara grids every equal sum has one number
    for (double beta : {1.0, 7.0, 10.0, 33.3, 1e3}) {
        const double pi = 3.14159265358979323846;
        for (int reach : {8, 40, 600}) {
            std::vector<double> z;
            std::vector<int> step;
            for (int i = 0; i < 16; ++i) step.push_back(reach <= 8 ? i - 8 : (i - 8) * reach / 8 + i % 3);
            for (int a : step)
                for (int b : step)
                    for (int c : step)
                        for (int n : {a, b, c}) {
                            z.push_back(0.0);
                            z.push_back(pi * (2 * n + 1) / beta);
                        }
            std::set<int> pairs, differences, all;
            for (int a : step)
                for (int b : step) {
                    pairs.insert(a + b + 1);
                    differences.insert(b - a);
                    for (int c : step) all.insert(a + b - c);
                }
            Points pt;
            build_points(pt, (int)z.size() / 6, z.data(), false);
            const int perm[3] = {0, 1, 2};
            PermIndex ix;
            index_perm(ix, perm, pt);
            number_sums(ix);
            EXPECT(ix.sval[0].size() == step.size());
            EXPECT(ix.sval[1].size() == all.size());
            EXPECT(ix.sval[2].size() == pairs.size());
            EXPECT(ix.sval[3].size() == differences.size());
        }
    }
    std::printf("%d failures\n", bad);
    return bad != 0;
}

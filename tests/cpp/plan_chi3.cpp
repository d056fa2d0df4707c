// The order of chi3's second frequencies with undefined and infinite values among
// them: distinct values stay distinct, every entry keeps its value, and each
// mirrored column is the conjugate of one that is computed.
#include <cmath>
#include <cstdio>

#include "pgx_numbers.h"

using namespace pgx;

int main() {
    const double nan = std::nan(""), inf = INFINITY;
    auto eq = [](double a, double b) { return a == b || (std::isnan(a) && std::isnan(b)); };
    auto same = [&](cd a, cd b) { return eq(a.x, b.x) && eq(a.y, b.y); };
    std::vector<cd> pool;
    for (double y : {-3.0, -1.0, 1.0, 3.0, 5.0, -7.0})
        for (double x : {0.0, 0.5}) pool.push_back(cd{x, y});
    for (cd v : {cd{nan, nan}, cd{nan, 3.0}, cd{nan, 7.0}, cd{nan, -5.0}, cd{0.0, nan}, cd{inf, -1.0}, cd{0.0, inf},
                 cd{0.0, -inf}, cd{0.25, 0.0}, cd{0.25, -0.0}})
        pool.push_back(v);
    int bad = 0;
    unsigned rnd = 1;
    for (int trial = 0; trial < 20000; ++trial) {
        std::vector<cd> list;
        for (int n = 1 + trial % 24; n > 0; --n) {
            rnd = rnd * 1664525u + 1013904223u;
            list.push_back(pool[(rnd >> 8) % pool.size()]);
        }
        std::vector<cd> v;
        std::vector<int> idx, src;
        const int n = distinct_index(list, v, idx), nu = conjugates_last(v, idx, src);
        bad += n != (int)v.size() || nu + (int)src.size() != n;
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < i; ++j) bad += same(v[i], v[j]);
        for (size_t q = 0; q < list.size(); ++q) bad += !same(v.at(idx[q]), list[q]);
        for (size_t i = 0; i < src.size(); ++i)
            bad += !(src[i] >= 0 && src[i] < nu && same(v.at(nu + i), conj(v.at(src[i]))));
    }
    std::printf("%d failures\n", bad);
    return bad != 0;
}

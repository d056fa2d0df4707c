// Numbering of complex values by their bits.  Undefined values equal only their
// own bits here; in a map ordered by < a NaN is equivalent to every key and
// disturbs the places of the others.  Host code only.
#pragma once

#include <cstring>
#include <unordered_map>
#include <vector>

#include "pgx_common.cuh"

namespace pgx {

struct CdKey {
    unsigned long long x, y;
    bool operator==(const CdKey& o) const { return x == o.x && y == o.y; }
};
struct CdHash {
    size_t operator()(const CdKey& k) const { return (k.x * 0x9E3779B97F4A7C15ull) ^ (k.y * 0xC2B2AE3D27D4EB4Full >> 7); }
};
inline CdKey cd_key(cd v) {
    v = cd{v.x + 0.0, v.y + 0.0};  // -0 and 0 are one value
    CdKey key;
    std::memcpy(&key, &v, sizeof(key));
    return key;
}
using CdMap = std::unordered_map<CdKey, int, CdHash>;

// Distinct values of a list in order of first appearance, and each entry's
// index into them.
inline int distinct_index(const std::vector<cd>& v, std::vector<cd>& uniq, std::vector<int>& idx) {
    CdMap seen;
    idx.resize(v.size());
    for (size_t q = 0; q < v.size(); ++q) {
        const auto it = seen.emplace(cd_key(v[q]), (int)uniq.size());
        if (it.second) uniq.push_back(v[q]);
        idx[q] = it.first->second;
    }
    return (int)uniq.size();
}

// Reorders distinct values so that those below the real axis whose conjugate is
// among them come last; returns how many come before, and for each of the last
// the place of its conjugate (src).  `idx` (indices into the values) follows.
inline int conjugates_last(std::vector<cd>& v, std::vector<int>& idx, std::vector<int>& src) {
    CdMap at;
    for (size_t b = 0; b < v.size(); ++b) at.emplace(cd_key(v[b]), (int)b);
    std::vector<int> order, low, up, pos(v.size());
    for (size_t b = 0; b < v.size(); ++b) {
        const auto it = v[b].y < 0.0 ? at.find(cd_key(conj(v[b]))) : at.end();
        if (it == at.end()) {
            order.push_back((int)b);
        } else {
            low.push_back((int)b);
            up.push_back(it->second);
        }
    }
    const int n = (int)order.size();
    order.insert(order.end(), low.begin(), low.end());
    std::vector<cd> sorted(v.size());
    for (size_t i = 0; i < v.size(); ++i) {
        pos[order[i]] = (int)i;
        sorted[i] = v[order[i]];
    }
    src.clear();
    for (int u : up) src.push_back(pos[u]);
    v = std::move(sorted);
    for (int& b : idx) b = pos[b];
    return n;
}

}  // namespace pgx

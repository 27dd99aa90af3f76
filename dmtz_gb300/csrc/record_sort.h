// record_sort.h — separatrix records in the order in which they are handed out.
#pragma once
#include <algorithm>
#include <cstddef>
#include <utility>
#include <vector>

namespace dmtz {

// Pairs (a, b) in increasing order, a >= 0: by a's digits of 11 bits, lowest first, then
// runs of equal a by b.  The detection's records arrive in no order, and a comparison sort
// of them took longer than the detection.
inline void sort_records(std::vector<std::pair<long long, long long>> &p) {
    long long top = 0;
    for (const auto &r : p) top = std::max(top, r.first);
    std::vector<std::pair<long long, long long>> q(p.size());
    for (int shift = 0; shift < 63 && (top >> shift) != 0; shift += 11) {
        size_t at[2049] = {};
        for (const auto &r : p) at[((r.first >> shift) & 2047) + 1]++;
        for (int k = 0; k < 2048; k++) at[k + 1] += at[k];
        for (const auto &r : p) q[at[(r.first >> shift) & 2047]++] = r;
        p.swap(q);
    }
    for (size_t i = 0, j; i < p.size(); i = j) {
        for (j = i + 1; j < p.size() && p[j].first == p[i].first;) j++;
        if (j - i > 1) std::sort(p.begin() + i, p.begin() + j);
    }
}

}  // namespace dmtz

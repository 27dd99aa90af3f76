// record_sort.h against std::sort.
#include <cstdio>
#include <random>

#include "../../dmtz_gb300/csrc/record_sort.h"

int main() {
    typedef std::vector<std::pair<long long, long long>> Pairs;
    std::mt19937_64 r(7);
    int bad = 0;
    for (int n : {0, 1, 2, 3, 1000, 50000})
        for (long long top : {1ll, 2ll, 2047ll, 2048ll, 2049ll, (1ll << 22) - 1, 1ll << 22, 1ll << 33, 6ll << 37, (1ll << 62) - 1})
            for (int order = 0; order < 3; order++) {
                Pairs p(n);
                for (auto &x : p) x = {(long long)(r() % (unsigned long long)top), (long long)(r() % 5) - 1};
                if (order == 1) std::sort(p.begin(), p.end());
                if (order == 2) std::sort(p.rbegin(), p.rend());
                Pairs q = p;
                std::sort(q.begin(), q.end());
                dmtz::sort_records(p);
                bad += p != q;
            }
    printf("%d wrong\n", bad);
    return bad != 0;
}

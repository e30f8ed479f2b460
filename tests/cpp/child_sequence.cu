// Host-side check of rq::child_sequence (trace_engine.cuh) against its
// statement, over every hit mask and every choice of entry distances from a
// set that holds ties, negative ones, the largest finite one and infinity.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>

#include "trace_engine.cuh"

int main() {
    const float values[] = {-1.0f, 0.0f, 1.0f, FLT_MAX, INFINITY};
    int bad = 0;
    for (int v = 0; v < 5 * 5 * 5 * 5; ++v)
        for (uint32_t hitm = 0; hitm < 16; ++hitm)
            for (int sorted = 0; sorted < 2; ++sorted) {
                const float t[4] = {values[v % 5], values[v / 5 % 5], values[v / 25 % 5], values[v / 125]};
                int order[4], n = 0;
                for (int k = 0; k < 4; ++k)
                    if ((hitm >> k) & 1u) order[n++] = k;
                if (sorted) std::stable_sort(order, order + n, [&](int a, int b) { return t[a] < t[b]; });
                uint32_t want = 0;
                for (int i = 0; i < n; ++i) want |= uint32_t(4 | order[i]) << (3 * i);
                const uint32_t got = rq::child_sequence<false>(hitm, t, sorted != 0),
                               mixed = rq::child_sequence<true>(hitm, t, sorted != 0);
                if ((got != want || mixed != want) && bad++ < 5)
                    std::printf("hits %x at %g %g %g %g, sorted %d: %o, %o for %o\n", hitm, t[0], t[1], t[2], t[3], sorted,
                                got, mixed, want);
            }
    std::printf("%d of 20000 wrong\n", bad);
    return bad != 0;
}

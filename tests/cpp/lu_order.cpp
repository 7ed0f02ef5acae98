// The row order from a panel's pivots (lu_order.cuh) against the exchanges
// themselves: every first step, panels of 1 to 16 steps, pivots anywhere below.
#include <cstdio>
#include <random>
#include <utility>
#include <vector>

#include "lu_order.cuh"

int main()
{
    std::mt19937 rng(1);
    for (int t = 0; t < 2000; ++t) {
        const int n = 1 + (int)(rng() % 16), rows = n + (int)(rng() % 40);
        std::vector<int> piv(n);
        for (int k = 0; k < n; ++k) piv[k] = k + (int)(rng() % (rows - k));
        for (int first = 0; first <= n; ++first) {
            std::vector<int> at(rows);
            for (int r = 0; r < rows; ++r) at[r] = r;
            for (int k = first; k < n; ++k) std::swap(at[k], at[piv[k]]);
            for (int r = 0; r < rows; ++r)
                if (piro::lu_row_before(piv.data(), first, n, r) != at[r]) {
                    std::printf("panel %d, step %d, row %d\n", t, first, r);
                    return 1;
                }
        }
    }
    return 0;
}

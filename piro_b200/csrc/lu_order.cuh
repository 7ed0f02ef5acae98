// lu_order.cuh -- the row order that a panel's exchanges leave.
//
// Step k of a panel exchanges the rows at positions k and piv[k] >= k (counted
// from the panel's first row).  The order follows from the panel's pivots
// alone, which stay where the factorization stores them: a block that comes to
// a panel late finds them, whatever has been factored since.
#pragma once

#ifdef __CUDACC__
#define PIRO_LU_HD __host__ __device__ __forceinline__
#else
#define PIRO_LU_HD inline
#endif

namespace piro {

// The position, before the exchanges of the steps first .. n - 1, of the row
// that stands at position r after them.
PIRO_LU_HD int lu_row_before(const int *piv, int first, int n, int r)
{
    for (int k = n - 1; k >= first; --k) {
        const int p = piv[k];
        r = r == k ? p : r == p ? k : r;
    }
    return r;
}

}  // namespace piro

// Kronecker inverse of the B-spline overlap, M^-1 = M_z^-1 (x) M_y^-1 (x) M_x^-1,
// by banded Cholesky line solves along each axis. Internal.
#pragma once

#include "space.h"

namespace tdz {

// Banded Cholesky factor of an SPD band: n rows x (p+1), entry j of row i is
// L(i, i-p+j); slot p holds 1/L(i, i).
struct BandChol {
    int n = 0, p = 0;
    std::vector<double> L;
    DevBuf L32, L64;
    DevBuf R32, R64;   // the rows of both recurrences scaled by 1/L(i, i) (linesolve.cu)
    void factor(const BandD &A);   // throws if A is not SPD
    void upload();
};

// Epilogue of a Chebyshev step on the solution z: d = a z + b d, x = d (set)
// or x + d. z itself is stored only with keep.
struct ChebStep {
    cd a, b;
    void *d, *x;
    bool set, keep;
};

// dst = (A_axis^-1 along one axis) src for an array of shape (n2, n1, n0), x
// fastest; dst may be src. With ch the epilogue takes the place of the store
// of dst where the kernel can (returns true); dst then holds z only with keep.
bool line_solve(const BandChol &F, int axis, const void *src, void *dst, int n0, int n1, int n2, int prec,
                cudaStream_t st, const ChebStep *ch = nullptr);

// Kronecker solve with one factor per axis (dim axes).
struct KronSolve {
    int dim = 0, n[3] = {1, 1, 1};
    BandChol f[3];
    void setup(const std::array<const BandD *, 3> &bands, int dim_);
    void apply(void *x, int prec, cudaStream_t st) const { apply(x, x, prec, st); }   // in place
    // x = M^-1 src (src may be x); with ch, x is scratch and the epilogue runs
    // on the solution, fused into the last axis's stores where it can be
    void apply(const void *src, void *x, int prec, cudaStream_t st, const ChebStep *ch = nullptr) const;
};

}  // namespace tdz

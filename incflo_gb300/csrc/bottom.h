// The coarsest level of a multigrid hierarchy (nodal or cell-centred): its operator as rows of a fixed number of
// entries, rebuilt on the device whenever the coefficients change, and the two solvers on it:
//   - up to kDenseBottom unknowns (nodal: kDenseNodal): the dense FP64 inverse (Gauss-Jordan in one CTA), applied as one product;
//   - above: Jacobi-preconditioned conjugate gradients in FP64 by one thread-block cluster (bottom_cg).
#pragma once

#include <cuda_runtime.h>

#include "gbp_internal.cuh"

namespace gbp {

// n unknowns: the inverse costs n^3 / 2 FP64 multiply-adds on one SM (2 per clock: about 75 us for 64, 230 us for 108, 480 us for
// 125) per coefficient set and a product of 1 to 3 us per V-cycle, where the cluster's conjugate gradients take 25 to 100 us per
// V-cycle; and a dense bottom lets the cluster tail cycle the small levels (MAC 112 x 16 x 24 cells, 84 unknowns: 3.7 ms
// per projection without, 1.5 with; 48 x 24 x 48, 108 unknowns: 1.84 and 1.27; 40^3, 125 unknowns: 1.6 and 1.4, and 1.6 and 0.9
// where the coefficients stay; nodal 112 x 48 x 48, 128 unknowns, whose sigma is set for every projection: 1.65 and 1.90). The
// limit of the cell-centred hierarchies is what one thread block's registers hold without a spill. (The inverse of up to 216
// unknowns by the host took 0.3 to 10 ms per coefficient set.)
constexpr int kDenseBottom = 127, kDenseNodal = 112;
// most unknowns of the cluster solver: the search direction is replicated in every CTA's shared memory
constexpr int kClusterBottom = 16384;
constexpr int kBottomThreads = 1024;

struct BottomRows {
    int n = 0, w = 0;          // unknowns, entries per row (27 nodal, 7 cell-centred)
    double* coef = nullptr;    // [w][n]
    int* idx = nullptr;        // [w][n] unknown of each entry
    double* diag = nullptr;    // [n]
    double* weight = nullptr;  // [n] null-space weight of each unknown (node volume / 1), 0: no equation (held at 0)
    size_t bytes() const { return (size_t)n * w * 12 + (size_t)n * 16 + 1024; }
    void carve(char* base);    // sets the arrays inside `bytes()` bytes at base (256-byte aligned)
};

// *empty += unknowns that are not held but have an empty row (sigma 0 in all their cells)
void bottom_rows_nodal(const NodalGeom& g, const double* s64, const BottomRows& r, unsigned* empty, cudaStream_t st);
void bottom_rows_mac(const CellGeom& g, const double* bx, const double* by, const double* bz, const BottomRows& r,
                     cudaStream_t st);
// M (n x n) = inverse of the rows' matrix (singular: of A + c 1 1^T over the unknowns that carry an equation), rows and
// columns of held unknowns 0; act (may be null): 1 where an unknown carries an equation. *bad = 1 when a pivot is 0.
void bottom_inverse(const BottomRows& r, int singular, double* M, unsigned char* act, unsigned* bad, cudaStream_t st);

struct BottomCG {
    BottomRows r;
    int singular, maxiter;
    double rtol, atol;
    int* info;  // most iterations so far (nullptr: not kept)
};
// x = A^-1 b on the coarsest level by one cluster
template <typename T>
int bottom_cg_nodal(const NodalGeom& g, const BottomCG& c, const T* b, T* x, cudaStream_t st);
template <typename T>
int bottom_cg_mac(const CellGeom& g, const BottomCG& c, const T* b, T* x, cudaStream_t st);

}  // namespace gbp

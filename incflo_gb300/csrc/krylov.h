// Conjugate-gradient acceleration of the multigrid solves: the vector kernels between the V-cycle (the preconditioner
// z = V r) and the operator q = -A p (the sign the residual kernels give with no right-hand side), on the padded layouts
// of the nodal and cell-centred levels.
//
// Flexible form: beta = (z.q) / (p.Ap) of the last direction makes the new one conjugate to it, and alpha = (r.p) / (p.Ap)
// is the exact minimum along it. Neither assumes that r is orthogonal to the last direction (as alpha = r.z / p.Ap and
// beta = z.(r_new - r_old) / (r.z)_old do): between two refinement steps of an FP32 solve the recursion's residual is
// replaced by the true one, and a solve that reached its rounding has lost the orthogonality anyway. With those forms the
// iteration kept its wrong steps from there on: 20 to 40 V-cycles instead of 8 on 2^3 cells, where a V-cycle is an exact
// solve, or a residual that grew from step to step. The scalars stay on the device (no host round trip inside an
// iteration); the dot products are folded in a fixed order by the last block to finish, so a solve is reproducible bit by
// bit.
//
// With a V-cycle that contracts the error by rho per application, the stationary iteration needs log(tol) / log(rho)
// of them; the accelerated one removes the few slow modes that set rho (a density jump, cut cells, stretched cells):
// V(2,2) cycles on the 256^3 interface problem 10 -> 7 (nodal, FP64, to 1e-10) and 12 -> 9 (MAC, FP64; FP32 in FP64
// 12 -> 10), to 1e-11 around a cylinder 22 -> 11 (nodal) and 13 -> 10 (MAC), on cells of aspect 1 : 0.8 : 1.25
// 38 -> 16 (both).
#pragma once

#include <cuda_runtime.h>

namespace gbp {

// unique points of a padded array: n0 x n1 x n2 from index (0, 0, 0), rows sy apart, planes sz apart
struct KrylovBox {
    int n[3];
    long long sy, sz, count;
    double null_inv;  // 1 / the number of unknowns of a system whose null space are the constants, or 0 (krylov_alpha)
};

struct KrylovState {
    double pap, alpha, beta;
    int it, restart;
    int plain;  // 1: stationary steps (beta 0, alpha 1)
    unsigned done[2];  // blocks that finished a dot product (reset by the last one)
    // power-of-two scale of an FP32 right-hand side, and its inverse: read on the device, so that a captured step
    // serves every right-hand side
    double scale, inv_scale;
};

constexpr double kNearRounding = 1e-12;

// most blocks of a dot product, and partial sums of each in the scratch
constexpr int kKrylovBlocks = 608, kKrylovSums = 4;

// beta = (z.q) / (p.Ap) of the last iteration (the first: 0); q: its -A p
template <typename T>
void krylov_beta(const KrylovBox& b, const T* z, const T* q, double* part, KrylovState* s, cudaStream_t st);
// p = z + beta p over the whole padded array (z carries its periodic aliases)
template <typename T>
void krylov_direction(const KrylovBox& b, const T* z, T* p, const KrylovState* s, cudaStream_t st);
// alpha = (r.p) / (p.Ap), q = -A p. In a singular system r carries the constant that its rounding errors sum up to, which no
// iteration removes, and p an arbitrary one; their product would drive alpha up without limit once the rest of r is smaller:
// run on below its rounding a 32 x 24 x 16 FP64 solve went from 3e-18 back to 0.06, and FP32 inner solves of strong V-cycles (8
// sweeps) spoiled a refinement step by a factor of 10 to 10^5. So r.p leaves the constants out (box.null_inv): always in FP32,
// and in FP64 below kNearRounding of the right-hand side, where the constant is still far smaller than r.
template <typename T>
void krylov_alpha(const KrylovBox& b, const T* p, const T* q, const T* r, double* part, KrylovState* s, cudaStream_t st);
// The max of |r| / V over the points that are not held, for krylov_update: *norm = max(*norm, it). nodal[d]: the points
// on the sides of direction d have half the volume; dlo / dhi: held sides; mask: 0 on held points (padded), or null.
struct KrylovNorm {
    unsigned long long* norm;
    int nodal[3], dlo[3], dhi[3];
    const unsigned char* mask;
    double ivol;
};
// x += alpha p over the whole padded array, r += alpha q on the unique points
template <typename T>
void krylov_update(const KrylovBox& b, const T* p, const T* q, T* x, T* r, const KrylovState* s, cudaStream_t st,
                   const KrylovNorm* norm = nullptr);

}  // namespace gbp

// TMA-staged level sweeps of the nodal operator (nodal_sweep64.cu: FP64 and FP32 sweeps, tensor maps and
// launch helpers).
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include "gbp_internal.cuh"

namespace gbp {

// mode 0: Jacobi sweep out = x + omega (b - A x) / diag(A); mode 1: residual out = b - A x (with the
// strong-form max norm into *norm when norm != nullptr). err: device word, bit 0 = a bounded wait ran out.
template <typename T>
int nodal_sweep(const NodalGeom& g, int mode, const T* s, const T* x, const T* b, T* out, double omega,
                unsigned* err, unsigned long long* norm, cudaStream_t st);
// Precomputed per padded node for the shared-sum FP64 sweep (nodal_qsweep64.cu), kc the far-corner coupling of the
// element: w5 = 5 kc (the 8 cells around the node), rd = 1 / the operator's diagonal; wx / wy / wz = kc (the 4 cells
// around the edge to the +x / +y / +z neighbour). rd may be null where only residuals are wanted.
struct KrylovState;
struct QWeights {
    double *w5, *rd, *wx, *wy, *wz;
};
bool qsweep_supported(const NodalGeom& g);
void nodal_qweights64(const NodalGeom& g, const double* s64, const QWeights& w, cudaStream_t st);
// mode 0: Jacobi sweep, 1: residual (+ strong-form max norm into *norm when norm != nullptr), 2: out = -A x (b unused),
// 3: mode 1 with the residual written as out32 = ks->scale (b - A x) instead
void nodal_qsweep64(const NodalGeom& g, int mode, const double* s64, const QWeights& w, const double* x,
                    const double* b, double* out, double omega, unsigned long long* norm, cudaStream_t st,
                    float* out32 = nullptr, const KrylovState* ks = nullptr);
// Jacobi sweep from zero: out = omega b / diag
void nodal_qzero64(const NodalGeom& g, const QWeights& w, const double* b, double* out, double omega, cudaStream_t st);

// whether the TMA sweep handles this level for elements of esize bytes (else the plain kernels do)
bool sweep_supported(const NodalGeom& g, int esize);
void sweep_forget_maps(const void* pool_base, size_t pool_bytes);

// helpers shared by the two sweep files
int make_tensor_map(const void* base, int esize, long long sy, long long sz, long long count, int boxx, int rows,
                    CUtensorMap* out);
// cuTensorMapEncodeTiled from the driver (nullptr when unavailable)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();
int sweep_z_chunks(const NodalGeom& g, int xy_tiles, int resident);
int sm_count_cached();
int sweep32_run(const NodalGeom& g, int mode, const float* s, const float* x, const float* b, float* out, float omega,
                unsigned* err, unsigned long long* norm, cudaStream_t st);

// FP32 whole-row sweeps with fused grid transfers (nodal_vsweep32.cu), isotropic levels whose rows hold
// at most 512 nodes (Jacobi and residual also with an overset mask: masked nodes are held at 0).
bool vsweep32_supported(const NodalGeom& g);
// ... and whose coarse level is the standard coarsening by 2 (residual + restriction, prolongation + sweep),
// neither of them with an overset mask
bool vsweep32_transfer_supported(const NodalGeom& g, const NodalGeom& gc);
// mode 0: Jacobi sweep, 1: residual (mix != 1: mix b - (mix - 1) A x = b + (mix - 1) (b - A x)); hold: masked nodes keep x
// in a Jacobi sweep instead of 0
int vsweep32(const NodalGeom& g, int mode, const float* s, const float* x, const float* b, float* out, float omega,
             unsigned* err, cudaStream_t st, bool hold = false, float mix = 1.f);
// bc (the coarse right-hand side) = full-weighting restriction of b - A x
int vsweep32_resid_restrict(const NodalGeom& g, const NodalGeom& gc, const float* s, const float* x, const float* b,
                            float* bc, unsigned* err, cudaStream_t st);
// out = one Jacobi sweep from x + P ec (ec: the coarse correction)
int vsweep32_prolong_jacobi(const NodalGeom& g, const NodalGeom& gc, const float* s, const float* x, const float* ec,
                            const float* b, float* out, float omega, unsigned* err, cudaStream_t st);
void vsweep32_forget_maps(const void* pool_base, size_t pool_bytes);

}  // namespace gbp

// Vector kernels of the conjugate-gradient acceleration (krylov.h). HBM bounds them on large levels: the dot product
// of three vectors, the direction and the update move 3, 3 and 6 vectors once each with 16-byte accesses; on small
// levels each is one launch.
#include "krylov.h"

#include <algorithm>

#include "gbp_internal.cuh"

namespace gbp {

namespace {

constexpr int kT = 256;

template <typename T>
struct Vec;
template <>
struct Vec<float> {
    static constexpr int N = 4;
    using type = float4;
};
template <>
struct Vec<double> {
    static constexpr int N = 2;
    using type = double2;
};

template <typename T>
__device__ __forceinline__ void ldv(const T* p, T (&v)[Vec<T>::N])
{
    const typename Vec<T>::type w = *reinterpret_cast<const typename Vec<T>::type*>(p);
    if constexpr (sizeof(T) == 4) {
        v[0] = w.x;
        v[1] = w.y;
        v[2] = w.z;
        v[3] = w.w;
    } else {
        v[0] = w.x;
        v[1] = w.y;
    }
}
template <typename T>
__device__ __forceinline__ void stv(T* p, const T (&v)[Vec<T>::N])
{
    if constexpr (sizeof(T) == 4)
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else
        *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}

// element e of the t-th vector of the unique points lies in the box; p: its offset (rows start 16-byte aligned)
template <typename T>
__device__ __forceinline__ long long vec_at(const KrylovBox& b, unsigned t, unsigned vr, int& i)
{
    const unsigned row = t / vr, k = row / (unsigned)b.n[1];
    i = (int)(t - row * vr) * Vec<T>::N;
    return pidx(b.sy, b.sz, i, (int)(row - k * (unsigned)b.n[1]), (int)k);
}

// The last block to get here sums the nb partial pairs in order and returns true in every thread, with the sums.
__device__ __forceinline__ bool fold_last(double v0, double v1, double* part, unsigned* done, double& s0, double& s1)
{
    __shared__ bool last;
    v0 = block_sum_all(v0);
    v1 = block_sum_all(v1);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = v0;
        part[2 * blockIdx.x + 1] = v1;
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    v0 = v1 = 0.0;
    for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) {
        v0 += __ldcg(part + 2 * q);
        v1 += __ldcg(part + 2 * q + 1);
    }
    s0 = block_sum_all(v0);
    s1 = block_sum_all(v1);
    if (threadIdx.x == 0) *done = 0;
    return true;
}

// a.b and a.c (c may be null) over the unique points. FP32 vectors are summed in FP32 per thread (a few hundred
// terms) and in FP64 from there: the FP64 pipe is 64 times slower than the FP32 one.
template <typename T, int WHAT>
__global__ void __launch_bounds__(kT) k_dots(KrylovBox b, const T* __restrict__ a, const T* __restrict__ v,
                                             const T* __restrict__ w, double* __restrict__ part, KrylovState* s)
{
    constexpr int N = Vec<T>::N;
    const unsigned vr = (unsigned)(b.n[0] + N - 1) / N;
    const unsigned total = vr * (unsigned)b.n[1] * (unsigned)b.n[2];
    const bool two = WHAT == 0 && s->it > 0;
    T acc0[N] = {}, acc1[N] = {};
    for (unsigned t = blockIdx.x * kT + threadIdx.x; t < total; t += gridDim.x * kT) {
        int i;
        const long long p = vec_at<T>(b, t, vr, i);
        T x[N], y[N], z[N];
        ldv<T>(a + p, x);
        ldv<T>(v + p, y);
        if (two) ldv<T>(w + p, z);
#pragma unroll
        for (int e = 0; e < N; ++e) {
            if (i + e >= b.n[0]) continue;
            acc0[e] += x[e] * y[e];
            if (two) acc1[e] += y[e] * z[e];
        }
    }
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int e = 0; e < N; ++e) {
        s0 += (double)acc0[e];
        s1 += (double)acc1[e];
    }
    if (!fold_last(s0, s1, part, s->done + WHAT, s0, s1) || threadIdx.x) return;
    if (WHAT == 0) {
        s->rz = s0;
        double beta = 0.0;
        if (two && !s->restart && s->rz_old > 0.0) {
            beta = s->alpha * s1 / s->rz_old;
            if (!(beta > 0.0 && beta < 1e30)) beta = 0.0;
        }
        s->beta = beta;
        s->rz_old = s0;
    } else {
        // a breakdown (rounding has the last word) takes the plain V-cycle step, or starts the directions again
        const double pap = -s0;
        const bool ok = pap > 0.0 && s->rz > 0.0;
        s->pq = pap;
        s->alpha = ok ? s->rz / pap : (s->beta == 0.0 ? 1.0 : 0.0);
        s->restart = !ok;
        s->it += 1;
    }
}

template <typename T>
__global__ void __launch_bounds__(kT) k_direction(long long nvec, const T* __restrict__ z, T* __restrict__ p,
                                                  const KrylovState* s)
{
    constexpr int N = Vec<T>::N;
    const long long t = blockIdx.x * (long long)kT + threadIdx.x;
    if (t >= nvec) return;
    const T beta = (T)s->beta;
    T x[N], y[N];
    ldv<T>(z + t * N, x);
    if (beta != T(0)) {
        ldv<T>(p + t * N, y);
#pragma unroll
        for (int e = 0; e < N; ++e) x[e] += beta * y[e];
    }
    stv<T>(p + t * N, x);
}

// one thread per vector of the padded array: x everywhere, r where the position is a unique point
template <typename T>
__global__ void __launch_bounds__(kT) k_update(KrylovBox b, long long nvec, const T* __restrict__ p,
                                               const T* __restrict__ q, T* __restrict__ x, T* __restrict__ r,
                                               const KrylovState* s)
{
    constexpr int N = Vec<T>::N;
    const long long t = blockIdx.x * (long long)kT + threadIdx.x;
    if (t >= nvec) return;
    const T alpha = (T)s->alpha;
    const unsigned rowv = (unsigned)(b.sy / N), rows = (unsigned)(b.sz / b.sy);
    const unsigned row = (unsigned)(t / rowv), k = row / rows;
    const int i = (int)(t - (long long)row * rowv) * N - kOX, j = (int)(row - k * rows) - 1;
    T u[N], v[N];
    ldv<T>(p + t * N, u);
    ldv<T>(x + t * N, v);
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] += alpha * u[e];
    stv<T>(x + t * N, v);
    if (j < 0 || j >= b.n[1] || k < 1 || (int)k - 1 >= b.n[2] || i + N <= 0 || i >= b.n[0]) return;
    ldv<T>(q + t * N, u);
    ldv<T>(r + t * N, v);
#pragma unroll
    for (int e = 0; e < N; ++e)
        if (i + e >= 0 && i + e < b.n[0]) v[e] += alpha * u[e];
    stv<T>(r + t * N, v);
}

unsigned dot_blocks(const KrylovBox& b, int vec)
{
    const long long nv = (long long)((b.n[0] + vec - 1) / vec) * b.n[1] * b.n[2];
    return (unsigned)std::max<long long>(1, std::min<long long>((nv + kT - 1) / kT, kKrylovBlocks));
}

}  // namespace

template <typename T>
void krylov_rz(const KrylovBox& b, const T* r, const T* z, const T* q, double* part, KrylovState* s, cudaStream_t st)
{
    k_dots<T, 0><<<dot_blocks(b, Vec<T>::N), kT, 0, st>>>(b, r, z, q, part, s);
}
template <typename T>
void krylov_direction(const KrylovBox& b, const T* z, T* p, const KrylovState* s, cudaStream_t st)
{
    const long long nv = b.count / Vec<T>::N;
    k_direction<T><<<(unsigned)((nv + kT - 1) / kT), kT, 0, st>>>(nv, z, p, s);
}
template <typename T>
void krylov_pq(const KrylovBox& b, const T* p, const T* q, double* part, KrylovState* s, cudaStream_t st)
{
    k_dots<T, 1><<<dot_blocks(b, Vec<T>::N), kT, 0, st>>>(b, p, q, nullptr, part, s);
}
template <typename T>
void krylov_update(const KrylovBox& b, const T* p, const T* q, T* x, T* r, const KrylovState* s, cudaStream_t st)
{
    const long long nv = b.count / Vec<T>::N;
    k_update<T><<<(unsigned)((nv + kT - 1) / kT), kT, 0, st>>>(b, nv, p, q, x, r, s);
}

#define GBP_KRYLOV(T)                                                                                               \
    template void krylov_rz<T>(const KrylovBox&, const T*, const T*, const T*, double*, KrylovState*, cudaStream_t); \
    template void krylov_direction<T>(const KrylovBox&, const T*, T*, const KrylovState*, cudaStream_t);             \
    template void krylov_pq<T>(const KrylovBox&, const T*, const T*, double*, KrylovState*, cudaStream_t);           \
    template void krylov_update<T>(const KrylovBox&, const T*, const T*, T*, T*, const KrylovState*, cudaStream_t);
GBP_KRYLOV(double)
GBP_KRYLOV(float)

}  // namespace gbp

// Vector kernels of the conjugate-gradient acceleration (krylov.h). HBM bounds them on large levels: the two dot
// products, the direction and the update move 2, 3, 3 and 6 vectors once each with 16-byte accesses; on small levels each is
// one launch.
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

// A sum carried by a thread: FP64 as it is, FP32 as an unevaluated pair hi + lo (Knuth's two-sum, about 48 bits: the
// FP64 pipe takes 16 cycles per warp for an addition or a conversion, the FP32 pipe takes the six additions of a
// two-sum in less).
template <typename T>
struct Sum;
template <>
struct Sum<double> {
    double v = 0.0;
};
template <>
struct Sum<float> {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float h, float l)
    {
        const float s = __fadd_rn(hi, h), t = __fsub_rn(s, hi);
        const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(h, t));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(l, e));
    }
    __device__ __forceinline__ void warp()
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            add(__shfl_xor_sync(0xffffffffu, hi, o), __shfl_xor_sync(0xffffffffu, lo, o));
    }
};

// Block sums of NV values per thread in a fixed order; the result lies in out[0 .. NV) after the next __syncthreads.
// FP64: one warp per value adds the threads' values (every warp reducing its own lanes would cost the pipe 8 times that).
template <int NV>
__device__ __forceinline__ void block_sums(const Sum<double> (&v)[NV], double* tab, double* out)
{
#pragma unroll
    for (int q = 0; q < NV; ++q) tab[q * kT + threadIdx.x] = v[q].v;
    __syncthreads();
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (wid < NV) {
        const double* t = tab + wid * kT + lane;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kT / 32; w += 4) s += (t[32 * w] + t[32 * w + 32]) + (t[32 * w + 64] + t[32 * w + 96]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[wid] = s;
    }
}
template <int NV>
__device__ __forceinline__ void block_sums(Sum<float> (&v)[NV], double* tab, double* out)
{
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        v[q].warp();
        if (lane == 0) tab[q * kT + wid] = (double)v[q].hi + (double)v[q].lo;
    }
    __syncthreads();
    if (wid < NV) {
        double s = lane < kT / 32 ? tab[wid * kT + lane] : 0.0;
#pragma unroll
        for (int o = kT / 64; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[wid] = s;
    }
}

// The last block to get here sums the blocks' partial sums in order and returns true in every thread, with the sums in out.
template <typename T, int NV>
__device__ __forceinline__ bool fold_last(Sum<T> (&v)[NV], double* part, unsigned* done, double* out)
{
    __shared__ double tab[NV * kT];
    __shared__ bool last;
    block_sums(v, tab, out);
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) part[kKrylovSums * blockIdx.x + q] = out[q];
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    Sum<double> f[NV];
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kT)
#pragma unroll
        for (int q = 0; q < NV; ++q) f[q].v += __ldcg(part + kKrylovSums * b + q);
    block_sums(f, tab, out);
    __syncthreads();
    if (threadIdx.x == 0) *done = 0;
    return true;
}

// a.b (WHAT 0: z.q and beta) or a.b and a.c (WHAT 1: p.q, p.r and alpha) over the unique points. FP32 vectors are summed in
// FP32 per thread (a few hundred terms), as pairs over the block and in FP64 from there. Latency and the FP64 pipe bound it
// below some 10^6 points: with FP64 sums in every warp 17.2 us (two products, 10^6 points FP32), 13.9 us (64^3 FP64), 9.8 us
// (16^3 FP64); now 10.5, 11.3 and 7.2 us.
// NULLSPACE (WHAT 1, singular systems): p.r without the constants of either, p.r - (sum p)(sum r) / n. In FP64 the two sums
// more bind it (117 against 62 us at 256^3, and 5 us more per launch on small levels).
template <typename T, int WHAT, bool NULLSPACE>
__global__ void __launch_bounds__(kT) k_dots(KrylovBox b, const T* __restrict__ a, const T* __restrict__ c,
                                             const T* __restrict__ d, double* __restrict__ part, KrylovState* s)
{
    constexpr int N = Vec<T>::N, NV = WHAT == 0 ? 1 : (NULLSPACE ? 4 : 2);
    const unsigned vr = (unsigned)(b.n[0] + N - 1) / N;
    const unsigned total = vr * (unsigned)b.n[1] * (unsigned)b.n[2];
    T acc[NV][N] = {};
    if (WHAT == 1 || s->it > 0)
        for (unsigned t = blockIdx.x * kT + threadIdx.x; t < total; t += gridDim.x * kT) {
            int i;
            const long long p = vec_at<T>(b, t, vr, i);
            T x[N], y[N], z[N];
            ldv<T>(a + p, x);
            ldv<T>(c + p, y);
            if (WHAT == 1) ldv<T>(d + p, z);
#pragma unroll
            for (int e = 0; e < N; ++e) {
                if (i + e >= b.n[0]) continue;
                acc[0][e] += x[e] * y[e];
                if constexpr (WHAT == 1) acc[1][e] += x[e] * z[e];
                if constexpr (NULLSPACE) {
                    acc[2][e] += x[e];
                    acc[3][e] += z[e];
                }
            }
        }
    __shared__ double out[NV];
    Sum<T> v[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
        for (int e = 0; e < N; ++e) {
            if constexpr (sizeof(T) == 4)
                v[q].add(acc[q][e], 0.f);
            else
                v[q].v += acc[q][e];
        }
    if (!fold_last<T, NV>(v, part, s->done + WHAT, out) || threadIdx.x) return;
    if constexpr (WHAT == 0) {
        double beta = s->it > 0 && !s->restart && !s->plain ? out[0] / s->pap : 0.0;
        if (!(beta > 0.0 && beta < 1e30)) beta = 0.0;
        s->beta = beta;
    } else {
        // p.r and p.Ap have one sign, that of the operator (coefficients may be negative throughout). A breakdown (rounding
        // has the last word) takes the plain V-cycle step, or starts the directions again.
        double rp = out[1];
        if constexpr (NULLSPACE) rp -= out[2] * out[3] * b.null_inv;
        const double pap = -out[0], alpha = rp / pap;
        const bool ok = alpha > 0.0 && alpha < 1e30;
        s->pap = pap;
        s->alpha = ok && !s->plain ? alpha : (s->beta == 0.0 ? 1.0 : 0.0);
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

// One thread per vector of the padded array: x everywhere, r where the position is a unique point. NORM: also the max
// of |r| / V, as integer keys of |r| (the points on non-periodic sides of a nodal box have half the volume per side: a
// power of two) and one multiplication per block; a pass over r of its own
// took 252 us at 256^3 (16 us at 64^3), the keys add 25 us (2 us).
template <typename T, bool NORM>
__global__ void __launch_bounds__(kT) k_update(KrylovBox b, long long nvec, const T* __restrict__ p,
                                               const T* __restrict__ q, T* __restrict__ x, T* __restrict__ r,
                                               const KrylovState* s, KrylovNorm nm)
{
    constexpr int N = Vec<T>::N;
    const long long t = blockIdx.x * (long long)kT + threadIdx.x;
    unsigned long long key = 0;
    if (t < nvec) {
        const T alpha = (T)s->alpha;
        const unsigned rowv = (unsigned)(b.sy / N), rows = (unsigned)(b.sz / b.sy);
        const unsigned row = (unsigned)(t / rowv), kp = row / rows;
        const int i = (int)(t - (long long)row * rowv) * N - kOX, j = (int)(row - kp * rows) - 1, k = (int)kp - 1;
        T u[N], v[N];
        ldv<T>(p + t * N, u);
        ldv<T>(x + t * N, v);
#pragma unroll
        for (int e = 0; e < N; ++e) v[e] += alpha * u[e];
        stv<T>(x + t * N, v);
        if (j >= 0 && j < b.n[1] && k >= 0 && k < b.n[2] && i + N > 0 && i < b.n[0]) {
            ldv<T>(q + t * N, u);
            ldv<T>(r + t * N, v);
#pragma unroll
            for (int e = 0; e < N; ++e) {
                if (i + e < 0 || i + e >= b.n[0]) continue;
                v[e] += alpha * u[e];
                if constexpr (NORM) {
                    const int at[3] = {i + e, j, k};
                    int halves = 0;
                    bool held = nm.mask && !nm.mask[t * N + e];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const bool lo = at[d] == 0, hi = at[d] == b.n[d] - 1;
                        halves += (nm.nodal[d] && (lo || hi)) ? 1 : 0;
                        held = held || (lo && nm.dlo[d]) || (hi && nm.dhi[d]);
                    }
                    const unsigned long long kv =
                        held ? 0 : abs_key(halves == 0 ? (double)v[e] : (double)v[e] * (double)(1 << halves));
                    key = kv > key ? kv : key;
                }
            }
            stv<T>(r + t * N, v);
        }
    }
    if constexpr (NORM) {
        key = block_max_key(key);
        if (threadIdx.x == 0) atomic_max_nonneg(nm.norm, key_value(key) * nm.ivol);
    }
}

unsigned dot_blocks(const KrylovBox& b, int vec)
{
    const long long nv = (long long)((b.n[0] + vec - 1) / vec) * b.n[1] * b.n[2];
    // a vector per thread until every SM has a block, then four (fewer blocks to sum in FP64), up to the scratch
    const long long blocks = std::max(std::min<long long>((nv + kT - 1) / kT, 152), (nv + 4 * kT - 1) / (4 * kT));
    return (unsigned)std::max<long long>(1, std::min<long long>(blocks, kKrylovBlocks));
}

}  // namespace

template <typename T>
void krylov_beta(const KrylovBox& b, const T* z, const T* q, double* part, KrylovState* s, cudaStream_t st)
{
    k_dots<T, 0, false><<<dot_blocks(b, Vec<T>::N), kT, 0, st>>>(b, z, q, nullptr, part, s);
}
template <typename T>
void krylov_direction(const KrylovBox& b, const T* z, T* p, const KrylovState* s, cudaStream_t st)
{
    const long long nv = b.count / Vec<T>::N;
    k_direction<T><<<(unsigned)((nv + kT - 1) / kT), kT, 0, st>>>(nv, z, p, s);
}
template <typename T>
void krylov_alpha(const KrylovBox& b, const T* p, const T* q, const T* r, double* part, KrylovState* s, cudaStream_t st)
{
    (b.null_inv != 0.0 ? k_dots<T, 1, true> : k_dots<T, 1, false>)<<<dot_blocks(b, Vec<T>::N), kT, 0, st>>>(b, p, q, r, part,
                                                                                                           s);
}
template <typename T>
void krylov_update(const KrylovBox& b, const T* p, const T* q, T* x, T* r, const KrylovState* s, cudaStream_t st,
                   const KrylovNorm* norm)
{
    const long long nv = b.count / Vec<T>::N;
    const unsigned nb = (unsigned)((nv + kT - 1) / kT);
    if (norm)
        k_update<T, true><<<nb, kT, 0, st>>>(b, nv, p, q, x, r, s, *norm);
    else
        k_update<T, false><<<nb, kT, 0, st>>>(b, nv, p, q, x, r, s, KrylovNorm{});
}

#define GBP_KRYLOV(T)                                                                                               \
    template void krylov_beta<T>(const KrylovBox&, const T*, const T*, double*, KrylovState*, cudaStream_t);         \
    template void krylov_direction<T>(const KrylovBox&, const T*, T*, const KrylovState*, cudaStream_t);             \
    template void krylov_alpha<T>(const KrylovBox&, const T*, const T*, const T*, double*, KrylovState*,             \
                                  cudaStream_t);                                                                     \
    template void krylov_update<T>(const KrylovBox&, const T*, const T*, T*, T*, const KrylovState*, cudaStream_t,   \
                                   const KrylovNorm*);
GBP_KRYLOV(double)
GBP_KRYLOV(float)

}  // namespace gbp

// Coarsest-level solvers (bottom.h).
//
// k_bottom_cg: hierarchies whose cell counts carry an odd factor end on a coarsest level of a few hundred to a few
// thousand unknowns, where one CTA's FP64 pipe (2 lanes per clock) bounds a 27-point product: 480 unknowns took 507 us
// per solve in one CTA with the operator evaluated from sigma (about 120 FP64 instructions per node), two thirds of a
// 144 x 80 x 112 projection (7.8 ms; 4.5 ms with this kernel). Here a cluster of 16 CTAs shares the rows, the coefficients are assembled once per
// sigma (one multiply-add per entry), each CTA holds the whole search direction in shared memory and sends its part to the
// others, and the dot products meet in a table of per-CTA sums in every CTA's shared memory: three cluster barriers
// per iteration and no global traffic.
#include "bottom.h"

#include <algorithm>

namespace gbp {

namespace {

__host__ __device__ inline size_t up(size_t v) { return (v + 255) & ~size_t(255); }

// ------------------------------------------------------------------------------------------------ rows
// *empty += unknowns whose row is 0
__global__ void __launch_bounds__(128) k_rows_nodal(NodalGeom g, const double* __restrict__ s, BottomRows r,
                                                    unsigned* empty)
{
    const int u = blockIdx.x * 128 + threadIdx.x;
    if (u >= r.n) return;
    const int i = u % g.nu[0], j = (u / g.nu[0]) % g.nu[1], k = u / (g.nu[0] * g.nu[1]);
    const bool held = node_is_dirichlet(g, i, j, k);
    double a[27];
#pragma unroll
    for (int q = 0; q < 27; ++q) a[q] = 0.0;
    if (!held) {
        const long long p = pidx(g.sy, g.sz, i, j, k);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int cx = c & 1, cy = (c >> 1) & 1, cz = c >> 2;
            const double sg = s[p + (cx - 1) + (cy - 1) * g.sy + (cz - 1) * g.sz];
            // corner (ax, ay, az) of the cell lies at offset c - 1 + a; this node is its corner 1 - c
#pragma unroll
            for (int a8 = 0; a8 < 8; ++a8) {
                const int ax = a8 & 1, ay = (a8 >> 1) & 1, az = a8 >> 2;
                const int mask = (ax != 1 - cx) | ((ay != 1 - cy) << 1) | ((az != 1 - cz) << 2);
                a[(cx + ax) + 3 * ((cy + ay) + 3 * (cz + az))] += sg * g.K[mask];
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        int c[3] = {i + q % 3 - 1, j + (q / 3) % 3 - 1, k + q / 9 - 1};
        bool in = true;
        for (int d = 0; d < 3; ++d) {
            if (g.per[d])
                c[d] = (c[d] + g.n[d]) % g.n[d];
            else
                in = in && c[d] >= 0 && c[d] <= g.n[d];
        }
        in = in && !node_is_dirichlet(g, c[0], c[1], c[2]);
        r.coef[(size_t)q * r.n + u] = in ? a[q] : 0.0;
        r.idx[(size_t)q * r.n + u] = in ? c[0] + g.nu[0] * (c[1] + g.nu[1] * c[2]) : u;
    }
    r.diag[u] = held ? 0.0 : a[13];
    r.weight[u] = held ? 0.0 : node_volume(g, i, j, k);
    if (!held && a[13] == 0.0) atomicAdd(empty, 1u);
}

__global__ void __launch_bounds__(128) k_rows_mac(CellGeom g, const double* __restrict__ bx, const double* __restrict__ by,
                                                  const double* __restrict__ bz, BottomRows r)
{
    const int u = blockIdx.x * 128 + threadIdx.x;
    if (u >= r.n) return;
    const int c[3] = {u % g.n[0], (u / g.n[0]) % g.n[1], u / (g.n[0] * g.n[1])};
    const long long p = pidx(g.sy, g.sz, c[0], c[1], c[2]);
    const long long sd[3] = {1, g.sy, g.sz};
    const double* b[3] = {bx, by, bz};
    double diag = g.a64 ? g.a64[p] : 0.0;
    for (int q = 0; q < 6; ++q) {
        const int d = q >> 1, side = q & 1;
        const double coef = g.w[d] * b[d][side ? p + sd[d] : p];
        diag += coef;
        int nb[3] = {c[0], c[1], c[2]};
        nb[d] += side ? 1 : -1;
        bool in = true;
        if (nb[d] < 0 || nb[d] >= g.n[d]) {
            in = g.per[d];  // else: ghost value 0 (Dirichlet) or no flux
            nb[d] = (nb[d] + g.n[d]) % g.n[d];
        }
        r.coef[(size_t)(q + 1) * r.n + u] = in ? -coef : 0.0;
        r.idx[(size_t)(q + 1) * r.n + u] = in ? nb[0] + g.n[0] * (nb[1] + g.n[1] * nb[2]) : u;
    }
    r.coef[u] = diag;
    r.idx[u] = u;
    r.diag[u] = diag;
    r.weight[u] = diag != 0.0 ? 1.0 : 0.0;
}

// ------------------------------------------------------------------------------------------------ dense inverse
// Symmetric and, for coefficients of one sign, definite, so no pivoting, and Gauss-Jordan as the sweep operator (Goodnight
// 1979, The American Statistician 33), which keeps the symmetry: one triangle in registers, the pivot's column passed
// through shared memory, one division per pivot in the warps that hold the column. (Coefficients of both signs or NaN go
// through as well: the inverse is a preconditioner, and the solve's residual decides.) A pivot that is rounding against its
// diagonal (up to 2e-13 with some 100 unknowns) closes a null space besides the constants, that of a region of fluid sealed off by covered cells: its unknown stays
// unswept, held at 0 (a generalised inverse, exact for a right-hand side that is consistent in the region). One SM's FP64 pipe bounds it (16 cycles per warp and instruction): 64
// unknowns took 243 us with the whole matrix and a division in every warp, now 75.
__global__ void __launch_bounds__(1024) k_bottom_inverse(BottomRows r, int singular, double* __restrict__ M,
                                                         unsigned char* __restrict__ act, unsigned* bad)
{
    constexpr int kMost = (kDenseBottom * (kDenseBottom + 1) / 2 + 1023) / 1024;  // entries of a thread
    __shared__ double col[2][kDenseBottom], scl[kDenseBottom], diag[kDenseBottom], shift;
    const int N = r.n, t = threadIdx.x;
    // entry (u, v) of the matrix
    auto entry = [&](int u, int v) {
        if (r.weight[u] == 0.0) return u == v ? 1.0 : 0.0;
        double sum = 0.0;
        for (int q = 0; q < r.w; ++q)
            if (r.idx[(size_t)q * N + u] == v) sum += r.coef[(size_t)q * N + u];
        return sum;
    };
    double tr = 0.0, na = 0.0;
    if (t < N) {
        const bool held = r.weight[t] == 0.0;
        scl[t] = held ? 0.0 : entry(t, t);
        col[0][t] = held ? 0.0 : 1.0;
        if (act) act[t] = !held;
    }
    __syncthreads();
    if (t < 32) {
        for (int u = t; u < N; u += 32) {
            tr += scl[u];
            na += col[0][u];
        }
        for (int o = 16; o > 0; o >>= 1) {
            tr += __shfl_xor_sync(0xffffffffu, tr, o);
            na += __shfl_xor_sync(0xffffffffu, na, o);
        }
        if (t == 0) shift = singular && na > 0.0 ? tr / (na * na) : 0.0;
    }
    __syncthreads();
    // entry e of the lower triangle: (u, v), v <= u, e = u (u + 1) / 2 + v
    int eu[kMost], ev[kMost];
    double a[kMost];
#pragma unroll
    for (int m = 0; m < kMost; ++m) {
        const int e = t + 1024 * m;
        int u = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
        while (u * (u + 1) / 2 > e) --u;
        while ((u + 1) * (u + 2) / 2 <= e) ++u;
        eu[m] = u < N ? u : -1;
        ev[m] = u < N ? e - u * (u + 1) / 2 : -1;
        a[m] = 0.0;
        if (u < N) {
            a[m] = entry(u, ev[m]);
            if (r.weight[u] != 0.0 && r.weight[ev[m]] != 0.0) a[m] += shift;
        }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kMost; ++m)  // the first pivot's column
        if (eu[m] >= 0) {
            if (ev[m] == 0) col[0][eu[m]] = a[m];
            if (ev[m] == eu[m]) diag[eu[m]] = fabs(a[m]);
        }
    __syncthreads();
    for (int c = 0; c < N; ++c) {
        const double* cc = col[c & 1];
        const double piv = cc[c];
        if (piv == 0.0) {  // uniform
            if (t == 0) *bad = 1u;
            return;
        }
        if (t < ((N + 31) & ~31)) {
            const double inv = fabs(piv) < 1e-12 * diag[c] ? 0.0 : 1.0 / piv;
            if (t < N) scl[t] = t == c ? -inv : cc[t] * inv;
        }
        __syncthreads();
        // a_uv -= a_uc a_cv / a_cc; the pivot's row and column a_uc / a_cc; the pivot -1 / a_cc: minus the inverse
        double* nx = col[(c + 1) & 1];
#pragma unroll
        for (int m = 0; m < kMost; ++m) {
            const int u = eu[m], v = ev[m];
            if (u < 0) continue;
            if (u == c || v == c)
                a[m] = scl[u == c ? v : u];
            else
                a[m] = fma(-cc[u], scl[v], a[m]);
            if (u == c + 1)
                nx[v] = a[m];
            else if (v == c + 1)
                nx[u] = a[m];
        }
        __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < kMost; ++m) {
        const int u = eu[m], v = ev[m];
        if (u < 0) continue;
        const double x = r.weight[u] != 0.0 && r.weight[v] != 0.0 ? -a[m] : 0.0;
        M[u * N + v] = x;
        M[v * N + u] = x;
    }
}

// ------------------------------------------------------------------------------------------------ conjugate gradients
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// store to the same shared-memory address of CTA `rank` of the cluster
__device__ __forceinline__ void st_cluster(double* p, unsigned rank, double v)
{
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

constexpr int kMostCtas = 16;

// Sums of two values over the vector threads (the first nvw warps) of the whole cluster, the same bits in every thread
// of every CTA (fixed order). An FP64 instruction takes 16 cycles of the SM per warp, so only warps that hold values
// add, and one warp adds the CTAs' sums. slots: one [2][kMostCtas][2] table per CTA, used alternately, so that a sum
// can be read while the next is written; every call is a cluster barrier.
struct ClusterSum {
    double* slots;
    double* warps;  // [32][2]
    double* out;    // [2]
    int nvw, flip;
    __device__ void operator()(double& a, double& b)
    {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (wid < nvw) {
            for (int o = 16; o > 0; o >>= 1) {
                a += __shfl_down_sync(0xffffffffu, a, o);
                b += __shfl_down_sync(0xffffffffu, b, o);
            }
            if (lane == 0) {
                warps[2 * wid] = a;
                warps[2 * wid + 1] = b;
            }
        }
        __syncthreads();
        const int nc = (int)cluster_nctas();
        double* table = slots + flip * 2 * kMostCtas;
        if (wid == 0) {
            double s0 = warps[0], s1 = warps[1];
            for (int q = 1; q < nvw; ++q) {
                s0 += warps[2 * q];
                s1 += warps[2 * q + 1];
            }
            if (lane < nc) {
                st_cluster(table + 2 * cluster_rank(), lane, s0);
                st_cluster(table + 2 * cluster_rank() + 1, lane, s1);
            }
        }
        cluster_barrier();
        if (wid == 0) {
            double s0 = lane < nc ? table[2 * lane] : 0.0, s1 = lane < nc ? table[2 * lane + 1] : 0.0;
            for (int o = 8; o > 0; o >>= 1) {
                s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            }
            if (lane == 0) {
                out[0] = s0;
                out[1] = s1;
            }
        }
        __syncthreads();
        a = out[0];
        b = out[1];
        flip ^= 1;
    }
};

__device__ __forceinline__ void unknown_at(const NodalGeom& g, int u, int& i, int& j, int& k)
{
    i = u % g.nu[0];
    j = (u / g.nu[0]) % g.nu[1];
    k = u / (g.nu[0] * g.nu[1]);
}
__device__ __forceinline__ void unknown_at(const CellGeom& g, int u, int& i, int& j, int& k)
{
    i = u % g.n[0];
    j = (u / g.n[0]) % g.n[1];
    k = u / (g.n[0] * g.n[1]);
}
template <typename T>
__device__ __forceinline__ void store_unknown(T* a, const NodalGeom& g, int i, int j, int k, T v)
{
    store_node(a, g, i, j, k, v);
}
template <typename T>
__device__ __forceinline__ void store_unknown(T* a, const CellGeom& g, int i, int j, int k, T v)
{
    store_cell(a, g, i, j, k, v);
}

// rows of one CTA, and the shared memory that the solver takes (the coefficients too when `held`)
__host__ __device__ inline int cg_rows(int n, int ctas) { return (n + ctas - 1) / ctas; }
__host__ __device__ inline size_t cg_bytes(int n, int w, int ctas, bool held)
{
    const size_t R = cg_rows(n, ctas);
    return sizeof(double) * (4 * kMostCtas + 66 + (size_t)n + 4 * R) + (held ? R * w * 12 + 16 : 0);
}

template <typename T, typename G>
__global__ void __launch_bounds__(kBottomThreads) k_bottom_cg(G g, BottomCG c, const T* __restrict__ bin,
                                                              T* __restrict__ xout, int held)
{
    extern __shared__ double sm[];
    const int N = c.r.n, W = c.r.w;
    const int C = (int)cluster_nctas(), me = (int)cluster_rank();
    const int R = cg_rows(N, C), u0 = min(N, me * R), nr = min(N, u0 + R) - u0;
    // vector threads: one row each where the block is large enough
    const int nvw = max(1, min((nr + 31) / 32, (int)blockDim.x / 32)), vstep = 32 * nvw;
    const bool vec = (int)threadIdx.x < vstep;
    ClusterSum sum{sm, sm + 4 * kMostCtas, sm + 4 * kMostCtas + 64, nvw, 0};
    double* p = sm + 4 * kMostCtas + 66;  // the whole search direction
    double *x = p + N, *r = x + R, *dinv = r + R, *qv = dinv + R;
    double* cf = qv + R;
    int* ix = reinterpret_cast<int*>(cf + (held ? (size_t)R * W : 0));
    // L lanes share a row of the product
    int L = 1;
    while (L < 8 && 2 * L * nr <= (int)blockDim.x) L *= 2;
    const int lane = threadIdx.x % L, row0 = threadIdx.x / L, rstep = blockDim.x / L;
    if (held)
        for (int q = threadIdx.x; q < nr * W; q += blockDim.x) {
            const int e = q / nr, u = q - e * nr;
            cf[e * R + u] = c.r.coef[(size_t)e * N + u0 + u];
            ix[e * R + u] = c.r.idx[(size_t)e * N + u0 + u];
        }
    double s = 0.0, ws = 0.0;
    if (vec)
        for (int u = threadIdx.x; u < nr; u += vstep) {
            int i, j, k;
            unknown_at(g, u0 + u, i, j, k);
            const double d = c.r.diag[u0 + u];
            const double b = d != 0.0 ? (double)bin[pidx(g.sy, g.sz, i, j, k)] : 0.0;
            x[u] = 0.0;
            r[u] = b;
            dinv[u] = d != 0.0 ? 1.0 / d : 0.0;
            s += b;
            ws += c.r.weight[u0 + u];
        }
    cluster_barrier();  // every CTA of the cluster runs before any of them is written to
    sum(s, ws);
    // singular: the right-hand side without its component along the null space
    double rz = 0.0, rr = 0.0;
    if (vec) {
        const double mean = c.singular && ws > 0.0 ? s / ws : 0.0;
        for (int u = threadIdx.x; u < nr; u += vstep) {
            r[u] -= mean * c.r.weight[u0 + u];
            const double z = r[u] * dinv[u];
            rz += r[u] * z;
            rr += r[u] * r[u];
            for (int q = 0; q < C; ++q) st_cluster(p + u0 + u, q, z);
        }
    }
    sum(rz, rr);
    const double target = fmax(c.rtol * c.rtol * rr, c.atol > 0.0 ? c.atol * c.atol : 0.0);
    int it = 0;
    if (rr > 0.0) {
        for (it = 1; it <= c.maxiter; ++it) {
            for (int base = 0; base < nr; base += rstep) {
                const int u = base + row0;
                double v = 0.0;
                if (u < nr) {
                    if (held)
                        for (int e = lane; e < W; e += L) v = fma(cf[e * R + u], p[ix[e * R + u]], v);
                    else
                        for (int e = lane; e < W; e += L)
                            v = fma(c.r.coef[(size_t)e * N + u0 + u], p[c.r.idx[(size_t)e * N + u0 + u]], v);
                }
                for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0 && u < nr) qv[u] = v;
            }
            __syncthreads();
            double pq = 0.0, unused = 0.0;
            if (vec)
                for (int u = threadIdx.x; u < nr; u += vstep) pq += p[u0 + u] * qv[u];
            sum(pq, unused);
            // (with the sign of r.z: the operator is negative for negative coefficients)
            if (!(__hiloint2double(__double2hiint(pq) ^ (__double2hiint(rz) & (int)0x80000000u), __double2loint(pq)) > 0.0)) break;
            double rz2 = 0.0;
            rr = 0.0;
            if (vec) {
                const double alpha = rz / pq;
                for (int u = threadIdx.x; u < nr; u += vstep) {
                    x[u] += alpha * p[u0 + u];
                    r[u] -= alpha * qv[u];
                    const double z = r[u] * dinv[u];
                    qv[u] = z;
                    rz2 += r[u] * z;
                    rr += r[u] * r[u];
                }
            }
            sum(rz2, rr);
            if (rr <= target) break;
            if (vec) {
                const double beta = rz2 / rz;
                for (int u = threadIdx.x; u < nr; u += vstep) {
                    const double v = qv[u] + beta * p[u0 + u];
                    for (int q = 0; q < C; ++q) st_cluster(p + u0 + u, q, v);
                }
            }
            rz = rz2;
            cluster_barrier();
        }
    }
    __syncthreads();
    for (int u = threadIdx.x; u < nr; u += blockDim.x) {
        int i, j, k;
        unknown_at(g, u0 + u, i, j, k);
        store_unknown(xout, g, i, j, k, (T)x[u]);
    }
    if (me == 0 && threadIdx.x == 0 && c.info) {
        const int used = it > c.maxiter ? c.maxiter : it;
        if (used > c.info[0]) c.info[0] = used;
    }
    cluster_barrier();  // no CTA leaves while another may still write to its shared memory
}

// the largest cluster the device co-schedules with `bytes` of shared memory per CTA
template <typename T, typename G>
int cg_cluster(size_t bytes)
{
    auto kern = k_bottom_cg<T, G>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int best = 8;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(kBottomThreads);
        cfg.dynamicSmemBytes = bytes;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 16;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) best = 16;
    }
    cudaGetLastError();
    return best;
}

template <typename T, typename G>
int launch_cg(const G& g, const BottomCG& c, const T* b, T* x, cudaStream_t st)
{
    constexpr size_t kMost = 227 * 1024;
    static const int ctas = cg_cluster<T, G>(kMost);
    if (ctas == 0 || c.r.n > kClusterBottom) {
        set_error("bottom solve: the coarsest level does not fit the cluster solver");
        return GBP_BAD_ARG;
    }
    const int held = cg_bytes(c.r.n, c.r.w, ctas, true) <= kMost ? 1 : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(std::min(kBottomThreads, std::max(64, (cg_rows(c.r.n, ctas) * 8 + 31) / 32 * 32)));
    cfg.dynamicSmemBytes = cg_bytes(c.r.n, c.r.w, ctas, held);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, k_bottom_cg<T, G>, g, c, b, x, held);
    return e == cudaSuccess ? GBP_OK : cuda_fail(e, "k_bottom_cg launch");
}

}  // namespace

void BottomRows::carve(char* base)
{
    size_t at = 0;
    auto take = [&](size_t b) {
        char* p = base + at;
        at = up(at + b);
        return p;
    };
    coef = reinterpret_cast<double*>(take(sizeof(double) * n * w));
    idx = reinterpret_cast<int*>(take(sizeof(int) * n * w));
    diag = reinterpret_cast<double*>(take(sizeof(double) * n));
    weight = reinterpret_cast<double*>(take(sizeof(double) * n));
}

void bottom_rows_nodal(const NodalGeom& g, const double* s64, const BottomRows& r, unsigned* empty, cudaStream_t st)
{
    k_rows_nodal<<<(r.n + 127) / 128, 128, 0, st>>>(g, s64, r, empty);
}
void bottom_rows_mac(const CellGeom& g, const double* bx, const double* by, const double* bz, const BottomRows& r,
                     cudaStream_t st)
{
    k_rows_mac<<<(r.n + 127) / 128, 128, 0, st>>>(g, bx, by, bz, r);
}
void bottom_inverse(const BottomRows& r, int singular, double* M, unsigned char* act, unsigned* bad, cudaStream_t st)
{
    k_bottom_inverse<<<1, 1024, 0, st>>>(r, singular, M, act, bad);
}

template <typename T>
int bottom_cg_nodal(const NodalGeom& g, const BottomCG& c, const T* b, T* x, cudaStream_t st)
{
    return launch_cg<T, NodalGeom>(g, c, b, x, st);
}
template <typename T>
int bottom_cg_mac(const CellGeom& g, const BottomCG& c, const T* b, T* x, cudaStream_t st)
{
    return launch_cg<T, CellGeom>(g, c, b, x, st);
}
template int bottom_cg_nodal<double>(const NodalGeom&, const BottomCG&, const double*, double*, cudaStream_t);
template int bottom_cg_nodal<float>(const NodalGeom&, const BottomCG&, const float*, float*, cudaStream_t);
template int bottom_cg_mac<double>(const CellGeom&, const BottomCG&, const double*, double*, cudaStream_t);
template int bottom_cg_mac<float>(const CellGeom&, const BottomCG&, const float*, float*, cudaStream_t);

}  // namespace gbp

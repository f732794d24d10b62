// FP64 sweep of the isotropic nodal operator in shared-sum form (levels of at least kQMinNodes nodes).
//
// With equal spacing the Q1 element couples a node only to its face and body diagonals
// (coefficient kc, K[1] = K[2] = K[4] = 0), and
//   (A x)_n = kc * ( sum_c sigma_c Q_c  -  5 x_n sum_c sigma_c  -  sum_e W_e x_e )
// over the 8 cells c around n (Q_c = the sum of the cell's 8 corner values) and the 6 edge
// neighbours e (W_e = the sigma of the 4 cells that contain both nodes). Q_c and sigma_c Q_c are
// computed once per cell and shared by its 8 nodes; kc W_e, 5 kc sum_c sigma_c and the reciprocal of the diagonal
// do not change between sweeps and are precomputed per node (k_qweights64), so that a residual is 17 FP64
// instructions per node and a Jacobi sweep 19 (29 when the diagonal's reciprocal, its range check and the factors
// kc and 5 were applied in every sweep, about 45 in the per-cell form): on GB300 the FP64 pipe (2 lanes per clock
// and SM), not HBM, bounds this kernel.
//
// Layout: a CTA of 10 warps marches a z range over a tile of 32 x 8 nodes. Warps 0-8 own the cell rows y0-1 ..
// y0+7 of columns x0 .. x0+31, warp 9 the 9 cells of column x0-1: an FP64 instruction occupies the pipe for a
// whole warp whatever its active lanes, so the node work runs on 8 full warps (a 33 x 9 thread tile spread it over
// 10 partly filled ones). Every thread forms sigma_c Q_c of its cell for the current cell layer into a
// double-buffered shared tile (one barrier per plane); warps 1-8 then add the four cells
// of the layer around their node and finish the node from the previous layer's sum, which they carry.
#include <cuda_runtime.h>

#include <algorithm>

#include "gbp_internal.cuh"
#include "krylov.h"
#include "nodal_sweep.h"

namespace gbp {

namespace {

constexpr int QX = 32, QY = 8;
constexpr int kQThreads = 32 * (QY + 2);    // k_qsweep64: QY + 1 cell rows and the halo column

__device__ __forceinline__ bool q_alias(const NodalGeom& g, int i, int j, int k)
{
    return (g.per[0] && (i <= 1 || i == g.n[0] - 1)) || (g.per[1] && (j <= 1 || j == g.n[1] - 1)) ||
           (g.per[2] && (k <= 1 || k == g.n[2] - 1));
}

// w5 = 5 kc (sum of the 8 cells around each node), rd = 1 / diagonal (single precision, where the diagonal is in
// its range: a smoother needs no more; nullptr: not wanted); wx / wy / wz = kc (sigma sum of the 4 cells around the edge
// from node (i,j,k) to (i+1,j,k) / (i,j+1,k) / (i,j,k+1)). The sweep also reads the edge to a node's low neighbour:
// across a periodic seam the last node's edge is stored at index -1 too, elsewhere index -1 keeps its 0.
// A CTA marches a z range over 32 x 8 node columns; separable sums of kc sigma per cell layer: Px = x pair, Q = Px +
// Px(j-1) (4 cells around a z edge), Y = y pair; then the 8 cells = Q(k-1) + Q(k), wz = Q(k), wx = Y(k-1) + Y(k), wy =
// Px(k-1) + Px(k): 9 FP64 instructions per node.
__global__ void __launch_bounds__(32 * QY) k_qweights64(NodalGeom g, const double* __restrict__ s, QWeights w,
                                                        int kchunk)
{
    __shared__ double T[2][QY + 1][QX + 1];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i = blockIdx.x * QX + tx, j = blockIdx.y * QY + ty;
    const int kbeg = blockIdx.z * kchunk, kend = min(kbeg + kchunk, g.nu[2]);
    const bool node = i < g.nu[0] && j < g.nu[1];
    const double kc = g.K[3];
    const long long sx = g.per[0] && i == g.n[0] - 1 ? -g.n[0] : 0, sy = g.per[1] && j == g.n[1] - 1 ? -g.n[1] * g.sy : 0;
    double Qp = 0.0, Yp = 0.0, Pp = 0.0;
    for (int L = kbeg - 1; L < kend; ++L) {
        const int buf = (L - kbeg + 1) & 1;
        // cells (x0-1 .. x0+31, y0-1 .. y0+7) of layer L
        for (int q = threadIdx.x; q < (QX + 1) * (QY + 1); q += 32 * QY) {
            const int cx = q % (QX + 1), cy = q / (QX + 1);
            const int a = blockIdx.x * QX - 1 + cx, b = blockIdx.y * QY - 1 + cy;
            T[buf][cy][cx] = a < g.nu[0] && b < g.nu[1] ? kc * s[pidx(g.sy, g.sz, a, b, L)] : 0.0;
        }
        __syncthreads();
        // this node's cells: (i-1, j-1) = (tx, ty) ... (i, j) = (tx+1, ty+1)
        const double Px = T[buf][ty + 1][tx] + T[buf][ty + 1][tx + 1];
        const double Q = Px + (T[buf][ty][tx] + T[buf][ty][tx + 1]);
        const double Y = T[buf][ty][tx + 1] + T[buf][ty + 1][tx + 1];
        if (node && L >= kbeg) {
            const long long p = pidx(g.sy, g.sz, i, j, L);
            const double w5 = 5.0 * (Qp + Q), wx = Yp + Y, wy = Pp + Px;
            w.w5[p] = w5;
            w.wx[p] = wx;
            w.wy[p] = wy;
            w.wz[p] = Q;
            if (sx) w.wx[p + sx] = wx;
            if (sy) w.wy[p + sy] = wy;
            if (g.per[2] && L == g.n[2] - 1) w.wz[p - g.n[2] * g.sz] = Q;
            if (w.rd) {
                // the diagonal is K0 = -4 kc times the 8 cells
                const double diag = -0.8 * w5;
                const float fd = (float)diag;
                w.rd[p] = (fd > 1e-30f && fd < 1e30f) ? (double)__frcp_rn(fd) : 1.0 / diag;
            }
        }
        Qp = Q;
        Yp = Y;
        Pp = Px;
    }
}

// MODE 0: Jacobi sweep out = x + omega (b - A x) / diag; 1: residual out = b - A x (with the max norm);
// 2: out = -A x; 3: the residual of mode 1 as the next FP32 right-hand side, out32 = scale (b - A x)
template <int MODE>
__global__ void __launch_bounds__(kQThreads, 3) k_qsweep64(NodalGeom g, const double* __restrict__ x,
                                                        const double* __restrict__ b, const double* __restrict__ s,
                                                        QWeights w, double* __restrict__ out, double omega,
                                                        int kchunk, unsigned long long* norm,
                                                        float* __restrict__ out32, const KrylovState* __restrict__ ks)
{
    __shared__ double T[2][QY + 1][QX + 1];
    const double scale = MODE == 3 ? ks->scale : 0.0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the cell of this thread: tile column cx (0 = the halo column x0-1), tile row cy (0 = the halo row y0-1)
    const bool halo = warp == QY + 1;
    const int cx = halo ? 0 : lane + 1, cy = halo ? lane : warp;
    const int i = blockIdx.x * QX - 1 + cx, j = blockIdx.y * QY - 1 + cy;
    const int kbeg = blockIdx.z * kchunk;
    const int kend = min(kbeg + kchunk, g.nu[2]);
    // a thread whose cell lies outside the padded box still takes part in the barriers
    const bool inbox = cy <= QY && i < g.nu[0] && j < g.nu[1];
    const bool owner = !halo && cy >= 1 && i < g.nu[0] && j < g.nu[1];
    const bool dxy = owner && ((g.dlo[0] && i == 0) || (g.dhi[0] && i == g.n[0]) || (g.dlo[1] && j == 0) ||
                               (g.dhi[1] && j == g.n[1]));
    const long long sy = g.sy, sz = g.sz;
    const double mkc = -g.K[3];
    long long pc = pidx(sy, sz, i, j, kbeg - 1);  // node (i, j, k) for the current k
    // q = sum of the 4 nodes (i..i+1, j..j+1) of a node plane
    auto qsum = [&](long long pp) { return (x[pp] + x[pp + 1]) + (x[pp + sy] + x[pp + sy + 1]); };
    double q_lo = inbox ? qsum(pc) : 0.0;  // plane kbeg-1
    double u_lo = 0.0;                     // layer kbeg-1 sum around the node
    unsigned long long nkey = 0;
    double xm = 0.0, xc = 0.0, wzm = 0.0;
    if (owner) {
        xm = x[pc];
        xc = x[pc + sz];
        wzm = w.wz[pc];
    }
    for (int k = kbeg - 1; k < kend; ++k, pc += sz) {
        // cell layer k: (i, j, k) .. (i+1, j+1, k+1)
        const double q_hi = inbox ? qsum(pc + sz) : 0.0;
        const int buf = (k - kbeg + 1) & 1;
        if (cy <= QY) T[buf][cy][cx] = inbox ? s[pc] * (q_lo + q_hi) : 0.0;
        q_lo = q_hi;
        // node (i, j, k): layers k-1 (u_lo) and k; its own terms do not need the tile
        const bool node = owner && k >= kbeg;
        const bool live = node && !(dxy || (g.dlo[2] && k == 0) || (g.dhi[2] && k == g.n[2]) || (g.mask && !g.mask[pc]));
        double xp = 0.0, wzp = 0.0, e = 0.0;
        if (node) {
            xp = x[pc + sz];
            wzp = w.wz[pc];
        }
        if (live) {
            e = MODE == 2 ? xc * w.w5[pc] : fma(xc, w.w5[pc], b[pc]);
            e = fma(x[pc + 1], w.wx[pc], e);
            e = fma(x[pc - 1], w.wx[pc - 1], e);
            e = fma(x[pc + sy], w.wy[pc], e);
            e = fma(x[pc - sy], w.wy[pc - sy], e);
            e = fma(xp, wzp, e);
            e = fma(xm, wzm, e);
        }
        __syncthreads();
        if (owner) {
            const double u = (T[buf][cy - 1][cx - 1] + T[buf][cy - 1][cx]) + (T[buf][cy][cx - 1] + T[buf][cy][cx]);
            if (node) {
                double v = 0.0;
                if (live) {
                    v = fma(mkc, u_lo + u, e);  // b - A x (MODE 2: -A x)
                    if (MODE == 0) {
                        v = fma(omega * v, w.rd[pc], xc);
                    } else if ((MODE == 1 || MODE == 3) && norm) {
                        // |v| / V_node as an integer key (boundary nodes: V / 2^e, exact scaling)
                        const int f = (!g.per[0] && (i == 0 || i == g.n[0])) + (!g.per[1] && (j == 0 || j == g.n[1])) +
                                      (!g.per[2] && (k == 0 || k == g.n[2]));
                        const unsigned long long kb = f == 0 ? abs_key(v) : abs_key(v * (double)(1 << f));
                        nkey = kb > nkey ? kb : nkey;
                    }
                }
                if (MODE == 3)
                    out32[pc] = (float)(scale * v);
                else if (q_alias(g, i, j, k))
                    store_node(out, g, i, j, k, v);
                else
                    out[pc] = v;
                wzm = wzp;
                xm = xc;
                xc = xp;
            }
            u_lo = u;
        }
    }
    if ((MODE == 1 || MODE == 3) && norm) {
        nkey = block_max_key(nkey);
        if (threadIdx.x == 0) atomic_max_nonneg(norm, key_value(nkey) * g.ivol);
    }
}

// first Jacobi sweep from zero: out = omega b / diag (the level sweeps' layout: z is a grid direction)
__global__ void __launch_bounds__(256) k_qzero64(NodalGeom g, const double* __restrict__ rd,
                                                 const double* __restrict__ b, double* __restrict__ out, double omega)
{
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, k = blockIdx.z;
    if (i >= g.nu[0] || j >= g.nu[1]) return;
    const long long p = pidx(g.sy, g.sz, i, j, k);
    const double v = node_is_dirichlet(g, i, j, k) ? 0.0 : omega * b[p] * rd[p];
    if (q_alias(g, i, j, k))
        store_node(out, g, i, j, k, v);
    else
        out[p] = v;
}

}  // namespace

// Levels of at least 100 k nodes (46^3): the precomputed sums cost 40 B per node and a launch per sigma, which the
// smaller levels, bound by launches and not by the FP64 pipe, do not earn back.
constexpr long long kQMinNodes = 100000;

bool qsweep_supported(const NodalGeom& g)
{
    return g.iso != 0 && (long long)g.nu[0] * g.nu[1] * g.nu[2] >= kQMinNodes;
}

// z chunk of a CTA: its planes and the extra cell layer below them all pass the SM's FP64 pipe, so the time is the
// largest number of CTAs on one SM times (chunk + 1); one CTA alone on an SM also waits for its own loads.
static int q_chunk(int tiles, int nz)
{
    const int sms = sm_count_cached();
    int best = nz;
    double cost = 1e300;
    for (int c = 1; c <= nz; ++c) {
        const int per = (tiles * ((nz + c - 1) / c) + sms - 1) / sms;
        const double t = per * (c + 1.0) * (1.0 + 0.35 / per);
        if (t < cost * (1.0 - 1e-9)) {
            cost = t;
            best = c;
        }
    }
    return best;
}

void nodal_qweights64(const NodalGeom& g, const double* s64, const QWeights& w, cudaStream_t st)
{
    const int bx = (g.nu[0] + QX - 1) / QX, by = (g.nu[1] + QY - 1) / QY;
    const int kchunk = q_chunk(bx * by, g.nu[2]);
    k_qweights64<<<dim3(bx, by, (g.nu[2] + kchunk - 1) / kchunk), 32 * QY, 0, st>>>(g, s64, w, kchunk);
}

void nodal_qsweep64(const NodalGeom& g, int mode, const double* s64, const QWeights& w, const double* x,
                    const double* b, double* out, double omega, unsigned long long* norm, cudaStream_t st,
                    float* out32, const KrylovState* ks)
{
    const int bx = (g.nu[0] + QX - 1) / QX, by = (g.nu[1] + QY - 1) / QY;
    const int kchunk = q_chunk(bx * by, g.nu[2]);
    const dim3 grid(bx, by, (g.nu[2] + kchunk - 1) / kchunk);
    if (mode == 0)
        k_qsweep64<0><<<grid, kQThreads, 0, st>>>(g, x, b, s64, w, out, omega, kchunk, norm, nullptr, nullptr);
    else if (mode == 1)
        k_qsweep64<1><<<grid, kQThreads, 0, st>>>(g, x, b, s64, w, out, omega, kchunk, norm, nullptr, nullptr);
    else if (mode == 2)
        k_qsweep64<2><<<grid, kQThreads, 0, st>>>(g, x, b, s64, w, out, omega, kchunk, norm, nullptr, nullptr);
    else
        k_qsweep64<3><<<grid, kQThreads, 0, st>>>(g, x, b, s64, w, nullptr, omega, kchunk, norm, out32, ks);
}

void nodal_qzero64(const NodalGeom& g, const QWeights& w, const double* b, double* out, double omega, cudaStream_t st)
{
    k_qzero64<<<dim3((g.nu[0] + 31) / 32, (g.nu[1] + 7) / 8, g.nu[2]), dim3(32, 8), 0, st>>>(g, w.rd, b, out, omega);
}

}  // namespace gbp

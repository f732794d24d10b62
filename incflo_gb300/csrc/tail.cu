// The small levels of a V-cycle in one launch, their data in the shared memory of a thread-block cluster.
//
// A level of a few thousand unknowns keeps the chip busy for a microsecond per sweep; what it costs is the step from
// one sweep to the next. Launches cost 2 to 4 us each, and a cluster that keeps the level data in L2 about 3 us per
// phase (coherent loads, a barrier that orders global memory): 80 us per V-cycle for the nodal levels from 17^3 down,
// 107 us for the cell-centred ones from 32^3 down. Here every CTA owns a slab of z planes of each level and keeps one
// more plane on either side; a sweep reads local shared memory only and a store also updates the copies of its plane in
// the other CTAs (distributed shared memory), so a phase ends with one cluster barrier and nothing travels through L2.
// The levels that one CTA's threads cover in a pass or two are cycled by CTA 0 alone between block barriers, which cost
// less than cluster barriers (1.2 k cycles). The kinds of phase are written once inside one loop over the phases:
// instantiated per level, the code was fetched cold phase after phase. 63 us per V-cycle for the nodal levels from 17^3
// down and 66 us for the cell-centred ones from 16^3 down; latency bounds both (a pass over 125 nodes costs 1.5 us).
//
// Which levels: FP32 from 5000 unknowns down (33^3 and 32^3 as well: 118 and 104 us per V-cycle, more than the launches
// over the chip take for them). FP64: the 16 SMs' FP64 pipes (2 lanes per clock) take 1.6 k cycles for a half sweep of
// 16^3 cells; the nodal levels from 9^3 down gain (16^3 cells, plain FP64: 1260 -> 1150 us per solve), the cell-centred ones
// do not (64^3: 2230 us from 16^3 down, 2170 us from 8^3 down, 2150 us with launches), so they have no tail.
#include "tail.h"

#include <algorithm>
#include <type_traits>

#include "bottom.h"
#include "nodal_op.cuh"

namespace gbp {

namespace {

__device__ __forceinline__ unsigned saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned a, unsigned rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_remote(unsigned a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_remote(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// what a phase needs of a level, in shared memory (a kernel parameter indexed by level is a cached constant that misses,
// and every conversion of a coefficient to FP32 an instruction of the FP64 pipe)
template <typename T>
struct Lev {
    int off[7];             // element offsets of its arrays
    int lo, np, sy, sz;     // slab, pitches (those of the global padded layout)
    int n[3], nu[3];        // cells, unique points
    unsigned m01, m0;       // ceil(2^32 / (points of a plane, of a row)): quotients by one multiplication
    int px, py, pz;         // period where periodic, else 0
    int copies;
    bool solo;
    int dir[6];             // the value of i, j, k on Dirichlet sides, else -1 (low and high)
    const unsigned char* mask;
    T K[8], w[3];           // element entries (nodal), face weights (cell-centred)
    const T* ac;            // alpha a V (cell-centred, may be null)
    __device__ __forceinline__ bool held(int i, int j, int k) const
    {
        return i == dir[0] || i == dir[1] || j == dir[2] || j == dir[3] || k == dir[4] || k == dir[5] ||
               (mask && !mask[pidx(sy, sz, i, j, k)]);
    }
};
__device__ __forceinline__ unsigned recip32(unsigned d) { return (unsigned)((0x100000000ull + d - 1) / d); }
// (t < 2^17 and points per plane < 2^15 in a tail, so the products below stay exact)
template <typename T>
__device__ __forceinline__ void split(const Lev<T>&, unsigned row, unsigned plane, unsigned m0, unsigned m01, unsigned t,
                                      int& i, int& j, int& kl)
{
    kl = m01 ? (int)__umulhi(t, m01) : (int)t;
    const unsigned r = t - (unsigned)kl * plane;
    j = m0 ? (int)__umulhi(r, m0) : (int)r;
    i = (int)(r - (unsigned)j * row);
}
// (p >= 4: a level above the bottom)
__device__ __forceinline__ int node_step(int i, int p) { return !p ? 0 : (i <= 1 ? p : (i == p - 1 ? -p : 0)); }
__device__ __forceinline__ int cell_step(int i, int p) { return !p ? 0 : (i == 0 ? p : (i == p - 1 ? -p : 0)); }

// contiguous planes between global and shared memory, 16 bytes per access (pitches are multiples of 8 elements)
template <typename T>
__device__ __forceinline__ void copy_planes(T* dst, const T* src, int n)
{
    const float4* s = reinterpret_cast<const float4*>(src);
    float4* d = reinterpret_cast<float4*>(dst);
    const int n4 = n * (int)sizeof(T) / 16;
#pragma unroll 4
    for (int t = threadIdx.x; t < n4; t += kTailThreads) d[t] = s[t];
}
template <typename T>
__device__ __forceinline__ void clear_planes(T* dst, int n)
{
    float4* d = reinterpret_cast<float4*>(dst);
    const int n4 = n * (int)sizeof(T) / 16;
    for (int t = threadIdx.x; t < n4; t += kTailThreads) d[t] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Store at padded position `at` of local slot `slot`: the aliases (steps ex, ey; ez in a level that one CTA holds whole),
// the copies of the plane in other CTAs, or (all > 1) every other CTA's same position.
template <typename T>
__device__ __forceinline__ void put(T* arr, const Lev<T>& L, int slot, int at, int ex, int ey, int ez, const int* copies, int all,
                                    T v)
{
    T* p = arr + slot * L.sz + at;
    *p = v;
    const int n = copies ? copies[0] : all - 1;
    if (!(ex | ey | ez) && n <= 0) return;
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
        if (((c & 1) && !ex) || ((c & 2) && !ey) || ((c & 4) && !ez)) continue;
        const int d = ((c & 1) ? ex : 0) + ((c & 2) ? ey : 0) + ((c & 4) ? ez : 0);
        p[d] = v;
        for (int m = 1; m <= n; ++m) {
            if (copies)
                st_remote(map_rank(saddr(arr + (copies[m] & 0xffff) * L.sz + at + d), (unsigned)copies[m] >> 16), v);
            else
                st_remote(map_rank(saddr(p + d), m), v);
        }
    }
}

// ------------------------------------------------------------------------------------------------ nodal
// A x at one node, and the diagonal (NodalOp with the element entries in T)
template <typename T, bool ISO>
__device__ __forceinline__ T node_op(const T* x, const T* s, int c, int sy, int sz, const T (&K)[8], T& diag)
{
    const T xc = x[c];
    T acc = T(0), ssum = T(0);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int cx = m & 1, cy = (m >> 1) & 1, cz = m >> 2;
        const T sg = s[c + (cx - 1) + (cy - 1) * sy + (cz - 1) * sz];
        const int ox = cx ? 1 : -1, oy = cy ? sy : -sy, oz = cz ? sz : -sz;
        ssum += sg;
        if (ISO && sizeof(T) == 8) {
            acc = fma(sg, (x[c + ox + oy] + x[c + ox + oz]) + (x[c + oy + oz] + x[c + ox + oy + oz]), acc);
        } else if (ISO) {
            acc += sg * (((x[c + ox + oy] - xc) + (x[c + ox + oz] - xc)) + ((x[c + oy + oz] - xc) + (x[c + ox + oy + oz] - xc)));
        } else {
            const T t = K[1] * (x[c + ox] - xc) + K[2] * (x[c + oy] - xc) + K[4] * (x[c + oz] - xc) +
                        K[3] * (x[c + ox + oy] - xc) + K[5] * (x[c + ox + oz] - xc) + K[6] * (x[c + oy + oz] - xc) +
                        K[7] * (x[c + ox + oy + oz] - xc);
            acc += sg * t;
        }
    }
    diag = K[0] * ssum;
    if (ISO && sizeof(T) == 8) return K[3] * fma(T(-4) * xc, ssum, acc);
    return ISO ? K[3] * acc : acc;
}

// Arrays of a level: 0 sigma (slot s holds the cell layer lo + s - 1), 1 and 2 the iterate and its ping-pong partner
// (node plane lo + s - 1), 3 the right-hand side (plane lo + s).
template <typename T, bool ISO>
__global__ void __launch_bounds__(kTailThreads, 1) k_nodal_tail(const __grid_constant__ NodalTail<T> a)
{
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ Lev<T> lev[kTailLevels];
    T* sm = reinterpret_cast<T*>(raw);
    int* tab = reinterpret_cast<int*>(raw + a.tab_off);
    const int me = (int)cluster_rank();
    const int last = a.nl - 1, solo = a.solo;
    for (int t = threadIdx.x; t < a.tab_ints; t += kTailThreads) tab[t] = a.table[t];
    if (threadIdx.x < a.nl) {
        const int q = threadIdx.x;
        const NodalGeom& g = a.g[q];
        Lev<T>& L = lev[q];
        L.lo = a.table[a.own[q] + 2 * me];
        L.np = a.table[a.own[q] + 2 * me + 1];
        L.sy = (int)g.sy;
        L.sz = (int)g.sz;
        for (int d = 0; d < 3; ++d) {
            L.n[d] = g.n[d];
            L.nu[d] = g.nu[d];
        }
        const int np = a.np[q], at[4] = {0, np + 1, 2 * np + 3, 3 * np + 5};
        for (int r = 0; r < 4; ++r) L.off[r] = a.off[q] + at[r] * L.sz;
        const unsigned row = g.nu[0], plane = row * g.nu[1];
        L.m0 = row > 1 ? recip32(row) : 0;
        L.m01 = plane > 1 ? recip32(plane) : 0;
        L.px = g.per[0] ? g.n[0] : 0;
        L.py = g.per[1] ? g.n[1] : 0;
        L.pz = g.per[2] ? g.n[2] : 0;
        L.copies = a.copies[q];
        L.solo = q >= solo;
        for (int d = 0; d < 3; ++d) {
            L.dir[2 * d] = g.dlo[d] ? 0 : -1;
            L.dir[2 * d + 1] = g.dhi[d] ? g.n[d] : -1;
        }
        L.mask = g.mask;
        for (int m = 0; m < 8; ++m) L.K[m] = (T)g.K[m];
    }
    __syncthreads();
    // bottom: right-hand side and inverse in CTA 0, the solution where it is prolonged
    const NodalGeom& gb = a.g[last];
    const int N = gb.nu[0] * gb.nu[1] * gb.nu[2];
    double* bb = reinterpret_cast<double*>(raw + a.dense_off);
    double* xb = bb + N;
    double* M = xb + N;
    if (me == 0)
        for (int t = threadIdx.x; t < N * N; t += kTailThreads) M[t] = a.M[t];
    for (int q = 0; q < last; ++q) {
        const Lev<T>& L = lev[q];
        if (q < solo || me == 0) copy_planes(sm + L.off[0], a.s[q] + (long long)L.lo * L.sz, (L.np + 1) * L.sz);
        if (q == 0 && (solo > 0 || me == 0)) copy_planes(sm + L.off[3], a.b0 + (L.lo + 1ll) * L.sz, L.np * L.sz);
        clear_planes(sm + L.off[1], 2 * (a.np[q] + 2) * L.sz);
    }
    cluster_barrier();  // every CTA's arrays are cleared before another stores into them
    // the pre-smoothing leaves a level's iterate in buffer pre, the post-smoothing in buffer done
    const int pre = (a.nu1 - 1) & 1, done = (pre + a.nu2) & 1;
    enum { kZero, kSweep, kResid, kRestrict, kBottom, kProlong };
    bool downward = true;
    int q = 0, sub = 0;
    for (;;) {
        int op, c = 0, p = 0;
        if (downward) {
            op = q == last ? kBottom : (sub == 0 ? kZero : (sub < a.nu1 ? kSweep : (sub == a.nu1 ? kResid : kRestrict)));
            c = sub == a.nu1 + 1 ? pre ^ 1 : (sub - 1) & 1;
            p = sub;
        } else {
            op = sub == 0 ? kProlong : kSweep;
            p = sub - 1;
            c = sub == 0 ? pre : (pre + p) & 1;
        }
        const bool mine = (q < solo && q < last) || me == 0;
        const bool final = !downward && sub == a.nu2;
        if (mine) {
            const Lev<T>& L = lev[q];
            if (op <= kResid || op == kProlong) {
                // over this CTA's nodes of the level
                const T w = downward ? a.wpre[p % kSweepWeights] : a.wpost[p % kSweepWeights];
                const int plane = L.nu[0] * L.nu[1], total = plane * L.np;
                T* x = sm + L.off[1 + c];
                const T* s = sm + L.off[0];
                const T* b = sm + L.off[3];
                T* out = sm + L.off[op == kZero ? 1 : (op == kProlong ? 1 + c : 2 - c)];
                const int* copies = L.solo ? nullptr : tab + L.copies;
                const int all = L.solo && final && q == solo ? a.ctas : 1;
                for (int t = threadIdx.x; t < total; t += kTailThreads) {
                    int i, j, kl;
                    split(L, L.nu[0], plane, L.m0, L.m01, t, i, j, kl);
                    const int k = L.lo + kl, at = (i + kOX) + (j + 1) * L.sy, o = (kl + 1) * L.sz + at;
                    T v = T(0);
                    if (!L.held(i, j, k)) {
                        if (op == kZero) {
                            const int sy = L.sy, sz = L.sz;
                            const T ssum = ((s[o - 1 - sy - sz] + s[o - sy - sz]) + (s[o - 1 - sz] + s[o - sz])) +
                                           ((s[o - 1 - sy] + s[o - sy]) + (s[o - 1] + s[o]));
                            v = w * b[o - L.sz] * approx_recip(L.K[0] * ssum);
                        } else if (op == kProlong) {
                            const Lev<T>& C = lev[q + 1];
                            const int oi = i & 1, oj = j & 1, ok = k & 1;
                            const T* xc = sm + C.off[1 + done];
                            T acc = T(0);
#pragma unroll 1
                            for (int m = 0; m < 8; ++m) {
                                if (((m & 1) > oi) || (((m >> 1) & 1) > oj) || ((m >> 2) > ok)) continue;
                                int I = (i >> 1) + (m & 1), J = (j >> 1) + ((m >> 1) & 1), K = (k >> 1) + (m >> 2);
                                if (q + 1 < last) {
                                    acc += xc[(K - C.lo + 1) * C.sz + (I + kOX) + (J + 1) * C.sy];
                                } else {
                                    I = I == C.nu[0] ? 0 : I;
                                    J = J == C.nu[1] ? 0 : J;
                                    K = K == C.nu[2] ? 0 : K;
                                    acc += (T)xb[I + C.nu[0] * (J + C.nu[1] * K)];
                                }
                            }
                            const int sh = oi + oj + ok;
                            v = x[o] + (sh == 0 ? T(1) : (sh == 1 ? T(0.5) : (sh == 2 ? T(0.25) : T(0.125)))) * acc;
                        } else {
                            T diag;
                            const T ax = node_op<T, ISO>(x, s, o, L.sy, L.sz, L.K, diag);
                            const T r = b[o - L.sz] - ax;
                            v = op == kResid ? r : x[o] + w * r * approx_recip(diag);
                        }
                    }
                    if (final && q == 0) {
                        store_node(a.xout, a.g[0], i, j, k, v);
                        continue;
                    }
                    const int* cp = copies ? copies + k * (kTailTargets + 1) : nullptr;
                    // (a level of one CTA keeps planes -1 .. n of a periodic z, no plane n + 1)
                    const int ez = L.solo ? cell_step(kl, L.pz) * L.sz : 0;
                    put(out, L, kl + 1, at, node_step(i, L.px), node_step(j, L.py) * L.sy, ez, cp, all, v);
                }
            } else if (op == kRestrict) {
                // full weighting into the next level's right-hand side: its own slab's, or CTA 0's
                const Lev<T>& C = lev[q + 1];
                const bool into0 = q + 1 == last || (C.solo && !L.solo);
                const int K0 = into0 ? (L.lo + 1) / 2 : C.lo;
                const int nk = into0 ? min((L.lo + L.np + 1) / 2, C.nu[2]) - K0 : C.np;
                const int plane = C.nu[0] * C.nu[1], total = plane * nk;
                const T* r = sm + L.off[1 + c];
                for (int t = threadIdx.x; t < total; t += kTailThreads) {
                    int I, J, kk;
                    split(C, C.nu[0], plane, C.m0, C.m01, t, I, J, kk);
                    const int K = K0 + kk;
                    T v = T(0);
                    if (!C.held(I, J, K)) {
                        const int f = (2 * K - L.lo + 1) * L.sz + (2 * I + kOX) + (2 * J + 1) * L.sy;
#pragma unroll
                        for (int dz = -1; dz <= 1; ++dz) {
                            T accy = T(0);
#pragma unroll
                            for (int dy = -1; dy <= 1; ++dy) {
                                const int row = f + dy * L.sy + dz * L.sz;
                                accy += (dy == 0 ? T(1) : T(0.5)) * (T(0.5) * (r[row - 1] + r[row + 1]) + r[row]);
                            }
                            v += (dz == 0 ? T(1) : T(0.5)) * accy;
                        }
                    }
                    T* cb = sm + C.off[3] + (K - C.lo) * C.sz + (I + kOX) + (J + 1) * C.sy;
                    if (q + 1 == last)
                        st_remote(map_rank(saddr(bb + I + C.nu[0] * (J + C.nu[1] * K)), 0), (double)v);
                    else if (into0)
                        st_remote(map_rank(saddr(cb), 0), v);
                    else
                        *cb = v;
                }
            } else {
                // x = M b (a singular system's right-hand side made consistent over the free nodes first), by the first
                // warps: an FP64 instruction costs the SM 16 cycles per warp
                if (threadIdx.x < 32 && a.singular) {
                    constexpr int kOwn = (kDenseBottom + 31) / 32;  // unknowns of a lane
                    double sb = 0.0, sv = 0.0, vu[kOwn] = {};
#pragma unroll
                    for (int h = 0; h < kOwn; ++h) {
                        const int u = threadIdx.x + 32 * h;
                        if (u >= N) break;
                        int ui, uj, uk;
                        split(L, L.nu[0], L.nu[0] * L.nu[1], L.m0, L.m01, u, ui, uj, uk);
                        if (node_is_dirichlet(gb, ui, uj, uk)) continue;
                        vu[h] = node_volume(gb, ui, uj, uk);
                        sb += bb[u];
                        sv += vu[h];
                    }
                    for (int o = 16; o > 0; o >>= 1) {
                        sb += __shfl_xor_sync(0xffffffffu, sb, o);
                        sv += __shfl_xor_sync(0xffffffffu, sv, o);
                    }
                    const double m = sv > 0.0 ? sb / sv : 0.0;
#pragma unroll
                    for (int h = 0; h < kOwn; ++h)
                        if (threadIdx.x + 32 * h < N) bb[threadIdx.x + 32 * h] -= m * vu[h];
                }
                __syncthreads();
                if (threadIdx.x < N) {
                    const int u = threadIdx.x;
                    double v0 = 0.0, v1 = 0.0;
                    int v = 0;
                    for (; v + 1 < N; v += 2) {
                        v0 = fma(M[v * N + u], bb[v], v0);
                        v1 = fma(M[(v + 1) * N + u], bb[v + 1], v1);
                    }
                    if (v < N) v0 = fma(M[v * N + u], bb[v], v0);
                    xb[u] = v0 + v1;
                    if (solo >= last)
                        for (int r = 1; r < a.ctas; ++r) st_remote(map_rank(saddr(xb + u), r), v0 + v1);
                }
            }
        }
        // advance
        if (final && q == 0) break;
        const int was = q;
        if (downward) {
            if (q == last) {
                downward = false;
                q = last - 1;
                sub = 0;
            } else if (++sub > a.nu1 + 1) {
                sub = 0;
                ++q;
            }
        } else if (++sub > a.nu2) {
            sub = 0;
            --q;
        }
        // a phase of one CTA ends in that CTA, until the cluster takes over again
        const bool alone = min(was, last) >= min(solo, last), next_alone = min(q, last) >= min(solo, last);
        if (alone && next_alone) {
            if (me == 0) __syncthreads();
        } else {
            cluster_barrier();
        }
    }
    // every store into another CTA lies before a cluster barrier that its owner takes part in
}

// ------------------------------------------------------------------------------------------------ cell-centred
template <typename T>
__device__ __forceinline__ const T* tail_acoef(const CellGeom& g);
template <>
__device__ __forceinline__ const double* tail_acoef<double>(const CellGeom& g) { return g.a64; }
template <>
__device__ __forceinline__ const float* tail_acoef<float>(const CellGeom& g) { return g.a32; }

// Arrays of a level (slot s holds plane lo + s - 1): 0 the iterate, 1 the residual, 2 the right-hand side, 3 1 / diag,
// 4 to 6 the face coefficients.
template <typename T>
__global__ void __launch_bounds__(kTailThreads, 1) k_mac_tail(const __grid_constant__ MacTail<T> a)
{
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ Lev<T> lev[kTailLevels];
    T* sm = reinterpret_cast<T*>(raw);
    int* tab = reinterpret_cast<int*>(raw + a.tab_off);
    const int me = (int)cluster_rank();
    const int last = a.nl - 1, solo = a.solo;
    for (int t = threadIdx.x; t < a.tab_ints; t += kTailThreads) tab[t] = a.table[t];
    if (threadIdx.x < a.nl) {
        const int q = threadIdx.x;
        const CellGeom& g = a.g[q];
        Lev<T>& L = lev[q];
        L.lo = a.table[a.own[q] + 2 * me];
        L.np = a.table[a.own[q] + 2 * me + 1];
        L.sy = (int)g.sy;
        L.sz = (int)g.sz;
        for (int d = 0; d < 3; ++d) L.n[d] = L.nu[d] = g.n[d];
        // (2 to 6 hold planes lo .. only: their slot 0 would lie before them)
        const int np = a.np[q], at[7] = {0, np + 2, 2 * np + 3, 3 * np + 3, 4 * np + 3, 5 * np + 3, 6 * np + 3};
        for (int r = 0; r < 7; ++r) L.off[r] = a.off[q] + at[r] * L.sz;
        // half a row: the cells of one colour
        const unsigned row = (g.n[0] + 1) / 2, plane = row * g.n[1];
        L.m0 = row > 1 ? recip32(row) : 0;
        L.m01 = plane > 1 ? recip32(plane) : 0;
        L.px = g.per[0] ? g.n[0] : 0;
        L.py = g.per[1] ? g.n[1] : 0;
        L.pz = g.per[2] ? g.n[2] : 0;
        L.copies = a.copies[q];
        L.solo = q >= solo;
        for (int d = 0; d < 3; ++d) L.w[d] = (T)g.w[d];
        L.ac = tail_acoef<T>(g);
    }
    __syncthreads();
    const CellGeom& gb = a.g[last];
    const int N = gb.n[0] * gb.n[1] * gb.n[2];
    double* bb = reinterpret_cast<double*>(raw + a.dense_off);
    double* xb = bb + N;
    double* M = xb + N;
    if (me == 0)
        for (int t = threadIdx.x; t < N * N; t += kTailThreads) M[t] = a.M[t];
    for (int q = 0; q < last; ++q) {
        const Lev<T>& L = lev[q];
        if (q < solo || me == 0) {
            const long long at = (L.lo + 1ll) * L.sz;
            copy_planes(sm + L.off[4] + L.sz, a.bx[q] + at, L.np * L.sz);
            copy_planes(sm + L.off[5] + L.sz, a.by[q] + at, L.np * L.sz);
            copy_planes(sm + L.off[6] + L.sz, a.bz[q] + at, (L.np + 1) * L.sz);
            if (q == 0) copy_planes(sm + L.off[2] + L.sz, a.b0 + at, L.np * L.sz);
        }
        clear_planes(sm + L.off[0], 2 * (a.np[q] + 2) * L.sz);
    }
    __syncthreads();
    for (int q = 0; q < last; ++q) {
        if (q >= solo && me != 0) break;
        const Lev<T>& L = lev[q];
        const T wx = L.w[0], wy = L.w[1], wz = L.w[2];
        const T* ac = L.ac;
        const T *bx = sm + L.off[4], *by = sm + L.off[5], *bz = sm + L.off[6];
        const int hx = (L.n[0] + 1) / 2, plane = hx * L.n[1];
        for (int t = threadIdx.x; t < plane * L.np; t += kTailThreads) {
            int h, j, kl;
            split(L, hx, plane, L.m0, L.m01, t, h, j, kl);
            for (int i = 2 * h; i < min(2 * h + 2, L.n[0]); ++i) {
                const int o = (kl + 1) * L.sz + (i + kOX) + (j + 1) * L.sy;
                T d = wx * (bx[o] + bx[o + 1]) + wy * (by[o] + by[o + L.sy]) + wz * (bz[o] + bz[o + L.sz]);
                if (ac) d += ac[pidx(L.sy, L.sz, i, j, L.lo + kl)];
                sm[L.off[3] + o] = d != T(0) ? T(1) / d : T(0);
            }
        }
    }
    cluster_barrier();  // every CTA's arrays are cleared before another stores into them
    // down a level: the half sweep from zero, black, (red, black) ..., the red residual, its restriction; up: the black
    // half sweep from the prolonged correction, red, (black, red) ...
    enum { kZero, kHalf, kResid, kRestrict, kBottom, kProlong };
    bool downward = true;
    int q = 0, sub = 0;
    for (;;) {
        int op, color = 0;
        if (downward) {
            op = q == last ? kBottom : (sub == 0 ? kZero : (sub < 2 * a.nu1 ? kHalf : (sub == 2 * a.nu1 ? kResid : kRestrict)));
            color = op == kHalf ? sub & 1 : 0;
        } else {
            op = sub == 0 ? kProlong : kHalf;
            color = (sub & 1) ^ 1;
        }
        const bool mine = (q < solo && q < last) || me == 0;
        const bool end = !downward && sub >= 2 * a.nu2 - 2;  // the last pair of half sweeps of a level
        if (mine) {
            const Lev<T>& L = lev[q];
            const auto cells = [&](auto what) {
                constexpr int OP = decltype(what)::value;
                const int hx = (L.n[0] + 1) / 2, plane = hx * L.n[1], total = plane * L.np, sy = L.sy, sz = L.sz;
                const T wx = L.w[0], wy = L.w[1], wz = L.w[2];
                const T *x = sm + L.off[0], *b = sm + L.off[2], *id = sm + L.off[3];
                const T *bx = sm + L.off[4], *by = sm + L.off[5], *bz = sm + L.off[6];
                T* out = sm + L.off[OP == kResid ? 1 : 0];
                const T* ac = L.ac;
                const int* copies = L.solo ? nullptr : tab + L.copies;
                const int all = L.solo && end && q == solo ? a.ctas : 1;  // the result goes to every CTA
                for (int t = threadIdx.x; t < total; t += kTailThreads) {
                    int h, j, kl;
                    split(L, hx, plane, L.m0, L.m01, t, h, j, kl);
                    const int k = L.lo + kl, i = 2 * h + ((j + k + color) & 1);
                    if (i >= L.n[0]) continue;
                    const int at = (i + kOX) + (j + 1) * sy, o = (kl + 1) * sz + at;
                    T v;
                    if constexpr (OP == kZero) {
                        v = b[o] * id[o];
                    } else {
                        T xw = x[o - 1], xe = x[o + 1], xs = x[o - sy], xn = x[o + sy], xd = x[o - sz], xu = x[o + sz];
                        if constexpr (OP == kProlong) {
                            // + the coarse correction of each neighbour's parent (one past the sides included: the
                            // periodic copy, or 0)
                            const Lev<T>& C = lev[q + 1];
                            T e0 = T(0);
#pragma unroll
                            for (int m = 0; m < 7; ++m) {
                                const int d = (m - 1) >> 1, st = m == 0 ? 0 : ((m & 1) ? -1 : 1);
                                int I = (i >> 1) + (m && d == 0 ? st : 0), J = (j >> 1) + (m && d == 1 ? st : 0),
                                    K = (k >> 1) + (m && d == 2 ? st : 0);
                                T r = T(0);
                                if (q + 1 < last) {
                                    r = sm[C.off[0] + (K - C.lo + 1) * C.sz + (I + kOX) + (J + 1) * C.sy];
                                } else {
                                    if (C.px) I = I < 0 ? I + C.px : (I >= C.px ? I - C.px : I);
                                    if (C.py) J = J < 0 ? J + C.py : (J >= C.py ? J - C.py : J);
                                    if (C.pz) K = K < 0 ? K + C.pz : (K >= C.pz ? K - C.pz : K);
                                    if (I >= 0 && I < C.n[0] && J >= 0 && J < C.n[1] && K >= 0 && K < C.n[2])
                                        r = (T)xb[I + C.n[0] * (J + C.n[1] * K)];
                                }
                                if (m == 0) e0 = r;
                                if (m == 1) xw += (i & 1) ? e0 : r;
                                if (m == 2) xe += (i & 1) ? r : e0;
                                if (m == 3) xs += (j & 1) ? e0 : r;
                                if (m == 4) xn += (j & 1) ? r : e0;
                                if (m == 5) xd += (k & 1) ? e0 : r;
                                if (m == 6) xu += (k & 1) ? r : e0;
                            }
                        }
                        // (the residual in differences to the cell, as the level kernels form it)
                        if (OP == kResid) {
                            const T xc = x[o];
                            xw -= xc, xe -= xc, xs -= xc, xn -= xc, xd -= xc, xu -= xc;
                        }
                        T acc = b[o];
                        acc += wx * (bx[o] * xw + bx[o + 1] * xe);
                        acc += wy * (by[o] * xs + by[o + sy] * xn);
                        acc += wz * (bz[o] * xd + bz[o + sz] * xu);
                        if (OP == kResid && ac) acc -= ac[pidx(sy, sz, i, j, k)] * x[o];
                        v = OP == kResid ? acc : acc * id[o];
                    }
                    put(out, L, kl + 1, at, cell_step(i, L.px), cell_step(j, L.py) * sy, L.solo ? cell_step(kl, L.pz) * sz : 0,
                        copies ? copies + k * (kTailTargets + 1) : nullptr, all, v);
                }
            };
            if (op == kZero) {
                cells(std::integral_constant<int, kZero>());
            } else if (op == kHalf) {
                cells(std::integral_constant<int, kHalf>());
            } else if (op == kResid) {
                cells(std::integral_constant<int, kResid>());
            } else if (op == kProlong) {
                cells(std::integral_constant<int, kProlong>());
            } else if (op == kRestrict) {
                const Lev<T>& C = lev[q + 1];
                const bool into0 = q + 1 == last || (C.solo && !L.solo);  // the coarse level lies in CTA 0
                const int K0 = into0 ? (L.lo + 1) / 2 : C.lo;
                const int nk = into0 ? min((L.lo + L.np + 1) / 2, C.n[2]) - K0 : C.np;
                const int hx = (C.n[0] + 1) / 2, plane = hx * C.n[1];
                for (int t = threadIdx.x; t < 2 * plane * nk; t += kTailThreads) {
                    int h, J, kk;
                    split(C, hx, plane, C.m0, C.m01, t >> 1, h, J, kk);
                    const int I = 2 * h + (t & 1), K = K0 + kk;
                    if (I >= C.n[0]) continue;
                    const T* f = sm + L.off[1] + (2 * K - L.lo + 1) * L.sz + (2 * I + kOX) + (2 * J + 1) * L.sy;
                    const T v = (f[0] + f[1 + L.sy]) + (f[1 + L.sz] + f[L.sy + L.sz]);
                    T* cb = sm + C.off[2] + (K - C.lo + 1) * C.sz + (I + kOX) + (J + 1) * C.sy;
                    if (q + 1 == last)
                        st_remote(map_rank(saddr(bb + I + C.n[0] * (J + C.n[1] * K)), 0), (double)v);
                    else if (into0)
                        st_remote(map_rank(saddr(cb), 0), v);
                    else
                        *cb = v;
                }
            } else {
                if (threadIdx.x < 32) {
                    double sb = 0.0, na = 0.0;
                    for (int u = threadIdx.x; u < N; u += 32) {
                        if (!a.act[u]) bb[u] = 0.0;
                        sb += bb[u];
                        na += a.act[u] ? 1.0 : 0.0;
                    }
                    if (a.singular) {
                        for (int o = 16; o > 0; o >>= 1) {
                            sb += __shfl_xor_sync(0xffffffffu, sb, o);
                            na += __shfl_xor_sync(0xffffffffu, na, o);
                        }
                        const double mean = na > 0.0 ? sb / na : 0.0;
                        for (int u = threadIdx.x; u < N; u += 32)
                            if (a.act[u]) bb[u] -= mean;
                    }
                }
                __syncthreads();
                if (threadIdx.x < N) {
                    const int u = threadIdx.x;
                    double v0 = 0.0;
                    for (int v = 0; v < N; ++v) v0 = fma(M[v * N + u], bb[v], v0);
                    xb[u] = v0;
                    if (solo >= last)
                        for (int r = 1; r < a.ctas; ++r) st_remote(map_rank(saddr(xb + u), r), v0);
                }
            }
        }
        // advance
        const int was = q;
        if (!downward && q == 0 && sub == 2 * a.nu2 - 1) break;
        if (downward) {
            if (q == last) {
                downward = false;
                q = last - 1;
                sub = 0;
            } else if (++sub > 2 * a.nu1 + 1) {
                sub = 0;
                ++q;
            }
        } else if (++sub > 2 * a.nu2 - 1) {
            sub = 0;
            --q;
        }
        const bool alone = min(was, last) >= min(solo, last), next_alone = min(q, last) >= min(solo, last);
        if (alone && next_alone) {
            if (me == 0) __syncthreads();
        } else {
            cluster_barrier();
        }
    }
    __syncthreads();
    // the result, with its aliases
    if (solo > 0 || me == 0) {
        const Lev<T>& L = lev[0];
        const CellGeom& g = a.g[0];
        const int hx = (L.n[0] + 1) / 2, plane = hx * L.n[1];
        for (int t = threadIdx.x; t < 2 * plane * L.np; t += kTailThreads) {
            int h, j, kl;
            split(L, hx, plane, L.m0, L.m01, t >> 1, h, j, kl);
            const int i = 2 * h + (t & 1);
            if (i < L.n[0]) store_cell(a.xout, g, i, j, L.lo + kl, sm[L.off[0] + (kl + 1) * L.sz + (i + kOX) + (j + 1) * L.sy]);
        }
    }
    // (the last half sweep's copies in other CTAs are not read, but no CTA may leave before they have arrived)
    cluster_barrier();
}

constexpr size_t kTailBytes = 224 * 1024;  // of the 227 KB of a CTA, beside the static part

template <typename K>
bool cluster_fits(K kern, int ctas, size_t bytes)
{
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailBytes) != cudaSuccess) return false;
    if (ctas > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = bytes;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    return cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0;
}

template <typename K, typename A>
int launch_tail(K kern, const A& a, size_t bytes, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.ctas);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = a.ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
    return e == cudaSuccess ? GBP_OK : cuda_fail(e, "tail of the V-cycle: launch");
}

}  // namespace

int tail_cluster_size()
{
    static const int ctas = [] {
        int n = 0;
        for (int c : {8, 16})
            if (cluster_fits(k_nodal_tail<float, true>, c, kTailBytes) && cluster_fits(k_nodal_tail<float, false>, c, kTailBytes) &&
                cluster_fits(k_nodal_tail<double, true>, c, kTailBytes) &&
                cluster_fits(k_nodal_tail<double, false>, c, kTailBytes) && cluster_fits(k_mac_tail<float>, c, kTailBytes))
                n = c;
        cudaGetLastError();  // a refused attribute or query leaves no sticky error behind
        return n;
    }();
    return ctas;
}

bool tail_layout(int nl, const int* planes, int per, const int* plane_elems, const long long* unknowns, int arrays,
                 int esize, int nbottom, long long solo_most, int ctas, TailLayout* out)
{
    TailLayout t;
    if (nl < 2 || nl > kTailLevels || ctas < 1) return false;
    t.nl = nl;
    while (t.solo < nl - 1 && unknowns[t.solo] > solo_most) ++t.solo;
    if (t.solo == 0) ctas = 1;
    t.ctas = ctas;
    std::vector<std::vector<int>> lo(nl, std::vector<int>(ctas)), np(nl, std::vector<int>(ctas));
    for (int q = 0; q < nl; ++q)
        for (int c = 0; c < ctas; ++c) {
            if (q >= t.solo) {
                lo[q][c] = 0;
                np[q][c] = planes[q];
            } else if (q == 0) {
                lo[q][c] = (int)((long long)planes[0] * c / ctas);
                np[q][c] = (int)((long long)planes[0] * (c + 1) / ctas) - lo[q][c];
            } else {
                // the coarse planes K with fine plane 2K in [lo, lo + np)
                const int f0 = lo[q - 1][c], f1 = f0 + np[q - 1][c];
                lo[q][c] = std::min((f0 + 1) / 2, planes[q]);
                np[q][c] = std::max(0, std::min((f1 + 1) / 2, planes[q]) - lo[q][c]);
            }
        }
    int elems = 0;
    for (int q = 0; q < nl; ++q) {
        t.np[q] = *std::max_element(np[q].begin(), np[q].end());
        t.plane[q] = plane_elems[q];
        t.own[q] = (int)t.table.size();
        for (int c = 0; c < ctas; ++c) {
            t.table.push_back(lo[q][c]);
            t.table.push_back(np[q][c]);
        }
        t.copies[q] = (int)t.table.size();
        for (int k = 0; k < planes[q] && q < t.solo; ++k) {
            std::vector<int> dst;
            for (int c = 0; c < ctas; ++c) {
                // its sweeps (planes of its own) or its prolongation to the finer level read the neighbours of its slab
                if (np[q][c] == 0 && (q == 0 || np[q - 1][c] == 0)) continue;
                for (int s : {-1, np[q][c]}) {
                    int p = lo[q][c] + s;
                    if (per) p = ((p % planes[q]) + planes[q]) % planes[q];
                    if (p == k) dst.push_back((c << 16) | (s + 1));
                }
            }
            if ((int)dst.size() > kTailTargets) return false;
            t.table.push_back((int)dst.size());
            for (int d : dst) t.table.push_back(d);
            t.table.resize(t.table.size() + (size_t)(kTailTargets - (int)dst.size()), 0);
        }
        t.off[q] = elems;
        if (q < nl - 1) elems += (arrays * t.np[q] + kTailHalo) * t.plane[q];
    }
    t.tab_ints = (int)t.table.size();
    t.tab_off = ((size_t)elems * esize + 15) & ~size_t(15);
    t.dense_off = (t.tab_off + sizeof(int) * t.tab_ints + 15) & ~size_t(15);
    t.bytes = t.dense_off + sizeof(double) * ((size_t)nbottom * nbottom + 2 * (size_t)nbottom);
    if (t.bytes > kTailBytes) return false;
    *out = t;
    return true;
}

template <typename T>
int nodal_tail(const NodalTail<T>& a, size_t bytes, cudaStream_t st)
{
    return a.g[0].iso ? launch_tail(k_nodal_tail<T, true>, a, bytes, st) : launch_tail(k_nodal_tail<T, false>, a, bytes, st);
}
template <typename T>
int mac_tail(const MacTail<T>& a, size_t bytes, cudaStream_t st)
{
    return launch_tail(k_mac_tail<T>, a, bytes, st);
}
template int nodal_tail<float>(const NodalTail<float>&, size_t, cudaStream_t);
template int nodal_tail<double>(const NodalTail<double>&, size_t, cudaStream_t);
template int mac_tail<float>(const MacTail<float>&, size_t, cudaStream_t);

}  // namespace gbp

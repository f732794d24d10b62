// BF16 3x3x3 convolutions of the warm-start U-Net as implicit GEMMs on tcgen05.
//
// Forward / data-gradient kernel (k_conv): a row of the GEMM is a group of G consecutive voxels of the zero-haloed
// channels-last grid (G = 4 for 16 channels, 2 for 32: a row of 64 elements, 128 bytes), because a TMA box costs about 8
// cycles per row however short the row is: with 32-byte rows the 16-channel convolutions at 128^3 ran at 13 k cycles per
// 128 voxels, 728 us, all of it TMA rows. The G output voxels of a group take G N accumulator columns. A persistent CTA
// walks output tiles of 128 groups. For each K step (input tensor, up to 64 channels, (dz, dy) of the taps) warp 0 issues
// the TMA loads of the groups' 130-row activation boxes (K-major, swizzled A operands; rows outside the array read as
// zeros); the weights lie in shared memory for the whole kernel where they fit, else they come with each step. Warp 1
// issues the MMAs, all of G N columns (one shape and accumulator, whose MMAs run in order): input voxel vi of the group
// feeds the output voxels vi - 1 to vi + 1, so its B operand is the stack of the three dx taps' weights at the rows of
// those voxels, with rows of zeros above and below; moving the start in one stack padded by zeros serves every vi. The
// group's last (first) voxel also feeds the first (last) output voxel of the next (previous) row: the box shifted by a
// row. (A value that is not finite so reaches the other voxels of the groups next to it as well.) Two FP32 accumulators
// in tensor memory: the epilogue of tile t overlaps the MMAs of tile t + 1.
// Warps 2..5 read the accumulator with tcgen05.ld (one group per thread), apply bias + GELU (forward) or gradient
// accumulation + GELU derivative (backward), zero the halo rows and store BF16.
//
// Weight-gradient kernel (k_wgrad): dw[tap][co][ci] = sum_p gout[p][co] in[p + off(tap)][ci] is a GEMM
// with M = (taps x input channels) in blocks of 128, N = output channels and K = grid rows. Both
// operands arrive MN-major (channels contiguous) straight from the activation arrays by TMA; each CTA
// reduces one slice of rows in tensor memory and adds its FP32 partial into dw.
//
// Every mbarrier wait is bounded; a wait that runs out sets the error word, stops the CTA's loops,
// drains the copies and MMAs it issued and frees its tensor memory.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <string>

#include "gbp_internal.cuh"
#include "nn.h"
#include "nn_tc.cuh"
#include "nodal_sweep.h"
#include "tma.cuh"

namespace gbp {
namespace nn {

namespace {

constexpr int kBM = 128;       // output rows per tile (MMA M)
constexpr int kThreads = 192;  // warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 epilogue
constexpr int kMaxStages = 32;
constexpr int kMostVoxels = 6;  // G + 2 input voxels feed a group
constexpr int kWgradRows = 64;  // K rows per pipeline stage of the weight-gradient kernel

struct ConvParams {
    CUtensorMap amap[2][2];  // per input: groups that start at voxel 0, at voxel `residue`
    CUtensorMap wmap[2];
    int nin, ntaps, N, ntiles, G;
    // per input: channels, channels of a K step, elements of a box row (voxels per box times those), boxes of a step
    int cin[2], cb[2], ab[2], nbox[2], wc0[2];
    // (dz, dy) of the taps: 9 of 3 taps (dx) each, or one of one; first box row relative to the tile's first group, and map
    int vsh[2];  // log2 of the voxels per box
    int ngroups, gtaps, a_rows, flip, wbox;  // wbox: taps per weight box (1, or all that lie in order)
    int grow[9], gmap[9];
    int X, Y, Z;
    long long PX, PXY, R;
    int nseg, flags;
    __nv_bfloat16* out[2];
    __nv_bfloat16* aux[2];
    int seg_c0[2], seg_nc[2];
    const float* bias;
    unsigned* err;
    int ns, wres;
    // weights of one (input, channel chunk, (dz, dy)): (G - 1) N rows of zeros, the taps' rows; zeros again at the end.
    // Resident: start, offset of an input, bytes of a channel chunk, bytes loaded, all bytes (else w_in: within a stage)
    uint32_t w_base, w_in[2], w_chunk[2], w_bytes, w_area;
    uint32_t box_bytes, a_bytes, stage_bytes, tmem_cols, idesc;
};

__device__ __forceinline__ void unpack16(const uint4 (&u)[2], float (&v)[16])
{
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[0]);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float2 f = __bfloat1622float2(h[q]);
        v[2 * q] = f.x;
        v[2 * q + 1] = f.y;
    }
}

__device__ __forceinline__ void pack16(const float (&v)[16], uint4 (&u)[2])
{
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u[0]);
#pragma unroll
    for (int q = 0; q < 8; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
}

__device__ __forceinline__ void load16(const __nv_bfloat16* p, float (&v)[16])
{
    uint4 u[2];
    u[0] = *reinterpret_cast<const uint4*>(p);
    u[1] = *reinterpret_cast<const uint4*>(p + 8);
    unpack16(u, v);
}

__device__ __forceinline__ void store16(__nv_bfloat16* p, const float (&v)[16])
{
    uint4 u[2];
    pack16(v, u);
    *reinterpret_cast<uint4*>(p) = u[0];
    *reinterpret_cast<uint4*>(p + 8) = u[1];
}

__device__ __forceinline__ uint32_t aligned_smem_base(unsigned char* raw)
{
    return (smem_u32(raw) + 1023u) & ~1023u;
}

__global__ void __launch_bounds__(kThreads, 1) k_conv(const __grid_constant__ ConvParams P)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], accf[2], acce[2], done, wfull;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;

    // (uniform by construction, so that the issue loops' values live in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t sbase = aligned_smem_base(smem_raw);
    unsigned char* sgen = smem_raw + (sbase - smem_u32(smem_raw));
    const int mid = P.ntaps > 1 ? 1 : 0;                 // box row of the tile's first group
    const uint32_t pad = (uint32_t)(P.G - 1);            // zero blocks of N rows before a weight stack
    const uint32_t per = (uint32_t)P.gtaps + pad;        // blocks from one stack to the next

    if (threadIdx.x == 0) {
        for (int s = 0; s < P.ns; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&accf[b], 1);
            mbar_init(&acce[b], 4);
        }
        mbar_init(&done, 1);
        mbar_init(&wfull, 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(&tmem_slot, 2 * P.tmem_cols);
        tc::tmem_relinquish();
    }
    if (P.G > 1) {
        // the zero rows of the weight stacks (the loads fill in the rest)
        const uint4 zero = make_uint4(0, 0, 0, 0);
        const uint32_t from = P.wres ? P.w_base : P.a_bytes, area = P.wres ? P.w_area : P.stage_bytes - P.a_bytes;
        for (int s = 0; s < (P.wres ? 1 : P.ns); ++s)
            for (uint32_t q = threadIdx.x * 16u; q < area; q += kThreads * 16u)
                *reinterpret_cast<uint4*>(sgen + s * P.stage_bytes + from + q) = zero;
        fence_proxy_async();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    if (warp == 0) {
        // the taps of a (dz, dy) in the order of the output voxels they feed: vi - 1, vi, vi + 1 (one voxel: as they lie)
        auto load_taps = [&](unsigned char* w, uint64_t* bar, int i, int cc, int gq) {
            const int x = P.wc0[i] + cc * P.cb[i], row0 = gq * P.gtaps * P.N;
            if (P.wbox > 1 || P.gtaps == 1) {
                tma_load_2d(w, &P.wmap[i], bar, x, row0);
                return;
            }
            for (int t = 0; t < P.gtaps; ++t) {
                const int q = P.flip || P.G == 1 ? t : P.gtaps - 1 - t;
                tma_load_2d(w + (uint32_t)(t * P.N) * P.cb[i] * 2u, &P.wmap[i], bar, x, row0 + q * P.N);
            }
        };
        if (P.wres && tc::elect_one()) {
            mbar_arrive_expect_tx(&wfull, P.w_bytes);
            for (int i = 0; i < P.nin; ++i)
                for (int cc = 0; cc < P.cin[i] / P.cb[i]; ++cc)
                    for (int gq = 0; gq < P.ngroups; ++gq)
                        load_taps(sgen + P.w_base + P.w_in[i] + cc * P.w_chunk[i] +
                                      (gq * per + pad) * (uint32_t)P.N * P.cb[i] * 2u,
                                  &wfull, i, cc, gq);
        }
        __syncwarp();
        uint32_t it = 0, s = 0, phase = 1;  // stage of the step, parity of its last release
        for (int tile = blockIdx.x; tile < P.ntiles && __all_sync(0xffffffffu, !abort_flag); tile += gridDim.x) {
            const int p0 = tile * kBM;
            for (int i = 0; i < P.nin; ++i) {
                const int nbox = P.nbox[i], ncc = P.cin[i] / P.cb[i], xstep = (P.ab[i] / P.cb[i]) * P.cin[i];
                const uint32_t bytes = (uint32_t)(nbox * P.a_rows * P.ab[i]) * 2u +
                                       (P.wres ? 0u : (uint32_t)(P.gtaps * P.N) * P.cb[i] * 2u);
                const uint32_t w_at = P.a_bytes + P.w_in[i] + pad * (uint32_t)P.N * P.cb[i] * 2u;
                for (int cc = 0; cc < ncc; ++cc)
                    for (int gq = 0; gq < P.ngroups; ++gq) {
                        if (it >= (uint32_t)P.ns && !tc::warp_wait(&empty[s], phase, P.err)) {
                            abort_flag = 1;
                            goto produced;
                        }
                        if (tc::elect_one()) {
                            mbar_arrive_expect_tx(&full[s], bytes);
                            unsigned char* a = sgen + s * P.stage_bytes;
                            const int arow = p0 + P.grow[gq];
                            const CUtensorMap* map = &P.amap[i][P.gmap[gq]];
                            for (int m = 0; m < nbox; ++m)
                                tma_load_2d(a + m * P.box_bytes, map, &full[s], m * xstep + cc * P.cb[i], arow);
                            if (!P.wres) load_taps(a + w_at, &full[s], i, cc, gq);
                        }
                        __syncwarp();
                        ++it;
                        if (++s == (uint32_t)P.ns) {
                            s = 0;
                            phase ^= 1u;
                        }
                    }
            }
        }
    produced:
        // drain: the last load into each stage must have landed before the CTA exits
        for (uint32_t q = 0; q < (uint32_t)P.ns && q < it; ++q) {
            const uint32_t last = it - 1 - ((it - 1 - q) % P.ns);
            (void)tc::warp_wait(&full[q], (last / P.ns) & 1, P.err);
        }
        if (P.wres) (void)tc::warp_wait(&wfull, 0, P.err);
    } else if (warp == 1) {
        uint32_t s = 0, phase = 0, tl = 0;
        if (P.wres && !tc::warp_wait(&wfull, 0, P.err)) abort_flag = 1;
        const int G = P.G;
        for (int tile = blockIdx.x; tile < P.ntiles && __all_sync(0xffffffffu, !abort_flag); tile += gridDim.x, ++tl) {
            const uint32_t buf = tl & 1;
            if (tl >= 2 && !tc::warp_wait(&acce[buf], ((tl >> 1) + 1) & 1, P.err)) {
                abort_flag = 1;
                break;
            }
            tc::fence_after_sync();
            const uint32_t d = tmem + buf * P.tmem_cols;
            uint32_t acc = 0;
            for (int i = 0; i < P.nin; ++i) {
                // descriptors: the addresses (16-byte units) are added to the low words
                const uint32_t rowa = P.ab[i] * 2u, roww = P.cb[i] * 2u, blk = ((uint32_t)P.N * roww) >> 4;
                const uint64_t da = tc::sdesc(0, 16, 8 * rowa, tc::swizzle_code((int)rowa));
                const uint64_t dw = tc::sdesc(0, 16, 8 * roww, tc::swizzle_code((int)roww));
                const int ks = P.cb[i] / 16, ncc = P.cin[i] / P.cb[i], vsh = P.vsh[i], vmask = (1 << vsh) - 1;
                // Input voxels -mid .. G - 1 + mid of the group, in the order of the taps: every output voxel sums its taps in
                // the same order whatever G is (the others add zeros), so the sums do not depend on it
                const int nvox = G + 2 * mid;
                uint32_t ao[kMostVoxels], wo[kMostVoxels];
#pragma unroll
                for (int n = 0; n < kMostVoxels; ++n) {
                    const int vi = P.flip ? G - 1 + mid - n : n - mid;
                    const int slot = vi < 0 ? G - 1 : (vi == G ? 0 : vi), r = vi < 0 ? 0 : (vi == G ? 2 : mid);
                    // (G = 1 keeps the taps in the order in which they lie)
                    const int t0 = (int)pad + (G == 1 && !P.flip ? vi + mid : mid - vi);
                    ao[n] = ((uint32_t)(slot >> vsh) * P.box_bytes + (uint32_t)r * rowa + (uint32_t)(slot & vmask) * roww) >> 4;
                    wo[n] = n < nvox ? (uint32_t)t0 * blk : 0;
                }
                for (int cc = 0; cc < ncc; ++cc) {
                    uint32_t wr = (sbase + P.w_base + P.w_in[i] + cc * P.w_chunk[i]) >> 4;
                    for (int gq = 0; gq < P.ngroups; ++gq) {
                        if (!tc::warp_wait(&full[s], phase, P.err)) {
                            abort_flag = 1;
                            goto issued;
                        }
                        tc::fence_after_sync();
                        const uint32_t a = sbase + s * P.stage_bytes;
                        const uint32_t w = P.wres ? wr : (a + P.a_bytes + P.w_in[i]) >> 4;
                        wr += per * blk;
                        const uint64_t ad = da + (a >> 4), wd = dw + w;
#pragma unroll
                        for (int n = 0; n < kMostVoxels; ++n) {
                            if (n >= nvox) break;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                if (kk >= ks) break;
                                tc::mma_bf16(d, ad + (ao[n] + 2u * kk), wd + (wo[n] + 2u * kk), P.idesc, acc);
                                acc = 1;
                            }
                        }
                        tc::mma_commit(&empty[s]);
                        if (++s == (uint32_t)P.ns) {
                            s = 0;
                            phase ^= 1u;
                        }
                    }
                }
            }
            tc::mma_commit(&accf[buf]);
        }
    issued:
        tc::mma_commit(&done);
        (void)tc::warp_wait(&done, 0, P.err);
    } else {
        const int q = warp & 3;  // tensor-memory lane quarter this warp may read
        const int row = q * 32 + lane;
        uint32_t tl = 0;
        for (int tile = blockIdx.x; tile < P.ntiles; tile += gridDim.x, ++tl) {
            const uint32_t buf = tl & 1;
            if (!mbar_wait_bounded(&accf[buf], (tl >> 1) & 1, P.err)) abort_flag = 1;
            if (__any_sync(0xffffffffu, abort_flag)) break;
            tc::fence_after_sync();
            const long long pg = ((long long)tile * kBM + row) * P.G;
            const bool valid = pg < P.R;  // (R is a multiple of G, below 2^30)
            const unsigned up = (unsigned)pg, pxy = (unsigned)P.PXY, px = (unsigned)P.PX;
            int z = (int)(up / pxy), y = (int)((up - z * pxy) / px), x = (int)(up - z * pxy - y * px);
            const uint32_t taddr = tmem + buf * P.tmem_cols + ((uint32_t)(q * 32) << 16);
            for (int vo = 0; vo < P.G; ++vo) {
                const long long p = pg + vo;
                const bool inside = x >= 1 && x <= P.X && y >= 1 && y <= P.Y && z >= 1 && z <= P.Z;
                if (++x == (int)px) {
                    x = 0;
                    if (++y == (int)(pxy / px)) {
                        y = 0;
                        ++z;
                    }
                }
                for (int sg = 0; sg < P.nseg; ++sg) {
                    const int nc = P.seg_nc[sg], c0 = P.seg_c0[sg];
                    __nv_bfloat16* orow = P.out[sg] + p * nc;
                    __nv_bfloat16* arow = P.aux[sg] ? P.aux[sg] + p * nc : nullptr;
                    for (int c = 0; c < nc; c += 16) {
                        float v[16];
                        tc::tmem_ld16(taddr + (uint32_t)(vo * P.N + c0 + c), v);
                        if (!valid) continue;
                        if (!inside) {
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] = 0.f;
                            store16(orow + c, v);
                            if (arow && (P.flags & kGelu)) store16(arow + c, v);
                            continue;
                        }
                        if (P.bias) {
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] += __ldg(P.bias + c0 + c + e);
                        }
                        if (P.flags & kAccum) {
                            float o[16];
                            load16(orow + c, o);
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] += o[e];
                        }
                        if (P.flags & kDGelu) {
                            float a[16];
                            load16(arow + c, a);
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] *= dgelu_f(a[e]);
                        }
                        if (P.flags & kGelu) {
                            if (arow) store16(arow + c, v);
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] = gelu_f(v[e]);
                        }
                        store16(orow + c, v);
                    }
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acce[buf]);
        }
    }

    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, 2 * P.tmem_cols);
    }
}

// ------------------------------------------------------------------ weight gradient
struct WgradParams {
    CUtensorMap amap;  // input activations, box {ca, kWgradRows}
    CUtensorMap gmap;  // output gradient, box {cg, kWgradRows}
    int ca, natom_a;   // channels per A atom (<= 64); atoms per 128-row M tile
    int cg, natom_g;   // channels per B atom; atoms (N = natom_g * cg = cout)
    int cin, ci0, cin_tot, cout, ntaps;
    int off[27];
    int k_steps_per_cta, k_steps_total;
    float* dw;
    unsigned* err;
    int ns;
    uint32_t a_bytes, stage_bytes, tmem_cols, idesc;
};

__global__ void __launch_bounds__(kThreads, 1) k_wgrad(const __grid_constant__ WgradParams P)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], accf;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ int2 atab[8];  // the A atoms of a K step: first channel, row offset

    // (uniform by construction, so that the issue loops' values live in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t sbase = aligned_smem_base(smem_raw);
    unsigned char* sgen = smem_raw + (sbase - smem_u32(smem_raw));
    const int mt = blockIdx.x;  // M tile: taps [mt * taps_per_tile, ...)
    const int taps_per_tile = kBM / P.cin >= 1 ? kBM / P.cin : 1;
    const int k_begin = blockIdx.y * P.k_steps_per_cta;
    const int k_end = min(P.k_steps_total, k_begin + P.k_steps_per_cta);

    if ((int)threadIdx.x < P.natom_a) {
        const int m = threadIdx.x, chunks = P.cin / P.ca, tap = mt * taps_per_tile + m / chunks;
        // taps past the last one load a valid tap (their rows of D are never stored)
        atab[m] = make_int2(m % chunks * P.ca, P.off[tap < P.ntaps ? tap : P.ntaps - 1]);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.ns; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&accf, 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(&tmem_slot, P.tmem_cols);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t a_atom_bytes = (uint32_t)kWgradRows * P.ca * 2u;
    const uint32_t g_atom_bytes = (uint32_t)kWgradRows * P.cg * 2u;

    if (warp == 0) {
        uint32_t it = 0, s = 0, phase = 1;  // stage of the step, parity of its last release
        const uint32_t bytes = a_atom_bytes * P.natom_a + g_atom_bytes * P.natom_g;
        for (int ks = k_begin; ks < k_end; ++ks, ++it) {
            if (it >= (uint32_t)P.ns && !tc::warp_wait(&empty[s], phase, P.err)) {
                abort_flag = 1;
                break;
            }
            if (tc::elect_one()) {
                const int q0 = ks * kWgradRows;
                mbar_arrive_expect_tx(&full[s], bytes);
                unsigned char* a = sgen + s * P.stage_bytes;
                const int natom_a = P.natom_a, natom_g = P.natom_g;
#pragma unroll 4
                for (int m = 0; m < natom_a; ++m) {
                    const int2 t = atab[m];
                    tma_load_2d(a + m * a_atom_bytes, &P.amap, &full[s], t.x, q0 + t.y);
                }
                a += P.a_bytes;
                for (int m = 0; m < natom_g; ++m) tma_load_2d(a + m * g_atom_bytes, &P.gmap, &full[s], m * P.cg, q0);
            }
            __syncwarp();
            if (++s == (uint32_t)P.ns) {
                s = 0;
                phase ^= 1u;
            }
        }
        for (uint32_t q = 0; q < (uint32_t)P.ns && q < it; ++q) {
            const uint32_t last = it - 1 - ((it - 1 - q) % P.ns);
            (void)tc::warp_wait(&full[q], (last / P.ns) & 1, P.err);
        }
    } else if (warp == 1) {
        // MN-major swizzled operands: MN atoms at LBO = atom bytes, 8-row K groups at SBO
        const uint64_t da = tc::sdesc(0, a_atom_bytes, 8u * P.ca * 2u, tc::swizzle_code(P.ca * 2));
        const uint64_t dg = tc::sdesc(0, g_atom_bytes, 8u * P.cg * 2u, tc::swizzle_code(P.cg * 2));
        const uint32_t stepa = 16u * P.ca * 2u >> 4, stepg = 16u * P.cg * 2u >> 4;
        uint32_t s = 0, phase = 0, acc = 0;
        for (int ks = k_begin; ks < k_end; ++ks) {
            if (!tc::warp_wait(&full[s], phase, P.err)) {
                abort_flag = 1;
                break;
            }
            tc::fence_after_sync();
            const uint32_t a = sbase + s * P.stage_bytes;
            uint64_t ad = da + (a >> 4), bd = dg + ((a + P.a_bytes) >> 4);
#pragma unroll
            for (int kk = 0; kk < kWgradRows / 16; ++kk) {
                tc::mma_bf16(tmem, ad, bd, P.idesc, acc);
                acc = 1;
                ad += stepa;
                bd += stepg;
            }
            tc::mma_commit(&empty[s]);
            if (++s == (uint32_t)P.ns) {
                s = 0;
                phase ^= 1u;
            }
        }
        tc::mma_commit(&accf);
    } else {
        const int q = warp & 3;
        const int row = q * 32 + lane;  // M row = (tap in tile, input channel)
        const bool ok = mbar_wait_bounded(&accf, 0, P.err);
        tc::fence_after_sync();
        const int tap = mt * taps_per_tile + row / P.cin;
        const int ci = row % P.cin;
        const bool store = ok && !abort_flag && k_end > k_begin && tap < P.ntaps && row < taps_per_tile * P.cin;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
        for (int c = 0; c < P.cout; c += 16) {
            float v[16];
            tc::tmem_ld16(taddr + (uint32_t)c, v);
            if (!store) continue;
            float* dst = P.dw + ((long long)tap * P.cout + c) * P.cin_tot + P.ci0 + ci;
#pragma unroll
            for (int e = 0; e < 16; ++e) atomicAdd(dst + (long long)e * P.cin_tot, v[e]);
        }
    }

    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, P.tmem_cols);
    }
}

// ------------------------------------------------------------------ host side
int encode_rows(const void* base, int C, long long R, int box_c, int box_rows, CUtensorMap* m)
{
    auto fn = tensor_map_encoder();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is unavailable from the driver");
        return GBP_CUDA_ERROR;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)C, (cuuint64_t)R};
    const cuuint64_t strides[1] = {(cuuint64_t)C * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_c, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUtensorMapSwizzle swz = box_c == 64   ? CU_TENSOR_MAP_SWIZZLE_128B
                                   : box_c == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                 : CU_TENSOR_MAP_SWIZZLE_32B;
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed for a BF16 activation map (code " + std::to_string((int)r) + ")");
        return GBP_CUDA_ERROR;
    }
    return GBP_OK;
}

int chunk_of(int c) { return c >= 64 ? 64 : c; }

bool channels_ok(int c) { return c == 16 || c == 32 || (c >= 64 && c % 64 == 0); }

uint32_t pow2_cols(int n)
{
    uint32_t c = 32;
    while (c < (uint32_t)n) c <<= 1;
    return c;
}

void tap_offsets(const Grid3& g, int ntaps, int flip, int* off)
{
    if (ntaps == 1) {
        off[0] = 0;
        return;
    }
    int t = 0;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx, ++t) {
                const long long o = dz * g.PXY + dy * g.PX + dx;
                off[t] = (int)(flip ? -o : o);
            }
}

}  // namespace

int conv3d(const ConvLaunch& L, cudaStream_t st)
{
    if (L.nin < 1 || L.nin > 2 || (L.ntaps != 1 && L.ntaps != 27) || L.N < 16 || L.N > 256 || L.N % 16 ||
        L.nseg < 1 || L.nseg > 2 || !L.w || L.g.R <= 0 || L.g.R > (1ll << 30)) {
        set_error("conv3d: bad launch shape");
        return GBP_BAD_ARG;
    }
    ConvParams P;
    memset(&P, 0, sizeof(P));
    int cin_tot = 0, cmin = 64;
    for (int i = 0; i < L.nin; ++i) {
        if (!L.in[i] || !channels_ok(L.cin[i]) || (reinterpret_cast<uintptr_t>(L.in[i]) & 15)) {
            set_error("conv3d: input channels must be 16, 32 or a multiple of 64, data 16-byte aligned");
            return GBP_BAD_ARG;
        }
        P.cin[i] = L.cin[i];
        P.cb[i] = chunk_of(L.cin[i]);
        P.wc0[i] = cin_tot;
        cin_tot += L.cin[i];
        cmin = std::min(cmin, P.cb[i]);
    }
    int segsum = 0;
    for (int s = 0; s < L.nseg; ++s) {
        if (!L.out[s] || L.seg_c[s] < 16 || L.seg_c[s] % 16 || (reinterpret_cast<uintptr_t>(L.out[s]) & 15) ||
            (reinterpret_cast<uintptr_t>(L.aux[s]) & 15) || (!L.aux[s] && (L.flags & kDGelu))) {
            set_error("conv3d: bad output segment");
            return GBP_BAD_ARG;
        }
        P.out[s] = L.out[s];
        P.aux[s] = L.aux[s];
        P.seg_c0[s] = segsum;
        P.seg_nc[s] = L.seg_c[s];
        segsum += L.seg_c[s];
    }
    if (segsum != L.N) {
        set_error("conv3d: output segments must cover N channels");
        return GBP_BAD_ARG;
    }
    P.nin = L.nin;
    P.ntaps = L.ntaps;
    P.N = L.N;
    P.flip = L.flip;
    P.ngroups = L.ntaps == 27 ? 9 : 1;
    P.gtaps = L.ntaps == 27 ? 3 : 1;
    P.a_rows = L.ntaps == 27 ? kBM + 2 : kBM;
    int off[27];
    tap_offsets(L.g, L.ntaps, L.flip, off);
    // voxels per GEMM row: rows of 64 elements (128 bytes) for the narrowest input, where the grid splits into such groups,
    // the (dz, dy) offsets fall on at most two positions within a group and the columns stay within an MMA's 256 (twice
    // that is the tensor memory)
    int residue = 0;
    for (P.G = 64 / cmin;; P.G >>= 1) {
        bool ok = L.g.R % P.G == 0 && P.G * L.N <= 256;
        residue = 0;
        for (int gq = 0; gq < P.ngroups; ++gq) {
            const int c = L.ntaps == 27 ? off[3 * gq + 1] : 0, r = ((c % P.G) + P.G) % P.G;
            if (r && residue && r != residue) ok = false;
            if (r) residue = r;
            P.gmap[gq] = r ? 1 : 0;
            P.grow[gq] = (c - r) / P.G - (L.ntaps == 27 ? 1 : 0);
        }
        if (ok || P.G == 1) break;
    }
    P.ntiles = (int)((L.g.R / P.G + kBM - 1) / kBM);
    P.wbox = (P.flip || P.G == 1) && P.gtaps * L.N <= 256 ? P.gtaps : 1;
    uint32_t wres_bytes = 0;
    int abmax = 16, nbmax = 1;
    for (int i = 0; i < L.nin; ++i) {
        P.ab[i] = std::min(64, P.G * P.cb[i]);
        P.nbox[i] = P.G * P.cb[i] / P.ab[i];
        for (P.vsh[i] = 0; P.cb[i] << P.vsh[i] < P.ab[i]; ++P.vsh[i]) {
        }
        abmax = std::max(abmax, P.ab[i]);
        nbmax = std::max(nbmax, P.nbox[i]);
        for (int m = 0; m < 2; ++m) {
            const int r = m ? residue : 0;
            const int rc = encode_rows(L.in[i] + (size_t)r * L.cin[i], P.G * L.cin[i], (L.g.R - r) / P.G, P.ab[i], P.a_rows,
                                       &P.amap[i][m]);
            if (rc) return rc;
        }
        const int rc = encode_rows(L.w, cin_tot, (long long)L.ntaps * L.N, P.cb[i], P.wbox * L.N, &P.wmap[i]);
        if (rc) return rc;
        P.w_in[i] = wres_bytes;
        P.w_chunk[i] = ((uint32_t)((P.gtaps + P.G - 1) * P.ngroups + P.G - 1) * L.N * P.cb[i] * 2u + 1023u) & ~1023u;
        wres_bytes += P.w_chunk[i] * (L.cin[i] / P.cb[i]);
        P.w_bytes += (uint32_t)L.ntaps * L.N * L.cin[i] * 2u;
    }
    P.X = L.g.X;
    P.Y = L.g.Y;
    P.Z = L.g.Z;
    P.PX = L.g.PX;
    P.PXY = L.g.PXY;
    P.R = L.g.R;
    P.nseg = L.nseg;
    P.flags = L.flags;
    P.bias = L.bias;
    P.err = L.err;
    P.box_bytes = ((uint32_t)P.a_rows * abmax * 2u + 1023u) & ~1023u;
    P.a_bytes = nbmax * P.box_bytes;
    P.tmem_cols = pow2_cols(P.G * L.N);
    P.idesc = tc::idesc_bf16(kBM, P.G * L.N, 0, 0);
    P.w_area = wres_bytes;
    // weights resident where at least 3 activation stages fit beside them, else with each step
    const uint32_t max_smem = 220 * 1024;
    P.wres = wres_bytes + 3 * P.a_bytes + 1024 <= max_smem;
    P.stage_bytes = P.a_bytes;
    if (!P.wres) {
        uint32_t w = 0;
        for (int i = 0; i < L.nin; ++i) {
            const uint32_t stack = ((uint32_t)((P.gtaps + 2 * (P.G - 1)) * L.N) * P.cb[i] * 2u + 1023u) & ~1023u;
            P.w_in[i] = P.G > 1 ? w : 0;  // (each input's zero rows stay where they are)
            w = P.G > 1 ? w + stack : std::max(w, stack);
        }
        P.stage_bytes += w;
    }
    P.ns = std::min(kMaxStages, (int)((max_smem - 1024 - (P.wres ? wres_bytes : 0)) / P.stage_bytes));
    if (P.ns < 2) {
        set_error("conv3d: stage does not fit in shared memory");
        return GBP_BAD_ARG;
    }
    P.w_base = (uint32_t)P.ns * P.stage_bytes;
    const size_t smem = (size_t)P.w_base + (P.wres ? wres_bytes : 0) + 1024;
    static bool attr_set = false;
    if (!attr_set) {
        GBP_CUDA(cudaFuncSetAttribute(k_conv, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
        attr_set = true;
    }
    const int grid = std::min(P.ntiles, sm_count_cached());
    k_conv<<<grid, kThreads, smem, st>>>(P);
    GBP_CUDA(cudaGetLastError());
    return GBP_OK;
}

int conv3d_wgrad(const WgradLaunch& L, cudaStream_t st)
{
    if (!L.in || !L.gout || !L.dw || (L.ntaps != 1 && L.ntaps != 27) || !channels_ok(L.cin) || L.cin > 128 ||
        !channels_ok(L.cout) || L.cout > 128 || L.ci0 < 0 || L.ci0 + L.cin > L.cin_tot || L.g.R <= 0 ||
        L.g.R > (1ll << 30)) {
        set_error("conv3d_wgrad: bad launch shape");
        return GBP_BAD_ARG;
    }
    WgradParams P;
    memset(&P, 0, sizeof(P));
    P.ca = chunk_of(L.cin);
    P.cg = chunk_of(L.cout);
    const int taps_per_tile = std::max(1, 128 / L.cin);
    P.natom_a = taps_per_tile * L.cin / P.ca;  // = 128 / ca
    P.natom_g = L.cout / P.cg;
    int rc = encode_rows(L.in, L.cin, L.g.R, P.ca, kWgradRows, &P.amap);
    if (!rc) rc = encode_rows(L.gout, L.cout, L.g.R, P.cg, kWgradRows, &P.gmap);
    if (rc) return rc;
    P.cin = L.cin;
    P.ci0 = L.ci0;
    P.cin_tot = L.cin_tot;
    P.cout = L.cout;
    P.ntaps = L.ntaps;
    tap_offsets(L.g, L.ntaps, 0, P.off);
    P.dw = L.dw;
    P.err = L.err;
    P.a_bytes = (uint32_t)kWgradRows * 128u * 2u;
    P.stage_bytes = P.a_bytes + (uint32_t)kWgradRows * L.cout * 2u;
    P.stage_bytes = (P.stage_bytes + 1023u) & ~1023u;
    P.tmem_cols = pow2_cols(L.cout);
    P.idesc = tc::idesc_bf16(kBM, L.cout, 1, 1);
    P.ns = std::min(kMaxStages, (int)((200 * 1024 - 1024) / P.stage_bytes));
    const int mtiles = (L.ntaps + taps_per_tile - 1) / taps_per_tile;
    P.k_steps_total = (int)((L.g.R + kWgradRows - 1) / kWgradRows);
    const int want = std::max(1, 2 * sm_count_cached() / mtiles);
    P.k_steps_per_cta = std::max(8, (P.k_steps_total + want - 1) / want);
    const int splits = (P.k_steps_total + P.k_steps_per_cta - 1) / P.k_steps_per_cta;
    static bool attr_set = false;
    if (!attr_set) {
        GBP_CUDA(cudaFuncSetAttribute(k_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_set = true;
    }
    const size_t smem = (size_t)P.ns * P.stage_bytes + 1024;
    k_wgrad<<<dim3(mtiles, splits), kThreads, smem, st>>>(P);
    GBP_CUDA(cudaGetLastError());
    return GBP_OK;
}

}  // namespace nn
}  // namespace gbp

// BF16 3x3x3 convolutions of the warm-start U-Net as implicit GEMMs on tcgen05.
//
// Forward / data-gradient kernel (k_conv): a row of the GEMM is a group of G consecutive voxels of the zero-haloed
// channels-last grid (G = 4 for 16 channels, 2 for 32: a row of 64 elements, 128 bytes). With a voxel per row the
// 16-channel convolutions at 128^3 took 728 us: 27 MMAs of 16 columns and 9 boxes of 32-byte rows per 128 voxels, every one
// of them some 400 cycles of scalar issue code. Now 81 us: 54 MMAs of 64 columns and 3 boxes per 512 voxels, at 150 cycles
// per MMA and issuing warp, which still bounds it (one issuer at 116 us: tensor pipe busy 21 %, DRAM 17 %). The G output
// voxels of a group take G N accumulator columns. A persistent CTA
// walks output tiles of 128 groups. For each K step (input tensor, up to 64 channels, (dz, dy) of the taps) warp 0 issues
// the TMA loads of the groups' 130-row activation boxes (K-major, swizzled A operands; rows outside the array read as
// zeros); the weights lie in shared memory for the whole kernel where they fit, else they come with each step. Warp 1
// issues the MMAs, all of G N columns (one shape and accumulator, whose MMAs run in order): input voxel vi of the group
// feeds the output voxels vi - 1 to vi + 1, so its B operand is the stack of the three dx taps' weights at the rows of
// those voxels, with rows of zeros above and below; moving the start in one stack padded by zeros serves every vi. The
// group's last (first) voxel also feeds the first (last) output voxel of the next (previous) row: the box shifted by a
// row. A value that is not finite meets those zeros too and spoils the sums of the other voxels of its group and of the groups
// next to it: the epilogue forms sums that are not finite once more, tap by tap (conv_at). Two FP32 accumulators
// (or four) in tensor memory: the epilogue of a tile overlaps the MMAs of the next. Two producer and issuer pairs take
// turns at the tiles where two rings of stages fit, since one warp's issue rate bounds a tile (116 us with one, 81 with two).
// The other warps read the accumulator with tcgen05.ld (one group per thread, 16 columns at a time), apply bias + GELU
// (forward) or gradient accumulation + GELU derivative (backward), zero the halo rows and store BF16.
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
constexpr int kThreads = 192;  // weight gradient: warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 epilogue
// convolution: four epilogue warps per lane quarter of tensor memory. The epilogue's chain (tensor-memory load, bias, GELU,
// two stores) bounded the level-0 convolutions with one: 4.6 k cycles per tile without a GELU, about 11 k with it.
constexpr int kEpiSets = 4, kConvThreads = 128 + 128 * kEpiSets;
constexpr int kMaxStages = 32;
constexpr int kConvSmem = 225 * 1024;  // of the 227 KB of a CTA, beside the convolution's static part (2 KB)
constexpr int kPairStages = kMaxStages / 2;  // stages of a producer / issuer pair of the convolution
constexpr int kWgradRows = 64;  // K rows per pipeline stage of the weight-gradient kernel

struct ConvParams {
    CUtensorMap amap[2];
    CUtensorMap wmap[2];
    int nin, ntaps, N, ntiles, G;
    // per input: channels, channels of a K step, elements of a box row (voxels per box times those), boxes of a step
    int cin[2], cb[2], ab[2], nbox[2], wc0[2];
    // (dz, dy) of the taps: 9 of 3 taps (dx) each, or one of one; first box row relative to the tile's first group, and map
    int vsh[2];  // log2 of the voxels per box
    // K steps of an input and channel chunk: nstep boxes of a_rows rows, the first at row grow[step] relative to the tile's
    // first group; a box holds the rows of ndy of the 9 (dz, dy), 3 taps (dx) each (a 1x1x1 convolution: one of one tap).
    // yoff[dy]: the voxel offset of a dy from the group, ybase: the one that box row 0 starts at or before (ndy = 1: per dy)
    int nstep, ndy, gtaps, a_rows, flip, wbox;  // wbox: taps per weight box (1, or all that lie in order)
    int grow[9], yoff[3], ybase[3];
    int X, Y, Z;
    long long PX, PXY, R;
    int nseg, flags;
    __nv_bfloat16* out[2];
    __nv_bfloat16* aux[2];
    int seg_c0[2], seg_nc[2];
    const float* bias;
    const __nv_bfloat16 *in[2], *w;  // as the caller gave them (conv_at)
    int cin_tot;
    unsigned* err;
    int ns, wres, npair, nbsh;  // stages of a pair, pairs (1 or 2), log2 of the accumulators (2 or 4)
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

// the MMAs of NV input voxels, KS slices of 16 channels each; vstep / wstep: descriptor steps (mod 2^32) from one to the next
template <int NV, int KS>
__device__ __forceinline__ void mma_voxels(uint32_t leader, uint32_t d, uint64_t ad, uint64_t wd, uint32_t vstep,
                                           uint32_t wstep, uint32_t idesc, uint32_t& acc)
{
#pragma unroll
    for (int n = 0; n < NV; ++n) {
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            tc::mma_bf16(leader, d, ad + 2u * kk, wd + 2u * kk, idesc, acc);
            acc = 1;
        }
        ad += (int32_t)vstep;
        wd += (int32_t)wstep;
    }
}

// The sum of output channel n at row p, from the arrays themselves
__device__ __noinline__ float conv_at(const ConvParams& P, long long p, int n)
{
    const int r = P.ntaps > 1 ? 1 : 0, sign = P.flip ? -1 : 1;
    float sum = 0.f;
    int t = 0;
    for (int dz = -r; dz <= r; ++dz)
        for (int dy = -r; dy <= r; ++dy)
            for (int dx = -r; dx <= r; ++dx, ++t) {
                const long long q = p + sign * (dz * P.PXY + dy * P.PX + dx);
                if (q < 0 || q >= P.R) continue;
                for (int i = 0; i < P.nin; ++i) {
                    const __nv_bfloat16* a = P.in[i] + q * P.cin[i];
                    const __nv_bfloat16* w = P.w + ((long long)t * P.N + n) * P.cin_tot + P.wc0[i];
                    for (int c = 0; c < P.cin[i]; ++c) sum = fmaf(__bfloat162float(a[c]), __bfloat162float(w[c]), sum);
                    if (sum != sum) return sum;  // NaN stays NaN
                }
            }
    return sum;
}

template <int G>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv(const __grid_constant__ ConvParams P)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_[2][kPairStages], empty_[2][kPairStages], accf[4], acce[4], done[2], wfull;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ __align__(16) float sbias[256];

    // (uniform by construction, so that the issue loops' values live in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t sbase = aligned_smem_base(smem_raw);
    unsigned char* sgen = smem_raw + (sbase - smem_u32(smem_raw));
    const int mid = P.ntaps > 1 ? 1 : 0;                 // box row of the tile's first group
    const uint32_t pad = (uint32_t)(G - 1);            // zero blocks of N rows before a weight stack
    const uint32_t per = (uint32_t)P.gtaps + pad;        // blocks from one stack to the next
    const int nstack = P.nstep * P.ndy;                  // stacks of a channel chunk: the (dz, dy)

    if (threadIdx.x == 0) {
        for (int s = 0; s < P.ns; ++s)
            for (int b = 0; b < 2; ++b) {
                mbar_init(&full_[b][s], 1);
                mbar_init(&empty_[b][s], 1);
            }
        for (int b = 0; b < 4; ++b) {
            mbar_init(&accf[b], 1);
            mbar_init(&acce[b], 4 * kEpiSets);
        }
        mbar_init(&done[0], 1);
        mbar_init(&done[1], 1);
        mbar_init(&wfull, 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(&tmem_slot, P.tmem_cols << P.nbsh);
        tc::tmem_relinquish();
    }
    if ((int)threadIdx.x < P.N) sbias[threadIdx.x] = P.bias ? P.bias[threadIdx.x] : 0.f;
    if (G > 1) {
        // the zero rows of the weight stacks (the loads fill in the rest)
        const uint4 zero = make_uint4(0, 0, 0, 0);
        const uint32_t from = P.wres ? P.w_base : P.a_bytes, area = P.wres ? P.w_area : P.stage_bytes - P.a_bytes;
        for (int s = 0; s < (P.wres ? 1 : P.npair * P.ns); ++s)
            for (uint32_t q = threadIdx.x * 16u; q < area; q += kConvThreads * 16u)
                *reinterpret_cast<uint4*>(sgen + s * P.stage_bytes + from + q) = zero;
        fence_proxy_async();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    // producer and issuer of pair p: warps 2 p and 2 p + 1; its tiles: every npair-th of the CTA's
    const int pair = warp >> 1 & 1;
    uint64_t *full = full_[pair], *empty = empty_[pair];
    const uint32_t ring = (uint32_t)(pair * P.ns) * P.stage_bytes;
    const int tstep = P.npair * (int)gridDim.x;
    if (warp < 4 && pair >= P.npair) {
        // no second pair where its stages do not fit
    } else if (warp < 4 && !(warp & 1)) {
        // the taps of a (dz, dy) in the order of the output voxels they feed: vi - 1, vi, vi + 1 (one voxel: as they lie)
        auto load_taps = [&](unsigned char* w, uint64_t* bar, int i, int cc, int gq) {
            const int x = P.wc0[i] + cc * P.cb[i], row0 = gq * P.gtaps * P.N;
            if (P.wbox > 1 || P.gtaps == 1) {
                tma_load_2d(w, &P.wmap[i], bar, x, row0);
                return;
            }
            for (int t = 0; t < P.gtaps; ++t) {
                const int q = P.flip || G == 1 ? t : P.gtaps - 1 - t;
                tma_load_2d(w + (uint32_t)(t * P.N) * P.cb[i] * 2u, &P.wmap[i], bar, x, row0 + q * P.N);
            }
        };
        if (P.wres && pair == 0 && tc::elect_one()) {
            mbar_arrive_expect_tx(&wfull, P.w_bytes);
            for (int i = 0; i < P.nin; ++i)
                for (int cc = 0; cc < P.cin[i] / P.cb[i]; ++cc)
                    for (int gq = 0; gq < nstack; ++gq)
                        load_taps(sgen + P.w_base + P.w_in[i] + cc * P.w_chunk[i] +
                                      (gq * per + pad) * (uint32_t)P.N * P.cb[i] * 2u,
                                  &wfull, i, cc, gq);
        }
        __syncwarp();
        uint32_t it = 0, s = 0, phase = 1;  // stage of the step, parity of its last release
        for (int tile = blockIdx.x + pair * gridDim.x; tile < P.ntiles && __all_sync(0xffffffffu, !abort_flag); tile += tstep) {
            const int p0 = tile * kBM;
            for (int i = 0; i < P.nin; ++i) {
                const int nbox = P.nbox[i], ncc = P.cin[i] / P.cb[i], xstep = (P.ab[i] / P.cb[i]) * P.cin[i];
                const uint32_t bytes = (uint32_t)(nbox * P.a_rows * P.ab[i]) * 2u +
                                       (P.wres ? 0u : (uint32_t)(P.gtaps * P.N) * P.cb[i] * 2u);
                const uint32_t w_at = P.a_bytes + P.w_in[i] + pad * (uint32_t)P.N * P.cb[i] * 2u;
                for (int cc = 0; cc < ncc; ++cc)
                    for (int gq = 0; gq < P.nstep; ++gq) {
                        if (it >= (uint32_t)P.ns && !tc::warp_wait(&empty[s], phase, P.err)) {
                            abort_flag = 1;
                            goto produced;
                        }
                        if (tc::elect_one()) {
                            mbar_arrive_expect_tx(&full[s], bytes);
                            unsigned char* a = sgen + ring + s * P.stage_bytes;
                            const int arow = p0 + P.grow[gq];
                            const CUtensorMap* map = &P.amap[i];
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
        if (P.wres && pair == 0) (void)tc::warp_wait(&wfull, 0, P.err);
    } else if (warp < 4) {
        uint32_t s = 0, phase = 0, tl = pair;
        const uint32_t leader = tc::elect_one();
        if (P.wres && !tc::warp_wait(&wfull, 0, P.err)) abort_flag = 1;
        for (int tile = blockIdx.x + pair * gridDim.x; tile < P.ntiles && __all_sync(0xffffffffu, !abort_flag);
             tile += tstep, tl += P.npair) {
            const uint32_t buf = tl & ((1u << P.nbsh) - 1u), use = tl >> P.nbsh;
            if (use > 0 && !tc::warp_wait(&acce[buf], (use + 1) & 1, P.err)) {
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
                const int ks = P.cb[i] / 16, ncc = P.cin[i] / P.cb[i];
                // first input voxel of a step's MMAs within the box, its step, and the same of the weight stacks. Every output
                // voxel sums its taps in their order whatever G is (the others add zeros), so the sums do not depend on it.
                // (G = 1 keeps the taps in the order in which they lie.)
                const int vfirst = P.flip ? G - 1 + mid : -mid;
                const uint32_t vstep = P.flip ? 0u - (roww >> 4) : roww >> 4, wstep = P.flip || G == 1 ? blk : 0u - blk;
                const uint32_t wfirst = P.flip || G == 1 ? 0u : (pad + 2u * mid) * blk;
                for (int cc = 0; cc < ncc; ++cc) {
                    uint32_t wr = (sbase + P.w_base + P.w_in[i] + cc * P.w_chunk[i]) >> 4;
                    for (int gq = 0, y1 = 0; gq < P.nstep; ++gq) {
                        if (!tc::warp_wait(&full[s], phase, P.err)) {
                            abort_flag = 1;
                            goto issued;
                        }
                        tc::fence_after_sync();
                        const uint32_t a = sbase + ring + s * P.stage_bytes;
                        for (int y = P.ndy == 1 ? y1 : 0, ye = P.ndy == 1 ? y1 + 1 : 3; y < ye; ++y) {
                            const int v0 = P.yoff[y] - P.ybase[y] + vfirst;
                            uint64_t wd = dw + ((P.wres ? wr : (a + P.a_bytes + P.w_in[i]) >> 4) + wfirst);
                            wr += per * blk;
                            if (P.nbox[i] == 1) {
                                // one box: its rows follow one another, voxel v at v * roww
                                uint64_t ad = da + ((a + (uint32_t)v0 * roww) >> 4);
                                if (mid) {
                                    if (ks == 4)
                                        mma_voxels<G + 2, 4>(leader, d, ad, wd, vstep, wstep, P.idesc, acc);
                                    else if (ks == 2)
                                        mma_voxels<G + 2, 2>(leader, d, ad, wd, vstep, wstep, P.idesc, acc);
                                    else
                                        mma_voxels<G + 2, 1>(leader, d, ad, wd, vstep, wstep, P.idesc, acc);
                                } else {
                                    for (int kk = 0; kk < ks; ++kk)
                                        mma_voxels<G, 1>(leader, d, ad + 2u * kk, wd + 2u * kk, vstep, wstep, P.idesc, acc);
                                }
                            } else {
                                // voxel v in row v / G, box (v % G) / (voxels per box)
                                const int vsh = P.vsh[i];
                                const uint32_t boxes = P.box_bytes >> 4, a16 = a >> 4, ra = rowa >> 4, rw = roww >> 4;
#pragma unroll
                                for (int n = 0; n < G + 2; ++n) {
                                    if (n >= G + 2 * mid) break;
                                    const int v = P.flip ? v0 - n : v0 + n, slot = v & (G - 1);
                                    const uint64_t ad = da + (a16 + (uint32_t)(slot >> vsh) * boxes + (uint32_t)(v / G) * ra +
                                                              (uint32_t)(slot & ((1 << vsh) - 1)) * rw);
#pragma unroll
                                    for (int kk = 0; kk < 4; ++kk) {
                                        if (kk >= ks) break;
                                        tc::mma_bf16(leader, d, ad + 2u * kk, wd + 2u * kk, P.idesc, acc);
                                        acc = 1;
                                    }
                                    wd += (int32_t)wstep;
                                }
                            }
                        }
                        if (P.gtaps > 1 && ++y1 == 3) y1 = 0;
                        tc::mma_commit(leader, &empty[s]);
                        if (++s == (uint32_t)P.ns) {
                            s = 0;
                            phase ^= 1u;
                        }
                    }
                }
            }
            tc::mma_commit(leader, &accf[buf]);
        }
    issued:
        tc::mma_commit(leader, &done[pair]);
        (void)tc::warp_wait(&done[pair], 0, P.err);
    } else {
        const int q = warp & 3;  // tensor-memory lane quarter this warp may read
        const int row = q * 32 + lane, set = (warp - 4) >> 2, cpv = P.N / 16, nchunk = G * cpv;
        uint32_t tl = 0;
        for (int tile = blockIdx.x; tile < P.ntiles; tile += gridDim.x, ++tl) {
            const uint32_t buf = tl & ((1u << P.nbsh) - 1u);
            if (!mbar_wait_bounded(&accf[buf], (tl >> P.nbsh) & 1, P.err)) abort_flag = 1;
            if (__any_sync(0xffffffffu, abort_flag)) break;
            tc::fence_after_sync();
            const long long pg = ((long long)tile * kBM + row) * G;
            const bool valid = pg < P.R;  // (R is a multiple of G, below 2^30)
            const unsigned up = (unsigned)pg, pxy = (unsigned)P.PXY, px = (unsigned)P.PX;
            const int z0 = (int)(up / pxy), y0 = (int)((up - z0 * pxy) / px), x0 = (int)(up - z0 * pxy - y0 * px);
            const uint32_t taddr = tmem + buf * P.tmem_cols + ((uint32_t)(q * 32) << 16);
            // 16 columns at a time, shared out over the sets of warps
            for (int ch = set; ch < nchunk; ch += kEpiSets) {
                const int vo = ch / cpv, col = 16 * (ch - vo * cpv);
                float v[16];
                if (G > 1) __syncwarp();  // (lanes may come from conv_at)
                tc::tmem_ld16(taddr + (uint32_t)(16 * ch), v);
                if (!valid) continue;
                int x = x0 + vo, y = y0, z = z0;
                if (x >= (int)px) {  // (G <= 4 voxels cross the end of one row at most)
                    x -= (int)px;
                    if (++y == P.Y + 2) {
                        y = 0;
                        ++z;
                    }
                }
                const bool inside = x >= 1 && x <= P.X && y >= 1 && y <= P.Y && z >= 1 && z <= P.Z;
                const int sg = P.nseg > 1 && col >= P.seg_c0[1] ? 1 : 0;
                const int nc = P.seg_nc[sg], c = col - P.seg_c0[sg];
                const long long at = (pg + vo) * nc + c;
                __nv_bfloat16* orow = P.out[sg] + at;
                __nv_bfloat16* arow = P.aux[sg] ? P.aux[sg] + at : nullptr;
                if (!inside) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] = 0.f;
                    store16(orow, v);
                    if (arow && (P.flags & kGelu)) store16(arow, v);
                    continue;
                }
                if (G > 1) {
                    float s = 0.f;
#pragma unroll
                    for (int e = 0; e < 16; ++e) s = fmaf(v[e], 0.f, s);
                    if (s != 0.f) {  // NaN: one of them is not finite
#pragma unroll 1
                        for (int e = 0; e < 16; ++e) {
                            const float x = conv_at(P, pg + vo, col + e);
#pragma unroll
                            for (int f = 0; f < 16; ++f) v[f] = f == e ? x : v[f];
                        }
                    }
                }
                if (P.bias) {
#pragma unroll
                    for (int e = 0; e < 16; e += 4) {
                        const float4 bq = *reinterpret_cast<const float4*>(sbias + col + e);
                        v[e] += bq.x;
                        v[e + 1] += bq.y;
                        v[e + 2] += bq.z;
                        v[e + 3] += bq.w;
                    }
                }
                if (P.flags & kAccum) {
                    float o[16];
                    load16(orow, o);
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] += o[e];
                }
                if (P.flags & kDGelu) {
                    float a[16];
                    load16(arow, a);
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] *= dgelu_f(a[e]);
                }
                if (P.flags & kGelu) {
                    if (arow) store16(arow, v);
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] = gelu_f(v[e]);
                }
                store16(orow, v);
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
        tc::tmem_dealloc(tmem, P.tmem_cols << P.nbsh);
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
        const uint32_t leader = tc::elect_one();
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
                tc::mma_bf16(leader, tmem, ad, bd, P.idesc, acc);
                acc = 1;
                ad += stepa;
                bd += stepg;
            }
            tc::mma_commit(leader, &empty[s]);
            if (++s == (uint32_t)P.ns) {
                s = 0;
                phase ^= 1u;
            }
        }
        tc::mma_commit(leader, &accf);
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

// The same for 16 and 32 input channels, with the groups of k_conv as K: A = the input's rows of G voxels (64 elements),
// two rows (2 G voxels, M = 128), B = the gradient's rows (N = G cout). One MMA sums 16 groups for a (dz, dy): D[(w, ci)]
// [(vo, co)], whose entries with the input voxel w next to the output voxel vo are the 3 taps dx. 3 boxes of 64 to 130 rows
// of 128 bytes per 256 voxels and 12 MMAs, where the taps one by one took 36 boxes of 64 32-byte rows and 64 MMAs (451 us
// for 16 x 16 channels at 128^3, now 70 us). The window of 2 G voxels starts at a voxel of one position within a group for
// all three dy (base), so they share a box.
struct WgradGroupParams {
    CUtensorMap amap, gmap;
    int cin, ci0, cin_tot, cout, G, ntaps, N;
    int ndy, box_rows;             // dy of a step: 3, or 1 (a 1x1x1 convolution)
    int row0[3];                   // per dz: first box row relative to the step's first group
    int yrow[3], ydelta[3];        // per dy: its row within the box; the window's first voxel relative to the group
    int cg, natom_g;
    int k_steps_per_cta, k_steps_total;
    float* dw;
    unsigned* err;
    int ns;
    uint32_t a_bytes, g_atom_bytes, stage_bytes, tmem_cols, idesc;
};

__global__ void __launch_bounds__(kThreads, 1) k_wgrad_groups(const __grid_constant__ WgradGroupParams P)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], accf;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t sbase = aligned_smem_base(smem_raw);
    unsigned char* sgen = smem_raw + (sbase - smem_u32(smem_raw));
    const int dz = blockIdx.x;
    const int k_begin = blockIdx.y * P.k_steps_per_cta;
    const int k_end = min(P.k_steps_total, k_begin + P.k_steps_per_cta);

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

    if (warp == 0) {
        uint32_t it = 0, s = 0, phase = 1;  // stage of the step, parity of its last release
        const uint32_t bytes = (uint32_t)P.box_rows * 128u + P.g_atom_bytes * P.natom_g;
        const int row0 = P.row0[dz];
        for (int ks = k_begin; ks < k_end; ++ks, ++it) {
            if (it >= (uint32_t)P.ns && !tc::warp_wait(&empty[s], phase, P.err)) {
                abort_flag = 1;
                break;
            }
            if (tc::elect_one()) {
                const int q0 = ks * kWgradRows;
                mbar_arrive_expect_tx(&full[s], bytes);
                unsigned char* a = sgen + s * P.stage_bytes;
                tma_load_2d(a, &P.amap, &full[s], 0, q0 + row0);
                for (int m = 0; m < P.natom_g; ++m)
                    tma_load_2d(a + P.a_bytes + m * P.g_atom_bytes, &P.gmap, &full[s], m * P.cg, q0);
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
        // MN-major operands: the second atom of A is the next row (LBO one row), 8-row K groups at SBO
        const uint32_t leader = tc::elect_one();
        const uint64_t da = tc::sdesc(0, 128, 1024, tc::kSwizzle128);
        const uint64_t dg = tc::sdesc(0, P.g_atom_bytes, 8u * P.cg * 2u, tc::swizzle_code(P.cg * 2));
        const uint32_t stepg = 16u * P.cg * 2u >> 4;
        const int ndy = P.ndy;
        const uint32_t y0 = (uint32_t)P.yrow[0] * 8u, y1 = (uint32_t)P.yrow[1] * 8u, y2 = (uint32_t)P.yrow[2] * 8u;
        uint32_t s = 0, phase = 0, acc = 0;
        for (int ks = k_begin; ks < k_end; ++ks) {
            if (!tc::warp_wait(&full[s], phase, P.err)) {
                abort_flag = 1;
                break;
            }
            tc::fence_after_sync();
            const uint32_t a = sbase + s * P.stage_bytes;
            const uint64_t ad = da + (a >> 4);
            uint64_t bd = dg + ((a + P.a_bytes) >> 4);
#pragma unroll
            for (int kk = 0; kk < kWgradRows / 16; ++kk) {
                tc::mma_bf16(leader, tmem, ad + (y0 + 128u * kk), bd, P.idesc, acc);
                if (ndy > 1) {
                    tc::mma_bf16(leader, tmem + P.N, ad + (y1 + 128u * kk), bd, P.idesc, acc);
                    tc::mma_bf16(leader, tmem + 2 * P.N, ad + (y2 + 128u * kk), bd, P.idesc, acc);
                }
                acc = 1;
                bd += stepg;
            }
            tc::mma_commit(leader, &empty[s]);
            if (++s == (uint32_t)P.ns) {
                s = 0;
                phase ^= 1u;
            }
        }
        tc::mma_commit(leader, &accf);
    } else {
        const int q = warp & 3;
        const int row = q * 32 + lane;  // M row = (window voxel, input channel)
        const bool ok = tc::warp_wait(&accf, 0, P.err) && k_end > k_begin;
        tc::fence_after_sync();
        const int w = row / P.cin, ci = row % P.cin;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
        const bool good = __all_sync(0xffffffffu, ok && !abort_flag);
        for (int y = 0; y < P.ndy; ++y)
            for (int vo = 0; vo < P.G; ++vo) {
                const int dx = P.ydelta[y] + w - vo;
                const bool store = good && (P.ntaps == 1 ? dx == 0 : dx >= -1 && dx <= 1);
                if (!__any_sync(0xffffffffu, store)) continue;
                const int tap = P.ntaps == 1 ? 0 : 9 * dz + 3 * y + dx + 1;
                for (int c = 0; c < P.cout; c += 16) {
                    float v[16];
                    tc::tmem_ld16(taddr + (uint32_t)(y * P.N + vo * P.cout + c), v);
                    if (!store) continue;
                    float* dst = P.dw + ((long long)tap * P.cout + c) * P.cin_tot + P.ci0 + ci;
#pragma unroll
                    for (int e = 0; e < 16; ++e) atomicAdd(dst + (long long)e * P.cin_tot, v[e]);
                }
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
        P.in[i] = L.in[i];
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
    P.w = L.w;
    P.cin_tot = cin_tot;
    P.ntaps = L.ntaps;
    P.N = L.N;
    P.flip = L.flip;
    P.gtaps = L.ntaps == 27 ? 3 : 1;
    const int nstack = L.ntaps == 27 ? 9 : 1;
    int off[27];
    tap_offsets(L.g, L.ntaps, L.flip, off);
    // voxels per GEMM row: rows of 64 elements (128 bytes) for the narrowest input, where the grid and its planes split into
    // such groups and the columns stay within an MMA's 256 (twice that is the tensor memory)
    for (P.G = 64 / cmin; P.G > 1; P.G >>= 1)
        if (L.g.R % P.G == 0 && L.g.PXY % P.G == 0 && P.G * L.N <= 256) break;
    auto rows_of = [&](int v) { return (int)((v >= 0 ? v : v - P.G + 1) / P.G); };  // floor
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
        const int rc = encode_rows(L.w, cin_tot, (long long)L.ntaps * L.N, P.cb[i], P.wbox * L.N, &P.wmap[i]);
        if (rc) return rc;
        P.w_in[i] = wres_bytes;
        P.w_chunk[i] = ((uint32_t)((P.gtaps + P.G - 1) * nstack + P.G - 1) * L.N * P.cb[i] * 2u + 1023u) & ~1023u;
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
    P.tmem_cols = pow2_cols(P.G * L.N);
    P.idesc = tc::idesc_bf16(kBM, P.G * L.N, 0, 0);
    P.w_area = wres_bytes;
    // weights resident where at least 3 activation stages fit beside them, else with each step
    const uint32_t max_smem = kConvSmem;
    auto box = [&](int rows) {
        P.a_rows = rows;
        P.box_bytes = ((uint32_t)rows * abmax * 2u + 1023u) & ~1023u;
        P.a_bytes = nbmax * P.box_bytes;
    };
    const int PX = (int)L.g.PX, mid = L.ntaps == 27 ? 1 : 0;
    box(kBM + (mid ? 2 + (P.G > 1) : 0));
    P.wres = wres_bytes + 3 * P.a_bytes + 1024 <= max_smem;
    P.ndy = 1;
    if (mid && P.wres) {
        // one box for the three dy of a dz where its rows fit a TMA box and two stages stay: the rows of neighbouring dy
        // overlap (194 rows instead of 3 x 130 at 128^3), and L2 reads bounded the level-0 convolutions at 5 TB/s
        // (two rings of single boxes go before one ring of these: 32 + 16 -> 16 channels at 128^3 263 us with one ring, 193
        // with two)
        const int rows = kBM + rows_of(PX + P.G) - rows_of(-PX - 1), was = P.a_rows;
        const bool two_rings = wres_bytes + 4 * P.a_bytes + 1024 <= max_smem;
        if (rows <= 256) {
            box(rows);
            P.ndy = 3;
            if (wres_bytes + (two_rings ? 4 : 2) * P.a_bytes + 1024 > max_smem) {
                box(was);
                P.ndy = 1;
            }
        }
    }
    P.nstep = nstack / P.ndy;
    for (int y = 0; y < 3; ++y) {
        P.yoff[y] = mid ? off[3 * (3 + y) + 1] : 0;  // dz = 0
        P.ybase[y] = rows_of(P.ndy == 3 ? -PX - 1 : P.yoff[y] - mid) * P.G;
    }
    for (int q = 0; q < P.nstep; ++q) {
        const int dz = mid ? off[3 * (3 * (q * P.ndy / 3) + 1) + 1] : 0;  // a multiple of G
        P.grow[q] = dz / P.G + P.ybase[P.ndy == 3 ? 0 : (mid ? q % 3 : 0)] / P.G;
    }
    for (int i = 0; i < L.nin; ++i) {
        const int rc = encode_rows(L.in[i], P.G * L.cin[i], L.g.R / P.G, P.ab[i], P.a_rows, &P.amap[i]);
        if (rc) return rc;
    }
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
    const int stages = (int)((max_smem - 1024 - (P.wres ? wres_bytes : 0)) / P.stage_bytes);
    P.npair = stages >= 4 ? 2 : 1;
    P.ns = std::min(kPairStages, stages / P.npair);
    if (P.ns < 2) {
        set_error("conv3d: stage does not fit in shared memory");
        return GBP_BAD_ARG;
    }
    P.nbsh = P.npair == 2 && 4 * P.tmem_cols <= 512 ? 2 : 1;
    P.w_base = (uint32_t)(P.npair * P.ns) * P.stage_bytes;
    const size_t smem = (size_t)P.w_base + (P.wres ? wres_bytes : 0) + 1024;
    static bool attr_set = false;
    if (!attr_set) {
        for (auto k : {k_conv<1>, k_conv<2>, k_conv<4>})
            GBP_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmem));
        attr_set = true;
    }
    const int grid = std::min(P.ntiles, sm_count_cached());
    (P.G == 4 ? k_conv<4> : P.G == 2 ? k_conv<2> : k_conv<1>)<<<grid, kConvThreads, smem, st>>>(P);
    GBP_CUDA(cudaGetLastError());
    return GBP_OK;
}

// The grouped weight gradient for 16 and 32 input channels; *done = false: not for this grid, nothing launched
static int wgrad_groups(const WgradLaunch& L, cudaStream_t st, bool* done)
{
    *done = false;
    const int G = 64 / std::max(L.cin, 1), PX = (int)L.g.PX;
    if ((L.cin != 16 && L.cin != 32) || L.g.R % G || L.g.PXY % G || 3 * G * L.cout > 512 || G * L.cout > 256) return GBP_OK;
    WgradGroupParams P;
    memset(&P, 0, sizeof(P));
    auto rows_of = [&](int v) { return (v >= 0 ? v : v - G + 1) / G; };  // floor
    const int mid = L.ntaps == 27 ? 1 : 0;
    P.ndy = mid ? 3 : 1;
    // the position within a group at which every dy's window of 2 G voxels can start: at or before its voxel -1, ending at or
    // after its voxel G
    int base = -1;
    for (int b = 0; b < G && base < 0; ++b) {
        bool all = true;
        for (int y = 0; y < P.ndy; ++y) {
            const int first = (mid ? (y - 1) * PX : 0) - mid;  // the window's start lies in (first - (G - 2 mid) - 1, first]
            const int start = b + rows_of(first - b) * G;
            all = all && start >= first - (G - 2 * mid);
        }
        if (all) base = b;
    }
    if (base < 0) return GBP_OK;
    int start[3], lo = 0, hi = 0;
    for (int y = 0; y < P.ndy; ++y) {
        const int off = mid ? (y - 1) * PX : 0;
        start[y] = rows_of(off - mid - base);
        P.ydelta[y] = base + start[y] * G - off;
        lo = y ? std::min(lo, start[y]) : start[y];
        hi = y ? std::max(hi, start[y]) : start[y];
    }
    P.box_rows = kWgradRows + hi - lo + 1;
    if (P.box_rows > 256) return GBP_OK;
    for (int y = 0; y < P.ndy; ++y) P.yrow[y] = start[y] - lo;
    for (int z = 0; z < 3; ++z) P.row0[z] = mid ? (int)((z - 1) * (L.g.PXY / G)) + lo : lo;
    P.cin = L.cin;
    P.ci0 = L.ci0;
    P.cin_tot = L.cin_tot;
    P.cout = L.cout;
    P.G = G;
    P.ntaps = L.ntaps;
    P.N = G * L.cout;
    P.cg = std::min(64, P.N);
    P.natom_g = P.N / P.cg;
    int rc = encode_rows(L.in + (size_t)base * L.cin, 64, (L.g.R - base) / G, 64, P.box_rows, &P.amap);
    if (!rc) rc = encode_rows(L.gout, P.N, L.g.R / G, P.cg, kWgradRows, &P.gmap);
    if (rc) return rc;
    P.dw = L.dw;
    P.err = L.err;
    P.a_bytes = ((uint32_t)P.box_rows * 128u + 1023u) & ~1023u;
    P.g_atom_bytes = (uint32_t)kWgradRows * P.cg * 2u;
    P.stage_bytes = P.a_bytes + ((P.g_atom_bytes * P.natom_g + 1023u) & ~1023u);
    P.tmem_cols = pow2_cols(P.ndy * P.N);
    P.idesc = tc::idesc_bf16(kBM, P.N, 1, 1);
    P.ns = std::min(kMaxStages, (int)((200 * 1024 - 1024) / P.stage_bytes));
    P.k_steps_total = (int)((L.g.R / G + kWgradRows - 1) / kWgradRows);
    const int nz = mid ? 3 : 1, want = std::max(1, sm_count_cached() / nz);
    P.k_steps_per_cta = std::max(8, (P.k_steps_total + want - 1) / want);
    const int splits = (P.k_steps_total + P.k_steps_per_cta - 1) / P.k_steps_per_cta;
    static bool attr_set = false;
    if (!attr_set) {
        GBP_CUDA(cudaFuncSetAttribute(k_wgrad_groups, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr_set = true;
    }
    k_wgrad_groups<<<dim3(nz, splits), kThreads, (size_t)P.ns * P.stage_bytes + 1024, st>>>(P);
    GBP_CUDA(cudaGetLastError());
    *done = true;
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
    bool done = false;
    const int grc = wgrad_groups(L, st, &done);
    if (grc || done) return grc;
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

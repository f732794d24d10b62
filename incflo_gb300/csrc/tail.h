// The small levels of a V-cycle in one launch: a thread-block cluster holds them in shared memory (tail.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "gbp_internal.cuh"
#include "nodal_kernels.h"

namespace gbp {

constexpr int kTailLevels = 8;     // most levels of a tail, the bottom included
constexpr int kTailThreads = 512;
constexpr int kTailTargets = 6;    // CTAs that keep a copy of one plane
constexpr int kTailHalo = 5;       // planes of a level's arrays beyond its own planes (nodal: 4 arrays, MAC: 7)

// How the planes of the levels are shared out: CTA c of the cluster owns planes lo .. lo + np - 1 of level q and keeps
// copies of planes lo - 1 and lo + np; a coarse plane K belongs to the owner of fine plane 2K. Levels from `solo` on are
// cycled by CTA 0 alone (lo = 0, all planes; the other CTAs hold room for the result of the first of them). The table (device
// memory, read once per launch): per level [lo, np] of each CTA, then per plane the copies that a store must update,
// [count, (cta << 16 | local slot) ...].
struct TailLayout {
    int nl = 0, ctas = 0, solo = 0;
    int np[kTailLevels] = {};       // most planes of a CTA on the level
    int plane[kTailLevels] = {};    // elements of one padded plane
    int off[kTailLevels] = {};      // first element of the level's arrays in shared memory
    int own[kTailLevels] = {};      // table position of the level's [lo, np]
    int copies[kTailLevels] = {};   // ... and of its planes' copies
    int tab_ints = 0;
    size_t tab_off = 0, dense_off = 0, bytes = 0;  // byte offsets in shared memory, and its size
    std::vector<int> table;
};
// planes[q] of the levels, periodic in z or not; plane elements, unknowns and arrays per level; esize: bytes of an
// element; nbottom: unknowns of the last level (its data are not distributed); solo_most: unknowns of a level that one
// CTA cycles. false: the tail does not fit.
bool tail_layout(int nl, const int* planes, int per, const int* plane_elems, const long long* unknowns, int arrays,
                 int esize, int nbottom, long long solo_most, int ctas, TailLayout* out);
// the largest cluster the device runs for the tail kernels: 16 (non-portable), 8, or 0
int tail_cluster_size();

template <typename T>
struct NodalTail {
    int nl, ctas, solo, tab_ints;
    NodalGeom g[kTailLevels];
    const T* s[kTailLevels];   // sigma of each level (global, padded)
    const T* b0;               // the first level's right-hand side
    T* xout;                   // its result (global, padded, with aliases)
    const double* M;           // dense inverse of the bottom operator
    int singular;
    T wpre[kSweepWeights], wpost[kSweepWeights];
    int nu1, nu2;              // >= 1
    const int* table;
    int np[kTailLevels], off[kTailLevels], own[kTailLevels], copies[kTailLevels];
    size_t tab_off, dense_off;
};
template <typename T>
int nodal_tail(const NodalTail<T>& a, size_t bytes, cudaStream_t st);

template <typename T>
struct MacTail {
    int nl, ctas, solo, tab_ints;
    CellGeom g[kTailLevels];
    const T *bx[kTailLevels], *by[kTailLevels], *bz[kTailLevels];
    const T* b0;
    T* xout;
    const double* M;
    const unsigned char* act;
    int singular;
    int nu1, nu2;              // >= 1
    const int* table;
    int np[kTailLevels], off[kTailLevels], own[kTailLevels], copies[kTailLevels];
    size_t tab_off, dense_off;
};
template <typename T>
int mac_tail(const MacTail<T>& a, size_t bytes, cudaStream_t st);

}  // namespace gbp

// The coarse part of a multigrid cycle in one thread-block-cluster launch (fhg_coarse.cu).
#pragma once

#include <cuda_runtime.h>

#include "fhg_pair.h"

namespace fhg {

constexpr int kClusterCtasPortable = 8;   // CTAs of the one cluster: the portable maximum, or
constexpr int kClusterCtasLarge = 16;     // the non-portable one where the device runs it
constexpr int kFusedThreads = 512;        // threads per CTA (128 registers)
constexpr int kFusedThreadsWide = 1024;   // or twice the warps per SM (64 registers)
constexpr int kFusedMaxLevels = 6;        // levels of a fused sub-cycle, the coarsest included
constexpr int kFusedMaxColours = 64;
constexpr int kFusedMaxRows = 65536;      // block rows of the largest level a fused sub-cycle takes

constexpr int kFusedDefaultRows = 768;    // the same without timing at setup (autotuning off)
constexpr int kChunkLog = 2, kChunk = 1 << kChunkLog;   // block rows dealt out to the CTAs at a time
constexpr int kFusedMaxSmem = 200 * 1024; // shared memory of a CTA for the levels' vectors

// Smoother directions of a fused sub-cycle (the GS codes; Jacobi is not fused).
enum { kFusedForward = 0, kFusedBackward = 1, kFusedSymmetric = 2, kFusedAlternatingForward = 3,
       kFusedAlternatingBackward = 4 };

// One level of the sub-cycle in the launch parameters: A in CSR form (all blocks, entry-major values,
// leading dimension a_ld), D^-1 entry-major (leading dimension nb), the colour offsets, P (this
// level's rows, the next level's columns) and R = P^T (the next level's rows), and the places of
// the level's vectors. Threads (2 to 32, a power of two) that walk one block row: `lanes` in a sweep, `a_lanes` in
// the residual, `r_lanes` and `p_lanes` in the transfers. On the coarsest level only those of x and b are
// used.
template <class T>
struct FusedLevel {
    int nb = 0, ncol = 0, lanes = 8, a_lanes = 8, r_lanes = 8, p_lanes = 8;
    int colour_start[kFusedMaxColours + 1] = {};
    const int* a_rowptr = nullptr;
    const int* a_colidx = nullptr;
    const T* a_vals = nullptr;
    long long a_ld = 0;
    const T* dinv = nullptr;
    const int* p_rowptr = nullptr;
    const int* p_colidx = nullptr;
    const T* p_vals = nullptr;
    long long p_ld = 0;
    const int* r_rowptr = nullptr;
    const int* r_colidx = nullptr;
    const T* r_vals = nullptr;
    long long r_ld = 0;
    int x_off = 0, b_off = 0, r_off = 0;   // the level's vectors in a CTA's shared memory (fused_layout)
    T* x = nullptr;                        // lev[0]: x and b in global memory
    const T* b = nullptr;
};

template <class T>
struct FusedCycle {
    int nlev = 0;                 // levels, the coarsest included (lev[nlev - 1])
    int n_coarse = 0;             // unknowns of the coarsest level
    int c_lanes = 8;              // threads per row of its dense solve
    int bc_off = 0;               // its b in FP64 in a CTA's shared memory (fused_layout)
    const double* cinv = nullptr; // its dense FP64 inverse, row-major
    int pre = 0, post = 1, npre = 1, npost = 1, w_loops = 1;
    int x_zero = 1;               // x of the first level starts at zero
    T omega = T(1);               // relaxation of the GS sweeps (block SOR when not 1)
    FusedLevel<T> lev[kFusedMaxLevels];
};

// Places the levels' vectors (nb of every level, nlev and n_coarse set) in the shared memory of `ctas`
// CTAs; the bytes a CTA needs, -1 when they do not fit.
template <class T>
int fused_layout(FusedCycle<T>& P, int bs, int ctas);
// One cluster of `ctas` CTAs (kClusterCtasPortable or kClusterCtasLarge) of `threads` threads
// (kFusedThreads or kFusedThreadsWide) with `smem` bytes of shared memory each.
template <class T>
cudaError_t launch_fused_cycle(const FusedCycle<T>& P, int bs, int ctas, int threads, int smem, cudaStream_t s);
// Clusters of `ctas` CTAs of `threads` threads with `smem` bytes each of the fused kernel that fit on the
// current device at once (0: it cannot run here).
template <class T>
int fused_cycle_clusters(int bs, int ctas, int threads, int smem);

}  // namespace fhg

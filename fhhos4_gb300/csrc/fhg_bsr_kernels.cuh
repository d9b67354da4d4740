#pragma once
// Block-sparse kernels of the fhhos4 solve phase for GB300 (sm_103a), templated on the value type
// (double, float, or the FP32 pair dfl) and instantiated by fhg_kernels.cu (float, double) and
// fhg_kernels_pair.cu (pairs).
//
// Every kernel is memory-bound: block-sparse products over face-block operators
// (bs = face DOFs: 2/3/4/6), colour sweeps of block Gauss-Seidel, and the FCG vector
// updates. The design targets HBM bandwidth:
//   * block values entry-major (vals[e*ld + p]) so a warp reading consecutive blocks
//     issues fully coalesced 8-byte (FP64) or 4-byte (FP32) loads per entry;
//   * a group of G lanes (G = 4..32, chosen per operator) per block row, partial sums
//     reduced with warp shuffles;
//   * reductions write fixed-size per-CTA partial arrays that every consumer reduces
//     in the same order (bitwise reproducible Krylov scalars, no atomics);
//   * Krylov scalars never leave the device: consumers read them from device memory,
//     so one whole iteration can be replayed as a CUDA graph.
#include "fhg_internal.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>
#include <utility>

namespace fhg {

namespace {


constexpr int kThreads = 256;

// Programmatic dependent launch: every kernel of this file is launched with programmatic stream
// serialization, so the next kernel's CTAs are scheduled while its predecessor drains instead of
// after it, and begins with pdl_wait() (griddepcontrol.wait), which returns once the predecessor
// grid has completed and its memory writes are visible. No global access precedes the wait, so
// the order of every read and write is that of plain stream order; only launch latency overlaps.
// Kernels launched without the attribute pass the wait at once. FHG_PDL=0 in the environment
// launches without it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

bool pdl_enabled()
{
    static const bool on = [] {
        const char* e = std::getenv("FHG_PDL");
        return !(e && e[0] == '0');
    }();
    return on;
}

template <class... KArgs, class... Args>
void pdl_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <int G, class T>
__device__ __forceinline__ T group_sum(T v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, G);
    return v;
}

// A pair's group sum: both parts shuffled, the partner's pair added with TwoSum.
template <int G>
__device__ __forceinline__ dfl group_sum(dfl v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, v.h, o, G);
        const float ol = __shfl_xor_sync(0xffffffffu, v.l, o, G);
        df_add(v.h, v.l, oh, ol);
    }
    return v;
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The warp of a kReduceThreads CTA that finishes its sums: one of four by the CTA's place in the grid, so that
// the CTAs of an SM use its four schedulers.
__device__ __forceinline__ int finishing_warp() { return (int)(blockIdx.x / (kReduceCtas / 4)) & 3; }

// Not +-0, without an instruction of the FP64 pipe.
__device__ __forceinline__ bool nonzero(double v) { return (__double_as_longlong(v) << 1) != 0; }

// N sums over a kReduceThreads CTA in one fixed order, valid in every thread. A warp's FP64 addition holds its
// scheduler for 64 cycles (2 lanes a clock on an SM), so what counts is the warp instructions of all CTAs of an
// SM: one warp a sum, each lane adding eight of the threads' values and five shuffles (12 additions), where
// a shuffle reduction of every warp and then of their results takes 45: with four CTAs on an SM 2,880 cycles of the
// pipe a sum against 770. Groups of zeros add nothing: a CTA without elements, and the partials of one, cost no
// addition. With cta_ratio below, an FCG iteration in FP64 at 6,000 unknowns went from 95 to 81 us, at 300,000 from
// 546 to 538.
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N])
{
    constexpr int kWarps = kReduceThreads / 32;
    __shared__ double sh[N * kReduceThreads + N];
    const int lane = threadIdx.x & 31, k = ((int)(threadIdx.x >> 5) - finishing_warp()) & (kWarps - 1);
    __syncthreads();   // the previous call's sums are read
#pragma unroll
    for (int q = 0; q < N; q++) sh[q * kReduceThreads + threadIdx.x] = v[q];
    __syncthreads();
    if (k < N) {
        const double* p = sh + k * kReduceThreads + lane;
        double t = p[0];
#pragma unroll
        for (int q = 1; q < kWarps; q++) {
            const double u = p[32 * q];
            if (__any_sync(0xffffffffu, nonzero(u))) t += u;
        }
        if (__any_sync(0xffffffffu, nonzero(t))) t = warp_sum(t);
        if (lane == 0) sh[N * kReduceThreads + k] = t;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < N; q++) v[q] = sh[N * kReduceThreads + q];
}

__device__ __forceinline__ double block_sum(double v)
{
    double s[1] = {v};
    block_sums(s);
    return s[0];
}

// Fixed-order sums of kReduceCtas-long partial arrays by one CTA.
template <int N>
__device__ __forceinline__ void reduce_partials(const double* const (&p)[N], double (&v)[N])
{
    constexpr int kRounds = (kReduceCtas + kReduceThreads - 1) / kReduceThreads;
    double u[N][kRounds];
#pragma unroll
    for (int k = 0; k < N; k++)
#pragma unroll
        for (int q = 0; q < kRounds; q++) {
            const int i = q * kReduceThreads + threadIdx.x;
            u[k][q] = i < kReduceCtas ? p[k][i] : 0.0;
        }
#pragma unroll
    for (int k = 0; k < N; k++) {
        v[k] = u[k][0];
#pragma unroll
        for (int q = 1; q < kRounds; q++)
            if (__any_sync(0xffffffffu, nonzero(u[k][q]))) v[k] += u[k][q];
    }
    block_sums(v);
}

__device__ __forceinline__ double reduce_partials(const double* __restrict__ p)
{
    const double* const ps[1] = {p};
    double v[1];
    reduce_partials(ps, v);
    return v[0];
}

// A Krylov scalar num / den and its FP32 pair in every thread, divided by one warp: an FP64 division is a
// chain of several instructions of the FP64 pipe, which all 32 warps of four CTAs on an SM would take in turn.
struct Scalar {
    double v;
    float h, l;
};
__device__ __forceinline__ Scalar cta_ratio(double num, double den)
{
    __shared__ Scalar s;
    if ((int)(threadIdx.x >> 5) == finishing_warp()) {
        Scalar q;
        q.v = num / den;
        df_split(q.v, q.h, q.l);
        if ((threadIdx.x & 31) == 0) s = q;
    }
    __syncthreads();
    return s;
}

// Element loop of the fixed-grid vector kernels: thread t of CTA c visits
// i = c * kReduceThreads + t, then i + S, i + 2 S, ... (S = kReduceCtas * kReduceThreads) in that
// order, so every per-thread sum is taken in one fixed order. Four elements go per step with all
// their loads issued before the first use: one element per thread per step leaves too few bytes
// in flight for HBM (a quarter of what the copy rate needs at 152 x 4 CTAs of 256 threads).
// `load(i)` returns the element's inputs, `use(i, v)` computes and stores; `ready()` runs once behind the
// first loads and in front of their use, for what the uses need of the grid's scalars.
constexpr long long kRedStride = (long long)kReduceCtas * kReduceThreads;
constexpr int kRedUnroll = 4;

// A CTA of those kernels without elements (the first one always works).
__device__ __forceinline__ bool idle_cta(long long n) { return blockIdx.x > 0 && (long long)blockIdx.x * kReduceThreads >= n; }

template <class Load, class Ready, class Use>
__device__ __forceinline__ void for_each_element(long long n, Load load, Ready ready, Use use)
{
    long long i = (long long)blockIdx.x * kReduceThreads + threadIdx.x;
    decltype(load(i)) v[kRedUnroll];
    auto fetch = [&] {
#pragma unroll
        for (int u = 0; u < kRedUnroll; u++)
            if (i + u * kRedStride < n) v[u] = load(i + u * kRedStride);
    };
    fetch();
    ready();
    while (i < n) {
#pragma unroll
        for (int u = 0; u < kRedUnroll; u++)
            if (i + u * kRedStride < n) use(i + u * kRedStride, v[u]);
        i += kRedUnroll * kRedStride;
        fetch();
    }
}

template <class Load, class Use>
__device__ __forceinline__ void for_each_element(long long n, Load load, Use use)
{
    for_each_element(n, load, [] {}, use);
}

template <class A, class B>
struct Pair2 {
    A a;
    B b;
};

template <class T>
struct Quad4 {
    T a, b, c, d;
};

// ---------------------------------------------------------------------------
// Row accumulation: acc[r] += sum over this lane's blocks of (A_block x_col)[r].
// `sel(col)` returns 0 (skip the block), 1 (use it) or 2 (stop: columns are sorted, nothing
// after it is used). With U = 2 (bs <= 3) each lane walks two blocks per step so that the loads
// of both (column index, bs^2 values, bs entries of x) are in flight together, at the cost of
// registers (fewer resident warps); U is chosen per operator by the autotuner. The
// accumulation order is block by block either way.
template <class T, int BS, int G, int U, class Sel>
__device__ __forceinline__ void accumulate_row(int p0, int p1, int lane, const int* __restrict__ colidx,
                                               const T* __restrict__ vals, long long ld, const T* x, T* acc,
                                               Sel sel)
{
    if constexpr (U == 2 && BS <= 3) {
        for (int p = p0 + lane; p < p1; p += 2 * G) {
            const int q = p + G;
            const int ca = colidx[p];
            const int cb = q < p1 ? colidx[q] : -1;
            const int ua = sel(ca);
            if (ua == 2) break;
            const int ub = cb >= 0 ? sel(cb) : 0;
            T va[BS * BS], vb[BS * BS], xa[BS], xb[BS];
            if (ua == 1) {
#pragma unroll
                for (int e = 0; e < BS * BS; e++) va[e] = vals[(long long)e * ld + p];
#pragma unroll
                for (int c = 0; c < BS; c++) xa[c] = x[(long long)ca * BS + c];
            }
            if (ub == 1) {
#pragma unroll
                for (int e = 0; e < BS * BS; e++) vb[e] = vals[(long long)e * ld + q];
#pragma unroll
                for (int c = 0; c < BS; c++) xb[c] = x[(long long)cb * BS + c];
            }
            if (ua == 1) {
#pragma unroll
                for (int r = 0; r < BS; r++)
#pragma unroll
                    for (int c = 0; c < BS; c++) acc[r] = fma(va[r * BS + c], xa[c], acc[r]);
            }
            if (ub == 1) {
#pragma unroll
                for (int r = 0; r < BS; r++)
#pragma unroll
                    for (int c = 0; c < BS; c++) acc[r] = fma(vb[r * BS + c], xb[c], acc[r]);
            }
            if (ub == 2) break;
        }
    } else {
        for (int p = p0 + lane; p < p1; p += G) {
            const int col = colidx[p];
            const int u = sel(col);
            if (u == 2) break;
            if (u == 0) continue;
            T xv[BS];
#pragma unroll
            for (int c = 0; c < BS; c++) xv[c] = x[(long long)col * BS + c];
#pragma unroll
            for (int r = 0; r < BS; r++)
#pragma unroll
                for (int c = 0; c < BS; c++) acc[r] = fma(vals[(long long)(r * BS + c) * ld + p], xv[c], acc[r]);
        }
    }
}

struct UseAll {
    __device__ __forceinline__ int operator()(int) const { return 1; }
};

// First and one-past-last stored position of a block row: padded views (ell > 0) put row i at
// i * ell, with no row-pointer load ahead of the row walk. Their empty slots hold zero values and
// a column inside the operator (the row's own in the off-diagonal GS view, where the sweep skips
// it as the diagonal; a stored column of the row otherwise, where a product adds an exact zero).
__device__ __forceinline__ void row_range(int row, int ell, const int* __restrict__ rowptr, int& p0, int& p1)
{
    if (ell > 0) {
        p0 = row * ell;
        p1 = p0 + ell;
    } else {
        p0 = rowptr[row];
        p1 = rowptr[row + 1];
    }
}

// ---------------------------------------------------------------------------
// y = A x  |  y = aux - A x  |  y = aux + A x      (aux may alias y)
template <class T, int BS, int G, int U, int MODE>
__global__ void __launch_bounds__(kThreads) k_bsr_spmv(int nbr, const int* __restrict__ rowptr,
                                                       const int* __restrict__ colidx,
                                                       const T* __restrict__ vals, long long ld,
                                                       const T* __restrict__ x, const T* aux, T* y, int ell)
{
    pdl_wait();
    const int lane = threadIdx.x & (G - 1);
    const int row = (int)(((long long)blockIdx.x * kThreads + threadIdx.x) / G);
    T acc[BS];
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = T(0);
    // Lane r < BS writes output r of the row (G >= BS here: G is at least 4 and bs at most 3 on
    // this path, or lanes loop over outputs below when bs > G). The added vector is loaded
    // before the row walk so that its latency overlaps it.
    T av = T(0);
    if (MODE != kSpmvAssign && G >= BS && row < nbr && lane < BS) av = aux[(long long)row * BS + lane];
    if (row < nbr) {
        int p0, p1;
        row_range(row, ell, rowptr, p0, p1);
        accumulate_row<T, BS, G, U>(p0, p1, lane, colidx, vals, ld, x, acc, UseAll());
    }
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = group_sum<G>(acc[r]);
    if (row < nbr) {
#pragma unroll
        for (int r = 0; r < BS; r++) {
            if (lane == r % G) {
                const long long i = (long long)row * BS + r;
                const T a = (G >= BS) ? av : ((MODE == kSpmvAssign) ? T(0) : aux[i]);
                if (MODE == kSpmvAssign) y[i] = fin(acc[r]);
                else if (MODE == kSpmvResidual) y[i] = a - acc[r];
                else y[i] = a + acc[r];
            }
        }
    }
}

// y = M x | y = y + M x on the sliced view: L lanes per row (1 for the short rows of P; 4 or 8 for those of
// R, 25 to 50 blocks, of which there are too few for a thread each), a warp per slice of 32 / L rows, so every
// load of the slice's columns and values is 32 consecutive words, with no padding but what the longest row of
// a slice adds (a few percent, the rows being sorted by length in windows of kSellWindow; the windows keep a
// slice's output rows within a few cache lines of each other). Few lanes: in FP64 a lane group's shuffle
// adds cost the pipe as much as its products. The columns of the next kGroup blocks are loaded ahead of the
// sums over the present ones. A lane's running sum in pairs is normalised every second product: left as it is, its
// low part gathers the errors of a dozen blocks and rounds at their size (R r 1.4 to 3 times further off than with a
// warp a row; so, 0.9 to 1.1 times). Against CSR rows of 8 (P) and 32 (R) lanes, or of the tuned lanes at 64^3: x += P e
// FP64 32^3 124 -> 47 us, FP32 64^3 183 -> 128 us (0.9 of HBM), pairs 48^3 122 -> 96; R r FP64 32^3 118 -> 43,
// FP32 64^3 148 -> 130, 32^3 23 -> 12, 24^3 k = 2 45 -> 30, pairs 48^3 113 -> 104.
template <class T, int BS, int MODE, int L>
__global__ void __launch_bounds__(kThreads) k_bsr_spmv_sell(int slices, const int* __restrict__ perm,
                                                            const int* __restrict__ ptr,
                                                            const int* __restrict__ colidx,
                                                            const T* __restrict__ vals, long long ld,
                                                            const T* __restrict__ x, const T* aux, T* y)
{
    constexpr int kBlockBytes = BS * BS * (int)sizeof(T);
    // blocks in flight: ~144 bytes; a thread a row of R, whose rows are long, takes twice that (pairs 64^3, 387,072
    // rows: 246 -> 239 us)
    constexpr bool kLong = L == 1 && MODE == kSpmvAssign;
    constexpr int kGroup = kBlockBytes <= (kLong ? 72 : 36) ? 4 : kBlockBytes <= 72 ? 2 : 1;
    const int slice = (int)((blockIdx.x * kThreads + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (slice >= slices) return;   // whole warps
    const int row = perm[slice * (32 / L) + lane / L];
    int p = ptr[slice] + lane;
    const int p1 = ptr[slice + 1];
    int col[kGroup];
#pragma unroll
    for (int g = 0; g < kGroup; g++) col[g] = p + 32 * g < p1 ? colidx[p + 32 * g] : -1;
    pdl_wait();
    T acc[BS], av[BS];   // M x is summed from zero and added once: from y on, every product would round at y's size
#pragma unroll
    for (int r = 0; r < BS; r++) {
        av[r] = MODE == kSpmvAssign || row < 0 ? T(0) : aux[(long long)row * BS + r];
        acc[r] = T(0);
    }
    while (p < p1) {   // the same number of steps in every lane
        T xv[kGroup][BS], v[kGroup][BS * BS];
#pragma unroll
        for (int g = 0; g < kGroup; g++) {
#pragma unroll
            for (int c = 0; c < BS; c++) xv[g][c] = col[g] >= 0 ? x[(long long)col[g] * BS + c] : T(0);
#pragma unroll
            for (int e = 0; e < BS * BS; e++) v[g][e] = col[g] >= 0 ? vals[(long long)e * ld + p + 32 * g] : T(0);
        }
        p += 32 * kGroup;
#pragma unroll
        for (int g = 0; g < kGroup; g++) {
            const int next = p + 32 * g < p1 ? colidx[p + 32 * g] : -1;
            if (col[g] >= 0) {
#pragma unroll
                for (int r = 0; r < BS; r++)
#pragma unroll
                    for (int c = 0; c < BS; c++) {
                        acc[r] = fma(v[g][r * BS + c], xv[g][c], acc[r]);
                        if (c % 2 || c + 1 == BS) acc[r] = fin(acc[r]);
                    }
            }
            col[g] = next;
        }
    }
    if (L > 1) {
#pragma unroll
        for (int r = 0; r < BS; r++) acc[r] = group_sum<L>(acc[r]);
    }
    if (row < 0) return;
#pragma unroll
    for (int r = 0; r < BS; r++)
        if (L == 1 || r % L == lane % L) y[(long long)row * BS + r] = MODE == kSpmvAssign ? fin(acc[r]) : av[r] + acc[r];
}

// w = D^-1 (b - A x) (block-Jacobi-scaled residual, the learned step's input): the residual of a
// row is reduced over the row's lanes, then lane r < BS applies row r of the row's D^-1.
template <class T, int BS, int G, int U>
__global__ void __launch_bounds__(kThreads) k_bsr_residual_dinv(int nbr, const int* __restrict__ rowptr,
                                                                const int* __restrict__ colidx,
                                                                const T* __restrict__ vals, long long ld,
                                                                const T* __restrict__ dinv, long long dld,
                                                                const T* __restrict__ x, const T* __restrict__ b,
                                                                T* __restrict__ w, int ell)
{
    pdl_wait();
    const int lane = threadIdx.x & (G - 1);
    const int row = (int)(((long long)blockIdx.x * kThreads + threadIdx.x) / G);
    T acc[BS];
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = T(0);
    T bv[BS], dv[BS];
    if (row < nbr) {
#pragma unroll
        for (int c = 0; c < BS; c++) bv[c] = b[(long long)row * BS + c];
        if (lane < BS)
#pragma unroll
            for (int c = 0; c < BS; c++) dv[c] = dinv[(long long)(lane * BS + c) * dld + row];
        int p0, p1;
        row_range(row, ell, rowptr, p0, p1);
        accumulate_row<T, BS, G, U>(p0, p1, lane, colidx, vals, ld, x, acc, UseAll());
    }
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = group_sum<G>(acc[r]);
    if (row < nbr && lane < BS) {
        T v = T(0);
#pragma unroll
        for (int c = 0; c < BS; c++) v += dv[c] * (bv[c] - acc[c]);
        w[(long long)row * BS + lane] = v;
    }
}

// One colour of block Gauss-Seidel: rows [row0, row1) are mutually uncoupled.
// x_i <- D_i^{-1} (b_i - sum_{j != i} A_ij x_j)
// Columns outside [col_lo, col_hi) are skipped: in a sweep that starts from x = 0 they hold
// zeros not yet overwritten (later colours of a forward sweep, earlier ones of a backward
// sweep), so skipping them changes no bit of the result and saves their loads. Block columns
// are sorted, so the skipped ones form a head and a tail of each row. The empty slots at the end
// of a padded (ell) row hold the row's own column and are skipped as the diagonal is; a stop on a
// column >= col_hi happens at a real block before them.
template <class T, int BS, int G, int U>
__global__ void __launch_bounds__(kThreads) k_bsr_gs(int row0, int row1, const int* __restrict__ rowptr,
                                                     const int* __restrict__ colidx,
                                                     const T* __restrict__ vals, long long ld,
                                                     const T* __restrict__ dinv, long long dld,
                                                     const T* __restrict__ b, T* x, int col_lo, int col_hi,
                                                     int ell, T omega)
{
    pdl_wait();
    const int lane = threadIdx.x & (G - 1);
    const int row = row0 + (int)(((long long)blockIdx.x * kThreads + threadIdx.x) / G);
    T acc[BS];
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = T(0);
    // b_i and the D_i^-1 row this lane applies (lane r < BS owns output r when G >= BS), loaded
    // before the row walk so that their latency overlaps it instead of following it.
    T bv[BS], dv[BS];
    if (G >= BS && row < row1) {
#pragma unroll
        for (int c = 0; c < BS; c++) bv[c] = b[(long long)row * BS + c];
        if (lane < BS)
#pragma unroll
            for (int c = 0; c < BS; c++) dv[c] = dinv[(long long)(lane * BS + c) * dld + row];
    }
    if (row < row1) {
        auto sel = [row, col_lo, col_hi](int col) -> int {
            if (col >= col_hi) return 2;
            return (col == row || col < col_lo) ? 0 : 1;
        };
        int p0, p1;
        row_range(row, ell, rowptr, p0, p1);
        accumulate_row<T, BS, G, U>(p0, p1, lane, colidx, vals, ld, x, acc, sel);
    }
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = group_sum<G>(acc[r]);
    if (row < row1) {
        if (G >= BS) {
            if (lane < BS) {
                T v = T(0);
#pragma unroll
                for (int c = 0; c < BS; c++) v = fma(dv[c], bv[c] - acc[c], v);
                const long long i = (long long)row * BS + lane;
                // block SOR: x_i <- omega D_i^-1 (b_i - sum_{j != i} A_ij x_j) + (1 - omega) x_i
                if (omega != T(1)) v = fma(omega, v, (T(1) - omega) * x[i]);
                x[i] = fin(v);
            }
        } else {
            T t[BS];
#pragma unroll
            for (int c = 0; c < BS; c++) t[c] = b[(long long)row * BS + c] - acc[c];
#pragma unroll
            for (int r = 0; r < BS; r++) {
                if (lane == r % G) {
                    T v = T(0);
#pragma unroll
                    for (int c = 0; c < BS; c++) v = fma(dinv[(long long)(r * BS + c) * dld + row], t[c], v);
                    const long long i = (long long)row * BS + r;
                    if (omega != T(1)) v = fma(omega, v, (T(1) - omega) * x[i]);
                    x[i] = fin(v);
                }
            }
        }
    }
}

// One colour of block GS over long rows (the Galerkin operators, whose rows hold 25 to 130 blocks in
// colours of tens to a thousand rows): TPR threads of a 128-thread CTA walk a row, one block each as far as
// it goes. Such a launch is bound by latency, not by bytes: a warp per row took the row's blocks 32 at a
// time, each step waiting for its columns and then for its x entries (9.5 us a colour of 40 rows of 124
// blocks in pairs). Here a thread has its block's column, values and its D^-1 row on the way before it waits
// for the kernel ahead, then one gather, the sums (shuffles, then shared memory across the row's warps) and
// the store remain. Column rules as in k_bsr_gs.
constexpr int kLongThreads = 128;

template <class T, int BS, int TPR>
__global__ void __launch_bounds__(kLongThreads) k_bsr_gs_long(int row0, int row1, const int* __restrict__ rowptr,
                                                              const int* __restrict__ colidx,
                                                              const T* __restrict__ vals, long long ld,
                                                              const T* __restrict__ dinv, long long dld,
                                                              const T* __restrict__ b, T* x, int col_lo, int col_hi, T omega)
{
    constexpr bool HOLD = BS * BS * (int)sizeof(T) <= 128;   // values in registers ahead of the wait
    constexpr int kWarps = kLongThreads / 32, kRowWarps = TPR / 32;
    __shared__ T part[kWarps][BS];
    const int tid = threadIdx.x, lane = tid % TPR;
    const int row = row0 + (int)blockIdx.x * (kLongThreads / TPR) + tid / TPR;
    const bool in = row < row1;
    int p = 0, p1 = 0;
    if (in) {
        p = rowptr[row] + lane;
        p1 = rowptr[row + 1];
    }
    int col = -1;
    T v[HOLD ? BS * BS : 1], dv[BS], bv[BS], acc[BS];
    auto load = [&]() {
        col = colidx[p];
        if (HOLD) {
#pragma unroll
            for (int e = 0; e < BS * BS; e++) v[e] = vals[(long long)e * ld + p];
        }
    };
    if (p < p1) load();
    const bool writes = in && lane < BS;
    if (writes)
#pragma unroll
        for (int c = 0; c < BS; c++) dv[c] = dinv[(long long)(lane * BS + c) * dld + row];
    pdl_wait();
    if (writes)
#pragma unroll
        for (int c = 0; c < BS; c++) bv[c] = b[(long long)row * BS + c];
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = T(0);
    while (p < p1) {
        if (col != row && col >= col_lo && col < col_hi) {
            T xv[BS];
#pragma unroll
            for (int c = 0; c < BS; c++) xv[c] = x[(long long)col * BS + c];
#pragma unroll
            for (int r = 0; r < BS; r++)
#pragma unroll
                for (int c = 0; c < BS; c++) {
                    const T a = HOLD ? v[r * BS + c] : vals[(long long)(r * BS + c) * ld + p];
                    acc[r] = fma(a, xv[c], acc[r]);
                }
        }
        p += TPR;
        if (p < p1) load();
    }
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = group_sum<32>(acc[r]);
    if (kRowWarps > 1) {
        const int warp = tid >> 5;
        if ((tid & 31) == 0)
#pragma unroll
            for (int r = 0; r < BS; r++) part[warp][r] = fin(acc[r]);
        __syncthreads();
        if (writes) {   // the row's first warp
#pragma unroll
            for (int w = 1; w < kRowWarps; w++)
#pragma unroll
                for (int r = 0; r < BS; r++) acc[r] += part[warp + w][r];
        }
    }
    if (writes) {
        T y = T(0);
#pragma unroll
        for (int c = 0; c < BS; c++) y = fma(dv[c], bv[c] - acc[c], y);
        const long long i = (long long)row * BS + lane;
        if (omega != T(1)) y = fma(omega, y, (T(1) - omega) * x[i]);   // block SOR
        x[i] = fin(y);
    }
}

// One colour of block GS on a slot-major padded view (slot_major, ell = W): one thread per block
// row. Slot s of row i of the colour [row0, row1) lives at row0 * W + s * (row1 - row0) + (i - row0),
// so a warp's loads of one slot are 32 consecutive words. The W column indices, then the used
// slots' values and x entries are loaded before the sums, so all of a row's loads are in flight
// together; no lane reduction follows. The column rules are those of k_bsr_gs (empty slots hold
// the row's own column). ZERO: a zero-start sweep, whose skipped blocks are not loaded; other
// sweeps load every slot and drop the diagonal ones by a select.
template <class T, int BS, int W, bool ZERO>
__global__ void __launch_bounds__(kThreads, 2) k_bsr_gs_slot(int row0, int row1, const int* __restrict__ colidx,
                                                            const T* __restrict__ vals, long long ld,
                                                            const T* __restrict__ dinv, long long dld,
                                                            const T* __restrict__ b, T* x, int col_lo, int col_hi,
                                                            T omega)
{
    pdl_wait();
    const int row = row0 + (int)(blockIdx.x * kThreads + threadIdx.x);
    if (row >= row1) return;
    const long long nrc = row1 - row0;
    const long long base = (long long)row0 * W + (row - row0);
    int col[W];
#pragma unroll
    for (int s = 0; s < W; s++) col[s] = colidx[base + s * nrc];
    T bv[BS], dv[BS * BS];
#pragma unroll
    for (int c = 0; c < BS; c++) bv[c] = b[(long long)row * BS + c];
#pragma unroll
    for (int e = 0; e < BS * BS; e++) dv[e] = dinv[(long long)e * dld + row];
    T acc[BS];
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = T(0);
#pragma unroll
    for (int s = 0; s < W; s++) {
        const int j = col[s];
        const bool use = j != row && (!ZERO || (j >= col_lo && j < col_hi));
        if (ZERO && !use) continue;
        const long long p = base + s * nrc;
        T xv[BS];
#pragma unroll
        for (int c = 0; c < BS; c++) xv[c] = x[(long long)j * BS + c];
#pragma unroll
        for (int r = 0; r < BS; r++)
#pragma unroll
            for (int c = 0; c < BS; c++) {
                const T a = vals[(long long)(r * BS + c) * ld + p];
                acc[r] = fma(use ? a : T(0), xv[c], acc[r]);
            }
    }
#pragma unroll
    for (int r = 0; r < BS; r++) {
        T v = T(0);
#pragma unroll
        for (int c = 0; c < BS; c++) v = fma(dv[r * BS + c], bv[c] - acc[c], v);
        const long long i = (long long)row * BS + r;
        if (omega != T(1)) v = fma(omega, v, (T(1) - omega) * x[i]);   // block SOR
        x[i] = fin(v);
    }
}

// y = A x | y = aux - A x on a slot-major padded view of all of A (slot_major, ell = W, one "colour"
// of every row): slot s of row i at s * nbr + i, one thread per block row. The W column indices,
// then every slot's values and x entries, are loaded before the sums, so all of a row's loads are in
// flight together and a warp's load of one slot is 32 consecutive values; no lane reduction follows.
// Empty slots hold zero values and a column of the row (an exact zero added). The summation order
// is block by block in column order, as in the row-major kernels.
template <class T, int BS, int W, int MODE>
__global__ void __launch_bounds__(kThreads, 2) k_bsr_spmv_slot(int nbr, const int* __restrict__ colidx,
                                                              const T* __restrict__ vals, long long ld,
                                                              const T* __restrict__ x, const T* aux, T* y)
{
    pdl_wait();
    const int row = (int)(blockIdx.x * kThreads + threadIdx.x);
    if (row >= nbr) return;
    int col[W];
#pragma unroll
    for (int k = 0; k < W; k++) col[k] = colidx[(long long)k * nbr + row];
    T av[BS];
    if (MODE != kSpmvAssign)
#pragma unroll
        for (int r = 0; r < BS; r++) av[r] = aux[(long long)row * BS + r];
    T acc[BS];
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = T(0);
#pragma unroll
    for (int k = 0; k < W; k++) {
        const long long p = (long long)k * nbr + row;
        T xv[BS];
#pragma unroll
        for (int c = 0; c < BS; c++) xv[c] = x[(long long)col[k] * BS + c];
#pragma unroll
        for (int r = 0; r < BS; r++)
#pragma unroll
            for (int c = 0; c < BS; c++) acc[r] = fma(vals[(long long)(r * BS + c) * ld + p], xv[c], acc[r]);
    }
#pragma unroll
    for (int r = 0; r < BS; r++) {
        const long long i = (long long)row * BS + r;
        if (MODE == kSpmvAssign) y[i] = fin(acc[r]);
        else if (MODE == kSpmvResidual) y[i] = av[r] - acc[r];
        else y[i] = av[r] + acc[r];
    }
}

// w = D^-1 (b - A x) on the slot-major view of all of A (the learned step's input), one thread per row.
template <class T, int BS, int W>
__global__ void __launch_bounds__(kThreads, 2) k_bsr_residual_dinv_slot(int nbr, const int* __restrict__ colidx,
                                                                       const T* __restrict__ vals, long long ld,
                                                                       const T* __restrict__ dinv, long long dld,
                                                                       const T* __restrict__ x,
                                                                       const T* __restrict__ b, T* __restrict__ w)
{
    pdl_wait();
    const int row = (int)(blockIdx.x * kThreads + threadIdx.x);
    if (row >= nbr) return;
    int col[W];
#pragma unroll
    for (int k = 0; k < W; k++) col[k] = colidx[(long long)k * nbr + row];
    T bv[BS], dv[BS * BS];
#pragma unroll
    for (int c = 0; c < BS; c++) bv[c] = b[(long long)row * BS + c];
#pragma unroll
    for (int e = 0; e < BS * BS; e++) dv[e] = dinv[(long long)e * dld + row];
    T acc[BS];
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = T(0);
#pragma unroll
    for (int k = 0; k < W; k++) {
        const long long p = (long long)k * nbr + row;
        T xv[BS];
#pragma unroll
        for (int c = 0; c < BS; c++) xv[c] = x[(long long)col[k] * BS + c];
#pragma unroll
        for (int r = 0; r < BS; r++)
#pragma unroll
            for (int c = 0; c < BS; c++) acc[r] = fma(vals[(long long)(r * BS + c) * ld + p], xv[c], acc[r]);
    }
#pragma unroll
    for (int r = 0; r < BS; r++) {
        T v = T(0);
#pragma unroll
        for (int c = 0; c < BS; c++) v = fma(dv[r * BS + c], bv[c] - acc[c], v);
        w[(long long)row * BS + r] = fin(v);
    }
}

// ---------------------------------------------------------------------------
// Row-class views. On a mesh of translated elements a block row is one of a few dozen (classes: see
// row_classes in fhg_host.h), so the values stay in L1 and only the class (2 bytes), the off-diagonal
// columns and the vectors are streamed: 62 bytes a row for an FP32 sweep with 3 x 3 blocks where the stored
// blocks take 312. One thread per block row; the column indices and then every neighbour's x entries are
// loaded before the sums, with registers for that (kClsBlocks CTAs of 128 threads per SM: at the compiler's
// own choice of 32 registers the x loads follow one another, and a launch too small to hide them
// takes twice as long). The sums run over the off-diagonal blocks in column order. What bounds a sweep now
// is the L1's rate of gathered lines (a warp's x loads of one slot touch 7 lines) and L2; FP64 stays bound
// by its pipe. 64^3, k = 1 (3.1 M rows, 77 classes), one sweep of stored blocks against classes:
// FP32 171 -> 73 us, pairs 326 -> 148 us, FP64 777 -> 413 us.
constexpr int kClsThreads = 128;

// CTAs per SM of a class kernel: 64, 80 or 128 registers, what W x BS gathered values in flight and
// 2 BS sums take (FP32 6 x 6 spills up to 40 bytes of 80 registers).
template <class T, int BS, int W>
constexpr int kClsBlocks = BS <= 3 ? 8 : sizeof(T) == 4 ? 6 : 4;

// The x entries of a row's off-diagonal slots; zeros for an empty slot (the row's own column) and, in a
// zero-start sweep, for a column outside [col_lo, col_hi).
template <class T, int BS, int W, bool ZERO>
__device__ __forceinline__ void gather_slots(const int (&col)[W], int row, int col_lo, int col_hi, const T* x, T (&xv)[W][BS])
{
#pragma unroll
    for (int s = 0; s < W; s++) {
        const int j = col[s];
        const bool use = j != row && (!ZERO || (j >= col_lo && j < col_hi));
#pragma unroll
        for (int c = 0; c < BS; c++) xv[s][c] = use ? x[(long long)j * BS + c] : T(0);
    }
}

// acc += sum over the off-diagonal slots of dict x (dict: the row's class). One thread sums a row's 21 to 42 products
// where stored blocks have eight lanes, so a running sum in pairs is normalised every second product (here and
// below): A x is then as near to exact as on eight lanes (root mean square over the rows, in 2^-47 of |A||x|: 3 x 3
// 0.28, 6 x 6 0.32; 0.45 and 0.68 without), for 1 to 4% of a cycle (48^3 k = 1 577 -> 591 us, 24^3 k = 2 442 -> 459).
template <class T, int BS, int W>
__device__ __forceinline__ void class_row(const T* __restrict__ dict, int ld, const T (&xv)[W][BS], T (&acc)[BS])
{
#pragma unroll
    for (int s = 0; s < W; s++)
#pragma unroll
        for (int r = 0; r < BS; r++)
#pragma unroll
            for (int c = 0; c < BS; c++) {
                acc[r] = fma(dict[((s * BS + r) * BS + c) * ld], xv[s][c], acc[r]);
                if (c % 2 || c + 1 == BS) acc[r] = fin(acc[r]);
            }
}

// v = M w, M the bs x bs block `slot` of the row's class.
template <class T, int BS>
__device__ __forceinline__ void class_block(const T* __restrict__ dict, int ld, int slot, const T (&w)[BS], T (&v)[BS])
{
#pragma unroll
    for (int r = 0; r < BS; r++)
#pragma unroll
        for (int c = 0; c < BS; c++) {
            v[r] = fma(dict[((slot * BS + r) * BS + c) * ld], w[c], v[r]);
            if (c % 2 || c + 1 == BS) v[r] = fin(v[r]);
        }
}

// One colour of block GS / SOR (the column rules of k_bsr_gs).
template <class T, int BS, int W, bool ZERO>
__global__ void __launch_bounds__(kClsThreads, kClsBlocks<T, BS, W>)
    k_bsr_gs_cls(int row0, int row1, int nbr, const unsigned short* __restrict__ cls, const int* __restrict__ colidx,
                 const T* __restrict__ dict, int ld, const T* __restrict__ b, T* x, int col_lo, int col_hi, T omega)
{
    const int row = row0 + (int)(blockIdx.x * kClsThreads + threadIdx.x);
    const bool in = row < row1;
    int col[W];   // the classes and columns never change after setup: read ahead of the wait
    const T* d = dict + (in ? cls[row] : 0);
#pragma unroll
    for (int s = 0; s < W; s++) col[s] = in ? colidx[(long long)s * nbr + row] : row;
    pdl_wait();
    if (!in) return;
    T xv[W][BS], t[BS], acc[BS], v[BS];
    gather_slots<T, BS, W, ZERO>(col, row, col_lo, col_hi, x, xv);
#pragma unroll
    for (int c = 0; c < BS; c++) {
        t[c] = b[(long long)row * BS + c];
        acc[c] = T(0);
        v[c] = T(0);
    }
    class_row<T, BS, W>(d, ld, xv, acc);
#pragma unroll
    for (int c = 0; c < BS; c++) t[c] = t[c] - acc[c];
    class_block<T, BS>(d, ld, W, t, v);
#pragma unroll
    for (int r = 0; r < BS; r++) {
        const long long i = (long long)row * BS + r;
        if (omega != T(1)) v[r] = fma(omega, v[r], (T(1) - omega) * x[i]);   // block SOR
        x[i] = fin(v[r]);
    }
}

// y = A x | y = aux - A x; with DINV y = D^-1 (aux - A x) (the learned step's input).
template <class T, int BS, int W, int MODE, bool DINV>
__global__ void __launch_bounds__(kClsThreads, kClsBlocks<T, BS, W>)
    k_bsr_spmv_cls(int nbr, const unsigned short* __restrict__ cls, const int* __restrict__ colidx,
                   const T* __restrict__ dict, int ld, const T* __restrict__ x, const T* aux, T* y)
{
    const int row = (int)(blockIdx.x * kClsThreads + threadIdx.x);
    const bool in = row < nbr;
    int col[W];
    const T* d = dict + (in ? cls[row] : 0);
#pragma unroll
    for (int s = 0; s < W; s++) col[s] = in ? colidx[(long long)s * nbr + row] : row;
    pdl_wait();
    if (!in) return;
    T xv[W][BS], xd[BS], acc[BS], av[BS];
    gather_slots<T, BS, W, false>(col, row, 0, 0, x, xv);
#pragma unroll
    for (int c = 0; c < BS; c++) {
        xd[c] = x[(long long)row * BS + c];
        av[c] = MODE == kSpmvAssign ? T(0) : aux[(long long)row * BS + c];
        acc[c] = T(0);
    }
    class_row<T, BS, W>(d, ld, xv, acc);
    class_block<T, BS>(d, ld, W + 1, xd, acc);
    if (DINV) {
        T v[BS];
#pragma unroll
        for (int c = 0; c < BS; c++) {
            av[c] = av[c] - acc[c];
            v[c] = T(0);
        }
        class_block<T, BS>(d, ld, W, av, v);
#pragma unroll
        for (int r = 0; r < BS; r++) y[(long long)row * BS + r] = fin(v[r]);
        return;
    }
#pragma unroll
    for (int r = 0; r < BS; r++) y[(long long)row * BS + r] = MODE == kSpmvAssign ? fin(acc[r]) : av[r] - acc[r];
}

// The same with one output per lane (BS lanes a row, 32 / BS rows a warp), for launches whose rows leave the
// GPU's 608 schedulers a warp or less each: a thread per row is then one long chain (63 multiply-adds
// with 3 x 3 blocks: 64 cycles each in FP64, 13 instructions in pairs), here a BS-th of it. The neighbours' x
// entries are loaded by every lane of the row (one request); t = b - A x goes round by shuffles for D^-1.
__device__ __forceinline__ float lane_value(float v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ double lane_value(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ dfl lane_value(dfl v, int lane)
{
    return dfl(__shfl_sync(0xffffffffu, v.h, lane), __shfl_sync(0xffffffffu, v.l, lane));
}

template <class T, int BS, int W>
struct ClassLane {
    static constexpr int kRows = 32 / BS;   // rows of a warp
    int row, r, first;                      // row, output, first lane of the row
    bool in;
    int col[W];
    const T* d;   // dictionary entry (0, r, 0) of the row's class

    __device__ __forceinline__ ClassLane(int row0, int row1, int nbr, const unsigned short* __restrict__ cls,
                                         const int* __restrict__ colidx, const T* __restrict__ dict, int ld)
    {
        const int lane = threadIdx.x & 31, q = lane / BS;
        row = row0 + (int)((blockIdx.x * kClsThreads + threadIdx.x) >> 5) * kRows + q;
        r = lane - q * BS;
        first = q * BS;
        in = q < kRows && row < row1;
        d = dict + (in ? cls[row] : 0) + r * BS * ld;
#pragma unroll
        for (int s = 0; s < W; s++) col[s] = in ? colidx[(long long)s * nbr + row] : row;
    }
    // Output r of block `slot` times w.
    __device__ __forceinline__ T block(int ld, int slot, const T (&w)[BS], T acc) const
    {
#pragma unroll
        for (int c = 0; c < BS; c++) {
            acc = fma(d[(slot * BS * BS + c) * ld], w[c], acc);
            if (c % 2 || c + 1 == BS) acc = fin(acc);
        }
        return acc;
    }
};

template <class T, int BS, int W, bool ZERO>
__global__ void __launch_bounds__(kClsThreads, kClsBlocks<T, BS, W>)
    k_bsr_gs_cls_lanes(int row0, int row1, int nbr, const unsigned short* __restrict__ cls, const int* __restrict__ colidx,
                       const T* __restrict__ dict, int ld, const T* __restrict__ b, T* x, int col_lo, int col_hi, T omega)
{
    const ClassLane<T, BS, W> L(row0, row1, nbr, cls, colidx, dict, ld);
    pdl_wait();
    const long long i = (long long)L.row * BS + L.r;
    T xv[W][BS], t[BS], acc = T(0);
    gather_slots<T, BS, W, ZERO>(L.col, L.row, col_lo, col_hi, x, xv);
    const T bv = L.in ? b[i] : T(0);
    if (L.in)
#pragma unroll
        for (int s = 0; s < W; s++) acc = L.block(ld, s, xv[s], acc);
    acc = bv - acc;
#pragma unroll
    for (int c = 0; c < BS; c++) t[c] = lane_value(acc, L.first + c);
    if (!L.in) return;
    T v = L.block(ld, W, t, T(0));
    if (omega != T(1)) v = fma(omega, v, (T(1) - omega) * x[i]);   // block SOR
    x[i] = fin(v);
}

template <class T, int BS, int W, int MODE>
__global__ void __launch_bounds__(kClsThreads, kClsBlocks<T, BS, W>)
    k_bsr_spmv_cls_lanes(int nbr, const unsigned short* __restrict__ cls, const int* __restrict__ colidx,
                         const T* __restrict__ dict, int ld, const T* __restrict__ x, const T* aux, T* y)
{
    const ClassLane<T, BS, W> L(0, nbr, nbr, cls, colidx, dict, ld);
    pdl_wait();
    if (!L.in) return;
    const long long i = (long long)L.row * BS + L.r;
    T xv[W][BS], xd[BS], acc = T(0);
    gather_slots<T, BS, W, false>(L.col, L.row, 0, 0, x, xv);
#pragma unroll
    for (int c = 0; c < BS; c++) xd[c] = x[(long long)L.row * BS + c];
    const T av = MODE == kSpmvAssign ? T(0) : aux[i];
#pragma unroll
    for (int s = 0; s < W; s++) acc = L.block(ld, s, xv[s], acc);
    acc = L.block(ld, W + 1, xd, acc);
    y[i] = MODE == kSpmvAssign ? fin(acc) : av - acc;
}

// Block Jacobi: xnew_i = D_i^{-1} (omega b_i + (1-omega) D_i xold_i - omega sum_{j!=i} A_ij xold_j)
template <class T, int BS, int G>
__global__ void __launch_bounds__(kThreads) k_bsr_jacobi(int nbr, const int* __restrict__ rowptr,
                                                         const int* __restrict__ colidx,
                                                         const T* __restrict__ vals, long long ld,
                                                         const T* __restrict__ dinv, long long dld, T omega,
                                                         const T* __restrict__ b, const T* __restrict__ xold,
                                                         T* __restrict__ xnew)
{
    pdl_wait();
    const int lane = threadIdx.x & (G - 1);
    const int row = (int)(((long long)blockIdx.x * kThreads + threadIdx.x) / G);
    T off[BS], dia[BS];
#pragma unroll
    for (int r = 0; r < BS; r++) { off[r] = T(0); dia[r] = T(0); }
    if (row < nbr) {
        const int p1 = rowptr[row + 1];
        for (int p = rowptr[row] + lane; p < p1; p += G) {
            const int col = colidx[p];
            T xv[BS];
#pragma unroll
            for (int c = 0; c < BS; c++) xv[c] = xold[(long long)col * BS + c];
            if (col == row) {
#pragma unroll
                for (int r = 0; r < BS; r++)
#pragma unroll
                    for (int c = 0; c < BS; c++) dia[r] = fma(vals[(long long)(r * BS + c) * ld + p], xv[c], dia[r]);
            } else {
#pragma unroll
                for (int r = 0; r < BS; r++)
#pragma unroll
                    for (int c = 0; c < BS; c++) off[r] = fma(vals[(long long)(r * BS + c) * ld + p], xv[c], off[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < BS; r++) { off[r] = group_sum<G>(off[r]); dia[r] = group_sum<G>(dia[r]); }
    if (row < nbr) {
        T t[BS];
#pragma unroll
        for (int c = 0; c < BS; c++)
            t[c] = omega * b[(long long)row * BS + c] + (T(1) - omega) * dia[c] - omega * off[c];
#pragma unroll
        for (int r = 0; r < BS; r++) {
            if (lane == r % G) {
                T v = T(0);
#pragma unroll
                for (int c = 0; c < BS; c++) v = fma(dinv[(long long)(r * BS + c) * dld + row], t[c], v);
                xnew[(long long)row * BS + r] = fin(v);
            }
        }
    }
}

// x = Cinv b, one warp per row, FP64 accumulation.
template <class T>
__global__ void __launch_bounds__(kThreads) k_coarse(int n, const double* __restrict__ cinv,
                                                     const T* __restrict__ b, T* __restrict__ x)
{
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int row = (blockIdx.x * kThreads + threadIdx.x) >> 5;
    if (row >= n) return;  // whole warps exit together
    const double* a = cinv + (long long)row * n;
    double acc = 0.0;
    for (int j = lane; j < n; j += 32) acc = fma(a[j], (double)b[j], acc);
    acc = warp_sum(acc);
    if (lane == 0) x[row] = (T)acc;
}

// Up to three dot products in one pass (K-cycle): partials[q * kReduceCtas + cta] of a_q . b_q,
// FP64 accumulation whatever T.
template <class T>
__global__ void __launch_bounds__(kReduceThreads) k_dots3(long long n, int nq, const T* __restrict__ a0,
                                                          const T* __restrict__ b0, const T* __restrict__ a1,
                                                          const T* __restrict__ b1, const T* __restrict__ a2,
                                                          const T* __restrict__ b2, double* __restrict__ partials)
{
    pdl_wait();
    double v0 = 0.0, v1 = 0.0, v2 = 0.0;
    struct E {
        T a0, b0, a1, b1, a2, b2;
    };
    for_each_element(
        n,
        [&](long long i) {
            E e{a0[i], b0[i], T(0), T(0), T(0), T(0)};
            if (nq > 1) { e.a1 = a1[i]; e.b1 = b1[i]; }
            if (nq > 2) { e.a2 = a2[i]; e.b2 = b2[i]; }
            return e;
        },
        [&](long long, const E& e) {
            v0 = fma((double)e.a0, (double)e.b0, v0);
            if (nq > 1) v1 = fma((double)e.a1, (double)e.b1, v1);
            if (nq > 2) v2 = fma((double)e.a2, (double)e.b2, v2);
        });
    double s[3] = {v0, v1, v2};
    block_sums(s);
    if (threadIdx.x < nq) partials[threadIdx.x * kReduceCtas + blockIdx.x] = threadIdx.x == 0 ? s[0] : threadIdx.x == 1 ? s[1] : s[2];
}

// y += alpha x; out = a c + b d (K-cycle updates, coefficients from the host).
template <class T>
__global__ void k_axpy(long long n, double alpha, const T* __restrict__ x, T* __restrict__ y)
{
    pdl_wait();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = y[i] + (T)alpha * x[i];
}

template <class T>
__global__ void k_lincomb(long long n, double a, const T* __restrict__ c, double b, const T* __restrict__ d,
                          T* __restrict__ out)
{
    pdl_wait();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = (T)a * c[i] + (T)b * d[i];
}

template <class Tin, class Tout>
__global__ void __launch_bounds__(kThreads) k_convert(long long n, const Tin* __restrict__ in, Tout* __restrict__ out)
{
    pdl_wait();
    const long long i = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (i < n) out[i] = (Tout)in[i];
}

template <class T>
__global__ void __launch_bounds__(kThreads) k_permute(int nb, int bs, const int* __restrict__ perm,
                                                      const T* __restrict__ in, T* __restrict__ out, int gather)
{
    pdl_wait();
    const long long i = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (i >= (long long)nb * bs) return;
    const int blk = (int)(i / bs), c = (int)(i - (long long)blk * bs);
    const long long o = (long long)perm[blk] * bs + c;
    if (gather) out[i] = in[o];
    else out[o] = in[i];
}

// The natural injection between two face degrees on the same faces (P_LevelForHHO::SetupProlongation,
// src/Solver/Multigrid/MultigridForHHO/P_MultigridForHHO.h:69-92): fine face block i (nh unknowns)
// is coarse block map[i] (nl < nh unknowns, the first nl functions of the hierarchical face basis).
// Restriction by P^T: out[map[i] * nl + q] = in[i * nh + q] for q < nl.
template <class T>
__global__ void __launch_bounds__(kThreads) k_inject_restrict(int nb, int nh, int nl, const int* __restrict__ map,
                                                              const T* __restrict__ in, T* __restrict__ out)
{
    pdl_wait();
    const long long i = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (i >= (long long)nb * nl) return;
    const int blk = (int)(i / nl), q = (int)(i - (long long)blk * nl);
    out[(long long)map[blk] * nl + q] = in[(long long)blk * nh + q];
}

// Prolongation by P: out[i * nh + q] = aux[i * nh + q] + (q < nl ? in[map[i] * nl + q] : 0), aux NULL
// reading as zero; out may be aux. The one entry of P is 1, so this is the product's arithmetic.
template <class T>
__global__ void __launch_bounds__(kThreads) k_inject_prolong(int nb, int nh, int nl, const int* __restrict__ map,
                                                             const T* __restrict__ in, const T* aux, T* out)
{
    pdl_wait();
    const long long i = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (i >= (long long)nb * nh) return;
    const int blk = (int)(i / nh), q = (int)(i - (long long)blk * nh);
    if (q < nl) {
        const T e = in[(long long)map[blk] * nl + q];
        out[i] = aux ? aux[i] + e : e;
    } else {
        out[i] = aux ? aux[i] : T(0);
    }
}

inline unsigned grid_for(long long work, int per_cta)
{
    long long g = (work + per_cta - 1) / per_cta;
    return (unsigned)(g > 0 ? g : 1);
}

}  // namespace

#define FHG_DISPATCH_BS_G(BSV, GV, ...)                                              \
    switch (BSV) {                                                                    \
    case 2: FHG_DISPATCH_G(2, GV, __VA_ARGS__); break;                                       \
    case 3: FHG_DISPATCH_G(3, GV, __VA_ARGS__); break;                                       \
    case 4: FHG_DISPATCH_G(4, GV, __VA_ARGS__); break;                                       \
    case 6: FHG_DISPATCH_G(6, GV, __VA_ARGS__); break;                                       \
    default: break;                                                                   \
    }
#define FHG_DISPATCH_G(BS_, GV, ...)                                                 \
    switch (GV) {                                                                     \
    case 4: { constexpr int BS = BS_, G = 4; __VA_ARGS__; } break;                          \
    case 8: { constexpr int BS = BS_, G = 8; __VA_ARGS__; } break;                          \
    case 16: { constexpr int BS = BS_, G = 16; __VA_ARGS__; } break;                        \
    default: { constexpr int BS = BS_, G = 32; __VA_ARGS__; } break;                        \
    }

template <class T, int BS, int G, int U>
void spmv_u(const BsrView<T>& A, unsigned grid, int mode, const T* x, const T* aux, T* y, cudaStream_t s)
{
    if (mode == kSpmvAssign)
        pdl_launch(k_bsr_spmv<T, BS, G, U, kSpmvAssign>, grid, kThreads, 0, s, A.nbr, A.rowptr, A.colidx, A.vals, A.ld, x, aux, y,
                   A.ell);
    else if (mode == kSpmvResidual)
        pdl_launch(k_bsr_spmv<T, BS, G, U, kSpmvResidual>, grid, kThreads, 0, s, A.nbr, A.rowptr, A.colidx, A.vals, A.ld, x, aux, y,
                   A.ell);
    else
        pdl_launch(k_bsr_spmv<T, BS, G, U, kSpmvAddTo>, grid, kThreads, 0, s, A.nbr, A.rowptr, A.colidx, A.vals, A.ld, x, aux, y,
                   A.ell);
}

// Slot-major products: dispatch on the block size and the slot count W (5..8).
template <class T, int BS, int W>
void spmv_slot_shape(const BsrView<T>& A, unsigned grid, int mode, const T* x, const T* aux, T* y, cudaStream_t s)
{
    if (mode == kSpmvAssign)
        pdl_launch(k_bsr_spmv_slot<T, BS, W, kSpmvAssign>, grid, kThreads, 0, s, A.nbr, A.colidx, A.vals, A.ld, x,
                   aux, y);
    else if (mode == kSpmvResidual)
        pdl_launch(k_bsr_spmv_slot<T, BS, W, kSpmvResidual>, grid, kThreads, 0, s, A.nbr, A.colidx, A.vals, A.ld, x,
                   aux, y);
    else
        pdl_launch(k_bsr_spmv_slot<T, BS, W, kSpmvAddTo>, grid, kThreads, 0, s, A.nbr, A.colidx, A.vals, A.ld, x,
                   aux, y);
}

template <class T, int BS>
void spmv_slot_w(const BsrView<T>& A, unsigned grid, int mode, const T* x, const T* aux, T* y, cudaStream_t s)
{
    switch (A.ell) {
    case 5: spmv_slot_shape<T, BS, 5>(A, grid, mode, x, aux, y, s); break;
    case 6: spmv_slot_shape<T, BS, 6>(A, grid, mode, x, aux, y, s); break;
    case 7: spmv_slot_shape<T, BS, 7>(A, grid, mode, x, aux, y, s); break;
    case 8: spmv_slot_shape<T, BS, 8>(A, grid, mode, x, aux, y, s); break;
    default: break;   // setup builds slot-major product views for W in 5..8 only
    }
}

// Row-class views: dispatch on the block size and the slot count (setup builds 4 and 6).
#define FHG_DISPATCH_CLS(BSV, WV, ...)                                     \
    switch (BSV * 10 + WV) {                                               \
    case 24: { constexpr int BS = 2, W = 4; __VA_ARGS__; } break;          \
    case 26: { constexpr int BS = 2, W = 6; __VA_ARGS__; } break;          \
    case 34: { constexpr int BS = 3, W = 4; __VA_ARGS__; } break;          \
    case 36: { constexpr int BS = 3, W = 6; __VA_ARGS__; } break;          \
    case 44: { constexpr int BS = 4, W = 4; __VA_ARGS__; } break;          \
    case 46: { constexpr int BS = 4, W = 6; __VA_ARGS__; } break;          \
    case 64: { constexpr int BS = 6, W = 4; __VA_ARGS__; } break;          \
    case 66: { constexpr int BS = 6, W = 6; __VA_ARGS__; } break;          \
    default: break;                                                        \
    }

template <class T, int BS>
void sell_bs(const BsrView<T>& A, int mode, const T* x, const T* aux, T* y, cudaStream_t s)
{
    const int rows = 32 / A.sell_lanes, slices = (A.nbr + rows - 1) / rows;
    const unsigned grid = grid_for(32LL * slices, kThreads);
    auto go = [&](auto kernel) {
        pdl_launch(kernel, grid, kThreads, 0, s, slices, A.sell_perm, A.sell_ptr, A.colidx, A.vals, A.ld, x, aux, y);
    };
    if (A.sell_lanes == 8) go(k_bsr_spmv_sell<T, BS, kSpmvAssign, 8>);
    else if (A.sell_lanes == 4) go(k_bsr_spmv_sell<T, BS, kSpmvAssign, 4>);
    else if (mode == kSpmvAssign) go(k_bsr_spmv_sell<T, BS, kSpmvAssign, 1>);
    else go(k_bsr_spmv_sell<T, BS, kSpmvAddTo, 1>);
}

// Rows up to which a launch on a row-class view takes one output per lane: 24,576 in FP64 and pairs, 12,288
// in FP32 (a thread per row gives the 608 schedulers 1.3 and 0.6 warps each there). us a sweep, a thread per row against
// a lane per output, at rows a colour: FP64 3 x 3 1,150: 20 / 14, 9,500: 22 / 18, 77,000: 61 / 70; pairs 3 x 3
// 4,000: 15 / 11, 32,000: 19 / 19; pairs 6 x 6 9,500: 40 / 23; FP32 3 x 3 9,500: 10.2 / 9.4, 77,000: 15 / 20;
// FP32 6 x 6 4,000: 22 / 12, 32,000: 30 / 32.
template <class T>
constexpr int kClsLaneRows = sizeof(T) == 4 ? 12288 : 24576;

template <int BS>
unsigned class_lanes_grid(int rows) { return grid_for(rows, kClsThreads / 32 * (32 / BS)); }

template <class T>
void launch_spmv(const BsrView<T>& A, int mode, const T* x, const T* aux, T* y, cudaStream_t s)
{
    if (A.nbr == 0) return;
    if (A.cls) {   // operators only (assign, residual)
        const bool lanes = A.nbr <= kClsLaneRows<T>;
        FHG_DISPATCH_CLS(A.bs, A.ell, {
            const unsigned grid = lanes ? class_lanes_grid<BS>(A.nbr) : grid_for(A.nbr, kClsThreads);
            if (lanes && mode == kSpmvAssign)
                pdl_launch(k_bsr_spmv_cls_lanes<T, BS, W, kSpmvAssign>, grid, kClsThreads, 0, s, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, x, aux, y);
            else if (lanes)
                pdl_launch(k_bsr_spmv_cls_lanes<T, BS, W, kSpmvResidual>, grid, kClsThreads, 0, s, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, x, aux, y);
            else if (mode == kSpmvAssign)
                pdl_launch(k_bsr_spmv_cls<T, BS, W, kSpmvAssign, false>, grid, kClsThreads, 0, s, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, x, aux, y);
            else
                pdl_launch(k_bsr_spmv_cls<T, BS, W, kSpmvResidual, false>, grid, kClsThreads, 0, s, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, x, aux, y);
        });
        g_kernel_launches++;
        return;
    }
    if (A.sell_perm) {
        // sliced views exist only for the transfers; they have no row pointers to fall back on
        if (mode != kSpmvAssign && (mode != kSpmvAddTo || A.sell_lanes != 1)) return;
        switch (A.bs) {
        case 2: sell_bs<T, 2>(A, mode, x, aux, y, s); break;
        case 3: sell_bs<T, 3>(A, mode, x, aux, y, s); break;
        case 4: sell_bs<T, 4>(A, mode, x, aux, y, s); break;
        case 6: sell_bs<T, 6>(A, mode, x, aux, y, s); break;
        default: break;
        }
        g_kernel_launches++;
        return;
    }
    if constexpr (!std::is_same<T, double>::value) {
        if (A.slot_major) {   // FP32 and pair product views (no FP64 slot-major view is built)
            const unsigned grid = grid_for(A.nbr, kThreads);
            switch (A.bs) {
            case 2: spmv_slot_w<T, 2>(A, grid, mode, x, aux, y, s); break;
            case 3: spmv_slot_w<T, 3>(A, grid, mode, x, aux, y, s); break;
            case 4: spmv_slot_w<T, 4>(A, grid, mode, x, aux, y, s); break;
            case 6: spmv_slot_w<T, 6>(A, grid, mode, x, aux, y, s); break;
            default: break;
            }
            g_kernel_launches++;
            return;
        }
    }
    // (the grid follows the dispatched lane count G, so every row is covered whatever A.lanes says)
    FHG_DISPATCH_BS_G(A.bs, A.lanes, {
        const unsigned grid = grid_for((long long)A.nbr * G, kThreads);
        if (A.unroll == 2) spmv_u<T, BS, G, 2>(A, grid, mode, x, aux, y, s);
        else spmv_u<T, BS, G, 1>(A, grid, mode, x, aux, y, s);
    });
    g_kernel_launches++;
}

// Slot-major sweeps: dispatch on the block size and the slot count W (4..8).
template <class T, int BS, int W>
void gs_slot_shape(const BsrView<T>& A, unsigned grid, int row0, int row1, const T* dinv, long long dld,
                   const T* b, T* x, cudaStream_t s, int col_lo, int col_hi, T omega)
{
    if (col_lo > 0 || col_hi < 0x7fffffff)
        pdl_launch(k_bsr_gs_slot<T, BS, W, true>, grid, kThreads, 0, s, row0, row1, A.colidx, A.vals, A.ld, dinv,
                   dld, b, x, col_lo, col_hi, omega);
    else
        pdl_launch(k_bsr_gs_slot<T, BS, W, false>, grid, kThreads, 0, s, row0, row1, A.colidx, A.vals, A.ld, dinv,
                   dld, b, x, col_lo, col_hi, omega);
}

template <class T, int BS>
void gs_slot_w(const BsrView<T>& A, unsigned grid, int row0, int row1, const T* dinv, long long dld,
               const T* b, T* x, cudaStream_t s, int col_lo, int col_hi, T omega)
{
    switch (A.ell) {
    case 4: gs_slot_shape<T, BS, 4>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 5: gs_slot_shape<T, BS, 5>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 6: gs_slot_shape<T, BS, 6>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 7: gs_slot_shape<T, BS, 7>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 8: gs_slot_shape<T, BS, 8>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    default: break;   // setup builds slot-major views for W in 4..8 only
    }
}

template <class T>
void launch_gs_slot(const BsrView<T>& A, int row0, int row1, const T* dinv, long long dld, const T* b,
                    T* x, cudaStream_t s, int col_lo, int col_hi, T omega)
{
    const unsigned grid = grid_for((long long)(row1 - row0), kThreads);
    switch (A.bs) {
    case 2: gs_slot_w<T, 2>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 3: gs_slot_w<T, 3>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 4: gs_slot_w<T, 4>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 6: gs_slot_w<T, 6>(A, grid, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    default: break;
    }
}

// Threads per row of k_bsr_gs_long: one block to a thread, but a single warp per row where the colour's rows
// fill the GPU by themselves (16 CTAs of 128 threads per SM).
template <class T, int BS>
void gs_long_bs(const BsrView<T>& A, int row0, int row1, const T* dinv, long long dld, const T* b, T* x, cudaStream_t s,
                int col_lo, int col_hi, T omega)
{
    const double mean = (double)A.nnzb / A.nbr;
    const int rows = row1 - row0;
    const int tpr = rows > 152 * 16 * 4 || mean <= 32.0 ? 32 : mean <= 64.0 ? 64 : 128;
    const unsigned grid = grid_for((long long)rows * tpr, kLongThreads);
    auto go = [&](auto kernel) {
        pdl_launch(kernel, grid, kLongThreads, 0, s, row0, row1, A.rowptr, A.colidx, A.vals, A.ld, dinv, dld, b, x, col_lo,
                   col_hi, omega);
    };
    if (tpr == 32) go(k_bsr_gs_long<T, BS, 32>);
    else if (tpr == 64) go(k_bsr_gs_long<T, BS, 64>);
    else go(k_bsr_gs_long<T, BS, 128>);
}

template <class T>
void gs_long(const BsrView<T>& A, int row0, int row1, const T* dinv, long long dld, const T* b, T* x, cudaStream_t s,
             int col_lo, int col_hi, T omega)
{
    switch (A.bs) {
    case 2: gs_long_bs<T, 2>(A, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 3: gs_long_bs<T, 3>(A, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 4: gs_long_bs<T, 4>(A, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    case 6: gs_long_bs<T, 6>(A, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega); break;
    default: break;
    }
}

template <class T>
void launch_gs(const BsrView<T>& A, int row0, int row1, const T* dinv, long long dld, const T* b, T* x, cudaStream_t s,
               int col_lo, int col_hi, T omega)
{
    if (row1 <= row0) return;
    if (A.cls) {
        const int rows = row1 - row0;
        const bool lanes = rows <= kClsLaneRows<T>, zero = col_lo > 0 || col_hi < 0x7fffffff;
        FHG_DISPATCH_CLS(A.bs, A.ell, {
            const unsigned grid = lanes ? class_lanes_grid<BS>(rows) : grid_for(rows, kClsThreads);
            if (lanes && zero)
                pdl_launch(k_bsr_gs_cls_lanes<T, BS, W, true>, grid, kClsThreads, 0, s, row0, row1, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, b, x, col_lo, col_hi, omega);
            else if (lanes)
                pdl_launch(k_bsr_gs_cls_lanes<T, BS, W, false>, grid, kClsThreads, 0, s, row0, row1, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, b, x, col_lo, col_hi, omega);
            else if (zero)
                pdl_launch(k_bsr_gs_cls<T, BS, W, true>, grid, kClsThreads, 0, s, row0, row1, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, b, x, col_lo, col_hi, omega);
            else
                pdl_launch(k_bsr_gs_cls<T, BS, W, false>, grid, kClsThreads, 0, s, row0, row1, A.nbr, A.cls, A.colidx,
                           A.vals, (int)A.ld, b, x, col_lo, col_hi, omega);
        });
        g_kernel_launches++;
        return;
    }
    if constexpr (!std::is_same<T, double>::value) {
        if (A.slot_major) {   // FP32 and pair views (setup builds no FP64 slot-major view)
            launch_gs_slot<T>(A, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega);
            g_kernel_launches++;
            return;
        }
    }
    if (A.lanes == 32 && A.ell == 0) {   // long rows
        gs_long<T>(A, row0, row1, dinv, dld, b, x, s, col_lo, col_hi, omega);
        g_kernel_launches++;
        return;
    }
    FHG_DISPATCH_BS_G(A.bs, A.lanes, {
        const unsigned grid = grid_for((long long)(row1 - row0) * G, kThreads);
        if (A.unroll == 2)
            pdl_launch(k_bsr_gs<T, BS, G, 2>, grid, kThreads, 0, s, row0, row1, A.rowptr, A.colidx, A.vals, A.ld, dinv,
                       dld, b, x, col_lo, col_hi, A.ell, omega);
        else
            pdl_launch(k_bsr_gs<T, BS, G, 1>, grid, kThreads, 0, s, row0, row1, A.rowptr, A.colidx, A.vals, A.ld, dinv,
                       dld, b, x, col_lo, col_hi, A.ell, omega);
    });
    g_kernel_launches++;
}

template <class T>
void launch_jacobi(const BsrView<T>& A, const T* dinv, long long dld, T omega, const T* b, const T* xold, T* xnew,
                   cudaStream_t s)
{
    if (A.nbr == 0 || A.ell > 0) return;   // the Jacobi row walk needs the row pointers (callers pass A)
    FHG_DISPATCH_BS_G(A.bs, A.lanes, {
        const unsigned grid = grid_for((long long)A.nbr * G, kThreads);
        pdl_launch(k_bsr_jacobi<T, BS, G>, grid, kThreads, 0, s, A.nbr, A.rowptr, A.colidx, A.vals, A.ld, dinv, dld, omega, b,
                                                         xold, xnew);
    });
    g_kernel_launches++;
}

template <class T>
void launch_coarse(int n, const double* cinv, const T* b, T* x, cudaStream_t s)
{
    pdl_launch(k_coarse<T>, grid_for((long long)n * 32, kThreads), kThreads, 0, s, n, cinv, b, x);
    g_kernel_launches++;
}

template <class T>
void launch_dots3(long long n, int nq, const T* a0, const T* b0, const T* a1, const T* b1, const T* a2, const T* b2,
                  double* partials, cudaStream_t s)
{
    pdl_launch(k_dots3<T>, kReduceCtas, kReduceThreads, 0, s, n, nq, a0, b0, a1 ? a1 : a0, b1 ? b1 : b0, a2 ? a2 : a0,
                                                      b2 ? b2 : b0, partials);
    g_kernel_launches++;
}

template <class T>
void launch_axpy(long long n, double alpha, const T* x, T* y, cudaStream_t s)
{
    const long long blocks = std::min<long long>((n + 255) / 256, 4 * 152);
    pdl_launch(k_axpy<T>, (unsigned)std::max<long long>(blocks, 1), 256, 0, s, n, alpha, x, y);
    g_kernel_launches++;
}

template <class T>
void launch_lincomb(long long n, double a, const T* c, double b, const T* d, T* out, cudaStream_t s)
{
    const long long blocks = std::min<long long>((n + 255) / 256, 4 * 152);
    pdl_launch(k_lincomb<T>, (unsigned)std::max<long long>(blocks, 1), 256, 0, s, n, a, c, b, d, out);
    g_kernel_launches++;
}

template <class Tin, class Tout>
void launch_convert(long long n, const Tin* in, Tout* out, cudaStream_t s)
{
    if (n == 0) return;
    pdl_launch(k_convert<Tin, Tout>, grid_for(n, kThreads), kThreads, 0, s, n, in, out);
    g_kernel_launches++;
}

template <class T>
void launch_permute(int nb, int bs, const int* perm, const T* in, T* out, bool gather, cudaStream_t s)
{
    if (nb == 0) return;
    pdl_launch(k_permute<T>, grid_for((long long)nb * bs, kThreads), kThreads, 0, s, nb, bs, perm, in, out, gather ? 1 : 0);
    g_kernel_launches++;
}

template <class T>
void launch_inject(int nb, int nh, int nl, const int* map, const T* in, const T* aux, T* out, bool prolong,
                   cudaStream_t s)
{
    if (nb == 0) return;
    if (prolong)
        pdl_launch(k_inject_prolong<T>, grid_for((long long)nb * nh, kThreads), kThreads, 0, s, nb, nh, nl, map, in,
                   aux, out);
    else
        pdl_launch(k_inject_restrict<T>, grid_for((long long)nb * nl, kThreads), kThreads, 0, s, nb, nh, nl, map, in,
                   out);
    g_kernel_launches++;
}

}  // namespace fhg

// The coarse part of a multigrid cycle in one kernel launch.
//
// Below some level the operators are small (thousands of block rows) and a cycle there is a long chain
// of short phases: every colour of every smoothing sweep, the residual, the restriction, the coarsest
// solve, the prolongation. Launched one kernel per phase, each costs 1.7 us or more (2.5 in pairs) while its
// work takes a fraction of that. Here one thread-block cluster (8 or 16 CTAs, co-scheduled by the
// hardware) runs the whole sub-cycle: every phase spreads its rows over the CTAs, and phases are separated
// by the hardware cluster barrier. The barrier cannot wait forever: all CTAs of a cluster are resident
// together and every thread takes the same path through the cycle.
//
// The vectors x, b and r of every level live in the cluster's distributed shared memory, so what one phase
// writes the next reads without a trip through L2: a store to global memory, the release and the load back
// take 0.9 us between two barriers, through distributed shared memory 0.4 us (measured, 512-thread CTAs; the
// barrier alone 0.24 us, with 8 CTAs as with 16). Block row i belongs to one CTA (chunks of kChunk rows dealt
// out in turn), which holds its entries and computes it; only the entries of other rows that a row walk
// gathers are remote. Matrix data stays in L2 and never changes: row bounds are loaded two phases ahead and
// block columns one, so that a phase waits for one round trip (values, D^-1 and the gathered entries
// together), the sums and the barrier. A block row is walked by a group of 2 to 32 threads, partial sums
// added by shuffles; warps without a row of the phase go straight to the barrier. The cycle runs as a loop
// over levels with a count of coarse corrections per level (no device recursion, so the stack is fixed at
// compile time).
//
// The arithmetic is the multigrid cycle of Multigrid::MultigridCycle (src/Solver/Multigrid/
// Multigrid.h:438-608) on the levels it covers: block Gauss-Seidel / SOR sweeps in colour order
// (BlockGaussSeidel.h:84-120, BlockSOR.h:199-227), r = b - A x (Multigrid.h:478), R r (Level.h:139-143),
// the coarse correction (V, or W with WLoops: repeated on the same right-hand side, except directly
// above the coarsest level), the coarsest dense solve, x += P e (Level.h:150-154, Multigrid.h:554).
// The FP32 and pair (dfl) value types are instantiated: in FP64 the phases are bound by the FP64 pipe of the
// cluster's SMs, and the launches are faster.
#include "fhg_coarse.h"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace fhg {

namespace {

// Every thread of the cluster arrives (release) when its writes of a phase are done and waits (acquire)
// before it reads what others wrote; the non-aligned form does not require the threads of a warp to
// arrive together. Each arrive is followed by exactly one wait.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }

__device__ __forceinline__ void pdl_wait_coarse() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Sum over the g lanes of a group (g a power of two <= 32; every lane of the warp calls it).
__device__ __forceinline__ float lanes_sum(float v, int g)
{
    for (int o = g >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, g);
    return v;
}

__device__ __forceinline__ dfl lanes_sum(dfl v, int g)
{
    for (int o = g >> 1; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, v.h, o, g);
        const float ol = __shfl_xor_sync(0xffffffffu, v.l, o, g);
        df_add(v.h, v.l, oh, ol);
    }
    return v;
}

__device__ __forceinline__ double lanes_sum(double v, int g)
{
    for (int o = g >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, g);
    return v;
}

// One block's BS values from distributed shared memory (address of the CTA that holds them, aligned to
// their own size), in the widest loads their size allows. Volatile: not moved across the barrier.
template <class T, int BS>
__device__ __forceinline__ void load_remote(unsigned addr, T (&out)[BS])
{
    constexpr int kBytes = BS * (int)sizeof(T);
    float f[kBytes / 4];
    if constexpr (kBytes % 16 == 0) {
#pragma unroll
        for (int q = 0; q < kBytes / 16; q++)
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                         : "=f"(f[4 * q]), "=f"(f[4 * q + 1]), "=f"(f[4 * q + 2]), "=f"(f[4 * q + 3]) : "r"(addr + 16 * q));
    } else if constexpr (kBytes % 8 == 0) {
#pragma unroll
        for (int q = 0; q < kBytes / 8; q++)
            asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(f[2 * q]), "=f"(f[2 * q + 1]) : "r"(addr + 8 * q));
    } else {
#pragma unroll
        for (int q = 0; q < kBytes / 4; q++)
            asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(f[q]) : "r"(addr + 4 * q));
    }
#pragma unroll
    for (int c = 0; c < BS; c++) {
        if constexpr (std::is_same<T, float>::value) out[c] = f[c];
        else if constexpr (std::is_same<T, double>::value)
            out[c] = __hiloint2double(__float_as_int(f[2 * c + 1]), __float_as_int(f[2 * c]));
        else out[c] = T(f[2 * c], f[2 * c + 1]);
    }
}

template <class T>
struct Ctx {
    const FusedCycle<T>& P;
    char* smem;                // the CTA's dynamic shared memory
    unsigned saddr;            // its shared-window address
    int rank, log_ctas;        // this CTA in the cluster, log2 of the cluster's CTAs
    int warp, nwarps, lane;    // of the CTA

    // Block row of local row u, and how many of the block rows below row are this CTA's.
    __device__ __forceinline__ int row(int u) const
    {
        return ((((u >> kChunkLog) << log_ctas) + rank) << kChunkLog) | (u & (kChunk - 1));
    }
    __device__ __forceinline__ int local_rows(int row) const
    {
        const int c = row >> kChunkLog, owner = c & ((1 << log_ctas) - 1), full = (c >> log_ctas) << kChunkLog;
        return full + (owner > rank ? kChunk : owner == rank ? (row & (kChunk - 1)) : 0);
    }
    // Where block row j's entries of the vector at byte offset `off` are: an address in the cluster.
    __device__ __forceinline__ unsigned remote(int off, int j, int bytes) const
    {
        const int c = j >> kChunkLog;
        const unsigned a = saddr + off + ((((c >> log_ctas) << kChunkLog) | (j & (kChunk - 1))) * bytes);
        unsigned r;
        asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(c & ((1 << log_ctas) - 1)));
        return r;
    }
    __device__ __forceinline__ T* local(int off) const { return reinterpret_cast<T*>(smem + off); }
};

// A block operator in CSR form, entry-major values.
template <class T>
struct Rows {
    const int* rowptr;
    const int* colidx;
    const T* vals;
    unsigned ld;   // entries of the levels here fit 32 bits (fused_layout)
};

// The local rows [lo, hi) of a phase, a row's bounds, and the columns of a lane's first blocks in it (-1:
// none); lane t of a row takes its blocks t, t + g, ... The bounds stay as loaded: an addition would wait for
// them there.
struct Span {
    int lo = 0, hi = 0;
};
struct Bounds {
    int p0 = 0, p1 = 0;
};
template <int N>
struct Columns {
    int col[N];
};

template <class T>
__device__ __forceinline__ Bounds row_bounds(const Ctx<T>& C, const Rows<T>& M, int u, int hi)
{
    Bounds b;
    if (u < hi) {
        const int i = C.row(u);
        b.p0 = M.rowptr[i];
        b.p1 = M.rowptr[i + 1];
    }
    return b;
}

template <int N, class T>
__device__ __forceinline__ Columns<N> row_columns(const Rows<T>& M, int p, int p1, int g)
{
    Columns<N> c;
#pragma unroll
    for (int q = 0; q < N; q++) c.col[q] = p + q * g < p1 ? M.colidx[p + q * g] : -1;
    return c;
}

// Blocks of a row a lane has in flight at once (columns ahead, then values and gathered entries), by the
// bytes of a block: 128 registers of a 512-thread CTA, 64 of a 1024-thread one. kHold: the values in registers
// (else as the sums reach them).
template <class T, int BS, int TH>
constexpr int kLaneBlocks = TH <= kFusedThreads && BS * BS * (int)sizeof(T) <= 16 ? 2 : 1;
template <class T, int BS, int TH>
constexpr bool kHold = BS * BS * (int)sizeof(T) <= (TH > kFusedThreads ? 16 : 36);

enum { kRowAssign = 0, kRowAdd = 1, kRowResidual = 2, kRowSweep = 3 };

// One phase over this CTA's rows `span` of M, `g` lanes per row, src: the byte offset of the gathered vector:
//   kRowAssign    out_i = (M src)_i, and zero_i = 0 (the next level's first x)
//   kRowAdd       out_i += (M src)_i
//   kRowResidual  out_i = b_i - (M src)_i
//   kRowSweep     out_i = omega D_i^-1 (b_i - sum_{j != i} M_ij src_j) + (1 - omega) out_i, out = src
// b, out and zero are the CTA's own parts. Output r of a row is written by lane r mod g. bounds, cols: the
// warp's first row, loaded ahead; on return those of the span `next`, with the bounds of `after` (the next
// two phases on M, empty spans where there are none). Waits for the barrier that the phase before arrived at,
// and arrives at the next.
template <class T, int BS, int TH, int KIND>
__device__ __forceinline__ void rows_phase(const Ctx<T>& C, Span span, int g, const Rows<T>& M, Bounds& bounds,
                                           Columns<kLaneBlocks<T, BS, TH>>& cols,
                                           Bounds& next_bounds, Span next, Span after, int src, const T* dinv, int nb,
                                           const T* b, T* out, T* zero)
{
    constexpr int NB = kLaneBlocks<T, BS, TH>;
    constexpr bool HOLD = kHold<T, BS, TH>, SWEEP = KIND == kRowSweep;
    const int lane = C.lane & (g - 1), group = C.warp * (32 / g) + C.lane / g, stride = C.nwarps * (32 / g);
    cluster_wait();
    bool ahead = false;   // the next phases' data asked for
    for (int base = span.lo + C.warp * (32 / g); base < span.hi || !ahead; base += stride) {   // warp-uniform
        const int u = base + C.lane / g;
        const bool in = u < span.hi;
        const int i = C.row(u);
        int p = bounds.p0 + lane;
        const int p1 = bounds.p1;
        Columns<NB> now = cols;
        T acc[BS], dv[BS];
#pragma unroll
        for (int r = 0; r < BS; r++) acc[r] = T(0);
        if (base < span.hi) {
            if (SWEEP) {
                unsigned dld = nb;
                asm volatile("" : "+r"(dld));
#pragma unroll
                for (int c = 0; c < BS; c++) dv[c] = in && lane < BS ? dinv[(unsigned)(lane * BS + c) * dld + (unsigned)i] : T(0);
            }
        }
        bool first = true;
        while (true) {
            unsigned ld = M.ld;   // opaque, so that the entries' offsets are not kept in registers between rows
            asm volatile("" : "+r"(ld));
            if (SWEEP) {
#pragma unroll
                for (int q = 0; q < NB; q++)
                    if (now.col[q] == i) now.col[q] = -1;   // the diagonal block: D^-1 instead
            }
            T xv[NB][BS], v[HOLD ? NB : 1][BS * BS];
#pragma unroll
            for (int q = 0; q < NB; q++) {
                const int j = now.col[q];
#pragma unroll
                for (int c = 0; c < BS; c++) xv[q][c] = T(0);
                if (j >= 0) {
                    if (HOLD) {
                        const T* vp = M.vals + (p + q * g);
#pragma unroll
                        for (int e = 0; e < BS * BS; e++, vp += ld) v[q][e] = *vp;
                    }
                    load_remote<T, BS>(C.remote(src, j, BS * (int)sizeof(T)), xv[q]);
                }
            }
            if (first) {   // behind the loads this row waits for
                first = false;
                if (base + stride < span.hi) {   // another pass of this phase
                    bounds = row_bounds(C, M, u + stride, span.hi);
                } else if (!ahead) {
                    ahead = true;
                    bounds = next_bounds;
                    cols = row_columns<NB>(M, bounds.p0 + lane, bounds.p1, g);
                    next_bounds = row_bounds(C, M, after.lo + group, after.hi);
                }
            }
#pragma unroll
            for (int q = 0; q < NB; q++) {
                if (now.col[q] < 0) continue;
#pragma unroll
                for (int r = 0; r < BS; r++)
#pragma unroll
                    for (int c = 0; c < BS; c++) {
                        const T a = HOLD ? v[q][r * BS + c] : M.vals[(unsigned)(r * BS + c) * ld + (unsigned)(p + q * g)];
                        acc[r] = fma(a, xv[q][c], acc[r]);
                    }
            }
            p += NB * g;
            if (p >= p1) break;   // per lane; no shuffle inside the loop
            now = row_columns<NB>(M, p, p1, g);
        }
        if (base >= span.hi) break;   // a warp without a row: only asked for the next phases' data
        if (base + stride < span.hi) cols = row_columns<NB>(M, bounds.p0 + lane, bounds.p1, g);
#pragma unroll
        for (int r = 0; r < BS; r++) acc[r] = lanes_sum(acc[r], g);
        if (!in) continue;
        if (SWEEP) {
            const T w = C.P.omega;
            T t[BS];
#pragma unroll
            for (int c = 0; c < BS; c++) t[c] = b[u * BS + c] - acc[c];
            auto output = [&](int r, const T (&d)[BS]) {
                T y = T(0);
#pragma unroll
                for (int c = 0; c < BS; c++) y = fma(d[c], t[c], y);
                if (w != T(1)) y = fma(w, y, (T(1) - w) * out[u * BS + r]);
                out[u * BS + r] = fin(y);
            };
            if (lane < BS) output(lane, dv);
            for (int r = lane + g; r < BS; r += g) {   // fewer lanes than outputs
                T d[BS];
#pragma unroll
                for (int c = 0; c < BS; c++) d[c] = dinv[(unsigned)(r * BS + c) * (unsigned)nb + (unsigned)i];
                output(r, d);
            }
        } else {
#pragma unroll
            for (int r = 0; r < BS; r++) {
                if (r % g != lane) continue;
                const int k = u * BS + r;
                if (KIND == kRowAssign) {
                    out[k] = fin(acc[r]);
                    zero[k] = T(0);
                } else if (KIND == kRowResidual) {
                    out[k] = b[k] - acc[r];
                } else {
                    out[k] = out[k] + acc[r];
                }
            }
        }
    }
    cluster_arrive();
}

// A phase of its own over all rows (residual, transfers): its first columns loaded between the barrier's
// arrive and wait.
template <class T, int BS, int TH, int KIND>
__device__ __forceinline__ void product(const Ctx<T>& C, int rows, int g, const Rows<T>& M, int src, const T* b, T* out, T* zero)
{
    constexpr int NB = kLaneBlocks<T, BS, TH>;
    const Span span{0, C.local_rows(rows)};
    Bounds bounds = row_bounds(C, M, C.warp * (32 / g) + C.lane / g, span.hi), none;
    Columns<NB> cols = row_columns<NB>(M, bounds.p0 + (C.lane & (g - 1)), bounds.p1, g);
    rows_phase<T, BS, TH, KIND>(C, span, g, M, bounds, cols, none, Span(), Span(), src, nullptr, 0, b, out, zero);
}

// `iters` smoothing steps on level L in the direction of the smoother code: the sweeps of
// BlockGaussSeidel::ExecuteOneIteration (alternating ones by iteration parity), one phase per colour.
template <class T, int BS, int TH>
__device__ void smooth(const Ctx<T>& C, const FusedLevel<T>& L, int code, int iters)
{
    const Rows<T> A{L.a_rowptr, L.a_colidx, L.a_vals, (unsigned)L.a_ld};
    const int sweeps = code == kFusedSymmetric ? 2 * iters : iters, g = L.lanes, group = C.warp * (32 / g) + C.lane / g;
    if (sweeps == 0) return;
    int s = 0, k = 0;   // sweep and colour of the next span
    auto next_span = [&]() {
        Span r;
        if (s >= sweeps) return r;
        const bool backward = code == kFusedBackward || (code == kFusedAlternatingBackward && !(s & 1)) ||
                              ((code == kFusedSymmetric || code == kFusedAlternatingForward) && (s & 1));
        const int c = backward ? L.ncol - 1 - k : k;
        r.lo = C.local_rows(L.colour_start[c]);
        r.hi = C.local_rows(L.colour_start[c + 1]);
        if (++k == L.ncol) {
            k = 0;
            s++;
        }
        return r;
    };
    Span now = next_span(), next = next_span(), after = next_span();
    Bounds bounds = row_bounds(C, A, now.lo + group, now.hi);
    Bounds next_bounds = row_bounds(C, A, next.lo + group, next.hi);
    Columns<kLaneBlocks<T, BS, TH>> cols =
        row_columns<kLaneBlocks<T, BS, TH>>(A, bounds.p0 + (C.lane & (g - 1)), bounds.p1, g);
    for (int phase = sweeps * L.ncol; phase > 0; phase--) {
        rows_phase<T, BS, TH, kRowSweep>(C, now, g, A, bounds, cols, next_bounds, next, after, L.x_off, L.dinv, L.nb,
                                         C.local(L.b_off), C.local(L.x_off), nullptr);
        now = next;
        next = after;
        after = next_span();
    }
}

// The coarsest level: x = C^{-1} b, C^{-1} dense FP64 row-major, FP64 accumulation. Every CTA gathers all
// of b in FP64, then computes its own rows, c_lanes lanes a row; the matrix is read eight entries a lane at
// a time, the first eight ahead of the barrier.
template <class T, int BS>
__device__ void coarse_solve(const Ctx<T>& C, const FusedLevel<T>& L)
{
    constexpr int kAtOnce = 8;
    const int n = C.P.n_coarse, g = C.P.c_lanes, tid = C.warp * 32 + C.lane;
    const int rows = C.local_rows(L.nb) * BS, lane = C.lane & (g - 1), stride = C.nwarps * (32 / g);
    double* bc = reinterpret_cast<double*>(C.smem + C.P.bc_off);
    T* x = C.local(L.x_off);
    double a[kAtOnce];
    auto load = [&](int k, int j) {
        const double* row = C.P.cinv + (long long)(C.row(k / BS) * BS + k % BS) * n;
#pragma unroll
        for (int q = 0; q < kAtOnce; q++) a[q] = k < rows && j + q * g < n ? row[j + q * g] : 0.0;
    };
    int k = C.warp * (32 / g) + C.lane / g;
    load(k, lane);
    cluster_wait();
    for (int j = tid; j < L.nb; j += C.nwarps * 32) {
        T v[BS];
        load_remote<T, BS>(C.remote(L.b_off, j, BS * (int)sizeof(T)), v);
#pragma unroll
        for (int c = 0; c < BS; c++) bc[j * BS + c] = (double)v[c];
    }
    __syncthreads();
    for (int base = C.warp * (32 / g); base < rows; base += stride, k += stride) {   // warp-uniform
        if (base >= stride) load(k, lane);
        double acc = 0.0;
        for (int j = lane; j < n; j += kAtOnce * g) {
            if (j != lane) load(k, j);
#pragma unroll
            for (int q = 0; q < kAtOnce; q++) acc = fma(a[q], j + q * g < n ? bc[j + q * g] : 0.0, acc);
        }
        acc = lanes_sum(acc, g);
        if (k < rows && lane == 0) x[k] = T(acc);
    }
    cluster_arrive();
}

// The cycle from lev[0] down: descend (pre-smooth, residual, restrict and zero the next x) to the
// coarsest, solve there, then ascend (prolongate, post-smooth) until a level still owes a coarse
// correction (W-cycle), from which the next descent starts with the coarser level's x kept. b and x of
// lev[0] come from and x goes back to global memory.
template <class T, int BS, int TH>
__device__ void run_cycle(const Ctx<T>& C)
{
    const FusedCycle<T>& P = C.P;
    const int last = P.nlev - 1;
    int done[kFusedMaxLevels];   // coarse corrections completed on each level of the current descent
    int l = 0;
    const FusedLevel<T>& L0 = P.lev[0];
    const int own = C.local_rows(L0.nb) * BS, tid = C.warp * 32 + C.lane;
    for (int k = tid; k < own; k += C.nwarps * 32) {
        const long long i = (long long)C.row(k / BS) * BS + k % BS;
        C.local(L0.b_off)[k] = L0.b[i];
        C.local(L0.x_off)[k] = P.x_zero ? T(0) : L0.x[i];
    }
    cluster_arrive();
    while (true) {
        for (; l < last; l++) {
            const FusedLevel<T>& L = P.lev[l];
            const FusedLevel<T>& N = P.lev[l + 1];
            smooth<T, BS, TH>(C, L, P.pre, P.npre);
            product<T, BS, TH, kRowResidual>(C, L.nb, L.a_lanes, {L.a_rowptr, L.a_colidx, L.a_vals, (unsigned)L.a_ld}, L.x_off,
                                             C.local(L.b_off), C.local(L.r_off), nullptr);
            product<T, BS, TH, kRowAssign>(C, N.nb, L.r_lanes, {L.r_rowptr, L.r_colidx, L.r_vals, (unsigned)L.r_ld}, L.r_off, nullptr,
                                           C.local(N.b_off), C.local(N.x_off));
            done[l] = 0;
        }
        coarse_solve<T, BS>(C, P.lev[last]);
        bool again = false;
        while (l > 0) {
            l--;
            done[l]++;
            const int loops = (l + 1 == last || P.w_loops < 1) ? 1 : P.w_loops;
            if (done[l] < loops) {
                again = true;
                break;
            }
            const FusedLevel<T>& L = P.lev[l];
            const FusedLevel<T>& N = P.lev[l + 1];
            product<T, BS, TH, kRowAdd>(C, L.nb, L.p_lanes, {L.p_rowptr, L.p_colidx, L.p_vals, (unsigned)L.p_ld}, N.x_off, nullptr,
                                        C.local(L.x_off), nullptr);
            smooth<T, BS, TH>(C, L, P.post, P.npost);
        }
        if (!again) break;
        l++;   // the next coarse correction of level l - 1 starts on level l, from the x the last one left
    }
    cluster_wait();   // the last phase's barrier: no CTA leaves before the others have read its memory
    for (int k = tid; k < own; k += C.nwarps * 32) L0.x[(long long)C.row(k / BS) * BS + k % BS] = C.local(L0.x_off)[k];
}

template <class T, int BS, int TH>
__global__ void __launch_bounds__(TH, 1) k_fused_cycle(const __grid_constant__ FusedCycle<T> P)
{
    extern __shared__ __align__(16) char fused_smem[];
    pdl_wait_coarse();
    const Ctx<T> C{P, fused_smem, (unsigned)__cvta_generic_to_shared(fused_smem), (int)blockIdx.x, 31 - __clz((int)gridDim.x),
                   (int)(threadIdx.x >> 5), (int)(blockDim.x >> 5), (int)(threadIdx.x & 31)};
    run_cycle<T, BS, TH>(C);
}

template <class T, int TH>
void* kernel_for_th(int bs)
{
    switch (bs) {
    case 2: return (void*)k_fused_cycle<T, 2, TH>;
    case 3: return (void*)k_fused_cycle<T, 3, TH>;
    case 4: return (void*)k_fused_cycle<T, 4, TH>;
    case 6: return (void*)k_fused_cycle<T, 6, TH>;
    default: return nullptr;
    }
}

template <class T>
void* kernel_for(int bs, int threads)
{
    if (threads == kFusedThreads) return kernel_for_th<T, kFusedThreads>(bs);
    if (threads == kFusedThreadsWide) return kernel_for_th<T, kFusedThreadsWide>(bs);
    return nullptr;
}

void fused_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int ctas, int threads, int smem, cudaStream_t s)
{
    cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
}

// Clusters above the portable size and shared memory above 48 KB need the kernel's opt-ins.
std::mutex g_fused_attr_mutex;

cudaError_t allow_fused(const void* k)
{
    std::lock_guard<std::mutex> lock(g_fused_attr_mutex);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kFusedMaxSmem);
    return e == cudaSuccess ? cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : e;
}

}  // namespace

template <class T>
int fused_layout(FusedCycle<T>& P, int bs, int ctas)
{
    long long at = 0;
    auto take = [&](long long bytes) {
        const long long o = at;
        at += (bytes + 15) / 16 * 16;
        return (int)std::min<long long>(o, 1 << 30);
    };
    for (int k = 0; k < P.nlev; k++) {
        FusedLevel<T>& L = P.lev[k];
        if (std::max({L.a_ld, L.p_ld, L.r_ld, (long long)L.nb}) * bs * bs >= 1LL << 31) return -1;   // 32-bit indices
        const long long chunks = (L.nb + kChunk - 1) / kChunk, own = (chunks + ctas - 1) / ctas * kChunk;
        L.x_off = take(own * bs * (long long)sizeof(T));
        L.b_off = take(own * bs * (long long)sizeof(T));
        if (k + 1 < P.nlev) L.r_off = take(own * bs * (long long)sizeof(T));
    }
    P.bc_off = take(8LL * P.n_coarse);
    return at <= kFusedMaxSmem ? (int)at : -1;
}

template <class T>
int fused_cycle_clusters(int bs, int ctas, int threads, int smem)
{
    const void* k = kernel_for<T>(bs, threads);
    if (!k || smem < 0 || (ctas != kClusterCtasPortable && ctas != kClusterCtasLarge)) return 0;
    if (allow_fused(k) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    fused_config(cfg, attr, ctas, threads, smem, nullptr);
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <class T>
cudaError_t launch_fused_cycle(const FusedCycle<T>& P, int bs, int ctas, int threads, int smem, cudaStream_t s)
{
    const void* k = kernel_for<T>(bs, threads);
    if (!k) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    fused_config(cfg, attr, ctas, threads, smem, s);
    void* args[] = {const_cast<FusedCycle<T>*>(&P)};
    return cudaLaunchKernelExC(&cfg, k, args);
}

#define FHG_FUSED_INSTANCES(T)                                                                      \
    template cudaError_t launch_fused_cycle<T>(const FusedCycle<T>&, int, int, int, int, cudaStream_t); \
    template int fused_cycle_clusters<T>(int, int, int, int);                                      \
    template int fused_layout<T>(FusedCycle<T>&, int, int);
FHG_FUSED_INSTANCES(float)
FHG_FUSED_INSTANCES(dfl)
#undef FHG_FUSED_INSTANCES

}  // namespace fhg

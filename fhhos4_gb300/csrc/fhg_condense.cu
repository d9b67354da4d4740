// Static condensation and assembly of the finest face system on the GPU.
//
// Reference: Diffusion_HHO::Assemble's condensation (src/Discretizations/HHO/Diffusion_HHO.h:627-638):
// with the cell unknowns of every element eliminated, the face operator is
//   A = A_FF - A_TF^T A_TT^{-1} A_TF,   b = b_F - A_TF^T A_TT^{-1} b_T,
// assembled element by element over the interior faces.
//
// Input: per class (elements that differ by a translation share their local operator; a caller
// without classes passes one class per element) the local operator before condensation, cells
// first; per element its class, its faces' unknown blocks (-1: Dirichlet) and b_T; per unknown face
// block its two elements with the face's local index in each. Steps, all in FP64:
//   1. per class: A_TT^{-1} by Gauss-Jordan elimination with partial pivoting; the Schur complement
//      S = A_FF - A_TF^T (A_TT^{-1} A_TF) and the source map G = -A_TF^T A_TT^{-1}
//      (n_face_dofs x n_cell) are kept;
//   2. per face block row: the sorted union of the unknown faces of its two elements is the row's
//      block columns (counted per CTA, then the CTAs' offsets by a scan);
//   3. per face block row: the values, S of the first element then of the second added into the
//      row's positions in that order, and b_I = sum over the two elements of G b_T, restricted to
//      the face's rows (the same order as the host assembly, so off-diagonal blocks are copies and
//      diagonal blocks one addition).
// Every entry is written once by one thread: no atomics, the result is bitwise reproducible. The output is
// the scalar CSR the solve phase takes (fhg_set_level): rows I * nf + a, columns J * nf + c.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <string>
#include <vector>

#include "fhg.h"

namespace {

constexpr int kCondThreads = 256;
constexpr int kCondMaxCell = 20;      // cell unknowns (3D, k = 3)
constexpr int kCondMaxFaceDofs = 40;  // faces per element x face DOFs (3D, k = 3)
constexpr int kCondMaxRowBlocks = 8;  // block columns of a face row: 2 (dim + 1) - 1 <= 7

struct CondData {
    int dim, ne, ncls, nC, nFF, nF, nf, nI;
    const int* cls;
    const int* elem_faces;
    const int* face_elems;
    const double* local;   // per class nH x nH
    const double* b_cell;  // per element nC
    double* S;             // per class nFF x nFF
    double* G;             // per class nFF x nC
    int* status;           // 1: a singular A_TT
};

// Step 1, one CTA per class: Gauss-Jordan elimination with partial pivoting of [A_TT | I] in shared
// memory gives A_TT^{-1}; then X = A_TT^{-1} A_TF, S = A_FF - A_TF^T X and G = -A_TF^T A_TT^{-1}, one
// entry per thread. NC = cell unknowns. A mesh has a few classes (tens), so a class is a serial chain
// of NC pivots whatever the launch: spreading a pivot's rows and the products over a CTA leaves NC
// barriers (one thread per class ran all of it, nFF NC (NC + nFF) multiply-adds, one after another).
// The sums run in the same order, so the values are the same bits.
constexpr int kClassThreads = 128;

template <int NC>
__global__ void __launch_bounds__(kClassThreads) k_condense_classes(CondData D)
{
    __shared__ double M[NC][NC], V[NC][NC], f[NC], X[NC][kCondMaxFaceDofs];
    __shared__ int piv;
    const int c = blockIdx.x, tid = threadIdx.x;
    const int nFF = D.nFF, nH = NC + nFF;
    const double* A = D.local + (long long)c * nH * nH;
    for (int e = tid; e < NC * NC; e += kClassThreads) {
        const int i = e / NC, j = e % NC;
        M[i][j] = A[i * nH + j];
        V[i][j] = i == j ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int k = 0; k < NC; k++) {
        if (tid == 0) {
            int p = k;
            for (int i = k + 1; i < NC; i++)
                if (fabs(M[i][k]) > fabs(M[p][k])) p = i;
            piv = M[p][k] == 0.0 ? -1 : p;
        }
        __syncthreads();
        const int p = piv;
        if (p < 0) {   // the whole CTA leaves together
            if (tid == 0) atomicExch(D.status, 1);
            return;
        }
        if (tid < NC && p != k) {
            double t = M[k][tid]; M[k][tid] = M[p][tid]; M[p][tid] = t;
            t = V[k][tid]; V[k][tid] = V[p][tid]; V[p][tid] = t;
        }
        __syncthreads();
        const double inv = 1.0 / M[k][k];
        if (tid < NC && tid != k) f[tid] = M[tid][k];
        __syncthreads();
        if (tid < NC) { M[k][tid] *= inv; V[k][tid] *= inv; }
        __syncthreads();
        for (int e = tid; e < NC * NC; e += kClassThreads) {
            const int i = e / NC, j = e % NC;
            if (i == k || f[i] == 0.0) continue;
            M[i][j] -= f[i] * M[k][j];
            V[i][j] -= f[i] * V[k][j];
        }
        __syncthreads();
    }
    double* S = D.S + (long long)c * nFF * nFF;
    double* G = D.G + (long long)c * nFF * NC;
    for (int e = tid; e < NC * nFF; e += kClassThreads) {
        const int t = e / nFF, j = e % nFF;
        double v = 0.0;
        for (int u = 0; u < NC; u++) v += V[t][u] * A[u * nH + NC + j];
        X[t][j] = v;
        double g = 0.0;
        const int i = e / NC, q = e % NC;
        for (int u = 0; u < NC; u++) g += A[u * nH + NC + i] * V[u][q];
        G[e] = -g;   // entry (i, q)
    }
    __syncthreads();
    for (int e = tid; e < nFF * nFF; e += kClassThreads) {
        const int i = e / nFF, j = e % nFF;
        double v = A[(NC + i) * nH + NC + j];
        for (int t = 0; t < NC; t++) v -= A[t * nH + NC + i] * X[t][j];
        S[e] = v;
    }
}

// The sorted block columns of face row I (the unknown faces of its two elements).
__device__ int row_columns(const CondData& D, int I, int* cols)
{
    int n = 0;
    for (int side = 0; side < 2; side++) {
        const int e = D.face_elems[(long long)I * 4 + 2 * side];
        if (e < 0) continue;
        for (int lf = 0; lf < D.nF; lf++) {
            const int g = D.elem_faces[(long long)e * D.nF + lf];
            if (g < 0) continue;
            bool seen = false;
            for (int q = 0; q < n; q++) seen |= cols[q] == g;
            if (!seen && n < kCondMaxRowBlocks) cols[n++] = g;
        }
    }
    for (int i = 1; i < n; i++) {   // insertion sort (n <= 7)
        const int v = cols[i];
        int j = i - 1;
        while (j >= 0 && cols[j] > v) { cols[j + 1] = cols[j]; j--; }
        cols[j + 1] = v;
    }
    return n;
}

// Step 2: block columns of the kCondThreads face rows of every CTA, summed.
__global__ void __launch_bounds__(kCondThreads) k_count(CondData D, long long* totals)
{
    __shared__ int sh[kCondThreads / 32];
    const int I = blockIdx.x * kCondThreads + threadIdx.x;
    int cols[kCondMaxRowBlocks];
    int n = I < D.nI ? row_columns(D, I, cols) : 0;
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long t = 0;
        for (int w = 0; w < kCondThreads / 32; w++) t += sh[w];
        totals[blockIdx.x] = t;
    }
}

// Exclusive scan of the totals by one CTA, in place; totals[nblocks] = the sum. Each thread sums a
// contiguous chunk, the chunk sums are scanned, and the chunk is written back.
constexpr int kScanThreads = 1024;

__global__ void __launch_bounds__(kScanThreads) k_scan_offsets(long long* totals, int nblocks)
{
    __shared__ long long warp_sum[kScanThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = (nblocks + kScanThreads - 1) / kScanThreads;
    const int lo = min(tid * chunk, nblocks), hi = min(lo + chunk, nblocks);
    long long sum = 0;
    for (int b = lo; b < hi; b++) sum += totals[b];
    long long run = sum;   // inclusive scan over the warp, then over the warps
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += t;
    }
    if (lane == 31) warp_sum[warp] = run;
    __syncthreads();
    if (warp == 0) {
        long long w = warp_sum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warp_sum[lane] = w;
    }
    __syncthreads();
    if (tid == kScanThreads - 1) totals[nblocks] = warp_sum[kScanThreads / 32 - 1];
    run += (warp ? warp_sum[warp - 1] : 0) - sum;
    for (int b = lo; b < hi; b++) {
        const long long t = totals[b];
        totals[b] = run;
        run += t;
    }
}

// Step 3: the scalar rows, column indices, values and right-hand side of kCondThreads face rows. The
// output is 12 bytes per entry and far larger than anything read (the class tables stay in L1), so
// the writes decide: a CTA first finds its rows' columns and sources one thread per row (shared
// memory), then each warp writes one face row's entries, which are contiguous, 32 at a time. One
// thread per face row, which cleared and then added to its own ~63 entries, and a serial scan of the
// offsets took a 48^3, k = 1 assembly (82 M entries, 0.98 GB) 2.56 ms; now 0.55 ms. NF: face DOFs (0: any).
template <int NF>
__global__ void __launch_bounds__(kCondThreads) k_fill(CondData D, const long long* offsets, int* rowptr,
                                                       int* colidx, double* vals, double* b)
{
    struct Row {
        int col[kCondMaxRowBlocks];     // block columns
        unsigned lf0, lf1;              // 4 bits per column: its local face in element 1 / 2 (15: none)
        long long s0, s1;               // first entry of S of element 1 / 2 at the face's rows
        short nb;                       // block columns
        short glued;                    // an element has a block on several faces (a periodic mesh one cell
                                        // across): the 4 bits of lf0, lf1 are then a bit per local face
        int start;                      // blocks before this row in the CTA
    };
    __shared__ Row rows[kCondThreads];
    __shared__ int warp_sum[kCondThreads / 32];
    const int nf = NF ? NF : D.nf, nC = D.nC, nFF = D.nFF;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int I = blockIdx.x * kCondThreads + tid;
    const long long block0 = offsets[blockIdx.x];
    Row& R = rows[tid];
    int nb = 0;
    if (I < D.nI) {
        int cols[kCondMaxRowBlocks];
        nb = row_columns(D, I, cols);
#pragma unroll
        for (int q = 0; q < kCondMaxRowBlocks; q++) R.col[q] = q < nb ? cols[q] : 0;
        unsigned lfs[2] = {0xffffffffu, 0xffffffffu}, faces[2] = {0u, 0u};
        R.glued = 0;
        long long first[2] = {0, 0};
        double acc[NF ? NF : kCondMaxFaceDofs];
        for (int a = 0; a < nf; a++) acc[a] = 0.0;
        for (int side = 0; side < 2; side++) {
            const int e = D.face_elems[(long long)I * 4 + 2 * side];
            const int lfi = D.face_elems[(long long)I * 4 + 2 * side + 1];
            if (e < 0 || lfi < 0) continue;
            const int c = D.cls[e];
            first[side] = ((long long)c * nFF + lfi * nf) * nFF;
            for (int lf = 0; lf < D.nF; lf++) {
                const int g = D.elem_faces[(long long)e * D.nF + lf];
                if (g < 0) continue;
                int q = 0;
                while (q < nb && cols[q] != g) q++;
                if ((faces[side] >> (4 * q)) & 15u) R.glued = 1;
                lfs[side] = (lfs[side] & ~(15u << (4 * q))) | ((unsigned)lf << (4 * q));
                faces[side] |= 1u << (4 * q + lf);
            }
            const double* G = D.G + ((long long)c * nFF + lfi * nf) * nC;
            const double* bT = D.b_cell + (long long)e * nC;
            for (int a = 0; a < nf; a++) {
                double s = 0.0;
                for (int t = 0; t < nC; t++) s += G[a * nC + t] * bT[t];
                acc[a] += s;
            }
        }
        for (int a = 0; a < nf; a++) b[(long long)I * nf + a] = acc[a];
        R.lf0 = R.glued ? faces[0] : lfs[0];
        R.lf1 = R.glued ? faces[1] : lfs[1];
        R.s0 = first[0]; R.s1 = first[1];
    }
    R.nb = (short)nb;
    int run = nb;   // blocks of the CTA's rows up to this one
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += t;
    }
    if (lane == 31) warp_sum[warp] = run;
    __syncthreads();
    for (int w = 0; w < warp; w++) run += warp_sum[w];
    R.start = run - nb;
    if (I < D.nI) {
        const long long base = (block0 + R.start) * nf * nf;
        for (int a = 0; a < nf; a++) rowptr[(long long)I * nf + a] = (int)(base + (long long)a * nb * nf);
        if (I == D.nI - 1) rowptr[(long long)D.nI * nf] = (int)(base + (long long)nb * nf * nf);
    }
    __syncthreads();
    const int n = min(kCondThreads, D.nI - (int)blockIdx.x * kCondThreads);
    for (int r = warp; r < n; r += kCondThreads / 32) {
        const Row& W = rows[r];
        const long long base = (block0 + W.start) * nf * nf;
        const int width = W.nb * nf, count = width * nf;
        // e / width by a rounded-up reciprocal: exact for e < 2^20 / width (count <= 8 * 13 * 13)
        const unsigned inv = ((1u << 20) + width - 1) / max(width, 1);
        for (int e = lane; e < count; e += 32) {
            const int a = (int)(((unsigned)e * inv) >> 20), j = e - a * width;
            const int q = j / nf, cc = j - q * nf;
            unsigned f0 = (W.lf0 >> (4 * q)) & 15u, f1 = (W.lf1 >> (4 * q)) & 15u;
            double v = 0.0;
            if (!W.glued) {
                if (f0 != 15u) v += D.S[W.s0 + a * nFF + (int)f0 * nf + cc];
                if (f1 != 15u) v += D.S[W.s1 + a * nFF + (int)f1 * nf + cc];
            } else {
                for (; f0; f0 &= f0 - 1) v += D.S[W.s0 + a * nFF + (__ffs(f0) - 1) * nf + cc];
                for (; f1; f1 &= f1 - 1) v += D.S[W.s1 + a * nFF + (__ffs(f1) - 1) * nf + cc];
            }
            colidx[base + e] = W.col[q] * nf + cc;
            vals[base + e] = v;
        }
    }
}

}  // namespace

struct fhg_cond {
    int device = 0;
    std::string err;
    CondData D{};
    std::vector<void*> allocs;
    long long* totals = nullptr;   // block columns before every CTA's rows, then their sum
    int* rowptr = nullptr;
    int* colidx = nullptr;
    double* vals = nullptr;
    double* b = nullptr;
    long long nnz = -1;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

namespace {

int cond_fail(fhg_cond* p, int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (p) p->err = buf;
    return code;
}

#define DCK(call)                                                                                         \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess) return cond_fail(p, FHG_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

template <class T>
int dev_alloc(fhg_cond* p, T** out, size_t n)
{
    void* d = nullptr;
    DCK(cudaMalloc(&d, sizeof(T) * std::max<size_t>(n, 1)));
    p->allocs.push_back(d);
    *out = (T*)d;
    return FHG_OK;
}

template <class T>
int dev_upload(fhg_cond* p, const T* host, size_t n, const T** out)
{
    T* d = nullptr;
    int rc = dev_alloc(p, &d, n);
    if (rc) return rc;
    DCK(cudaMemcpy(d, host, sizeof(T) * n, cudaMemcpyHostToDevice));
    *out = d;
    return FHG_OK;
}

}  // namespace

extern "C" {

int fhg_cond_create(fhg_cond** out, int device, int dim, int n_elements, int n_classes, int n_cell, int n_face_dofs,
                    int n_face_blocks, const int* elem_class, const int* elem_faces, const int* face_elems,
                    const double* local, const double* b_cell)
{
    if (!out) return FHG_ERR_INVALID_ARG;
    fhg_cond* p = new fhg_cond();
    *out = p;
    p->device = device;
    if (dim != 2 && dim != 3) return cond_fail(p, FHG_ERR_INVALID_ARG, "dimension %d", dim);
    if (n_elements <= 0 || n_classes <= 0 || n_cell <= 0 || n_face_blocks <= 0 || n_face_dofs <= 0 ||
        n_face_dofs % (dim + 1) != 0)
        return cond_fail(p, FHG_ERR_INVALID_ARG, "bad table sizes");
    if (n_cell > kCondMaxCell || n_face_dofs > kCondMaxFaceDofs ||
        (n_cell != 3 && n_cell != 4 && n_cell != 6 && n_cell != 10 && n_cell != 20))
        return cond_fail(p, FHG_ERR_UNSUPPORTED, "element larger than supported (%d cell, %d face unknowns)", n_cell,
                         n_face_dofs);
    if (!elem_class || !elem_faces || !face_elems || !local || !b_cell) return cond_fail(p, FHG_ERR_INVALID_ARG, "null table");
    const int nF = dim + 1;
    for (int e = 0; e < n_elements; e++) {
        if (elem_class[e] < 0 || elem_class[e] >= n_classes)
            return cond_fail(p, FHG_ERR_INVALID_ARG, "element %d: class %d out of range", e, elem_class[e]);
        for (int lf = 0; lf < nF; lf++)
            if (elem_faces[(size_t)e * nF + lf] >= n_face_blocks)
                return cond_fail(p, FHG_ERR_INVALID_ARG, "element %d: face block out of range", e);
    }
    for (int I = 0; I < n_face_blocks; I++)
        for (int side = 0; side < 2; side++) {
            const int e = face_elems[(size_t)I * 4 + 2 * side], lf = face_elems[(size_t)I * 4 + 2 * side + 1];
            if (e >= n_elements || (e >= 0 && (lf < 0 || lf >= nF || elem_faces[(size_t)e * nF + lf] != I)))
                return cond_fail(p, FHG_ERR_INVALID_ARG, "face block %d: element %d / local face %d inconsistent", I, e, lf);
        }
    DCK(cudaSetDevice(device));
    CondData& D = p->D;
    D.dim = dim;
    D.ne = n_elements;
    D.ncls = n_classes;
    D.nC = n_cell;
    D.nFF = n_face_dofs;
    D.nF = nF;
    D.nf = n_face_dofs / nF;
    D.nI = n_face_blocks;
    const size_t ne = n_elements, nc = n_classes, nH = n_cell + n_face_dofs;
    int rc;
    if ((rc = dev_upload(p, elem_class, ne, &D.cls)) || (rc = dev_upload(p, elem_faces, ne * nF, &D.elem_faces)) ||
        (rc = dev_upload(p, face_elems, (size_t)n_face_blocks * 4, &D.face_elems)) ||
        (rc = dev_upload(p, local, nc * nH * nH, &D.local)) || (rc = dev_upload(p, b_cell, ne * n_cell, &D.b_cell)) ||
        (rc = dev_alloc(p, &D.S, nc * n_face_dofs * n_face_dofs)) || (rc = dev_alloc(p, &D.G, nc * n_face_dofs * n_cell)) ||
        (rc = dev_alloc(p, &D.status, 1)) ||
        (rc = dev_alloc(p, &p->totals, (size_t)(n_face_blocks + kCondThreads - 1) / kCondThreads + 1)) ||
        (rc = dev_alloc(p, &p->b, (size_t)n_face_blocks * D.nf)) ||
        (rc = dev_alloc(p, &p->rowptr, (size_t)n_face_blocks * D.nf + 1)))
        return rc;
    DCK(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
    DCK(cudaEventCreate(&p->ev0));
    DCK(cudaEventCreate(&p->ev1));
    return FHG_OK;
}

int fhg_cond_run(fhg_cond* p, long long* nnz, double* elapsed_ms)
{
    if (!p || !p->stream) return FHG_ERR_INVALID_ARG;
    DCK(cudaSetDevice(p->device));
    CondData& D = p->D;
    const int nI = D.nI, nf = D.nf;
    const int grid = (nI + kCondThreads - 1) / kCondThreads;
    cudaStream_t s = p->stream;
    DCK(cudaMemsetAsync(D.status, 0, sizeof(int), s));
    DCK(cudaEventRecord(p->ev0, s));
    switch (D.nC) {
    case 3: k_condense_classes<3><<<D.ncls, kClassThreads, 0, s>>>(D); break;
    case 4: k_condense_classes<4><<<D.ncls, kClassThreads, 0, s>>>(D); break;
    case 6: k_condense_classes<6><<<D.ncls, kClassThreads, 0, s>>>(D); break;
    case 10: k_condense_classes<10><<<D.ncls, kClassThreads, 0, s>>>(D); break;
    case 20: k_condense_classes<20><<<D.ncls, kClassThreads, 0, s>>>(D); break;
    default: return cond_fail(p, FHG_ERR_UNSUPPORTED, "%d cell unknowns per element", D.nC);
    }
    k_count<<<grid, kCondThreads, 0, s>>>(D, p->totals);
    k_scan_offsets<<<1, kScanThreads, 0, s>>>(p->totals, grid);
    DCK(cudaGetLastError());
    long long blocks = 0;
    int status = 0;
    DCK(cudaMemcpyAsync(&blocks, p->totals + grid, sizeof(long long), cudaMemcpyDeviceToHost, s));
    DCK(cudaMemcpyAsync(&status, D.status, sizeof(int), cudaMemcpyDeviceToHost, s));
    DCK(cudaStreamSynchronize(s));
    if (status) return cond_fail(p, FHG_ERR_SINGULAR_BLOCK, "singular cell block in a local operator");
    const long long n_scalar = blocks * nf * nf;
    if (n_scalar > 0x7fffffffLL) return cond_fail(p, FHG_ERR_TOO_LARGE, "%lld entries exceed 32-bit indices", n_scalar);
    if (n_scalar != p->nnz) {
        for (void* d : {(void*)p->colidx, (void*)p->vals})
            if (d) {
                cudaFree(d);
                p->allocs.erase(std::find(p->allocs.begin(), p->allocs.end(), d));
            }
        p->colidx = nullptr;
        p->vals = nullptr;
        int rc;
        if ((rc = dev_alloc(p, &p->colidx, (size_t)n_scalar)) || (rc = dev_alloc(p, &p->vals, (size_t)n_scalar))) return rc;
        p->nnz = n_scalar;
    }
    switch (nf) {   // the face blocks of the supported degrees; any other size by the general kernel
    case 2: k_fill<2><<<grid, kCondThreads, 0, s>>>(D, p->totals, p->rowptr, p->colidx, p->vals, p->b); break;
    case 3: k_fill<3><<<grid, kCondThreads, 0, s>>>(D, p->totals, p->rowptr, p->colidx, p->vals, p->b); break;
    case 4: k_fill<4><<<grid, kCondThreads, 0, s>>>(D, p->totals, p->rowptr, p->colidx, p->vals, p->b); break;
    case 6: k_fill<6><<<grid, kCondThreads, 0, s>>>(D, p->totals, p->rowptr, p->colidx, p->vals, p->b); break;
    default: k_fill<0><<<grid, kCondThreads, 0, s>>>(D, p->totals, p->rowptr, p->colidx, p->vals, p->b); break;
    }
    DCK(cudaGetLastError());
    DCK(cudaEventRecord(p->ev1, s));
    DCK(cudaStreamSynchronize(s));
    if (nnz) *nnz = n_scalar;
    if (elapsed_ms) {
        float ms = 0.f;
        DCK(cudaEventElapsedTime(&ms, p->ev0, p->ev1));
        *elapsed_ms = ms;
    }
    return FHG_OK;
}

int fhg_cond_result(fhg_cond* p, int** rowptr, int** colidx, double** vals, double** b)
{
    if (!p || p->nnz < 0) return FHG_ERR_NOT_READY;
    if (rowptr) *rowptr = p->rowptr;
    if (colidx) *colidx = p->colidx;
    if (vals) *vals = p->vals;
    if (b) *b = p->b;
    return FHG_OK;
}

int fhg_cond_download(fhg_cond* p, int* rowptr, int* colidx, double* vals, double* b)
{
    if (!p || p->nnz < 0) return FHG_ERR_NOT_READY;
    DCK(cudaSetDevice(p->device));
    const size_t n = (size_t)p->D.nI * p->D.nf;
    if (rowptr) DCK(cudaMemcpy(rowptr, p->rowptr, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost));
    if (colidx) DCK(cudaMemcpy(colidx, p->colidx, sizeof(int) * (size_t)p->nnz, cudaMemcpyDeviceToHost));
    if (vals) DCK(cudaMemcpy(vals, p->vals, sizeof(double) * (size_t)p->nnz, cudaMemcpyDeviceToHost));
    if (b) DCK(cudaMemcpy(b, p->b, sizeof(double) * n, cudaMemcpyDeviceToHost));
    return FHG_OK;
}

const char* fhg_cond_last_error(const fhg_cond* p) { return p ? p->err.c_str() : "null condensation handle"; }

void fhg_cond_destroy(fhg_cond* p)
{
    if (!p) return;
    cudaSetDevice(p->device);
    if (p->stream) cudaStreamSynchronize(p->stream);
    for (void* d : p->allocs) cudaFree(d);
    if (p->ev0) cudaEventDestroy(p->ev0);
    if (p->ev1) cudaEventDestroy(p->ev1);
    if (p->stream) cudaStreamDestroy(p->stream);
    delete p;
}

}  // extern "C"

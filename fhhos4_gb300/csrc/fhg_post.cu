// Post-processing of a face solution on the GPU: cell-unknown recovery, the k+1 reconstruction and
// its L2 error against a closed-form solution, element by element.
//
// Reference: Diffusion_HHO::HybridCoeffsBySolvingCellUnknowns (src/Discretizations/HHO/
// Diffusion_HHO.h:855-882: x_T = A_TT^{-1} (b_T - A_TF x_F) per element),
// ReconstructHigherOrderApproximationFromHybridCoeffs (:896-912: the reconstruction operator applied to
// [x_T; x_F]) and Diffusion_HHO::L2Error (:120-150: sqrt(sum_T |u_h - u|^2_T) / sqrt(sum_T |u|^2_T) by
// cell quadrature).
//
// Layout: per element its class, the unknown block of each local face (-1: Dirichlet), its centroid
// and A_TT^{-1} b_T; per class the dense local operators -A_TT^{-1} A_TF and the reconstruction, and
// at the cell quadrature points the weights, offsets from the centroid and reconstruction basis values.
// Elements of one class differ by a translation, so the class tables are shared (they stay in L1/L2);
// a caller without classes passes one class per element. Class tables are stored entry by entry
// (entry e of class c at e * n_classes + c), so that a warp whose elements have a few classes reads each
// entry from one cache line, and consecutive lines when every element has its own class.
//
// The L2 sums. With centroid c and quadrature point offset o, sin(pi (c + o)) = sin(pi c) cos(pi o) +
// cos(pi c) sin(pi o), so u at the points of an element is Phi t: 2^dim class functions Phi (products of
// cos / sin of pi o) times 2^dim element coefficients t. With u_h = B c_h there, sum_q w_q (u_h - u)^2 is
// the squared 2-norm of sqrt(W) [Phi B] (t, -c_h), and a QR factorisation of that matrix per distinct
// table (on the first run that asks) leaves the same number as |R (t, -c_h)|^2 with R of 2^dim + n_recon rows: 171 multiply-adds
// per element in 3D, k = 1, instead of 216 points with three sines each on the FP64 pipe (2 per clock and
// SM), and the differences u_h - u are formed before they are squared, as at the points. A 32^3, k = 1
// solution takes 0.23 ms, 7.09 ms with the points. One thread per element in FP64, bound by the FP64 pipe; the L2
// sums go through per-CTA partials reduced in a fixed order, so the result is bitwise reproducible.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "fhg.h"

namespace {

constexpr int kPostThreads = 256;
constexpr int kPostMaxCtas = 152 * 8;
constexpr int kPostMaxCell = 20;       // cell basis functions (3D, k = 3)
constexpr int kPostMaxFaceDofs = 40;   // faces per element x face DOFs (3D, k = 3)
constexpr int kPostMaxRecon = 35;      // reconstruction basis functions (3D, degree 4)
constexpr int kPostMaxPoints = 512;

constexpr int kPostMaxGeometries = 256;   // distinct quadrature tables that are factorised (else: the points)
// Tables that are factorised however few elements share them, and elements to a table above that. A table takes
// 0.34 ms of one core in 3D, k = 1 (0.03 in 2D), on the first run with an exact solution; the points take 1.1 ms
// there for 1,300 elements (a thread's 216 points one after another), 7.1 ms for 197,000, and the factors 0.05 and
// 0.21 ms. So 32 tables on 16 cores repay themselves within that run, more of them from 500 elements each on: 13
// tables of 10,368 elements: first run and set-up 1.31 ms against 1.43 at the points.
constexpr int kPostFewTables = 32, kPostFactorElements = 512;

struct PostData {
    int dim, ne, ncls, ngeo, nC, nFF, nF, nf, nR, nq;
    const int* cls;
    const int* geo;       // per class: its factorised quadrature table
    const int* faces;
    const double* centre;
    const double* cell_rhs;
    const double* sc;     // nC x nFF per class
    const double* rc;     // nR x (nC + nFF) per class
    const double* R;      // (2^dim + nR)^2 per table, zero below the diagonal (null: the points)
    const double* w;      // nq per class (the points only, as the next two)
    const double* off;    // nq x 3 per class
    const double* basis;  // nq x nR per class
};

__device__ double block_sum_post(double v, double* sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += sh[i];
    return t;  // valid in thread 0
}

// x_cells (optional) and, with exact = FHG_EXACT_SINE, per-CTA partial sums of |u_h - u|^2 and |u|^2.
// NC, NFF, NR: the element's sizes (0: those of D).
template <int DIM, int NC, int NFF, int NR>
__global__ void __launch_bounds__(kPostThreads) k_post(PostData D, const double* __restrict__ x, double* x_cells,
                                                       int exact, double* partials)
{
    __shared__ double sh[kPostThreads / 32];
    const int nC = NC ? NC : D.nC, nFF = NFF ? NFF : D.nFF, nR = NR ? NR : D.nR, nf = nFF / (DIM + 1);
    const long long ncls = D.ncls, ngeo = D.ngeo;
    double err = 0.0, nrm = 0.0;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < D.ne; e += (long long)gridDim.x * blockDim.x) {
        const int c = D.cls[e];
        double cell[NC ? NC : kPostMaxCell], face[NFF ? NFF : kPostMaxFaceDofs], coef[NR ? NR : kPostMaxRecon];
        for (int k = 0; k < DIM + 1; k++) {
            const int g = D.faces[e * (DIM + 1) + k];
            for (int j = 0; j < nf; j++) face[k * nf + j] = g >= 0 ? x[(long long)g * nf + j] : 0.0;
        }
        const double* sc = D.sc + c;
        for (int i = 0; i < nC; i++) {
            double v = D.cell_rhs[e * nC + i];
            for (int j = 0; j < nFF; j++) v += sc[(i * nFF + j) * ncls] * face[j];
            cell[i] = v;
            if (x_cells) x_cells[e * nC + i] = v;
        }
        if (exact != FHG_EXACT_SINE) continue;
        const int nh = nC + nFF;
        const double* rc = D.rc + c;
        for (int i = 0; i < nR; i++) {
            double s = 0.0;
            for (int j = 0; j < nC; j++) s += rc[(i * nh + j) * ncls] * cell[j];
            for (int j = 0; j < nFF; j++) s += rc[(i * nh + nC + j) * ncls] * face[j];
            coef[i] = s;
        }
        if (D.R) {
            constexpr int M = 1 << DIM;
            double t[M];
            t[0] = 1.0;
#pragma unroll
            for (int d = 0; d < DIM; d++) {
                double sn, cs;
                sincospi(D.centre[e * 3 + d], &sn, &cs);
#pragma unroll
                for (int m = (1 << d) - 1; m >= 0; m--) {
                    t[m | (1 << d)] = t[m] * cs;   // bit d set: cos(pi c_d) sin(pi o_d)
                    t[m] *= sn;
                }
            }
            const double* R = D.R + D.geo[c];
            const int nv = M + nR;
#pragma unroll
            for (int r = 0; r < M; r++) {
                double u = 0.0;
#pragma unroll
                for (int m = r; m < M; m++) u += R[(r * nv + m) * ngeo] * t[m];
                nrm += u * u;
                for (int i = 0; i < nR; i++) u -= R[(r * nv + M + i) * ngeo] * coef[i];
                err += u * u;
            }
            for (int r = 0; r < nR; r++) {
                double u = 0.0;
                for (int i = r; i < nR; i++) u += R[((M + r) * nv + M + i) * ngeo] * coef[i];
                err += u * u;
            }
            continue;
        }
        const double *w = D.w + c, *off = D.off + c, *B = D.basis + c;
        for (int q = 0; q < D.nq; q++) {
            double uh = 0.0;
            for (int i = 0; i < nR; i++) uh += coef[i] * B[(long long)(q * nR + i) * ncls];
            double u = 1.0;
            for (int d = 0; d < DIM; d++) u *= sinpi(D.centre[e * 3 + d] + off[(long long)(q * 3 + d) * ncls]);
            err += w[q * ncls] * (uh - u) * (uh - u);
            nrm += w[q * ncls] * u * u;
        }
    }
    if (exact != FHG_EXACT_SINE) return;
    const double te = block_sum_post(err, sh);
    const double tn = block_sum_post(nrm, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = te;
        partials[2 * blockIdx.x + 1] = tn;
    }
}

// Fixed-order sum of the partials by one CTA (at most kPostMaxCtas pairs): each thread's strided share,
// then the block sum.
__global__ void __launch_bounds__(kPostThreads) k_post_finish(const double* partials, int n, double* out)
{
    __shared__ double sh[kPostThreads / 32];
    double e = 0.0, u = 0.0;
    for (int i = threadIdx.x; i < n; i += kPostThreads) {
        e += partials[2 * i];
        u += partials[2 * i + 1];
    }
    e = block_sum_post(e, sh);
    u = block_sum_post(u, sh);
    if (threadIdx.x == 0) {
        out[0] = e;
        out[1] = u;
    }
}

// Numbers of 106 bits as a sum of two doubles (Dekker 1971), on the host: the same results on every machine,
// and ten times faster than a long double where that is emulated.
struct Dd {
    double h, l;
};
inline Dd dd_fast(double a, double b) { const double s = a + b; return {s, b - (s - a)}; }   // |a| >= |b|
inline Dd operator+(Dd a, Dd b)
{
    const double s = a.h + b.h, t = s - a.h;
    return dd_fast(s, ((a.h - (s - t)) + (b.h - t)) + (a.l + b.l));
}
inline Dd operator-(Dd a, Dd b) { return a + Dd{-b.h, -b.l}; }
inline Dd operator*(Dd a, Dd b)
{
    const double p = a.h * b.h;
    return dd_fast(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
inline Dd operator/(Dd a, Dd b)
{
    const double q = a.h / b.h;
    return dd_fast(q, (a - b * Dd{q, 0.0}).h / b.h);
}
inline Dd dd_sqrt(double a)
{
    const double s = std::sqrt(a);
    return s > 0.0 ? dd_fast(s, (Dd{a, 0.0} - Dd{s, 0.0} * Dd{s, 0.0}).h / (2.0 * s)) : Dd{s, 0.0};
}

// sin(pi o) and cos(pi o): o = 2 m + n / 2 + f exactly, |f| <= 1/4, and the Taylor series of pi f to
// y^22 / 22! (5e-24).
void dd_sincospi(double o, Dd& sn, Dd& cs)
{
    constexpr int kTerms = 11;
    const Dd pi = {3.141592653589793, 1.2246467991473532e-16};
    const double r = o - 2.0 * std::round(0.5 * o), n = std::round(2.0 * r), f = r - 0.5 * n;
    const Dd y = pi * Dd{f, 0.0}, y2 = y * y;
    Dd s = {1.0, 0.0}, c = {1.0, 0.0};   // Horner: 1 - y^2 / ((k - 1) k) (1 - ...)
    for (int k = 2 * kTerms; k > 0; k -= 2) {
        c = Dd{1.0, 0.0} - y2 * c / Dd{(double)(k - 1) * k, 0.0};
        s = Dd{1.0, 0.0} - y2 * s / Dd{(double)k * (k + 1), 0.0};
    }
    s = s * y;
    const Dd ms = {-s.h, -s.l}, mc = {-c.h, -c.l};
    switch ((int)n & 3) {
    case 0: sn = s; cs = c; break;
    case 1: sn = c; cs = ms; break;
    case 2: sn = ms; cs = mc; break;
    default: sn = mc; cs = s; break;
    }
}

// sum over q of a[q] b[q], four sums side by side.
inline Dd dd_dot(const Dd* a, const Dd* b, int n)
{
    Dd t[4] = {};
    int q = 0;
    for (; q + 4 <= n; q += 4)
        for (int u = 0; u < 4; u++) t[u] = t[u] + a[q + u] * b[q + u];
    for (; q < n; q++) t[0] = t[0] + a[q] * b[q];
    return (t[0] + t[1]) + (t[2] + t[3]);
}

// R of the QR factorisation (Householder) of sqrt(W) [Phi B] of one quadrature table, in pairs of doubles
// so that R adds no more than its own rounding to FP64; column m < 2^dim of Phi is the product
// over d of sin(pi o_d) (bit d of m set) or cos(pi o_d). Rows past the number of points are zero.
void factor_table(int dim, int nq, int nR, const double* w, const double* off, const double* basis, double* R)
{
    const int M = 1 << dim, nv = M + nR;
    std::vector<Dd> A((size_t)nv * nq);   // column-major
    for (int q = 0; q < nq; q++) {
        const Dd sw = dd_sqrt(w[q]);
        Dd s[3], c[3];
        for (int d = 0; d < dim; d++) dd_sincospi(off[q * 3 + d], s[d], c[d]);
        for (int m = 0; m < M; m++) {
            Dd v = sw;
            for (int d = 0; d < dim; d++) v = v * ((m >> d & 1) ? s[d] : c[d]);
            A[(size_t)m * nq + q] = v;
        }
        for (int i = 0; i < nR; i++) A[(size_t)(M + i) * nq + q] = sw * Dd{basis[(size_t)q * nR + i], 0.0};
    }
    for (int k = 0; k < std::min(nv, nq); k++) {
        Dd* a = &A[(size_t)k * nq];
        const Dd nn = dd_dot(a + k, a + k, nq - k);
        Dd alpha = {0.0, 0.0};
        if (!(nn.h <= 0.0)) {
            const Dd root = dd_sqrt(nn.h);   // of the pair: one Newton step more
            alpha = root + (nn - root * root) / Dd{2.0 * root.h, 0.0};
            if (a[k].h > 0.0) alpha = Dd{-alpha.h, -alpha.l};
        }
        const Dd vv = nn - alpha * a[k];   // v = a - alpha e_k, v.v / 2 = nn - alpha a_k
        a[k] = a[k] - alpha;
        if (!(vv.h <= 0.0))
            for (int j = k + 1; j < nv; j++) {
                Dd* b = &A[(size_t)j * nq];
                const Dd dot = dd_dot(a + k, b + k, nq - k) / vv;
                for (int q = k; q < nq; q++) b[q] = b[q] - dot * a[q];
            }
        a[k] = alpha;
    }
    for (int r = 0; r < nv; r++)
        for (int m = 0; m < nv; m++) R[(size_t)r * nv + m] = r < nq && m >= r ? A[(size_t)m * nq + r].h : 0.0;
}

}  // namespace

struct fhg_post {
    int device = 0;
    std::string err;
    PostData D{};
    std::vector<void*> allocs;
    double* partials = nullptr;
    double* sums = nullptr;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // The distinct quadrature tables (weights, offsets, basis values) and each class's, held until the first
    // run with an exact solution factorises them; empty when the points are used.
    std::vector<double> w, off, basis;
    std::vector<int> geo;
};

namespace {

int post_fail(fhg_post* p, int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (p) p->err = buf;
    return code;
}

#define PCK(call)                                                                                         \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess) return post_fail(p, FHG_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

template <class T>
int upload(fhg_post* p, const T* host, size_t n, const T** dev)
{
    void* d = nullptr;
    PCK(cudaMalloc(&d, sizeof(T) * std::max<size_t>(n, 1)));
    p->allocs.push_back(d);
    PCK(cudaMemcpy(d, host, sizeof(T) * n, cudaMemcpyHostToDevice));
    *dev = (const T*)d;
    return FHG_OK;
}

// A table of n entries per class, given class by class (of = null) or table by table (class c's is of[c]),
// entry by entry (entry e of class c at e * classes + c).
int upload_interleaved(fhg_post* p, const double* host, size_t classes, size_t n, const double** dev, const int* of = nullptr)
{
    std::vector<double> t(classes * n);
    for (size_t c = 0; c < classes; c++)
        for (size_t e = 0; e < n; e++) t[e * classes + c] = host[(of ? (size_t)of[c] : c) * n + e];
    return upload(p, t.data(), t.size(), dev);
}

int upload_points(fhg_post* p, const double* weights, const double* offsets, const double* basis, const int* of = nullptr)
{
    PostData& D = p->D;
    const size_t nc = D.ncls, nq = D.nq;
    int rc;
    if ((rc = upload_interleaved(p, weights, nc, nq, &D.w, of)) || (rc = upload_interleaved(p, offsets, nc, nq * 3, &D.off, of)))
        return rc;
    return upload_interleaved(p, basis, nc, nq * D.nR, &D.basis, of);
}

// The distinct quadrature tables: classes with the same weights, offsets and basis values share one
// (coefficients change an element's operators, not its quadrature), found by hashing. Left in p for factorise
// where they repay it (kPostFewTables) and no weight is negative; false: the points are used.
bool distinct_tables(fhg_post* p, const double* weights, const double* offsets, const double* basis)
{
    const PostData& D = p->D;
    const size_t nc = D.ncls, nq = D.nq, nR = D.nR;
    const size_t limit = std::min(kPostMaxGeometries, std::max(kPostFewTables, D.ne / kPostFactorElements));
    for (size_t i = 0; i < nc * nq; i++)
        if (!(weights[i] >= 0.0)) return false;
    std::vector<int> geo(nc);
    std::vector<size_t> hash, rep;
    auto same = [](const double* a, const double* b, size_t n) { return std::memcmp(a, b, sizeof(double) * n) == 0; };
    for (size_t c = 0; c < nc; c++) {
        const double *w = weights + c * nq, *o = offsets + c * nq * 3, *B = basis + c * nq * nR;
        size_t h = 1469598103934665603ull;
        for (const auto& [t, n] : {std::pair<const double*, size_t>{w, nq}, {o, nq * 3}, {B, nq * nR}})
            for (size_t i = 0; i < n; i++) {
                unsigned long long u;
                std::memcpy(&u, t + i, 8);
                h = (h ^ u) * 1099511628211ull;
                h ^= h >> 29;
            }
        int g = -1;
        for (size_t k = 0; k < rep.size() && g < 0; k++)
            if (hash[k] == h && same(weights + rep[k] * nq, w, nq) && same(offsets + rep[k] * nq * 3, o, nq * 3) &&
                same(basis + rep[k] * nq * nR, B, nq * nR))
                g = (int)k;
        if (g < 0) {
            if (rep.size() == limit) return false;
            g = (int)rep.size();
            rep.push_back(c);
            hash.push_back(h);
        }
        geo[c] = g;
    }
    for (size_t c : rep) {
        p->w.insert(p->w.end(), weights + c * nq, weights + (c + 1) * nq);
        p->off.insert(p->off.end(), offsets + c * nq * 3, offsets + (c + 1) * nq * 3);
        p->basis.insert(p->basis.end(), basis + c * nq * nR, basis + (c + 1) * nq * nR);
    }
    p->geo = std::move(geo);
    return true;
}

// The factors of the distinct tables, on the host's threads; where one is not finite, the points. The tables held
// for it are given back.
int factorise(fhg_post* p)
{
    PostData& D = p->D;
    const size_t nq = D.nq, nR = D.nR, nv = (size_t)(1 << D.dim) + nR, tables = p->w.size() / nq;
    std::vector<double> R(tables * nv * nv);
    std::atomic<size_t> next{0};
    std::atomic<bool> bad{false};
    auto work = [&]() {
        try {
            for (size_t k = next++; k < tables; k = next++)
                factor_table(D.dim, (int)nq, (int)nR, &p->w[k * nq], &p->off[k * nq * 3], &p->basis[k * nq * nR], &R[k * nv * nv]);
        } catch (const std::bad_alloc&) {
            bad = true;
        }
    };
    std::vector<std::thread> th;
    const size_t nt = std::min<size_t>(tables, std::max(1u, std::min(32u, std::thread::hardware_concurrency())));
    th.reserve(nt);   // no allocation between the first thread and the joins
    try {
        for (size_t t = 1; t < nt; t++) th.emplace_back(work);
    } catch (...) {
        // no more threads to be had: those that run and this one share the tables
    }
    work();
    for (auto& t : th) t.join();
    for (double v : R) bad = bad || !std::isfinite(v);
    int rc;
    if (bad) {
        if ((rc = upload_points(p, p->w.data(), p->off.data(), p->basis.data(), p->geo.data()))) return rc;
    } else {
        const double* dev = nullptr;
        if ((rc = upload(p, p->geo.data(), p->geo.size(), &D.geo)) || (rc = upload_interleaved(p, R.data(), tables, nv * nv, &dev)))
            return rc;
        D.ngeo = (int)tables;
        D.R = dev;
    }
    for (auto* t : {&p->w, &p->off, &p->basis}) std::vector<double>().swap(*t);
    std::vector<int>().swap(p->geo);
    return FHG_OK;
}

typedef void (*PostKernel)(PostData, const double*, double*, int, double*);

// The kernel of an element's sizes: the degrees 1 to 3, else the one that takes them at run time.
PostKernel post_kernel(const PostData& D)
{
    auto is = [&](int dim, int nC, int nFF, int nR) { return D.dim == dim && D.nC == nC && D.nFF == nFF && D.nR == nR; };
    if (is(2, 3, 6, 6)) return k_post<2, 3, 6, 6>;
    if (is(2, 6, 9, 10)) return k_post<2, 6, 9, 10>;
    if (is(2, 10, 12, 15)) return k_post<2, 10, 12, 15>;
    if (is(3, 4, 12, 10)) return k_post<3, 4, 12, 10>;
    if (is(3, 10, 24, 20)) return k_post<3, 10, 24, 20>;
    return D.dim == 2 ? k_post<2, 0, 0, 0> : k_post<3, 0, 0, 0>;
}

}  // namespace

extern "C" {

int fhg_post_create(fhg_post** out, int device, int dim, int n_elements, int n_classes, int n_cell, int n_face_dofs,
                    int n_recon, int n_points, const int* elem_class, const int* elem_faces, const double* elem_centre,
                    const double* cell_rhs, const double* solve_cells, const double* recon, const double* weights,
                    const double* offsets, const double* basis)
{
    if (!out) return FHG_ERR_INVALID_ARG;
    fhg_post* p = new fhg_post();
    *out = p;
    p->device = device;
    if (dim != 2 && dim != 3) return post_fail(p, FHG_ERR_INVALID_ARG, "dimension %d", dim);
    if (n_elements <= 0 || n_classes <= 0 || n_cell <= 0 || n_recon <= 0 || n_points <= 0 ||
        n_face_dofs <= 0 || n_face_dofs % (dim + 1) != 0)
        return post_fail(p, FHG_ERR_INVALID_ARG, "bad table sizes");
    if (n_cell > kPostMaxCell || n_face_dofs > kPostMaxFaceDofs || n_recon > kPostMaxRecon || n_points > kPostMaxPoints)
        return post_fail(p, FHG_ERR_UNSUPPORTED, "element tables larger than supported (%d cell, %d face, %d recon, %d points)",
                         n_cell, n_face_dofs, n_recon, n_points);
    if (!elem_class || !elem_faces || !elem_centre || !cell_rhs || !solve_cells || !recon || !weights || !offsets || !basis)
        return post_fail(p, FHG_ERR_INVALID_ARG, "null table");
    for (int e = 0; e < n_elements; e++)
        if (elem_class[e] < 0 || elem_class[e] >= n_classes)
            return post_fail(p, FHG_ERR_INVALID_ARG, "element %d: class %d out of range", e, elem_class[e]);
    PCK(cudaSetDevice(device));
    PostData& D = p->D;
    D.dim = dim;
    D.ne = n_elements;
    D.ncls = n_classes;
    D.nC = n_cell;
    D.nFF = n_face_dofs;
    D.nF = dim + 1;
    D.nf = n_face_dofs / (dim + 1);
    D.nR = n_recon;
    D.nq = n_points;
    const size_t ne = n_elements, nc = n_classes;
    int rc;
    try {
        if ((rc = upload(p, elem_class, ne, &D.cls)) || (rc = upload(p, elem_faces, ne * D.nF, &D.faces)) ||
            (rc = upload(p, elem_centre, ne * 3, &D.centre)) || (rc = upload(p, cell_rhs, ne * n_cell, &D.cell_rhs)) ||
            (rc = upload_interleaved(p, solve_cells, nc, (size_t)n_cell * n_face_dofs, &D.sc)) ||
            (rc = upload_interleaved(p, recon, nc, (size_t)n_recon * (n_cell + n_face_dofs), &D.rc)))
            return rc;
        if (!distinct_tables(p, weights, offsets, basis) && (rc = upload_points(p, weights, offsets, basis))) return rc;
    } catch (const std::bad_alloc&) {
        return post_fail(p, FHG_ERR_TOO_LARGE, "out of host memory for the element tables");
    }
    void* d = nullptr;
    PCK(cudaMalloc(&d, sizeof(double) * (2 * kPostMaxCtas + 2)));
    p->allocs.push_back(d);
    p->partials = (double*)d;
    p->sums = p->partials + 2 * kPostMaxCtas;
    PCK(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
    PCK(cudaEventCreate(&p->ev0));
    PCK(cudaEventCreate(&p->ev1));
    return FHG_OK;
}

int fhg_post_run(fhg_post* p, const double* x_faces, double* x_cells, int exact, double* rel_l2_error, double* elapsed_ms)
{
    if (!p || !p->stream) return FHG_ERR_INVALID_ARG;
    if (!x_faces) return post_fail(p, FHG_ERR_INVALID_ARG, "null face solution");
    if (exact != FHG_EXACT_NONE && exact != FHG_EXACT_SINE) return post_fail(p, FHG_ERR_INVALID_ARG, "unknown exact solution %d", exact);
    if (exact == FHG_EXACT_SINE && !rel_l2_error) return post_fail(p, FHG_ERR_INVALID_ARG, "null error output");
    PCK(cudaSetDevice(p->device));
    if (exact == FHG_EXACT_SINE && !p->geo.empty()) {
        try {
            const int rc = factorise(p);
            if (rc) return rc;
        } catch (const std::bad_alloc&) {
            return post_fail(p, FHG_ERR_TOO_LARGE, "out of host memory for the element tables");
        }
    }
    const int grid = (int)std::min<long long>(kPostMaxCtas, ((long long)p->D.ne + kPostThreads - 1) / kPostThreads);
    PCK(cudaEventRecord(p->ev0, p->stream));
    post_kernel(p->D)<<<grid, kPostThreads, 0, p->stream>>>(p->D, x_faces, x_cells, exact, p->partials);
    PCK(cudaGetLastError());
    if (exact == FHG_EXACT_SINE) {
        k_post_finish<<<1, kPostThreads, 0, p->stream>>>(p->partials, grid, p->sums);
        PCK(cudaGetLastError());
    }
    PCK(cudaEventRecord(p->ev1, p->stream));
    double s[2] = {0.0, 0.0};
    if (exact == FHG_EXACT_SINE) PCK(cudaMemcpyAsync(s, p->sums, sizeof(s), cudaMemcpyDeviceToHost, p->stream));
    PCK(cudaStreamSynchronize(p->stream));
    if (exact == FHG_EXACT_SINE) *rel_l2_error = s[1] > 0 ? std::sqrt(s[0]) / std::sqrt(s[1]) : std::sqrt(s[0]);
    if (elapsed_ms) {
        float ms = 0.f;
        PCK(cudaEventElapsedTime(&ms, p->ev0, p->ev1));
        *elapsed_ms = ms;
    }
    return FHG_OK;
}

int fhg_post_factors(const fhg_post* p) { return p ? p->D.ngeo : 0; }

const char* fhg_post_last_error(const fhg_post* p) { return p ? p->err.c_str() : "null post-processing handle"; }

void fhg_post_destroy(fhg_post* p)
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

// symops.cu -- block updates on vectors with X^T = s X (s = 1 singlet, -1
// triplet), the ZGEMM 'N','N' updates of gplmr.F90:101-103,298-320 and
// harmonic_ritz_small.F90:145,313-316 where the iteration keeps the exchange
// sector exactly (Solver::detect_symmetry).
//
// HBM-bound: a combination of n columns moves n + 1 vectors.  Here a CTA forms
// the 32 x 32 tile at (p0, q0), p0 <= q0, from the upper halves of its inputs
// and writes it and s times its transpose: n/2 + 1 vectors.  The results are
// (anti)symmetric bit for bit, as the general update's are.  A block that only
// such sums and updates read next needs its upper tiles alone (`upper`): n/2 +
// 1/2 vectors.
#include "de_kernels.h"
#include "pdl.h"

#include <algorithm>

namespace de {
namespace {

__device__ __forceinline__ double2 wide(double2 v) { return v; }
__device__ __forceinline__ double2 wide(float2 v) { return make_double2(v.x, v.y); }

// tile pair of block b: bi <= bj
__device__ __forceinline__ void tile_pair(int b, int &bi, int &bj)
{
    bj = (int)((sqrtf(8.0f * b + 1.0f) - 1.0f) * 0.5f);
    while ((bj + 1) * (bj + 2) / 2 <= b) ++bj;
    while (bj * (bj + 1) / 2 > b) --bj;
    bi = b - bj * (bj + 1) / 2;
}

// Y_j = beta_j Y_j + alpha sum_i X_i C(i,j); IC inputs of E elements a thread
// in flight.
template <class SI, int NOUT, int E, int IC>
__global__ void __launch_bounds__(1024 / E, E == 4 ? 2 : 1)
    update_sym_kernel(const __grid_constant__ UpdListT<SI, double2> U, const double2 *C, int ldc, int64_t m,
                      double s, int upper)
{
    pdl_enter();
    constexpr int RY = 32 / E;
    extern __shared__ __align__(16) unsigned char us_smem[];
    double2 *cs = reinterpret_cast<double2 *>(us_smem);  // [nin][NOUT]
    __shared__ double2 tile[32][33];
    const int nin = U.nin, nout = U.nout;
    for (int e = threadIdx.x; e < nin * NOUT; e += blockDim.x) {
        const int i = e / NOUT, j = e % NOUT;
        const double2 c = j < nout ? C[i + (int64_t)ldc * j] : make_double2(0.0, 0.0);
        cs[e] = make_double2(U.alpha.x * c.x - U.alpha.y * c.y, U.alpha.x * c.y + U.alpha.y * c.x);
    }
    int bi, bj;
    tile_pair(blockIdx.x, bi, bj);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t p = bi * 32 + tx, pt = bj * 32 + tx;
    int64_t row[E];
    bool in[E];
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int64_t q = bj * 32 + ty + RY * u;
        in[u] = p < m && q < m;
        row[u] = in[u] ? p + m * q : 0;
    }
    __syncthreads();
    double ar[E][NOUT], ai[E][NOUT];
#pragma unroll
    for (int u = 0; u < E; ++u)
#pragma unroll
        for (int j = 0; j < NOUT; ++j) {
            ar[u][j] = ai[u][j] = 0.0;
            if (j < nout && (U.beta[j].x != 0.0 || U.beta[j].y != 0.0) && in[u]) {
                const double2 y = U.y[j][row[u]], b = U.beta[j];
                ar[u][j] = b.x * y.x - b.y * y.y;
                ai[u][j] = b.x * y.y + b.y * y.x;
            }
        }
    auto add = [&](double2 v, const double2 *c, int u) {
#pragma unroll
        for (int j = 0; j < NOUT; ++j) {
            ar[u][j] = fma(v.x, c[j].x, ar[u][j]);
            ai[u][j] = fma(v.x, c[j].y, ai[u][j]);
        }
#pragma unroll
        for (int j = 0; j < NOUT; ++j) {
            ar[u][j] = fma(-v.y, c[j].y, ar[u][j]);
            ai[u][j] = fma(v.y, c[j].x, ai[u][j]);
        }
    };
    int i = 0;
    for (; i + IC <= nin; i += IC) {
        SI v[IC][E];
#pragma unroll
        for (int k = 0; k < IC; ++k)
#pragma unroll
            for (int u = 0; u < E; ++u) v[k][u] = U.x[i + k][row[u]];
#pragma unroll
        for (int k = 0; k < IC; ++k)
#pragma unroll
            for (int u = 0; u < E; ++u) add(wide(v[k][u]), cs + (i + k) * NOUT, u);
    }
    for (; i < nin; ++i) {
        SI v[E];
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = U.x[i][row[u]];
#pragma unroll
        for (int u = 0; u < E; ++u) add(wide(v[u]), cs + i * NOUT, u);
    }
#pragma unroll
    for (int j = 0; j < NOUT; ++j) {
        if (j >= nout) break;
        double2 *y = U.y[j];
#pragma unroll
        for (int u = 0; u < E; ++u)
            if (in[u]) y[row[u]] = make_double2(ar[u][j], ai[u][j]);
        if (bi == bj || upper) continue;
        if (j > 0) __syncthreads();
#pragma unroll
        for (int u = 0; u < E; ++u) tile[tx][ty + RY * u] = make_double2(s * ar[u][j], s * ai[u][j]);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int c = ty + RY * u;  // Y(q0 + tx, p0 + c) = s Y(p0 + c, q0 + tx)
            const int64_t q = bi * 32 + c;
            if (pt < m && q < m) y[pt + m * q] = tile[c][tx];
        }
    }
}

// out = (complex64) (a + s0 c b), one column, c from the device
__global__ void __launch_bounds__(512)
    axpc_f32_sym_kernel(float2 *out, const double2 *a, const double2 *b, double2 s0, const double2 *c_dev, int64_t m,
                        float s)
{
    pdl_enter();
    constexpr int E = 2, RY = 16;
    __shared__ float2 tile[32][33];
    int bi, bj;
    tile_pair(blockIdx.x, bi, bj);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const double2 c = c_dev[0];
    const double2 sc = make_double2(s0.x * c.x - s0.y * c.y, s0.x * c.y + s0.y * c.x);
    const int64_t p = bi * 32 + tx, pt = bj * 32 + tx;
    double2 av[E], bv[E];
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int64_t q = bj * 32 + ty + RY * u;
        const bool in = p < m && q < m;
        av[u] = in ? ld_prev(a + p + m * q) : make_double2(0.0, 0.0);
        bv[u] = in ? ld_prev(b + p + m * q) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int64_t q = bj * 32 + ty + RY * u;
        const float2 v = make_float2((float)(av[u].x + sc.x * bv[u].x - sc.y * bv[u].y),
                                     (float)(av[u].y + sc.x * bv[u].y + sc.y * bv[u].x));
        if (p < m && q < m) out[p + m * q] = v;
        tile[tx][ty + RY * u] = make_float2(s * v.x, s * v.y);
    }
    if (bi == bj) return;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int cc = ty + RY * u;
        const int64_t q = bi * 32 + cc;
        if (pt < m && q < m) out[pt + m * q] = tile[cc][tx];
    }
}

struct ResArgs {
    double2 *x[16], *ax[16];
    void *w[16];
    const double2 *n2, *e;  // <x, x> and <x, A x> (conjugated: <A x, x>) of the columns as they come in
    double2 *e_out;
    int conj;
};

// The end of an outer iteration (lamod.f90:94-126, gplmr.F90:128-139) in one
// pass: x and A x scaled to |x| = 1, E = <x, A x>, the residual w = A x - E x in
// SW (complex64 where the inner solve takes it next) and the partial sums of
// |w|^2.  x and A x are read and written in their upper tiles, w is written in
// full: 3 vector passes (2.5 for complex64) against 9 in separate kernels.
template <class SW>
__global__ void __launch_bounds__(256, 2)
    residual_sym_kernel(const __grid_constant__ ResArgs A, int64_t m, double s, double2 *partial)
{
    pdl_enter();
    constexpr int E = 4, RY = 8;
    __shared__ SW tile[32][33];
    __shared__ double2 ec;
    __shared__ double sc, red[8];
    const int col = blockIdx.y;
    if (threadIdx.x == 0) {
        const double2 n = A.n2[col], e = A.e[col];
        const double c = 1.0 / sqrt(hypot(n.x, n.y)), c2 = c * c;
        sc = c;
        ec = make_double2(c2 * e.x, A.conj ? -c2 * e.y : c2 * e.y);
        if (blockIdx.x == 0) A.e_out[col] = ec;
    }
    int bi, bj;
    tile_pair(blockIdx.x, bi, bj);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t p = bi * 32 + tx, pt = bj * 32 + tx;
    double2 *x = A.x[col], *ax = A.ax[col];
    SW *w = static_cast<SW *>(A.w[col]);
    double2 xv[E], av[E];
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int64_t q = bj * 32 + ty + RY * u;
        const bool in = p < m && q < m;
        xv[u] = in ? x[p + m * q] : make_double2(0.0, 0.0);
        av[u] = in ? ax[p + m * q] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    const double c = sc;
    const double2 e = ec;
    double sum = 0.0;
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int64_t q = bj * 32 + ty + RY * u;
        xv[u].x *= c;
        xv[u].y *= c;
        av[u].x *= c;
        av[u].y *= c;
        const double2 v = make_double2(av[u].x - e.x * xv[u].x + e.y * xv[u].y, av[u].y - e.x * xv[u].y - e.y * xv[u].x);
        SW o;
        o.x = v.x;
        o.y = v.y;
        if (p < m && q < m) {
            x[p + m * q] = xv[u];
            ax[p + m * q] = av[u];
            w[p + m * q] = o;
        }
        sum = fma(v.x, v.x, sum);
        sum = fma(v.y, v.y, sum);
        o.x = s * o.x;
        o.y = s * o.y;
        tile[tx][ty + RY * u] = o;
    }
    __syncthreads();
    if (bi != bj) {
        sum *= 2.0;  // the tile below the diagonal
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int cc = ty + RY * u;
            const int64_t q = bi * 32 + cc;
            if (pt < m && q < m) w[pt + m * q] = tile[cc][tx];
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
    if (tx == 0) red[ty] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < 8; ++k) t += red[k];
        partial[(int64_t)col * gridDim.x + blockIdx.x] = make_double2(t, 0.0);
    }
}

template <class SW>
cudaError_t residual_go(double2 *const *x, double2 *const *ax, SW *const *w, int n, const double2 *n2, const double2 *e,
                        int conj, double2 *e_out, double2 *r2, int64_t m, double s, double2 *work, cudaStream_t st)
{
    if (!sym_rows_supported(m) || n < 1 || n > 16) return cudaErrorInvalidValue;
    ResArgs A{};
    for (int j = 0; j < n; ++j) {
        A.x[j] = x[j];
        A.ax[j] = ax[j];
        A.w[j] = w[j];
    }
    A.n2 = n2;
    A.e = e;
    A.e_out = e_out;
    A.conj = conj;
    const int64_t nblk = residual_sym_work_elems(1, m);
    cudaError_t er = pdl_launch(residual_sym_kernel<SW>, dim3((unsigned)nblk, n), 256, 0, st, A, m, s, work + 1);
    return er != cudaSuccess ? er : dotdiag_reduce_launch(work + 1, (int)nblk, n, r2, st);
}

template <class SI, int NOUT, int E, int IC>
cudaError_t go(const UpdListT<SI, double2> &U, const double2 *c, int ldc, int64_t m, double s, bool upper, cudaStream_t st)
{
    const int64_t t = (m + 31) / 32;
    return pdl_launch(update_sym_kernel<SI, NOUT, E, IC>, (unsigned)(t * (t + 1) / 2), 1024 / E,
                      (size_t)U.nin * NOUT * sizeof(double2), st, U, c, ldc, m, s, (int)upper);
}

template <class SI>
cudaError_t any(const UpdListT<SI, double2> &U, const double2 *c, int ldc, int64_t m, double s, bool upper,
                cudaStream_t st)
{
    if (!update_sym_supported(m, U.nout) || U.nin < 1 || U.nin > kMaxCols) return cudaErrorInvalidValue;
    if (U.nout <= 1) return go<SI, 1, 4, 4>(U, c, ldc, m, s, upper, st);
    if (U.nout <= 2) return go<SI, 2, 4, 2>(U, c, ldc, m, s, upper, st);
    if (U.nout <= 4) return go<SI, 4, 4, 2>(U, c, ldc, m, s, upper, st);
    return go<SI, 8, 2, 2>(U, c, ldc, m, s, upper, st);
}

}  // namespace

// Small grids have too few tile pairs for the SMs (276 at M = 729, 903 at
// 1331); there the vectors sit in L2 and the general update is as fast.
bool sym_rows_supported(int64_t m) { return m >= 1000 && m <= 46000; }
bool update_sym_supported(int64_t m, int nout) { return sym_rows_supported(m) && nout >= 1 && nout <= 8; }

cudaError_t update_sym_launch(const UpdList &U, const double2 *c_dev, int ldc, int64_t m, double s, cudaStream_t st,
                              bool upper)
{
    return any(U, c_dev, ldc, m, s, upper, st);
}

cudaError_t update_sym_launch(const UpdListT<float2, double2> &U, const double2 *c_dev, int ldc, int64_t m, double s,
                              cudaStream_t st)
{
    return any(U, c_dev, ldc, m, s, false, st);
}

cudaError_t axpc_f32_sym_launch(float2 *out, const double2 *a, const double2 *b, double2 s0, const double2 *c_dev,
                                int64_t m, double s, cudaStream_t st)
{
    if (!sym_rows_supported(m) || !c_dev) return cudaErrorInvalidValue;
    const int64_t t = (m + 31) / 32;
    return pdl_launch(axpc_f32_sym_kernel, (unsigned)(t * (t + 1) / 2), 512, 0, st, out, a, b, s0, c_dev, m, (float)s);
}

int64_t residual_sym_work_elems(int n, int64_t m)
{
    const int64_t t = (m + 31) / 32;
    return n * (t * (t + 1) / 2);
}

cudaError_t residual_sym_launch(double2 *const *x, double2 *const *ax, double2 *const *w, int n, const double2 *n2,
                                const double2 *e, int conj, double2 *e_out, double2 *r2, int64_t m, double s,
                                double2 *work, cudaStream_t st)
{
    return residual_go(x, ax, w, n, n2, e, conj, e_out, r2, m, s, work, st);
}

cudaError_t residual_sym_launch(double2 *const *x, double2 *const *ax, float2 *const *w, int n, const double2 *n2,
                                const double2 *e, int conj, double2 *e_out, double2 *r2, int64_t m, double s,
                                double2 *work, cudaStream_t st)
{
    return residual_go(x, ax, w, n, n2, e, conj, e_out, r2, m, s, work, st);
}

}  // namespace de

// blockops.cu -- tall-skinny FP64 complex block operations of the GPLMR
// eigensolver and its inner solve, for sm_100a.
//
// Reference: crossmult / crossmult_diag / colnorms / normalize / cholQR
// lamod.f90:21-180, the K/M projection ZGEMMs gplmr.F90:201-277, the
// 'N','N' ZGEMM updates gplmr.F90:101-103,298-320 and the inner-solve
// products harmonic_ritz_small.F90:28-75,145,313-316.  The MPI_ALLREDUCE
// of every k x k result becomes a deterministic two-stage on-device
// reduction (per-CTA partials, then a fixed-order sum), so repeated runs
// are bitwise identical.
//
// Every kernel here streams its vectors once; they are HBM-bound except the
// 64 x 128 projection Gram, which runs on the FP64 tensor cores (gram_tc).
// The vector kernels are templated on the storage type S (double2, or
// float2 for the mixed form's inner solve); reductions accumulate in FP64,
// and only the complex64 block update (a preconditioner's combination of at
// most 40 columns) computes in FP32.
#include "de_internal.h"
#include "de_kernels.h"
#include "pdl.h"
#include "tri.h"

#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>

namespace de {

static std::atomic<int64_t> g_launches{0};
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
int64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }
bool programmatic_launch()
{
    static const bool on = [] {
        const char *v = std::getenv("DE_PDL");
        return !(v && v[0] == '0' && v[1] == 0);
    }();
    return on;
}

namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ---------------------------------------------------------------- Gram

constexpr int kGramRT = 32;  // row granularity of the Gram split over blocks
constexpr int kSmallBlocks = 296;  // grid of the fused small reductions

// element load widened to FP64
__device__ __forceinline__ double2 ld2(const double2 *p) { return __ldg(p); }
__device__ __forceinline__ double2 ld2(const float2 *p)
{
    const float2 v = __ldg(p);
    return make_double2(v.x, v.y);
}
// plain (coherent) loads, for data the same kernel may have written
__device__ __forceinline__ double2 ldp(const double2 *p) { return *p; }
__device__ __forceinline__ double2 ldp(const float2 *p)
{
    const float2 v = *p;
    return make_double2(v.x, v.y);
}
// a predecessor's data, widened
template <class S>
__device__ __forceinline__ double2 ldw_prev(const S *p)
{
    const S v = ld_prev(p);
    return make_double2(v.x, v.y);
}
template <class S>
__device__ __forceinline__ S st2(double x, double y);
template <>
__device__ __forceinline__ double2 st2<double2>(double x, double y)
{
    return make_double2(x, y);
}
template <>
__device__ __forceinline__ float2 st2<float2>(double x, double y)
{
    return make_float2((float)x, (float)y);
}

template <class S>
__device__ __forceinline__ double2 col_elem(const ColListT<S> &L, int c, int64_t r)
{
    double2 v = ld2(L.a[c] + r);
    if (L.b[c] != nullptr) {
        const double2 w = ld2(L.b[c] + r);
        v.x -= L.sigma.x * w.x - L.sigma.y * w.y;
        v.y -= L.sigma.x * w.y + L.sigma.y * w.x;
    }
    return v;
}

// One 256-thread block per 8 outputs: 32 groups take the partials of every
// 32nd block, 16 loads in flight, then a fixed tree (29 us with 8 groups of one
// warp and 1184 partials, 18 us so).
__global__ void __launch_bounds__(256)
    gram_reduce(const double2 *work, int nblk, int nl, int nr, double2 *out, int ldo)
{
    pdl_enter();
    __shared__ double2 acc[32][8];
    const int k = threadIdx.x & 7, g = threadIdx.x >> 3, o = blockIdx.x * 8 + k;
    const int nout = nl * nr;
    double sx = 0.0, sy = 0.0;
    for (int b = g; b < nblk && o < nout; b += 16 * 32) {
        double2 v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u)
            v[u] = b + 32 * u < nblk ? ld_prev(work + (int64_t)(b + 32 * u) * nout + o) : make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            sx += v[u].x;
            sy += v[u].y;
        }
    }
    acc[g][k] = make_double2(sx, sy);
    __syncthreads();
    for (int half = 16; half > 0; half >>= 1) {
        if (g < half) {
            acc[g][k].x += acc[g + half][k].x;
            acc[g][k].y += acc[g + half][k].y;
        }
        __syncthreads();
    }
    if (g == 0 && o < nout) out[o % nl + (int64_t)ldo * (o / nl)] = acc[0][k];
}

int gram_blocks(int nl, int nr, int64_t len)
{
    const int64_t tiles = (len + kGramRT - 1) / kGramRT;
    const int64_t cap = (int64_t)nl * nr > 1024 ? 296 : 148 * 8;
    return (int)std::max<int64_t>(1, std::min(tiles, cap));
}

// ---------------------------------------------------------------- update

// Arithmetic of the block update: FP32 when input and output are both
// complex64 (the mixed form's inner solve, where the sums run over at most
// 40 terms and feed a preconditioner), FP64 otherwise.
template <class SI, class SO>
struct UpdArith {
    using T = double;
    using T2 = double2;
};
template <>
struct UpdArith<float2, float2> {
    using T = float;
    using T2 = float2;
};

template <class SI, class SO, int NOUT>
__global__ void __launch_bounds__(256)
    update_kernel(const __grid_constant__ UpdListT<SI, SO> U, const double2 *C, int ldc, int64_t len)
{
    pdl_enter();
    using T = typename UpdArith<SI, SO>::T;
    using T2 = typename UpdArith<SI, SO>::T2;
    extern __shared__ __align__(16) unsigned char upd_sm[];
    T2 *cs = reinterpret_cast<T2 *>(upd_sm);  // [nin][NOUT]
    const int nin = U.nin, nout = U.nout;
    for (int idx = threadIdx.x; idx < nin * NOUT; idx += blockDim.x) {
        const int i = idx / NOUT, j = idx % NOUT;
        const double2 c = (j < nout) ? C[i + (int64_t)ldc * j] : make_double2(0.0, 0.0);
        cs[idx].x = (T)c.x;
        cs[idx].y = (T)c.y;
    }
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // from the last row to the first: an update follows the Gram that read the
    // same columns from first to last, and finds its last rows in L2
    for (int64_t r = len - 1 - ((int64_t)blockIdx.x * blockDim.x + threadIdx.x); r >= 0; r -= stride) {
        T ar[NOUT], ai[NOUT];
        double2 yb[NOUT];
#pragma unroll
        for (int j = 0; j < NOUT; ++j) {
            ar[j] = ai[j] = T(0);
            yb[j] = make_double2(0.0, 0.0);
            if (j < nout && (U.beta[j].x != 0.0 || U.beta[j].y != 0.0)) yb[j] = cmul(U.beta[j], ldp(U.y[j] + r));
        }
        // eight input columns a step, their loads issued together
        int i = 0;
        for (; i + 8 <= nin; i += 8) {
            double2 xv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) xv[u] = ldp(U.x[i + u] + r);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const T xr = (T)xv[u].x, xi = (T)xv[u].y;
#pragma unroll
                for (int j = 0; j < NOUT; ++j) {
                    const T2 c = cs[(i + u) * NOUT + j];
                    ar[j] = fma(xr, c.x, ar[j]);
                    ar[j] = fma(-xi, c.y, ar[j]);
                    ai[j] = fma(xr, c.y, ai[j]);
                    ai[j] = fma(xi, c.x, ai[j]);
                }
            }
        }
        for (; i < nin; ++i) {
            const double2 xv = ldp(U.x[i] + r);
            const T xr = (T)xv.x, xi = (T)xv.y;
#pragma unroll
            for (int j = 0; j < NOUT; ++j) {
                const T2 c = cs[i * NOUT + j];
                ar[j] = fma(xr, c.x, ar[j]);
                ar[j] = fma(-xi, c.y, ar[j]);
                ai[j] = fma(xr, c.y, ai[j]);
                ai[j] = fma(xi, c.x, ai[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < NOUT; ++j) {
            const double2 sj = cmul(U.alpha, make_double2((double)ar[j], (double)ai[j]));
            if (j < nout) U.y[j][r] = st2<SO>(yb[j].x + sj.x, yb[j].y + sj.y);
        }
    }
}

// Y = alpha sum_i X_i c_i of NC columns (one output, nothing kept of Y): the
// loads of two rows in flight before the sums.  HBM-bound; us at 4.8 M rows,
// update_kernel -> here (HBM time): 3 columns 64 -> 50 (47), 5 88 -> 76 (71),
// 7 113 -> 94 (94), 8 152 -> 105 (106).
template <int NC>
__global__ void __launch_bounds__(256, 3)
    update_col(const __grid_constant__ UpdListT<double2, double2> U, const double2 *C, int64_t len)
{
    pdl_enter();
    __shared__ double2 cs[NC];
    if (threadIdx.x < NC) cs[threadIdx.x] = cmul(U.alpha, C[threadIdx.x]);
    __syncthreads();
    const double2 *x[NC];
    double2 c[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        x[i] = U.x[i];
        c[i] = cs[i];
    }
    double2 *y = U.y[0];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // from the last row to the first, as update_kernel
    for (int64_t r = len - 1 - ((int64_t)blockIdx.x * blockDim.x + threadIdx.x); r >= 0; r -= 2 * stride) {
        const int64_t r1 = r - stride;
        double2 v0[NC], v1[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            v0[i] = ldp(x[i] + r);
            v1[i] = r1 >= 0 ? ldp(x[i] + r1) : make_double2(0.0, 0.0);
        }
        double2 s0 = make_double2(0.0, 0.0), s1 = s0;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            s0.x = fma(v0[i].x, c[i].x, s0.x);
            s0.x = fma(-v0[i].y, c[i].y, s0.x);
            s0.y = fma(v0[i].x, c[i].y, s0.y);
            s0.y = fma(v0[i].y, c[i].x, s0.y);
            s1.x = fma(v1[i].x, c[i].x, s1.x);
            s1.x = fma(-v1[i].y, c[i].y, s1.x);
            s1.y = fma(v1[i].x, c[i].y, s1.y);
            s1.y = fma(v1[i].y, c[i].x, s1.y);
        }
        y[r] = s0;
        if (r1 >= 0) y[r1] = s1;
    }
}

template <int NOUT, class SI, class SO>
cudaError_t update_go(const UpdListT<SI, SO> &U, const double2 *c, int ldc, int64_t len, cudaStream_t st)
{
    const size_t smem = (size_t)U.nin * NOUT * sizeof(typename UpdArith<SI, SO>::T2);
    const int64_t want = (len + 255) / 256;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(want, 148 * 8));
    return pdl_launch(update_kernel<SI, SO, NOUT>, blocks, 256, smem, st, U, c, ldc, len);
}

// ---------------------------------------------------------------- small

struct PtrPack {
    double2 *out[64];
    const double2 *a[64];
    const double2 *b[64];
};

__global__ void axpc_kernel(const __grid_constant__ PtrPack P, double2 s, const double2 *c_dev,
                            int64_t len)
{
    pdl_enter();
    const int j = blockIdx.y;
    double2 c = c_dev ? c_dev[j] : make_double2(1.0, 0.0);
    const double2 sc = cmul(s, c);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        const double2 av = P.a[j][r], bv = P.b[j][r];
        P.out[j][r] = make_double2(av.x + sc.x * bv.x - sc.y * bv.y, av.y + sc.x * bv.y + sc.y * bv.x);
    }
}

// out = (complex64) (a + s c b) for one column (c = c_dev[0], or 1)
__global__ void axpc_f32_kernel(float2 *out, const double2 *a, const double2 *b, double2 s, const double2 *c_dev,
                                int64_t len)
{
    pdl_enter();
    const double2 c = c_dev ? c_dev[0] : make_double2(1.0, 0.0);
    const double2 sc = cmul(s, c);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        const double2 av = a[r], bv = b[r];
        out[r] = make_float2((float)(av.x + sc.x * bv.x - sc.y * bv.y), (float)(av.y + sc.x * bv.y + sc.y * bv.x));
    }
}

// out = a + s b over n contiguous elements (FP64 arithmetic, storage S)
template <class S>
__global__ void axpy_kernel(S *out, const S *a, const S *b, double2 s, int64_t n)
{
    pdl_enter();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const double2 av = ldp(a + r), bv = ldp(b + r);
        out[r] = st2<S>(av.x + s.x * bv.x - s.y * bv.y, av.y + s.x * bv.y + s.y * bv.x);
    }
}

__global__ void scale_kernel(const __grid_constant__ PtrPack P, const double2 *c_dev, int64_t len)
{
    pdl_enter();
    const int j = blockIdx.y;
    const double2 c = c_dev[j];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride)
        P.out[j][r] = cmul(P.out[j][r], c);
}

template <bool TRI>
__global__ void dotdiag_partial(const __grid_constant__ PtrPack P, int64_t len, unsigned m, int herm,
                                double2 *__restrict__ work)
{
    pdl_enter();
    const int j = blockIdx.y;
    double sr = 0.0, si = 0.0;
    const double sg = herm ? -1.0 : 1.0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        int64_t row = r;
        double w = 1.0;
        if constexpr (TRI) {
            if (!tri_row((unsigned)r, m, row, w)) continue;
        }
        double2 a = P.a[j][row];
        const double2 b = P.b[j][row];
        if constexpr (TRI) {
            a.x *= w;
            a.y *= w;
        }
        const double ay = sg * a.y;
        sr = fma(a.x, b.x, sr);
        sr = fma(-ay, b.y, sr);
        si = fma(a.x, b.y, si);
        si = fma(ay, b.x, si);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        sr += __shfl_down_sync(0xffffffffu, sr, off);
        si += __shfl_down_sync(0xffffffffu, si, off);
    }
    __shared__ double red[2][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        red[0][w] = sr;
        red[1][w] = si;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tr = 0.0, ti = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            tr += red[0][k];
            ti += red[1][k];
        }
        work[(int64_t)j * gridDim.x + blockIdx.x] = make_double2(tr, ti);
    }
}

// One 256-thread block per output j: strided partial sums, then a fixed
// shuffle/shared-memory tree (deterministic).
__global__ void __launch_bounds__(256)
    dotdiag_reduce(const double2 *work, int nblk, int n, double2 *out)
{
    pdl_enter();
    __shared__ double2 acc[8];
    const int j = blockIdx.x;
    double sr = 0.0, si = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        const double2 v = work[(int64_t)j * nblk + b];
        sr += v.x;
        si += v.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        sr += __shfl_down_sync(0xffffffffu, sr, off);
        si += __shfl_down_sync(0xffffffffu, si, off);
    }
    if ((threadIdx.x & 31) == 0) acc[threadIdx.x >> 5] = make_double2(sr, si);
    __syncthreads();
    if (threadIdx.x == 0) {
        double x = 0.0, y = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            x += acc[k].x;
            y += acc[k].y;
        }
        out[j] = make_double2(x, y);
    }
}

__global__ void inv_sqrt_abs_kernel(const double2 *d, double2 *c, int n)
{
    pdl_enter();
    const int j = threadIdx.x;
    if (j < n) {
        const double a = sqrt(hypot(d[j].x, d[j].y));
        c[j] = make_double2(1.0 / a, 0.0);
    }
}

__global__ void tables_kernel(int nn, int n, double charge, double delta,
                              const double *__restrict__ tinv, int nbd, double *__restrict__ t1a,
                              double *__restrict__ v12)
{
    const int nb = nn;  // TINV is (-NB..NB)^3 with NB = 2N+1 (initmod.F90:39)
    const double d3 = delta * delta * delta;
    const double a = -charge / d3;
    const int64_t m = (int64_t)nn * nn * nn;
    const int w = 2 * nn - 1;
    const int64_t nv = (int64_t)w * w * w;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < m + nv; idx += stride) {
        if (idx < m) {
            const int i = (int)(idx % nn) - n, j = (int)((idx / nn) % nn) - n, k = (int)(idx / ((int64_t)nn * nn)) - n;
            t1a[idx] = a * tinv[(i + nb) + (int64_t)nbd * ((j + nb) + (int64_t)nbd * (k + nb))];
        } else {
            const int64_t v = idx - m;
            const int di = (int)(v % w) - (nn - 1), dj = (int)((v / w) % w) - (nn - 1),
                      dk = (int)(v / ((int64_t)w * w)) - (nn - 1);
            v12[v] = tinv[(di + nb) + (int64_t)nbd * ((dj + nb) + (int64_t)nbd * (dk + nb))] / d3;
        }
    }
}

// ---------------------------------------------------------------- fused
// Deterministic grid reduction without a second launch: every block writes
// its partials, then the last block to finish (atomic ticket) sums them in
// block order.  work[0] holds the ticket (zero between launches; the last
// block resets it), partials start at work + 1.

__device__ __forceinline__ bool last_block(unsigned *ticket, unsigned nblocks)
{
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = (atomicAdd(ticket, 1u) == nblocks - 1);
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

// Block-wide sum of n complex values per thread (vals[k]) into partial[k].
template <int N>
__device__ __forceinline__ void block_sum(double (&re)[N], double (&im)[N], double2 *partial, int n)
{
    __shared__ double red[2][8][32];  // [re/im][warp][value] (blockDim <= 256, N <= 32)
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        double a = re[k], b = im[k];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            a += __shfl_down_sync(0xffffffffu, a, off);
            b += __shfl_down_sync(0xffffffffu, b, off);
        }
        if (lane == 0 && k < n) {
            red[0][w][k] = a;
            red[1][w][k] = b;
        }
    }
    __syncthreads();
    if (threadIdx.x < n) {
        double a = 0.0, b = 0.0;
        for (int k = 0; k < nw; ++k) {
            a += red[0][k][threadIdx.x];
            b += red[1][k][threadIdx.x];
        }
        partial[threadIdx.x] = make_double2(a, b);
    }
}

// Final sum of nblk per-block partials part[b*stride + o], o < nout <= 32,
// by the whole 256-thread block in a fixed order: with np = nout rounded up
// to a power of two, thread t sums output t % np over the blocks
// b = t / np (mod 256 / np), then a pairwise tree in shared memory adds the
// 256 / np group sums.  The result does not depend on block timing.
template <bool DEEP = true>
__device__ __forceinline__ void reduce_partials(const double2 *__restrict__ part, unsigned nblk, int stride,
                                                int nout, double2 *res)
{
    __shared__ double2 acc[256];
    int np = 1;
    while (np < nout) np <<= 1;
    const int groups = 256 / np;
    const int o = threadIdx.x % np, g = threadIdx.x / np;
    double sx = 0.0, sy = 0.0;
    if (!DEEP && o < nout) {
#pragma unroll 4
        for (unsigned b = g; b < nblk; b += groups) {
            const double2 v = ld_l2(part + (int64_t)b * stride + o);
            sx += v.x;
            sy += v.y;
        }
    } else if (o < nout) {
        // 16 loads in flight: this tail is latency, paid by every reduction.
        // (Not in gram_small, whose main loop the compiler then schedules worse:
        // 12 x 1 at 4.8 M rows 454 us with 4 loads, 487 with 16.)
        for (unsigned b = g; b < nblk; b += 16 * groups) {
            double2 v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u)
                v[u] = b + u * groups < nblk ? ld_l2(part + (int64_t)(b + u * groups) * stride + o)
                                             : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                sx += v[u].x;
                sy += v[u].y;
            }
        }
    }
    acc[threadIdx.x] = make_double2(sx, sy);
    __syncthreads();
    for (int half = groups >> 1; half > 0; half >>= 1) {
        if (g < half) {
            const double2 u = acc[threadIdx.x + half * np];
            acc[threadIdx.x].x += u.x;
            acc[threadIdx.x].y += u.y;
        }
        __syncthreads();
    }
    if ((int)threadIdx.x < nout) res[threadIdx.x] = acc[threadIdx.x];
    __syncthreads();
}

// Grid of the fused single-launch reductions: up to 8 blocks of 256 per
// SM, capped so blocks x (outputs rounded to a power of two) fits the
// kSmallBlocks x 32 partials the scratch holds.
// One full wave: SMs x resident 256-thread blocks of the kernel (cached per
// kernel and device).
template <auto kernel>
int wave_blocks()
{
    // atomic entries: the handle-free entry point (de_dots_noalloc_d) can
    // reach this from several host threads at once; every thread computes
    // the same value, so relaxed order suffices
    static std::atomic<int> cache[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 296;
    int v = cache[dev].load(std::memory_order_relaxed);
    if (!v) {
        int sms = 0, per = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 256, 0);
        v = std::max(1, sms) * std::max(1, std::min(per, 8));
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

template <auto kernel>
int fused_blocks(int64_t len, int nout)
{
    int np = 1;
    while (np < nout) np <<= 1;
    const int64_t cap = std::min<int64_t>(wave_blocks<kernel>(), (int64_t)kSmallBlocks * 32 / np);
    return (int)std::max<int64_t>(1, std::min<int64_t>((len + 255) / 256, cap));
}

// G = op(L)^T R for nl*nr <= NLM*NRM <= 32, register accumulation over a
// grid-stride loop of rows, fused reduction.
template <class S, int NLM, int NRM>
__global__ void __launch_bounds__(256)
    gram_small(const __grid_constant__ ColListT<S> L, const __grid_constant__ ColListT<S> R, int64_t len, int herm,
               double2 *__restrict__ work, double2 *__restrict__ out, int ldo)
{
    const int nl = L.n, nr = R.n;
    double ar[NLM * NRM], ai[NLM * NRM];
#pragma unroll
    for (int k = 0; k < NLM * NRM; ++k) ar[k] = ai[k] = 0.0;
    const double sg = herm ? -1.0 : 1.0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        double2 rv[NRM];
#pragma unroll
        for (int j = 0; j < NRM; ++j) rv[j] = (j < nr) ? col_elem(R, j, r) : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < NLM; ++i) {
            if (i < nl) {
                double2 lv = col_elem(L, i, r);
                lv.y *= sg;
#pragma unroll
                for (int j = 0; j < NRM; ++j) {
                    const int k = i * NRM + j;
                    ar[k] = fma(lv.x, rv[j].x, ar[k]);
                    ar[k] = fma(-lv.y, rv[j].y, ar[k]);
                    ai[k] = fma(lv.x, rv[j].y, ai[k]);
                    ai[k] = fma(lv.y, rv[j].x, ai[k]);
                }
            }
        }
    }
    unsigned *ticket = reinterpret_cast<unsigned *>(work);
    double2 *part = work + 1;
    const int nout = NLM * NRM;
    block_sum<NLM * NRM>(ar, ai, part + (int64_t)blockIdx.x * nout, nout);
    if (last_block(ticket, gridDim.x)) {
        __shared__ double2 res[32];
        reduce_partials<false>(part, gridDim.x, nout, nout, res);
        for (int o = threadIdx.x; o < nl * nr; o += blockDim.x) {
            const int i = o / nr, j = o % nr;
            out[i + (int64_t)ldo * j] = res[i * NRM + j];
        }
        if (threadIdx.x == 0) *ticket = 0u;
    }
}

// NC columns against one: all of a row pair's loads in flight before the sums
// (gram_small checks each column's presence in between).  SELF: the one is
// the last of the NC, as in orthogonalise-and-normalise, and is read once.
// HBM-bound; inside the mixed solve at 4.8 M rows, us before -> now (HBM time):
// 3-4 columns 79 -> 44-56 (35-47), 5-8 columns 133 -> 70-108 (59-94).
template <int NC, bool SELF, bool TRI>
__global__ void __launch_bounds__(256, 2)
    gram_col(const __grid_constant__ ColListT<double2> L, const double2 *b, int64_t len, unsigned m, int herm, double2 *work,
             double2 *out)
{
    pdl_enter();
    constexpr int U = 2;
    const double2 *col[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) col[i] = L.a[i];
    double ar[NC], ai[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) ar[i] = ai[i] = 0.0;
    const double sg = herm ? -1.0 : 1.0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += U * stride) {
        double2 l[U][NC], x[U];
        double wt[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            wt[u] = 1.0;
            int64_t ru = r + u * stride;
            bool in = ru < len;
            if constexpr (TRI) in = in && tri_row((unsigned)ru, m, ru, wt[u]);
#pragma unroll
            for (int i = 0; i < NC; ++i) l[u][i] = in ? ld_prev(col[i] + ru) : make_double2(0.0, 0.0);
            if constexpr (!SELF) x[u] = in ? ld_prev(b + ru) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if constexpr (SELF) x[u] = l[u][NC - 1];
            if constexpr (TRI) {
                x[u].x *= wt[u];
                x[u].y *= wt[u];
            }
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                ar[i] = fma(l[u][i].x, x[u].x, ar[i]);
                ai[i] = fma(l[u][i].x, x[u].y, ai[i]);
            }
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                const double ly = sg * l[u][i].y;
                ar[i] = fma(-ly, x[u].y, ar[i]);
                ai[i] = fma(ly, x[u].x, ai[i]);
            }
        }
    }
    unsigned *ticket = reinterpret_cast<unsigned *>(work);
    double2 *part = work + 1;
    block_sum<NC>(ar, ai, part + (int64_t)blockIdx.x * NC, NC);
    if (last_block(ticket, gridDim.x)) {
        __shared__ double2 res[32];
        reduce_partials(part, gridDim.x, NC, NC, res);
        if (threadIdx.x < NC) out[threadIdx.x] = res[threadIdx.x];
        if (threadIdx.x == 0) *ticket = 0u;
    }
}

// Gram-Schmidt step of myhgramschmidt_many (harmonic_ritz_small.F90:52-59):
//   q -= sum_i Qp_i d_i ; v -= sum_i Vp_i d_i ; c = 1/sqrt(|<q,q>|)
// with d (m values) and the output c in device memory.
template <class S>
struct GsArgs {
    const S *qp[64];
    const S *vp[64];
    S *q, *v;
    int m;
};

template <class S>
__global__ void __launch_bounds__(256)
    gs_update(const __grid_constant__ GsArgs<S> A, const double2 *__restrict__ d, int64_t len,
              double2 *__restrict__ work, double2 *__restrict__ cout)
{
    __shared__ double2 ds[64];
    if (threadIdx.x < A.m) ds[threadIdx.x] = d[threadIdx.x];
    __syncthreads();
    double nr[1] = {0.0}, ni[1] = {0.0};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        double2 q = ldp(A.q + r), v = ldp(A.v + r);
        for (int i = 0; i < A.m; ++i) {
            const double2 c = ds[i];
            const double2 a = ldp(A.qp[i] + r), b = ldp(A.vp[i] + r);
            q.x -= a.x * c.x - a.y * c.y;
            q.y -= a.x * c.y + a.y * c.x;
            v.x -= b.x * c.x - b.y * c.y;
            v.y -= b.x * c.y + b.y * c.x;
        }
        const S qs = st2<S>(q.x, q.y);
        A.q[r] = qs;
        A.v[r] = st2<S>(v.x, v.y);
        const double2 qr = ldp(&qs);  // the norm of the stored vector
        nr[0] = fma(qr.x, qr.x, nr[0]);
        nr[0] = fma(qr.y, qr.y, nr[0]);
    }
    unsigned *ticket = reinterpret_cast<unsigned *>(work);
    double2 *part = work + 1;
    block_sum<1>(nr, ni, part + blockIdx.x, 1);
    if (last_block(ticket, gridDim.x)) {
        __shared__ double2 res[32];
        reduce_partials(part, gridDim.x, 1, 1, res);
        if (threadIdx.x == 0) {
            cout[0] = make_double2(1.0 / sqrt(fabs(res[0].x)), 0.0);
            *ticket = 0u;
        }
    }
}

template <class S>
__global__ void gs_scale(S *__restrict__ q, S *__restrict__ v, const double2 *__restrict__ c, int64_t len)
{
    const double s = c[0].x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        const double2 a = ldp(q + r), b = ldp(v + r);
        q[r] = st2<S>(a.x * s, a.y * s);
        v[r] = st2<S>(b.x * s, b.y * s);
    }
}

// Second pass of the fused two-pass Gram-Schmidt: with the pass-1
// coefficients d (device), q -= Qp d and v -= Vp d, then the pass-2
// coefficients <Qp_i, q> (i < m) are reduced into dout (m values).
template <class S, int MM>
__global__ void __launch_bounds__(256)
    gs_pass1(const __grid_constant__ GsArgs<S> A, const double2 *__restrict__ d, int64_t len,
             double2 *__restrict__ work, double2 *__restrict__ dout)
{
    __shared__ double2 ds[64];
    if (threadIdx.x < A.m) ds[threadIdx.x] = d[threadIdx.x];
    __syncthreads();
    double ar[MM + 1], ai[MM + 1];
#pragma unroll
    for (int i = 0; i <= MM; ++i) ar[i] = ai[i] = 0.0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        double2 q = ldp(A.q + r), v = ldp(A.v + r);
        double2 a[MM];
#pragma unroll
        for (int i = 0; i < MM; ++i) {
            if (i < A.m) {
                const double2 c = ds[i];
                a[i] = ldp(A.qp[i] + r);
                const double2 b = ldp(A.vp[i] + r);
                q.x -= a[i].x * c.x - a[i].y * c.y;
                q.y -= a[i].x * c.y + a[i].y * c.x;
                v.x -= b.x * c.x - b.y * c.y;
                v.y -= b.x * c.y + b.y * c.x;
            }
        }
        {
            const S qs = st2<S>(q.x, q.y);
            A.q[r] = qs;
            A.v[r] = st2<S>(v.x, v.y);
            q = ldp(&qs);  // coefficients of the stored vector
        }
#pragma unroll
        for (int i = 0; i < MM; ++i) {
            if (i < A.m) {  // conj(a_i) q
                ar[i] = fma(a[i].x, q.x, ar[i]);
                ar[i] = fma(a[i].y, q.y, ar[i]);
                ai[i] = fma(a[i].x, q.y, ai[i]);
                ai[i] = fma(-a[i].y, q.x, ai[i]);
            }
        }
        ar[MM] = fma(q.x, q.x, ar[MM]);
        ar[MM] = fma(q.y, q.y, ar[MM]);
    }
    unsigned *ticket = reinterpret_cast<unsigned *>(work);
    double2 *part = work + 1;
    block_sum<MM + 1>(ar, ai, part + (int64_t)blockIdx.x * (MM + 1), MM + 1);
    if (last_block(ticket, gridDim.x)) {
        __shared__ double2 res[32];
        reduce_partials(part, gridDim.x, MM + 1, MM + 1, res);
        for (int o = threadIdx.x; o <= MM; o += blockDim.x)
            if (o < A.m || o == MM) dout[o == MM ? 64 : o] = res[o];  // |u|^2 goes to dout[64]
        if (threadIdx.x == 0) *ticket = 0u;
    }
}

// Second pass with the normalisation folded in: q <- (q - Qp d2)/|w|,
// v <- (v - Vp d2)/|w| where |w|^2 = |u|^2 - |d2|^2 (Pythagoras; u is the
// pass-1 vector, whose component in span(Qp) is already at rounding level,
// so the subtraction loses nothing).
template <class S, int MM>
__global__ void __launch_bounds__(256)
    gs_pass2(const __grid_constant__ GsArgs<S> A, const double2 *__restrict__ d2, int64_t len, double2 *cout)
{
    __shared__ double2 ds[64];
    __shared__ double scale;
    __shared__ int project;
    if (threadIdx.x < A.m) ds[threadIdx.x] = d2[threadIdx.x];
    if (threadIdx.x == 0) {
        const double u2 = d2[64].x;
        double dd = 0.0;
        for (int i = 0; i < A.m; ++i) dd += d2[i].x * d2[i].x + d2[i].y * d2[i].y;
        scale = 1.0 / sqrt(fabs(u2 - dd));
        // complex64 storage: when the pass-2 coefficients are at its own
        // rounding level (|d2| <= 1e-6 |u|) the projection would change the
        // vectors by less than storing them does, so only the normalisation
        // is applied.  Cancellation in pass 1 (larger d2) keeps the full
        // second pass.  complex128 always projects, as the reference does.
        project = sizeof(S) == 16 || dd > 1e-12 * u2;
        if (blockIdx.x == 0) cout[0] = make_double2(scale, 0.0);
    }
    __syncthreads();
    const double sc = scale;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    if (!project) {
        for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
            const double2 q = ldp(A.q + r), v = ldp(A.v + r);
            A.q[r] = st2<S>(q.x * sc, q.y * sc);
            A.v[r] = st2<S>(v.x * sc, v.y * sc);
        }
        return;
    }
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < len; r += stride) {
        double2 q = ldp(A.q + r), v = ldp(A.v + r);
        double2 a[MM], b[MM];  // all loads first: MM independent requests in flight
#pragma unroll
        for (int i = 0; i < MM; ++i)
            if (i < A.m) {
                a[i] = ldp(A.qp[i] + r);
                b[i] = ldp(A.vp[i] + r);
            }
#pragma unroll
        for (int i = 0; i < MM; ++i)
            if (i < A.m) {
                const double2 c = ds[i];
                q.x -= a[i].x * c.x - a[i].y * c.y;
                q.y -= a[i].x * c.y + a[i].y * c.x;
                v.x -= b[i].x * c.x - b[i].y * c.y;
                v.y -= b[i].x * c.y + b[i].y * c.x;
            }
        A.q[r] = st2<S>(q.x * sc, q.y * sc);
        A.v[r] = st2<S>(v.x * sc, v.y * sc);
    }
}

// ---------------------------------------------------------------- k x k
// Dense k x k work kept on the device (k <= 16) so the solver does not stop
// for the host: one thread each, column-major, flags reported through `flag`.

// flag[0] accumulates every raised bit, flag[1] keeps the first one, so the
// error reported is the one the reference would have stopped at.
__device__ __forceinline__ void raise_flag(int *flag, int bit)
{
    atomicOr(flag, bit);
    atomicCAS(flag + 1, 0, bit);
}

// Coefficients that orthogonalise one column b against orthonormal columns
// Q (n of them) and normalise it, from g = [Q^H b; b^H b]: with |w|^2 =
// b^H b - |Q^H b|^2 (Pythagoras), coef = [-(Q^H b)/|w|; 1/|w|], so that
// w/|w| = [Q, b] coef.  A |w|^2 not above 1e-28 b^H b raises flag bit 1, as
// a cholQR breakdown does, and leaves b unchanged.
__global__ void orth_norm_coef(const double2 *g, int n, double2 *coef, int *flag)
{
    pdl_enter();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double bb = g[n].x;
    double w2 = bb;
    for (int i = 0; i < n; ++i) w2 -= g[i].x * g[i].x + g[i].y * g[i].y;
    if (!(w2 > 1e-28 * bb)) {
        raise_flag(flag, 1);
        for (int i = 0; i < n; ++i) coef[i] = make_double2(0.0, 0.0);
        coef[n] = make_double2(1.0, 0.0);
        return;
    }
    const double r = 1.0 / sqrt(w2);
    for (int i = 0; i < n; ++i) coef[i] = make_double2(-g[i].x * r, -g[i].y * r);
    coef[n] = make_double2(r, 0.0);
}

// Right-looking Cholesky of the k x k matrix A in shared memory by the whole
// block: A's upper triangle becomes R, inv its reciprocal diagonal; false on
// breakdown.  The entries of a step are independent; one thread walking them
// (and waiting for global memory at each) took 10 us at k = 4, 14 us for the 5
// x 5 system of the power basis, against 4-5 us.
__device__ __forceinline__ bool block_cholesky(double2 *A, double *inv, int k)
{
    for (int j = 0; j < k; ++j) {
        const double dj = A[j + k * j].x;  // the same for every thread
        if (!(dj > 0.0) || !isfinite(dj)) return false;
        const double rjj = sqrt(dj), r = 1.0 / rjj;
        __syncthreads();
        if (threadIdx.x == 0) {
            A[j + k * j] = make_double2(rjj, 0.0);
            inv[j] = r;
        }
        for (int l = j + 1 + threadIdx.x; l < k; l += blockDim.x) {
            A[j + k * l].x *= r;
            A[j + k * l].y *= r;
        }
        __syncthreads();
        const int n = k - j - 1;
        for (int o = threadIdx.x; o < n * n; o += blockDim.x) {
            const int i = j + 1 + o % n, l = j + 1 + o / n;
            if (i > l) continue;
            const double2 p = A[j + k * i], q = A[j + k * l];  // A(i,l) -= conj(R(j,i)) R(j,l)
            A[i + k * l].x -= p.x * q.x + p.y * q.y;
            A[i + k * l].y -= p.x * q.y - p.y * q.x;
        }
        __syncthreads();
    }
    return true;
}

// X = R^-1 of the upper factor of block_cholesky, a column per thread by back
// substitution; X is zero below the diagonal on entry.
__device__ __forceinline__ void block_upper_inverse(const double2 *R, const double *inv, double2 *X, int k)
{
    if ((int)threadIdx.x < k) {
        const int j = threadIdx.x;
        for (int i = j; i >= 0; --i) {
            double2 s = make_double2(i == j ? 1.0 : 0.0, 0.0);
            for (int l = i + 1; l <= j; ++l) {
                const double2 a = R[i + k * l], b = X[l + k * j];
                s.x -= a.x * b.x - a.y * b.y;
                s.y -= a.x * b.y + a.y * b.x;
            }
            X[i + k * j] = make_double2(s.x * inv[i], s.y * inv[i]);
        }
    }
}

// Upper Cholesky R of the Hermitian G (upper triangle read, as zpotrf 'U')
// and R^{-1}.  flag |= 1 on breakdown, 2 when G is all zero.
__global__ void __launch_bounds__(64)
    small_cholinv(const double2 *G, int k, double2 *Rinv, int *flag)
{
    pdl_enter();
    __shared__ double2 R[16 * 16], X[16 * 16];
    __shared__ double inv[16];
    bool nonzero = false;
    for (int o = threadIdx.x; o < k * k; o += blockDim.x) {
        R[o] = G[o];
        X[o] = make_double2(0.0, 0.0);
        nonzero = nonzero || !(R[o].x == 0.0 && R[o].y == 0.0);
    }
    const bool any = __syncthreads_or(nonzero);
    if (!any || !block_cholesky(R, inv, k)) {
        if (threadIdx.x == 0) raise_flag(flag, any ? 1 : 2);
        return;
    }
    block_upper_inverse(R, inv, X, k);
    __syncthreads();
    for (int o = threadIdx.x; o < k * k; o += blockDim.x) Rinv[o] = X[o];
}

// The second Gram-Schmidt pass and the first CholQR of a block in one update:
// with B = Q^H W (g's first m rows), |W - Q B|^2 = W^H W - B^H B (Pythagoras), so
// the factor R needs no further Gram.  W has been through the first pass, so B is
// of the order of its rounding and nothing cancels -- unless all of W is
// rounding, when half of a column or more may go: then the pass is done alone (R
// = 1) and the CholQR that follows normalises.
__global__ void __launch_bounds__(256)
    small_orth_chol(const double2 *g, int m, int k, double2 *rinv, double2 *c, int *flag)
{
    pdl_enter();
    __shared__ double2 B[64 * 16], R[16 * 16], X[16 * 16];
    __shared__ double inv[16];
    const int ld = m + k;
    for (int o = threadIdx.x; o < ld * k; o += blockDim.x) {
        const int i = o % ld, j = o / ld;
        if (i < m) B[i + m * j] = g[o];
        else R[i - m + k * j] = g[o];
    }
    for (int o = threadIdx.x; o < k * k; o += blockDim.x) X[o] = make_double2(0.0, 0.0);
    __syncthreads();
    bool lost = false;
    if ((int)threadIdx.x < k * k) {
        const int i = threadIdx.x % k, j = threadIdx.x / k;
        double2 s = R[threadIdx.x];
        const double before = s.x;
        for (int l = 0; l < m; ++l) {
            const double2 p = B[l + m * i], q = B[l + m * j];
            s.x -= p.x * q.x + p.y * q.y;
            s.y -= p.x * q.y - p.y * q.x;
        }
        R[threadIdx.x] = s;
        lost = i == j && !(s.x > 0.5 * before);
    }
    if (__syncthreads_or(lost)) {
        for (int j = threadIdx.x; j < k; j += blockDim.x) X[j + k * j] = make_double2(1.0, 0.0);
    } else {
        if (!block_cholesky(R, inv, k)) {
            if (threadIdx.x == 0) raise_flag(flag, 1);
            return;
        }
        block_upper_inverse(R, inv, X, k);
    }
    __syncthreads();
    for (int o = threadIdx.x; o < k * k; o += blockDim.x) rinv[o] = X[o];
    for (int o = threadIdx.x; o < ld * k; o += blockDim.x) {
        const int i = o % ld, j = o / ld;
        double2 s = i >= m ? X[i - m + k * j] : make_double2(0.0, 0.0);
        for (int l = 0; i < m && l <= j; ++l) {
            const double2 p = cmul(B[i + m * l], X[l + k * j]);
            s.x -= p.x;
            s.y -= p.y;
        }
        c[o] = s;
    }
}

// C = [-(G1 + G2) W; W] with W = R1^-1 R2^-1: G1, G2 m x k (ld m and ld2), the
// rest k x k, C (m + k) x k (ld m + k), k <= 16.
__global__ void __launch_bounds__(256)
    small_block_coef(const double2 *g1, const double2 *g2, int ld2, int m, int k, const double2 *r1, const double2 *r2,
                     double2 *c)
{
    pdl_enter();
    __shared__ double2 w[16 * 16];
    if ((int)threadIdx.x < k * k) {
        const int i = threadIdx.x % k, j = threadIdx.x / k;
        double2 s = make_double2(0.0, 0.0);
        for (int l = 0; l < k; ++l) {
            const double2 p = cmul(r1[i + k * l], r2[l + k * j]);
            s.x += p.x;
            s.y += p.y;
        }
        w[threadIdx.x] = s;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < (m + k) * k; o += blockDim.x) {
        const int i = o % (m + k), j = o / (m + k);
        double2 s = i >= m ? w[i - m + k * j] : make_double2(0.0, 0.0);
        for (int l = 0; i < m && l < k; ++l) {
            const double2 a = g1[i + m * l], b = g2[i + ld2 * l];
            const double2 p = cmul(make_double2(a.x + b.x, a.y + b.y), w[l + k * j]);
            s.x -= p.x;
            s.y -= p.y;
        }
        c[o] = s;
    }
}

// 1 x 1 case of gen_cmatsub flag 2 (hr_eigen.f90:223-291): g > 0 real.
__global__ void small_hsqrt1(const double2 *__restrict__ g, double2 *__restrict__ ginvh, double2 *__restrict__ gsq,
                             int *flag)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double s = hypot(g[0].x, g[0].y);  // the singular value of the 1 x 1 matrix
    if (!(s > 0.0)) {
        raise_flag(flag, 8);
        return;
    }
    ginvh[0] = make_double2(sqrt(1.0 / s), 0.0);
    gsq[0] = make_double2(sqrt(s), 0.0);
}

// harm_orthog_oneblock's self-check (harmonic_ritz_small.F90:221-242):
// flag |= 4 when any |T - I| > 1e-10.
__global__ void small_ortho_check(const double2 *t, int k, double tol, int *flag)
{
    pdl_enter();
    const int o = threadIdx.x;
    if (o < k * k) {
        const int i = o % k, j = o / k;
        const double re = t[o].x - (i == j ? 1.0 : 0.0);
        if (!(hypot(re, t[o].y) <= tol)) raise_flag(flag, 4);
    }
}

// C (m x n) = A (m x k) B (k x n), all small, column-major.
__global__ void small_gemm(const double2 *__restrict__ A, const double2 *__restrict__ B, double2 *__restrict__ C,
                           int m, int k, int n)
{
    const int o = threadIdx.x + blockIdx.x * blockDim.x;
    if (o >= m * n) return;
    const int i = o % m, j = o / m;
    double2 s = make_double2(0.0, 0.0);
    for (int l = 0; l < k; ++l) {
        const double2 a = A[i + (int64_t)m * l], b = B[l + (int64_t)k * j];
        s.x += a.x * b.x - a.y * b.y;
        s.y += a.x * b.y + a.y * b.x;
    }
    C[o] = s;
}

// Electron-exchange symmetry of an M x M block X (column-major, X(p,q) at
// p + M q).  Tile pair (bi <= bj) of 32 x 32 tiles: PROJECT replaces X by
// (X + s X^T)/2 in place (s = +1 singlet, -1 triplet); otherwise the block's
// shares of |(X - X^T)/2|^2 and |(X + X^T)/2|^2 go to work[block].  The parts are
// summed, and not <X, X^T> = their difference, in which a part of norm 1e-8
// leaves no digit.
template <bool PROJECT>
__global__ void __launch_bounds__(256)
    exch_kernel(double2 *__restrict__ x, int64_t m, double s, double2 *__restrict__ work)
{
    __shared__ double2 ta[32][33], tb[32][33];
    const int bi = blockIdx.x, bj = blockIdx.y;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    double sr = 0.0, si = 0.0;
    if (bi <= bj) {
        const int64_t p0 = (int64_t)bi * 32, q0 = (int64_t)bj * 32;
        // ta[r][c] = X(p0 + r, q0 + c); tb[r][c] = X(q0 + r, p0 + c)
        for (int c = ty; c < 32; c += 8) {
            const int64_t pa = p0 + tx, qa = q0 + c, pb = q0 + tx, qb = p0 + c;
            ta[tx][c] = (pa < m && qa < m) ? x[pa + m * qa] : make_double2(0.0, 0.0);
            tb[tx][c] = (pb < m && qb < m) ? x[pb + m * qb] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        if (PROJECT) {
            for (int c = ty; c < 32; c += 8) {
                const int64_t pa = p0 + tx, qa = q0 + c, pb = q0 + tx, qb = p0 + c;
                // X^T(p,q) = X(q,p): ta[r][c]^T partner is tb[c][r]
                const double2 a = ta[tx][c], at = tb[c][tx], b = tb[tx][c], bt = ta[c][tx];
                if (pa < m && qa < m) x[pa + m * qa] = make_double2(0.5 * (a.x + s * at.x), 0.5 * (a.y + s * at.y));
                if (bi != bj && pb < m && qb < m)
                    x[pb + m * qb] = make_double2(0.5 * (b.x + s * bt.x), 0.5 * (b.y + s * bt.y));
            }
        } else {
            for (int c = ty; c < 32; c += 8) {
                // pairs (p0+tx, q0+c) and its transpose partner
                const double2 a = ta[tx][c], at = tb[c][tx];
                const double dx = a.x - at.x, dy = a.y - at.y, ex = a.x + at.x, ey = a.y + at.y;
                const double w = bi != bj ? 0.5 : 0.25;  // the partner tile's pair has the same two parts
                sr += w * (dx * dx + dy * dy);
                si += w * (ex * ex + ey * ey);
            }
        }
    }
    if (!PROJECT) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            sr += __shfl_down_sync(0xffffffffu, sr, off);
            si += __shfl_down_sync(0xffffffffu, si, off);
        }
        __shared__ double2 red[8];
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_double2(sr, si);
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = 0.0, b = 0.0;
            for (int k = 0; k < 8; ++k) {
                a += red[k].x;
                b += red[k].y;
            }
            work[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = make_double2(a, b);
        }
    }
}

__global__ void cvt_c2f_kernel(const double2 *x, float2 *y, int64_t n)
{
    pdl_enter();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const double2 v = x[i];
        y[i] = make_float2((float)v.x, (float)v.y);
    }
}

__global__ void cvt_r2f_kernel(const double *__restrict__ x, float *__restrict__ y, int64_t n)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) y[i] = (float)x[i];
}

// Y = sum_i Z_i a_i (complex64 columns, coefficients on the device) and the
// exchange projection Y <- (Y + s Y^T)/2 in one pass: a block forms the
// 32 x 32 tile of Y at (p0, q0) and its transpose partner at (q0, p0) from
// the inputs, then writes both projected.  Blocks below the diagonal leave
// at once (their tiles are their partners').
constexpr int kUxMaxIn = 8;
struct UxArgs {
    const float2 *z[kUxMaxIn];
    int nz;
};

template <int NZ>
__global__ void __launch_bounds__(256)
    update_exch_kernel(const __grid_constant__ UxArgs A, const double2 *__restrict__ coef, double2 *__restrict__ y,
                       int64_t m, double s, int t)
{
    __shared__ double2 ta[32][33], tb[32][33];
    // blocks enumerate the tiles on and above the diagonal: bi <= bj
    int bj = (int)((sqrt(8.0 * blockIdx.x + 1.0) - 1.0) * 0.5);
    while ((bj + 1) * (bj + 2) / 2 <= (int)blockIdx.x) ++bj;
    while (bj * (bj + 1) / 2 > (int)blockIdx.x) --bj;
    const int bi = (int)blockIdx.x - bj * (bj + 1) / 2;
    if (bj >= t) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const int64_t p0 = (int64_t)bi * 32, q0 = (int64_t)bj * 32;
    double2 c[NZ];
#pragma unroll
    for (int i = 0; i < NZ; ++i) c[i] = coef[i];
    const int64_t pa = p0 + tx, pb = q0 + tx;
    // every input of the thread's 4 + 4 elements in flight before the sums
    float2 za[4][NZ], zb[4][NZ];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int cc = ty + 8 * u;
        const int64_t qa = q0 + cc, qb = p0 + cc;
        const bool oka = pa < m && qa < m, okb = pb < m && qb < m;
#pragma unroll
        for (int i = 0; i < NZ; ++i) {
            za[u][i] = oka ? __ldg(A.z[i] + pa + m * qa) : make_float2(0.f, 0.f);
            zb[u][i] = okb ? __ldg(A.z[i] + pb + m * qb) : make_float2(0.f, 0.f);
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int cc = ty + 8 * u;
        double ar = 0.0, ai = 0.0, br = 0.0, bim = 0.0;
#pragma unroll
        for (int i = 0; i < NZ; ++i) {
            ar += (double)za[u][i].x * c[i].x - (double)za[u][i].y * c[i].y;
            ai += (double)za[u][i].x * c[i].y + (double)za[u][i].y * c[i].x;
            br += (double)zb[u][i].x * c[i].x - (double)zb[u][i].y * c[i].y;
            bim += (double)zb[u][i].x * c[i].y + (double)zb[u][i].y * c[i].x;
        }
        // ta[r][cc] = Y(p0 + r, q0 + cc), tb[r][cc] = Y(q0 + r, p0 + cc)
        ta[tx][cc] = make_double2(ar, ai);
        tb[tx][cc] = make_double2(br, bim);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int cc = ty + 8 * u;
        const int64_t qa = q0 + cc, qb = p0 + cc;
        // Y^T(p, q) = Y(q, p): the partner of ta[r][cc] is tb[cc][r]
        const double2 a = ta[tx][cc], at = tb[cc][tx], b = tb[tx][cc], bt = ta[cc][tx];
        if (pa < m && qa < m) y[pa + m * qa] = make_double2(0.5 * (a.x + s * at.x), 0.5 * (a.y + s * at.y));
        if (bi != bj && pb < m && qb < m) y[pb + m * qb] = make_double2(0.5 * (b.x + s * bt.x), 0.5 * (b.y + s * bt.y));
    }
}

int stream_blocks(int64_t len)
{
    return (int)std::max<int64_t>(1, std::min<int64_t>((len + 255) / 256, 148 * 4));
}

// Reflection sectors.  The grid is symmetric under c -> nn-1-c of each
// Cartesian axis (applied to both electrons at once), and H commutes with
// the three reflections; they generate a group of 8 elements, indexed by a
// 3-bit mask r (bit a: axis a reflected).  Its characters chi_c(r) =
// (-1)^popcount(c & r) label 8 sectors.  Element index of a vector:
// x1 + nn y1 + nn^2 z1 + nn^3 (x2 + nn y2 + nn^2 z2).
__device__ __forceinline__ int64_t refl_image(const int c[6], int r, int nn)
{
    const int m = nn - 1;
    int d[6];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const bool f = (r >> a) & 1;
        d[a] = f ? m - c[a] : c[a];
        d[a + 3] = f ? m - c[a + 3] : c[a + 3];
    }
    const int64_t n1 = nn, n2 = n1 * nn, n3 = n2 * nn;
    return d[0] + n1 * d[1] + n2 * d[2] + n3 * (d[3] + n1 * d[4] + n2 * d[5]);
}

// work[r * gridDim.x + block] = the block's share of <x, R_r x> =
// sum_i conj(x_i) x_{R_r(i)}
__global__ void __launch_bounds__(256) refl_corr_kernel(const double2 *__restrict__ x, int nn, int64_t d,
                                                        double2 *__restrict__ work)
{
    double sr[8], si[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) sr[r] = si[r] = 0.0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < d; i += stride) {
        int c[6];
        int64_t t = i;
#pragma unroll
        for (int a = 0; a < 5; ++a) {
            c[a] = (int)(t % nn);
            t /= nn;
        }
        c[5] = (int)t;
        const double2 a = x[i];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const double2 b = x[refl_image(c, r, nn)];
            sr[r] += a.x * b.x + a.y * b.y;
            si[r] += a.x * b.y - a.y * b.x;
        }
    }
    __shared__ double2 red[8][8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            sr[r] += __shfl_down_sync(0xffffffffu, sr[r], off);
            si[r] += __shfl_down_sync(0xffffffffu, si[r], off);
        }
        if ((threadIdx.x & 31) == 0) red[r][threadIdx.x >> 5] = make_double2(sr[r], si[r]);
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            a += red[threadIdx.x][w].x;
            b += red[threadIdx.x][w].y;
        }
        work[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = make_double2(a, b);
    }
}

// 8-point Walsh-Hadamard transform in place: v[c] <- sum_r (-1)^popcount(c & r) v[r]
__device__ __forceinline__ void wht8(double2 v[8])
{
#pragma unroll
    for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (!(r & h)) {
                const double2 a = v[r], b = v[r | h];
                v[r] = make_double2(a.x + b.x, a.y + b.y);
                v[r | h] = make_double2(a.x - b.x, a.y - b.y);
            }
}

// In-place projection onto the sectors whose bit is set in keep: one thread
// per orbit of the group.  The orbit's canonical element has, on every axis,
// its electron pair (c1, c2) with c1 < N, or c1 = N and c2 <= N (N = nn/2),
// so there are K = N nn + N + 1 canonical pairs per axis and K^3 orbits.
// The thread reads the orbit's 8 values, transforms them to the sector
// components (wht8), zeroes the sectors not kept, transforms back (/8) and
// writes the 8 values.  A pair (N, N) is its own reflection; the orbit then
// repeats elements, and every copy of an element receives the same value.
__global__ void __launch_bounds__(256) refl_project_kernel(double2 *__restrict__ x, int nn, unsigned keep)
{
    const int n = nn / 2, k = n * nn + n + 1;
    const int64_t orbits = (int64_t)k * k * k;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < orbits; t += stride) {
        int c[6];
        int64_t u = t;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int q = (int)(u % k);
            u /= k;
            if (q < n * nn) {
                c[a] = q % n;
                c[a + 3] = q / n;
            } else {
                c[a] = n;
                c[a + 3] = q - n * nn;
            }
        }
        double2 v[8];
        int64_t idx[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            idx[r] = refl_image(c, r, nn);
            v[r] = x[idx[r]];
        }
        wht8(v);
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (!((keep >> r) & 1)) v[r] = make_double2(0.0, 0.0);
        wht8(v);
#pragma unroll
        for (int r = 0; r < 8; ++r) x[idx[r]] = make_double2(0.125 * v[r].x, 0.125 * v[r].y);
    }
}

}  // namespace

int64_t gram_work_elems(int nl, int nr, int64_t len)
{
    // tiled partials, or one 32-output partial per block of a fused launch
    // (at most one wave: 8 blocks on each of up to 512 SMs)
    return 1 + std::max<int64_t>((int64_t)gram_blocks(nl, nr, len) * nl * nr, 4096LL * 32);
}

template <int A, int B, class S>
static cudaError_t gram_small_go(const ColListT<S> &L, const ColListT<S> &R, int64_t len, int herm, double2 *out,
                                 int ldo, double2 *work, cudaStream_t st)
{
    const int blocks = fused_blocks<gram_small<S, A, B>>(len, A * B);
    gram_small<S, A, B><<<blocks, 256, 0, st>>>(L, R, len, herm, work, out, ldo);
    count_launch();
    return cudaGetLastError();
}

template <class S>
static cudaError_t gs_update_go(const S *const *qp, const S *const *vp, int m, S *q, S *v, const double2 *d,
                                int64_t len, double2 *work, double2 *cout, cudaStream_t st)
{
    if (m < 0 || m > 64) return cudaErrorInvalidValue;
    GsArgs<S> A{};
    for (int i = 0; i < m; ++i) {
        A.qp[i] = qp[i];
        A.vp[i] = vp[i];
    }
    A.q = q;
    A.v = v;
    A.m = m;
    const int blocks = fused_blocks<gs_update<S>>(len, 1);
    gs_update<S><<<blocks, 256, 0, st>>>(A, d, len, work, cout);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    gs_scale<S><<<blocks, 256, 0, st>>>(q, v, cout, len);
    count_launch();
    return cudaGetLastError();
}

cudaError_t gs_update_launch(const double2 *const *qp, const double2 *const *vp, int m, double2 *q, double2 *v,
                             const double2 *d, int64_t len, double2 *work, double2 *cout, cudaStream_t st)
{
    return gs_update_go(qp, vp, m, q, v, d, len, work, cout, st);
}

cudaError_t gs_update_launch(const float2 *const *qp, const float2 *const *vp, int m, float2 *q, float2 *v,
                             const double2 *d, int64_t len, double2 *work, double2 *cout, cudaStream_t st)
{
    return gs_update_go(qp, vp, m, q, v, d, len, work, cout, st);
}

// ---------------------------------------------------------------- Gram on the FP64 tensor cores
// G = op(L)^T R as real GEMMs over the rows on DMMA (mma.sync m8n8k4 f64):
// with L = Lr + i Li, R = Rr + i Ri,
//   Re G = Lr^T Rr + s Li^T Ri,  Im G = Lr^T Ri - s Li^T Rr  (s = +1 for
//   conj(L), -1 for L),
// A fragments straight from L (lane: row r0 + lane%4, column i0 + lane/4),
// B fragments from R (row r0 + lane%4, column j0 + lane/4): one 16-byte
// load gives a lane both components.  A warp owns MTW x NTW 8x8 output
// tiles; a block holds WM x WN warps covering all outputs, times RG row
// groups that take interleaved 4-row steps of the block's row range.  Block
// partials go to work[block][nl*nr] (column-major) for gram_reduce.

__device__ __forceinline__ void dmma_g(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// KM8: the harmonic projection of one column with a P block (8 x 16): L
// columns are b_c = a_c - sigma v_c (c < 8) and R is [b_0..b_7, v_0..v_7],
// so a lane's two loads (a_c, v_c of its column c) give its L fragment and
// both R fragments.
template <class S, int MTW, int NTW, bool KM8, bool TRI>
__global__ void __launch_bounds__(512)
    gram_tc(const __grid_constant__ ColListT<S> L, const __grid_constant__ ColListT<S> R, int64_t len, int64_t chunk,
            unsigned m, int herm, int wm, int wn, int rg, double2 *__restrict__ work)
{
    pdl_enter();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = wm * wn;
    const int g = warp / per, wt = warp - g * per;
    const int wi = wt % wm, wj = wt / wm;
    const int nl = L.n, nr = R.n;
    const double sg = herm ? 1.0 : -1.0;
    const int q4 = lane & 3, r8 = lane >> 2;
    double re[MTW][NTW][2], im[MTW][NTW][2];
#pragma unroll
    for (int a = 0; a < MTW; ++a)
#pragma unroll
        for (int b = 0; b < NTW; ++b) re[a][b][0] = re[a][b][1] = im[a][b][0] = im[a][b][1] = 0.0;
    const int64_t r0 = (int64_t)blockIdx.x * chunk;
    const int64_t r1 = min(len, r0 + chunk);
    // The lane's column pointers, read once: indexing the parameter lists
    // with a lane-dependent column inside the loop would serialise the
    // constant-cache reads of every load.
    const S *la[MTW], *lb[MTW], *ra[NTW], *rbp[NTW];
#pragma unroll
    for (int a = 0; a < MTW; ++a) {
        const int i = 8 * (wi * MTW + a) + r8;
        la[a] = i < nl ? L.a[i] : nullptr;
        lb[a] = i < nl ? L.b[i] : nullptr;
    }
#pragma unroll
    for (int b = 0; b < NTW; ++b) {
        const int j = 8 * (wj * NTW + b) + r8;
        ra[b] = j < nr ? R.a[j] : nullptr;
        rbp[b] = j < nr ? R.b[j] : nullptr;
    }
    auto elem = [](const S *pa, const S *pb, double2 sgm, int64_t r) {
        double2 v = ldw_prev(pa + r);
        if (pb) {
            const double2 w = ldw_prev(pb + r);
            v.x -= sgm.x * w.x - sgm.y * w.y;
            v.y -= sgm.x * w.y + sgm.y * w.x;
        }
        return v;
    };
    // two 4-row steps an iteration for the small warp tiles, their loads
    // issued first
    constexpr int US = MTW * NTW >= 4 ? 1 : 2;
    for (int64_t rb = r0 + 4 * (int64_t)g; rb < r1; rb += 4 * US * (int64_t)rg) {
        double2 lv[US][MTW], rv[US][NTW];
#pragma unroll
        for (int u = 0; u < US; ++u) {
            int64_t r = rb + 4 * (int64_t)rg * u + q4;
            bool rok = r < r1;
            double wt = 1.0;
            if constexpr (TRI) rok = rok && tri_row((unsigned)r, m, r, wt);
            if constexpr (KM8) {
                const double2 av = rok ? ldw_prev(la[0] + r) : make_double2(0.0, 0.0);
                const double2 v = rok ? ldw_prev(lb[0] + r) : make_double2(0.0, 0.0);
                const double2 sgm = L.sigma;
                lv[u][0] = make_double2(av.x - (sgm.x * v.x - sgm.y * v.y), av.y - (sgm.x * v.y + sgm.y * v.x));
                rv[u][0] = lv[u][0];
                rv[u][NTW - 1] = v;
            } else {
#pragma unroll
                for (int a = 0; a < MTW; ++a)
                    lv[u][a] = (rok && la[a]) ? elem(la[a], lb[a], L.sigma, r) : make_double2(0.0, 0.0);
#pragma unroll
                for (int b = 0; b < NTW; ++b)
                    rv[u][b] = (rok && ra[b]) ? elem(ra[b], rbp[b], R.sigma, r) : make_double2(0.0, 0.0);
            }
            if constexpr (TRI) {
#pragma unroll
                for (int b = 0; b < NTW; ++b) {
                    rv[u][b].x *= wt;
                    rv[u][b].y *= wt;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < US; ++u)
#pragma unroll
            for (int a = 0; a < MTW; ++a)
#pragma unroll
                for (int b = 0; b < NTW; ++b) {
                    dmma_g(re[a][b][0], re[a][b][1], lv[u][a].x, rv[u][b].x);
                    dmma_g(re[a][b][0], re[a][b][1], lv[u][a].y, sg * rv[u][b].y);
                    dmma_g(im[a][b][0], im[a][b][1], lv[u][a].x, rv[u][b].y);
                    dmma_g(im[a][b][0], im[a][b][1], lv[u][a].y, -sg * rv[u][b].x);
                }
    }
    // sum the row groups in shared memory (fixed order), then one partial per block
    extern __shared__ double2 gtc_sm[];  // [rg][per*32][MTW*NTW*2]
    constexpr int V = MTW * NTW * 2;
    double2 *mine = gtc_sm + ((int64_t)g * per * 32 + wt * 32 + lane) * V;
#pragma unroll
    for (int a = 0; a < MTW; ++a)
#pragma unroll
        for (int b = 0; b < NTW; ++b)
#pragma unroll
            for (int c = 0; c < 2; ++c) mine[(a * NTW + b) * 2 + c] = make_double2(re[a][b][c], im[a][b][c]);
    __syncthreads();
    if (g == 0) {
        double2 *part = work + (int64_t)blockIdx.x * nl * nr;
#pragma unroll
        for (int a = 0; a < MTW; ++a)
#pragma unroll
            for (int b = 0; b < NTW; ++b)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int k = (a * NTW + b) * 2 + c;
                    double x = 0.0, y = 0.0;
                    for (int gg = 0; gg < rg; ++gg) {
                        const double2 v = gtc_sm[((int64_t)gg * per * 32 + wt * 32 + lane) * V + k];
                        x += v.x;
                        y += v.y;
                    }
                    const int i = 8 * (wi * MTW + a) + r8, j = 8 * (wj * NTW + b) + 2 * q4 + c;
                    if (i < nl && j < nr) part[i + (int64_t)nl * j] = make_double2(x, y);
                }
    }
}

template <class S, int MTW, int NTW, bool KM8 = false, bool TRI = false>
static cudaError_t gram_tc_go(const ColListT<S> &L, const ColListT<S> &R, int64_t len, int herm, double2 *out, int ldo,
                              double2 *work, cudaStream_t st, int64_t tri)
{
    if constexpr (!TRI) {
        if (tri) return gram_tc_go<S, MTW, NTW, KM8, true>(L, R, tri_slots(tri), herm, out, ldo, work, st, tri);
    }
    const int mt = (L.n + 7) / 8, nt = (R.n + 7) / 8;
    const int wm = (mt + MTW - 1) / MTW, wn = (nt + NTW - 1) / NTW;
    const int per = wm * wn;
    if (per > 16) return cudaErrorInvalidValue;
    const int rg = std::max(1, 8 / per);
    const int threads = 32 * per * rg;
    const size_t smem = (size_t)threads * MTW * NTW * 2 * sizeof(double2);
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gram_tc<S, MTW, NTW, KM8, TRI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             512 * MTW * NTW * 2 * (int)sizeof(double2));
        if (e != cudaSuccess) return e;
        attr[dev] = true;
    }
    // about four blocks per SM; the partials (nblk x nl x nr) fit the work
    // buffer that gram_work_elems sizes for them
    const int nblk = gram_blocks(L.n, R.n, len);
    int64_t chunk = (len + nblk - 1) / nblk;
    chunk = (chunk + 3) / 4 * 4;
    work += 1;
    cudaError_t e = pdl_launch(gram_tc<S, MTW, NTW, KM8, TRI>, nblk, threads, smem, st,
                      L, R, len, chunk, (unsigned)tri, herm, wm, wn, rg, work);
    if (e != cudaSuccess) return e;
    const int nout = L.n * R.n;
    return pdl_launch(gram_reduce, (nout + 7) / 8, 256, 0, st, work, nblk, L.n, R.n, out, ldo);
}

template <int NC, bool SELF>
static cudaError_t gram_col_go(const ColList &L, const double2 *b, int64_t len, int herm, double2 *out, double2 *work,
                               cudaStream_t st, int64_t tri)
{
    if (tri) {
        len = tri_slots(tri);
        const int blocks = fused_blocks<gram_col<NC, SELF, true>>((len + 1) / 2, NC);
        return pdl_launch(gram_col<NC, SELF, true>, blocks, 256, 0, st, L, b, len, (unsigned)tri, herm, work, out);
    }
    const int blocks = fused_blocks<gram_col<NC, SELF, false>>((len + 1) / 2, NC);
    return pdl_launch(gram_col<NC, SELF, false>, blocks, 256, 0, st, L, b, len, 0u, herm, work, out);
}

// L unshifted, 2 <= L.n <= 9, one unshifted column in R
template <bool SELF>
static cudaError_t gram_col_any(const ColList &L, const double2 *b, int64_t len, int herm, double2 *out, double2 *work,
                                cudaStream_t st, int64_t tri)
{
    switch (L.n) {
    case 2: return gram_col_go<2, SELF>(L, b, len, herm, out, work, st, tri);
    case 3: return gram_col_go<3, SELF>(L, b, len, herm, out, work, st, tri);
    case 4: return gram_col_go<4, SELF>(L, b, len, herm, out, work, st, tri);
    case 5: return gram_col_go<5, SELF>(L, b, len, herm, out, work, st, tri);
    case 6: return gram_col_go<6, SELF>(L, b, len, herm, out, work, st, tri);
    case 7: return gram_col_go<7, SELF>(L, b, len, herm, out, work, st, tri);
    case 8: return gram_col_go<8, SELF>(L, b, len, herm, out, work, st, tri);
    case 9: return gram_col_go<9, SELF>(L, b, len, herm, out, work, st, tri);
    default: return cudaErrorInvalidValue;
    }
}

template <class S>
static cudaError_t gram_any(const ColListT<S> &L, const ColListT<S> &R, int64_t len, int herm, double2 *out, int ldo,
                            double2 *work, cudaStream_t st, int64_t tri)
{
    if (L.n < 1 || L.n > 64 || R.n < 1 || R.n > 128 || len < 1) return cudaErrorInvalidValue;
    if constexpr (sizeof(S) == 16) {
        bool plain = R.n == 1 && L.n >= 2 && L.n <= 9 && !R.b[0];
        for (int i = 0; i < L.n && plain; ++i) plain = !L.b[i];
        if (plain)
            return L.a[L.n - 1] == R.a[0] ? gram_col_any<true>(L, R.a[0], len, herm, out, work, st, tri)
                                          : gram_col_any<false>(L, R.a[0], len, herm, out, work, st, tri);
    }
    // one ket: a thread holds all sums, up to 8 of them, or up to 32 of a short
    // vector; longer ones go to the tiles (4.8 M rows: 12 x 1 454 us against 215,
    // 24 x 1 1645 against 351).  These read whole vectors.
    if (R.n == 1 && (L.n <= 8 || (L.n <= 32 && len < (1 << 18))) && !tri) {
        if (L.n <= 1) return gram_small_go<1, 1>(L, R, len, herm, out, ldo, work, st);
        if (L.n <= 2) return gram_small_go<2, 1>(L, R, len, herm, out, ldo, work, st);
        if (L.n <= 4) return gram_small_go<4, 1>(L, R, len, herm, out, ldo, work, st);
        if (L.n <= 8) return gram_small_go<8, 1>(L, R, len, herm, out, ldo, work, st);
        if (L.n <= 16) return gram_small_go<16, 1>(L, R, len, herm, out, ldo, work, st);
        return gram_small_go<32, 1>(L, R, len, herm, out, ldo, work, st);
    }
    // a block against itself: half the sums, one read of each column (4 x 4 at
    // 1.8 M rows 24 us against 32 on the tiles)
    if constexpr (sizeof(S) == 16) {
        bool self = herm && L.n == R.n && L.n >= 2 && L.n <= 7;
        for (int i = 0; i < L.n && self; ++i) self = L.a[i] == R.a[i] && !L.b[i] && !R.b[i];
        if (self) return gram_herm_launch(L, len, out, ldo, work, st, tri);
    }
    // up to 4 x 4 of a short vector in one fused launch, all operands straight
    // into registers: 13 us against 15 for the tiles at 118 K rows, 70 against
    // 33 at 1.8 M; 1 x 2 at any length, where the tiles pad one bra to four (44
    // us against 32 at 1.8 M rows), and 2 x 2 up to 2^20 rows (36 against 31 at
    // 531 K)
    if (!tri && L.n <= 2 && R.n <= 2 && (L.n == 1 || len < (1 << 20)))
        return gram_small_go<2, 2>(L, R, len, herm, out, ldo, work, st);
    if (!tri && L.n <= 4 && R.n <= 4 && len < (1 << 18)) return gram_small_go<4, 4>(L, R, len, herm, out, ldo, work, st);
    if (L.n == 8 && R.n == 16 && herm) {  // the projection of one column with a P block
        bool km8 = R.sigma.x == L.sigma.x && R.sigma.y == L.sigma.y;
        for (int c = 0; c < 8 && km8; ++c)
            km8 = L.b[c] && R.a[c] == L.a[c] && R.b[c] == L.b[c] && R.a[8 + c] == L.b[c] && !R.b[8 + c];
        if (km8) return gram_tc_go<S, 1, 2, true>(L, R, len, herm, out, ldo, work, st, tri);
    }
    // the tiles keep one shift; no caller has two
    bool one_shift = true;
    if (R.sigma.x != L.sigma.x || R.sigma.y != L.sigma.y)
        for (int j = 0; j < R.n; ++j) one_shift = one_shift && !R.b[j];
    if (one_shift && gram_tile_supported(L, R)) return gram_tile_launch(L, R, len, herm, out, ldo, work, st, tri);
    // everything else on the FP64 tensor cores, warp tiles sized to the output
    const int mt = (L.n + 7) / 8, nt = (R.n + 7) / 8;
    if (mt == 1) return gram_tc_go<S, 1, 4>(L, R, len, herm, out, ldo, work, st, tri);
    if (nt <= 4) return gram_tc_go<S, 2, 2>(L, R, len, herm, out, ldo, work, st, tri);
    return gram_tc_go<S, 2, 4>(L, R, len, herm, out, ldo, work, st, tri);
}

cudaError_t gram_launch(const ColList &L, const ColList &R, int64_t len, int herm, double2 *out, int ldo,
                        double2 *work, cudaStream_t st, int64_t tri)
{
    return gram_any(L, R, len, herm, out, ldo, work, st, tri);
}

cudaError_t gram_launch(const ColListF &L, const ColListF &R, int64_t len, int herm, double2 *out, int ldo,
                        double2 *work, cudaStream_t st, int64_t tri)
{
    return gram_any(L, R, len, herm, out, ldo, work, st, tri);
}

namespace {
// Hermitian Gram Z^H Z of n <= 7 vectors (28 packed upper-triangle sums).
// Each row is read once per thread pair: the two threads of a pair take
// the first and the second 14 sums of the same rows, so a thread keeps 14
// FP64 complex accumulators; every thread has two rows in flight.  Warp
// shuffles reduce the even and odd lanes separately, then the block, then
// the last block sums the per-block partials in a fixed order.
// packed index k of the pair (i <= j) of NZ columns, row-major over i
template <int NZ>
__host__ __device__ constexpr int herm_i(int k)
{
    int i = 0;
    while (k >= NZ - i) {
        k -= NZ - i;
        ++i;
    }
    return i;
}
template <int NZ>
__host__ __device__ constexpr int herm_j(int k)
{
    int i = 0;
    while (k >= NZ - i) {
        k -= NZ - i;
        ++i;
    }
    return i + k;
}

// conj(z_i) z_j of one row added to the packed sums; K walks the pairs at
// compile time.  Products of two floats are exact in double.
template <int NZ, int K, int HALF>
__device__ __forceinline__ void herm_half(double (&ar)[NZ * (NZ + 1) / 2], double (&ai)[NZ * (NZ + 1) / 2],
                                          const double (&zr)[NZ], const double (&zi)[NZ])
{
    if constexpr (K < NZ * (NZ + 1) / 2) {
        constexpr int i = herm_i<NZ>(K), j = herm_j<NZ>(K);
        if constexpr (HALF == 0) {
            ar[K] = fma(zr[i], zr[j], ar[K]);
            if constexpr (i != j) ai[K] = fma(zr[i], zi[j], ai[K]);
        } else {
            ar[K] = fma(zi[i], zi[j], ar[K]);
            if constexpr (i != j) ai[K] = fma(-zi[i], zr[j], ai[K]);
        }
        herm_half<NZ, K + 1, HALF>(ar, ai, zr, zi);
    }
}

// The two halves of every sum are NZ (NZ + 1) multiply-adds apart, so that none
// waits for the one before it (6 complex64 columns of the upper half at N = 6:
// 45 -> 36 us; prefetched rows at one block per SM gained nothing); a diagonal
// sum has no imaginary part.
template <int NZ>
__device__ __forceinline__ void herm_acc(double (&ar)[NZ * (NZ + 1) / 2], double (&ai)[NZ * (NZ + 1) / 2],
                                         const double (&zr)[NZ], const double (&zi)[NZ])
{
    herm_half<NZ, 0, 0>(ar, ai, zr, zi);
    herm_half<NZ, 0, 1>(ar, ai, zr, zi);
}

// G = Z^H Z (n = NZ complex64 columns, FP64 sums) in one read: each thread
// adds all NZ (NZ + 1) / 2 packed sums of two rows per step; warps, blocks
// and the last block's fixed-order tree reduce them.
template <class S, int NZ, bool TRI>
__global__ void __launch_bounds__(256, 2)
    gram_herm_kernel(const __grid_constant__ ColListT<S> Z, int64_t len, unsigned m, double2 *__restrict__ work,
                     double2 *__restrict__ out, int ldo)
{
    pdl_enter();
    constexpr int NP = NZ * (NZ + 1) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double ar[NP], ai[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) ar[k] = ai[k] = 0.0;
    const S *zc[NZ];
#pragma unroll
    for (int j = 0; j < NZ; ++j) zc[j] = Z.a[j];
    // upper half: the sums are doubled at the end, so a diagonal row enters by half
    auto halve = [](double(&xr)[NZ], double(&xi)[NZ]) {
#pragma unroll
        for (int j = 0; j < NZ; ++j) {
            xr[j] *= 0.70710678118654752440;
            xi[j] *= 0.70710678118654752440;
        }
    };
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r0 < len; r0 += 2 * stride) {
        int64_t ra = r0, r1 = r0 + stride;
        bool has0 = true, has1 = r1 < len;
        double w0 = 1.0, w1 = 1.0;
        if constexpr (TRI) {
            has0 = tri_row((unsigned)r0, m, ra, w0);
            has1 = has1 && tri_row((unsigned)r1, m, r1, w1);
        }
        S z0[NZ], z1[NZ];
#pragma unroll
        for (int j = 0; j < NZ; ++j) {
            z0[j] = has0 ? ld_prev(zc[j] + ra) : S{0, 0};
            z1[j] = has1 ? ld_prev(zc[j] + r1) : S{0, 0};
        }
        double xr[NZ], xi[NZ];
#pragma unroll
        for (int j = 0; j < NZ; ++j) {
            xr[j] = z0[j].x;
            xi[j] = z0[j].y;
        }
        if (TRI && w0 == 1.0) halve(xr, xi);
        herm_acc<NZ>(ar, ai, xr, xi);
#pragma unroll
        for (int j = 0; j < NZ; ++j) {
            xr[j] = z1[j].x;
            xi[j] = z1[j].y;
        }
        if (TRI && w1 == 1.0) halve(xr, xi);
        herm_acc<NZ>(ar, ai, xr, xi);
    }
    __shared__ double2 wsum[8][NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            ar[k] += __shfl_xor_sync(0xffffffffu, ar[k], off);
            ai[k] += __shfl_xor_sync(0xffffffffu, ai[k], off);
        }
        if (lane == 0) wsum[warp][k] = make_double2(ar[k], ai[k]);
    }
    __syncthreads();
    unsigned *ticket = reinterpret_cast<unsigned *>(work);
    double2 *part_out = work + 1;
    const int nw = blockDim.x >> 5;
    if (threadIdx.x < NP) {
        double2 t = make_double2(0.0, 0.0);
        for (int w = 0; w < nw; ++w) {
            t.x += wsum[w][threadIdx.x].x;
            t.y += wsum[w][threadIdx.x].y;
        }
        part_out[(int64_t)blockIdx.x * NP + threadIdx.x] = t;
    }
    if (last_block(ticket, gridDim.x)) {
        __shared__ double2 res[32];
        reduce_partials(part_out, gridDim.x, NP, NP, res);
        for (int o = threadIdx.x; o < NZ * NZ; o += blockDim.x) {
            const int i = o % NZ, j = o / NZ;
            const int a = i < j ? i : j, b = i < j ? j : i;
            const int kk = a * NZ - a * (a - 1) / 2 + (b - a);  // packed index of (a, b)
            double2 v = res[kk];
            if constexpr (TRI) v = make_double2(2.0 * v.x, 2.0 * v.y);
            if (i > j) v.y = -v.y;
            out[i + (int64_t)ldo * j] = v;
        }
        if (threadIdx.x == 0) *ticket = 0u;
    }
}

template <class S, int NZ, bool TRI>
cudaError_t gram_herm_go(const ColListT<S> &Z, int64_t len, double2 *out, int ldo, double2 *work, cudaStream_t st,
                         int64_t tri)
{
    // partials: NZ (NZ + 1) / 2 per block must fit the reduction scratch (kSmallBlocks * 32)
    if constexpr (TRI) len = tri_slots(tri);
    const int64_t want = (len + 511) / 512;
    const int blocks = (int)std::max<int64_t>(
        1, std::min<int64_t>(want, std::min(wave_blocks<gram_herm_kernel<S, NZ, TRI>>(), kSmallBlocks)));
    return pdl_launch(gram_herm_kernel<S, NZ, TRI>, blocks, 256, 0, st, Z, len, (unsigned)tri, work, out, ldo);
}

template <class S, int NZ>
cudaError_t gram_herm_go(const ColListT<S> &Z, int64_t len, double2 *out, int ldo, double2 *work, cudaStream_t st,
                         int64_t tri)
{
    return tri ? gram_herm_go<S, NZ, true>(Z, len, out, ldo, work, st, tri)
               : gram_herm_go<S, NZ, false>(Z, len, out, ldo, work, st, 0);
}
}  // namespace

template <class S>
static cudaError_t gram_herm_any(const ColListT<S> &Z, int64_t len, double2 *out, int ldo, double2 *work,
                                 cudaStream_t st, int64_t tri)
{
    if (len < 1) return cudaErrorInvalidValue;
    switch (Z.n) {
    case 2: return gram_herm_go<S, 2>(Z, len, out, ldo, work, st, tri);
    case 3: return gram_herm_go<S, 3>(Z, len, out, ldo, work, st, tri);
    case 4: return gram_herm_go<S, 4>(Z, len, out, ldo, work, st, tri);
    case 5: return gram_herm_go<S, 5>(Z, len, out, ldo, work, st, tri);
    case 6: return gram_herm_go<S, 6>(Z, len, out, ldo, work, st, tri);
    case 7: return gram_herm_go<S, 7>(Z, len, out, ldo, work, st, tri);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t gram_herm_launch(const ColListF &Z, int64_t len, double2 *out, int ldo, double2 *work, cudaStream_t st,
                             int64_t tri)
{
    return gram_herm_any(Z, len, out, ldo, work, st, tri);
}

cudaError_t gram_herm_launch(const ColList &Z, int64_t len, double2 *out, int ldo, double2 *work, cudaStream_t st,
                             int64_t tri)
{
    return gram_herm_any(Z, len, out, ldo, work, st, tri);
}

template <int NC>
static cudaError_t update_col_go(const UpdList &U, const double2 *c_dev, int64_t len, cudaStream_t st)
{
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((len + 511) / 512, wave_blocks<update_col<NC>>()));
    return pdl_launch(update_col<NC>, blocks, 256, 0, st, U, c_dev, len);
}

template <class SI, class SO>
static cudaError_t update_any(const UpdListT<SI, SO> &U, const double2 *c_dev, int ldc, int64_t len, cudaStream_t st)
{
    if (U.nin < 1 || U.nin > kMaxCols || U.nout < 1 || U.nout > 16 || len < 1)
        return cudaErrorInvalidValue;
    if constexpr (sizeof(SI) == 16 && sizeof(SO) == 16) {
        if (U.nout == 1 && U.nin >= 2 && U.nin <= 9 && U.beta[0].x == 0.0 && U.beta[0].y == 0.0) {
            switch (U.nin) {
            case 2: return update_col_go<2>(U, c_dev, len, st);
            case 3: return update_col_go<3>(U, c_dev, len, st);
            case 4: return update_col_go<4>(U, c_dev, len, st);
            case 5: return update_col_go<5>(U, c_dev, len, st);
            case 6: return update_col_go<6>(U, c_dev, len, st);
            case 7: return update_col_go<7>(U, c_dev, len, st);
            case 8: return update_col_go<8>(U, c_dev, len, st);
            default: return update_col_go<9>(U, c_dev, len, st);
            }
        }
    }
    if (U.nout <= 1) return update_go<1>(U, c_dev, ldc, len, st);
    if (U.nout <= 2) return update_go<2>(U, c_dev, ldc, len, st);
    if (U.nout <= 4) return update_go<4>(U, c_dev, ldc, len, st);
    if (U.nout <= 8) return update_go<8>(U, c_dev, ldc, len, st);
    return update_go<16>(U, c_dev, ldc, len, st);
}

cudaError_t update_launch(const UpdList &U, const double2 *c_dev, int ldc, int64_t len, cudaStream_t st)
{
    return update_any(U, c_dev, ldc, len, st);
}
cudaError_t update_launch(const UpdListT<float2, float2> &U, const double2 *c_dev, int ldc, int64_t len,
                          cudaStream_t st)
{
    return update_any(U, c_dev, ldc, len, st);
}
cudaError_t update_launch(const UpdListT<float2, double2> &U, const double2 *c_dev, int ldc, int64_t len,
                          cudaStream_t st)
{
    return update_any(U, c_dev, ldc, len, st);
}

cudaError_t axpc_launch(double2 *const *out, const double2 *const *a, const double2 *const *b,
                        int n, double2 s, const double2 *c_dev, int64_t len, cudaStream_t st)
{
    if (n < 1 || n > 64) return cudaErrorInvalidValue;
    PtrPack P{};
    for (int j = 0; j < n; ++j) {
        P.out[j] = out[j];
        P.a[j] = a[j];
        P.b[j] = b[j];
    }
    return pdl_launch(axpc_kernel, dim3(stream_blocks(len) / n + 1, n), 256, 0, st, P, s, c_dev, len);
}

cudaError_t axpc_f32_launch(float2 *out, const double2 *a, const double2 *b, double2 s, const double2 *c_dev,
                            int64_t len, cudaStream_t st)
{
    if (len < 1) return cudaErrorInvalidValue;
    return pdl_launch(axpc_f32_kernel, stream_blocks(len) * 2, 256, 0, st, out, a, b, s, c_dev, len);
}

cudaError_t axpy_launch(double2 *out, const double2 *a, const double2 *b, double2 s, int64_t n, cudaStream_t st)
{
    if (n < 1) return cudaErrorInvalidValue;
    return pdl_launch(axpy_kernel<double2>, stream_blocks(n) * 2, 256, 0, st, out, a, b, s, n);
}

cudaError_t axpy_launch(float2 *out, const float2 *a, const float2 *b, double2 s, int64_t n, cudaStream_t st)
{
    if (n < 1) return cudaErrorInvalidValue;
    return pdl_launch(axpy_kernel<float2>, stream_blocks(n) * 2, 256, 0, st, out, a, b, s, n);
}

cudaError_t scale_cols_launch(double2 *const *x, int n, const double2 *c_dev, int64_t len,
                              cudaStream_t st)
{
    if (n < 1 || n > 64) return cudaErrorInvalidValue;
    PtrPack P{};
    for (int j = 0; j < n; ++j) P.out[j] = x[j];
    return pdl_launch(scale_kernel, dim3(stream_blocks(len) / n + 1, n), 256, 0, st, P, c_dev, len);
}

cudaError_t dotdiag_reduce_launch(const double2 *work, int nblk, int n, double2 *out, cudaStream_t st)
{
    if (n < 1 || nblk < 1) return cudaErrorInvalidValue;
    return pdl_launch(dotdiag_reduce, n, 256, 0, st, work, nblk, n, out);
}

int64_t dotdiag_work_elems(int n, int64_t len)
{
    (void)len;
    return 1 + (int64_t)n * 296;
}

cudaError_t dotdiag_launch(const double2 *const *a, const double2 *const *b, int n, int64_t len,
                           int herm, double2 *out, double2 *work, cudaStream_t st, int64_t tri)
{
    if (n < 1 || n > 64) return cudaErrorInvalidValue;
    if (tri) len = tri_slots(tri);
    PtrPack P{};
    for (int j = 0; j < n; ++j) {
        P.a[j] = a[j];
        P.b[j] = b[j];
    }
    work += 1;
    const int nblk = (int)std::max<int64_t>(1, std::min<int64_t>((len + 255) / 256, std::max(1, 296 / n)));
    cudaError_t e = tri ? pdl_launch(dotdiag_partial<true>, dim3(nblk, n), 256, 0, st, P, len, (unsigned)tri, herm, work)
                        : pdl_launch(dotdiag_partial<false>, dim3(nblk, n), 256, 0, st, P, len, 0u, herm, work);
    if (e != cudaSuccess) return e;
    return dotdiag_reduce_launch(work, nblk, n, out, st);
}

template <class S>
static cudaError_t gs_pass1_go(const S *const *qp, const S *const *vp, int m, S *q, S *v, const double2 *d,
                               int64_t len, double2 *work, double2 *dout, cudaStream_t st)
{
    if (m < 1 || m > 16) return cudaErrorInvalidValue;
    GsArgs<S> A{};
    for (int i = 0; i < m; ++i) {
        A.qp[i] = qp[i];
        A.vp[i] = vp[i];
    }
    A.q = q;
    A.v = v;
    A.m = m;
#define GS1(MM) gs_pass1<S, MM><<<fused_blocks<gs_pass1<S, MM>>(len, MM + 1), 256, 0, st>>>(A, d, len, work, dout)
    if (m <= 1) GS1(1);
    else if (m <= 2) GS1(2);
    else if (m <= 4) GS1(4);
    else if (m <= 8) GS1(8);
    else GS1(16);
#undef GS1
    count_launch();
    return cudaGetLastError();
}

cudaError_t gs_pass1_launch(const double2 *const *qp, const double2 *const *vp, int m, double2 *q, double2 *v,
                            const double2 *d, int64_t len, double2 *work, double2 *dout, cudaStream_t st)
{
    return gs_pass1_go(qp, vp, m, q, v, d, len, work, dout, st);
}
cudaError_t gs_pass1_launch(const float2 *const *qp, const float2 *const *vp, int m, float2 *q, float2 *v,
                            const double2 *d, int64_t len, double2 *work, double2 *dout, cudaStream_t st)
{
    return gs_pass1_go(qp, vp, m, q, v, d, len, work, dout, st);
}

template <class S>
static cudaError_t gs_pass2_go(const S *const *qp, const S *const *vp, int m, S *q, S *v, const double2 *d2,
                               int64_t len, double2 *cout, cudaStream_t st)
{
    if (m < 1 || m > 16) return cudaErrorInvalidValue;
    GsArgs<S> A{};
    for (int i = 0; i < m; ++i) {
        A.qp[i] = qp[i];
        A.vp[i] = vp[i];
    }
    A.q = q;
    A.v = v;
    A.m = m;
    const int blocks = stream_blocks(len) * 2;
    if (m <= 1) gs_pass2<S, 1><<<blocks, 256, 0, st>>>(A, d2, len, cout);
    else if (m <= 2) gs_pass2<S, 2><<<blocks, 256, 0, st>>>(A, d2, len, cout);
    else if (m <= 4) gs_pass2<S, 4><<<blocks, 256, 0, st>>>(A, d2, len, cout);
    else if (m <= 8) gs_pass2<S, 8><<<blocks, 256, 0, st>>>(A, d2, len, cout);
    else gs_pass2<S, 16><<<blocks, 256, 0, st>>>(A, d2, len, cout);
    count_launch();
    return cudaGetLastError();
}

cudaError_t gs_pass2_launch(const double2 *const *qp, const double2 *const *vp, int m, double2 *q, double2 *v,
                            const double2 *d2, int64_t len, double2 *cout, cudaStream_t st)
{
    return gs_pass2_go(qp, vp, m, q, v, d2, len, cout, st);
}
cudaError_t gs_pass2_launch(const float2 *const *qp, const float2 *const *vp, int m, float2 *q, float2 *v,
                            const double2 *d2, int64_t len, double2 *cout, cudaStream_t st)
{
    return gs_pass2_go(qp, vp, m, q, v, d2, len, cout, st);
}

// The mixed inner solve's normal equations for one column: from the
// Hermitian Gram G of the power basis z_0..z_nq (nz = nq + 1 <= 8,
// column-major, ld nz), with D = sqrt(diag(G[1:,1:])), solves
// (D^-1 G[1:,1:] D^-1 + 1e-13 I) y = D^-1 G[1:,0] by Cholesky and returns
// a = D^-1 y (nq values).  Flag 8 if the system is not positive definite.
__global__ void __launch_bounds__(64)
    small_sstep_solve(const double2 *G, int nz, double2 *a, int *flag)
{
    pdl_enter();
    __shared__ double2 R[8 * 8], y[8];
    __shared__ double d[8], inv[8];
    const int n = nz - 1, t = threadIdx.x;
    double v = 1.0;
    if (t < n) {
        v = G[(t + 1) + nz * (t + 1)].x;
        d[t] = 1.0 / sqrt(v);
    }
    if (__syncthreads_or(!(v > 0.0) || !isfinite(v))) {
        if (t == 0) raise_flag(flag, 8);
        return;
    }
    if (t < n * n) {
        const int i = t % n, j = t / n;
        const double2 g = G[(i + 1) + nz * (j + 1)];
        const double s = d[i] * d[j];
        R[t] = make_double2(i == j ? g.x * s + 1e-13 : g.x * s, g.y * s);
    }
    if (t < n) {
        const double2 g = G[t + 1];
        y[t] = make_double2(g.x * d[t], g.y * d[t]);
    }
    __syncthreads();
    if (!block_cholesky(R, inv, n)) {
        if (t == 0) raise_flag(flag, 8);
        return;
    }
    for (int i = 0; i < n; ++i) {  // R^H y = D^-1 G[1:, 0]
        const double2 yi = make_double2(y[i].x * inv[i], y[i].y * inv[i]);
        __syncthreads();
        if (t == i) y[i] = yi;
        if (t > i && t < n) {  // y(t) -= conj(R(i,t)) y(i)
            const double2 p = R[i + n * t];
            y[t].x -= p.x * yi.x + p.y * yi.y;
            y[t].y -= p.x * yi.y - p.y * yi.x;
        }
        __syncthreads();
    }
    for (int i = n - 1; i >= 0; --i) {  // R x = y
        const double2 xi = make_double2(y[i].x * inv[i], y[i].y * inv[i]);
        __syncthreads();
        if (t == i) y[i] = xi;
        if (t < i) {  // y(t) -= R(t,i) x(i)
            const double2 p = R[t + n * i];
            y[t].x -= p.x * xi.x - p.y * xi.y;
            y[t].y -= p.x * xi.y + p.y * xi.x;
        }
        __syncthreads();
    }
    if (t < n) a[t] = make_double2(y[t].x * d[t], y[t].y * d[t]);
}

cudaError_t small_sstep_solve_launch(const double2 *g, int nz, double2 *a, int *flag, cudaStream_t st)
{
    if (nz < 2 || nz > 9) return cudaErrorInvalidValue;
    return pdl_launch(small_sstep_solve, 1, 64, 0, st, g, nz, a, flag);
}

cudaError_t orth_norm_coef_launch(const double2 *g, int n, double2 *coef, int *flag, cudaStream_t st)
{
    if (n < 0 || n > 127) return cudaErrorInvalidValue;
    return pdl_launch(orth_norm_coef, 1, 32, 0, st, g, n, coef, flag);
}

cudaError_t small_cholinv_launch(const double2 *g, int k, double2 *rinv, int *flag, cudaStream_t st)
{
    if (k < 1 || k > 16) return cudaErrorInvalidValue;
    return pdl_launch(small_cholinv, 1, 64, 0, st, g, k, rinv, flag);
}

cudaError_t small_orth_chol_launch(const double2 *g, int m, int k, double2 *rinv, double2 *c, int *flag,
                                   cudaStream_t st)
{
    if (m < 1 || k < 1 || k > 16 || m > 64) return cudaErrorInvalidValue;
    return pdl_launch(small_orth_chol, 1, 256, 0, st, g, m, k, rinv, c, flag);
}

cudaError_t small_block_coef_launch(const double2 *g1, const double2 *g2, int ld2, int m, int k, const double2 *r1,
                                    const double2 *r2, double2 *c, cudaStream_t st)
{
    if (m < 0 || k < 1 || k > 16) return cudaErrorInvalidValue;
    return pdl_launch(small_block_coef, 1, 256, 0, st, g1, g2, ld2, m, k, r1, r2, c);
}

cudaError_t small_hsqrt1_launch(const double2 *g, double2 *ginvh, double2 *gsq, int *flag, cudaStream_t st)
{
    small_hsqrt1<<<1, 32, 0, st>>>(g, ginvh, gsq, flag);
    count_launch();
    return cudaGetLastError();
}

cudaError_t small_ortho_check_launch(const double2 *t, int k, int *flag, cudaStream_t st, double tol)
{
    if (k < 1 || k > 16) return cudaErrorInvalidValue;
    return pdl_launch(small_ortho_check, 1, 256, 0, st, t, k, tol, flag);
}

cudaError_t small_gemm_launch(const double2 *a, const double2 *b, double2 *c, int m, int k, int n, cudaStream_t st)
{
    if (m * n < 1) return cudaErrorInvalidValue;
    small_gemm<<<(m * n + 127) / 128, 128, 0, st>>>(a, b, c, m, k, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t inv_sqrt_abs_launch(const double2 *d, double2 *c, int n, cudaStream_t st)
{
    if (n < 1 || n > 64) return cudaErrorInvalidValue;
    return pdl_launch(inv_sqrt_abs_kernel, 1, 64, 0, st, d, c, n);
}

cudaError_t update_exch_launch(const float2 *const *z, int nz, const double2 *coef, double2 *y, int64_t m, double s,
                               cudaStream_t st)
{
    const int64_t t = (m + 31) / 32;
    if (m < 1 || t > 4096 || nz < 1 || nz > kUxMaxIn) return cudaErrorInvalidValue;
    UxArgs A{};
    for (int i = 0; i < nz; ++i) A.z[i] = z[i];
    A.nz = nz;
    const unsigned blocks = (unsigned)(t * (t + 1) / 2);
    switch (nz) {
#define UX_CASE(K) \
    case K: update_exch_kernel<K><<<blocks, 256, 0, st>>>(A, coef, y, m, s, (int)t); break;
        UX_CASE(1) UX_CASE(2) UX_CASE(3) UX_CASE(4) UX_CASE(5) UX_CASE(6) UX_CASE(7) UX_CASE(8)
#undef UX_CASE
    }
    count_launch();
    return cudaGetLastError();
}

cudaError_t exch_parts_launch(const double2 *x, int64_t m, double2 *out, double2 *work, cudaStream_t st)
{
    const int64_t t = (m + 31) / 32;
    if (m < 1 || t > 65535) return cudaErrorInvalidValue;
    exch_kernel<false><<<dim3((unsigned)t, (unsigned)t), 256, 0, st>>>(const_cast<double2 *>(x), m, 0.0, work + 1);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return pdl_launch(dotdiag_reduce, 1, 256, 0, st, work + 1, (int)(t * t), 1, out);
}

cudaError_t exch_project_launch(double2 *x, int64_t m, double s, cudaStream_t st)
{
    const int64_t t = (m + 31) / 32;
    if (m < 1 || t > 65535) return cudaErrorInvalidValue;
    exch_kernel<true><<<dim3((unsigned)t, (unsigned)t), 256, 0, st>>>(x, m, s, nullptr);
    count_launch();
    return cudaGetLastError();
}

cudaError_t refl_corr_launch(const double2 *x, int nn, double2 *out, double2 *work, cudaStream_t st)
{
    if (nn < 3 || !(nn & 1)) return cudaErrorInvalidValue;
    const int64_t d = (int64_t)nn * nn * nn * nn * nn * nn;
    const int blocks = stream_blocks(d);
    // work[0] is the fused reductions' ticket: the partials start at work + 1
    refl_corr_kernel<<<blocks, 256, 0, st>>>(x, nn, d, work + 1);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return pdl_launch(dotdiag_reduce, 8, 256, 0, st, work + 1, blocks, 8, out);
}

cudaError_t refl_project_launch(double2 *x, int nn, unsigned keep, cudaStream_t st)
{
    if (nn < 3 || !(nn & 1) || keep > 255u) return cudaErrorInvalidValue;
    const int64_t k = (int64_t)(nn / 2) * nn + nn / 2 + 1;
    refl_project_kernel<<<stream_blocks(k * k * k), 256, 0, st>>>(x, nn, keep);
    count_launch();
    return cudaGetLastError();
}

cudaError_t to_f32_launch(const double2 *x, float2 *y, int64_t n, cudaStream_t st)
{
    if (n < 1) return cudaErrorInvalidValue;
    return pdl_launch(cvt_c2f_kernel, stream_blocks(n) * 2, 256, 0, st, x, y, n);
}

cudaError_t to_f32_launch(const double *x, float *y, int64_t n, cudaStream_t st)
{
    if (n < 1) return cudaErrorInvalidValue;
    cvt_r2f_kernel<<<stream_blocks(n), 256, 0, st>>>(x, y, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t build_tables_launch(int nn, int n, double charge, double delta, const double *tinv,
                                int nbd, double *t1a, double *v12, cudaStream_t st)
{
    tables_kernel<<<148, 256, 0, st>>>(nn, n, charge, delta, tinv, nbd, t1a, v12);
    count_launch();
    return cudaGetLastError();
}

}  // namespace de

// ---------------------------------------------------------------- no-alloc
// Allocation-free variant of the device dot products, for callers that cannot
// call cudaMalloc: code embedded in a host application that owns all device
// memory through its own pool or a fixed reservation (a serving process that
// reserved its HBM up front), where an allocation from this library would
// fail or push the process past its reservation.  Its reduction scratch
// (ticket plus one partial per block and output of the fused small Gram) is
// a file-scope device array of 1 + 296*32 complex values (151,568 bytes) that
// every GPU loading this library holds until the process exits.

namespace de {

static __device__ __align__(256) double2 g_dots_scratch[1 + kSmallBlocks * 32];

namespace {
// The array's device address per device, valid for the context it was looked
// up in: after cudaDeviceReset (or a released and re-created primary
// context) the module is loaded again and the address changes, so the
// cache is keyed on the driver's context id as well.
struct ScratchAddr {
    unsigned long long ctx_id;
    double2 *ptr;
};
std::mutex g_scratch_mu;
ScratchAddr g_scratch_addr[64] = {};

using CtxGetCurrentFn = CUresult (*)(CUcontext *);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long *);

// Id of the calling thread's current context (0: none current, or the
// driver offers no id).  The driver entry points come through the runtime,
// so the library does not link libcuda.
unsigned long long current_ctx_id()
{
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<CtxGetIdFn>(f);
    });
    if (!get_current || !get_id) return 0;
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
    if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}
}  // namespace

}  // namespace de

extern "C" DE_API int de_dots_noalloc_d(const de_complex *bras_d, const de_complex *kets_d, int64_t size, int nbra,
                                        int nket, de_complex *out_d, int hermitian, void *cuda_stream)
{
    using namespace de;
    if (!bras_d || !kets_d || !out_d) return set_error(DE_E_INVALID, "de_dots_noalloc_d: null pointer");
    if (size < 1 || nbra < 1 || nket < 1) return set_error(DE_E_INVALID, "de_dots_noalloc_d: empty dot");
    const bool shape_ok = (nket == 1 && nbra <= 32) || (nbra <= 4 && nket <= 4) || (nbra <= 8 && nket <= 4) ||
                          (nbra <= 4 && nket <= 8);
    if (!shape_ok)
        return set_error(DE_E_INVALID,
                         "de_dots_noalloc_d: %d x %d outputs exceed the allocation-free maximum "
                         "(nket == 1 with nbra <= 32, or nbra*nket <= 32 with both <= 8 and one <= 4)",
                         nbra, nket);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
    if (dev < 0 || dev >= 64) return set_error(DE_E_INVALID, "de_dots_noalloc_d: device ordinal %d", dev);
    double2 *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        ScratchAddr &a = g_scratch_addr[dev];
        const unsigned long long id = current_ctx_id();
        if (!a.ptr || id == 0 || id != a.ctx_id) {
            // First call on this device (or in a new context of it): host code
            // needs the device address of the array, whose host-side symbol is
            // only a stand-in.  This also creates the context if none is
            // current yet, so the id is read again afterwards.
            double2 *p = nullptr;
            e = cudaGetSymbolAddress((void **)&p, g_dots_scratch);
            if (e != cudaSuccess) {
                a = ScratchAddr{0, nullptr};
                return cuda_error(e, "cudaGetSymbolAddress(dots scratch)");
            }
            a = ScratchAddr{current_ctx_id(), p};
        }
        scratch = a.ptr;
    }
    cudaStream_t st = (cudaStream_t)cuda_stream;
    // the reduction ticket must start at zero whatever the previous call left
    e = cudaMemsetAsync(scratch, 0, sizeof(double2), st);
    if (e != cudaSuccess) return cuda_error(e, "cudaMemsetAsync(dots scratch)");
    ColList L{}, R{};
    L.n = nbra;
    R.n = nket;
    for (int i = 0; i < nbra; ++i) L.a[i] = (const double2 *)bras_d + (int64_t)i * size;
    for (int j = 0; j < nket; ++j) R.a[j] = (const double2 *)kets_d + (int64_t)j * size;
    double2 *out = (double2 *)out_d;
    const int herm = hermitian ? 1 : 0;
    if (nket == 1) {
        if (nbra <= 1) e = gram_small_go<1, 1>(L, R, size, herm, out, nbra, scratch, st);
        else if (nbra <= 2) e = gram_small_go<2, 1>(L, R, size, herm, out, nbra, scratch, st);
        else if (nbra <= 4) e = gram_small_go<4, 1>(L, R, size, herm, out, nbra, scratch, st);
        else if (nbra <= 8) e = gram_small_go<8, 1>(L, R, size, herm, out, nbra, scratch, st);
        else if (nbra <= 16) e = gram_small_go<16, 1>(L, R, size, herm, out, nbra, scratch, st);
        else e = gram_small_go<32, 1>(L, R, size, herm, out, nbra, scratch, st);
    } else if (nbra <= 4 && nket <= 4) {
        e = gram_small_go<4, 4>(L, R, size, herm, out, nbra, scratch, st);
    } else if (nket <= 4) {
        e = gram_small_go<8, 4>(L, R, size, herm, out, nbra, scratch, st);
    } else {
        e = gram_small_go<4, 8>(L, R, size, herm, out, nbra, scratch, st);
    }
    if (e != cudaSuccess) return cuda_error(e, "de_dots_noalloc_d launch");
    return DE_OK;
}


// gram_tile.cu -- Gram matrices of a few columns against a few columns,
// G(i,j) = sum_r op(L_i[r]) R_j[r] (crossmult lamod.f90:51-125, the K/M
// projection ZGEMMs gplmr.F90:207-267), up to 36 4 x 4 output tiles.
//
// Bound by HBM: 16 bytes per row and distinct column (8 in complex64) against
// 8 nl nr FP64 flops.  The earlier kernels read every column straight into
// registers, once per output tile and with a few loads in flight.  Here a CTA
// streams row tiles of the distinct columns through a cp.async ring (a column
// that occurs in L and in R, or as the partner of a shift, is read once), and
// each warp forms one 4 x 4 tile of outputs, a lane per row: 8 shared-memory
// reads for 64 FP64 multiply-adds, so shared memory and the FP64 pipe take
// about the same time, both below the HBM time up to 8 x 16 outputs.
//
// us on B200, complex128, before -> now (HBM time of the distinct columns in
// brackets):
//   4.8 M rows   8 x 16    837 -> 384 [283]      5 x 3   547 -> 117 [94]
//                16 x 16  1440 -> 769 [378]      24 x 8 1443 -> 606 [378]
//                7 x 14 shifted projection       460 -> 433 [165]
//   1.8 M rows   8 x 4     308 ->  73 [52]      20 x 4   494 -> 123 [104]
//                4 x 4 of itself  70 ->  33 [17]
//   118 K rows   8 x 16     46 ->  23           20 x 4    52 ->  21
// complex64 (1.8 M rows): 10 x 12 502 -> 196, 20 x 24 1259 -> 737.  The shifted
// 8 x 16 projection stays on gram_tc's one-load form (294 us against 446).
#include "de_kernels.h"
#include "pdl.h"
#include "tile_slots.h"
#include "tri.h"

#include <algorithm>
#include <atomic>

namespace de {
namespace {

constexpr int kFusedOut = 32;  // up to as many outputs the last CTA adds the partials

template <class S>
struct GramTileArgs {
    const S *col[kMaxSlots];  // as TileSlots
    unsigned char shifted[kMaxSlots], partner[kMaxSlots];
    unsigned char lslot[kTile * kTileWarps], rslot[kTile * kTileWarps];
    double2 sigma;
    int64_t len;
    unsigned m;  // TRI: rows are the slots of an M x M upper half
    int nslots, nshift, nl, nr, tl, tr, stages;
    double sign;  // -1: conj(L)
    double2 *work, *out;  // work[0]: the fused reductions' ticket, zero between launches
    int ldo;
};

template <class S>
__device__ __forceinline__ void copy_async(S *s, const S *g, bool in)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
    const int n = in ? (int)sizeof(S) : 0;  // rows past the end read as zero
    if constexpr (sizeof(S) == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(g), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(g), "r"(n) : "memory");
}

// Output o: its nblk partials added by one warp in a fixed order.
__device__ __forceinline__ void sum_partials(const double2 *work, int nblk, int nl, int nout, int o, int lane,
                                             double2 *out, int ldo)
{
    double x = 0.0, y = 0.0;
    for (int b = lane; b < nblk; b += 32 * 10) {  // all of 296 CTAs' partials in flight
        double2 v[10];
#pragma unroll
        for (int u = 0; u < 10; ++u)
            v[u] = b + 32 * u < nblk ? ld_l2(work + (int64_t)(b + 32 * u) * nout + o) : make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < 10; ++u) {
            x += v[u].x;
            y += v[u].y;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        x += __shfl_down_sync(0xffffffffu, x, off);
        y += __shfl_down_sync(0xffffffffu, y, off);
    }
    if (lane == 0) out[o % nl + (int64_t)ldo * (o / nl)] = make_double2(x, y);
}

// RT rows a stage.  Warp w: tile
// w % (tl tr), row group w / (tl tr).
template <class S, int RT, bool TRI>
__global__ void __launch_bounds__(32 * kTileWarps) gram_tile_kernel(const __grid_constant__ GramTileArgs<S> a)
{
    pdl_enter();
    extern __shared__ __align__(16) unsigned char gt_smem[];
    S *ring = reinterpret_cast<S *>(gt_smem);  // [stage][slot][RT]
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nt = blockDim.x;
    const int tiles = a.tl * a.tr, tile = warp % tiles, group = warp / tiles, groups = (nt >> 5) / tiles;
    const int i0 = tile % a.tl * kTile, j0 = tile / a.tl * kTile;
    int ls[kTile], rs[kTile];
#pragma unroll
    for (int i = 0; i < kTile; ++i) {
        ls[i] = a.lslot[i0 + i] * RT;
        rs[i] = a.rslot[j0 + i] * RT;
    }
    const int64_t ntiles = (a.len + RT - 1) / RT;
    const int elems = a.nslots * RT, stride = elems;
    auto issue = [&](int64_t tl, int st) {
        if (tl < ntiles) {
            const int64_t r0 = tl * RT;
            for (int e = t; e < elems; e += nt) {
                const int s = e / RT, r = e % RT;
                bool in = r0 + r < a.len;
                int64_t row = r0 + r;
                if constexpr (TRI) {
                    double w;
                    in = in && tri_row((unsigned)row, a.m, row, w);
                }
                copy_async<S>(ring + st * stride + e, a.col[s] + (in ? row : 0), in);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    double gr[kTile][kTile], gi[kTile][kTile];
#pragma unroll
    for (int i = 0; i < kTile; ++i)
#pragma unroll
        for (int j = 0; j < kTile; ++j) gr[i][j] = gi[i][j] = 0.0;
    const int ns = a.stages;
    for (int k = 0; k + 1 < ns; ++k) issue(blockIdx.x + (int64_t)k * gridDim.x, k);
    int st = 0;
    for (int64_t tl = blockIdx.x; tl < ntiles; tl += gridDim.x, st = st + 1 == ns ? 0 : st + 1) {
        if (ns == 4) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        else if (ns == 3) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        S *xs = ring + st * stride;
        // the slot freed by the previous step takes the copies ns - 1 ahead
        issue(tl + (int64_t)(ns - 1) * gridDim.x, st == 0 ? ns - 1 : st - 1);
        if (a.nshift) {  // a <- a - sigma b; partners are never shifted themselves
            for (int e = t; e < a.nshift * RT; e += nt) {
                const int k = e / RT, r = e % RT;
                S *xa = xs + a.shifted[k] * RT + r;
                const S av = *xa, bv = xs[a.partner[k] * RT + r];
                S v;
                v.x = av.x - (a.sigma.x * bv.x - a.sigma.y * bv.y);
                v.y = av.y - (a.sigma.x * bv.y + a.sigma.y * bv.x);
                *xa = v;
            }
            __syncthreads();
        }
        for (int r = group * 32 + lane; r < RT; r += groups * 32) {
            double2 l[kTile], x[kTile];
#pragma unroll
            for (int i = 0; i < kTile; ++i) {
                const S lv = xs[ls[i] + r], xv = xs[rs[i] + r];
                l[i] = make_double2(lv.x, a.sign * lv.y);
                x[i] = make_double2(xv.x, xv.y);
            }
            if constexpr (TRI) {
                int64_t row;
                double w;
                tri_row((unsigned)(tl * RT + r), a.m, row, w);
#pragma unroll
                for (int i = 0; i < kTile; ++i) {
                    x[i].x *= w;
                    x[i].y *= w;
                }
            }
            // the second terms 32 multiply-adds after the first: none waits for the one before it
#pragma unroll
            for (int i = 0; i < kTile; ++i)
#pragma unroll
                for (int j = 0; j < kTile; ++j) {
                    gr[i][j] = fma(l[i].x, x[j].x, gr[i][j]);
                    gi[i][j] = fma(l[i].x, x[j].y, gi[i][j]);
                }
#pragma unroll
            for (int i = 0; i < kTile; ++i)
#pragma unroll
                for (int j = 0; j < kTile; ++j) {
                    gr[i][j] = fma(-l[i].y, x[j].y, gr[i][j]);
                    gi[i][j] = fma(l[i].y, x[j].x, gi[i][j]);
                }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    // lanes, then row groups, then one partial per CTA; the last CTA or
    // gram_reduce adds the partials in a fixed order
    double2 *acc = reinterpret_cast<double2 *>(gt_smem);  // [warp][16]
#pragma unroll
    for (int i = 0; i < kTile; ++i)
#pragma unroll
        for (int j = 0; j < kTile; ++j) {
            double x = gr[i][j], y = gi[i][j];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                x += __shfl_down_sync(0xffffffffu, x, off);
                y += __shfl_down_sync(0xffffffffu, y, off);
            }
            if (lane == 0) acc[warp * 16 + i * kTile + j] = make_double2(x, y);
        }
    __syncthreads();
    const int nout = a.nl * a.nr;
    double2 *part = a.work + 1 + (int64_t)blockIdx.x * nout;
    for (int o = t; o < nout; o += nt) {
        const int i = o % a.nl, j = o / a.nl;
        const int w = i / kTile + a.tl * (j / kTile), k = (i % kTile) * kTile + j % kTile;
        double x = 0.0, y = 0.0;
        for (int g = 0; g < groups; ++g) {
            x += acc[(g * tiles + w) * 16 + k].x;
            y += acc[(g * tiles + w) * 16 + k].y;
        }
        part[o] = make_double2(x, y);
    }
    if (nout > kFusedOut) return;  // gram_tile_reduce follows
    __shared__ bool last;
    unsigned *ticket = reinterpret_cast<unsigned *>(a.work);
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int o = warp; o < nout; o += nt >> 5) sum_partials(a.work + 1, gridDim.x, a.nl, nout, o, lane, a.out, a.ldo);
    if (t == 0) *ticket = 0u;
}

// Sum of the nblk partials, a warp per output.
__global__ void __launch_bounds__(256)
    gram_tile_reduce(const double2 *work, int nblk, int nl, int nr, double2 *out, int ldo)
{
    pdl_enter();
    const int o = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (o < nl * nr) sum_partials(work, nblk, nl, nl * nr, o, threadIdx.x & 31, out, ldo);
}

template <class S, int RT, bool TRI>
cudaError_t tile_launch(const GramTileArgs<S> &a, int threads, size_t smem, cudaStream_t st)
{
    static std::atomic<int> sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    int n = sms[dev].load(std::memory_order_relaxed);
    if (!n) {
        cudaError_t e = cudaFuncSetAttribute(gram_tile_kernel<S, RT, TRI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kTileSmem);
        if (e != cudaSuccess) return e;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
        sms[dev].store(n, std::memory_order_relaxed);
    }
    // two CTAs per SM: 112 KB of shared memory and 128 registers a thread
    const int nblk = (int)std::max<int64_t>(1, std::min<int64_t>((a.len + RT - 1) / RT, std::min(2 * n, 296)));
    cudaError_t e = pdl_launch(gram_tile_kernel<S, RT, TRI>, nblk, threads, smem, st, a);
    if (e != cudaSuccess || a.nl * a.nr <= kFusedOut) return e;
    return pdl_launch(gram_tile_reduce, (a.nl * a.nr + 7) / 8, 256, 0, st, a.work + 1, nblk, a.nl, a.nr, a.out, a.ldo);
}

// One launch: L columns [l0, l0 + nl) against R columns [r0, r0 + nr), at
// most kTileWarps tiles.
template <class S>
cudaError_t tile_go(const ColListT<S> &L, const ColListT<S> &R, int l0, int nl, int r0, int nr, int64_t len, int herm,
                    double2 *out, int ldo, double2 *work, cudaStream_t st, int64_t tri)
{
    GramTileArgs<S> a{};
    a.sigma = L.sigma;
    TileSlots<S> t{};
    if (!tile_slots(t, L.a + l0, L.b + l0, nl, R.a + r0, R.b + r0, nr)) return cudaErrorInvalidValue;
    std::copy_n(t.col, t.n, a.col);
    std::copy_n(t.shifted, t.nshift, a.shifted);
    std::copy_n(t.partner, t.nshift, a.partner);
    std::copy_n(t.l, sizeof t.l, a.lslot);
    std::copy_n(t.r, sizeof t.r, a.rslot);
    a.nslots = t.n;
    a.nshift = t.nshift;
    a.tl = (nl + kTile - 1) / kTile;
    a.tr = (nr + kTile - 1) / kTile;
    a.len = tri ? tri_slots(tri) : len;
    a.m = (unsigned)tri;
    a.nl = nl;
    a.nr = nr;
    a.sign = herm ? -1.0 : 1.0;
    a.work = work;
    a.out = out + l0 + (int64_t)ldo * r0;
    a.ldo = ldo;
    const int tiles = a.tl * a.tr, threads = 32 * tiles * tile_groups(tiles), rt = tile_rows(tiles);
    const size_t stage = (size_t)a.nslots * rt * sizeof(S);
    a.stages = (int)std::max<size_t>(2, std::min<size_t>(4, (kTileSmem - 1024) / stage));
    const size_t smem = std::max<size_t>(stage * a.stages, kTileWarps * 16 * sizeof(double2));
    if (tri) {
        if (rt == 256) return tile_launch<S, 256, true>(a, threads, smem, st);
        if (rt == 128) return tile_launch<S, 128, true>(a, threads, smem, st);
        return tile_launch<S, 64, true>(a, threads, smem, st);
    }
    if (rt == 256) return tile_launch<S, 256, false>(a, threads, smem, st);
    if (rt == 128) return tile_launch<S, 128, false>(a, threads, smem, st);
    return tile_launch<S, 64, false>(a, threads, smem, st);
}

template <class S>
cudaError_t tiles_go(const ColListT<S> &L, const ColListT<S> &R, int64_t len, int herm, double2 *out, int ldo,
                     double2 *work, cudaStream_t st, int64_t tri)
{
    int bl, br;
    tile_block(L.n, R.n, bl, br);
    for (int i = 0; i < L.n; i += bl)
        for (int j = 0; j < R.n; j += br) {
            cudaError_t e = tile_go(L, R, i, std::min(bl, L.n - i), j, std::min(br, R.n - j), len, herm, out, ldo, work,
                                    st, tri);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

}  // namespace

// Up to 24 x 24 (4.8 M rows: 2150 us against 3940 on the FP64 tensor cores); more
// tiles re-read the columns of the other side too often, and shifted columns
// with too many distinct partners do not fit: those go to gram_tc.
bool gram_tile_supported(const ColList &L, const ColList &R) { return tiles_fit(L.a, L.b, L.n, R.a, R.b, R.n); }
bool gram_tile_supported(const ColListF &L, const ColListF &R) { return tiles_fit(L.a, L.b, L.n, R.a, R.b, R.n); }

cudaError_t gram_tile_launch(const ColList &L, const ColList &R, int64_t len, int herm, double2 *out, int ldo,
                             double2 *work, cudaStream_t st, int64_t tri)
{
    return tiles_go(L, R, len, herm, out, ldo, work, st, tri);
}

cudaError_t gram_tile_launch(const ColListF &L, const ColListF &R, int64_t len, int herm, double2 *out, int ldo,
                             double2 *work, cudaStream_t st, int64_t tri)
{
    return tiles_go(L, R, len, herm, out, ldo, work, st, tri);
}

}  // namespace de

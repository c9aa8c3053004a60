// hammult_line.cu -- the two-electron matvec on even/odd-split lines held in
// registers; the default kernels of every grid, NN = 3..23, both storages.
//
// Reference: HAMMULT hammod.F90:19-67 -> KEMULT2 :138-187 -> KEMULTS
// :264-286, plus Y = Y + V*X (:58-59) with V from POTENTIAL2 :502-582.
//
// X(p, q), p = i1 + NN j1 + NN^2 k1 fastest, q = i2 + NN j2 + NN^2 k2.  The
// six axes are done by three kernels, two of them pass A (electron 2, V) and
// one pass B (electron 1):
//
//   plane_kernel  Y  = S2 (T_i2 + T_j2) X      tile: a run of PW adjacent p
//                                              times one (i2, j2) plane
//   kline_kernel  Y += S2 T_k2 X + V X         one k2 line per thread
//   cube_kernel   Y += S2 (T_i1 + T_j1 + T_k1) X   one contiguous column
//
// What bounds them and why this split:
//
// * A thread keeps a whole line in registers and makes all its outputs: one
//   load per point and axis.  T is symmetric Toeplitz, so it commutes with
//   the reflection of the line: with u_b = v(N+b) + v(N-b), w_b = v(N+b) -
//   v(N-b), out(N +- a) = sum_b ce(a,b) u_b +- sum_b co(a,b) w_b, (N+1)^2 +
//   N^2 multiply-adds instead of NN^2.  delta^2 T depends on NN alone, so
//   ce and co are literals and 1/delta^2 goes into the final factor; read
//   from the kernel's parameters, the 85 coefficients of NN = 13 were kept
//   in registers across the axes and spilled (complex128 cube at NN = 13:
//   62 us from parameters, 47 us as literals).
// * complex64 arithmetic is packed (fma.rn.f32x2 on (re, im) pairs): half
//   the issue slots of scalar FMAs for the same arithmetic.
// * No kernel gathers with a large stride.  The cubes X(p, :) of electron 2
//   do not fit shared memory for more than 2-4 adjacent p, and reading them
//   in 16-32 byte pieces is bound by L2 requests: at NN = 13 complex64 a
//   one-kernel pass A took 58, 52, 33 us with 1, 2, 4 adjacent p, against
//   13 + 11 us for the two kernels here, which read and write whole 128-byte
//   runs.  The price is 8 vector passes instead of 5.
// * The kernel that only writes runs first; the accumulating ones cost more
//   (their old values are on the critical path).  complex64 adds into Y with
//   red.global.add.v2.f32, one per element and kernel, so the order of the
//   sums is fixed and no load of Y is waited for (a product at NN = 17: 260 us
//   against 314 with Y prefetched as below).  That add flushes subnormals, so
//   tiny values take a load, an add and a store (add_to).  complex128 would
//   need two scalar adds per element and measured no faster; it prefetches Y
//   two outputs ahead instead.
//
// Measured on B200, us per vector, one vector per call, before (the even/odd
// slab, streaming or cube kernels, whichever the grid had) and now; in
// parentheses the two passes by events between them (plane + kline, cube), in
// brackets the HBM time of 8 vector passes at 6.54 TB/s where the vectors
// exceed L2:
//
//   NN        complex128                       complex64
//    7    16.8 ->    8.0                    14.2 ->    7.9
//   11    64.8 ->   34.1 (  25 +   18)      33.7 ->   18.5 (  16 +   12)
//   13   169   ->  121   (  80 +   49) [94]  80.3 ->   42.9 (  29 +   22)
//   15   450   ->  315   ( 189 +  134) [223]  239 ->  119   (  82 +   47) [111]
//   17  1130   ->  683   ( 405 +  287) [472]  640 ->  257   ( 170 +   96) [236]
//   19  2100   -> 1640   ( 828 +  635) [921] 1430 ->  648   ( 338 +  230) [460]
//   21  6250   -> 2985   (1608 + 1266) [1680] 3460 -> 1070  ( 617 +  449) [839]
//   23 23700   -> 7950   (3046 + 4061) [2900] 15400 -> 1975 (1084 +  851) [1450]
//
// From NN = 19 on the passes' sum is below the product: back to back under
// programmatic launch the kernels cost more than by themselves (NN = 19 without
// it: 1446 and 570).
//
// complex64 is at 71-93 % of the HBM time from NN = 15 on.  complex128 is held
// back by the cube kernel: one CTA of NN^2 threads per SM from NN = 17 on (two
// cubes of shared memory), whose load, FP64 and store phases do not overlap.
// Staging part of the cube to fit two CTAs measured slower (340-460 us at NN
// = 17), as did L2 prefetches of the next column (the phases wait on the SM,
// not on DRAM) and running the two electron-2 kernels in p chunks that fit L2.
#include "de_kernels.h"
#include "pdl.h"

#include <algorithm>
#include <atomic>
#include <type_traits>

namespace de {
namespace {

// delta^2 T(a, b) for d = |a - b| (KEMATRIX hammod.F90:235-260) and its
// even / odd halves
constexpr double kPi = 3.14159265358979323846;
constexpr double tcoef(int d) { return d == 0 ? kPi * kPi / 6.0 : ((d % 2 == 0) ? 1.0 : -1.0) / ((double)d * d); }
constexpr double ecoef(int a, int b) { return b == 0 ? tcoef(a) : 0.5 * (tcoef(a > b ? a - b : b - a) + tcoef(a + b)); }
constexpr double ocoef(int a, int b) { return 0.5 * (tcoef(a > b ? a - b : b - a) - tcoef(a + b)); }

// Complex arithmetic with real coefficients: double2, or (re, im) packed in
// 64 bits for the f32x2 instructions.
template <class R>
struct Cx;
template <>
struct Cx<float> {
    using C = unsigned long long;
    static __device__ __forceinline__ C add(C a, C b)
    {
        C d;
        asm("add.rn.f32x2 %0,%1,%2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ C sub(C a, C b)
    {
        C d;
        asm("sub.rn.f32x2 %0,%1,%2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ C dup(float c)
    {
        C d;
        asm("mov.b64 %0,{%1,%1};" : "=l"(d) : "f"(c));
        return d;
    }
    static __device__ __forceinline__ C mul(float c, C v)
    {
        C d;
        asm("mul.rn.f32x2 %0,%1,%2;" : "=l"(d) : "l"(dup(c)), "l"(v));
        return d;
    }
    static __device__ __forceinline__ C fma(float c, C v, C acc)
    {
        C d;
        asm("fma.rn.f32x2 %0,%1,%2,%3;" : "=l"(d) : "l"(dup(c)), "l"(v), "l"(acc));
        return d;
    }
    static __device__ __forceinline__ C make(float a, float b)
    {
        C d;
        asm("mov.b64 %0,{%1,%2};" : "=l"(d) : "f"(a), "f"(b));
        return d;
    }
    static __device__ __forceinline__ void split(C a, float &re, float &im)
    {
        asm("mov.b64 {%0,%1},%2;" : "=f"(re), "=f"(im) : "l"(a));
    }
};
template <>
struct Cx<double> {
    using C = double2;
    static __device__ __forceinline__ C add(C a, C b) { return make_double2(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ C sub(C a, C b) { return make_double2(a.x - b.x, a.y - b.y); }
    static __device__ __forceinline__ C mul(double c, C v) { return make_double2(c * v.x, c * v.y); }
    static __device__ __forceinline__ C fma(double c, C v, C acc)
    {
        return make_double2(::fma(c, v.x, acc.x), ::fma(c, v.y, acc.y));
    }
    static __device__ __forceinline__ C make(double a, double b) { return make_double2(a, b); }
    static __device__ __forceinline__ void split(C a, double &re, double &im)
    {
        re = a.x;
        im = a.y;
    }
};
template <class R>
using CC = typename Cx<R>::C;
template <class R>
using G2 = std::conditional_t<sizeof(R) == 8, double2, float2>;

template <int I, int E, class F>
__device__ __forceinline__ void static_for(F f)
{
    if constexpr (I < E) {
        f(std::integral_constant<int, I>());
        static_for<I + 1, E>(f);
    }
}

struct Nothing {};

// One line: v holds its NN values and is overwritten; emit(pos, value,
// loaded) receives delta^2 T v at every point.  loaded = fetch(pos) is what
// the caller adds there, fetched LA outputs ahead.  ORDER keeps the memory
// operations in that order: without it the compiler gathers all of a line's
// loads in front of the sums, and complex128 lines do not leave it the
// registers.
template <class R, int NN, int LA, bool ORDER, class Q, class F, class P = Nothing>
__device__ __forceinline__ void line_transform(CC<R> (&v)[NN], Q fetch, F emit, P emit_pair = P())
{
    using X = Cx<R>;
    constexpr int N = NN / 2;
    using L = decltype(fetch(0));
    L lp[N + 1], lm[N + 1];
#pragma unroll
    for (int a = 0; a < (LA < N + 1 ? LA : N + 1); ++a) {
        lp[a] = fetch(N + a);
        if (a > 0) lm[a] = fetch(N - a);
    }
#pragma unroll
    for (int b = 1; b <= N; ++b) {
        const CC<R> p = v[N + b], m = v[N - b];
        v[N + b] = X::add(p, m);
        v[N - b] = X::sub(p, m);
    }
    static_for<0, N + 1>([&](auto ac) {
        constexpr int a = decltype(ac)::value;
        if constexpr (ORDER) asm volatile("" ::: "memory");
        if constexpr (a + LA <= N) {
            lp[a + LA] = fetch(N + a + LA);
            if constexpr (a + LA > 0) lm[a + LA] = fetch(N - a - LA);
        }
        constexpr R c0 = (R)ecoef(a, 0);
        CC<R> e = X::mul(c0, v[N]);
        static_for<1, N + 1>([&](auto bc) {
            constexpr int b = decltype(bc)::value;
            constexpr R c = (R)ecoef(a, b);
            e = X::fma(c, v[N + b], e);
        });
        if constexpr (a == 0) {
            emit(N, e, lp[0]);
        } else {
            constexpr R d1 = (R)ocoef(a, 1);
            CC<R> o = X::mul(d1, v[N - 1]);
            static_for<2, N + 1>([&](auto bc) {
                constexpr int b = decltype(bc)::value;
                constexpr R d = (R)ocoef(a, b);
                o = X::fma(d, v[N - b], o);
            });
            if constexpr (std::is_same_v<P, Nothing>) {
                emit(N + a, X::add(e, o), lp[a]);
                emit(N - a, X::sub(e, o), lm[a]);
            } else {
                emit_pair(N + a, X::add(e, o), lp[a], N - a, X::sub(e, o), lm[a]);
            }
        }
    });
}

template <class R>
struct LineArgs {
    const CC<R> *x;
    CC<R> *y;
    const R *t1a, *v12;
    int64_t vstride;
    int nvec;
    R s2r, s2i;  // 1 / (SCALE delta)^2
    R vsr, vsi;  // 1 / SCALE
    R shr, shi;  // diagonal shift
};

template <class R>
__device__ __forceinline__ void times_s2(const LineArgs<R> &a, CC<R> z, R &yr, R &yi)
{
    R zr, zi;
    Cx<R>::split(z, zr, zi);
    yr = a.s2r * zr - a.s2i * zi;
    yi = a.s2r * zi + a.s2i * zr;
}

// y += v of complex64 values, one add per element and kernel, without waiting
// for y.  The add in L2 flushes subnormals, and a vector of values below 1e-36
// lost 0.1 % of its norm, one below 1e-40 all of it; a value with a part below
// 2^-100 is therefore added here.  At or above that nothing is lost: y's
// subnormal part is below half an ulp of the sum, and a sum that cancels is
// zero or at least 2^-123.  One test serves the two outputs of a step: us per
// product without a test, with one per output, with one per pair: NN = 13
// 47.3, 44.1, 43.6; NN = 17 256, 264, 260; NN = 19 665, 643, 632.
__device__ __forceinline__ bool l2_add(float2 v, float2 w)
{
    return fminf(fminf(fabsf(v.x), fabsf(v.y)), fminf(fabsf(w.x), fabsf(w.y))) >= 0x1p-100f;
}
__device__ __forceinline__ void add_l2(unsigned long long *y, float2 v)
{
    asm volatile("red.global.add.v2.f32 [%0], {%1,%2};" ::"l"(y), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void add_here(unsigned long long *y, float2 v)
{
    *y = Cx<float>::add(*y, Cx<float>::make(v.x, v.y));
}
__device__ __forceinline__ void add_to(unsigned long long *y, float2 v)
{
    if (l2_add(v, v)) add_l2(y, v);
    else add_here(y, v);
}
__device__ __forceinline__ void add_to(unsigned long long *y, float2 v, unsigned long long *z, float2 w)
{
    if (l2_add(v, w)) {
        add_l2(y, v);
        add_l2(z, w);
    } else {
        add_here(y, v);
        add_here(z, w);
    }
}

// Programmatic dependent launch (a no-op when the launch carries no
// programmatic attribute).  Nothing is read before the wait, and every CTA
// waits, so a grid never completes before its predecessor.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;"); }

// Launch shapes, from sweeps over each grid on B200 (registers decide: a
// line takes 4 NN of them in complex128, 2 NN in complex64, and shapes with
// more resident CTAs than that allows spill or serialise the loads).
//   PW, PB  plane: run of adjacent p (128 bytes where it fits), min CTAs/SM
//   KT, KB  kline: threads, min CTAs/SM; KS stash the line in shared memory
//           for the V x term instead of reading it again
//   CT, CB  cube: threads, min CTAs/SM; CG slabs of x staged at a time (NN =
//           the whole cube; less where two cubes exceed shared memory)
template <class R, int NN>
struct Shape;
#define LINE_SHAPE(RT, NNV, PWV, PBV, KTV, KBV, KSV, CTV, CBV, CGV)                          \
    template <>                                                                              \
    struct Shape<RT, NNV> {                                                                  \
        static constexpr int PW = PWV, PB = PBV, KT = KTV, KB = KBV, KS = KSV;               \
        static constexpr int CT = CTV, CB = CBV, CG = CGV;                                   \
    };
LINE_SHAPE(double, 3, 32, 8, 128, 5, 1, 32, 31, 3)
LINE_SHAPE(double, 5, 16, 8, 128, 5, 1, 32, 28, 5)
LINE_SHAPE(double, 7, 16, 5, 128, 3, 1, 64, 6, 7)
LINE_SHAPE(double, 9, 16, 2, 128, 4, 1, 96, 3, 9)
LINE_SHAPE(double, 11, 8, 6, 128, 3, 1, 128, 3, 11)
LINE_SHAPE(double, 13, 16, 2, 128, 3, 1, 192, 2, 13)
LINE_SHAPE(double, 15, 8, 3, 128, 3, 1, 128, 2, 8)
LINE_SHAPE(double, 17, 8, 2, 128, 3, 1, 320, 1, 17)
LINE_SHAPE(double, 19, 8, 2, 128, 3, 1, 384, 1, 19)
LINE_SHAPE(double, 21, 4, 2, 128, 3, 1, 224, 1, 7)
LINE_SHAPE(double, 23, 4, 2, 256, 1, 0, 96, 1, 3)
LINE_SHAPE(float, 3, 64, 8, 128, 10, 1, 32, 31, 3)
LINE_SHAPE(float, 5, 64, 4, 128, 9, 1, 32, 31, 5)
LINE_SHAPE(float, 7, 32, 4, 128, 8, 1, 64, 20, 7)
LINE_SHAPE(float, 9, 32, 2, 128, 6, 1, 96, 13, 9)
LINE_SHAPE(float, 11, 16, 5, 128, 6, 1, 128, 7, 11)
LINE_SHAPE(float, 13, 16, 3, 128, 6, 1, 192, 6, 13)
LINE_SHAPE(float, 15, 16, 3, 128, 4, 1, 256, 3, 15)
LINE_SHAPE(float, 17, 16, 2, 256, 2, 1, 320, 2, 17)
LINE_SHAPE(float, 19, 16, 2, 256, 3, 1, 192, 2, 19)
LINE_SHAPE(float, 21, 8, 2, 128, 3, 1, 448, 1, 21)
LINE_SHAPE(float, 23, 8, 2, 128, 3, 1, 544, 1, 23)
#undef LINE_SHAPE

template <class R, int NN>
struct Cfg : Shape<R, NN> {
    using S = Shape<R, NN>;
    static constexpr int P2 = NN * NN, M = NN * NN * NN;
    static constexpr int PT = (S::PW * NN + 31) / 32 * 32;  // plane threads
    static constexpr int RUNS = (M + S::PW - 1) / S::PW;
    // kline: all of a line's potential values loaded before the sums, where
    // loads wait for their turn among the ordered memory operations.  complex64
    // has the registers for them (us per product without, with, at NN = 11 19.0,
    // 18.5; 17 262, 257; 21 1084, 1066; equal up to 9); complex128 has not
    // (without, with: NN = 17 682, 693; equal elsewhere, but 21 3014, 2980).
    static constexpr bool KV = sizeof(R) == 4;
    static constexpr size_t PSMEM = (size_t)2 * S::PW * P2 * sizeof(CC<R>);
    static constexpr size_t KSMEM = S::KS ? (size_t)S::KT * NN * sizeof(CC<R>) : 0;
    static constexpr size_t CSMEM = (size_t)(NN + S::CG) * P2 * sizeof(CC<R>);
    static_assert(PSMEM <= 227 * 1024 && KSMEM <= 227 * 1024 && CSMEM <= 227 * 1024, "shared memory of a CTA");
};

// Y = S2 (T_i2 + T_j2) X on one (i2, j2) plane of PW adjacent p; lanes run
// along p.  Thread (p, j) makes the i line, thread (p, i) the j line and the
// result.
template <class R, int NN>
__global__ void __launch_bounds__(Cfg<R, NN>::PT, Cfg<R, NN>::PB) plane_kernel(const __grid_constant__ LineArgs<R> a)
{
    using K = Cfg<R, NN>;
    using X = Cx<R>;
    constexpr int PW = K::PW, P2 = K::P2, M = K::M;
    extern __shared__ __align__(16) unsigned char line_smem[];
    CC<R> *xs = reinterpret_cast<CC<R> *>(line_smem), *ys = xs + PW * P2;  // [j][i][p]
    const int k2 = blockIdx.x / K::RUNS, run = blockIdx.x % K::RUNS;
    const int pp = threadIdx.x % PW, l = threadIdx.x / PW;
    const int p0 = run * PW + pp;
    const bool active = l < NN, valid = active && p0 < M;
    const int64_t base = (p0 < M ? p0 : M - 1) + (int64_t)M * P2 * k2;
    grid_wait();
    grid_release();
    for (int vec = blockIdx.y; vec < a.nvec; vec += gridDim.y) {
        const CC<R> *x = a.x + vec * a.vstride + base;
        CC<R> *y = a.y + vec * a.vstride + base;
        CC<R> v[NN];
        if (active) {
            const CC<R> *g = x + (int64_t)M * NN * l;
            CC<R> *xl = xs + pp + PW * NN * l, *yl = ys + pp + PW * NN * l;
#pragma unroll
            for (int i = 0; i < NN; ++i) v[i] = ld_prev(g + (int64_t)M * i);
#pragma unroll
            for (int i = 0; i < NN; ++i) xl[PW * i] = v[i];
            line_transform<R, NN, 0, sizeof(R) == 8>(
                v, [](int) { return Nothing{}; }, [&](int i, CC<R> z, Nothing) { yl[PW * i] = z; });
        }
        __syncthreads();
        if (active) {
            const CC<R> *xl = xs + pp + PW * l, *yl = ys + pp + PW * l;
            CC<R> *g = y + (int64_t)M * l;
#pragma unroll
            for (int j = 0; j < NN; ++j) v[j] = xl[PW * NN * j];
            line_transform<R, NN, 0, sizeof(R) == 8>(
                v, [&](int j) { return yl[PW * NN * j]; },
                [&](int j, CC<R> z, CC<R> zi) {
                    R yr, yi;
                    times_s2(a, X::add(zi, z), yr, yi);
                    if (valid) g[(int64_t)M * NN * j] = X::make(yr, yi);
                });
        }
        if (vec + (int)gridDim.y < a.nvec) __syncthreads();
    }
}

// Y += S2 T_k2 X + (V + shift) X, one k2 line per thread, lanes along p:
// registers only, every access a contiguous run.
template <class R, int NN>
__global__ void __launch_bounds__(Cfg<R, NN>::KT, Cfg<R, NN>::KB) kline_kernel(const __grid_constant__ LineArgs<R> a)
{
    using K = Cfg<R, NN>;
    using X = Cx<R>;
    constexpr int P2 = K::P2, M = K::M, T = K::KT, W = 2 * NN - 1;
    constexpr int64_t KS = (int64_t)M * P2;
    extern __shared__ __align__(16) unsigned char line_smem[];
    CC<R> *stash = reinterpret_cast<CC<R> *>(line_smem) + threadIdx.x;
    const int idx = blockIdx.x * T + threadIdx.x;  // p + M (i2 + NN j2)
    grid_wait();
    grid_release();
    if (idx >= M * P2) return;
    const int ij = idx / M, p = idx - ij * M;
    // V(p,q) = A TINV(r_p) + A TINV(r_q) + TINV(r_q - r_p)/delta^3 (hammod.F90:576-578)
    const int ip = p % NN, jp = (p / NN) % NN, kp = p / P2;
    const R *vt = a.v12 + (ij % NN - ip + NN - 1) + W * ((ij / NN - jp + NN - 1) + W * (NN - 1 - kp));
    const R *tq = a.t1a + ij;
    const R tp = __ldg(a.t1a + p);
    struct L {
        CC<R> x, y;
        R v;
    };
    for (int vec = blockIdx.y; vec < a.nvec; vec += gridDim.y) {
        const CC<R> *x = a.x + vec * a.vstride + idx;
        CC<R> *y = a.y + vec * a.vstride + idx;
        CC<R> v[NN];
#pragma unroll
        for (int k = 0; k < NN; ++k) v[k] = ld_prev(x + KS * k);
        if constexpr (K::KS) {
#pragma unroll
            for (int k = 0; k < NN; ++k) stash[T * k] = v[k];
        }
        auto potential = [&](int k) { return (__ldg(tq + P2 * k) + tp) + __ldg(vt + W * W * k); };
        R pot[K::KV ? NN : 1];
        if constexpr (K::KV) {
#pragma unroll
            for (int k = 0; k < NN; ++k) pot[k] = potential(k);
        }
        auto sum = [&](CC<R> z, L l) {
            R yr, yi, xr, xi;
            times_s2(a, z, yr, yi);
            X::split(l.x, xr, xi);
            const R pr = fma(l.v, a.vsr, a.shr), pi = fma(l.v, a.vsi, a.shi);
            return G2<R>{yr + (pr * xr - pi * xi), yi + (pr * xi + pi * xr)};
        };
        line_transform<R, NN, K::KV ? 0 : 2, true>(
            v,
            [&](int k) {
                L l;
                if constexpr (K::KS) l.x = stash[T * k];
                else l.x = ld_prev(x + KS * k);
                if constexpr (sizeof(R) == 8) l.y = y[KS * k];
                if constexpr (K::KV) l.v = pot[k];
                else l.v = potential(k);
                return l;
            },
            [&](int k, CC<R> z, L l) {
                const G2<R> s = sum(z, l);
                if constexpr (sizeof(R) == 8) y[KS * k] = X::make(l.y.x + s.x, l.y.y + s.y);
                else add_to(y + KS * k, s);
            },
            [&] {
                if constexpr (sizeof(R) == 8) return Nothing{};
                else return [&](int k1, CC<R> z1, L l1, int k2, CC<R> z2, L l2) {
                    add_to(y + KS * k1, sum(z1, l1), y + KS * k2, sum(z2, l2));
                };
            }());
    }
}

// Y += S2 (T_i1 + T_j1 + T_k1) X (ADD; else Y = ...) on one column X(:, q): k
// lines straight from global memory (lanes along i, j), the i and j lines
// through shared memory.
//
// A CTA per column, so the loop over units makes one turn.  Without it the
// compiler keeps fewer of a line's loads in flight (complex64 at NN = 11: 52
// registers instead of 70), and the launch shapes above fit no more: blocks of 8
// at NN = 11 took 172 us instead of 143 in complex64, 320 instead of 325 in
// complex128.
template <class R, int NN, bool ADD>
__global__ void __launch_bounds__(Cfg<R, NN>::CT, Cfg<R, NN>::CB) cube_line_kernel(const __grid_constant__ LineArgs<R> a)
{
    using K = Cfg<R, NN>;
    using X = Cx<R>;
    constexpr int P2 = K::P2, M = K::M, T = K::CT, G = K::CG;
    constexpr bool ORDER = sizeof(R) == 8;
    extern __shared__ __align__(16) unsigned char line_smem[];
    CC<R> *ys = reinterpret_cast<CC<R> *>(line_smem), *xs = ys + M;  // [k][j][i], G slabs of x
    const int t = threadIdx.x;
    const int64_t nunits = (int64_t)M * a.nvec;
    grid_wait();
    CC<R> v[NN];
    for (int64_t u = blockIdx.x; u < nunits; u += gridDim.x) {
        const bool more = u + gridDim.x < nunits;
        if (!more) grid_release();
        const int64_t vec = u / M, off = vec * a.vstride + (u - vec * M) * M;
        const CC<R> *x = a.x + off;
        CC<R> *y = a.y + off;
#pragma unroll 1
        for (int l = t; l < P2; l += T) {
#pragma unroll
            for (int k = 0; k < NN; ++k) v[k] = ld_prev(x + l + P2 * k);
            if constexpr (G == NN) {
#pragma unroll
                for (int k = 0; k < NN; ++k) xs[l + P2 * k] = v[k];
            }
            CC<R> *yk = ys + l;
            line_transform<R, NN, 0, ORDER>(
                v, [](int) { return Nothing{}; }, [&](int k, CC<R> z, Nothing) { yk[P2 * k] = z; });
        }
#pragma unroll 1
        for (int k0 = 0; k0 < NN; k0 += G) {
            const int gn = G == NN ? NN : min(G, NN - k0);
            if constexpr (G < NN) {
                for (int e = t; e < gn * P2; e += T) xs[e] = ld_prev(x + k0 * P2 + e);
            }
            __syncthreads();
#pragma unroll 1
            for (int l = t; l < gn * NN; l += T) {
                const CC<R> *xl = xs + NN * l;
                CC<R> *yl = ys + k0 * P2 + NN * l;
#pragma unroll
                for (int i = 0; i < NN; ++i) v[i] = xl[i];
                line_transform<R, NN, 0, ORDER>(
                    v, [&](int i) { return yl[i]; }, [&](int i, CC<R> z, CC<R> s) { yl[i] = X::add(s, z); });
            }
            __syncthreads();
#pragma unroll 1
            for (int l = t; l < gn * NN; l += T) {
                const int o = l % NN + P2 * (l / NN);
                const CC<R> *xl = xs + o, *yl = ys + k0 * P2 + o;
                CC<R> *g = y + k0 * P2 + o;
                struct L {
                    CC<R> s, y;
                };
#pragma unroll
                for (int j = 0; j < NN; ++j) v[j] = xl[NN * j];
                line_transform<R, NN, ADD && sizeof(R) == 8 ? 2 : 0, ORDER>(
                    v,
                    [&](int j) {
                        L r;
                        r.s = yl[NN * j];
                        if constexpr (ADD && sizeof(R) == 8) r.y = g[NN * j];
                        return r;
                    },
                    [&](int j, CC<R> z, L r) {
                        G2<R> s;
                        times_s2(a, X::add(r.s, z), s.x, s.y);
                        if constexpr (!ADD) g[NN * j] = X::make(s.x, s.y);
                        else if constexpr (sizeof(R) == 8) g[NN * j] = X::make(r.y.x + s.x, r.y.y + s.y);
                        else add_to(g + NN * j, s);
                    },
                    [&] {
                        if constexpr (!ADD || sizeof(R) == 8) return Nothing{};
                        else return [&](int j1, CC<R> z1, L r1, int j2, CC<R> z2, L r2) {
                            G2<R> s1, s2;
                            times_s2(a, X::add(r1.s, z1), s1.x, s1.y);
                            times_s2(a, X::add(r2.s, z2), s2.x, s2.y);
                            add_to(g + NN * j1, s1, g + NN * j2, s2);
                        };
                    }());
            }
            if (G < NN || more) __syncthreads();
        }
    }
}

// Electron exchange: for X^T = s X (s = 1 or -1) the electron-2 axes need no
// pass of their own, T_2 X = s (T_1 X)^T, so from Z = T_1 X in Y
//   Y <- Z + s Z^T + (V + shift) X
// in place on pairs of 32 x 32 tiles (bi <= bj).  V is symmetric, so the
// partner tile is s times the transpose: only the upper half of X is read,
// and Y is exactly (anti)symmetric.  Memory-bound: 2.5 vector passes after
// the cube kernel's 2, against 8 for the general product.
// Inside the mixed solve at NN = 13 the two take 44 us a product against 59.
// 512 threads with two elements each and three CTAs per SM, measured there (ms
// per outer iteration of 30 products): 5.18; four CTAs 5.39, two 5.26; 256
// threads 5.18 at four CTAs, 5.26 at three; 128 threads 5.38.
constexpr int kExchThreads = 512;
template <class R>
__global__ void __launch_bounds__(kExchThreads, 3)
    exch_add_kernel(const __grid_constant__ LineArgs<R> a, int nn, R s)
{
    using G = G2<R>;
    constexpr int RY = kExchThreads / 32, E = 32 / RY;
    __shared__ G ta[32][33], tb[32][33];
    __shared__ int bp[32], bq[32];
    const int m = nn * nn * nn, w = 2 * nn - 1;
    // the tile pair: blocks enumerate bi <= bj
    int bj = (int)((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while ((bj + 1) * (bj + 2) / 2 <= (int)blockIdx.x) ++bj;
    while (bj * (bj + 1) / 2 > (int)blockIdx.x) --bj;
    const int bi = (int)blockIdx.x - bj * (bj + 1) / 2;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int p0 = bi * 32, q0 = bj * 32;
    if (threadIdx.x < 64) {  // TINV(r_q - r_p) sits at bq - bp of the table
        const int r = min((threadIdx.x < 32 ? p0 : q0) + tx, m - 1);
        const int b = r % nn + w * ((r / nn) % nn + w * (r / (nn * nn)));
        if (threadIdx.x < 32) bp[tx] = b;
        else bq[tx] = b + (nn - 1) * (1 + w + w * w);
    }
    __syncthreads();
    const int p = p0 + tx, pt = q0 + tx;
    const R tp = __ldg(a.t1a + min(p, m - 1));
    grid_wait();
    grid_release();
    for (int vec = blockIdx.y; vec < a.nvec; vec += gridDim.y) {
        const G *x = reinterpret_cast<const G *>(a.x) + vec * a.vstride;
        G *y = reinterpret_cast<G *>(a.y) + vec * a.vstride;
        G za[E], zb[E], xa[E];
        R v[E];
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int c = ty + RY * u;
            const bool oka = p < m && q0 + c < m, okb = pt < m && p0 + c < m;
            zb[u] = okb ? y[pt + (int64_t)m * (p0 + c)] : G{R(0), R(0)};
            za[u] = oka ? y[p + (int64_t)m * (q0 + c)] : G{R(0), R(0)};
            xa[u] = oka ? ld_prev(x + p + (int64_t)m * (q0 + c)) : G{R(0), R(0)};
            // in a diagonal tile both orders of a pair take the same table entry
            // (TINV's two halves agree to rounding only)
            const int lo = bi == bj ? min(c, tx) : tx, hi = bi == bj ? max(c, tx) : c;
            v[u] = (__ldg(a.t1a + min(q0 + c, m - 1)) + tp) + __ldg(a.v12 + bq[hi] - bp[lo]);
        }
#pragma unroll
        for (int u = 0; u < E; ++u) tb[tx][ty + RY * u] = zb[u];  // tb[r][c] = Z(q0 + r, p0 + c)
        __syncthreads();
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int c = ty + RY * u, q = q0 + c;
            const R pr = fma(v[u], a.vsr, a.shr), pi = fma(v[u], a.vsi, a.shi);
            const G zt = tb[c][tx];
            R yr = za[u].x + s * zt.x, yi = za[u].y + s * zt.y;
            yr += pr * xa[u].x - pi * xa[u].y;
            yi += pr * xa[u].y + pi * xa[u].x;
            ta[tx][c] = G{yr, yi};  // ta[r][c] = Y(p0 + r, q0 + c)
            if (p < m && q < m) y[p + (int64_t)m * q] = G{yr, yi};
        }
        __syncthreads();
        if (bi != bj) {
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const int c = ty + RY * u;
                const G t = ta[c][tx];  // Y(p0 + c, q0 + tx)
                if (pt < m && p0 + c < m) y[pt + (int64_t)m * (p0 + c)] = G{s * t.x, s * t.y};
            }
        }
    }
}

template <class R>
cudaError_t launch(void (*kernel)(LineArgs<R>), dim3 grid, int threads, size_t smem, const LineArgs<R> &a,
                   cudaStream_t st)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = programmatic_launch() ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

// Shared-memory limits of one grid's kernels, set once per device.
template <class R, int NN>
cudaError_t prepare()
{
    using K = Cfg<R, NN>;
    static std::atomic<bool> done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(plane_kernel<R, NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::PSMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kline_kernel<R, NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::KSMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(cube_line_kernel<R, NN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)K::CSMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(cube_line_kernel<R, NN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)K::CSMEM);
    if (e == cudaSuccess) done[dev].store(true, std::memory_order_release);
    return e;
}

template <class R, int NN>
cudaError_t pass(const LineArgs<R> &a, int which, cudaStream_t st)
{
    using K = Cfg<R, NN>;
    cudaError_t e = prepare<R, NN>();
    if (e != cudaSuccess) return e;
    const unsigned ny = (unsigned)std::min(a.nvec, 65535);
    if (which == 0) {
        e = launch<R>(plane_kernel<R, NN>, dim3(NN * K::RUNS, ny), K::PT, K::PSMEM, a, st);
        if (e != cudaSuccess) return e;
        return launch<R>(kline_kernel<R, NN>, dim3((K::M * K::P2 + K::KT - 1) / K::KT, ny), K::KT, K::KSMEM, a, st);
    }
    const unsigned units = (unsigned)std::min<int64_t>((int64_t)K::M * a.nvec, 0x7fffffff);
    return launch<R>(which == 1 ? cube_line_kernel<R, NN, true> : cube_line_kernel<R, NN, false>, dim3(units), K::CT,
                     K::CSMEM, a, st);
}

template <class R, class G>
LineArgs<R> line_args(const HamDev &h, const G *x, G *y, int nvec, int64_t vstride, double2 shift)
{
    LineArgs<R> a{};
    a.x = reinterpret_cast<const CC<R> *>(x);
    a.y = reinterpret_cast<CC<R> *>(y);
    if constexpr (sizeof(R) == 8) {
        a.t1a = h.t1a;
        a.v12 = h.v12;
    } else {
        a.t1a = h.t1af;
        a.v12 = h.v12f;
    }
    a.vstride = vstride;
    a.nvec = nvec;
    a.s2r = (R)(h.s2re * h.id2);
    a.s2i = (R)(h.s2im * h.id2);
    a.vsr = (R)h.vsre;
    a.vsi = (R)h.vsim;
    a.shr = (R)shift.x;
    a.shi = (R)shift.y;
    return a;
}

template <class R>
cudaError_t go(const HamDev &h, const LineArgs<R> &a, int which, cudaStream_t st)
{
    switch (h.nn) {
    case 3: return pass<R, 3>(a, which, st);
    case 5: return pass<R, 5>(a, which, st);
    case 7: return pass<R, 7>(a, which, st);
    case 9: return pass<R, 9>(a, which, st);
    case 11: return pass<R, 11>(a, which, st);
    case 13: return pass<R, 13>(a, which, st);
    case 15: return pass<R, 15>(a, which, st);
    case 17: return pass<R, 17>(a, which, st);
    case 19: return pass<R, 19>(a, which, st);
    case 21: return pass<R, 21>(a, which, st);
    case 23: return pass<R, 23>(a, which, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t hammult_line_pass_launch(const HamDev &h, const double2 *x, double2 *y, int nvec, int64_t vstride,
                                     int pass, cudaStream_t st, double2 shift)
{
    return go<double>(h, line_args<double>(h, x, y, nvec, vstride, shift), pass, st);
}

cudaError_t hammult_line_pass_launch(const HamDev &h, const float2 *x, float2 *y, int nvec, int64_t vstride,
                                     int pass, cudaStream_t st, double2 shift)
{
    return go<float>(h, line_args<float>(h, x, y, nvec, vstride, shift), pass, st);
}

template <class R, class G>
static cudaError_t exch_pass(const HamDev &h, const G *x, G *y, int nvec, int64_t vstride, int pass, double sign,
                             cudaStream_t st, double2 shift)
{
    if (h.nelec != 2 || nvec <= 0) return cudaErrorInvalidValue;
    const LineArgs<R> a = line_args<R>(h, x, y, nvec, vstride, shift);
    if (!a.t1a || !a.v12) return cudaErrorInvalidValue;
    if (pass == 0) return go<R>(h, a, 2, st);
    const int tiles = (int)((h.m + 31) / 32);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles * (tiles + 1) / 2), (unsigned)std::min(nvec, 65535));
    cfg.blockDim = dim3(kExchThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = programmatic_launch() ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, exch_add_kernel<R>, a, h.nn, (R)sign);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t hammult_exch_pass_launch(const HamDev &h, const float2 *x, float2 *y, int nvec, int64_t vstride, int pass,
                                     double sign, cudaStream_t st, double2 shift)
{
    return exch_pass<float>(h, x, y, nvec, vstride, pass, sign, st, shift);
}

cudaError_t hammult_exch_pass_launch(const HamDev &h, const double2 *x, double2 *y, int nvec, int64_t vstride, int pass,
                                     double sign, cudaStream_t st, double2 shift)
{
    return exch_pass<double>(h, x, y, nvec, vstride, pass, sign, st, shift);
}

}  // namespace de

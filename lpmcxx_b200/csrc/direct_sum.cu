// Direct (all-pairs) sums: the pair loops of DirectSum::meshSolve (src/LpmDirectSum.cpp:94-167)
// and DirectSum::meshfreeSolve (src/LpmDirectSum.cpp:175-254) as shared-memory-tiled sm_100a
// kernels.
//
// Layout: sources are packed n x 4 (x, y, z, w) with w = strength (vorticity * area, or charge);
// a block stages kTile sources in shared memory and its threads sweep them against their
// TPT register-resident targets, so each source is read once per block from HBM/L2 and once
// per thread from shared memory as a broadcast 128-bit load.  The sources are split over thread groups
// and over the blocks of a cluster (Split below).
//
// FP64 kernels: den = (R^2 - x.y) + delta^2, the term is dropped when |den| <= 1e-13
// (src/LpmVectorKernel.h:24-28).  The sum is reorganised as u = mult * (x cross sum_j (w_j/den_j) y_j),
// since x cross (.) is linear, which saves the per-pair cross product (close pairs: see BsF64).
//
// FP32 kernels use 1 - x.y = |x - y|^2 / 2 for points on the sphere (no cancellation for close
// pairs), accumulate sum_j (2 w_j / (r_j^2 + 2 delta^2)) (x - y_j) in FP32 over one shared-memory
// tile and add each tile's partial into FP64 accumulators (a compensated two-level sum); the
// final u = -mult * (x cross D) uses the FP64 target position.
#include "lpm_internal.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace lpm {

namespace {

constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr double kZeroTol = 1.0e-13;  // ZERO_TOL (src/LpmTypeDefs.h:33-34)

// The hardware's approximate reciprocal and reciprocal square root of a double (about 20 bits).
__device__ __forceinline__ double rcp64_approx(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    return r;
}
__device__ __forceinline__ double rsqrt64_approx(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    return y;
}

// Reciprocal: hardware approximation refined by two Newton-Raphson steps r <- r + r(1 - d r)
// (quadratic convergence from ~2^-22 gives full double precision, within one ulp).
__device__ __forceinline__ double rcp64(double d) {
    double r = rcp64_approx(d);
    double e = fma(-d, r, 1.0);
    r = fma(r, e, r);
    e = fma(-d, r, 1.0);
    return fma(r, e, r);
}

// Reciprocal square root: hardware approximation refined by two Newton-Raphson steps
// y <- y + (y/2)(1 - a y^2).
__device__ __forceinline__ double rsqrt64(double a) {
    double y = rsqrt64_approx(a);
    double t = a * y;
    double e = fma(-t, y, 1.0);
    y = fma(0.5 * y, e, y);
    t = a * y;
    e = fma(-t, y, 1.0);
    return fma(0.5 * y, e, y);
}

__device__ __forceinline__ float rcp32(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt32(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

constexpr int kThreads = 256;    // FP32 kernels
constexpr int kThreads64 = 128;  // FP64 kernels
constexpr int kTile = 256;       // sources staged per tile

// ------------------------------------------------------------------ source splits
// The threads of a block form G groups (G = 1 << gshift): each group holds the block's threads x TPT / G targets and
// sums its own share of the block's sources, and the blocks of a cluster of C share one set of targets and split the
// sources C ways, so that a small or ragged problem gets up to 32 times the blocks and warps its targets alone would
// make.  At the end every thread leaves its FP64 sums in shared memory and the cluster's blocks add the G C sums of a
// target in a fixed order (their own block's and, through distributed shared memory, the others'): the result does
// not depend on timing, and no workspace is needed.  One block per 512 (FP64) or 1,024 (FP32) targets, as before,
// left most SMs idle below 10^5 targets: 1,280 sources x 1,922 targets 121 -> 12.3 us, 5,120 x 7,682 482 -> 57.5 us
// (FP64); 24,576 x 49,154 878 -> 536 us (FP32).
struct Split {
    int gshift;  // log2 of the thread groups per block
    int parts;   // blocks per cluster = source parts
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The threads have left their sums in red[group][target][component][thread of the group]: adds them over the groups
// and the cluster's blocks and hands each target (in block order u = target * (threads per group) + thread) to
// finish(u, sums) once, in the block that owns it.
template <int TPT, int NC, int NT, class Finish>
__device__ __forceinline__ void reduce_split(double* red, Split sp, int rank, Finish finish) {
    const int gw = NT >> sp.gshift, groups = 1 << sp.gshift;
    if (sp.parts > 1) cluster_barrier();
    else __syncthreads();
    const int tb = gw * TPT, own = tb / sp.parts;  // powers of two, tb >= 64 and parts <= 8
    for (int u = rank * own + (int)threadIdx.x; u < (rank + 1) * own; u += NT) {
        const int t = u / gw, l = u - t * gw;
        double s[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) s[c] = 0.0;
        for (int p = 0; p < sp.parts; ++p)
#pragma unroll 4
            for (int g = 0; g < groups; ++g)
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const double* at = red + ((g * TPT + t) * NC + c) * gw + l;
                    s[c] += sp.parts > 1 ? cluster_load(at, p) : *at;
                }
        finish(u, s);
    }
    if (sp.parts > 1) cluster_barrier();  // no block leaves while another reads its sums
}

// ------------------------------------------------------------------ FP64 pair sums
// One op per kernel: TPT targets per thread; init() makes what a thread keeps for the launch, prepare() forms what a
// staged source needs beside its coordinates and strength, tile() sums a run of staged sources (src and aux, m of them)
// into the thread's targets, finish() writes one target's result from its NC sums.

struct NoState {};

// The common paths take finite points and strengths of ordinary size only, so that no intermediate overflows or
// becomes NaN; a tile that holds another source, and every tile of a warp that holds another target, is summed by the
// pair-by-pair path, which treats such values as the reference's expression does.
__device__ __forceinline__ bool odd_point(const double4& p) {
    return !(fabs(p.x) < 1e150 && fabs(p.y) < 1e150 && fabs(p.z) < 1e150);
}
__device__ __forceinline__ bool odd_strength(double w) {
    return !(fabs(w) < 1e150 && (w == 0.0 || fabs(w) > 1e-150));
}

// FP64 Biot-Savart.  The bound is the FP64 pipe; 9 operations a pair on the common path against 18 with the
// reference's expression:
//   den = R^2 + delta^2 - x.y by three fused steps instead of six rounded ones,
//   r = 1/den by Householder's third-order step r0 (1 + e + e^2), e = 1 - den r0 (remainder e^3 < 2^-57), three
//       operations against four of two Newton steps,
//   S += r (w y), three operations: x cross y = x cross (y - x), so S needs no y - x, and w y is formed once per
//       staged source.
// A pair whose den is small beside R^2 (below 2^-10 R^2, below the kernel's own 1e-13, or not finite) takes the
// reference's rounding step by step instead: (x x' + y y') + z z' without fused multiply-adds, as
// XyzVector::dotProduct, and S += f (y - x), so that den carries the same rounding error where cancellation magnifies
// it and the sum loses no digits to terms much larger than their cross product.  Elsewhere the fused den errs by at
// most 3 2^-53 R^2, as the unfused one, and S is summed tile by tile (kTile sources, then the tiles), which keeps
// its rounding below that of one long sum: relative L2 error of the result against 80-bit sums 4.5e-15 / 2.0e-14 /
// 7.7e-14 at 1,500 / 6,000 / 24,000 sources, against 7.4e-15 / 2.5e-14 / 7.7e-14 of the reference's expression.
// The test for small dens runs on the integer pipe, on high words, once per source as a warp vote; the dens of the
// next source are formed beside the current one's reciprocals and sums, so that the two chains overlap.  What bounds
// the kernel now is the register file beside the pipe: an FP64 FMA of three distinct register operands issues every
// three cycles instead of two (a probe of the instruction alone), and the ~9 other instructions a pair share its
// ports.  81,920 sources x 122,882 targets: 14.26 -> 8.0 ms (12.0 -> 21.4 TFLOP/s at 17 flops a pair).  Two or four
// sources a vote, two targets a thread, or more resident warps with fewer registers: 8.3 - 10.2 ms where this form took
// 8.35 (with missing targets on the long path).
template <bool kDelta, int kTPT>
struct BsF64 {
    static constexpr int NC = 3, TPT = kTPT;
    static constexpr bool kSelf = false, kAux = true, kCheck = true;
    static constexpr int kCrowd = 5;
    double r2, d2, c0;   // R^2, delta^2, R^2 + delta^2
    int lo;              // a den whose high word is at least lo takes the common path

    __device__ __forceinline__ static NoState init() { return NoState{}; }
    __device__ __forceinline__ static double4 prepare(const double4& y) {
        return make_double4(y.w * y.x, y.w * y.y, y.w * y.z, 0.0);
    }
    __device__ __forceinline__ void pair(double (&s)[NC], double tx, double ty, double tz, const double4& y) const {
        const double dot = __dadd_rn(__dadd_rn(__dmul_rn(tx, y.x), __dmul_rn(ty, y.y)), __dmul_rn(tz, y.z));
        double den = r2 - dot;
        if (kDelta) den += d2;
        double f = y.w * rcp64(den);
        f = fabs(den) > kZeroTol ? f : 0.0;
        s[0] = fma(f, y.x - tx, s[0]);
        s[1] = fma(f, y.y - ty, s[1]);
        s[2] = fma(f, y.z - tz, s[2]);
    }
    // the dens of one source; returns the smallest high word (as a signed number: a negative den is small too)
    __device__ __forceinline__ int dens(const double4& y, const double (&tx)[TPT], const double (&ty)[TPT],
                                        const double (&tz)[TPT], double (&den)[TPT]) const {
        int least = 0x7fffffff;
#pragma unroll
        for (int t = 0; t < TPT; ++t) den[t] = fma(-tx[t], y.x, c0);
#pragma unroll
        for (int t = 0; t < TPT; ++t) den[t] = fma(-ty[t], y.y, den[t]);
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
            den[t] = fma(-tz[t], y.z, den[t]);
            least = min(least, __double2hiint(den[t]));
        }
        return least;
    }
    // source *src of the run, whose dens are formed: its reciprocals and sums, beside the dens of *next_src
    __device__ __forceinline__ void step(const double4* src, const double4* aux, const double4* next_src,
                                         const double (&tx)[TPT], const double (&ty)[TPT], const double (&tz)[TPT],
                                         const double (&den)[TPT], int least, double (&next)[TPT], int& next_least,
                                         double (&s)[TPT][NC]) const {
        if (__all_sync(0xffffffffu, least >= lo)) {
            next_least = dens(*next_src, tx, ty, tz, next);
            const double4 wy = *aux;
#pragma unroll
            for (int t = 0; t < TPT; ++t) {
                const double r = rcp64_approx(den[t]), e = fma(-den[t], r, 1.0);
                const double f = fma(r, fma(e, e, e), r);
                s[t][0] = fma(f, wy.x, s[t][0]);
                s[t][1] = fma(f, wy.y, s[t][1]);
                s[t][2] = fma(f, wy.z, s[t][2]);
            }
        } else {
#pragma unroll
            for (int t = 0; t < TPT; ++t) pair(s[t], tx[t], ty[t], tz[t], *src);
            next_least = dens(*next_src, tx, ty, tz, next);
        }
    }
    __device__ __forceinline__ void tile(const NoState&, const double4* src, const double4* aux, int m, bool plain, int64_t,
                                         const double (&tx)[TPT], const double (&ty)[TPT], const double (&tz)[TPT],
                                         const int64_t (&)[TPT], double (&s)[TPT][NC]) const {
        int k = 0;
        if (plain && m >= 2) {
            double a[TPT], b[TPT];
            int la = dens(src[0], tx, ty, tz, a), lb = 0;
            do {  // two sources a round; after the last round's second source its first is formed again, unused
                step(src + k, aux + k, src + k + 1, tx, ty, tz, a, la, b, lb, s);
                step(src + k + 1, aux + k + 1, src + min(k + 2, m - 2), tx, ty, tz, b, lb, a, la, s);
                k += 2;
            } while (k <= m - 2);
        }
#pragma unroll 1
        for (; k < m; ++k)
#pragma unroll
            for (int t = 0; t < TPT; ++t) pair(s[t], tx[t], ty[t], tz[t], src[k]);
    }
    __device__ __forceinline__ void finish(int64_t i, const double (&s)[NC], const double4* tgt, double mult,
                                           double* out, int64_t stride) const {
        const double4 x = tgt[i];
        out[i] = mult * (x.y * s[2] - x.z * s[1]);
        out[stride + i] = mult * (x.z * s[0] - x.x * s[2]);
        out[2 * stride + i] = mult * (x.x * s[1] - x.y * s[0]);
    }
};

// FP64 Poisson 1/(4 pi r): 12 FP64 operations a pair against 17.  1/r by Householder's third-order step
// y (1 + e (1/2 + 3/8 e)), e = 1 - r^2 y^2, in place of two Newton steps; a coincident pair (or one whose r^2 is
// subnormal) adds nothing, by a select of the approximation's high word on the integer pipe (its low word is 0).
// 20,011 points: 2.85 ms -> 0.35 ms (with the split), 100,011 points 8.5 ms.
template <int kTPT>
struct PoissonF64 {
    static constexpr int NC = 1, TPT = kTPT;
    static constexpr bool kSelf = false, kAux = false, kCheck = true;
    static constexpr int kCrowd = 5;

    __device__ __forceinline__ static NoState init() { return NoState{}; }
    __device__ __forceinline__ static double4 prepare(const double4& y) { return y; }
    __device__ __forceinline__ void tile(const NoState&, const double4* src, const double4*, int m, bool plain, int64_t,
                                         const double (&tx)[TPT], const double (&ty)[TPT], const double (&tz)[TPT],
                                         const int64_t (&)[TPT], double (&s)[TPT][NC]) const {
        if (plain) {
#pragma unroll 4
            for (int k = 0; k < m; ++k) {
                const double4 p = src[k];
#pragma unroll
                for (int t = 0; t < TPT; ++t) {
                    const double dx = tx[t] - p.x, dy = ty[t] - p.y, dz = tz[t] - p.z;
                    const double rr = dx * dx + dy * dy + dz * dz;
                    // high word of the smallest normal number: below it the pair adds nothing
                    const int hi = __double2hiint(rr) >= 0x00100000 ? __double2hiint(rsqrt64_approx(rr)) : 0;
                    const double y = __hiloint2double(hi, 0);
                    const double e = fma(-(rr * y), y, 1.0);
                    s[t][0] = fma(p.w, fma(y, e * fma(0.375, e, 0.5), y), s[t][0]);
                }
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < m; ++k)
#pragma unroll
                for (int t = 0; t < TPT; ++t) {
                    const double4 p = src[k];
                    const double dx = tx[t] - p.x, dy = ty[t] - p.y, dz = tz[t] - p.z;
                    const double rr = dx * dx + dy * dy + dz * dz;
                    s[t][0] = fma(p.w, rr > 0.0 ? rsqrt64(rr) : 0.0, s[t][0]);
                }
        }
    }
    __device__ __forceinline__ void finish(int64_t i, const double (&s)[NC], const double4*, double mult, double* out,
                                           int64_t) const {
        out[i] = mult * s[0];
    }
};

// The ScalarKernel family.  Pair values without the constant factor (applied once per target as `mult`), each
// formed as the reference forms it (products and sums without contraction where the reference has no FMA):
//   SphereGreensFn        -log(R^2 - y.x) / (4 pi R)           (src/LpmScalarKernel.h:31-45)
//   PlanarGreens...       log(|x - y|^2) / (4 pi)              (src/LpmScalarKernel.h:19-29)
//   SecondOrderDelta3d    3 exp(-(|x - y|/eps)^3) / (4 pi eps^3) (src/LpmScalarKernel.h:47-62)
//   SphereDelta           (2 eps^2 d - (1 - d)^2) / (4 pi (1 - d + eps^2)^2) - 1/(4 pi), d = x.y
//                                                               (src/LpmScalarKernel.h:64-78)
struct Delta3dPair {
    double inv_eps;
    __device__ double operator()(double tx, double ty, double tz, double sx, double sy, double sz) const {
        const double dx = tx - sx, dy = ty - sy, dz = tz - sz;
        const double q = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz))) * inv_eps;
        return exp(-(q * q * q));
    }
};
struct SphereDeltaPair {
    double eps2;
    __device__ double operator()(double tx, double ty, double tz, double sx, double sy, double sz) const {
        const double d = __dadd_rn(__dadd_rn(__dmul_rn(tx, sx), __dmul_rn(ty, sy)), __dmul_rn(tz, sz));
        const double numer = 2.0 * eps2 * d - (1.0 - d) * (1.0 - d);
        const double den = 1.0 - d + eps2;
        return numer / (den * den) - 1.0;
    }
};

// sum_j w_j K(x_i, y_j) of the kernels that are not singular.
template <class K>
struct ScalarF64 {
    static constexpr int NC = 1, TPT = 2;
    static constexpr bool kSelf = false, kAux = false, kCheck = false;
    static constexpr int kCrowd = 24;
    K kern;

    __device__ __forceinline__ static NoState init() { return NoState{}; }
    __device__ __forceinline__ static double4 prepare(const double4& y) { return y; }
    __device__ __forceinline__ void tile(const NoState&, const double4* src, const double4*, int m, bool, int64_t,
                                         const double (&tx)[TPT], const double (&ty)[TPT], const double (&tz)[TPT],
                                         const int64_t (&)[TPT], double (&s)[TPT][NC]) const {
        for (int k = 0; k < m; ++k) {
            const double4 y = src[k];
#pragma unroll
            for (int t = 0; t < TPT; ++t) {
                s[t][0] = fma(y.w, kern(tx[t], ty[t], tz[t], y.x, y.y, y.z), s[t][0]);
            }
        }
    }
    __device__ __forceinline__ void finish(int64_t i, const double (&s)[NC], const double4*, double mult, double* out,
                                           int64_t) const {
        out[i] = mult * s[0];
    }
};

// The two logarithmic kernels.  z() is the argument of the logarithm as the reference rounds it, fast_z() by fused steps.
struct SphereGreensArg {
    double r2;
    int lo;  // high word below which z counts as small: 2^-10 R^2, as BsF64's
    __device__ __forceinline__ double z(double tx, double ty, double tz, const double4& y) const {
        return r2 - __dadd_rn(__dadd_rn(__dmul_rn(y.x, tx), __dmul_rn(y.y, ty)), __dmul_rn(y.z, tz));
    }
    __device__ __forceinline__ double fast_z(double tx, double ty, double tz, const double4& y) const {
        return fma(-tz, y.z, fma(-ty, y.y, fma(-tx, y.x, r2)));
    }
};
struct PlanarLogArg {
    int lo;  // high word of the smallest normal number
    __device__ __forceinline__ double z(double tx, double ty, double tz, const double4& y) const {
        const double dx = tx - y.x, dy = ty - y.y, dz = tz - y.z;
        return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    }
    __device__ __forceinline__ double fast_z(double tx, double ty, double tz, const double4& y) const {
        const double dx = tx - y.x, dy = ty - y.y, dz = tz - y.z;
        return fma(dz, dz, fma(dy, dy, dx * dx));
    }
};

// sum_j w_j log z(x_i, y_j), skipping j == self[t].  The CUDA library's log takes about 130 issue cycles a pair here; the
// common path forms it after Tang (Table-driven implementation of the logarithm function in IEEE floating-point
// arithmetic, ACM TOMS 16, 1990): z = 2^k m with m in [0.742, 1.484), c = 1/v to 20 bits for the nearest of 32 points
// v = 0.75, 0.75 + 1/64, ..., 1, 1 + 1/32, ... 1.46875, r = m c - 1 (exact before one rounding, |r| <= 2^-6, c = 1 about
// m = 1), log z = k log 2 - log c + log1p(r), log1p by its series to r^9 (the remainder is below 2^-57 of r).  The table is
// one entry per lane, read by shuffles.  k log 2 is summed as sum w k and multiplied once a target.  17 FP64 operations
// a pair; a pair with a small or not finite z, a tile that holds a target's own source and every other special case take
// the library's log on the reference's rounding.  20,480 sources x 30,722 targets from host arrays: 2.64 -> 1.6 ms (9.17
// before the sources were split); relative L2 error against 64-bit sums 2.8e-16, as with the library's log.
template <class Arg>
struct LogF64 {
    static constexpr int NC = 2, TPT = 2;  // sum w (log z - k log 2), sum w k
    static constexpr bool kSelf = true, kAux = false, kCheck = true;
    static constexpr int kCrowd = 24;
    Arg arg;

    struct State {  // the lane's entry of the table: the high word of c, -log c
        int c_hi, t_hi, t_lo;
    };
    __device__ __forceinline__ static State init() {
        const int lane = threadIdx.x & 31;
        const double v = lane < 16 ? 0.75 + lane / 64.0 : 1.0 + (lane - 16) / 32.0;
        State st;
        st.c_hi = __double2hiint(1.0 / v);
        const double t = -log(__hiloint2double(st.c_hi, 0));
        st.t_hi = __double2hiint(t);
        st.t_lo = __double2loint(t);
        return st;
    }
    __device__ __forceinline__ static double4 prepare(const double4& y) { return y; }
    __device__ __forceinline__ void tile(const State& st, const double4* src, const double4*, int m, bool plain, int64_t j0,
                                         const double (&tx)[TPT], const double (&ty)[TPT], const double (&tz)[TPT],
                                         const int64_t (&self)[TPT], double (&s)[TPT][NC]) const {
        bool own = false;
#pragma unroll
        for (int t = 0; t < TPT; ++t) own = own || (self[t] >= j0 && self[t] < j0 + m);
        const bool fast = plain && !__any_sync(0xffffffffu, own);
#pragma unroll 1
        for (int k = 0; k < m; ++k) {
            const double4 y = src[k];
            double z[TPT];
            int least = 0x7fffffff;
#pragma unroll
            for (int t = 0; t < TPT; ++t) {
                z[t] = arg.fast_z(tx[t], ty[t], tz[t], y);
                least = min(least, __double2hiint(z[t]));
            }
            if (__all_sync(0xffffffffu, fast && least >= arg.lo)) {
#pragma unroll
                for (int t = 0; t < TPT; ++t) {
                    constexpr int kBase = 0x3fe7c000;  // 0.75 less half a step of the table
                    const int off = __double2hiint(z[t]) - kBase, e = off >> 20, j = (off >> 15) & 31;
                    const double c = __hiloint2double(__shfl_sync(0xffffffffu, st.c_hi, j), 0);
                    const double lc = __hiloint2double(__shfl_sync(0xffffffffu, st.t_hi, j),
                                                       __shfl_sync(0xffffffffu, st.t_lo, j));
                    const double r = fma(__hiloint2double(__double2hiint(z[t]) - (e << 20), __double2loint(z[t])), c, -1.0);
                    double q = fma(r, 1.0 / 9.0, -1.0 / 8.0);
                    q = fma(q, r, 1.0 / 7.0);
                    q = fma(q, r, -1.0 / 6.0);
                    q = fma(q, r, 1.0 / 5.0);
                    q = fma(q, r, -1.0 / 4.0);
                    q = fma(q, r, 1.0 / 3.0);
                    q = fma(q, r, -1.0 / 2.0);
                    const double l = lc + fma(r * r, q, r);
                    // e as a double: the integer in the last bits of 2^52 + 2^31
                    const double ed = __hiloint2double(0x43300000, e ^ (int)0x80000000) - 4503601774854144.0;
                    s[t][0] = fma(y.w, l, s[t][0]);
                    s[t][1] = fma(y.w, ed, s[t][1]);
                }
            } else {
#pragma unroll
                for (int t = 0; t < TPT; ++t)
                    if (j0 + k != self[t]) s[t][0] = fma(y.w, log(arg.z(tx[t], ty[t], tz[t], y)), s[t][0]);
            }
        }
    }
    __device__ __forceinline__ void finish(int64_t i, const double (&s)[NC], const double4*, double mult, double* out,
                                           int64_t) const {
        out[i] = mult * fma(s[1], 0.69314718055994530942, s[0]);
    }
};

// FP64 direct sum: each block sums its part of the sources (n_src / parts consecutive ones), staged kTile at a time by
// cp.async one tile ahead of the tile being summed; the groups take consecutive shares of every tile.  A tile's sums
// start from zero and are then added to the thread's totals, which stay in shared memory between tiles (one read and
// write a tile).  Blocks of 128 threads: a barrier a tile holds four warps together, and the warps' times differ
// where close pairs send some of them through the long path (8.35 against 8.8 ms by 256 threads on 81,920
// sources x 122,882 targets).
template <class Op>
struct Shape64 {
    static constexpr int kRow = Op::kAux ? 2 * kTile : kTile;  // a stage: the sources, then what prepare() made
    static constexpr size_t kSmem = sizeof(double4) * 2 * kRow + sizeof(double) * kThreads64 * Op::TPT * Op::NC;
};

template <class Op>
__global__ void __launch_bounds__(kThreads64, 4) direct64_kernel(const double4* __restrict__ src, int64_t n_src,
                                                                 const double4* __restrict__ tgt, int64_t n_tgt, Op op,
                                                                 double mult, double* __restrict__ out, int64_t stride,
                                                                 int64_t coinc_n, int64_t coinc_off, Split sp) {
    constexpr int TPT = Op::TPT, NC = Op::NC, kRow = Shape64<Op>::kRow;
    extern __shared__ __align__(32) double4 smem64[];  // two stages, then the totals
    double* totals = (double*)(smem64 + 2 * kRow);     // [group][target][component][thread of the group]
    const int gw = kThreads64 >> sp.gshift;
    const int grp = (int)threadIdx.x / gw, lt = (int)threadIdx.x - grp * gw;
    const int rank = (int)(blockIdx.x % (unsigned)sp.parts);
    const int64_t blk0 = (int64_t)(blockIdx.x / (unsigned)sp.parts) * (gw * TPT);
    const bool live = blk0 + (lt & ~31) < n_tgt;  // warp-uniform
    double* mine = totals + grp * TPT * NC * gw + lt;
    double tx[TPT], ty[TPT], tz[TPT];
    int64_t self[TPT];
    bool odd = false;
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
        const int64_t i = blk0 + lt + t * gw;
        const double4 p = i < n_tgt ? tgt[i] : make_double4(0.0, 0.0, 0.0, 0.0);  // den R^2: never a close pair
        tx[t] = p.x; ty[t] = p.y; tz[t] = p.z;
        odd = odd || odd_point(p);
        self[t] = Op::kSelf && i < coinc_n ? coinc_off + i : -1;
#pragma unroll
        for (int c = 0; c < NC; ++c) mine[(t * NC + c) * gw] = 0.0;
    }
    const auto state = op.init();
    const bool plain_targets = !__any_sync(0xffffffffu, odd);
    const int64_t begin = n_src * rank / sp.parts, end = n_src * (rank + 1) / sp.parts;
    auto load = [&](int64_t j0, int buf) {
#pragma unroll
        for (int q = threadIdx.x; q < kTile; q += kThreads64)
            if (j0 + q < end) {
                double4* at = smem64 + buf * kRow + q;
                cp_async16(at, src + j0 + q);
                cp_async16((char*)at + 16, (const char*)(src + j0 + q) + 16);
            }
    };
    if (begin < end) load(begin, 0);
    int buf = 0;
    for (int64_t j0 = begin; j0 < end; j0 += kTile, buf ^= 1) {
        const int n = (int)min((int64_t)kTile, end - j0);
        double4* st = smem64 + buf * kRow;
        cp_async_wait_all();
        bool plain = plain_targets;
        if constexpr (Op::kCheck) {  // each thread on the sources it copied
            bool bad = false;
#pragma unroll
            for (int q = threadIdx.x; q < kTile; q += kThreads64)
                if (q < n) {
                    bad = bad || odd_point(st[q]) || odd_strength(st[q].w);
                    if constexpr (Op::kAux) st[kTile + q] = Op::prepare(st[q]);
                }
            plain = !__syncthreads_or(bad) && plain;
        } else {
            __syncthreads();
        }
        // this tile has landed, and the other buffer's readers are done
        if (j0 + kTile < end) load(j0 + kTile, buf ^ 1);
        const int share = (n + (1 << sp.gshift) - 1) >> sp.gshift;
        const int lo = min(n, grp * share), m = min(n - lo, share);
        if (live && m > 0) {
            double s[TPT][NC];
#pragma unroll
            for (int t = 0; t < TPT; ++t)
#pragma unroll
                for (int c = 0; c < NC; ++c) s[t][c] = 0.0;
            op.tile(state, st + lo, st + kTile + lo, m, plain, j0 + lo, tx, ty, tz, self, s);
#pragma unroll
            for (int t = 0; t < TPT; ++t)
#pragma unroll
                for (int c = 0; c < NC; ++c) mine[(t * NC + c) * gw] += s[t][c];
        }
    }
    reduce_split<TPT, NC, kThreads64>(totals, sp, rank, [&](int u, const double (&v)[NC]) {
        if (blk0 + u < n_tgt) op.finish(blk0 + u, v, tgt, mult, out, stride);
    });
}

// FP64 direct sum of at most kFew sources: one per thread to stage, no groups, parts or totals; a thread sums its targets
// over all of them and writes its results.  Bound by the targets' loads and the results' stores: at few sources the
// totals' way through shared memory costs more than the pairs (1 source x 300,000 / 1M targets 14.7 / 41 us by
// direct64_kernel in four groups, 10.6 / 27 in one).
constexpr int kFew = kThreads64;
template <class Op>
__global__ void __launch_bounds__(kThreads64) direct64_few_kernel(const double4* __restrict__ src, int n_src,
                                                                  const double4* __restrict__ tgt, int64_t n_tgt, Op op,
                                                                  double mult, double* __restrict__ out, int64_t stride,
                                                                  int64_t coinc_n, int64_t coinc_off) {
    constexpr int TPT = Op::TPT, NC = Op::NC;
    __shared__ double4 st[Op::kAux ? 2 * kFew : kFew];
    const int64_t first = (int64_t)blockIdx.x * (kThreads64 * TPT) + threadIdx.x;
    double tx[TPT], ty[TPT], tz[TPT], s[TPT][NC];
    int64_t self[TPT];
    bool odd = false, bad = false;
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
        const int64_t i = first + t * kThreads64;
        const double4 p = i < n_tgt ? tgt[i] : make_double4(0.0, 0.0, 0.0, 0.0);  // as in direct64_kernel
        tx[t] = p.x; ty[t] = p.y; tz[t] = p.z;
        odd = odd || odd_point(p);
        self[t] = Op::kSelf && i < coinc_n ? coinc_off + i : -1;
#pragma unroll
        for (int c = 0; c < NC; ++c) s[t][c] = 0.0;
    }
    if ((int)threadIdx.x < n_src) {
        const double4 y = src[threadIdx.x];
        st[threadIdx.x] = y;
        bad = odd_point(y) || odd_strength(y.w);
        if constexpr (Op::kAux) st[kFew + threadIdx.x] = Op::prepare(y);
    }
    const auto state = op.init();
    const bool plain = !__syncthreads_or(bad) && !__any_sync(0xffffffffu, odd);
    op.tile(state, st, st + kFew, n_src, plain, 0, tx, ty, tz, self, s);
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
        const int64_t i = first + t * kThreads64;
        if (i < n_tgt) op.finish(i, s[t], tgt, mult, out, stride);
    }
}

// ------------------------------------------------------------------ FP32 Biot-Savart
// src.w holds 2*strength.  Coincident (target, source) pairs -- a face-centroid target and its
// own source -- can only sit at equal indices (see coinc_* arguments); tiles that may contain one
// run the guarded loop, all others the unguarded one.
template <bool kDelta>
struct BsF32 {
    static constexpr int NC = 3;
    float d2x2;

    template <bool kGuard, int TPT>
    __device__ __forceinline__ void tile(const float4* src, int m, const float (&tx)[TPT], const float (&ty)[TPT],
                                         const float (&tz)[TPT], double (&D)[TPT][NC]) const {
        // Targets go in pairs through packed FMAs (fma.rn.f32x2); each lane rounds as the scalar form
        // d = t - s, rr = fma(dz, dz, fma(dy, dy, dx dx)), f = w / rr, a += f d:  t - s is fma(s, -1, t) and
        // a product is fma(a, b, -0), both exact restatements of the single-rounded operation.
        static_assert(TPT % 2 == 0, "targets are processed in pairs");
        float ax[TPT], ay[TPT], az[TPT];
#pragma unroll
        for (int t = 0; t < TPT; ++t) { ax[t] = 0.f; ay[t] = 0.f; az[t] = 0.f; }
#pragma unroll 32  // 1.3M sources x 1.97M targets: 884 ms by 4, 866 by 8, 859 by 16, 850 by 32 (80 registers in all)
        for (int k = 0; k < m; ++k) {
            const float4 s = src[k];
#pragma unroll
            for (int t = 0; t < TPT; t += 2) {
                float dx0, dx1, dy0, dy1, dz0, dz1, r0, r1, f0, f1;
                fma2p(dx0, dx1, s.x, s.x, -1.0f, tx[t], tx[t + 1]);
                fma2p(dy0, dy1, s.y, s.y, -1.0f, ty[t], ty[t + 1]);
                fma2p(dz0, dz1, s.z, s.z, -1.0f, tz[t], tz[t + 1]);
                fma2v(r0, r1, dx0, dx1, dx0, dx1, -0.0f, -0.0f);
                fma2v(r0, r1, dy0, dy1, dy0, dy1, r0, r1);
                fma2v(r0, r1, dz0, dz1, dz0, dz1, r0, r1);
                if (kDelta) { r0 += d2x2; r1 += d2x2; }
                float i0 = rcp32(r0), i1 = rcp32(r1);
                if (kGuard) {
                    i0 = r0 > 2.0e-13f ? i0 : 0.0f;
                    i1 = r1 > 2.0e-13f ? i1 : 0.0f;
                }
                fma2p(f0, f1, i0, i1, s.w, -0.0f, -0.0f);
                fma2v(ax[t], ax[t + 1], f0, f1, dx0, dx1, ax[t], ax[t + 1]);
                fma2v(ay[t], ay[t + 1], f0, f1, dy0, dy1, ay[t], ay[t + 1]);
                fma2v(az[t], az[t + 1], f0, f1, dz0, dz1, az[t], az[t + 1]);
            }
        }
#pragma unroll
        for (int t = 0; t < TPT; ++t) { D[t][0] += ax[t]; D[t][1] += ay[t]; D[t][2] += az[t]; }
    }
    __device__ __forceinline__ void finish(int64_t i, const double (&D)[NC], const double4* tgt64, double mult,
                                           double* out, int64_t stride) const {
        const double4 p = tgt64[i];
        const double nm = -mult;
        out[i] = nm * (p.y * D[2] - p.z * D[1]);
        out[stride + i] = nm * (p.z * D[0] - p.x * D[2]);
        out[2 * stride + i] = nm * (p.x * D[1] - p.y * D[0]);
    }
};

// ------------------------------------------------------------------ FP32 Poisson
struct PoissonF32 {
    static constexpr int NC = 1;

    template <bool kGuard, int TPT>
    __device__ __forceinline__ void tile(const float4* src, int m, const float (&tx)[TPT], const float (&ty)[TPT],
                                         const float (&tz)[TPT], double (&D)[TPT][NC]) const {
        // targets in pairs through packed FMAs, rounded as the scalar form (see BsF32)
        float acc[TPT];
#pragma unroll
        for (int t = 0; t < TPT; ++t) acc[t] = 0.f;
#pragma unroll 64  // 1.3M sources x 1.97M targets: 629 ms by 4, 613 by 8, 614 by 16, 637 by 32, 592 by 64
        for (int k = 0; k < m; ++k) {
            const float4 s = src[k];
#pragma unroll
            for (int t = 0; t < TPT; t += 2) {
                float dx0, dx1, dy0, dy1, dz0, dz1, r0, r1;
                fma2p(dx0, dx1, s.x, s.x, -1.0f, tx[t], tx[t + 1]);
                fma2p(dy0, dy1, s.y, s.y, -1.0f, ty[t], ty[t + 1]);
                fma2p(dz0, dz1, s.z, s.z, -1.0f, tz[t], tz[t + 1]);
                fma2v(r0, r1, dx0, dx1, dx0, dx1, -0.0f, -0.0f);
                fma2v(r0, r1, dy0, dy1, dy0, dy1, r0, r1);
                fma2v(r0, r1, dz0, dz1, dz0, dz1, r0, r1);
                float i0 = rsqrt32(r0), i1 = rsqrt32(r1);
                if (kGuard) {
                    i0 = r0 > 0.0f ? i0 : 0.0f;
                    i1 = r1 > 0.0f ? i1 : 0.0f;
                }
                fma2p(acc[t], acc[t + 1], i0, i1, s.w, acc[t], acc[t + 1]);
            }
        }
#pragma unroll
        for (int t = 0; t < TPT; ++t) D[t][0] += acc[t];
    }
    __device__ __forceinline__ void finish(int64_t i, const double (&D)[NC], const double4*, double mult, double* out,
                                           int64_t) const {
        out[i] = mult * D[0];
    }
};

// FP32 direct sum, TPT targets per thread (2, 4 or 8: at most the context's "direct_targets").  A tile of kTile sources is
// always summed by one thread per target in FP32 and folded into FP64 once, so the FP32 sums are the same however
// the tiles are shared out: every stage holds one tile per group.
template <class Op, int TPT>
__global__ void __launch_bounds__(kThreads) direct32_kernel(const float4* __restrict__ src, int64_t n_src,
                                                            const float4* __restrict__ tgt,
                                                            const double4* __restrict__ tgt64, int64_t n_tgt, Op op,
                                                            double mult, double* __restrict__ out, int64_t stride,
                                                            int64_t coinc_n, int64_t coinc_off, Split sp) {
    extern __shared__ __align__(16) float4 stages[];  // 2 x groups x kTile sources, later the sums
    const int gw = kThreads >> sp.gshift, groups = 1 << sp.gshift;
    const int grp = (int)threadIdx.x / gw, lt = (int)threadIdx.x - grp * gw;
    const int rank = (int)(blockIdx.x % (unsigned)sp.parts);
    const int64_t blk0 = (int64_t)(blockIdx.x / (unsigned)sp.parts) * (gw * TPT);
    const bool live = blk0 + (lt & ~31) < n_tgt;  // warp-uniform
    float tx[TPT], ty[TPT], tz[TPT];
    double D[TPT][Op::NC];
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
        const int64_t i = blk0 + lt + t * gw;
        const float4 p = i < n_tgt ? tgt[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        tx[t] = p.x; ty[t] = p.y; tz[t] = p.z;
#pragma unroll
        for (int c = 0; c < Op::NC; ++c) D[t][c] = 0.0;
    }
    // source indices that may coincide with this block's targets
    const int64_t c_lo = blk0 < coinc_n ? blk0 + coinc_off : INT64_MAX;
    const int64_t c_hi = blk0 < coinc_n ? min(blk0 + gw * TPT, coinc_n) + coinc_off : INT64_MIN;
    const int64_t tiles = (n_src + kTile - 1) / kTile;
    const int64_t t0 = tiles * rank / sp.parts, t1 = tiles * (rank + 1) / sp.parts;
    auto load = [&](int64_t tile, int buf) {  // tiles tile .. tile + groups - 1 of the part
        for (int g = 0; g < groups; ++g) {
            const int64_t j = (tile + g) * kTile + threadIdx.x;
            if (tile + g < t1 && j < n_src) cp_async16(&stages[(buf * groups + g) * kTile + threadIdx.x], src + j);
        }
    };
    if (t0 < t1) load(t0, 0);
    int buf = 0;
    for (int64_t tile = t0; tile < t1; tile += groups, buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();  // these tiles have landed, and the other buffer's readers are done
        if (tile + groups < t1) load(tile + groups, buf ^ 1);
        if (live && tile + grp < t1) {
            const int64_t j0 = (tile + grp) * kTile;
            const int m = (int)min((int64_t)kTile, n_src - j0);
            const float4* s = &stages[(buf * groups + grp) * kTile];
            if (j0 < c_hi && j0 + m > c_lo)
                op.template tile<true, TPT>(s, m, tx, ty, tz, D);
            else
                op.template tile<false, TPT>(s, m, tx, ty, tz, D);
        }
    }
    if (sp.gshift == 0 && sp.parts == 1) {  // uniform per launch
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
            const int64_t i = blk0 + lt + t * gw;
            if (i < n_tgt) op.finish(i, D[t], tgt64, mult, out, stride);
        }
    } else {
        double* red = (double*)stages;
        __syncthreads();  // the staged sources are read: the sums take their space
#pragma unroll
        for (int t = 0; t < TPT; ++t)
#pragma unroll
            for (int c = 0; c < Op::NC; ++c) red[((grp * TPT + t) * Op::NC + c) * gw + lt] = D[t][c];
        reduce_split<TPT, Op::NC, kThreads>(red, sp, rank, [&](int u, const double (&v)[Op::NC]) {
            if (blk0 + u < n_tgt) op.finish(blk0 + u, v, tgt64, mult, out, stride);
        });
    }
}

__global__ void pack_f32_kernel(const double4* __restrict__ in, int64_t n, float4* __restrict__ out, float wscale) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const double4 p = in[i];
        out[i] = make_float4((float)p.x, (float)p.y, (float)p.z, (float)(p.w * wscale));
    }
}

}  // namespace

int pack_f32(lpm_ctx* ctx, const double4* in, int64_t n, float4* out, bool scale_w2) {
    if (n <= 0) return LPM_OK;
    LPM_LAUNCH(ctx, "pack_f32_kernel", pack_f32_kernel, grid_for(n, 256), 256, 0, in, n, out,
               scale_w2 ? 2.0f : 1.0f);
    return LPM_OK;
}

namespace {
// Splits of a direct sum of n_tgt targets.  FP64: four groups per block at every size (more blocks of fewer targets fill
// the last wave better; 81,920 sources x 122,882 targets took 1.4 times as long with one group and part), and eight parts
// while the blocks alone are fewer than the four resident per SM, two above (1,500 sources x 5,000 targets / 16,000 x 20,000
// 22 / 312 us with eight parts, 31 / 433 with two; 16,000 x 150,000 2.10 ms with eight, 2.02 with two).  A part keeps at least 64 sources (a warp 16), and 256
// where blocks x parts are more than Op::kCrowd per SM: a block's fixed cost (targets, totals, the sums' reduction) then
// outweighs a short run of sources.  75,000 targets, Biot-Savart, 130 / 257 / 700 / 1,000 sources: 16.7 / 27 / 56 / 76 us so
// and 20.8 / 40 / 97 / 111 us with 64 everywhere; the scalar kernels, with fewer targets a block and longer pairs, gain
// from parts up to 16 blocks per SM (Green's function, 40,000 targets, 400 sources: 41 us with two parts, 51 with one) and
// lose beyond (300,000 targets, 130 sources: 107 and 84).
int64_t blocks64(int64_t n_tgt, int tpt) {
    const int64_t tb = (kThreads64 * tpt) >> 2;
    return (n_tgt + tb - 1) / tb;
}
Split split64(int sms, int64_t blocks, int64_t n_src, int crowd) {
    int parts = blocks < 4 * (int64_t)sms ? 8 : 2;
    while (parts > 1 && n_src < (int64_t)parts * (blocks * parts > crowd * (int64_t)sms ? 256 : 64)) parts /= 2;
    return Split{2, parts};
}

// Whether a sum goes to direct64_few_kernel, which has a quarter of direct64_kernel's blocks: by targets per SM.  1 / 8 / 30
// / 128 sources by either (Biot-Savart, us): 75,000 targets 5.0 / 5.1 / 9.0 / 20.8 against 6.0 / 6.5 / 8.5 / 16.7, 150,000
// 5.5 / 5.9 / 10.5 / 24.9 against 9.0 / 10.5 / 12.7 / 25.3, 1M 10.5 / 18.8 / 35.2 / 119 against 41 / 47 / 62 / 135.
bool few_sources(int sms, int64_t n_tgt, int64_t n_src) {
    return n_src <= kFew && n_tgt >= sms * std::min<int64_t>(1000, 100 + 40 * n_src);
}

// FP32: the estimated time of `rounds` of stages (one tile per group) at the blocks each SM holds, in units fitted to
// 640 ... 327,680 sources (a round takes 19 / 30 / 55 us with 1 / 2 / 4 blocks of 256 x 4 targets on the SM); clusters
// of four and eight blocks lose 15% and 30% where the blocks are many times the resident ones.  Few tiles on many
// targets share out badly: groups that have none hold their block's place on the SM while the others work, so there fewer
// groups count too, a round of the last tile alone as long as that tile is, and a round's time by how full its groups
// are.  Biot-Savart, 257 / 700 / 1,100 / 1,300 sources x 1M targets 134 / 292 / 504 / 599 us with four groups and two parts
// from three and five tiles on, 112 / 274 / 416 / 495 so; 1,000 sources (four tiles) 368 us with four groups, 383 with one.
struct Split32 {
    int tpt;
    Split split;
};
Split32 split32(int sms, int64_t n_tgt, int64_t n_src, int max_tpt) {
    const int64_t tiles = std::max<int64_t>(1, (n_src + kTile - 1) / kTile);
    const double last = (double)(n_src - (tiles - 1) * kTile) / kTile;
    const bool uneven = tiles <= 8 && n_tgt >= 1000 * (int64_t)sms;
    const int most = tiles >= 3 ? 2 : (tiles == 2 ? 1 : 0);
    Split32 best{max_tpt, Split{most, 1}};
    double best_cost = 0.0;
    for (int tpt = max_tpt; tpt >= 2; tpt /= 2)
        for (int gs = most; gs >= (uneven ? 0 : most); --gs)
            for (int parts = 1; parts <= 8 && parts <= tiles; parts *= 2) {
                const int64_t per_part = (tiles + parts - 1) / parts, tb = (kThreads * tpt) >> gs;
                const int64_t blocks = (n_tgt + tb - 1) / tb * parts;
                if (tpt < max_tpt && blocks > 2 * (int64_t)sms) break;  // fewer targets per thread read more per pair
                double rounds = (double)((per_part + (1 << gs) - 1) >> gs), fill = 1.0;
                if (uneven && parts == 1) {
                    if (((tiles - 1) & ((1 << gs) - 1)) == 0) rounds += last - 1.0;
                    fill = (double)n_src / std::max(1.0, rounds * (kTile << gs));
                }
                const double loss = blocks > 4 * (int64_t)sms && parts > 2 ? (parts == 8 ? 1.3 : 1.15) : 1.0;
                const double cost = loss * rounds * tpt *
                                    (7.0 + (3.0 + 9.0 * fill) * std::ceil((double)blocks / std::max(sms, 1)));
                if ((tpt == max_tpt && gs == most && parts == 1) || cost < 0.985 * best_cost) {
                    best = Split32{tpt, Split{gs, parts}};
                    best_cost = cost;
                }
            }
    return best;
}

// Whether the vector and 1/r kernels take two targets per thread instead of four: while four leave less than two
// blocks to an SM even in eight parts (1,280 sources x 1,922 targets: 12.4 against 16.5 us; 5,120 x 7,682: 60.0
// against 57.5 us).
bool few_targets(const lpm_ctx* ctx, int64_t n_tgt) { return blocks64(n_tgt, 4) * 8 < 2 * (int64_t)ctx->num_sms; }

template <class Op>
int launch64(lpm_ctx* ctx, const char* name, Op op, const double4* src, int64_t n_src, const double4* tgt,
             int64_t n_tgt, double mult, double* out, int64_t stride, int64_t coinc_n, int64_t coinc_off) {
    if (few_sources(ctx->num_sms, n_tgt, n_src)) {
        LPM_LAUNCH(ctx, name, direct64_few_kernel<Op>, grid_for(n_tgt, kThreads64 * Op::TPT), kThreads64, 0, src, (int)n_src,
                   tgt, n_tgt, op, mult, out, stride, coinc_n, coinc_off);
        return LPM_OK;
    }
    const int64_t blocks = blocks64(n_tgt, Op::TPT);
    const Split sp = split64(ctx->num_sms, blocks, n_src, Op::kCrowd);
    const size_t smem = Shape64<Op>::kSmem;
    static_assert(Shape64<Op>::kSmem <= 48 * 1024, "no opt-in needed");
    return launch_cluster(ctx, name, direct64_kernel<Op>, (unsigned)(blocks * sp.parts), kThreads64, smem, sp.parts, src,
                          n_src, tgt, n_tgt, op, mult, out, stride, coinc_n, coinc_off, sp);
}

template <class Op, int TPT>
int launch32(lpm_ctx* ctx, const char* name, Op op, const float4* src, int64_t n_src, const float4* tgt,
             const double4* tgt64, int64_t n_tgt, double mult, double* out, int64_t stride, int64_t coinc_n,
             int64_t coinc_off, Split sp) {
    const int64_t tb = (kThreads * TPT) >> sp.gshift;
    const size_t smem = std::max(2 * sizeof(float4) * (kTile << sp.gshift), sizeof(double) * kThreads * TPT * Op::NC);
    return launch_cluster(ctx, name, direct32_kernel<Op, TPT>, (unsigned)((n_tgt + tb - 1) / tb * sp.parts), kThreads, smem,
                          sp.parts, src, n_src, tgt, tgt64, n_tgt, op, mult, out, stride, coinc_n, coinc_off, sp);
}
}  // namespace

// The high word of 2^-10 R^2, but at least the kernels' zero tolerance: a smaller R^2 - x.y (+ delta^2) takes the
// reference's rounding.
static int small_den(double radius) {
    uint64_t bits = 0;
    const double close = std::max(radius * radius * 0x1p-10, 2.0 * kZeroTol);
    std::memcpy(&bits, &close, sizeof(bits));
    return (int)std::min((unsigned)(bits >> 32), 0x7ff00000u);
}

int direct_sum_f64(lpm_ctx* ctx, const lpm_kernel_desc& k, const double4* src, int64_t n_src, const double4* tgt,
                   int64_t n_tgt, double* out, int64_t out_stride, int64_t coinc_n, int64_t coinc_off) {
    if (n_tgt <= 0) return LPM_OK;
    if (k.kind == LPM_KERNEL_BIOT_SAVART_SPHERE) {
        const double mult = -1.0 / (4.0 * kPi * k.radius);
        const double r2 = k.radius * k.radius, d2 = k.delta * k.delta;
        const int lo = small_den(k.radius);
        const bool few = few_targets(ctx, n_tgt);
        auto run = [&](auto op) {
            return launch64(ctx, "bs_f64_kernel", op, src, n_src, tgt, n_tgt, mult, out, out_stride, 0, 0);
        };
        if (k.delta != 0.0)
            return few ? run(BsF64<true, 2>{r2, d2, r2 + d2, lo}) : run(BsF64<true, 4>{r2, d2, r2 + d2, lo});
        return few ? run(BsF64<false, 2>{r2, d2, r2, lo}) : run(BsF64<false, 4>{r2, d2, r2, lo});
    }
    if (k.kind == LPM_KERNEL_POISSON_3D) {
        auto run = [&](auto op) {
            return launch64(ctx, "poisson_f64_kernel", op, src, n_src, tgt, n_tgt, 1.0 / (4.0 * kPi), out, out_stride,
                            0, 0);
        };
        return few_targets(ctx, n_tgt) ? run(PoissonF64<2>{}) : run(PoissonF64<4>{});
    }
    if (k.kind == LPM_KERNEL_SPHERE_GREENS)
        return launch64(ctx, "scalar_f64_kernel", LogF64<SphereGreensArg>{{k.radius * k.radius, small_den(k.radius)}}, src,
                        n_src, tgt, n_tgt, -1.0 / (4.0 * kPi * k.radius), out, out_stride, coinc_n, coinc_off);
    if (k.kind == LPM_KERNEL_PLANAR_LOG)
        return launch64(ctx, "scalar_f64_kernel", LogF64<PlanarLogArg>{{0x00100000}}, src, n_src, tgt, n_tgt,
                        1.0 / (4.0 * kPi), out, out_stride, coinc_n, coinc_off);
    if (k.kind == LPM_KERNEL_DELTA_3D)
        return launch64(ctx, "scalar_f64_kernel", ScalarF64<Delta3dPair>{{1.0 / k.delta}}, src, n_src, tgt,
                        n_tgt, 3.0 / (4.0 * kPi * (k.delta * k.delta * k.delta)), out, out_stride, 0, 0);
    if (k.kind == LPM_KERNEL_SPHERE_DELTA)
        return launch64(ctx, "scalar_f64_kernel", ScalarF64<SphereDeltaPair>{{k.delta * k.delta}}, src, n_src,
                        tgt, n_tgt, 1.0 / (4.0 * kPi), out, out_stride, 0, 0);
    set_error("invalid kernel");
    return LPM_ERR_KERNEL;
}

// FP32 sums take FP32 copies of sources (w pre-scaled by 2 for Biot-Savart) and targets, plus the
// FP64 targets for the Biot-Savart epilogue.  Targets 0..coinc_n-1 may coincide with sources
// coinc_off..coinc_off+coinc_n-1 (face-centroid targets and their own sources).
template <int TPT>
static int direct_sum_f32_tpt(lpm_ctx* ctx, const lpm_kernel_desc& k, const float4* src, int64_t n_src,
                              const float4* tgt, const double4* tgt64, int64_t n_tgt, double* out, int64_t out_stride,
                              int64_t coinc_n, int64_t coinc_off, Split sp) {
    if (k.kind == LPM_KERNEL_BIOT_SAVART_SPHERE) {
        const double mult = -1.0 / (4.0 * kPi * k.radius);
        if (k.delta != 0.0)
            return launch32<BsF32<true>, TPT>(ctx, "bs_f32_kernel", BsF32<true>{(float)(2.0 * k.delta * k.delta)}, src,
                                              n_src, tgt, tgt64, n_tgt, mult, out, out_stride, coinc_n, coinc_off,
                                              sp);
        return launch32<BsF32<false>, TPT>(ctx, "bs_f32_kernel", BsF32<false>{0.0f}, src, n_src, tgt, tgt64, n_tgt,
                                           mult, out, out_stride, coinc_n, coinc_off, sp);
    }
    if (k.kind == LPM_KERNEL_POISSON_3D)
        return launch32<PoissonF32, TPT>(ctx, "poisson_f32_kernel", PoissonF32{}, src, n_src, tgt, tgt64, n_tgt,
                                         1.0 / (4.0 * kPi), out, out_stride, coinc_n, coinc_off, sp);
    set_error("invalid kernel");
    return LPM_ERR_KERNEL;
}

int direct_sum_f32_impl(lpm_ctx* ctx, const lpm_kernel_desc& k, const float4* src, int64_t n_src, const float4* tgt,
                        const double4* tgt64, int64_t n_tgt, double* out, int64_t out_stride, int64_t coinc_n,
                        int64_t coinc_off) {
    if (n_tgt <= 0) return LPM_OK;
    // the context's "direct_targets" is the most targets per thread; a sum that would leave SMs idle takes fewer
    // (every target's FP32 sums are the same: its tiles are summed by one thread whatever the count)
    const Split32 c = split32(ctx->num_sms, n_tgt, n_src, ctx->direct_tpt);
    switch (c.tpt) {
        case 2:
            return direct_sum_f32_tpt<2>(ctx, k, src, n_src, tgt, tgt64, n_tgt, out, out_stride, coinc_n, coinc_off,
                                         c.split);
        case 8:
            return direct_sum_f32_tpt<8>(ctx, k, src, n_src, tgt, tgt64, n_tgt, out, out_stride, coinc_n, coinc_off,
                                         c.split);
        default:
            return direct_sum_f32_tpt<4>(ctx, k, src, n_src, tgt, tgt64, n_tgt, out, out_stride, coinc_n, coinc_off,
                                         c.split);
    }
}

int check_kernel_desc(const lpm_kernel_desc* k) {
    if (!k) {
        set_error("null kernel descriptor");
        return LPM_ERR_ARG;
    }
    if (k->kind < LPM_KERNEL_BIOT_SAVART_SPHERE || k->kind > LPM_KERNEL_SPHERE_DELTA) {
        set_error("invalid kernel");
        return LPM_ERR_KERNEL;
    }
    if ((k->kind == LPM_KERNEL_BIOT_SAVART_SPHERE || k->kind == LPM_KERNEL_SPHERE_GREENS) && !(k->radius > 0.0)) {
        set_error("sphere kernels need radius > 0");
        return LPM_ERR_ARG;
    }
    if ((k->kind == LPM_KERNEL_DELTA_3D || k->kind == LPM_KERNEL_SPHERE_DELTA) && !(k->delta > 0.0)) {
        set_error("delta kernels need eps (the delta field) > 0");
        return LPM_ERR_ARG;
    }
    return LPM_OK;
}

// The FP32 direct sums exist for the Biot-Savart and 3D Poisson kernels only; every FP32 entry point checks
// this before it launches anything.
int check_f32_kind(const lpm_kernel_desc& k) {
    if (k.kind != LPM_KERNEL_BIOT_SAVART_SPHERE && k.kind != LPM_KERNEL_POISSON_3D) {
        set_error("invalid kernel: the FP32 direct sum takes the Biot-Savart and 3D Poisson kernels (use LPM_PREC_F64)");
        return LPM_ERR_KERNEL;
    }
    return LPM_OK;
}

// Device entry shared by the C ABI: FP64 or FP32 (FP32 copies go to scratch slots).
int direct_sum_any(lpm_ctx* ctx, const lpm_kernel_desc& k, int precision, const double4* src, int64_t n_src,
                   const double4* tgt, int64_t n_tgt, double* out, int64_t coinc_n, int64_t coinc_off) {
    if (precision == LPM_PREC_F64) return direct_sum_f64(ctx, k, src, n_src, tgt, n_tgt, out, n_tgt, coinc_n, coinc_off);
    if (precision != LPM_PREC_F32) {
        set_error("unknown precision %d", precision);
        return LPM_ERR_ARG;
    }
    int rc = check_f32_kind(k);
    if (rc) return rc;
    float4* s32 = (float4*)scratch(ctx, kSlotSrc32, sizeof(float4) * (size_t)std::max<int64_t>(n_src, 1));
    float4* t32 = (float4*)scratch(ctx, kSlotTgt32, sizeof(float4) * (size_t)std::max<int64_t>(n_tgt, 1));
    if (!s32 || !t32) return LPM_ERR_OOM;
    rc = pack_f32(ctx, src, n_src, s32, k.kind == LPM_KERNEL_BIOT_SAVART_SPHERE);
    if (rc) return rc;
    rc = pack_f32(ctx, tgt, n_tgt, t32, false);
    if (rc) return rc;
    return direct_sum_f32_impl(ctx, k, s32, n_src, t32, tgt, n_tgt, out, n_tgt, coinc_n, coinc_off);
}

}  // namespace lpm

using namespace lpm;

extern "C" int lpm_direct_sum_dev(lpm_ctx* ctx, const lpm_kernel_desc* kernel, int precision, const double* src,
                                  int64_t n_src, const double* tgt, int64_t n_tgt, int64_t n_coincident,
                                  double* out) {
    if (!ctx) {
        set_error("null context");
        return LPM_ERR_ARG;
    }
    int rc = check_kernel_desc(kernel);
    if (rc) return rc;
    if (n_src < 0 || n_tgt < 0 || (n_src > 0 && !src) || (n_tgt > 0 && (!tgt || !out)) || n_coincident < 0 ||
        n_coincident > std::min(n_src, n_tgt)) {
        set_error("lpm_direct_sum_dev: bad sizes or null pointers");
        return LPM_ERR_ARG;
    }
    LPM_CUDA_TRY(cudaSetDevice(ctx->device));
    return direct_sum_any(ctx, *kernel, precision, (const double4*)src, n_src, (const double4*)tgt, n_tgt, out,
                          n_coincident, 0);
}

extern "C" int lpm_direct_sum_mesh(lpm_ctx* ctx, const lpm_kernel_desc* kernel, int precision, int64_t n_verts,
                                   const double* vx, const double* vy, const double* vz, int64_t n_faces,
                                   const double* fx, const double* fy, const double* fz, const double* face_area,
                                   const uint8_t* face_divided, const double* face_src, int64_t vert_begin,
                                   int64_t vert_end, int64_t face_begin, int64_t face_end, double* vert_out0,
                                   double* vert_out1, double* vert_out2, double* face_out0, double* face_out1,
                                   double* face_out2) {
    if (!ctx) {
        set_error("null context");
        return LPM_ERR_ARG;
    }
    int rc = check_kernel_desc(kernel);
    if (rc) return rc;
    const bool vec = kernel->kind == LPM_KERNEL_BIOT_SAVART_SPHERE;
    const int comps = vec ? 3 : 1;
    if (n_verts < 0 || n_faces < 0 || (n_verts > 0 && (!vx || !vy || !vz)) ||
        (n_faces > 0 && (!fx || !fy || !fz || !face_area || !face_divided || !face_src))) {
        set_error("lpm_direct_sum_mesh: null input arrays");
        return LPM_ERR_ARG;
    }
    // empty ranges (end < begin) are allowed, as for a rank with no items
    const bool do_v = vert_end >= vert_begin, do_f = face_end >= face_begin;
    if ((do_v && (vert_begin < 0 || vert_end >= n_verts || !vert_out0 || (vec && (!vert_out1 || !vert_out2)))) ||
        (do_f && (face_begin < 0 || face_end >= n_faces || !face_out0 || (vec && (!face_out1 || !face_out2))))) {
        set_error("lpm_direct_sum_mesh: target range out of bounds or null outputs");
        return LPM_ERR_ARG;
    }
    LPM_CUDA_TRY(cudaSetDevice(ctx->device));
    // sources: undivided faces in index order; face targets: undivided faces in [face_begin, face_end]
    int64_t n_src = 0, src_before_fb = 0, n_ft = 0;
    for (int64_t i = 0; i < n_faces; ++i) {
        if (!face_divided[i]) {
            if (i < face_begin) ++src_before_fb;
            if (do_f && i >= face_begin && i <= face_end) ++n_ft;
            ++n_src;
        }
    }
    const int64_t n_vt = do_v ? vert_end - vert_begin + 1 : 0;
    const int64_t n_tgt = n_ft + n_vt;
    const size_t in_bytes = sizeof(double4) * (size_t)(n_src + n_tgt);
    const size_t out_bytes = sizeof(double) * comps * (size_t)n_tgt;
    double* host = (double*)pinned(ctx, in_bytes + out_bytes);
    if (!host) return LPM_ERR_OOM;
    double4* hsrc = (double4*)host;
    double4* htgt = hsrc + n_src;
    double* hout = (double*)(htgt + n_tgt);
    int64_t s = 0, t = 0;
    for (int64_t i = 0; i < n_faces; ++i) {
        if (face_divided[i]) continue;
        hsrc[s++] = make_double4(fx[i], fy[i], fz[i], face_src[i] * face_area[i]);
        if (do_f && i >= face_begin && i <= face_end) htgt[t++] = make_double4(fx[i], fy[i], fz[i], 0.0);
    }
    for (int64_t i = 0; i < n_vt; ++i) {
        const int64_t v = vert_begin + i;
        htgt[t++] = make_double4(vx[v], vy[v], vz[v], 0.0);
    }
    double4* dsrc = (double4*)scratch(ctx, kSlotSrcPack, sizeof(double4) * (size_t)std::max<int64_t>(n_src, 1));
    double4* dtgt = (double4*)scratch(ctx, kSlotTgtPack, sizeof(double4) * (size_t)std::max<int64_t>(n_tgt, 1));
    double* dout = (double*)scratch(ctx, kSlotOut, std::max<size_t>(out_bytes, 8));
    if (!dsrc || !dtgt || !dout) return LPM_ERR_OOM;
    if (n_tgt > 0) {
        if (n_src > 0)
            LPM_CUDA_TRY(cudaMemcpyAsync(dsrc, hsrc, sizeof(double4) * (size_t)n_src, cudaMemcpyHostToDevice,
                                         ctx->stream));
        LPM_CUDA_TRY(cudaMemcpyAsync(dtgt, htgt, sizeof(double4) * (size_t)n_tgt, cudaMemcpyHostToDevice, ctx->stream));
        // face targets come first and sit on sources src_before_fb.. in order: the self pairs a singular
        // scalar kernel skips (the FP32 paths use the same indices to guard coincident pairs)
        rc = direct_sum_any(ctx, *kernel, precision, dsrc, n_src, dtgt, n_tgt, dout, n_ft, src_before_fb);
        if (rc) return rc;
        LPM_CUDA_TRY(cudaMemcpyAsync(hout, dout, out_bytes, cudaMemcpyDeviceToHost, ctx->stream));
        LPM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    }
    t = 0;
    for (int64_t i = face_begin; do_f && i <= face_end; ++i) {
        if (face_divided[i]) continue;
        face_out0[i] = hout[t];
        if (vec) {
            face_out1[i] = hout[n_tgt + t];
            face_out2[i] = hout[2 * n_tgt + t];
        }
        ++t;
    }
    for (int64_t i = 0; i < n_vt; ++i, ++t) {
        vert_out0[vert_begin + i] = hout[t];
        if (vec) {
            vert_out1[vert_begin + i] = hout[n_tgt + t];
            vert_out2[vert_begin + i] = hout[2 * n_tgt + t];
        }
    }
    return LPM_OK;
}

extern "C" int lpm_direct_sum_meshfree(lpm_ctx* ctx, const lpm_kernel_desc* kernel, int precision, int64_t n,
                                       const double* x, const double* y, const double* z, const double* src,
                                       const double* weights, int64_t begin, int64_t end, double* out) {
    if (!ctx) {
        set_error("null context");
        return LPM_ERR_ARG;
    }
    int rc = check_kernel_desc(kernel);
    if (rc) return rc;
    if (kernel->kind == LPM_KERNEL_BIOT_SAVART_SPHERE) {
        set_error("invalid kernel: lpm_direct_sum_meshfree takes a scalar kernel");
        return LPM_ERR_KERNEL;
    }
    if (n < 0 || (n > 0 && (!x || !y || !z || !src))) {
        set_error("lpm_direct_sum_meshfree: null input arrays");
        return LPM_ERR_ARG;
    }
    const bool any = end >= begin;
    if (any && (begin < 0 || end >= n || !out)) {
        set_error("lpm_direct_sum_meshfree: target range out of bounds");
        return LPM_ERR_ARG;
    }
    if (!any || n == 0) return LPM_OK;
    LPM_CUDA_TRY(cudaSetDevice(ctx->device));
    const int64_t n_tgt = end - begin + 1;
    const size_t in_bytes = sizeof(double4) * (size_t)n;
    const size_t out_bytes = sizeof(double) * (size_t)n_tgt;
    double* host = (double*)pinned(ctx, in_bytes + out_bytes);
    if (!host) return LPM_ERR_OOM;
    double4* hsrc = (double4*)host;
    double* hout = (double*)(hsrc + n);
    for (int64_t i = 0; i < n; ++i)
        hsrc[i] = make_double4(x[i], y[i], z[i], weights ? src[i] * weights[i] : src[i]);
    double4* dsrc = (double4*)scratch(ctx, kSlotSrcPack, in_bytes);
    double* dout = (double*)scratch(ctx, kSlotOut, out_bytes);
    if (!dsrc || !dout) return LPM_ERR_OOM;
    LPM_CUDA_TRY(cudaMemcpyAsync(dsrc, hsrc, in_bytes, cudaMemcpyHostToDevice, ctx->stream));
    rc = direct_sum_any(ctx, *kernel, precision, dsrc, n, dsrc + begin, n_tgt, dout, n_tgt, begin);
    if (rc) return rc;
    LPM_CUDA_TRY(cudaMemcpyAsync(hout, dout, out_bytes, cudaMemcpyDeviceToHost, ctx->stream));
    LPM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    for (int64_t i = 0; i < n_tgt; ++i) out[begin + i] = hout[i];
    return LPM_OK;
}

// A cell's mass and momentum as exact 64-bit fixed point (units of 2^-61),
// for the diagnostics.  The float64 pipe issues 1.67 operations per clock
// per SM against ~64 on the integer pipes, so moments formed and summed in
// float64 bound every diagnostic; formed in integers they leave it idle.
//
//   float64 storage   the 27 values converted exactly (fx_math.cuh) and
//                     summed exactly.
//   reduced precision the deviations h = kScale (f - w) summed in float32,
//                     pair by pair as the collision sums them (or, EXACT,
//                     the stored values exactly); mass = 1 +
//                     sum h, momentum = sum h e.  The float32 sums are
//                     multiples of 2^-37 or more for stored values of the
//                     weights' size, so their conversion drops nothing.
//
// Outside the range `ok` is false and the caller uses moments_f64_of.  In the
// range are: float64 values in [2^-9, 1) for f_0 and [2^-9, 1/8) for the others
// with 3p < 2; float32 sums below 1 in magnitude (sum h, and each of sum h e);
// EXACT, stored values (or deviations, in units of f) below 1/2 and 1/8 in
// magnitude, whose sums may reach 3.75 (3p) and 2.25 (u, v, w).
#pragma once

#include "fx_math.cuh"
#include "imexlbm.h"
#include "kernels_common.cuh"
#include "lowp_math.cuh"

namespace imex {
namespace mom {

constexpr int kBits = fx::kFrac;  // 61
static_assert(kBits == 61, "the shifts below assume units of 2^-61");

template <int P>
struct Elem {
    using T = typename lowp::Storage<P>::T;
    static constexpr int kScaleLog2 = P == IMEX_F16DEV ? 12 : 0;
    static_assert(lowp::Storage<P>::kScale == (float)(1 << kScaleLog2), "kScale is 2^kScaleLog2");
};
template <>
struct Elem<IMEX_F64> {
    using T = double;
};

// x / 2^S in units of 2^-61, bits below dropped; clears ok for |x| >= 2^(S -
// LIM) (NaN and Inf included).
template <int S, int LIM = 0>
__device__ __forceinline__ int64_t fixed_of_float(float x, bool& ok)
{
    const uint32_t b = __float_as_uint(x);
    const int e = (int)((b >> 23) & 255u);
    ok = ok && e <= 126 + S - LIM;
    // mantissa * 2^(e - 150) * 2^61 / 2^S = (mantissa << 37) >> (126 + S - e)
    const int sh = 126 + S - e;
    const uint64_t v = ((uint64_t)((b & 0x007FFFFFu) | 0x00800000u) << 37) >> (sh < 63 ? sh : 63);
    return (b >> 31) ? -(int64_t)v : (int64_t)v;
}

// One cell: M = {3p, u, v, w} 2^61 and u, v, w again as numbers in units of
// 2^-kVelBits<P> (vel), the form whose squares make the kinetic energy.
template <int P>
struct Cell {
    int64_t M[4];
    double vel[3];
};
template <int P>
inline constexpr int kVelBits = P == IMEX_F64 ? kBits : P == IMEX_F16DEV ? 12 : 0;

// Sum of the 27 weights.
__device__ __forceinline__ constexpr uint64_t weights_fixed()
{
    uint64_t w = 0;
    for (int a = 0; a < kQ; ++a) w += lowp::weight_fixed(a);
    return w;
}

// EXACT (reduced precision): the stored values summed exactly instead of in
// float32; the velocities in units of 2^-61.
template <int P, bool EXACT>
__device__ __forceinline__ bool moments(const typename Elem<P>::T* src, const Geom& g, const PullIndex& pi,
                                        Cell<P>& c)
{
    bool ok = true;
    if constexpr (P == IMEX_F64) {
        double f[kQ];
        gather27<double>(src, g, pi, f);
        uint64_t S = 0, A[3] = {0, 0, 0}, B[3] = {0, 0, 0};
#pragma unroll
        for (int a = 0; a < kQ; ++a) {  // f_0 < 1, others < 1/8: every sum below 2^64
            const uint64_t X = fx::to_fixed(f[a], a == 0 ? 8u : 5u, ok);
            S += X;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (ex(a, d) == 1) A[d] += X;
                if (ex(a, d) == -1) B[d] += X;
            }
        }
        ok = ok && (S >> 62) == 0;
        c.M[0] = (int64_t)S;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            c.M[1 + d] = (int64_t)(A[d] - B[d]);
            c.vel[d] = __ll2double_rn(c.M[1 + d]);
        }
    } else if constexpr (EXACT) {
        // float32: f itself; float16: the deviations, the weights added after
        int64_t S = 0, U[3] = {0, 0, 0};
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
            const auto v = load_state(src + pi.at_dyn(g, a));
            constexpr int S2 = P == IMEX_F32 ? 0 : Elem<P>::kScaleLog2;
            float x;
            if constexpr (P == IMEX_F32) x = v;
            else x = __half2float(v);
            // below 1/2 (rest) and 1/8: every sum below 2^63
            const int64_t X = a == 0 ? fixed_of_float<S2, 1>(x, ok) : fixed_of_float<S2, 3>(x, ok);
            S += X;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (ex(a, d) == 1) U[d] += X;
                if (ex(a, d) == -1) U[d] -= X;
            }
        }
        if constexpr (P == IMEX_F16DEV) {
            ok = ok && S < (int64_t)3 << 61;  // the weights' 2^61 more stays below 2^63
            S += (int64_t)weights_fixed();
        }
        c.M[0] = S;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            c.M[1 + d] = U[d];
            c.vel[d] = __ll2double_rn(U[d]);
        }
    } else {
        using A = lowp::F1;
        constexpr int S = Elem<P>::kScaleLog2;
        float h[kQ];
#pragma unroll
        for (int a = 0; a < kQ; ++a) h[a] = lowp::Storage<P>::dev(load_state(src + pi.at_dyn(g, a)), a);
        float d[kPairs + 1], sig = h[0];
#pragma unroll
        for (int q = 1; q <= kPairs; ++q) {
            d[q] = A::sub(h[2 * q - 1], h[2 * q]);
            sig = A::add(sig, A::add(h[2 * q - 1], h[2 * q]));
        }
        c.M[0] = (int64_t)(1ull << kBits) + fixed_of_float<S>(sig, ok);
#pragma unroll
        for (int dim = 0; dim < 3; ++dim) {
            float u = 0.f;
#pragma unroll
            for (int q = 1; q <= kPairs; ++q) {
                const int e = ex(2 * q - 1, dim);
                if (e == 1) u = A::add(u, d[q]);
                if (e == -1) u = A::sub(u, d[q]);
            }
            c.M[1 + dim] = fixed_of_float<S>(u, ok);
            c.vel[dim] = (double)u;
        }
    }
    return ok;
}

// The same moments in float64, for a cell outside the range; out[0] only if MASS.
template <int P, bool MASS = true>
__device__ __noinline__ void moments_f64_of(const typename Elem<P>::T* src, Geom g, int i, int j, int k, bool pull,
                                            double* out)
{
    const PullIndex pi(g, i, j, k, pull);
    for (int q = 0; q < 4; ++q) out[q] = 0.0;
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
        double f;
        const auto v = load_state(src + pi.at_dyn(g, a));
        if constexpr (P == IMEX_F64) f = v;
        else f = lowp::Storage<P>::to_f64(v, a);
        if (MASS) out[0] += f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (ex(a, d) == 1) out[1 + d] += f;
            if (ex(a, d) == -1) out[1 + d] -= f;
        }
    }
}

// Reduced precision again with a wider range: the exact sums of the values (float16: of
// the deviations, without the weights' part of 3p) in units of 2^-(61 - kWide), for densities up
// to several thousand.  ok: every value is below 2^(kWide - 1) (rest) or
// 2^(kWide - 3) in magnitude and a multiple of the unit (a float16 / 2^12 always is).
constexpr int kWide = 12;
struct WideMoments {
    int64_t M[4];
    bool ok;
};
template <int S, int LIM>
__device__ __forceinline__ int64_t exact_of_float(float x, bool& ok)
{
    const uint32_t b = __float_as_uint(x), mant = (b & 0x007FFFFFu) | 0x00800000u;
    const int over = 89 + S - (int)((b >> 23) & 255u);  // bits of the mantissa below the unit
    ok = ok && (over <= 0 || (b << 1) == 0 || (over < 24 && (mant & ((1u << over) - 1u)) == 0));
    return fixed_of_float<S, LIM>(x, ok);
}
template <int P>
__device__ __forceinline__ WideMoments moments_wide(const typename Elem<P>::T* src, Geom g, int i, int j, int k, bool pull)
{
    constexpr int S = Elem<P>::kScaleLog2 + kWide;
    const PullIndex pi(g, i, j, k, pull);
    WideMoments w = {{0, 0, 0, 0}, true};
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
        float x;
        if constexpr (P == IMEX_F32) x = load_state(src + pi.at_dyn(g, a));
        else x = __half2float(load_state(src + pi.at_dyn(g, a)));
        int64_t X;
        if constexpr (P == IMEX_F32) X = a == 0 ? exact_of_float<S, 1>(x, w.ok) : exact_of_float<S, 3>(x, w.ok);
        else X = a == 0 ? fixed_of_float<S, 1>(x, w.ok) : fixed_of_float<S, 3>(x, w.ok);
        w.M[0] += X;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (ex(a, d) == 1) w.M[1 + d] += X;
            if (ex(a, d) == -1) w.M[1 + d] -= X;
        }
    }
    return w;
}

// (x, y, z) of a flat cell index (z fastest); lattices in device memory
// hold fewer than 2^32 cells.
__device__ __forceinline__ void cell_of(const Geom& g, unsigned idx, int& i, int& j, int& k)
{
    const unsigned row = idx / (unsigned)g.nz;
    k = (int)(idx - row * (unsigned)g.nz);
    i = (int)(row / (unsigned)g.ny);
    j = (int)(row - (unsigned)i * (unsigned)g.ny);
}

}  // namespace mom
}  // namespace imex

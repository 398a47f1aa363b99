// Taylor-Green initial field and its equilibrium distributions for one cell,
// src/lbm.cpp:78-108.  The trigonometric factors depend on one coordinate
// each and come in as per-axis tables t[3 i + {0, 1, 2}] = sin, cos, cos 2x
// of x = (double)i / (double)n * 2.0 * 3.1415926, computed on the host with
// that expression.  Products and sums use round-to-nearest intrinsics in the
// reference's order, so no FMA contraction changes its rounding.
//
// Bound: the float64 pipe (1.67 operations per clock per SM), not memory.
// The 27 populations written out one by one take ~300 float64 operations;
// they hold only 18 different values.  w = 0, so e.u depends on (ex, ey)
// alone: 0, +-u, +-v, +-(u + v), +-(u - v), and adding ez w = +-0 changes no
// bit of 3p + 3 e.u.  Negation is exact, so the two members of +-e.u share
// 3 e.u and 4.5 (e.u)^2, and one bracket serves the ez = 0 direction (its
// weight) and the ez = +-1 pair (theirs): 70 operations, the same bits.
// imex_initialize at 256^3: float64 8.21 -> 2.38 ms, float32 8.94 -> 2.37,
// float16 deviations 10.65 -> 2.37 (memory alone would take 0.54 / 0.27 / 0.14).
#pragma once

#include "d3q27.cuh"

namespace imex {

// What does not depend on the cell, formed on the host (the same roundings;
// 2.50 -> 2.38 ms).
struct TgParams {
    double u0, amp, p0;  // rho0 u0^2 / 16, rho0 / 3
};
inline TgParams tg_params(double rho0, double u0) { return TgParams{u0, rho0 * u0 * u0 / 16.0, rho0 * (1.0 / 3.0)}; }

__device__ __forceinline__ void tg_init_cell(double (&fe)[kQ], const double* __restrict__ tx,
                                             const double* __restrict__ ty, const double* __restrict__ tz, int i,
                                             int j, int k, const TgParams& tg)
{
    const double sx = tx[3 * i], cx = tx[3 * i + 1], c2x = tx[3 * i + 2];
    const double sy = ty[3 * j], cy = ty[3 * j + 1], c2y = ty[3 * j + 2];
    const double cz = tz[3 * k + 1], c2z = tz[3 * k + 2];
    const double u = __dmul_rn(__dmul_rn(__dmul_rn(tg.u0, sx), cy), cz);
    const double v = __dmul_rn(__dmul_rn(__dmul_rn(-tg.u0, cx), sy), cz);
    const double p = __dadd_rn(tg.p0, __dmul_rn(__dmul_rn(tg.amp, __dadd_rn(c2x, c2y)), __dadd_rn(c2z, 2.0)));
    const double udu = __dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v));
    const double p3 = __dmul_rn(3.0, p), u15 = __dmul_rn(1.5, udu);
    // e.u by (|ex|, |ey|) and the relative sign of ex and ey: x, y, same, opposite
    const double edu[4] = {u, v, __dadd_rn(u, v), __dsub_rn(u, v)};
    double e3[4], e45[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        e3[q] = __dmul_rn(3.0, edu[q]);
        e45[q] = __dmul_rn(__dmul_rn(4.5, edu[q]), edu[q]);
    }
    // bracket [0]: e.u = 0; [1 + 2 q]: +edu[q]; [2 + 2 q]: -edu[q]
    double br[9];
    br[0] = __dsub_rn(p3, u15);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        br[1 + 2 * q] = __dsub_rn(__dadd_rn(__dadd_rn(p3, e3[q]), e45[q]), u15);
        br[2 + 2 * q] = __dsub_rn(__dadd_rn(__dsub_rn(p3, e3[q]), e45[q]), u15);
    }
    // the weight times the bracket, formed once per (ex, ey) and |ez|
    double val[9][2];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int moves = q == 0 ? 0 : q < 5 ? 1 : 2;  // nonzero components among ex, ey
#pragma unroll
        for (int ez = 0; ez < 2; ++ez) {
            const int n = moves + ez;
            val[q][ez] = __dmul_rn(n == 0 ? 8.0 / 27.0 : n == 1 ? 2.0 / 27.0 : n == 2 ? 1.0 / 54.0 : 1.0 / 216.0, br[q]);
        }
    }
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
        const int x = ex(a, 0), y = ex(a, 1);
        const int q = x == 0 && y == 0 ? 0
                    : y == 0           ? (x > 0 ? 1 : 2)
                    : x == 0           ? (y > 0 ? 3 : 4)
                    : x == y           ? (x > 0 ? 5 : 6)
                                       : (x > 0 ? 7 : 8);
        fe[a] = val[q][ex(a, 2) != 0 ? 1 : 0];
    }
}

}  // namespace imex

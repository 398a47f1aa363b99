// Per-cell pressure and velocity (src/lbm.cpp:218-236) of one lattice.
//
// Bound: memory, 27 values read and 3 or 4 float64 written a cell.  The
// moments are the exact fixed-point ones (moments_fixed.cuh), each rounded
// once to float64; the reference's float64 sums (81 additions a cell, and 27
// conversions from reduced precision) held the kernels to the float64 pipe
// (2.7 ms at 256^3 float64, now 0.7).  A cell outside the fixed-point range is summed in
// float64.
//
// The largest difference of two lattices' velocities needs no float64 at
// all: the difference of exact integers is exact, and largest among integers.
// One kernel reads both lattices; two field kernels, 6 arrays between and a
// float64 maximum took 7.3 / 8.9 / 10.3 ms at 256^3 (float64 / float32 / float16
// against itself), this takes 1.09 / 1.03 / 1.07 (memory: 1.08 / 0.54 / 0.27).
#pragma once

#include "moments_fixed.cuh"

namespace imex {
namespace macro {

constexpr int kThreads = 128;

template <int P, bool PULL>
__global__ void __launch_bounds__(kThreads) k_macro(const typename mom::Elem<P>::T* __restrict__ src, Geom g, unsigned cells,
                                                    double* __restrict__ p, double* __restrict__ u,
                                                    double* __restrict__ v, double* __restrict__ w)
{
    const unsigned cell = blockIdx.x * kThreads + threadIdx.x;
    if (cell >= cells) return;
    int i, j, k;
    mom::cell_of(g, cell, i, j, k);
    const PullIndex pi(g, i, j, k, PULL);
    mom::Cell<P> c;
    double m[4];
    if (mom::moments<P, true>(src, g, pi, c)) {
        m[0] = (double)c.M[0] * 0x1p-61;
        for (int d = 0; d < 3; ++d) m[1 + d] = c.vel[d] * 0x1p-61;
    } else {
        mom::moments_f64_of<P>(src, g, i, j, k, PULL, m);
    }
    if (p) p[cell] = m[0] * (1.0 / 3.0);
    u[cell] = m[1];
    v[cell] = m[2];
    w[cell] = m[3];
}

template <int P>
cudaError_t launch(bool pull, const void* src, const Geom& g, double* p, double* u, double* v, double* w, cudaStream_t s)
{
    if (g.plane > 0xffffffffull - kThreads) return cudaErrorInvalidValue;  // above device memory
    const unsigned cells = (unsigned)g.plane, grid = (cells + kThreads - 1) / kThreads;
    const auto* f = static_cast<const typename mom::Elem<P>::T*>(src);
    if (pull) k_macro<P, true><<<grid, kThreads, 0, s>>>(f, g, cells, p, u, v, w);
    else k_macro<P, false><<<grid, kThreads, 0, s>>>(f, g, cells, p, u, v, w);
    return cudaGetLastError();
}

// CTAs an SM holds, with the registers that two cells' sums and loads take, and a
// grid of four turns of them. (Six CTAs an SM where four or five fit left a second
// turn nearly empty, for one pair of formats or another as their registers came out:
// 256^3 1.08 to 2.46 ms; now 0.96 to 1.09.  One turn 1.03 to 1.18,
// four CTAs and four turns 0.98 to 1.12.)
constexpr int kDiffCtas = 3;

// max over cells and components of |u_a - u_b| and of |u_b|: res[0], res[1]
// as integers in units of 2^-61; res[2], res[3] as float64 bit patterns over
// the cells where either lattice is outside the fixed-point range (NaN
// skipped, as fmax skips it).
template <int PA, int PB>
__global__ void __launch_bounds__(kThreads, kDiffCtas) k_velocity_diff(const typename mom::Elem<PA>::T* __restrict__ fa, bool pull_a,
                                                            const typename mom::Elem<PB>::T* __restrict__ fb, bool pull_b,
                                                            Geom g, unsigned cells, unsigned long long* __restrict__ res)
{
    unsigned long long best[4] = {0, 0, 0, 0};
    auto take = [&](int q, unsigned long long v) { best[q] = v > best[q] ? v : best[q]; };
    for (unsigned long long q = (unsigned long long)blockIdx.x * kThreads + threadIdx.x; q < cells;
         q += (unsigned long long)gridDim.x * kThreads) {
        int i, j, k;
        mom::cell_of(g, (unsigned)q, i, j, k);
        mom::Cell<PA> ca;
        mom::Cell<PB> cb;
        const bool oka = mom::moments<PA, true>(fa, g, PullIndex(g, i, j, k, pull_a), ca);
        const bool okb = mom::moments<PB, true>(fb, g, PullIndex(g, i, j, k, pull_b), cb);
        if (oka && okb) {
#pragma unroll
            for (int d = 1; d < 4; ++d) {
                // a component is below 2.25 (18 values below 1/8), so a difference can pass
                // the 4 at which the signed form ends
                const int64_t x = ca.M[d], y = cb.M[d];
                const uint64_t diff = (uint64_t)x - (uint64_t)y;
                take(0, x < y ? 0 - diff : diff);
                take(1, (uint64_t)(y < 0 ? -y : y));
            }
        } else {
            double ma[4], mb[4];
            // velocities alone: the float64 pipe bounds a lattice of such cells (256^3
            // float32 of density 1000 against float64 4.8 ms; with the mass, and six CTAs an
            // SM, 8.7; two field kernels and a maximum 8.1)
            mom::moments_f64_of<PA, false>(fa, g, i, j, k, pull_a, ma);
            mom::moments_f64_of<PB, false>(fb, g, i, j, k, pull_b, mb);
            for (int d = 1; d < 4; ++d) {
                const double x = fabs(ma[d] - mb[d]), y = fabs(mb[d]);
                if (x >= 0.0) take(2, (unsigned long long)__double_as_longlong(x));
                if (y >= 0.0) take(3, (unsigned long long)__double_as_longlong(y));
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) take(q, __shfl_xor_sync(0xffffffffu, best[q], o));
        if ((threadIdx.x & 31) == 0 && best[q]) atomicMax(res + q, best[q]);
    }
}

template <int PA, int PB>
cudaError_t launch_diff(const void* fa, bool pull_a, const void* fb, bool pull_b, const Geom& g, unsigned long long* res,
                        cudaStream_t s)
{
    if (g.plane > 0xffffffffull) return cudaErrorInvalidValue;
    const unsigned need = (unsigned)((g.plane + kThreads - 1) / kThreads), most = (unsigned)current_sm_count() * 4 * kDiffCtas;
    k_velocity_diff<PA, PB><<<need < most ? need : most, kThreads, 0, s>>>(
        static_cast<const typename mom::Elem<PA>::T*>(fa), pull_a, static_cast<const typename mom::Elem<PB>::T*>(fb), pull_b, g,
        (unsigned)g.plane, res);
    return cudaGetLastError();
}

}  // namespace macro
}  // namespace imex

// Conserved sums {mass, px, py, pz, ke} (src/lbm.cpp:266-306) of one lattice
// in one launch.
//
// Bound: memory, 27 values a cell (float64 storage), and for float16
// deviations the float64 pipe, which the kinetic energy's 6 operations a
// cell still need.  Mass and momentum are summed exactly, as 128-bit
// integers of the cells' fixed-point moments (moments_fixed.cuh), so only
// the kinetic energy depends on an order: each thread sums its cells in
// float64, then the block its threads, then the last block to finish the
// blocks, all in a fixed order.  Summing all five in float64 through warp
// shuffles (25 float64 additions a cell beside the moments' own) and then
// over one partial per 128-cell row segment with a single CTA took 1.75 /
// 1.50 / 1.59 ms at 256^3 (float64 / float32 / float16 deviations); this
// takes 0.56 / 0.36 / 0.36 ms (memory alone: 0.54 / 0.27 / 0.14), and 30 us
// instead of 66 at 32^3.
//
// Work split: cells in flat order, 256 consecutive ones per CTA and round,
// so the CTAs of a round read one contiguous region and the +-1 shifted
// pulls meet in L2; a row's end leaves no thread idle whatever nz is.
#pragma once

#include "moments_fixed.cuh"

namespace imex {
namespace cons {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// One block's sums: 4 integers of 128 bits, the kinetic energy in units of
// 2^-(2 kVelBits), and the float64 sums of cells outside the fixed-point range.
struct Partial {
    unsigned long long lo[4];
    long long hi[4];
    double ke;
    double out[5];
    int any_out;
    int pad;
};

struct Int128 {
    unsigned long long lo;
    long long hi;
    __device__ __forceinline__ void add(unsigned long long l, long long h)
    {
        lo += l;
        hi += h + (lo < l ? 1 : 0);
    }
    __device__ __forceinline__ void add(long long v) { add((unsigned long long)v, v >> 63); }
};

// Sums over the block's threads, valid in thread 0.  The integers go down
// the warp by shuffles; a float64 value through shared memory, where
// warp 0 adds a fixed eight per lane before its own shuffles (1.6 float64
// additions a thread instead of 5).
struct BlockSum {
    unsigned long long lo[kWarps][4];
    long long hi[kWarps][4];
    double ke[kThreads];
};
__device__ __forceinline__ double block_sum(double v, BlockSum& s)
{
    const int lane = threadIdx.x & 31;
    s.ke[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = s.ke[lane];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) v += s.ke[w * 32 + lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}
__device__ __forceinline__ void block_sum(Int128 (&m)[4], double& ke, BlockSum& s)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            m[q].add(__shfl_down_sync(0xffffffffu, m[q].lo, o), __shfl_down_sync(0xffffffffu, m[q].hi, o));
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s.lo[warp][q] = m[q].lo;
            s.hi[warp][q] = m[q].hi;
        }
    ke = block_sum(ke, s);
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            for (int w = 1; w < kWarps; ++w) m[q].add(s.lo[w][q], s.hi[w][q]);
}

// value * 2^-61, rounded twice at most (the high word is exact).
__device__ __forceinline__ double to_double(Int128 v)
{
    const bool neg = v.hi < 0;
    if (neg) {
        v.lo = ~v.lo + 1ull;
        v.hi = ~v.hi + (v.lo == 0 ? 1 : 0);
    }
    const double d = fma((double)v.hi, 0x1p64, __ull2double_rn(v.lo)) * 0x1p-61;
    return neg ? -d : d;
}

// Sums of a thread's cells outside the fixed-point range, in local memory: those of
// reduced precision in the wider range (moments_wide) as integers, the kinetic energy in
// the other cells' units; the rest in float64.  Written from the first such cell on:
// cleared at the start, by every thread, they cost 3 us at 128^3 (of 93).
struct Outside {
    Int128 m[4];
    double ke, sums[5];
    int any;  // float64 sums
};

// Adds such a cell (src/lbm.cpp:271-294).  The wider range covers lattices of densities of 2 to
// thousands: in float64, on the pipe that the integers are there to leave alone, 256^3
// float32 of density 1000 takes 3.9 ms, in integers 1.12.
template <int P>
__device__ __noinline__ void add_outside(const typename mom::Elem<P>::T* src, Geom g, int i, int j, int k, bool pull,
                                         Outside* o, bool first)
{
    if (first) *o = Outside{};
    if constexpr (P != IMEX_F64) {
        const mom::WideMoments w = mom::moments_wide<P>(src, g, i, j, k, pull);
        if (w.ok) {
            constexpr double kVel = (double)(1ull << (mom::kWide + mom::kVelBits<P>)) * 0x1p-61;
            for (int d = 0; d < 4; ++d)
                o->m[d].add((unsigned long long)w.M[d] << mom::kWide, (long long)w.M[d] >> (64 - mom::kWide));
            if (P == IMEX_F16DEV) o->m[0].add((long long)mom::weights_fixed());
            for (int d = 1; d < 4; ++d) {
                const double v = __ll2double_rn(w.M[d]) * kVel;
                o->ke = fma(v, v, o->ke);
            }
            return;
        }
    }
    double m[4];
    mom::moments_f64_of<P>(src, g, i, j, k, pull, m);
    for (int q = 0; q < 4; ++q) o->sums[q] += m[q];
    o->sums[4] += 0.5 * (m[1] * m[1] + m[2] * m[2] + m[3] * m[3]);
    o->any = 1;
}

template <int P, bool PULL, int MINB>
__global__ void __launch_bounds__(kThreads, MINB)
    k_conserved(const typename mom::Elem<P>::T* src, Geom g, unsigned cells, Partial* __restrict__ part,
                unsigned* __restrict__ ticket, const unsigned long long* __restrict__ status, double* __restrict__ out)
{
    __shared__ BlockSum s;
    __shared__ int s_last;
    chain_begin<true>();
    Int128 m[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
    double ke = 0.0;
    Outside outside;
    bool met = false;  // a cell for it
    for (unsigned long long q = (unsigned long long)blockIdx.x * kThreads + threadIdx.x; q < cells;
         q += (unsigned long long)gridDim.x * kThreads) {
        int i, j, k;
        mom::cell_of(g, (unsigned)q, i, j, k);
        const PullIndex pi(g, i, j, k, PULL);
        mom::Cell<P> c;
        if (mom::moments<P, false>(src, g, pi, c)) {
#pragma unroll
            for (int d = 0; d < 4; ++d) m[d].add((long long)c.M[d]);
#pragma unroll
            for (int d = 0; d < 3; ++d) ke = fma(c.vel[d], c.vel[d], ke);
        } else {
            add_outside<P>(src, g, i, j, k, PULL, &outside, !met);
            met = true;
        }
    }
    if (P != IMEX_F64 && met) {
#pragma unroll
        for (int d = 0; d < 4; ++d) m[d].add(outside.m[d].lo, outside.m[d].hi);
        ke += outside.ke;
    }
    block_sum(m, ke, s);
    int any = __syncthreads_or(met && outside.any);
    Partial& mine = part[blockIdx.x];
    if (any)
        for (int q = 0; q < 5; ++q) {
            __syncthreads();  // s is read
            const double v = block_sum(met ? outside.sums[q] : 0.0, s);
            if (threadIdx.x == 0) mine.out[q] = v;
        }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            mine.lo[q] = m[q].lo;
            mine.hi[q] = m[q].hi;
        }
        mine.ke = ke;
        mine.any_out = any;
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    // the last block: every partial is visible
    __threadfence();
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = Int128{0, 0};
    ke = 0.0;
    any = 0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kThreads) {
#pragma unroll
        for (int q = 0; q < 4; ++q) m[q].add(__ldcg(&part[b].lo[q]), __ldcg(&part[b].hi[q]));
        ke += __ldcg(&part[b].ke);
        any |= __ldcg(&part[b].any_out);
    }
    block_sum(m, ke, s);
    any = __syncthreads_or(any);
    double sums[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (any)
        for (int q = 0; q < 5; ++q) {
            for (unsigned b = threadIdx.x; b < gridDim.x; b += kThreads)
                if (__ldcg(&part[b].any_out)) sums[q] += __ldcg(&part[b].out[q]);
            __syncthreads();  // s is read
            sums[q] = block_sum(sums[q], s);
        }
    if (threadIdx.x == 0) {
        constexpr double kUnit = 1.0 / (double)(1ull << mom::kVelBits<P>);
        double r[5];
        for (int q = 0; q < 4; ++q) r[q] = to_double(m[q]);
        r[4] = 0.5 * ((ke * kUnit) * kUnit);
        for (int q = 0; q < 5; ++q) out[q] = any ? r[q] + sums[q] : r[q];
        if (status)
            for (int q = 0; q < 2; ++q) reinterpret_cast<unsigned long long*>(out)[5 + q] = __ldcg(status + q);
        *ticket = 0;  // for the next launch
    }
}

// CTAs of a launch over `cells` cells with `per_sm` CTAs per SM: no more
// than there are 256-cell rounds.
inline unsigned blocks_for(size_t cells, int sms, int per_sm)
{
    const size_t need = (cells + kThreads - 1) / kThreads, most = (size_t)sms * per_sm;
    return (unsigned)(need < most ? need : most);
}
constexpr int kMostPerSm = 4;

template <int P, int MINB>
cudaError_t launch(bool pull, const void* src, const Geom& g, void* part, unsigned* ticket,
                   const unsigned long long* status, double* out, cudaStream_t s)
{
    const size_t cells = (size_t)g.nx * g.ny * g.nz;
    if (cells > 0xffffffffull) return cudaErrorInvalidValue;
    const unsigned grid = blocks_for(cells, current_sm_count(), MINB);
    const auto* p = static_cast<const typename mom::Elem<P>::T*>(src);
    auto* pt = static_cast<Partial*>(part);
    return pull ? launch_chained(k_conserved<P, true, MINB>, grid, kThreads, 0, s, p, g, (unsigned)cells, pt, ticket, status, out)
                : launch_chained(k_conserved<P, false, MINB>, grid, kThreads, 0, s, p, g, (unsigned)cells, pt, ticket, status, out);
}

}  // namespace cons
}  // namespace imex

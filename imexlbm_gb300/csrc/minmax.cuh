// Largest and smallest u, v, w, p of a lattice (src/lbm.cpp:351-372), bit for
// bit those of the reference's float64 sums, found with integers.
//
// Bound: memory, each value read once (and the integer pipes beside it).
// Four float64 sums of a cell are 81 additions, and the float64 pipe issues
// 1.67 a clock and SM: summing every cell took 3.23 / 4.05 / 4.80 ms at 256^3
// (float64 / float32 / float16).  Here k_extremes forms the exact integer
// moments of every cell (moments_fixed.cuh) and k_pick sums in float64
// only the cells whose moment is within 2 kSlack of the extreme one: the two
// sums of a cell differ by less than kSlack, so no other cell can hold the
// float64 extreme.  The cells are taken in chunks; a chunk with no such cell
// ends at once, so k_pick is a few chunks' work unless a component is constant
// to the last bits.  0.62 / 0.67 / 0.67 ms at 256^3 (memory: 0.54 / 0.27 / 0.14);
// with w = 0 everywhere, as in an initial flow in x and y, that one component
// is summed again everywhere: 1.33 / 1.20 / 1.81.  Of cells that repeat, as in a fluid at
// rest, the first is summed (1.91 / 1.39 / 1.54; each of them 3.73 / 1.33 / 3.69, more
// than the float64 sums of all in one kernel).  Cells outside the integers' range are
// summed by k_extremes, where they are met: a lattice of density 1000 3.32 / 4.16 / 4.47
// (in k_pick 3.94 / 4.58 / 5.26).
#pragma once

#include <cfloat>
#include <type_traits>

#include "moments_fixed.cuh"

namespace imex {
namespace mm {

constexpr int kThreads = 128;
constexpr unsigned kLeastChunk = 256, kMostChunk = 2048;

// |float64 sum - exact moment| of an in-range cell, in units of 2^-61: 26
// additions whose partial sums are below 8 in magnitude, so each rounds by at
// most 2^-51 (26 * 2^10 units); reduced precision: 27 conversions within 2^-54
// of values below 1 (27 * 2^7), and bits below a unit dropped (2 * 27).
constexpr unsigned long long kSlack = 1ull << 15;
static_assert(26 * 1024 + 27 * 128 + 2 * 27 < kSlack, "kSlack covers the roundings");

// Keys whose order is the values' and whose 0 is below every value: [0..3] the
// largest of M (3p, u, v, w), [4..7] the smallest (the complement's largest).
__device__ __forceinline__ unsigned long long up(int64_t m) { return (unsigned long long)m + (1ull << 63); }
__device__ __forceinline__ unsigned long long up(double d)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// Integer extremes of one chunk of cells.
struct Chunk {
    unsigned long long key[8];
};
// The whole lattice's: the integer extremes, and the float64 ones as keys.
struct Result {
    unsigned long long whole[8], picked[8];
};

struct Split {
    unsigned cells, chunk, count;
};
// Chunks for a few CTAs on every SM, between the sizes whose start-up and
// whose scan by one CTA show.
inline Split split_of(const Geom& g, int sms)
{
    Split s;
    s.cells = (unsigned)g.plane;
    const unsigned even = (unsigned)(g.plane / ((size_t)sms * 8) + kThreads) / kThreads * kThreads;
    s.chunk = even < kLeastChunk ? kLeastChunk : even > kMostChunk ? kMostChunk : even;
    s.count = (unsigned)((g.plane + s.chunk - 1) / s.chunk);
    return s;
}
// Scratch for any split of the lattice.
inline size_t scratch_bytes(const Geom& g)
{
    return sizeof(Result) + (g.plane + kLeastChunk - 1) / kLeastChunk * sizeof(Chunk);
}

__device__ __forceinline__ void lift(unsigned long long* p, unsigned long long v)
{
    if (v > __ldcg(p)) atomicMax(p, v);
}

// Largest of each key over the CTA, valid in threads 0..7 (thread q: key q).
__device__ __forceinline__ unsigned long long block_largest(unsigned long long (&best)[8],
                                                            unsigned long long (*red)[8])
{
#pragma unroll
    for (int q = 0; q < 8; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, best[q], o);
            best[q] = v > best[q] ? v : best[q];
        }
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = best[q];
    }
    __syncthreads();
    unsigned long long v = 0;
    if (threadIdx.x < 8)
        for (int w = 0; w < kThreads / 32; ++w) v = red[w][threadIdx.x] > v ? red[w][threadIdx.x] : v;
    return v;
}

template <int P>
__device__ __forceinline__ double value_of(const typename mom::Elem<P>::T* src, const Geom& g, const PullIndex& pi, int a)
{
    const auto v = load_state(src + pi.at_dyn(g, a));
    if constexpr (P == IMEX_F64) return v;
    else return lowp::Storage<P>::to_f64(v, a);
}

// The float64 sums of a cell in the reference's order: x[0] = 3p, x[1..3] = u, v, w.
// Out of line: few cells need them.  sum_one forms one of them alone.
template <int P>
__device__ __noinline__ void sum_all(const typename mom::Elem<P>::T* src, const Geom& g, const PullIndex& pi, double* x)
{
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
        const double f = value_of<P>(src, g, pi, a);
        s[0] += f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (ex(a, d) == 1) s[1 + d] += f;
            if (ex(a, d) == -1) s[1 + d] -= f;
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = s[q];
}
template <int P>
__device__ __noinline__ double sum_one(const typename mom::Elem<P>::T* src, const Geom& g, const PullIndex& pi, int q)
{
    double s = 0.0;
    if (q == 0) {
#pragma unroll
        for (int a = 0; a < kQ; ++a) s += value_of<P>(src, g, pi, a);
        return s;
    }
    auto along = [&](auto dim) {
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
            if (ex(a, decltype(dim)::value) == 1) s += value_of<P>(src, g, pi, a);
            if (ex(a, decltype(dim)::value) == -1) s -= value_of<P>(src, g, pi, a);
        }
    };
    if (q == 1) along(std::integral_constant<int, 0>{});
    else if (q == 2) along(std::integral_constant<int, 1>{});
    else along(std::integral_constant<int, 2>{});
    return s;
}

// Whether every float64 sum of an in-range cell is exact, so that the moment is the sum:
// float32 values of 2^-27 and more are multiples of 2^-50, their partial sums
// below 8.
template <int P>
__device__ __noinline__ bool sums_exact(const typename mom::Elem<P>::T* src, const Geom& g, const PullIndex& pi)
{
    if constexpr (P != IMEX_F32) return false;
    else {
        float least = 1.f;
#pragma unroll
        for (int a = 0; a < kQ; ++a) least = fminf(least, fabsf(load_state(src + pi.at_dyn(g, a))));
        return least >= 0x1p-27f;
    }
}

// Whether cells c and d hold the same 27 values, so that their sums are the same:
// in a fluid at rest all do.  Ends at the first difference.
constexpr unsigned kNoCell = 0xffffffffu;
template <int P>
__device__ __noinline__ bool same_values(const typename mom::Elem<P>::T* src, Geom g, unsigned c, unsigned d, bool pull)
{
    int i, j, k;
    mom::cell_of(g, c, i, j, k);
    const PullIndex pc(g, i, j, k, pull);
    mom::cell_of(g, d, i, j, k);
    const PullIndex pd(g, i, j, k, pull);
    bool same = true;
#pragma unroll
    for (int a = 0; a < kQ && same; ++a) {
        const auto v = load_state(src + pc.at_dyn(g, a)), w = load_state(src + pd.at_dyn(g, a));
        if constexpr (P == IMEX_F64) same = __double_as_longlong(v) == __double_as_longlong(w);
        else if constexpr (P == IMEX_F32) same = __float_as_uint(v) == __float_as_uint(w);
        else same = __half_as_ushort(v) == __half_as_ushort(w);
    }
    return same;
}

// Component q of a cell by the reference's comparisons: from -DBL_MAX and DBL_MAX on,
// NaN skipped.
__device__ __forceinline__ void take(unsigned long long* best, int q, double x)
{
    if (x > -DBL_MAX && up(x) > best[q]) best[q] = up(x);
    if (x < DBL_MAX && ~up(x) > best[4 + q]) best[4 + q] = ~up(x);
}

// The float64 sums of a cell outside the range, for k_extremes, unless the thread's last such
// cell (kNoCell: none yet) has the same; best lies in local memory, cleared by the first.
template <int P>
__device__ __noinline__ void take_outside(const typename mom::Elem<P>::T* src, Geom g, unsigned cell, unsigned last,
                                          bool pull, unsigned long long* best)
{
    if (last == kNoCell) {
        for (int q = 0; q < 8; ++q) best[q] = 0;
    } else if (same_values<P>(src, g, cell, last, pull)) {
        return;
    }
    double x[4];
    int i, j, k;
    mom::cell_of(g, cell, i, j, k);
    mom::moments_f64_of<P>(src, g, i, j, k, pull, x);
    x[0] *= 1.0 / 3.0;
    for (int q = 0; q < 4; ++q) take(best, q, x[q]);
}

template <int P, bool PULL>
__global__ void __launch_bounds__(kThreads) k_extremes(const typename mom::Elem<P>::T* src, Geom g, Split s,
                                                       Chunk* __restrict__ chunks, Result* __restrict__ res)
{
    __shared__ unsigned long long red[kThreads / 32][8];
    chain_begin<false>();
    unsigned long long best[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    unsigned long long summed[8];  // of cells outside the range
    unsigned last = kNoCell;       // the last of them
    const unsigned begin = blockIdx.x * s.chunk, end = s.cells - begin < s.chunk ? s.cells : begin + s.chunk;
    for (unsigned cell = begin + threadIdx.x; cell < end && cell >= begin; cell += kThreads) {
        int i, j, k;
        mom::cell_of(g, cell, i, j, k);
        mom::Cell<P> c;
        if (mom::moments<P, true>(src, g, PullIndex(g, i, j, k, PULL), c)) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned long long v = up(c.M[q]);
                best[q] = v > best[q] ? v : best[q];
                best[4 + q] = ~v > best[4 + q] ? ~v : best[4 + q];
            }
        } else {
            take_outside<P>(src, g, cell, last, PULL, summed);
            last = cell;
        }
    }
    const unsigned long long v = block_largest(best, red);
    if (threadIdx.x < 8) {
        chunks[blockIdx.x].key[threadIdx.x] = v;
        lift(&res->whole[threadIdx.x], v);
    }
    if (__syncthreads_or(last != kNoCell)) {
#pragma unroll
        for (int q = 0; q < 8; ++q) best[q] = last != kNoCell ? summed[q] : 0;
        const unsigned long long w = block_largest(best, red);
        if (threadIdx.x < 8) lift(&res->picked[threadIdx.x], w);
    }
    chain_end<false>();
}

template <int P, bool PULL>
__global__ void __launch_bounds__(kThreads) k_pick(const typename mom::Elem<P>::T* src, Geom g, Split s,
                                                   const Chunk* __restrict__ chunks, Result* __restrict__ res)
{
    __shared__ unsigned long long red[kThreads / 32][8];
    chain_begin<false>();
    // least key of a cell to be summed; keys are far above 2 kSlack or 0 (no
    // in-range cell at all: none is compared)
    unsigned long long least[8];
    bool any = false;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const unsigned long long w = __ldcg(&res->whole[q]);
        least[q] = w > 2 * kSlack ? w - 2 * kSlack : 1;
        any = any || __ldcg(&chunks[blockIdx.x].key[q]) >= least[q];
    }
    if (!any) return;  // the same in every thread
    unsigned last = kNoCell;  // the last cell summed
    int last_need = 0;
    bool differ = false;      // a comparison failed: no more of them in this chunk (16 cells a thread)
    unsigned long long best[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const unsigned begin = blockIdx.x * s.chunk, end = s.cells - begin < s.chunk ? s.cells : begin + s.chunk;
    for (unsigned cell = begin + threadIdx.x; cell < end && cell >= begin; cell += kThreads) {
        int i, j, k;
        mom::cell_of(g, cell, i, j, k);
        const PullIndex pi(g, i, j, k, PULL);
        mom::Cell<P> c;
        if (!mom::moments<P, true>(src, g, pi, c)) continue;  // k_extremes has summed it
        int need = 0;  // components to be summed
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const unsigned long long v = up(c.M[q]);
            if (v >= least[q] || ~v >= least[4 + q]) need |= 1 << q;
        }
        if (!need) continue;
        double x[4];
        if (sums_exact<P>(src, g, pi)) {
#pragma unroll
            for (int q = 0; q < 4; ++q) x[q] = (double)c.M[q] * 0x1p-61;
        } else {
            if (need == last_need && !differ) {
                if (same_values<P>(src, g, cell, last, PULL)) continue;
                differ = true;
            }
            last = cell;
            last_need = need;
            if (need & (need - 1)) {
                sum_all<P>(src, g, pi, x);
            } else {
                x[0] = sum_one<P>(src, g, pi, __ffs(need) - 1);
                x[1] = x[2] = x[3] = x[0];
            }
        }
        x[0] *= 1.0 / 3.0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (need >> q & 1) take(best, q, x[q]);
    }
    const unsigned long long v = block_largest(best, red);
    if (threadIdx.x < 8) lift(&res->picked[threadIdx.x], v);
}

template <int P, bool PULL>
cudaError_t launch_as(const void* src, const Geom& g, const Split& s, Chunk* chunks, Result* res, cudaStream_t st)
{
    const auto* f = static_cast<const typename mom::Elem<P>::T*>(src);
    cudaError_t e = launch_chained(k_extremes<P, PULL>, s.count, kThreads, 0, st, f, g, s, chunks, res);
    if (e != cudaSuccess) return e;
    return launch_chained(k_pick<P, PULL>, s.count, kThreads, 0, st, f, g, s, chunks, res);
}

// Two launches; `scratch` (scratch_bytes) begins with the Result on completion.
inline cudaError_t launch(int prec, bool pull, const void* src, const Geom& g, void* scratch, cudaStream_t st)
{
    if (g.plane > 0xffffffffull) return cudaErrorInvalidValue;  // above device memory
    const Split s = split_of(g, current_sm_count());
    Result* res = static_cast<Result*>(scratch);
    Chunk* chunks = reinterpret_cast<Chunk*>(res + 1);
    cudaError_t e = cudaMemsetAsync(res, 0, sizeof(Result), st);
    if (e != cudaSuccess) return e;
    switch (prec) {
    case IMEX_F64:
        return pull ? launch_as<IMEX_F64, true>(src, g, s, chunks, res, st) : launch_as<IMEX_F64, false>(src, g, s, chunks, res, st);
    case IMEX_F32:
        return pull ? launch_as<IMEX_F32, true>(src, g, s, chunks, res, st) : launch_as<IMEX_F32, false>(src, g, s, chunks, res, st);
    case IMEX_F16DEV:
        return pull ? launch_as<IMEX_F16DEV, true>(src, g, s, chunks, res, st)
                    : launch_as<IMEX_F16DEV, false>(src, g, s, chunks, res, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace mm
}  // namespace imex

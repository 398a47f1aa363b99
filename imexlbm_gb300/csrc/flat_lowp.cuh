// Fused step of the reduced-precision formats over flat cell pairs: a thread
// takes cells 2 p and 2 p + 1 of the lattice's flat order (z fastest),
// whatever row they lie in, straight from global memory.  Any sizes; the
// row-staged kernel (rows_lowp.cuh) takes float16 rows that are whole 16-byte
// pieces, the two-step kernel (two_f32.cuh) most large float32 lattices, this one the
// rest.
//
// Why pairs in flat order.  One thread per cell and 128 of them per row
// segment (the form before) leaves the threads behind a row's end idle and
// spends ~815 instructions on a float16 cell: issue-bound.  Two cells go
// through the packed f32x2 collision together; pairs of the flat order are
// the pairs that share a random word (sr_word), so one cvt.rs rounds
// both; no thread is idle whatever nz is.  The two cells' sources are
// separate sums of an x, a y and a z offset, so a pair may lie across a
// row's end.
// Of an odd number of cells the even directions' pairs still lie on a 4-byte
// boundary and are stored at once; the number's parity is a template argument
// (255^3 float16 377 -> 350 us, 45^3 4.9 -> 4.0).
// Measured per step, one cell per thread -> now: float16 131 x 77 x 90 37.0 -> 18.0
// us, 107 x 99 x 84 33.0 -> 17.3, 255^3 469 -> 350, 256^3 468 -> 335 (the row-staged
// kernel: 281); float32 97 x 150 x 121 69.9 -> 59.1, 255^3 575 -> 546, 256^3 527 -> 520
// (memory alone: 543 at the copy rate).  Bound: memory for float32, issue for float16.
#pragma once

#include "kernels_common.cuh"
#include "lowp_math.cuh"

namespace imex {
namespace flat {

constexpr int kThreads = 128;
constexpr int kCells = 2 * kThreads;  // cells of a CTA

// A thread's pair is two neighbours, cells 2 t and 2 t + 1 of its CTA's
// kCells (near), or cells t and t + kThreads.  Float32 results of an odd number of
// cells lie off their 8-byte boundary in every other direction: there the
// second form keeps lanes on consecutive cells, so that the 4-byte accesses
// coalesce (61 x 65 x 63: 10.3 us against 12.3; 64^3 8.4 in the first form,
// 10.3 in the second).
template <int P, bool kEven>
inline constexpr bool kNear = kEven || P == IMEX_F16DEV;
template <int P, bool kEven>
__device__ __forceinline__ unsigned first_cell(unsigned block, unsigned t)
{
    return block * kCells + (kNear<P, kEven> ? 2 * t : t);
}

// Fused step of the pair whose first cell is c < plane (the second may lie
// beyond the last cell) of a lattice of fewer than 2^32 cells; kEven: of an even
// number of them.  Ends its kernel's chain (chain_end).
template <int P, bool kEven, bool kEarly>
__device__ __forceinline__ void step_pair(const typename lowp::Storage<P>::T* src,
                                          typename lowp::Storage<P>::T* __restrict__ dst, int nx, int ny, int nz,
                                          size_t plane, unsigned c, const CollideF32& cp)
{
    using S = lowp::Storage<P>;
    using T = typename S::T;
    using A = lowp::F2;
    constexpr unsigned kNext = kNear<P, kEven> ? 1 : kThreads;  // float16 pairs share a random word
    const bool two = c + kNext < (unsigned)plane;
    const FlatPull p0(nx, ny, nz, c), p1(nx, ny, nz, two ? c + kNext : c);
    float2 h[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
        const T* p = src + (size_t)a * plane;
        const T v0 = load_state(p + p0.at(a)), v1 = load_state(p + p1.at(a));
        h[a] = make_float2(S::dev(v0, a), S::dev(v1, a));
    }
    lowp::collide_dev<P, A>(h, cp);
    chain_end<kEarly>();
    T* const o = dst + c;
    if constexpr (P == IMEX_F16DEV) {
        // an odd number of cells puts the odd directions' pairs off their
        // 4-byte boundary
        auto put = [&](int a, __half2 r) {
            T* const q = o + (size_t)a * plane;
            if ((kEven || !(a & 1)) && two) {
                *reinterpret_cast<__half2*>(q) = r;
            } else {
                q[0] = __low2half(r);
                if (two) q[1] = __high2half(r);
            }
        };
        if (cp.sr) {
            const uint32_t ph = lowp::sr_hash(c >> 1, cp.seed), pc = lowp::sr_corner_hash(ph);
            lowp::round_f16_conserving<A>(h, [&](int a, float2 v) -> float2 {
                const uint32_t w = lowp::cvt_rs_f16x2(v.y, v.x, lowp::sr_word(ph, pc, a));
                const __half2 r = *reinterpret_cast<const __half2*>(&w);
                put(a, r);
                return make_float2(lowp::sub_f16_f32(__low2half(r), v.x), lowp::sub_f16_f32(__high2half(r), v.y));
            });
        } else {
            lowp::round_f16_conserving<A>(h, [&](int a, float2 v) -> float2 {
                const __half2 r = __floats2half2_rn(v.x, v.y);
                put(a, r);
                return make_float2(lowp::sub_f16_f32(__low2half(r), v.x), lowp::sub_f16_f32(__high2half(r), v.y));
            });
        }
    } else {
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
            T* const q = o + (size_t)a * plane;
            const float2 v = make_float2(S::store(h[a].x, a), S::store(h[a].y, a));
            if (kEven && two) {  // plane even: 8-byte aligned
                *reinterpret_cast<float2*>(q) = v;
            } else {
                q[0] = v.x;
                if (two) q[kNext] = v.y;
            }
        }
    }
}

}  // namespace flat
}  // namespace imex

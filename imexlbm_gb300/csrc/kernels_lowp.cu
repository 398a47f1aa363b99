// Reduced-precision storage kernels: float32 distributions (IMEX_F32) and
// float16 deviations 2^12 (f - w) (IMEX_F16DEV), collided in float32 by
// lowp::collide_dev_f32 (lowp_math.cuh, which explains the arithmetic);
// diagnostics accumulate in float64.
#include <atomic>
#include <cmath>

#include <cuda_fp16.h>

#include "conserved.cuh"
#include "flat_lowp.cuh"
#include "kernels_lowp.cuh"
#include "lowp_math.cuh"
#include "macro.cuh"
#include "rows.cuh"
#include "rows_lowp.cuh"
#include "tg_init.cuh"

namespace imex {

namespace {

using lowp::Storage;
using lowp::collide_dev_f32;

// Collision in place (src == dst), or streaming alone.
template <int P, bool COLLIDE>
__global__ void __launch_bounds__(kStepBlock) k_step_lowp(const typename Storage<P>::T* src, typename Storage<P>::T* dst,
                                                          Geom g, CollideF32 cp)
{
    using S = Storage<P>;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, i = blockIdx.z;
    if (k >= g.nz) return;
    const size_t cell = ((size_t)i * g.ny + j) * g.nz + k;
    if constexpr (!COLLIDE) {
        // streaming alone moves the stored bits unchanged
        const PullIndex pi(g, i, j, k, true);
#pragma unroll
        for (int a = 0; a < kQ; ++a) dst[(size_t)a * g.plane + cell] = src[pi.at_dyn(g, a)];
        return;
    }
    float h[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) h[a] = S::load_plain(src + (size_t)a * g.plane + cell, a);
    collide_dev_f32<P>(h, cp);
    if constexpr (P == IMEX_F16DEV) {
        auto at = [&](int a) -> __half& { return dst[(size_t)a * g.plane + cell]; };
        lowp::store_f16_cell(h, cp.sr, cell, cp.seed, at);
    } else {
#pragma unroll
        for (int a = 0; a < kQ; ++a) dst[(size_t)a * g.plane + cell] = S::store(h[a], a);
    }
}

// The fused step over flat cell pairs (flat_lowp.cuh).
// CTAs per SM the registers are held to; 0: as the compiler has it (90 at most,
// 5 CTAs).  Six fit without a spill where nothing is drawn at random (float16 to
// nearest: 107 x 99 x 84 17.25 -> 17.08 us a step, 64 x 64 x 63 6.50 -> 6.00, 45^3 4.24 ->
// 3.51; float32 with 6: 64^3 6.44 -> 6.92); a lattice whose CTAs all run at once
// gains from room for its loads' addresses instead (1; stochastic 64 x 64 x 63
// 6.55 -> 6.16, 45^3 3.87 -> 3.57; float32 61 x 65 x 63 7.79 -> 7.44, but 64^3 6.44 -> 6.62).
template <int P, bool kEven, bool SR, bool kEarly>
inline constexpr int kFlatCtas = P == IMEX_F16DEV && !SR                      ? 6
                                 : !kEarly && (P == IMEX_F16DEV || !kEven) ? 1
                                                                              : 0;
template <int P, bool kEven, bool SR, bool kEarly>
__global__ void __launch_bounds__(flat::kThreads, kFlatCtas<P, kEven, SR, kEarly>) k_flat_lowp(const typename Storage<P>::T* src,
                                                              typename Storage<P>::T* __restrict__ dst, Geom g,
                                                              CollideF32 cp)
{
    chain_begin<kEarly>();
    const unsigned c = flat::first_cell<P, kEven>(blockIdx.x, threadIdx.x);
    if (c >= (unsigned)g.plane) return;
    cp.sr = SR;
    flat::step_pair<P, kEven, kEarly>(src, dst, g.nx, g.ny, g.nz, g.plane, c, cp);
}

// Taylor-Green initial state (float64 equilibrium, src/lbm.cpp:78-108),
// rounded once into the storage format.
template <int P>
__global__ void __launch_bounds__(kStepBlock) k_init_lowp(typename Storage<P>::T* __restrict__ f, Geom g,
                                                          const double* __restrict__ tx, const double* __restrict__ ty,
                                                          const double* __restrict__ tz, TgParams tg)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, i = blockIdx.z;
    if (k >= g.nz) return;
    double fe[kQ];
    tg_init_cell(fe, tx, ty, tz, i, j, k, tg);
    const size_t cell = ((size_t)i * g.ny + j) * g.nz + k;
#pragma unroll
    for (int a = 0; a < kQ; ++a) f[(size_t)a * g.plane + cell] = Storage<P>::from_f64(fe[a], a);
}

// Conversions between float64 reference-order f and the storage format,
// bound by memory (10 or 12 bytes a value).  From float64: one direction per
// grid row, so its weight is uniform over the CTA and no thread divides by
// the plane's size.
constexpr int kConvThreads = 256, kConvPer = 4;
template <int P>
__global__ void __launch_bounds__(kConvThreads) k_from_f64(const double* __restrict__ f,
                                                           typename Storage<P>::T* __restrict__ out, size_t plane)
{
    const int a = blockIdx.y;
    f += (size_t)a * plane;
    out += (size_t)a * plane;
    const size_t q0 = (size_t)blockIdx.x * (kConvThreads * kConvPer) + threadIdx.x;
    double v[kConvPer];
#pragma unroll
    for (int c = 0; c < kConvPer; ++c) v[c] = q0 + c * kConvThreads < plane ? __ldg(f + q0 + c * kConvThreads) : 1.0;
#pragma unroll
    for (int c = 0; c < kConvPer; ++c)
        if (q0 + c * kConvThreads < plane) out[q0 + c * kConvThreads] = Storage<P>::from_f64(v[c], a);
}

// One cell again in float64, for values off the exact integer grid.
template <int P>
__device__ __noinline__ void to_f64_cell_wide(const typename Storage<P>::T* src, Geom g, int i, int j, int k, bool pull,
                                              unsigned cell, double* out)
{
    const PullIndex pi(g, i, j, k, pull);
#pragma unroll
    for (int a = 0; a < kQ; ++a) out[(size_t)a * g.plane + cell] = Storage<P>::to_f64(src[pi.at_dyn(g, a)], a);
}

// To float64: a thread per cell in flat order (a row's end leaves no thread
// idle), pulling through a pending streaming.
template <int P, bool PULL>
__global__ void __launch_bounds__(kStepBlock) k_to_f64(const typename Storage<P>::T* __restrict__ src, Geom g,
                                                         unsigned cells, double* __restrict__ out)
{
    const unsigned cell = blockIdx.x * kStepBlock + threadIdx.x;
    if (cell >= cells) return;
    int i, j, k;
    mom::cell_of(g, cell, i, j, k);
    const PullIndex pi(g, i, j, k, PULL);
    bool ok = true;
#pragma unroll
    for (int a = 0; a < kQ; ++a)
        out[(size_t)a * g.plane + cell] = Storage<P>::to_f64_exact(__ldg(src + pi.at_dyn(g, a)), a, ok);
    if (!ok) to_f64_cell_wide<P>(src, g, i, j, k, PULL, cell, out);
}

dim3 step_grid(const Geom& g) { return dim3((g.nz + kStepBlock - 1) / kStepBlock, g.ny, g.nx); }

template <int P>
cudaError_t step_impl(int mode, const void* src, void* dst, const Geom& g, const CollideF32& cp, cudaStream_t s)
{
    using T = typename Storage<P>::T;
    const T* a = static_cast<const T*>(src);
    T* b = static_cast<T*>(dst);
    switch (mode) {
    case kModeFused: {
        if (g.plane > 0xffffffffull - flat::kCells) return cudaErrorInvalidValue;  // above device memory
        const unsigned grid = (unsigned)((g.plane + flat::kCells - 1) / flat::kCells);
        // CTAs an SM, us a step early and late: float16 to nearest 4 4.06, 4.20; 6 5.4, 5.5; 8 6.7, 6.8; float32
        // 4 6.2, 4.8; 6 6.9, 6.6; 8 8.1, 7.7; 11 11.0, 10.7; 14 15.8, 16.2
        const bool early = chain_early((unsigned long long)grid * flat::kThreads, 8 * flat::kThreads);
        auto go = [&](auto kernel) { return launch_chained(kernel, grid, flat::kThreads, 0, s, a, b, g, cp); };
        auto of = [&](auto even, auto sr) {
            constexpr bool kEven = decltype(even)::value, kSr = decltype(sr)::value;
            return early ? go(k_flat_lowp<P, kEven, kSr, true>) : go(k_flat_lowp<P, kEven, kSr, false>);
        };
        const bool even = !(g.plane & 1);
        if constexpr (P == IMEX_F16DEV) {
            if (cp.sr) return even ? of(std::true_type{}, std::true_type{}) : of(std::false_type{}, std::true_type{});
        }
        return even ? of(std::true_type{}, std::false_type{}) : of(std::false_type{}, std::false_type{});
    }
    case kModeCollide: k_step_lowp<P, true><<<step_grid(g), kStepBlock, 0, s>>>(a, b, g, cp); break;
    case kModeStream: k_step_lowp<P, false><<<step_grid(g), kStepBlock, 0, s>>>(a, b, g, cp); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace

CollideF32 make_collide_f32(double tau0)
{
    CollideF32 cp;
    const double omega = 1.0 / (tau0 + 0.5);  // src/lbm.cpp:133
    cp.eps = (float)(2.0 - omega);              // exact in float64 for omega in [1, 2]
    const double w[4] = {8.0 / 27.0, 2.0 / 27.0, 1.0 / 54.0, 1.0 / 216.0};  // src/lbm.cpp:10-17
    for (int c = 0; c < 4; ++c) cp.w[c] = (float)w[c];
    // e.u coefficients 3 w with the momentum identity exact in float32:
    // b_face on the 2^-27 grid, b_corner on the 2^-28 grid, so that
    // 1/2 - 4 b_face - 4 b_corner lands on the 2^-26 grid of b_axis.
    const double bf = std::nearbyint(3.0 * w[2] * 0x1p27) * 0x1p-27;
    const double bc = std::nearbyint(3.0 * w[3] * 0x1p28) * 0x1p-28;
    const double ba = 0.5 - 4.0 * bf - 4.0 * bc;
    cp.w3[0] = 0.f;
    cp.w3[1] = (float)ba;
    cp.w3[2] = (float)bf;
    cp.w3[3] = (float)bc;
    cp.sr = 0;
    cp.seed = 0;
    return cp;
}

cudaError_t launch_init_lowp(int prec, void* f, const Geom& g, const double* tx, const double* ty, const double* tz,
                             double rho0, double u0, cudaStream_t s)
{
    if (prec == IMEX_F32)
        k_init_lowp<IMEX_F32><<<step_grid(g), kStepBlock, 0, s>>>(static_cast<float*>(f), g, tx, ty, tz, tg_params(rho0, u0));
    else
        k_init_lowp<IMEX_F16DEV><<<step_grid(g), kStepBlock, 0, s>>>(static_cast<__half*>(f), g, tx, ty, tz, tg_params(rho0, u0));
    return cudaGetLastError();
}

cudaError_t launch_step_lowp(int prec, int mode, const void* src, void* dst, const Geom& g, const CollideF32& cp,
                             cudaStream_t s)
{
    return prec == IMEX_F32 ? step_impl<IMEX_F32>(mode, src, dst, g, cp, s)
                            : step_impl<IMEX_F16DEV>(mode, src, dst, g, cp, s);
}

bool rows_lowp_eligible(int prec, const Geom& g)
{
    const size_t row = (size_t)g.nz * (prec == IMEX_F32 ? 4 : 2);
    return row % 16 == 0 && row <= (size_t)kRowsLowpDirMax && (size_t)g.nx * g.ny < 0x7fffffffu;
}

template <int D, int MINB>
cudaError_t launch_rows_lowp_d(int prec, const void* src, void* dst, const Geom& g, const CollideF32& cp,
                               const RowConfig& rc, unsigned* err, cudaStream_t s, unsigned grid)
{
    const size_t smem = rowslp::smem_bytes(D, rc.stages);
    // raise the kernel's shared-memory limit once per device and size, not
    // per launch (the attribute belongs to the device's context)
    static std::atomic<int> allowed[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || (int)smem > allowed[dev].load()) {
        e = cudaFuncSetAttribute(rowslp::k_rows_lowp<D, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
        if (e != cudaSuccess) return e;
        if (dev < 64) allowed[dev].store((int)smem);
    }
    return launch_chained(rowslp::k_rows_lowp<D, MINB>, grid, rowslp::kThreads, smem, s, src, dst, g, prec, rc.rows, cp,
                          rc.stages, make_wait_ctl(err));
}

cudaError_t launch_rows_lowp(int prec, const void* src, void* dst, const Geom& g, const CollideF32& cp,
                             const RowConfig& rc, unsigned* err, cudaStream_t s)
{
    const int sms = current_sm_count();
    const size_t es = prec == IMEX_F32 ? 4 : 2;
    if (rc.rows < 1 || (size_t)rc.rows * g.nz * es > (size_t)rc.dir_bytes || rc.stages < 2)
        return cudaErrorInvalidValue;
    const long long items = (long long)g.nx * rowslp::y_blocks(g.ny, rc.rows);
    long long grid = (long long)sms * rc.ctas_per_sm;
    if (grid > items) grid = items;
    const bool one = rc.ctas_per_sm <= 1;  // one resident CTA: the full register file
    switch (rc.dir_bytes) {
    case 1024:
        return one ? launch_rows_lowp_d<1024, 1>(prec, src, dst, g, cp, rc, err, s, (unsigned)grid)
                   : launch_rows_lowp_d<1024, 2>(prec, src, dst, g, cp, rc, err, s, (unsigned)grid);
    case 2048:
        return one ? launch_rows_lowp_d<2048, 1>(prec, src, dst, g, cp, rc, err, s, (unsigned)grid)
                   : launch_rows_lowp_d<2048, 2>(prec, src, dst, g, cp, rc, err, s, (unsigned)grid);
    case 4096: return launch_rows_lowp_d<4096, 1>(prec, src, dst, g, cp, rc, err, s, (unsigned)grid);
    default: return cudaErrorInvalidValue;
    }
}

size_t rows_lowp_stage_bytes(int prec, int nz) { return (size_t)kQ * nz * (prec == IMEX_F32 ? 4 : 2); }

cudaError_t launch_from_f64(int prec, const double* f, void* out, const Geom& g, cudaStream_t s)
{
    const dim3 grid((unsigned)((g.plane + kConvThreads * kConvPer - 1) / (kConvThreads * kConvPer)), kQ);
    if (prec == IMEX_F32)
        k_from_f64<IMEX_F32><<<grid, kConvThreads, 0, s>>>(f, static_cast<float*>(out), g.plane);
    else
        k_from_f64<IMEX_F16DEV><<<grid, kConvThreads, 0, s>>>(f, static_cast<__half*>(out), g.plane);
    return cudaGetLastError();
}

cudaError_t launch_to_f64(int prec, bool pull, const void* src, const Geom& g, double* out, cudaStream_t s)
{
    if (g.plane > 0xffffffffull - kStepBlock) return cudaErrorInvalidValue;  // above device memory
    const unsigned cells = (unsigned)g.plane, grid = (cells + kStepBlock - 1) / kStepBlock;
    if (prec == IMEX_F32) {
        const float* p = static_cast<const float*>(src);
        if (pull) k_to_f64<IMEX_F32, true><<<grid, kStepBlock, 0, s>>>(p, g, cells, out);
        else k_to_f64<IMEX_F32, false><<<grid, kStepBlock, 0, s>>>(p, g, cells, out);
    } else {
        const __half* p = static_cast<const __half*>(src);
        if (pull) k_to_f64<IMEX_F16DEV, true><<<grid, kStepBlock, 0, s>>>(p, g, cells, out);
        else k_to_f64<IMEX_F16DEV, false><<<grid, kStepBlock, 0, s>>>(p, g, cells, out);
    }
    return cudaGetLastError();
}

cudaError_t launch_macro(int prec, bool pull, const void* src, const Geom& g, double* p, double* u, double* v, double* w,
                         cudaStream_t s)
{
    switch (prec) {
    case IMEX_F64: return macro::launch<IMEX_F64>(pull, src, g, p, u, v, w, s);
    case IMEX_F32: return macro::launch<IMEX_F32>(pull, src, g, p, u, v, w, s);
    default: return macro::launch<IMEX_F16DEV>(pull, src, g, p, u, v, w, s);
    }
}

cudaError_t launch_velocity_diff(int prec_a, const void* fa, bool pull_a, int prec_b, const void* fb, bool pull_b,
                                 const Geom& g, unsigned long long* res, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(res, 0, 4 * sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    switch (3 * prec_a + prec_b) {
    case 3 * IMEX_F64 + IMEX_F64: return macro::launch_diff<IMEX_F64, IMEX_F64>(fa, pull_a, fb, pull_b, g, res, s);
    case 3 * IMEX_F64 + IMEX_F32: return macro::launch_diff<IMEX_F64, IMEX_F32>(fa, pull_a, fb, pull_b, g, res, s);
    case 3 * IMEX_F64 + IMEX_F16DEV: return macro::launch_diff<IMEX_F64, IMEX_F16DEV>(fa, pull_a, fb, pull_b, g, res, s);
    case 3 * IMEX_F32 + IMEX_F64: return macro::launch_diff<IMEX_F32, IMEX_F64>(fa, pull_a, fb, pull_b, g, res, s);
    case 3 * IMEX_F32 + IMEX_F32: return macro::launch_diff<IMEX_F32, IMEX_F32>(fa, pull_a, fb, pull_b, g, res, s);
    case 3 * IMEX_F32 + IMEX_F16DEV: return macro::launch_diff<IMEX_F32, IMEX_F16DEV>(fa, pull_a, fb, pull_b, g, res, s);
    case 3 * IMEX_F16DEV + IMEX_F64: return macro::launch_diff<IMEX_F16DEV, IMEX_F64>(fa, pull_a, fb, pull_b, g, res, s);
    case 3 * IMEX_F16DEV + IMEX_F32: return macro::launch_diff<IMEX_F16DEV, IMEX_F32>(fa, pull_a, fb, pull_b, g, res, s);
    default: return macro::launch_diff<IMEX_F16DEV, IMEX_F16DEV>(fa, pull_a, fb, pull_b, g, res, s);
    }
}

cudaError_t launch_conserved_lowp(int prec, bool pull, const void* src, const Geom& g, void* partial, unsigned* ticket,
                                  const unsigned long long* status, double* out, cudaStream_t s)
{
    return prec == IMEX_F32 ? cons::launch<IMEX_F32, 3>(pull, src, g, partial, ticket, status, out, s)
                            : cons::launch<IMEX_F16DEV, 3>(pull, src, g, partial, ticket, status, out, s);
}

size_t conserved_scratch_bytes(const Geom& g)
{
    return cons::blocks_for((size_t)g.nx * g.ny * g.nz, current_sm_count(), cons::kMostPerSm) * sizeof(cons::Partial);
}

}  // namespace imex

// Two float32 steps per launch (two_f32.cuh): plans, tensor maps and the
// one-lattice kernel.
#include <algorithm>
#include <atomic>
#include <new>
#include <utility>
#include <vector>

#include "two_f32.cuh"
#include "two_f32.hpp"

namespace imex {
namespace two {

namespace {

template <bool kPadded>
__global__ void __launch_bounds__(kThreads, 1)
    k_two_f32(const __grid_constant__ Maps maps, const float* __restrict__ src, float* __restrict__ dst, Geom g, Plan p,
              CollideF32 cp, WaitCtl wc)
{
    extern __shared__ __align__(128) unsigned char smem[];
    chain_next();
    run_box<false, kPadded>(&maps, src, dst, g.nx, g.ny, g.nz, kPadded ? (size_t)g.nx * g.ny * pitch_of(g.nz) : g.plane,
                           box_of(p, g.nx, g.ny, g.nz, blockIdx.x), cp, smem, wc);
}

// One fused step between the layouts, two cells a thread (flat_lowp.cuh's
// separate pairs: neither layout's rows are 8-byte aligned in every direction).
constexpr int kEdgeThreads = 128;
template <bool kOut>
__global__ void __launch_bounds__(kEdgeThreads) k_edge_f32(const float* src, float* __restrict__ dst, Geom g,
                                                           CollideF32 cp)
{
    using S = lowp::Storage<IMEX_F32>;
    using A = lowp::F2;
    chain_begin<true>();
    const unsigned cells = (unsigned)g.plane, c0 = blockIdx.x * (2 * kEdgeThreads) + threadIdx.x;
    if (c0 >= cells) return;
    const bool two = c0 + kEdgeThreads < cells;
    const unsigned c1 = two ? c0 + kEdgeThreads : c0;
    const int pitch = pitch_of(g.nz);
    const size_t padded = (size_t)g.nx * g.ny * pitch, from = kOut ? padded : g.plane, to = kOut ? g.plane : padded;
    const FlatPull p0(g.nx, g.ny, g.nz, c0, kOut ? pitch : g.nz), p1(g.nx, g.ny, g.nz, c1, kOut ? pitch : g.nz);
    float2 h[kQ];
#pragma unroll
    for (int a = 0; a < kQ; ++a) {
        const float* p = src + (size_t)a * from;
        h[a] = make_float2(S::dev(load_state(p + p0.at(a)), a), S::dev(load_state(p + p1.at(a)), a));
    }
    lowp::collide_dev<IMEX_F32, A>(h, cp);
    if (kOut) {
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
            dst[(size_t)a * to + c0] = S::store(h[a].x, a);
            if (two) dst[(size_t)a * to + c1] = S::store(h[a].y, a);
        }
        return;
    }
    auto put = [&](unsigned c, bool second) {
        const unsigned row = c / (unsigned)g.nz;
        const int z = (int)(c - row * (unsigned)g.nz);
        const bool copy = z == 0 && (g.nz & 1);
        float* const o = dst + (size_t)row * pitch + z;
#pragma unroll
        for (int a = 0; a < kQ; ++a) {
            const float v = S::store(second ? h[a].y : h[a].x, a);
            o[(size_t)a * to] = v;
            if (copy) o[(size_t)a * to + g.nz] = v;
        }
    };
    put(c0, false);
    if (two) put(c1, true);
}

using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                            const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled of the driver, through the runtime (the library
// links no driver library).
Encode encode_fn()
{
    static std::atomic<void*> fn{nullptr};
    void* f = fn.load();
    if (!f) {
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess)
            f = nullptr;
        fn.store(f);
    }
    return reinterpret_cast<Encode>(f);
}

// Iterations a CTA spends beside its planes: the pipeline's 3 and the set-up.
constexpr int kExtra = 5;
// Planes of a brief part at least.
constexpr int kLeastPart = 4;

// Iterations until the last SM is done, one CTA each at a time, taken in order by
// the SM free first.
int iterations(const Geom& g, const Plan& p, int sms)
{
    std::vector<std::pair<int, int>> free{{0, sms}}, next;  // (time, SMs), in order of time
    int end = 0;
    for (int c = 0; c < p.chunks; ++c) {
        const int len = p.begin(c + 1, g.nx) - p.begin(c, g.nx) + kExtra;
        int left = p.nty * p.ntz;
        while (left > 0) {
            const int n = std::min(left, free[0].second), t = free[0].first + len;
            left -= n;
            next.clear();
            if (free[0].second > n) next.emplace_back(free[0].first, free[0].second - n);
            bool in = false;
            for (size_t q = 1; q < free.size(); ++q) {
                if (!in && t <= free[q].first) {
                    in = true;
                    if (t == free[q].first) {
                        next.emplace_back(t, free[q].second + n);
                        continue;
                    }
                    next.emplace_back(t, n);
                }
                next.push_back(free[q]);
            }
            if (!in) next.emplace_back(t, n);
            free.swap(next);
            end = std::max(end, t);
        }
    }
    return end;
}

Plan tiles_of(const Geom& g)
{
    Plan p = {};
    // full tiles and one narrower: every full tile's rows are whole 128-byte
    // lines where nz is a multiple of 32 values, and of 16 bytes always (evened
    // out, 4 x 28 for 112, each row took two lines: 112^3 43.2 us a step, now 35.8)
    p.tz = kTileZ;
    p.ntz = (g.nz + kTileZ - 1) / kTileZ;
    p.nty = (g.ny + kTileY - 1) / kTileY;
    p.ty = (g.ny + p.nty - 1) / p.nty;
    p.chunks = 1;
    return p;
}

// The tiles cut along x so that the last SM is done soonest: in even parts, or in
// even ones and up to three brief ones that fill the SMs left over in the end.
// The parts of neighbouring tiles begin and end at the same planes: they share
// rows and sectors, and read them once while they march together (cut so that
// every SM has the same number of planes, 256^3 takes 514 us a step).  Even
// parts alone -> with brief ones: 256^3 (399 iterations, 376) 337 -> 317 us a
// step, 128^3 (62, 56) 50.9 -> 47.1, 96^3 (25, 25) 20.7 as before.
Plan plan_for(const Geom& g, int sms)
{
    Plan best = tiles_of(g);
    if (best.nty * best.ntz > 32 * sms) return best;  // no last wave to speak of
    int least = iterations(g, best, sms);
    auto offer = [&](const Plan& p) {
        const int n = iterations(g, p, sms);
        if (n < least) {
            least = n;
            best = p;
        }
    };
    Plan p = best;
    for (p.chunks = 2; p.chunks <= std::min(g.nx, 32); ++p.chunks) offer(p);
    for (p.briefs = 1; p.briefs <= 3; ++p.briefs)
        for (int evens = 1; evens <= 6; ++evens) {
            p.chunks = evens + p.briefs;
            for (p.brief = kLeastPart; p.brief * p.chunks < g.nx; ++p.brief) offer(p);
        }
    return best;
}

cudaError_t encode_maps(const float* buf, const Geom& g, const Plan& p, bool padded, Maps* out)
{
    const Encode f = encode_fn();
    if (!f) return cudaErrorNotSupported;
    const cuuint64_t row = (cuuint64_t)(padded ? pitch_of(g.nz) : g.nz);
    const cuuint64_t dims[3] = {row, (cuuint64_t)g.ny, (cuuint64_t)kQ * g.nx};
    const cuuint64_t strides[2] = {row * 4, row * g.ny * 4};
    const cuuint32_t step[3] = {1, 1, 1};
    for (int q = 0; q < kMaps; ++q) {
        // fewer rows than one: never used, a valid box all the same
        const cuuint32_t box[3] = {(cuuint32_t)kTileZ, (cuuint32_t)std::max(1, p.ty + 2 - q), 1};
        if (f(&out->m[q], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(buf), dims, strides, box, step,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}

}  // namespace

bool eligible(const Geom& g)
{
    return g.nz % 4 == 0 && g.nz >= kTileZ && g.ny >= 4 && g.nx >= 4 && g.plane < (1ull << 32) / kQ;
}

bool padded_eligible(const Geom& g)
{
    return g.nz % 4 != 0 && g.nz >= kTileZ && g.ny >= 4 && g.nx >= 4 && padded_plane(g) < (1ull << 32) / kQ;
}

int item_iterations(const Geom& g, const Plan& p) { return (g.nx + p.chunks - 1) / p.chunks + kExtra; }

Plan plan_tiles(const Geom& g, int planes)
{
    Plan p = tiles_of(g);
    p.chunks = std::max(1, (g.nx + planes / 2) / planes);
    return p;
}

// Measured: two steps in one launch take 1.5 us and 1.65 us per iteration of
// the busiest SM (96^3 41 us, 128^3 94, 256^3 635), in two launches of the
// one-step kernel cells / 31 per ns each (96^3 59 us, 128^3 134, 256^3 1034;
// below 80^3 less, the lattice then stays in L2: 80^3 28 us against 35). So
// small lattices, whose tiles leave SMs idle or spend most iterations filling
// the pipeline, and shapes that fit the tiles badly keep one step per launch;
// the line lies near 85^3.  Padded layout, single -> two steps, us a step: 255^3
// 546 -> 343, 131 x 128 x 128 68.8 -> 57.0, 97 x 150 x 121 (four tiles for
// three and a value) 59.1 -> 52.4, 111^3 48.5 -> 38.9, 85^3 20.3 -> 19.9 (not taken),
// 65 x 160 x 160 54.0 -> 53.8.
bool worth_alone(const Geom& g, int sms)
{
    if (!eligible(g) && !padded_eligible(g)) return false;
    const bool plain = eligible(g);
    const double singles = 2.0 * (double)g.plane * (plain ? kCellUs : kPaddedCellUs);
    auto beats = [&](double its) {
        return kLaunchUs + (plain ? kIterationUs : kPaddedIterationUs) * its < 0.97 * singles;
    };
    // no plan has fewer iterations than all the tiles' spread evenly (imex_create asks: the plan takes 40 us)
    const Plan t = tiles_of(g);
    const double least = std::max<double>(1 + kExtra, (double)t.nty * t.ntz * (g.nx + kExtra) / sms);
    return beats(least) && beats((double)iterations(g, plan_for(g, sms), sms));
}

void cut_alone(Lattice* l, const Geom& g)
{
    l->plan = plan_for(g, current_sm_count());
    l->cut = true;
}

cudaError_t make_lattice(const float* buf0, const float* buf1, const Geom& g, LatticePtr* out)
{
    LatticePtr l(new (std::nothrow) Lattice);
    if (!l) return cudaErrorMemoryAllocation;
    l->plan = tiles_of(g);
    l->padded = !eligible(g);
    cudaError_t e = encode_maps(buf0, g, l->plan, l->padded, &l->maps[0]);
    if (e == cudaSuccess) e = encode_maps(buf1, g, l->plan, l->padded, &l->maps[1]);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(l->padded ? k_two_f32<true> : k_two_f32<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSmemBytes);
    if (e == cudaSuccess) *out = std::move(l);
    return e;
}

cudaError_t launch(const Lattice& l, int from, const float* src, float* dst, const Geom& g, const CollideF32& cp,
                   unsigned* err, cudaStream_t s)
{
    return launch_chained(l.padded ? k_two_f32<true> : k_two_f32<false>, (unsigned)l.plan.items(), kThreads, kSmemBytes, s,
                          l.maps[from], src, dst, g, l.plan, cp, make_wait_ctl(err));
}

cudaError_t launch_edge(bool out, const float* src, float* dst, const Geom& g, const CollideF32& cp, cudaStream_t s)
{
    const unsigned grid = (unsigned)((g.plane + 2 * kEdgeThreads - 1) / (2 * kEdgeThreads));
    return launch_chained(out ? k_edge_f32<true> : k_edge_f32<false>, grid, kEdgeThreads, 0, s, src, dst, g, cp);
}

}  // namespace two
}  // namespace imex

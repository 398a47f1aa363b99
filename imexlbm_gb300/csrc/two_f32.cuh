// Two fused float32 steps in one pass over memory.
//
// Why.  A float32 step is bound by memory: 27 values read and written per
// cell, 102% of the copy bandwidth at 256^3 with the float32 pipe 30% busy.
// Here a CTA marches along x over a (y, z) tile and keeps the state between
// the two steps in shared memory, so memory moves one read and one write per
// two steps.  256^3: 1048 us per two steps -> 635 (52.8 GLUPS where the copy
// bandwidth allows 31 of one step); 128^3: 134 -> 94.  Bound now: 85% of the
// copy bandwidth, then the packed float32 pipe (304 two-cell operations a
// pair of cells and step) and the latency of a plane's phases.
//
// Order.  Iteration i of a tile:
//   loaders (3 warps)  bring the 27 pulled sources of middle plane i + 2
//                      (x = x0 - 1 + i + 2) into one of two stages;
//   A (7 warps)        collide middle plane i (the tile and one cell around
//                      it) from its stage: the first step, stored - as the
//                      float32 values a step would store - in the ring;
//   B (5 warps)        pull plane i - 2 from the ring (ex = -1 values of middle
//                      plane i - 1, ex = 0 of i - 2, ex = +1 of i - 3),
//                      collide, and store the second step's values.
// So loading, the first and the second step of different planes overlap. The
// ring holds 1 plane of the ex = -1 values, 2 of ex = 0 and 3 of ex = +1: A
// stores plane i over the values B has read at the start of the iteration
// (barrier 1), and barrier 0 ends the iteration.  A stage is handed over by
// mbarriers (full: the copies' bytes and the loaders' arrivals; empty: one
// arrival per A warp).  The results are those of two single steps, bit for
// bit: the cell arithmetic is lowp::collide_dev on two z-neighbours at a time.
//
// Tile.  32 z cells x 10 rows of destinations at most: 34 x 12 middle cells,
// 1.275 times the work of the first step.  12 working warps put 3 on each of the SM's four
// schedulers; 2 loader warps measured 703 us, 4 691; 12 rows (8 + 6 warps, 4 on two
// of the schedulers) 774, 13 rows with the ex = -1, 0, +1 ring one plane deeper each (no barrier
// 1) and a single stage 835.  Half the time of the first versions was the
// loads: 34-float rows through L1 (ld or 4-byte cp.async) have too little of
// L1 left beside 220 KB of shared memory (1290 us), 16-byte cp.async writes
// shared memory a sector at a time (917), a tensor copy of 40-float rows
// costs three 128-byte requests per row, 2.5 clocks each (956).  So the 32 aligned values
// of a row come as tensor copies (one 128-byte request a row, each direction's box
// issued by its own lane), and the 4 values left and right of it as 16-byte
// cp.async, for the directions that need them.
//
// Edges.  x wraps through the box's coordinate, the side pieces through their
// addresses; rows that wrap in y are left out of the box (tensor maps of ty +
// 2 down to ty - 1 rows) and copied one by one.
//
// Requirements (eligible): nz a multiple of 4 (16-byte pieces and tensor
// strides), nz >= 32, ny >= 4, nx >= 4, 27 * cells below 2^32.  Other nz >= 32:
// the padded layout, in which rows lie a multiple of 8 values apart.  A run's
// first and last steps are single ones there (k_edge_f32), from the plain layout
// and back to it.  An odd row's last pair computes z = nz, which is z = 0 once
// more, and stores it behind the row, where the next launch's boxes read it;
// of the pieces that wrap, those off a 16-byte boundary come as two values.
// (Copies of all the cells that wrap, stored behind both ends by B's edge
// threads, kept every load whole and cost B up to twice its time: 255^3 459 us a step.)
#pragma once

#include <cuda_runtime.h>

#include "bulk.cuh"
#include "kernels_common.cuh"
#include "lowp_math.cuh"
#include "two_f32.hpp"

namespace imex {
namespace two {

constexpr int kThreadsA = 224, kThreadsB = 160, kThreadsL = 96;
constexpr int kThreads = kThreadsA + kThreadsB + kThreadsL;
constexpr int kTileZ = 32;                   // staged values of a row, destination columns at most
constexpr int kTileY = 10;                   // destination rows of a tile at most
constexpr int kRows = kTileY + 2;            // middle rows
constexpr int kMid = kRows * (kTileZ + 2);   // middle cells of a plane
constexpr int kStage = kRows * (kTileZ + 8);  // staged values of a direction: rows, then 2 x 4 side values a row
constexpr int kRing = 9 * (1 + 2 + 3);       // ring arrays of kMid values
constexpr int kSide = 5;                     // side pieces of a loader thread
constexpr int kLoadWarps = kThreadsL / 32;
constexpr unsigned kTwoValues = 1u << 29;    // mark of a side piece of two values
static_assert(kMid / 2 <= kThreadsA && kTileY * kTileZ / 2 <= kThreadsB, "one pair of cells per thread");
static_assert(36 * kRows <= kSide * kThreadsL, "side pieces");
static_assert(kStage * 4 % 128 == 0 && kMid % 2 == 0, "128-byte aligned boxes, 8-byte pairs");
static_assert(kLoadWarps * 32 >= kQ, "a loader thread per direction");

// Shared memory: two stages, the ring, four mbarriers and a flag.
constexpr size_t kDataBytes = (size_t)(2 * kQ * kStage + kRing * kMid) * sizeof(float);
constexpr size_t kSmemBytes = kDataBytes + 64;
static_assert(kSmemBytes <= 227 * 1024, "shared memory of a CTA");

// One CTA's destinations.
struct Box {
    int x0, planes, y0, rows, z0, cols;
    int box_rows;  // rows of maps->m[0]'s box (ty + 2)
};

__device__ __forceinline__ Box box_of(const Plan& p, int nx, int ny, int nz, int item)
{
    const int tiles = p.nty * p.ntz, chunk = item / tiles, t = item - chunk * tiles;
    const int iy = t / p.ntz, iz = t - iy * p.ntz;
    Box b;  // part i of n balanced parts of a length starts at i * length / n
    b.x0 = p.begin(chunk, nx);
    b.planes = p.begin(chunk + 1, nx) - b.x0;
    b.y0 = (int)((long long)iy * ny / p.nty);
    b.rows = (int)((long long)(iy + 1) * ny / p.nty) - b.y0;
    b.z0 = iz * p.tz;
    b.cols = ((iz + 1 == p.ntz ? nz : b.z0 + p.tz) - b.z0 + 1) & ~1;  // odd: the last one is z = 0 once more
    b.box_rows = p.ty + 2;
    return b;
}

__device__ __forceinline__ int wrap(int v, int n) { return v < 0 ? v + n : v >= n ? v - n : v; }

// Direction with velocity (x, y, z), and a component of a direction that is
// not a compile-time constant.
__device__ __forceinline__ int dir_of(int x, int y, int z)
{
    int d = 0;
#pragma unroll
    for (int a = 0; a < kQ; ++a)
        if (ex(a, 0) == x && ex(a, 1) == y && ex(a, 2) == z) d = a;
    return d;
}
__device__ __forceinline__ int ex_rt(int a, int dim)
{
    int e = 0;
#pragma unroll
    for (int q = 0; q < kQ; ++q)
        if (q == a) e = ex(q, dim);
    return e;
}

template <int ID, int N>
__device__ __forceinline__ void bar_sync()
{
    asm volatile("barrier.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void bar_arrive()
{
    asm volatile("barrier.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* mbar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bulk::smem_u32(mbar)) : "memory");
}
__device__ __forceinline__ void tma_load(void* dst, const CUtensorMap* map, int z, int y, int x, uint64_t* mbar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            bulk::smem_u32(dst)),
        "l"(map), "r"(z), "r"(y), "r"(x), "r"(bulk::smem_u32(mbar))
        : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(bulk::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(bulk::smem_u32(dst)), "l"(src) : "memory");
}

// The two-step march of one box of the lattice at src into dst.  kMapsInMemory:
// the tensor maps lie in global memory (a batch's table) rather than in the
// kernel's parameters.  Every wait
// on an mbarrier is bounded: one that runs out sets wc.err, the loaders stop
// bringing planes, and the CTA runs to its end on what the stages hold (its
// results are reported invalid).  The set-up before the roles' loops touches
// no lattice, so each role waits for the kernels before (chain_wait) only then;
// the caller has let the next kernel in.  kPadded: both buffers in the
// padded layout (two_f32.hpp), `plane` the values of a direction there.
template <bool kMapsInMemory, bool kPadded>
__device__ __forceinline__ void run_box(const Maps* __restrict__ maps, const float* __restrict__ src,
                                        float* __restrict__ dst, int nx, int ny, int nz, size_t plane, const Box& b,
                                        const CollideF32& cp, unsigned char* smem, const WaitCtl& wc)
{
    using S = lowp::Storage<IMEX_F32>;
    using A2 = lowp::F2;
    float* const stages = reinterpret_cast<float*>(smem);
    float* const ring = stages + 2 * kQ * kStage;
    uint64_t* const full = reinterpret_cast<uint64_t*>(smem + kDataBytes);
    uint64_t* const empty = full + 2;
    volatile int* const failed = reinterpret_cast<volatile int*>(full + 4);
    const int half = b.cols >> 1;                 // destination pairs of a row
    const int W = b.cols + 2, R = b.rows + 2;     // middle cells of a row, middle rows
    const int side0 = b.box_rows * kTileZ;        // a direction's side pieces follow its rows
    const int pitch = kPadded ? pitch_of(nz) : nz;
    const unsigned sheet = (unsigned)ny * (unsigned)pitch;
    const int last = b.planes + 2;                // middle planes
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; ++q) {
            bulk::mbar_init(full + q, kQ + kThreadsL);
            bulk::mbar_init(empty + q, kThreadsA / 32);
        }
        *failed = 0;
        bulk::fence_mbar_init();
    }
    __syncthreads();

    if (threadIdx.x >= kThreadsA + kThreadsB) {
        const int lid = threadIdx.x - (kThreadsA + kThreadsB);
        // Thread `dir` brings direction dir's rows of a plane.
        const int dir = (lid & 31) * kLoadWarps + (lid >> 5);
        const bool on = dir < kQ;
        const int ey = ex_rt(on ? dir : 0, 1), exd = ex_rt(on ? dir : 0, 0);
        const int ylo = b.y0 - 1 - ey, top = ylo < 0 ? -ylo : 0, bot = ylo + R > ny ? ylo + R - ny : 0;
        // the box ends with the tile's rows where the next would wrap, and
        // with the map's otherwise (a tile one row short brings one too many)
        const int rows = bot ? R - top - bot : b.box_rows - top;
        const CUtensorMap* const map = &maps->m[b.box_rows - rows];
        if constexpr (kMapsInMemory)  // written through the generic proxy (an upload before the launch)
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
        const uint32_t row_bytes = (((uint32_t)b.cols + 3u) & ~3u) * 4u;
        const uint32_t my_bytes = (uint32_t)rows * (kTileZ * 4u) + (uint32_t)(top + bot) * row_bytes;
        unsigned from[kSide], at[kSide];
#pragma unroll
        for (int q = 0; q < kSide; ++q) {
            const int p = lid + q * kThreadsL;
            at[q] = 0xffffffffu;
            from[q] = 0;
            if (p >= 36 * R) continue;
            // left for ez = 0 and +1 (18 directions), right for ez = 0 and -1
            const int k = p / R, r = p - k * R, right = k >= 18, kk = k - 18 * right, c9 = kk >> 1;
            const int a = dir_of(c9 / 3 - 1, c9 % 3 - 1, (kk & 1) ? (right ? -1 : 1) : 0);
            const int y = b.y0 - 1 + r - ex_rt(a, 1), z = right ? b.z0 + b.cols : b.z0 - 4;
            from[q] = (unsigned)(a * plane) + (unsigned)wrap(y, ny) * (unsigned)pitch + (unsigned)wrap(z, nz);
            at[q] = (unsigned)(a * kStage + side0 + r * 8 + 4 * right) | ((unsigned)(ex_rt(a, 0) + 1) << 30);
            // a piece that wraps off its 16-byte boundary: only the two values used
            // of it, z = nz - 2 and nz - 1 on the left, 1 and 2 on the right of an odd row
            if (kPadded && (z < 0 || z > nz)) {
                at[q] = (at[q] + (right ? 0 : 2)) | kTwoValues;
                from[q] += right ? 0 : 2;
            }
        }
        auto bring = [&](int i) {  // middle plane i into stage i & 1
            const int x = wrap(b.x0 - 1 + i, nx);
            const int xs[3] = {x + 1 == nx ? 0 : x + 1, x, x == 0 ? nx - 1 : x - 1};  // [ex + 1]
            float* const stage = stages + (i & 1) * (kQ * kStage);
            uint64_t* const mb = full + (i & 1);
            bulk::fence_proxy_async_smem();
            if (on) {
                const int xd = exd == -1 ? xs[0] : exd == 0 ? xs[1] : xs[2];
                float* const to = stage + dir * kStage;
                bulk::mbar_arrive_expect_tx(mb, my_bytes);
                if (i > 0 || (int)blockIdx.x != wc.starve_cta) {  // test hook: the first plane never arrives
                    tma_load(to + top * kTileZ, map, b.z0, ylo + top, dir * nx + xd, mb);
                    if (top + bot) {
                        const float* p = src + ((size_t)dir * plane + (size_t)xd * sheet + b.z0);
                        for (int r = 0; r < top; ++r)
                            bulk::copy_g2s(to + r * kTileZ, p + (size_t)(ylo + r + ny) * pitch, row_bytes, mb);
                        for (int r = R - bot; r < R; ++r)
                            bulk::copy_g2s(to + r * kTileZ, p + (size_t)(ylo + r - ny) * pitch, row_bytes, mb);
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < kSide; ++q)
                if (at[q] != 0xffffffffu) {
                    const unsigned e = at[q] >> 30;
                    float* const t = stage + (at[q] & (kTwoValues - 1));
                    const float* const f = src + ((size_t)from[q] + (size_t)(e == 0 ? xs[0] : e == 1 ? xs[1] : xs[2]) * sheet);
                    if (kPadded && (at[q] & kTwoValues)) {
                        cp4(t, f);
                        cp4(t + 1, f + 1);
                    } else {
                        cp16(t, f);
                    }
                }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bulk::smem_u32(mb)) : "memory");
        };
        chain_wait();
        int brought = 0;
        bool good = true;
        for (int i = 0; i < last; ++i) {
            if (i >= 2) {  // plane i - 2 read
                good = bulk::mbar_wait(empty + (i & 1), (uint32_t)((i >> 1) & 1) ^ 1u, wc.cycles) && !*failed;
                if (__any_sync(0xffffffffu, !good)) break;
            }
            bring(i);
            brought = i + 1;
        }
        // the copies must be over before the CTA's shared memory is another's
        for (int i = brought > 2 ? brought - 2 : 0; i < brought; ++i)
            if (!bulk::mbar_wait(full + (i & 1), (uint32_t)((i >> 1) & 1), wc.cycles)) atomicOr(wc.err, 1u);
        return;
    }

    if (threadIdx.x < kThreadsA) {
        const int tid = threadIdx.x;
        const bool on = tid < (half + 1) * R;
        int pa, pb;  // staged values z - 1, z and z + 1, z + 2 of the middle pair z, z + 1 with z = z0 - 1 + 2 q
        {
            const int m = on ? tid : 0, r = m / (half + 1), q = m - r * (half + 1);
            pa = q == 0 ? side0 + r * 8 + 2 : r * kTileZ + 2 * q - 2;
            pb = q == half ? side0 + r * 8 + 4 : r * kTileZ + 2 * q;
        }
        chain_wait();
        bool good = true;
        int s2 = 0, s3 = 0;  // ring slots of this plane's ex = 0 and ex = +1 values
        for (int i = 0; i < last + 1; ++i) {
            if (i < last) {
                if (good && !bulk::mbar_wait(full + (i & 1), (uint32_t)((i >> 1) & 1), wc.cycles)) {
                    good = false;
                    *failed = 1;
                    atomicOr(wc.err, 1u);
                }
                float2 h[kQ];
                const float* const stage = stages + (i & 1) * (kQ * kStage);
                if (on) {
#pragma unroll
                    for (int a = 0; a < kQ; ++a) {
                        const float* v = stage + a * kStage;
                        if (ex(a, 2) == 0) h[a] = make_float2(v[pa + 1], v[pb]);
                        else h[a] = *reinterpret_cast<const float2*>(v + (ex(a, 2) == 1 ? pa : pb));
                    }
                }
                __syncwarp();
                if ((tid & 31) == 0) mbar_arrive(empty + (i & 1));  // the warp has read its part of the stage
                if (on) {
#pragma unroll
                    for (int a = 0; a < kQ; ++a) h[a] = A2::add(h[a], A2::splat(-(float)weight(a)));
                    lowp::collide_dev<IMEX_F32, A2>(h, cp);
                }
                bar_sync<1, kThreadsA + kThreadsB>();  // B has read what the stores below overwrite
                if (on) {
#pragma unroll
                    for (int a = 0; a < kQ; ++a) {
                        const int k = (ex(a, 1) + 1) * 3 + ex(a, 2) + 1;
                        const int slot = ex(a, 0) == -1 ? k : ex(a, 0) == 0 ? (9 + k) + 9 * s2 : (27 + k) + 9 * s3;
                        *reinterpret_cast<float2*>(ring + slot * kMid + 2 * tid) =
                            make_float2(S::store(h[a].x, a), S::store(h[a].y, a));
                    }
                }
            } else {
                bar_sync<1, kThreadsA + kThreadsB>();
            }
            bar_sync<0, kThreadsA + kThreadsB>();
            s2 ^= 1;
            s3 = s3 == 2 ? 0 : s3 + 1;
        }
        return;
    }

    const int tid = threadIdx.x - kThreadsA;
    const bool on = tid < half * b.rows;
    int pos;  // the destination pair's place in the middle plane, one column left of it
    unsigned to;
    {
        const int m = on ? tid : 0, r = m / half, q = m - r * half;
        pos = (r + 1) * W + 2 * q;
        to = (unsigned)(b.y0 + r) * (unsigned)pitch + (unsigned)(b.z0 + 2 * q);
    }
    chain_wait();
    int s2 = 0, s3 = 0;  // slots of middle planes i - 2 (ex = 0) and i - 3 (ex = +1): those plane i is about to take
    for (int i = 0; i < last + 1; ++i) {
        float2 h[kQ];
        const bool run = i >= 3 && on;
        if (run) {
#pragma unroll
            for (int a = 0; a < kQ; ++a) {
                const int k = (ex(a, 1) + 1) * 3 + ex(a, 2) + 1;
                const int slot = ex(a, 0) == -1 ? k : ex(a, 0) == 0 ? (9 + k) + 9 * s2 : (27 + k) + 9 * s3;
                const float* v = ring + slot * kMid - ex(a, 1) * W + pos;
                if (ex(a, 2) == 0) h[a] = make_float2(v[1], v[2]);
                else h[a] = *reinterpret_cast<const float2*>(v + (ex(a, 2) == 1 ? 0 : 2));
            }
#pragma unroll
            for (int a = 0; a < kQ; ++a) h[a] = A2::add(h[a], A2::splat(-(float)weight(a)));
        }
        bar_arrive<1, kThreadsA + kThreadsB>();
        if (run) {
            lowp::collide_dev<IMEX_F32, A2>(h, cp);
            float* const d = dst + (size_t)(b.x0 + i - 3) * sheet + to;
#pragma unroll
            for (int a = 0; a < kQ; ++a)
                __stcs(reinterpret_cast<float2*>(d + (size_t)a * plane), make_float2(S::store(h[a].x, a), S::store(h[a].y, a)));
        }
        bar_sync<0, kThreadsA + kThreadsB>();
        s2 ^= 1;
        s3 = s3 == 2 ? 0 : s3 + 1;
    }
}

}  // namespace two
}  // namespace imex

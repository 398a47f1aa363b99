// Shared device code: lattice geometry, periodic pull gather, block
// reductions.  Used by every engine's kernels.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

#include "d3q27.cuh"

namespace imex {

// Lattice of nx*ny*nz cells stored as f[a][x][y][z], z fastest; one
// direction plane holds nx*ny*nz values.
struct Geom {
    int nx, ny, nz;
    size_t plane;
};

// Threads of the step kernels: one block covers `kStepBlock` consecutive z
// cells of one (x, y) row; grid = (ceil(nz / kStepBlock), ny, nx).
constexpr int kStepBlock = 128;

// SM count of the calling thread's current device, for persistent grids.
// Queried per call: the runtime answers from its own cache, and a process
// that drives several devices gets each one's count.
inline int current_sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) return 1;
    return sms;
}

// Chained launches: the kernels of a run of steps are launched with
// programmatic stream serialization, so that a kernel's CTAs may take their
// places while the one before it in the stream still runs, and only the
// launch's own latency overlaps: 1.5 to 3 us a step (float32
// 32^3 4.1 -> 2.3 us, 64^3 8.4 -> 6.5; float64 32^3 6.2 -> 4.6, 64^3 22.6 -> 20.0,
// 131 x 77 x 90 69.5 -> 66.3; float16 64^3 8.8 -> 6.6).
//
// Every thread of such a kernel calls chain_begin before its first access to
// memory and before any return: it waits until the kernels before have
// completed and their stores are visible (a kernel that completed without
// waiting would let the one after it overtake the one before).  The kernel
// exists while the one before still writes, so what it reads of a lattice it
// reads by load_state, tensor or bulk copies.  chain_end
// comes once its sources are read.  Where the CTAs take turns on the SMs
// (early) the next kernel is let in at the beginning: its CTAs come up as
// these finish.  Where all CTAs run at once it is let in at the end: let in
// earlier, its CTAs pile up on whichever SMs have room and run unevenly
// (float64 32^3 7.8 us; the late form, even as an untaken branch, costs 256^3 1%).
// The batch's segment kernel is launched plainly (chained 32.2 GLUPS, plainly 33.2).
template <class... Params, class... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                  Args... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// Whether a grid of `threads` threads runs in turns on SMs that hold `resident` of them.
inline bool chain_early(unsigned long long threads, unsigned resident)
{
    return threads > (unsigned long long)resident * (unsigned)current_sm_count();
}

__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <bool EARLY>
__device__ __forceinline__ void chain_begin()
{
    if (EARLY) chain_next();
    chain_wait();
}
template <bool EARLY>
__device__ __forceinline__ void chain_end()
{
    if (!EARLY) chain_next();
}

// Load of lattice state.  An ordinary cached load: the read-only path (__ldg, and what the
// compiler may take for a const __restrict__ pointer) is for memory that nothing
// writes as long as the kernel exists, which does not hold for a chained one.
template <class T>
__device__ __forceinline__ T load_state(const T* p)
{
    return __ldca(p);
}

// Source indices of the pull for cell (i, j, k): the value streaming into
// the cell along direction a comes from (i - ex, j - ey, k - ez), wrapped
// periodically.  This is the one-rank image of the reference's ghost layer
// (src/mpi_view_transfer.cpp:260-456 fills ghost cells with the periodic
// image; src/lbm.cpp:194-195 pulls from x - e).
struct PullIndex {
    size_t row[3][3];  // [ex + 1][ey + 1] -> offset of source row (x, y)
    int zk[3];         // [ez + 1] -> source z

    __device__ __forceinline__ PullIndex(const Geom& g, int i, int j, int k, bool pull)
    {
        const int im = i == 0 ? g.nx - 1 : i - 1, ip = i == g.nx - 1 ? 0 : i + 1;
        const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
        const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
        // ex = +1 pulls from x - 1, ex = -1 from x + 1.
        const int xs[3] = {pull ? ip : i, i, pull ? im : i};
        const int ys[3] = {pull ? jp : j, j, pull ? jm : j};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)
                row[a][b] = ((size_t)xs[a] * g.ny + ys[b]) * g.nz;
        zk[0] = pull ? kp : k;
        zk[1] = k;
        zk[2] = pull ? km : k;
    }

    template <int A>
    __device__ __forceinline__ size_t at(const Geom& g) const
    {
        return (size_t)A * g.plane + row[ex(A, 0) + 1][ex(A, 1) + 1] + zk[ex(A, 2) + 1];
    }

    // Same for a direction that is a compile-time constant only after
    // unrolling.
    __device__ __forceinline__ size_t at_dyn(const Geom& g, int a) const
    {
        return (size_t)a * g.plane + row[ex(a, 0) + 1][ex(a, 1) + 1] + zk[ex(a, 2) + 1];
    }
};

// The same for a cell given by its flat index (z fastest) in a lattice of
// fewer than 2^32 cells: the source offset within a direction's plane is the
// sum of a part for each of ex, ey and ez ([e + 1]).
struct FlatPull {
    unsigned x[3], y[3], z[3];
    __device__ __forceinline__ FlatPull(int nx, int ny, int nz, unsigned cell) : FlatPull(nx, ny, nz, cell, nz) {}
    // rows `pitch` values apart
    __device__ __forceinline__ FlatPull(int nx, int ny, int nz, unsigned cell, int pitch)
    {
        const unsigned row = cell / (unsigned)nz, k = cell - row * (unsigned)nz;
        const unsigned i = row / (unsigned)ny, j = row - i * (unsigned)ny;
        const unsigned sheet = (unsigned)ny * (unsigned)pitch;
        x[0] = (i == (unsigned)nx - 1 ? 0 : i + 1) * sheet;
        x[1] = i * sheet;
        x[2] = (i == 0 ? (unsigned)nx - 1 : i - 1) * sheet;
        y[0] = (j == (unsigned)ny - 1 ? 0 : j + 1) * (unsigned)pitch;
        y[1] = j * (unsigned)pitch;
        y[2] = (j == 0 ? (unsigned)ny - 1 : j - 1) * (unsigned)pitch;
        z[0] = k == (unsigned)nz - 1 ? 0 : k + 1;
        z[1] = k;
        z[2] = k == 0 ? (unsigned)nz - 1 : k - 1;
    }
    __device__ __forceinline__ unsigned at(int a) const { return x[ex(a, 0) + 1] + y[ex(a, 1) + 1] + z[ex(a, 2) + 1]; }
};

// Unrolled gather of the 27 pulled (or in-place) values.
template <typename T, int A = 0>
__device__ __forceinline__ void gather27(const T* src, const Geom& g, const PullIndex& p, T (&f)[kQ])
{
    if constexpr (A < kQ) {
        f[A] = load_state(src + p.at<A>(g));
        gather27<T, A + 1>(src, g, p, f);
    }
}

// Deterministic block sum of NV doubles: warp shuffle tree, then the warps'
// results in warp order.  Result valid in thread 0.  blockDim.x <= 1024.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* smem /* 32*NV */)
{
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) smem[warp * NV + q] = v[q];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double s = 0.0;
            for (int w = 0; w < nw; ++w) s += smem[w * NV + q];
            v[q] = s;
        }
    }
}

}  // namespace imex

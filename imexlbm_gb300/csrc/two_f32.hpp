// Two float32 steps per launch (two_f32.cuh): host side.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <memory>

#include "kernels_lowp.cuh"

namespace imex {
namespace two {

// Tensor maps of one buffer of a lattice: boxes of ty + 2, ty + 1, ty and
// ty - 1 rows of 32 values.
constexpr int kMaps = 4;
struct alignas(64) Maps {
    CUtensorMap m[kMaps];
};

// How a lattice is cut: nty x ntz tiles of at most ty x tz destinations, each
// marched in `chunks` parts along x, the last `briefs` of `brief` planes and the
// others even.
struct Plan {
    int ty, tz, nty, ntz, chunks, briefs, brief;
    int items() const { return nty * ntz * chunks; }
    // Plane at which part i of nx planes begins.
    __host__ __device__ int begin(int i, int nx) const
    {
        const int evens = chunks - briefs;
        return i > evens ? nx - (chunks - i) * brief : (int)((long long)i * (nx - briefs * brief) / evens);
    }
};

// The padded layout of a lattice whose rows are no multiple of 4 values: within
// a direction, row (x, y) begins at (x ny + y) pitch_of(nz) values, on a 32-byte
// sector; where nz is odd a copy of z = 0 follows z = nz - 1, which completes
// the row's last pair of cells.
__host__ __device__ constexpr int pitch_of(int nz) { return (nz + 8) / 8 * 8; }

// What a lattice handle keeps: its tiles, once it has stepped alone cut for
// that, and the maps of its two buffers (the same whatever the cut along x).
struct Lattice {
    Plan plan;
    bool cut = false;
    bool padded;
    Maps maps[2];
};
using LatticePtr = std::unique_ptr<Lattice>;

// Whether a float32 lattice can take two steps per launch as it lies in
// memory, or else in the padded layout.
bool eligible(const Geom& g);
bool padded_eligible(const Geom& g);
// Values of a direction in the padded layout.
inline size_t padded_plane(const Geom& g) { return (size_t)g.nx * g.ny * pitch_of(g.nz); }
// Whether two steps per launch beat two launches for one lattice alone, as it
// lies or in the padded layout.
bool worth_alone(const Geom& g, int sms);
// An eligible lattice's tiles, cut along x into parts of about `planes` planes.
Plan plan_tiles(const Geom& g, int planes);
// Iterations one item (CTA) of the plan takes.
int item_iterations(const Geom& g, const Plan& p);
// Microseconds: an SM's iteration, a launch, and a float32 cell's step in the
// one-step kernels on the whole GPU (see worth_alone).
constexpr double kIterationUs = 1.65, kLaunchUs = 1.5, kCellUs = 1.0 / 31000.0;
// The same in the padded layout, whose first and last tiles bring twice the
// side pieces, and of the one-step kernel on such rows.
constexpr double kPaddedIterationUs = 1.85, kPaddedCellUs = 1.0 / 30000.0;

// The tiles cut along x for the lattice alone (0.1 ms on the host: not for a
// batch's members, which are cut together).
void cut_alone(Lattice* l, const Geom& g);
cudaError_t make_lattice(const float* buf0, const float* buf1, const Geom& g, LatticePtr* out);
// Two fused steps of one lattice from buffer `from` into the other one.
cudaError_t launch(const Lattice& l, int from, const float* src, float* dst, const Geom& g, const CollideF32& cp,
                   unsigned* err, cudaStream_t s);
// One fused step from the plain into the padded layout, or (out) back.
cudaError_t launch_edge(bool out, const float* src, float* dst, const Geom& g, const CollideF32& cp, cudaStream_t s);

}  // namespace two
}  // namespace imex

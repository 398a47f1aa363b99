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
// marched in `chunks` parts along x.
struct Plan {
    int ty, tz, nty, ntz, chunks;
    int items() const { return nty * ntz * chunks; }
};

// What a lattice handle keeps: its tiles, cut for the lattice alone, and the
// maps of its two buffers (the same whatever the cut along x).
struct Lattice {
    Plan plan;
    Maps maps[2];
};
using LatticePtr = std::unique_ptr<Lattice>;

// Whether a float32 lattice can take two steps per launch at all.
bool eligible(const Geom& g);
// Whether two steps per launch beat two launches for one such lattice alone.
bool worth_alone(const Geom& g, int sms);
// An eligible lattice's tiles, cut along x into parts of about `planes` planes.
Plan plan_tiles(const Geom& g, int planes);
// Iterations one item (CTA) of the plan takes.
int item_iterations(const Geom& g, const Plan& p);
// Microseconds: an SM's iteration, a launch, and a float32 cell's step in the
// one-step kernels on the whole GPU (see worth_alone).
constexpr double kIterationUs = 1.65, kLaunchUs = 1.5, kCellUs = 1.0 / 31000.0;

cudaError_t make_lattice(const float* buf0, const float* buf1, const Geom& g, LatticePtr* out);
// Two fused steps of one lattice from buffer `from` into the other one.
cudaError_t launch(const Lattice& l, int from, const float* src, float* dst, const Geom& g, const CollideF32& cp,
                   unsigned* err, cudaStream_t s);

}  // namespace two
}  // namespace imex

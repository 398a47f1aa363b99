// Two float32 steps per launch (two_f32.cuh): host side.
#pragma once

#include <cuda_runtime.h>

#include <memory>

#include "kernels_lowp.cuh"

namespace imex {
namespace two {

struct Maps;
struct Plan;

// Whether a float32 lattice can take two steps per launch at all.
bool eligible(const Geom& g);
// The tiles of an eligible lattice, marched in the number of x chunks that
// spreads them best over `sms` SMs.
Plan plan_for(const Geom& g, int sms);
// The tiles, each marched in chunks of about `planes` planes.
Plan plan_tiles(const Geom& g, int planes);
// Whether two steps per launch beat two launches for one such lattice alone.
bool worth_alone(const Geom& g, int sms);
// Tensor maps of the lattice's buffer for tiles of plan p.
cudaError_t encode_maps(const float* buf, const Geom& g, const Plan& p, Maps* out);
// Raise the shared-memory limit of a kernel of this file's size once per device.
cudaError_t allow_smem(const void* kernel);

// What a lattice handle keeps: its plan and the maps of its two buffers.
struct Lattice;
struct LatticeDelete {
    void operator()(Lattice* p) const;
};
using LatticePtr = std::unique_ptr<Lattice, LatticeDelete>;
cudaError_t make_lattice(const float* buf0, const float* buf1, const Geom& g, LatticePtr* out);
// Two fused steps from buffer `from` into the other one.
cudaError_t launch(const Lattice& l, int from, const float* src, float* dst, const Geom& g, const CollideF32& cp,
                   unsigned* err, cudaStream_t s);

}  // namespace two
}  // namespace imex

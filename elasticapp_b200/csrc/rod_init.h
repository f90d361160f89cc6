// Initial data of straight rods on the device, and their final state to the
// host (rod_init.cu).  The lists and velocities may be pinned host memory.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "eb_internal.h"

namespace eb {

struct RodSpec {
  double origin[3], step[3];  // node j is at origin + j step
  double rows[9];             // directors of every element
  double area, density, youngs, shear, nu_f, nu_t;
  int64_t start;              // first slot
  int64_t velocity;           // offset (doubles) of 3 x (n + 1) node velocities, or -1
  int32_t n, damped;
  uint32_t rod;               // rod id of the metadata words
  uint32_t pad;
  RodInfo info;               // the rod's table entry
};

// a rod of the device table in a list of rods, and where its results go
struct RodRef {
  int64_t rod;
  double gravity[3];   // of its request (zero: none)
  double* result;      // kStateFields x (n + 1) rows
  double* energies;    // 5 initial values; the final ones at energies + final_at
  int64_t final_at;
};

// writes the state, parameters and metadata of every slot of `count` rods, and
// their entries of the rod table, first slots and element counts (at the rods'
// ids)
cudaError_t launch_rod_init(const RodSpec* specs, int64_t count, const double* velocities, int64_t stride,
                            double* state, double* par, uint32_t* meta, RodInfo* rods, int64_t* rod_start,
                            int32_t* rod_n, cudaStream_t stream);

// writes the listed rods' states and energies (5 values a rod of e0 and of e1)
// to the places their entries name, which may be pinned host memory
cudaError_t launch_rod_result(const RodRef* refs, int64_t count, int64_t stride, const double* state,
                              const int64_t* rod_start, const int32_t* rod_n, const double* e0, const double* e1,
                              cudaStream_t stream);

// energies of the listed rods (rod_energy.cu): out[5 r + k] of rod r, k = 0..3
// translational, rotational, shear and bend, 4 the gravitational potential
cudaError_t launch_rod_energy_list(const RodRef* refs, int64_t count, int64_t stride, const int64_t* rod_start,
                                   const int32_t* rod_n, const double* state, const double* params, double* out,
                                   cudaStream_t stream);

}  // namespace eb

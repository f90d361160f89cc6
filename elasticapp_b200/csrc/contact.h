// Device data of the collision system (rod elements as capsules), shared by
// the contact kernels (contact.cu) and the host side (eb_capi.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "eb_internal.h"

namespace eb {

// capsule table rows, in units of stride, indexed by element slot
enum CapsuleRow : int {
  kCapC = 0,     // 3: centre
  kCapL = 3,     // length
  kCapR = 4,     // radius
  kCapU = 5,     // 3: axis (third row of the capsule rotation)
  kCapVel = 8,   // 3: velocity
  kCapW = 11,    // 3: angular velocity taken to the world frame
  kCapLo = 14,   // 3: bounding box lower corner
  kCapHi = 17,   // 3: bounding box upper corner
  kCapRows = 20
};

// a capsule filed in the grid: its box rounded outward to FP32 and its slot,
// one 32-byte sector
struct alignas(32) ContactRecord {
  float lo[3], hi[3];
  int32_t slot;
  int32_t pad;
};

// partners a capsule keeps in its fixed-stride list; a capsule with more
// (a pile-up) gets its whole list in the overflow lists instead
constexpr int kFixedPartners = 32;

struct ContactPlane {
  double p[3];   // point on the plane
  double n[3];   // unit normal
  double lo[3];  // bounding box
  double hi[3];
  int32_t material;
  int32_t pad;
};

// contact parameters of a material pair (series rule for stiffness and
// damping, sum for the friction coefficients)
struct ContactPair {
  double k, cn, ct, mu_s, mu_d;
};

// the grid of one evaluation and what chooses it (device memory, zeroed once)
struct ContactGrid {
  double inv_edge;             // 1 / cell edge of this evaluation
  double reach;                // largest box extent with its margin: how far below a box's lower
                               // corner the lower corner of an overlapping box may lie
  int32_t first[3], last[3];   // lowest and highest cell of a lower corner, each axis
  int32_t dense;               // 1: a bucket a cell (the cells fit the table), 0: hashed
  int32_t by_float;            // 1: a capsule's cell is that of its FP32 lower corner, 0: of the FP64 one
  int32_t row, slab;           // dense: cells a row (x) and a slab (x, y)
  float sure;                  // FP32 boxes that overlap by this much overlap
  int32_t edge;                // cell edge of this evaluation in units of reach (1 or 2)
  int32_t edge_before;         // of the evaluation before (0: none yet)
  unsigned long long scanned;  // records the evaluation before read in its search
  int32_t filed;               // capsules filed in the grid
  int32_t live;                // capsules in the list of those the narrow phase evaluates
  // entries and listed capsules that the search's and the narrow phase's
  // warps have taken beyond their first
  uint32_t searched, evaluated;
  // bounds of the boxes' lower corners, rounded outward to FP32: the largest
  // and the negated smallest as order-preserving integers (zero: none yet)
  uint32_t top[3], bottom[3];
};

struct ContactArgs {
  int64_t stride;
  int64_t n_slots;
  const double* state;  // state buffer read by the step (slot layout)
  const double* par;
  const uint32_t* meta;
  const RodInfo* rods;
  const int32_t* cap_material;  // per slot: material of the capsule, -1 if none
  double half_dt;
  uint32_t sim_flags;
  double* cap;                       // kCapRows x stride
  unsigned long long* extent_bits;   // largest box extent (bits of a non-negative double)
  uint32_t* bucket;                  // stride; all ones: not filed (no finite box)
  uint32_t table_mask;               // hash table size - 1 (power of two)
  uint32_t max_cells;                // buckets of the tables below: cells a dense grid may have (at least
                                     // the hash table's size)
  int2* cell;                        // max_cells: the capsules filed in a bucket and the first one's entry
  ContactGrid* grid;
  ContactRecord* sorted_rec;         // n_caps: the capsules grouped by bucket
  int32_t* pair_count;               // stride (zero outside capsules): partners per capsule (between
                                     // the cell kernel and the scatter: the capsule's rank in its bucket)
  // per element slot: 1 if its capsule and the next one of its rod meet end to
  // end and plainly bent, so that the narrow phase finds no contact between them
  uint8_t* plain_joint;
  int32_t* live;                     // n_caps: the capsules with any other partner
  int32_t* fixed;                    // kFixedPartners x stride: partner lists of up to kFixedPartners
  int64_t* pair_offset;              // n_slots + 1: a capsule's overflow list (if it has more than
                                     // kFixedPartners partners); [n_slots] their total
  int32_t* partners;                 // capacity: overflow lists
  int64_t capacity;
  unsigned long long* required;      // largest pair total seen when over capacity
  const ContactPlane* planes;
  int32_t n_planes;
  int32_t n_materials;
  const ContactPair* pair_table;     // n_materials x n_materials
  double* cf;                        // 3 x stride, capsule force (lab frame)
  double* ct;                        // 3 x stride, capsule torque (lab frame)
  int32_t n_caps;                    // number of capsules (fixed at finalize)
  uint32_t* status;
};

// one whole contact evaluation (capsules, candidate pairs, contact loads)
// for the state a.state at the start of a step; launches counted into *launches
cudaError_t launch_contact(const ContactArgs& a, cudaStream_t stream, int64_t* launches);

}  // namespace eb

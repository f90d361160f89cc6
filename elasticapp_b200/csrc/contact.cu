// Collision system for rods: capsules, candidate pairs, contact loads.
//
// Every element of a participating rod is a capsule (Systems/Customization/
// CosseratRods/Transfer/Common.hpp:57-93): centre = mid-point of the element's
// nodes, length = dilatation * rest length, radius = the element dimension
// sqrt(V / (pi l)), rotation from the tangent (Utilities/Math/Orthogonal.cpp:
// 118-129), mass-weighted node velocity and the element's angular velocity.
// One evaluation per step, at the state after the first half drift, in
// five stages:
//
//   1. capsule_kernel: capsules and their axis-aligned bounding boxes
//      (Primitives/detail/CapsulePrimitiveBase.cpp:163-180), and the largest
//      box extent (block max, one atomic per CTA).
//   2. cell_kernel + range_kernel + scatter_kernel: a uniform grid with the
//      cell edge one or two of the largest extent, a bucket a cell or hashed
//      into a power-of-two table; every capsule is filed under the cell of its
//      box's lower corner (a counting sort by bucket).
//   3. pairs_kernel<0>: every capsule tests the capsules filed in the cells
//      its box can reach, then every plane, in one pass, writing up to
//      kFixedPartners partners into its fixed-stride list (sorted) and its
//      count; a capsule with more partners takes a region of the overflow
//      lists (one atomic on their total), and pairs_kernel<1> writes its
//      whole sorted list there.  A box that overlaps has its lower corner no
//      further below than the largest extent, so the candidate set equals the
//      exhaustive search's (Detection/Coarse/ExhaustiveSearch.hpp:322-435,
//      closed intervals of BoundingBox.hpp:532-540), which the reference's
//      hash grids reproduce (tests/.../Test_HashGrids.cpp).
//   4. force_kernel: each capsule with a partner other than its neighbours on
//      its rod evaluates the narrow phase with every
//      partner in ascending id order (RodCapsuleRodCapsule.hpp:70-186,
//      CapsulePlane.hpp:60-113), the pair always oriented with the smaller id
//      as the first body, and sums the spring-dashpot loads
//      (LinearSpringDashpot.cpp:32-85) that act on itself.  Each pair is
//      evaluated by both of its capsules; no atomics, so the loads are
//      deterministic.
//   5. the step kernel adds half the capsule force to each node and the
//      torque, recast as Q tau, to the element (Transfer/Common.hpp:32-55).
//
// This file is compiled without contraction of multiply-adds, so every
// product and sum is rounded as written; the capsules, boxes and candidate
// pairs are then bit-identical to a scalar FP64 evaluation of the same
// expressions.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "bulk_copy.cuh"
#include "contact.h"
#include "rod_fast.cuh"

namespace eb {
namespace {

using D3 = Vec3<double>;

constexpr double kContactThreshold = 1e-8;   // Utilities/Thresholds.hpp:138
constexpr double kParallelThreshold = 1e-8;  // Utilities/Thresholds.hpp:159
constexpr double kFrictionThreshold = 1e-8;  // Utilities/Thresholds.hpp:149
constexpr double kZeroLength = 1e-8;         // is_zero_length bound (Utilities/Math/Zero.hpp:46-49)
constexpr double kCellMargin = 1.0 + 1.0 / 1048576.0;
constexpr double kCellClamp = 1073741824.0;  // 2^30 cells from the origin

constexpr int kThreads = 256;
// the narrow phase: 128-thread CTAs, three per SM at 168 registers a thread
// (12 warps; 256 threads at 192 registers held 8, and a 128-register bound
// spilled 500 bytes a thread): 0.91 -> 0.82 ms a contact step
constexpr int kForceThreads = 128;
constexpr int kForceCtasPerSm = 3;

__device__ __forceinline__ D3 ld3(const double* p, int64_t S, int64_t s) { return {p[s], p[S + s], p[2 * S + s]}; }
__device__ __forceinline__ void st3(double* p, int64_t S, int64_t s, D3 a) {
  p[s] = a.x;
  p[S + s] = a.y;
  p[2 * S + s] = a.z;
}
__device__ __forceinline__ D3 mul3(double k, D3 a) { return {k * a.x, k * a.y, k * a.z}; }
__device__ __forceinline__ D3 neg3(D3 a) { return {-a.x, -a.y, -a.z}; }
// quotients and roots in the correctly rounded forms of rod_fast.cuh (their
// fused operations are written out, so nothing is contracted here)
__device__ __forceinline__ D3 quotient3(D3 a, double b) {
  if (!ordinary(b)) return {a.x / b, a.y / b, a.z / b};
  const double y = rcp_from(b, rcp_near(b));
  return {div_from(a.x, b, y), div_from(a.y, b, y), div_from(a.z, b, y)};
}
__device__ __forceinline__ double root(double a) { return ordinary(a) ? sqrt_from(a, rsqrt_near(a)) : sqrt(a); }
__device__ __forceinline__ double squared(D3 a) { return a.x * a.x + a.y * a.y + a.z * a.z; }
__device__ __forceinline__ double norm3(D3 a) { return root(squared(a)); }
// blaze::normalize: a * (1 / |a|), a zero vector stays zero
__device__ __forceinline__ D3 normalize3(D3 a) {
  const Length len = length_of(squared(a));
  const double il = len.l != 0.0 ? len.il : 0.0;
  return {a.x * il, a.y * il, a.z * il};
}

// a capsule's shape (centre, axis, length, radius); its velocity and
// angular velocity are read from the table only where a contact point needs
// them, so they are not held in registers through the closest-point search
// (that took the contact step from 0.71 to 0.69 ms; 68 B a thread of the
// narrow phase are still spilled)
struct Capsule {
  D3 c, u;
  double L, r;
};

__device__ __forceinline__ Capsule load_capsule(const double* cap, int64_t S, int64_t s) {
  Capsule k;
  k.c = ld3(cap + kCapC * S, S, s);
  k.L = cap[kCapL * S + s];
  k.r = cap[kCapR * S + s];
  k.u = ld3(cap + kCapU * S, S, s);
  return k;
}

__device__ __forceinline__ uint32_t cell_hash(int32_t cx, int32_t cy, int32_t cz) {
  uint64_t h = static_cast<uint64_t>(static_cast<uint32_t>(cx)) * 0x9E3779B97F4A7C15ull ^
               static_cast<uint64_t>(static_cast<uint32_t>(cy)) * 0xC2B2AE3D27D4EB4Full ^
               static_cast<uint64_t>(static_cast<uint32_t>(cz)) * 0x165667B19E3779F9ull;
  h ^= h >> 29;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 32;
  return static_cast<uint32_t>(h);
}

// FP32 values as integers of the same order, above zero for every number
__device__ __forceinline__ uint32_t ordered(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// ---- stage 1: capsules and boxes ------------------------------------------

constexpr uint32_t kNotFiled = 0xffffffffu;

__global__ void __launch_bounds__(kThreads) capsule_kernel(const ContactArgs a) {
  grid_dependency_launch();
  const int64_t s = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  const int64_t S = a.stride;
  double ext = 0.0;
  bool bad = false;
  // bounds of the lower corners (see ContactGrid): zero takes no part
  uint32_t top[3] = {0u, 0u, 0u}, bottom[3] = {0u, 0u, 0u};
  if (s < a.n_slots && a.cap_material[s] >= 0) {
    const double* x = a.state + kStX * S;
    const double* v = a.state + kStV * S;
    const double* w = a.state + kStW * S;
    const double c = a.half_dt;
    // everything the capsule is made of is asked for before anything is
    // written (a load after a store waits for it)
    const uint32_t meta = a.meta[s];
    const D3 xa = ld3(x, S, s), xb = ld3(x, S, s + 1), va = ld3(v, S, s), vb = ld3(v, S, s + 1), om = ld3(w, S, s);
    const double l0 = a.par[kL0 * S + s], volume = a.par[kVol * S + s];
    const double m0 = a.par[kMass * S + s], m1 = a.par[kMass * S + s + 1];
    // the bucket the capsule was filed in last time holds nothing any more
    // (those of its capsules all write the same; a bucket no capsule was
    // filed in is empty already)
    const uint32_t old = a.bucket[s];
    if (old < a.max_cells) a.cell[old] = make_int2(0, 0);
    // positions after the first half drift (PositionVerlet.hpp:60-69) and
    // the clamp's value constraint
    D3 x0 = {xa.x + c * va.x, xa.y + c * va.y, xa.z + c * va.z};
    D3 x1 = {xb.x + c * vb.x, xb.y + c * vb.y, xb.z + c * vb.z};
    // the far node of the next element of the rod
    const bool joint = (meta & kVor) != 0;
    D3 x2 = x1;
    if (joint) x2 = {x[s + 2] + c * v[s + 2], x[S + s + 2] + c * v[S + s + 2], x[2 * S + s + 2] + c * v[2 * S + s + 2]};
    if (a.sim_flags & kSimClamp) {
      // any of the nodes may be held by a clamp
      const RodInfo& ri = a.rods[meta >> kRodShift];
      double t[3];
      if (clamp_position(ri, s, t)) x0 = {t[0], t[1], t[2]};
      if (clamp_position(ri, s + 1, t)) x1 = {t[0], t[1], t[2]};
      if (joint && clamp_position(ri, s + 2, t)) x2 = {t[0], t[1], t[2]};
    }
    const D3 dx = x1 - x0;
    const Length len = length_of(squared(dx));
    const double l = len.l;
    // Consecutive capsules of a rod share a node, so the narrow phase finds
    // them no distance apart and no contact.  Its tolerance on the projections
    // (1e-8 m^2) can only pick another region for elements shorter than a
    // millimetre or folded back on one another, or where the ends part by so
    // much rounding that it passes the tolerance: they part by up to
    // 1.2e-15 (X + 2 L), L the longer element's length and X the coordinates,
    // and the projections by L times that, 3.5e-9 m^2 within the bound below
    // (and the ends by 1.2e-9 m, of 1e-8).  Other joints are evaluated.
    {
      const D3 dn = x2 - x1;
      const double l2 = dot(dx, dx), n2 = dot(dn, dn), along = dot(dx, dn), big = fmax(l2, n2);
      const double far = fmax(fabs(x1.x), fmax(fabs(x1.y), fabs(x1.z)));
      a.plain_joint[s] = joint && l2 > 1e-6 && n2 > 1e-6 && far < 1e6 && (far * far + big) * big < 1e12 &&
                         along > 0.0 && along * along > 0.01 * (l2 * n2);
    }
    D3 t;
    double area;  // volume / (pi l)
    if (ordinary(l)) {
      t = {div_from(dx.x, l, len.il), div_from(dx.y, l, len.il), div_from(dx.z, l, len.il)};
      area = div_from(M_1_PI * volume, l, len.il);
    } else {
      t = {dx.x / l, dx.y / l, dx.z / l};
      area = M_1_PI * volume / l;
    }
    const double e = quotient(l, l0);
    const double L = e * l0;
    const double r = root(area);
    const D3 cen = {0.5 * (x0.x + x1.x), 0.5 * (x0.y + x1.y), 0.5 * (x0.z + x1.z)};
    // Orthogonal.cpp:32-55 with the tangent as the third row
    const D3 v1 = normalize3(t);
    D3 v2 = {0.8, 0.6, 0.0};
    D3 v3 = cross(v1, v2);
    v2 = cross(v3, v1);
    if (dot(v2, v2) < kZeroLength) {
      v2 = {0.6, -0.8, 0.0};
      v3 = normalize3(cross(v1, v2));
      v2 = cross(v3, v1);
    }
    const D3 r0 = normalize3(v2), r1 = normalize3(v3), r2 = v1;
    const D3 num = mul3(m0, va) + mul3(m1, vb);
    const double den = m0 + m1;
    const D3 vel = quotient3(num, den);
    const D3 ww = {r0.x * om.x + r1.x * om.y + r2.x * om.z, r0.y * om.x + r1.y * om.y + r2.y * om.z,
                   r0.z * om.x + r1.z * om.y + r2.z * om.z};
    // the narrow phase writes only the capsules it evaluates
    st3(a.cf, S, s, D3{0.0, 0.0, 0.0});
    st3(a.ct, S, s, D3{0.0, 0.0, 0.0});
    double* cap = a.cap;
    st3(cap + kCapC * S, S, s, cen);
    cap[kCapL * S + s] = L;
    cap[kCapR * S + s] = r;
    st3(cap + kCapU * S, S, s, r2);
    st3(cap + kCapVel * S, S, s, vel);
    st3(cap + kCapW * S, S, s, ww);
    const double ua[3] = {r2.x, r2.y, r2.z}, ca[3] = {cen.x, cen.y, cen.z};
    // a capsule whose box is not finite (a diverged state) takes no part: it
    // would overlap every box
    bool filed = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double len = fabs(ua[d] * L) * 0.5 + r + kContactThreshold;
      const double lo = ca[d] - len, hi = ca[d] + len;
      cap[(kCapLo + d) * S + s] = lo;
      cap[(kCapHi + d) * S + s] = hi;
      const double xt = hi - lo;
      if (!(xt >= 0.0 && xt < 1e300)) bad = true;  // NaN or infinite box
      else ext = fmax(ext, xt);
      filed = filed && (xt >= 0.0) && (xt < 1e300) && (fabs(lo) < 1e300);
      top[d] = ordered(__double2float_ru(lo));
      bottom[d] = ordered(-__double2float_rd(lo));
    }
    a.bucket[s] = filed ? 0u : kNotFiled;
    if (!filed) {
      a.pair_count[s] = 0;
      top[0] = top[1] = top[2] = bottom[0] = bottom[1] = bottom[2] = 0u;
    }
  }
  // block max of the extents, one atomic per CTA (non-negative doubles order
  // like their bit patterns)
  for (int o = 16; o > 0; o >>= 1) ext = fmax(ext, __shfl_xor_sync(0xffffffffu, ext, o));
  __shared__ double wmax[kThreads / 32];
  __shared__ uint32_t bounds[6];
  if (threadIdx.x < 6) bounds[threadIdx.x] = 0u;
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = ext;
  __syncthreads();
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const uint32_t t = __reduce_max_sync(0xffffffffu, top[d]), b = __reduce_max_sync(0xffffffffu, bottom[d]);
    if ((threadIdx.x & 31) == 0) {
      atomicMax(bounds + d, t);
      atomicMax(bounds + 3 + d, b);
    }
  }
  if (bad) atomicOr(a.status, kStatusContactNonFinite);
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int i = 0; i < kThreads / 32; ++i) m = fmax(m, wmax[i]);
    if (m > 0.0) atomicMax(a.extent_bits, static_cast<unsigned long long>(__double_as_longlong(m)));
  }
  if (threadIdx.x < 6 && bounds[threadIdx.x])
    atomicMax(threadIdx.x < 3 ? a.grid->top + threadIdx.x : a.grid->bottom + (threadIdx.x - 3), bounds[threadIdx.x]);
}

// ---- stage 2: grid cells, counting sort by bucket --------------------------

// Cell edge in units of the largest extent (with its margin): one capsule
// searches the cells its box can reach, 2.7 an axis for an edge of one
// (unless its box is as large as the largest, in which case three) and 1.8
// for an edge of two, whose cells hold eight times the space.  Two wins where
// the lookups outnumber the records read, which the evaluation before tells
// (it changes the time only, never the pairs).  Records read a capsule with an
// edge of two, and a step's time with an edge of one and of two, in us: 8.4:
// 332 and 265, 11.4: 84 and 69, 18.8: 582 and 445, 42: 396 and 397, 54: 558 and
// 572, 213: 1316 and 1500, 670: 2765 and 3157; so the line to an edge of one is
// at 48.  An edge of one reads 2.4 times fewer; the line back, at 8 of them
// (19 with an edge of two), lies well below so that the choice does not
// alternate.
__device__ __forceinline__ int32_t choose_edge(const ContactArgs& a) {
  const int32_t before = a.grid->edge_before;
  const unsigned long long n = static_cast<unsigned long long>(a.n_caps);
  const unsigned long long scanned = a.grid->scanned;
  if (before == 1) return scanned < 8 * n ? 2 : 1;
  return before == 2 && scanned > 48 * n ? 1 : 2;
}

__device__ __forceinline__ int32_t cell_of(double x, double inv_edge) {
  return static_cast<int32_t>(fmin(fmax(floor(x * inv_edge), -kCellClamp), kCellClamp));
}

// The grid of this evaluation: a bucket a cell when the cells between the
// lowest and the highest lower corner fit the table, else cells hashed into
// it.  A bucket a cell needs no hash (four 64-bit multiplications a lookup)
// and no comparison of cells, and the cells of a row are neighbours in memory.
__device__ __forceinline__ ContactGrid make_grid(const ContactArgs& a) {
  ContactGrid g;
  const double h = __longlong_as_double(static_cast<long long>(*a.extent_bits)) * kCellMargin;
  g.edge = choose_edge(a);
  g.reach = h > 0.0 ? h : 1.0;
  g.inv_edge = 1.0 / (g.edge * g.reach);
  double total = 1.0;
  float far = 0.0f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const bool any = a.grid->top[d] != 0u;
    const float hi = any ? unordered(a.grid->top[d]) : 0.0f, lo = any ? -unordered(a.grid->bottom[d]) : 0.0f;
    g.first[d] = cell_of(lo, g.inv_edge);
    g.last[d] = cell_of(hi, g.inv_edge);
    total *= static_cast<double>(g.last[d]) - static_cast<double>(g.first[d]) + 1.0;
    far = fmaxf(far, fmaxf(fabsf(lo), fabsf(hi)));
  }
  g.dense = total <= static_cast<double>(a.max_cells);
  g.row = g.dense ? g.last[0] - g.first[0] + 1 : 0;
  g.slab = g.dense ? g.row * (g.last[1] - g.first[1] + 1) : 0;
  // a corner rounded outward lies within 2^-23 of its value (and 1e-44 of
  // zero), and no corner lies further out than the farthest plus the reach
  // (beyond FP32's range a NaN: no FP32 comparison decides)
  const float out = far + static_cast<float>(g.reach);
  g.sure = out < 1e30f ? out * 1e-6f + 1e-30f : __int_as_float(0x7fffffff);
  // cells by the FP32 corners, which the records hold, as long as their
  // rounding (the margin added to the reach) is small against a box
  const double margin = static_cast<double>(out) * 2.5e-7;
  g.by_float = margin < 0.125 * g.reach;
  if (g.by_float) g.reach += margin;
  return g;
}

// cell of a lower corner: of its FP32 value rounded down, or of itself
__device__ __forceinline__ int32_t corner_cell(const ContactGrid& g, double lo) {
  return cell_of(g.by_float ? static_cast<double>(__double2float_rd(lo)) : lo, g.inv_edge);
}

// bucket of a cell (in the dense grid: of a cell inside it)
__device__ __forceinline__ uint32_t bucket_of(const ContactGrid& g, bool dense, uint32_t mask, int32_t cx, int32_t cy,
                                              int32_t cz) {
  if (dense)
    return static_cast<uint32_t>((cz - g.first[2]) * g.slab + (cy - g.first[1]) * g.row + (cx - g.first[0]));
  return cell_hash(cx, cy, cz) & mask;
}

__global__ void __launch_bounds__(kThreads) cell_kernel(const ContactArgs a) {
  grid_dependency_launch();
  grid_dependency_wait();
  const int64_t s = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  const ContactGrid g = make_grid(a);
  if (s == 0) {
    a.pair_offset[a.n_slots] = 0;  // the pair search's overflow total
    // (none of these is read before the next kernel)
    a.grid->inv_edge = g.inv_edge;
    a.grid->reach = g.reach;
    for (int d = 0; d < 3; ++d) {
      a.grid->first[d] = g.first[d];
      a.grid->last[d] = g.last[d];
    }
    a.grid->dense = g.dense;
    a.grid->by_float = g.by_float;
    a.grid->row = g.row;
    a.grid->slab = g.slab;
    a.grid->sure = g.sure;
    a.grid->edge = g.edge;
    a.grid->filed = 0;
    a.grid->live = 0;
    a.grid->searched = a.grid->evaluated = 0u;
  }
  if (s >= a.n_slots || a.cap_material[s] < 0 || a.bucket[s] == kNotFiled) return;
  const int64_t S = a.stride;
  int32_t c[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) c[d] = corner_cell(g, a.cap[(kCapLo + d) * S + s]);
  const uint32_t b = bucket_of(g, g.dense, a.table_mask, c[0], c[1], c[2]);
  if (b >= a.max_cells) {  // cannot happen: the bounds hold every lower corner
    atomicOr(a.status, kStatusContactIndex);
    a.bucket[s] = kNotFiled;
    a.pair_count[s] = 0;
    return;
  }
  a.bucket[s] = b;
  // the capsule's rank in its bucket, kept in its pair count until the
  // scatter has filed it (the pair search then writes the count)
  a.pair_count[s] = atomicAdd(&a.cell[b].x, 1);
}

// The buckets' first entries, in whatever order the CTAs come: the capsule of
// rank 0 stands for its bucket, and a CTA scans the counts of its buckets and
// takes their entries with one atomic.  (No reader needs the buckets in order,
// and only those in use are looked at: a pass over every bucket, which also
// set the counts back to zero, took 22 us for four million of them, this one
// 9 us for the half million capsules in them.)
__global__ void __launch_bounds__(kThreads) range_kernel(const ContactArgs a) {
  grid_dependency_launch();
  grid_dependency_wait();
  const int64_t s = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  int2* cell = nullptr;
  if (s < a.n_slots) {
    const int32_t mat = a.cap_material[s], rank = a.pair_count[s];
    const uint32_t b = a.bucket[s];
    if (mat >= 0 && rank == 0 && b < a.max_cells) cell = a.cell + b;  // (past the last bucket: not filed)
  }
  const int32_t n = cell ? cell->x : 0;
  __shared__ int32_t warp_sum[kThreads / 32];
  __shared__ int32_t base;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t x = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sum[wid] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    int32_t total = 0;
    for (int i = 0; i < kThreads / 32; ++i) {
      const int32_t t = warp_sum[i];
      warp_sum[i] = total;
      total += t;
    }
    base = total ? atomicAdd(&a.grid->filed, total) : 0;
  }
  __syncthreads();
  if (cell) cell->y = base + warp_sum[wid] + x - n;
}

__global__ void __launch_bounds__(kThreads) scatter_kernel(const ContactArgs a) {
  grid_dependency_launch();
  grid_dependency_wait();
  const int64_t s = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  if (s == 0) {
    *a.extent_bits = 0;  // read only by the cell kernel: zero for the next evaluation
    a.grid->edge_before = a.grid->edge;
    a.grid->scanned = 0;
    for (int d = 0; d < 3; ++d) a.grid->top[d] = a.grid->bottom[d] = 0u;
  }
  if (s >= a.n_slots) return;
  const int64_t S = a.stride;
  const int32_t mat = a.cap_material[s], rank = a.pair_count[s];  // the rank the cell kernel took
  const uint32_t b = a.bucket[s];
  if (mat < 0 || b >= a.max_cells) return;  // no capsule, or excluded (not finite)
  const int32_t pos = a.cell[b].y + rank;
  if (pos < 0 || pos >= a.n_caps) {  // cannot happen with consistent counts; never write out of range
    atomicOr(a.status, kStatusContactIndex);
    return;
  }
  const double* cap = a.cap;
  float4* rec = reinterpret_cast<float4*>(a.sorted_rec + pos);
  rec[0] = make_float4(__double2float_rd(cap[kCapLo * S + s]), __double2float_rd(cap[(kCapLo + 1) * S + s]),
                       __double2float_rd(cap[(kCapLo + 2) * S + s]), __double2float_ru(cap[kCapHi * S + s]));
  rec[1] = make_float4(__double2float_ru(cap[(kCapHi + 1) * S + s]), __double2float_ru(cap[(kCapHi + 2) * S + s]),
                       __int_as_float(static_cast<int32_t>(s)), 0.0f);
}

// ---- stage 3: candidate pairs ----------------------------------------------

__device__ __forceinline__ void sort_ids(int32_t* v, int32_t n) {
  for (int32_t i = 1; i < n; ++i) {
    const int32_t x = v[i];
    int32_t j = i - 1;
    while (j >= 0 && v[j] > x) {
      v[j + 1] = v[j];
      --j;
    }
    v[j + 1] = x;
  }
}

struct FloatBox {
  float lo[3], hi[3];
};

// whether the boxes of slots i and j overlap, from their FP64 corners
__device__ __forceinline__ bool boxes_overlap(const ContactArgs& a, int64_t i, int64_t j) {
  const int64_t S = a.stride;
  bool yes = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double* lo = a.cap + (kCapLo + d) * S;
    const double* hi = a.cap + (kCapHi + d) * S;
    yes = yes & !(lo[j] > hi[i]) & !(hi[j] < lo[i]);
  }
  return yes;
}

// The search of one capsule.  kPass 0 (idx: a filed entry) counts the
// partners and fills the fixed-stride list; kPass 1 (idx: a slot, leaving at
// once unless its coalesced count is above kFixedPartners) writes the overflow
// list of a capsule with more partners.
//
// A box that overlaps has its lower corner at most `reach` below this box's
// lower corner (no box is larger) and at or below its upper corner, so the
// search visits the cells of that range (rounding is monotone, and the margins
// in `reach` are above it): at most eight with an edge of two.  It is
// bound by dependent round trips to L2 and by its instructions on diverged
// lanes, so the ranges of two neighbouring cells are loaded together and their
// entries scanned in one loop, the next two ranges on their way meanwhile, and
// an entry is one 32-byte record of FP32 corners.  Rounded outward, they
// decide every pair but those that overlap by less than `sure`; only these
// take the FP64 corners.  Against 27 hashed
// lookups in turn and 64-byte FP64 records, the search of 524,288 capsules
// went from 160 to 73 us.
template <int kPass, bool kDense>
__device__ __forceinline__ uint32_t search_one(const ContactArgs& a, const ContactGrid& g, int32_t n_caps, int64_t idx) {
  int32_t id;
  FloatBox me;
  int32_t* out;
  if (kPass == 1) {
    const int64_t s = idx;
    // only filed capsules have a count; the others hold zero
    if (s >= a.n_slots || a.pair_count[s] <= kFixedPartners) return 0;
    const int64_t total = a.pair_offset[a.n_slots];
    if (total > a.capacity) {
      atomicOr(a.status, kStatusPairOverflow);
      atomicMax(a.required, static_cast<unsigned long long>(total));
      return 0;
    }
    out = a.partners + a.pair_offset[s];  // within [0, capacity)
    id = static_cast<int32_t>(s);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      me.lo[d] = __double2float_rd(a.cap[(kCapLo + d) * a.stride + s]);
      me.hi[d] = __double2float_ru(a.cap[(kCapHi + d) * a.stride + s]);
    }
  } else {
    const float4* own = reinterpret_cast<const float4*>(a.sorted_rec + idx);
    const float4 r0 = own[0], r1 = own[1];
    me = {{r0.x, r0.y, r0.z}, {r0.w, r1.x, r1.y}};
    id = __float_as_int(r1.z);
    out = a.fixed + static_cast<int64_t>(id) * kFixedPartners;
  }
  // joints with the neighbours on the rod that the narrow phase may skip
  // (slot id - 1 of a rod's first element is a node slot, which holds zero)
  const int32_t next = kPass == 0 && a.plain_joint[id] ? id + 1 : -1;
  const int32_t prev = kPass == 0 && id > 0 && a.plain_joint[id - 1] ? id - 1 : -1;
  int32_t c0[3], c1[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double lo = g.by_float ? me.lo[d] : a.cap[(kCapLo + d) * a.stride + id];
    const double hi = g.by_float ? me.hi[d] : a.cap[(kCapHi + d) * a.stride + id];
    c0[d] = max(cell_of(lo - g.reach, g.inv_edge), g.first[d]);
    c1[d] = min(cell_of(hi, g.inv_edge), g.last[d]);
  }
  int32_t cnt = 0;
  uint32_t scanned = 0;
  bool live = false;
  int32_t cx = c0[0], cy = c0[1], cz = c0[2];
  bool more = c0[0] <= c1[0] && c0[1] <= c1[1] && c0[2] <= c1[2];
  // the counts and first entries of cells cx and cx + 1 of the row
  int2 ra = make_int2(0, 0), rb = make_int2(0, 0);
  auto fetch = [&]() {
    ra = a.cell[bucket_of(g, kDense, a.table_mask, cx, cy, cz)];
    rb = cx < c1[0] ? a.cell[bucket_of(g, kDense, a.table_mask, cx + 1, cy, cz)] : make_int2(0, 0);
  };
  if (more) fetch();
  while (more) {
    const int32_t hx = cx, hy = cy, hz = cz;
    const int32_t a0 = max(ra.y, 0), na = max(min(ra.x, n_caps - a0), 0);
    const int32_t b0 = max(rb.y, 0), n = na + max(min(rb.x, n_caps - b0), 0);
    cx += 2;
    if (cx > c1[0]) {
      cx = c0[0];
      if (++cy > c1[1]) {
        cy = c0[1];
        ++cz;
      }
    }
    more = cz <= c1[2];
    if (more) fetch();
    scanned += n;
    for (int32_t k = 0; k < n; ++k) {
      const float4* r = reinterpret_cast<const float4*>(a.sorted_rec + (k < na ? a0 + k : b0 + (k - na)));
      const float4 e0 = r[0], e1 = r[1];
      const int32_t o = __float_as_int(e1.z);
      // how far the boxes overlap, the least of the axes and sides
      const float by = fminf(fminf(fminf(me.hi[0] - e0.x, me.hi[1] - e0.y), fminf(me.hi[2] - e0.z, e0.w - me.lo[0])),
                             fminf(e1.x - me.lo[1], e1.y - me.lo[2]));
      if (by < 0.0f || o == id) continue;
      if (!(by >= g.sure) && !boxes_overlap(a, id, o)) continue;
      if (!kDense) {  // the entry may be of another cell of this bucket
        const double* lo = a.cap + kCapLo * a.stride + o;
        const int64_t S = a.stride;
        const double x = g.by_float ? e0.x : lo[0], y = g.by_float ? e0.y : lo[S], z = g.by_float ? e0.z : lo[2 * S];
        if (cell_of(x, g.inv_edge) != (k < na ? hx : hx + 1) || cell_of(y, g.inv_edge) != hy ||
            cell_of(z, g.inv_edge) != hz)
          continue;
      }
      if (kPass == 1 || cnt < kFixedPartners) out[cnt] = o;
      ++cnt;
      live = live || (o != next && o != prev);
    }
  }
  for (int32_t p = 0; p < a.n_planes; ++p) {
    const ContactPlane& P = a.planes[p];
    bool yes = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) yes = yes & !(P.lo[d] > me.hi[d]) & !(P.hi[d] < me.lo[d]);
    if (!yes) continue;
#pragma unroll
    for (int d = 0; d < 3; ++d)
      yes = yes & !(P.lo[d] > a.cap[(kCapHi + d) * a.stride + id]) & !(P.hi[d] < a.cap[(kCapLo + d) * a.stride + id]);
    if (!yes) continue;
    if (kPass == 1 || cnt < kFixedPartners) out[cnt] = static_cast<int32_t>(a.n_slots) + p;
    ++cnt;
    live = true;
  }
  if (kPass == 0) {
    a.pair_count[id] = cnt;
    // a capsule with more partners takes a region of the overflow lists
    // (in whatever order the atomics come; every list is whole and sorted)
    if (cnt > kFixedPartners)
      a.pair_offset[id] = static_cast<int64_t>(atomicAdd(
          reinterpret_cast<unsigned long long*>(a.pair_offset + a.n_slots), static_cast<unsigned long long>(cnt)));
    if (cnt <= kFixedPartners) sort_ids(out, cnt);  // ascending partner order
    // the narrow phase's list, one atomic for the lanes that come here together
    if (live) {
      const unsigned lanes = __activemask();
      const int lane = threadIdx.x & 31, first = __ffs(lanes) - 1;
      int32_t base = 0;
      if (lane == first) base = atomicAdd(&a.grid->live, __popc(lanes));
      base = __shfl_sync(lanes, base, first);
      a.live[base + __popc(lanes & ((1u << lane) - 1u))] = id;  // one entry a filed capsule: below n_caps
    }
  } else {
    sort_ids(out, cnt);
  }
  return scanned;
}

// The items 0 .. n - 1 in groups of 32: a warp of a grid of resident CTAs
// takes its first by its place in the grid and each other one from *taken
// (zero before the launch), so none waits for a slower one and none takes more
// rounds than its share: with fixed strides some threads step four times
// through half a million entries and others three (8192 4-mm rods, every
// capsule in the narrow phase: 0.492 -> 0.445 ms a step; 4096 rods in a box of
// 0.25 1.39 -> 1.31; few in the narrow phase: 243 -> 241 us; one group a warp
// or less: no change).  The next group is asked for when the one in hand is
// done: before it, at a register more across the search, 0.459 ms.
template <typename Body>
__device__ __forceinline__ void take_groups(uint32_t* taken, uint32_t n, Body&& body) {
  const uint32_t lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  uint32_t at = 32u * (blockIdx.x * warps + (threadIdx.x >> 5));
  while (at < n) {
    if (at + lane < n) body(static_cast<int64_t>(at + lane));
    __syncwarp();
    if (lane == 0) at = 32u * gridDim.x * warps + atomicAdd(taken, 32u);
    at = __shfl_sync(0xffffffffu, at, 0);
  }
}

// a grid of resident CTAs whose warps take the entries (pass 0) or whose
// threads step through the slots (pass 1, which leaves at once when no
// capsule overflowed)
// (At four CTAs an SM the search has 64 registers a thread and spills 172 B of
// stores and 180 of loads, of both searches' bodies together; at three CTAs and
// 80 registers it was 0 to 16 % slower.)
template <int kPass>
__global__ void __launch_bounds__(kThreads, 4) pairs_kernel(const ContactArgs a) {
  grid_dependency_wait();
  if (kPass == 1 && a.pair_offset[a.n_slots] == 0) return;
  // entries filed this evaluation (the capsules with finite boxes)
  const int32_t n_caps = min(a.grid->filed, a.n_caps);
  // (read from shared memory where it is used: in registers it costs the
  // search two of five CTAs an SM)
  __shared__ ContactGrid g;
  if (threadIdx.x == 0) g = *a.grid;
  __syncthreads();
  uint32_t scanned = 0;
  auto search = [&](auto dense) {
    constexpr bool kDense = decltype(dense)::value;
    if (kPass == 0) {
      take_groups(&a.grid->searched, static_cast<uint32_t>(n_caps),
                  [&](int64_t i) { scanned += search_one<kPass, kDense>(a, g, n_caps, i); });
    } else {
      const int64_t stride = static_cast<int64_t>(gridDim.x) * kThreads;
      for (int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x; i < a.n_slots; i += stride)
        search_one<kPass, kDense>(a, g, n_caps, i);
    }
  };
  if (g.dense)
    search(std::true_type{});
  else
    search(std::false_type{});
  if (kPass == 0) {
    scanned = __reduce_add_sync(0xffffffffu, scanned);
    if ((threadIdx.x & 31) == 0) atomicAdd(&a.grid->scanned, static_cast<unsigned long long>(scanned));
  }
}

// ---- stage 4: narrow phase and spring-dashpot loads ------------------------

struct ContactPoint {
  D3 pos, n;
  double dist;
};

// Utilities/Geometry/GetClosestLineSegmentPoints.cpp, branch for branch
__device__ void closest_segment_points(D3 a1, D3 a2, D3 b1, D3 b2, D3& cp1, D3& cp2) {
  const D3 a1a2 = a2 - a1, b1b2 = b2 - b1, a1b1 = b1 - a1;
  const double da1 = dot(a1a2, a1b1), db1 = dot(b1b2, a1b1);
  if (da1 <= 0.0 && db1 >= 0.0) {
    cp1 = a1;
    cp2 = b1;
    return;
  }
  const D3 a1b2 = b2 - a1;
  const double da2 = dot(a1a2, a1b2), db2 = dot(b1b2, a1b2);
  if (da2 <= 0.0 && db2 <= 0.0) {
    cp1 = a1;
    cp2 = b2;
    return;
  }
  const D3 a2b1 = b1 - a2;
  const double da3 = dot(a1a2, a2b1), db3 = dot(b1b2, a2b1);
  if (da3 >= 0.0 && db3 >= 0.0) {
    cp1 = a2;
    cp2 = b1;
    return;
  }
  const D3 a2b2 = b2 - a2;
  const double da4 = dot(a1a2, a2b2), db4 = dot(b1b2, a2b2);
  if (da4 >= 0.0 && db4 <= 0.0) {
    cp1 = a2;
    cp2 = b2;
    return;
  }
  const double la = dot(a1a2, a1a2);
  if (da1 >= -kParallelThreshold && da3 <= kParallelThreshold) {
    const D3 k = mul3(quotient(da1, la), a1a2);
    const D3 n = a1b1 - k;
    if (dot(b1b2, n) >= -kParallelThreshold) {
      cp1 = a1 + k;
      cp2 = b1;
      return;
    }
  }
  if (da2 >= -kParallelThreshold && da4 <= kParallelThreshold) {
    const D3 k = mul3(quotient(da2, la), a1a2);
    const D3 n = a1b2 - k;
    if (dot(b1b2, n) <= kParallelThreshold) {
      cp1 = a1 + k;
      cp2 = b2;
      return;
    }
  }
  const double lb = dot(b1b2, b1b2);
  if (db1 <= kParallelThreshold && db2 >= -kParallelThreshold) {
    const D3 k = mul3(quotient(-db1, lb), b1b2);
    const D3 n = neg3(a1b1) - k;
    if (dot(a1a2, n) >= -kParallelThreshold) {
      cp1 = a1;
      cp2 = b1 + k;
      return;
    }
  }
  if (db3 <= kParallelThreshold && db4 >= -kParallelThreshold) {
    const D3 k = mul3(quotient(-db3, lb), b1b2);
    const D3 n = neg3(a2b1) - k;
    if (dot(a1a2, n) <= kParallelThreshold) {
      cp1 = a2;
      cp2 = b1 + k;
      return;
    }
  }
  const double sc = dot(a1a2, b1b2);
  double div = la * lb - sc * sc;
  div = reciprocal(div);
  const double sp = (lb * da1 - sc * db1) * div;
  const double tp = (sc * da1 - la * db1) * div;
  cp1 = a1 + mul3(sp, a1a2);
  cp2 = b1 + mul3(tp, b1b2);
}

// RodCapsuleRodCapsule.hpp:70-186 (c1 has the smaller id)
__device__ __forceinline__ int rod_capsule_contacts(const Capsule& c1, const Capsule& c2, ContactPoint out[2]) {
  const D3 up1 = mul3(0.5 * c1.L, c1.u), up2 = mul3(0.5 * c2.L, c2.u);
  D3 cp1, cp2;
  closest_segment_points(c1.c + up1, c1.c - up1, c2.c + up2, c2.c - up2, cp1, cp2);
  D3 nrm = cp1 - cp2;
  const double ln = norm3(nrm);
  if (ln < kContactThreshold) return 0;
  const double dist = ln - c1.r - c2.r;
  if (!(dist < kContactThreshold)) return 0;
  nrm = normalize3(nrm);
  const double c2x = dot(c1.u, c2.c - c1.c);
  if ((fabs(dot(c1.u, c2.u)) - 1.0) > -kParallelThreshold && fabs(c2x) < c1.L) {
    const double hl1 = 0.5 * c1.L, hl2 = 0.5 * c2.L;
    if (hl1 < c2x + hl2) {
      const double k = c1.r + 0.5 * dist;
      out[0] = {(c1.c + up1) - mul3(k, nrm), nrm, dist};
    } else {
      const double k = c2.r + 0.5 * dist;
      out[0] = {(c2.c + mul3(hl2, c1.u)) + mul3(k, nrm), nrm, dist};
    }
    if (-hl1 > c2x - hl2) {
      const double k = c1.r + 0.5 * dist;
      out[1] = {(c1.c - up1) - mul3(k, nrm), nrm, dist};
    } else {
      const double k = c2.r + 0.5 * dist;
      out[1] = {(c2.c - mul3(hl2, c1.u)) + mul3(k, nrm), nrm, dist};
    }
    return 2;
  }
  const double k = c2.r + 0.5 * dist;
  out[0] = {cp2 + mul3(k, nrm), nrm, dist};
  return 1;
}

// CapsulePlane.hpp:60-113
// (the points are written at constant indices, so they stay in registers)
__device__ __forceinline__ int capsule_plane_contacts(const Capsule& c, const ContactPlane& p, ContactPoint out[2]) {
  const D3 up = mul3(0.5 * c.L, c.u);
  const D3 pu = c.c + up, pl = c.c - up;
  const D3 pp = {p.p[0], p.p[1], p.p[2]}, n = {p.n[0], p.n[1], p.n[2]};
  const double du = fabs(dot(n, pu - pp)) - c.r;
  const double dl = fabs(dot(n, pl - pp)) - c.r;
  const bool hu = du < kContactThreshold, hl = dl < kContactThreshold;
  if (hu) out[0] = {pu - mul3(c.r + du, n), n, du};
  if (hl) {
    const ContactPoint q = {pl - mul3(c.r + dl, n), n, dl};
    if (hu)
      out[1] = q;
    else
      out[0] = q;
  }
  return (hu ? 1 : 0) + (hl ? 1 : 0);
}

// velocity of the material point at pos of capsule s (centre c)
__device__ __forceinline__ D3 point_velocity(const double* cap, int64_t S, int64_t s, D3 c, D3 pos) {
  const D3 vel = ld3(cap + kCapVel * S, S, s), ww = ld3(cap + kCapW * S, S, s);
  return vel + cross(ww, pos - c);
}

// Contact.cpp:150-215 and LinearSpringDashpot.cpp:32-85; false: separated
__device__ bool spring_dashpot(const ContactPoint& ct, D3 rvel, const ContactPair& pm, D3& net) {
  if (!(ct.dist < -kContactThreshold)) return false;
  const D3 n = ct.n;
  const double rvn = dot(n, rvel);
  const double rvt = dot(n, rvel - mul3(rvn, n));
  const double mu = fabs(rvt) > kFrictionThreshold ? pm.mu_d : pm.mu_s;
  const double delta = -ct.dist;
  const double relvn = -dot(n, rvel);
  const D3 relvt = neg3(rvel) - mul3(relvn, n);
  const double fn = fmax(0.0, pm.k * delta + pm.cn * relvn);
  const double ft = fmin(pm.ct * norm3(relvt), mu * fn);
  net = mul3(fn, n) + mul3(ft, normalize3(relvt));
  return true;
}

__device__ __forceinline__ void force_one(const ContactArgs& a, int64_t s) {
  const int32_t mat = a.cap_material[s];
  if (mat < 0) return;
  const int64_t S = a.stride;
  D3 F = {0.0, 0.0, 0.0}, T = {0.0, 0.0, 0.0};
  const int32_t cnt = a.pair_count[s];
  const int32_t* list = a.fixed + s * kFixedPartners;
  bool ok = true;
  if (cnt > kFixedPartners) {
    const int64_t total = a.pair_offset[a.n_slots];
    ok = total <= a.capacity;
    list = a.partners + a.pair_offset[s];
  }
  if (ok) {
    const Capsule me = load_capsule(a.cap, S, s);
    ContactPoint pts[2];
    for (int32_t k = 0; k < cnt; ++k) {
      const int64_t o = list[k];
      if (o == s + 1 ? a.plain_joint[s] : (o == s - 1 && a.plain_joint[o])) continue;  // no contact (capsule_kernel)
      if (o >= 0 && o < a.n_slots) {
        const int32_t om = a.cap_material[o];
        if (om < 0) continue;
        const bool first = s < o;
        const Capsule other = load_capsule(a.cap, S, o);
        const Capsule& c1 = first ? me : other;
        const Capsule& c2 = first ? other : me;
        const ContactPair pm = a.pair_table[(first ? mat : om) * a.n_materials + (first ? om : mat)];
        const int np = rod_capsule_contacts(c1, c2, pts);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i >= np) break;
          const D3 rvel = point_velocity(a.cap, S, first ? s : o, c1.c, pts[i].pos) -
                          point_velocity(a.cap, S, first ? o : s, c2.c, pts[i].pos);
          D3 net;
          if (!spring_dashpot(pts[i], rvel, pm, net)) continue;
          // RigidBodyPrimitive.hpp:500-504 add_force_at_position
          const D3 f = first ? net : neg3(net);
          F = F + f;
          T = T + cross(pts[i].pos - me.c, f);
        }
      } else if (o >= a.n_slots && o < a.n_slots + a.n_planes) {
        const ContactPlane& P = a.planes[o - a.n_slots];
        const ContactPair pm = a.pair_table[mat * a.n_materials + P.material];
        const int np = capsule_plane_contacts(me, P, pts);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i >= np) break;
          const D3 rvel = point_velocity(a.cap, S, s, me.c, pts[i].pos) - D3{0.0, 0.0, 0.0};  // the plane is fixed
          D3 net;
          if (!spring_dashpot(pts[i], rvel, pm, net)) continue;
          F = F + net;
          T = T + cross(pts[i].pos - me.c, net);
        }
      }
    }
  }
  st3(a.cf, S, s, F);
  st3(a.ct, S, s, T);
}

// a grid of resident CTAs whose warps take the listed capsules in turn, as the
// pair search does: a warp whose capsules had few partners goes on to the next
// ones instead of waiting for the slowest
__global__ void __launch_bounds__(kForceThreads, kForceCtasPerSm) force_kernel(const ContactArgs a) {
  grid_dependency_wait();
  take_groups(&a.grid->evaluated, static_cast<uint32_t>(min(a.grid->live, a.n_caps)),
              [&](int64_t i) { force_one(a, a.live[i]); });
}

}  // namespace

cudaError_t launch_contact(const ContactArgs& a, cudaStream_t stream, int64_t* launches) {
  if (a.n_slots <= 0) return cudaSuccess;
  const unsigned gs = static_cast<unsigned>((a.n_slots + kThreads - 1) / kThreads);
  // the largest box extent and the bucket counts are zero when they are added
  // to: allocated zeroed, the extent set back to zero by the scatter once the
  // cell kernel has used it, and each count by the next evaluation's capsule
  // kernel; the cell kernel zeroes the running totals
  // A programmatic launch is resident before the one before it has ended, and
  // waits for that first; the kernels of one slot a thread also let the next
  // in at their start.  The capsules' launch is plain: its CTAs and those of
  // the launches after it would take the room of the step kernel that still
  // runs (8192 4-mm rods 0.51 -> 0.64 ms a step).  So is the pairs' launch,
  // whose CTAs stay for the whole search and so start on an empty chip (4096
  // rods in a box of 0.25, 1.375 -> 1.39 ms otherwise).  A step of 64 rods:
  // 76 us with plain launches, 69 so; 8192 64-element rods 267 -> 257.
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kern, unsigned grid, int threads, bool early) {
    if (e != cudaSuccess || grid == 0) return;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(static_cast<unsigned>(threads));
    lc.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = early;
    lc.attrs = at;
    lc.numAttrs = 1;
    e = cudaLaunchKernelEx(&lc, kern, a);
    ++*launches;
  };
  go(capsule_kernel, gs, kThreads, false);
  go(cell_kernel, gs, kThreads, true);
  go(range_kernel, gs, kThreads, true);
  go(scatter_kernel, gs, kThreads, true);
  const unsigned ge = static_cast<unsigned>((a.n_caps + kThreads - 1) / kThreads);
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int pper = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pper, pairs_kernel<0>, kThreads, 0);
  go(pairs_kernel<0>, static_cast<unsigned>(std::min<int64_t>(ge, static_cast<int64_t>(sms) * std::max(pper, 1))),
     kThreads, false);
  go(pairs_kernel<1>, static_cast<unsigned>(std::min<int64_t>(gs, 4 * static_cast<int64_t>(sms))), kThreads, true);
  go(force_kernel, static_cast<unsigned>(std::min<int64_t>((a.n_caps + kForceThreads - 1) / kForceThreads,
                                                           static_cast<int64_t>(sms) * kForceCtasPerSm)),
     kForceThreads, true);
  return e;
}

}  // namespace eb

// Initial data of straight rods, written on the device: one CTA a rod, one
// thread a slot, from a few hundred bytes a rod (and the velocities, if any)
// instead of 340 bytes a slot computed, staged and copied by the host.  The
// formulas are init_straight_rod's (eb_capi.cu), rounded as written there
// (this file is compiled without contraction), so the data are the same bits.
// Admitting 24 requests of four rods (62 k slots) takes 0.2 ms of host time
// instead of 3.6 ms.
#include "rod_init.h"

#include <cmath>

namespace eb {
namespace {

constexpr int kThreads = 256;

struct Nodes {
  double x, y, z;
};

__device__ __forceinline__ Nodes node(const RodSpec& r, int j) {
  const double d = static_cast<double>(j);
  return {r.origin[0] + d * r.step[0], r.origin[1] + d * r.step[1], r.origin[2] + d * r.step[2]};
}

// rest length of element i
__device__ __forceinline__ double rest_length(const RodSpec& r, int i) {
  const Nodes a = node(r, i), b = node(r, i + 1);
  const double dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
  return sqrt(dx * dx + dy * dy + dz * dz);
}

// second moment of area of an element of rest length l0 about a bending axis
// (twice it about the tangent), from its volume as the reference has it, and
// its cross section
__device__ __forceinline__ double bending_moment(const RodSpec& r, double l0, double* section) {
  const double radius = sqrt(M_1_PI * (r.area * l0) / l0);
  const double A = M_PI * (radius * radius);
  *section = A;
  return (0.25 * M_1_PI) * (A * A);
}

__global__ void __launch_bounds__(kThreads) rod_init_kernel(const RodSpec* __restrict__ specs,
                                                            const double* __restrict__ velocities, int64_t S,
                                                            double* __restrict__ state, double* __restrict__ par,
                                                            uint32_t* __restrict__ meta, RodInfo* __restrict__ rods,
                                                            int64_t* __restrict__ rod_start,
                                                            int32_t* __restrict__ rod_n) {
  __shared__ RodSpec r;
  for (unsigned i = threadIdx.x; i < sizeof(RodSpec) / sizeof(uint32_t); i += kThreads)
    reinterpret_cast<uint32_t*>(&r)[i] = reinterpret_cast<const uint32_t*>(specs + blockIdx.x)[i];
  __syncthreads();
  const int n = r.n;
  if (threadIdx.x == 0) {
    rods[r.rod] = r.info;
    rod_start[r.rod] = r.start;
    rod_n[r.rod] = n;
  }
  for (int j = threadIdx.x; j <= n; j += kThreads) {
    const int64_t g = r.start + j;
    const bool elem = j < n, vor = j < n - 1;
    auto st = [&](int f, double v) { state[f * S + g] = v; };
    auto pr = [&](int f, double v) { par[f * S + g] = v; };
    const Nodes x = node(r, j);
    st(kStX, x.x);
    st(kStX + 1, x.y);
    st(kStX + 2, x.z);
    for (int d = 0; d < 3; ++d) {
      st(kStV + d, r.velocity >= 0 ? velocities[r.velocity + static_cast<int64_t>(d) * (n + 1) + j] : 0.0);
      st(kStW + d, 0.0);
    }
    for (int k = 0; k < 9; ++k) st(kStQ + k, elem ? r.rows[k] : 0.0);
    for (int f = 0; f < kParamFields; ++f) pr(f, 0.0);
    const double before = j > 0 ? rest_length(r, j - 1) : 0.0;
    // each node takes half the mass of the element before it, then of its own
    double mass = 0.0;
    if (j > 0) mass = mass + 0.5 * (r.density * (r.area * before));
    // benign values in the entries without an element or Voronoi point
    double l0 = 1.0, D0 = 1.0, J[3] = {1.0, 1.0, 1.0}, Jinv[3] = {1.0, 1.0, 1.0};
    if (elem) {
      l0 = rest_length(r, j);
      mass = mass + 0.5 * (r.density * (r.area * l0));
      pr(kVol, r.area * l0);
      double A;
      const double I = bending_moment(r, l0, &A);
      const double alpha_c = 13.5 / 14.0;
      pr(kShear, r.shear * (A * alpha_c));
      pr(kShear + 1, r.shear * (A * alpha_c));
      pr(kShear + 2, r.youngs * A);
      for (int d = 0; d < 3; ++d) {
        J[d] = (d == 2 ? 2.0 * I : I) * r.density * l0;
        Jinv[d] = 1.0 / J[d];
      }
      if (vor) {
        const double l1 = rest_length(r, j + 1);
        double A1;
        const double I1 = bending_moment(r, l1, &A1);
        D0 = 0.5 * (l0 + l1);
        for (int d = 0; d < 3; ++d) {
          const double stiff = d == 2 ? r.shear : r.youngs;
          pr(kBend + d, (l0 * stiff * (d == 2 ? 2.0 * I : I) + l1 * stiff * (d == 2 ? 2.0 * I1 : I1)) / (l0 + l1));
        }
      }
      if (r.damped) pr(kNuT, r.nu_t);
    }
    if (r.damped) pr(kNuF, r.nu_f);
    pr(kMass, mass);
    pr(kL0, l0);
    pr(kD0, D0);
    for (int d = 0; d < 3; ++d) {
      pr(kJ + d, J[d]);
      pr(kJinv + d, Jinv[d]);
    }
    uint32_t m = r.rod << kRodShift;
    if (elem) m |= kElem;
    if (vor) m |= kVor;
    if (j == 0) m |= kFirst;
    if (j == n) m |= kLastNode;
    if (j == n - 1) m |= kLastElem;
    meta[g] = m;
  }
}

// A rod's rows straight into the pinned host arena, one CTA a rod.  (A copy of
// 18 rows of 4 KB a bin through the copy engine, and an energy kernel a
// request, took 3.6 ms for 24 requests of four rods; 1.2 ms so.)
__global__ void __launch_bounds__(kThreads) rod_result_kernel(const RodRef* __restrict__ refs, int64_t S,
                                                              const double* __restrict__ state,
                                                              const int64_t* __restrict__ rod_start,
                                                              const int32_t* __restrict__ rod_n,
                                                              const double* __restrict__ e0,
                                                              const double* __restrict__ e1) {
  const RodRef r = refs[blockIdx.x];
  const int64_t g = rod_start[r.rod];
  const int W = rod_n[r.rod] + 1;
  for (int f = 0; f < kStateFields; ++f)
    for (int j = threadIdx.x; j < W; j += kThreads) r.result[f * W + j] = state[f * S + g + j];
  if (threadIdx.x < 5) {
    r.energies[threadIdx.x] = e0[5 * r.rod + threadIdx.x];
    r.energies[r.final_at + threadIdx.x] = e1[5 * r.rod + threadIdx.x];
  }
}

}  // namespace

cudaError_t launch_rod_init(const RodSpec* specs, int64_t count, const double* velocities, int64_t stride,
                            double* state, double* par, uint32_t* meta, RodInfo* rods, int64_t* rod_start,
                            int32_t* rod_n, cudaStream_t stream) {
  if (count <= 0) return cudaSuccess;
  rod_init_kernel<<<static_cast<unsigned>(count), kThreads, 0, stream>>>(specs, velocities, stride, state, par, meta,
                                                                        rods, rod_start, rod_n);
  return cudaGetLastError();
}

cudaError_t launch_rod_result(const RodRef* refs, int64_t count, int64_t stride, const double* state,
                              const int64_t* rod_start, const int32_t* rod_n, const double* e0, const double* e1,
                              cudaStream_t stream) {
  if (count <= 0) return cudaSuccess;
  rod_result_kernel<<<static_cast<unsigned>(count), kThreads, 0, stream>>>(refs, stride, state, rod_start, rod_n, e0,
                                                                          e1);
  return cudaGetLastError();
}

}  // namespace eb

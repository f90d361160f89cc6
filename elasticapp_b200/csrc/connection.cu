// Connections (joints) between rods.
//
// The reference connects two rods with a user-written force and torque rule
// (simulator->connect(rod_a, at(i)).to(rod_b, at(j)).with(generator),
// elastica/Simulator/Connections/, applied among the pre-dynamic updates
// after the internal loads).  Here the rules are built in: the joint of the
// reference's hinge-joint example (examples/hinge_joint/
// HingeJointCaseStudy.cpp:96-150), with its index conventions:
//
//   force (every joint): d = x_b[j] - x_a[i + 1],
//     F = k d - nu ((v_b[j] - v_a[i + 1]) . u) u,  u = d / |d|
//     (Blaze's normalize multiplies by 1/|d|, or by 0 when |d| = 0),
//     rod a's node i + 1 gains F, rod b's node j loses it;
//   torque (hinge joints): l = x_b[j + 1] - x_b[j], f = -k_rot (l . n) n,
//     tau = l x f; rod a's element i loses Q_a tau and rod b's element j
//     gains Q_b tau (material frame).
//
// Positions are those of the force evaluation: drifted by the substep's
// first drift, with the clamp's value constraint.  One thread per loaded slot
// evaluates and sums the joints acting on it in connection order (rod a's
// share before rod b's), so the sums are deterministic; where a slot carries
// many joints, one thread per joint evaluates them in a launch before.  Torques
// are summed in the lab frame; the step kernel recasts them by the element's
// directors.  Built with --fmad=false, like the CPU restatement.
#include <cuda_runtime.h>

#include "bulk_copy.cuh"
#include "eb_internal.h"
#include "joint.h"

namespace eb {
namespace {

struct P3 {
  double x, y, z;
};

// joints a slot may carry for its thread to evaluate them itself.  A joint
// more is a chain of loads, a root and divisions more in that thread: 64 rods
// with k others jointed to one node, us a step with one launch and with two,
// k = 2: 10.3 and 10.7, 4: 13.4 and 11.5, 8: 18.3 and 12.7, 16: 27.9 and 15.0
// (hinges 10.4 and 11.8, 13.4 and 12.4, 18.4 and 13.4, 27.9 and 16.1)
constexpr int kFewJoints = 2;

__device__ __forceinline__ P3 node_position(const JointArgs& a, int64_t g) {
  const uint32_t m = a.meta[g];
  double t[3];
  if (clamp_position(a.rods[m >> kRodShift], g, t)) return {t[0], t[1], t[2]};
  const int64_t S = a.stride;
  const double* in = a.state;
  return {in[kStX * S + g] + a.pre * in[kStV * S + g], in[(kStX + 1) * S + g] + a.pre * in[(kStV + 1) * S + g],
          in[(kStX + 2) * S + g] + a.pre * in[(kStV + 2) * S + g]};
}

__device__ __forceinline__ P3 node_velocity(const JointArgs& a, int64_t g) {
  const int64_t S = a.stride;
  return {a.state[kStV * S + g], a.state[(kStV + 1) * S + g], a.state[(kStV + 2) * S + g]};
}

// force of a joint on rod a's node (rod b's loses it)
__device__ __forceinline__ P3 joint_force(const JointArgs& a, const JointDev& J) {
  const P3 xa = node_position(a, J.node_a), xb = node_position(a, J.node_b);
  const P3 va = node_velocity(a, J.node_a), vb = node_velocity(a, J.node_b);
  const P3 d = {xb.x - xa.x, xb.y - xa.y, xb.z - xa.z};
  const P3 fel = {J.k * d.x, J.k * d.y, J.k * d.z};
  const double len = sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
  const double il = len != 0.0 ? 1.0 / len : len;
  const P3 u = {d.x * il, d.y * il, d.z * il};
  const P3 dv = {vb.x - va.x, vb.y - va.y, vb.z - va.z};
  const double vr = dv.x * u.x + dv.y * u.y + dv.z * u.z;
  const P3 vel = {vr * u.x, vr * u.y, vr * u.z};
  const double mnu = -J.nu;
  return {fel.x + mnu * vel.x, fel.y + mnu * vel.y, fel.z + mnu * vel.z};
}

// torque of a hinge on rod b's element (rod a's loses it), lab frame
__device__ __forceinline__ P3 joint_torque(const JointArgs& a, const JointDev& J) {
  const P3 xb = node_position(a, J.node_b), xb1 = node_position(a, J.node_b + 1);
  const P3 l = {xb1.x - xb.x, xb1.y - xb.y, xb1.z - xb.z};
  const double s = (-J.k_rot) * (l.x * J.normal[0] + l.y * J.normal[1] + l.z * J.normal[2]);
  const P3 f = {s * J.normal[0], s * J.normal[1], s * J.normal[2]};
  return {l.y * f.z - l.z * f.y, l.z * f.x - l.x * f.z, l.x * f.y - l.y * f.x};
}

__global__ void joint_eval_kernel(const JointArgs a) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  grid_dependency_launch();
  grid_dependency_wait();
  if (c >= a.n_joints) return;
  const JointDev J = a.joints[c];
  const P3 f = joint_force(a, J);
  const P3 tau = J.kind == kJointHinge ? joint_torque(a, J) : P3{0.0, 0.0, 0.0};
  double* o = a.out + 6 * static_cast<int64_t>(c);
  o[0] = f.x;
  o[1] = f.y;
  o[2] = f.z;
  o[3] = tau.x;
  o[4] = tau.y;
  o[5] = tau.z;
}

// slots [0, n_force_slots) of the combined index range sum forces, the rest
// torques; entry e of a slot's list is 2 * joint + (1 if subtracted).
// kEvaluate: the joints' loads are evaluated here (by every slot they act on)
// instead of read from the table that joint_eval_kernel wrote
template <bool kEvaluate>
__global__ void joint_apply_kernel(const JointArgs a) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  grid_dependency_launch();
  grid_dependency_wait();
  const bool force = t < a.n_force_slots;
  const int64_t k = force ? t : t - a.n_force_slots;
  if (!force && k >= a.n_torque_slots) return;
  const int64_t* slot = force ? a.force_slot : a.torque_slot;
  const int64_t* off = force ? a.force_off : a.torque_off;
  const int32_t* src = force ? a.force_src : a.torque_src;
  double* dst = force ? a.joint_force : a.joint_torque;
  const int col = force ? 0 : 3;
  double sx = 0.0, sy = 0.0, sz = 0.0;
  for (int64_t e = off[k]; e < off[k + 1]; ++e) {
    const int32_t v = src[e];
    P3 o;
    if (kEvaluate) {
      const JointDev J = a.joints[v >> 1];
      o = force ? joint_force(a, J) : joint_torque(a, J);
    } else {
      const double* r = a.out + 6 * static_cast<int64_t>(v >> 1) + col;
      o = {r[0], r[1], r[2]};
    }
    if (v & 1) {
      sx = sx - o.x;
      sy = sy - o.y;
      sz = sz - o.z;
    } else {
      sx = sx + o.x;
      sy = sy + o.y;
      sz = sz + o.z;
    }
  }
  const int64_t g = slot[k], S = a.stride;
  dst[g] = sx;
  dst[S + g] = sy;
  dst[2 * S + g] = sz;
}

}  // namespace

// A launch is a few microseconds of latency and more of host time, so where no
// slot carries more than two joints one launch evaluates and sums (a joint
// is then evaluated by each slot it acts on), and a launch begins before the
// one before it has ended, as the step kernel after it does.  A chain of 32
// links: 17.5 us a step with two plain launches, 10.3 with two of these,
// 8.7 with one.
cudaError_t launch_joints(const JointArgs& a, cudaStream_t stream, int64_t* launches) {
  if (a.n_joints <= 0) return cudaSuccess;
  constexpr int kThreads = 128;
  cudaLaunchConfig_t lc = {};
  lc.blockDim = dim3(kThreads);
  lc.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  const int64_t n = a.n_force_slots + a.n_torque_slots;
  const dim3 apply(static_cast<unsigned>((n + kThreads - 1) / kThreads));
  if (a.max_per_slot <= kFewJoints) {
    lc.gridDim = apply;
    ++*launches;
    return cudaLaunchKernelEx(&lc, joint_apply_kernel<true>, a);
  }
  lc.gridDim = dim3(static_cast<unsigned>((a.n_joints + kThreads - 1) / kThreads));
  if (cudaError_t e = cudaLaunchKernelEx(&lc, joint_eval_kernel, a)) return e;
  lc.gridDim = apply;
  *launches += 2;
  return cudaLaunchKernelEx(&lc, joint_apply_kernel<false>, a);
}

}  // namespace eb

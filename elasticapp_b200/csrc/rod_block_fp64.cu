// Resident multi-step PositionVerlet kernel for batches of whole rods.
//
// The streaming step kernel (rod_step_fp64.cu) moves the full state through
// HBM every step.  Rods are independent, so a CTA can instead own a group of
// whole rods, stage their state and parameters into shared memory once, run
// many steps entirely on chip and write the state back once: HBM traffic per
// element-step falls by the number of steps per launch and the step becomes
// arithmetic-bound.
//
// Work list: CTA c owns the slots gmap[cta_start[c] .. cta_start[c + 1]),
// always whole rods (the host packs rods best fit decreasing into CTAs of at
// most kCap slots; serving launches read consecutive slot ranges from a CTA
// table instead).  Every phase loops its threads over the CTA's slots; all
// per-slot data lives in shared-memory rows, so any thread count works.
//
// Step structure: the substeps of the streaming kernel in two phases with one
// barrier after each (element and Voronoi terms; loads, kick and drifts).
//
// Rod pairs (kPair): a rod of up to 1039 elements runs on a cluster of two
// CTAs, each holding half of its slots.  The threads of the slots at the split
// write what the partner's neighbours read to copies in the partner's shared
// memory as well (distributed shared memory), so every read is local, and the
// barriers that order a phase's writes before the next phase's neighbour
// reads become cluster barriers.  (Reads that go to the partner past the
// split cost every slot a test and an address, and registers spilled.)  Serving
// launches mix pairs and single CTAs in one cluster launch; a single CTA takes
// only CTA barriers.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "eb_internal.h"
#include "rod_fast.cuh"

namespace eb {
namespace {

using D3 = Vec3<double>;

// shared-memory rows (each kCap doubles)
enum BlockRow : int {
  bX = 0, bV = 3, bQ = 6, bW = 15,  // state (kStateFields rows)
  // parameters (of the divisors l0 and D0 also the reciprocals, formed once a
  // launch; explicit damping's rates stay in global memory)
  bMass = 18, bL0 = 19, bD0 = 20, bSig0 = 21, bKap0 = 24, bShear = 27, bBend = 30, bJ = 33, bJinv = 36,
  bInvL0 = 39, bInvD0 = 40,
  // exchanged once per force evaluation: internal force of the element, the
  // couple terms of the Voronoi point
  bF = 41, bG = 44, bH = 47,
  // element-local torque terms and dilatation, where a thread steps several slots
  bTl = 50, bE = 53,
  kBlockRows = 54
};

template <int kRow>
struct BRows {
  double* base;
  __device__ __forceinline__ double& at(int r, int s) const { return base[r * kRow + s]; }
  __device__ __forceinline__ D3 get3(int r, int s) const {
    return {base[r * kRow + s], base[(r + 1) * kRow + s], base[(r + 2) * kRow + s]};
  }
  __device__ __forceinline__ void put3(int r, int s, D3 v) const {
    base[r * kRow + s] = v.x;
    base[(r + 1) * kRow + s] = v.y;
    base[(r + 2) * kRow + s] = v.z;
  }
};

// entries of a row: a CTA of a pair also holds copies of the partner's
// neighbouring slots, one before its first slot and two after its last
template <int kCap, bool kPair>
constexpr int block_row() { return kPair ? kCap + 4 : kCap; }

// kServe: the CTA's slot range, step count, time step and environment come
// from serve[blockIdx.x] (serving launches)
// kGather: cta_start indexes gmap, the list of the CTA's slots (rods that
// need not be neighbours in the slot layout)
// kPair: cluster launch of CTA pairs; with kServe, CTAs 2i and 2i + 1 form a
// pair when both serve entries say so and run the same step count, and are
// single CTAs otherwise; without kServe every cluster is a pair
// kStepper: 0 PositionVerlet, 1 PEFRL (four force evaluations a step), 2
// VelocityVerlet (two: kick dt/2, drift dt, kick dt/2)
// two CTAs per SM for the CTAs of at most 264 slots (437 B a slot)
template <int kCap>
constexpr int block_min_ctas() { return kCap <= 264 ? 2 : 1; }

__device__ __forceinline__ double squared_length(D3 d) {
  return __fma_rn(d.z, d.z, __fma_rn(d.y, d.y, __dmul_rn(d.x, d.x)));
}

// a slot's state and what its force evaluation hands to its kick
struct SlotState {
  D3 x, v, w;
  double q[9];
};
struct SlotTerms {
  D3 f, g, h, tl;  // internal force of the element, couple terms of the Voronoi point, element-local torque terms
  double e;        // dilatation
};

template <int kCap, int kThreads, bool kDamped, bool kServe, bool kGather = false, bool kPair = false,
          int kStepper = 0>
__global__ void __launch_bounds__(kThreads, block_min_ctas<kCap>()) rod_block_fp64_kernel(const StepArgs a, const int64_t* cta_start,
                                                                    int n_steps_launch, const ServeCta* serve,
                                                                    const int32_t* gmap) {
  extern __shared__ __align__(128) double smem[];
  constexpr int kRow = block_row<kCap, kPair>();
  const BRows<kRow> R{smem + (kPair ? 1 : 0)};
  uint32_t* meta_s = reinterpret_cast<uint32_t*>(smem + kBlockRows * kRow);
  // per slot: which clamp holds it, the torque, the damper (SlotHits)
  uint8_t* hit_s = reinterpret_cast<uint8_t*>(meta_s + kCap);

  const int tid = threadIdx.x;
  int64_t g0;
  int count, n_steps = n_steps_launch;
  double dt = a.dt, hdt = a.half_dt;
  uint32_t flags = a.sim_flags;
  double gvec[3] = {a.gravity[0], a.gravity[1], a.gravity[2]};
  if constexpr (kServe) {
    const ServeCta& sc = serve[blockIdx.x];
    g0 = sc.start;
    count = sc.count;
    n_steps = min(n_steps_launch, sc.steps);
    dt = sc.dt;
    hdt = sc.half_dt;
    flags = sc.flags;
    gvec[0] = sc.gravity[0];
    gvec[1] = sc.gravity[1];
    gvec[2] = sc.gravity[2];
  } else {
    g0 = cta_start[blockIdx.x];
    count = static_cast<int>(cta_start[blockIdx.x + 1] - g0);
  }
  if (n_steps <= 0) return;
  const int64_t S = a.stride;
  // the partner's rows, at the place of this CTA's slot 0 (left half: past the
  // end of the right half's left copy; right half: the left half's count)
  BRows<kRow> peer = R;
  bool paired = false, left = false;
  if constexpr (kPair) {
    const unsigned partner = blockIdx.x ^ 1u;
    int pcount = 0;
    if constexpr (kServe) {
      const ServeCta& sc = serve[blockIdx.x];
      const ServeCta& o = serve[partner];
      paired = sc.pair != 0 && o.pair != 0 && sc.steps == o.steps;
      pcount = o.count;
    } else {
      paired = true;
      pcount = static_cast<int>(cta_start[partner + 1] - cta_start[partner]);
    }
    if (paired) {
      cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
      left = cl.block_rank() == 0;
      peer.base = cl.map_shared_rank(R.base, cl.block_rank() ^ 1u) + (left ? -count : pcount);
    }
  }
  // orders this phase's writes before the next phase's neighbour reads
  auto sync_neighbours = [&]() {
    if constexpr (kPair) {
      if (paired) {
        cooperative_groups::this_cluster().sync();
        return;
      }
    }
    __syncthreads();
  };
  const bool any_rod = (flags & (kSimClamp | kSimDamper | kSimEndTorque)) != 0;

  // global slot of the CTA's slot s
  auto slot_of = [&](int s) -> int64_t { return kGather ? static_cast<int64_t>(gmap[g0 + s]) : g0 + s; };

  // ---- stage state, parameters and slot metadata (coalesced loads)
  for (int s = tid; s < count; s += kThreads) {
    const int64_t g = slot_of(s);
    const uint32_t m = a.meta[g];
    meta_s[s] = m;
    hit_s[s] = static_cast<uint8_t>(any_rod ? slot_hits(a.rods[m >> kRodShift], g) : 0u);
    // loads in flight together, a group at a time: one CTA fills an SM, so
    // nothing else hides their latency
    auto stage = [&](const double* field, int n, int row, auto group) {
      constexpr int kGroup = decltype(group)::value;
#pragma unroll 1
      for (int f = 0; f < n; f += kGroup) {
        double v[kGroup];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) v[k] = field[(f + k) * S + g];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) R.at(row + f + k, s) = v[k];
      }
    };
    stage(a.in, kStateFields, bX, std::integral_constant<int, 18>{});
    // (kSig0 .. kBend and kJ, kJinv are consecutive fields and rows)
    stage(a.par + kSig0 * S, 12, bSig0, std::integral_constant<int, 12>{});
    stage(a.par + kJ * S, 6, bJ, std::integral_constant<int, 6>{});
    const double l0 = a.par[kL0 * S + g], d0 = a.par[kD0 * S + g], m0 = a.par[kMass * S + g];
    R.at(bL0, s) = l0;
    R.at(bD0, s) = d0;
    R.at(bMass, s) = m0;
    R.at(bInvL0, s) = 1.0 / l0;
    R.at(bInvD0, s) = 1.0 / d0;
  }
  sync_neighbours();

  // Substeps: PositionVerlet (drift dt/2, kick dt, drift dt/2), or PEFRL's
  // four kicks with their drifts (in units of dt; compile-time constants)
  constexpr bool kPefrl = kStepper == 1, kVelocity = kStepper == 2;
  constexpr int nsub = kPefrl ? 4 : (kVelocity ? 2 : 1);
  auto pefrl_pre = [](int j) -> double {  // drift before force evaluation j
    return j == 0 ? kPefrlXi : (j == 2 ? 1.0 - 2.0 * (kPefrlChi + kPefrlXi) : kPefrlChi);
  };
  auto pefrl_kick = [](int j) -> double {
    return (j == 0 || j == 3) ? 0.5 * (1.0 - 2.0 * kPefrlLambda) : kPefrlLambda;
  };

  auto load_state = [&](int s, SlotState& m) {
    m.x = R.get3(bX, s);
    m.v = R.get3(bV, s);
    m.w = R.get3(bW, s);
#pragma unroll
    for (int k = 0; k < 9; ++k) m.q[k] = R.at(bQ + k, s);
  };
  // the state the neighbours read (their positions, velocities, directors)
  auto publish = [&](int s, const SlotState& m) {
    R.put3(bX, s, m.x);
    R.put3(bV, s, m.v);
#pragma unroll
    for (int k = 0; k < 9; ++k) R.at(bQ + k, s) = m.q[k];
    if (kPair && paired && !left && s < 2) {  // the left half's copies after its last slot
      peer.put3(bX, s, m.x);
      peer.put3(bV, s, m.v);
#pragma unroll
      for (int k = 0; k < 9; ++k) peer.at(bQ + k, s) = m.q[k];
    }
  };
  // drift of a slot by c (x += c v, Q <- exp(-c [w]x) Q), once or twice:
  // the closing drift of a step and the first of the next are two rotations
  // by the same coefficients, formed once and applied one after the other, so a run
  // rounds alike however it is cut into launches (and one rotation by 2 c
  // would not be the same: the axis guard of the reference makes it differ by
  // 1e-14 a step, which stiff rods amplify)
  auto drift = [&](SlotState& m, uint32_t meta, double c, bool twice) {
    m.x = {m.x.x + c * m.v.x, m.x.y + c * m.v.y, m.x.z + c * m.v.z};
    if (twice) m.x = {m.x.x + c * m.v.x, m.x.y + c * m.v.y, m.x.z + c * m.v.z};
    if (meta & kElem) {
      const Rotation r = rotation(c * m.w.x, c * m.w.y, c * m.w.z);
      rotate(m.q, r);
      if (twice) rotate(m.q, r);
    }
  };
  auto clamp_value = [&](SlotState& m, uint32_t meta, uint32_t hit) {
    if (!(hit & (kHitClamp0 | kHitClamp1))) return;
    const RodInfo& ri = a.rods[meta >> kRodShift];
    const double* tx = (hit & kHitClamp0) ? ri.clamp_x : ri.clamp2_x;
    const double* tq = (hit & kHitClamp0) ? ri.clamp_Q : ri.clamp2_Q;
    m.x = {tx[0], tx[1], tx[2]};
    if (meta & kElem) {
#pragma unroll
      for (int k = 0; k < 9; ++k) m.q[k] = tq[k];
    }
  };

  // Element s (strain, internal force, element-local torque terms) and
  // Voronoi point s (curvature and couple; the length of element s + 1 is
  // recomputed rather than exchanged).  The quotients are those of the plain
  // expressions (rod_fast.cuh): one reciprocal square root gives l and 1 / l,
  // 1 / e starts from l0 / l and 1 / (e l0) from 1 / l, and division by the
  // rest lengths uses their stored reciprocals.
  auto evaluate = [&](int s, uint32_t meta, const SlotState& m, SlotTerms& o) {
    o.f = o.g = o.h = o.tl = D3{0.0, 0.0, 0.0};
    o.e = 1.0;
    if (meta & kElem) {
      const D3 xn = R.get3(bX, s + 1);
      const D3 dx = xn - m.x;
      const Length len = length_of(squared_length(dx));
      const double l = len.l, il = len.il;
      const D3 t = {dx.x * il, dx.y * il, dx.z * il};
      const double l0 = R.at(bL0, s);
      const double e = div_from(l, l0, R.at(bInvL0, s));
      const D3 qt = matvec(m.q, t);
      const D3 sigma = {qt.x * e, qt.y * e, qt.z * e - 1.0};
      const D3 d = sigma - R.get3(bSig0, s);
      const D3 sh = R.get3(bShear, s);
      const D3 nl = {sh.x * d.x, sh.y * d.y, sh.z * d.z};
      const double ie = rcp_from_rough(e, l0 * il);
      o.f = scale(mattranspvec(m.q, nl), ie);
      const D3 J = R.get3(bJ, s);
      const D3 jwe = {J.x * m.w.x * ie, J.y * m.w.y * ie, J.z * m.w.z * ie};
      const D3 dv = R.get3(bV, s + 1) - m.v;
      const double el0 = e * l0;
      const double rate = div_from(dot(t, dv), el0, rcp_from_rough(el0, il));
      o.tl = scale(cross(qt, nl), l0) + cross(jwe, m.w) + scale(jwe, rate);
      o.e = e;
      if (meta & kVor) {
        double qn[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) qn[k] = R.at(bQ + k, s + 1);
        const double D0 = R.at(bD0, s);
        const D3 kappa = curvature(m.q, qn, D0);
        const double ln = length_of(squared_length(R.get3(bX, s + 2) - xn)).l;
        const double eps = div_from(0.5 * (l + ln), D0, R.at(bInvD0, s));
        const double cube = eps * eps * eps;
        const double ic = rcp_from(cube, rcp_near(cube));
        const D3 dk = kappa - R.get3(bKap0, s);
        const D3 B = R.get3(bBend, s);
        const D3 tau = {B.x * dk.x, B.y * dk.y, B.z * dk.z};
        o.g = scale(tau, ic);
        o.h = scale(cross(kappa, tau), ic * D0);
      }
    }
    R.put3(bF, s, o.f);
    R.put3(bG, s, o.g);
    R.put3(bH, s, o.h);
    if (kPair && paired && left && s == count - 1) {  // the right half's copy before its first slot
      peer.put3(bF, s, o.f);
      peer.put3(bG, s, o.g);
      peer.put3(bH, s, o.h);
    }
  };

  // loads, torques, accelerations, kick (by kc dt) and rate constraints
  // what a slot's kick needs of its mass and its rod's damper
  struct SlotConst {
    double im, damper_t, damp;  // 1 / m, exp(-nu_t dt), -nu_r m_e
  };
  auto slot_const = [&](int s, int64_t g, uint32_t meta, uint32_t hit) -> SlotConst {
    const double m = R.at(bMass, s);
    SlotConst c{1.0 / m, 1.0, 0.0};
    if (hit & kHitDamper) {
      const RodInfo& ri = a.rods[meta >> kRodShift];
      c.damper_t = ri.damper_t;
      if (meta & kElem) {
        const double mn = a.par[kMass * S + g + 1];  // the element's other node
        double em = 0.5 * (m + mn);
        if (meta & kFirst) em += 0.5 * m;
        if (meta & kLastElem) em += 0.5 * mn;
        c.damp = -ri.damper_r * em;
      }
    }
    return c;
  };
  // (g: the global slot)
  auto kick = [&](int s, int64_t g, uint32_t meta, uint32_t hit, const SlotTerms& o, const SlotConst& c, double kc,
                  SlotState& n) {
    const bool first = (meta & kFirst) != 0;
    const double kdt = kc == 1.0 ? dt : kc * dt;
    // the damper's time: the kick's share of dt for PEFRL, the full dt for
    // VelocityVerlet (its constants hold dt and act after each kick)
    const double dc = kVelocity ? 1.0 : kc;
    const double ddt = dc == 1.0 ? dt : kdt;
    const double m = R.at(bMass, s);
    D3 v = n.v, w = n.w;
    D3 F = o.f;
    if (!first) F = F - R.get3(bF, s - 1);
    if (kDamped) {
      const double cf = m * a.par[kNuF * S + g];
      F = {F.x - cf * v.x, F.y - cf * v.y, F.z - cf * v.z};
    }
    if (flags & kSimGravity) F = F + D3{gvec[0] * m, gvec[1] * m, gvec[2] * m};
    v = {v.x + kdt * (F.x * c.im), v.y + kdt * (F.y * c.im), v.z + kdt * (F.z * c.im)};
    if (meta & kElem) {
      const double e = o.e;
      D3 T = o.g;
      D3 Q2 = o.h;
      if (!first) {
        T = T - R.get3(bG, s - 1);
        Q2 = Q2 + R.get3(bH, s - 1);
      }
      T = T + scale(Q2, 0.5) + o.tl;
      if (kDamped) {
        const double ct = 0.5 * (m + a.par[kMass * S + g + 1]) * a.par[kNuT * S + g];
        T = {T.x - ct * w.x, T.y - ct * w.y, T.z - ct * w.z};
      }
      if (hit & kHitTorque) {
        const RodInfo& ri = a.rods[meta >> kRodShift];
        T = T + matvec(n.q, D3{ri.end_torque[0], ri.end_torque[1], ri.end_torque[2]});
      }
      const D3 ji = R.get3(bJinv, s);
      w = {w.x + kdt * (ji.x * T.x * e), w.y + kdt * (ji.y * T.y * e), w.z + kdt * (ji.z * T.z * e)};
      if (hit & kHitDamper) {
        const double y = c.damp * ddt * e;
        const double ex = exp(y * ji.x);
        // (a circular cross section: one factor for both bending directions)
        w = {w.x * ex, w.y * (ji.y == ji.x ? ex : exp(y * ji.y)), w.z * exp(y * ji.z)};
      }
    }
    if (hit & (kHitClamp0 | kHitClamp1)) {
      v = D3{0.0, 0.0, 0.0};
      w = D3{0.0, 0.0, 0.0};
    }
    // exp(-nu_t dt) for a kick of dt; a fractional kick scales the exponent
    if (hit & kHitDamper) v = scale(v, dc == 1.0 ? c.damper_t : exp(log(c.damper_t) * dc));
    n.v = v;
    n.w = w;
  };
  // the drifts between one kick and the next force evaluation, the
  // constraint's value and the write-out
  auto advance = [&](int s, uint32_t meta, uint32_t hit, bool last_of_step, int sub, SlotState& m) {
    if (!last_of_step)
      drift(m, meta, kVelocity ? dt : pefrl_pre(sub + 1) * dt, false);
    else if (!kVelocity)  // (VelocityVerlet's next step starts with a kick: the clamp's value alone)
      drift(m, meta, kPefrl ? kPefrlXi * dt : hdt, true);
    clamp_value(m, meta, hit);
    publish(s, m);
  };
  // closing drift of the last step and write-back
  const double fin = kPefrl ? kPefrlXi * dt : (kVelocity ? 0.0 : hdt);
  auto finish = [&](int64_t g, uint32_t meta, SlotState& m) {
    if (!kVelocity) drift(m, meta, fin, false);
    a.out[kStX * S + g] = m.x.x;
    a.out[(kStX + 1) * S + g] = m.x.y;
    a.out[(kStX + 2) * S + g] = m.x.z;
    a.out[kStV * S + g] = m.v.x;
    a.out[(kStV + 1) * S + g] = m.v.y;
    a.out[(kStV + 2) * S + g] = m.v.z;
    if (meta & kElem) {
#pragma unroll
      for (int k = 0; k < 9; ++k) a.out[(kStQ + k) * S + g] = m.q[k];
      a.out[kStW * S + g] = m.w.x;
      a.out[(kStW + 1) * S + g] = m.w.y;
      a.out[(kStW + 2) * S + g] = m.w.z;
    }
  };
  // Two phases per force evaluation, one barrier after each (for a pair, the
  // partner must also not leave, and free its rows, while this CTA still
  // reads them).  A CTA of at most kThreads slots keeps each slot's state and
  // terms in its thread's registers from phase to phase and launch to end; a
  // longer one keeps them in their rows.
  if (count <= kThreads) {
    const bool on = tid < count;
    const uint32_t meta = on ? meta_s[tid] : 0u, hit = on ? hit_s[tid] : 0u;
    int64_t g = 0;
    SlotConst c;
    SlotState m;
    SlotTerms t;
    if (on) {
      g = slot_of(tid);
      c = slot_const(tid, g, meta, hit);
      load_state(tid, m);
      // first drift of the first step and the clamp's value constraint
      // (VelocityVerlet starts with a kick: no drift, the clamp's value alone)
      if (!kVelocity) drift(m, meta, kPefrl ? kPefrlXi * dt : hdt, false);
      clamp_value(m, meta, hit);
      publish(tid, m);
    }
    sync_neighbours();
    for (int step = 0; step < n_steps; ++step)
      for (int sub = 0; sub < nsub; ++sub) {
        if (on) evaluate(tid, meta, m, t);
        sync_neighbours();
        if (on) {
          kick(tid, g, meta, hit, t, c, kPefrl ? pefrl_kick(sub) : (kVelocity ? 0.5 : 1.0), m);
          if (sub + 1 < nsub || step + 1 < n_steps) advance(tid, meta, hit, sub + 1 == nsub, sub, m);
        }
        sync_neighbours();
      }
    if (on) finish(g, meta, m);
    return;
  }
  for (int s = tid; s < count; s += kThreads) {
    SlotState m;
    load_state(s, m);
    if (!kVelocity) drift(m, meta_s[s], kPefrl ? kPefrlXi * dt : hdt, false);
    clamp_value(m, meta_s[s], hit_s[s]);
    publish(s, m);
  }
  sync_neighbours();
  for (int step = 0; step < n_steps; ++step)
    for (int sub = 0; sub < nsub; ++sub) {
      for (int s = tid; s < count; s += kThreads) {
        SlotState m;
        SlotTerms t;
        load_state(s, m);
        evaluate(s, meta_s[s], m, t);
        R.put3(bTl, s, t.tl);
        R.at(bE, s) = t.e;
      }
      sync_neighbours();
      for (int s = tid; s < count; s += kThreads) {
        const uint32_t meta = meta_s[s], hit = hit_s[s];
        SlotState m;
        load_state(s, m);
        const SlotTerms t = {R.get3(bF, s), R.get3(bG, s), R.get3(bH, s), R.get3(bTl, s), R.at(bE, s)};
        const int64_t g = slot_of(s);
        kick(s, g, meta, hit, t, slot_const(s, g, meta, hit), kPefrl ? pefrl_kick(sub) : (kVelocity ? 0.5 : 1.0), m);
        if (sub + 1 < nsub || step + 1 < n_steps)
          advance(s, meta, hit, sub + 1 == nsub, sub, m);
        else
          publish(s, m);
        R.put3(bW, s, m.w);
      }
      sync_neighbours();
    }
  for (int s = tid; s < count; s += kThreads) {
    SlotState m;
    load_state(s, m);
    finish(slot_of(s), meta_s[s], m);
  }
}

template <int kCap, int kThreads, bool kServe = false, bool kGather = false, bool kPair = false>
cudaError_t launch_block_cfg(const StepArgs& args, const int64_t* cta_start, int n_ctas, int n_steps, bool damped,
                             cudaStream_t stream, const ServeCta* serve = nullptr, const int32_t* gmap = nullptr) {
  const size_t bytes = size_t(kBlockRows) * block_row<kCap, kPair>() * sizeof(double) +
                       size_t(kCap) * (sizeof(uint32_t) + sizeof(uint8_t));
  auto go = [&](auto kern) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
    if constexpr (kPair) {
      // clusters of two CTAs; the grid is a whole number of clusters
      if (n_ctas % 2 != 0) return cudaErrorInvalidValue;
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3(static_cast<unsigned>(n_ctas));
      lc.blockDim = dim3(kThreads);
      lc.dynamicSmemBytes = bytes;
      lc.stream = stream;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      lc.attrs = at;
      lc.numAttrs = 1;
      return cudaLaunchKernelEx(&lc, kern, args, cta_start, n_steps, serve, gmap);
    } else {
      kern<<<n_ctas, kThreads, bytes, stream>>>(args, cta_start, n_steps, serve, gmap);
      return cudaGetLastError();
    }
  };
  if constexpr (!kServe) {  // serving launches are PositionVerlet
    if (args.n_sub == 4)
      return damped ? go(rod_block_fp64_kernel<kCap, kThreads, true, kServe, kGather, kPair, 1>)
                    : go(rod_block_fp64_kernel<kCap, kThreads, false, kServe, kGather, kPair, 1>);
    if (args.n_sub == 2)
      return damped ? go(rod_block_fp64_kernel<kCap, kThreads, true, kServe, kGather, kPair, 2>)
                    : go(rod_block_fp64_kernel<kCap, kThreads, false, kServe, kGather, kPair, 2>);
  }
  return damped ? go(rod_block_fp64_kernel<kCap, kThreads, true, kServe, kGather, kPair>)
                : go(rod_block_fp64_kernel<kCap, kThreads, false, kServe, kGather, kPair>);
}

}  // namespace

// Configurations offered to the autotuner.  The capacity bounds the longest
// rod a configuration can hold (n + 1 slots).
namespace {
// {slots per CTA, threads per CTA}
constexpr int kBlockConfigs[][2] = {{520, 512}, {520, 256}, {264, 256}, {320, 320}};
constexpr int kNumConfigs = 4;
}  // namespace

int block_config_count() { return kNumConfigs; }

int block_config_capacity(int config) {
  return (config >= 0 && config < kNumConfigs) ? kBlockConfigs[config][0] : 0;
}

int block_config_threads(int config) {
  return (config >= 0 && config < kNumConfigs) ? kBlockConfigs[config][1] : 0;
}

// Serving launches (see launch_rod_block_mixed_serve): 520-slot CTAs in a
// cluster launch (n_ctas even) in which serve entries 2i and 2i + 1 may hold
// the two halves of one rod.
cudaError_t launch_rod_block_fp64_serve(const StepArgs& args, const ServeCta* serve, int n_ctas, int n_steps,
                                        bool damped, cudaStream_t stream) {
  if (n_ctas <= 0 || n_steps <= 0) return cudaSuccess;
  return launch_block_cfg<520, 512, true, false, true>(args, nullptr, n_ctas, n_steps, damped, stream, serve);
}

// Rod pairs on gathered CTAs: CTAs 2i and 2i + 1 own the two halves of one
// rod (slots gmap[cta_start[c] .. cta_start[c + 1])); config 0: 512 threads,
// 1: 256 threads per CTA.
cudaError_t launch_rod_block_fp64_pairs(const StepArgs& args, const int64_t* cta_start, const int32_t* gmap,
                                        int n_ctas, int n_steps, int config, bool damped, cudaStream_t stream) {
  if (n_ctas <= 0 || n_steps <= 0) return cudaSuccess;
  switch (config) {
    case 0: return launch_block_cfg<520, 512, false, true, true>(args, cta_start, n_ctas, n_steps, damped, stream, nullptr, gmap);
    case 1: return launch_block_cfg<520, 256, false, true, true>(args, cta_start, n_ctas, n_steps, damped, stream, nullptr, gmap);
    default: return cudaErrorInvalidValue;
  }
}

// Gathered CTAs: CTA c owns the slots gmap[cta_start[c] .. cta_start[c + 1]),
// whole rods in slot order (the per-size-bucket plans).
cudaError_t launch_rod_block_fp64_gather(const StepArgs& args, const int64_t* cta_start, const int32_t* gmap,
                                         int n_ctas, int n_steps, int config, bool damped, cudaStream_t stream) {
  if (n_ctas <= 0 || n_steps <= 0) return cudaSuccess;
  switch (config) {
    case 0: return launch_block_cfg<520, 512, false, true>(args, cta_start, n_ctas, n_steps, damped, stream, nullptr, gmap);
    case 1: return launch_block_cfg<520, 256, false, true>(args, cta_start, n_ctas, n_steps, damped, stream, nullptr, gmap);
    case 2: return launch_block_cfg<264, 256, false, true>(args, cta_start, n_ctas, n_steps, damped, stream, nullptr, gmap);
    case 3: return launch_block_cfg<320, 320, false, true>(args, cta_start, n_ctas, n_steps, damped, stream, nullptr, gmap);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace eb

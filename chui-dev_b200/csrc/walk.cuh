// Arguments and device helpers shared by the short-range walk kernels
// (walk.cu: per-node, adaptive and counting walks; walk_strict.cu: the strict
// policy's production walk).
#pragma once

#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>

#include "context.cuh"

namespace chui {

struct WalkArgs {
  int64_t nt;       // targets
  int64_t v0, v1;   // visit positions walked: [v0, v1) of the nt
  float* chunk_cost;  // SM cycles spent per 32 visit positions (index position / 32), nullable
  int out_compact;    // outputs at visit position - v0 (a visit-range solve) instead of the slot
  int64_t n;        // sources
  const uint32_t* order;   // visit position -> active slot
  const uint32_t* active;  // slot -> source row (nullable: slot == row)
  const double* tx;        // explicit target positions (nullable)
  const double* ty;
  const double* tz;
  const double* sx;        // caller source positions
  const double* sy;
  const double* sz;
  const uint32_t* pos_of_row;
  const double4* geom;
  const double4* com;
  const double* quad;
  const uint32_t* child;
  const uint4* range;
  const float4* src_f4;
  const double4* src_d4;
  const float4* node_f4;
  const float4* node_mq;   // per node 2 x float4: {mass, Mxx, Mxy, Mxz}, {Myy, Myz, Mzz, trace}
  const double4* src_u4;   // tree-ordered unwrapped positions + mass
  const double* prev;      // per slot |a_previous| (nullable: no history)
  // per-particle softening (all nullable: uniform wp.eps): tree-order and
  // row-order source epsilons, per-slot target epsilons, per-node {min, max}
  const double* src_eps;
  const double* row_eps;
  const double* tgt_eps;
  const double2* node_soft;
  // group walk
  const uint32_t* leaf_of_pos;  // tree position -> leaf node
  uint32_t* grp_start;          // visit position -> visit position of its group's first target
  double4* grp_rec;             // at a group start v: [2v] {centre, a_min}, [2v+1] {half, targets or 0 if ineligible}
  uint32_t* grp_list;           // eligible group starts
  unsigned char* grp_done;      // per slot: evaluated by the group walk
  const double2* gauss;         // Gaussian Hermite table {value, slope} (4097 knots)
  double* out_x;   // per slot, short-range part
  double* out_y;
  double* out_z;
  double* out_near;
  unsigned long long* counters;
  uint32_t* work;
  uint32_t* status;
  PolyH poly;
  PolyH dpoly;     // H'(t)
  PolyH ddpoly;    // H''(t)
  float inv_16rs5_f;
  float inv_32rs7_f;
  int mult_f32;    // accepted multipoles in FP32 (the split constants are normal floats)
  int mpoly12;     // H' and H'' fits have at most 12 terms
  // Packed (f32x2) operands of the pair loop, each value in both halves, so
  // that two queued sources share every FP32 instruction: the coefficients
  // of -H(t)/(8 r_s^3) (minus the long-range kernel K_long), the scale and
  // offset taking r^2 + eps^2 to the polynomial variable s = r^2 sc - 1, and
  // eps^2. cut2e = r_cut^2 + eps^2 is the cutoff test on r^2 + eps^2.
  float2 pk2[kPolyMaxTerms];
  float2 sc2, soff2, eps2_2;
  float2 mone2;  // {-1, -1}: s from r^2 itself (per-pair softening)
  float cut2e;
  // diagnostics 2 (or a requested nearest-pair lane): the counting instances
  // walk with subtree blocks (the production traversal) -- blocks -- and the
  // FP64 production walk counts and records nearest pairs -- instrument
  int blocks;
  int instrument;
  // groups of nearby targets ({first visit position, targets}) and their number
  const uint2* groups;
  const uint32_t* group_count;
  WalkParams wp;
};

// Bounds of the sources in the tree frame.
struct SourceFrame {
  double lo[3], hi[3];
};

// The strict production walk's own arguments (walk_strict.cu).
struct StrictArgs {
  int targets_per_group;        // at most; a power of two
  int stack_cap, batch_cap;     // stack entries, and those open to taking several nodes at once
  double block_half;            // largest half-size of a subtree block
  float cut_f;                  // r_cut
  float accept_half;            // nodes from this half-size on are never accepted as multipoles
  float sc_r2;                  // r^2 -> polynomial variable
  double h64[kPoly64Terms];     // FP64: H(t)/(8 r_s^3) in s = 1 - r^2 h64_scale
  double h64_scale;
  int canonical;                // FP64: every coordinate lies in [0, L)
  double anchor[3];             // ... and the tree frame moves those below the anchor up by L
  SourceFrame frame;
};

namespace {

__device__ __forceinline__ float polyH(const PolyH& p, float t) {
  const float s = fmaf(t, p.scale, -1.0f);
  float h = p.c[p.terms - 1];
  for (int k = p.terms - 2; k >= 0; --k) h = fmaf(h, s, p.c[k]);
  return h;
}

// monopolePlusQuadrupoleAccelPeriodicReference (tree_pm_coupling.cpp:743-827), FP64.
__device__ __forceinline__ void multipoleForce(const WalkArgs& a, uint32_t node, double dx, double dy, double dz,
                               double eps_t, double& ax, double& ay, double& az) {
  const WalkParams& w = a.wp;
  const double rs = w.rs;
  const double4 cm = a.com[node];
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double safe_r2 = fmax(r2, 1.0e-30);
  const double r = sqrt(safe_r2);
  // max(node softening maximum, target) (tree_pm_coupling.cpp:749-757)
  const double pe = fmax(a.node_soft ? a.node_soft[node].y : w.eps, eps_t);
  const double denom = fmax(r2 + pe * pe, 1.0e-30);
  const double soft = 1.0 / (denom * sqrt(denom));
  const double split = shortRangeFactor(r, rs);
  const double newton = 1.0 / (safe_r2 * r);
  const double radial = soft + (split - 1.0) * newton;
  const double G = w.G;
  double fx = G * cm.w * radial * dx;
  double fy = G * cm.w * radial * dy;
  double fz = G * cm.w * radial * dz;
  if (w.quadrupole) {
    const double* q = a.quad + 8 * static_cast<size_t>(node);
    const double tr = q[6];
    const double mxx = (q[0] + tr) / 3.0, mxy = q[1] / 3.0, mxz = q[2] / 3.0;
    const double myy = (q[3] + tr) / 3.0, myz = q[4] / 3.0, mzz = (q[5] + tr) / 3.0;
    const double mdx = mxx * dx + mxy * dy + mxz * dz;
    const double mdy = mxy * dx + myy * dy + myz * dz;
    const double mdz = mxz * dx + myz * dy + mzz * dz;
    const double dmd = dx * mdx + dy * mdy + dz * mdz;
    const double k = 0.564189583547756286948079451560772586;
    const double rs2 = rs * rs;
    const double ex = exp(-r2 / (4.0 * rs2));
    const double sf = -0.5 * k * r2 * ex / (rs * rs2);
    const double ss = k * ex * (-r / (rs * rs2) + 0.25 * r * r2 / (rs * rs2 * rs2));
    const double s1 = -3.0 * r / (denom * denom * sqrt(denom));
    const double s2 = -3.0 / (denom * denom * sqrt(denom)) + 15.0 * r2 / (denom * denom * denom * sqrt(denom));
    const double n1 = -3.0 / (safe_r2 * safe_r2);
    const double n2 = 12.0 / (safe_r2 * safe_r2 * r);
    const double rf = s1 + sf * newton + (split - 1.0) * n1;
    const double rsec = s2 + ss * newton + 2.0 * sf * n1 + (split - 1.0) * n2;
    const double f1 = rf / r;
    const double cr = rsec / r2 - rf / (r2 * r);
    fx += G * (mdx * f1 + 0.5 * tr * dx * f1 + 0.5 * dx * dmd * cr);
    fy += G * (mdy * f1 + 0.5 * tr * dy * f1 + 0.5 * dy * dmd * cr);
    fz += G * (mdz * f1 + 0.5 * tr * dz * f1 + 0.5 * dz * dmd * cr);
  }
  ax += fx;
  ay += fy;
  az += fz;
}

// |d|^2 summed as the reference does, ((dx dx + dy dy) + dz dz) with every
// operation rounded on its own (no FMA contraction), so acceptance decisions
// see the reference's exact value.
__device__ __forceinline__ double norm2rn(double dx, double dy, double dz) {
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Per-target acceleration history: present and finite
// (tree_pm_coupling.cpp:4467-4472); magnitude 0 when absent.
struct History {
  bool avail;
  double mag;
};

__device__ __forceinline__ History loadHistory(const double* prev, uint32_t slot, bool valid) {
  History h{false, 0.0};
  if (prev && valid) {
    const double v = prev[slot];
    h.avail = isfinite(v);
    h.mag = h.avail ? v : 0.0;
  }
  return h;
}

// residualAccuracyProxy (internal/tree_pm_acceptance.hpp:20-51) with uniform
// softening (node softening max = the target's). Scalars by value: a
// reference into the kernel's parameter block would force a local copy of it.
__device__ __noinline__ double residualProxy(double G, double eps, double rs, double half, double com_offset,
                                            double mass, double r2) {
  if (!(r2 > 0.0) || !isfinite(r2)) return INFINITY;
  const double r = sqrt(r2);
  const double d = r2 + eps * eps;
  const double inv_d5 = 1.0 / (d * d * sqrt(d));
  const double inv_r3 = 1.0 / (r2 * r);
  const double inv_r4 = 1.0 / (r2 * r2);
  const double long_factor = longRangeFactor(r, rs);
  const double q = r / (2.0 * rs);
  const double exponential = exp(-q * q);
  const double k_inv_sqrt_pi = 0.564189583547756286948079451560772586;
  const double scale3 = rs * rs * rs;
  const double s_first = -0.5 * k_inv_sqrt_pi * r2 * exponential / scale3;
  const double s_second = k_inv_sqrt_pi * exponential * (-r / scale3 + 0.25 * r * r2 / (scale3 * rs * rs));
  const double first = -3.0 * r * inv_d5 + s_first * inv_r3 - 3.0 * (-long_factor) * inv_r4;
  const double second = -3.0 * inv_d5 + 15.0 * r2 * inv_d5 / d + s_second * inv_r3 - 6.0 * s_first * inv_r4 +
                        12.0 * (-long_factor) * inv_r4 / r;
  const double width = 2.0 * half;
  const double rho = sqrt(3.0) * half + com_offset;
  const double proxy =
      G * mass * fmax(width * width * inv_r4, 0.5 * rho * rho * (3.0 * fabs(first) + fabs(r * second - first)));
  return isfinite(proxy) && proxy >= 0.0 ? proxy : INFINITY;
}

// A target's softening: its own lane, else its source row's epsilon, else
// the configured one (targetSofteningEpsilonUnchecked, tree_softening.hpp:90-110).
__device__ __forceinline__ double targetEps(const WalkArgs& a, uint32_t slot, uint32_t row, bool valid) {
  if (!valid) return a.wp.eps;
  if (a.tgt_eps) return a.tgt_eps[slot];
  if (a.row_eps && row < a.n) return a.row_eps[row];
  return a.wp.eps;
}

// A source's softening by tree position.
__device__ __forceinline__ double sourceEps(const WalkArgs& a, uint32_t pos) {
  return a.src_eps ? a.src_eps[pos] : a.wp.eps;
}

// max(node softening maximum, target): the multipole and proxy softening.
__device__ __forceinline__ double nodeEps(const WalkArgs& a, uint32_t node, double eps_t) {
  return fmax(a.node_soft ? a.node_soft[node].y : a.wp.eps, eps_t);
}

// passesSofteningEnvelopeGuard (internal/tree_interaction_common.hpp:77-89)
// at r = sqrt(max(r^2, 1e-30)): nodes whose sources' softenings differ are
// accepted only beyond 2h + 2 max(node maximum, target).
__device__ __forceinline__ bool softeningGuard(const WalkArgs& a, uint32_t node, double half, double r2,
                                               double eps_t) {
  if (!a.node_soft) return true;
  const double2 ns = a.node_soft[node];
  if (ns.y - ns.x <= 1.0e-12) return true;
  return sqrt(fmax(r2, 1.0e-30)) > 2.0 * half + 2.0 * fmax(ns.y, eps_t);
}

// Acceptance of an internal node (acceptTreePmNode, internal/tree_pm_acceptance.hpp:53-139,
// with acceptNodeByMac and acceptNodeByComDistanceMac of
// internal/tree_interaction_common.hpp:36-75). Softening is uniform, so the
// softening envelope guard passes.
template <bool kAdaptive>
__device__ __forceinline__ bool acceptNode(const WalkParams& w, double half, double com_offset, double mass,
                                           bool inside, bool within, double r2, const History& hist,
                                           bool soft_ok = true, double eps_node = -1.0) {
  const double r = sqrt(fmax(r2, 1.0e-30));
  const double width = 2.0 * half;
  if (eps_node < 0.0) eps_node = w.eps;
  if (!soft_ok) return false;  // passesSofteningEnvelopeGuard
  if constexpr (!kAdaptive) {
    const bool envelope_ok = w.quadrupole && (width / r) < 0.08;
    bool mac_ok;
    if (inside) {
      mac_ok = false;
    } else if (w.criterion == 0) {
      mac_ok = (width / sqrt(r2 + 1.0e-30)) < w.theta;
    } else if (w.criterion == 1 || !hist.avail) {
      mac_ok = ((width + com_offset) / sqrt(r2 + 1.0e-30)) < w.theta;
    } else {
      const double scale = fmax(fabs(hist.mag), w.floor_);
      mac_ok = w.G * mass * width * width <= w.rel_tol * scale * r2 * r2;
    }
    return mac_ok && envelope_ok && within && !inside && isfinite(r2);
  }
  const bool envelope_ok = (width / r) < w.angle;
  if (!envelope_ok || inside || !within || !isfinite(r2)) return false;
  if (hist.avail && hist.mag > w.floor_) {
    const double allowance = w.rel_tol * hist.mag;
    const double inv_r4 = 1.0 / (r2 * r2);
    const double lower = w.G * mass * (width * width * inv_r4);
    if (isfinite(allowance) && isfinite(lower) && lower > allowance) return false;
    if (w.estimator == 1) return isfinite(allowance) && isfinite(lower);
    const double est = residualProxy(w.G, eps_node, w.rs, half, com_offset, mass, r2);
    return isfinite(est) && isfinite(allowance) && est <= allowance;
  }
  return ((width + com_offset) / sqrt(r2 + 1.0e-30)) < w.theta;
}

// ---- Gaussian pair lookup and the group walk (FP64) ------------------------

constexpr int kGaussCells = 4096;                  // tree_pm_split_kernel.hpp:136-138
constexpr double kGaussStep = 64.0 / kGaussCells;

// Cubic Hermite evaluation of H(t) from the reference's table
// (TreePmGaussianCoefficientTable::dimensionlessCoefficient, :150-164).
__device__ __forceinline__ double gaussHermite(const double2* g, double t) {
  const double cell = t / kGaussStep;
  const int i = static_cast<int>(cell);
  const double u = cell - static_cast<double>(i);
  const double u2 = u * u;
  const double u3 = u2 * u;
  const double2 k0 = g[i], k1 = g[i + 1];
  return (2 * u3 - 3 * u2 + 1) * k0.x + (u3 - 2 * u2 + u) * k0.y + (-2 * u3 + 3 * u2) * k1.x + (u3 - u2) * k1.y;
}

// Per-target direct pair with the Gaussian lookup (tree_pm_coupling.cpp:4221-4226).
__device__ __forceinline__ double gaussResidualInvR3(const WalkArgs& a, double r2, double eps) {
  const double rs = a.wp.rs;
  const double inv_2a2 = (0.25 / rs) / rs, inv_8a3 = ((0.125 / rs) / rs) / rs;
  const double t = r2 * inv_2a2;
  double long_inv_r3;
  if (t < 64.0) {
    const double coeff = t < 0.015625 ? coefficientSeries(t) : gaussHermite(a.gauss, t);
    long_inv_r3 = coeff * inv_8a3;
  } else {
    long_inv_r3 = longRangeInvR3(sqrt(r2), rs);
  }
  return softenedInvR3(r2, eps) - long_inv_r3;
}

// The fitted polynomial at t = r^2 / (4 r_s^2), straight from r^2: s =
// r^2 * sc - 1 with sc = scale / (4 r_s^2), then Horner (kTerms - 1 FMAs).
// The walk is issue-bound, so the fewest instructions win over a shorter
// dependency chain (the unrolled queue loop supplies the parallelism).
template <int kTerms>
__device__ __forceinline__ float hornerR2(const PolyH& p, float r2, float sc) {
  const float s = fmaf(r2, sc, -1.0f);
  float h = p.c[kTerms - 1];
#pragma unroll
  for (int k = kTerms - 2; k >= 0; --k) h = fmaf(h, s, p.c[k]);
  return h;
}

// The same Horner chain for two sources at once (packed FP32: one f32x2 FMA
// per term serves both halves); c2 holds each coefficient in both halves,
// s = r2 * sc2 + off2.
template <int kTerms>
__device__ __forceinline__ float2 hornerR2x2(const float2* c2, float2 r2, float2 sc2, float2 off2) {
  const float2 s = __ffma2_rn(r2, sc2, off2);
  float2 h = c2[kTerms - 1];
#pragma unroll
  for (int k = kTerms - 2; k >= 0; --k) h = __ffma2_rn(h, s, c2[k]);
  return h;
}

// monopolePlusQuadrupoleAccelPeriodicReference (tree_pm_coupling.cpp:743-827)
// in FP32, without the G factor, added to (fx, fy, fz). With t = r^2/(4 r_s^2)
// and H the fitted long-range kernel: K = (r^2+eps^2)^-3/2 - H(t)/(8 r_s^3),
// K'/r = -3 (r^2+eps^2)^-5/2 - H'(t)/(16 r_s^5) and
// (K'' - K'/r)/r^2 = 15 (r^2+eps^2)^-7/2 - H''(t)/(32 r_s^7); the force is
// M K d + f1 (Md + tr d / 2) + cr (d.Md) d / 2 with f1 = K'/r, cr the last.
template <bool kEpsZero, int kTerms>
__device__ __forceinline__ void multipoleF32(const WalkArgs& a, uint32_t node, float dx, float dy, float dz, float sc,
                                             float& fx, float& fy, float& fz, float eps2) {
  const float4 q0 = a.node_mq[2 * static_cast<size_t>(node)];
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  const float den = kEpsZero ? r2 : r2 + eps2;
  const float rinv = rsqrtf(den);
  const float rinv2 = rinv * rinv;
  const float rinv3 = rinv2 * rinv;
  const float k = fmaf(-hornerR2<kTerms>(a.poly, r2, sc), a.wp.inv_8rs3_f, rinv3);
  float s = q0.x * k;
  if (a.wp.quadrupole) {
    const float4 q1 = a.node_mq[2 * static_cast<size_t>(node) + 1];
    const float rinv5 = rinv3 * rinv2;
    // H' and H'' have their own fitted lengths (warp-uniform choice)
    const float h1 = a.mpoly12 ? hornerR2<12>(a.dpoly, r2, sc) : hornerR2<kPolyMaxTerms>(a.dpoly, r2, sc);
    const float h2 = a.mpoly12 ? hornerR2<12>(a.ddpoly, r2, sc) : hornerR2<kPolyMaxTerms>(a.ddpoly, r2, sc);
    const float f1 = fmaf(-h1, a.inv_16rs5_f, -3.0f * rinv5);
    const float cr = fmaf(-h2, a.inv_32rs7_f, 15.0f * rinv5 * rinv2);
    const float mdx = fmaf(q0.y, dx, fmaf(q0.z, dy, q0.w * dz));
    const float mdy = fmaf(q0.z, dx, fmaf(q1.x, dy, q1.y * dz));
    const float mdz = fmaf(q0.w, dx, fmaf(q1.y, dy, q1.z * dz));
    const float dmd = fmaf(dx, mdx, fmaf(dy, mdy, dz * mdz));
    s = fmaf(0.5f, fmaf(q1.w, f1, dmd * cr), s);
    fx = fmaf(mdx, f1, fmaf(s, dx, fx));
    fy = fmaf(mdy, f1, fmaf(s, dy, fy));
    fz = fmaf(mdz, f1, fmaf(s, dz, fz));
  } else {
    fx = fmaf(s, dx, fx);
    fy = fmaf(s, dy, fy);
    fz = fmaf(s, dz, fz);
  }
}

// Exact (FP64, reference formulas) decision for one lane at one node: prune,
// and for internal nodes accept/open, plus the COM offset for a multipole.
struct ExactDecision {
  bool prune, accept;
  double dx, dy, dz;
};

template <bool kAdaptive>
__device__ __forceinline__ ExactDecision exactNodeDecision(const WalkArgs& a, uint32_t node, double px, double py,
                                                        double pz, bool skip_self, const History& hist,
                                                        double eps_t) {
  const WalkParams& w = a.wp;
  ExactDecision d{};
  const double4 g = a.geom[node];
  const uint4 rg4 = a.range[node];
  const Metric mx = makeMetric(w.node_lo[0], w.node_hi[0], px, w.box[0]);
  const Metric my = makeMetric(w.node_lo[1], w.node_hi[1], py, w.box[1]);
  const Metric mz = makeMetric(w.node_lo[2], w.node_hi[2], pz, w.box[2]);
  const double h = g.w;
  const double ndx = applyMetric(mx, g.x - px), ndy = applyMetric(my, g.y - py), ndz = applyMetric(mz, g.z - pz);
  const double ax = fabs(ndx), ay = fabs(ndy), az = fabs(ndz);
  const double ex = fmax(0.0, ax - h), ey = fmax(0.0, ay - h), ez = fmax(0.0, az - h);
  d.prune = !withinCutoff(ex * ex + ey * ey + ez * ez, w.cutoff, w.cutoff2);
  d.accept = false;
  if (d.prune || rg4.z == 0) return d;
  const double4 cm = a.com[node];
  const double off = a.quad[8 * static_cast<size_t>(node) + 7];
  const bool inside = (skip_self || kAdaptive) && ax <= h && ay <= h && az <= h;
  const double qx = ax + h, qy = ay + h, qz = az + h;
  const bool within = (kAdaptive && w.com_cutoff) || withinCutoff(qx * qx + qy * qy + qz * qz, w.cutoff, w.cutoff2);
  d.dx = applyMetric(mx, cm.x - px);
  d.dy = applyMetric(my, cm.y - py);
  d.dz = applyMetric(mz, cm.z - pz);
  const double r2 = norm2rn(d.dx, d.dy, d.dz);
  d.accept = acceptNode<kAdaptive>(w, h, off, cm.w, inside, within, r2, hist, softeningGuard(a, node, h, r2, eps_t),
                                   nodeEps(a, node, eps_t));
  if (kAdaptive && d.accept && w.com_cutoff && r2 > w.cutoff2) {  // accepted beyond r_cut: pruned
    d.accept = false;
    d.prune = true;
  }
  return d;
}

// Nearest image of a frame offset on an axis of length L (inv_l = 1/L); L = 0
// (isolated/open boundaries) has no images. The reciprocal replaces a division
// per axis and node: the shared frame is only used where offsets stay well
// inside half a box, so the rounding of d/L cannot pick another image.
__device__ __forceinline__ double frameImage(double d, double L, double inv_l) {
  return L > 0.0 ? d - L * rint(d * inv_l) : d;
}

// Comparison a < b decided in FP32 with a guard band (relative, plus an
// absolute bound `err` on the inputs' own error): returns +1 (certainly true),
// -1 (certainly false) or 0 (too close to call in FP32).
__device__ __forceinline__ int certainLess(float a, float b, float err = 0.f) {
  const float band = fmaf(2.0e-5f, fabsf(a) + fabsf(b), err) + 1.0e-30f;
  if (a < b - band) return 1;
  if (a > b + band) return -1;
  return 0;
}

// order-preserving signed integer image of a float
__device__ __forceinline__ int floatOrder(float f) {
  const int i = __float_as_int(f);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float fromFloatOrder(int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }

// The group's centre to FP32: offsets of nearby FP64 positions from it are
// exact, so a pair's separation is rounded once.
__device__ __forceinline__ double coarse(double v) {
  const float f = static_cast<float>(v);
  return isfinite(f) ? static_cast<double>(f) : v;
}

constexpr int kBatchStack = 224;         // stack entries beyond the depth-first bound, for nodes taken together
constexpr float kFar = 1.0e15f;          // padding entry of a source queue, outside every cutoff
constexpr uint32_t kWideRun = 1u << 31;  // group record: the 32 visit positions around it spread wide

// The box of a warp's targets (FP64 positions, one per lane, near each other
// in one frame): centre and half extents, rounding included.
struct GroupFrame {
  double cx, cy, cz;
  float hx, hy, hz;
};

__device__ __forceinline__ void groupAxis(double p, float off, double& c, float& h) {
  const float lo = fromFloatOrder(__reduce_min_sync(0xffffffffu, floatOrder(off)));
  const float hi = fromFloatOrder(__reduce_max_sync(0xffffffffu, floatOrder(off)));
  c = coarse(p + static_cast<double>(0.5f * (lo + hi)));
  const float mid = static_cast<float>(c - p);
  h = fmaxf(hi - mid, mid - lo) + 3.0e-7f * (hi - lo + fabsf(mid));
}

__device__ __forceinline__ GroupFrame groupFrame(double px, double py, double pz, bool valid) {
  GroupFrame f;
  const double rx = __shfl_sync(0xffffffffu, px, 0), ry = __shfl_sync(0xffffffffu, py, 0),
               rz = __shfl_sync(0xffffffffu, pz, 0);
  groupAxis(rx, valid ? static_cast<float>(px - rx) : 0.f, f.cx, f.hx);
  groupAxis(ry, valid ? static_cast<float>(py - ry) : 0.f, f.cy, f.hy);
  groupAxis(rz, valid ? static_cast<float>(pz - rz) : 0.f, f.cz, f.hz);
  return f;
}

// One node per lane against the box of the targets: the nearest image of its
// centre (whole box lengths k, offset nd), the squared distance from the box
// to the cube's nearest point (low side of rounding) and the squared reach of
// all targets to its farthest corner (high side).
struct NodeReach {
  uint4 rg;
  double half;
  double kx, ky, kz, ndx, ndy, ndz;
  float ax, ay, az, hf, gap2, far2;
};

__device__ __forceinline__ NodeReach nodeReach(const double4* __restrict__ geom, const uint4* __restrict__ range,
                                               uint32_t node, bool have, const GroupFrame& f, const WalkParams& w) {
  NodeReach r;
  double4 g = make_double4(0.0, 0.0, 0.0, 0.0);
  r.rg = make_uint4(0u, 0u, 0u, 0u);
  if (have) {
    g = geom[node];
    r.rg = range[node];
  }
  r.half = g.w;
  // L = 0: no images
  r.kx = w.box[0] > 0.0 ? rint((g.x - f.cx) * w.inv_box[0]) : 0.0;
  r.ky = w.box[1] > 0.0 ? rint((g.y - f.cy) * w.inv_box[1]) : 0.0;
  r.kz = w.box[2] > 0.0 ? rint((g.z - f.cz) * w.inv_box[2]) : 0.0;
  r.ndx = (g.x - f.cx) - w.box[0] * r.kx;
  r.ndy = (g.y - f.cy) - w.box[1] * r.ky;
  r.ndz = (g.z - f.cz) - w.box[2] * r.kz;
  r.hf = __double2float_ru(g.w);
  r.ax = fabsf(static_cast<float>(r.ndx));
  r.ay = fabsf(static_cast<float>(r.ndy));
  r.az = fabsf(static_cast<float>(r.ndz));
  const float gx = fmaxf(fmaf(r.ax, 0.9999995f, -(r.hf + f.hx)), 0.f), gy = fmaxf(fmaf(r.ay, 0.9999995f, -(r.hf + f.hy)), 0.f),
              gz = fmaxf(fmaf(r.az, 0.9999995f, -(r.hf + f.hz)), 0.f);
  r.gap2 = fmaf(gx, gx, fmaf(gy, gy, gz * gz));
  const float wx = r.ax + r.hf + f.hx, wy = r.ay + r.hf + f.hy, wz = r.az + r.hf + f.hz;
  r.far2 = fmaf(wx, wx, fmaf(wy, wy, wz * wz));
  return r;
}

// One axis of the images of a node that some target may reach: its sources lie
// in the part of its cube (centre nd from the image k of the box centre c,
// half-size h) inside the bounds of all sources, and come within r_cut of the
// targets' box (half extent hb) when moved back by k, k + 1, ... k + count - 1
// box lengths. The cube of a sparse leaf can span several short sides of an
// elongated box, its centre lengths away from its sources, so the images are
// counted from the sources' interval (three at most: it is no wider than L, and
// r_cut + hb stays below 0.63 L).
__device__ __forceinline__ void nodeImages(const WalkParams& w, const SourceFrame& s, int axis, double nd, double h,
                                           double c, double hb, double& k, int& count) {
  const double L = w.box[axis];
  if (!(L > 0.0)) return;
  const double centre = nd + L * k, reach = w.cutoff + hb + 1.0e-5 * L;  // with room for rounding
  const double lo = fmax(centre - h, s.lo[axis] - c) - reach, hi = fmin(centre + h, s.hi[axis] - c) + reach;
  k = ceil(lo * w.inv_box[axis]);
  count = 1 + static_cast<int>(fmin(fmax(floor(hi * w.inv_box[axis]) - k, 0.0), 3.0));
}

// The children of the lanes' nodes that are opened (push) go on the stack, each
// with `flag` set; returns the new height, or sets overflow.
__device__ __forceinline__ int pushChildren(const uint32_t* __restrict__ child, uint32_t node, bool push,
                                            uint32_t children, uint32_t flag, uint32_t* stack, int sp, int cap,
                                            bool& overflow, uint32_t* stack_mask = nullptr, uint32_t mask = 0u) {
  const int lane = threadIdx.x & 31;
  const uint32_t n = push ? children : 0u;
  uint32_t incl = n;
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += y;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  if (sp + static_cast<int>(total) > cap) {
    overflow = true;
    return sp;
  }
  if (push) {
    uint32_t at = static_cast<uint32_t>(sp) + incl - n;
    const uint4* ch = reinterpret_cast<const uint4*>(child + 8 * static_cast<size_t>(node));
    const uint4 c0 = ch[0], c1 = ch[1];
    const uint32_t c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      if (c[o] != kInvalid) {
        stack[at] = c[o] | flag;
        if (stack_mask) stack_mask[at] = mask;
        ++at;
      }
    }
  }
  __syncwarp();
  return sp + static_cast<int>(total);
}

inline SourceFrame sourceFrame(const Context& c) {
  SourceFrame f;
  for (int a = 0; a < 3; ++a) {
    f.lo[a] = c.frame_lo[a];
    f.hi[a] = c.frame_hi[a];
  }
  return f;
}

}  // namespace

// Groups of at most `most` (a power of two, <= 32) nearby targets over the
// visit positions [a.v0, a.v1), each within `limit` per axis.
int targetGroups(Context& c, const WalkArgs& a, int most, double limit, const uint2** groups, const uint32_t** count,
                 cudaStream_t s);
// The strict policy's production walk (mixed precision, or FP64 pairs); tiny: a
// box in which a group of targets reaches two images of a leaf.
int walkStrictRun(Context& c, WalkArgs& a, bool f64, bool tiny, cudaStream_t s);

}  // namespace chui

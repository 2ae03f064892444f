// Production walk of the strict policy (diagnostics off).
//
// The answer is that of walkFastKernel (walk.cu): each target takes every source inside r_cut
// of it as a direct pair, except the subtrees the strict policy accepts as a
// multipole for that target (decided as the reference decides them), and a
// node of at most kStrictBlock sources that is not accepted itself is summed
// as pairs whatever its descendants would have been.
//
// Organisation: the visit order is cut into groups of at most 32 / S targets
// that lie close together (targetGroupsKernel); one warp walks the tree once
// for a group, S lanes sharing each target.
//  - Traversal takes up to 32 stacked nodes at a time, a node per lane, and
//    tests them against the bounding box of the group's targets: out of reach
//    of every target, enqueued whole, or replaced by its children. Only the
//    few nodes some target might accept as a multipole (width below 0.08 of
//    the distance, wholly inside r_cut) are decided per target.
//  - Enqueue forms each source's FP64 offset from the box centre, rounds it
//    once to FP32, and keeps the sources within r_cut of the box (a third of
//    the volume of the sphere around one of the targets in a near-uniform
//    region).
//  - The pair loop reads four queued sources at a time from x, y, z arrays in
//    shared memory and evaluates them two by two in packed FP32.
// Bound by the FMA pipe of the pair loop (78 % of the walk at 256^3 clustered:
// 2552 quads of sources per 32 targets at 54 ns per quad and scheduler is 122 of
// 156 ms). Before, with one warp per 32 consecutive targets whatever their spread,
// every node decided per lane and sources culled by a sphere: 193 ms at 256^3,
// 33 to 46 ms against 15.6 at 128^3, 20 against 1.8 ms for 200 k particles (a
// warp straddling a jump of the tree order walked for milliseconds).
// No lane masks travel with the sources: a target's own entry is at distance
// zero and adds nothing (targets and sources round the same tree-frame
// position the same way; EpsForm), sources beyond r_cut fail the pair's cutoff test, and
// the rare source whose node some target has accepted as a multipole is queued
// in a batch of its own that those targets' lanes sit out.
//
// Periodic images: a node is placed at its nearest image of the box centre, and
// where the reach of the group (box + r_cut + node) spans more than one image
// its sources are queued once per image that brings some of them into reach
// (nodeImages); a pair is inside r_cut < L/2 in one image at most.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>

#include "walk.cuh"

namespace chui {
namespace {

// subtree blocks: an opened node of at most kStrictBlock sources and half-size
// at most kStrictHalf r_cut has no multipoles inside
constexpr uint32_t kStrictBlock = 2048;
constexpr double kStrictHalf = 1.0;
// Inside a block, a node that straddles the reach of the group is opened down
// to this many sources (fewer sources to test against the box, more nodes to
// visit). 64 / 128 / 256 / 512 / 1024 sources: 171.5 / 165.9 / 162.9 / 161.4 /
// 160.6 ms at 256^3 clustered, 9.1 / 5.8 / 5.8 / 5.8 / 6.6 ms for a lattice of
// 2.65 M particles.
constexpr uint32_t kStrictCull = 512;
// queued sources per batch (128: 2 % slower at 256^3)
constexpr int kQueue32 = 256;
constexpr int kQueue64 = 128;
constexpr uint32_t kInBlock = 1u << 31;  // stack entry inside a subtree block (node ids stay below 2^31)

// Resident blocks per SM the FP32 registers are sized for. 4, 5 and 6 (128, 96
// and 80 registers) are equal to 1 % (160.9 / 160.9 / 161.8 ms at 256^3), 7 and
// 8 spill in the pair loop (166.4, 170.3): with four warps per scheduler the
// FMA pipe is already the limit of the pair loop, 54 ns per 4 sources and warp
// where two or more warps evaluate (the loop alone, measured with 2 to 8).
constexpr int kBlocks32 = 5;

enum SourceLanes { kUniformMass = 0, kMassLane = 1, kMassEpsLanes = 2 };

// What a target's own entry, and a source that coincides with it, need (FP32,
// one softening): nothing with kEpsFinite, where the pair's factor m K(0) is a
// finite number times d = 0; otherwise the pair loop drops pairs at distance
// zero, on r^2 itself (kEpsGuard: two more instructions per two pairs).
enum EpsForm { kEpsNone = 0, kEpsFinite = 1, kEpsGuard = 2 };

// A target's position: its source's tree-frame position, or the explicit one.
__device__ __forceinline__ void targetPosition(const WalkArgs& a, int64_t v, uint32_t slot, uint32_t row, double& x,
                                               double& y, double& z) {
  if (a.tx) {
    x = a.tx[slot];
    y = a.ty[slot];
    z = a.tz[slot];
  } else {
    const double4 u = a.src_u4[a.active ? a.pos_of_row[row] : static_cast<uint32_t>(v)];
    x = u.x;
    y = u.y;
    z = u.z;
  }
}

// Offset of a target from a point near it. Tree-frame positions are unwrapped:
// targets on opposite faces of the frame stay apart, and the offset has the
// bits of the queued source's. Explicit positions may be anywhere.
__device__ __forceinline__ double targetOffset(const WalkArgs& a, double d, int axis) {
  return a.tx ? frameImage(d, a.wp.box[axis], a.wp.inv_box[axis]) : d;
}

// FP64: c + q L in two parts {hi, lo}, so that p - c - q L of a position p at the
// caller's coordinate is (p - hi) - lo, rounded on the scale of the offset (p lies
// near hi). The tree frame's copy of a position below the anchor is p + L rounded
// to an ulp of L, which is no rounding for a close pair; formed this way for
// targets and sources alike, coincident particles are at distance zero.
__device__ __forceinline__ double2 movedOrigin(double c, double q, double length) {
  const double ql = __dmul_rn(q, length);
  const double hi = __dadd_rn(c, ql);
  const double part = __dsub_rn(hi, c);
  return make_double2(hi, __dadd_rn(__dsub_rn(c, __dsub_rn(hi, part)), __dsub_rn(ql, part)));
}

// FP64: offset from c of a position at the caller's coordinate p, at the image at
// (about) `near`.
__device__ __forceinline__ double callerOffset(double p, double near, double c, double length, double inv_length) {
  const double2 o = movedOrigin(c, length > 0.0 ? rint(((p - c) - near) * inv_length) : 0.0, length);
  return __dsub_rn(__dsub_rn(p, o.x), o.y);
}

// Cuts each run of 32 visit positions into groups: maximal runs of consecutive
// targets, at most `most` of them, whose extent stays within `limit` per axis
// (a run that straddles a jump of the tree order would walk the tree with a
// box that spans the jump). One warp per 32 positions.
// A run whose targets spread beyond a quarter of r_cut, but not beyond the reach
// of the nearest image (r_cut + spread below half a box), is marked kWideRun:
// its groups keep the run's first target as the origin of their FP32 offsets.
// That origin is coarser than the box centre (offsets of up to half a box are
// rounded to 24 bits; 3 % active targets of a clustered box are 1.6e-5 off the
// FP64 sums, a full solve 1.3e-6). It is kept because a caller's results under
// sparse active sets were rounded in that frame before groups existed, and with
// the box centre they would move by as much as they are off.
__global__ void __launch_bounds__(256) targetGroupsKernel(WalkArgs a, int most, double limit, uint2* groups,
                                                          uint32_t* count) {
  const int lane = threadIdx.x & 31;
  const WalkParams& w = a.wp;
  const float lim = static_cast<float>(limit);
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t b = blockIdx.x * static_cast<int64_t>(blockDim.x >> 5) + (threadIdx.x >> 5); a.v0 + 32 * b < a.v1;
       b += warps) {
    const int64_t v = a.v0 + 32 * b + lane;
    const bool valid = v < a.v1;
    double px = 0.0, py = 0.0, pz = 0.0;
    if (valid) {
      const uint32_t slot = a.order[v];
      targetPosition(a, v, slot, a.active ? a.active[slot] : slot, px, py, pz);
    }
    unsigned todo = __ballot_sync(0xffffffffu, valid);
    uint32_t wide = 0u;
    {
      const double sx = frameImage(px - __shfl_sync(0xffffffffu, px, 0), w.box[0], w.inv_box[0]);
      const double sy = frameImage(py - __shfl_sync(0xffffffffu, py, 0), w.box[1], w.inv_box[1]);
      const double sz = frameImage(pz - __shfl_sync(0xffffffffu, pz, 0), w.box[2], w.inv_box[2]);
      const double spread = fmax(fabs(sx), fmax(fabs(sy), fabs(sz)));
      const double nearest = w.box[0] > 0.0 ? 0.5 * fmin(w.box[0], fmin(w.box[1], w.box[2])) : INFINITY;
      const bool far = __any_sync(0xffffffffu, valid && spread > 0.25 * w.cutoff);
      const bool ambiguous = __any_sync(0xffffffffu, valid && w.cutoff + spread >= nearest);
      if (far && !ambiguous) wide = kWideRun;
    }
    int size = 0;  // group size, on the group's first lane
    while (todo) {
      const int lead = __ffs(todo) - 1;
      const float ox = static_cast<float>(targetOffset(a, px - __shfl_sync(0xffffffffu, px, lead), 0));
      const float oy = static_cast<float>(targetOffset(a, py - __shfl_sync(0xffffffffu, py, lead), 1));
      const float oz = static_cast<float>(targetOffset(a, pz - __shfl_sync(0xffffffffu, pz, lead), 2));
      // running extents from the lead lane on
      const bool in = valid && lane >= lead;
      float lx = in ? ox : INFINITY, hx = in ? ox : -INFINITY, ly = in ? oy : INFINITY, hy = in ? oy : -INFINITY;
      float lz = in ? oz : INFINITY, hz = in ? oz : -INFINITY;
      for (int off = 1; off < 32; off <<= 1) {
        const float a0 = __shfl_up_sync(0xffffffffu, lx, off), a1 = __shfl_up_sync(0xffffffffu, hx, off);
        const float b0 = __shfl_up_sync(0xffffffffu, ly, off), b1 = __shfl_up_sync(0xffffffffu, hy, off);
        const float c0 = __shfl_up_sync(0xffffffffu, lz, off), c1 = __shfl_up_sync(0xffffffffu, hz, off);
        if (lane >= off) {
          lx = fminf(lx, a0);
          hx = fmaxf(hx, a1);
          ly = fminf(ly, b0);
          hy = fmaxf(hy, b1);
          lz = fminf(lz, c0);
          hz = fmaxf(hz, c1);
        }
      }
      const bool fits = in && lane < lead + most && hx - lx <= lim && hy - ly <= lim && hz - lz <= lim;
      // the run ends before the first lane from the lead on that does not fit
      const unsigned stop = ~__ballot_sync(0xffffffffu, fits) & (0xffffffffu << lead);
      const int end = max(stop ? __ffs(stop) - 1 : 32, lead + 1);
      if (lane == lead) size = end - lead;
      todo &= end < 32 ? (0xffffffffu << end) : 0u;
    }
    const unsigned leads = __ballot_sync(0xffffffffu, size > 0);
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(count, static_cast<uint32_t>(__popc(leads)));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (size > 0)
      groups[base + __popc(leads & ((1u << lane) - 1u))] =
          make_uint2(static_cast<uint32_t>(v), static_cast<uint32_t>(size) | wide);
  }
}

// Shared memory of one warp.
template <class Real, int kLanes, bool kIndex>
struct WarpShared {
  static constexpr int kQ = sizeof(Real) == 4 ? kQueue32 : kQueue64;
  static constexpr size_t kArrays = 3 + (kLanes >= kMassLane ? 1 : 0) + (kLanes >= kMassEpsLanes ? 1 : 0);
  __host__ __device__ static constexpr size_t queueBytes() { return kArrays * kQ * sizeof(Real) + (kIndex ? kQ * sizeof(uint32_t) : 0); }
  __host__ __device__ static constexpr size_t accBytes() { return 3 * 32 * sizeof(double); }
  // FP64: the sources' origin per axis, for positions the tree frame keeps and moves
  __host__ __device__ static constexpr size_t originBytes() { return sizeof(Real) == 8 ? 6 * sizeof(double2) : 0; }
  __host__ __device__ static constexpr size_t bytes(int stack_cap) {
    return queueBytes() + accBytes() + originBytes() + static_cast<size_t>(stack_cap) * 8;
  }
};

// kTerms: terms of the long-range coefficient's polynomial; FP64 with 0: the
// reference's erf/exp form (or its Gaussian table).
template <class Real, int kEps, int kTerms, int kLanes, bool kIndex>
__global__ void __launch_bounds__(kWalkWarpsPerBlock * 32, sizeof(Real) == 4 ? kBlocks32 : 4)
    walkStrictKernel(WalkArgs a, StrictArgs sa) {
  constexpr bool kF64 = sizeof(Real) == 8;
  constexpr bool kEpsZero = kEps == kEpsNone;
  constexpr bool kPairEps = kLanes == kMassEpsLanes;      // FP32: softening per pair
  constexpr bool kFolded = !kPairEps && kEps == kEpsFinite;  // FP32: r^2 + eps^2 in one chain
  using Shared = WarpShared<Real, kLanes, kIndex>;
  constexpr int kQ = Shared::kQ;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  unsigned char* mine = smem + (threadIdx.x >> 5) * Shared::bytes(sa.stack_cap);
  Real* qx = reinterpret_cast<Real*>(mine);
  Real* qy = qx + kQ;
  Real* qz = qy + kQ;
  Real* qm = qz + kQ;  // kLanes >= kMassLane
  Real* qe = qm + kQ;  // kLanes >= kMassEpsLanes
  uint32_t* qi = reinterpret_cast<uint32_t*>(mine + Shared::kArrays * kQ * sizeof(Real));
  double* acc = reinterpret_cast<double*>(mine + Shared::queueBytes());
  double2* origin = reinterpret_cast<double2*>(mine + Shared::queueBytes() + Shared::accBytes());  // FP64
  uint32_t* stack = reinterpret_cast<uint32_t*>(mine + Shared::queueBytes() + Shared::accBytes() + Shared::originBytes());
  uint32_t* stack_mask = stack + sa.stack_cap;

  const WalkParams& w = a.wp;
  const int per = sa.targets_per_group;  // 32 / S
  const int share = 32 / per;            // S
  const int t = lane & (per - 1);        // this lane's target within the group
  const int sub = lane / per;            // its share of the sources
  const float cut2 = w.cut2_f;
  const float cut_hi2 = cut2 * 1.00002f, cut_lo2 = cut2 * 0.99998f;
  const float never_half = w.quadrupole ? sa.accept_half : 0.f;  // nodes from this half-size on are never accepted
  const float theta2 = static_cast<float>(w.theta * w.theta);
  const float env2 = 0.0064f;  // 0.08^2
  const uint32_t groups = *a.group_count;

  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(a.work, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= groups) break;
    long long started = 0;
    if (a.chunk_cost) started = clock64();
    const uint2 gr = a.groups[item];
    const int64_t v = static_cast<int64_t>(gr.x) + t;
    const bool valid = t < static_cast<int>(gr.y & ~kWideRun);
    uint32_t slot = 0, row = kInvalid;
    double px = 0.0, py = 0.0, pz = 0.0;
    if (valid) {
      slot = a.order[v];
      row = a.active ? a.active[slot] : slot;
      targetPosition(a, v, slot, row, px, py, pz);
    }
    // FP64 takes targets and sources at the caller's coordinates (callerOffset)
    const double ux = px, uy = py, uz = pz;
    if constexpr (kF64) {
      if (valid && !a.tx) {
        px = a.sx[row];
        py = a.sy[row];
        pz = a.sz[row];
      }
    }
    const uint32_t self_pos = kIndex && valid && row < a.n ? a.pos_of_row[row] : kInvalid;
    // the box of the targets
    GroupFrame frame;
    {
      const double rx = __shfl_sync(0xffffffffu, ux, 0), ry = __shfl_sync(0xffffffffu, uy, 0),
                   rz = __shfl_sync(0xffffffffu, uz, 0);
      groupAxis(rx, valid ? static_cast<float>(targetOffset(a, ux - rx, 0)) : 0.f, frame.cx, frame.hx);
      groupAxis(ry, valid ? static_cast<float>(targetOffset(a, uy - ry, 1)) : 0.f, frame.cy, frame.hy);
      groupAxis(rz, valid ? static_cast<float>(targetOffset(a, uz - rz, 2)) : 0.f, frame.cz, frame.hz);
    }
    const double cx = frame.cx, cy = frame.cy, cz = frame.cz;
    const float hbx = frame.hx, hby = frame.hy, hbz = frame.hz;
    // the origin of the FP32 offsets: the centre, or the first target of a run of
    // 32 that spreads wide (its pairs keep the rounding of that frame)
    double fx0 = cx, fy0 = cy, fz0 = cz;
    if constexpr (!kF64) {
      if (gr.y & kWideRun) {
        const int64_t v0 = static_cast<int64_t>(gr.x & ~31u);
        const uint32_t s0 = a.order[v0];
        targetPosition(a, v0, s0, a.active ? a.active[s0] : s0, fx0, fy0, fz0);
        fx0 = cx - frameImage(cx - fx0, w.box[0], w.inv_box[0]);
        fy0 = cy - frameImage(cy - fy0, w.box[1], w.inv_box[1]);
        fz0 = cz - frameImage(cz - fz0, w.box[2], w.inv_box[2]);
      }
    }
    const float bx = static_cast<float>(cx - fx0), by = static_cast<float>(cy - fy0), bz = static_cast<float>(cz - fz0);
    // target offsets from the origin: the arithmetic of the queued sources, so
    // a target meets its own entry at distance exactly zero
    Real tx = Real(0), ty = Real(0), tz = Real(0);
    if (valid) {
      if constexpr (kF64) {
        tx = callerOffset(px, targetOffset(a, ux - cx, 0), cx, w.box[0], w.inv_box[0]);
        ty = callerOffset(py, targetOffset(a, uy - cy, 1), cy, w.box[1], w.inv_box[1]);
        tz = callerOffset(pz, targetOffset(a, uz - cz, 2), cz, w.box[2], w.inv_box[2]);
      } else {
        tx = static_cast<Real>(targetOffset(a, px - fx0, 0));
        ty = static_cast<Real>(targetOffset(a, py - fy0, 1));
        tz = static_cast<Real>(targetOffset(a, pz - fz0, 2));
      }
    }
    const double eps_d = kLanes == kMassEpsLanes ? targetEps(a, slot, row, valid) : w.eps;
    const float eps_f = static_cast<float>(eps_d);
    acc[lane] = 0.0;
    acc[32 + lane] = 0.0;
    acc[64 + lane] = 0.0;
    int qn = 0;              // queued sources
    uint32_t on = ~0u;       // lanes taking the queued sources
    int sp = 1;
    if (lane == 0) {
      stack[0] = 0u;
      stack_mask[0] = ~0u;
    }
    __syncwarp();

    // Pair loop over the queue.
    auto flush = [&]() {
      if (qn == 0) return;
      if constexpr (!kF64) {
        const int quads = (qn + 4 * share - 1) / (4 * share) * share;
        for (int i = qn + lane; i < 4 * quads; i += 32) {
          qx[i] = kFar;
          qy[i] = 0.f;
          qz[i] = 0.f;
          if constexpr (kLanes >= kMassLane) qm[i] = 0.f;
          if constexpr (kLanes >= kMassEpsLanes) qe[i] = 0.f;
          if constexpr (kIndex) qi[i] = kInvalid;
        }
        __syncwarp();
        const float2 ntx = make_float2(-tx, -tx), nty = make_float2(-ty, -ty), ntz = make_float2(-tz, -tz);
        // two sets of sums: each takes a quarter of the batch per half, so FP32
        // sums stay short (near-uniform regions cancel to a small force)
        float2 fx = make_float2(0.f, 0.f), fy = fx, fz = fx, hx = fx, hy = fx, hz = fx;
        auto pairStep = [&](float2 sx, float2 sy, float2 sz, float2 m, float2 es, bool ok0, bool ok1, float2& fx,
                            float2& fy, float2& fz) {
          const float2 dx = __fadd2_rn(sx, ntx);
          const float2 dy = __fadd2_rn(sy, nty);
          const float2 dz = __fadd2_rn(sz, ntz);
          // r^2 + eps^2 in one chain (eps^2 folded into the cutoff test and the
          // polynomial variable), or r^2 apart
          float2 r2e, r2;
          if constexpr (kFolded) {
            r2e = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, a.eps2_2)));
            r2 = r2e;
          } else {
            r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
            r2e = r2;
            if constexpr (kPairEps) {
              const float2 ep = make_float2(fmaxf(es.x, eps_f), fmaxf(es.y, eps_f));
              r2e = __ffma2_rn(ep, ep, r2);
            } else if constexpr (kEps == kEpsGuard) {
              r2e = __fadd2_rn(r2, a.eps2_2);
            }
          }
          const float cut_t = kFolded ? a.cut2e : cut2;
          bool in0 = r2.x <= cut_t, in1 = r2.y <= cut_t;
          if constexpr (kIndex) {
            in0 = in0 && ok0;
            in1 = in1 && ok1;
          }
          // coincident particles add nothing
          if constexpr (!kFolded) {
            in0 = in0 && r2.x > 0.f;
            in1 = in1 && r2.y > 0.f;
          }
          const float2 klong = hornerR2x2<kTerms>(a.pk2, r2, a.sc2, kFolded ? a.soff2 : a.mone2);
          const float2 rinv = make_float2(rsqrtf(r2e.x), rsqrtf(r2e.y));
          float2 k3 = __ffma2_rn(__fmul2_rn(rinv, rinv), rinv, klong);  // K_soft - K_long
          if constexpr (kLanes >= kMassLane) k3 = __fmul2_rn(k3, m);
          const float2 f = make_float2(in0 ? k3.x : 0.f, in1 ? k3.y : 0.f);
          fx = __ffma2_rn(f, dx, fx);
          fy = __ffma2_rn(f, dy, fy);
          fz = __ffma2_rn(f, dz, fz);
        };
#pragma unroll 2
        for (int q = sub; q < quads; q += share) {
          const float4 X = reinterpret_cast<const float4*>(qx)[q];
          const float4 Y = reinterpret_cast<const float4*>(qy)[q];
          const float4 Z = reinterpret_cast<const float4*>(qz)[q];
          float4 M = make_float4(0.f, 0.f, 0.f, 0.f), E = M;
          uint4 I = make_uint4(0u, 0u, 0u, 0u);
          if constexpr (kLanes >= kMassLane) M = reinterpret_cast<const float4*>(qm)[q];
          if constexpr (kLanes >= kMassEpsLanes) E = reinterpret_cast<const float4*>(qe)[q];
          if constexpr (kIndex) I = reinterpret_cast<const uint4*>(qi)[q];
          pairStep(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), make_float2(M.x, M.y),
                   make_float2(E.x, E.y), I.x != self_pos, I.y != self_pos, fx, fy, fz);
          pairStep(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), make_float2(M.z, M.w),
                   make_float2(E.z, E.w), I.z != self_pos, I.w != self_pos, hx, hy, hz);
        }
        if ((on >> lane) & 1u) {
          const float g = kLanes == kUniformMass ? w.G_f * w.m0_f : w.G_f;
          acc[lane] += static_cast<double>(g * ((fx.x + fx.y) + (hx.x + hx.y)));
          acc[32 + lane] += static_cast<double>(g * ((fy.x + fy.y) + (hy.x + hy.y)));
          acc[64 + lane] += static_cast<double>(g * ((fz.x + fz.y) + (hz.x + hz.y)));
        }
      } else {
        double fx = 0.0, fy = 0.0, fz = 0.0;
#pragma unroll 2
        for (int k = sub; k < qn; k += share) {
          const double dx = qx[k] - tx, dy = qy[k] - ty, dz = qz[k] - tz;
          const double r2 = dx * dx + dy * dy + dz * dz;
          bool in = r2 <= w.cutoff2 && r2 > 0.0;
          if constexpr (kIndex) in = in && qi[k] != self_pos;
          const double pe = fmax(qe[k], eps_d);
          double kr;
          if constexpr (kTerms > 0) {
            kr = softMinusLong64(r2, pe, sa.h64_scale, sa.h64);
          } else {
            kr = !in ? 0.0 : (w.gauss_lookup ? gaussResidualInvR3(a, r2, pe) : residualInvR3(r2, pe, w.rs));
          }
          const double f = in ? kr * qm[k] : 0.0;
          fx = fma(f, dx, fx);
          fy = fma(f, dy, fy);
          fz = fma(f, dz, fz);
        }
        if ((on >> lane) & 1u) {
          acc[lane] += w.G * fx;
          acc[32 + lane] += w.G * fy;
          acc[64 + lane] += w.G * fz;
        }
      }
      qn = 0;
      __syncwarp();
    };

    // FP64: the sources' origin at the image (ix, iy, iz)
    auto setOrigin = [&](double ix, double iy, double iz) {
      if (lane < 6) {
        const int axis = lane >> 1;
        origin[lane] = movedOrigin(axis == 0 ? cx : (axis == 1 ? cy : cz),
                                   (axis == 0 ? ix : (axis == 1 ? iy : iz)) - (lane & 1),
                                   axis == 0 ? w.box[0] : (axis == 1 ? w.box[1] : w.box[2]));
      }
      __syncwarp();
    };

    // Queue the sources [begin, begin + count) within r_cut of the box, as
    // offsets from the origin moved by (ix, iy, iz) box lengths to the sources'
    // image. `lanes` take them; `inside`: every one is within r_cut of every target.
    auto enqueue = [&](uint32_t begin, uint32_t count, uint32_t lanes, bool inside, double ix, double iy, double iz) {
      const bool caller = kF64 && sa.canonical != 0;  // positions as the caller gave them
      const double4* src = (caller ? a.src_d4 : a.src_u4) + begin;
      // unmoved sources keep the origin's bits (FP32: a target's own entry stays at
      // distance zero)
      const double sx = fx0 + w.box[0] * ix, sy = fy0 + w.box[1] * iy, sz = fz0 + w.box[2] * iz;
      // rounding of the box's position in the frame
      const float slack = 2.4e-7f * fmaxf(fabsf(bx), fmaxf(fabsf(by), fabsf(bz)));
      uint32_t k = lane;
      double4 u = make_double4(0.0, 0.0, 0.0, 0.0);
      if (k < count) u = src[k];
      for (uint32_t chunk = 0; chunk < count; chunk += 32) {
        const double4 cur = u;
        const bool have = k < count;
        const uint32_t pos = begin + k;
        k += 32;
        if (k < count) u = src[k];  // the next chunk's sources, on their way during this one
        if (qn > kQ - 32 || lanes != on) flush();
        on = lanes;
        double dx = cur.x - sx, dy = cur.y - sy, dz = cur.z - sz;
        if constexpr (kF64) {
          if (caller) {
            // a position below the anchor is a box length further up in the tree frame
            const double2 px0 = origin[cur.x < sa.anchor[0] ? 1 : 0], py0 = origin[cur.y < sa.anchor[1] ? 3 : 2],
                          pz0 = origin[cur.z < sa.anchor[2] ? 5 : 4];
            dx = __dsub_rn(__dsub_rn(cur.x, px0.x), px0.y);
            dy = __dsub_rn(__dsub_rn(cur.y, py0.x), py0.y);
            dz = __dsub_rn(__dsub_rn(cur.z, pz0.x), pz0.y);
          } else if (have) {
            // coordinates outside the box: the image the tree frame took
            const double4 p = a.src_d4[pos];
            dx = callerOffset(p.x, dx, cx, w.box[0], w.inv_box[0]);
            dy = callerOffset(p.y, dy, cy, w.box[1], w.inv_box[1]);
            dz = callerOffset(p.z, dz, cz, w.box[2], w.inv_box[2]);
          }
        }
        const float ex = static_cast<float>(dx), ey = static_cast<float>(dy), ez = static_cast<float>(dz);
        bool keep = have;
        if (!inside) {
          const float gx = fmaxf(fabsf(ex - bx) - (hbx + slack), 0.f), gy = fmaxf(fabsf(ey - by) - (hby + slack), 0.f),
                      gz = fmaxf(fabsf(ez - bz) - (hbz + slack), 0.f);
          keep = have && fmaf(gx, gx, fmaf(gy, gy, gz * gz)) <= cut_hi2;
        }
        const uint32_t kept = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int o = qn + __popc(kept & ((1u << lane) - 1u));
          if constexpr (kF64) {
            qx[o] = dx;
            qy[o] = dy;
            qz[o] = dz;
          } else {
            qx[o] = ex;
            qy[o] = ey;
            qz[o] = ez;
          }
          if constexpr (kLanes >= kMassLane) qm[o] = static_cast<Real>(cur.w);
          if constexpr (kLanes >= kMassEpsLanes) qe[o] = static_cast<Real>(sourceEps(a, pos));
          if constexpr (kIndex) qi[o] = pos;
        }
        qn += __popc(kept);
        __syncwarp();
      }
    };

    if constexpr (kF64) setOrigin(0.0, 0.0, 0.0);
    bool overflow = false;
    while (sp > 0) {
      // take up to 32 nodes, leaving room for a depth-first descent below them
      const int room = sa.batch_cap - sp;
      const int k = room >= 7 ? min(min(sp, 32), room / 7) : 1;
      const bool have = lane < k;
      const uint32_t entry = have ? stack[sp - 1 - lane] : 0u;
      const uint32_t mask = have ? stack_mask[sp - 1 - lane] : 0u;
      sp -= k;
      __syncwarp();
      const uint32_t node = entry & ~kInBlock;
      bool in_block = (entry & kInBlock) != 0u;
      const NodeReach r = nodeReach(a.geom, a.range, node, have, frame, w);
      const uint4 rg = r.rg;
      const float hf = r.hf;
      const bool reach = have && r.gap2 <= cut_hi2;
      const bool leaf = rg.z == 0u;
      // could some target accept the node as a multipole? It must lie inside
      // r_cut of the target and be narrower than 0.08 of its distance.
      bool may = false;
      if (reach && !leaf && !in_block && hf < never_half) {
        const float nx = fmaxf(r.ax - hbx, 0.f) + hf, ny = fmaxf(r.ay - hby, 0.f) + hf, nz = fmaxf(r.az - hbz, 0.f) + hf;
        may = fmaf(nx, nx, fmaf(ny, ny, nz * nz)) <= cut_hi2 && 4.0f * hf * hf < 0.00641f * r.far2;
      }
      if (!may && !leaf && rg.y <= kStrictBlock && r.half <= sa.block_half) in_block = true;
      const bool whole = leaf || (in_block && (rg.y <= kStrictCull || r.far2 <= cut_lo2));
      const bool emit = reach && !may && whole;
      const bool push = reach && !may && !whole;

      // children of the opened nodes
      sp = pushChildren(a.child, node, push, rg.z, in_block ? kInBlock : 0u, stack, sp, sa.stack_cap, overflow,
                        stack_mask, mask);
      if (overflow) break;

      // nodes some target may accept: decided per target (every lane, one node
      // at a time); the rest of the targets see the node again, opened
      for (unsigned todo = __ballot_sync(0xffffffffu, may); todo; todo &= todo - 1u) {
        const int j = __ffs(todo) - 1;
        const uint32_t nd = __shfl_sync(0xffffffffu, node, j);
        const uint32_t lanes = __shfl_sync(0xffffffffu, mask, j);
        const double4 ng = a.geom[nd];
        const uint4 nr = a.range[nd];
        const double ox = __shfl_sync(0xffffffffu, r.ndx, j), oy = __shfl_sync(0xffffffffu, r.ndy, j),
                     oz = __shfl_sync(0xffffffffu, r.ndz, j);
        bool accept = false;
        if (valid && ((lanes >> lane) & 1u)) {
          float mx = 0.f, my = 0.f, mz = 0.f;  // COM offset of an accepted node
          const float h = static_cast<float>(ng.w);
          const float omax = fmaxf(fabsf(static_cast<float>(ox)), fmaxf(fabsf(static_cast<float>(oy)), fabsf(static_cast<float>(oz))));
          const float hb = fmaxf(hbx, fmaxf(hby, hbz));
          // bound on the error of each FP32 offset component
          const float fe = 2.4e-7f * (omax + hb + h + fmaxf(fabsf(bx), fmaxf(fabsf(by), fabsf(bz))));
          const float cut_e = 4.0f * sa.cut_f * fe;
          const float dx = static_cast<float>(ox) - (static_cast<float>(tx) - bx), dy = static_cast<float>(oy) - (static_cast<float>(ty) - by),
                      dz = static_cast<float>(oz) - (static_cast<float>(tz) - bz);
          // the node lies inside r_cut (< L/2) of this target only if this is
          // its nearest image; other images fail the containment test
          const float qx_ = fabsf(dx) + h, qy_ = fabsf(dy) + h, qz_ = fabsf(dz) + h;
          const int within = certainLess(fmaf(qx_, qx_, fmaf(qy_, qy_, qz_ * qz_)), cut2, cut_e);
          bool exact = within == 0;
          if (within > 0) {
            const float4 nf = a.node_f4[nd];
            mx = dx + nf.x;
            my = dy + nf.y;
            mz = dz + nf.z;
            const float r2 = fmaf(mx, mx, fmaf(my, my, mz * mz));
            const float w2 = 4.0f * h * h;
            const float r2_e = 4.0f * (r2 * rsqrtf(r2)) * fe;
            const int env = certainLess(w2, env2 * r2, env2 * r2_e);
            int mac = 0;
            History hist = loadHistory(w.criterion == 2 ? a.prev : nullptr, slot, true);
            if (w.criterion == 2 && hist.avail) {
              // relative-force MAC: G M w^2 / r^4 against alpha max(|a_prev|, floor)
              float allow = static_cast<float>(w.rel_tol * fmax(fabs(hist.mag), w.floor_));
              if (!(allow >= FLT_MIN && allow <= FLT_MAX)) allow = 0.f;
              const float ir = __fdividef(1.0f, r2);
              const float lower = w.G_f * a.node_mq[2 * static_cast<size_t>(nd)].x * (w2 * ir) * ir;
              mac = allow > 0.f && isfinite(lower) ? -certainLess(allow, lower, 2.0f * lower * (r2_e / r2)) : 0;
            } else {
              const float l2 = w.criterion == 0 ? w2 : (2.0f * h + nf.w) * (2.0f * h + nf.w);
              mac = certainLess(l2, theta2 * r2, theta2 * r2_e);
            }
            if (env < 0 || mac < 0) accept = false;
            else if (env == 0 || mac == 0) exact = true;
            else accept = true;
            if constexpr (kLanes == kMassEpsLanes) {
              // sources of differing softenings: the FP64 envelope guard
              if (a.node_soft) {
                const double2 ns = a.node_soft[nd];
                if (ns.y - ns.x > 1.0e-12) exact = true;
              }
            }
          }
          if (exact || (accept && kF64)) {
            // the reference's FP64 decision at the caller's coordinates
            const double ex = a.tx ? a.tx[slot] : a.sx[row], ey = a.ty ? a.ty[slot] : a.sy[row],
                         ez = a.tz ? a.tz[slot] : a.sz[row];
            const History hist = loadHistory(w.criterion == 2 ? a.prev : nullptr, slot, true);
            const ExactDecision d = exactNodeDecision<false>(a, nd, ex, ey, ez, row < a.n, hist, eps_d);
            accept = accept || (d.accept && !d.prune);
            if (exact) accept = d.accept && !d.prune;
            mx = static_cast<float>(d.dx);
            my = static_cast<float>(d.dy);
            mz = static_cast<float>(d.dz);
            if (kF64 && accept && sub == 0) {
              double fx = 0.0, fy = 0.0, fz = 0.0;
              multipoleForce(a, nd, d.dx, d.dy, d.dz, eps_d, fx, fy, fz);
              acc[lane] += fx;
              acc[32 + lane] += fy;
              acc[64 + lane] += fz;
            }
          }
          if (!kF64 && accept && sub == 0) {
            if (a.mult_f32 && fmaf(mx, mx, fmaf(my, my, mz * mz)) >= fmaxf(1.0e-8f * cut2, 1.0e-10f)) {
              float me2 = kEpsZero ? 0.f : w.eps2_f;
              if constexpr (kLanes == kMassEpsLanes) {
                const float me = static_cast<float>(nodeEps(a, nd, eps_d));
                me2 = me * me;
              }
              float fx = 0.f, fy = 0.f, fz = 0.f;
              multipoleF32<kEpsZero, kF64 ? 9 : kTerms>(a, nd, mx, my, mz, sa.sc_r2, fx, fy, fz, me2);
              acc[lane] += static_cast<double>(w.G_f * fx);
              acc[32 + lane] += static_cast<double>(w.G_f * fy);
              acc[64 + lane] += static_cast<double>(w.G_f * fz);
            } else {
              // FP32 powers of 1/r could overflow this close to the COM, or the
              // FP32 split constants are out of range for this r_s
              const double ex = a.tx ? a.tx[slot] : a.sx[row], ey = a.ty ? a.ty[slot] : a.sy[row],
                           ez = a.tz ? a.tz[slot] : a.sz[row];
              const History hist = loadHistory(w.criterion == 2 ? a.prev : nullptr, slot, true);
              const ExactDecision d = exactNodeDecision<false>(a, nd, ex, ey, ez, row < a.n, hist, eps_d);
              double fx = 0.0, fy = 0.0, fz = 0.0;
              multipoleForce(a, nd, d.dx, d.dy, d.dz, eps_d, fx, fy, fz);
              acc[lane] += fx;
              acc[32 + lane] += fy;
              acc[64 + lane] += fz;
            }
          }
        }
        const uint32_t rest = lanes & ~__ballot_sync(0xffffffffu, accept);
        if ((rest & __ballot_sync(0xffffffffu, valid)) == 0u) continue;
        const bool block = nr.y <= kStrictBlock && ng.w <= sa.block_half;
        const int add = block ? 1 : static_cast<int>(nr.z);
        if (sp + add > sa.stack_cap) {
          overflow = true;
          break;
        }
        if (block) {
          if (lane == 0) {
            stack[sp] = nd | kInBlock;
            stack_mask[sp] = rest;
          }
        } else {
          const uint32_t ch = lane < 8 ? a.child[8 * static_cast<size_t>(nd) + lane] : kInvalid;
          const unsigned cm = __ballot_sync(0xffffffffu, ch != kInvalid);
          if (ch != kInvalid) {
            const int at = sp + __popc(cm & ((1u << lane) - 1u));
            stack[at] = ch;
            stack_mask[at] = rest;
          }
        }
        sp += add;
        __syncwarp();
      }
      if (overflow) break;

      // sources of the nodes taken whole
      const float Lx = static_cast<float>(w.box[0]), Ly = static_cast<float>(w.box[1]), Lz = static_cast<float>(w.box[2]);
      // reach of the group spans more than the nearest image on some axis
      const float rc = sa.cut_f * 1.00001f + hf;
      const bool images = emit && ((Lx > 0.f && r.ax + hbx + rc >= Lx * 0.99999f) ||
                                   (Ly > 0.f && r.ay + hby + rc >= Ly * 0.99999f) ||
                                   (Lz > 0.f && r.az + hbz + rc >= Lz * 0.99999f));
      const unsigned moved = __ballot_sync(0xffffffffu, emit && (r.kx != 0.0 || r.ky != 0.0 || r.kz != 0.0));
      const unsigned many = __ballot_sync(0xffffffffu, images);
      const unsigned within = __ballot_sync(0xffffffffu, r.far2 <= cut_lo2);  // no source to cull
      for (unsigned todo = __ballot_sync(0xffffffffu, emit); todo; todo &= todo - 1u) {
        const int j = __ffs(todo) - 1;
        const uint32_t begin = __shfl_sync(0xffffffffu, rg.x, j), count = __shfl_sync(0xffffffffu, rg.y, j);
        const uint32_t lanes = __shfl_sync(0xffffffffu, mask, j);
        const bool shift = ((moved >> j) & 1u) != 0u, each = ((many >> j) & 1u) != 0u;
        double jx = 0.0, jy = 0.0, jz = 0.0;
        int nx = 1, ny = 1, nz = 1;
        if (shift || each) {
          jx = __shfl_sync(0xffffffffu, r.kx, j);
          jy = __shfl_sync(0xffffffffu, r.ky, j);
          jz = __shfl_sync(0xffffffffu, r.kz, j);
        }
        if (each) {
          const double h = __shfl_sync(0xffffffffu, r.half, j);
          nodeImages(w, sa.frame, 0, __shfl_sync(0xffffffffu, r.ndx, j), h, cx, hbx, jx, nx);
          nodeImages(w, sa.frame, 1, __shfl_sync(0xffffffffu, r.ndy, j), h, cy, hby, jy, ny);
          nodeImages(w, sa.frame, 2, __shfl_sync(0xffffffffu, r.ndz, j), h, cz, hbz, jz, nz);
        }
        for (int ix = 0, iy = 0, iz = 0; iz < nz;) {
          if constexpr (kF64) {
            if (shift || each) setOrigin(jx + ix, jy + iy, jz + iz);
          }
          enqueue(begin, count, lanes, !each && ((within >> j) & 1u) != 0u, jx + ix, jy + iy, jz + iz);
          if (++ix == nx) {
            ix = 0;
            if (++iy == ny) {
              iy = 0;
              ++iz;
            }
          }
        }
        if constexpr (kF64) {
          if (shift || each) setOrigin(0.0, 0.0, 0.0);
        }
      }
    }
    flush();
    if (overflow && lane == 0) atomicOr(a.status, kStatusStackOverflow);
    // the lanes sharing a target
    double rx = acc[lane], ry = acc[32 + lane], rz = acc[64 + lane];
    for (int off = 16; off >= per; off >>= 1) {
      rx += __shfl_xor_sync(0xffffffffu, rx, off);
      ry += __shfl_xor_sync(0xffffffffu, ry, off);
      rz += __shfl_xor_sync(0xffffffffu, rz, off);
    }
    if (valid && sub == 0) {
      const int64_t o = a.out_compact ? v - a.v0 : slot;
      a.out_x[o] = rx;
      a.out_y[o] = ry;
      a.out_z[o] = rz;
    }
    if (a.chunk_cost && lane == 0) atomicAdd(a.chunk_cost + (gr.x >> 5), static_cast<float>(clock64() - started));
    __syncwarp();
  }
}

template <class Real, int kEps, int kTerms, int kLanes, bool kIndex>
int launchStrict(const WalkArgs& a, const StrictArgs& sa, cudaStream_t s) {
  auto kernel = walkStrictKernel<Real, kEps, kTerms, kLanes, kIndex>;
  const size_t smem = kWalkWarpsPerBlock * WarpShared<Real, kLanes, kIndex>::bytes(sa.stack_cap);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess)
    return CHUI_TREEPM_EDEVICE;
  int dev = 0, sms = 148, per_sm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWalkWarpsPerBlock * 32, smem);
  // groups are counted on the device; no more warps than there can be groups
  const int64_t most = a.v1 - a.v0;
  const int64_t blocks = std::min<int64_t>(static_cast<int64_t>(sms) * std::max(per_sm, 1),
                                           (most + kWalkWarpsPerBlock - 1) / kWalkWarpsPerBlock);
  noteLaunch();
  kernel<<<static_cast<unsigned>(std::max<int64_t>(blocks, 1)), kWalkWarpsPerBlock * 32, smem, s>>>(a, sa);
  return cudaGetLastError() == cudaSuccess ? 0 : CHUI_TREEPM_EDEVICE;
}

}  // namespace

int targetGroups(Context& c, const WalkArgs& a, int most, double limit, const uint2** groups, const uint32_t** count,
                 cudaStream_t s) {
  const int64_t targets = a.v1 - a.v0;
  if (ensure(c.walk_groups, static_cast<size_t>(targets) * sizeof(uint2)) || ensure(c.work_counter, 16))
    return CHUI_TREEPM_ENOMEM;
  uint32_t* n = c.work_counter.as<uint32_t>() + 2;
  cudaMemsetAsync(n, 0, 4, s);
  const int64_t blocks = std::min<int64_t>((targets + 255) / 256, 148 * 16);
  noteLaunch();
  targetGroupsKernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(a, most, limit, c.walk_groups.as<uint2>(), n);
  *groups = c.walk_groups.as<uint2>();
  *count = n;
  return cudaGetLastError() == cudaSuccess ? 0 : CHUI_TREEPM_EDEVICE;
}

int walkStrictRun(Context& c, WalkArgs& a, bool f64, bool tiny, cudaStream_t s) {
  StrictArgs sa{};
  // Lanes per target: a group of 32 / S targets has a smaller box and keeps
  // fewer sources for nothing, but each group walks the tree; S > 1 pays where
  // there are too few groups to fill the schedulers (592) evenly. Measured with
  // S = 1 / 2 / 4 / 8: 33 k targets 0.128 / 0.105 / 0.110 / 0.140 ms, 50 k 1.90 /
  // 1.35 / 1.08 / 1.29, 70 k 0.92 / 0.69 / 0.69 / 0.90, 200 k 2.20 / 2.09 / 2.39 /
  // 3.19, 262 k 1.38 / 1.45 / 1.82 / 2.66. FP64 pairs cost more against the
  // traversal: 262 k 4.10 / 3.51 / 3.41 / 4.06.
  const int64_t targets = a.v1 - a.v0;
  int per = 32;
  while (per > 8 && targets / per < (f64 ? 12000 : 4000)) per >>= 1;
  if (targets / 8 < 592) per = 4;
  sa.targets_per_group = per;
  // Largest extent of a group: 1.0 / 1.5 / 2.5 r_cut take 170.9 / 165.9 / 168.2 ms
  // at 256^3 clustered.
  double limit = 1.5 * c.cutoff;
  if (a.wp.box[0] > 0.0) limit = std::min(limit, 0.25 * std::min({a.wp.box[0], a.wp.box[1], a.wp.box[2]}));
  if (int rc = targetGroups(c, a, per, limit, &a.groups, &a.group_count, s)) return rc;
  const int depth_first = 1 + 7 * std::max<int>(static_cast<int>(c.max_depth), 1);
  sa.batch_cap = kBatchStack;
  sa.stack_cap = (kBatchStack + depth_first + 7 + 1) & ~1;  // even: 16-byte aligned warps
  // In a tiny box the reference's own decisions are kept for every node (its
  // multipoles are few and its box is checked pair by pair), unless no internal
  // node is small enough to be accepted anyway.
  const double smallest = std::ldexp(c.root_half, -std::max<int>(static_cast<int>(c.max_depth) - 1, 0));
  const bool blocks = !tiny || !a.wp.quadrupole || smallest > 0.0401 * c.cutoff;
  sa.block_half = blocks ? kStrictHalf * c.cutoff : -1.0;
  sa.cut_f = static_cast<float>(c.cutoff);
  sa.frame = sourceFrame(c);
  sa.accept_half = static_cast<float>(0.04 * c.cutoff * 1.0001);
  sa.sc_r2 = a.wp.inv_4rs2_f * a.poly.scale;
  const bool index = a.tx != nullptr;
  const bool soft = a.src_eps || a.tgt_eps;
  if (f64) {
    if (!c.poly64_fitted) {
      c.poly64 = fitPoly64(c.rs, c.cutoff);
      c.poly64_fitted = true;
    }
    for (int j = 0; j < kPoly64Terms; ++j) sa.h64[j] = c.poly64.c[j];
    sa.h64_scale = c.poly64.scale;
    sa.canonical = 1;
    for (int a0 = 0; a0 < 3; ++a0) {
      const double L = a.wp.box[a0];
      if (L > 0.0 && !(a.wp.src_lo[a0] >= 0.0 && a.wp.src_hi[a0] < L)) sa.canonical = 0;
      sa.anchor[a0] = L > 0.0 ? c.tree_anchor[a0] : -INFINITY;
    }
    return a.wp.gauss_lookup || c.poly64.terms == 0
               ? launchStrict<double, kEpsGuard, 0, kMassEpsLanes, true>(a, sa, s)
               : launchStrict<double, kEpsGuard, kPoly64Terms, kMassEpsLanes, true>(a, sa, s);
  }
  if (soft)
    return index ? launchStrict<float, kEpsGuard, kPolyMaxTerms, kMassEpsLanes, true>(a, sa, s)
                 : launchStrict<float, kEpsGuard, kPolyMaxTerms, kMassEpsLanes, false>(a, sa, s);
  const bool eps_zero = a.wp.eps == 0.0;
  const bool shortp = a.poly.terms <= kPairPolyTerms;
  // m K(0) = m (eps^-3 - 0.094 / r_s^3) of the heaviest source must be well
  // inside FP32 (a source's mass is a factor of each pair, a common mass is not)
  const double heaviest = std::max(1.0, a.wp.m_max);
  const bool finite = heaviest * (std::pow(a.wp.eps, -3.0) + 0.1 / (c.rs * c.rs * c.rs)) < 1.0e36;
#define CHUI_STRICT32(EPS, T)                                                                       \
  return index ? launchStrict<float, EPS, T, kMassLane, true>(a, sa, s)                             \
               : (a.wp.uniform_mass ? launchStrict<float, EPS, T, kUniformMass, false>(a, sa, s)    \
                                    : launchStrict<float, EPS, T, kMassLane, false>(a, sa, s))
  if (eps_zero) {
    if (shortp) CHUI_STRICT32(kEpsNone, kPairPolyTerms);
    CHUI_STRICT32(kEpsNone, kPolyMaxTerms);
  }
  if (!finite) CHUI_STRICT32(kEpsGuard, kPolyMaxTerms);
  if (shortp) CHUI_STRICT32(kEpsFinite, kPairPolyTerms);
  CHUI_STRICT32(kEpsFinite, kPolyMaxTerms);
#undef CHUI_STRICT32
}

}  // namespace chui

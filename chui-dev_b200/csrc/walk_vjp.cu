// Adjoint walk: vector-Jacobian product of the short-range force over every
// pair inside r_cut. FP64: one warp per 32 consecutive targets (walkVjpKernel).
// Mixed precision: the groups, box culling and batches of walk_strict.cu
// (walkVjpGroupKernel); nothing is ever accepted as a multipole here.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>

#include "walk.cuh"

namespace chui {
namespace {

constexpr int kQueue = 64;              // FP64: sources per warp batch
constexpr uint32_t kBulkCountVjp = 1024;  // FP64: nodes enqueued whole
constexpr double kBulkHalf = 1.0;         // ... of at most this half-size in r_cut

// ---- adjoint: vector-Jacobian product of the short-range force ----------

struct VjpArgs {
  int64_t n;                    // particles (every particle is a target)
  const uint32_t* order;        // visit position -> row (tree order)
  const double* sx;             // caller positions
  const double* sy;
  const double* sz;
  const double* m;              // masses (nullable: uniform_mass)
  double uniform_mass;
  const double* cx;             // cotangents a_bar per row
  const double* cy;
  const double* cz;
  const double4* geom;
  const uint4* range;
  const uint32_t* child;
  const double4* src_d4;        // tree order: caller position + mass
  const double4* src_c4;        // tree order: cotangent
  double* out_x;                // per row: x_bar of the short-range force (times G)
  double* out_y;
  double* out_z;
  uint32_t* work;
  uint32_t* status;
  WalkParams wp;
  // the FP32 pair loop: each coefficient in both halves (of -H/(8 r_s^3) and
  // -H'/(16 r_s^5)), the polynomial variables' scales and the constants as pairs
  float2 pk2[kPolyMaxTerms];
  float2 dk2[kPolyMaxTerms];
  float2 sc2, dsc2, mone2, eps2_2, mthree2;
  // the FP32 walk: groups of targets, source positions in the tree frame
  const double4* src_u4;
  const uint2* groups;
  const uint32_t* group_count;
  int targets_per_group;
  int stack_cap, batch_cap;
  float cut_f;
  SourceFrame frame;
};

// x_bar_k = G sum_j M(d) (m_k a_bar_j - m_j a_bar_k), d = x_j - x_k, over every
// source j within r_cut of target k (j != k, d != 0), M(d) = K I + (K'/r) d d^T
// the Jacobian of the pair force d -> K(|d|) d. Because M is even in d and the
// pair set {|d| <= r_cut} is symmetric, this gathers both the target-side and
// the source-side derivatives without scattering.
//
// This is the FP64 walk (the FP32 one, over groups of targets, follows).
// Traversal: a node is kept while the r_cut sphere of some lane may reach its
// cube (each lane with its own minimum image, so groups of targets that are
// far apart in the box still prune); leaves and nodes of at most kBulkCountVjp
// sources are enqueued whole, keeping sources inside the sphere of the lanes
// that need the node; every pair decision is the per-pair cutoff test. Queue
// entries are FP64-formed minimum-image offsets from the warp's reference
// target; when r_cut plus the group radius reaches half the box, each pair
// takes its own minimum image.
__global__ void __launch_bounds__(kWalkWarpsPerBlock * 32, 4) walkVjpKernel(VjpArgs a) {
  __shared__ uint32_t stack_sm[kWalkWarpsPerBlock][kStackCap];
  __shared__ double4 q_pos[kWalkWarpsPerBlock][kQueue];
  __shared__ double4 q_cot[kWalkWarpsPerBlock][kQueue];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  uint32_t* stack = stack_sm[warp];
  const WalkParams& w = a.wp;
  const double half_min_box = 0.5 * fmin(w.box[0], fmin(w.box[1], w.box[2]));
  const double inv_box[3] = {1.0 / w.box[0], 1.0 / w.box[1], 1.0 / w.box[2]};
  const double cut2 = w.cutoff2;
  const double box_r[3] = {w.box[0], w.box[1], w.box[2]};
  const double inv_box_r[3] = {inv_box[0], inv_box[1],
                             inv_box[2]};
  const double bulk_half = kBulkHalf * w.cutoff;

  while (true) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(a.work, 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= a.n) break;
    const int64_t v = static_cast<int64_t>(base) + lane;
    const bool valid = v < a.n;
    uint32_t row = 0;
    double px = 0.0, py = 0.0, pz = 0.0, mk = 0.0, ckx = 0.0, cky = 0.0, ckz = 0.0;
    if (valid) {
      row = a.order[v];
      px = a.sx[row];
      py = a.sy[row];
      pz = a.sz[row];
      mk = a.m ? a.m[row] : a.uniform_mass;
      ckx = a.cx[row];
      cky = a.cy[row];
      ckz = a.cz[row];
    }
    const double rx = __shfl_sync(0xffffffffu, px, 0);
    const double ry = __shfl_sync(0xffffffffu, py, 0);
    const double rz = __shfl_sync(0xffffffffu, pz, 0);
    double ox = px - rx, oy = py - ry, oz = pz - rz;
    ox -= w.box[0] * rint(ox * inv_box[0]);
    oy -= w.box[1] * rint(oy * inv_box[1]);
    oz -= w.box[2] * rint(oz * inv_box[2]);
    double rg2 = valid ? ox * ox + oy * oy + oz * oz : 0.0;
    for (int off = 16; off > 0; off >>= 1) rg2 = fmax(rg2, __shfl_xor_sync(0xffffffffu, rg2, off));
    const double reach = w.cutoff + sqrt(rg2);       // group sphere radius
    const bool pair_image = reach >= half_min_box * (1.0 - 1.0e-9);
    const double tx = ox, ty = oy, tz = oz;
    const double mkr = mk;
    const double ckxr = ckx, ckyr = cky, ckzr = ckz;
    double acc_x = 0.0, acc_y = 0.0, acc_z = 0.0;
    int qn = 0;
    if (lane == 0) stack[0] = 0u;
    int sp = 1;
    __syncwarp();
    bool overflow = false;

    auto flush = [&]() {
      double gx = 0.0, gy = 0.0, gz = 0.0;
#pragma unroll 2
      for (int k = 0; k < qn; ++k) {
        const double4 e = q_pos[warp][k], cj = q_cot[warp][k];
        double dx = e.x - tx, dy = e.y - ty, dz = e.z - tz;
        if (pair_image) {
          dx -= box_r[0] * rint(dx * inv_box_r[0]);
          dy -= box_r[1] * rint(dy * inv_box_r[1]);
          dz -= box_r[2] * rint(dz * inv_box_r[2]);
        }
        const double r2 = dx * dx + dy * dy + dz * dz;
        const bool in = valid && r2 <= cut2 && r2 > 0.0;
        const double rr = in ? r2 : 1.0;
        const double K = residualInvR3(rr, w.eps, w.rs), Kp = residualDerivOverR(rr, w.eps, w.rs);
        const double c0 = mkr * cj.x - e.w * ckxr;
        const double c1 = mkr * cj.y - e.w * ckyr;
        const double c2 = mkr * cj.z - e.w * ckzr;
        const double dc = (dx * c0 + dy * c1 + dz * c2) * Kp;
        // select, not multiply: K and K' are infinite for the excluded self pair
        gx += in ? K * c0 + dc * dx : 0.0;
        gy += in ? K * c1 + dc * dy : 0.0;
        gz += in ? K * c2 + dc * dz : 0.0;
      }
      acc_x += static_cast<double>(gx);
      acc_y += static_cast<double>(gy);
      acc_z += static_cast<double>(gz);
      qn = 0;
      __syncwarp();
    };

    auto enqueue = [&](uint32_t begin, uint32_t count, uint32_t mask) {
      // sphere of the lanes that need the node (their offsets, FP64)
      const int first = __ffs(mask) - 1;
      const double scx = __shfl_sync(0xffffffffu, ox, first);
      const double scy = __shfl_sync(0xffffffffu, oy, first);
      const double scz = __shfl_sync(0xffffffffu, oz, first);
      double d2 = 0.0;
      if ((mask >> lane) & 1u) {
        const double ux = ox - scx, uy = oy - scy, uz = oz - scz;
        d2 = ux * ux + uy * uy + uz * uz;
      }
      for (int off = 16; off > 0; off >>= 1) d2 = fmax(d2, __shfl_xor_sync(0xffffffffu, d2, off));
      const double sr = w.cutoff + sqrt(d2);
      const double sr2 = sr * sr * (1.0 + 1.0e-6);
      // a sphere reaching half the box keeps everything; in warps whose pairs
      // take their own minimum image, the distance to its centre is wrapped too
      const bool keep_all = sr >= half_min_box * (1.0 - 1.0e-9);
      for (uint32_t chunk = 0; chunk < count; chunk += 32) {
        const uint32_t k = chunk + lane;
        bool keep = false;
        double ex = 0.0, ey = 0.0, ez = 0.0;
        double4 sv = make_double4(0.0, 0.0, 0.0, 0.0), cv = sv;
        if (k < count) {
          sv = a.src_d4[begin + k];
          ex = sv.x - rx;
          ey = sv.y - ry;
          ez = sv.z - rz;
          ex -= w.box[0] * rint(ex * inv_box[0]);
          ey -= w.box[1] * rint(ey * inv_box[1]);
          ez -= w.box[2] * rint(ez * inv_box[2]);
          double qx = ex - scx, qy = ey - scy, qz = ez - scz;
          if (pair_image) {
            qx -= w.box[0] * rint(qx * inv_box[0]);
            qy -= w.box[1] * rint(qy * inv_box[1]);
            qz -= w.box[2] * rint(qz * inv_box[2]);
          }
          keep = keep_all || qx * qx + qy * qy + qz * qz <= sr2;
          if (keep) cv = a.src_c4[begin + k];
        }
        const uint32_t keep_mask = __ballot_sync(0xffffffffu, keep);
        const int c = __popc(keep_mask);
        if (qn + c > kQueue) flush();
        if (keep) {
          const int slot_q = qn + __popc(keep_mask & ((1u << lane) - 1u));
          q_pos[warp][slot_q] = make_double4(ex, ey, ez, sv.w);
          q_cot[warp][slot_q] = cv;
        }
        __syncwarp();
        qn += c;
      }
    };

    while (sp > 0) {
      const uint32_t node = stack[sp - 1];
      --sp;
      __syncwarp();
      const double4 g = a.geom[node];
      const uint4 rg4 = a.range[node];
      const double h = g.w;
      // lanes whose r_cut sphere may reach the node cube: each lane takes its
      // own minimum image of the cube centre, so the test holds however far
      // apart the warp's targets are (only cubes with h + r_cut >= L/2, near
      // the root, are never pruned)
      bool need = valid;
      if (valid && h + w.cutoff < half_min_box * (1.0 - 1.0e-9)) {
        double dx = g.x - px, dy = g.y - py, dz = g.z - pz;
        dx -= w.box[0] * rint(dx * inv_box[0]);
        dy -= w.box[1] * rint(dy * inv_box[1]);
        dz -= w.box[2] * rint(dz * inv_box[2]);
        const double ex = fmax(0.0, fabs(dx) - h), ey = fmax(0.0, fabs(dy) - h), ez = fmax(0.0, fabs(dz) - h);
        need = ex * ex + ey * ey + ez * ez <= w.cutoff2 * (1.0 + 1.0e-9);
      }
      const uint32_t need_mask = __ballot_sync(0xffffffffu, need);
      if (need_mask == 0u) continue;
      if (rg4.z == 0 || (rg4.y <= kBulkCountVjp && h <= bulk_half)) {
        enqueue(rg4.x, rg4.y, need_mask);
        continue;
      }
      const uint32_t ch = lane < 8 ? a.child[8 * static_cast<size_t>(node) + lane] : kInvalid;
      const unsigned cmask = __ballot_sync(0xffffffffu, ch != kInvalid) & 0xFFu;
      const int nc = __popc(cmask);
      if (sp + nc > kStackCap) {
        overflow = true;
        break;
      }
      if (ch != kInvalid) stack[sp + __popc(cmask >> (lane + 1))] = ch;
      sp += nc;
      __syncwarp();
    }
    if (qn > 0) flush();
    if (overflow && lane == 0) atomicOr(a.status, kStatusStackOverflow);
    if (valid) {
      a.out_x[row] = w.G * acc_x;
      a.out_y[row] = w.G * acc_y;
      a.out_z[row] = w.G * acc_z;
    }
    __syncwarp();
  }
}

// FP32 walk over groups of targets. A node that straddles the reach of the
// group is opened down to kVjpCull sources (256 / 512 / 1024: 28.4 / 27.8 / 27.7 ms
// for the clustered box at 128^3); sources carry their position, cotangent and
// (unless every mass is equal) mass. Bound by the FMA pipe: about 48 packed FMAs
// per pair of sources, 2.4 times the forward walk's. 36.5 -> 27.8 ms at 128^3,
// 3.5 -> 2.3 ms for a 64^3 lattice, whose sources the sphere around the first
// target let through 6.7 volumes of r_cut for 2.6 of the box.
constexpr uint32_t kVjpCull = 512;
// resident blocks per SM (3 / 4 / 5: 27.7 / 27.8 / 28.3 ms)
constexpr int kVjpBlocks = 4;
constexpr int kVjpQueue = 128;
constexpr size_t kVjpAccBytes = 3 * 32 * sizeof(double);
__host__ __device__ constexpr size_t vjpQueueBytes(bool uniform) { return (uniform ? 6 : 7) * kVjpQueue * sizeof(float); }

template <bool kEpsZero, int kTerms, bool kUniform>
__global__ void __launch_bounds__(kWalkWarpsPerBlock * 32, kVjpBlocks) walkVjpGroupKernel(VjpArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  unsigned char* mine = smem + (threadIdx.x >> 5) * (vjpQueueBytes(kUniform) + kVjpAccBytes + static_cast<size_t>(a.stack_cap) * 4);
  float* q = reinterpret_cast<float*>(mine);  // x, y, z, cotangent x, y, z (, mass), kVjpQueue each
  double* acc = reinterpret_cast<double*>(mine + vjpQueueBytes(kUniform));
  uint32_t* stack = reinterpret_cast<uint32_t*>(mine + vjpQueueBytes(kUniform) + kVjpAccBytes);
  const WalkParams& w = a.wp;
  const int per = a.targets_per_group;
  const int share = 32 / per;
  const int t = lane & (per - 1);
  const int sub = lane / per;
  const float cut2 = w.cut2_f, cut_hi2 = cut2 * 1.00002f, cut_lo2 = cut2 * 0.99998f;
  const uint32_t groups = *a.group_count;
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(a.work, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= groups) break;
    const uint2 gr = a.groups[item];
    const int64_t v = static_cast<int64_t>(gr.x) + t;
    const bool valid = t < static_cast<int>(gr.y & ~kWideRun);
    uint32_t row = 0;
    double px = 0.0, py = 0.0, pz = 0.0;
    float ckx = 0.f, cky = 0.f, ckz = 0.f, mk = 1.f;
    if (valid) {
      row = a.order[v];
      const double4 u = a.src_u4[v];
      px = u.x;
      py = u.y;
      pz = u.z;
      const double4 c = a.src_c4[v];
      ckx = static_cast<float>(c.x);
      cky = static_cast<float>(c.y);
      ckz = static_cast<float>(c.z);
      if constexpr (!kUniform) mk = static_cast<float>(u.w);
    }
    const GroupFrame f = groupFrame(px, py, pz, valid);
    // the arithmetic of the queued sources: a target meets its own entry at
    // distance exactly zero, which the pair test excludes
    const float tx = static_cast<float>(px - f.cx), ty = static_cast<float>(py - f.cy), tz = static_cast<float>(pz - f.cz);
    acc[lane] = 0.0;
    acc[32 + lane] = 0.0;
    acc[64 + lane] = 0.0;
    int qn = 0, sp = 1;
    if (lane == 0) stack[0] = 0u;
    __syncwarp();

    auto flush = [&]() {
      const int quads = (qn + 4 * share - 1) / (4 * share) * share;
      for (int i = qn + lane; i < 4 * quads; i += 32) {
        q[i] = kFar;
#pragma unroll
        for (int c = 1; c < (kUniform ? 6 : 7); ++c) q[c * kVjpQueue + i] = 0.f;
      }
      __syncwarp();
      const float2 ntx = make_float2(-tx, -tx), nty = make_float2(-ty, -ty), ntz = make_float2(-tz, -tz);
      const float2 nc0 = make_float2(-ckx, -ckx), nc1 = make_float2(-cky, -cky), nc2 = make_float2(-ckz, -ckz);
      const float2 mk2 = make_float2(mk, mk);
      // two sets of sums, as in the forward walk: FP32 sums stay short
      float2 g0 = make_float2(0.f, 0.f), g1 = g0, g2 = g0, h0 = g0, h1 = g0, h2 = g0;
      auto pairStep = [&](float2 sx, float2 sy, float2 sz, float2 c0, float2 c1, float2 c2, float2 mj, float2& g0,
                          float2& g1, float2& g2) {
        const float2 dx = __fadd2_rn(sx, ntx);
        const float2 dy = __fadd2_rn(sy, nty);
        const float2 dz = __fadd2_rn(sz, ntz);
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        const bool in0 = r2.x <= cut2 && r2.x > 0.f;
        const bool in1 = r2.y <= cut2 && r2.y > 0.f;
        const float2 hh = hornerR2x2<(kTerms == 12 ? kPairPolyTerms : kTerms)>(a.pk2, r2, a.sc2, a.mone2);
        const float2 hp = hornerR2x2<kTerms>(a.dk2, r2, a.dsc2, a.mone2);
        const float2 s2 = kEpsZero ? r2 : __fadd2_rn(r2, a.eps2_2);
        const float2 rinv = make_float2(rsqrtf(s2.x), rsqrtf(s2.y));
        const float2 rinv2 = __fmul2_rn(rinv, rinv);
        const float2 rinv3 = __fmul2_rn(rinv2, rinv);
        const float2 K = __fadd2_rn(rinv3, hh);                                     // r^-3 - H/(8 r_s^3)
        const float2 Kp = __ffma2_rn(__fmul2_rn(rinv3, rinv2), a.mthree2, hp);      // -3 r^-5 - H'/(16 r_s^5)
        // m_k a_bar_j - m_j a_bar_k (equal masses: their common factor is applied to the sum)
        if constexpr (kUniform) {
          c0 = __fadd2_rn(c0, nc0);
          c1 = __fadd2_rn(c1, nc1);
          c2 = __fadd2_rn(c2, nc2);
        } else {
          c0 = __ffma2_rn(mk2, c0, __fmul2_rn(mj, nc0));
          c1 = __ffma2_rn(mk2, c1, __fmul2_rn(mj, nc1));
          c2 = __ffma2_rn(mk2, c2, __fmul2_rn(mj, nc2));
        }
        const float2 dc = __fmul2_rn(__ffma2_rn(dx, c0, __ffma2_rn(dy, c1, __fmul2_rn(dz, c2))), Kp);
        // select, not multiply: K and K' are infinite for the excluded self pair
        const float2 Ks = make_float2(in0 ? K.x : 0.f, in1 ? K.y : 0.f);
        const float2 dcs = make_float2(in0 ? dc.x : 0.f, in1 ? dc.y : 0.f);
        g0 = __ffma2_rn(Ks, c0, __ffma2_rn(dcs, dx, g0));
        g1 = __ffma2_rn(Ks, c1, __ffma2_rn(dcs, dy, g1));
        g2 = __ffma2_rn(Ks, c2, __ffma2_rn(dcs, dz, g2));
      };
      const float4* q4 = reinterpret_cast<const float4*>(q);
      constexpr int kStride = kVjpQueue / 4;
      for (int i = sub; i < quads; i += share) {
        const float4 X = q4[i], Y = q4[kStride + i], Z = q4[2 * kStride + i];
        const float4 A = q4[3 * kStride + i], B = q4[4 * kStride + i], C = q4[5 * kStride + i];
        float4 M = make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr (!kUniform) M = q4[6 * kStride + i];
        pairStep(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), make_float2(A.x, A.y),
                 make_float2(B.x, B.y), make_float2(C.x, C.y), make_float2(M.x, M.y), g0, g1, g2);
        pairStep(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), make_float2(A.z, A.w),
                 make_float2(B.z, B.w), make_float2(C.z, C.w), make_float2(M.z, M.w), h0, h1, h2);
      }
      acc[lane] += static_cast<double>((g0.x + g0.y) + (h0.x + h0.y));
      acc[32 + lane] += static_cast<double>((g1.x + g1.y) + (h1.x + h1.y));
      acc[64 + lane] += static_cast<double>((g2.x + g2.y) + (h2.x + h2.y));
      qn = 0;
      __syncwarp();
    };

    auto enqueue = [&](uint32_t begin, uint32_t count, double sx, double sy, double sz) {
      const double4* src = a.src_u4 + begin;
      uint32_t k = lane;
      double4 u = make_double4(0.0, 0.0, 0.0, 0.0);
      if (k < count) u = src[k];
      for (uint32_t chunk = 0; chunk < count; chunk += 32) {
        const double4 cur = u;
        const bool have = k < count;
        const uint32_t pos = begin + k;
        k += 32;
        if (k < count) u = src[k];
        if (qn > kVjpQueue - 32) flush();
        const float ex = static_cast<float>(cur.x - sx), ey = static_cast<float>(cur.y - sy), ez = static_cast<float>(cur.z - sz);
        const float gx = fmaxf(fabsf(ex) - f.hx, 0.f), gy = fmaxf(fabsf(ey) - f.hy, 0.f), gz = fmaxf(fabsf(ez) - f.hz, 0.f);
        const bool keep = have && fmaf(gx, gx, fmaf(gy, gy, gz * gz)) <= cut_hi2;
        const uint32_t kept = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int o = qn + __popc(kept & ((1u << lane) - 1u));
          const double4 c = a.src_c4[pos];
          q[o] = ex;
          q[kVjpQueue + o] = ey;
          q[2 * kVjpQueue + o] = ez;
          q[3 * kVjpQueue + o] = static_cast<float>(c.x);
          q[4 * kVjpQueue + o] = static_cast<float>(c.y);
          q[5 * kVjpQueue + o] = static_cast<float>(c.z);
          if constexpr (!kUniform) q[6 * kVjpQueue + o] = static_cast<float>(cur.w);
        }
        qn += __popc(kept);
        __syncwarp();
      }
    };

    bool overflow = false;
    while (sp > 0) {
      // up to 32 nodes at a time, leaving room for a depth-first descent
      const int room = a.batch_cap - sp;
      const int k = room >= 7 ? min(min(sp, 32), room / 7) : 1;
      const bool have = lane < k;
      const uint32_t node = have ? stack[sp - 1 - lane] : 0u;
      sp -= k;
      __syncwarp();
      const NodeReach r = nodeReach(a.geom, a.range, node, have, f, w);
      const bool reach = have && r.gap2 <= cut_hi2;
      const bool whole = r.rg.z == 0u || r.rg.y <= kVjpCull || r.far2 <= cut_lo2;
      const bool emit = reach && whole;
      const bool push = reach && !whole;
      sp = pushChildren(a.child, node, push, r.rg.z, 0u, stack, sp, a.stack_cap, overflow);
      if (overflow) break;
      // nodes taken whole, at each periodic image in reach
      const float rc = a.cut_f * 1.00001f + r.hf;
      const bool images = emit && (r.ax + f.hx + rc >= static_cast<float>(w.box[0]) * 0.99999f ||
                                   r.ay + f.hy + rc >= static_cast<float>(w.box[1]) * 0.99999f ||
                                   r.az + f.hz + rc >= static_cast<float>(w.box[2]) * 0.99999f);
      const unsigned moved = __ballot_sync(0xffffffffu, emit && (r.kx != 0.0 || r.ky != 0.0 || r.kz != 0.0));
      const unsigned many = __ballot_sync(0xffffffffu, images);
      for (unsigned todo = __ballot_sync(0xffffffffu, emit); todo; todo &= todo - 1u) {
        const int j = __ffs(todo) - 1;
        const uint32_t begin = __shfl_sync(0xffffffffu, r.rg.x, j), count = __shfl_sync(0xffffffffu, r.rg.y, j);
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
          nodeImages(w, a.frame, 0, __shfl_sync(0xffffffffu, r.ndx, j), h, f.cx, f.hx, jx, nx);
          nodeImages(w, a.frame, 1, __shfl_sync(0xffffffffu, r.ndy, j), h, f.cy, f.hy, jy, ny);
          nodeImages(w, a.frame, 2, __shfl_sync(0xffffffffu, r.ndz, j), h, f.cz, f.hz, jz, nz);
        }
        for (int ix = 0, iy = 0, iz = 0; iz < nz;) {
          enqueue(begin, count, f.cx + w.box[0] * (jx + ix), f.cy + w.box[1] * (jy + iy), f.cz + w.box[2] * (jz + iz));
          if (++ix == nx) {
            ix = 0;
            if (++iy == ny) {
              iy = 0;
              ++iz;
            }
          }
        }
      }
    }
    if (qn > 0) flush();
    if (overflow && lane == 0) atomicOr(a.status, kStatusStackOverflow);
    double rx = acc[lane], ry = acc[32 + lane], rz = acc[64 + lane];
    for (int off = 16; off >= per; off >>= 1) {
      rx += __shfl_xor_sync(0xffffffffu, rx, off);
      ry += __shfl_xor_sync(0xffffffffu, ry, off);
      rz += __shfl_xor_sync(0xffffffffu, rz, off);
    }
    if (valid && sub == 0) {
      const double g = kUniform ? w.G * a.uniform_mass : w.G;
      a.out_x[row] = g * rx;
      a.out_y[row] = g * ry;
      a.out_z[row] = g * rz;
    }
    __syncwarp();
  }
}

// Cotangents gathered into tree order (double4 {a_bar, 0}).
__global__ void packCotangentKernel(int64_t n, const uint32_t* __restrict__ sorted, const double* __restrict__ cx,
                                    const double* __restrict__ cy, const double* __restrict__ cz, double4* out) {
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < n;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const uint32_t s = sorted[t];
    out[t] = make_double4(cx[s], cy[s], cz[s], 0.0);
  }
}

int launchVjp(const VjpArgs& args, cudaStream_t s) {
  int dev = 0, sms = 148, per_sm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, walkVjpKernel, kWalkWarpsPerBlock * 32, 0);
  const int64_t warps_needed = (args.n + 31) / 32;
  const int64_t blocks = std::min<int64_t>(static_cast<int64_t>(sms) * std::max(per_sm, 1),
                                           (warps_needed + kWalkWarpsPerBlock - 1) / kWalkWarpsPerBlock);
  { noteLaunch(); walkVjpKernel<<<static_cast<unsigned>(std::max<int64_t>(blocks, 1)), kWalkWarpsPerBlock * 32, 0, s>>>(args); }
  return cudaGetLastError() == cudaSuccess ? 0 : CHUI_TREEPM_EDEVICE;
}

template <bool kEpsZero, int kTerms, bool kUniform>
int launchVjpGroups(const VjpArgs& args, cudaStream_t s) {
  auto kernel = walkVjpGroupKernel<kEpsZero, kTerms, kUniform>;
  const size_t smem =
      kWalkWarpsPerBlock * (vjpQueueBytes(kUniform) + kVjpAccBytes + static_cast<size_t>(args.stack_cap) * 4);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess)
    return CHUI_TREEPM_EDEVICE;
  int dev = 0, sms = 148, per_sm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWalkWarpsPerBlock * 32, smem);
  const int64_t blocks = std::min<int64_t>(static_cast<int64_t>(sms) * std::max(per_sm, 1),
                                           (args.n + kWalkWarpsPerBlock - 1) / kWalkWarpsPerBlock);
  noteLaunch();
  kernel<<<static_cast<unsigned>(std::max<int64_t>(blocks, 1)), kWalkWarpsPerBlock * 32, smem, s>>>(args);
  return cudaGetLastError() == cudaSuccess ? 0 : CHUI_TREEPM_EDEVICE;
}

}  // namespace

int walkVjpRun(Context& c, int64_t n, const double* sx, const double* sy, const double* sz, const double* m,
               double uniform_mass, const double* cx, const double* cy, const double* cz, const WalkParams& wp,
               double* gx, double* gy, double* gz, cudaStream_t s) {
  if (n == 0) return 0;
  if (ensure(c.src_cot, static_cast<size_t>(n) * sizeof(double4)) || ensure(c.work_counter, 16))
    return CHUI_TREEPM_ENOMEM;
  { noteLaunch(); packCotangentKernel<<<static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 148 * 32)), 256, 0, s>>>(
      n, c.sorted_index.as<uint32_t>(), cx, cy, cz, c.src_cot.as<double4>()); }
  cudaMemsetAsync(c.work_counter.ptr, 0, 4, s);
  VjpArgs a;
  a.n = n;
  a.order = c.target_order.as<uint32_t>();
  a.sx = sx;
  a.sy = sy;
  a.sz = sz;
  a.m = m;
  a.uniform_mass = uniform_mass;
  a.cx = cx;
  a.cy = cy;
  a.cz = cz;
  a.geom = c.node_geom.as<double4>();
  a.range = c.node_range.as<uint4>();
  a.child = c.node_child.as<uint32_t>();
  a.src_d4 = c.src_d4.as<double4>();
  a.src_c4 = c.src_cot.as<double4>();
  a.out_x = gx;
  a.out_y = gy;
  a.out_z = gz;
  a.work = c.work_counter.as<uint32_t>();
  a.status = c.status.as<uint32_t>();
  a.wp = wp;
  const double rs2 = c.rs * c.rs;
  for (int k = 0; k < kPolyMaxTerms; ++k) {
    const float h = static_cast<float>(-0.125 * static_cast<double>(c.poly.c[k]) / (rs2 * c.rs));
    const float d = static_cast<float>(-0.0625 * static_cast<double>(c.dpoly.c[k]) / (rs2 * rs2 * c.rs));
    a.pk2[k] = make_float2(h, h);
    a.dk2[k] = make_float2(d, d);
  }
  const float sc = wp.inv_4rs2_f * c.poly.scale, dsc = wp.inv_4rs2_f * c.dpoly.scale;
  a.sc2 = make_float2(sc, sc);
  a.dsc2 = make_float2(dsc, dsc);
  a.mone2 = make_float2(-1.f, -1.f);
  a.eps2_2 = make_float2(wp.eps2_f, wp.eps2_f);
  a.mthree2 = make_float2(-3.f, -3.f);
  if (c.cfg.precision != CHUI_TREEPM_MIXED) return launchVjp(a, s);
  // groups of targets; lanes per target as in the forward walk (whose pairs cost
  // less than half as much). S = 1 / 2 / 4: 64 k targets 0.88 / 0.68 / 0.67 ms,
  // 2.1 M 28.0 / 28.4 / 33.4.
  a.src_u4 = c.src_u4.as<double4>();
  WalkArgs g{};
  g.nt = n;
  g.v1 = n;
  g.n = n;
  g.order = a.order;
  g.src_u4 = a.src_u4;
  g.wp = wp;
  int per = 32;
  while (per > 8 && n / per < 6000) per >>= 1;
  if (n / 8 < 592) per = 4;
  a.targets_per_group = per;
  const double limit = std::min(1.5 * c.cutoff, 0.25 * std::min({wp.box[0], wp.box[1], wp.box[2]}));
  if (int rc = targetGroups(c, g, per, limit, &a.groups, &a.group_count, s)) return rc;
  a.work = c.work_counter.as<uint32_t>();
  a.batch_cap = kBatchStack;
  a.stack_cap = (kBatchStack + 1 + 7 * std::max<int>(static_cast<int>(c.max_depth), 1) + 7 + 3) & ~3;
  a.cut_f = static_cast<float>(c.cutoff);
  a.frame = sourceFrame(c);
  const bool eps_zero = wp.eps == 0.0;
  const bool shortp = c.poly.terms <= kPairPolyTerms && c.dpoly.terms <= 12;
#define CHUI_VJP(EPS, T) return m ? launchVjpGroups<EPS, T, false>(a, s) : launchVjpGroups<EPS, T, true>(a, s)
  if (eps_zero) {
    if (shortp) CHUI_VJP(true, 12);
    CHUI_VJP(true, kPolyMaxTerms);
  }
  if (shortp) CHUI_VJP(false, 12);
  CHUI_VJP(false, kPolyMaxTerms);
#undef CHUI_VJP
}

}  // namespace chui

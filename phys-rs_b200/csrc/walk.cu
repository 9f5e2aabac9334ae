// K6: theta-criterion walk (OctreeNode::compute_force, gravity_tree.rs:171-209).
//
// Warp-coherent, stackless union traversal over the pre-order node array.
// A warp owns 32 consecutive key-sorted targets (spatially close) and visits
// nodes in pre-order; each lane applies the reference's own criterion
// (s*s < theta*theta*d2 -> monopole at the centre of mass) and the warp
// descends into a node's children when any lane opened it (__any_sync),
// otherwise it jumps over the subtree with the skip pointer.  A lane is
// active at a node only if it opened every ancestor (tracked by `open_to`,
// the number of consecutive opened levels on the current path), so no lane
// ever double-counts a cell.  All lanes read the same node: every node load
// is one broadcast transaction.
//
// Variants:
//   F64_EXACT  reference arithmetic (no FMA, IEEE sqrt/div) and the
//              reference's nested summation: the force of an opened cell is
//              0 + sum of its children in octant order, added into the parent
//              as one term.  Per-lane accumulators per depth live in local
//              memory; closing a level adds it into the level above.
//   F64        flat f64 sum of m_j r / s^3, FMA + inv_cubed.
//   F32C       f32 pair terms on double-float relative coordinates
//              r = (hi_j - hi_i) + (lo_j - lo_i); f32 partial sums folded
//              into a (hi, lo) accumulator with two-sum every 16 nodes.
#include <algorithm>
#include <type_traits>

#include "bh.cuh"

#ifndef WALK_BRANCHY
#define WALK_BRANCHY 0
#endif
#ifndef WALK_PAIRED
#define WALK_PAIRED 1
#endif
#ifndef WALK_UNROLL
#define WALK_UNROLL 0
#endif

namespace phys {
namespace {

constexpr int kWalkBlock = 128;

__device__ __forceinline__ void warp_count(unsigned ninter, unsigned long long* counter) {
  unsigned long long v = ninter;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(counter, v);
}

template <bool kF32>
__global__ void __launch_bounds__(kWalkBlock)
walk_kernel(int q0, int n, int nnodes, const Rec32* __restrict__ w32, const Rec64* __restrict__ w64,
            const double4* __restrict__ body64, const float4* __restrict__ body_hi,
            const float4* __restrict__ body_lo, const uint32_t* __restrict__ perm,
            const TreeHeader* __restrict__ hdr, double G, double eps2, int want_force,
            double* __restrict__ ox, double* __restrict__ oy, double* __restrict__ oz,
            unsigned long long* counter, int32_t* status) {
  wait_for_previous();
  __shared__ double s2d[kWDepth + 1];
  if (!kF32) {
    for (int d = threadIdx.x; d <= kWDepth; d += blockDim.x)
      s2d[d] = d < kMaxLevels ? hdr->s2[d] : 0.0;
    __syncthreads();
  }
  const double theta2 = hdr->theta2;
  const float eps2f = (float)eps2;
  const int p = q0 + blockIdx.x * kWalkBlock + threadIdx.x;  // targets [q0, n)
  const bool valid = p < n;

  double tx = 0, ty = 0, tz = 0;
  float thx = 0, thy = 0, thz = 0, tlx = 0, tly = 0, tlz = 0;
  if (valid) {
    if (kF32) {
      const float4 h = body_hi[p], l = body_lo[p];
      thx = h.x; thy = h.y; thz = h.z;
      tlx = l.x; tly = l.y; tlz = l.z;
    } else {
      const double4 b = body64[p];
      tx = b.x; ty = b.y; tz = b.z;
    }
  }
  double ax = sum_start(eps2), ay = ax, az = ax;  // F64 sums
  float hx = 0, hy = 0, hz = 0;             // F32C compensated sums (hi)
  float lx = 0, ly = 0, lz = 0;             //                      (lo)
  float px = 0, py = 0, pz = 0;             // F32C partial since last flush
  unsigned ninter = 0;
  // open_to = number of consecutive opened levels on the current path; a
  // lane is active at a node of depth d iff open_to == d.  Lanes past the end
  // start at -1 and are never active.
  int open_to = valid ? 0 : -1;
  int node = 0;

  auto flush = [&]() {
    float s, e;
    two_sum(hx, px, s, e);
    hx = s;
    lx += e;
    two_sum(hy, py, s, e);
    hy = s;
    ly += e;
    two_sum(hz, pz, s, e);
    hz = s;
    lz += e;
    px = py = pz = 0.f;
  };

  // Visit body.  Returns the next node; always > node, so the loop ends
  // even on a malformed tree.
  auto visit = [&](int nd) -> int {
    int4 L;
    float4 A, B;
    double4 A64;
    if (kF32) {
      const Rec32* rp = w32 + nd;
      A = rp->a;
      B = rp->b;
      L = rp->l;
    } else {
      const Rec64* rp = w64 + nd;
      A64 = rp->a;
      L = rp->l;
    }
    const int d = L.w & kWDepth;
    open_to = min(open_to, d);
    const bool act = open_to == d;
    bool acc;
    if (kF32) {
      const float rx = (A.x - thx) + (B.x - tlx);
      const float ry = (A.y - thy) + (B.y - tly);
      const float rz = (A.z - thz) + (B.z - tlz);
      const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
      acc = d2 > B.w;  // one-body leaves carry -1: always an exact pair
      const bool use = act && acc && L.y != p;
#if WALK_BRANCHY
      if (use) {
        const float inv = rsqrt_sfu(d2 + eps2f);
        const float w = A.w * (inv * inv * inv);
        px = fmaf(rx, w, px);
        py = fmaf(ry, w, py);
        pz = fmaf(rz, w, pz);
      }
#else
      const float inv = rsqrt_sfu(d2 + eps2f);
      const float w = use ? A.w * (inv * inv * inv) : 0.f;
      px = fmaf(rx, w, px);
      py = fmaf(ry, w, py);
      pz = fmaf(rz, w, pz);
#endif
      ninter += use;
    } else {
      const double rx = A64.x - tx, ry = A64.y - ty, rz = A64.z - tz;
      const double d2 = fma(rx, rx, fma(ry, ry, rz * rz));
      acc = L.y >= 0 || s2d[d] < theta2 * d2;  // gravity_tree.rs:194
      const bool use = act && acc && L.y != p;
      if (use) {
        const double w = A64.w * inv_cubed(d2 + eps2);
        ax = fma(rx, w, ax);
        ay = fma(ry, w, ay);
        az = fma(rz, w, az);
      }
      ninter += use;
    }
    const bool open = act && !acc;
    int nxt = L.x;
    if (__any_sync(0xffffffffu, open)) {
      if (L.w & kWLeaf) {
        // Bucket leaf opened: exact pairs with its bodies (skipping self).
        const int q1 = L.z + (L.w >> 8);
        for (int q = L.z; q < q1; ++q) {
          const bool use = open && q != p;
          if (kF32) {
            const float4 h = body_hi[q], l = body_lo[q];
            const float rx = (h.x - thx) + (l.x - tlx);
            const float ry = (h.y - thy) + (l.y - tly);
            const float rz = (h.z - thz) + (l.z - tlz);
            const float inv = rsqrt_sfu(fmaf(rx, rx, fmaf(ry, ry, fmaf(rz, rz, eps2f))));
            const float w = use ? h.w * (inv * inv * inv) : 0.f;
            px = fmaf(rx, w, px);
            py = fmaf(ry, w, py);
            pz = fmaf(rz, w, pz);
          } else {
            const double4 b = body64[q];
            if (use) {
              const double rx = b.x - tx, ry = b.y - ty, rz = b.z - tz;
              const double w = b.w * inv_cubed(fma(rx, rx, fma(ry, ry, fma(rz, rz, eps2))));
              ax = fma(rx, w, ax);
              ay = fma(ry, w, ay);
              az = fma(rz, w, az);
            }
          }
          ninter += use;
        }
      } else {
        if (open) open_to = d + 1;
        nxt = nd + 1;
      }
    }
    return max(nxt, nd + 1);
  };

  // Sixteen visits per flush of the f32 partial sums into the compensated
  // accumulator.
#if WALK_UNROLL
  while (node < nnodes) {
#pragma unroll
    for (int k = 0; k < WALK_UNROLL; ++k) {
      if (node >= nnodes) break;
      node = visit(node);
    }
    if (kF32) flush();
  }
#else
  unsigned iter = 0;
  while (node < nnodes) {
    node = visit(node);
    if (kF32 && ((++iter & 15u) == 0u)) flush();
  }
#endif
  warp_count(ninter, counter);
  if (!valid) return;
  double fx, fy, fz;
  if (kF32) {
    flush();
    fx = (double)hx + (double)lx;
    fy = (double)hy + (double)ly;
    fz = (double)hz + (double)lz;
  } else {
    fx = ax;
    fy = ay;
    fz = az;
  }
  const double sc = want_force ? G * body64[p].w : G;
  fx *= sc;
  fy *= sc;
  fz *= sc;
  const uint32_t i = perm[p];
  ox[i] = fx;
  oy[i] = fy;
  oz[i] = fz;
  if (!isfinite(fx) || !isfinite(fy) || !isfinite(fz)) atomicOr(status, kStatNonfinite);
}

// ---------------------------------------------------------------------------
// F32C walk, two key-adjacent targets per lane (64 per warp).  The per-target
// arithmetic runs on packed f32x2 instructions (one instruction for both
// targets), which halves the issue slots of the floating-point work; node
// and body records are stored pre-duplicated (x, x, y, y, ...) so the packed
// operands come straight from the 16-byte loads.  Decisions stay per target.
// ---------------------------------------------------------------------------
constexpr int kWalk2Block = 128;

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

__global__ void __launch_bounds__(kWalk2Block)
walk2_kernel(int q64, int n, int nnodes, const Rec32x2* __restrict__ w, const Body32x2* __restrict__ body2,
             const double4* __restrict__ body64, const uint32_t* __restrict__ perm, double G,
             double eps2, int want_force, double* __restrict__ ox, double* __restrict__ oy,
             double* __restrict__ oz, unsigned long long* counter, int32_t* status) {
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  // targets [64 q64, n), 64 per warp (a multiple of 64: pa even)
  const int base = (q64 + blockIdx.x * (kWalk2Block / 32) + (threadIdx.x >> 5)) * 64;
  const int pa = base + 2 * lane, pb = pa + 1;
  const bool va = pa < n, vb = pb < n;
  float2 nhx, nhy, nhz, nlx, nly, nlz;  // negated target coordinates (a, b)
  {
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 a0 = va ? body2[pa].q0 : z4, a1 = va ? body2[pa].q1 : z4;
    const float4 a2 = va ? body2[pa].q2 : z4, a3 = va ? body2[pa].q3 : z4;
    const float4 b0 = vb ? body2[pb].q0 : z4, b1 = vb ? body2[pb].q1 : z4;
    const float4 b2 = vb ? body2[pb].q2 : z4, b3 = vb ? body2[pb].q3 : z4;
    nhx = make_float2(-a0.x, -b0.x);
    nhy = make_float2(-a0.z, -b0.z);
    nhz = make_float2(-a1.x, -b1.x);
    nlx = make_float2(-a2.x, -b2.x);
    nly = make_float2(-a2.z, -b2.z);
    nlz = make_float2(-a3.x, -b3.x);
  }
  const float eps2f = (float)eps2;
  const float2 e2 = make_float2(eps2f, eps2f);
  float2 px = make_float2(0.f, 0.f), py = px, pz = px;  // partial sums since last flush
  float hxa = 0, hya = 0, hza = 0, lxa = 0, lya = 0, lza = 0;  // compensated, target a
  float hxb = 0, hyb = 0, hzb = 0, lxb = 0, lyb = 0, lzb = 0;  // compensated, target b
  int oa = va ? 0 : -1, ob = vb ? 0 : -1;  // opened levels on the current path
  unsigned ninter = 0;

  auto flush = [&]() {
    float s, e;
    two_sum(hxa, px.x, s, e); hxa = s; lxa += e;
    two_sum(hya, py.x, s, e); hya = s; lya += e;
    two_sum(hza, pz.x, s, e); hza = s; lza += e;
    two_sum(hxb, px.y, s, e); hxb = s; lxb += e;
    two_sum(hyb, py.y, s, e); hyb = s; lyb += e;
    two_sum(hzb, pz.y, s, e); hzb = s; lzb += e;
    px = py = pz = make_float2(0.f, 0.f);
  };
  // Packed separation from a paired record (q0..q3) to both targets.
  auto sep = [&](float4 q0, float4 q1, float4 q2, float4 q3, float2& rx, float2& ry,
                 float2& rz) {
    rx = __fadd2_rn(__fadd2_rn(lo2(q0), nhx), __fadd2_rn(lo2(q2), nlx));
    ry = __fadd2_rn(__fadd2_rn(hi2(q0), nhy), __fadd2_rn(hi2(q2), nly));
    rz = __fadd2_rn(__fadd2_rn(lo2(q1), nhz), __fadd2_rn(lo2(q3), nlz));
  };
  auto accum = [&](float2 rx, float2 ry, float2 rz, float2 r2, float2 m2, bool ua, bool ub) {
    const float2 inv = make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
    float2 wg = __fmul2_rn(m2, __fmul2_rn(__fmul2_rn(inv, inv), inv));
    wg.x = ua ? wg.x : 0.f;
    wg.y = ub ? wg.y : 0.f;
    px = __ffma2_rn(rx, wg, px);
    py = __ffma2_rn(ry, wg, py);
    pz = __ffma2_rn(rz, wg, pz);
    ninter += (unsigned)ua + (unsigned)ub;
  };

  auto visit = [&](int nd) -> int {
    const Rec32x2* rp = w + nd;
    const float4 q0 = rp->q0, q1 = rp->q1, q2 = rp->q2, q3 = rp->q3;
    const int4 L = rp->l;
    const int d = L.w & kWDepth;
    oa = min(oa, d);
    ob = min(ob, d);
    const bool acta = oa == d, actb = ob == d;
    float2 rx, ry, rz;
    sep(q0, q1, q2, q3, rx, ry, rz);
    const float2 d2 = __ffma2_rn(rx, rx, __ffma2_rn(ry, ry, __fmul2_rn(rz, rz)));
    const bool acca = d2.x > q3.z, accb = d2.y > q3.w;  // -1 for one-body leaves
    accum(rx, ry, rz, __fadd2_rn(d2, e2), hi2(q1), acta && acca && L.y != pa,
          actb && accb && L.y != pb);
    const bool opa = acta && !acca, opb = actb && !accb;
    int nxt = L.x;
    if (__any_sync(0xffffffffu, opa || opb)) {
      if (L.w & kWLeaf) {
        const int qe = L.z + (L.w >> 8);
        for (int q = L.z; q < qe; ++q) {
          const Body32x2* bp = body2 + q;
          const float4 b0 = bp->q0, b1 = bp->q1, b2 = bp->q2, b3 = bp->q3;
          float2 bx, by, bz;
          sep(b0, b1, b2, b3, bx, by, bz);
          const float2 r2 = __ffma2_rn(bx, bx, __ffma2_rn(by, by, __ffma2_rn(bz, bz, e2)));
          accum(bx, by, bz, r2, hi2(b1), opa && q != pa, opb && q != pb);
        }
      } else {
        if (opa) oa = d + 1;
        if (opb) ob = d + 1;
        nxt = nd + 1;
      }
    }
    return max(nxt, nd + 1);
  };

  int node = 0;
  unsigned iter = 0;
  while (node < nnodes) {
    node = visit(node);
    if ((++iter & 15u) == 0u) flush();
  }
  flush();
  warp_count(ninter, counter);
  auto out = [&](int pp, float hx, float hy, float hz, float lx, float ly, float lz) {
    double fx = (double)hx + (double)lx, fy = (double)hy + (double)ly,
           fz = (double)hz + (double)lz;
    const double sc = want_force ? G * body64[pp].w : G;
    fx *= sc;
    fy *= sc;
    fz *= sc;
    const uint32_t i = perm[pp];
    ox[i] = fx;
    oy[i] = fy;
    oz[i] = fz;
    if (!isfinite(fx) || !isfinite(fy) || !isfinite(fz)) atomicOr(status, kStatNonfinite);
  };
  if (va) out(pa, hxa, hya, hza, lxa, lya, lza);
  if (vb) out(pb, hxb, hyb, hzb, lxb, lyb, lzb);
}

// ---------------------------------------------------------------------------
// F64_EXACT walk (leaf capacity 1).
//
// A warp walks for its 32 targets together.  The traversal only decides: a
// node that some target takes (a monopole or a stored body) becomes an entry
// of the warp's queue in shared memory, in pre-order, with the mask of those
// lanes and the levels that the open partial sums close to and open to before
// it.  A full queue is evaluated kXU entries at a time: every lane forms the
// weights (exact_scale, independent chains), then the terms are added in
// order, 0 for the lanes outside the mask.  Levels are opened and closed by
// the warp's path for all lanes at once: a lane that did not open a cell has
// +0 in its level, and adding that changes nothing.  The deepest level's sum
// is in registers, the ones around it in local memory; closing a level adds it
// to the one above, as the reference's nested sums do.
//
// The traversal works on 32 cells at a time, a cell per lane: the children of
// up to four opened cells of one depth.  Each is first tested against the box
// of the warp's targets, nearest and farthest point; the f32 operations are
// the ones of a single target's test and monotone, so a cell that all targets
// take or all open is found without looking at them.  Only the others (one in
// six) are tested per target.
//
// Opening is decided in f32 on coordinates relative to the root cube: each
// coordinate is within 2^-25 of its value, their difference within 2^-23, so
// the distance is within 2.1e-7 of the half size and the lane's choice is the
// f64 one outside a band of 4e-7 (and 1e-6 relative) around side / theta;
// inside it, and for a centre of mass outside the cube (masses of both signs;
// its f32 position is NaN), the warp takes the reference's f64 test.
//
// Few targets would leave most of the chip idle behind the longest walk, so
// up to 131072 of them are split: the children of the cells of more than a
// 16th to a 5th of the bodies become tasks of their own, each leaving its
// cell's contribution to each target in `part`; exact_combine_kernel walks
// the cells above and sums them with the reference's nesting.  Warps take
// pairs of a task and 32 targets from a queue, large tasks first: the longest
// pair (halo targets, spread out, against a dense cell) takes 0.27 ms at
// 10 000 bodies and n/8, so it must not start last.  Split against whole
// walks: 0.29 / 0.96 ms at 10 000 bodies, 0.58 / 1.21 at 32768, 1.05 / 1.54 at
// 65536, 1.57 / 1.89 at 100 000, 4.8 / 4.9 at 300 000 (and a block per pair in
// grid order: 0.32 at 10 000, 0.86 at 32768, 1.27 at 65536).  Masses of both
// signs: 0.20 ms at 10 000, 1.7 at 100 000, 13.9 at 2^20 (a node per step 1.19,
// 2.5 and 18.0; every cell in f64 with the library's weights 0.26, 3.25, 24.8).
//
// Bound by the terms: 3300 entries a warp at 300 000 bodies (2100 per target),
// 38 FP64 instructions and about as many others each, at 47 % of the FP64
// pipe; without them the traversal takes 1.1 of 5.0 ms.  Two entries at a time
// and 24 warps an SM do best on a full chip (four: 17.3 ms at 2^20), four with
// 16 warps when the tasks' tails show (0.32 against 0.34 ms at 10 000, in grid
// order).  One walk per target, a node per step and its term evaluated in place, took 19.8
// ms at 2^20 bodies against 15.5; split, a node per step, 0.44 at 10 000.
// ---------------------------------------------------------------------------
constexpr unsigned kFull = 0xffffffffu;
constexpr int kXQ = 32;  // queue entries per warp
constexpr float kXBand = 4e-7f;

// Whether every pair of an evaluation is in exact_scale's range: masses within
// [2^-190, 2^240 / n] or 0, bodies within 2^98, softening.  With masses of one
// sign the sums over cells and the centres of mass are then in range as well;
// with both (kSigns) record_in_range looks at the queued ones, in a kernel of
// its own (the look, or only the flag for it, costs masses of one sign 2 to 7 %).
__device__ __forceinline__ bool record_in_range(double4 r) {
  return scale_pos_ok(r.x, r.y, r.z) && scale_mass_ok(r.w);
}
__device__ __forceinline__ bool walk_in_range(const TreeHeader* hdr, int64_t n, double eps2) {
  const double c = fmax(fmax(fabs(hdr->center[0]), fabs(hdr->center[1])), fabs(hdr->center[2]));
  return scale_eps2_ok(eps2) && hdr->min_abs >= 0x1p-190 &&
         hdr->max_abs * (double)n < 0x1p240 && c + 2.0 * hdr->half < 0x1p98;
}

struct ExactTarget {
  double x, y, z, gm;
};

// Term of compute_gravity_pair (gravity_tree.rs:218-234): its weight, and
// the separation.
template <bool kFast>
__device__ __forceinline__ double exact_weight(const ExactTarget& t, double4 s, double eps2,
                                               double& rx, double& ry, double& rz) {
  rx = xsub(s.x, t.x), ry = xsub(s.y, t.y), rz = xsub(s.z, t.z);
  const double s2 = xadd(xlen2(rx, ry, rz), eps2), a = xmul(t.gm, s.w);
  return kFast ? exact_scale(a, s2) : exact_scale_ieee(a, s2);
}

// The nested sums of one target: the deepest level with a term in registers,
// the levels around it in an array of the caller's (one struct with the array
// inside would be written back to local memory after every term).
struct NestedSum {
  double x, y, z;
  int d;
  __device__ __forceinline__ void init(int depth) {
    x = y = z = 0.0;
    d = depth;
  }
  // close the levels below m
  __device__ __forceinline__ void close_to(int m, double (*st)[3]) {
#pragma unroll 1
    while (d > m) {
      --d;
      x = xadd(st[d][0], x);
      y = xadd(st[d][1], y);
      z = xadd(st[d][2], z);
    }
  }
  // open levels up to depth, at 0
  __device__ __forceinline__ void open_to(int depth, double (*st)[3]) {
#pragma unroll 1
    while (d < depth) {
      st[d][0] = x;
      st[d][1] = y;
      st[d][2] = z;
      x = y = z = 0.0;
      ++d;
    }
  }
  __device__ __forceinline__ void add(double tx, double ty, double tz) {
    x = xadd(x, tx);
    y = xadd(y, ty);
    z = xadd(z, tz);
  }
};

// The reference's opening test in f64 (gravity_tree.rs:192-194).
__device__ __forceinline__ bool exact_open(double4 s, const ExactTarget& t, double s2,
                                           double theta2) {
  const double rx = xsub(s.x, t.x), ry = xsub(s.y, t.y), rz = xsub(s.z, t.z);
  return !(s2 < xmul(theta2, xlen2(rx, ry, rz)));
}

__device__ __forceinline__ ExactTarget exact_target(const double4* body64, int64_t p, bool valid,
                                                    double G) {
  const double4 b = valid ? body64[p] : make_double4(0.0, 0.0, 0.0, 0.0);
  return ExactTarget{b.x, b.y, b.z, xmul(G, b.w)};
}

// Force -> output of one target (a = F / m unless the force is wanted).
__device__ __forceinline__ void exact_store(double fx, double fy, double fz, double mi,
                                            uint32_t i, int want_force, double* ox, double* oy,
                                            double* oz, int32_t* status) {
  if (!want_force) {  // a = F / m (integrators.rs:115)
    fx = xdiv(fx, mi);
    fy = xdiv(fy, mi);
    fz = xdiv(fz, mi);
  }
  ox[i] = fx;
  oy[i] = fy;
  oz[i] = fz;
  if (!isfinite(fx) || !isfinite(fy) || !isfinite(fz)) atomicOr(status, kStatNonfinite);
}

constexpr int kXWarps = 4;  // warps per block
constexpr int kXTargets = 32 * kXWarps;

template <bool kWhole, bool kSigns>
__global__ void __launch_bounds__(32 * kXWarps, kWhole ? 6 : 4)
walk_exact_kernel(int64_t q0, int64_t n, int64_t nbody, int nnodes, const float4* __restrict__ wx,
                  const Kids* __restrict__ kids, const double4* __restrict__ rec64,
                  const double4* __restrict__ body64, const uint32_t* __restrict__ perm,
                  const TreeHeader* __restrict__ hdr, TopTree top, double G, double eps2,
                  int want_force, double* __restrict__ part, double* __restrict__ ox,
                  double* __restrict__ oy, double* __restrict__ oz, unsigned long long* counter,
                  int32_t* status) {
  wait_for_previous();
  constexpr int kXU = kWhole ? 2 : 4;  // entries evaluated together
  static_assert(kXQ % kXU == 0, "whole rounds");
  __shared__ double s2d[kMaxLevels];
  __shared__ float2 band[kMaxLevels];
  __shared__ __align__(16) double4 srec[kXWarps][kXQ];
  __shared__ int qnode[kXWarps][kXQ];
  __shared__ unsigned qmask[kXWarps][kXQ];    // lanes that take it
  __shared__ unsigned qlevels[kXWarps][kXQ];  // 0: those of the entry before
  const int ntask = kWhole ? 1 : top.ntask;
  const double theta2 = hdr->theta2, half = hdr->half;
  for (int d = threadIdx.x; d < kMaxLevels; d += blockDim.x) {
    s2d[d] = hdr->s2[d];
    // side / theta in units of the half size, and the band around it
    const double r = sqrt(hdr->s2[d] / theta2) / half;
    const double lo = fmax(r - (double)kXBand, 0.0), hi = r + (double)kXBand;
    band[d] = make_float2((float)(lo * lo * (1.0 - 1e-6)), (float)(hi * hi * (1.0 + 1e-6)));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned bit = 1u << lane;
  unsigned ninter = 0;
  // a warp's work: one task for 32 of the targets [q0, n)
  const int nrun = (int)((n - q0 + 31) / 32);
  for (;;) {
    int task = 0, run = blockIdx.x * kXWarps + wid;
    if (!kWhole) {
      int it = 0;
      if (lane == 0) it = atomicAdd(top.queue, 1);
      it = __shfl_sync(kFull, it, 0);
      task = it / nrun;
      run = it - task * nrun;
    }
    if (run >= nrun || task >= ntask) break;
    if (!kWhole) task = top.order[task];
    const int root = kWhole ? 0 : top.task[task];
    const int64_t p = q0 + run * 32 + lane;
    const bool valid = p < n;
    const int p0 = (int)(p - lane);
    const ExactTarget t = exact_target(body64, p, valid, G);
    const bool fast = __all_sync(kFull, scale_mass_ok(t.gm)) && walk_in_range(hdr, nbody, eps2);
    const double ih = 1.0 / half;
    const float fx = (float)((t.x - hdr->center[0]) * ih), fy = (float)((t.y - hdr->center[1]) * ih),
                fz = (float)((t.z - hdr->center[2]) * ih);
    const bool coarse = __all_sync(kFull, !valid || (isfinite(fx) && isfinite(fy) && isfinite(fz)));
    // the box around the warp's targets
    float bl[3] = {valid ? fx : INFINITY, valid ? fy : INFINITY, valid ? fz : INFINITY};
    float bh[3] = {valid ? fx : -INFINITY, valid ? fy : -INFINITY, valid ? fz : -INFINITY};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        bl[k] = fminf(bl[k], __shfl_xor_sync(kFull, bl[k], o));
        bh[k] = fmaxf(bh[k], __shfl_xor_sync(kFull, bh[k], o));
      }
    }

    NestedSum sum;
    double outer[kMaxLevels + 1][3];
    int cnt = 0;
    unsigned* const qm = qmask[wid];
    unsigned* const ql = qlevels[wid];
    int* const qn = qnode[wid];
    double4* const sr = srec[wid];
    // add the queue's terms: bit k of `on`: entry k is the lane's, of `ev`: it
    // changes levels
    auto terms = [&](auto quick, unsigned on, unsigned ev) {
      constexpr bool kQuick = decltype(quick)::value;
#pragma unroll 1
      for (int k0 = 0; k0 < cnt; k0 += kXU) {
        double rx[kXU], ry[kXU], rz[kXU], w[kXU];
#pragma unroll
        for (int u = 0; u < kXU; ++u)
          w[u] = exact_weight<kQuick>(t, sr[k0 + u], eps2, rx[u], ry[u], rz[u]);
#pragma unroll
        for (int u = 0; u < kXU; ++u) {
          if (ev >> u & 1) {
            const unsigned l = ql[k0 + u];
            sum.close_to((int)(l & 0xffff), outer);
            sum.open_to((int)(l >> 17), outer);
          }
          // a lane outside the mask adds 0, which changes no sum
          const bool mine = on >> u & 1;
          const double wu = mine ? w[u] : 0.0;
          if (!kQuick && !mine) rx[u] = ry[u] = rz[u] = 0.0;  // may be infinite
          sum.add(xmul(rx[u], wu), xmul(ry[u], wu), xmul(rz[u], wu));
        }
        on >>= kXU;
        ev >>= kXU;
      }
    };
    auto drain = [&]() {
      __syncwarp();
      unsigned on = lane < cnt ? qm[lane] : 0;
      const unsigned ev = __ballot_sync(kFull, lane < cnt && ql[lane] != 0);
      sr[lane] = rec64[qn[min(lane, cnt - 1)]];
      // transpose: from a lane mask per entry to an entry mask per lane
#pragma unroll
      for (int j = 16; j > 0; j >>= 1) {
        const unsigned m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu
                                       : j == 2 ? 0x33333333u : 0x55555555u;
        const unsigned y = __shfl_xor_sync(kFull, on, j);
        on = lane & j ? (on & ~m) | (y >> j & m) : (on & m) | (y & m) << j;
      }
      __syncwarp();
      if (fast && (!kSigns || __all_sync(kFull, record_in_range(sr[lane]))))
        terms(std::true_type{}, on, ev);
      else
        terms(std::false_type{}, on, ev);
      __syncwarp();
      cnt = 0;
    };

    // the task's cells above were all opened by the lane?
    const int base = __float_as_int(wx[root].w) & kMetaDepth;
    bool in = valid;
    if (!kWhole && valid) {
      for (int k = root, d = base - 1; d >= 0; --d) {
        k = top.parent[k];
        in = in && (k == 0 || (__float_as_int(wx[k].w) & kMetaGate)) &&
             exact_open(rec64[k], t, s2d[d], theta2);
      }
    }
    const unsigned start = __ballot_sync(kFull, in);
    sum.init(base);
    // A frame per depth: in lanes 8g..8g+7 the children of the g-th of up to
    // four opened cells of the frame above (set `above`), with the targets that
    // take (tk) and open (op) each.  The walk goes through a group of lanes
    // [pos, end) at a time; the other groups wait until it comes to their cell.
    int4 frame[kMaxLevels];     // cell, tk, op, pos | end << 8
    unsigned above[kMaxLevels + 1];
    int d = base, cn = lane == 0 ? root : -1, pos = 0, end = 8;
    unsigned tk, op, act = start;
    auto classify = [&]() {
      tk = op = 0;
      bool mixed = false;
      float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
      const float2 bd = band[d];
      if (cn >= 0) {
        A = __ldg(&wx[cn]);
        const int meta = __float_as_int(A.w);
        if ((meta & kMetaGate) || cn == 0) {
          if (meta & kMetaLeaf) {  // every target but the body itself
            const unsigned self = (unsigned)(__float_as_int(A.x) - p0);
            tk = self < 32 ? act & ~(1u << self) : act;
          } else {
            const float nx = fmaxf(fmaxf(bl[0] - A.x, A.x - bh[0]), 0.f),
                        ny = fmaxf(fmaxf(bl[1] - A.y, A.y - bh[1]), 0.f),
                        nz = fmaxf(fmaxf(bl[2] - A.z, A.z - bh[2]), 0.f);
            const float mx = fmaxf(A.x - bl[0], bh[0] - A.x), my = fmaxf(A.y - bl[1], bh[1] - A.y),
                        mz = fmaxf(A.z - bl[2], bh[2] - A.z);
            const float near2 = fmaf(nx, nx, fmaf(ny, ny, nz * nz)),
                        far2 = fmaf(mx, mx, fmaf(my, my, mz * mz));
            if (coarse && cn != 0 && near2 > bd.y && far2 >= near2)
              tk = act;
            else if (coarse && cn != 0 && far2 < bd.x)
              op = act;
            else
              mixed = true;
          }
        }
      }
#pragma unroll 1
      for (unsigned mm = __ballot_sync(kFull, mixed); mm; mm &= mm - 1) {
        const int j = __ffs(mm) - 1;
        const float rx = __shfl_sync(kFull, A.x, j) - fx, ry = __shfl_sync(kFull, A.y, j) - fy,
                    rz = __shfl_sync(kFull, A.z, j) - fz;
        const unsigned a = __shfl_sync(kFull, act, j);
        const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
        bool open = d2 < bd.x;
        if (__any_sync(kFull, (a & bit) && !(coarse && (d2 < bd.x || d2 > bd.y))))
          open = exact_open(rec64[__shfl_sync(kFull, cn, j)], t, s2d[d], theta2);
        const unsigned o = __ballot_sync(kFull, open) & a;
        if (lane == j) {
          op = o;
          tk = a & ~o;
        }
      }
      frame[d] = make_int4(cn, (int)tk, (int)op, 0);
      above[d + 1] = 0;
    };
    if (start) classify();
    // low: the least depth of the path since the last entry
    int low = base, steps = 0;
    while (start) {
      const unsigned group = (unsigned)((1ull << end) - (1ull << pos));
      const unsigned all_op = __ballot_sync(kFull, op != 0);
      const unsigned opens = all_op & group, takes = __ballot_sync(kFull, tk != 0) & group;
      const unsigned put = opens ? takes & (opens ^ (opens - 1)) : takes;  // up to the first opened
      low = min(low, d);
      if (put) {
        if (put & bit) {
          const int r = __popc(put & (bit - 1));
          qn[cnt + r] = cn;
          // levels: the one the open sums close to, then the entry's own
          qm[cnt + r] = tk;
          ql[cnt + r] = r == 0 ? (unsigned)(low | 0x10000 | d << 17) : 0u;
          ninter += __popc(tk);
        }
        low = d;
        cnt += __popc(put);
        if (cnt > kXQ - 8) drain();
      }
      if (!opens) {  // group done: on with the frame above
        if (d == base) break;
        --d;
        const int4 f = frame[d];
        cn = f.x;
        tk = (unsigned)f.y;
        op = (unsigned)f.z;
        pos = f.w & 0xff;
        end = f.w >> 8;
        continue;
      }
      const int j = __ffs(opens) - 1;
      frame[d].w = (j + 1) | end << 8;
      unsigned done = above[d + 1];
      if (done >> j & 1) {  // its children are in the frame below already
        pos = 8 * __popc(done & ((1u << j) - 1));
        ++d;
        const int4 f = frame[d];
        cn = f.x;
        tk = (unsigned)f.y;
        op = (unsigned)f.z;
      } else {  // the children of this and of the next opened cells, four at most
        if (d + 1 >= kMaxLevels || ++steps > nnodes) {  // malformed tree: report, never spin
          if (lane == 0) atomicOr(status, kStatOverflow);
          break;
        }
        const unsigned s0 = all_op & ~((1u << j) - 1), s1 = s0 & (s0 - 1), s2 = s1 & (s1 - 1),
                       s3 = s2 & (s2 - 1);
        done = s0 & ~(s3 & (s3 - 1));
        const unsigned mine = lane < 16 ? (lane < 8 ? s0 : s1) : (lane < 24 ? s2 : s3);
        const int from = __ffs(mine) - 1;
        const int cell = __shfl_sync(kFull, cn, from & 31);
        act = __shfl_sync(kFull, op, from & 31);
        cn = -1;
        if (mine) cn = __ldg(&kids[cell].id[lane & 7]);
        if (cn <= cell || cn >= nnodes) cn = -1;
        above[d + 1] = done;
        ++d;
        classify();
        pos = 0;
      }
      end = pos + 8;
    }
    if (cnt) drain();
    sum.close_to(base, outer);
    if (kWhole) {
      if (valid)
        exact_store(sum.x, sum.y, sum.z, body64[p].w, perm[p], want_force, ox, oy, oz, status);
    } else if (in) {
      double* o = part + ((size_t)task * (size_t)(n - q0) + (size_t)(p - q0)) * 3;
      o[0] = sum.x;
      o[1] = sum.y;
      o[2] = sum.z;
    }
    if (kWhole) break;
  }
  warp_count(ninter, counter);
}

// A target's force from its tasks' contributions: the walk over the upper
// cells, nested as in compute_force (gravity_tree.rs:194-205).
constexpr int kStage = 64;  // top nodes in shared memory at a time
constexpr int kAhead = 8;

__global__ void __launch_bounds__(kStage)
exact_combine_kernel(int64_t q0, int64_t n, const float4* __restrict__ wx,
                     const double4* __restrict__ rec64, const double4* __restrict__ body64,
                     const uint32_t* __restrict__ perm, const TreeHeader* __restrict__ hdr,
                     TopTree top, double G, double eps2, int want_force,
                     const double* __restrict__ part, double* __restrict__ ox,
                     double* __restrict__ oy, double* __restrict__ oz,
                     unsigned long long* counter, int32_t* status) {
  wait_for_previous();
  __shared__ int4 se[kStage];
  __shared__ __align__(16) double4 sr[kStage];
  const int64_t p = q0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = p < n;
  const ExactTarget t = exact_target(body64, valid ? p : q0, true, G);
  const double theta2 = hdr->theta2;
  const int ntop = top.ntop;
  unsigned ninter = 0;
  NestedSum sum;
  double outer[kMaxLevels + 1][3];
  sum.init(0);
  int open_to = 0;
  for (int i0 = 0; i0 < ntop; i0 += kStage) {
    __syncthreads();
    const int i = i0 + (int)threadIdx.x;
    const int4 e = i < ntop ? top.top[i] : make_int4(0, -1, 0, 0);
    const bool gate = e.x == 0 || (__float_as_int(wx[e.x].w) & kMetaGate);
    se[threadIdx.x] = make_int4(e.x, e.y, e.z, gate);
    sr[threadIdx.x] = rec64[e.x];
    __syncthreads();
    for (int k0 = 0; k0 < min(kStage, ntop - i0); k0 += kAhead) {
      // the contributions of several tasks are read together
      double v[kAhead][3];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const int task = se[k0 + k].y;
        const double* q = part + ((size_t)max(task, 0) * (size_t)(n - q0) + (size_t)(p - q0)) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[k][c] = task >= 0 && valid ? q[c] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        if (i0 + k0 + k >= ntop) break;
        const int4 e = se[k0 + k];
        const int d = e.z;
        open_to = min(open_to, d);
        sum.close_to(d, outer);
        const bool act = open_to == d && e.w;
        if (e.y >= 0) {
          sum.open_to(d, outer);
          if (act && valid) sum.add(v[k][0], v[k][1], v[k][2]);
        } else {
          const double4 r = sr[k0 + k];
          const bool open = act && exact_open(r, t, hdr->s2[d], theta2);
          if (open) open_to = d + 1;
          if (act && !open) {  // taken as a monopole
            double rx, ry, rz;
            const double w = exact_weight<false>(t, r, eps2, rx, ry, rz);
            sum.open_to(d, outer);
            sum.add(xmul(rx, w), xmul(ry, w), xmul(rz, w));
            ninter += valid;
          }
        }
      }
    }
  }
  sum.close_to(0, outer);
  warp_count(ninter, counter);
  if (!valid) return;
  exact_store(sum.x, sum.y, sum.z, body64[p].w, perm[p], want_force, ox, oy, oz, status);
}

}  // namespace

int exact_walk_tasks(const phys_ctx* c, int64_t n) {
  int64_t q0 = 0, q1 = n;
  target_range(c, n, q0, q1);
  const int64_t nt = q1 - q0;
  // `part` holds 24 bytes per task that the tree has and target: at most 100 MB,
  // 200 MB for more than 65536 targets (64 tasks)
  if (nt <= 0 || nt > 131072) return 0;
  return (int)std::max<int64_t>(64, min64(512, (int64_t(1) << 22) / nt));
}

int bh_walk(phys_ctx* c, const phys_params* p, const BhTree& t, bool want_force, double* ox,
            double* oy, double* oz) {
  const int64_t n = t.n;
  const double eps2 = p->eps * p->eps;
  // targets: sorted positions [q0, q1), all or the share
  int64_t q0 = 0, q1 = n;
  target_range(c, n, q0, q1);
  const int64_t nt = q1 > q0 ? q1 - q0 : 0;
  const int grid = (int)ceil_div(nt > 0 ? nt : 1, kWalkBlock);
  PHYS_CUDA(c, cudaMemsetAsync(c->d_counter, 0, 2 * sizeof(unsigned long long), c->stream));
  PHYS_CUDA(c, cudaEventRecord(c->ev[6], c->stream));
  if (p->flags & PHYS_FLAG_GROUP_WALK) {
    PHYS_TRY(bh_group_walk(c, p, t, want_force, ox, oy, oz));
  } else if (p->precision == PHYS_F64_EXACT) {
    const int tasks = t.top.ntask;
    const int xgrid = (int)ceil_div(nt > 0 ? nt : 1, kXTargets);
    if (tasks > 0) {
      double* part = nullptr;
      PHYS_TRY(ws_alloc(c, WS_DIRECT_PART, 3 * nt * tasks, &part));
      auto kernel = t.signs ? walk_exact_kernel<false, true> : walk_exact_kernel<false, false>;
      PHYS_LAUNCH(c, kernel, (int)min64(148 * 4, (int64_t)xgrid * tasks),
                  32 * kXWarps, 0, q0, q1, n,
                  (int)t.nnodes, t.wx, t.kids, t.rec64, t.body64, t.perm, t.hdr, t.top, p->G, eps2,
                  (int)want_force, part, ox, oy, oz, c->d_counter, c->d_status);
      PHYS_LAUNCH(c, exact_combine_kernel, (int)ceil_div(nt > 0 ? nt : 1, kStage), kStage, 0, q0, q1, t.wx, t.rec64,
                  t.body64, t.perm, t.hdr, t.top, p->G, eps2, want_force, part, ox, oy, oz,
                  c->d_counter, c->d_status);
    } else {
      auto kernel = t.signs ? walk_exact_kernel<true, true> : walk_exact_kernel<true, false>;
      PHYS_LAUNCH(c, kernel, xgrid, 32 * kXWarps, 0, q0, q1, n, (int)t.nnodes, t.wx,
                  t.kids, t.rec64, t.body64, t.perm, t.hdr, t.top, p->G, eps2, (int)want_force,
                  (double*)nullptr, ox, oy, oz, c->d_counter, c->d_status);
    }
  } else if (p->precision == PHYS_F64) {
    PHYS_LAUNCH(c, walk_kernel<false>, grid, kWalkBlock, 0, (int)q0, (int)q1, (int)t.nnodes, t.w32, t.w64,
                t.body64, t.body_hi, t.body_lo, t.perm, t.hdr, p->G, eps2, (int)want_force, ox, oy,
                oz, c->d_counter, c->d_status);
  } else if (WALK_PAIRED && t.w32x2) {
    if (q0 % 64) return fail(c, PHYS_ERR_ARG, "per-body walk share must start at a multiple of 64");
    const int grid2 = (int)ceil_div(nt > 0 ? nt : 1, 64 * (kWalk2Block / 32));
    PHYS_LAUNCH(c, walk2_kernel, grid2, kWalk2Block, 0, (int)(q0 / 64), (int)q1, (int)t.nnodes, t.w32x2, t.body2,
                t.body64, t.perm, p->G, eps2, (int)want_force, ox, oy, oz, c->d_counter,
                c->d_status);
  } else {
    PHYS_LAUNCH(c, walk_kernel<true>, grid, kWalkBlock, 0, (int)q0, (int)q1, (int)t.nnodes, t.w32, t.w64,
                t.body64, t.body_hi, t.body_lo, t.perm, t.hdr, p->G, eps2, (int)want_force, ox, oy,
                oz, c->d_counter, c->d_status);
  }
  PHYS_CUDA(c, cudaEventRecord(c->ev[7], c->stream));
  return PHYS_OK;
}

}  // namespace phys

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
  double ax = 0, ay = 0, az = 0;            // F64 sums
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
// The traversal only decides: a node that some lane takes (a monopole or a
// stored body) becomes an entry of the warp's queue in shared memory, with
// the mask of those lanes, the level that the open partial sums close to
// before it and its own level.  A full queue is evaluated kXU entries at a
// time: every lane forms the weights (exact_scale, independent chains, the
// node's record read once for the warp), then the terms are added in order,
// the masked lanes' only.  Levels are opened and closed by the warp's path
// for all lanes at once: a lane that did not open a cell has +0 in its level,
// and adding that changes nothing.  The deepest level's sum is in registers,
// the ones around it in local memory; closing a level adds it to the one
// above, as the reference's nested sums do.
//
// Opening is decided in f32 on coordinates relative to the root cube: each
// coordinate is within 2^-25 of its value, their difference within 2^-23, so
// the distance is within 2.1e-7 of the half size and the lane's choice is the
// f64 one outside a band of 4e-7 (and 1e-6 relative) around side / theta;
// inside it, or when the masses do not all have one sign (a centre of mass
// may then lie outside the cube), the warp takes the reference's f64 test.
//
// Few targets would leave most of the chip idle behind the longest walk, so
// the children of the cells of more than n/8 bodies become tasks of their own
// (grid.y; n/16 to n/64 make more tasks than they save walking: 10 000 bodies
// 0.44 ms against 0.45, 0.55 and 0.68), each leaving its cell's contribution to each target in `part`;
// exact_combine_kernel walks the cells above and sums them with the
// reference's nesting.  Bound by the issue of the traversal and of the terms,
// about 125 instructions per visit and warp, 37 of them on the FP64 pipe.
// ---------------------------------------------------------------------------
constexpr int kXQ = 32;  // queue entries per warp
constexpr int kXU = 4;   // entries evaluated together
constexpr float kXBand = 4e-7f;

// Whether every pair of an evaluation is in exact_scale's range: masses of
// one sign within [2^-190, 2^240 / n] or 0 (so are the sums over cells),
// bodies and centres of mass within 2^98, softening.
__device__ __forceinline__ bool walk_in_range(const TreeHeader* hdr, int64_t n, double eps2) {
  const double c = fmax(fmax(fabs(hdr->center[0]), fabs(hdr->center[1])), fabs(hdr->center[2]));
  return scale_eps2_ok(eps2) && hdr->min_mass >= 0.0 && hdr->min_abs >= 0x1p-190 &&
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

// The nested sums of one target: the deepest level with a term in registers.
struct NestedSum {
  double st[kMaxLevels + 1][3];
  double x, y, z;
  int d;
  __device__ __forceinline__ void init(int depth) {
    x = y = z = 0.0;
    d = depth;
  }
  // close the levels below m
  __device__ __forceinline__ void close_to(int m) {
    while (d > m) {
      --d;
      x = xadd(st[d][0], x);
      y = xadd(st[d][1], y);
      z = xadd(st[d][2], z);
    }
  }
  // open levels up to depth, at 0
  __device__ __forceinline__ void open_to(int depth) {
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

// Number of tasks; a tree with more top nodes than there is room for is
// walked as one task, the root.
__device__ __forceinline__ int top_tasks(const TopTree& top) {
  const int c = *top.counts, nt = c >> 16;
  return nt <= top.max_tasks && (c & 0xffff) <= top.max_top ? nt : 1;
}

__global__ void __launch_bounds__(kWalkBlock, 4)
walk_task_kernel(int64_t q0, int64_t n, int64_t nbody, int nnodes, const RecX* __restrict__ wx,
                 const double4* __restrict__ rec64, const double4* __restrict__ body64,
                 const TreeHeader* __restrict__ hdr, TopTree top, double G, double eps2,
                 double* __restrict__ part, unsigned long long* counter, int32_t* status) {
  wait_for_previous();
  __shared__ double s2d[kMaxLevels];
  __shared__ float2 band[kMaxLevels];
  __shared__ uint4 queue[kWalkBlock / 32][kXQ];  // node, lane mask, close to, level
  const int task = (int)blockIdx.y;
  const int ntask = top_tasks(top);
  if (task >= ntask) return;
  const int root = ntask == 1 ? 0 : top.task[task];
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
  const int64_t p = q0 + blockIdx.x * (int64_t)kWalkBlock + threadIdx.x;  // targets [q0, n)
  const bool valid = p < n;
  const ExactTarget t = exact_target(body64, p, valid, G);
  const bool coarse = hdr->min_mass >= 0.0;
  const bool fast =
      !__any_sync(0xffffffffu, !scale_mass_ok(t.gm)) && walk_in_range(hdr, nbody, eps2);
  const double ih = 1.0 / half;
  const float fx = (float)((t.x - hdr->center[0]) * ih), fy = (float)((t.y - hdr->center[1]) * ih),
              fz = (float)((t.z - hdr->center[2]) * ih);

  NestedSum sum;
  unsigned ninter = 0;
  int cnt = 0;
  uint4* const q = queue[wid];
  auto drain = [&]() {
    __syncwarp();
    for (int k0 = 0; k0 < cnt; k0 += kXU) {
      double rx[kXU], ry[kXU], rz[kXU], w[kXU];
      uint4 e[kXU];
      if (fast) {
#pragma unroll
        for (int u = 0; u < kXU; ++u) {
          e[u] = q[min(k0 + u, cnt - 1)];
          w[u] = exact_weight<true>(t, rec64[e[u].x], eps2, rx[u], ry[u], rz[u]);
        }
      } else {
#pragma unroll
        for (int u = 0; u < kXU; ++u) {
          e[u] = q[min(k0 + u, cnt - 1)];
          w[u] = exact_weight<false>(t, rec64[e[u].x], eps2, rx[u], ry[u], rz[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < kXU; ++u) {
        if (k0 + u < cnt) {
          sum.close_to((int)e[u].z);
          sum.open_to((int)e[u].w);
          if ((e[u].y >> lane) & 1u) {
            sum.add(xmul(rx[u], w[u]), xmul(ry[u], w[u]), xmul(rz[u], w[u]));
            ++ninter;
          }
        }
      }
    }
    __syncwarp();
    cnt = 0;
  };

  // open_to: opened levels on the current path (a lane is active at a node
  // of depth d iff open_to == d); low: the least depth of the warp's path
  // since its last entry
  // the task's cells above were all opened by the lane?
  const int base = wx[root].b.x & kMetaDepth;
  int open_to = -1;
  if (valid) {
    bool in = true;
    for (int k = root, d = base - 1; d >= 0; --d) {
      k = top.parent[k];
      in = in && (k == 0 || (wx[k].b.x & kMetaGate)) && exact_open(rec64[k], t, s2d[d], theta2);
    }
    if (in) open_to = base;
  }
  const bool counted = open_to >= 0;
  sum.init(base);
  int low = base;
  int node = root;
  const int end = __float_as_int(wx[root].a.w);
  auto ld_a = [&](int k) { return __ldg(&wx[k].a); };
  auto ld_b = [&](int k) { return __ldg(reinterpret_cast<const int2*>(&wx[k].b)); };
  float4 A = ld_a(node);
  int2 B = ld_b(node);
  while (node < end) {
    const int next = __float_as_int(A.w);
    if (next <= node || next > nnodes) {  // malformed tree: report, never spin
      if (lane == 0) atomicOr(status, kStatOverflow);
      break;
    }
    // both nodes that may follow are read while this one is decided
    const int k0 = min(node + 1, nnodes - 1), k1 = min(next, nnodes - 1);
    const float4 A0 = ld_a(k0), A1 = ld_a(k1);
    const int2 B0 = ld_b(k0), B1 = ld_b(k1);
    const int d = B.x & kMetaDepth;
    open_to = min(open_to, d);
    low = min(low, d);
    const bool act = open_to == d && ((B.x & kMetaGate) || node == 0);
    bool take;
    int go = next;
    if (B.x & kMetaLeaf) {
      take = act && B.y != (int)p;
    } else {
      const float rx = A.x - fx, ry = A.y - fy, rz = A.z - fz;
      const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
      const float2 bd = band[d];
      bool open = act && d2 < bd.x;
      if (__any_sync(0xffffffffu, act && !(coarse && (d2 < bd.x || d2 > bd.y))))
        open = act && exact_open(rec64[node], t, s2d[d], theta2);
      take = act && !open;
      if (open) open_to = d + 1;
      if (__any_sync(0xffffffffu, open)) go = node + 1;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, take);
    if (mask) {
      if (lane == 0) q[cnt] = make_uint4((unsigned)node, mask, (unsigned)low, (unsigned)d);
      low = d;
      if (++cnt == kXQ) drain();
    }
    A = go == next ? A1 : A0;
    B = go == next ? B1 : B0;
    node = go;
  }
  drain();
  sum.close_to(base);
  warp_count(ninter, counter);
  if (counted) {
    double* o = part + ((size_t)task * (size_t)(n - q0) + (size_t)(p - q0)) * 3;
    o[0] = sum.x;
    o[1] = sum.y;
    o[2] = sum.z;
  }
}

// A target's force from its tasks' contributions: the walk over the upper
// cells, nested as in compute_force (gravity_tree.rs:194-205).
__global__ void __launch_bounds__(kWalkBlock)
exact_combine_kernel(int64_t q0, int64_t n, const RecX* __restrict__ wx,
                     const double4* __restrict__ rec64, const double4* __restrict__ body64,
                     const uint32_t* __restrict__ perm, const TreeHeader* __restrict__ hdr,
                     TopTree top, double G, double eps2, int want_force,
                     const double* __restrict__ part, double* __restrict__ ox,
                     double* __restrict__ oy, double* __restrict__ oz,
                     unsigned long long* counter, int32_t* status) {
  wait_for_previous();
  const int64_t p = q0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = p < n;
  const ExactTarget t = exact_target(body64, valid ? p : q0, true, G);
  const double theta2 = hdr->theta2;
  const int ntop = top_tasks(top) == 1 ? 1 : *top.counts & 0xffff;
  unsigned ninter = 0;
  NestedSum sum;
  sum.init(0);
  int open_to = 0;
  for (int i = 0; i < ntop; ++i) {
    const int4 e = ntop == 1 ? make_int4(0, 0, 0, 0) : top.top[i];
    const int node = e.x, d = e.z;
    open_to = min(open_to, d);
    sum.close_to(d);
    const bool act = open_to == d && (node == 0 || (wx[node].b.x & kMetaGate));
    if (e.y >= 0) {
      sum.open_to(d);
      if (act && valid) {
        const double* q = part + ((size_t)e.y * (size_t)(n - q0) + (size_t)(p - q0)) * 3;
        sum.add(q[0], q[1], q[2]);
      }
    } else {
      const double4 r = rec64[node];
      const bool open = act && exact_open(r, t, hdr->s2[d], theta2);
      if (open) open_to = d + 1;
      if (act && !open) {  // taken as a monopole
        double rx, ry, rz;
        const double w = exact_weight<false>(t, r, eps2, rx, ry, rz);
        sum.open_to(d);
        sum.add(xmul(rx, w), xmul(ry, w), xmul(rz, w));
        ninter += valid;
      }
    }
  }
  sum.close_to(0);
  warp_count(ninter, counter);
  if (!valid) return;
  double f[3] = {sum.x, sum.y, sum.z};
  const double mi = body64[p].w;
  const uint32_t i = perm[p];
  double* o[3] = {ox, oy, oz};
  bool bad = false;
  for (int k = 0; k < 3; ++k) {
    if (!want_force) f[k] = xdiv(f[k], mi);  // a = F / m (integrators.rs:115)
    o[k][i] = f[k];
    bad |= !isfinite(f[k]);
  }
  if (bad) atomicOr(status, kStatNonfinite);
}

// One walk per target over the whole tree, terms evaluated as they are
// taken: 48 registers and more warps per SM hide the latency of a visit, so
// with enough targets to fill the SMs this is the faster form (2^20 bodies:
// 19.8 ms against 28.7 for walk_task_kernel over the root, 100 000: 2.9
// against 3.0; 65 536: 2.7 against 2.1, 10 000: 1.64 against 0.44).
__global__ void __launch_bounds__(kWalkBlock)
walk_exact_kernel(int64_t q0, int64_t n, int64_t nnodes, const int4* __restrict__ link,
                  const double4* __restrict__ rec64, const double4* __restrict__ body64,
                  const uint32_t* __restrict__ perm, const TreeHeader* __restrict__ hdr, double G,
                  double eps2, int want_force, double* __restrict__ ox, double* __restrict__ oy,
                  double* __restrict__ oz, unsigned long long* counter, int32_t* status) {
  wait_for_previous();
  __shared__ double s2d[kMaxLevels];
  for (int d = threadIdx.x; d < kMaxLevels; d += blockDim.x) s2d[d] = hdr->s2[d];
  __syncthreads();
  const double theta2 = hdr->theta2;
  const int64_t p = q0 + blockIdx.x * (int64_t)kWalkBlock + threadIdx.x;  // targets [q0, n)
  const bool valid = p < n;
  double tx = 0, ty = 0, tz = 0, mi = 0;
  if (valid) {
    const double4 b = body64[p];
    tx = b.x;
    ty = b.y;
    tz = b.z;
    mi = b.w;
  }
  const double gm = xmul(G, mi);
  // acc[d] collects the terms of the nodes at depth d (children of the lane's
  // opened node at depth d-1); acc[0] is the root's own term.
  double acc[kMaxLevels + 1][3];
  acc[0][0] = acc[0][1] = acc[0][2] = 0.0;
  unsigned ninter = 0;
  int open_to = 0;
  int32_t node = 0;

  // compute_gravity_pair (gravity_tree.rs:218-234)
  auto pair = [&](double4 s, int slot) {
    const double rx = xsub(s.x, tx), ry = xsub(s.y, ty), rz = xsub(s.z, tz);
    const double r2 = xlen2(rx, ry, rz);
    const double s2 = xadd(r2, eps2);
    const double s3 = xmul(s2, xsqrt(s2));
    const double sc = xdiv(xmul(gm, s.w), s3);
    acc[slot][0] = xadd(acc[slot][0], xmul(rx, sc));
    acc[slot][1] = xadd(acc[slot][1], xmul(ry, sc));
    acc[slot][2] = xadd(acc[slot][2], xmul(rz, sc));
  };
  auto close_to = [&](int d) {  // finish the lane's opened cells at depths >= d
    for (int k = open_to; k > d; --k) {
      acc[k - 1][0] = xadd(acc[k - 1][0], acc[k][0]);
      acc[k - 1][1] = xadd(acc[k - 1][1], acc[k][1]);
      acc[k - 1][2] = xadd(acc[k - 1][2], acc[k][2]);
    }
    if (open_to > d) open_to = d;
  };

  while (node < nnodes) {
    const int4 lk = link[node];
    if (lk.x <= node || lk.x > nnodes) {  // malformed tree: report, never spin
      if ((threadIdx.x & 31) == 0) atomicOr(status, kStatOverflow);
      break;
    }
    const int d = lk.w & kMetaDepth;
    close_to(d);
    const bool act = valid && open_to == d && ((lk.w & kMetaGate) || node == 0);
    if (lk.w & kMetaLeaf) {
      const int sp = (lk.z - lk.y) == 1 ? lk.y : lk.z - 1;
      if (act && sp != p) {
        pair(rec64[node], d);
        ++ninter;
      }
      node = lk.x;
    } else {
      const double4 s = rec64[node];
      const double rx = xsub(s.x, tx), ry = xsub(s.y, ty), rz = xsub(s.z, tz);
      const double d2 = xlen2(rx, ry, rz);
      const bool open = act && !(s2d[d] < xmul(theta2, d2));
      if (act && !open) {
        pair(s, d);
        ++ninter;
      }
      if (open) {
        acc[d + 1][0] = acc[d + 1][1] = acc[d + 1][2] = 0.0;
        open_to = d + 1;
      }
      node = __any_sync(0xffffffffu, open) ? node + 1 : lk.x;
    }
  }
  close_to(0);
  warp_count(ninter, counter);
  if (!valid) return;
  double fx = acc[0][0], fy = acc[0][1], fz = acc[0][2];
  if (!want_force) {  // a = F / m (integrators.rs:115)
    fx = xdiv(fx, mi);
    fy = xdiv(fy, mi);
    fz = xdiv(fz, mi);
  }
  const uint32_t i = perm[p];
  ox[i] = fx;
  oy[i] = fy;
  oz[i] = fz;
  if (!isfinite(fx) || !isfinite(fy) || !isfinite(fz)) atomicOr(status, kStatNonfinite);
}

}  // namespace

int exact_walk_tasks(const phys_ctx* c, int64_t n) {
  int64_t q0 = 0, q1 = n;
  target_range(c, n, q0, q1);
  const int64_t nt = q1 - q0;
  // `part` holds 24 bytes per task and target: at most 100 MB
  return nt > 0 && nt <= 65536 ? (int)min64(512, (int64_t(1) << 22) / nt) : 0;
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
    const int tasks = t.top.max_tasks;
    if (tasks > 0) {
      double* part = nullptr;
      PHYS_TRY(ws_alloc(c, WS_DIRECT_PART, 3 * nt * tasks, &part));
      PHYS_LAUNCH(c, walk_task_kernel, dim3(grid, tasks), kWalkBlock, 0, q0, q1, n, t.nnodes,
                  t.wx, t.rec64, t.body64, t.hdr, t.top, p->G, eps2, part, c->d_counter,
                  c->d_status);
      PHYS_LAUNCH(c, exact_combine_kernel, (int)ceil_div(nt, 64), 64, 0, q0, q1, t.wx, t.rec64,
                  t.body64, t.perm, t.hdr, t.top, p->G, eps2, want_force, part, ox, oy, oz,
                  c->d_counter, c->d_status);
    } else {
      PHYS_LAUNCH(c, walk_exact_kernel, grid, kWalkBlock, 0, q0, q1, t.nnodes, t.link, t.rec64,
                  t.body64, t.perm, t.hdr, p->G, eps2, want_force, ox, oy, oz, c->d_counter,
                  c->d_status);
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

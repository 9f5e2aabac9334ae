// K1: softened all-pairs direct sum (brute_force_gravity_system,
// src/physics/gravity.rs:53-69), in three precisions.
//
// Layout: sources are staged through shared memory in tiles; every lane of a
// warp reads the same source (shared-memory broadcast) while owning one
// target.  For small N the source range is split into `slices` so the grid
// covers all SMs; slice partials are reduced in slice order (deterministic).
#include <utility>

#include "common.cuh"

namespace phys {
namespace {

// ---------------------------------------------------------------------------
// F64_EXACT: the reference's arithmetic, j in order 0..N-1, no FMA.
//   r = x_j - x_i; r2 = len2(r); s2 = r2 + eps2; s3 = s2 * sqrt(s2)
//   sc = ((G*m_i)*m_j)/s3; F += r*sc            (gravity.rs:58-65)
// Only the additions into F are ordered; the terms r*sc are independent.  A
// block takes kXT targets.  Producer warps evaluate the terms: producer p
// takes the chunks p, p + kProd, ... of 32 sources, a lane holding one
// source against half of the targets at a time (that many independent chains of
// exact_scale), and hands each chunk to warp 0 through its own shared-memory
// slot.  Lane l of warp 0 adds component l / kXT of target l % kXT in j
// order: one dependent f64 addition per source and nothing else on the chain
// (the next chunk's terms are read while the current chunk's are added).  A
// skipped term (j == i, past the end) is stored as +-0: the sum starts from
// +0 and so is never -0, and adding a zero leaves every value as it is.  A
// chunk with a source, or a block with a target, outside exact_scale's range
// takes the library's square root and division instead.
//
// The floor of any exact form is the ordered chain, N - 1 additions of 8.2
// cycles (4.3 us at N = 1024; the adding warp takes 10.6 per source), and for
// many targets the FP64 pipe, 37 operations per pair.  A tick of 1024 bodies
// (force pass, velocity and position step) takes 12.7 us where the form with
// one round barrier and the library's operations took 21.1 us in two
// kernels; 20000 bodies 1.40 ms against 2.46 (about 60 % of the FP64 pipe, the
// shared-memory traffic of the terms close behind).
// kTick also performs the velocity step of the tick and the position step of
// the next one on the finished components, the new positions going to a
// second set of arrays because other blocks still read the old ones.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void pair_sync(int id) {  // one producer warp and warp 0
  asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void pair_arrive(int id) {
  asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}

// A tick's integration state beside the force pass: kicked velocities,
// previous accelerations, positions written to nx/ny/nz.
struct TickArgs {
  double dt;
  double *vx, *vy, *vz, *pax, *pay, *paz, *nx, *ny, *nz;
};

// kProd = 6, 8 warps, 8 targets: warps 1-3 and 5-7 produce, so that no
// producer shares warp 0's scheduler (warps go to an SM's four schedulers by
// index) while a block has an SM to itself (N = 1024: 9.5 us a launch inside a
// graph, 13.0 with the other layout), and up to two such blocks an SM (a tick
// of 1500 bodies 19.1 against 22.0 us, of 2368 26.9 against 32.4); kProd = 4, 5
// warps, 10 targets, four blocks per SM: more adding warps per SM once there
// are more blocks (N = 4096: 68 us against 78).
// kSoft: eps^2 alone keeps |r|^2 + eps^2 in exact_scale's range; else (no
// softening) every pair is looked at, and a chunk with one outside (coincident
// bodies) is formed again.  Against library operations for all of these, and
// for masses or positions out of range against both forms in turn: a tick of
// 1500 bodies 35.8 -> 19.3 us without softening, 50.1 -> 28.6 with masses of
// 1e-103 (31.8 before either form had the branch-free weight).
constexpr int x_block(int prod) { return prod == 6 ? 256 : 32 * (prod + 1); }
constexpr int x_targets(int prod) { return prod == 6 ? 8 : 10; }

template <int kProd, bool kTick, bool kSoft>
__global__ void __launch_bounds__(x_block(kProd), kProd == 6 ? 2 : 4)
direct_exact_kernel(int64_t n, int64_t t0, int64_t t1, const double* __restrict__ x,
                    const double* __restrict__ y, const double* __restrict__ z,
                    const double* __restrict__ m, double G, double eps2, int want_force,
                    double* __restrict__ ox, double* __restrict__ oy, double* __restrict__ oz,
                    TickArgs tick, int32_t* status) {
  wait_for_previous();
  constexpr int kXT = x_targets(kProd), kXGroup = kXT / 2;
  constexpr int kXRows = 3 * kXT;  // ordered sums per block, one per lane
  static_assert(kXRows <= 32, "one adding warp");
  __shared__ double term[kProd][kXRows][33];  // [producer][component, target][source]
  __shared__ double4 tgt[kXT];                // x_i, y_i, z_i, G*m_i
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i0 = t0 + blockIdx.x * (int64_t)kXT;
  if (threadIdx.x < kXT) {
    const int64_t i = i0 + threadIdx.x;
    tgt[threadIdx.x] = i < t1 ? make_double4(x[i], y[i], z[i], xmul(G, m[i]))
                              : make_double4(0.0, 0.0, 0.0, 0.0);
  }
  __syncthreads();
  const int chunks = (int)ceil_div(n, 32);
  // barrier ids: 1 + p a full slot, 1 + kProd + p a slot read out
  if (w > 0) {
    if (kProd == 6 && w == 4) return;
    const int p = kProd == 6 ? w - 1 - (w > 4) : w - 1;
    bool targets_ok = true;
    for (int t = 0; t < kXT; ++t)
      targets_ok &= scale_mass_ok(tgt[t].w) && scale_pos_ok(tgt[t].x, tgt[t].y, tgt[t].z);
    auto load = [&](int64_t j) {
      return j < n ? make_double4(x[j], y[j], z[j], m[j]) : make_double4(0.0, 0.0, 0.0, 0.0);
    };
    for (int k = p; k < chunks; k += kProd) {
      const int64_t j = k * (int64_t)32 + lane;
      const double4 src = load(j);
      if (k >= kProd) pair_sync(1 + kProd + p);
      bool in_range = __all_sync(0xffffffffu, targets_ok && scale_pos_ok(src.x, src.y, src.z) &&
                                                  scale_mass_ok(src.w));
      bool pairs_ok = true;
#pragma unroll 1
      for (int tg = 0; tg < kXT && in_range; tg += kXGroup) {
        // every weight of the group first: a store between two of them would
        // keep the second pair's chain behind the first's
        double rx[kXGroup], ry[kXGroup], rz[kXGroup], wt[kXGroup];
#pragma unroll
        for (int u = 0; u < kXGroup; ++u) {
          const int t = tg + u;
          const double4 T = tgt[t];
          rx[u] = xsub(src.x, T.x), ry[u] = xsub(src.y, T.y), rz[u] = xsub(src.z, T.z);
          const double x2 = xadd(xlen2(rx[u], ry[u], rz[u]), eps2);
          wt[u] = exact_scale(xmul(T.w, src.w), x2);
          const bool none = j >= n || j == i0 + t;
          if (!kSoft) pairs_ok &= none || scale_square_ok(x2);
          if (none) wt[u] = 0.0;
        }
#pragma unroll
        for (int u = 0; u < kXGroup; ++u) {
          term[p][tg + u][lane] = xmul(rx[u], wt[u]);
          term[p][kXT + tg + u][lane] = xmul(ry[u], wt[u]);
          term[p][2 * kXT + tg + u][lane] = xmul(rz[u], wt[u]);
        }
      }
      if (!kSoft) in_range &= __all_sync(0xffffffffu, pairs_ok);
      if (!in_range) {
        for (int t = 0; t < kXT; ++t) {
          const double4 T = tgt[t];
          const double rx = xsub(src.x, T.x), ry = xsub(src.y, T.y), rz = xsub(src.z, T.z);
          double wt = exact_scale_ieee(xmul(T.w, src.w), xadd(xlen2(rx, ry, rz), eps2));
          if (j >= n || j == i0 + t) wt = 0.0;
          term[p][t][lane] = xmul(rx, wt);
          term[p][kXT + t][lane] = xmul(ry, wt);
          term[p][2 * kXT + t][lane] = xmul(rz, wt);
        }
      }
      __syncwarp();
      pair_arrive(1 + p);
    }
    return;
  }
  const int row = lane < kXRows ? lane : 0;
  double f = 0.0, cur[32];
  pair_sync(1);
#pragma unroll
  for (int q = 0; q < 32; ++q) cur[q] = term[0][row][q];
  if (kProd < chunks) pair_arrive(1 + kProd);
  for (int k = 1, p = 1; k < chunks; ++k) {
    double nxt[32];
    pair_sync(1 + p);
#pragma unroll
    for (int q = 0; q < 32; ++q) {
      nxt[q] = term[p][row][q];
      f = xadd(f, cur[q]);
    }
    if (k + kProd < chunks) pair_arrive(1 + kProd + p);
#pragma unroll
    for (int q = 0; q < 32; ++q) cur[q] = nxt[q];
    p = p + 1 == kProd ? 0 : p + 1;
  }
#pragma unroll
  for (int q = 0; q < 32; ++q) f = xadd(f, cur[q]);

  const int c = row / kXT;
  const int64_t i = i0 + row % kXT;
  const bool valid = lane < kXRows && i < t1;
  bool bad = false;
  if (valid) {
    // compute_acceleration_system: a = F / m (integrators.rs:115)
    if (kTick || !want_force) f = xdiv(f, m[i]);
    (c == 0 ? ox : c == 1 ? oy : oz)[i] = f;
    bad = !isfinite(f);
    if (kTick) {  // kick_drift_kernel's operations on this component
      double* v = c == 0 ? tick.vx : c == 1 ? tick.vy : tick.vz;
      double* pa = c == 0 ? tick.pax : c == 1 ? tick.pay : tick.paz;
      const double* xo = c == 0 ? x : c == 1 ? y : z;
      const double hdt = xmul(0.5, tick.dt), h2 = xmul(xmul(0.5, tick.dt), tick.dt);
      const double v1 = xadd(v[i], xmul(xadd(pa[i], f), hdt));
      const double x1 = xadd(xo[i], xadd(xmul(v1, tick.dt), xmul(f, h2)));
      v[i] = v1;
      pa[i] = f;
      (c == 0 ? tick.nx : c == 1 ? tick.ny : tick.nz)[i] = x1;
      bad |= !isfinite(v1) || !isfinite(x1);
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(status, kStatNonfinite);
}

template <bool kTick>
int launch_exact(phys_ctx* c, const phys_params* p, int64_t t0, int64_t t1, const double* x,
                 const double* y, const double* z, int want_force, double* ox, double* oy,
                 double* oz, const TickArgs& tick) {
  const bool solo = t1 - t0 <= 2 * 148 * x_targets(6);
  const int64_t blocks = ceil_div(t1 - t0, solo ? x_targets(6) : x_targets(4));
  const double eps2 = p->eps * p->eps;
  const bool soft = scale_eps2_ok(eps2);
  auto kernel = solo ? (soft ? direct_exact_kernel<6, kTick, true>
                             : direct_exact_kernel<6, kTick, false>)
                     : (soft ? direct_exact_kernel<4, kTick, true>
                             : direct_exact_kernel<4, kTick, false>);
  PHYS_LAUNCH(c, kernel, (int)blocks, solo ? x_block(6) : x_block(4), 0, c->n, t0, t1, x, y, z,
              c->m, p->G, eps2, want_force, ox, oy, oz, tick, c->d_status);
  return PHYS_OK;
}

// ---------------------------------------------------------------------------
// F64: same law with FMA and inv_cubed, accumulating sum m_j r / s^3 (G applied
// at the end).  A thread takes two targets, so that a source read from shared
// memory (two 16-byte broadcasts, 8 cycles of an SM's load path a warp) serves
// two pair terms of 16 FP64 operations (8 cycles of its FP64 pipe each): with
// one target per thread the loads were as long as the arithmetic.  65 536
// bodies: 5.40 -> 4.51 ms (84 % of the FP64 pipe's rate), 20 011: 500 -> 443
// us, 1024: 28 -> 16 us (the slices also follow the chip now); four targets
// per thread 4.79 ms.  A tile that overlaps the block's own targets takes the checked
// loop (j == i skipped).
// ---------------------------------------------------------------------------
constexpr int kTile = 128;
constexpr int kDThreads = 64;
constexpr int kT = 2;  // targets per thread, kDThreads apart

template <bool kChecked>
__device__ __forceinline__ void f64_tile(const double4* __restrict__ t, int cnt, const int* self,
                                         const double (&xi)[kT], const double (&yi)[kT],
                                         const double (&zi)[kT], double eps2, double (&ax)[kT],
                                         double (&ay)[kT], double (&az)[kT]) {
#pragma unroll 4
  for (int k = 0; k < cnt; ++k) {
    const double4 s = t[k];
#pragma unroll
    for (int q = 0; q < kT; ++q) {
      const double rx = s.x - xi[q], ry = s.y - yi[q], rz = s.z - zi[q];
      double r2 = fma(rx, rx, fma(ry, ry, fma(rz, rz, eps2)));
      double mj = s.w;
      if (kChecked && k == self[q]) {
        mj = 0.0;
        r2 = 1.0;
      }
      const double w = mj * inv_cubed(r2);
      ax[q] = fma(rx, w, ax[q]);
      ay[q] = fma(ry, w, ay[q]);
      az[q] = fma(rz, w, az[q]);
    }
  }
}

// part: partial sums per slice (or, null with one slice, the results).
__global__ void __launch_bounds__(kDThreads)
direct_f64_kernel(int64_t n, int64_t t0, int64_t t1, int64_t slice_len,
                  const double* __restrict__ x, const double* __restrict__ y,
                  const double* __restrict__ z, const double* __restrict__ m, double G,
                  double eps2, int want_force, double* __restrict__ ox, double* __restrict__ oy,
                  double* __restrict__ oz, double* __restrict__ part, int32_t* status) {
  wait_for_previous();
  __shared__ double4 tile[kTile];
  const int64_t tbase = t0 + blockIdx.x * (int64_t)(kDThreads * kT);
  double xi[kT], yi[kT], zi[kT], ax[kT], ay[kT], az[kT];
#pragma unroll
  for (int q = 0; q < kT; ++q) {
    const int64_t i = tbase + threadIdx.x + q * kDThreads;
    const bool valid = i < t1;
    xi[q] = valid ? x[i] : 0.0;
    yi[q] = valid ? y[i] : 0.0;
    zi[q] = valid ? z[i] : 0.0;
    ax[q] = ay[q] = az[q] = sum_start(eps2);
  }
  const int64_t lo = blockIdx.y * slice_len;
  const int64_t hi = min64(n, lo + slice_len);
  for (int64_t base = lo; base < hi; base += kTile) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kTile / kDThreads; ++r) {
      const int64_t j = base + threadIdx.x + r * kDThreads;
      tile[threadIdx.x + r * kDThreads] =
          j < hi ? make_double4(x[j], y[j], z[j], m[j]) : make_double4(0, 0, 0, 0);
    }
    __syncthreads();
    const int cnt = (int)min64(kTile, hi - base);
    int self[kT];
#pragma unroll
    for (int q = 0; q < kT; ++q) {
      const int64_t d = tbase + threadIdx.x + q * kDThreads - base;
      self[q] = d >= 0 && d < kTile ? (int)d : -1;
    }
    if (base < tbase + kDThreads * kT && base + kTile > tbase)
      f64_tile<true>(tile, cnt, self, xi, yi, zi, eps2, ax, ay, az);
    else
      f64_tile<false>(tile, cnt, self, xi, yi, zi, eps2, ax, ay, az);
  }
#pragma unroll
  for (int q = 0; q < kT; ++q) {
    const int64_t i = tbase + threadIdx.x + q * kDThreads;
    if (i >= t1) continue;
    if (!part) {
      const double s = want_force ? G * m[i] : G;
      ox[i] = ax[q] * s;
      oy[i] = ay[q] * s;
      oz[i] = az[q] * s;
      if (!isfinite(ax[q]) || !isfinite(ay[q]) || !isfinite(az[q]))
        atomicOr(status, kStatNonfinite);
    } else {
      double* p = part + (size_t)blockIdx.y * 3 * n;
      p[i] = ax[q];
      p[n + i] = ay[q];
      p[2 * n + i] = az[q];
    }
  }
}

// ---------------------------------------------------------------------------
// F32C: f32 pair terms.  Positions are double-float pairs (hi, lo); the
// separation r = (hi_j - hi_i) + (lo_j - lo_i) keeps ~1e-7 relative accuracy
// however close the pair is compared with |x|.  Each group of 32 terms is
// summed in plain f32 and folded into a per-target (hi, lo) accumulator with
// Knuth's two-sum.
// ---------------------------------------------------------------------------
__global__ void split_bodies_kernel(int64_t n, const double* __restrict__ x,
                                    const double* __restrict__ y, const double* __restrict__ z,
                                    const double* __restrict__ m, float4* __restrict__ bh,
                                    float4* __restrict__ bl, int32_t* status) {
  wait_for_previous();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float4 h, l;
    split_df(x[i], h.x, l.x);
    split_df(y[i], h.y, l.y);
    split_df(z[i], h.z, l.z);
    h.w = (float)m[i];
    l.w = 0.f;
    bh[i] = h;
    bl[i] = l;
    if (!isfinite(x[i]) || !isfinite(y[i]) || !isfinite(z[i]) || !isfinite(m[i]))
      atomicOr(status, kStatNonfinite);
  }
}

// The thread's two targets, packed (f32x2).
struct F32Targets {
  float2 nhx, nhy, nhz, nlx, nly, nlz;  // negated positions
};

template <bool kChecked>
__device__ __forceinline__ void f32_group(const float4* __restrict__ th,
                                          const float4* __restrict__ tl, int k0, int k1,
                                          const int (&self)[kT], const F32Targets& t, float2 e2,
                                          float2& px, float2& py, float2& pz) {
#pragma unroll 8
  for (int k = k0; k < k1; ++k) {
    const float4 h = th[k];
    const float4 l = tl[k];
    auto both = [](float v) { return make_float2(v, v); };
    const float2 rx = __fadd2_rn(__fadd2_rn(both(h.x), t.nhx), __fadd2_rn(both(l.x), t.nlx));
    const float2 ry = __fadd2_rn(__fadd2_rn(both(h.y), t.nhy), __fadd2_rn(both(l.y), t.nly));
    const float2 rz = __fadd2_rn(__fadd2_rn(both(h.z), t.nhz), __fadd2_rn(both(l.z), t.nlz));
    const float2 r2 = __ffma2_rn(rx, rx, __ffma2_rn(ry, ry, __ffma2_rn(rz, rz, e2)));
    const float2 inv = make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
    float2 w = __fmul2_rn(both(h.w), __fmul2_rn(__fmul2_rn(inv, inv), inv));
    if (kChecked && k == self[0]) w.x = 0.f;
    if (kChecked && k == self[1]) w.y = 0.f;
    px = __ffma2_rn(rx, w, px);
    py = __ffma2_rn(ry, w, py);
    pz = __ffma2_rn(rz, w, pz);
  }
}

// Two targets per thread, both in one packed instruction: half the issue
// slots and half the shared-memory broadcasts per pair term (18 FP32
// operations).  The arithmetic per target and its order are those of one
// target per thread.  20 011 bodies: 324 -> 271 us (87 % of the packed FMA
// rate), 65 536: 3.40 -> 2.78 ms; four targets per thread 304 us, two scalar
// ones 315.
__global__ void __launch_bounds__(kDThreads)
direct_f32c_kernel(int64_t n, int64_t t0, int64_t t1, int64_t slice_len,
                   const float4* __restrict__ bh, const float4* __restrict__ bl,
                   const double* __restrict__ m, double G, float eps2, int want_force,
                   double* __restrict__ ox, double* __restrict__ oy, double* __restrict__ oz,
                   double* __restrict__ part, int32_t* status) {
  wait_for_previous();
  __shared__ float4 th[kTile];
  __shared__ float4 tl[kTile];
  const int64_t tbase = t0 + blockIdx.x * (int64_t)(kDThreads * kT);  // t0: a multiple of kTile
  const int64_t i0 = tbase + threadIdx.x, i1 = i0 + kDThreads;
  const float4 zero = make_float4(0, 0, 0, 0);
  const float4 ha = i0 < t1 ? bh[i0] : zero, la = i0 < t1 ? bl[i0] : zero;
  const float4 hb = i1 < t1 ? bh[i1] : zero, lb = i1 < t1 ? bl[i1] : zero;
  const F32Targets t{make_float2(-ha.x, -hb.x), make_float2(-ha.y, -hb.y),
                     make_float2(-ha.z, -hb.z), make_float2(-la.x, -lb.x),
                     make_float2(-la.y, -lb.y), make_float2(-la.z, -lb.z)};
  const int64_t lo = blockIdx.y * slice_len;
  const int64_t hi = min64(n, lo + slice_len);
  const float2 e2 = make_float2(eps2, eps2);
  float ahx[kT] = {}, ahy[kT] = {}, ahz[kT] = {}, alx[kT] = {}, aly[kT] = {}, alz[kT] = {};
  auto fold = [](float& ah, float& al, float p) {
    float s, e;
    two_sum(ah, p, s, e);
    ah = s;
    al += e;
  };
  for (int64_t base = lo; base < hi; base += kTile) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kTile / kDThreads; ++r) {
      const int k = threadIdx.x + r * kDThreads;
      const int64_t j = base + k;
      th[k] = j < hi ? bh[j] : zero;
      tl[k] = j < hi ? bl[j] : zero;
    }
    __syncthreads();
    const int cnt = (int)min64(kTile, hi - base);
    // slices and blocks both start on tiles: the block's own tile, or none
    const bool diag = base == tbase;
    const int self[kT] = {(int)threadIdx.x, (int)threadIdx.x + kDThreads};
    for (int k0 = 0; k0 < cnt; k0 += 32) {
      const int k1 = min(cnt, k0 + 32);
      float2 px = make_float2(0.f, 0.f), py = px, pz = px;
      if (diag)
        f32_group<true>(th, tl, k0, k1, self, t, e2, px, py, pz);
      else
        f32_group<false>(th, tl, k0, k1, self, t, e2, px, py, pz);
      fold(ahx[0], alx[0], px.x);
      fold(ahy[0], aly[0], py.x);
      fold(ahz[0], alz[0], pz.x);
      fold(ahx[1], alx[1], px.y);
      fold(ahy[1], aly[1], py.y);
      fold(ahz[1], alz[1], pz.y);
    }
  }
  static_assert(kTile == kDThreads * kT, "a block's targets are one tile");
#pragma unroll
  for (int q = 0; q < kT; ++q) {
    const int64_t i = q ? i1 : i0;
    if (i >= t1) continue;
    const double ax = (double)ahx[q] + (double)alx[q];
    const double ay = (double)ahy[q] + (double)aly[q];
    const double az = (double)ahz[q] + (double)alz[q];
    if (gridDim.y == 1) {
      const double s = want_force ? G * m[i] : G;
      ox[i] = ax * s;
      oy[i] = ay * s;
      oz[i] = az * s;
      if (!isfinite(ax) || !isfinite(ay) || !isfinite(az)) atomicOr(status, kStatNonfinite);
    } else {
      double* p = part + (size_t)blockIdx.y * 3 * n;
      p[i] = ax;
      p[n + i] = ay;
      p[2 * n + i] = az;
    }
  }
}

// Sum slice partials in slice order and apply G (and m_i for forces), for
// targets [t0, t1) of partials laid out with stride n per component: one
// thread per (target, component), its slices' loads in flight together.
__global__ void slice_reduce_kernel(int64_t n, int64_t t0, int64_t t1, int nslices,
                                    const double* __restrict__ part,
                                    const double* __restrict__ m, double G, int want_force,
                                    double* __restrict__ ox, double* __restrict__ oy,
                                    double* __restrict__ oz, int32_t* status) {
  wait_for_previous();
  const int64_t nt = t1 - t0;
  bool bad = false;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 3 * nt;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(e / nt);
    const int64_t i = t0 + (e - k * nt);
    const double a = slice_sum(part + k * n + i, 3 * (size_t)n, nslices);
    const double sc = want_force ? G * m[i] : G;
    (k == 0 ? ox : k == 1 ? oy : oz)[i] = a * sc;
    bad |= !isfinite(a);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, kStatNonfinite);
}

// Subset of targets (index list), all sources; one thread per (target,
// slice).  The self pair is skipped by index.  F64_EXACT keeps the reference
// op order with one slice; F64 / F32C use FMA + inv_cubed (the subset
// serves as the f64 reference, so F32C is not used here).
__global__ void __launch_bounds__(kTile)
direct_targets_kernel(int64_t n, int64_t nt, const int64_t* __restrict__ tidx, int64_t slice_len,
                      const double* __restrict__ x, const double* __restrict__ y,
                      const double* __restrict__ z, const double* __restrict__ m, double G,
                      double eps2, int exact, double* __restrict__ part, double* __restrict__ ox,
                      double* __restrict__ oy, double* __restrict__ oz, int32_t* status) {
  wait_for_previous();
  __shared__ double4 tile[kTile];
  const int64_t t = blockIdx.x * (int64_t)kTile + threadIdx.x;
  const bool valid = t < nt;
  const int64_t i = valid ? tidx[t] : -1;
  const bool ok = valid && i >= 0 && i < n;
  if (valid && !ok) atomicOr(status, kStatOverflow);
  const double xi = ok ? x[i] : 0.0, yi = ok ? y[i] : 0.0, zi = ok ? z[i] : 0.0;
  const double mi = ok ? m[i] : 0.0;
  const double gm = xmul(G, mi);
  const int64_t lo = blockIdx.y * slice_len;
  const int64_t hi = min64(n, lo + slice_len);
  double ax = exact ? 0.0 : sum_start(eps2), ay = ax, az = ax;
  for (int64_t base = lo; base < hi; base += kTile) {
    const int64_t j = base + threadIdx.x;
    __syncthreads();
    tile[threadIdx.x] = j < hi ? make_double4(x[j], y[j], z[j], m[j]) : make_double4(0, 0, 0, 0);
    __syncthreads();
    const int cnt = (int)min64(kTile, hi - base);
    if (exact) {
      for (int k = 0; k < cnt; ++k) {
        if (base + k == i) continue;
        const double4 s = tile[k];
        const double rx = xsub(s.x, xi), ry = xsub(s.y, yi), rz = xsub(s.z, zi);
        const double s2 = xadd(xlen2(rx, ry, rz), eps2);
        const double sc = xdiv(xmul(gm, s.w), xmul(s2, xsqrt(s2)));
        ax = xadd(ax, xmul(rx, sc));
        ay = xadd(ay, xmul(ry, sc));
        az = xadd(az, xmul(rz, sc));
      }
    } else {
#pragma unroll 4
      for (int k = 0; k < cnt; ++k) {
        const double4 s = tile[k];
        const double rx = s.x - xi, ry = s.y - yi, rz = s.z - zi;
        const bool self = base + k == i;
        const double r2 = self ? 1.0 : fma(rx, rx, fma(ry, ry, fma(rz, rz, eps2)));
        const double w = self ? 0.0 : s.w * inv_cubed(r2);
        ax = fma(rx, w, ax);
        ay = fma(ry, w, ay);
        az = fma(rz, w, az);
      }
    }
  }
  if (!valid) return;
  if (exact) {  // a = F / m
    ox[t] = xdiv(ax, mi);
    oy[t] = xdiv(ay, mi);
    oz[t] = xdiv(az, mi);
    return;
  }
  double* pp = part + (size_t)blockIdx.y * 3 * nt;
  pp[t] = ax;
  pp[nt + t] = ay;
  pp[2 * nt + t] = az;
}

// F32C slices: about two waves of 148 SMs x 2048 one-target threads; every
// slice spans whole tiles.  (The slices order a target's sum: they follow
// from n alone.)
int64_t f32c_slice_len(int64_t n, int64_t most) {
  int64_t s = ceil_div(148LL * 2048, ceil_div(n, kTile) * kTile);
  s = min64(min64(s, ceil_div(n, kTile)), most);
  return ceil_div(ceil_div(n, s < 1 ? 1 : s), kTile) * kTile;
}

void launch_f32c(cudaStream_t s, int64_t n, int64_t t0, int64_t t1, int64_t slice_len,
                 const float4* bh, const float4* bl, const double* m, double G, float eps2,
                 int want_force, double* ox, double* oy, double* oz, double* part,
                 int32_t* status) {
  const int64_t nsl = ceil_div(n, slice_len);
  const dim3 grid((unsigned)ceil_div(t1 - t0, kDThreads * kT), (unsigned)nsl);
  launch_kernel(s, grid, kDThreads, 0, direct_f32c_kernel, n, t0, t1, slice_len, bh, bl, m, G,
                eps2, want_force, ox, oy, oz, part, status);
}

}  // namespace

// Slices of the F64 sum of n bodies (at most `most`): sixteen 64-thread
// blocks per SM, the number of slices chosen so that the last round of blocks
// is nearly full (eight per SM left 65 536 bodies at 5.8 ms, 24 at 4.55).
F64Plan f64_plan(int64_t n, int64_t most) {
  const int64_t xb = ceil_div(n, kDThreads * kT), round = 148 * 16;
  int64_t best = 1;
  double best_use = 0.0;
  for (int k = 1; k <= 3; ++k) {
    const int64_t sl = round * k / xb > 0 ? round * k / xb : 1;
    const double use = (double)(xb * sl) / (double)(ceil_div(xb * sl, round) * round);
    if (use > best_use + 0.04) {
      best = sl;
      best_use = use;
    }
  }
  best = min64(min64(best, ceil_div(n, 32)), most);
  F64Plan p;
  p.slice_len = ceil_div(ceil_div(n, best), 4) * 4;
  p.slices = ceil_div(n, p.slice_len);
  return p;
}

void direct_f64_launch(cudaStream_t s, const F64Plan& plan, int64_t n, int64_t t0, int64_t t1,
                       const double* x, const double* y, const double* z, const double* m,
                       double G, double eps2, int want_force, double* ox, double* oy, double* oz,
                       double* part, int32_t* status) {
  const dim3 grid((unsigned)ceil_div(t1 - t0, kDThreads * kT), (unsigned)plan.slices);
  launch_kernel(s, grid, kDThreads, 0, direct_f64_kernel, n, t0, t1, plan.slice_len, x, y, z, m,
                G, eps2, want_force, ox, oy, oz, part, status);
}

int direct_eval(phys_ctx* c, const phys_params* p, bool want_force, double* ox, double* oy,
                double* oz) {
  const int64_t n = c->n;
  const double eps2 = p->eps * p->eps;
  if (!c->capturing) PHYS_CUDA(c, cudaEventRecord(c->ev[6], c->stream));
  // targets [t0, t1): all, or the share (t0 a multiple of kTile); the slices
  // follow from n alone, so a target's sum does not depend on the share
  int64_t t0 = 0, t1 = n;
  target_range(c, n, t0, t1);
  if (t0 % kTile) return fail(c, PHYS_ERR_ARG, "direct-sum share must start on a tile");
  const int64_t nt = t1 - t0;
  if (nt <= 0) {
    if (!c->capturing) PHYS_CUDA(c, cudaEventRecord(c->ev[7], c->stream));
    c->tm.interactions = 0;
    return PHYS_OK;
  }
  if (p->precision == PHYS_F64_EXACT) {
    PHYS_TRY(launch_exact<false>(c, p, t0, t1, c->x, c->y, c->z, (int)want_force, ox, oy, oz,
                                 TickArgs{}));
  } else {
    const bool f64 = p->precision == PHYS_F64;
    const F64Plan plan = f64_plan(n, INT64_MAX);
    const int64_t slice_len = f64 ? plan.slice_len : f32c_slice_len(n, INT64_MAX);
    const int64_t nsl = ceil_div(n, slice_len);
    double* part = nullptr;
    int st = PHYS_OK;
    if (nsl > 1) {
      part = (double*)ws_get(c, WS_DIRECT_PART, sizeof(double) * 3 * n * nsl, &st);
      if (st) return st;
    }
    if (f64) {
      direct_f64_launch(c->stream, plan, n, t0, t1, c->x, c->y, c->z, c->m, p->G, eps2,
                        (int)want_force, ox, oy, oz, part, c->d_status);
    } else {
      float4* bh = (float4*)ws_get(c, WS_BODY_HI, sizeof(float4) * n, &st);
      if (st) return st;
      float4* bl = (float4*)ws_get(c, WS_BODY_LO, sizeof(float4) * n, &st);
      if (st) return st;
      int g = (int)min64(ceil_div(n, 256), 148 * 8);
      PHYS_LAUNCH(c, split_bodies_kernel, g, 256, 0, n, c->x, c->y, c->z, c->m, bh, bl,
                  c->d_status);
      launch_f32c(c->stream, n, t0, t1, slice_len, bh, bl, c->m, p->G, (float)eps2,
                  (int)want_force, ox, oy, oz, part, c->d_status);
    }
    c->launches++;
    PHYS_TRY(check_launch(c, "direct sum"));
    if (nsl > 1) {
      int g = (int)min64(ceil_div(3 * nt, 256), 148 * 8);
      PHYS_LAUNCH(c, slice_reduce_kernel, g, 256, 0, n, t0, t1, (int)nsl, part, c->m, p->G,
                  (int)want_force, ox, oy, oz, c->d_status);
    }
  }
  if (!c->capturing) PHYS_CUDA(c, cudaEventRecord(c->ev[7], c->stream));
  c->tm.interactions = (uint64_t)nt * (uint64_t)(n - 1);
  c->tm.bbox_ms = c->tm.keys_ms = c->tm.sort_ms = c->tm.tree_ms = 0.0;
  c->tm.nodes = 0;
  c->tm.max_depth = 0;
  return PHYS_OK;
}

// The force pass of an F64_EXACT tick fused with its velocity step and the
// next position step: positions from x/y/z into the force scratch arrays
// (to_scratch) or back, so a run takes these in pairs.
int direct_exact_tick(phys_ctx* c, const phys_params* p, double dt, bool to_scratch) {
  double *from[3] = {c->x, c->y, c->z}, *to[3] = {c->fx, c->fy, c->fz};
  if (!to_scratch)
    for (int k = 0; k < 3; ++k) std::swap(from[k], to[k]);
  const TickArgs tick{dt, c->vx, c->vy, c->vz, c->pax, c->pay, c->paz, to[0], to[1], to[2]};
  return launch_exact<true>(c, p, 0, c->n, from[0], from[1], from[2], 0, c->ax, c->ay, c->az,
                            tick);
}

// Sliced F64 / F32C direct sum on caller-owned device buffers and stream,
// with caller-provided scratch: `part` (3 * n * nslices doubles), `bh`/`bl`
// (n float4 each, F32C only) and the status word.  Launches the same kernels
// as direct_eval; allocates nothing.
cudaError_t direct_accel_launch_scratch(cudaStream_t s, int64_t n, const double* x,
                                        const double* y,
                                const double* z, const double* m, double G, double eps,
                                int precision, int64_t nslices, double* part, float4* bh,
                                float4* bl, int32_t* status, double* ox, double* oy,
                                double* oz) {
  const double eps2 = eps * eps;
  const F64Plan plan = f64_plan(n, nslices);
  const bool f64 = precision == PHYS_F64;
  const int64_t slice_len = f64 ? plan.slice_len : f32c_slice_len(n, nslices);
  const int64_t nsl = ceil_div(n, slice_len);
  double* out = nsl > 1 ? part : nullptr;
  const int g = (int)min64(ceil_div(n, 256), 148 * 8);
  if (f64) {
    direct_f64_launch(s, plan, n, 0, n, x, y, z, m, G, eps2, 0, ox, oy, oz, out, status);
  } else {
    launch_kernel(s, g, 256, 0, split_bodies_kernel, n, x, y, z, m, bh, bl, status);
    launch_f32c(s, n, 0, n, slice_len, bh, bl, m, G, (float)eps2, 0, ox, oy, oz, out, status);
  }
  if (nsl > 1)
    launch_kernel(s, (int)min64(ceil_div(3 * n, 256), 148 * 8), 256, 0, slice_reduce_kernel, n,
                  0, n, nsl, part, m, G, 0, ox, oy, oz, status);
  return cudaGetLastError();  // the launch error, if any (and clears it)
}

int direct_targets(phys_ctx* c, const phys_params* p, int64_t nt, const int64_t* d_tidx,
                   double* ox, double* oy, double* oz) {
  const int64_t n = c->n;
  const double eps2 = p->eps * p->eps;
  const bool exact = p->precision == PHYS_F64_EXACT;
  int64_t nsl = 1;
  if (!exact) {
    nsl = ceil_div(148LL * 2048, ceil_div(nt, kTile) * kTile);
    if (nsl > ceil_div(n, kTile)) nsl = ceil_div(n, kTile);
    if (nsl < 1) nsl = 1;
  }
  const int64_t slice_len = ceil_div(ceil_div(n, nsl), kTile) * kTile;
  nsl = ceil_div(n, slice_len);
  int st = PHYS_OK;
  double* part = (double*)ws_get(c, WS_DIRECT_PART, sizeof(double) * 3 * nt * nsl, &st);
  if (st) return st;
  dim3 grid((unsigned)ceil_div(nt, kTile), (unsigned)nsl);
  PHYS_LAUNCH(c, direct_targets_kernel, grid, kTile, 0, n, nt, d_tidx, slice_len, c->x, c->y,
              c->z, c->m, p->G, eps2, (int)exact, part, ox, oy, oz, c->d_status);
  if (!exact) {
    int g = (int)min64(ceil_div(3 * nt, 256), 148 * 8);
    PHYS_LAUNCH(c, slice_reduce_kernel, g, 256, 0, nt, 0, nt, (int)nsl, part, c->m, p->G, 0, ox,
                oy, oz, c->d_status);
  }
  return PHYS_OK;
}

}  // namespace phys

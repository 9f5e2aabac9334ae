// K9: hand-written adjoint of the direct-sum acceleration and the
// Velocity-Verlet step (integrators.rs:63-104 with gravity.rs:53-69 and
// a = F/m), for the gradient of a trajectory loss
//     L = sum_i |x_i(T) - target_i|^2
// with respect to initial positions, velocities and masses.
//
// Forward program (f64, the sliced direct sum of direct.cu):
//     a_0 = A(x_0)
//     x_{k+1} = x_k + (v_k dt + a_k dt^2/2)
//     a_{k+1} = A(x_{k+1})
//     v_{k+1} = v_k + (a_k + a_{k+1}) dt/2
// Reverse sweep (bars are adjoints), k = T-1 .. 0:
//     abar_{k+1} += (dt/2) vbar_{k+1}
//     xbar_{k+1} += J(x_{k+1})^T abar_{k+1};  mbar += (dA/dm)^T abar_{k+1}
//     abar_k      = (dt/2) vbar_{k+1} + (dt^2/2) xbar_{k+1}
//     vbar_k      = vbar_{k+1} + dt xbar_{k+1};  xbar_k = xbar_{k+1}
// then xbar_0 += J(x_0)^T abar_0, mbar += (dA/dm)^T abar_0.
// With a_i = G sum_{j != i} m_j r_ij / s^3 (r_ij = x_j - x_i,
// s^2 = |r_ij|^2 + eps^2) and K_ij = I/s^3 - 3 r r^T / s^5 (symmetric):
//     (J^T w)_j = G sum_{i != j} K_ij (m_j w_i - m_i w_j)
//     (dA/dm)^T w)_j = G sum_{i != j} (r_ij . w_i) / s^3
// Positions are kept for a whole segment of steps (the trajectory, where it
// fits in kHistoryBytes and can be allocated; else `checkpoint` steps, with
// (x, v) kept at the segment starts and the segments before the last recomputed,
// deterministically, bit for bit, during the reverse sweep).
//
// A forward step is two kernels, the sliced force sum and one that adds up the
// slices and performs the velocity step and the next position step; a reverse
// step is two as well, the VJP and one that adds up its slices and updates
// xbar, abar and vbar for the next step.  4096 bodies, 100 steps:
// 14.1 -> 7.7 ms per gradient (31 us per VJP and 17 per force sum of FP64
// arithmetic at the pipe's rate, of 74 us per step).
#include <algorithm>
#include <vector>

#include "common.cuh"

namespace phys {
namespace {

constexpr int kTile = 128;
constexpr int kBlock = 256;

int grid_for(int64_t n) { return (int)std::min<int64_t>(std::max<int64_t>(ceil_div(n, kBlock), 1), 148 * 8); }

// x += v dt + a dt^2/2 ; per component arrays of n; also written to `hist`.
__global__ void adj_drift(int64_t n, double dt, double* __restrict__ x,
                          const double* __restrict__ v, const double* __restrict__ a,
                          double* __restrict__ hist) {
  wait_for_previous();
  const double h2 = xmul(xmul(0.5, dt), dt);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 3 * n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double x1 = xadd(x[i], xadd(xmul(v[i], dt), xmul(a[i], h2)));
    x[i] = x1;
    if (hist) hist[i] = x1;
  }
}

// a = G sum_slices; v += (a_old + a) dt/2; with kDrift the next position
// step: x += v dt + a dt^2/2, also written to `hist`.  One thread per (body,
// component).
template <bool kDrift>
__global__ void __launch_bounds__(kBlock)
adj_kick(int64_t n, int nsl, const double* __restrict__ part, double G, double dt,
         double* __restrict__ x, double* __restrict__ v, double* __restrict__ a,
         double* __restrict__ hist, int32_t* status) {
  wait_for_previous();
  const double hdt = xmul(0.5, dt), h2 = xmul(xmul(0.5, dt), dt);
  bool bad = false;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 3 * n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const double a1 = slice_sum(part + e, 3 * (size_t)n, nsl) * G;
    const double v1 = xadd(v[e], xmul(xadd(a[e], a1), hdt));
    v[e] = v1;
    a[e] = a1;
    if (kDrift) {
      const double x1 = xadd(x[e], xadd(xmul(v1, dt), xmul(a1, h2)));
      x[e] = x1;
      if (hist) hist[e] = x1;
    }
    bad |= !isfinite(a1);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, kStatNonfinite);
}

// a = G sum_slices.
__global__ void __launch_bounds__(kBlock)
adj_accel(int64_t n, int nsl, const double* __restrict__ part, double G, double* __restrict__ a,
          int32_t* status) {
  wait_for_previous();
  bool bad = false;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 3 * n;
       e += (int64_t)gridDim.x * blockDim.x) {
    a[e] = slice_sum(part + e, 3 * (size_t)n, nsl) * G;
    bad |= !isfinite(a[e]);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, kStatNonfinite);
}

// Per-block partial sums of (x - t)^2 and xbar = 2 (x - t).
__global__ void loss_kernel(int64_t n, const double* __restrict__ x,
                            const double* __restrict__ t, double* __restrict__ xbar,
                            double* __restrict__ part) {
  wait_for_previous();
  __shared__ double sh[kBlock];
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 3 * n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double d = x[i] - t[i];
    s = fma(d, d, s);
    if (xbar) xbar[i] = 2.0 * d;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int k = kBlock / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) sh[threadIdx.x] += sh[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void sum_kernel(int nparts, const double* __restrict__ part, double* __restrict__ out) {
  wait_for_previous();
  if (threadIdx.x != 0) return;
  double s = 0.0;
  for (int b = 0; b < nparts; ++b) s += part[b];
  out[0] = s;
}

// VJP of the acceleration at positions (x, y, z) with weights w (SoA, n
// each): per target j and source slice, partial (ux, uy, uz, gm).  Two
// targets per thread: a source (four 16-byte broadcasts from shared memory, 16
// cycles a warp) serves two terms of 35 FP64 operations (17.5 cycles each).
constexpr int kVThreads = 64;
constexpr int kVT = 2;

template <bool kChecked>
__device__ __forceinline__ void vjp_tile(const double4* __restrict__ ts,
                                         const double4* __restrict__ tw, int cnt,
                                         const int (&self)[kVT], const double4 (&xj)[kVT],
                                         const double4 (&wj)[kVT], double eps2,
                                         double4 (&u)[kVT]) {
#pragma unroll 2
  for (int k = 0; k < cnt; ++k) {
    const double4 s = ts[k];
    const double4 w = tw[k];
#pragma unroll
    for (int q = 0; q < kVT; ++q) {
      // r_ij = x_j - x_i
      const double rx = xj[q].x - s.x, ry = xj[q].y - s.y, rz = xj[q].z - s.z;
      double s2 = fma(rx, rx, fma(ry, ry, fma(rz, rz, eps2)));
      if (kChecked && k == self[q]) s2 = 1.0;
      const double inv = inv_root(s2);
      const double inv2 = inv * inv;
      double inv3 = inv2 * inv;
      if (kChecked && k == self[q]) inv3 = 0.0;
      // q = m_j w_i - m_i w_j ; K q = q / s^3 - 3 r (r . q) / s^5
      const double qx = fma(xj[q].w, w.x, -(s.w * wj[q].x));
      const double qy = fma(xj[q].w, w.y, -(s.w * wj[q].y));
      const double qz = fma(xj[q].w, w.z, -(s.w * wj[q].z));
      const double c = -3.0 * (inv3 * inv2) * fma(rx, qx, fma(ry, qy, rz * qz));
      u[q].x = fma(rx, c, fma(qx, inv3, u[q].x));
      u[q].y = fma(ry, c, fma(qy, inv3, u[q].y));
      u[q].z = fma(rz, c, fma(qz, inv3, u[q].z));
      u[q].w = fma(fma(rx, w.x, fma(ry, w.y, rz * w.z)), inv3, u[q].w);
    }
  }
}

__global__ void __launch_bounds__(kVThreads)
vjp_kernel(int64_t n, int64_t slice_len, const double* __restrict__ x,
           const double* __restrict__ y, const double* __restrict__ z,
           const double* __restrict__ m, const double* __restrict__ wx,
           const double* __restrict__ wy, const double* __restrict__ wz, double eps2,
           double* __restrict__ part) {
  wait_for_previous();
  __shared__ double4 ts[kTile];
  __shared__ double4 tw[kTile];
  const int64_t tbase = blockIdx.x * (int64_t)(kVThreads * kVT);
  double4 xj[kVT], wj[kVT], u[kVT];
#pragma unroll
  for (int q = 0; q < kVT; ++q) {
    const int64_t j = tbase + threadIdx.x + q * kVThreads;
    const double4 zero = make_double4(0, 0, 0, 0);
    xj[q] = j < n ? make_double4(x[j], y[j], z[j], m[j]) : zero;
    wj[q] = j < n ? make_double4(wx[j], wy[j], wz[j], 0.0) : zero;
    const double s = sum_start(eps2);
    u[q] = make_double4(s, s, s, s);
  }
  const int64_t lo = blockIdx.y * slice_len;
  const int64_t hi = min64(n, lo + slice_len);
  for (int64_t base = lo; base < hi; base += kTile) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kTile / kVThreads; ++r) {
      const int k = threadIdx.x + r * kVThreads;
      const int64_t i = base + k;
      if (i < hi) {
        ts[k] = make_double4(x[i], y[i], z[i], m[i]);
        tw[k] = make_double4(wx[i], wy[i], wz[i], 0.0);
      }
    }
    __syncthreads();
    const int cnt = (int)min64(kTile, hi - base);
    int self[kVT];
#pragma unroll
    for (int q = 0; q < kVT; ++q) {
      const int64_t d = tbase + threadIdx.x + q * kVThreads - base;
      self[q] = d >= 0 && d < kTile ? (int)d : -1;
    }
    if (base < tbase + kVThreads * kVT && base + kTile > tbase)
      vjp_tile<true>(ts, tw, cnt, self, xj, wj, eps2, u);
    else
      vjp_tile<false>(ts, tw, cnt, self, xj, wj, eps2, u);
  }
  double* p = part + (size_t)blockIdx.y * 4 * n;
#pragma unroll
  for (int q = 0; q < kVT; ++q) {
    const int64_t j = tbase + threadIdx.x + q * kVThreads;
    if (j >= n) continue;
    p[j] = u[q].x;
    p[n + j] = u[q].y;
    p[2 * n + j] = u[q].z;
    p[3 * n + j] = u[q].w;
  }
}

// xbar += G sum_slices u ; mbar += G sum_slices gm (slice order fixed), one
// thread per (body, component).  kPost: the rest of the reverse step,
// abar = h vbar + h2 xbar ; vbar += dt xbar, and with `pre` the next one's
// abar += h vbar.
template <bool kPost>
__global__ void __launch_bounds__(kBlock)
vjp_reduce(int64_t n, int nsl, const double* __restrict__ part, double G, double dt, int pre,
           double* __restrict__ xbar, double* __restrict__ mbar, double* __restrict__ vbar,
           double* __restrict__ abar) {
  wait_for_previous();
  const double h = 0.5 * dt, h2 = 0.5 * dt * dt;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 4 * n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const double u = slice_sum(part + e, 4 * (size_t)n, nsl);
    if (e >= 3 * n) {
      mbar[e - 3 * n] += G * u;
      continue;
    }
    const double xb = xbar[e] + G * u;
    xbar[e] = xb;
    if (kPost) {
      const double vb = vbar[e], vn = fma(dt, xb, vb);
      const double ab = fma(h, vb, h2 * xb);
      vbar[e] = vn;
      abar[e] = pre ? fma(h, vn, ab) : ab;
    }
  }
}

// Room for the positions of every step (24 bytes per body and step).
constexpr int64_t kHistoryBytes = int64_t(256) << 20;

struct Adj {
  int64_t n, T, K, nck;      // bodies, steps, steps per segment, segments
  double *X, *V, *A;         // 3n each
  double *ckpt;              // nck * 6n
  double *seg;               // (K+1) * 3n: positions of a segment's steps
  double *xbar, *vbar, *abar, *mbar, *tgt;
  double *fpart, *vpart, *lpart, *loss;
  F64Plan plan;              // slices of the force sum and of the VJP
};

// Slice partials of the force at a.X.
int force(phys_ctx* c, const phys_params* p, Adj& a) {
  const int64_t n = a.n;
  direct_f64_launch(c->stream, a.plan, n, 0, n, a.X, a.X + n, a.X + 2 * n, c->m, p->G,
                    p->eps * p->eps, 0, nullptr, nullptr, nullptr, a.fpart, c->d_status);
  c->launches++;
  return check_launch(c, "adjoint force");
}

// `len` steps from (X, V, A); the positions after step j to hist + 3n j.
int steps(phys_ctx* c, const phys_params* p, Adj& a, double dt, int64_t len, double* hist) {
  const int64_t n = a.n;
  auto at = [&](int64_t j) { return hist ? hist + 3 * n * j : nullptr; };
  const int g = grid_for(3 * n), nsl = (int)a.plan.slices;
  for (int64_t j = 0; j < len; ++j) {
    if (j == 0) PHYS_LAUNCH(c, adj_drift, g, kBlock, 0, n, dt, a.X, a.V, a.A, at(0));
    PHYS_TRY(force(c, p, a));
    if (j + 1 < len)
      PHYS_LAUNCH(c, adj_kick<true>, g, kBlock, 0, n, nsl, a.fpart, p->G, dt, a.X, a.V, a.A,
                  at(j + 1), c->d_status);
    else
      PHYS_LAUNCH(c, adj_kick<false>, g, kBlock, 0, n, nsl, a.fpart, p->G, dt, a.X, a.V, a.A,
                  nullptr, c->d_status);
  }
  return PHYS_OK;
}

int accel(phys_ctx* c, const phys_params* p, Adj& a) {  // a.A at a.X
  PHYS_TRY(force(c, p, a));
  PHYS_LAUNCH(c, adj_accel, grid_for(3 * a.n), kBlock, 0, a.n, (int)a.plan.slices, a.fpart, p->G,
              a.A, c->d_status);
  return PHYS_OK;
}

int vjp(phys_ctx* c, const phys_params* p, Adj& a, const double* x) {
  const int64_t n = a.n;
  dim3 grid((unsigned)ceil_div(n, kVThreads * kVT), (unsigned)a.plan.slices);
  PHYS_LAUNCH(c, vjp_kernel, grid, kVThreads, 0, n, a.plan.slice_len, x, x + n, x + 2 * n, c->m,
              a.abar, a.abar + n, a.abar + 2 * n, p->eps * p->eps, a.vpart);
  return PHYS_OK;
}

// Everything but the partial sums, for segments of K steps.
int setup_segments(phys_ctx* c, int64_t K, bool reverse, Adj& a) {
  const int64_t n = a.n, T = a.T;
  a.K = reverse ? std::min<int64_t>(K, std::max<int64_t>(T, 1)) : 0;
  a.nck = reverse ? std::max<int64_t>(ceil_div(T, a.K), 1) : 0;
  const size_t doubles = 9 * n + a.nck * 6 * n + (a.K + 1) * 3 * n + 13 * n;
  int st = PHYS_OK;
  double* b = (double*)ws_get(c, WS_ADJ0, sizeof(double) * doubles, &st);
  if (st) return st;
  a.X = b; b += 3 * n;
  a.V = b; b += 3 * n;
  a.A = b; b += 3 * n;
  a.ckpt = b; b += a.nck * 6 * n;
  a.seg = b; b += (a.K + 1) * 3 * n;
  a.xbar = b; b += 3 * n;
  a.vbar = b; b += 3 * n;
  a.abar = b; b += 3 * n;
  a.mbar = b; b += n;
  a.tgt = b; b += 3 * n;
  return PHYS_OK;
}

int setup(phys_ctx* c, int64_t T, int64_t K, bool reverse, Adj& a) {
  const int64_t n = c->n;
  a.n = n;
  a.T = T;
  a.plan = f64_plan(n, INT64_MAX);
  int st = PHYS_OK;
  a.fpart = (double*)ws_get(c, WS_ADJ1, sizeof(double) * 3 * n * a.plan.slices, &st);
  if (st) return st;
  a.vpart = (double*)ws_get(c, WS_ADJ2, sizeof(double) * 4 * n * a.plan.slices, &st);
  if (st) return st;
  a.lpart = (double*)ws_get(c, WS_ADJ3, sizeof(double) * (148 * 8 + 8), &st);
  if (st) return st;
  a.loss = a.lpart + 148 * 8;
  if (reverse && K < T && (T + 1) * 3 * n * (int64_t)sizeof(double) <= kHistoryBytes) {
    st = setup_segments(c, T, reverse, a);
    if (st != PHYS_ERR_OOM) return st;
    c->err.clear();  // no room for every step: the caller's interval
  }
  return setup_segments(c, K, reverse, a);
}

int copy_d2d(phys_ctx* c, double* dst, const double* src, int64_t count) {
  PHYS_CUDA(c, cudaMemcpyAsync(dst, src, sizeof(double) * count, cudaMemcpyDeviceToDevice,
                               c->stream));
  return PHYS_OK;
}

// x0, v0 of the context state into a.X, a.V (SoA blocks of 3n).
int load_initial(phys_ctx* c, Adj& a) {
  const int64_t n = a.n;
  PHYS_TRY(copy_d2d(c, a.X, c->x, n));
  PHYS_TRY(copy_d2d(c, a.X + n, c->y, n));
  PHYS_TRY(copy_d2d(c, a.X + 2 * n, c->z, n));
  PHYS_TRY(copy_d2d(c, a.V, c->vx, n));
  PHYS_TRY(copy_d2d(c, a.V + n, c->vy, n));
  PHYS_TRY(copy_d2d(c, a.V + 2 * n, c->vz, n));
  return PHYS_OK;
}

// The whole trajectory; with checkpoints, (x, v) at the segment starts and
// the last segment's positions.
int forward(phys_ctx* c, const phys_params* p, Adj& a, double dt, bool keep_ckpt) {
  const int64_t n = a.n;
  PHYS_TRY(load_initial(c, a));
  PHYS_TRY(accel(c, p, a));
  if (!keep_ckpt) return steps(c, p, a, dt, a.T, nullptr);
  for (int64_t k0 = 0; k0 < a.T; k0 += a.K) {
    double* ck = a.ckpt + (k0 / a.K) * 6 * n;
    PHYS_TRY(copy_d2d(c, ck, a.X, 3 * n));
    PHYS_TRY(copy_d2d(c, ck + 3 * n, a.V, 3 * n));
    const bool last = k0 + a.K >= a.T;
    if (last) PHYS_TRY(copy_d2d(c, a.seg, a.X, 3 * n));
    PHYS_TRY(steps(c, p, a, dt, std::min<int64_t>(a.K, a.T - k0), last ? a.seg + 3 * n : nullptr));
  }
  return PHYS_OK;
}

int loss_of(phys_ctx* c, Adj& a, bool grad, double* out) {
  const int g = grid_for(3 * a.n);
  PHYS_LAUNCH(c, loss_kernel, g, kBlock, 0, a.n, a.X, a.tgt, grad ? a.xbar : nullptr, a.lpart);
  PHYS_LAUNCH(c, sum_kernel, 1, 32, 0, g, a.lpart, a.loss);
  PHYS_CUDA(c, cudaMemcpyAsync(out, a.loss, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  return PHYS_OK;
}

int check_args(phys_ctx* c, const phys_params* p, int64_t nsteps, int64_t K, const double* tx,
               const double* ty, const double* tz) {
  if (!p) return fail(c, PHYS_ERR_ARG, "params is NULL");
  if (p->precision != PHYS_F64) return fail(c, PHYS_ERR_ARG, "adjoint runs in PHYS_F64");
  if (nsteps < 0 || K <= 0) return fail(c, PHYS_ERR_ARG, "nsteps >= 0 and checkpoint > 0");
  if (!tx || !ty || !tz) return fail(c, PHYS_ERR_ARG, "targets are required");
  if (c->n < 2) return fail(c, PHYS_ERR_STATE, "need at least 2 bodies");
  return PHYS_OK;
}

int upload_targets(phys_ctx* c, Adj& a, const double* tx, const double* ty, const double* tz) {
  const int64_t n = a.n;
  PHYS_CUDA(c, cudaMemcpyAsync(a.tgt, tx, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
  PHYS_CUDA(c, cudaMemcpyAsync(a.tgt + n, ty, sizeof(double) * n, cudaMemcpyHostToDevice,
                               c->stream));
  PHYS_CUDA(c, cudaMemcpyAsync(a.tgt + 2 * n, tz, sizeof(double) * n, cudaMemcpyHostToDevice,
                               c->stream));
  return PHYS_OK;
}

}  // namespace

int trajectory_loss(phys_ctx* c, const phys_params* p, double dt, int64_t nsteps,
                    const double* tx, const double* ty, const double* tz, double* loss,
                    double* xT, double* yT, double* zT) {
  PHYS_TRY(check_args(c, p, nsteps, 1, tx, ty, tz));
  Adj a{};
  PHYS_TRY(setup(c, nsteps, 1, false, a));
  PHYS_TRY(upload_targets(c, a, tx, ty, tz));
  PHYS_TRY(forward(c, p, a, dt, false));
  double l = 0.0;
  PHYS_TRY(loss_of(c, a, false, &l));
  double* outs[3] = {xT, yT, zT};
  for (int k = 0; k < 3; ++k)
    if (outs[k])
      PHYS_CUDA(c, cudaMemcpyAsync(outs[k], a.X + k * a.n, sizeof(double) * a.n,
                                   cudaMemcpyDeviceToHost, c->stream));
  PHYS_CUDA(c, cudaStreamSynchronize(c->stream));
  *loss = l;
  return PHYS_OK;
}

int adjoint(phys_ctx* c, const phys_params* p, double dt, int64_t nsteps, int64_t K,
            const double* tx, const double* ty, const double* tz, double* loss, double* gxyz[3],
            double* gvxyz[3], double* gm) {
  PHYS_TRY(check_args(c, p, nsteps, K, tx, ty, tz));
  Adj a{};
  PHYS_TRY(setup(c, nsteps, K, true, a));
  const int64_t n = a.n;
  PHYS_TRY(upload_targets(c, a, tx, ty, tz));
  PHYS_TRY(forward(c, p, a, dt, true));
  double l = 0.0;
  PHYS_TRY(loss_of(c, a, true, &l));  // xbar = dL/dx_T
  PHYS_CUDA(c, cudaMemsetAsync(a.vbar, 0, sizeof(double) * 3 * n, c->stream));
  PHYS_CUDA(c, cudaMemsetAsync(a.abar, 0, sizeof(double) * 3 * n, c->stream));
  PHYS_CUDA(c, cudaMemsetAsync(a.mbar, 0, sizeof(double) * n, c->stream));
  const int nsl = (int)a.plan.slices, g4 = grid_for(4 * n);
  // abar_T = 0 + (dt/2) vbar_T = 0: nothing to add before the first step
  for (int64_t s = a.nck - 1; s >= 0 && a.T > 0; --s) {
    const int64_t k0 = s * a.K;
    const int64_t len = std::min<int64_t>(a.K, a.T - k0);
    if (s + 1 < a.nck) {  // recompute the segment: seg[j] = x_{k0 + j}
      const double* ck = a.ckpt + s * 6 * n;
      PHYS_TRY(copy_d2d(c, a.X, ck, 3 * n));
      PHYS_TRY(copy_d2d(c, a.V, ck + 3 * n, 3 * n));
      PHYS_TRY(copy_d2d(c, a.seg, ck, 3 * n));
      PHYS_TRY(accel(c, p, a));
      PHYS_TRY(steps(c, p, a, dt, len, a.seg + 3 * n));
    }
    for (int64_t j = len - 1; j >= 0; --j) {  // reverse of step k = k0 + j
      PHYS_TRY(vjp(c, p, a, a.seg + (j + 1) * 3 * n));
      PHYS_LAUNCH(c, vjp_reduce<true>, g4, kBlock, 0, n, nsl, a.vpart, p->G, dt,
                  (int)(k0 + j > 0), a.xbar, a.mbar, a.vbar, a.abar);
    }
  }
  // a_0 = A(x_0)
  PHYS_TRY(load_initial(c, a));
  PHYS_TRY(vjp(c, p, a, a.X));
  PHYS_LAUNCH(c, vjp_reduce<false>, g4, kBlock, 0, n, nsl, a.vpart, p->G, dt, 0, a.xbar, a.mbar,
              a.vbar, a.abar);
  for (int k = 0; k < 3; ++k) {
    if (gxyz[k])
      PHYS_CUDA(c, cudaMemcpyAsync(gxyz[k], a.xbar + k * n, sizeof(double) * n,
                                   cudaMemcpyDeviceToHost, c->stream));
    if (gvxyz[k])
      PHYS_CUDA(c, cudaMemcpyAsync(gvxyz[k], a.vbar + k * n, sizeof(double) * n,
                                   cudaMemcpyDeviceToHost, c->stream));
  }
  if (gm)
    PHYS_CUDA(c, cudaMemcpyAsync(gm, a.mbar, sizeof(double) * n, cudaMemcpyDeviceToHost,
                                 c->stream));
  PHYS_CUDA(c, cudaStreamSynchronize(c->stream));
  *loss = l;
  return PHYS_OK;
}

}  // namespace phys

// Reference-form centre of mass (gravity_tree.rs:113-118) of cells of many
// bodies: com <- (com M + x m) / (M + m) per body in insertion order, every
// operation rounded, a chain that no reordering may shorten without changing
// the bits.  The chain is cut into segments that run at the same time.
//
// Running masses (segment_mass_kernel, mass_stitch_kernel).  While M stays in
// one binade, adding an even number of its ulps to M shifts every later
// RN(M + m) by the same amount (a tie goes to the even neighbour either way).
// A segment is summed from an approximate start and from the next double, and
// the one of the true start's parity, shifted, is the true sum; a segment
// that crosses into another binade is summed again from the true start.
//
// Centre of mass.  The reference's value at a segment's start is the exact
// mean of the bodies so far plus the roundings it has gathered, of the order
// of u |com| sqrt(k) after k bodies (u = 2^-53).  Most of what a segment adds
// to that does not depend on the value that it starts from, so
// first_pass_kernel runs every segment from the mean and predict_kernel adds
// up the differences; what is left is some tens of ulps (110 at most in
// chains of 3 x 10^5 bodies).  segment_kernel then runs each segment from
// every double in a window around the prediction.  A step is monotone in com
// (a product with M > 0, a sum and a quotient by M' > 0, each rounded to
// nearest), so the candidates stay in order and those that have met stay
// together: where the steps' roundings differ between neighbours a few dozen
// values are left after some hundred steps, and only these go on; where they
// do not, the prediction is close.  stitch_kernel follows the true value from
// segment to segment by looking its candidate up: the candidate's end is the
// reference's, bit for bit.  Where it has none, refine_kernel goes on from an
// estimate, and the segments it found outside their windows are run again
// around where it passed them (twice, for the longest chains); what is left
// then is run from the true value in turn.
//
// The division is by a precomputed reciprocal (div_recip).  A candidate that
// leaves its range ends as NaN and counts as unknown: in a plane the centre of
// mass is 0, in range, and its neighbours are not.  Only a segment whose
// running masses, or whose true value, leave the range is run with the IEEE
// division, by itself.  Masses of both signs have the same steps wherever the
// running mass is positive; their running masses are summed in turn.
//
// Tree phase of an exact evaluation, one chain per cell before against
// segments: Plummer spheres of 10 000 bodies 0.82 -> 0.35 ms, 100 000 4.2 ->
// 1.28 ms, 300 000 7.3 -> 2.1 ms, 2^20 16.1 -> 8.6 and 18.3 -> 9.9 ms (two
// seeds; the longest chain decides); in a plane 0.84 -> 0.46, 4.4 -> 1.5 and
// 25.6 -> 9.3 ms at 10 000, 100 000 and 2^20; masses of both signs 7.0 -> 3.3
// and 66 -> 33 ms at 100 000 and 2^20.  The candidates' steps bound it: 7 FP64
// operations each, a dependent chain of 57 cycles a body.
#include "bh.cuh"

namespace phys {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kCand = 512;   // candidates per segment and coordinate, at most
constexpr int kRound = 256;  // steps between two looks at which have met

// Bodies per segment: a power of two, about a hundredth of the longest chain.
int segment_len(int64_t n) {
  int len = 256;
  while ((int64_t)len * 2 <= n / 256) len *= 2;
  return len;
}

struct LongCells {
  int64_t nnodes;
  int len;               // bodies per segment
  const int32_t* eoff;   // node -> first (cell, body) pair
  const double4* eb;     // bodies in pair order (x, y, z, m)
  const TreeHeader* hdr;
  const int32_t* longs;  // nodes of the long cells, count in longs[nnodes]
  double4* mc;           // result per node
  int32_t* ctr;          // [0] segments, [1] segments with candidates
  int2* first;           // per long cell: its first segment, first candidate slot
  int2* seg;             // per segment: long cell, number within it
  double4* sum;          // per segment: sum of m x, m y, m z, m
  double4* start;        // per segment: com x, y, z and running mass at its start
                         // (first the sums before it, then the mean, then the
                         // prediction)
  double2* mass_end;     // per segment: masses at its end from the two starts
  int32_t* bad;          // per segment: its masses (for a cell's first segment, its
                         // steps) leave div_recip's range
  int32_t* redo;         // per segment: coordinates to run again (bits 0-2)
  double4* pass;         // per segment: com at its end from the mean
  double* end;           // per candidate slot: com at the segment's end, [3][kCand]; NaN
                         // where the candidate left div_recip's range
  const int32_t* status;
};

__device__ __forceinline__ int long_count(const LongCells& a) {
  return min(a.longs[a.nnodes], (int32_t)a.nnodes);
}
__device__ __forceinline__ double next_up(double v) {  // v >= 0
  return __longlong_as_double(__double_as_longlong(v) + 1);
}

// The candidates at the start of a cell's segment s: consecutive doubles
// around its prediction (few where that is the true value, s = 1, or 0: then
// the bodies lie in a plane, and its neighbours are out of range).
struct Window {
  double mid, ulp;
  int n;
  __device__ __forceinline__ Window(double m, int s, int64_t len)
      : mid(m), ulp(xsub(next_up(fabs(m)), fabs(m))),
        n(s == 1 || m == 0.0 ? 32
          : s * len < 8192   ? kCand / 4
          : s * len < 100000 ? kCand / 2
                             : kCand) {}
  __device__ __forceinline__ double at(int i) const {
    return xadd(mid, xmul((double)(i - n / 2), ulp));
  }
  // the last candidate not above c, in [0, n - 2]
  __device__ __forceinline__ int find(double c) const {
    int lo = (int)fmin(fmax(floor((c - mid) / ulp) + n / 2, 0.0), (double)(n - 2));
    while (lo > 0 && at(lo) > c) --lo;
    while (lo < n - 2 && at(lo + 1) <= c) ++lo;
    return lo;
  }
};

__global__ void segments_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  const int nl = long_count(a);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nl; i += gridDim.x * blockDim.x) {
    const int k = a.longs[i];
    const int ns = (a.eoff[k + 1] - a.eoff[k] + a.len - 1) / a.len;
    const int base = atomicAdd(&a.ctr[0], ns);
    a.first[i] = make_int2(base, atomicAdd(&a.ctr[1], ns - 1));
    for (int s = 0; s < ns; ++s) a.seg[base + s] = make_int2(i, s);
  }
}

// Ordinary sums of m x and m over each segment, a warp per segment.
__global__ void __launch_bounds__(128) segment_sum_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  const int lane = threadIdx.x & 31, nseg = a.ctr[0];
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < nseg;
       g += (gridDim.x * blockDim.x) >> 5) {
    const int k = a.longs[a.seg[g].x];
    const int64_t e0 = a.eoff[k] + (int64_t)a.seg[g].y * a.len;
    const int64_t e1 = min64(a.eoff[k + 1], e0 + a.len);
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t e = e0 + lane; e < e1; e += 32) {
      const double4 b = a.eb[e];
      s[0] = fma(b.w, b.x, s[0]);
      s[1] = fma(b.w, b.y, s[1]);
      s[2] = fma(b.w, b.z, s[2]);
      s[3] += b.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < 4; ++c) s[c] += __shfl_xor_sync(kFull, s[c], o);
    if (lane == 0) {
      a.sum[g] = make_double4(s[0], s[1], s[2], s[3]);
      a.bad[g] = 0;
    }
  }
}

// The sums before each segment, a warp per long cell (lane c: component c).
__global__ void __launch_bounds__(32) prefix_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  const int lane = threadIdx.x, nl = long_count(a);
  for (int i = blockIdx.x; i < nl; i += gridDim.x) {
    const int k = a.longs[i], base = a.first[i].x;
    const int ns = (a.eoff[k + 1] - a.eoff[k] + a.len - 1) / a.len;
    if (lane < 4) {
      double s = 0.0;
#pragma unroll 8
      for (int g = 0; g < ns; ++g) {
        reinterpret_cast<double*>(&a.start[base + g])[lane] = s;
        s += reinterpret_cast<const double*>(&a.sum[base + g])[lane];
      }
    }
  }
}

// RN sums of the masses eb[e0, e1) onto M in order (warp-collective; lanes
// may differ in M), four batches of 32 masses in flight.
__device__ __forceinline__ double mass_run(const double4* __restrict__ eb, int64_t e0, int64_t e1,
                                           double M, double (&ms)[2][32], int lane) {
  auto load = [&](int64_t e) { return e + lane < e1 ? eb[e + lane].w : 0.0; };
  constexpr int kAhead = 4;
  double v[kAhead];
#pragma unroll
  for (int j = 0; j < kAhead; ++j) v[j] = load(e0 + 32 * j);
  for (int64_t e = e0; e < e1; e += 32 * kAhead) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      ms[j & 1][lane] = v[j];
      __syncwarp();
      v[j] = load(e + 32 * (j + kAhead));
#pragma unroll
      for (int u = 0; u < 32; ++u) M = xadd(M, ms[j & 1][u]);  // past the end: + 0
    }
  }
  __syncwarp();
  return M;
}

__global__ void __launch_bounds__(32) segment_mass_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  __shared__ double ms[2][32];
  const int lane = threadIdx.x, nseg = a.ctr[0];
  for (int g = blockIdx.x; g < nseg; g += gridDim.x) {
    const int k = a.longs[a.seg[g].x];
    const int64_t e0 = a.eoff[k] + (int64_t)a.seg[g].y * a.len;
    const int64_t e1 = min64(a.eoff[k + 1], e0 + a.len);
    const double from = a.start[g].w;
    const double M = mass_run(a.eb, e0, e1, lane & 1 ? next_up(from) : from, ms, lane);
    const double other = __shfl_sync(kFull, M, 1);
    if (lane == 0) a.mass_end[g] = make_double2(M, other);
  }
}

// A warp per long cell: the true running masses and the means at the segment
// starts.
__global__ void __launch_bounds__(32) mass_stitch_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  __shared__ double ms[2][32];
  const int lane = threadIdx.x, nl = long_count(a);
  const bool positive = a.hdr->min_mass >= 0.0;
  for (int i = blockIdx.x; i < nl; i += gridDim.x) {
    const int k = a.longs[i], base = a.first[i].x;
    const int64_t e0 = a.eoff[k], e1 = a.eoff[k + 1];
    const int ns = (int)((e1 - e0 + a.len - 1) / a.len);
    auto expo = [](double v) { return __double2hiint(v) >> 20; };
    double M = 0.0;
    for (int s = 0; s < ns; ++s) {
      const double2 en = a.mass_end[base + s];
      const double from = a.start[base + s].w;
      __syncwarp();
      if (lane < 4) {  // the prefix sums become the means and the true mass
        double* st = reinterpret_cast<double*>(&a.start[base + s]);
        st[lane] = lane == 3 ? M : M > 0.0 ? st[lane] / M : 0.0;
      }
      const bool odd = ((__double_as_longlong(M) ^ __double_as_longlong(from)) & 1) != 0;
      const double f = odd ? next_up(from) : from, e = odd ? en.y : en.x;
      const double to = xadd(e, xsub(M, f));
      const int ex = expo(M);
      if (s == 0 || (positive && expo(f) == ex && expo(e) == ex && expo(to) == ex)) {
        M = s ? to : en.x;  // segment 0 was summed from 0 itself
      } else {
        const int64_t b0 = e0 + (int64_t)s * a.len;
        M = mass_run(a.eb, b0, min64(e1, b0 + a.len), M, ms, lane);
      }
      __syncwarp();
    }
    if (lane == 0) a.mc[k].w = M;
  }
}

// kN bodies of a chain as its steps take them.
template <int kN>
struct Batch {
  double M[kN], nt[kN], y[kN];  // running mass before and after, RN(1 / after)
  double p[3][kN];              // RN(x m) per coordinate
};

// Fills the batch's places [at, at + 32) from a lane's body (warp-collective):
// the running masses in order, the reciprocals on all lanes.  Returns whether
// the lane's mass is in div_recip's range.
template <int kN>
__device__ __forceinline__ bool fill_batch(Batch<kN>& B, int at, double4 body, int cnt, int lane,
                                           double& M) {
  B.p[0][at + lane] = xmul(body.x, body.w);
  B.p[1][at + lane] = xmul(body.y, body.w);
  B.p[2][at + lane] = xmul(body.z, body.w);
  B.y[at + lane] = lane < cnt ? body.w : 0.0;  // the masses, until the reciprocals
  __syncwarp();
  double before = M, after = M;
#pragma unroll
  for (int u = 0; u < 32; ++u) {  // every lane adds, lane u keeps its own
    const double acc = xadd(M, B.y[at + u]);
    if (lane == u) {
      before = M;
      after = acc;
    }
    M = acc;
  }
  __syncwarp();
  B.M[at + lane] = before;
  B.nt[at + lane] = after;
  B.y[at + lane] = __drcp_rn(after);
  return lane >= cnt || div_recip_den_ok(after);
}

// cnt steps of kQ chains; ok: they stayed in div_recip's range.
template <int kQ, int kN>
__device__ __forceinline__ void chain_steps(const Batch<kN>& B, const double* __restrict__ p,
                                            int cnt, double (&c)[kQ], bool& ok) {
  auto step = [&](int u) {
    const double M = B.M[u], nt = B.nt[u], y = B.y[u], pu = p[u];
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      const double t = xadd(xmul(c[q], M), pu);
      ok &= div_recip_num_ok(t);
      c[q] = div_recip(t, nt, y);
    }
  };
  int u = 0;
  for (; u + 8 <= cnt; u += 8) {
#pragma unroll
    for (int v = 0; v < 8; ++v) step(u + v);
  }
  for (; u < cnt; ++u) step(u);
}

// The steps of segment eb[f0, f0 + len) from mass M and com c, lane j < 3
// coordinate j (warp-collective).  masses_ok: of the lane's own bodies.
__device__ __forceinline__ void run_warp(const double4* __restrict__ eb, int64_t f0, int len,
                                         double M, double& c, Batch<32>& B, int lane,
                                         bool& masses_ok, bool& steps_ok) {
  const int j = lane < 3 ? lane : 0;
  const double4 zero = make_double4(0.0, 0.0, 0.0, 0.0);
  double cc[1] = {c};
  masses_ok = true;
  bool ok = true;
  double4 body = lane < len ? eb[f0 + lane] : zero;
  for (int b = 0; b < len; b += 32) {
    const int cnt = min(32, len - b);
    const double4 next = b + 32 + lane < len ? eb[f0 + b + 32 + lane] : zero;
    masses_ok &= fill_batch(B, 0, body, cnt, lane, M);
    __syncwarp();
    chain_steps<1>(B, B.p[j], cnt, cc, ok);
    __syncwarp();
    body = next;
  }
  c = cc[0];
  steps_ok = ok;
}

// Every segment from the mean at its start (the first one of a cell from 0,
// its true start), a warp per segment.
__global__ void __launch_bounds__(32) first_pass_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  __shared__ Batch<32> B;
  const int lane = threadIdx.x, nseg = a.ctr[0];
  for (int g = blockIdx.x; g < nseg; g += gridDim.x) {
    const int2 sg = a.seg[g];
    const int k = a.longs[sg.x];
    const int64_t f0 = a.eoff[k] + (int64_t)sg.y * a.len;
    const int len = (int)min64(a.len, a.eoff[k + 1] - f0);
    const double4 st = a.start[g];
    double c = lane == 0 ? st.x : lane == 1 ? st.y : st.z;
    bool masses_ok, steps_ok;
    run_warp(a.eb, f0, len, st.w, c, B, lane, masses_ok, steps_ok);
    if (lane < 3) reinterpret_cast<double*>(&a.pass[g])[lane] = c;
    // beyond the first segment the steps are a mean's and only predict
    if (__any_sync(kFull, !masses_ok || (sg.y == 0 && !steps_ok)) && lane == 0) a.bad[g] = 1;
  }
}

// The predictions: the segment's end from the mean plus the difference at
// its start, shrunk by the ratio of the masses.  Warp per long cell, lane
// j < 3: coordinate j.
__global__ void __launch_bounds__(32) predict_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  const int lane = threadIdx.x, nl = long_count(a);
  for (int i = blockIdx.x; i < nl; i += gridDim.x) {
    const int k = a.longs[i], base = a.first[i].x;
    const int ns = (a.eoff[k + 1] - a.eoff[k] + a.len - 1) / a.len;
    if (lane < 3) {
      double diff = 0.0, M = 0.0;  // of the true value from the mean, mass
#pragma unroll 4
      for (int s = 1; s < ns; ++s) {
        double* st = reinterpret_cast<double*>(&a.start[base + s]);
        const double mean = st[lane], Ms = st[3];
        double at = reinterpret_cast<const double*>(&a.pass[base + s - 1])[lane] +
                    diff * (M / Ms);
        if (!isfinite(at)) at = mean;  // no mass yet, or out of range
        diff = at - mean;
        M = Ms;
        st[lane] = at;
      }
    }
  }
}

// kQ chains per lane of the places [g, g + 32 kQ) of val[0, live).  A candidate
// that leaves the range, or has, ends as the one NaN; which of a lane's it is
// shows only with one per lane: of several, false and nothing written.
template <int kQ>
__device__ __forceinline__ bool run_places(const Batch<kRound>& B, const double* p, int cnt,
                                           double* val, int g, int live, int lane) {
  double c[kQ];
#pragma unroll
  for (int q = 0; q < kQ; ++q) c[q] = val[min(g + 32 * q + lane, live - 1)];
  bool ok = true;
  chain_steps<kQ>(B, p, cnt, c, ok);
  if (kQ > 1 && __any_sync(kFull, !ok)) return false;
  if (!ok) c[0] = __longlong_as_double(0x7ff8000000000000ll);
  __syncwarp();
#pragma unroll
  for (int q = 0; q < kQ; ++q)
    if (g + 32 * q + lane < live) val[g + 32 * q + lane] = c[q];
  return true;
}

// A block per segment: warps 0-2 run the candidates of x, y and z, warp 3
// prepares the next round's bodies meanwhile.
__global__ void __launch_bounds__(128) segment_kernel(LongCells a, int again) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  __shared__ Batch<kRound> B[2];
  __shared__ double vals[3][kCand];      // the values still apart, in order
  __shared__ uint16_t map[3][kCand];     // candidate -> its place in vals
  __shared__ uint16_t moved[3][kCand];   // place before a look -> place after
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nseg = a.ctr[0];
  for (int g = blockIdx.x; g < nseg; g += gridDim.x) {
    const int2 sg = a.seg[g];
    if (sg.y == 0) continue;  // the first pass started at the true value
    const int redo = again ? a.redo[g] : 7;
    if (!redo || a.bad[g]) continue;
    const int k = a.longs[sg.x];
    const int64_t f0 = a.eoff[k] + (int64_t)sg.y * a.len;
    const int len = (int)min64(a.len, a.eoff[k + 1] - f0);
    const double4 st = a.start[g];
    const int rounds = (len + kRound - 1) / kRound;
    double M = st.w;
    auto fill = [&](int r) {  // round r's bodies into its buffer
      const int cnt = min(kRound, len - r * kRound);
      const double4* eb = a.eb + f0 + (int64_t)r * kRound;
      const double4 zero = make_double4(0.0, 0.0, 0.0, 0.0);
      double4 body = lane < cnt ? eb[lane] : zero;
      for (int j = 0; j < cnt; j += 32) {
        const double4 next = j + 32 + lane < cnt ? eb[j + 32 + lane] : zero;
        fill_batch(B[r & 1], j, body, min(32, cnt - j), lane, M);
        body = next;
      }
    };
    const Window win(w == 0 ? st.x : w == 1 ? st.y : st.z, sg.y, a.len);
    int live = (redo >> w) & 1 ? win.n : 0;
    if (w == 3) {
      fill(0);
    } else {
      for (int i = lane; i < live; i += 32) {
        vals[w][i] = win.at(i);
        map[w][i] = (uint16_t)i;
      }
    }
    __syncthreads();
    for (int r = 0; r < rounds; ++r) {
      if (w == 3) {
        if (r + 1 < rounds) fill(r + 1);
      } else {
        const Batch<kRound>& C = B[r & 1];
        const int cnt = min(kRound, len - r * kRound);
        double* val = vals[w];
        int apart = 0;  // places before this one go one per lane
        for (int g0 = 0; g0 < live;) {
          if (live - g0 > 64 && g0 >= apart) {
            if (run_places<4>(C, C.p[w], cnt, val, g0, live, lane))
              g0 += 128;
            else
              apart = g0 + 128;
          } else if (live - g0 > 32 && g0 >= apart) {
            if (run_places<2>(C, C.p[w], cnt, val, g0, live, lane))
              g0 += 64;
            else
              apart = g0 + 64;
          } else {
            run_places<1>(C, C.p[w], cnt, val, g0, live, lane);
            g0 += 32;
          }
        }
        __syncwarp();
        if (live > 32) {  // keep one place of each run of equal values
          int kept = 0;
          long long last = 0;
          for (int g0 = 0; g0 < live; g0 += 32) {
            const int i = g0 + lane;
            const double v = val[min(i, live - 1)];
            const long long bits = __double_as_longlong(v), up = __shfl_up_sync(kFull, bits, 1);
            const bool first = i < live && (i == 0 || bits != (lane ? up : last));
            const unsigned m = __ballot_sync(kFull, first);
            const int place = kept + __popc(m & (0xffffffffu >> (31 - lane))) - 1;
            last = __shfl_sync(kFull, bits, 31);
            if (i < live) moved[w][i] = (uint16_t)place;
            if (first) val[place] = v;
            kept += __popc(m);
            __syncwarp();
          }
          if (kept < live) {
            for (int i = lane; i < win.n; i += 32) map[w][i] = moved[w][map[w][i]];
            live = kept;
          }
          __syncwarp();
        }
      }
      __syncthreads();
    }
    if (live > 0) {
      double* out = a.end + ((size_t)(a.first[sg.x].y + sg.y - 1) * 3 + w) * kCand;
      for (int i = lane; i < win.n; i += 32) out[i] = vals[w][map[w][i]];
    }
    __syncthreads();
  }
}

// The reference's form over a segment, from mass M and com c: the fallback.
// Lane j < 3: coordinate j; the others return lane 0's.
__device__ double segment_ieee(const double4* __restrict__ eb, int64_t f0, int len, double M,
                               double c, double4* rec, int lane) {
  for (int b = 0; b < len; b += 32) {
    __syncwarp();
    if (b + lane < len) rec[lane] = eb[f0 + b + lane];
    __syncwarp();
    const int cnt = min(32, len - b);
    if (lane < 3) {
      const double* q = reinterpret_cast<const double*>(rec);
      for (int u = 0; u < cnt; ++u) {
        const double p = q[4 * u + lane], mm = q[4 * u + 3];
        const double nt = xadd(M, mm);
        if (nt > 0.0) c = xdiv(xadd(xmul(c, M), xmul(p, mm)), nt);
        M = nt;
      }
    }
  }
  __syncwarp();
  return __shfl_sync(kFull, c, lane < 3 ? lane : 0);
}

// Whether one of the segments [g0, g0 + ns) is marked (warp-collective).
__device__ __forceinline__ bool any_segment_bad(const LongCells& a, int g0, int ns, int lane) {
  int bad = 0;
  for (int g = lane; g < ns; g += 32) bad |= a.bad[g0 + g];
  return __any_sync(kFull, bad != 0);
}

// A warp per long cell follows the true value through the segments, or past
// a segment whose candidates do not hold it an estimate, and leaves the
// segments to run again with their new middles.  Lane j < 3: coordinate j.
__global__ void __launch_bounds__(32) refine_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  const int lane = threadIdx.x, nl = long_count(a);
  const int j = lane < 3 ? lane : 0;
  for (int i = blockIdx.x; i < nl; i += gridDim.x) {
    const int k = a.longs[i];
    const int2 first = a.first[i];
    const int ns = (a.eoff[k + 1] - a.eoff[k] + a.len - 1) / a.len;
    const bool any_bad = any_segment_bad(a, first.x, ns, lane);
    double c = reinterpret_cast<const double*>(&a.pass[first.x])[j];
    for (int s = 1; s < ns; ++s) {
      double* st = reinterpret_cast<double*>(&a.start[first.x + s]);
      auto predicted = [&]() { return s + 1 < ns ? st[4 + j] : 0.0; };  // at its end
      if (any_bad && a.bad[first.x + s]) {
        if (lane == 0) a.redo[first.x + s] = 0;
        c = predicted();
        continue;
      }
      const Window win(st[j], s, a.len);
      const int lo = win.find(c);
      const double* en = a.end + ((size_t)(first.y + s - 1) * 3 + j) * kCand + lo;
      const double cl = win.at(lo), ch = win.at(lo + 1), el = en[0], eh = en[1];
      const bool in = cl <= c && c <= ch;
      const unsigned out = __ballot_sync(kFull, !in) & 7u;
      if (!in && lane < 3) st[j] = c;
      if (lane == 0) a.redo[first.x + s] = (int)out;
      // outside the window: the nearer end, shifted
      c = in ? (c == ch ? eh : el) : c < cl ? el + (c - cl) : eh + (c - ch);
      if (!isfinite(c)) c = predicted();  // left the range
    }
  }
}

// A warp per long cell follows the true value; lane j < 3: coordinate j.
__global__ void __launch_bounds__(32) stitch_kernel(LongCells a) {
  wait_for_previous();
  if (sort_failed(a.status)) return;
  __shared__ Batch<32> B;
  __shared__ double4 rec[32];
  const int lane = threadIdx.x, nl = long_count(a);
  const int j = lane < 3 ? lane : 0;
  for (int i = blockIdx.x; i < nl; i += gridDim.x) {
    const int k = a.longs[i];
    const int64_t e0 = a.eoff[k], e1 = a.eoff[k + 1];
    const int2 first = a.first[i];
    const int ns = (int)((e1 - e0 + a.len - 1) / a.len);
    const bool any_bad = any_segment_bad(a, first.x, ns, lane);
    auto run_again = [&](int s, double4 st, bool in_range, double c) {  // from the true value
      const int64_t f0 = e0 + (int64_t)s * a.len;
      const int len = (int)min64(a.len, e1 - f0);
      double to = c;
      bool masses_ok = false, steps_ok = false;
      if (in_range) run_warp(a.eb, f0, len, st.w, to, B, lane, masses_ok, steps_ok);
      if (__any_sync(kFull, !masses_ok || !steps_ok))
        to = segment_ieee(a.eb, f0, len, st.w, c, rec, lane);
      return to;
    };
    double c = reinterpret_cast<const double*>(&a.pass[first.x])[j];
    if (any_bad && a.bad[first.x]) c = run_again(0, a.start[first.x], false, 0.0);
    for (int s = 1; s < ns; ++s) {
      const double4 st = a.start[first.x + s];
      if (any_bad && a.bad[first.x + s]) {
        c = run_again(s, st, false, c);
        continue;
      }
      const Window win(j == 0 ? st.x : j == 1 ? st.y : st.z, s, a.len);
      const int lo = win.find(c);
      const double* en = a.end + ((size_t)(first.y + s - 1) * 3 + j) * kCand + lo;
      const double cl = win.at(lo), ch = win.at(lo + 1), el = en[0], eh = en[1];
      const double to = c == ch ? eh : el;
      const bool known =
          (c == cl || c == ch || (cl < c && c < ch && el == eh)) && to == to;
      c = __all_sync(kFull, known) ? to : run_again(s, st, true, c);
    }
    if (lane < 3) reinterpret_cast<double*>(&a.mc[k])[lane] = c;
    __syncwarp();
  }
}

}  // namespace

// Cells of fewer bodies run on one thread (about 140 cycles a body; a segment
// costs a block three warps at about 100).
int com_long_chain(int64_t n) {
  const int len = segment_len(n);
  return len < 512 ? 512 : len > 4096 ? 4096 : len;
}

int com_long_cells(phys_ctx* c, int64_t n, int64_t nnodes, int64_t total, const int32_t* eoff,
                   const double4* eb, const TreeHeader* hdr, const int32_t* longs, double4* mc) {
  LongCells a{};
  a.nnodes = nnodes;
  a.len = segment_len(n);
  a.eoff = eoff;
  a.eb = eb;
  a.hdr = hdr;
  a.longs = longs;
  a.mc = mc;
  a.status = c->d_status;
  // at most total / com_long_chain cells, a partial segment each
  const int64_t cells = total / com_long_chain(n) + 1, slots = total / a.len + 1,
                segs = slots + cells;
  char* b = nullptr;
  PHYS_TRY(ws_alloc(c, WS_COM_SEG,
                    256 + segs * (32 + 32 + 32 + 16 + 8 + 4 + 4) + cells * 8, &b));
  a.ctr = reinterpret_cast<int32_t*>(b);
  b += 256;
  a.sum = reinterpret_cast<double4*>(b);
  b += segs * 32;
  a.start = reinterpret_cast<double4*>(b);
  b += segs * 32;
  a.pass = reinterpret_cast<double4*>(b);
  b += segs * 32;
  a.mass_end = reinterpret_cast<double2*>(b);
  b += segs * 16;
  a.first = reinterpret_cast<int2*>(b);
  b += cells * 8;
  a.seg = reinterpret_cast<int2*>(b);
  b += segs * 8;
  a.bad = reinterpret_cast<int32_t*>(b);
  b += segs * 4;
  a.redo = reinterpret_cast<int32_t*>(b);
  PHYS_TRY(ws_alloc(c, WS_COM_TRAJ, slots * 3 * kCand, &a.end));
  PHYS_CUDA(c, cudaMemsetAsync(a.ctr, 0, 256, c->stream));
  const int warps = (int)min64(segs, 148 * 32), per_cell = (int)min64(cells, 148 * 16);
  PHYS_LAUNCH(c, segments_kernel, (int)min64(ceil_div(cells, 128), 148), 128, 0, a);
  PHYS_LAUNCH(c, segment_sum_kernel, (int)min64(ceil_div(segs, 4), 148 * 8), 128, 0, a);
  PHYS_LAUNCH(c, prefix_kernel, per_cell, 32, 0, a);
  PHYS_LAUNCH(c, segment_mass_kernel, warps, 32, 0, a);
  PHYS_LAUNCH(c, mass_stitch_kernel, per_cell, 32, 0, a);
  PHYS_LAUNCH(c, first_pass_kernel, warps, 32, 0, a);
  PHYS_LAUNCH(c, predict_kernel, per_cell, 32, 0, a);
  // chains of more than some 10^5 bodies leave the windows in a fifth of their
  // segments (2^20: 13.6 ms without refinement, 9.8 with); below that the two
  // more passes cost more than the few segments run in turn (300 000: 2.1
  // against 2.8 ms)
  const int refine = n > 500000 ? 2 : 0;
  for (int again = 0; again <= refine; ++again) {
    if (again) PHYS_LAUNCH(c, refine_kernel, per_cell, 32, 0, a);
    PHYS_LAUNCH(c, segment_kernel, (int)min64(segs, 148 * 16), 128, 0, a, again);
  }
  PHYS_LAUNCH(c, stitch_kernel, per_cell, 32, 0, a);
  return PHYS_OK;
}

}  // namespace phys

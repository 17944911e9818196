// Adjoint of the Langevin velocity-Verlet step (no reference counterpart: the
// reference has no derivatives).  One loop iteration of MD.cpp:335-729 with
// the box fixed maps the state (x_n, h_n), h the half-step velocity, to
//   h_{n+1} = (1 - gamma dt) h_n + dt F(x_n; theta) + dt sigma psi_n
//   x_{n+1} = x_n + dt h_{n+1}
// (verlet.h:288-355, 463-491 and langevin.h:284-331 composed), and the
// observable is J = (1/T) sum_{n=1..T} U(x_n; theta).  With the Langevin
// noise fixed by its seed, the discrete adjoint runs backwards as
//   w_n    = hbar_{n+1} + dt xbar_{n+1}
//   xbar_n = xbar_{n+1} + dt K(x_n) w_n - (1/T) F(x_n)
//   hbar_n = (1 - gamma dt) w_n
//   dJ/dtheta = sum_n [ dt w_n . dF(x_n)/dtheta + (1/T) dU(x_n)/dtheta ]
// where K = dF/dx is the symmetric force Jacobian (minus the Hessian of U).
// K w is a Hessian-vector product over the same Verlet list as the forces:
// for a pair force g(r) d, d = x_i - x_j,
//   (K w)_i = sum_j g (w_i - w_j) + (g'(r)/r) (d . (w_i - w_j)) d.
// The parameters enter linearly: Umin of a type pair through the table rows
// (include/potentials/laradjiRevalee.h:84-152), kbond and kbend as the CHAIN
// constants 1 and 3 (include/MD.h:384-431, 683-789), so their derivatives
// are the same kernels evaluated with derivative rows or unit constants.
//
// MIXED: pair terms in FP32 from the exact fractional mirror, summed in three
// FP32 words (Sum3, more bits than FP64), the adjoint state in FP64.  PLAIN: FP64 throughout.  The
// CHAIN terms are FP64 in both, their K w the directional derivative of the
// force formulas, written out.
#pragma once

#include "smd_kernels.cuh"

namespace smd {

// A sum of FP32 terms held as three FP32 words (Knuth's TwoSum, cascaded: the
// rounding error of each addition to a word, exact, is added to the next one;
// Ogita, Rump and Oishi's K-fold summation with K = 3).  Its error is some
// n^2 2^-70 of the terms' magnitude, below that of FP64 additions: on 52 terms
// of which 40 cancel, in units of 2^-53 of the terms' total, FP64 0.42 at most,
// three words 1e-6, two words 21.  Thirteen FP32 instructions a term cost a
// fifth of an FP64 conversion and addition (two FP64 instructions).
struct Sum3 {
  float hi = 0.f, mid = 0.f, lo = 0.f;
  // a + b in a, its rounding error returned
  static __device__ __forceinline__ float two_sum(float& a, float b) {
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
    a = s;
    return e;
  }
  __device__ __forceinline__ void add(float x) { lo = __fadd_rn(lo, two_sum(mid, two_sum(hi, x))); }
  __device__ __forceinline__ void add(const Sum3& o) {
    add(o.hi);
    lo = __fadd_rn(lo, __fadd_rn(two_sum(mid, o.mid), o.lo));
  }
  __device__ __forceinline__ Sum3 from(int x) const {  // lane lane ^ x's
    Sum3 o;
    o.hi = __shfl_xor_sync(0xffffffffu, hi, x);
    o.mid = __shfl_xor_sync(0xffffffffu, mid, x);
    o.lo = __shfl_xor_sync(0xffffffffu, lo, x);
    return o;
  }
  // (an infinite or undefined sum is hi alone: the lower words of one are NaN)
  __device__ __forceinline__ double value() const {
    return isfinite(hi) ? (double)hi + ((double)mid + (double)lo) : (double)hi;
  }
};
struct Sum1 {  // the plain form's sums
  double v = 0.0;
  __device__ __forceinline__ void add(double x) { v += x; }
  __device__ __forceinline__ void add(const Sum1& o) { v += o.v; }
  __device__ __forceinline__ Sum1 from(int x) const {
    Sum1 o;
    o.v = __shfl_xor_sync(0xffffffffu, v, x);
    return o;
  }
  __device__ __forceinline__ double value() const { return v; }
};

// CHAIN terms of one bead in FP64, with unit force constants (the forces are
// linear in them): bonds and bends summed apart, each with its directional
// derivative along the beads' w, and the energies the bead owns.  For a bond
// d with tangent t, r = |d|:
//   f = -(1 - l/r) d,   f' = -(1 - l/r) t - (l/r^3)(d . t) d;
// for a bend of unit vectors a, b (lengths p, q), c = a . b, m = c0 - c:
//   g1 = (m/p)(b - a c) on the first bead, g2 = (m/q)(a - b c) off the third,
//   the second taking g2 - g1, with a' = (t_a - a (a . t_a)) / p and so on.
// One reciprocal root per vector serves everything, its quotients rounded by a
// residual step: the same terms by dual numbers through sqrt and divisions took
// 1,280 FP64 instructions per warp and 95 us at 15,000 beads, these 28 us in the
// same CTAs of 256 threads (17 in CTAs of 64) with the same error (3.91e-16 and 2.46e-16 of the rms derivative for a bilayer and
// a vesicle, the dual numbers 3.92e-16 and 2.45e-16; with plain products by the
// reciprocal 24 us, but 3.97e-16 and 2.63e-16).
struct ChainDual {
  double fb[3] = {0, 0, 0}, tb[3] = {0, 0, 0};  // bonds: force, derivative
  double fn[3] = {0, 0, 0}, tn[3] = {0, 0, 0};  // bends
  double ub = 0.0, un = 0.0;                    // energies
};
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return fma(a[2], b[2], fma(a[1], b[1], a[0] * b[0]));
}
// e[k] = x(p-2+k) - x(p-1+k) and t[k] the same difference of w, k = 0 .. 3.
// sums: 1 with the forces themselves and energies, 0 derivatives only.
template <bool SUMS>
__device__ __forceinline__ void chain_dual(const Vec3<double> e[4], const double t[4][3], const bool valid[4],
                                           const double* cd, ChainDual& c) {
  double u[4][3], rr[4], ri[4];  // unit vectors, lengths and their reciprocals
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    u[k][0] = u[k][1] = u[k][2] = rr[k] = ri[k] = 0.0;
    if (!valid[k]) continue;
    const double d[3] = {e[k].x, e[k].y, e[k].z};
    const double r2 = dot3(d, d);
    const double r = rr[k] = root64(r2, ri[k]);
    for (int a = 0; a < 3; ++a) u[k][a] = div64(d[a], r, ri[k]);
    if (k == 1 || k == 2) {  // bonds (p-1, p) as second, (p, p+1) as first
      const double sg = k == 1 ? -1.0 : 1.0;
      const double l = cd[0], lr = div64(l, r, ri[k]), A = sg * (lr - 1.0);
      const double B = sg * lr * dot3(u[k], t[k]);  // (l/r)(u . t)
      for (int a = 0; a < 3; ++a) {
        if constexpr (SUMS) c.fb[a] = fma(A, d[a], c.fb[a]);
        c.tb[a] += fma(A, t[k][a], -B * u[k][a]);
      }
      if constexpr (SUMS) {
        if (k == 2) {
          const double x = r - l;
          c.ub = 0.5 * x * x;
        }
      }
    }
  }
  // bends (e[k], e[k+1]): the bead is the third, second, first for k = 0, 1, 2;
  // one turn per bend the bead has (one for three-bead chains, whichever it is)
  unsigned int todo = (valid[0] && valid[1] ? 1u : 0u) | (valid[1] && valid[2] ? 2u : 0u) | (valid[2] && valid[3] ? 4u : 0u);
  while (todo) {
    const int k = __ffs(todo) - 1;
    todo &= todo - 1;
    double a[3], b[3], ta[3], tb[3];
    for (int x = 0; x < 3; ++x) {
      a[x] = k == 0 ? u[0][x] : (k == 1 ? u[1][x] : u[2][x]);
      b[x] = k == 0 ? u[1][x] : (k == 1 ? u[2][x] : u[3][x]);
      ta[x] = k == 0 ? t[0][x] : (k == 1 ? t[1][x] : t[2][x]);
      tb[x] = k == 0 ? t[1][x] : (k == 1 ? t[2][x] : t[3][x]);
    }
    const double ia = k == 0 ? ri[0] : (k == 1 ? ri[1] : ri[2]), ib = k == 0 ? ri[1] : (k == 1 ? ri[2] : ri[3]);
    const double ra = k == 0 ? rr[0] : (k == 1 ? rr[1] : rr[2]), rb = k == 0 ? rr[1] : (k == 1 ? rr[2] : rr[3]);
    const double cs = dot3(a, b), m = cd[2] - cs;
    const double pa = dot3(a, ta), pb = dot3(b, tb);  // rates of the lengths
    double da[3], db[3];
    for (int x = 0; x < 3; ++x) {
      da[x] = div64(fma(-a[x], pa, ta[x]), ra, ia);
      db[x] = div64(fma(-b[x], pb, tb[x]), rb, ib);
    }
    const double dc = dot3(da, b) + dot3(a, db);
    const double ma = div64(m, ra, ia), mb = div64(m, rb, ib);
    const double na = div64(fma(-ma, pa, -dc), ra, ia), nb = div64(fma(-mb, pb, -dc), rb, ib);  // rates of m/p, m/q
    const double s1 = k == 0 ? 0.0 : (k == 1 ? -1.0 : 1.0), s2 = k == 0 ? -1.0 : (k == 1 ? 1.0 : 0.0);
    for (int x = 0; x < 3; ++x) {
      const double va = fma(-a[x], cs, b[x]), vb = fma(-b[x], cs, a[x]);
      const double wa = fma(-a[x], dc, fma(-da[x], cs, db[x])), wb = fma(-b[x], dc, fma(-db[x], cs, da[x]));
      if constexpr (SUMS) c.fn[x] = fma(s1 * ma, va, fma(s2 * mb, vb, c.fn[x]));
      c.tn[x] = fma(s1, fma(ma, wa, na * va), fma(s2, fma(mb, wb, nb * vb), c.tn[x]));
    }
    if constexpr (SUMS) {
      if (k == 2) c.un = 0.5 * m * m;
    }
  }
}

// Device accumulators of one adjoint run.
struct AdjAcc {
  double J;         // (1/T) sum U
  double grad[3];   // dJ/d(Umin(a,b), kbond, kbend)
  double kw_norm;   // unused by the recursion; kept for diagnostics
};

// Derivative rows of the pair tables for Umin of one type pair (zero rows
// elsewhere), FP32 and FP64.
struct AdjTables {
  float fF[6 * kMaxTypes * kMaxTypes];
  float fU[6 * kMaxTypes * kMaxTypes];
  double dF[6 * kMaxTypes * kMaxTypes];
  double dU[6 * kMaxTypes * kMaxTypes];
};

// Positions of the state in file order (xs: 3n) written into the sorted
// arrays and the current mirror; the displacement from the list-build
// positions decides whether the list must be rebuilt before the next pass.
template <bool MIXED>
__global__ void __launch_bounds__(kBlock) k_adj_load(DevPtrs P, int cur, const double* xs, const double* vs) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  float vmax = 0.f;
  if (i < P.n) {
    const RepState& rs = P.rs[rep_of(P, i)];
    const int o = P.orig[i];
    const double x = xs[3 * o], y = xs[3 * o + 1], z = xs[3 * o + 2];
    P.x[i] = x;
    P.y[i] = y;
    P.z[i] = z;
    if (vs) {
      P.vx[i] = vs[3 * o];
      P.vy[i] = vs[3 * o + 1];
      P.vz[i] = vs[3 * o + 2];
    }
    const unsigned int fx = to_frac(x, rs.frac_per_len[0]), fy = to_frac(y, rs.frac_per_len[1]),
                       fz = to_frac(z, rs.frac_per_len[2]);
    vmax = displacement(P.ref[i], fx, fy, fz, rs);
    P.m4[cur][i] = make_uint4(fx, fy, fz, P.m4[cur][i].w);
    if constexpr (!MIXED) {
      const double4 me = P.d4[cur][i];
      P.d4[cur][i] = make_double4(x, y, z, me.w);
    }
  }
  vmax = warp_max(vmax);
  __shared__ float smax[kBlock / 32];
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = vmax;
  __syncthreads();
  float bm = 0.f;
  if (threadIdx.x == 0)
    for (int w = 0; w < kBlock / 32; ++w) bm = fmaxf(bm, smax[w]);
  finalize_step(P, bm, StepEnd{0, 0, 0, 0, 0});
}

// Sorted-order copy of the adjoint direction w (file order) for the pair
// gathers.
template <typename V>
__global__ void __launch_bounds__(kBlock) k_adj_wsort(DevPtrs P, const double* w, V* ws) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= P.n) return;
  const int o = P.orig[i];
  if constexpr (std::is_same<V, float4>::value)
    ws[i] = make_float4((float)w[3 * o], (float)w[3 * o + 1], (float)w[3 * o + 2], 0.f);
  else
    ws[i] = make_double4(w[3 * o], w[3 * o + 1], w[3 * o + 2], 0.0);
}

// Adds v to *dst once per CTA, where any lane of it has a part: one address
// takes one atomic after another, 2-3 ns each.  Called by the whole CTA, N
// quantities at once.
template <int NT, int N>
__device__ __forceinline__ void adj_add(const double (&v)[N], double* const (&dst)[N]) {
  __shared__ double part[N][NT / 32];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double x = warp_sum(v[k]);
    if ((threadIdx.x & 31) == 0) part[k][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double x = 0.0;
    for (int u = 0; u < NT / 32; ++u) x += part[threadIdx.x][u];
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (threadIdx.x == k && x != 0.0) atomicAdd(dst[k], x);
  }
}

// Pair part of step n: for bead i the non-bonded force F_i, (K w)_i, and the
// replica sums of U, dU/dUmin and w_i . dF_i/dUmin.  Eight lanes per bead walk
// the Verlet list in stretches of kPairQueue entries: they first queue the
// entries in range (about half) by a cheap FP32 test with a slightly wider cut,
// then take the terms of full groups of queued entries.  The mixed form's sums
// are Sum3, and the eight sums of a bead end on one lane each by a butterfly
// that halves what every lane still carries.  At 15,000 beads, per pass: each
// term converted and added in FP64 92 us, with Sum3, the queue, the butterfly and one
// atomic per CTA 30.  Sum3's words take 84 registers, which leave an SM 20 warps;
// CTAs of 128 threads held to seven per SM (72 registers) leave it 28 and a finer
// last wave.  A 40-step call at 15,000 and 18,300 beads (chain pass in CTAs of 256):
// 5.61 and 6.77 ms, with six per SM (80 registers) 5.75 and 6.92, with eight (64,
// 92 bytes spilled) 5.72 and 6.56 but 2 % more at 1,176 and 24,000, as three CTAs
// of 256 threads 5.74 and 6.95.
constexpr int kAdjThreads = 128;
template <bool MIXED>
__global__ void __launch_bounds__(kAdjThreads, MIXED ? 7 : 1) k_adj_pair(DevPtrs P, int cur, const AdjTables* AT,
                                                     const typename std::conditional<MIXED, float4, double4>::type* ws,
                                                     double* kw, double* fpair, AdjAcc* acc, double dt, double invT) {
  constexpr int G = 8;
  using R = typename std::conditional<MIXED, float, double>::type;
  using Sum = typename std::conditional<MIXED, Sum3, Sum1>::type;
  __shared__ R tabs[4][6 * kMaxTypes * kMaxTypes];  // F, U and their Umin derivatives
  __shared__ int queues[kAdjThreads / G][kPairQueue];
  const Tables& T = *P.tab;
  for (int k = threadIdx.x; k < 6 * T.nT * T.nT; k += kAdjThreads) {
    if constexpr (MIXED) {
      tabs[0][k] = T.fF[k];
      tabs[1][k] = T.fU[k];
      tabs[2][k] = AT->fF[k];
      tabs[3][k] = AT->fU[k];
    } else {
      tabs[0][k] = T.dF[k];
      tabs[1][k] = T.dU[k];
      tabs[2][k] = AT->dF[k];
      tabs[3][k] = AT->dU[k];
    }
  }
  __syncthreads();
  const int t = blockIdx.x * kAdjThreads + threadIdx.x;
  const int sub = t % G, lane = threadIdx.x & 31;
  const bool active = t / G < P.n;
  const int i = active ? t / G : 0, nn = active ? P.nnbr[i] : 0;
  const unsigned int below = (1u << lane) - 1u, mine = 0xffu << (lane & ~(G - 1));
  Sum S[8], swft;  // F, K w, U and dU/dUmin (each pair's from both its beads)
  {
    const RepState& rs = P.rs[rep_of(P, i)];
    const int* nb = P.nbr + (size_t)i * P.kmax;
    int* queue = queues[threadIdx.x / G];
    const auto wi = ws[i];
    const uint4 mu = P.m4[cur][i];
    R mx = 0, my = 0, mz = 0;
    if constexpr (!MIXED) {
      const double4 me = P.d4[cur][i];
      mx = me.x;
      my = me.y;
      mz = me.z;
    }
    const int row = 6 * (mu.w & 0xff) * T.nT;
    const R rc2 = MIXED ? (R)T.rc2f : (R)T.rc2;
    const float s0 = rs.len_per_frac[0], s1 = rs.len_per_frac[1], s2 = rs.len_per_frac[2];
    const float cut = T.rcf * (1.f + 4e-6f) + 4.f * fmaxf(s0, fmaxf(s1, s2)), cut2 = cut * cut;
    const int longest = __reduce_max_sync(0xffffffffu, nn);
    for (int base = 0; base < longest; base += kPairQueue) {
      const int end = min(kPairQueue, longest - base);
      int queued = 0;
#pragma unroll 4
      for (int k0 = 0; k0 < end; k0 += G) {
        const int k = base + k0 + sub;
        bool near = false;
        int j = 0;
        if (k < nn) {
          j = __ldg(nb + k);
          const uint4 o = P.m4[cur][j];
          const float dx = frac_delta(mu.x, o.x, s0), dy = frac_delta(mu.y, o.y, s1), dz = frac_delta(mu.z, o.z, s2);
          near = dx * dx + dy * dy + dz * dz < cut2;
        }
        const unsigned int hits = __ballot_sync(0xffffffffu, near) & mine;
        if (near) queue[queued + __popc(hits & below)] = j;
        queued += __popc(hits);
      }
      __syncwarp();
      for (int k = sub; k < queued; k += G) {
        const int j = queue[k];
        R dx, dy, dz;
        const uint4 o = P.m4[cur][j];
        const int tj = o.w & 0xff;
        if constexpr (MIXED) {
          dx = frac_delta(mu.x, o.x, s0);
          dy = frac_delta(mu.y, o.y, s1);
          dz = frac_delta(mu.z, o.z, s2);
        } else {
          const double4 e = P.d4[cur][j];
          double ox = e.x, oy = e.y, oz = e.z;
          if (mx - ox > rs.box[0] / 2.0) ox += rs.box[0];
          if (mx - ox < -rs.box[0] / 2.0) ox -= rs.box[0];
          if (my - oy > rs.box[1] / 2.0) oy += rs.box[1];
          if (my - oy < -rs.box[1] / 2.0) oy -= rs.box[1];
          if (mz - oz > rs.box[2] / 2.0) oz += rs.box[2];
          if (mz - oz < -rs.box[2] / 2.0) oz -= rs.box[2];
          dx = mx - ox;
          dy = my - oy;
          dz = mz - oz;
        }
        const R r2 = dx * dx + dy * dy + dz * dz;
        if (!(r2 < rc2)) continue;
        const R rr = ::sqrt(r2);
        const R* c = tabs[0] + row + 6 * tj;
        const int ci = (rr >= c[0]) ? 3 : 0;
        const R m = c[ci] - rr;
        const R g = ((c[ci + 1] - c[ci + 2] * m) * m) / rr;
        // g'(r)/r = -((C1 - 2 C2 m) + g) / r^2
        const R q = -((c[ci + 1] - (R)2 * c[ci + 2] * m) + g) / r2;
        const auto wj = ws[j];
        const R ex = (R)wi.x - (R)wj.x, ey = (R)wi.y - (R)wj.y, ez = (R)wi.z - (R)wj.z;
        const R dd = q * (dx * ex + dy * ey + dz * ez);
        S[0].add(g * dx);
        S[1].add(g * dy);
        S[2].add(g * dz);
        S[3].add(g * ex + dd * dx);
        S[4].add(g * ey + dd * dy);
        S[5].add(g * ez + dd * dz);
        S[6].add((R)0.5 * pair_pot<R>(tabs[1] + row + 6 * tj, rr));
        const R* ct = tabs[2] + row + 6 * tj;
        if (ct[1] != (R)0 || ct[4] != (R)0) {
          const R mt = ct[ci] - rr;
          const R gt = ((ct[ci + 1] - ct[ci + 2] * mt) * mt) / rr;
          swft.add(gt * (dx * (R)wi.x + dy * (R)wi.y + dz * (R)wi.z));
          S[7].add((R)0.5 * pair_pot<R>(tabs[3] + row + 6 * tj, rr));
        }
      }
      __syncwarp();
    }
  }
  // lane sub ends with the group's sum of S[sub]
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const bool upper = (sub & o) != 0;
#pragma unroll
    for (int k = 0; k < o; ++k) {
      const Sum give = upper ? S[k] : S[k + o];
      Sum keep = upper ? S[k + o] : S[k];
      keep.add(give.from(o));
      S[k] = keep;
    }
    swft.add(swft.from(o));
  }
  const double mysum = S[0].value();
  if (active && sub < 6) (sub < 3 ? fpair : kw)[i + (sub % 3) * P.n] = mysum;
  // replica sums (single-system handles): J and the Umin component
  const double gJ = sub == 6 ? invT * mysum : 0.0, g0 = sub == 7 ? dt * swft.value() + invT * mysum : 0.0;
  adj_add<kAdjThreads, 2>({gJ, g0}, {&acc->J, &acc->grad[0]});
}

// Differences of w along the chain of file-order bead o (file order is chain
// order), 0 where a vector does not exist.
__device__ __forceinline__ void chain_tangents(const double* w, int o, const bool valid[4], double t[4][3]) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
    for (int d = 0; d < 3; ++d) t[k][d] = valid[k] ? w[3 * (o - 2 + k) + d] - w[3 * (o - 1 + k) + d] : 0.0;
}

// CHAIN part of step n and the adjoint update of every bead (file order):
//   F_i = F_pair + F_chain, (K w)_i = (K w)_pair + (K w)_chain,
//   xbar += dt (K w)_i - invT F_i, hbar = (1 - gamma dt) w_i,
//   w_next = hbar + dt xbar.
// Adds invT U_chain and the kbond / kbend components to the accumulators.
// Bound by FP64: 15,000 beads are 59 CTAs of 256 threads, on as many SMs, 28 us;
// CTAs of 64 reach every SM's pipe, 17 us (a 40-step call of 1,176, 15,000 and
// 24,000 beads: 4.14, 5.61 and 7.25 ms against 3.65, 5.21 and 6.99).
constexpr int kChainThreads = 64;
template <bool MIXED>
__global__ void __launch_bounds__(kChainThreads) k_adj_chain(DevPtrs P, int cur, const double* w, double* w_next,
                                                      double* xbar, double* hbar, const double* kw,
                                                      const double* fpair, AdjAcc* acc, double dt, double invT) {
  const int i = blockIdx.x * kChainThreads + threadIdx.x;
  double gJ = 0.0, g1 = 0.0, g2 = 0.0;
  if (i < P.n) {
    const Tables& T = *P.tab;
    const int r = rep_of(P, i);
    const RepParams& rp = P.rp[r];
    const RepState& rs = P.rs[r];
    const double box[3] = {rs.box[0], rs.box[1], rs.box[2]};
    const int o = P.orig[i];
    const double wi[3] = {w[3 * o], w[3 * o + 1], w[3 * o + 2]};
    double F[3] = {fpair[i], fpair[i + P.n], fpair[i + 2 * P.n]};
    double K[3] = {kw[i], kw[i + P.n], kw[i + 2 * P.n]};
    const int ci = P.cinfo[i];
    if (ci < 0 && !(ci & 0x40000000)) {
      const int p = ci & 0xfff, len = (ci >> 12) & 0xfff, set = (ci >> 24) & 0x1f;
      Vec3<double> e[4];
      bool valid[4];
      chain_vectors<MIXED, double>(P, cur, i, p, len, box, rs, e, valid);
      double t[4][3];
      chain_tangents(w, o, valid, t);
      const double* cd = T.chainD[set];
      ChainDual c;
      chain_dual<true>(e, t, valid, cd, c);
      for (int d = 0; d < 3; ++d) {
        F[d] += fma(cd[1], c.fb[d], cd[3] * c.fn[d]);
        K[d] += fma(cd[1], c.tb[d], cd[3] * c.tn[d]);
      }
      gJ = invT * (cd[1] * c.ub + cd[3] * c.un);
      g1 = dt * dot3(wi, c.fb) + invT * c.ub;
      g2 = dt * dot3(wi, c.fn) + invT * c.un;
    }
    const double damp = 1.0 - rp.gamma * dt;
    for (int d = 0; d < 3; ++d) {
      const double xb = xbar[3 * o + d] + dt * K[d] - invT * F[d];
      const double hb = damp * wi[d];
      xbar[3 * o + d] = xb;
      hbar[3 * o + d] = hb;
      w_next[3 * o + d] = hb + dt * xb;
    }
  }
  adj_add<kChainThreads, 3>({gJ, g1, g2}, {&acc->J, &acc->grad[1], &acc->grad[2]});
}

// (K w)_i of the full conservative force at the current positions, file
// order, for a caller-supplied w: the pair part from k_adj_pair (kw) plus
// the CHAIN part, written to out (3n).
template <bool MIXED>
__global__ void __launch_bounds__(kBlock) k_adj_hvp_out(DevPtrs P, int cur, const double* w, const double* kw,
                                                        double* out) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= P.n) return;
  const Tables& T = *P.tab;
  const RepState& rs = P.rs[rep_of(P, i)];
  const double box[3] = {rs.box[0], rs.box[1], rs.box[2]};
  const int o = P.orig[i];
  double K[3] = {kw[i], kw[i + P.n], kw[i + 2 * P.n]};
  const int ci = P.cinfo[i];
  if (ci < 0 && !(ci & 0x40000000)) {
    const int p = ci & 0xfff, len = (ci >> 12) & 0xfff, set = (ci >> 24) & 0x1f;
    Vec3<double> e[4];
    bool valid[4];
    chain_vectors<MIXED, double>(P, cur, i, p, len, box, rs, e, valid);
    double t[4][3];
    chain_tangents(w, o, valid, t);
    const double* cd = T.chainD[set];
    ChainDual c;
    chain_dual<false>(e, t, valid, cd, c);
    for (int d = 0; d < 3; ++d) K[d] += fma(cd[1], c.tb[d], cd[3] * c.tn[d]);
  }
  for (int d = 0; d < 3; ++d) out[3 * o + d] = K[d];
}

}  // namespace smd

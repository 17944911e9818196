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
// MIXED: pair terms in FP32 from the exact fractional mirror, summed as pairs
// of FP32 (TwoSum), the adjoint state in FP64.  PLAIN: FP64 throughout.  The
// CHAIN terms are FP64 in both, their K w the directional derivative of the
// force formulas, written out.
#pragma once

#include "smd_kernels.cuh"

namespace smd {

// A sum of FP32 terms held as an unevaluated pair hi + lo (Knuth's TwoSum: the
// rounding error of each addition, exact, is added to lo).  Its error, some
// 2^-45 of the terms' magnitude, is far below the terms' own FP32 rounding, and
// its seven FP32 instructions cost a tenth of an FP64 conversion and addition.
struct Sum2 {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float s = __fadd_rn(hi, x);
    const float b = __fsub_rn(s, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(x, b)));
    hi = s;
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};
struct Sum1 {  // the plain form's sums
  double v = 0.0;
  __device__ __forceinline__ void add(double x) { v += x; }
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
// One reciprocal root per vector serves everything: the same terms by dual
// numbers through sqrt and divisions took 1,280 FP64 instructions per warp and
// 95 us at 15,000 beads, these 260 and 24 us.
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
  double u[4][3], ri[4];  // unit vectors and reciprocal lengths
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    u[k][0] = u[k][1] = u[k][2] = ri[k] = 0.0;
    if (!valid[k]) continue;
    const double d[3] = {e[k].x, e[k].y, e[k].z};
    const double r2 = dot3(d, d);
    ri[k] = rsqrt(r2);
    for (int a = 0; a < 3; ++a) u[k][a] = d[a] * ri[k];
    if (k == 1 || k == 2) {  // bonds (p-1, p) as second, (p, p+1) as first
      const double sg = k == 1 ? -1.0 : 1.0;
      const double l = cd[0], lr = l * ri[k], A = sg * (lr - 1.0);
      const double B = sg * lr * dot3(u[k], t[k]);  // (l/r)(u . t)
      for (int a = 0; a < 3; ++a) {
        if constexpr (SUMS) c.fb[a] = fma(A, d[a], c.fb[a]);
        c.tb[a] += fma(A, t[k][a], -B * u[k][a]);
      }
      if constexpr (SUMS) {
        if (k == 2) {
          const double x = fma(r2, ri[k], -l);
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
    const double cs = dot3(a, b), m = cd[2] - cs;
    const double pa = dot3(a, ta), pb = dot3(b, tb);  // rates of the lengths
    double da[3], db[3];
    for (int x = 0; x < 3; ++x) {
      da[x] = fma(-a[x], pa, ta[x]) * ia;
      db[x] = fma(-b[x], pb, tb[x]) * ib;
    }
    const double dc = dot3(da, b) + dot3(a, db);
    const double ma = m * ia, mb = m * ib;
    const double na = fma(-ma, pa, -dc) * ia, nb = fma(-mb, pb, -dc) * ib;  // rates of m/p, m/q
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

// Pair part of step n: for bead i the non-bonded force F_i, (K w)_i, and the
// replica sums of U, dU/dUmin and w_i . dF_i/dUmin.  G lanes per bead walk
// the Verlet list as k_force does.  The mixed form's sums are Sum2: 39 us per
// pass at 15,000 beads against 92 with each term converted and added in FP64.
template <bool MIXED, int G>
__global__ void __launch_bounds__(kBlock) k_adj_pair(DevPtrs P, int cur, const AdjTables* AT,
                                                     const typename std::conditional<MIXED, float4, double4>::type* ws,
                                                     double* kw, double* fpair, AdjAcc* acc, double dt, double invT) {
  using R = typename std::conditional<MIXED, float, double>::type;
  const Tables& T = *P.tab;
  const int t = blockIdx.x * kBlock + threadIdx.x;
  const int i = t / G, sub = t % G;
  const bool active = i < P.n;
  using Sum = typename std::conditional<MIXED, Sum2, Sum1>::type;
  Sum sF[3], sK[3], su, sut, swft;
  if (active) {
    const RepState& rs = P.rs[rep_of(P, i)];
    const int nn = P.nnbr[i];
    const int* nb = P.nbr + (size_t)i * P.kmax;
    const auto wi = ws[i];
    int ti;
    R mx, my, mz;
    uint4 mu = make_uint4(0, 0, 0, 0);
    if constexpr (MIXED) {
      mu = P.m4[cur][i];
      ti = mu.w & 0xff;
    } else {
      const double4 me = P.d4[cur][i];
      ti = __double_as_longlong(me.w) & 0xff;
      mx = me.x;
      my = me.y;
      mz = me.z;
    }
    const R* rowF;
    const R* rowU;
    const R* rowFt;
    const R* rowUt;
    if constexpr (MIXED) {
      rowF = T.fF + 6 * ti * T.nT;
      rowU = T.fU + 6 * ti * T.nT;
      rowFt = AT->fF + 6 * ti * T.nT;
      rowUt = AT->fU + 6 * ti * T.nT;
    } else {
      rowF = T.dF + 6 * ti * T.nT;
      rowU = T.dU + 6 * ti * T.nT;
      rowFt = AT->dF + 6 * ti * T.nT;
      rowUt = AT->dU + 6 * ti * T.nT;
    }
    const R rc2 = MIXED ? (R)T.rc2f : (R)T.rc2;
    for (int k = sub; k < nn; k += G) {
      const int j = __ldg(nb + k);
      R dx, dy, dz;
      int tj;
      if constexpr (MIXED) {
        const uint4 o = P.m4[cur][j];
        tj = o.w & 0xff;
        dx = frac_delta(mu.x, o.x, rs.len_per_frac[0]);
        dy = frac_delta(mu.y, o.y, rs.len_per_frac[1]);
        dz = frac_delta(mu.z, o.z, rs.len_per_frac[2]);
      } else {
        const double4 o = P.d4[cur][j];
        tj = __double_as_longlong(o.w) & 0xff;
        double ox = o.x, oy = o.y, oz = o.z;
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
      const R* c = rowF + 6 * tj;
      const int ci = (rr >= c[0]) ? 3 : 0;
      const R m = c[ci] - rr;
      const R g = ((c[ci + 1] - c[ci + 2] * m) * m) / rr;
      // g'(r)/r = -((C1 - 2 C2 m) + g) / r^2
      const R q = -((c[ci + 1] - (R)2 * c[ci + 2] * m) + g) / r2;
      const auto wj = ws[j];
      const R ex = (R)wi.x - (R)wj.x, ey = (R)wi.y - (R)wj.y, ez = (R)wi.z - (R)wj.z;
      const R dd = q * (dx * ex + dy * ey + dz * ez);
      sF[0].add(g * dx);
      sF[1].add(g * dy);
      sF[2].add(g * dz);
      sK[0].add(g * ex + dd * dx);
      sK[1].add(g * ey + dd * dy);
      sK[2].add(g * ez + dd * dz);
      su.add((R)0.5 * pair_pot<R>(rowU + 6 * tj, rr));
      const R* ct = rowFt + 6 * tj;
      if (ct[1] != (R)0 || ct[4] != (R)0) {
        const R mt = ct[ci] - rr;
        const R gt = ((ct[ci + 1] - ct[ci + 2] * mt) * mt) / rr;
        swft.add(gt * (dx * (R)wi.x + dy * (R)wi.y + dz * (R)wi.z));
        sut.add((R)0.5 * pair_pot<R>(rowUt + 6 * tj, rr));
      }
    }
  }
  double F[3], K[3];
  for (int d = 0; d < 3; ++d) {
    F[d] = sF[d].value();
    K[d] = sK[d].value();
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    for (int d = 0; d < 3; ++d) {
      F[d] += __shfl_xor_sync(0xffffffffu, F[d], o);
      K[d] += __shfl_xor_sync(0xffffffffu, K[d], o);
    }
  }
  if (active && sub == 0) {
    for (int d = 0; d < 3; ++d) {
      kw[i + d * P.n] = K[d];
      fpair[i + d * P.n] = F[d];
    }
  }
  // replica sums (single-system handles): J and the Umin component
  const double gJ = invT * su.value(), g0 = dt * swft.value() + invT * sut.value();
  const double sJ = warp_sum(gJ), s0 = warp_sum(g0);
  if ((threadIdx.x & 31) == 0) {
    if (sJ != 0.0) atomicAdd(&acc->J, sJ);
    if (s0 != 0.0) atomicAdd(&acc->grad[0], s0);
  }
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
template <bool MIXED>
__global__ void __launch_bounds__(kBlock) k_adj_chain(DevPtrs P, int cur, const double* w, double* w_next,
                                                      double* xbar, double* hbar, const double* kw,
                                                      const double* fpair, AdjAcc* acc, double dt, double invT) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
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
  gJ = warp_sum(gJ);
  g1 = warp_sum(g1);
  g2 = warp_sum(g2);
  if ((threadIdx.x & 31) == 0) {
    if (gJ != 0.0) atomicAdd(&acc->J, gJ);
    if (g1 != 0.0) atomicAdd(&acc->grad[1], g1);
    if (g2 != 0.0) atomicAdd(&acc->grad[2], g2);
  }
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

// The MD loop as one persistent kernel, for systems and batches whose replicas
// have up to 65,000 beads each.
//
// Kernel by kernel, a loop step of a few thousand beads is all latency: two
// step kernels and, every second step, four list kernels of 5-25 us each that
// keep at most a tenth of the chip's warps busy.  At tens of thousands the
// launches' starts and tails, the reordered state's way through memory and one
// list cell per CTA still cost a quarter of a step.  us per step at a skin of
// 0.5, kernel by kernel and here: 1,176 beads 32 and 12, 15,000 41 and 21, 22,500
// 51 and 32, 29,400 57 and 35, 45,000 63 and 47, 60,000 75 and 61 (57 at a skin
// of 0.42).  Here every CTA owns a contiguous range of the
// cell-sorted beads and keeps their positions, velocities and bookkeeping in
// shared memory; only the position mirror goes through global memory.  A step
// is one grid barrier: each CTA forms its beads' pair sums (and beside them
// the bonded forces and the noise), integrates them, writes the next mirror
// and arrives.  A list rebuild adds one barrier (between the reordering and
// the stencil scans), a barostat trial one (its summed energy difference).
// Every barrier waits with a limit.  The CTAs of a batch are dealt out to its
// replicas, which share the barriers and, as kernel by kernel, the decision to
// rebuild.
//
// The arithmetic of a step is that of k_force, k_integ, k_mc and k_finish, and
// the mixed form's sums are exact in any order, so a mixed run has the same
// bits here and there.
#pragma once

#include "smd_kernels.cuh"

namespace smd {

// Warps per CTA at most, which set the registers per thread: 24 (80 registers)
// where a CTA has few beads; with many, 28 (72) or 32 (64), whichever takes
// their pair and bonded tasks in fewer rounds, 28 if both do: fewer spills then
// count for more.  us per step with 28 and 32 warps, by beads per CTA (tasks),
// bilayers in the mixed form: 60 (17) 19.4 and 19.8, 79 (23) 20.8 and 21.1, 98
// (29) 21.7 and 22.0, 109 (32) 26.9 and 23.9, 119 (34) 29.0 and 26.4 (the rule
// takes 28), 139 (40) 30.4 and 32.1, 168 (48) 32.8 and 34.2, 198 (57) 35.2 and
// 35.8, 227 (65) 40.2 and 37.2, 257 (74) 44.6 and 46.3, 297 (85) 46.7 and 48.3,
// 336 (95) 55.2 and 52.3, 390 (111) 59.5 and 61.9, 422 (120) 64.0 and 63.7.  The
// plain form, bound by FP64, differs by 1 % (227: 234 and 229, the others 28).
__host__ __device__ constexpr int run_tasks(int beads, int lanes) {
  return (beads * lanes + 31) / 32 + (beads + 31) / 32;
}
__host__ __device__ constexpr int run_warps(int beads, int lanes) {
  const int tasks = run_tasks(beads, lanes);
  return lanes != 8 ? 24 : (beads <= 896 && (tasks + 27) / 28 == (tasks + 31) / 32 ? 28 : 32);
}
// What 16-bit cell starts can count.  It still gains a quarter there (63,654
// beads: 84 us per step kernel by kernel, 67 here).
constexpr int kRunMaxBeads = 65000;
constexpr int kRunCells = 81920;    // largest list-cell grid (its starts, 160 KB, are kept in shared memory)
constexpr int kRunSpinLimit = 1 << 22;  // polls of a barrier: some seconds

// A CTA's place: its replica, its number among the replica's CTAs, and where
// the replica's cell counts begin.
struct RunPlace {
  int rep, index, ctas, cnt;
};

// Grid-wide words of the persistent loop (zero between launches).
struct RunSync {
  // arrivals in the low 40 bits, then three 8-bit counts (by step modulo 3) of
  // the CTAs with a bead beyond the list's margin: they ride on the arrival,
  // so the barrier itself tells whether the list must be rebuilt
  unsigned long long arrive;
  unsigned int left;             // CTAs that are done with the kernel
  // of trial steps, alternating: the largest displacement (FP32 bits) and the
  // largest change of a pair distance by an accepted trial (FP64 bits)
  unsigned int dmax[2];
  unsigned long long shift[2];
};
// A replica's trial sums, alternating (zero between launches).
struct RunTrial {
  long long dq_pair[2], dq_bond[2];
  double du_pair[2], du_bond[2];
};

struct RunArgs {
  long long it;   // loop step of the first iteration
  int cur;        // current mirror
  int steps;      // iterations to run
  int rate;       // barostat period
  int barostat;
  int beads;      // beads per CTA
  int* cnt;       // 2 x run_cells(cells) cell counts per replica, zero between launches
  RunSync* sync;
  RunTrial* trial;  // per replica
  const RunPlace* place;  // per CTA
  double* save;   // positions after every step in file order (3n each), or null
};

// Shared memory per CTA beyond the static part.
__host__ __device__ constexpr size_t run_align(size_t b) { return (b + 15) & ~(size_t)15; }
__host__ __device__ constexpr int run_cells(int cells) { return (cells + 3) & ~3; }
__host__ __device__ constexpr size_t run_smem(int beads, int cells, bool mixed, int threads, int lanes) {
  return run_align(sizeof(unsigned short) * ((size_t)run_cells(cells) + 1)) + run_align(sizeof(double) * 6 * (size_t)beads) +  // starts, x v
         run_align(sizeof(double) * 3 * (size_t)beads) + run_align(sizeof(double) * 3 * (size_t)beads) +  // sums, bonded
         run_align(sizeof(uint4) * (size_t)beads) + run_align(sizeof(int) * 4 * (size_t)beads) +
         (mixed ? 0 : run_align(sizeof(int) * (size_t)kPairQueue * (threads / lanes)));
}

// Both bounds of the periodic wrap decided on the bits, in the integer pipe:
// doubles order like signed integers when one of them is positive, and x < 0
// is a set sign bit other than -0.
__device__ __forceinline__ double wrap64(double x, double box) {
  if (__double_as_longlong(x) > __double_as_longlong(box)) x -= box;
  if ((unsigned long long)__double_as_longlong(x) > 0x8000000000000000ull) x += box;
  return x;
}

// The stencil of cell (cx, cy, cz) as contiguous bead ranges with prefix sums,
// formed by one warp: lane l < 18 takes half of row l / 2 (dy, dz), whose
// cells cx - 1 .. cx + 1 are one range unless it wraps in x; axes with fewer
// than 3 cells take every cell once.  seg: first bead less first slot [0, 18),
// the slot after the last [18, 36), none after the last segment's.  Returns the
// number of slots.
__device__ __forceinline__ int run_stencil(const int ncell[3], const unsigned short* starts, int first, int cx,
                                           int cy, int cz, int* seg) {
  const int lane = threadIdx.x & 31;
  const int n0 = ncell[0], n1 = ncell[1], n2 = ncell[2];
  int start = 0, len = 0;
  if (lane < 18) {
    const int t = lane >> 1, half = lane & 1, oy = t % 3 - 1, oz = t / 3 - 1;
    if (!((oy < 0 && n1 < 3) || (oy > 0 && n1 < 2) || (oz < 0 && n2 < 3) || (oz > 0 && n2 < 2))) {
      int yy = cy + oy, zz = cz + oz;
      yy += yy < 0 ? n1 : (yy >= n1 ? -n1 : 0);
      zz += zz < 0 ? n2 : (zz >= n2 ? -n2 : 0);
      const int row = n0 * (yy + n1 * zz);
      int u0 = n0 < 3 ? 0 : cx - 1, u1 = n0 < 3 ? n0 - 1 : cx + 1;
      if (u0 < 0) {
        u0 = half ? 0 : n0 - 1;
        u1 = half ? u1 : n0 - 1;
      } else if (u1 >= n0) {
        u0 = half ? 0 : u0;
        u1 = half ? 0 : n0 - 1;
      } else if (half) {
        u1 = u0 - 1;
      }
      if (u1 >= u0) {
        start = first + starts[row + u0];
        len = starts[row + u1 + 1] - starts[row + u0];
      }
    }
  }
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const unsigned int full = __ballot_sync(0xffffffffu, len > 0);
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  __syncwarp();
  if (len > 0) {
    const int k = __popc(full & ((1u << lane) - 1u));
    seg[k] = start - (incl - len);
    seg[18 + k] = incl == total ? 0x7fffffff : incl;
  }
  __syncwarp();
  return total;
}

// The beads of a stencil's slots, 32 at a time.  The segment of the first slot
// is the warp's; lanes behind a boundary take the next one, so a round costs a
// few uniform instructions per boundary it crosses instead of a search per lane.
struct SlotWalk {
  const int* seg;
  int t = 0, off, end;
  __device__ __forceinline__ explicit SlotWalk(const int* s) : seg(s), off(s[0]), end(s[18]) {}
  // bead of slot min(k0 + lane, M - 1); k0 increases from call to call
  __device__ __forceinline__ int round(int k0, int lane, int M) {
    const int g = min(k0 + lane, M - 1);
    int o = off;
    while (end < k0 + 32) {
      ++t;
      off = seg[t];
      o = g >= end ? off : o;
      end = seg[18 + t];
    }
    return o + g;
  }
};

// Lists of beads a = ia and b = ia + 1 of the same cell from the stencil's M
// slots, by one warp.  Distances come from the exact fractional differences,
// whose wrap is the minimum image, so thin grids need no other path.
__device__ __forceinline__ void run_scan_pair(const uint4* m, const int* seg, int M, uint4 ma, uint4 mb, int ia,
                                              float x0, float x1, float x2, float lc2, int* oa, int kmax, int* cnt) {
  const int lane = threadIdx.x & 31;
  const unsigned int below = (1u << lane) - 1u;
  int ca = 0, cb = 0;
  SlotWalk walk(seg);
  int j = walk.round(0, lane, M);
  uint4 o = m[j];
  for (int k0 = 0; k0 < M; k0 += 32) {
    const int jc = j;
    const uint4 c = o;
    const float lim = k0 + lane < M ? lc2 : -1.f;
    if (k0 + 32 < M) {  // the next round's candidate, a round ahead
      j = walk.round(k0 + 32, lane, M);
      o = m[j];
    }
    const float ax = frac_delta(ma.x, c.x, x0), ay = frac_delta(ma.y, c.y, x1), az = frac_delta(ma.z, c.z, x2);
    const float bx = frac_delta(mb.x, c.x, x0), by = frac_delta(mb.y, c.y, x1), bz = frac_delta(mb.z, c.z, x2);
    keep_hits(ax * ax + ay * ay + az * az, lim, jc - ia, 0, below, jc, oa, kmax, ca);
    keep_hits(bx * bx + by * by + bz * bz, lim, jc - ia, 1, below, jc, oa + kmax, kmax, cb);
  }
  if (lane == 0) {
    cnt[0] = ca;
    cnt[1] = cb;
  }
}

// Rounds `part`, part + parts, ... of bead ia's list, by one of the `parts` warps
// that share it; count (shared memory) starts at 0.
__device__ __forceinline__ void run_scan_part(const uint4* m, const int* seg, int M, uint4 ma, int ia, int part,
                                              int parts, float x0, float x1, float x2, float lc2, int* out, int kmax,
                                              int* count) {
  const int lane = threadIdx.x & 31;
  const unsigned int below = (1u << lane) - 1u;
  SlotWalk walk(seg);
  for (int k0 = 32 * part; k0 < M; k0 += 32 * parts) {
    const int j = walk.round(k0, lane, M);
    const uint4 c = m[j];
    const float ax = frac_delta(ma.x, c.x, x0), ay = frac_delta(ma.y, c.y, x1), az = frac_delta(ma.z, c.z, x2);
    const bool hit = k0 + lane < M && j != ia && ax * ax + ay * ay + az * az < lc2;
    const unsigned int hits = __ballot_sync(0xffffffffu, hit);
    int at = 0;
    if (lane == 0 && hits) at = atomicAdd(count, __popc(hits));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(hits & below);
    if (hit && at < kmax) out[at] = j;
  }
}

// Lists of n <= Q neighbouring beads of one cell, from bead ia on, by one warp
// (grids of five cells on every axis: no candidate of the stencil is then near
// half the box from the first bead and in range of another).  With c a
// candidate's and x a bead's offset from the first of them, |c - x|^2 < L^2 is
// |c|^2 - 2 x . c < L^2 - |x|^2: three FMAs and a comparison per bead, and one
// load and conversion of a candidate for all: 104,000 cycles per build at 395
// beads per CTA against 150,000 in pairs with six operations per distance.
template <int Q>
__device__ __forceinline__ void run_scan_group(const uint4* m, const int* seg, int M, const uint4* own, int n, int ia,
                                               float x0, float x1, float x2, float lc2, int* out, int kmax, int* cnt) {
  const int lane = threadIdx.x & 31;
  const unsigned int below = (1u << lane) - 1u;
  const uint4 ma = own[0];
  float fx[Q], fy[Q], fz[Q], lim[Q];
  int count[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint4 mq = own[q < n ? q : 0];
    const float x = frac_delta(mq.x, ma.x, x0), y = frac_delta(mq.y, ma.y, x1), z = frac_delta(mq.z, ma.z, x2);
    fx[q] = -2.f * x;
    fy[q] = -2.f * y;
    fz[q] = -2.f * z;
    lim[q] = q < n ? lc2 - (x * x + y * y + z * z) : -1e30f;  // past the last bead: no hit
    count[q] = q * kmax;
  }
  SlotWalk walk(seg);
  int j = walk.round(0, lane, M);
  uint4 o = m[j];
  for (int k0 = 0; k0 < M; k0 += 32) {
    const int jc = j;
    const float cx = frac_delta(o.x, ma.x, x0), cy = frac_delta(o.y, ma.y, x1), cz = frac_delta(o.z, ma.z, x2);
    const float cc = k0 + lane < M ? cx * cx + cy * cy + cz * cz : 1e30f;
    if (k0 + 32 < M) {  // the next round's candidate, a round ahead
      j = walk.round(k0 + 32, lane, M);
      o = m[j];
    }
#pragma unroll
    for (int q = 0; q < Q; ++q)
      keep_hits(fmaf(fz[q], cz, fmaf(fy[q], cy, fmaf(fx[q], cx, cc))), lim[q], jc - ia, q, below, jc, out,
                (q + 1) * kmax, count[q]);
  }
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (lane == q && q < n) cnt[q] = count[q] - q * kmax;
}

template <bool MIXED, int G, int NW>
__global__ void __launch_bounds__(NW * 32, 1) k_run(DevPtrs P, RunArgs A) {
  using R = typename std::conditional<MIXED, float, double>::type;
  using Sum = typename std::conditional<MIXED, long long, double>::type;
  extern __shared__ uint4 run_dyn[];
  __shared__ RepState rs;
  __shared__ __align__(8) R sF[6 * kMaxTypes * kMaxTypes], sU[6 * kMaxTypes * kMaxTypes];
  __shared__ int wsum[NW];
  __shared__ int segs[NW][36];
  __shared__ float smax[NW];
  __shared__ long long sdq[2];
  __shared__ double sdu[2];
  __shared__ double slack, shift_s;
  __shared__ int rebuild, slot, abort_s, n_groups;
  __shared__ unsigned long long seen;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  // kept in shared memory, as what follows from it: registers are short here
  __shared__ RunPlace me;
  __shared__ RepParams rp;
  if (tid == 0) {
    me = A.place[blockIdx.x];
    rp = P.rp[me.rep];
  }
  __syncthreads();
  const int b0 = rp.bead_begin + me.index * A.beads, nb = min(A.beads, rp.bead_end - b0);
  const int ncell = rp.cell_cap, ncell4 = run_cells(ncell);
  // dynamic shared memory (run_smem)
  unsigned char* at = reinterpret_cast<unsigned char*>(run_dyn);
  static_assert(kRunMaxBeads < 65536, "16-bit cell starts");
  unsigned short* starts = reinterpret_cast<unsigned short*>(at);
  at += run_align(sizeof(unsigned short) * ((size_t)ncell4 + 1));
  double* st = reinterpret_cast<double*>(at);  // x, y, z, vx, vy, vz of the CTA's beads
  at += run_align(sizeof(double) * 6 * (size_t)A.beads);
  Sum* fsum = reinterpret_cast<Sum*>(at);
  at += run_align(sizeof(double) * 3 * (size_t)A.beads);
  R* fbond = reinterpret_cast<R*>(at);  // mixed: bonded force + noise in FP32; plain: bonded force
  at += run_align(sizeof(double) * 3 * (size_t)A.beads);
  uint4* ref = reinterpret_cast<uint4*>(at);
  at += run_align(sizeof(uint4) * (size_t)A.beads);
  int* orig = reinterpret_cast<int*>(at);
  int* cinfo = orig + A.beads;
  int* key = cinfo + A.beads;
  int* cnt = key + A.beads;
  at += run_align(sizeof(int) * 4 * (size_t)A.beads);
  int* queue = reinterpret_cast<int*>(at);
  const Tables& T = *P.tab;
  const int nT = T.nT;
  const int NB = A.beads;

  // ---- entry
  for (int k = tid; k < (int)(sizeof(RepState) / 4); k += nt)
    reinterpret_cast<int*>(&rs)[k] = reinterpret_cast<const int*>(P.rs + me.rep)[k];
  for (int k = tid; k < 6 * nT * nT; k += nt) {
    if constexpr (MIXED) {
      sF[pack_force_row(k)] = T.fF[k];
      sU[k] = T.fU[k];
    } else {
      sF[k] = T.dF[k];
      sU[k] = T.dU[k];
    }
  }
  if (*(volatile int*)&P.g->error & 8) return;  // an earlier launch gave up: its words are not clean
  if (tid == 0) {
    slack = P.g->slack;
    slot = P.g->trial_slot;
    rebuild = P.g->rebuild;
    abort_s = 0;
    n_groups = 0;
  }
  if (tid < nb) {
    const int i = b0 + tid;
    st[tid] = P.x[i];
    st[NB + tid] = P.y[i];
    st[2 * NB + tid] = P.z[i];
    st[3 * NB + tid] = P.vx[i];
    st[4 * NB + tid] = P.vy[i];
    st[5 * NB + tid] = P.vz[i];
    ref[tid] = P.ref[i];
    orig[tid] = P.orig[i];
    cinfo[tid] = P.cinfo[i];
  }
  __syncthreads();
  const double gamma = rp.gamma, dt = rp.dt, h = dt * 0.5;
  long long it = A.it;
  int cur = A.cur;
  unsigned long long waited = 0;  // barriers so far

  // Arrives with inc and waits for every CTA; false when the limit ran out.
  auto barrier = [&](unsigned long long inc) -> bool {
    __syncthreads();
    ++waited;
    if (tid == 0) {
      const unsigned long long target = waited * gridDim.x;
      // release: the CTA's writes (ordered before by the block barrier) are
      // visible to whoever sees the arrival; the acquire below is its other end
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&A.sync->arrive), "l"(inc) : "memory");
      unsigned long long v = 0;
      int polls = 0;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&A.sync->arrive) : "memory");
        if ((v & ((1ull << 40) - 1)) >= target) break;
        if (++polls > kRunSpinLimit) {
          atomicOr(&P.g->error, 8);
          abort_s = 1;
          break;
        }
      }
      seen = v;
    }
    __syncthreads();
    return abort_s == 0;
  };
  int phase = (int)(((it % A.rate) + A.rate) % A.rate);  // of the barostat period
  // list cell of own bead t on the current grid
  auto cell_of = [&](const uint4& m) {
    const int n0 = rs.ncell[0], n1 = rs.ncell[1], n2 = rs.ncell[2];
    return (int)__umulhi(m.x, (unsigned)n0) +
           n0 * ((int)__umulhi(m.y, (unsigned)n1) + n1 * (int)__umulhi(m.z, (unsigned)n2));
  };
  // own bead t's cell on the reference's grid (the size-change passes)
  auto ref_key = [&](const double x[3]) {
    unsigned long long k = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d)
      k |= (unsigned long long)(ref_cell_coord(x[d], rs.ref_cs[d], rs.ref_inv_cs[d], rs.refn[d]) & 0x1fffff) << (21 * d);
    return k;
  };
  // exclusive sum of v over the block's threads, and the total (scratch: 32
  // words; the caller synchronises before it is used again)
  auto block_scan = [&](int v, int* scratch, int& total) {
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) scratch[warp] = x;
    __syncthreads();
    int t = lane < nw ? scratch[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    total = __shfl_sync(0xffffffffu, t, 31);
    const int before = __shfl_sync(0xffffffffu, t, warp > 0 ? warp - 1 : 0);
    return (warp > 0 ? before : 0) + x - v;
  };
  // the trial of a barostat step: every CTA draws it into its own copy
  auto draw = [&]() {
    if (tid == 0) draw_trial(rs, rp, P.trial_u[((size_t)slot * P.n_rep + me.rep) * 2]);
  };
  bool trial = A.barostat && phase == 0 && it != 0;
  {
    const bool stale = rebuild != 0;
    if (trial) draw();
    if (stale && tid < nb) {
      const int c = cell_of(P.m4[cur][b0 + tid]);
      key[tid] = c;
      atomicAdd(A.cnt + me.cnt + ncell4 + c, 1);
    }
    if (trial && !stale && tid < nb) {
      const double x[3] = {st[tid], st[NB + tid], st[2 * NB + tid]};
      P.refcell[b0 + tid] = ref_key(x);
    }
    if ((stale || trial) && !barrier(1)) return;
  }

  int trials = 0, rebuilds = 0;
  for (int s = 0; s < A.steps; ++s) {
    const bool last = s + 1 == A.steps;
    if (rebuild) {
      // ---- exclusive scan of the cell counts, by every CTA for itself
      {
        const int4* counts = reinterpret_cast<const int4*>(A.cnt + me.cnt + (size_t)((s + 1) & 1) * ncell4);
        constexpr int kQuads = 4;  // 16 consecutive counts per thread and pass, loaded together
        int carry = 0, most = 0;
        for (int q0 = 0; q0 < ncell4 / 4; q0 += kQuads * nt) {
          int4 v[kQuads];
          int sum = 0;
#pragma unroll
          for (int u = 0; u < kQuads; ++u) {
            const int q = q0 + kQuads * tid + u;
            v[u] = q < ncell4 / 4 ? __ldcg(counts + q) : make_int4(0, 0, 0, 0);
          }
#pragma unroll
          for (int u = 0; u < kQuads; ++u) {
            sum += v[u].x + v[u].y + v[u].z + v[u].w;
            most = max(max(most, max(v[u].x, v[u].y)), max(v[u].z, v[u].w));
          }
          int total;
          int ex = carry + block_scan(sum, wsum, total);
#pragma unroll
          for (int u = 0; u < kQuads; ++u) {
            const int q = q0 + kQuads * tid + u;
            ushort4 f;
            f.x = (unsigned short)ex;
            f.y = (unsigned short)(ex += v[u].x);
            f.z = (unsigned short)(ex += v[u].y);
            f.w = (unsigned short)(ex += v[u].z);
            ex += v[u].w;
            if (q < ncell4 / 4) reinterpret_cast<ushort4*>(starts)[q] = f;
          }
          carry += total;
          __syncthreads();  // wsum is used again
        }
        if (most > kNbrMaxCell) atomicOr(&P.g->error, 2);
        if (tid == 0) starts[ncell4] = (unsigned short)(rp.bead_end - rp.bead_begin);
      }
      __syncthreads();
      // ---- scatter to the new order (cell_count: the cells' fill)
      if (tid < nb) {
        const int c = key[tid], nw_i = rp.bead_begin + starts[c] + atomicAdd(P.cell_count + rp.cell_begin + c, 1);
        P.tx[nw_i] = st[tid];
        P.ty[nw_i] = st[NB + tid];
        P.tz[nw_i] = st[2 * NB + tid];
        P.tvx[nw_i] = st[3 * NB + tid];
        P.tvy[nw_i] = st[4 * NB + tid];
        P.tvz[nw_i] = st[5 * NB + tid];
        const int o = orig[tid];
        P.torig[nw_i] = o;
        P.tcinfo[nw_i] = cinfo[tid];
        P.inv[o] = nw_i;
        P.m4[cur ^ 1][nw_i] = P.m4[cur][b0 + tid];
        if constexpr (!MIXED) P.d4[cur ^ 1][nw_i] = P.d4[cur][b0 + tid];
        if (trial) {
          const double x[3] = {st[tid], st[NB + tid], st[2 * NB + tid]};
          P.refcell[nw_i] = ref_key(x);
        }
      }
      if (!barrier(1)) return;
      cur ^= 1;
      if (tid < nb) {
        const int i = b0 + tid;
        st[tid] = __ldcg(P.tx + i);
        st[NB + tid] = __ldcg(P.ty + i);
        st[2 * NB + tid] = __ldcg(P.tz + i);
        st[3 * NB + tid] = __ldcg(P.tvx + i);
        st[4 * NB + tid] = __ldcg(P.tvy + i);
        st[5 * NB + tid] = __ldcg(P.tvz + i);
        const int o = __ldcg(P.torig + i);
        orig[tid] = o;
        P.orig[i] = o;
        cinfo[tid] = __ldcg(P.tcinfo + i);
        ref[tid] = P.m4[cur][i];
      }
      if (tid == 0) {
        n_groups = 0;
        slack = 0.0;
        ++rebuilds;
      }
      __syncthreads();
      // ---- lists: a warp takes up to four neighbouring beads of one cell at a time,
      // fewer where that leaves warps idle
      const bool offset = rs.ncell[0] >= 5 && rs.ncell[1] >= 5 && rs.ncell[2] >= 5;
      int* const groups = reinterpret_cast<int*>(fsum);  // first bead and size (free until the force pass)
      {
        const int most = nb <= nw ? 1 : (nb <= 2 * nw || !offset ? 2 : 4);
        int n = 0, c = 0;
        if (tid < nb) {
          const int i = b0 + tid;
          key[tid] = c = cell_of(ref[tid]);
          cnt[tid] = 0;
          const int rank = i - max(rp.bead_begin + starts[c], b0);
          if (rank % most == 0) n = min(min(most, rp.bead_begin + starts[c + 1] - i), nb - tid);
        }
        const unsigned int heads = __ballot_sync(0xffffffffu, n > 0);
        int at = 0;
        if (lane == 0 && heads) at = atomicAdd(&n_groups, __popc(heads));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(heads & ((1u << lane) - 1u));
        if (n > 0) groups[at] = tid | n << 16;
      }
      __syncthreads();
      {
        const float lcut = list_reach<MIXED>(rs, T.list_cut_f);
        const float lc2 = lcut * lcut;
        const float x0 = rs.len_per_frac[0], x1 = rs.len_per_frac[1], x2 = rs.len_per_frac[2];
        const uint4* m = P.m4[cur];
        const int kmax = P.kmax, ng = n_groups;
        int* seg = segs[warp];
        // where there are warps for it, several share a bead's candidates
        const int parts = max(1, min(8, nw / max(ng, 1)));
        for (int t = warp; t < ng * parts; t += nw) {
          const int g = t / parts, q = groups[g] & 0xffff, n = groups[g] >> 16, c = key[q], i = b0 + q;
          const int n0 = rs.ncell[0], n1 = rs.ncell[1], row = c / n0;
          const int M = run_stencil(rs.ncell, starts, rp.bead_begin, c - row * n0, row % n1, row / n1, seg);
          int* out = P.nbr + (size_t)i * kmax;
          const uint4 ma = ref[q];
          if (n > 2) run_scan_group<4>(m, seg, M, ref + q, n, i, x0, x1, x2, lc2, out, kmax, cnt + q);
          else if (n == 2 && offset) run_scan_group<2>(m, seg, M, ref + q, n, i, x0, x1, x2, lc2, out, kmax, cnt + q);
          else if (n == 2) run_scan_pair(m, seg, M, ma, ref[q + 1], i, x0, x1, x2, lc2, out, kmax, cnt + q);
          else run_scan_part(m, seg, M, ma, i, t - g * parts, parts, x0, x1, x2, lc2, out, kmax, cnt + q);
        }
      }
      __syncthreads();
      if (tid < nb) {
        const int count = cnt[tid];
        P.nnbr[b0 + tid] = min(count, P.kmax);
        if (count > *(volatile int*)&P.g->max_nbr) atomicMax(&P.g->max_nbr, count);
        if (count > P.kmax) {
          atomicOr(&P.g->error, 1);
          atomicMax(&P.g->need_nbr, count);
        }
      }
      for (int c = me.index * nt + tid; c < ncell; c += me.ctas * nt) P.cell_count[rp.cell_begin + c] = 0;
      __syncthreads();
    }
    // the counts of the step before this one: read above at the latest
    for (int c = me.index * nt + tid; c < ncell; c += me.ctas * nt) A.cnt[me.cnt + (size_t)((s + 1) & 1) * ncell4 + c] = 0;
    if (tid == 0) {
      sdq[0] = sdq[1] = 0;
      sdu[0] = sdu[1] = 0.0;
    }
    if (trial) __syncthreads();

    // ---- forces: warps take the bonded terms and the noise, then the pair sums
    const int bond_tasks = (nb + 31) >> 5, pair_tasks = (nb * G + 31) >> 5;
    for (int task = warp; task < bond_tasks + pair_tasks; task += nw) {
      if (task < bond_tasks) {
        const int b = task * 32 + lane;
        double dU = 0.0, unused = 0.0;
        if (b < nb) {
          const int ci = cinfo[b];
          const double box[3] = {rs.box[0], rs.box[1], rs.box[2]};
          const Vec3<R> f = bonded_force<MIXED, false>(P, cur, b0 + b, ci, box, rs);
          if (trial) bonded_sums<MIXED, F_DU>(P, cur, b0 + b, ci, box, rs, dU, unused);
          if constexpr (MIXED) {
            float nf[3];
            langevin_noise_f(rp.seed, orig[b] - rp.bead_begin, it, 0, rp.sig31f, nf);
            fbond[3 * b] = f.x + nf[0];
            fbond[3 * b + 1] = f.y + nf[1];
            fbond[3 * b + 2] = f.z + nf[2];
          } else {
            fbond[3 * b] = f.x;
            fbond[3 * b + 1] = f.y;
            fbond[3 * b + 2] = f.z;
          }
        }
        if (trial) {
          if constexpr (MIXED) {
            long long q = __double2ll_rn(dU * 4294967296.0);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
            if (lane == 0) atomicAdd((unsigned long long*)&sdq[1], (unsigned long long)q);
          } else {
            dU = warp_sum(dU);
            if (lane == 0) atomicAdd(&sdu[1], dU);
          }
        }
      } else {
        const int g = (task - bond_tasks) * 32 + lane;
        const int b = g / G, sub = g % G;
        const bool active = b < nb;
        const int i = b0 + (active ? b : 0);
        if constexpr (MIXED) {
          long long qx = 0, qy = 0, qz = 0, dq = 0;
          float unused = 0.f;
          if (active) {
            const BeadList<false> list{P.nbr + (size_t)i * P.kmax, P.m4[cur]};
            const int nn = P.nnbr[i];
            if (trial) pair_sum_q<F_DU, G>(P, list, nn, i, sub, rs, sF, sU, nT, qx, qy, qz, dq, unused);
            else pair_sum_q<0, G>(P, list, nn, i, sub, rs, sF, sU, nT, qx, qy, qz, dq, unused);
          }
#pragma unroll
          for (int o = G / 2; o > 0; o >>= 1) {
            qx += __shfl_xor_sync(0xffffffffu, qx, o);
            qy += __shfl_xor_sync(0xffffffffu, qy, o);
            qz += __shfl_xor_sync(0xffffffffu, qz, o);
          }
          if (active && sub == 0) {
            fsum[3 * b] = qx;
            fsum[3 * b + 1] = qy;
            fsum[3 * b + 2] = qz;
          }
          if (trial) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) dq += __shfl_xor_sync(0xffffffffu, dq, o);
            if (lane == 0) atomicAdd((unsigned long long*)&sdq[0], (unsigned long long)dq);
          }
        } else {
          double fx = 0, fy = 0, fz = 0, ep = 0, dU = 0;
          int* q = queue + (size_t)(tid / G) * kPairQueue;
          const BeadList<false> list{P.nbr + (size_t)i * P.kmax, P.m4[cur]};
          const int nn = active ? P.nnbr[i] : 0;
          if (trial) pair_sum_d<F_DU, G>(P, cur, list, nn, i, sub, rs, sF, sU, nT, q, fx, fy, fz, ep, dU);
          else pair_sum_d<0, G>(P, cur, list, nn, i, sub, rs, sF, sU, nT, q, fx, fy, fz, ep, dU);
#pragma unroll
          for (int o = G / 2; o > 0; o >>= 1) {
            fx += __shfl_xor_sync(0xffffffffu, fx, o);
            fy += __shfl_xor_sync(0xffffffffu, fy, o);
            fz += __shfl_xor_sync(0xffffffffu, fz, o);
          }
          if (active && sub == 0) {
            fsum[3 * b] = fx;
            fsum[3 * b + 1] = fy;
            fsum[3 * b + 2] = fz;
          }
          if (trial) {
            dU = warp_sum(dU);
            if (lane == 0) atomicAdd(&sdu[0], dU);
          }
        }
      }
    }
    __syncthreads();

    // ---- acceleration of own bead tid
    double a[3] = {0, 0, 0}, x[3] = {0, 0, 0}, v[3] = {0, 0, 0};
    int ti = 0;
    unsigned int w = 0;
    if (tid < nb) {
      w = ref[tid].w;
      ti = w & 0xff;
      for (int d = 0; d < 3; ++d) {
        x[d] = st[d * NB + tid];
        v[d] = st[(3 + d) * NB + tid];
      }
      if constexpr (MIXED) {
        for (int d = 0; d < 3; ++d)
          a[d] = fma(-gamma, v[d], fma((double)fsum[3 * tid + d], T.inv_fscale, (double)fbond[3 * tid + d]));
      } else {
        double noise[3];
        langevin_noise(rp.seed, orig[tid] - rp.bead_begin, it, 0, rp.sig31, noise);
        for (int d = 0; d < 3; ++d) a[d] = fma(-gamma, v[d], fsum[3 * tid + d] + fbond[3 * tid + d]) + noise[d];
      }
      if (ti != 0)
        for (int d = 0; d < 3; ++d) v[d] = fma(a[d], h, v[d]);  // second half-kick
    }
    bool scaled = false;
    if (trial) {
      // ---- the trial's energy difference over the grid, and the decision by every CTA
      const int par = trials & 1;
      if (tid == 0) {
        if constexpr (MIXED) {
          atomicAdd((unsigned long long*)&A.trial[me.rep].dq_pair[par], (unsigned long long)sdq[0]);
          atomicAdd((unsigned long long*)&A.trial[me.rep].dq_bond[par], (unsigned long long)sdq[1]);
        } else {
          atomicAdd(&A.trial[me.rep].du_pair[par], sdu[0]);
          atomicAdd(&A.trial[me.rep].du_bond[par], sdu[1]);
        }
        if (me.index == 0) {  // the previous trial's words: every CTA read them before the barrier that ended its step
          A.trial[me.rep].dq_pair[par ^ 1] = A.trial[me.rep].dq_bond[par ^ 1] = 0;
          A.trial[me.rep].du_pair[par ^ 1] = A.trial[me.rep].du_bond[par ^ 1] = 0.0;
        }
      }
      if (!barrier(1)) return;
      // Past this barrier every CTA has read the previous trial's largest
      // displacement and shift (after the barrier that ended its step, the last
      // one before this where a period is one step); they are added to again
      // after the barrier that ends this step.  (Not by thread 0, whose decision
      // the whole CTA waits for.)
      if (tid == 32 && blockIdx.x == 0) {
        A.sync->dmax[par ^ 1] = 0;
        A.sync->shift[par ^ 1] = 0;
      }
      if (tid == 0) {
        rs.dUq_pair = __ldcg(&A.trial[me.rep].dq_pair[par]);
        rs.dUq_bond = __ldcg(&A.trial[me.rep].dq_bond[par]);
        rs.dU_pair = __ldcg(&A.trial[me.rep].du_pair[par]);
        rs.dU_bond = __ldcg(&A.trial[me.rep].du_bond[par]);
        rs.accept = 0;
        shift_s = 0.0;
        if (rp.dlxy != 0) {
          shift_s = decide_trial(rs, rp, T, P.trial_u[((size_t)slot * P.n_rep + me.rep) * 2 + 1]);
          if (me.index == 0) {
            P.accept_log[(size_t)slot * P.n_rep + me.rep] = rs.accept;
            if (rs.accept)
              atomicMax(&A.sync->shift[par], (unsigned long long)__double_as_longlong(shift_s));
          }
        }
        ++slot;
      }
      __syncthreads();
      scaled = rs.accept != 0;
      ++trials;
    }
    // ---- first half-kick and drift of the next step, its mirror and cell count
    phase = phase + 1 == A.rate ? 0 : phase + 1;
    const bool next_trial = A.barostat && phase == 0 && it + 1 != 0;
    float vmax = 0.f;
    if (tid < nb) {
      const int i = b0 + tid;
      if (scaled)
        for (int d = 0; d < 3; ++d) x[d] *= rs.scale[d];
      if (ti != 0) {
        for (int d = 0; d < 3; ++d) {
          v[d] = fma(a[d], h, v[d]);
          x[d] = wrap64(fma(v[d], dt, x[d]), rs.box[d]);
          st[(3 + d) * NB + tid] = v[d];
        }
      }
      for (int d = 0; d < 3; ++d) st[d * NB + tid] = x[d];
      if (A.save) {
        double* to = A.save + 3 * ((size_t)s * P.n + orig[tid]);
        for (int d = 0; d < 3; ++d) to[d] = x[d];
      }
      const uint4 mn = make_uint4(to_frac(x[0], rs.frac_per_len[0]), to_frac(x[1], rs.frac_per_len[1]),
                                  to_frac(x[2], rs.frac_per_len[2]), w);
      vmax = displacement(ref[tid], mn.x, mn.y, mn.z, rs);
      P.m4[cur ^ 1][i] = mn;
      if constexpr (!MIXED) P.d4[cur ^ 1][i] = make_double4(x[0], x[1], x[2], __longlong_as_double((long long)w));
      const int c = cell_of(mn);
      key[tid] = c;
      if (!last) atomicAdd(A.cnt + me.cnt + (size_t)(s & 1) * ncell4 + c, 1);
      if (next_trial && !last) P.refcell[i] = ref_key(x);
    }
    vmax = warp_max(vmax);
    if (lane == 0) smax[warp] = vmax;
    __syncthreads();
    // ---- arrive: a bead beyond the margin (half the skin less the slack) asks for new lists
    unsigned long long inc = 1;
    if (warp == 0) {
      const float bm = warp_max(lane < nw ? smax[lane] : 0.f);
      if (trial) {  // (the slack is not known yet)
        if (lane == 0 && bm > 0.f) atomicMax(&A.sync->dmax[(trials - 1) & 1], __float_as_uint(bm));
      } else if ((double)bm + slack > P.half_skin) {
        inc += 1ull << (40 + 8 * (s % 3));
      }
      if (last && lane == 0 && bm > 0.f) atomicMax(&P.g->dmax_bits, __float_as_uint(bm));
      // the first CTA clears the field of two steps ago (the next step's), which every CTA has read
      if (blockIdx.x == 0 && s >= 2) inc -= ((seen >> (40 + 8 * ((s + 1) % 3))) & 0xffull) << (40 + 8 * ((s + 1) % 3));
    }
    if (!barrier(inc)) return;
    if (tid == 0) {
      if (trial) {
        const int par = (trials - 1) & 1;
        slack += __longlong_as_double((long long)__ldcg(&A.sync->shift[par]));
        rebuild = (double)__uint_as_float(__ldcg(&A.sync->dmax[par])) + slack > P.half_skin;
      } else {
        rebuild = ((seen >> (40 + 8 * (s % 3))) & 0xffull) != 0;
      }
    }
    cur ^= 1;
    ++it;
    trial = next_trial;
    if (trial && !last) draw();
    __syncthreads();
  }

  // ---- exit: the CTA's beads back to global memory, the mirror where the host expects it
  const int want = A.cur ^ (A.steps & 1);
  if (tid < nb) {
    const int i = b0 + tid;
    P.x[i] = st[tid];
    P.y[i] = st[NB + tid];
    P.z[i] = st[2 * NB + tid];
    P.vx[i] = st[3 * NB + tid];
    P.vy[i] = st[4 * NB + tid];
    P.vz[i] = st[5 * NB + tid];
    P.ref[i] = ref[tid];
    P.cinfo[i] = cinfo[tid];
    if (cur != want) {
      P.m4[want][i] = P.m4[cur][i];
      if constexpr (!MIXED) P.d4[want][i] = P.d4[cur][i];
    }
  }
  if (me.index == 0) {
    for (int k = tid; k < (int)(sizeof(RepState) / 4); k += nt)
      reinterpret_cast<int*>(P.rs + me.rep)[k] = reinterpret_cast<const int*>(&rs)[k];
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&A.sync->left, 1u) == gridDim.x - 1) {  // every CTA has passed its last barrier
      __threadfence();
      *A.sync = RunSync{};
      for (int r = 0; r < P.n_rep; ++r) A.trial[r] = RunTrial{};
      P.g->slack = slack;
      P.g->rebuild = rebuild;
      P.g->n_rebuilds += rebuilds;
      P.g->trial_slot = slot;
      P.g->it = it;
      P.g->last_disp = __uint_as_float(atomicExch(&P.g->dmax_bits, 0u));
    }
  }
}

}  // namespace smd

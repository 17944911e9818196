// Non-bonded forces without any device allocation.
//
// Some callers cannot call cudaMalloc: code that runs while another framework
// owns the device memory through its own pool, or a latency-critical loop in
// which cudaMalloc's implicit device-wide synchronisation is not allowed.
// smd_pair_forces_static serves them: the caller passes device pointers for
// the inputs and the output, and the scratch of the cell list lives in the
// file-scope array below, reserved once on every GPU that loads the library
// (SMD_STATIC_MAX_BEADS / SMD_STATIC_MAX_CELLS bound what fits; about 2.1 MB).
//
// The array is shared by every call and keeps the last call's contents, so
// each call clears the cell counts before use; calls whose kernels overlap on
// the GPU (different streams, or different host threads on one device) race on
// it and must be serialised by the caller.  The first call on a device looks
// up the array's device address (cudaGetSymbolAddress); make that first call
// before any stream capture.  The cached address belongs to the CUDA context
// it was looked up in: after cudaDeviceReset of a device, this entry point
// must not be called on that device again in the same process.
//
// The inputs come from another framework and are not checked on the host.
// Every index the kernels derive from them stays inside the arrays whatever
// their values (smd_static_cell.h): cell coordinates are clamped into the
// grid and types are range-checked before any table lookup.  A bead whose
// position is not finite, or whose type or a neighbour's type is outside
// [0, n_types), gets a NaN force.  Positions must be wrapped into [0, L] for
// the forces to be those of the reference.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <atomic>
#include <cmath>
#include <string>

#include "../../include/softmold_gb300.h"
#include "smd_pair64.cuh"
#include "smd_static_cell.h"

namespace smd {
void set_last_error(const std::string& msg);
}

namespace {

constexpr int kMaxBeads = SMD_STATIC_MAX_BEADS;
constexpr int kMaxCells = SMD_STATIC_MAX_CELLS;
constexpr int kMaxDevices = 64;
constexpr int kThreads = 256;

// [sorted positions (double4) | sorted positions in FP32 (float4) | cell counts
// | cell starts (+1) | bead keys | bead slots]
struct Scratch {
  double4 pos[kMaxBeads];  // x, y, z, (type | file index << 32) as bits, cell order
  float4 posf[kMaxBeads];  // the same positions rounded to FP32
  int count[kMaxCells];
  int start[kMaxCells + 1];
  int key[kMaxBeads];
  int slot[kMaxBeads];
};
static __device__ __align__(256) unsigned char g_scratch[sizeof(Scratch)];

// Host side: device address of g_scratch, looked up once per device.  Two
// host threads making a first call on one device at the same time both look
// it up and store the same value.
std::atomic<Scratch*> g_scratch_addr[kMaxDevices];

struct Grid {
  int n[3];
  double cs[3];
  double box[3];
  float inv_cs[3];  // 1 / cs
  float boxf[3];
};

__global__ void k_static_clear(int* count, int ncells) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += gridDim.x * blockDim.x) count[c] = 0;
}

// Cell along one axis: smd_static::cell_coord, its FP64 division taken only
// where an FP32 quotient cannot decide.  Three roundings of 2^-24 put the FP32
// quotient within 1.8e-7 q of p / cs, below 7.4e-4 for q < 4096, so one more
// than 1e-3 from an integer has the division's integer part.
__device__ __forceinline__ int bin_coord(double p, double cs, float inv_cs, int n, int* flags) {
  const float q = (float)p * inv_cs;
  const float fr = q - floorf(q);
  if (q > 0.f && q < 4096.f && fr > 1e-3f && fr < 1.f - 1e-3f) {
    const int c = (int)q;
    return c >= n ? n - 1 : c;
  }
  return smd_static::cell_coord(p, cs, n, flags);
}

// CellOpt key with the reference's formula (int(p/cellSize), x>=n -> n-1),
// clamped into the grid (smd_static_cell.h): the key is always < ncells.
__global__ void __launch_bounds__(kThreads) k_static_bin(const double* pos, int n, Grid g, int* key, int* slot,
                                                         int* count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int flags = 0, c[3];
  for (int d = 0; d < 3; ++d) c[d] = bin_coord(pos[3 * i + d], g.cs[d], g.inv_cs[d], g.n[d], &flags);
  const int k = c[0] + c[1] * g.n[0] + c[2] * g.n[0] * g.n[1];
  key[i] = k;
  slot[i] = atomicAdd(&count[k], 1);
}

// Exclusive scan of the counts, one block: each thread sums 8 consecutive
// counts, so the largest grid takes four rounds (a 256-thread scan of one
// count each took 10.5 us of latency at 8,700 cells).
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) k_static_scan(const int* count, int* start, int ncells) {
  __shared__ int warp_sums[kScanThreads / 32];
  int carry = 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < ncells; base += 8 * kScanThreads) {
    const int c0 = base + 8 * threadIdx.x;
    int v[8], s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k] = c0 + k < ncells ? count[c0 + k] : 0;
      s += v[k];
    }
    int x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    int t = warp_sums[lane];  // every warp scans the warps' sums itself
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    const int total = __shfl_sync(0xffffffffu, t, 31);
    const int before = __shfl_sync(0xffffffffu, t, w > 0 ? w - 1 : 0);
    int ex = carry + (w > 0 ? before : 0) + x - s;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (c0 + k < ncells) start[c0 + k] = ex;
      ex += v[k];
    }
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) start[ncells] = carry;
}

__global__ void __launch_bounds__(kThreads) k_static_scatter(const double* pos, const int* type, const int* key,
                                                             const int* slot, const int* start, double4* spos,
                                                             float4* sposf, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int to = start[key[i]] + slot[i];
  const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  const long long w = ((long long)i << 32) | (unsigned int)type[i];
  spos[to] = make_double4(x, y, z, __longlong_as_double(w));
  sposf[to] = make_float4((float)x, (float)y, (float)z, 0.f);
}

// FP64 non-bonded force on every bead from the 27 surrounding cells, with the
// Force functor of include/MD.h:795-848 and the neighbour-shift minimum image.
// The table row is int(r/C0) (0 or 3 for the reference's tables, rc = 2 rm),
// taken as r >= C0 so that no table value can move the lookup outside the
// pair's 6 constants.  A bead with a non-finite position or a type outside
// [0, nT), or with a neighbour within rc whose type is outside it, gets NaN.
//
// GB300's FP64 pipe bounds this: an FP64 warp instruction holds it for ~25
// clocks of an SM, an FP32 one a quarter of a clock, and only one in seven of
// the 27 cells' beads lies within rc.  So eight lanes per bead (four beads of
// neighbouring cells per warp) first test the stencil in FP32, with a cut
// widened by the FP32 rounding of the positions, and queue what passes in
// shared memory; the FP64 distance, its exact test against rc and the force
// then run on full groups of queued beads.  A call on 29,400 beads: 170 us,
// against 2,176 us with one thread per bead and every test in FP64.
constexpr int kForceLanes = 8;
constexpr int kForceQueue = 128;  // queued neighbours per bead
constexpr int kSharedTypes = 8;   // tables up to this size are copied to shared memory
__global__ void __launch_bounds__(kThreads, 4) k_static_force(int n, Grid g, double rc2, int nT, const double* fC,
                                                              const int* start, const double4* spos,
                                                              const float4* sposf, float rcf, double* force) {
  __shared__ double tab_s[6 * kSharedTypes * kSharedTypes];
  __shared__ int queue_s[kThreads / kForceLanes][kForceQueue];
  const double* tab = fC;
  if (nT <= kSharedTypes) {
    for (int k = threadIdx.x; k < 6 * nT * nT; k += kThreads) tab_s[k] = fC[k];
    tab = tab_s;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, sub = lane & (kForceLanes - 1), grp = lane / kForceLanes;
  const int i = (blockIdx.x * kThreads + threadIdx.x) / kForceLanes;
  const bool active = i < n;
  double4 me = make_double4(0.0, 0.0, 0.0, 0.0);
  float4 mf = make_float4(0.f, 0.f, 0.f, 0.f);
  int ti = 0, flags = 0, cx = 0, cy = 0, cz = 0;
  if (active) {
    me = spos[i];
    mf = sposf[i];
    ti = (int)(__double_as_longlong(me.w) & 0xffffffffll);
    cx = bin_coord(me.x, g.cs[0], g.inv_cs[0], g.n[0], &flags);
    cy = bin_coord(me.y, g.cs[1], g.inv_cs[1], g.n[1], &flags);
    cz = bin_coord(me.z, g.cs[2], g.inv_cs[2], g.n[2], &flags);
    if (!smd_static::type_ok(ti, nT)) flags |= smd_static::kStaticBadType;
  }
  // x-rows of the stencil: cells cx-1 .. cx+1 of a row are contiguous, or two
  // ranges where they wrap; lane k of the group holds rows k and k + 8
  int s0[2] = {0, 0}, l0[2] = {0, 0}, s1[2] = {0, 0}, l1[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = sub + h * kForceLanes;
    if (t < 9 && active && flags == 0) {
      const int yy = (cy + t % 3 - 1 + g.n[1]) % g.n[1], zz = (cz + t / 3 - 1 + g.n[2]) % g.n[2];
      const int row = g.n[0] * (yy + g.n[1] * zz);
      const int xa = cx - 1, xb = cx + 1;
      s0[h] = start[row + (xa < 0 ? g.n[0] - 1 : xa)];
      l0[h] = start[row + (xa < 0 || xb >= g.n[0] ? g.n[0] : xb + 1)] - s0[h];
      if (xa < 0 || xb >= g.n[0]) {
        s1[h] = start[row];
        l1[h] = start[row + (xa < 0 ? xb + 1 : 1)] - s1[h];
      }
    }
  }
  // FP32 cut: per axis the rounding of both positions, of L and of the two
  // subtractions stays below 4e-7 (|x_i| + L + rc) for every neighbour within rc
  const float slop = 4e-7f * (fabsf(mf.x) + fabsf(mf.y) + fabsf(mf.z) + g.boxf[0] + g.boxf[1] + g.boxf[2] + 3.f * rcf);
  const float cut = rcf * (1.f + 2e-6f) + slop;
  const float cut2 = cut * cut;
  const float hx = 0.5f * g.boxf[0], hy = 0.5f * g.boxf[1], hz = 0.5f * g.boxf[2];
  const int bhx = __double2hiint(0.5 * g.box[0]), bhy = __double2hiint(0.5 * g.box[1]),
            bhz = __double2hiint(0.5 * g.box[2]);
  int* queue = queue_s[threadIdx.x / kForceLanes];
  int queued = 0;
  double fx = 0, fy = 0, fz = 0;
  auto drain = [&]() {
    __syncwarp();
    for (int k = sub; k < queued; k += kForceLanes) {
      const double4 o = spos[queue[k]];
      const double dx = smd::image64(me.x, o.x, g.box[0], bhx), dy = smd::image64(me.y, o.y, g.box[1], bhy),
                   dz = smd::image64(me.z, o.z, g.box[2], bhz);
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (r2 < rc2) {  // false for a neighbour whose position is not finite
        const int tj = (int)(__double_as_longlong(o.w) & 0xffffffffll);
        if (!smd_static::type_ok(tj, nT)) {
          flags |= smd_static::kStaticBadType;
          continue;
        }
        const double mag = smd::pair_mag64(tab + 6 * (ti * nT + tj), r2);
        fx += dx * mag;
        fy += dy * mag;
        fz += dz * mag;
      }
    }
    queued = 0;
    __syncwarp();
  };
  const unsigned int below = (1u << lane) - 1u;
  const unsigned int mine = ((1u << kForceLanes) - 1u) << (grp * kForceLanes);
  for (int t = 0; t < 9; ++t) {
    const int src = grp * kForceLanes + (t & (kForceLanes - 1));
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int a = __shfl_sync(0xffffffffu, half ? (t < kForceLanes ? s1[0] : s1[1]) : (t < kForceLanes ? s0[0] : s0[1]), src);
      const int len = __shfl_sync(0xffffffffu, half ? (t < kForceLanes ? l1[0] : l1[1]) : (t < kForceLanes ? l0[0] : l0[1]), src);
      const int longest = __reduce_max_sync(0xffffffffu, len);
      for (int k0 = 0; k0 < longest; k0 += kForceLanes) {
        const int j = a + k0 + sub;
        bool near = false;
        if (k0 + sub < len) {
          const float4 o = sposf[j];
          float dx = mf.x - o.x, dy = mf.y - o.y, dz = mf.z - o.z;
          if (fabsf(dx) > hx) dx -= copysignf(g.boxf[0], dx);
          if (fabsf(dy) > hy) dy -= copysignf(g.boxf[1], dy);
          if (fabsf(dz) > hz) dz -= copysignf(g.boxf[2], dz);
          near = !(dx * dx + dy * dy + dz * dz > cut2) && j != i;  // a NaN goes on to the FP64 test
        }
        const unsigned int hits = __ballot_sync(0xffffffffu, near) & mine;
        if (near) queue[queued + __popc(hits & below)] = j;
        queued += __popc(hits);
        if (__any_sync(0xffffffffu, queued > kForceQueue - kForceLanes)) drain();
      }
    }
  }
  drain();
#pragma unroll
  for (int o = kForceLanes / 2; o > 0; o >>= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o);
    fy += __shfl_xor_sync(0xffffffffu, fy, o);
    fz += __shfl_xor_sync(0xffffffffu, fz, o);
    flags |= __shfl_xor_sync(0xffffffffu, flags, o);
  }
  if (active && sub == 0) {
    if (flags != 0) fx = fy = fz = CUDART_NAN;
    const size_t o = 3 * (size_t)(__double_as_longlong(me.w) >> 32);
    force[o] = fx;
    force[o + 1] = fy;
    force[o + 2] = fz;
  }
}

int error(int code, const std::string& msg) {
  smd::set_last_error(msg);
  return code;
}

}  // namespace

extern "C" int smd_pair_forces_static(const double* d_pos, const int* d_type, int n, const double box[3],
                                      double cutoff, int n_types, const double* d_fconst, double* d_force,
                                      void* stream) {
  if (!d_pos || !d_type || !d_fconst || !d_force || !box || n < 0)
    return error(1, "smd_pair_forces_static: null pointer or negative size");
  if (n > kMaxBeads)
    return error(1, "smd_pair_forces_static: " + std::to_string(n) + " beads exceed the static maximum of " +
                        std::to_string(kMaxBeads));
  if (!(cutoff > 0) || !std::isfinite(cutoff) || n_types <= 0)
    return error(1, "smd_pair_forces_static: bad cutoff or n_types");
  Grid g;
  long long cells = 1;
  for (int d = 0; d < 3; ++d) {
    if (!std::isfinite(box[d]) || !(box[d] > 0))
      return error(1, "smd_pair_forces_static: box edges must be finite and positive");
    const double per_axis = box[d] / cutoff;  // compared before any conversion to int
    if (!(per_axis < (double)kMaxCells + 1.0))
      return error(1, "smd_pair_forces_static: box edge / cutoff exceeds the static maximum of " +
                          std::to_string(kMaxCells) + " cells");
    g.box[d] = box[d];
    g.n[d] = int(per_axis);
    if (g.n[d] < 3) return error(1, "smd_pair_forces_static: box edge shorter than 3 cutoffs");
    g.cs[d] = box[d] / g.n[d];
    g.inv_cs[d] = (float)(1.0 / g.cs[d]);
    g.boxf[d] = (float)box[d];
    cells *= g.n[d];
    if (cells > kMaxCells)
      return error(1, "smd_pair_forces_static: the grid's cells exceed the static maximum of " +
                          std::to_string(kMaxCells));
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();  // reported here, not by the caller's next launch check
    return error(100 + (int)e, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  }
  if (dev < 0 || dev >= kMaxDevices) return error(1, "smd_pair_forces_static: device index out of range");
  Scratch* w = g_scratch_addr[dev].load(std::memory_order_acquire);
  if (!w) {
    e = cudaGetSymbolAddress((void**)&w, g_scratch);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return error(100 + (int)e, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    }
    g_scratch_addr[dev].store(w, std::memory_order_release);
  }
  if (n == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const int nc = (int)cells;
  const int gb = (n + kThreads - 1) / kThreads;
  k_static_clear<<<(nc + kThreads - 1) / kThreads, kThreads, 0, s>>>(w->count, nc);
  k_static_bin<<<gb, kThreads, 0, s>>>(d_pos, n, g, w->key, w->slot, w->count);
  k_static_scan<<<1, kScanThreads, 0, s>>>(w->count, w->start, nc);
  k_static_scatter<<<gb, kThreads, 0, s>>>(d_pos, d_type, w->key, w->slot, w->start, w->pos, w->posf, n);
  const int gf = (n * kForceLanes + kThreads - 1) / kThreads;
  k_static_force<<<gf, kThreads, 0, s>>>(n, g, cutoff * cutoff, n_types, d_fconst, w->start, w->pos, w->posf,
                                         (float)cutoff, d_force);
  e = cudaGetLastError();
  if (e != cudaSuccess) return error(200 + (int)e, std::string("kernel launch: ") + cudaGetErrorString(e));
  return 0;
}

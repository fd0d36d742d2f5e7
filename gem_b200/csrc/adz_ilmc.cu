// ILMC shape-preserving filter (B/ILMC_LAM.F90:16-388 with
// B/ilmc_lam_loop.inc): each point outside its [min, max] bounds moves its
// excess (or deficit) of air-mass-weighted tracer into the room its
// neighbours have, shell by shell (sweeps), then an optional clip.
//
// The reference visits the points in loop order (k, then j, then i) and
// every visit changes the point's neighbourhood, so later visits see earlier
// results.  This file keeps that order exactly and still runs in parallel.
// A visit reads and writes only the cube of radius S = sweep_max around its
// point, so a visit can depend only on earlier points within R = 2 S
// (Chebyshev).  The region is cut into tiles of one row and R columns,
// numbered (k, j, it); every earlier point within R of a
// tile's point lies in the same tile (handled in order by one warp) or in a
// tile of strictly smaller wavefront number
//     t = (2 R + 2) k + 2 j + it
// (a level below: at most R rows and one tile column away; the same level: an
// earlier row, at most one tile column away; the same row: the tile before).
// Tiles of one wavefront therefore never interact, and running the wavefronts
// in increasing t, each tile by one warp in loop order, reproduces the
// sequential result bit for bit.  Within a visit the lanes split the shell's
// loads and updates; every lane forms the capacity sum in the reference's order.
//
// A visit moves a neighbour only toward its bounds (it gains up to its max or
// loses down to its min) and its own point into them, so a point inside its
// bounds when the filter starts stays inside, and the reference's visit of it
// does nothing.  Candidate tiles (a point outside its bounds at the start)
// are therefore listed per wavefront once (count, scan, scatter), and a warp
// loads a tile's points at once and visits, in order, only those that were
// outside.
//
// What bounds the filter is the chain of wavefronts (10 per level, 2 per row
// at two sweeps), each as long as its slowest tile: a few dependent loads.
// One cooperative kernel runs them all, with a barrier over the grid between
// two non-empty wavefronts; a launch per wavefront costs several times the
// barrier.  A visit loads every shell's values at once (the shells are
// disjoint, so a sweep changes only its own shell and the centre), each
// lane's cells stay in registers, and the list entry and bounds of a warp's
// next tile are loaded before the barrier.  Bounds and cubes of 3 tracers at
// 301 x 262 x 80, 3.4 % of the points outside, two sweeps: 20.4 ms with a launch
// per wavefront (15 us each), 8.1 ms here (6 us).  1 % outside, one to four
// sweeps: 8.1, 17.6, 39.0, 84.0 ms with launches, 4.3, 6.5, 8.9, 38.6 here (FP64 8.4,
// 18.8, 43.3, 92.3 and 4.6, 6.5, 10.8, 58.9).  The values of four sweeps do not fit the
// registers (552 bytes a lane in local memory, 960 in FP64): 30 % outside, 1024
// x 512 x 80, FP64, took 704 ms with launches and takes 750.
// Built with -fmad=false: the REAL arithmetic is the reference's, without
// contraction.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/adz_b200.h"
#include "adz_internal.h"
#include "adz_types.h"

namespace adz {
namespace ilmc {

struct Box {
  int il, ir, jl, jr, k0, nk;
  int lminx, lminy, nit;
  long long nij;
  __host__ __device__ int bx() const { return ir - il + 1; }
  __host__ __device__ int by() const { return jr - jl + 1; }
  __host__ __device__ long long n() const { return (long long)bx() * by() * (nk - k0 + 1); }
};

__device__ __forceinline__ long long ext(const Box& b, int i, int j, int k) {
  return (long long)(i - b.lminx) + (long long)(j - b.lminy) * b.nit + (long long)(k - 1) * b.nij;
}

template <typename T>
__device__ __forceinline__ T rmax(T a, T b) { return a > b ? a : b; }
template <typename T>
__device__ __forceinline__ T rmin(T a, T b) { return a < b ? a : b; }

constexpr int kWarps = 16;  // tiles (warps) per block of k_waves
constexpr unsigned long long kBarrierSpins = 1ull << 24;  // several seconds
// columns per tile: R = 2 sweep_max, the narrowest width the wavefront order
// allows (a tile's visits are sequential, so narrow tiles shorten each wave)
inline int tile_width(int sweep_max) { return 2 * sweep_max; }

template <typename T>
struct Fields {
  T* f[ADZC_ILMC_MAX_TRACERS];
  const T* mn[ADZC_ILMC_MAX_TRACERS];
  const T* mx[ADZC_ILMC_MAX_TRACERS];
};

// cells of sweep sw's unclipped shell, its 32-cell slots, and the slots of
// the sweeps before it (sw 1..4)
__host__ __device__ constexpr int shell_len(int sw) { return 24 * sw * sw + 2; }
__host__ __device__ constexpr int shell_slots(int sw) { return (shell_len(sw) + 31) / 32; }
__host__ __device__ constexpr int first_slot(int sw) { return sw == 1 ? 0 : sw == 2 ? 1 : sw == 3 ? 5 : 12; }

// cell q of sweep sw's unclipped shell in the order of the reference's
// sweep_rd list (B/ILMC_LAM.F90:118-169: dj, then dk, then di; inside the
// shell's faces only the two ends of di).  A shell clipped to the region is
// this list filtered to the region, in the same order.
__device__ inline void shell_cell(int sw, int q, int& di, int& dj, int& dk) {
  const int side = 2 * sw + 1, ring = 2 * side + 2 * (side - 2);  // cells of an inner plane: two full rows, the rest ends
  const int face = side * side;
  if (q < face) {
    dj = -sw;
    dk = q / side - sw;
    di = q % side - sw;
    return;
  }
  q -= face;
  if (q >= (side - 2) * ring) {
    q -= (side - 2) * ring;
    dj = sw;
    dk = q / side - sw;
    di = q % side - sw;
    return;
  }
  dj = q / ring - sw + 1;
  q %= ring;
  if (q < side) {
    dk = -sw;
    di = q - sw;
  } else if (q >= ring - side) {
    dk = sw;
    di = q - (ring - side) - sw;
  } else {
    q -= side;
    dk = q / 2 - sw + 1;
    di = (q & 1) ? sw : -sw;
  }
}

// a lane's shell cells: offset in the extended array, packed (di, dj, dk)
template <int S>
struct Cells {
  static constexpr int N = first_slot(S) + shell_slots(S);
  int off[N], d[N];  // d < 0: no cell
};

// one visit by a warp of the point e = (i, j, k) with its value and bounds.
// Lane l owns the cells l, l + 32, ... of each shell; every lane adds up the
// capacities in the reference's order, from shared memory.  f is read and
// written past L1: other SMs' wavefronts wrote it.
template <typename T, int S>
__device__ __forceinline__ void visit_warp(const Box& b, const Cells<S>& cl, T* f, const T* mn, const T* mx,
                                           const T* air, int i, int j, int k, long long e, T fe, T mne, T mxe,
                                           int lane, T* prod) {
  T o_shoot = rmax((T)0, fe - mxe);
  T u_shoot = rmax((T)0, mne - fe);
  if (o_shoot == (T)0 && u_shoot == (T)0) return;
  const bool over = o_shoot > (T)0;
  const T* bound = over ? mx : mn;
  constexpr int N = Cells<S>::N;
  T fv[N], bv[N], av[N];
  unsigned in = 0;
  const bool inner = i - S >= b.il && i + S <= b.ir && j - S >= b.jl && j + S <= b.jr && k - S >= b.k0 && k + S <= b.nk;
#pragma unroll
  for (int q = 0; q < N; q++) {
    bool use = cl.d[q] >= 0;
    if (!inner && use) {
      const int ix = i + (cl.d[q] & 15) - 4, jx = j + ((cl.d[q] >> 4) & 15) - 4, kx = k + (cl.d[q] >> 8) - 4;
      use = ix >= b.il && ix <= b.ir && jx >= b.jl && jx <= b.jr && kx >= b.k0 && kx <= b.nk;
    }
    fv[q] = bv[q] = av[q] = (T)0;
    if (use) {
      fv[q] = __ldcg(f + e + cl.off[q]);
      bv[q] = __ldg(bound + e + cl.off[q]);
      av[q] = __ldg(air + e + cl.off[q]);
      in |= 1u << q;
    }
  }
  const T aire = __ldg(air + e);
#pragma unroll
  for (int sw = 1; sw <= S; sw++) {
    if ((over ? o_shoot : u_shoot) == (T)0) break;  // nothing left to move: the later sweeps change nothing
    const int q0 = first_slot(sw), nq = shell_len(sw);
    T cap[shell_slots(S)];
#pragma unroll
    for (int q = 0; q < shell_slots(sw); q++) {
      const int s = q0 + q;
      cap[q] = (in >> s) & 1u ? (over ? rmax((T)0, bv[s] - fv[s]) : rmax((T)0, fv[s] - bv[s])) : (T)0;
      prod[lane + 32 * q] = cap[q] * av[s];
    }
    __syncwarp();
    // the reference skips cells outside the region; their prod is +0 and
    // msum >= +0, so adding it leaves msum unchanged bit for bit
    T msum = 0;
    constexpr int V = 16 / sizeof(T);  // the shell's last vector is filled up with +0
    struct alignas(16) Vec {
      T x[V];
    };
#pragma unroll 8
    for (int q = 0; q < (nq + V - 1) / V; q++) {
      const Vec p = reinterpret_cast<const Vec*>(prod)[q];
#pragma unroll
      for (int c = 0; c < V; c++) msum = p.x[c] + msum;
    }
    __syncwarp();  // prod is written again in the next sweep
    const T use = rmin(msum, (over ? o_shoot : u_shoot) * aire);
    if (use > (T)0) {
      if (over) {
        fe = rmax(fe - (T)(use / aire), mne);
        o_shoot = rmax((T)0, fe - mxe);
      } else {
        fe = rmin(fe + (T)(use / aire), mxe);
        u_shoot = rmax((T)0, mne - fe);
      }
      if (lane == 0) __stcg(f + e, fe);
      const T ratio = use / msum;
#pragma unroll
      for (int q = 0; q < shell_slots(sw); q++) {
        const int s = q0 + q;
        if (cap[q] > (T)0)
          __stcg(f + e + cl.off[s],
                 over ? rmin(fv[s] + (T)(cap[q] * ratio), bv[s]) : rmax(fv[s] - (T)(cap[q] * ratio), bv[s]));
      }
    }
  }
}

// tile id (tracer, level, tile column) and the row it has in wavefront t
__device__ __forceinline__ int tile_row(int t, int c1, int kk, int it) { return (t - c1 * kk - it) >> 1; }

// candidate tiles per wavefront.  pass 0 counts them, pass 1 lists their ids
// (order inside a wave is free: its tiles never interact)
template <typename T, int PASS>
__global__ void __launch_bounds__(256) k_candidates(Box b, Fields<T> fl, int ntr, int c1, int ntile, int tw,
                                                    int* __restrict__ count, const int* __restrict__ wstart,
                                                    int* __restrict__ list) {
  const int nz = b.nk - b.k0 + 1, ny = b.by();
  const long long n = (long long)ntr * nz * ny * ntile;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n; g += (long long)gridDim.x * blockDim.x) {
    const int it = (int)(g % ntile);
    const int jr = (int)((g / ntile) % ny);
    const long long rest = g / ((long long)ntile * ny);
    const int kk = (int)(rest % nz), tr = (int)(rest / nz);
    const int j = b.jl + jr, k = b.k0 + kk;
    const int i0 = b.il + it * tw, i1 = min(i0 + tw - 1, b.ir);
    const T* f = fl.f[tr];
    const T* mn = fl.mn[tr];
    const T* mx = fl.mx[tr];
    bool any = false;
    for (int i = i0; i <= i1; i++) {
      const long long e = ext(b, i, j, k);
      const T v = f[e];
      any |= (v > mx[e]) || (v < mn[e]);
    }
    if (!any) continue;
    const int t = c1 * kk + 2 * jr + it;
    if (PASS == 0) {
      atomicAdd(count + t, 1);
    } else {
      list[wstart[t] + atomicAdd(count + t, 1)] = (tr * nz + kk) * ntile + it;
    }
  }
}

// exclusive scan of the per-wave counts (one block): wstart[0..n]
__global__ void __launch_bounds__(1024) k_scan(const int* __restrict__ count, int n, int* __restrict__ wstart) {
  __shared__ int part[1024];
  const int per = (n + 1023) / 1024, a = threadIdx.x * per, z = min(a + per, n);
  int sum = 0;
  for (int q = a; q < z; q++) sum += count[q];
  part[threadIdx.x] = sum;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {  // inclusive Hillis-Steele
    const int v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  int run = part[threadIdx.x] - sum;
  for (int q = a; q < z; q++) {
    wstart[q] = run;
    run += count[q];
  }
  if (threadIdx.x == 1023) wstart[n] = part[1023];
}

// every wavefront in turn: a warp per listed tile, its points in loop order,
// then a barrier over the grid.  64 registers up to two FP32 sweeps (10.5 ms at
// the 74 that ptxas takes, 9.6 at 64).  bar counts the blocks that have arrived.
// The wait is bounded: when it runs out the block raises kErrTimeout and
// leaves, and so do the others.
template <typename T, int S>
__global__ void __launch_bounds__(32 * kWarps, S <= 2 && sizeof(T) == 4 ? 2 : 1) k_waves(Box b, Fields<T> fl, const T* __restrict__ air, int nwave, int c1,
                                                       int ntile, const int* __restrict__ wstart,
                                                       const int* __restrict__ list, unsigned long long* bar,
                                                       int* status) {
  constexpr int TW = 2 * S, PAD = 32 * shell_slots(S);
  extern __shared__ __align__(16) unsigned char ilmc_dyn[];
  __shared__ int s_stop;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T* prod = reinterpret_cast<T*>(ilmc_dyn) + w * PAD;
  const int nz = b.nk - b.k0 + 1;
  Cells<S> cl;
#pragma unroll
  for (int sw = 1; sw <= S; sw++)
#pragma unroll
    for (int q = 0; q < shell_slots(sw); q++) {
      const int c = lane + 32 * q, s = first_slot(sw) + q;
      int di = 0, dj = 0, dk = 0;
      if (c < shell_len(sw)) shell_cell(sw, c, di, dj, dk);
      cl.d[s] = c < shell_len(sw) ? (di + 4) | ((dj + 4) << 4) | ((dk + 4) << 8) : -1;
      cl.off[s] = di + dj * b.nit + dk * (int)b.nij;
    }
  unsigned long long arrived = 0;
  // tile of this warp in a wavefront: consecutive tiles on consecutive blocks
  const int first = blockIdx.x + w * gridDim.x, stride = gridDim.x * kWarps;
  int beg = wstart[0], end = wstart[1];
  int id = beg + first < end ? list[beg + first] : -1;  // the warp's next tile
  T vmn = 0, vmx = 0;
  long long e = 0;
  int i0 = 0, j = 0, k = 0, n = 0;
  T* f = nullptr;
  const T* mn = nullptr;
  const T* mx = nullptr;
  // where tile id of wavefront t lies, and its points' bounds (a lane each)
  auto open = [&](int t) {
    const int it = id % ntile, r = id / ntile, kk = r % nz, tr = r / nz;
    j = b.jl + tile_row(t, c1, kk, it);
    k = b.k0 + kk;
    i0 = b.il + it * TW;
    n = min(TW, b.ir - i0 + 1);
    f = fl.f[tr];
    mn = fl.mn[tr];
    mx = fl.mx[tr];
    e = ext(b, i0, j, k) + min(lane, n - 1);
    vmn = __ldg(mn + e);
    vmx = __ldg(mx + e);
  };
  if (id >= 0) open(0);
  for (int t = 0; t < nwave; t++) {
    const bool any = beg < end;
    for (int q = beg + first; q < end; q += stride) {
      if (q != beg + first) {
        id = list[q];
        open(t);
      }
      T v = __ldcg(f + e);
      unsigned todo = __ballot_sync(0xffffffffu, lane < n && ((v > vmx) || (v < vmn)));
      while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1;
        const T fe = __shfl_sync(0xffffffffu, v, l), mne = __shfl_sync(0xffffffffu, vmn, l);
        const T mxe = __shfl_sync(0xffffffffu, vmx, l);
        visit_warp<T, S>(b, cl, f, mn, mx, air, i0 + l, j, k, ext(b, i0 + l, j, k), fe, mne, mxe, lane, prod);
        __syncwarp();
        if (todo) v = __ldcg(f + e);  // the visit may have moved the tile's other points
      }
    }
    if (t == nwave - 1) break;
    beg = end;
    end = wstart[t + 2];
    if (beg + first < end) {
      id = list[beg + first];
      open(t + 1);
    }
    if (!any) continue;
    // barrier over the grid
    arrived += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
      s_stop = 0;
      __threadfence();
      atomicAdd(bar, 1ull);
      unsigned long long v, spins = 0;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
        if (v >= arrived) break;
        if (++spins > kBarrierSpins) {
          s_stop = 1;
          if (status) atomicOr(status, kErrTimeout);
          break;
        }
      }
    }
    __syncthreads();
    if (s_stop) return;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_clip(Box b, T* __restrict__ f, const T* __restrict__ mn,
                                              const T* __restrict__ mx) {
  const int by = b.by();
  for (long long row = blockIdx.x; row < (long long)by * (b.nk - b.k0 + 1); row += gridDim.x) {
    const int j = b.jl + (int)(row % by), k = b.k0 + (int)(row / by);
    for (int i = b.il + threadIdx.x; i <= b.ir; i += blockDim.x) {
      const long long e = ext(b, i, j, k);
      T v = f[e];
      if (v < mn[e]) v = mn[e];
      if (v > mx[e]) v = mx[e];
      f[e] = v;
    }
  }
}

}  // namespace ilmc
}  // namespace adz

namespace {

using namespace adz::ilmc;

// SMs that the kernels of a stream run on: all of the device's, or those of
// the green context that the stream belongs to
int stream_sms(cudaStream_t s, int sms) {
  struct Driver {
    CUresult (*stream_ctx)(CUstream, CUcontext*, CUgreenCtx*) = nullptr;
    CUresult (*resource)(CUgreenCtx, CUdevResource*, CUdevResourceType) = nullptr;
    Driver() {  // through the runtime: the library loads without a driver
      cudaDriverEntryPointQueryResult q;
      void* p = nullptr;
      if (cudaGetDriverEntryPointByVersion("cuStreamGetCtx", &p, 12050, cudaEnableDefault, &q) != cudaSuccess || !p)
        return;
      stream_ctx = (decltype(stream_ctx))p;
      p = nullptr;
      if (cudaGetDriverEntryPointByVersion("cuGreenCtxGetDevResource", &p, 12040, cudaEnableDefault, &q) == cudaSuccess)
        resource = (decltype(resource))p;
    }
  };
  static const Driver d;
  CUcontext ctx = nullptr;
  CUgreenCtx green = nullptr;
  CUdevResource r{};
  if (!d.stream_ctx || !d.resource || d.stream_ctx((CUstream)s, &ctx, &green) != CUDA_SUCCESS || !green ||
      d.resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS || r.sm.smCount < 1)
    return sms;
  return std::min(sms, (int)r.sm.smCount);
}

// the cooperative launch of every wavefront, one block per SM of the stream
// (all of them run at once; a tile loop strides by the grid, so any number does)
template <typename T, int S>
cudaError_t launch_waves(const Box& b, const Fields<T>& fl, const T* air, int nwave, int c1, int ntile,
                         const int* wstart, const int* list, unsigned long long* bar, int* status, cudaStream_t s) {
  constexpr int smem = kWarps * 32 * shell_slots(S) * (int)sizeof(T);
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaFuncSetAttribute(k_waves<T, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_waves<T, S>, 32 * kWarps, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  const int grid = stream_sms(s, sms);  // two per SM lengthen the barrier: 9.9 against 9.6 ms (8 tracers at 1024 x 1024 x 80: 77.9, 77.0)
  Box bb = b;
  Fields<T> ff = fl;
  void* args[] = {&bb, &ff, &air, &nwave, &c1, &ntile, &wstart, &list, &bar, &status};
  return cudaLaunchCooperativeKernel((const void*)k_waves<T, S>, dim3(grid), dim3(32 * kWarps), args, (size_t)smem, s);
}

template <typename T>
int run_ilmc(adzc_handle* h, const Box& b, int ntr, void* const* f, const void* const* mn, const void* const* mx,
             const T* air, int sweep_max, int min_max, int* waves, int* status, cudaStream_t s) {
  Fields<T> fl{};
  for (int q = 0; q < ntr; q++) {
    fl.f[q] = (T*)f[q];
    fl.mn[q] = (const T*)mn[q];
    fl.mx[q] = (const T*)mx[q];
  }
  const int R = 2 * sweep_max, c1 = 2 * R + 2;
  const int tw = tile_width(sweep_max);
  const int nz = b.nk - b.k0 + 1, ny = b.by(), ntile = (b.bx() + tw - 1) / tw;
  const int nwave = c1 * (nz - 1) + 2 * (ny - 1) + (ntile - 1) + 1;
  const long long ntiles = (long long)ntr * nz * ny * ntile;
  if ((long long)ntr * nz * ntile > (1LL << 31) - 1 || ntiles > (1LL << 31) - 1) return ADZC_ERR_SIZE;
  // scratch: barrier counter (8 B), count[nwave], wstart[nwave + 1], list[ntiles] (ints)
  void* scratch = nullptr;
  const size_t nint = 2 + (size_t)nwave * 2 + 1 + (size_t)ntiles;
  if (adz_internal_aux(h, nint * sizeof(int), &scratch) != ADZC_OK) return ADZC_ERR_ALLOC;
  unsigned long long* bar = (unsigned long long*)scratch;
  int* count = (int*)scratch + 2;
  int* wstart = count + nwave;
  int* list = wstart + nwave + 1;
  const int gc = (int)std::max<long long>(1, std::min<long long>((ntiles + 255) / 256, 148LL * 16));
  if (cudaMemsetAsync(bar, 0, (size_t)(nwave + 2) * sizeof(int), s) != cudaSuccess) return ADZC_ERR_CUDA;
  k_candidates<T, 0><<<gc, 256, 0, s>>>(b, fl, ntr, c1, ntile, tw, count, nullptr, nullptr);
  k_scan<<<1, 1024, 0, s>>>(count, nwave, wstart);
  if (cudaMemsetAsync(count, 0, (size_t)nwave * sizeof(int), s) != cudaSuccess) return ADZC_ERR_CUDA;
  k_candidates<T, 1><<<gc, 256, 0, s>>>(b, fl, ntr, c1, ntile, tw, count, wstart, list);
  cudaError_t le;
  switch (sweep_max) {
    case 1: le = launch_waves<T, 1>(b, fl, air, nwave, c1, ntile, wstart, list, bar, status, s); break;
    case 2: le = launch_waves<T, 2>(b, fl, air, nwave, c1, ntile, wstart, list, bar, status, s); break;
    case 3: le = launch_waves<T, 3>(b, fl, air, nwave, c1, ntile, wstart, list, bar, status, s); break;
    default: le = launch_waves<T, 4>(b, fl, air, nwave, c1, ntile, wstart, list, bar, status, s); break;
  }
  if (le != cudaSuccess) return ADZC_ERR_CUDA;
  if (min_max) {
    const long long rows = (long long)ny * nz;
    const int gr = (int)std::min<long long>(rows, 148LL * 16);
    for (int q = 0; q < ntr; q++) k_clip<T><<<gr, 256, 0, s>>>(b, fl.f[q], fl.mn[q], fl.mx[q]);
  }
  if (waves) *waves = nwave;
  return cudaGetLastError() == cudaSuccess ? ADZC_OK : ADZC_ERR_CUDA;
}

}  // namespace

extern "C" int adzc_ilmc(adzc_handle* h, int prec, int ntr, void* const* f, const void* const* mn,
                         const void* const* mx, const void* air, int sweep_max, int min_max, int* rounds,
                         void* stream) {
  AdzRange nvtx_range("ILMC_LAM");
  adz::DGrid D;
  adzc_info I;
  adzc_grid G;
  int niter = 0, cold = 0;
  if (!h || (prec != ADZC_REF32 && prec != ADZC_MIXED && prec != ADZC_FP64) || ntr < 0 ||
      ntr > ADZC_ILMC_MAX_TRACERS || (ntr > 0 && (!f || !mn || !mx)) || !air || sweep_max < 1 || sweep_max > 4 ||
      adz_internal_view(h, &D, &I, &G, &niter, &cold) != ADZC_OK)
    return adz_internal_fail(ADZC_ERR_ARG);
  for (int q = 0; q < ntr; q++)
    if (!f[q] || !mn[q] || !mx[q]) return adz_internal_fail(ADZC_ERR_ARG);
  if (rounds) *rounds = 0;
  if (ntr == 0) return ADZC_OK;
  // single LAM domain: il..ir, jl..jr = Adz_i0..Adz_in, Adz_j0..Adz_jn (B/ILMC_LAM.F90:57-63), levels k0t..nk
  Box b{I.i0, I.in, I.j0, I.jn, I.k0t, D.nk, D.lminx, D.lminy, D.nit, D.nij};
  if (b.n() <= 0) return adz_internal_fail(ADZC_ERR_ARG);
  const cudaStream_t s = (cudaStream_t)stream;
  const int st = prec == ADZC_FP64 ? run_ilmc<double>(h, b, ntr, f, mn, mx, (const double*)air, sweep_max,
                                                      min_max, rounds, D.status, s)
                                   : run_ilmc<float>(h, b, ntr, f, mn, mx, (const float*)air, sweep_max, min_max,
                                                     rounds, D.status, s);
  return st == ADZC_OK ? ADZC_OK : adz_internal_fail(st);
}

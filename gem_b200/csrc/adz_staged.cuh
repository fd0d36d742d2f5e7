// The gather kernels of the step on shared-memory boxes.
//
// A departure point's stencil is 64 values at addresses that are consecutive
// in x across a warp, but the points of a warp depart from two or more levels
// (a departure point lies within a layer of its arrival level, a grid node,
// so its cell is the one above or below almost at random).  A global gather
// then touches several lines per request: 2.2 data-pipe wavefronts for 32
// scalars, and that pipe bounds the direct kernels.  Here a block of
// 32 x TJ x TK arrival points copies the box of source cells its points
// depart from into shared memory once (cp.async) and gathers there.  Row and
// plane pitches are multiples of the 32 banks, so lanes with different x fall
// in different banks whatever row or plane each of them reads: one wavefront
// per request.
//
// The sums are those of the direct kernels (adz_kernels.cuh), in the same
// order, so results are the same bit for bit.  A point whose stencil leaves
// the box (larger spreads inside one tile occur where the flow is sheared
// over a few cells) is done by the direct code, which also reports stencils
// outside the array.
#pragma once
// included by adz_kernels.cuh after the per-point code

namespace adz {

// ---------------------------------------------------------------------------
// a tile of 32 x TJ x TK points, MINB resident blocks, and room for a box of
// BY rows by BZ planes of RP cells in x (RP a multiple of 32 four-byte or 16
// eight-byte elements).  DYN: the room is for any ny rows by nz planes with ny
// * nz <= BY * BZ, the plane pitch (ny rows) being known at run time only.  A
// sheared flow needs many rows and few planes, a scattered one near the ground
// many planes; points left out go to the direct code, which is slow here (the
// boxes leave it little L1).  At 512 x 512 x 60, gyres of 24 cells at Courant
// number 1.9, two updates: FP64 4.24 ms with the fixed split, 2.96 with any,
// direct 4.04; REF32 3.07, 2.21, 3.10; in smooth flows the same within 2 %.
// The pitch costs MIXED's kernels a register that they do not have (2 to 7 %
// in smooth flows, and two pitches known at compile time 4 to 6 %), so only
// its tolerance kernel, with 80 registers, takes it
template <int TJ_, int TK_, int MINB_, int RP_, int BY_, int BZ_, bool DYN_ = false>
struct StShape {
  static constexpr int TJ = TJ_, TK = TK_, MINB = MINB_, RP = RP_, BY = BY_, BZ = BZ_;
  static constexpr int NT = 32 * TJ * TK, ROWS = BY * BZ, BOX = RP * ROWS;
  static constexpr bool DYN = DYN_;
  static constexpr long long WAVE = 148LL * MINB * NT;  // points of the blocks that run at once
  static_assert(ROWS < 256, "StCopy::plan divides by multiplication");
};
// trajectory.  MIXED: three component boxes per block; two updates at 1024 x
// 1024 x 80 6.89 ms, direct 9.57 (4 x 4 points at 2 blocks 2 % slower, 4 x 2
// points 0.5 %, 3 x 4 points 10 %, 80 registers instead of 64 3 %).
// The iteration to a tolerance takes 3 blocks (80 registers): the first step
// of a run at 768 x 640 x 80 8.77 ms, 9.07 at 4 blocks, 9.65 with the direct kernel
// (boxes of 96 rows leave less L1: 4 to 13 % slower).
// FP64: one box of interleaved (u, v, w) cells; 1024 x 512 x 80 6.01 ms,
// direct 8.43 (2 x 4 points at 2 blocks 6.20); REF32, the same box of FP32
// cells at 4 blocks (80 registers), 5.81, direct 6.25
template <int PREC>
struct TrajBox;
template <>
struct TrajBox<kMixed> : StShape<2, 4, 4, 64, 7, 10> {};
template <>
struct TrajBox<kFp64> : StShape<3, 2, 3, 48, 8, 8, true> {};
template <>
struct TrajBox<kRef32> : StShape<3, 2, 4, 64, 7, 10, true> {};
struct TolBox : StShape<2, 4, 3, 64, 7, 10, true> {};
// the shape of a trajectory kernel and of its launch
template <int PREC, bool TOL>
using TrajShape = typename std::conditional<TOL, TolBox, TrajBox<PREC>>::type;
template <int PREC>
struct SetBox;
// 8 fields of set t at 1024 x 1024 x 80: 7.93 ms, direct 11.19 (rows that are
// no multiple of 16 bytes, 1021: 10.9 and 13.4); 4 x 4 points 8.21, 4 x 2
// points 8.59
template <>
struct SetBox<kMixed> : StShape<2, 4, 4, 64, 7, 10> {};
// FP64, 8 fields at 1024 x 512 x 80: 7.38 ms, direct 9.08 (7 rows by 11 planes).
// 8 clipped fields in the sheared flow above: 5.61 ms with 7 by 11, 4.02 with 8
// by 10, direct 5.11; in a smooth one 3.25, 3.29, 3.61 (8 by 11 spills: 3.47)
template <>
struct SetBox<kFp64> : StShape<2, 4, 2, 48, 8, 10> {};
constexpr int kStRing = 3;  // boxes in flight of the sets kernel
// A launch whose blocks all run at once takes as long as one block, and the
// staged block's chain is longer, so small launches stay direct (C::WAVE points
// are one wave).  Staged against direct speed, smooth flow / gyres at Courant
// number 1.9, at 48 x 40 x 20, 64 x 64 x 24 (98 K points), 30 x 200 x 24 (144 K), 96 x 90 x
// 40 (346 K):
//   two updates, MIXED  1.09 / 0.68, 1.15 / 0.83, 1.08 / 0.92, 1.34 / 1.08: one wave
//                       (152 K)
//   FP64, DYN           1.11 / 1.19, 1.11 / 1.08, 1.24 / 1.23, 1.30 / 1.33; REF32 1.00 /
//                       1.11, 1.14 / 1.23, 0.96 / 1.11, 1.10 / 1.17: half a wave (43 K, 57 K)
//   six from the arrival points, which place their box twice, MIXED 0.57, 1.10,
//                       0.68, 1.15 (smooth), FP64 0.76, 0.91, 1.07, 1.18: 1.5 waves (227 K,
//                       128 K).  REF32 0.65, 0.79, 0.72, 0.93, at 512 x 512 x 60 0.95: direct
//   sets, MIXED         3 fields 0.90 / 0.73, 1.06 / 0.85, 0.98 / 0.91, 1.24 / 1.06; 8 fields
//                       1.01 / 0.79, 1.29 / 0.94, 1.00 / 0.95, 1.44 / 1.22: one wave, half
//                       a wave where the rows are copied in 16-byte pieces (all but 30 x
//                       200), and four waves of points times fields
//   BICUBH_QV           3 fields 0.95 / 0.85, 1.27 / 0.94, 1.03 / 0.94, 1.34 / 1.16: half a
//                       wave (57 K)
// The iteration to a tolerance is staged at every size: from the arrival points
// 0.97 to 1.20 at those sizes, from a converged start 1.35 to 1.57

// fields from which a part of a sets launch is staged: placing and filling
// the boxes costs about what two fields gain (MIXED at 1024 x 1024 x 80, 2
// fields: 3.44 ms staged, 3.36 direct; 5 fields 5.64 and 7.19), in FP64 with bounds
// three (1024 x 512 x 80, 3 fields 4.13 and 3.89 ms, 4 4.79 and 4.91; 3 fields
// without bounds 3.77 and 3.69, at 250 x 60 x 70 110 and 138 us).  The sets of REF32
// stay direct (8 fields: 6.88 staged, 6.37 direct).  Rows that are no
// multiple of 16 bytes gain less (MIXED, 1021 x 512 x 80: 3 fields 2.41 ms staged,
// 2.63 direct, 5 3.68 and 4.18; BICUBH_QV at 637 x 512 x 80, 2 fields 1.57 and 1.95),
// and so does a single update of the trajectory (640 x 512 x 80: MIXED 1.29 times
// as fast as direct, two updates 1.36; FP64 1.17, 1.40; REF32 1.04, 1.09)
constexpr int kStQvMinFields = 2;
template <int PREC>
bool st_fields_ok(const FieldPtrs& fp) {
  return fp.nf >= (PREC == kFp64 && fp.mono_mask ? 4 : 3);
}

// a staged box: first cell in the extended array, extents in cells
struct StBox {
  int ox, oy, oz, nx, ny, nz;
  int pp;  // plane pitch
};

// the cell of a position: stencil corner column and row (0-based in the
// extended array), the level pair iz0, iz0+1 and whether z is linear there
struct StCell {
  int ci, cj, iz0;
  bool zl;
  __device__ __forceinline__ int zmin() const { return zl ? iz0 : iz0 - 1; }
  __device__ __forceinline__ int zmax() const { return zl ? iz0 + 1 : iz0 + 2; }
};

__device__ __forceinline__ StCell st_cell(const DGrid& g, const DZtab& lv, double px, double py, double pz) {
  int ix, iy, iz;
  cell_of(px, ix);
  cell_of(py, iy);
  cell_of(pz, iz);
  iz = imin_(imax_(iz, 1), lv.nk - 1);
  StCell c;
  c.ci = (int)((unsigned)ix + (unsigned)(lv.offi - 1 - g.lminx));  // a cell at the end of the range of int wraps
  c.cj = (int)((unsigned)iy + (unsigned)(lv.offj - 1 - g.lminy));
  c.iz0 = iz - 1;
  c.zl = c.iz0 < 1 || c.iz0 > lv.nk - 3;
  return c;
}
// the 4 x 4 columns lie in the extended array (planes always do; nit and njt
// are 5 or more).  Unsigned: c.ci + 3 would wrap for the last three ints, the
// cells of REF32's stored positions (not clipped) beyond the range of int
__device__ __forceinline__ bool st_inside(const DGrid& g, const StCell& c) {
  return (unsigned)c.ci < (unsigned)(g.nit - 3) && (unsigned)c.cj < (unsigned)(g.njt - 3);
}
// the stencil lies in the box
template <class Cell>
__device__ __forceinline__ bool st_in_box(const StBox& b, const Cell& c) {
  return c.ci >= b.ox && c.ci + 4 <= b.ox + b.nx && c.cj >= b.oy && c.cj + 4 <= b.oy + b.ny && c.zmin() >= b.oz &&
         c.zmax() < b.oz + b.nz;
}

// least and greatest stencil corner over the block's stencils (use: the
// thread has one): minima of (ci, cj, zmin, -ci, -cj, -zmax) into red[0..5]
// (INT_MAX before; a barrier must follow)
template <class Cell>
__device__ __forceinline__ void st_reduce(int* red, bool use, const Cell& c) {
  const int big = 0x7fffffff;
  const int m0 = __reduce_min_sync(0xffffffffu, use ? c.ci : big), m1 = __reduce_min_sync(0xffffffffu, use ? c.cj : big);
  const int m2 = __reduce_min_sync(0xffffffffu, use ? c.zmin() : big);
  const int m3 = __reduce_min_sync(0xffffffffu, use ? -c.ci : big);
  const int m4 = __reduce_min_sync(0xffffffffu, use ? -c.cj : big);
  const int m5 = __reduce_min_sync(0xffffffffu, use ? -c.zmax() : big);
  const int lane = threadIdx.x & 31;
  const int lo = lane == 0 ? m0 : lane == 1 ? m1 : m2, hi = lane == 3 ? m3 : lane == 4 ? m4 : m5;
  if (lane < 6) atomicMin(red + lane, lane < 3 ? lo : hi);
}

// the box that holds every reduced stencil, or the middle of their range
// where that is larger than a box of shape C; al: x origin a multiple of al
// cells; empty when there is no stencil.  MARGIN: with a cell around them
template <class C, bool MARGIN>
__device__ __forceinline__ StBox st_box(const DGrid& g, const int* red, int al) {
  StBox b{0, 0, 0, 0, 0, 0, 0};
  int x0 = red[0], y0 = red[1], z0 = red[2];
  if (x0 == 0x7fffffff) return b;
  int x1 = 4 - red[3], y1 = 4 - red[4], z1 = 1 - red[5];
  if (MARGIN) {
    x0 = imax_(x0 - 1, 0);
    y0 = imax_(y0 - 1, 0);
    z0 = imax_(z0 - 1, 0);
    x1 = imin_(x1 + 1, g.nit);
    y1 = imin_(y1 + 1, g.njt);
    z1 = imin_(z1 + 1, g.nk);
  }
  b.ox = (x1 - (x0 & ~(al - 1)) > C::RP ? imax_(x0, (x0 + x1 - C::RP) / 2) : x0) & ~(al - 1);
  b.nx = imin_(x1 - b.ox, C::RP);
  if constexpr (!C::DYN) {
    b.oy = y1 - y0 > C::BY ? (y0 + y1 - C::BY) / 2 : y0;
    b.ny = imin_(y1 - b.oy, C::BY);
    b.oz = z1 - z0 > C::BZ ? (z0 + z1 - C::BZ) / 2 : z0;
    b.nz = imin_(z1 - b.oz, C::BZ);
    b.pp = C::BY * C::RP;
    return b;
  }
  b.ny = y1 - y0;
  b.nz = z1 - z0;
  if (b.ny * b.nz > C::ROWS) {  // BY rows, or those that the planes leave
    b.ny = imin_(b.ny, imax_(C::BY, C::ROWS / b.nz));
    b.nz = imin_(b.nz, C::ROWS / b.ny);
  }
  b.oy = (y0 + y1 - b.ny) / 2;
  b.oz = (z0 + z1 - b.nz) / 2;
  b.pp = b.ny * C::RP;
  return b;
}

// the reduced stencils span more than a box of shape C (uniform over the block)
template <class C>
__device__ __forceinline__ bool st_overflow(const int* red, int al) {
  const int nx = 4 - red[3] - (red[0] & ~(al - 1)), ny = 4 - red[4] - red[1], nz = 1 - red[5] - red[2];
  return red[0] != 0x7fffffff && (nx > C::RP || (C::DYN ? ny * nz > C::ROWS : ny > C::BY || nz > C::BZ));
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The copies of a thread: its places in a box, the same for every array of
// one layout.  With rows of the extended array and the box's origin on
// 16-byte boundaries (vec) LPR lanes copy a row in 16-byte chunks, else a warp
// copies it element by element.  A row's last chunk may run past the box into
// the row, never past the row's end (vec implies rows of whole chunks).
template <typename T, class C>
struct StCopy {
  static constexpr int CH = 16 / sizeof(T);
  static constexpr int LPR = C::RP / CH <= 16 ? 16 : 32;   // lanes of a row (vec)
  static constexpr int VR = C::NT / LPR, ER = C::NT / 32;  // rows of a pass
  static constexpr int SLOTS = (C::ROWS + VR - 1) / VR;
  static_assert(C::RP % CH == 0 && C::RP / CH <= 32, "box shape");
  int off[SLOTS], dst[SLOTS];  // vec: source and shared offsets, dst < 0 for none
  float inv;                   // 1 / rows of a plane
  __device__ __forceinline__ void plan(const StBox& b, const DGrid& g, bool vec) {
    inv = __fdividef(1.0f, (float)imax_(b.ny, 1));
    if (!vec) return;
    const int c = (int)(threadIdx.x % LPR) * CH, r0 = threadIdx.x / LPR, rows = c < b.nx ? b.ny * b.nz : 0;
#pragma unroll
    for (int t = 0; t < SLOTS; t++) {
      const int r = r0 + t * VR;
      // r < 256 and ny < 128: the half keeps the product clear of the next integer
      const int z = (int)(((float)r + 0.5f) * inv), y = r - z * b.ny;
      off[t] = z * (int)g.nij + y * g.nit + c;
      dst[t] = r < rows ? z * b.pp + y * C::RP + c : -1;
    }
  }
  __device__ __forceinline__ void copy(T* sm, const T* __restrict__ a, const StBox& b, const DGrid& g,
                                       bool vec) const {
    const T* base = a + ((long long)(b.ox + b.oy * g.nit) + b.oz * g.nij);
    if (vec) {
#pragma unroll
      for (int t = 0; t < SLOTS; t++)
        if (dst[t] >= 0) cp_async<16>(sm + dst[t], base + off[t]);
    } else {
      const int lane = threadIdx.x & 31, rows = b.ny * b.nz;
#pragma unroll 1
      for (int r = threadIdx.x >> 5; r < rows; r += ER) {
        const int z = (int)(((float)r + 0.5f) * inv), y = r - z * b.ny;
        const T* s = base + (z * (int)g.nij + y * g.nit + lane);
        T* d = sm + z * b.pp + y * C::RP + lane;
#pragma unroll
        for (int x = 0; x < C::RP; x += 32)
          if (lane + x < b.nx) cp_async<(int)sizeof(T)>(d + x, s + x);
      }
    }
  }
};

// one box of cells of three interleaved values, a row per warp at a time
template <typename T, class C>
__device__ __forceinline__ void st_fill3(T* sm, const T* __restrict__ a, const StBox& b, const DGrid& g, bool vec) {
  constexpr int CH = 16 / sizeof(T);
  const T* base = a + 3 * ((long long)(b.ox + b.oy * g.nit) + b.oz * g.nij);
  const int lane = threadIdx.x & 31, rows = b.ny * b.nz, ne = 3 * b.nx;
  const float inv = __fdividef(1.0f, (float)imax_(b.ny, 1));
#pragma unroll 1
  for (int r = threadIdx.x >> 5; r < rows; r += C::NT / 32) {
    const int z = (int)(((float)r + 0.5f) * inv), y = r - z * b.ny;
    const T* s = base + 3 * (z * g.nij + y * g.nit);
    T* d = sm + 3 * (z * b.pp + y * C::RP);
    if (vec) {
#pragma unroll
      for (int c = 0; c < 3 * C::RP; c += 32 * CH)
        if (c + lane * CH < ne) cp_async<16>(d + c + lane * CH, s + c + lane * CH);
    } else {
      for (int c = lane; c < ne; c += 32) cp_async<(int)sizeof(T)>(d + c, s + c);
    }
  }
}

// ---------------------------------------------------------------------------
// sums over a staged box; s: the stencil corner on plane iz0, pp, d0 and d3
// the offsets of the next plane, the lower outer and the upper outer one from s
// (those of the inner planes where z is linear)
template <int RP>
__device__ __forceinline__ float st_interp1_mixed(const float* s, int pp, int d0, int d3, const float* cx,
                                                  const float* cy, const float* cz) {
  const float* p0 = s + d0;
  const float* p1 = s;
  const float* p2 = s + pp;
  const float* p3 = s + d3;
  const float2 cz0 = f2(cz[0], cz[0]), cz1 = f2(cz[1], cz[1]);
  const float2 cz2 = f2(cz[2], cz[2]), cz3 = f2(cz[3], cz[3]);
  float2 ya = f2(0.f, 0.f), yb = f2(0.f, 0.f);
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int o = r * RP;
    float2 za = __fmul2_rn(f2(p0[o], p0[o + 1]), cz0);
    float2 zb = __fmul2_rn(f2(p0[o + 2], p0[o + 3]), cz0);
    za = __ffma2_rn(f2(p1[o], p1[o + 1]), cz1, za);
    zb = __ffma2_rn(f2(p1[o + 2], p1[o + 3]), cz1, zb);
    za = __ffma2_rn(f2(p2[o], p2[o + 1]), cz2, za);
    zb = __ffma2_rn(f2(p2[o + 2], p2[o + 3]), cz2, zb);
    za = __ffma2_rn(f2(p3[o], p3[o + 1]), cz3, za);
    zb = __ffma2_rn(f2(p3[o + 2], p3[o + 3]), cz3, zb);
    const float2 cyr = f2(cy[r], cy[r]);
    ya = __ffma2_rn(za, cyr, ya);
    yb = __ffma2_rn(zb, cyr, yb);
  }
  float2 x = __fmul2_rn(ya, f2(cx[0], cx[1]));
  x = __ffma2_rn(yb, f2(cx[2], cx[3]), x);
  return x.x + x.y;
}

template <int RP>
__device__ __forceinline__ void st_mono_mixed(const float* s, int pp, int d0, int d3, float fx, float fy, float dz,
                                              const float* cx, const float* cy, const float* cz, float& d, float& lin,
                                              float& mn, float& mx) {
  const float* p0 = s + d0;
  const float* p1 = s;
  const float* p2 = s + pp;
  const float* p3 = s + d3;
  const float2 cz0 = f2(cz[0], cz[0]), cz1 = f2(cz[1], cz[1]);
  const float2 cz2 = f2(cz[2], cz[2]), cz3 = f2(cz[3], cz[3]);
  const float2 lz0 = f2(1.0f - dz, 1.0f - dz), lz1 = f2(dz, dz);
  float2 ya = f2(0.f, 0.f), yb = f2(0.f, 0.f), yl = f2(0.f, 0.f);
  float lo = 3.402823466e38f, hi = -3.402823466e38f;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int o = r * RP;
    const float2 a1 = f2(p1[o], p1[o + 1]), b1 = f2(p1[o + 2], p1[o + 3]);
    const float2 a2 = f2(p2[o], p2[o + 1]), b2 = f2(p2[o + 2], p2[o + 3]);
    float2 za = __fmul2_rn(f2(p0[o], p0[o + 1]), cz0);
    float2 zb = __fmul2_rn(f2(p0[o + 2], p0[o + 3]), cz0);
    za = __ffma2_rn(a1, cz1, za);
    zb = __ffma2_rn(b1, cz1, zb);
    za = __ffma2_rn(a2, cz2, za);
    zb = __ffma2_rn(b2, cz2, zb);
    za = __ffma2_rn(f2(p3[o], p3[o + 1]), cz3, za);
    zb = __ffma2_rn(f2(p3[o + 2], p3[o + 3]), cz3, zb);
    const float2 cyr = f2(cy[r], cy[r]);
    ya = __ffma2_rn(za, cyr, ya);
    yb = __ffma2_rn(zb, cyr, yb);
    lo = fminf(lo, fminf(fminf(a1.y, b1.x), fminf(a2.y, b2.x)));
    hi = fmaxf(hi, fmaxf(fmaxf(a1.y, b1.x), fmaxf(a2.y, b2.x)));
    if (r == 1 || r == 2) {
      const float2 zl = __ffma2_rn(f2(a2.y, b2.x), lz1, __fmul2_rn(f2(a1.y, b1.x), lz0));
      const float cyl = (r == 1) ? 1.0f - fy : fy;
      yl = __ffma2_rn(zl, f2(cyl, cyl), yl);
    }
  }
  float2 x = __fmul2_rn(ya, f2(cx[0], cx[1]));
  x = __ffma2_rn(yb, f2(cx[2], cx[3]), x);
  d = x.x + x.y;
  lin = fmaf(yl.y, fx, yl.x * (1.0f - fx));
  mn = lo;
  mx = hi;
}

// interp1_exact
template <typename T, int RP>
__device__ __forceinline__ double st_interp_exact(const T* s, int pp, int d0, int d3, const double* c) {
  const T* p0 = s + d0;
  const T* p1 = s;
  const T* p2 = s + pp;
  const T* p3 = s + d3;
  double ya[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const int o = r * RP + x;
      double za = (double)p0[o] * c[8];
      za = fma((double)p1[o], c[9], za);
      za = fma((double)p2[o], c[10], za);
      za = fma((double)p3[o], c[11], za);
      ya[x] = (r == 0) ? za * c[4] : fma(za, c[4 + r], ya[x]);
    }
  }
  return (ya[0] * c[0] + ya[2] * c[2]) + (ya[1] * c[1] + ya[3] * c[3]);
}

// one component of interp3_exact, from cells of three interleaved values
template <typename T, int RP>
__device__ __forceinline__ double st_interp3_exact(const T* s, int pp, int d0, int d3, const double* c) {
  const T* p0 = s + 3 * d0;
  const T* p1 = s;
  const T* p2 = s + 3 * pp;
  const T* p3 = s + 3 * d3;
  double ya[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const int o = 3 * (r * RP + x);
      double za = (double)p0[o] * c[8];
      za = fma((double)p1[o], c[9], za);
      za = fma((double)p2[o], c[10], za);
      za = fma((double)p3[o], c[11], za);
      ya[x] = (r == 0) ? za * c[4] : fma(za, c[4 + r], ya[x]);
    }
  }
  double x0 = ya[0] * c[0];
  x0 = fma(ya[1], c[1], x0);
  x0 = fma(ya[2], c[2], x0);
  return fma(ya[3], c[3], x0);
}

// interp_mono_exact with the 4-row box
template <typename T, int RP>
__device__ __forceinline__ void st_mono_exact(const T* s, int pp, int d0, int d3, const double* c, double& d,
                                              double& lin, T& mn, T& mx) {
  const T* p0 = s + d0;
  const T* p1 = s;
  const T* p2 = s + pp;
  const T* p3 = s + d3;
  double ya[4], vyl[4];
  T mi[4], ma[4];  // the bounds of values of type T
#pragma unroll
  for (int r = 0; r < 4; r++) {
#pragma unroll
    for (int x = 0; x < 4; x++) {
      const int o = r * RP + x;
      const T t1 = p1[o], t2 = p2[o];
      const double v0 = (double)p0[o], v1 = (double)t1, v2 = (double)t2, v3 = (double)p3[o];
      double za = v0 * c[8];
      if (r == 0) {
        mi[x] = t1;
        ma[x] = t1;
      } else {
        mi[x] = vmin(mi[x], t1);
        ma[x] = vmax(ma[x], t1);
      }
      za = fma(v1, c[9], za);
      mi[x] = vmin(mi[x], t2);
      ma[x] = vmax(ma[x], t2);
      za = fma(v2, c[10], za);
      za = fma(v3, c[11], za);
      ya[x] = (r == 0) ? za * c[4] : fma(za, c[4 + r], ya[x]);
      if (r == 1 || r == 2) {
        double vzl = v1 * c[18];
        vzl = fma(v2, c[19], vzl);
        vyl[x] = (r == 1) ? vzl * c[16] : fma(vzl, c[17], vyl[x]);
      }
    }
  }
  mn = vmin(mi[1], mi[2]);
  mx = vmax(ma[1], ma[2]);
  const double l0 = vyl[0] * c[12], l1 = vyl[1] * c[13], l2 = vyl[2] * c[14], l3 = vyl[3] * c[15];
  lin = (l0 + l2) + (l1 + l3);
  d = (ya[0] * c[0] + ya[2] * c[2]) + (ya[1] * c[1] + ya[3] * c[3]);
}

// FP32 weights of coef_mixed from the offsets inside the cell
__device__ __forceinline__ void st_weights(const DZtab& lv, int iz0, bool zl, float fx, float fy, float dz, float* cx,
                                           float* cy, float* cz) {
  cubic_w(fx, cx);
  cubic_w(fy, cy);
  if (zl) {
    cz[0] = 0.0f;
    cz[1] = 1.0f - dz;
    cz[2] = dz;
    cz[3] = 0.0f;
  } else {
    const float4 a = __ldg(reinterpret_cast<const float4*>(lv.zn + 8 * iz0));
    const float2 b = __ldg(reinterpret_cast<const float2*>(lv.zn + 8 * iz0 + 4));
    const float t = dz;
    const float d0 = t - a.x, d1 = t, d2 = t - 1.0f, d3 = t - a.y;
    cz[0] = d1 * d2 * d3 * a.z;
    cz[1] = d0 * d2 * d3 * a.w;
    cz[2] = d0 * d1 * d3 * b.x;
    cz[3] = d0 * d1 * d2 * b.y;
  }
}

// ---------------------------------------------------------------------------
// trajectory
struct TrajState {
  double ua, va, wa, px, py, pz, xm, ym, w3, wd;
};
// one update by the direct gather, for a point whose stencil is not staged
template <int PREC>
__device__ __noinline__ int traj_update_direct(const DGrid* g, const TrajArgs* a, int i, int j, int k, TrajState* s) {
  return traj_update<PREC, false>(*g, *a, i, j, k, s->ua, s->va, s->wa, s->px, s->py, s->pz, s->xm, s->ym, s->w3,
                                    s->wd);
}

// departure winds at (px, py, pz) from the staged boxes
template <int PREC, class C>
__device__ __forceinline__ void st_winds(const DGrid& g, const typename Types<PREC>::F* sm, const StBox& b,
                                         const StCell& c, double px, double py, double pz, double& ud, double& vd,
                                         double& wd) {
  using F = typename Types<PREC>::F;
  constexpr int RP = C::RP;
  const int pp = C::DYN ? b.pp : C::BY * RP;
  const int d0 = c.zl ? 0 : -pp, d3 = c.zl ? pp : 2 * pp;
  const int o = (c.iz0 - b.oz) * pp + (c.cj - b.oy) * RP + (c.ci - b.ox);
  if constexpr (PREC == kMixed) {
    const int ix = c.ci - g.tab_m.offi + 1 + g.lminx, iy = c.cj - g.tab_m.offj + 1 + g.lminy;
    const float fx = (float)(px - ix), fy = (float)(py - iy), dz = (float)(pz - (c.iz0 + 1));
    float cx[4], cy[4], cz[4];
    st_weights(g.tab_m, c.iz0, c.zl, fx, fy, dz, cx, cy, cz);
    const float* s = sm + o;
    ud = st_interp1_mixed<RP>(s, pp, d0, d3, cx, cy, cz);
    vd = st_interp1_mixed<RP>(s + C::BOX, pp, d0, d3, cx, cy, cz);
    wd = st_interp1_mixed<RP>(s + 2 * C::BOX, pp, d0, d3, cx, cy, cz);
  } else {
    double cf[20];
    int off;
    if constexpr (PREC == kRef32) coef_f32pos(cf, off, (float)px, (float)py, (float)pz, g.tab_m);
    else coef_f64pos(cf, off, px, py, pz, g.tab_m);
    const F* s = sm + 3 * o;
    // Tricublin_zyx3_n returns ``real`` (F)
    ud = (double)(F)st_interp3_exact<F, RP>(s, pp, d0, d3, cf);
    vd = (double)(F)st_interp3_exact<F, RP>(s + 1, pp, d0, d3, cf);
    wd = (double)(F)st_interp3_exact<F, RP>(s + 2, pp, d0, d3, cf);
  }
}

// All updates of a block of 32 i x TJ j x TK k points of a box of the tile
// (columns i0.., rows j0.., levels from a.k00).  The departure cells of the
// first update place the box, and later updates stay in it.  A cold start's
// points move by their whole displacement, so there the box is placed again
// when more than 1/16 of the block's points left it.
// TOL: the iteration to a tolerance (traject_point_tol), MIXED; its start is
// smooth and the first update scatters the levels, so its box has a margin
// (a margin of levels only: 8.98 against 8.76 ms).
// Else a.niter updates.
template <int PREC, bool TOL>
__global__ void __launch_bounds__(TrajShape<PREC, TOL>::NT, TrajShape<PREC, TOL>::MINB)
    k_traject_st(const __grid_constant__ DGrid g, const __grid_constant__ TrajArgs a, int i0, int nx, int j0, int ny,
                 double tol, int maxit, unsigned char* iters, unsigned long long* stats,
                 const __grid_constant__ GuessStart gs) {
  using F = typename Types<PREC>::F;
  using C = TrajShape<PREC, TOL>;
  constexpr int TK = C::TK, TJ = C::TJ, AL = 16 / sizeof(F);
  extern __shared__ uint4 st_dyn[];
  F* sm = reinterpret_cast<F*>(st_dyn);
  __shared__ int red[6];
  // the box in shared memory leaves more registers to the sums (FP64: nothing
  // spills, else 16 bytes); MIXED keeps it in registers (96 bytes instead of 32)
  constexpr bool RB = PREC == kMixed;
  __shared__ StBox sbox;
  StBox rbox;
  StBox& box = RB ? rbox : sbox;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = i0 + (int)blockIdx.x * 32 + lane;
  const int k = a.k00 + (int)blockIdx.y * TK + w % TK;
  const int j = j0 + (int)blockIdx.z * TJ + w / TK;
  const bool vec = g.nit % AL == 0 && ((unsigned long long)a.uvw_d & 15) == 0;
  const bool active = i < i0 + nx && k <= g.nk && j < j0 + ny;
  if (threadIdx.x < 6) red[threadIdx.x] = 0x7fffffff;
  TrajState s;
  s.xm = s.ym = s.w3 = s.wd = 0.0;
  s.px = s.py = s.pz = s.ua = s.va = s.wa = 0.0;
  if (active) {
    if (a.cold) {
      s.px = (double)(i + g.i0g - 1);
      s.py = (double)(j + g.j0g - 1);
      s.pz = (double)k;
    } else if (TOL && gs.d) {
      guess_start(g, a, gs, i, j, k, s.px, s.py, s.pz);
    } else {
      warm_start<PREC>(g, a, i, j, k, s.px, s.py, s.pz);
    }
  }
  auto place = [&](bool use, const StCell& c) {  // place the box and start its copies
    st_reduce(red, use, c);
    __syncthreads();
    StBox b = st_box<C, TOL>(g, red, vec ? AL : 1);
    // FP64, REF32: where more than a quarter of the points would be left out
    // (strong shear inside the tile), the direct code takes them all (83 x 192 x
    // 59 at Courant numbers up to 2: 0.217 against 0.25 ms).  In the MIXED
    // kernel the test costs more in spills (7.8 against 6.9 ms) than it saves
    if constexpr (PREC != kMixed)
      if (st_overflow<C>(red, vec ? AL : 1) && __syncthreads_count(use && !st_in_box(b, c)) > C::NT / 4) {
        b.nx = 0;
        if (RB || threadIdx.x == 0) box = b;
        return;
      }
    if (RB || threadIdx.x == 0) box = b;  // seen after the barrier that ends the copies
    const F* uvw = (const F*)a.uvw_d;
    if constexpr (PREC == kMixed) {
      StCopy<F, C> cp;
      cp.plan(b, g, vec);
#pragma unroll
      for (int q = 0; q < 3; q++) cp.copy(sm + q * C::BOX, uvw + q * g.nij * g.nk, b, g, vec);
    } else {
      st_fill3<F, C>(sm, uvw, b, g, vec);
    }
    cp_async_commit();
  };
  StCell c = st_cell(g, g.tab_m, s.px, s.py, s.pz);
  bool ok = active && st_inside(g, c);
  __syncthreads();
  place(ok, c);
  if (active) arrival_winds<PREC>(g, a, j, k, ext_index(g, i, j, k), s.ua, s.va, s.wa);
  cp_async_wait<0>();
  __syncthreads();

  int st = 0, used = 0, left = TOL ? maxit : a.niter;
  bool conv = false, second = a.cold != 0;  // second: the plain iteration of a guess that did not converge
  bool run = active && left > 0;
  for (;;) {
    if (run) {
      const double qx = s.px, qy = s.py, qz = s.pz;
      if (ok && st_in_box(box, c)) {
        double ud, vd;
        st_winds<PREC, C>(g, sm, box, c, s.px, s.py, s.pz, ud, vd, s.wd);
        st = traj_advance<PREC>(g, a, i, j, k, s.ua, s.va, s.wa, ud, vd, s.wd, s.px, s.py, s.pz, s.xm, s.ym, s.w3);
      } else {
        TrajState t = s;
        st = traj_update_direct<PREC>(&g, &a, i, j, k, &t);
        s = t;
      }
      left--;
      if (st) {
        run = false;
      } else {
        used++;
        if (TOL && fabs(s.px - qx) <= tol && fabs(s.py - qy) <= tol && fabs(s.pz - qz) <= tol) {
          conv = true;
          run = false;
        } else if (left == 0) {
          run = TOL && !second;
          if (run) {  // fallback: plain iteration from the arrival point
            second = true;
            left = maxit;
            s.px = (double)(i + g.i0g - 1);
            s.py = (double)(j + g.j0g - 1);
            s.pz = (double)k;
          }
        }
      }
    }
    if (a.cold) {
      if (!__syncthreads_or(run)) break;
    } else if (!__any_sync(0xffffffffu, run)) {
      break;
    }
    c = st_cell(g, g.tab_m, s.px, s.py, s.pz);
    ok = run && st_inside(g, c);
    if (a.cold && __syncthreads_count(ok && !st_in_box(box, c)) > C::NT / 16) {
      if (threadIdx.x < 6) red[threadIdx.x] = 0x7fffffff;
      __syncthreads();
      place(ok, c);
      cp_async_wait<0>();
      __syncthreads();
    }
  }
  if (TOL && active && iters)
    iters[arr_index(g, i, j, k)] = (unsigned char)(imin_(used, 127) + ((second && !a.cold) ? 128 : 0));
  if (active && st) raise_status(g.status, st);
  if (active && !st && used > 0) traj_store<PREC>(g, a, i, j, k, s.xm, s.ym, s.w3, s.px, s.py, s.pz, s.wd);
  if (TOL && stats) {
    const unsigned cnt[3] = {(unsigned)used, (unsigned)(active && second && !a.cold), (unsigned)(active && !conv)};
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const unsigned v = __reduce_add_sync(0xffffffffu, cnt[q]);
      if (lane == 0 && v) atomicAdd(stats + q, (unsigned long long)v);
    }
  }
}

// ---------------------------------------------------------------------------
// position sets
template <int PREC>  // 32-bit offsets: in 64 bits the FP64 kernel spills and is 4 % slower
__device__ __noinline__ void set_point_direct(const DGrid* g, int set, const SetArgs* a, const FieldPtrs* fp, int i,
                                              int j, int k) {
  set_point<PREC, false, false, int>(*g, set, *a, *fp, i, j, k);
}

// the fields of the position sets' parts on tiles of 32 i x TJ j x TK k
// points, consecutive blocks taking consecutive parts (u, v, t ...).  A block's
// fields go one after another through a ring of boxes: the copies of the next
// two run while one is summed.
template <int PREC>
__global__ void __launch_bounds__(SetBox<PREC>::NT, SetBox<PREC>::MINB)
    k_sets_st(const __grid_constant__ DGrid g, const __grid_constant__ SetArgs a, const __grid_constant__ SetParts sp) {
  using F = typename Types<PREC>::F;
  using C = SetBox<PREC>;
  constexpr int TK = C::TK, TJ = C::TJ, RP = C::RP, BOX = C::BOX;
  extern __shared__ uint4 st_dyn[];
  F* ring = reinterpret_cast<F*>(st_dyn);
  __shared__ int red[6];
  const unsigned part = blockIdx.x % (unsigned)sp.n;
  const SetPart& P = sp.p[part];
  const FieldPtrs& fp = P.fp;
  const DZtab& lv = (P.set == 3) ? g.tab_t : g.tab_m;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int fi = (int)(blockIdx.x / (unsigned)sp.n) * 32, fk = (int)blockIdx.y * TK, fj = (int)blockIdx.z * TJ;
  if (fi >= P.nx || fk >= P.nz || fj >= P.ny) return;
  const int i = P.i0 + fi + lane, k = P.k0 + fk + w % TK, j = P.j0 + fj + w / TK;
  const bool active = fi + lane < P.nx && fk + w % TK < P.nz && fj + w / TK < P.ny;
  constexpr int AL = 16 / sizeof(F);
  const bool vec = P.vec != 0;
  if (threadIdx.x < 6) red[threadIdx.x] = 0x7fffffff;
  __syncthreads();
  StCell c{};
  bool in = false;
  double px = 0.0, py = 0.0, pz = 0.0;
  if (active) {
    set_position<PREC, false>(g, a, P.set, i, j, k, px, py, pz);
    c = st_cell(g, lv, px, py, pz);
    in = st_inside(g, c);
  }
  st_reduce(red, in, c);
  __syncthreads();
  const StBox box = st_box<C, false>(g, red, vec ? AL : 1);
  StCopy<F, C> cp;
  cp.plan(box, g, vec);
  // copies of field q into its slot; always one group, so that group q is
  // field q's
  auto copy = [&](int q, int slot) {
    if (q < fp.nf) cp.copy(ring + slot * BOX, (const F*)fp.src[q], box, g, vec);
    cp_async_commit();
  };
#pragma unroll
  for (int q = 0; q < kStRing - 1; q++) copy(q, q);
  in = in && st_in_box(box, c);
  const int pp = C::DYN ? box.pp : C::BY * RP;
  const int o = (c.iz0 - box.oz) * pp + (c.cj - box.oy) * RP + (c.ci - box.ox);
  const int d0 = c.zl ? 0 : -pp, d3 = c.zl ? pp : 2 * pp;
  typename std::conditional<PREC == kMixed, float, double>::type cf[20];
  float fx = 0.f, fy = 0.f, dz = 0.f;
  if (in) {
    if constexpr (PREC == kMixed) {
      fx = (float)(px - (c.ci - lv.offi + 1 + g.lminx));
      fy = (float)(py - (c.cj - lv.offj + 1 + g.lminy));
      dz = (float)(pz - (c.iz0 + 1));
      st_weights(lv, c.iz0, c.zl, fx, fy, dz, cf, cf + 4, cf + 8);
    } else {
      int off;
      coef_f64pos(cf, off, px, py, pz, lv);
    }
  }
  const int e = (int)ext_index(g, i, j, k);
  int use = 0, next = kStRing - 1;
#pragma unroll 1
  for (int q = 0; q < fp.nf; q++) {
    cp_async_wait<kStRing - 2>();
    __syncthreads();  // field q has arrived, and everyone is done with the slot of the next copy
    copy(q + kStRing - 1, next);
    next = next == kStRing - 1 ? 0 : next + 1;
    const F* s = ring + use * BOX + o;
    use = use == kStRing - 1 ? 0 : use + 1;
    if (!in) continue;
    if constexpr (PREC == kMixed) {
      if ((fp.mono_mask >> q) & 1u) {
        float d, lin, mn, mx;
        st_mono_mixed<RP>(s, pp, d0, d3, fx, fy, dz, cf, cf + 4, cf + 8, d, lin, mn, mx);
        if ((fp.clip_mask >> q) & 1u) d = fmaxf(mn, fminf(mx, d));
        if (fp.lin[q]) ((float*)fp.lin[q])[e] = fmaxf(mn, fminf(mx, lin));
        if (fp.mn[q]) ((float*)fp.mn[q])[e] = mn;
        if (fp.mx[q]) ((float*)fp.mx[q])[e] = mx;
        ((float*)fp.dst[q])[e] = d;
      } else {
        ((float*)fp.dst[q])[e] = st_interp1_mixed<RP>(s, pp, d0, d3, cf, cf + 4, cf + 8);
      }
    } else {
      if ((fp.mono_mask >> q) & 1u) {
        double d, lin;
        F mnf, mxf;
        st_mono_exact<F, RP>(s, pp, d0, d3, cf, d, lin, mnf, mxf);
        F df = (F)d, lf = (F)lin;
        if ((fp.clip_mask >> q) & 1u) df = (mnf > ((mxf < df) ? mxf : df)) ? mnf : ((mxf < df) ? mxf : df);
        if (fp.lin[q]) ((F*)fp.lin[q])[e] = (mnf > ((mxf < lf) ? mxf : lf)) ? mnf : ((mxf < lf) ? mxf : lf);
        if (fp.mn[q]) ((F*)fp.mn[q])[e] = mnf;
        if (fp.mx[q]) ((F*)fp.mx[q])[e] = mxf;
        ((F*)fp.dst[q])[e] = df;
      } else {
        ((F*)fp.dst[q])[e] = (F)st_interp_exact<F, RP>(s, pp, d0, d3, cf);
      }
    }
  }
  if (active && !in) set_point_direct<PREC>(&g, P.set, &a, &fp, i, j, k);
}

// ---------------------------------------------------------------------------
// BICUBH_QV, MIXED
// 8 fields with bounds at 640 x 600 x 80: 4.29 ms, direct 6.04 (637: 5.28 and
// 6.48); 2 fields 1.75 and 1.97, 1 field 1.40 and 1.39
struct QvBox : StShape<2, 4, 3, 64, 7, 12> {};
struct QvCell {
  int ci, cj, k0, k1;
  __device__ __forceinline__ int zmin() const { return k0; }
  __device__ __forceinline__ int zmax() const { return k1; }
};

// interp_qv_mixed over a staged box: s the stencil's corner, p1..p5 the
// offsets of the planes of the vertical terms
template <int RP>
__device__ __forceinline__ void st_qv_mixed(const float* s, int p1, int p2, int p3, int p4, int p5, const QvCoefF& w,
                                            float& xyz, float& li, float& mi, float& ma) {
  const float *s1 = s + p1, *s2 = s + p2, *s3 = s + p3, *s4 = s + p4, *s5 = s + p5;
  float dst[4], dsl[2] = {0.f, 0.f};
  float hi = s2[1 + RP], lo = hi;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float v[4], b2 = 0.f, b3 = 0.f, c2 = 0.f, c3 = 0.f;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int o = i + r * RP;
      const float t2 = s2[o], t3 = s3[o];
      float a = s[o] * w.qz[0];
      a = fmaf(s1[o], w.qz[1], a);
      a = fmaf(t2, w.qz[2], a);
      a = fmaf(t3, w.qz[3], a);
      a = fmaf(s4[o], w.qz[4], a);
      v[r] = fmaf(s5[o], w.qz[5], a);
      if (r == 1) {
        b2 = t2;
        b3 = t3;
      } else if (r == 2) {
        c2 = t2;
        c3 = t3;
      }
    }
    dst[i] = fmaf(v[3], w.cy[3], fmaf(v[2], w.cy[2], fmaf(v[1], w.cy[1], v[0] * w.cy[0])));
    if (i == 1 || i == 2) {
      dsl[i - 1] = fmaf(fmaf(c3, w.lz[1], c2 * w.lz[0]), w.ly[1], fmaf(b3, w.lz[1], b2 * w.lz[0]) * w.ly[0]);
      hi = fmaxf(fmaxf(hi, b2), fmaxf(b3, fmaxf(c2, c3)));
      lo = fminf(fminf(lo, b2), fminf(b3, fminf(c2, c3)));
    }
  }
  xyz = fmaf(dst[3], w.cx[3], fmaf(dst[2], w.cx[2], fmaf(dst[1], w.cx[1], dst[0] * w.cx[0])));
  li = fmaf(dsl[1], w.lx[1], dsl[0] * w.lx[0]);
  mi = lo;
  ma = hi;
}

template <int PREC>
__device__ __noinline__ void qv_point_direct(const DGrid* g, const SetArgs* a, const FieldPtrs* fp, int i, int j,
                                             int k) {
  qv_point<PREC, false>(*g, *a, *fp, i, j, k);
}

// the fields at the t-set positions of a region, as k_sets_st: 96 values per
// point and field instead of 64
template <int PREC>
__global__ void __launch_bounds__(QvBox::NT, QvBox::MINB)
    k_qv_st(const __grid_constant__ DGrid g, const __grid_constant__ SetArgs a, const __grid_constant__ FieldPtrs fp,
            int i0, int nx, int j0, int ny, int k0, int nz, int vec) {
  static_assert(PREC == kMixed, "FP32 sums");
  using C = QvBox;
  constexpr int TK = C::TK, TJ = C::TJ, RP = C::RP, BOX = C::BOX;
  extern __shared__ uint4 st_dyn[];
  float* ring = reinterpret_cast<float*>(st_dyn);
  __shared__ int red[6];
  const int w = threadIdx.x >> 5;
  const int i = i0 + (int)blockIdx.x * 32 + (int)(threadIdx.x & 31), k = k0 + (int)blockIdx.y * TK + w % TK;
  const int j = j0 + (int)blockIdx.z * TJ + w / TK;
  const bool active = i < i0 + nx && k < k0 + nz && j < j0 + ny;
  if (threadIdx.x < 6) red[threadIdx.x] = 0x7fffffff;
  __syncthreads();
  QvCell cell{};
  QvCoefF f{};
  bool in = false;
  int nc = 0, nl = 0;
  if (active) {
    double px, py, pz;
    set_position<PREC, false>(g, a, 3, i, j, k, px, py, pz);
    QvCoef c;
    qv_coef<PREC>(g, px, py, pz, c);
    qv_to_float(c, f);
    nc = c.pl[1];
    nl = c.pl[2] - c.pl[1];
    cell.ci = (int)(float)px - g.i0g - g.lminx;
    cell.cj = (int)(float)py - g.j0g - g.lminy;
    cell.k0 = c.kb - 1;
    cell.k1 = cell.k0 + c.pl[5];
    in = cell.ci >= 0 && cell.ci + 3 < g.nit && cell.cj >= 0 && cell.cj + 3 < g.njt && cell.k0 >= 0 && cell.k1 < g.nk;
  }
  st_reduce(red, in, cell);
  __syncthreads();
  const StBox box = st_box<C, false>(g, red, vec ? 4 : 1);
  // more than a quarter of the points outside the box: the direct code for all
  if (st_overflow<C>(red, vec ? 4 : 1) && __syncthreads_count(in && !st_in_box(box, cell)) > C::NT / 4) {
    if (active) qv_point_direct<PREC>(&g, &a, &fp, i, j, k);
    return;
  }
  StCopy<float, C> cp;
  cp.plan(box, g, vec != 0);
  auto copy = [&](int q, int slot) {
    if (q < fp.nf) cp.copy(ring + slot * BOX, (const float*)fp.src[q], box, g, vec != 0);
    cp_async_commit();
  };
#pragma unroll
  for (int q = 0; q < kStRing - 1; q++) copy(q, q);
  in = in && st_in_box(box, cell);
  const int pp = C::DYN ? box.pp : C::BY * RP;
  const int o = (cell.k0 - box.oz) * pp + (cell.cj - box.oy) * RP + (cell.ci - box.ox);
  const int p1 = nc * pp, p2 = p1 + nl * pp, p3 = p2 + pp, p4 = p3 + nl * pp, p5 = p4 + nc * pp;
  const int e = (int)ext_index(g, i, j, k);
  int use = 0, next = kStRing - 1;
#pragma unroll 1
  for (int q = 0; q < fp.nf; q++) {
    cp_async_wait<kStRing - 2>();
    __syncthreads();  // field q has arrived, and everyone is done with the slot of the next copy
    copy(q + kStRing - 1, next);
    next = next == kStRing - 1 ? 0 : next + 1;
    const float* s = ring + use * BOX + o;
    use = use == kStRing - 1 ? 0 : use + 1;
    if (!in) continue;
    float d, lin, mn, mx;
    st_qv_mixed<RP>(s, p1, p2, p3, p4, p5, f, d, lin, mn, mx);
    if ((fp.clip_mask >> q) & 1u) d = fmaxf(mn, fminf(mx, d));
    if (fp.lin[q]) ((float*)fp.lin[q])[e] = fmaxf(mn, fminf(mx, lin));
    if (fp.mn[q]) ((float*)fp.mn[q])[e] = mn;
    if (fp.mx[q]) ((float*)fp.mx[q])[e] = mx;
    ((float*)fp.dst[q])[e] = d;
  }
  if (active && !in) qv_point_direct<PREC>(&g, &a, &fp, i, j, k);
}

// ---------------------------------------------------------------------------
// whether the staged kernel runs the trajectory of nx columns by ny rows: from
// the sizes above on, and its grid's y and z extents have to be below 65536
template <int PREC, bool TOL>
bool st_traject_ok(const DGrid& g, const TrajArgs& a, int nx, int ny) {
  using C = TrajShape<PREC, TOL>;
  const long long nk = g.nk - a.k00 + 1, n = (long long)nx * ny * nk;
  if ((nk + C::TK - 1) / C::TK > 65535 || (ny + C::TJ - 1) / C::TJ > 65535) return false;
  if (TOL) return true;
  if (a.cold) return PREC != kRef32 && 2 * n >= 3 * C::WAVE;
  return n >= (C::DYN ? C::WAVE / 2 : C::WAVE);
}
// whether the staged kernel runs a part of a sets launch: one of enough points
// and fields whose box is like the launch's largest extents nx, ny, nz (it fills
// at least half of them; not so the boxes of a band) and whose grid fits
template <int PREC>
bool st_part_ok(const DGrid& g, const SetPart& P, long long nx, long long ny, long long nz) {
  if constexpr (PREC == kRef32) return false;
  else {
    using C = SetBox<PREC>;
    const long long n = (long long)P.nx * P.ny * P.nz;
    const bool rows16 = g.nit % (16 / (int)sizeof(typename Types<PREC>::F)) == 0;
    return st_fields_ok<PREC>(P.fp) && (rows16 ? 2 * n : n) >= C::WAVE && n * P.fp.nf >= 4 * C::WAVE && 2 * n >= nx * ny * nz &&
           (nz + C::TK - 1) / C::TK <= 65535 && (ny + C::TJ - 1) / C::TJ <= 65535;
  }
}
inline void st_extents(const SetParts& sp, long long& nx, long long& ny, long long& nz) {
  nx = ny = nz = 0;
  for (int q = 0; q < sp.n; q++) {
    nx = sp.p[q].nx > nx ? sp.p[q].nx : nx;
    ny = sp.p[q].ny > ny ? sp.p[q].ny : ny;
    nz = sp.p[q].nz > nz ? sp.p[q].nz : nz;
  }
}
template <int PREC>
bool st_takes_some(const DGrid& g, const SetParts& sp) {
  long long nx, ny, nz;
  st_extents(sp, nx, ny, nz);
  for (int q = 0; q < sp.n; q++)
    if (st_part_ok<PREC>(g, sp.p[q], nx, ny, nz)) return true;
  return false;
}
// takes the parts of a sets launch that the staged kernel runs out of sp
template <int PREC>
SetParts st_take_parts(const DGrid& g, SetParts& sp) {
  SetParts st{}, rest{};
  long long nx, ny, nz;
  st_extents(sp, nx, ny, nz);
  for (int q = 0; q < sp.n; q++) {
    if (st_part_ok<PREC>(g, sp.p[q], nx, ny, nz)) st.p[st.n++] = sp.p[q];
    else rest.p[rest.n++] = sp.p[q];
  }
  sp = rest;
  return st;
}

template <int PREC, bool TOL>
cudaError_t st_launch_traject(const DGrid& g, const TrajArgs& a, int i0, int nx, int j0, int ny, double tol, int maxit,
                              unsigned char* iters, unsigned long long* stats, const GuessStart& gs, cudaStream_t s) {
  using C = TrajShape<PREC, TOL>;
  const int nkp = g.nk - a.k00 + 1;
  if (nx <= 0 || ny <= 0 || nkp <= 0) return cudaSuccess;
  constexpr int smem = 3 * C::BOX * (int)sizeof(typename Types<PREC>::F);
  const cudaError_t e =
      cudaFuncSetAttribute(k_traject_st<PREC, TOL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((nx + 31) / 32, (nkp + C::TK - 1) / C::TK, (ny + C::TJ - 1) / C::TJ);
  k_traject_st<PREC, TOL><<<grid, C::NT, smem, s>>>(g, a, i0, nx, j0, ny, tol, maxit, iters, stats, gs);
  return cudaGetLastError();
}

template <int PREC>
cudaError_t st_launch_sets(const DGrid& g, const SetArgs& a, const SetParts& parts, cudaStream_t s) {
  using C = SetBox<PREC>;
  using F = typename Types<PREC>::F;
  SetParts sp = parts;
  int nx = 0, ny = 0, nz = 0;
  for (int q = 0; q < sp.n; q++) {
    SetPart& P = sp.p[q];
    nx = P.nx > nx ? P.nx : nx;
    ny = P.ny > ny ? P.ny : ny;
    nz = P.nz > nz ? P.nz : nz;
    bool vec = g.nit % (16 / (int)sizeof(F)) == 0;
    for (int f = 0; f < P.fp.nf; f++) vec = vec && ((uintptr_t)P.fp.src[f] & 15) == 0;
    P.vec = vec;
  }
  if (nx <= 0 || ny <= 0 || nz <= 0) return cudaSuccess;
  constexpr int smem = kStRing * C::BOX * (int)sizeof(F);
  const cudaError_t e = cudaFuncSetAttribute(k_sets_st<PREC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((nx + 31) / 32 * sp.n, (nz + C::TK - 1) / C::TK, (ny + C::TJ - 1) / C::TJ);
  k_sets_st<PREC><<<grid, C::NT, smem, s>>>(g, a, sp);
  return cudaGetLastError();
}

// whether the staged kernel runs nf BICUBH_QV fields of nx x ny x nz points
inline bool st_qv_ok(int nf, int nx, int ny, int nz) {
  using C = QvBox;
  return nf >= kStQvMinFields && 2LL * nx * ny * nz >= C::WAVE && (nz + C::TK - 1) / C::TK <= 65535 &&
         (ny + C::TJ - 1) / C::TJ <= 65535;
}

template <int PREC>
cudaError_t st_launch_qv(const DGrid& g, int i0, int nx, int j0, int ny, int k0, int nz, const SetArgs& a,
                         const FieldPtrs& fp, cudaStream_t s) {
  using C = QvBox;
  bool vec = g.nit % 4 == 0;
  for (int f = 0; f < fp.nf; f++) vec = vec && ((uintptr_t)fp.src[f] & 15) == 0;
  constexpr int smem = kStRing * C::BOX * (int)sizeof(float);
  const cudaError_t e = cudaFuncSetAttribute(k_qv_st<PREC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((nx + 31) / 32, (nz + C::TK - 1) / C::TK, (ny + C::TJ - 1) / C::TJ);
  k_qv_st<PREC><<<grid, C::NT, smem, s>>>(g, a, fp, i0, nx, j0, ny, k0, nz, vec);
  return cudaGetLastError();
}

}  // namespace adz

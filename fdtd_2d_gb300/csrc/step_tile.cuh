// The register-tile kernel of single shots (step_tile.cu has its description): the
// device code that its instances are made of.
#pragma once

#include "internal.h"
#include "step_common.cuh"
#include "tile_common.cuh"
#include "tma_common.cuh"

namespace fdtd2d {

namespace {

constexpr int kHalo = kTileSteps;                 // columns and rows around the stored part
constexpr int kUse = kTileCols - 2 * kHalo;       // stored columns of a tile
constexpr int kWarps = 8;
constexpr int kREdge = 4;                         // rows per warp of a tile with CPML work
constexpr int kRowsEdge = kREdge * kWarps;
// Rows per warp of the plain tiles, by shape (Jz in shared memory).
constexpr int kShapes[] = {7, 5};
constexpr int kNumShapes = 2;

// Four elements (not by the read-only path, whose loads the compiler may
// move up across the wait above).
template <class T>
__device__ __forceinline__ void load4(float (&d)[4], const T* p, bool in) {
  if (!in) {
    zero4(d);
  } else if constexpr (sizeof(T) == 4) {
    get4(d, *reinterpret_cast<const float4*>(p));
  } else {
    Sto<T>::cvt(d, *reinterpret_cast<const uint2*>(p));
  }
}

// The part of the grid a tile answers for: rows [r0, r1), and of the thread's
// columns all (15) or none.  A plain tile's is what its halo leaves; the others
// read theirs again wherever they need it, for both kinds share the kernel's
// registers: kept in them, or read for plain tiles too, it took 8192^2 from 114
// to 123 and 132 us per step.
struct Part {
  int r0, r1;
  unsigned own;
};
template <bool PLAIN>
__device__ __forceinline__ Part tile_part(const int4& tile, const int4* at, int lane, bool in) {
  if (PLAIN) return {tile.z + kHalo, tile.w, lane >= kHalo / 4 && lane < 32 - kHalo / 4 && in ? 15u : 0u};
  int w;
  asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(w) : "l"(&at->w));
  return {tile.z + (w & 255), tile.z + (w >> 8 & 255), lane >= (w >> 16 & 255) && lane < w >> 24 && in ? 15u : 0u};
}

// How the sources and detectors of a tile are stepped: not at all (the tile holds
// none), tile_points, tile_few_points.
enum Points : int { kNoPoints, kManyPoints, kFewPoints };

template <int R, int NW, bool JS, bool LOSSLESS, bool PLAIN, int POINTS, bool AUX, class T>
__device__ __forceinline__ void tile_pass(const DevShot& S, const TileAux& A, const int4 tile, const int4* at, int n, int steps, float4* smem) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int rows = NW * R, threads = NW * 32;
  const int c0 = tile.y, r0 = tile.z;
  const int nx = S.nx, ny = S.ny;
  const int64_t pitch = S.pitch;
  const int row0 = warp * R, j0 = r0 + row0;
  const TilePos p = tile_pos(S, c0, r0, R, warp, lane);
  const Coef<T> C(S);
  float4* ex = smem;                                   // [2][NW][2][32]
  float4* kps = ex + 4 * NW * 32 + tid;                // [R][threads]
  float4* jzs = kps + R * threads;                     // [R][threads] where JS
  float4* rest = ex + 4 * NW * 32 + (JS ? 2 : 1) * R * threads;
  float* tc = reinterpret_cast<float*>(rest);          // the tables and psi of a tile with CPML work
  float* tr = tc + kTcRows * kTileCols;
  const TilePsi psi = tile_psi(rest + tile_table_f4(rows), p, rows, R, lane);

  // Everything the tile reads is asked for together: drive, Jz (JS) and psi by
  // copies into shared memory (FP32; 16-bit elements pass through registers to be
  // converted), the fields into registers.
  TileRegs<R, JS> s;
  constexpr bool kCopy = sizeof(T) == 4;
  const bool in = PLAIN || (p.i >= 0 && p.i < nx);
  const T* ez = field_ptr_t<T>(S, kEz, 0) + p.i;
  const T* hx = field_ptr_t<T>(S, kHx, 0) + p.i;
  const T* hy = field_ptr_t<T>(S, kHy, 0) + p.i;
  const T* jz = field_ptr_t<T>(S, kJz, 0) + p.i;
  const T* kp = reinterpret_cast<const T*>(S.kp);
  earlier_launches_done();
  if (!PLAIN) tile_psi_load<R, true>(S, S.psi, p, psi, rows, row0);
  float kv[kCopy ? 1 : R][4], jv[JS && !kCopy ? R : 1][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = j0 + r;
    const bool ok = in && (PLAIN || (j >= 0 && j < ny));
    const int64_t o = (int64_t)j * pitch;
    if (kCopy) {
      const bool has = ok && kp != nullptr;
      copy16(kps + r * threads, has ? (const void*)(kp + p.i + o) : (const void*)S.fb[0], has);
      if (JS) copy16(jzs + r * threads, ok ? (const void*)(jz + o) : (const void*)S.fb[0], ok);
    } else {
      load4(kv[kCopy ? 0 : r], kp + p.i + o, ok && kp != nullptr);
      if (JS) load4(jv[JS && !kCopy ? r : 0], jz + o, ok);
    }
  }
  load4(s.hx[0], hx + (int64_t)(j0 - 1) * pitch, in && (PLAIN || (j0 >= 1 && j0 <= ny)));
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = j0 + r;
    const bool ok = in && (PLAIN || (j >= 0 && j < ny));
    const int64_t o = (int64_t)j * pitch;
    load4(s.ez[r + 1], ez + o, ok);
    load4(s.hx[r + 1], hx + o, ok);
    load4(s.hy[r], hy + o, ok);
    if (!JS) load4(s.jz[JS ? 0 : r], jz + o, ok);
  }
  if (!PLAIN) tile_tables<T>(S, C, tc, tr, c0, r0, rows, tid, threads);
  if (!kCopy) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float (&v)[4] = kv[kCopy ? 0 : r];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = __fmul_rn(v[k], C.rk);
      kps[r * threads] = put4(v);
      if (JS) jzs[r * threads] = put4(jv[JS && !kCopy ? r : 0]);
    }
  }
  int p0 = 0, p1 = 0;
  if (POINTS && (POINTS == kFewPoints || (tile.x & kTilePoints)) && j0 + R > 0 && j0 < ny) {
    p0 = __ldg(S.row_start + max(j0, 0));
    p1 = __ldg(S.row_start + min(j0 + R, ny));
  }
  copies_done();   // (a thread reads only what it copied)
  const unsigned slots = AUX ? tile_tracked(A, p.i, tile_part<PLAIN>(tile, at, lane, p.i < nx).own) : 0u;
  // the loop in the form the warp needs (its barriers pair across the forms)
  auto loop = [&](auto x, auto y) {
    for (int t = 0; t < steps; ++t) {
      float4* e = ex + (t & 1) * 2 * NW * 32;
      e[(2 * warp) * 32 + lane] = put4(s.ez[1]);
      e[(2 * warp + 1) * 32 + lane] = put4(s.ez[R]);
      cta_sync();
      // the tile's first and last rows have no neighbour here: any value does
      get4(s.ez[0], e[(warp > 0 ? 2 * warp - 1 : 0) * 32 + lane]);
      get4(s.ez[R + 1], e[(warp < NW - 1 ? 2 * warp + 2 : 2 * warp + 1) * 32 + lane]);
      tile_step<R, JS, LOSSLESS, decltype(x)::value, decltype(y)::value, T>(s, S, C, p, psi, tc, tr, rows, row0, kps, jzs, threads, lane);
      if (AUX || (POINTS && p1 > p0)) {
        const Part u = tile_part<PLAIN>(tile, at, lane, p.i < nx);
        if (POINTS == kManyPoints && p1 > p0) tile_points<R, JS, T>(s, S, p, p0, p1, n + t, u.own, u.r0, u.r1, lane);
        if (POINTS == kFewPoints && p1 > p0) tile_few_points<R, JS, T>(s, S, p, p0, p1, n + t, u.own, u.r0, u.r1);
        if (AUX) tile_record<R, JS>(s, A, slots, p, u.own, u.r0, u.r1, n + t);
      }
      tile_round<R, JS, T>(s);
    }
  };
  if (PLAIN || !(p.x || p.y)) loop(No{}, No{});
  else if (!p.y) loop(Yes{}, No{});
  else if (!p.x) loop(No{}, Yes{});
  else loop(Yes{}, Yes{});
  const Part u = tile_part<PLAIN>(tile, at, lane, p.i < nx);
  if (u.own) {
    T* ez_w = field_ptr_t<T>(S, kEz, 1) + p.i;
    T* hx_w = field_ptr_t<T>(S, kHx, 1) + p.i;
    T* hy_w = field_ptr_t<T>(S, kHy, 1) + p.i;
    T* jz_w = field_ptr_t<T>(S, kJz, 1) + p.i;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = j0 + r;
      if (j < u.r0 || j >= u.r1) continue;
      const int64_t o = (int64_t)j * pitch;
      Sto<T>::stcs4(ez_w + o, s.ez[r + 1]);
      Sto<T>::stcs4(hx_w + o, s.hx[r + 1]);
      Sto<T>::stcs4(hy_w + o, s.hy[r]);
      if (JS) {
        float v[4];
        get4(v, jzs[r * threads]);
        Sto<T>::stcs4(jz_w + o, v);
      } else {
        Sto<T>::stcs4(jz_w + o, s.jz[JS ? 0 : r]);
      }
    }
  }
  if (!PLAIN) tile_psi_store<R, true>(S, S.psi + S.psi_buf, p, psi, rows, row0, u.own, u.r0, u.r1);
}

template <int RP>
struct Tile {
  static constexpr int kRows = RP;
};

// Plain tiles with points, in FP32 in a function of their own: their code in the
// kernel took registers of the loop of the plain tiles without any (8192^2 113 us per
// step, 114.4 with it, 126 with the points in the one loop; with 16-bit fields the call
// is the slower of the two, F16 103.3 against 103.6 and 104.5).
template <class Shape, bool LOSSLESS, bool AUX, class T>
__device__ __noinline__ void points_pass(const DevShot& S, const TileAux& A, const int4 tile, const int4* at, int n, int steps, float4* smem) {
  tile_pass<Shape::kRows, kWarps, true, LOSSLESS, true, kManyPoints, AUX, T>(S, A, tile, at, n, steps, smem);
}

// A tile in its form.
template <class Shape, bool LOSSLESS, bool AUX, bool FEW, class T>
__device__ __forceinline__ void any_tile(const DevShot& S, const TileAux& A, const int4 tile, const int4* at, int n, int steps, float4* smem) {
  if constexpr (FEW) {
    if (tile.x & kTilePlain) {
      tile_pass<Shape::kRows, kWarps, true, LOSSLESS, true, kFewPoints, AUX, T>(S, A, tile, at, n, steps, smem);
    } else {
      tile_pass<kREdge, kWarps, false, LOSSLESS, false, kFewPoints, AUX, T>(S, A, tile, at, n, steps, smem);
    }
  } else if (!(tile.x & kTilePlain)) {
    tile_pass<kREdge, kWarps, false, LOSSLESS, false, kManyPoints, AUX, T>(S, A, tile, at, n, steps, smem);
  } else if (!(tile.x & kTilePoints)) {
    tile_pass<Shape::kRows, kWarps, true, LOSSLESS, true, kNoPoints, AUX, T>(S, A, tile, at, n, steps, smem);
  } else if constexpr (sizeof(T) == 4) {
    points_pass<Shape, LOSSLESS, AUX, T>(S, A, tile, at, n, steps, smem);
  } else {
    tile_pass<Shape::kRows, kWarps, true, LOSSLESS, true, kManyPoints, AUX, T>(S, A, tile, at, n, steps, smem);
  }
}

// FEW: for shots with few points (tile_few), by tile_few_points.
template <class Shape, bool LOSSLESS, bool AUX, bool FEW, class T>
__global__ void __launch_bounds__(kWarps * 32, 2)
step_tmat_kernel(const __grid_constant__ DevShot S, const __grid_constant__ TileAux A, const int4* __restrict__ tiles, int n_global, int steps) {
  extern __shared__ float4 smem[];
  const int4 tile = __ldg(tiles + blockIdx.x);
  const int n = n_global - S.base_n;
  any_tile<Shape, LOSSLESS, AUX, FEW, T>(S, A, tile, tiles + blockIdx.x, n, steps, smem);
}

}  // namespace
}  // namespace fdtd2d

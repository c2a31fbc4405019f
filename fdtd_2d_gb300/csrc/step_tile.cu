// Several time steps per pass over the fields, a tile at a time in registers
// (uniform medium, the CPML included).
//
// step_tmat_kernel<Tile<R>, ...>: a CTA of 8 warps loads a tile of 128 columns
// x 8 R rows of state n, steps it up to kTileSteps = 4 times in registers
// (tile_common.cuh) and stores state n+4 of the part that no step has eaten
// into: a cell at distance d from the tile's edge is right for d steps, so 4
// columns and 4 rows on every side are read again by the neighbouring tiles.
// Tiles read one buffer and write the other, so nothing orders them but the
// launch: one launch per four steps, where the two-step path took four per
// two (interior, CPML bands twice, frame).
//
// Why this shape: 4 columns of halo are one lane, so every access stays a
// whole vector; the rows are what registers allow at 2 CTAs per SM (128 per
// thread: while one CTA loads or stores, the other computes), which with Jz in
// shared memory is 7 (FP32) or 5 to 7 (16-bit, whose rounding takes registers).  Tiles
// with CPML work keep 4 rows per warp and their psi in shared memory.
//
// Bytes: 20 x (halo) + 16 per stored cell and 4 steps, 10.1 B per cell-update
// with R = 7 (the two-step path 18).  Measured on GB300 against that path,
// Gcell/s: 8192^2 FP32 591 (315), F16 648 (413); 4096^2 536 (249) and 576
// (281); 2048^2 445 (165).  Bound by latency at 16 warps per SM: a 4096^2 pass
// issues in 43 % of the cycles, DRAM moves 4.4 TB/s (0.65 of the copy peak); the
// loads of a tile take a third of its time, overlapped with the SM's other CTA.
// us per step with 7 / 6 / 5 rows per warp: FP32 8192^2 114 / 119 / 127, 4096^2
// 31.4 / 32.6 / 33.2, 2048^2 9.8 / 9.6 / 9.4, 1024^2 4.5 / 4.4 / 4.0, F16 8192^2
// 104 / 125 / 112; 6 is best at few sizes (1400^2 4.9 against 5.0 with 5) and left
// out.  CTAs of CPML tiles with 5 or 6 rows need the shared memory of two (8192^2:
// 363 and 370 Gcell/s).
#include <algorithm>

#include "internal.h"
#include "tile_common.cuh"

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

// POINTS: there are sources or detectors in the tile.
template <int R, int NW, bool JS, bool LOSSLESS, bool PLAIN, bool POINTS, bool AUX, class T>
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
  if (POINTS && (tile.x & kTilePoints) && j0 + R > 0 && j0 < ny) {
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
        if (POINTS && p1 > p0) tile_points<R, JS, T>(s, S, p, p0, p1, n + t, u.own, u.r0, u.r1, lane);
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
// kernel took registers of the loop of the plain tiles without any (8192^2 112.8 us per
// step, 114.4 with it, 126 with the points in the one loop; with 16-bit fields the call
// is the slower of the two, F16 103.3 against 103.6 and 104.5).
template <class Shape, bool LOSSLESS, bool AUX, class T>
__device__ __noinline__ void points_pass(const DevShot& S, const TileAux& A, const int4 tile, const int4* at, int n, int steps, float4* smem) {
  tile_pass<Shape::kRows, kWarps, true, LOSSLESS, true, true, AUX, T>(S, A, tile, at, n, steps, smem);
}

// A tile in its form.
template <class Shape, bool LOSSLESS, bool AUX, class T>
__device__ __forceinline__ void any_tile(const DevShot& S, const TileAux& A, const int4 tile, const int4* at, int n, int steps, float4* smem) {
  if (!(tile.x & kTilePlain)) {
    tile_pass<kREdge, kWarps, false, LOSSLESS, false, true, AUX, T>(S, A, tile, at, n, steps, smem);
  } else if (!(tile.x & kTilePoints)) {
    tile_pass<Shape::kRows, kWarps, true, LOSSLESS, true, false, AUX, T>(S, A, tile, at, n, steps, smem);
  } else if constexpr (sizeof(T) == 4) {
    points_pass<Shape, LOSSLESS, AUX, T>(S, A, tile, at, n, steps, smem);
  } else {
    tile_pass<Shape::kRows, kWarps, true, LOSSLESS, true, true, AUX, T>(S, A, tile, at, n, steps, smem);
  }
}

template <class Shape, bool LOSSLESS, bool AUX, class T>
__global__ void __launch_bounds__(kWarps * 32, 2)
step_tmat_kernel(const __grid_constant__ DevShot S, const __grid_constant__ TileAux A, const int4* __restrict__ tiles, int n_global, int steps) {
  extern __shared__ float4 smem[];
  const int4 tile = __ldg(tiles + blockIdx.x);
  const int n = n_global - S.base_n;
  any_tile<Shape, LOSSLESS, AUX, T>(S, A, tile, tiles + blockIdx.x, n, steps, smem);
}

// The same for the shots of a batch: the tile's shot from a device array, its
// own step and the buffers its passes so far have left it in.
template <class Shape, bool LOSSLESS>
__global__ void __launch_bounds__(kWarps * 32, 2)
step_tma_batch_kernel(const DevShot* __restrict__ shots, const int4* __restrict__ tiles, int g, int steps, int pass) {
  extern __shared__ float4 smem[];
  __shared__ __align__(16) DevShot S;
  const int4 tile = __ldg(tiles + blockIdx.x);
  const int* src = reinterpret_cast<const int*>(shots + (tile.x >> kTileSlot));
  for (int t = threadIdx.x; t < (int)(sizeof(DevShot) / 4); t += kWarps * 32) reinterpret_cast<int*>(&S)[t] = __ldg(src + t);
  __syncthreads();
  if (threadIdx.x == 0 && ((pass - S.base_pass) & 1)) {
    float* f = S.fb[0];
    S.fb[0] = S.fb[1];
    S.fb[1] = f;
    S.psi += S.psi_buf;
    S.psi_buf = -S.psi_buf;
  }
  __syncthreads();
  const int n = g + 1 - S.base_n, k = min(steps, S.n_steps - n + 1);
  if (k <= 0) return;
  const TileAux none{};
  any_tile<Shape, LOSSLESS, false, float>(S, none, tile, tiles + blockIdx.x, n, k, smem);
}

// A launch that may start while the one before it in the stream ends; its tiles
// wait for the earlier launches before they read anything those write
// (earlier_launches_done).  Saves ~3 us of the ~5 us between two passes: 700^2
// 4.10 -> 3.46 us per step, 2048^2 11.25 -> 10.3.  (Loading the tables and the
// points' values before that wait gained nothing more and cost the plain tiles,
// compiled into the same kernel, 8 % at 8192^2.)
cudaError_t launch_early(const void* fn, int n_tiles, void** args, size_t smem, cudaStream_t stream) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(n_tiles);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, args);
}

bool lossless(const DevShot& s) { return s.ca == 1.f && s.da == 1.f; }

template <int RP, bool AUX, class T>
const void* tile_kernel(const DevShot& s) {
  return lossless(s) ? (const void*)step_tmat_kernel<Tile<RP>, true, AUX, T> : (const void*)step_tmat_kernel<Tile<RP>, false, AUX, T>;
}
template <int RP>
const void* tile_kernel(const DevShot& s, bool aux) {
  if (aux) return s.store == 0 ? tile_kernel<RP, true, float>(s) : nullptr;
  return s.store == 0 ? tile_kernel<RP, false, float>(s)
       : s.store == 1 ? tile_kernel<RP, false, __half>(s) : tile_kernel<RP, false, __nv_bfloat16>(s);
}
const void* tile_kernel(int shape, const DevShot& s, bool aux) {
  return shape == 0 ? tile_kernel<kShapes[0]>(s, aux) : tile_kernel<kShapes[1]>(s, aux);
}

}  // namespace

int tile_shape_count() { return kNumShapes; }
int tile_shape_rows(int shape) { return kShapes[shape]; }

namespace {

// A column of tiles: it answers for grid columns [a, b), a a multiple of 4, with
// tiles from column c0 on.  plain: no CPML, no border.
struct TileColumn {
  int c0, a, b;
  bool plain;
};

// Plain columns (whole: 120 grid columns each), as few as it takes, between a first and a last one on
// the borders, which need no halo there: up to 124 grid columns each.
std::vector<TileColumn> tile_columns(const DevShot& s) {
  const int nx = s.nx, clear = s.npml + kHalo, most = kTileCols - kHalo;
  std::vector<TileColumn> v;
  const int n = s.den_uniform ? std::max(0, (nx - 2 * most + kUse - 1) / kUse) : 0, both = nx - n * kUse;
  if (n < 1 || both < 2 * ((clear + 3) & ~3)) {
    for (int a = 0, b; a < nx; a = b) {
      const int c0 = std::max(a - kHalo, 0);
      b = c0 + kTileCols >= nx ? nx : c0 + most;
      v.push_back({c0, a, b, false});
    }
    return v;
  }
  int a = std::min(most, (both - clear) & ~3);
  v.push_back({0, 0, a, false});
  for (int q = 0; q < n; ++q, a += kUse) v.push_back({a - kHalo, a, a + kUse, true});
  v.push_back({a - kHalo, a, nx, false});
  return v;
}

}  // namespace

// Tiles over the grid: plain ones, whole, where no cell of the tile has CPML, the
// others (slower: first) over the rest.  Every cell below the last row belongs to
// one tile.  Tiles on a border have no halo there, so a CPML of 20 cells takes one
// column of them on each side and 2 to 4 rows, where tiles that began 4 cells
// outside took 2 or 3 columns and 4 or 5 rows.  us per step, before and now: 2048^2
// 10.35 and 9.43 (with 5 rows per warp 10.68 and 9.43), 4096^2 32.1 and 31.3, F16
// 31.9 and 29.1, 2300 x 1531 BF16 8.43 and 8.07, 8192^2 F16 110 and 104.
std::vector<int4> make_tiles(const DevShot& s, int shape, const std::vector<int3>& points) {
  const int ny = s.ny, P = s.npml, up = kShapes[shape] * kWarps - 2 * kHalo;
  std::vector<int4> edge, plain;
  // plain rows between `top` and `bottom` rows of others: as many as fit, the rest
  // split so that it takes the fewest tiles (a tile reads one row below its first)
  const int top0 = P + 1 + kHalo, bottom0 = P + kHalo - 1, n = (ny - 1 - top0 - bottom0) / up;
  int top = 0, least = 1 << 30;
  if (n >= 1) {
    const int rest = ny - 1 - n * up, ue = kRowsEdge - 2 * kHalo, on = kRowsEdge - kHalo;
    auto count = [&](int r, int first) { return r <= first ? 1 : 1 + (r - first + ue - 1) / ue; };
    for (int r = top0; r <= rest - bottom0; ++r)
      if (const int k = count(r, on) + count(rest - r, on - 1); k < least) {
        least = k;
        top = r;
      }
  }
  for (const TileColumn& c : tile_columns(s)) {
    const int lanes = (c.a - c.c0) / 4 << 16 | (c.b - c.c0 + 3) / 4 << 24;
    auto others = [&](int a, int stop) {
      while (a < stop) {
        const int r0 = std::max(a - kHalo, 0), b = std::min(stop, r0 + kRowsEdge >= ny ? ny - 1 : r0 + kRowsEdge - kHalo);
        edge.push_back(make_int4(0, c.c0, r0, (a - r0) | (b - r0) << 8 | lanes));
        a = b;
      }
    };
    if (!c.plain || n < 1) {
      others(0, ny - 1);
      continue;
    }
    others(0, top);
    others(top + n * up, ny - 1);
    for (int q = 0; q < n; ++q) plain.push_back(make_int4(kTilePlain, c.c0, top + q * up - kHalo, top + (q + 1) * up));
  }
  edge.insert(edge.end(), plain.begin(), plain.end());
  // the tiles that hold points, halo included
  for (int4& t : edge) {
    const int rows = t.x & kTilePlain ? kShapes[shape] * kWarps : kRowsEdge;
    auto q = std::lower_bound(points.begin(), points.end(), t.z, [](const int3& p, int row) { return p.y < row; });
    for (; q != points.end() && q->y < t.z + rows && !(t.x & kTilePoints); ++q)
      if (q->x >= t.y && q->x < t.y + kTileCols) t.x |= kTilePoints;
  }
  return edge;
}

size_t tile_smem(const DevShot& s, int shape) {
  int nxl = 0, yw = 0;
  for (const TileColumn& c : tile_columns(s))
    if (!c.plain) nxl = std::max(nxl, strip_lanes(s, c.c0));
  for (int r = 0; r < s.ny - 1; ++r) yw = std::max(yw, y_warps(s, r, kWarps, kREdge));
  const size_t ex = 4 * kWarps * 32;
  const size_t edge = ex + kREdge * kWarps * 32 + tile_table_f4(kRowsEdge) + tile_psi_x(kRowsEdge, nxl) +
                      (size_t)yw * (2 * kREdge + 1) * 32;
  const size_t plain = ex + 2 * (size_t)kShapes[shape] * kWarps * 32;
  return std::max(edge, plain) * 16;
}

namespace {

// The most shared memory a tile takes: tile_smem with every lane of the tile in an
// x strip and every warp in a y strip (a CPML of 120 cells comes to that).
constexpr size_t most_smem() {
  size_t most = 0;
  for (const int rows : kShapes) {
    const size_t plain = 4 * kWarps * 32 + 2 * (size_t)rows * kWarps * 32;
    most = most > plain ? most : plain;
  }
  const size_t edge = 4 * kWarps * 32 + kREdge * kWarps * 32 + kTcRows * (kTileCols + kRowsEdge + 4) / 4 +
                      2 * kRowsEdge * 32 + (size_t)kWarps * (2 * kREdge + 1) * 32;
  return (most > edge ? most : edge) * 16;
}

// The attribute belongs to the kernel, in every thread that launches it: always
// set to the same value, so that no thread takes away what another one's launch is
// about to ask for.
cudaError_t allow_smem(const void* fn) {
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most_smem());
}

}  // namespace

cudaError_t launch_step_tile(int shape, const DevShot& shot, const int4* tiles, int n_tiles, size_t smem, int n_global,
                             int steps, const TileAux* aux, cudaStream_t stream) {
  if (steps < 1 || steps > kTileSteps || n_tiles <= 0) return cudaErrorInvalidValue;
  const void* fn = tile_kernel(shape, shot, aux != nullptr);
  if (!fn) return cudaErrorInvalidValue;
  const cudaError_t e = allow_smem(fn);
  if (e != cudaSuccess) return e;
  DevShot s = shot;
  TileAux a = aux ? *aux : TileAux{};
  void* args[] = {&s, &a, (void*)&tiles, &n_global, &steps};
  return launch_early(fn, n_tiles, args, smem, stream);
}

cudaError_t launch_batch_tile(bool lossless, const DevShot* shots, const int4* tiles, int n_tiles, size_t smem,
                              int g, int steps, int pass, cudaStream_t stream) {
  if (steps < 1 || steps > kTileSteps) return cudaErrorInvalidValue;
  if (n_tiles <= 0) return cudaSuccess;
  const void* fn = lossless ? (const void*)step_tma_batch_kernel<Tile<kShapes[kBatchShape]>, true>
                            : (const void*)step_tma_batch_kernel<Tile<kShapes[kBatchShape]>, false>;
  const cudaError_t e = allow_smem(fn);
  if (e != cudaSuccess) return e;
  void* args[] = {&shots, &tiles, &g, &steps, &pass};
  return launch_early(fn, n_tiles, args, smem, stream);
}

}  // namespace fdtd2d

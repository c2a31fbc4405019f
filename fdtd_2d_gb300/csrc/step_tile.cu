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
#include <map>

#include "step_tile.cuh"

namespace fdtd2d {

namespace {

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
  any_tile<Shape, LOSSLESS, false, false, float>(S, none, tile, tiles + blockIdx.x, n, k, smem);
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
  return lossless(s) ? (const void*)step_tmat_kernel<Tile<RP>, true, AUX, false, T>
                     : (const void*)step_tmat_kernel<Tile<RP>, false, AUX, false, T>;
}
template <int RP>
const void* tile_kernel(const DevShot& s, bool aux) {
  if (aux) return s.store == 0 ? tile_kernel<RP, true, float>(s) : nullptr;
  return s.store == 0 ? tile_kernel<RP, false, float>(s)
       : s.store == 1 ? tile_kernel<RP, false, __half>(s) : tile_kernel<RP, false, __nv_bfloat16>(s);
}
const void* tile_kernel(int shape, bool few, const DevShot& s, bool aux) {
  if (few) return tile_kernel_few(shape, s.store, lossless(s), aux);
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

// FP32 shots with at most 4 points in any 8 rows of 128 columns (an array of sources
// and detectors every 5 rows along y): us per step with tile_few_points and tile_points,
// 1400^2 5.16 and 5.30, 2048^2 9.51 and 9.73, 8192^2 113.7 and 114.5; an array with an
// element in every row 2048^2 9.98 and 9.74.  F16 shots too from 4e7 cells on (3300^2
// 20.7 and 20.7, 5000^2 41.9 and 41.7, 8192^2 104.2 and 104.9), BF16 ones never (4096^2
// 31.5 and 30.9 at the better shape, 8192^2 110.1 and 109.9).
bool tile_few(const DevShot& s, const std::vector<int3>& points) {
  if (s.store == 2 || (s.store == 1 && (int64_t)s.nx * s.ny < 40000000)) return false;
  std::map<std::pair<int, int>, int> blocks;
  for (const int3& p : points)
    if (++blocks[{p.y / 8, p.x / kTileCols}] > 4) return false;
  return true;
}

cudaError_t launch_step_tile(int shape, bool few, const DevShot& shot, const int4* tiles, int n_tiles, size_t smem, int n_global,
                             int steps, const TileAux* aux, cudaStream_t stream) {
  if (steps < 1 || steps > kTileSteps || n_tiles <= 0) return cudaErrorInvalidValue;
  const void* fn = tile_kernel(shape, few, shot, aux != nullptr);
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

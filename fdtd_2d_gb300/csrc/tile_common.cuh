// A tile of the grid held in registers, stepped in place: the device code
// shared by the kernels that advance several time steps per pass
// (step_tile.cu).
//
// A tile is 128 columns (a warp's 32 lanes x 4) by kWarps x R rows, R rows
// per warp.  A thread keeps Ez, Hx, Hy and Jz of its 4 x R cells in
// registers; Ez(i+1) and Hy(i-1) come by shuffle, the rows above and below a
// warp's by shared memory (its first and last Ez rows, published once per
// step), and Hx of the row below is recomputed by every warp, so a step needs
// one CTA barrier.  The plasma drive sits in shared memory (a float4 per
// thread and row), and so do the CPML psi of the tiles that touch a strip.
//
// Arithmetic is in stored units (Ez/sE, H/sH, Jz/sJ; the scales are powers of
// two, folded into the coefficients, 1 for FP32 storage) with the one-row
// kernels' operations in their order; with 16-bit storage every array is
// rounded to its element at the end of the step, as a store and a load would.
// So a tile gives the bits of that many one-step launches.
#pragma once

#include "internal.h"
#include "step_common.cuh"
#include "tma_common.cuh"

namespace fdtd2d {
namespace {

constexpr unsigned kFull = 0xffffffffu;

struct Yes { static constexpr bool value = true; };
struct No { static constexpr bool value = false; };

// The CTA's barrier, from any point of the code: the warps of a tile run
// differently specialised loops that meet at it.
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

// Column and row tables of a tile that is not plain, in shared memory.
// Columns: b and c/d of the Hy and Ez recursions (the column's strip), and
// the denominators; rows likewise for Hx and Ez.
enum TabCol : int { kTcBh = 0, kTcCh, kTcBe, kTcCe, kTcDe, kTcDh, kTcRows };
constexpr int kTileCols = 128;

// Coefficients of a shot in stored units (Hx and Hy share one scale, as
// set_storage_scales gives them).
template <class T>
struct Coef {
  float da, db, ca, cb, ja, rj, rk;   // upd_h, upd_es, upd_j and the drive's factor
  float sE, sH, pdb, pcb;             // psi: scale of its differences, factor into H (db/sH) and Ez (cb/sE)
  __device__ __forceinline__ explicit Coef(const DevShot& S) {
    constexpr bool sc = sizeof(T) == 2;
    da = S.da;
    ca = S.ca;
    ja = S.ja;
    sE = sc ? S.sc[0] : 1.f;
    sH = sc ? S.sc[1] : 1.f;
    db = sc ? __fmul_rn(__fmul_rn(S.db, sE), S.isc[1]) : S.db;
    cb = sc ? __fmul_rn(__fmul_rn(S.cb, sH), S.isc[0]) : S.cb;
    rj = sc ? __fmul_rn(S.sc[3], S.isc[1]) : 1.f;
    rk = sc ? __fmul_rn(__fmul_rn(S.sc[4], sE), S.isc[3]) : 1.f;
    pdb = sc ? __fmul_rn(S.db, S.isc[1]) : S.db;
    pcb = sc ? __fmul_rn(S.cb, S.isc[0]) : S.cb;
  }
};

// LOSSLESS: CA = DA = 1, whose products are exact and are left out.
template <bool LOSSLESS>
__device__ __forceinline__ float tile_h(float da, float h, float db, float ea, float eb, float den) {
  return __fmaf_rn(db, __fmul_rn(__fsub_rn(ea, eb), den), LOSSLESS ? h : __fmul_rn(da, h));
}
template <bool LOSSLESS, class T>
__device__ __forceinline__ float tile_e(const Coef<T>& C, float e, float dhy, float dex, float dhx, float dey, float jz) {
  const float c = __fmaf_rn(dhy, dex, __fmul_rn(dhx, dey));
  const float curl = sizeof(T) == 2 ? __fmaf_rn(-C.rj, jz, c) : __fsub_rn(c, jz);
  return __fmaf_rn(C.cb, curl, LOSSLESS ? e : __fmul_rn(C.ca, e));
}

// A thread's cells: rows j0 .. j0+R-1, columns i .. i+3.  ez[0] and ez[R+1]
// are Ez of the rows below and above, hx[0] is Hx of the row below.  JS: Jz is
// kept in shared memory beside the drive (a float4 per row, `stride` apart)
// instead of in registers, which leaves room for more rows.
template <int R, bool JS>
struct TileRegs {
  float ez[R + 2][4], hx[R + 1][4], hy[R][4], jz[JS ? 1 : R][4];
};

// Where a thread and its warp sit in the grid, and what of the CPML they hold.
// x: the tile touches a border or a strip in x (the same for its whole CTA);
// y: the warp's rows, or the row below them, do in y.  Elsewhere the update
// needs no masks, no psi and no tables.
struct TilePos {
  int i, j0;          // first column and row
  bool x, y;
  // columns whose H (bits 0-3) and Ez (4-7) are updated, that lie in an x strip
  // for Hy (8-11) and for Ez (12-15)
  unsigned mask;
  int xslot, nxl;     // the thread's slot among the row's strip lanes, their number
  int yslot;          // the warp's slot among the CTA's y warps
  __device__ __forceinline__ bool mh(int k) const { return mask >> k & 1; }
  __device__ __forceinline__ bool me(int k) const { return mask >> (4 + k) & 1; }
  __device__ __forceinline__ bool xh(int k) const { return mask >> (8 + k) & 1; }
  __device__ __forceinline__ bool xe(int k) const { return mask >> (12 + k) & 1; }
  __device__ __forceinline__ bool strip() const { return mask >> 8; }
};

// psi of a tile in shared memory: x strips [Hy, Ez][rows][nxl]; y strips, per y
// warp, R + 1 rows of Hx (the row below first) and R of Ez, a float4 per lane.
struct TilePsi {
  float4 *x, *y;      // y: this thread's first
};

__device__ __forceinline__ void get4(float (&d)[4], const float4& v) { d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w; }
__device__ __forceinline__ float4 put4(const float (&d)[4]) { return make_float4(d[0], d[1], d[2], d[3]); }

// Strip rows of Hx: 0 .. P-2 and ny-P .. ny-2.
__host__ __device__ __forceinline__ bool y_strip_h(int j, int ny, int P) { return (j >= 0 && j <= P - 2) || (j >= ny - P && j <= ny - 2); }
// Strip rows of Ez: 1 .. P-1 and ny-P .. ny-2.
__host__ __device__ __forceinline__ bool y_strip_e(int j, int ny, int P) { return (j >= 1 && j <= P - 1) || (j >= ny - P && j <= ny - 2); }
// Whether rows j0-1 .. j0+R-1 need the y form, columns c0 .. c0+127 the x form.
__host__ __device__ __forceinline__ bool tile_y(const DevShot& s, int j0, int R) {
  return !s.den_uniform || j0 - 1 < s.npml || j0 + R - 1 >= s.ny - s.npml;
}
__host__ __device__ __forceinline__ bool tile_x(const DevShot& s, int c0) {
  return !s.den_uniform || c0 < s.npml || c0 + kTileCols - 1 >= s.nx - s.npml;
}

__device__ __forceinline__ TilePos tile_pos(const DevShot& S, int c0, int r0, int R, int warp, int lane) {
  TilePos p{};
  p.i = c0 + 4 * lane;
  p.j0 = r0 + warp * R;
  p.x = tile_x(S, c0);
  p.y = tile_y(S, p.j0, R);
  const int nx = S.nx, P = S.npml;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = p.i + k;
    if (c >= 0 && c <= nx - 2) p.mask |= 1u << k;
    if (c >= 1 && c <= nx - 2) p.mask |= 16u << k;
    if ((c >= 0 && c <= P - 2) || (c >= nx - P && c <= nx - 2)) p.mask |= 256u << k;
    if ((c >= 1 && c <= P - 1) || (c >= nx - P && c <= nx - 2)) p.mask |= 4096u << k;
  }
  const unsigned m = __ballot_sync(kFull, p.strip());
  p.xslot = p.strip() ? __popc(m & ((1u << lane) - 1)) : 0;
  p.nxl = __popc(m);
  for (int w = 0; w < warp; ++w) p.yslot += tile_y(S, r0 + w * R, R) ? 1 : 0;
  return p;
}

// float4s of a tile's tables and of its x psi
__host__ __device__ __forceinline__ int tile_table_f4(int rows) { return kTcRows * (kTileCols + rows + 4) / 4; }
__host__ __device__ __forceinline__ int tile_psi_x(int rows, int nxl) { return 2 * rows * nxl; }
__device__ __forceinline__ TilePsi tile_psi(float4* base, const TilePos& p, int rows, int R, int lane) {
  TilePsi s;
  s.x = base;
  s.y = base + tile_psi_x(rows, p.nxl) + p.yslot * (2 * R + 1) * 32 + lane;
  return s;
}

// The tables of a tile with borders or strips: tc[kTcRows][128] by column,
// tr[kTcRows][rows+1] by row (row r0-1 first); c/d in stored units.
template <class T>
__device__ __forceinline__ void tile_tables(const DevShot& S, const Coef<T>& C, float* tc, float* tr, int c0, int r0,
                                            int rows, int tid, int threads) {
  const int nx = S.nx, ny = S.ny, P = S.npml;
  for (int t = tid; t < kTileCols + rows + 1; t += threads) {
    const bool col = t < kTileCols;
    const int c = col ? c0 + t : r0 - 1 + (t - kTileCols);
    const int n = col ? nx : ny;
    float* out = col ? tc + t : tr + (t - kTileCols);
    const int st = col ? kTileCols : rows + 1;
    // every entry's six loads are issued together, from a clamped place where
    // there is none
    const int h0 = col ? kBhX1 : kBhY1, e0 = col ? kBeX1 : kBeY1;
    const bool lo_h = c >= 0 && c <= P - 2, hi_h = c >= n - P && c <= n - 2;
    const bool lo_e = c >= 1 && c <= P - 1, hi_e = hi_h, in = c >= 0 && c < n - 1;
    const int qh = lo_h ? h0 * P + c : hi_h ? (h0 + 2) * P + n - 2 - c : 0;
    const int qe = lo_e ? e0 * P + c : hi_e ? (e0 + 2) * P + n - 1 - c : 0;
    const int qd = in ? c : 0;
    float bh = __ldg(S.cpml + qh), ch = __ldg(S.cpml + qh + P), be = __ldg(S.cpml + qe), ce = __ldg(S.cpml + qe + P);
    float de = __ldg((col ? S.den_ex : S.den_ey) + qd), dh = __ldg((col ? S.den_hx : S.den_hy) + qd);
    if (!(lo_h || hi_h)) bh = ch = 0.f;
    if (!(lo_e || hi_e)) be = ce = 0.f;
    if (!in) de = dh = 0.f;
    out[kTcBh * st] = bh; out[kTcCh * st] = __fmul_rn(ch, C.sE); out[kTcBe * st] = be; out[kTcCe * st] = __fmul_rn(ce, C.sH);
    out[kTcDe * st] = de; out[kTcDh * st] = dh;
  }
}

// Copies of 4 and 16 bytes into shared memory, without a register or a wait
// (cp.async; the issuing thread waits for its own with copies_done()).  The
// 16-byte form gives zeros where `in` is false and reads nothing.
__device__ __forceinline__ void copy4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16(void* dst, const void* src, bool in) {
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// psi of the tile from the slab, every slot of the thread (copies in flight at
// return), and back: the columns of the mask `own` in rows [u0, u1).  ALIGNED:
// the thread's first column is a multiple of 4 (then `own` is all or none).
// (A load at a time in a loop, each waiting for the one before, made up half the
// time of a pass's CPML tiles.)
template <int R, bool ALIGNED>
__device__ __forceinline__ void tile_psi_load(const DevShot& S, const float* slab, const TilePos& p, const TilePsi& psi,
                                              int rows, int row0) {
  const int nx = S.nx, ny = S.ny, P = S.npml;
  const int64_t pitch = S.pitch;
  if (p.strip()) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = p.j0 + r;
      const bool row = j >= 0 && j <= ny - 1;
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        float* ps = reinterpret_cast<float*>(psi.x + (f * rows + row0 + r) * p.nxl + p.xslot);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int c = p.i + k;
          const int side = c >= P ? 1 : 0, q = side ? nx - (f ? 1 : 2) - c : c;
          if (row && (f ? p.xe(k) : p.xh(k))) copy4(ps + k, slab + (f ? S.o_ezx : S.o_hyx) + ((int64_t)side * ny + j) * P + q);
          else ps[k] = 0.f;
        }
      }
    }
  }
  if (p.y) {
#pragma unroll
    for (int r = -1; r < R; ++r) {
      const int j = p.j0 + r;
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        if (r < 0 && f) continue;
        const bool strip = f ? y_strip_e(j, ny, P) : y_strip_h(j, ny, P);
        const int side = j >= P ? 1 : 0, q = side ? ny - (f ? 1 : 2) - j : j;
        const float* g = slab + (strip ? (f ? S.o_ezy + ((int64_t)side * P + q) * pitch : ((int64_t)side * (P - 1) + q) * pitch) + p.i : 0);
        float4* ps = psi.y + (f ? R + 1 + r : r + 1) * 32;
        if (ALIGNED) {   // a thread left of column 0 holds no strip cell
          const bool in = strip && p.i >= 0 && p.i < nx;
          copy16(ps, in ? g : slab, in);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (strip && p.i + k >= 0 && p.i + k < nx) copy4(reinterpret_cast<float*>(ps) + k, g + k);
            else reinterpret_cast<float*>(ps)[k] = 0.f;
          }
        }
      }
    }
  }
}

template <int R, bool ALIGNED>
__device__ __forceinline__ void tile_psi_store(const DevShot& S, float* slab, const TilePos& p, const TilePsi& psi, int rows,
                                               int row0, unsigned own, int u0, int u1) {
  const int nx = S.nx, ny = S.ny, P = S.npml;
  const int64_t pitch = S.pitch;
  if (!own) return;
#pragma unroll 1
  for (int r = 0; r < R; ++r) {
    const int j = p.j0 + r;
    if (j < u0 || j >= u1) continue;
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      if (p.strip()) {
        float v[4];
        get4(v, psi.x[(f * rows + row0 + r) * p.nxl + p.xslot]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (!(f ? p.xe(k) : p.xh(k)) || !(own >> k & 1)) continue;
          const int c = p.i + k;
          const int side = c >= P ? 1 : 0, q = side ? nx - (f ? 1 : 2) - c : c;
          slab[(f ? S.o_ezx : S.o_hyx) + ((int64_t)side * ny + j) * P + q] = v[k];
        }
      }
      if (p.y && (f ? y_strip_e(j, ny, P) : y_strip_h(j, ny, P))) {
        const int side = j >= P ? 1 : 0, q = side ? ny - (f ? 1 : 2) - j : j;
        float* g = slab + (f ? S.o_ezy + ((int64_t)side * P + q) * pitch : ((int64_t)side * (P - 1) + q) * pitch) + p.i;
        const float4 v = psi.y[(f ? R + 1 + r : r + 1) * 32];
        if (ALIGNED) {
          if (p.i >= 0 && p.i < nx) *reinterpret_cast<float4*>(g) = v;
        } else {
          const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if ((own >> k & 1) && p.i + k >= 0 && p.i + k < nx) g[k] = w[k];
        }
      }
    }
  }
}

// The material-ID medium: tables by material in shared memory, and per thread
// and row one word for 4 cells in place of the drive: their ids in the Hx, Hy and
// Ez maps, and which of the reference's eight update launches reach them (bit
// 4 q + k: kernel q, column k).  Row R of the thread's words is the row below.
// (The one-step kernel reads 3 ids and compares 8 indexes per cell and step; here
// both are done once per launch, and a step costs one 16-byte read per 4 cells.)
struct MatTables {
  const float2* h = nullptr;   // da, db
  const float4* e = nullptr;   // ca, cb, drive, PEC
};
__device__ __forceinline__ uint4 mat_word(const float4* words, int r, int stride) {
  return *reinterpret_cast<const uint4*>(words + r * stride);
}
__device__ __forceinline__ bool mat_covered(const uint4& w, int kernel, int k) { return w.w >> (4 * kernel + k) & 1; }

// The word of columns i .. i+3 of row j (zeros outside the grid).
__device__ __forceinline__ uint4 mat_make(const DevShot& S, int i, int j) {
  uint4 w = make_uint4(0, 0, 0, 0);
  const int nx = S.nx, ny = S.ny, P = S.npml;
  if (j < 0 || j >= ny) return w;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = i + k;
    if (c < 0 || c >= nx) continue;
    const int64_t o = (int64_t)j * S.pitch + c;
    w.x |= (unsigned)__ldg(S.id1 + o) << 8 * k;
    w.y |= (unsigned)__ldg(S.id2 + o) << 8 * k;
    w.z |= (unsigned)__ldg(S.id3 + o) << 8 * k;
    // the reference's thread index of the cell in each launch
    const int ry = j >= P ? ny - 2 - j : j, rx = c >= P ? nx - 2 - c : c;
    const long long l[8] = {(long long)j * (nx - 1) + c, (long long)ry * (nx - 1) + c, (long long)j * (nx - 1) + c,
                            (long long)j * (P - 1) + rx, (long long)(j - 1) * (nx - 2) + (c - 1),
                            (long long)(j - 1) * (nx - 2) + (c - 1),
                            (long long)(j - 1) * (P - 1) + ((c >= P ? nx - 1 - c : c) - 1),
                            (long long)((j >= P ? ny - 1 - j : j) - 1) * (nx - 2) + (c - 1)};
#pragma unroll
    for (int q = 0; q < 8; ++q) w.w |= (l[q] < S.cov[q] ? 1u : 0u) << (4 * q + k);
  }
  return w;
}

// One time step of the thread's cells up to Ez, without sources, detectors
// and the rounding to the storage type; s.ez[0] and s.ez[R+1] hold the rows
// around the thread's.  X, Y: the tile's and the warp's forms (TilePos).  The
// body has no branches (a strip row or lane is a select, every psi slot of an
// X tile or Y warp is read and written) and stores to shared memory only
// after several rows' loads, which the compiler may not move across a store,
// so that the rows' chains overlap: with a branch per strip row a warp took
// ~1800 cycles a row, and the tiles in the corners of the grid set the step
// time of all.
// kp: the thread's drive, js its Jz where JS, `stride` float4 from row to row.
// MED: the material-ID medium (FP32): kp holds the cells' words.
template <int R, bool JS, bool LOSSLESS, bool X, bool Y, class T, bool MED = false>
__device__ __forceinline__ void tile_step(TileRegs<R, JS>& s, const DevShot& S, const Coef<T>& C, const TilePos& p,
                                          const TilePsi& psi, const float* tc, const float* tr, int rows, int row0,
                                          const float4* kp, float4* js, int stride, int lane, const MatTables& M = MatTables()) {
  static_assert(!MED || (!LOSSLESS && sizeof(T) == 4), "the material medium: FP32, coefficients by cell");
  const int ny = S.ny, P = S.npml;
  const int ts = rows + 1;             // row tables start at row r0 - 1
  const float* trw = tr + row0;        // this warp's: entry r is row j0 - 1 + r
  // ---- Hx: row j0 - 1 (the warp below owns it), then the thread's rows
  constexpr int kBatch = 2;   // rows whose psi is held before it is stored
  float pq[kBatch][4];
#pragma unroll
  for (int r = 0; r <= R; ++r) {
    const float den = Y ? trw[kTcDh * ts + r] : S.den_c[3];
    float (&pn)[4] = pq[r % kBatch];
    float b = 0.f, c = 0.f;
    bool strip = false;
    if (Y) {
      get4(pn, psi.y[r * 32]);
      b = trw[kTcBh * ts + r];
      c = trw[kTcCh * ts + r];
      strip = y_strip_h(p.j0 - 1 + r, ny, P);
    }
    if constexpr (MED) {
      const uint4 w = mat_word(kp, r == 0 ? R : r - 1, stride);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 m = M.h[w.x >> 8 * k & 255];
        const bool in = !X || p.mh(k);
        float v = tile_h<false>(m.x, s.hx[r][k], m.y, s.ez[r][k], s.ez[r + 1][k], den);
        v = in && mat_covered(w, kCovHx, k) ? v : s.hx[r][k];
        if (Y) {
          const bool add = strip && in && mat_covered(w, kCovHxPml, k);
          const float q = upd_psi(b, pn[k], c, s.ez[r][k], s.ez[r + 1][k]);
          v = add ? __fmaf_rn(m.y, q, v) : v;
          pn[k] = add ? q : pn[k];
        }
        s.hx[r][k] = v;
      }
    } else
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = !X || p.mh(k);
      float v = tile_h<LOSSLESS>(C.da, s.hx[r][k], C.db, s.ez[r][k], s.ez[r + 1][k], den);
      if (Y) {
        const float q = upd_psi(b, pn[k], c, s.ez[r][k], s.ez[r + 1][k]);
        const float w = __fmaf_rn(C.pdb, q, v);
        v = strip ? w : v;
        pn[k] = strip && in ? q : pn[k];
      }
      s.hx[r][k] = in ? v : s.hx[r][k];
    }
    if (Y && (r % kBatch == kBatch - 1 || r == R)) {
#pragma unroll
      for (int q = r - r % kBatch; q <= r; ++q) psi.y[q * 32] = put4(pq[q % kBatch]);
    }
  }
  // ---- Hy
  float dhx[4], b[4], c[4];
  if (X) {
    lds4f(dhx, tc + kTcDh * kTileCols + 4 * lane);
    lds4f(b, tc + kTcBh * kTileCols + 4 * lane);
    lds4f(c, tc + kTcCh * kTileCols + 4 * lane);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) dhx[k] = S.den_c[1];
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float e4 = __shfl_down_sync(kFull, s.ez[r + 1][0], 1);
    const float er[4] = {s.ez[r + 1][1], s.ez[r + 1][2], s.ez[r + 1][3], e4};
    float (&pn)[4] = pq[r % kBatch];
    if (X) get4(pn, psi.x[(row0 + r) * p.nxl + p.xslot]);
    if constexpr (MED) {
      const uint4 w = mat_word(kp, r, stride);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 m = M.h[w.y >> 8 * k & 255];
        float v = tile_h<false>(m.x, s.hy[r][k], m.y, er[k], s.ez[r + 1][k], dhx[k]);
        v = (!X || p.mh(k)) && mat_covered(w, kCovHy, k) ? v : s.hy[r][k];
        if (X) {
          const bool add = p.xh(k) && mat_covered(w, kCovHyPml, k);
          const float q = upd_psi(b[k], pn[k], c[k], er[k], s.ez[r + 1][k]);
          v = add ? __fmaf_rn(m.y, q, v) : v;
          pn[k] = add ? q : pn[k];
        }
        s.hy[r][k] = v;
      }
    } else
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float v = tile_h<LOSSLESS>(C.da, s.hy[r][k], C.db, er[k], s.ez[r + 1][k], dhx[k]);
      if (X) {
        const bool strip = p.xh(k);
        const float q = upd_psi(b[k], pn[k], c[k], er[k], s.ez[r + 1][k]);
        const float w = __fmaf_rn(C.pdb, q, v);
        v = strip ? w : v;
        pn[k] = strip ? q : pn[k];
      }
      s.hy[r][k] = !X || p.mh(k) ? v : s.hy[r][k];
    }
    if (X && p.strip() && (r % kBatch == kBatch - 1 || r == R - 1)) {
#pragma unroll
      for (int q = r - r % kBatch; q <= r; ++q) psi.x[(row0 + q) * p.nxl + p.xslot] = put4(pq[q % kBatch]);
    }
  }
  // ---- Jz and Ez
  float dex[4];
  if (X) {
    lds4f(dex, tc + kTcDe * kTileCols + 4 * lane);
    lds4f(b, tc + kTcBe * kTileCols + 4 * lane);
    lds4f(c, tc + kTcCe * kTileCols + 4 * lane);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) dex[k] = S.den_c[0];
  }
  float pxq[kBatch][4], pyq[kBatch][4], jq[kBatch][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float hl = __shfl_up_sync(kFull, s.hy[r][3], 1);
    const float hyl[4] = {hl, s.hy[r][0], s.hy[r][1], s.hy[r][2]};
    const int j = p.j0 + r;
    const bool row_in = !Y || (j >= 1 && j <= ny - 2);
    float (&px)[4] = pxq[r % kBatch], (&py)[4] = pyq[r % kBatch], (&jv)[4] = jq[r % kBatch];
    float kv[4];
    get4(kv, kp[r * stride]);
    if (JS) get4(jv, js[r * stride]);
    float (&jz)[4] = s.jz[JS ? 0 : r];
    const float dey = Y ? trw[kTcDe * ts + r + 1] : S.den_c[2];
    float yb = 0.f, yc = 0.f;
    bool ystrip = false;
    if (X) get4(px, psi.x[(rows + row0 + r) * p.nxl + p.xslot]);
    if (Y) {
      get4(py, psi.y[(R + 1 + r) * 32]);
      yb = trw[kTcBe * ts + r + 1];
      yc = trw[kTcCe * ts + r + 1];
      ystrip = y_strip_e(j, ny, P);
    }
    if constexpr (MED) {
      const uint4 w = mat_word(kp, r, stride);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 m = M.e[w.z >> 8 * k & 255];   // ca, cb, drive, PEC
        const bool in = row_in && (!X || p.me(k));
        const float jo = JS ? jv[k] : jz[k];
        const float jn = in && mat_covered(w, kCovJz, k) ? upd_j(C.ja, jo, m.z, s.ez[r + 1][k]) : jo;
        float v = upd_e(m.x, s.ez[r + 1][k], m.y, __fsub_rn(s.hy[r][k], hyl[k]), dex[k], __fsub_rn(s.hx[r][k], s.hx[r + 1][k]), dey, jn);
        v = m.w != 0.f ? 0.f : v;
        v = in && mat_covered(w, kCovEz, k) ? v : s.ez[r + 1][k];
        if (X) {
          const bool add = row_in && p.xe(k) && mat_covered(w, kCovEzPmlI, k);
          const float q = upd_psi(b[k], px[k], c[k], s.hy[r][k], hyl[k]);
          v = add ? __fmaf_rn(m.y, q, v) : v;
          px[k] = add ? q : px[k];
        }
        if (Y) {
          const bool add = ystrip && in && mat_covered(w, kCovEzPmlJ, k);
          const float q = upd_psi(yb, py[k], yc, s.hx[r][k], s.hx[r + 1][k]);
          v = add ? __fmaf_rn(m.y, q, v) : v;
          py[k] = add ? q : py[k];
        }
        if (JS) jv[k] = jn; else jz[k] = jn;
        s.ez[r + 1][k] = v;
      }
    } else
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = row_in && (!X || p.me(k));
      const float jo = JS ? jv[k] : jz[k];
      const float jn = upd_j(C.ja, jo, kv[k], s.ez[r + 1][k]);
      float v = tile_e<LOSSLESS, T>(C, s.ez[r + 1][k], __fsub_rn(s.hy[r][k], hyl[k]), dex[k], __fsub_rn(s.hx[r][k], s.hx[r + 1][k]),
                                    dey, jn);
      if (X) {
        const bool strip = p.xe(k) && row_in;
        const float q = upd_psi(b[k], px[k], c[k], s.hy[r][k], hyl[k]);
        const float w = __fmaf_rn(C.pcb, q, v);
        v = strip ? w : v;
        px[k] = strip ? q : px[k];
      }
      if (Y) {
        const float q = upd_psi(yb, py[k], yc, s.hx[r][k], s.hx[r + 1][k]);
        const float w = __fmaf_rn(C.pcb, q, v);
        v = ystrip ? w : v;
        py[k] = ystrip && in ? q : py[k];
      }
      if (JS) jv[k] = in ? jn : jo; else jz[k] = in ? jn : jo;
      s.ez[r + 1][k] = in ? v : s.ez[r + 1][k];
    }
    if (JS && sizeof(T) == 2) Sto<T>::rt4(jv, jv);
    if (r % kBatch == kBatch - 1 || r == R - 1) {
#pragma unroll
      for (int q = r - r % kBatch; q <= r; ++q) {
        if (X && p.strip()) psi.x[(rows + row0 + q) * p.nxl + p.xslot] = put4(pxq[q % kBatch]);
        if (Y) psi.y[(R + 1 + q) * 32] = put4(pyq[q % kBatch]);
        if (JS) js[q * stride] = put4(jq[q % kBatch]);
      }
    }
  }
}

// Strip lanes of the 128 columns at c0, y warps among `warps` of R rows from r0.
inline int strip_lanes(const DevShot& s, int c0) {
  int n = 0;
  for (int l = 0; l < 32; ++l) {
    bool any = false;
    for (int k = 0; k < 4; ++k) {
      const int c = c0 + 4 * l + k;
      any = any || (c >= 0 && c <= s.npml - 1) || (c >= s.nx - s.npml && c <= s.nx - 2);
    }
    n += any;
  }
  return n;
}
inline int y_warps(const DevShot& s, int r0, int warps, int R) {
  int n = 0;
  for (int w = 0; w < warps; ++w) n += tile_y(s, r0 + w * R, R) ? 1 : 0;
  return n;
}

// Sources, then detectors, of the warp's rows at step n (points [p0, p1) of the
// shot's table are those of its rows, a row's sources before its detectors, the
// sources of a cell in the order in which they are subtracted).  Detectors record in
// the columns of the mask `own` and rows [u0, u1), the ones this tile answers for.
//
// 32 points at a time, one per lane, which loads and stores what belongs to its point
// (its entry, the source's value, the detector's trace and sum) beside the others; the
// cells' values come and go by shuffle.  A point at a time, its loads one after
// another, took 0.1 to 0.4 us a step for each point of a warp's rows.  us per step then
// and now: 16 sources and detectors along y, 700^2 6.0 and 3.7; 40 along x, 1500^2 30
// and 9.0; 40 x 40 detectors, 512^2 90 and 8.3; 400 sources along x, 1500^2 75 and 17.
template <int R, bool JS, class T>
__device__ __forceinline__ void tile_points(TileRegs<R, JS>& s, const DevShot& S, const TilePos& p, int p0, int p1, int n,
                                            unsigned own, int u0, int u1, int lane) {
  constexpr bool sc = sizeof(T) == 2;
  const int c0 = p.i - 4 * lane;
#pragma unroll 1
  for (int q0 = p0; q0 < p1; q0 += 32) {
    int4 pt = make_int4(c0 - 1, 0, 0, 0);
    if (q0 + lane < p1) pt = __ldg(S.pts + q0 + lane);
    const int x = pt.x - c0;
    const bool in = x >= 0 && x < kTileCols, src = in && pt.y == kPointSource;
    if (!__any_sync(kFull, in)) continue;
    const int at = in ? x >> 2 : 0, slot = (pt.w - p.j0) * 4 + (x & 3);
    const unsigned owned = __shfl_sync(kFull, own, at);
    const bool det = in && !src && pt.w >= u0 && pt.w < u1 && (owned >> (x & 3) & 1);
    const bool sum = det && pt.y == kPointDetEz && S.dft;
    // everything the points need from memory is asked for together
    float v = 0.f;
    double2 tw = make_double2(0., 0.), acc = tw;
    if (src) v = __ldg(S.src_val + (int64_t)n * S.n_src + pt.z);
    if (sum) {
      tw = __ldg(S.twiddle + n);
      acc = S.dft[pt.z];
    }
    if (sc) v = __fmul_rn(v, S.isc[0]);
    for (unsigned m = __ballot_sync(kFull, src); m; m &= m - 1) {
      const int k = __ffs(m) - 1;
      const int owner = __shfl_sync(kFull, at, k), cell = __shfl_sync(kFull, slot, k), to = owner == lane ? cell : -1;
      const float w = __shfl_sync(kFull, v, k);
#pragma unroll
      for (int t = 0; t < 4 * R; ++t)
        if (t == to) s.ez[t / 4 + 1][t % 4] = __fsub_rn(s.ez[t / 4 + 1][t % 4], w);
    }
    if (!__any_sync(kFull, det)) continue;
    float e = 0.f;
#pragma unroll
    for (int t = 0; t < 4 * R; ++t) {
      const float z = __shfl_sync(kFull, s.ez[t / 4 + 1][t % 4], at);
      e = t == slot ? z : e;
    }
    if (sc) e = __fmul_rn(e, S.sc[0]);
    if (det && pt.y == kPointDetEz && S.record) S.trace[(int64_t)(n - 1) * S.n_det + pt.z] = e;
    if (sum) {
      acc.x = fma((double)e, tw.x, acc.x);
      acc.y = fma(-(double)e, tw.y, acc.y);
      S.dft[pt.z] = acc;
    }
    const bool comp = det && pt.y == kPointDetComp;
    if (S.record && __any_sync(kFull, comp)) {
      float hxv = 0.f, hyv = 0.f;
#pragma unroll
      for (int t = 0; t < 4 * R; ++t) {
        const float a = __shfl_sync(kFull, s.hx[t / 4 + 1][t % 4], at), b = __shfl_sync(kFull, s.hy[t / 4][t % 4], at);
        hxv = t == slot ? a : hxv;
        hyv = t == slot ? b : hyv;
      }
      if (comp) {
        float* dst = S.ctrace + ((int64_t)(n - 1) * S.n_comp + pt.z) * 3;
        dst[0] = e;
        dst[1] = sc ? __fmul_rn(hxv, S.sc[1]) : hxv;
        dst[2] = sc ? __fmul_rn(hyv, S.sc[2]) : hyv;
      }
    }
  }
}

// The same, a point at a time by the thread that holds its cell: its loads wait for one
// another, but the tiles without points keep more of their registers (tile_few).
template <int R, bool JS, class T>
__device__ __forceinline__ void tile_few_points(TileRegs<R, JS>& s, const DevShot& S, const TilePos& p, int p0, int p1, int n,
                                            unsigned own, int u0, int u1) {
  constexpr bool sc = sizeof(T) == 2;
  for (int q = p0; q < p1; ++q) {
    const int4 pt = __ldg(S.pts + q);
    const int k = pt.x - p.i, r = pt.w - p.j0;
    if (k < 0 || k > 3) continue;
    const int at = r * 4 + k;
    float e = 0.f;
#pragma unroll
    for (int t = 0; t < 4 * R; ++t)
      if (t == at) e = s.ez[t / 4 + 1][t % 4];
    if (pt.y == kPointSource) {
      const float v = __ldg(S.src_val + (int64_t)n * S.n_src + pt.z);
      e = __fsub_rn(e, sc ? __fmul_rn(v, S.isc[0]) : v);
#pragma unroll
      for (int t = 0; t < 4 * R; ++t)
        if (t == at) s.ez[t / 4 + 1][t % 4] = e;
    } else if (!(own >> k & 1) || pt.w < u0 || pt.w >= u1) {
      continue;
    } else if (pt.y == kPointDetEz) {
      if (sc) e = __fmul_rn(e, S.sc[0]);
      if (S.record) S.trace[(int64_t)(n - 1) * S.n_det + pt.z] = e;
      if (S.dft) {
        const double2 tw = __ldg(S.twiddle + n);
        double2 acc = S.dft[pt.z];
        acc.x = fma((double)e, tw.x, acc.x);
        acc.y = fma(-(double)e, tw.y, acc.y);
        S.dft[pt.z] = acc;
      }
    } else if (S.record) {
      float hxv = 0.f, hyv = 0.f;
#pragma unroll
      for (int t = 0; t < 4 * R; ++t)
        if (t == at) { hxv = s.hx[t / 4 + 1][t % 4]; hyv = s.hy[t / 4][t % 4]; }
      float* dst = S.ctrace + ((int64_t)(n - 1) * S.n_comp + pt.z) * 3;
      dst[0] = sc ? __fmul_rn(e, S.sc[0]) : e;
      dst[1] = sc ? __fmul_rn(hxv, S.sc[1]) : hxv;
      dst[2] = sc ? __fmul_rn(hyv, S.sc[2]) : hyv;
    }
  }
}

// Slots of the thread's columns in the tracked list (TileAux::cols), 8 bits per
// column, 0 for none: the columns of the mask `own`.
__device__ __forceinline__ unsigned tile_tracked(const TileAux& A, int i, unsigned own) {
  unsigned slots = 0;
  for (int u = 0; u < A.n_cols; ++u) {
    const int k = __ldg(A.cols + u) - i;
    if (k >= 0 && k < 4 && (own >> k & 1)) slots |= (unsigned)(u + 1) << 8 * k;
  }
  return slots;
}

// Records state n of the rows [u0, u1) among the thread's: its tracked columns
// and its part of the line probe.
template <int R, bool JS>
__device__ __forceinline__ void tile_record(const TileRegs<R, JS>& s, const TileAux& A, unsigned slots, const TilePos& p,
                                            unsigned own, int u0, int u1, int n) {
  if (slots) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int u = slots >> 8 * k & 255;
      if (!u) continue;
      float* h = A.hist + ((int64_t)(n - A.n0) * A.n_cols + u - 1) * A.rows + p.j0;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (p.j0 + r >= u0 && p.j0 + r < u1) h[r] = s.ez[r + 1][k];
    }
  }
  if (A.line_n > 0 && n >= A.line_first && n <= A.line_last && A.line_j >= max(u0, p.j0) && A.line_j < min(u1, p.j0 + R)) {
    float* dst = A.line + (int64_t)(n - A.line_first) * A.line_n;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (p.j0 + r != A.line_j) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = p.i + k - A.line_i0;
        if ((own >> k & 1) && c >= 0 && c < A.line_n) dst[c] = s.ez[r + 1][k];
      }
    }
  }
}

// 16-bit storage: the values a store and a load would give back.
template <int R, bool JS, class T>
__device__ __forceinline__ void tile_round(TileRegs<R, JS>& s) {
  if constexpr (sizeof(T) == 2) {
    using St = Sto<T>;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      St::rt4(s.ez[r + 1], s.ez[r + 1]);
      St::rt4(s.hx[r + 1], s.hx[r + 1]);
      St::rt4(s.hy[r], s.hy[r]);
      if (!JS) St::rt4(s.jz[JS ? 0 : r], s.jz[JS ? 0 : r]);
    }
    St::rt4(s.hx[0], s.hx[0]);
  }
}

}  // namespace
}  // namespace fdtd2d

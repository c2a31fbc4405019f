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

// Column and row tables of a tile that is not plain, in shared memory.
// Columns: b and c/d of the Hy and Ez recursions (the column's strip), and
// the denominators; rows likewise for Hx and Ez.
enum TabCol : int { kTcBh = 0, kTcCh, kTcBe, kTcCe, kTcDe, kTcDh, kTcRows };
constexpr int kTileCols = 128;

// Coefficients of a shot in stored units.
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
struct TilePos {
  int i, j0;          // first column and row
  unsigned mh, me;    // columns (bits 0-3) whose H / Ez are updated
  unsigned xh, xe;    // columns in an x strip for Hy / Ez
  int xslot, nxl;     // the thread's slot among the row's strip lanes, their number
  int ylo, yhi, nyl;  // strip rows: slot of row j is j - ylo (j < npml) or j - yhi; their number
};

// psi of a tile in shared memory.
struct TilePsi {
  float4* x;   // [Hy, Ez][rows][nxl]
  float4* y;   // [Hx, Ez][nyl][32]
  float4* b;   // [warps][32]: Hx of the row below each warp
};

__device__ __forceinline__ void get4(float (&d)[4], const float4& v) { d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w; }
__device__ __forceinline__ float4 put4(const float (&d)[4]) { return make_float4(d[0], d[1], d[2], d[3]); }

// Strip row of Hx (side -1: none): rows 0 .. P-2 and ny-P .. ny-2.
__device__ __forceinline__ bool y_strip_h(int j, int ny, int P) { return (j >= 0 && j <= P - 2) || (j >= ny - P && j <= ny - 2); }
// Strip row of Ez: rows 1 .. P-1 and ny-P .. ny-2.
__device__ __forceinline__ bool y_strip_e(int j, int ny, int P) { return (j >= 1 && j <= P - 1) || (j >= ny - P && j <= ny - 2); }

// Geometry of a thread in the tile at (c0, r0) of `rows` rows; `plain` tiles
// have no CPML and no border.
__device__ __forceinline__ TilePos tile_pos(const DevShot& S, int c0, int r0, int rows, int j0, int lane, bool plain) {
  TilePos p{};
  p.i = c0 + 4 * lane;
  p.j0 = j0;
  if (plain) return p;
  const int nx = S.nx, ny = S.ny, P = S.npml;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = p.i + k;
    if (c >= 0 && c <= nx - 2) p.mh |= 1u << k;
    if (c >= 1 && c <= nx - 2) p.me |= 1u << k;
    if ((c >= 0 && c <= P - 2) || (c >= nx - P && c <= nx - 2)) p.xh |= 1u << k;
    if ((c >= 1 && c <= P - 1) || (c >= nx - P && c <= nx - 2)) p.xe |= 1u << k;
  }
  const unsigned m = __ballot_sync(kFull, (p.xh | p.xe) != 0);
  p.xslot = __popc(m & ((1u << lane) - 1));
  p.nxl = __popc(m);
  const int top = r0 + rows;                      // one past the tile's last row
  const int lo0 = max(r0, 0), lo = max(0, min(top, P) - lo0);
  const int hi0 = max(r0, ny - P), hi = max(0, min(top, ny - 1) - hi0);
  p.ylo = lo0;
  p.yhi = hi0 - lo;
  p.nyl = lo + hi;
  return p;
}

__device__ __forceinline__ TilePsi tile_psi(float4* base, const TilePos& p, int rows) {
  TilePsi s;
  s.x = base;
  s.y = s.x + 2 * rows * p.nxl;
  s.b = s.y + 2 * p.nyl * 32;
  return s;
}

// The tables of a tile that is not plain: tc[kTcRows][128] by column, tr[kTcRows][rows+1] by row (row r0-1 first).
__device__ __forceinline__ void tile_tables(const DevShot& S, float* tc, float* tr, int c0, int r0, int rows, int tid,
                                            int threads) {
  const int nx = S.nx, ny = S.ny, P = S.npml;
  for (int t = tid; t < kTileCols + rows + 1; t += threads) {
    const bool col = t < kTileCols;
    const int c = col ? c0 + t : r0 - 1 + (t - kTileCols);
    const int n = col ? nx : ny;
    float* out = col ? tc + t : tr + (t - kTileCols);
    const int st = col ? kTileCols : rows + 1;
    float bh = 0.f, ch = 0.f, be = 0.f, ce = 0.f, de = 0.f, dh = 0.f;
    const int h0 = col ? kBhX1 : kBhY1, e0 = col ? kBeX1 : kBeY1;
    if (c >= 0 && c <= P - 2) { bh = S.cpml[h0 * P + c]; ch = S.cpml[(h0 + 1) * P + c]; }
    else if (c >= n - P && c <= n - 2) { bh = S.cpml[(h0 + 2) * P + n - 2 - c]; ch = S.cpml[(h0 + 3) * P + n - 2 - c]; }
    if (c >= 1 && c <= P - 1) { be = S.cpml[e0 * P + c]; ce = S.cpml[(e0 + 1) * P + c]; }
    else if (c >= n - P && c <= n - 2) { be = S.cpml[(e0 + 2) * P + n - 1 - c]; ce = S.cpml[(e0 + 3) * P + n - 1 - c]; }
    if (c >= 0 && c < n - 1) { de = (col ? S.den_ex : S.den_ey)[c]; dh = (col ? S.den_hx : S.den_hy)[c]; }
    out[kTcBh * st] = bh; out[kTcCh * st] = ch; out[kTcBe * st] = be; out[kTcCe * st] = ce;
    out[kTcDe * st] = de; out[kTcDh * st] = dh;
  }
}

// One time step of the thread's cells up to Ez, without sources, detectors
// and the rounding to the storage type; s.ez[0] and s.ez[R+1] hold the rows
// around the thread's.  PLAIN: no CPML, no border, the denominators are the shot's
// constants.  kp: the thread's drive, `stride` float4 from row to row.
template <int R, bool JS, bool LOSSLESS, bool PLAIN, class T>
__device__ __forceinline__ void tile_step(TileRegs<R, JS>& s, const DevShot& S, const Coef<T>& C, const TilePos& p,
                                          const TilePsi& psi, const float* tc, const float* tr, int rows, int row0,
                                          const float4* kp, float4* js, int stride, int warp, int lane) {
  const int ny = S.ny, P = S.npml;
  const float dhx_c = S.den_c[1], dhy_c = S.den_c[3], dex_c = S.den_c[0], dey_c = S.den_c[2];
  const int ts = rows + 1;             // row tables start at row r0 - 1
  // ---- Hx: row j0 - 1 (the warp below owns it), then the thread's rows
#pragma unroll
  for (int r = 0; r <= R; ++r) {
    const float den = PLAIN ? dhy_c : tr[kTcDh * ts + row0 + r];
    const int j = p.j0 - 1 + r;
    if (!PLAIN && !(j >= 0 && j <= ny - 2)) continue;
    const bool strip = !PLAIN && y_strip_h(j, ny, P);
    float4* ps = r == 0 ? psi.b + warp * 32 + lane : psi.y + (j - (j < P ? p.ylo : p.yhi)) * 32 + lane;
    float pn[4] = {0.f, 0.f, 0.f, 0.f};
    if (strip) get4(pn, *ps);
    const float b = strip ? tr[kTcBh * ts + row0 + r] : 0.f;
    const float c = strip ? __fmul_rn(tr[kTcCh * ts + row0 + r], C.sE) : 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = PLAIN || (p.mh >> k & 1);
      float v = tile_h<LOSSLESS>(C.da, s.hx[r][k], C.db, s.ez[r][k], s.ez[r + 1][k], den);
      if (strip) {
        const float q = upd_psi(b, pn[k], c, s.ez[r][k], s.ez[r + 1][k]);
        v = __fmaf_rn(C.pdb, q, v);
        pn[k] = in ? q : pn[k];
      }
      s.hx[r][k] = in ? v : s.hx[r][k];
    }
    if (strip) *ps = put4(pn);
  }
  // ---- Hy
  float dhx[4], dex[4];
  if (PLAIN) {
#pragma unroll
    for (int k = 0; k < 4; ++k) { dhx[k] = dhx_c; dex[k] = dex_c; }
  } else {
    lds4f(dhx, tc + kTcDh * kTileCols + 4 * lane);
    lds4f(dex, tc + kTcDe * kTileCols + 4 * lane);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float e4 = __shfl_down_sync(kFull, s.ez[r + 1][0], 1);
    const float er[4] = {s.ez[r + 1][1], s.ez[r + 1][2], s.ez[r + 1][3], e4};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float v = tile_h<LOSSLESS>(C.da, s.hy[r][k], C.db, er[k], s.ez[r + 1][k], dhx[k]);
      s.hy[r][k] = PLAIN || (p.mh >> k & 1) ? v : s.hy[r][k];
    }
    if (!PLAIN && p.xh) {
      float b[4], c[4], pn[4];
      lds4f(b, tc + kTcBh * kTileCols + 4 * lane);
      lds4f(c, tc + kTcCh * kTileCols + 4 * lane);
      float4* ps = psi.x + (row0 + r) * p.nxl + p.xslot;
      get4(pn, *ps);
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
        const bool in = p.xh >> k & 1;
        const float q = upd_psi(b[k], pn[k], __fmul_rn(c[k], C.sE), er[k], s.ez[r + 1][k]);
        const float v = __fmaf_rn(C.pdb, q, s.hy[r][k]);
        pn[k] = in ? q : pn[k];
        s.hy[r][k] = in ? v : s.hy[r][k];
      }
      *ps = put4(pn);
    }
  }
  // ---- Jz and Ez
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float hl = __shfl_up_sync(kFull, s.hy[r][3], 1);
    const float hyl[4] = {hl, s.hy[r][0], s.hy[r][1], s.hy[r][2]};
    const int j = p.j0 + r;
    if (!PLAIN && !(j >= 1 && j <= ny - 2)) continue;
    float kv[4];
    get4(kv, kp[r * stride]);
    float (&jz)[4] = s.jz[JS ? 0 : r];
    if (JS) get4(jz, js[r * stride]);
    const float dey = PLAIN ? dey_c : tr[kTcDe * ts + row0 + 1 + r];
    float ep[4] = {0.f, 0.f, 0.f, 0.f};
    if (!PLAIN && p.xe) {
      float b[4], c[4];
      lds4f(b, tc + kTcBe * kTileCols + 4 * lane);
      lds4f(c, tc + kTcCe * kTileCols + 4 * lane);
      float4* ps = psi.x + (rows + row0 + r) * p.nxl + p.xslot;
      get4(ep, *ps);
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
        const float q = upd_psi(b[k], ep[k], __fmul_rn(c[k], C.sH), s.hy[r][k], hyl[k]);
        ep[k] = p.xe >> k & 1 ? q : ep[k];
      }
      *ps = put4(ep);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = PLAIN || (p.me >> k & 1);
      const float jn = upd_j(C.ja, jz[k], kv[k], s.ez[r + 1][k]);
      float v = tile_e<LOSSLESS, T>(C, s.ez[r + 1][k], __fsub_rn(s.hy[r][k], hyl[k]), dex[k], __fsub_rn(s.hx[r][k], s.hx[r + 1][k]), dey, jn);
      if (!PLAIN && p.xe) {
        const float w = __fmaf_rn(C.pcb, ep[k], v);
        v = p.xe >> k & 1 ? w : v;
      }
      jz[k] = in ? jn : jz[k];
      s.ez[r + 1][k] = in ? v : s.ez[r + 1][k];
    }
    if (JS) {
      if (sizeof(T) == 2) Sto<T>::rt4(jz, jz);
      js[r * stride] = put4(jz);
    }
    if (!PLAIN && y_strip_e(j, ny, P)) {
      const float b = tr[kTcBe * ts + row0 + 1 + r], c = __fmul_rn(tr[kTcCe * ts + row0 + 1 + r], C.sH);
      float4* ps = psi.y + (p.nyl + j - (j < P ? p.ylo : p.yhi)) * 32 + lane;
      float pn[4];
      get4(pn, *ps);
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
        const bool in = p.me >> k & 1;
        const float q = upd_psi(b, pn[k], c, s.hx[r][k], s.hx[r + 1][k]);
        const float v = __fmaf_rn(C.pcb, q, s.ez[r + 1][k]);
        pn[k] = in ? q : pn[k];
        s.ez[r + 1][k] = in ? v : s.ez[r + 1][k];
      }
      *ps = put4(pn);
    }
  }
}

// Sources, then detectors, of the thread's rows at step n (points [p0, p1) of
// the shot's table are those of the warp's rows).  Detectors record where
// `own`; rows [u0, u1) are the ones this tile answers for.
template <int R, bool JS, class T>
__device__ __forceinline__ void tile_points(TileRegs<R, JS>& s, const DevShot& S, const TilePos& p, int p0, int p1, int n,
                                            bool own, int u0, int u1) {
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
    } else if (!own || pt.w < u0 || pt.w >= u1) {
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

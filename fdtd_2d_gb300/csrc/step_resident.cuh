// Many steps per launch with the whole shot on chip (grids whose cells fit the
// registers of the GPU's SMs).
//
// step_persist_tile_kernel<R> (T: the fields' element; MED: the material-ID medium): one cooperative launch whose CTAs, one per SM,
// each keep a tile of the grid in registers (tile_common.cuh) for every step
// of a run call.  CTAs are nb bands of w columns cut into strips of rows; a
// warp has R rows.  Strips are cut by cost (a row of a band with x strips takes
// about 1.8 plain rows, a warp in a y strip 0.6 more), so that the corners and
// edges of the grid do not set every step's time.  Of a neighbouring tile a step needs only Ez: one row above and
// below (Hx of the row below is recomputed here), one column left and right
// (Hy of the column left is recomputed here, its Ez column replaced by the
// neighbour's after every step).  These go through L2 as 64-bit words that
// carry the value and the step's tag together, so a reader polls the data
// itself: one trip through L2 per step, no flag, no fence, no grid barrier.
// Two slots by the step's parity are enough: a warp overwrites a word it sent
// two steps ago only after its reader, the CTAs across the same edge, have
// sent the word that followed from it.  One warp of each CTA does nothing but
// send and receive: the others leave their edges in shared memory, meet it at
// one barrier and find the neighbours' edges in shared memory after the next,
// so that addresses, tags and polling cost the stepping warps no registers (a
// version in which every warp polled spilled 200 to 400 B per thread, and its
// step took 1.5x as long).
//
// Waits are bounded as in the other kernels: after wait_ns without progress, or
// another CTA's error, the error word is set and the CTA polls for nothing more
// until its steps are through.
//
// What bounds it: the loop between neighbouring CTAs, a step of each and the trip
// of their edges through L2 (~1100 cycles for a poll's round trip alone, ~2800 in
// all at 512^2, where the step itself takes 400 to 1500), and from ~1 M cells on
// the updates themselves.  us per step on GB300 against the kernels before it
// (L2-resident persistent kernel, two-step path): 256 x 192 1.70 (6.0), 512^2 1.9
// (6.1), 777 x 1301 2.87 (16.4), 1024^2 2.90 (13.0); the tile passes of
// step_tile.cu take 3.55 at 512^2 and 4.5 at 1024^2.
#pragma once

#include "internal.h"
#include "tile_common.cuh"

namespace fdtd2d {

namespace {

constexpr int kOwn = kTileCols - 2;   // most columns a band owns: one halo column on each side

// Warps a CTA may have at R rows per warp, from the registers a thread needs.
// (an SM's four register files hold 16 K words each: 3, 4, 5 warps of 168, 128,
// 96 registers).
__host__ __device__ constexpr int all_warps(int R) { return R >= 6 ? 12 : R == 4 ? 16 : 20; }
__host__ __device__ constexpr int max_warps(int R) { return all_warps(R) - 1; }   // one sends and receives
// Jz in shared memory where the rows leave no registers for it.
__host__ __device__ constexpr bool jz_shared(int R) { return R >= 6; }

__device__ __forceinline__ uint64_t tagged(float v, uint32_t tag) { return ((uint64_t)tag << 32) | __float_as_uint(v); }
__device__ __forceinline__ void send1(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void send2(uint64_t* p, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void poll2(const uint64_t* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ uint64_t poll1(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

struct Waiter {
  volatile int* dead;   // shared: this CTA waits no more
  int* err;
  uint64_t ns;
  // False when the wait is over without the data.
  __device__ __forceinline__ bool again(int& it, uint64_t& t0) const {
    if (*dead) return false;
    if (++it & 63) return true;
    const uint64_t t = global_ns();
    if (it == 64) {
      t0 = t;
    } else if (t - t0 > ns) {
      atomicExch(err, kErrWaitTimeout);
      *dead = 1;
      return false;
    }
    if (*(volatile int*)err != kErrNone) {
      *dead = 1;
      return false;
    }
    return true;
  }
};

// Named barriers of a CTA: 1 when the stepping warps have left their edges, 2
// when the neighbours' are there.
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// A CTA's edges in shared memory: columns out and in ([left, right][rows]),
// rows in ([below, above][32] float4).
struct Edges {
  float *col_out, *col_in;
  float4* row_in;
};
__host__ __device__ constexpr int edge_f4(int rows) { return (4 * rows + 3) / 4 + 64; }

// The warp that sends and receives, for every step of a launch.
__device__ __forceinline__ void exchange(const ResidentPlan& G, const Edges& E, const float4* ex, int nw, int rows, int r0, int b,
                                         int k, bool has_u, int steps, uint64_t* link, const Waiter& wait, uint32_t tag_add,
                                         int threads, int lane) {
  // Words by the step's parity: per CTA its first and last row of 128, then
  // per band its first and last column over all rows (neighbouring bands cut
  // their rows differently).
  const int64_t n_rows = (int64_t)gridDim.x * 2 * kTileCols, height = (int64_t)G.groups * G.R;
  const int64_t per = n_rows + 2 * G.nb * height;
  const bool has_l = b > 0, has_r = b + 1 < G.nb, has_d = k > 0;
  uint64_t* my_row = link + (int64_t)blockIdx.x * 2 * kTileCols + 4 * lane;
  // column words of this lane: number q = lane + 32 i, left ones first
  constexpr int kMost = 2 * 96 / 32;
  const int nl = has_l ? rows : 0, nc = nl + (has_r ? rows : 0);
  uint64_t* left = link + n_rows + 2 * b * height + r0;       // this band's first column; its last one `height` on
  for (int t = 0; t < steps; ++t) {
    const int par = t & 1;
    const uint32_t tag = (uint32_t)t + 1, want = tag + tag_add;
    bar_sync(1, threads);
    const float4* e = ex + par * 2 * G.nw * 32;
    uint64_t* row = my_row + par * per;
    uint64_t* col = left + par * per;
#pragma unroll
    for (int i = 0; i < kMost; ++i) {
      if (32 * i >= nc) break;
      const int q = lane + 32 * i;
      if (q < nl) send1(col + q, tagged(E.col_out[q], tag));
      else if (q < nc) send1(col + height + (q - nl), tagged(E.col_out[rows + q - nl], tag));
    }
    if (has_d) {
      const float4 v = e[lane];
      send2(row, tagged(v.x, tag), tagged(v.y, tag));
      send2(row + 2, tagged(v.z, tag), tagged(v.w, tag));
    }
    if (has_u) {
      const float4 v = e[(2 * nw - 1) * 32 + lane];
      send2(row + kTileCols, tagged(v.x, tag), tagged(v.y, tag));
      send2(row + kTileCols + 2, tagged(v.z, tag), tagged(v.w, tag));
    }
    // everything the neighbours send is asked for together: one trip through L2
    uint64_t c[kMost], d[4], u[4], t0 = 0;
    int it = 0;
    for (;;) {
#pragma unroll
      for (int i = 0; i < kMost; ++i) {
        if (32 * i >= nc) break;
        const int q = lane + 32 * i;
        if (q < nc) c[i] = poll1(q < nl ? col - height + q : col + 2 * height + (q - nl));
      }
      if (has_d) {
        poll2(row - kTileCols, d[0], d[1]);
        poll2(row - kTileCols + 2, d[2], d[3]);
      }
      if (has_u) {
        poll2(row + 2 * kTileCols, u[0], u[1]);
        poll2(row + 2 * kTileCols + 2, u[2], u[3]);
      }
      bool ok = true;
#pragma unroll
      for (int i = 0; i < kMost; ++i) {
        if (32 * i >= nc) break;
        ok = ok && (lane + 32 * i >= nc || (uint32_t)(c[i] >> 32) == want);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        ok = ok && (!has_d || (uint32_t)(d[i] >> 32) == want) && (!has_u || (uint32_t)(u[i] >> 32) == want);
      if (__all_sync(kFull, ok)) break;
      if (!__all_sync(kFull, wait.again(it, t0))) break;
    }
    auto f = [](uint64_t v) { return __uint_as_float((uint32_t)v); };
#pragma unroll
    for (int i = 0; i < kMost; ++i) {
      if (32 * i >= nc) break;
      const int q = lane + 32 * i;
      if (q < nc) E.col_in[q < nl ? q : rows + q - nl] = f(c[i]);
    }
    if (has_d) E.row_in[lane] = make_float4(f(d[0]), f(d[1]), f(d[2]), f(d[3]));
    if (has_u) E.row_in[32 + lane] = make_float4(f(u[0]), f(u[1]), f(u[2]), f(u[3]));
    __syncwarp();
    bar_arrive(2, threads);
  }
}

// A source or detector of a warp's rows, in shared memory with its running
// state: lane q of the warp serves point q.
struct ResPoint {
  int kind, slot, idx;   // slot: its cell's place among the warp's source or detector cells
  float val;             // the step's source value
  double2 tw, acc;       // the step's DFT twiddle, the running sum
};
constexpr int kWarpPoints = 32;
// A warp's points in shared memory: per lane a word of its source cells, of its
// detector cells (bit 4 r + k) and of the first slots of both; the source values
// and the detector cells' Ez, Hx, Hy by slot; the points.
constexpr int kPointF4 = 32 + 4 * kWarpPoints / 4 + kWarpPoints * (int)sizeof(ResPoint) / 16;

// The points of a warp.  A step's source values and twiddles are copied in
// from its start on (cp.async), the sums stay in shared memory for the whole
// launch, and the rows that hold points pass their cells' values through slots in
// shared memory, a predicated access per cell, so that no register is indexed by a
// point's position.  (Points read from global memory and cells found by selects
// took 0.4 us of a 512^2 step; loops over a warp's points that touch its cells'
// registers slowed the whole step by up to 2x.  Buffers of all the warp's cells
// cost 8 KB more shared memory per warp with points at 8 rows, and the registers
// spilled there no longer fit the L1 cache beside it: 500 x 3000 5.25 us per step,
// 3.80 now, 1600 x 900 5.18 and 3.98.)
struct ResPoints {
  float4* mem;
  // 0: no points; bits 0-5 their number, 6 sources, 7 detectors, 8 component ones
  // among them; 9 + r source cells in row r, 17 + r detector cells
  int state;
  static constexpr int kSrc = 64, kDet = 128, kComp = 256, kSrcRow = 9, kDetRow = 17;
  __device__ __forceinline__ uint4* words() const { return reinterpret_cast<uint4*>(mem); }
  __device__ __forceinline__ float* vals() const { return reinterpret_cast<float*>(mem + 32); }
  __device__ __forceinline__ float* cells() const { return vals() + kWarpPoints; }
  __device__ __forceinline__ ResPoint* points() const { return reinterpret_cast<ResPoint*>(mem + 32 + kWarpPoints); }
  __device__ __forceinline__ int count() const { return state & 63; }
  // the slot of the cell of bit b
  __device__ __forceinline__ static int slot(unsigned mask, unsigned first, int b) { return (int)first + __popc(mask & ((1u << b) - 1)); }

  template <int R>
  __device__ __forceinline__ void begin(const DevShot& S, int j0, int c0, int lo, int hi, float4* smem, int* slots, int lane) {
    state = 0;
    mem = smem;
    int flags = 0;
    if (j0 >= S.ny) return;
    const int p0 = __ldg(S.row_start + j0), p1 = __ldg(S.row_start + min(j0 + R, S.ny));
    // where they start: first whether there are any
    for (int pass = 0; pass < 2; ++pass) {
      int n = 0;
      for (int q = p0; q < p1; q += 32) {
        bool in = q + lane < p1;
        int4 pt = make_int4(0, 0, 0, 0);
        if (in) pt = __ldg(S.pts + q + lane);
        const int x = pt.x - c0;
        in = in && x >= lo && x < hi;
        const unsigned m = __ballot_sync(kFull, in);
        const bool src = pt.y == kPointSource;
        if (pass && in) {
          ResPoint& p = points()[n + __popc(m & ((1u << lane) - 1))];
          p.kind = pt.y;
          p.slot = (x >> 2) * 32 + 4 * (pt.w - j0) + (x & 3);   // lane and bit, until the slots are known
          p.idx = pt.z;
          if (pt.y == kPointDetEz && S.dft) p.acc = S.dft[pt.z];
          unsigned* w = reinterpret_cast<unsigned*>(words() + (x >> 2));
          atomicOr(w + (src ? 0 : 1), 1u << (4 * (pt.w - j0) + (x & 3)));
        }
        flags |= (__any_sync(kFull, in && src) ? kSrc : 0) | (__any_sync(kFull, in && !src) ? kDet : 0) |
                 (__any_sync(kFull, in && pt.y == kPointDetComp) ? kComp : 0);
        for (int r = 0; r < R; ++r)
          flags |= (__any_sync(kFull, in && src && pt.w - j0 == r) ? 1 << (kSrcRow + r) : 0) |
                   (__any_sync(kFull, in && !src && pt.w - j0 == r) ? 1 << (kDetRow + r) : 0);
        n += __popc(m);
      }
      if (n == 0) return;
      if (pass == 0) {
        int at = 0;
        if (lane == 0) at = atomicAdd(slots, 1);
        at = __shfl_sync(kFull, at, 0);
        mem = smem + at * kPointF4;
        state = n | flags;
        words()[lane] = make_uint4(0, 0, 0, 0);
        __syncwarp();
      }
    }
    __syncwarp();
    const uint4 w = words()[lane];
    int s = __popc(w.x), d = __popc(w.y);
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int a = __shfl_up_sync(kFull, s, o), b = __shfl_up_sync(kFull, d, o);
      s += lane >= o ? a : 0;
      d += lane >= o ? b : 0;
    }
    words()[lane] = make_uint4(w.x, w.y, s - __popc(w.x), d - __popc(w.y));
    __syncwarp();
    if (lane < count()) {
      ResPoint& p = points()[lane];
      const uint4 v = words()[p.slot >> 5];
      p.slot = p.kind == kPointSource ? slot(v.x, v.z, p.slot & 31) : slot(v.y, v.w, p.slot & 31);
    }
    __syncwarp();
  }
  __device__ __forceinline__ void end(const DevShot& S, int lane) const {
    const ResPoint* at = points();
    if (lane < count() && at[lane].kind == kPointDetEz && S.dft) S.dft[at[lane].idx] = at[lane].acc;
  }
  __device__ __forceinline__ void load_step(const DevShot& S, int n, int lane) const {
    if (lane < count()) {
      ResPoint& p = points()[lane];
      if (p.kind == kPointSource)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&p.val)),
                     "l"(S.src_val + (int64_t)n * S.n_src + p.idx));
      else if (S.dft)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&p.tw)), "l"(S.twiddle + n));
    }
  }
  // A step's sources, on the cells after their Ez update.
  template <int R, bool JS, class T>
  __device__ __forceinline__ void sources(TileRegs<R, JS>& s, const DevShot& S, int lane) const {
    if (!(state & kSrc)) return;
    const ResPoint* at = points();
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (lane < count() && at[lane].kind == kPointSource)
      vals()[at[lane].slot] = sizeof(T) == 2 ? __fmul_rn(at[lane].val, S.isc[0]) : at[lane].val;
    __syncwarp();
    const uint4 w = words()[lane];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!(state >> (kSrcRow + r) & 1)) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (w.x >> (4 * r + k) & 1) s.ez[r + 1][k] = __fsub_rn(s.ez[r + 1][k], vals()[slot(w.x, w.z, 4 * r + k)]);
    }
    __syncwarp();
  }
  // The detectors' cells as they are after the step (16-bit storage: before the
  // step is rounded), left for record().
  template <int R, bool JS>
  __device__ __forceinline__ void leave(const TileRegs<R, JS>& s, int lane) const {
    if (!(state & kDet)) return;
    const uint4 w = words()[lane];
    float* out = cells();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!(state >> (kDetRow + r) & 1)) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!(w.y >> (4 * r + k) & 1)) continue;
        const int q = slot(w.y, w.w, 4 * r + k);
        out[q] = s.ez[r + 1][k];
        if (state & kComp) {
          out[kWarpPoints + q] = s.hx[r + 1][k];
          out[2 * kWarpPoints + q] = s.hy[r][k];
        }
      }
    }
  }
  // Step n's detectors, of the values left.
  template <class T>
  __device__ __forceinline__ void record(const DevShot& S, int n, int lane) const {
    if (!(state & kDet)) return;
    constexpr bool sc = sizeof(T) == 2;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (lane < count() && points()[lane].kind != kPointSource) {
      ResPoint& p = points()[lane];
      const float* in = cells() + p.slot;
      const float e = sc ? __fmul_rn(in[0], S.sc[0]) : in[0];
      if (p.kind == kPointDetEz) {
        if (S.record) S.trace[(int64_t)(n - 1) * S.n_det + p.idx] = e;
        if (S.dft) {
          p.acc.x = fma((double)e, p.tw.x, p.acc.x);
          p.acc.y = fma(-(double)e, p.tw.y, p.acc.y);
        }
      } else if (S.record) {
        float* dst = S.ctrace + ((int64_t)(n - 1) * S.n_comp + p.idx) * 3;
        dst[0] = e;
        dst[1] = sc ? __fmul_rn(in[kWarpPoints], S.sc[1]) : in[kWarpPoints];
        dst[2] = sc ? __fmul_rn(in[2 * kWarpPoints], S.sc[2]) : in[2 * kWarpPoints];
      }
    }
    __syncwarp();
  }
};

template <int R, bool LOSSLESS, bool AUX, bool MED, class T>
__device__ __forceinline__ void resident_run(const DevShot& S, const TileAux& A, const ResidentPlan& G, int n, int steps, uint64_t* link,
                                             const Waiter& wait, uint32_t tag_add, float4* smem, int* slots) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x;
  const int nx = S.nx, ny = S.ny;
  const int64_t pitch = S.pitch;
  // CTAs: the strips of the first band, of the last, then of the others
  const int cta = blockIdx.x, ns0 = G.ns[0], edges = min(G.nb, 2) * ns0;
  const bool edge = cta < edges;
  const int b = edge ? (cta < ns0 ? 0 : G.nb - 1) : 1 + (cta - edges) / G.ns[1];
  const int k = edge ? (cta < ns0 ? cta : cta - ns0) : (cta - edges) % G.ns[1];
  const int g0 = G.start[edge ? 0 : 1][k], g1 = G.start[edge ? 0 : 1][k + 1];
  const int nw = g1 - g0, rows = nw * R, r0 = g0 * R;
  const bool has_u = k + 1 < G.ns[edge ? 0 : 1];
  const bool work = warp < nw;
  const int ww = work ? warp : 0, row0 = ww * R, j0 = r0 + row0;
  const int c0 = b * G.w - 1;                   // the left halo column
  const int own_n = min(G.w, nx - (c0 + 1));    // columns owned: c0+1 .. c0+own_n
  constexpr bool JS = jz_shared(R);
  float4* ex = smem;                            // [2][nw][2][32]
  Edges E;
  E.row_in = ex + 4 * G.nw * 32;
  E.col_out = reinterpret_cast<float*>(E.row_in + 64);
  E.col_in = E.col_out + 2 * rows;
  float4* rest = E.row_in + edge_f4(G.nw * R);
  const int wt = G.nw * 32;                     // threads that step
  constexpr int kWords = MED ? R + 1 : R;
  float4* kps = rest + tid;                     // [kWords][wt]
  float4* jzs = kps + kWords * wt;              // [R][wt] where JS
  rest += (kWords + (JS ? R : 0)) * wt;
  MatTables mat;
  if (MED) {
    float4* e = rest;
    float2* h = reinterpret_cast<float2*>(e + 256);
    for (int t = tid; t < 256; t += threads) {
      e[t] = __ldg(reinterpret_cast<const float4*>(S.mat_e) + t);
      h[t] = __ldg(reinterpret_cast<const float2*>(S.mat_h) + t);
    }
    mat.e = e;
    mat.h = h;
    rest += 256 + 128;
  }
  float4* point_mem = rest;
  rest += G.point_warps * kPointF4;
  float* tc = reinterpret_cast<float*>(rest);
  float* tr = tc + kTcRows * kTileCols;
  const Coef<T> C(S);
  tile_tables<T>(S, C, tc, tr, c0, r0, rows, tid, threads);
  __syncthreads();
  if (warp == G.nw) {
    exchange(G, E, ex, nw, rows, r0, b, k, has_u, steps, link, wait, tag_add, threads, lane);
    return;
  }
  const TilePos p = tile_pos(S, c0, r0, R, ww, lane);
  const TilePsi psi = tile_psi(rest + tile_table_f4(rows), p, rows, R, lane);
  unsigned own = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) own |= (4 * lane + q >= 1 && 4 * lane + q <= own_n ? 1u : 0u) << q;

  TileRegs<R, JS> s;
  {
    const T* f[4];
    const T* drive = reinterpret_cast<const T*>(S.kp);
#pragma unroll
    for (int a = 0; a < 4; ++a) f[a] = field_ptr_t<T>(S, a, 0) + p.i;
#pragma unroll
    for (int r = -1; r <= R; ++r) {
      const int j = j0 + r;
      const bool rin = work && j >= 0 && j < ny;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = p.i + q;
        const bool in = rin && c >= 0 && c < nx;
        const int64_t o = (int64_t)j * pitch + q;
        s.ez[r + 1][q] = in ? Sto<T>::ld1(f[kEz] + o) : 0.f;
        if (r < R) s.hx[r + 1 < R + 1 ? r + 1 : 0][q] = in ? Sto<T>::ld1(f[kHx] + o) : 0.f;
        if (r >= 0 && r < R) {
          s.hy[r >= 0 && r < R ? r : 0][q] = in ? Sto<T>::ld1(f[kHy] + o) : 0.f;
          if (!JS) s.jz[!JS && r >= 0 && r < R ? r : 0][q] = in ? Sto<T>::ld1(f[kJz] + o) : 0.f;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float kv[4], jv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = p.i + q, j = j0 + r;
        const bool in = work && j < ny && c >= 0 && c < nx;
        kv[q] = !MED && drive && in ? Sto<T>::ldg1(drive + (int64_t)j * pitch + c) : 0.f;
        if (sizeof(T) == 2) kv[q] = __fmul_rn(kv[q], C.rk);
        if (JS) jv[q] = in ? Sto<T>::ld1(f[kJz] + (int64_t)j * pitch + q) : 0.f;
      }
      if (!MED) kps[r * wt] = put4(kv);
      if (JS) jzs[r * wt] = put4(jv);
    }
  }
  if (MED && work) {
    for (int r = -1; r < R; ++r)
      *reinterpret_cast<uint4*>(kps + (r < 0 ? R : r) * wt) = mat_make(S, p.i, j0 + r);
  }
  if (work) tile_psi_load<R, false>(S, S.psi, p, psi, rows, row0);
  copies_done();
  // rows around the strip that nobody sends (beyond the grid, or its last row) stay as loaded
  if (work && warp == 0 && k == 0) E.row_in[lane] = put4(s.ez[0]);
  if (work && warp == nw - 1 && !has_u) E.row_in[32 + lane] = put4(s.ez[R + 1]);
  // (a halo column's Ez comes from its owner: own columns only)
  ResPoints pts;
  pts.begin<R>(S, work ? j0 : ny, c0, 1, own_n + 1, point_mem, slots, lane);
  const int lr = G.w >> 2;               // lane of the last own column (k = 2) and the right halo (k = 3)
  const bool l = lane == 0, rr = lane == lr;
  const bool take_l = l && b > 0, take_r = rr && b + 1 < G.nb;
  const int col_at = (rr ? rows : 0) + row0;

  const unsigned tracked = AUX && work ? tile_tracked(A, p.i, own) : 0u;
  // the loop in the form the warp needs
  auto loop = [&](auto x, auto y) {
    for (int t = 0; t < steps; ++t) {
      float4* e = ex + (t & 1) * 2 * G.nw * 32;
      e[(2 * warp) * 32 + lane] = put4(s.ez[1]);
      e[(2 * warp + 1) * 32 + lane] = put4(s.ez[R]);
      if (l || rr) {
#pragma unroll
        for (int r = 0; r < R; ++r) E.col_out[col_at + r] = l ? s.ez[r + 1][1] : s.ez[r + 1][2];
      }
      bar_arrive(1, threads);
      if (AUX && t > 0) tile_record<R, JS>(s, A, tracked, p, own, r0, min(r0 + rows, ny - 1), n + t - 1);
      if (pts.state) {
        if (t > 0) {
          if (sizeof(T) == 4) pts.leave<R, JS>(s, lane);
          pts.record<T>(S, n + t - 1, lane);
        }
        pts.load_step(S, n + t, lane);
      }
      bar_sync(2, threads);
      get4(s.ez[0], warp > 0 ? e[(2 * warp - 1) * 32 + lane] : E.row_in[lane]);
      get4(s.ez[R + 1], warp < nw - 1 ? e[(2 * warp + 2) * 32 + lane] : E.row_in[32 + lane]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float z = E.col_in[col_at + r];
        s.ez[r + 1][0] = take_l ? z : s.ez[r + 1][0];
        s.ez[r + 1][3] = take_r ? z : s.ez[r + 1][3];
      }
      tile_step<R, JS, LOSSLESS, decltype(x)::value, decltype(y)::value, T, MED>(s, S, C, p, psi, tc, tr, rows, row0, kps, jzs, wt, lane, mat);
      if (pts.state) {
        pts.sources<R, JS, T>(s, S, lane);
        if (sizeof(T) == 2) pts.leave<R, JS>(s, lane);
      }
      tile_round<R, JS, T>(s);
    }
  };
  if (!work) {
    for (int t = 0; t < steps; ++t) {
      bar_arrive(1, threads);
      bar_sync(2, threads);
    }
    return;
  }
  if (!p.x) {
    if (!p.y) loop(No{}, No{});
    else loop(No{}, Yes{});
  } else {
    if (!p.y) loop(Yes{}, No{});
    else loop(Yes{}, Yes{});
  }
  if (AUX) tile_record<R, JS>(s, A, tracked, p, own, r0, min(r0 + rows, ny - 1), n + steps - 1);
  if (pts.state) {
    if (sizeof(T) == 4) pts.leave<R, JS>(s, lane);
    pts.record<T>(S, n + steps - 1, lane);
    pts.end(S, lane);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = j0 + r;
    if (j >= ny - 1) continue;
    float jv[4];
    if (JS) get4(jv, jzs[r * wt]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!(own >> q & 1)) continue;
      const int64_t o = (int64_t)j * pitch + p.i + q;
      Sto<T>::st1(field_ptr_t<T>(S, kEz, 1) + o, s.ez[r + 1][q]);
      Sto<T>::st1(field_ptr_t<T>(S, kHx, 1) + o, s.hx[r + 1][q]);
      Sto<T>::st1(field_ptr_t<T>(S, kHy, 1) + o, s.hy[r][q]);
      Sto<T>::st1(field_ptr_t<T>(S, kJz, 1) + o, JS ? jv[q] : s.jz[JS ? 0 : r][q]);
    }
  }
  tile_psi_store<R, false>(S, S.psi + S.psi_buf, p, psi, rows, row0, own, r0, min(r0 + rows, ny - 1));
}

template <int R, bool LOSSLESS, bool AUX, bool MED, class T>
__global__ void __launch_bounds__(all_warps(R) * 32, 1)
step_persist_tile_kernel(const __grid_constant__ DevShot S, const __grid_constant__ TileAux A,
                         const __grid_constant__ ResidentPlan G, int n_global, int steps,
                         uint64_t* link, int* err, unsigned long long wait_ns, int tag_add) {
  extern __shared__ float4 smem[];
  __shared__ int dead, slots;
  if (threadIdx.x == 0) dead = slots = 0;
  __syncthreads();
  const Waiter wait{&dead, err, wait_ns};
  resident_run<R, LOSSLESS, AUX, MED, T>(S, A, G, n_global - S.base_n, steps, link, wait, (uint32_t)tag_add, smem, &slots);
}

}  // namespace
}  // namespace fdtd2d

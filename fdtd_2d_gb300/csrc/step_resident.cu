// Many steps per launch with the whole shot on chip (uniform medium, grids
// whose cells fit the registers of the GPU's SMs).
//
// step_persist_tile_kernel<R>: one cooperative launch whose CTAs, one per SM,
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
// (L2-resident persistent kernel, two-step path): 256 x 192 1.67 (6.0), 512^2 1.77
// (6.1), 777 x 1301 2.81 (16.4), 1024^2 2.87 (13.0); the tile passes of
// step_tile.cu take 4.6 at 512^2 and 5.1 at 1024^2.
#include <algorithm>
#include <map>
#include <set>

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
  int kind, cell, idx;   // cell: its float in the warp's buffer of R rows
  float val;             // the step's source value
  double2 tw, acc;       // the step's DFT twiddle, the running sum
};
constexpr int kWarpPoints = 32;
__host__ __device__ constexpr int point_f4(int R) { return 2 * R * 32 + kWarpPoints * (int)sizeof(ResPoint) / 16; }

// The points of a warp.  A step's source values and twiddles are copied in
// from its start on (cp.async), the sums stay in shared memory for the whole
// launch, and the cells are reached through a buffer of the warp's rows in
// shared memory: a source is subtracted with every other cell's zero, which
// changes nothing, so no register is indexed by a point's position.  (Points
// read from global memory and cells found by selects took 0.4 us of a 512^2
// step; loops over a warp's points that touch its cells' registers slowed the
// whole step by up to 2x.)
struct ResPoints {
  float4* buf;
  int state;   // 0: no points; bits 0-5 their number, 6 sources, 7 detectors, 8 of them component ones
  static constexpr int kSrc = 64, kDet = 128, kComp = 256;
  template <int R>
  __device__ __forceinline__ ResPoint* points() const { return reinterpret_cast<ResPoint*>(buf + 2 * R * 32); }
  __device__ __forceinline__ int count() const { return state & 63; }

  template <int R>
  __device__ __forceinline__ void begin(const DevShot& S, int j0, int c0, int lo, int hi, float4* smem, int* slots, int lane) {
    state = 0;
    buf = smem;
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
        if (pass && in) {
          ResPoint& p = points<R>()[n + __popc(m & ((1u << lane) - 1))];
          p.kind = pt.y;
          p.cell = ((pt.w - j0) * 32 + (x >> 2)) * 4 + (x & 3);
          p.idx = pt.z;
          if (pt.y == kPointDetEz && S.dft) p.acc = S.dft[pt.z];
        }
        flags |= (__any_sync(kFull, in && pt.y == kPointSource) ? kSrc : 0) |
                 (__any_sync(kFull, in && pt.y != kPointSource) ? kDet : 0) |
                 (__any_sync(kFull, in && pt.y == kPointDetComp) ? kComp : 0);
        n += __popc(m);
      }
      if (n == 0) return;
      if (pass == 0) {
        int slot = 0;
        if (lane == 0) slot = atomicAdd(slots, 1);
        slot = __shfl_sync(kFull, slot, 0);
        buf = smem + slot * point_f4(R);
        state = n | flags;
        for (int r = 0; r < R; ++r) buf[r * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    __syncwarp();
  }
  template <int R>
  __device__ __forceinline__ void end(const DevShot& S, int lane) const {
    const ResPoint* at = points<R>();
    if (lane < count() && at[lane].kind == kPointDetEz && S.dft) S.dft[at[lane].idx] = at[lane].acc;
  }
  template <int R>
  __device__ __forceinline__ void load_step(const DevShot& S, int n, int lane) const {
    if (lane < count()) {
      ResPoint& p = points<R>()[lane];
      if (p.kind == kPointSource)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&p.val)),
                     "l"(S.src_val + (int64_t)n * S.n_src + p.idx));
      else if (S.dft)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&p.tw)), "l"(S.twiddle + n));
    }
  }
  // A step's sources, on the cells after their Ez update.
  template <int R, bool JS>
  __device__ __forceinline__ void sources(TileRegs<R, JS>& s, int lane) const {
    if (!(state & kSrc)) return;
    const ResPoint* at = points<R>();
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (lane < count() && at[lane].kind == kPointSource) reinterpret_cast<float*>(buf)[at[lane].cell] = at[lane].val;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float a[4];
      get4(a, buf[r * 32 + lane]);
#pragma unroll
      for (int k = 0; k < 4; ++k) s.ez[r + 1][k] = __fsub_rn(s.ez[r + 1][k], a[k]);
    }
    __syncwarp();
  }
  // Step n's detectors, on the state after it.
  template <int R, bool JS>
  __device__ __forceinline__ void detectors(const TileRegs<R, JS>& s, const DevShot& S, int n, int lane) const {
    if (!(state & kDet)) return;
    float4* out = buf + R * 32;
    const float* cells = reinterpret_cast<const float*>(out);
    ResPoint* at = points<R>();
    asm volatile("cp.async.wait_all;" ::: "memory");
    const int kind = lane < count() ? at[lane].kind : -1;
    float e = 0.f, hx = 0.f, hy = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) out[r * 32 + lane] = put4(s.ez[r + 1]);
    __syncwarp();
    if (kind > kPointSource) e = cells[at[lane].cell];
    __syncwarp();
    if (state & kComp) {
#pragma unroll
      for (int r = 0; r < R; ++r) out[r * 32 + lane] = put4(s.hx[r + 1]);
      __syncwarp();
      if (kind == kPointDetComp) hx = cells[at[lane].cell];
      __syncwarp();
#pragma unroll
      for (int r = 0; r < R; ++r) out[r * 32 + lane] = put4(s.hy[r]);
      __syncwarp();
      if (kind == kPointDetComp) hy = cells[at[lane].cell];
    }
    if (kind == kPointDetEz) {
      ResPoint& p = at[lane];
      if (S.record) S.trace[(int64_t)(n - 1) * S.n_det + p.idx] = e;
      if (S.dft) {
        p.acc.x = fma((double)e, p.tw.x, p.acc.x);
        p.acc.y = fma(-(double)e, p.tw.y, p.acc.y);
      }
    } else if (kind == kPointDetComp && S.record) {
      float* dst = S.ctrace + ((int64_t)(n - 1) * S.n_comp + at[lane].idx) * 3;
      dst[0] = e;
      dst[1] = hx;
      dst[2] = hy;
    }
    __syncwarp();
  }
};

template <int R, bool LOSSLESS, bool AUX, bool MED>
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
  rest += G.point_warps * point_f4(R);
  float* tc = reinterpret_cast<float*>(rest);
  float* tr = tc + kTcRows * kTileCols;
  const Coef<float> C(S);
  tile_tables<float>(S, C, tc, tr, c0, r0, rows, tid, threads);
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
    const float* f[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) f[a] = field_ptr(S, a, 0) + p.i;
#pragma unroll
    for (int r = -1; r <= R; ++r) {
      const int j = j0 + r;
      const bool rin = work && j >= 0 && j < ny;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = p.i + q;
        const bool in = rin && c >= 0 && c < nx;
        const int64_t o = (int64_t)j * pitch + q;
        s.ez[r + 1][q] = in ? __ldcg(f[kEz] + o) : 0.f;
        if (r < R) s.hx[r + 1 < R + 1 ? r + 1 : 0][q] = in ? __ldcg(f[kHx] + o) : 0.f;
        if (r >= 0 && r < R) {
          s.hy[r >= 0 && r < R ? r : 0][q] = in ? __ldcg(f[kHy] + o) : 0.f;
          if (!JS) s.jz[!JS && r >= 0 && r < R ? r : 0][q] = in ? __ldcg(f[kJz] + o) : 0.f;
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
        kv[q] = !MED && S.kp && in ? __ldg(S.kp + (int64_t)j * pitch + c) : 0.f;
        if (JS) jv[q] = in ? __ldcg(f[kJz] + (int64_t)j * pitch + q) : 0.f;
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
        if (t > 0) pts.detectors<R, JS>(s, S, n + t - 1, lane);
        pts.load_step<R>(S, n + t, lane);
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
      tile_step<R, JS, LOSSLESS, decltype(x)::value, decltype(y)::value, float, MED>(s, S, C, p, psi, tc, tr, rows, row0, kps, jzs, wt, lane, mat);
      if (pts.state) pts.sources<R, JS>(s, lane);
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
    pts.detectors<R, JS>(s, S, n + steps - 1, lane);
    pts.end<R>(S, lane);
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
      field_ptr(S, kEz, 1)[o] = s.ez[r + 1][q];
      field_ptr(S, kHx, 1)[o] = s.hx[r + 1][q];
      field_ptr(S, kHy, 1)[o] = s.hy[r][q];
      field_ptr(S, kJz, 1)[o] = JS ? jv[q] : s.jz[JS ? 0 : r][q];
    }
  }
  tile_psi_store<R, false>(S, S.psi + S.psi_buf, p, psi, rows, row0, own, r0, min(r0 + rows, ny - 1));
}

template <int R, bool LOSSLESS, bool AUX, bool MED>
__global__ void __launch_bounds__(all_warps(R) * 32, 1)
step_persist_tile_kernel(const __grid_constant__ DevShot S, const __grid_constant__ TileAux A,
                         const __grid_constant__ ResidentPlan G, int n_global, int steps,
                         uint64_t* link, int* err, unsigned long long wait_ns, int tag_add) {
  extern __shared__ float4 smem[];
  __shared__ int dead, slots;
  if (threadIdx.x == 0) dead = slots = 0;
  __syncthreads();
  const Waiter wait{&dead, err, wait_ns};
  resident_run<R, LOSSLESS, AUX, MED>(S, A, G, n_global - S.base_n, steps, link, wait, (uint32_t)tag_add, smem, &slots);
}

template <int R, bool AUX>
const void* resident_kernel(const DevShot& s) {
  return s.ca == 1.f && s.da == 1.f ? (const void*)step_persist_tile_kernel<R, true, AUX, false>
                                    : (const void*)step_persist_tile_kernel<R, false, AUX, false>;
}
template <int R>
const void* resident_kernel(const DevShot& s, bool aux) {
  if (s.mat_e) return (const void*)step_persist_tile_kernel<R, false, true, true>;   // (one form: such shots have a tracker)
  return aux ? resident_kernel<R, true>(s) : resident_kernel<R, false>(s);
}
const void* resident_kernel(int R, const DevShot& s, bool aux) {
  switch (R) {
    case 8: return resident_kernel<8>(s, aux);
    case 6: return resident_kernel<6>(s, aux);
    case 4: return resident_kernel<4>(s, aux);
    default: return resident_kernel<2>(s, aux);
  }
}

}  // namespace

// Rows per warp, tried in this order: the fewest that fit, for a step's time is
// a warp's chain of its rows.  us per step on GB300 with 2 / 4 / 6 / 8 rows: 512^2
// 1.77 / 2.11 / 2.49 / 3.26, 900^2 - / 2.50 / 2.65 / 3.26, 1024^2 - / - / 2.87 /
// 3.29; 500 x 3000 fits 8 rows only, 4.16.
const std::vector<int>& resident_rows() {
  static const std::vector<int> rows = {2, 4, 6, 8};
  return rows;
}

// The split of a shot over the device's SMs at R rows per warp; false when it
// does not fit.
bool resident_plan(const DevShot& s, const std::vector<int3>& points, int R, int device, ResidentPlan* out) {
  int sms = 0, most = 0, coop = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  if (!coop || s.store != 0) return false;
  ResidentPlan g{};
  g.R = R;
  g.nb = (s.nx + kOwn - 1) / kOwn;
  if (g.nb > sms) return false;
  // the narrowest width 4 m + 2 that covers the grid in nb bands
  const int need = (s.nx + g.nb - 1) / g.nb;
  g.w = std::max(6, (need + 1) / 4 * 4 + 2);
  if (g.w < need) g.w += 4;
  if (g.w > kOwn) return false;
  g.nb = (s.nx + g.w - 1) / g.w;
  g.groups = (s.ny - 1 + R - 1) / R;
  if (g.groups > 65535 || (int64_t)g.nb * g.groups > (int64_t)sms * max_warps(R)) return false;
  // The cuts: for each number of strips of the inner bands, as many as are
  // left for the two edge bands; the split whose dearest strip is cheapest.
  std::vector<float> y_cost(g.groups);
  double cum[2] = {0, 0};
  for (int gr = 0; gr < g.groups; ++gr) {
    y_cost[gr] = tile_y(s, gr * R, R) ? 0.6f : 0.f;
    cum[0] += 1.8 + y_cost[gr];
    cum[1] += 1.0 + y_cost[gr];
  }
  auto cost = [&](int t, int gr) { return (t == 0 ? 1.8 : 1.0) + y_cost[gr]; };
  auto cut = [&](int t, int ns, uint16_t* start, double* dearest) {
    // strip k ends where the cost so far reaches (k + 1) / ns of the whole
    double sum = 0, strip = 0;
    int k = 0;
    *dearest = 0;
    start[0] = 0;
    for (int gr = 0; gr < g.groups; ++gr) {
      const double w = cost(t, gr);
      const int left = g.groups - gr, open = ns - k;   // strips not closed, this one included
      const int have = gr - start[k];
      const bool must = have >= max_warps(R) || (have > 0 && left < open);
      if (k < ns - 1 && have > 0 && (must || (left >= open - 1 && sum + 0.5 * w > cum[t] * (k + 1) / ns))) {
        *dearest = std::max(*dearest, strip);
        start[++k] = (uint16_t)gr;
        strip = 0;
      }
      sum += w;
      strip += w;
    }
    *dearest = std::max(*dearest, strip);
    start[k + 1] = (uint16_t)g.groups;
    auto fits = [&] {
      for (int q = 0; q < ns; ++q)
        if (start[q + 1] <= start[q] || start[q + 1] - start[q] > max_warps(R)) return false;
      return true;
    };
    if (k == ns - 1 && fits()) return true;
    // no room to weigh: strips of equal rows
    for (int q = 0; q <= ns; ++q) start[q] = (uint16_t)((int64_t)g.groups * q / ns);
    *dearest = 0;
    for (int q = 0; q < ns; ++q) {
      strip = 0;
      for (int gr = start[q]; gr < start[q + 1]; ++gr) strip += cost(t, gr);
      *dearest = std::max(*dearest, strip);
    }
    return fits();
  };
  const int edge_bands = std::min(g.nb, 2), inner = g.nb - edge_bands;
  double best = 1e30;
  ResidentPlan c = g;
  // (an inner band never has more strips than an edge band: its rows are cheaper)
  for (int ni = inner ? (g.groups + max_warps(R) - 1) / max_warps(R) : 0; ni <= (inner ? sms / g.nb : 0); ++ni) {
    c.ns[1] = std::min(ni, g.groups);
    c.ns[0] = std::min({(sms - inner * ni) / edge_bands, g.groups, kMaxStrips});
    if (ni > g.groups || ni > kMaxStrips || c.ns[0] < 1) continue;
    double d0 = 0, d1 = 0;
    if (!cut(0, c.ns[0], c.start[0], &d0) || (inner && !cut(1, c.ns[1], c.start[1], &d1))) continue;
    if (std::max(d0, d1) < best) {
      best = std::max(d0, d1);
      g = c;
    }
  }
  if (best > 1e29) return false;
  // the largest strip of each kind, for the launch's shared memory
  int f4 = 0;
  for (int t = 0; t < (inner ? 2 : 1); ++t) {
    int nxl = 0;
    for (int b = 0; b < g.nb; ++b)
      if ((b == 0 || b == g.nb - 1) == (t == 0)) nxl = std::max(nxl, strip_lanes(s, b * g.w - 1));
    for (int k = 0; k < g.ns[t]; ++k) {
      const int n = g.start[t][k + 1] - g.start[t][k];
      g.nw = std::max(g.nw, n);
      f4 = std::max(f4, tile_table_f4(n * R) + tile_psi_x(n * R, nxl) + y_warps(s, g.start[t][k] * R, n, R) * (2 * R + 1) * 32);
    }
  }
  // the warps with points: at most kWarpPoints each, no two sources in a cell
  std::map<std::pair<int, int>, int> per_warp;    // (band, group) -> points
  std::map<std::pair<int, int>, int> per_cta;     // (band, strip) -> warps with points
  std::set<std::pair<int, int>> cells;
  for (const int3& q : points) {
    const std::pair<int, int> w(q.x / g.w, q.y / R);
    if (++per_warp[w] > kWarpPoints || (q.z == kPointSource && !cells.insert({q.x, q.y}).second)) return false;
    if (per_warp[w] == 1) {
      const int t = w.first == 0 || w.first == g.nb - 1 ? 0 : 1;
      const int strip = (int)(std::upper_bound(g.start[t], g.start[t] + g.ns[t] + 1, (uint16_t)w.second) - g.start[t]);
      g.point_warps = std::max(g.point_warps, ++per_cta[{w.first, strip}]);
    }
  }
  f4 += g.point_warps * point_f4(R);
  f4 += 4 * g.nw * 32 + edge_f4(g.nw * R) + (jz_shared(R) ? 2 : 1) * R * g.nw * 32;
  if (s.mat_e) f4 += g.nw * 32 + 256 + 128;   // the words of the rows below, the tables
  g.smem = f4 * 16;
  if (g.smem + 64 > most) return false;
  g.link_words = 2 * ((int64_t)(edge_bands * g.ns[0] + inner * g.ns[1]) * 2 * kTileCols + 2 * (int64_t)g.nb * g.groups * R);
  if (g.link_words >= (int64_t)1 << 31) return false;
  *out = g;
  return true;
}

int resident_ctas(const ResidentPlan& p) {
  const int edges = std::min(p.nb, 2);
  return edges * p.ns[0] + (p.nb - edges) * p.ns[1];
}

cudaError_t launch_resident(const DevShot& shot, const ResidentPlan& plan, int n_global, int steps, const TileAux* aux,
                            uint64_t* link, int* err, unsigned long long wait_ns, int tag_add, cudaStream_t stream) {
  const void* fn = resident_kernel(plan.R, shot, aux != nullptr);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, plan.smem);
  // tags count from 1 in every launch: clear the words of earlier ones
  if (e == cudaSuccess) e = cudaMemsetAsync(link, 0, (size_t)plan.link_words * sizeof(uint64_t), stream);
  if (e != cudaSuccess) return e;
  DevShot s = shot;
  ResidentPlan g = plan;
  if (wait_ns == 0) wait_ns = kWaitNs;
  TileAux a = aux ? *aux : TileAux{};
  void* args[] = {&s, &a, &g, &n_global, &steps, &link, &err, &wait_ns, &tag_add};
  return cudaLaunchCooperativeKernel(fn, dim3(resident_ctas(plan)), dim3((plan.nw + 1) * 32), args, (size_t)plan.smem, stream);
}

}  // namespace fdtd2d

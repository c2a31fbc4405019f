// The on-chip kernel (step_resident.cuh) in FP32: its instances, the split of a
// shot over the SMs and the launch.
#include <algorithm>
#include <map>
#include <set>

#include "step_resident.cuh"

namespace fdtd2d {

namespace {

template <int R, bool AUX>
const void* resident_kernel(const DevShot& s) {
  return s.ca == 1.f && s.da == 1.f ? (const void*)step_persist_tile_kernel<R, true, AUX, false, float>
                                    : (const void*)step_persist_tile_kernel<R, false, AUX, false, float>;
}
template <int R>
const void* resident_kernel(const DevShot& s, bool aux) {
  if (s.mat_e) return (const void*)step_persist_tile_kernel<R, false, true, true, float>;   // (one form: such shots have a tracker)
  return aux ? resident_kernel<R, true>(s) : resident_kernel<R, false>(s);
}
const void* resident_kernel(int R, const DevShot& s, bool aux) {
  if (s.store != 0) return resident_kernel16(R, s.store);
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
// 1.77 / 2.11 / 2.49 / 3.26, 900^2 - / 2.37 / 2.65 / 3.26, 1024^2 - / - / 2.90 /
// 3.29; 500 x 3000 fits 8 rows only, 3.80.
// 16-bit fields take at most 6 (1024^2 3.4 us, the tile passes 4.6): what 8 rows
// spill is no longer in the L1 cache, 900 x 1600 5.6 against 4.9 in passes, 1200^2
// 4.9 on both.
const std::vector<int>& resident_rows() {
  static const std::vector<int> rows = {2, 4, 6, 8};
  return rows;
}

constexpr int kMost16 = 6;

// The split of a shot over the device's SMs at R rows per warp; false when it
// does not fit.
bool resident_plan(const DevShot& s, const std::vector<int3>& points, int R, int device, ResidentPlan* out) {
  int sms = 0, most = 0, coop = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  if (!coop || (s.store != 0 && R > kMost16)) return false;
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
  f4 += g.point_warps * kPointF4;
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

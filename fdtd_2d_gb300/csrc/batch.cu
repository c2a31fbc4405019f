// Batched and continuous stepping of many shots on one GPU (fdtd2d_batch_*).
//
// The reference runs one shot per process (global state, FDTD_2D_Full/
// kernel.cu:1928-2818).  A batch owns many shots, each a full fdtd2d_ctx
// (fields, CPML state, tables, traces and DFT accumulators resident in HBM),
// and advances all of them with one launch per pass of up to four time steps
// (step_tile.cu's batch kernel): the register tiles of every unfinished shot in
// one grid, each shot at its own step n = global step - its admission step, so
// shots admitted at different times advance together (continuous batching).
// Admission is by a device-memory budget.
//
// Host-side state changes (admit, finish, remove) take effect between passes:
// the tile list is rebuilt on the host and uploaded in the order of the batch's
// stream before the next pass.  Two lists can be on their way: the host waits for
// the device only when a third change follows while the first one's list is still
// behind queued passes.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <vector>

#include "ctx.h"

using namespace fdtd2d;

namespace {

constexpr int kMaxShots = 512;     // descriptor slots per batch

struct Member {
  fdtd2d_ctx* ctx = nullptr;
  int64_t bytes = 0;
  int32_t base = 0;     // global steps issued before its first step
  bool live = false;
  bool done = false;    // all its steps issued
  // its register tiles (a member of the batch kernel) and the passes issued
  std::vector<int4> tiles;
  int32_t passes = 0;
  // A solo member is a full single shot on its own streams, stepped by
  // fdtd2d_run from the batch's run calls; `ev` holds the events recorded after its recent run calls on
  // its stream, oldest first.
  bool solo = false;
  std::vector<cudaEvent_t> ev;
  int64_t seq = 0;      // admission order
};

// Solo members stepped at a time (the oldest admitted first; the others
// wait): a few chains of passes keep the GPU busy, and every extra one only
// adds streams and shares the device among more shots, which delays each.
// FDTD2D_BATCH_SOLO_ACTIVE overrides it.
int solo_active() {
  const char* v = std::getenv("FDTD2D_BATCH_SOLO_ACTIVE");
  const int k = v ? std::atoi(v) : 8;
  return k > 0 ? k : 8;
}

// Grids of at least this many cells (2^21, about 1448^2) join a batch as
// solo members (their own launches fill the GPU); smaller ones
// share the batch kernel.  FDTD2D_BATCH_SOLO_CELLS overrides it (0: none
// solo).
int64_t solo_cells() {
  const char* v = std::getenv("FDTD2D_BATCH_SOLO_CELLS");
  return v ? std::atoll(v) : (int64_t)1 << 21;
}

}  // namespace

struct fdtd2d_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  int64_t budget = 0, used = 0;
  std::vector<Member> m;
  std::vector<DevShot> h_shots;        // host copies of the slots' descriptors
  DevShot* d_shots = nullptr;          // [kMaxShots]
  int4* d_tiles = nullptr;
  int tile_cap = 0, n_tiles = 0;
  // the list's host copies, pinned: two, so that one can be filled while the
  // stream still copies from the other (its event marks that copy)
  struct Staging {
    int4* p = nullptr;
    int cap = 0;
    cudaEvent_t ev = nullptr;
  } staging[2];
  int next_staging = 0;
  size_t smem = 0;
  bool lossless = true;                // CA = DA = 1 in every member
  int32_t g = 0;                       // global steps issued
  int32_t passes = 0;                  // and passes
  bool dirty = true;
  int64_t launches = 0;
  int last_cuda = 0;
  char name[64] = {0};
  int64_t admitted = 0;                // admissions so far (Member::seq)
};

namespace {

int fail(fdtd2d_batch* b, cudaError_t e) {
  if (b) b->last_cuda = (int)e;
  return e == cudaErrorMemoryAllocation ? FDTD2D_ERR_NOMEM : FDTD2D_ERR_CUDA;
}

// The tile list of every live shot with steps left, tiles with CPML work (the
// slower ones) of all shots first, uploaded in the stream's order.
int upload_tiles(fdtd2d_batch* b) {
  int n = 0;
  b->smem = 0;
  b->lossless = true;
  for (int k = 0; k < (int)b->m.size(); ++k) {
    const Member& x = b->m[k];
    if (!x.live || x.done || x.solo) continue;
    const DevShot& s = b->h_shots[k];
    n += (int)x.tiles.size();
    b->smem = std::max(b->smem, tile_smem(s, kBatchShape));
    b->lossless = b->lossless && s.ca == 1.f && s.da == 1.f;
  }
  cudaError_t e = cudaSuccess;
  fdtd2d_batch::Staging& st = b->staging[b->next_staging];
  if (!st.ev) e = cudaEventCreateWithFlags(&st.ev, cudaEventDisableTiming);
  else e = cudaEventSynchronize(st.ev);   // the list before the last one has been copied
  if (e == cudaSuccess && n > st.cap) {
    if (st.p) cudaFreeHost(st.p);
    st.p = nullptr;
    st.cap = 0;
    const int cap = std::max(n * 2, 4096);
    e = cudaHostAlloc(&st.p, (size_t)cap * sizeof(int4), cudaHostAllocDefault);
    if (e == cudaSuccess) st.cap = cap;
  }
  if (e == cudaSuccess && n > b->tile_cap) {
    // (stream-ordered: the passes issued before still read the old list)
    if (b->d_tiles) cudaFreeAsync(b->d_tiles, b->stream);
    b->d_tiles = nullptr;
    b->tile_cap = 0;
    const int cap = std::max(n * 2, 4096);
    e = cudaMallocAsync(&b->d_tiles, (size_t)cap * sizeof(int4), b->stream);
    if (e == cudaSuccess) b->tile_cap = cap;
  }
  if (e != cudaSuccess) return fail(b, e);
  int at = 0;
  for (int plain = 0; plain < 2; ++plain)
    for (int k = 0; k < (int)b->m.size(); ++k) {
      const Member& x = b->m[k];
      if (!x.live || x.done || x.solo) continue;
      for (const int4& t : x.tiles)
        if (((t.x & kTilePlain) != 0) == (plain != 0)) st.p[at++] = make_int4(t.x | k << kTileSlot, t.y, t.z, t.w);
    }
  if (n) e = cudaMemcpyAsync(b->d_tiles, st.p, (size_t)n * sizeof(int4), cudaMemcpyHostToDevice, b->stream);
  if (e == cudaSuccess) e = cudaEventRecord(st.ev, b->stream);
  if (e != cudaSuccess) return fail(b, e);
  b->n_tiles = n;
  b->next_staging ^= 1;
  b->dirty = false;
  return FDTD2D_OK;
}

// A member's host descriptor after a pass: the state after step n is in slot
// n & 1 for the readers, whatever buffer its passes have left it in (slot
// `passes & 1` of the descriptor it was admitted with, which the kernel reads).
void settle(Member& x, const DevShot& s) {
  DevShot& h = x.ctx->h;
  const int at = x.passes & 1, slot = x.ctx->step & 1;
  h.fb[slot] = s.fb[at];
  h.fb[slot ^ 1] = s.fb[at ^ 1];
  h.psi = at == slot ? s.psi : s.psi + s.psi_buf;
  h.psi_buf = at == slot ? s.psi_buf : -s.psi_buf;
}

// Room a solo member must find beside its device bytes: the two more field buffers
// of the two-step path, where a variable sends it there.
int64_t solo_extra(const fdtd2d_setup* s) {
  return tiles_off() ? 2 * (int64_t)buffer_floats(s->nx, s->ny) * 4 * store_bytes(s->storage) : 0;
}

int add_solo(fdtd2d_batch* b, const fdtd2d_setup* s, int64_t bytes, int32_t* shot) {
  int slot = -1;
  for (int k = 0; k < (int)b->m.size(); ++k)
    if (!b->m[k].live) { slot = k; break; }
  if (slot < 0) {
    if ((int)b->m.size() >= kMaxShots) return FDTD2D_ERR_BUDGET;
    b->m.emplace_back();
    slot = (int)b->m.size() - 1;
  }
  // Its own streams; its kernel choice is timed at create while the batch
  // has no device work in flight.  Timing trials run beside other shots'
  // kernels measure nothing useful, and on a GB300 with some 150 shots in
  // flight a trial kernel's bounded wait ran out; such an admission takes
  // the class's stored choice or the default one.
  bool busy = cudaStreamQuery(b->stream) == cudaErrorNotReady;
  for (const Member& m : b->m)
    if (m.live && m.solo && !busy)
      busy = cudaStreamQuery(m.ctx->stream) == cudaErrorNotReady ||
             (m.ctx->side && cudaStreamQuery(m.ctx->side) == cudaErrorNotReady);
  cudaGetLastError();
  fdtd2d_ctx* c = nullptr;
  const int rc = create_ctx(s, b->device, false, &c, true, busy);
  if (rc) return rc;
  // the bytes it holds: two more field buffers on the two-step path
  if (c->tb) bytes += 2 * c->h.cells * 4 * store_bytes(c->h.store);
  Member& x = b->m[slot];
  x.ctx = c;
  x.bytes = bytes;
  x.base = b->g;
  x.live = true;
  x.done = c->n_steps <= 0;
  x.solo = true;
  x.seq = b->admitted++;
  b->used += bytes;
  *shot = slot;
  return FDTD2D_OK;
}

// Issue up to n more steps of the solo_active() oldest unfinished solo
// members on their own streams (the host does not wait), keeping at most two
// run calls of each in flight.
int run_solo(fdtd2d_batch* b, int32_t n) {
  // the solo_active() oldest unfinished solo members
  std::vector<std::pair<int64_t, int>> order;
  for (int k = 0; k < (int)b->m.size(); ++k) {
    const Member& x = b->m[k];
    if (x.live && x.solo && !x.done) order.push_back({x.seq, k});
  }
  std::sort(order.begin(), order.end());
  if ((int)order.size() > solo_active()) order.resize(solo_active());
  for (const auto& o : order) {
    Member& x = b->m[o.second];
    fdtd2d_ctx* c = x.ctx;
    while (x.ev.size() >= 2) {
      const cudaError_t e = cudaEventSynchronize(x.ev.front());
      if (e != cudaSuccess) return fail(b, e);
      cudaEventDestroy(x.ev.front());
      x.ev.erase(x.ev.begin());
    }
    const int32_t last = std::min(c->n_steps, c->step + n);
    const int64_t l0 = c->launches;
    const int rc = fdtd2d_run(c, c->step + 1, last);
    if (rc) {
      b->last_cuda = c->last_cuda;
      return rc;
    }
    b->launches += c->launches - l0;
    cudaEvent_t e = nullptr;
    cudaError_t ce = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    if (ce == cudaSuccess) ce = cudaEventRecord(e, c->stream);
    if (ce != cudaSuccess) return fail(b, ce);
    x.ev.push_back(e);
    if (c->step >= c->n_steps) x.done = true;
  }
  return FDTD2D_OK;
}

// A solo member whose steps have all been issued and have completed.
bool solo_complete(const Member& x) {
  return x.solo && x.done && (x.ev.empty() || cudaEventQuery(x.ev.back()) == cudaSuccess);
}

void release_events(Member& x) {
  for (cudaEvent_t e : x.ev) cudaEventDestroy(e);
  x.ev.clear();
}

}  // namespace

extern "C" {

int fdtd2d_batch_create(int device, int64_t hbm_budget_bytes, fdtd2d_batch** out) {
  if (!out) return FDTD2D_ERR_INVALID;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return FDTD2D_ERR_NODEVICE;
  if (device < 0 || device >= ndev) return FDTD2D_ERR_INVALID;
  fdtd2d_batch* b = new (std::nothrow) fdtd2d_batch();
  if (!b) return FDTD2D_ERR_NOMEM;
  b->device = device;
  cudaSetDevice(device);
  if (hbm_budget_bytes <= 0) {
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    hbm_budget_bytes = (int64_t)(free_b * 0.9);
  }
  b->budget = hbm_budget_bytes;
  // host descriptors first: a failure here leaves no device resource behind
  try {
    b->h_shots.resize(kMaxShots);
  } catch (...) {
    delete b;
    return FDTD2D_ERR_NOMEM;
  }
  std::memset(b->h_shots.data(), 0, kMaxShots * sizeof(DevShot));
  cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&b->d_shots, kMaxShots * sizeof(DevShot));
  if (e != cudaSuccess) {
    fdtd2d_batch_destroy(b);
    return e == cudaErrorMemoryAllocation ? FDTD2D_ERR_NOMEM : FDTD2D_ERR_CUDA;
  }
  *out = b;
  return FDTD2D_OK;
}

static int fdtd2d_batch_add_body(fdtd2d_batch* b, const fdtd2d_setup* s, int32_t* shot);

// The entry point: its body, below, runs behind abi_guard.
int fdtd2d_batch_add(fdtd2d_batch* b, const fdtd2d_setup* s, int32_t* shot) {
  return abi_guard([&] { return fdtd2d_batch_add_body(b, s, shot); });
}

static int fdtd2d_batch_add_body(fdtd2d_batch* b, const fdtd2d_setup* s, int32_t* shot) {
  if (!b || !s || !shot) return FDTD2D_ERR_INVALID;
  *shot = -1;
  if (s->medium != FDTD2D_MEDIUM_UNIFORM || s->npml > tma_max_pml() || s->n_rc > 0 || s->line_n > 0)
    return FDTD2D_ERR_INVALID;
  const int64_t bytes = fdtd2d_device_bytes(s);
  if (bytes < 0) return FDTD2D_ERR_INVALID;
  if (b->used + bytes > b->budget) return FDTD2D_ERR_BUDGET;
  // A large grid goes solo.  The batch kernel steps FP32 fields only, so a shot
  // with 16-bit storage is a solo member whatever its size (the single-shot
  // path, 16-bit forms included).
  const int64_t cells = (int64_t)s->nx * s->ny;
  const int64_t sc = solo_cells();
  const bool fits2 = b->used + bytes + solo_extra(s) <= b->budget;
  if (s->storage != FDTD2D_STORE_F32) return fits2 ? add_solo(b, s, bytes, shot) : FDTD2D_ERR_BUDGET;
  if (sc > 0 && cells >= sc && fits2) return add_solo(b, s, bytes, shot);
  int slot = -1;
  for (int k = 0; k < (int)b->m.size(); ++k)
    if (!b->m[k].live) { slot = k; break; }
  if (slot < 0) {
    if ((int)b->m.size() >= kMaxShots) return FDTD2D_ERR_BUDGET;
    b->m.emplace_back();
    slot = (int)b->m.size() - 1;
  }
  fdtd2d_ctx* c = nullptr;
  const int rc = create_ctx(s, b->device, true, &c);   // uploads on its own stream
  if (rc) return rc;
  adopt_ctx(c, b->stream);
  c->h.base_n = b->g;
  c->h.base_pass = b->passes;
  // nothing of the batch's changes before all that can fail has been done
  Member& x = b->m[slot];
  cudaError_t e = cudaSuccess;
  try {
    if (c->fail_here()) throw std::bad_alloc();
    x.tiles = make_tiles(c->h, kBatchShape, c->points);
    b->h_shots[slot] = c->h;
    cudaSetDevice(b->device);
    e = cudaMemcpyAsync(b->d_shots + slot, &b->h_shots[slot], sizeof(DevShot), cudaMemcpyHostToDevice, b->stream);
  } catch (const std::bad_alloc&) {
    e = cudaErrorMemoryAllocation;
  }
  if (e != cudaSuccess) {
    fdtd2d_destroy(c);
    return fail(b, e);
  }
  x.ctx = c;
  x.bytes = bytes;
  x.base = b->g;
  x.live = true;
  x.done = false;
  x.passes = 0;
  b->used += bytes;
  b->dirty = true;
  *shot = slot;
  return FDTD2D_OK;
}

static int fdtd2d_batch_run_body(fdtd2d_batch* b, int32_t n_steps);

// The entry point: its body, below, runs behind abi_guard.
int fdtd2d_batch_run(fdtd2d_batch* b, int32_t n_steps) {
  return abi_guard([&] { return fdtd2d_batch_run_body(b, n_steps); });
}

static int fdtd2d_batch_run_body(fdtd2d_batch* b, int32_t n_steps) {
  if (!b || n_steps < 0) return FDTD2D_ERR_INVALID;
  cudaSetDevice(b->device);
  if (n_steps > 0) {
    const int rc = run_solo(b, n_steps);
    if (rc) return rc;
  }
  while (n_steps > 0) {
    bool any = false;
    for (const Member& x : b->m) any = any || (x.live && !x.done && !x.solo);
    if (!any) return FDTD2D_OK;
    if (b->dirty) {
      const int rc = upload_tiles(b);
      if (rc) return rc;
    }
    const int K = std::min<int>(n_steps, kTileSteps);
    const cudaError_t e = launch_batch_tile(b->lossless, b->d_shots, b->d_tiles, b->n_tiles, b->smem, b->g, K,
                                            b->passes, b->stream);
    if (e != cudaSuccess) return fail(b, e);
    b->g += K;
    ++b->passes;
    ++b->launches;
    n_steps -= K;
    for (int k = 0; k < (int)b->m.size(); ++k) {
      Member& x = b->m[k];
      if (!x.live || x.solo || x.done) continue;
      x.ctx->step = std::min(x.ctx->n_steps, b->g - x.base);
      ++x.passes;
      settle(x, b->h_shots[k]);
      if (x.ctx->step >= x.ctx->n_steps) {
        x.done = true;
        b->dirty = true;
      }
    }
  }
  return FDTD2D_OK;
}

int fdtd2d_batch_synchronize(fdtd2d_batch* b) {
  if (!b) return FDTD2D_ERR_INVALID;
  cudaSetDevice(b->device);
  for (Member& x : b->m)
    if (x.live && x.solo) {
      const int rc = fdtd2d_synchronize(x.ctx);
      if (rc) return rc;
    }
  const cudaError_t e = cudaStreamSynchronize(b->stream);
  return e == cudaSuccess ? FDTD2D_OK : fail(b, e);
}

fdtd2d_ctx* fdtd2d_batch_shot(fdtd2d_batch* b, int32_t shot) {
  if (!b || shot < 0 || shot >= (int)b->m.size() || !b->m[shot].live) return nullptr;
  return b->m[shot].ctx;
}

int32_t fdtd2d_batch_shot_step(const fdtd2d_batch* b, int32_t shot) {
  if (!b || shot < 0 || shot >= (int)b->m.size() || !b->m[shot].live) return -1;
  return b->m[shot].ctx->step;
}

int fdtd2d_batch_remove(fdtd2d_batch* b, int32_t shot) {
  if (!b || shot < 0 || shot >= (int)b->m.size() || !b->m[shot].live) return FDTD2D_ERR_INVALID;
  cudaSetDevice(b->device);
  Member& x = b->m[shot];
  fdtd2d_destroy(x.ctx);   // memory released behind the queued kernels (a solo shot waits for its own)
  release_events(x);
  b->used -= x.bytes;
  x = Member();
  b->dirty = true;
  return FDTD2D_OK;
}

int64_t fdtd2d_batch_free_bytes(const fdtd2d_batch* b) { return b ? b->budget - b->used : -1; }

int64_t fdtd2d_batch_launch_count(const fdtd2d_batch* b) { return b ? b->launches : -1; }

const char* fdtd2d_batch_kernel_name(const fdtd2d_batch* b) {
  if (!b) return "";
  std::snprintf(const_cast<char*>(b->name), sizeof b->name, "step_tma_batch_kernel<tile,%d>", tile_shape_rows(kBatchShape));
  return b->name;
}

int fdtd2d_batch_destroy(fdtd2d_batch* b) {
  if (!b) return FDTD2D_ERR_INVALID;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (Member& x : b->m)
    if (x.live) {
      fdtd2d_destroy(x.ctx);
      release_events(x);
    }
  for (auto& st : b->staging) {
    if (st.ev) cudaEventDestroy(st.ev);
    if (st.p) cudaFreeHost(st.p);
  }
  if (b->d_tiles) cudaFreeAsync(b->d_tiles, b->stream);
  if (b->d_shots) cudaFree(b->d_shots);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return FDTD2D_OK;
}

}  // extern "C"

// ---- Serving loop -----------------------------------------------------------
//
// A request loop on top of a batch: shots are queued as they arrive, admitted
// in arrival order while they fit the device-memory budget, stepped together
// in blocks, and retired as soon as the block that issued their last step has
// completed on the GPU (a CUDA event per block; no device-wide wait): their
// DFT accumulators and Ez traces are copied out and their memory is released
// behind the queued kernels.  The caller drives it with fdtd2d_server_step and
// collects results with fdtd2d_server_pop.

namespace {

struct Queued {
  const fdtd2d_setup* s;
  int64_t tag;
};
struct Running {
  int32_t slot;
  int64_t tag;
  int32_t last_g;   // global step that completes the shot
};
struct Finished {
  int64_t tag;
  int32_t n_det, n_steps;
  std::vector<double> dft;    // re, im per detector
  std::vector<float> trace;   // [n_steps][n_det] Ez samples
};

}  // namespace

struct fdtd2d_server {
  fdtd2d_batch* b = nullptr;
  int32_t block = 64;
  std::vector<Queued> queue;            // FIFO (front = index 0)
  std::vector<Running> running;
  std::vector<Finished> finished;       // FIFO
  std::vector<std::pair<int32_t, cudaEvent_t>> blocks;   // (global step after the block, event)
  std::vector<cudaEvent_t> spare;
  int32_t g_complete = 0;               // global steps known complete on the GPU
};

namespace {

cudaEvent_t take_event(fdtd2d_server* s) {
  if (!s->spare.empty()) {
    cudaEvent_t e = s->spare.back();
    s->spare.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  return e;
}

// Retire every running shot whose last step has completed.
int retire(fdtd2d_server* s, int* n_done) {
  fdtd2d_batch* b = s->b;
  size_t k = 0;
  for (; k < s->blocks.size(); ++k) {
    if (cudaEventQuery(s->blocks[k].second) != cudaSuccess) break;
    s->g_complete = std::max(s->g_complete, s->blocks[k].first);
    s->spare.push_back(s->blocks[k].second);
  }
  s->blocks.erase(s->blocks.begin(), s->blocks.begin() + k);
  for (size_t r = 0; r < s->running.size();) {
    const Running x = s->running[r];
    const Member& mem = b->m[x.slot];
    if (mem.solo ? !solo_complete(mem) : x.last_g > s->g_complete) {
      ++r;
      continue;
    }
    fdtd2d_ctx* c = b->m[x.slot].ctx;
    // A solo member whose kernels gave up on a bounded wait has skipped work:
    // its results are not handed out, and the call reports the timeout (the
    // batch's own kernel waits for nothing).  The word was allocated and zeroed
    // on the member's own stream: it is read in that stream's order, which has
    // completed.
    if (mem.solo) {
      int derr = 0;
      cudaError_t re = cudaMemcpyAsync(&derr, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
      if (re == cudaSuccess) re = cudaStreamSynchronize(c->stream);
      if (re != cudaSuccess) return fail(b, re);
      if (derr) return FDTD2D_ERR_TIMEOUT;
    }
    Finished f;
    f.tag = x.tag;
    f.n_det = c->n_det;
    f.n_steps = c->n_steps;
    cudaError_t e = cudaSuccess;
    if (c->dft && c->n_det > 0) {
      f.dft.resize((size_t)2 * c->n_det);
      e = cudaMemcpy(f.dft.data(), c->h.dft, f.dft.size() * sizeof(double), cudaMemcpyDeviceToHost);
    }
    if (e == cudaSuccess && c->record && c->n_det > 0) {
      f.trace.resize((size_t)c->n_steps * c->n_det);
      e = cudaMemcpy(f.trace.data(), c->h.trace, f.trace.size() * sizeof(float), cudaMemcpyDeviceToHost);
    }
    if (e != cudaSuccess) return fail(b, e);
    fdtd2d_batch_remove(b, x.slot);
    s->finished.push_back(std::move(f));
    s->running.erase(s->running.begin() + r);
    ++*n_done;
  }
  return FDTD2D_OK;
}

}  // namespace

extern "C" {

int fdtd2d_server_create(int device, int64_t hbm_budget_bytes, int32_t block_steps, fdtd2d_server** out) {
  if (!out || block_steps < 1) return FDTD2D_ERR_INVALID;
  *out = nullptr;
  fdtd2d_server* s = new (std::nothrow) fdtd2d_server();
  if (!s) return FDTD2D_ERR_NOMEM;
  const int rc = fdtd2d_batch_create(device, hbm_budget_bytes, &s->b);
  if (rc) {
    delete s;
    return rc;
  }
  s->block = block_steps;
  *out = s;
  return FDTD2D_OK;
}

static int fdtd2d_server_submit_body(fdtd2d_server* s, const fdtd2d_setup* setup, int64_t tag);

// The entry point: its body, below, runs behind abi_guard.
int fdtd2d_server_submit(fdtd2d_server* s, const fdtd2d_setup* setup, int64_t tag) {
  return abi_guard([&] { return fdtd2d_server_submit_body(s, setup, tag); });
}

static int fdtd2d_server_submit_body(fdtd2d_server* s, const fdtd2d_setup* setup, int64_t tag) {
  if (!s || !setup) return FDTD2D_ERR_INVALID;
  if (setup->medium != FDTD2D_MEDIUM_UNIFORM || setup->npml > tma_max_pml() || setup->n_rc > 0 ||
      setup->line_n > 0)
    return FDTD2D_ERR_INVALID;
  // a setup fdtd2d_create would refuse is refused here, not at admission
  const int vrc = validate_setup(setup);
  if (vrc) return vrc;
  const int64_t bytes = fdtd2d_device_bytes(setup);
  if (bytes < 0) return FDTD2D_ERR_INVALID;
  // could never be admitted (a 16-bit shot is a solo member)
  const int64_t extra = setup->storage == FDTD2D_STORE_F32 ? 0 : solo_extra(setup);
  if (bytes + extra > s->b->budget) return FDTD2D_ERR_BUDGET;
  s->queue.push_back({setup, tag});
  return FDTD2D_OK;
}

static int fdtd2d_server_step_body(fdtd2d_server* s);

// The entry point: its body, below, runs behind abi_guard.
int fdtd2d_server_step(fdtd2d_server* s) {
  return abi_guard([&] { return fdtd2d_server_step_body(s); });
}

static int fdtd2d_server_step_body(fdtd2d_server* s) {
  if (!s) return FDTD2D_ERR_INVALID;
  fdtd2d_batch* b = s->b;
  cudaSetDevice(b->device);
  int n_done = 0;
  // 1. admit in arrival order while the head fits (uploads overlap the queued
  // steps).  Each shot leaves the queue as soon as it is admitted and
  // recorded, so an error on a later one returns with every earlier one
  // running exactly once; the failing shot stays at the head of the queue.
  // The running list grows before the add, so nothing can throw between a
  // successful add and its record.
  while (!s->queue.empty()) {
    s->running.reserve(s->running.size() + 1);
    const Queued head = s->queue.front();
    int32_t slot = -1;
    const int arc = fdtd2d_batch_add(b, head.s, &slot);
    if (arc == FDTD2D_ERR_BUDGET) break;
    if (arc) return arc;
    const fdtd2d_ctx* c = b->m[slot].ctx;
    s->running.push_back({slot, head.tag, b->m[slot].base + c->n_steps});
    s->queue.erase(s->queue.begin());
  }
  // 2. retire what the GPU has finished
  int rc = retire(s, &n_done);
  if (rc) return rc;
  // 3. issue one block while any shot has steps left
  bool steps_left = false, solo_left = false;
  for (const Running& x : s->running) {
    const Member& mem = b->m[x.slot];
    if (mem.solo)
      solo_left = solo_left || !mem.done;
    else
      steps_left = steps_left || x.last_g > b->g;
  }
  if (solo_left && !steps_left) {
    // only solo members have steps left: issue theirs, then wait for the
    // oldest run call of one of them instead of spinning
    rc = run_solo(b, s->block);
    if (rc) return rc;
    for (const Running& x : s->running) {
      Member& mem = b->m[x.slot];
      if (mem.solo && !mem.ev.empty()) {
        const cudaError_t we = cudaEventSynchronize(mem.ev.front());
        if (we != cudaSuccess) return fail(b, we);
        break;
      }
    }
    rc = retire(s, &n_done);
    if (rc) return rc;
  } else if (steps_left) {
    rc = fdtd2d_batch_run(b, s->block);
    if (rc) return rc;
    cudaEvent_t e = take_event(s);
    const cudaError_t ce = cudaEventRecord(e, b->stream);
    if (ce != cudaSuccess) return fail(b, ce);
    s->blocks.push_back({b->g, e});
    // keep at most two blocks ahead of the GPU
    while (s->blocks.size() > 2) {
      const cudaError_t we = cudaEventSynchronize(s->blocks.front().second);
      if (we != cudaSuccess) return fail(b, we);
      rc = retire(s, &n_done);
      if (rc) return rc;
    }
  } else if (!s->blocks.empty()) {
    // nothing more to issue: wait for the oldest block instead of spinning
    const cudaError_t we = cudaEventSynchronize(s->blocks.front().second);
    if (we != cudaSuccess) return fail(b, we);
    rc = retire(s, &n_done);
    if (rc) return rc;
  } else {
    // only solo members still running, all issued: wait for one of them
    for (const Running& x : s->running) {
      const Member& mem = b->m[x.slot];
      if (mem.solo && !mem.ev.empty()) {
        const cudaError_t we = cudaEventSynchronize(mem.ev.back());
        if (we != cudaSuccess) return fail(b, we);
        break;
      }
    }
    rc = retire(s, &n_done);
    if (rc) return rc;
  }
  return n_done;
}

int fdtd2d_server_pop(fdtd2d_server* s, int64_t* tag, int32_t* n_det, int32_t* n_steps, double* dft,
                      int32_t max_det, float* trace, int64_t max_trace) {
  if (!s) return FDTD2D_ERR_INVALID;
  if (s->finished.empty()) return 0;
  Finished& f = s->finished.front();
  if (tag) *tag = f.tag;
  if (n_det) *n_det = f.n_det;
  if (n_steps) *n_steps = f.n_steps;
  if (dft && !f.dft.empty())
    std::memcpy(dft, f.dft.data(), std::min<size_t>(f.dft.size(), 2 * (size_t)std::max<int32_t>(0, max_det)) * 8);
  if (trace && !f.trace.empty())
    std::memcpy(trace, f.trace.data(), std::min<size_t>(f.trace.size(), (size_t)std::max<int64_t>(0, max_trace)) * 4);
  s->finished.erase(s->finished.begin());
  return 1;
}

static int fdtd2d_server_cancel_body(fdtd2d_server* s, int64_t tag);

// The entry point: its body, below, runs behind abi_guard.
int fdtd2d_server_cancel(fdtd2d_server* s, int64_t tag) {
  return abi_guard([&] { return fdtd2d_server_cancel_body(s, tag); });
}

// Queued shots of the tag leave the queue; running ones are removed from the
// batch (a batch-kernel member's memory is released behind the blocks already
// queued for it, which the batch's stream orders before any reuse, and the
// unit list is rebuilt before the next block; a solo member waits for its own
// streams); finished ones not yet popped are dropped.
static int fdtd2d_server_cancel_body(fdtd2d_server* s, int64_t tag) {
  if (!s) return FDTD2D_ERR_INVALID;
  cudaSetDevice(s->b->device);
  int n = 0;
  for (size_t q = 0; q < s->queue.size();) {
    if (s->queue[q].tag == tag) {
      s->queue.erase(s->queue.begin() + q);
      ++n;
    } else {
      ++q;
    }
  }
  for (size_t r = 0; r < s->running.size();) {
    if (s->running[r].tag != tag) {
      ++r;
      continue;
    }
    const int rc = fdtd2d_batch_remove(s->b, s->running[r].slot);
    if (rc) return rc;
    s->running.erase(s->running.begin() + r);
    ++n;
  }
  for (size_t f = 0; f < s->finished.size();) {
    if (s->finished[f].tag == tag) {
      s->finished.erase(s->finished.begin() + f);
      ++n;
    } else {
      ++f;
    }
  }
  return n;
}

int fdtd2d_server_counts(const fdtd2d_server* s, int32_t* queued, int32_t* running, int32_t* finished) {
  if (!s) return FDTD2D_ERR_INVALID;
  if (queued) *queued = (int32_t)s->queue.size();
  if (running) *running = (int32_t)s->running.size();
  if (finished) *finished = (int32_t)s->finished.size();
  return FDTD2D_OK;
}

fdtd2d_batch* fdtd2d_server_batch(fdtd2d_server* s) { return s ? s->b : nullptr; }

int fdtd2d_server_destroy(fdtd2d_server* s) {
  if (!s) return FDTD2D_ERR_INVALID;
  if (s->b) fdtd2d_batch_destroy(s->b);
  for (auto& x : s->blocks) cudaEventDestroy(x.second);
  for (cudaEvent_t e : s->spare) cudaEventDestroy(e);
  delete s;
  return FDTD2D_OK;
}

}  // extern "C"

// Host runtime of the GB300 sweep library and its C ABI (include/subsweep_gpu.h).
//
// Mirrors the reference's Sweep<HydrogenOnly> driver (src/sweep/mod.rs:171-610): the
// sweep parameters, the hierarchical timestep state and the per-step sequence of
// level sweeps live here on the host; every per-cell and per-(cell, direction)
// computation runs in the kernels of sweep_fp64.cu / sweep_mixed.cu.  There is no
// CPU fallback: every entry point fails with SW_ERR_CUDA when no device is usable.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/subsweep_gpu.h"
#include "host_checks.h"
#include "launch.h"
#include "sweep_types.h"

#include "direction_bins.inc"

namespace {

thread_local std::string g_create_error;

// TimestepState, src/sweep/timestep_state.rs:5-90.
struct TimestepState {
  double max_timestep = 0.0;
  int max_num_levels = 1;
  int lowest = 0;
  bool first_done = false;

  void init(double m, int n) {
    max_timestep = m;
    max_num_levels = n;
    lowest = n - 1;
    first_done = false;
  }
  // iter_levels_in_sweep_order (22-27) with lowest_active_from_iteration (70-75)
  std::vector<int> sweep_order() const {
    int num = max_num_levels - lowest;
    std::vector<int> out;
    for (uint32_t i = 0; i < (1u << (num - 1)); ++i) {
      int first_bit = (i == 0) ? (num - 1) : __builtin_ctz(i);
      out.push_back(lowest + (num - 1 - first_bit));
    }
    return out;
  }
  // advance_allowed_levels (37-48)
  void advance() {
    if (first_done && lowest > 0) lowest -= 1;
    if (!first_done) first_done = true;
  }
  // current_max_timestep (77-79): max_timestep * 0.5^lowest
  double current_max_timestep() const { return std::ldexp(max_timestep, -lowest); }
};

template <typename T>
cudaError_t dalloc(T** p, size_t count) {
  *p = nullptr;
  if (count == 0) count = 1;
  return cudaMalloc((void**)p, count * sizeof(T));
}

}  // namespace

int32_t sw_host_sweep_order(int32_t num_levels, int32_t advances, int32_t* out, int32_t cap) {
  if (num_levels < 1 || num_levels > 16 || advances < 0 || cap < 0 || (cap > 0 && !out)) return -1;
  TimestepState ts;
  ts.init(1.0, num_levels);
  for (int32_t i = 0; i < advances; ++i) ts.advance();
  const std::vector<int> order = ts.sweep_order();
  for (size_t i = 0; i < order.size() && (int32_t)i < cap; ++i) out[i] = order[i];
  return (int32_t)order.size();
}

int32_t sw_host_lowest_allowed(int32_t num_levels, int32_t advances) {
  if (num_levels < 1 || num_levels > 16 || advances < 0) return -1;
  TimestepState ts;
  ts.init(1.0, num_levels);
  for (int32_t i = 0; i < advances; ++i) ts.advance();
  return ts.lowest;
}

struct sw_handle {
  sw_params params{};
  const swh::PrecisionOps* ops = nullptr;
  std::vector<double> dirs;
  int D = 0, L = 1;
  uint32_t Np = 0;
  int64_t N = 0, E = 0;
  TimestepState ts;
  double sim_time = 0.0;
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[8] = {};
  // sweeps of a step in flight: their events (start, transport start and end, transport and
  // fold end, chemistry end) and their error flags, read when the host waits for them
  static constexpr int kMaxInFlight = 64;
  std::vector<std::array<cudaEvent_t, 5>> sweep_ev;
  struct Pinned {
    swk::SweepCtl ctl;
    uint32_t error[kMaxInFlight];
  }* pinned = nullptr;
  swh::DevicePtrs p{};
  std::vector<void*> allocations;
  std::vector<uint32_t> n_ge_host;  // cells with level >= l at the start of the next step
  swk::SweepCtl ctl_host{};
  sw_stats stats{};
  std::string last_error;
  double* scratch = nullptr;  // N doubles for field export
  uint32_t stats_schedule_levels = 0;
  // direction streams: whether the schedule is to be laid out in streams, the closed cell
  // ranges of the grid ([parts] offsets), and the layout until the records are built
  bool want_streams = false, force_streams = false;
  uint64_t stream_limit = ~0ull;  // bytes that their pieces may take (SUBSWEEP_STREAM_BYTES)
  int64_t stream_allocs_left = INT64_MAX;  // of their arrays (SUBSWEEP_STREAM_ARRAYS)
  // whether sweeps pull (and are numbered): the mixed path and the FP64 streams
  bool pulls() const { return ops->pull || p.stream_mode; }
  std::vector<uint32_t> parts;
  std::vector<uint32_t> stream_seg;
  std::vector<uint16_t> kept_levels;  // of every task, until the streams are laid out or given up
  std::vector<std::vector<uint8_t>> stream_gmax;  // per stream: the largest count of every group
  std::vector<swk::StreamDesc> streams;
  // fingerprint of the levelled schedule (direction groups and segment offsets): the pull
  // path's checkpointed words are indexed by schedule position
  uint64_t schedule_hash = 0;
  int64_t device_bytes = 0;  // device memory held by the handle (its allocations)
  int64_t stats_upwind_slots = 0;
  int force_path = 0;  // 0 automatic, 1 always levelled, 2 always dependency-driven
  bool trace = false;  // SUBSWEEP_TRACE: one stderr line per level sweep
  uint32_t no_act_list = 0;  // streams: levels whose compacted list found no room
  uint32_t act_valid = 0;  // pull path: levels whose compacted list is current this step
  double* series_dev = nullptr;  // time-series partial sums and result (allocated on first use)
  // graph replay of a step (pull path): the instantiated graph, the step shape it was
  // captured for, and the pinned scalars its first node copies to the control block
  bool graph_mode = false;
  cudaGraphExec_t graph_exec = nullptr;
  std::vector<int64_t> graph_key;
  struct GraphScalars {
    uint32_t epoch_base, pad;
    double time;
  }* graph_scalars = nullptr;
  int64_t graph_captures = 0;
  int64_t graph_kernels = 0;  // kernel launches in the captured step
  // autotuning of the pull transport kernel: trials of ops->tune_variants, one per sweep
  bool autotune = false;
  bool tuned = false;
  int tune_index = 0;
  std::vector<double> tune_ns;  // ns per task of each candidate
  std::vector<cudaEvent_t> graph_ev;  // start / end of each sweep's transport inside the graph
  // whether a cell's x_HII may lie above what the chemistry's clamp takes for a floor
  bool floor_unsafe = false;
  void look_at_floors(const double* x) {
    floor_unsafe = !(params.chemistry_timestep_safety_factor < 1.0);  // (a change of any size may pass)
    for (int64_t c = 0; c < N && !floor_unsafe; ++c) floor_unsafe = !(x[c] <= 1.0 - 1e-10);
  }
  uint32_t last_epoch = 0;  // pull path: sweep number of the last sweep of the last step

  ~sw_handle() {
    if (graph_exec) cudaGraphExecDestroy(graph_exec);
    for (cudaEvent_t e : graph_ev) cudaEventDestroy(e);
    if (graph_scalars) cudaFreeHost(graph_scalars);
    for (auto& set : sweep_ev)
      for (cudaEvent_t e : set)
        if (e) cudaEventDestroy(e);
    if (pinned) cudaFreeHost(pinned);
    for (void* a : allocations) cudaFree(a);
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
    if (stream) cudaStreamDestroy(stream);
  }

  template <typename T>
  bool alloc(T** ptr, size_t count) {
    cudaError_t e = dalloc(ptr, count);
    if (e != cudaSuccess) return false;
    allocations.push_back((void*)*ptr);
    device_bytes += (int64_t)(count * sizeof(T));
    return true;
  }

  // The stream does not wait for the default stream, nor that for it: copies and sets of the arrays
  // that kernels use go by the stream.  Returns when the host's side of the copy is free.
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, kind, stream);
    return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
  }

  // one of the streams' arrays: counted, so that a test can let any of them find no memory
  template <typename T>
  bool stream_alloc(T** ptr, size_t count) {
    return stream_allocs_left-- > 0 && alloc(ptr, count);
  }

  sw_status fail(sw_status st, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    last_error = buf;
    return st;
  }
  sw_status cuda_fail(cudaError_t e, const char* where) {
    return fail(e == cudaErrorMemoryAllocation ? SW_ERR_OOM : SW_ERR_CUDA, "%s: %s", where,
                cudaGetErrorString(e));
  }
};

namespace {

#define SW_CUDA(h, call, where)                   \
  do {                                            \
    cudaError_t _e = (call);                      \
    if (_e != cudaSuccess) return (h)->cuda_fail(_e, where); \
  } while (0)

// The handle's device is current until the entry point returns; the caller's device
// is current again afterwards.
#define SW_DEVICE_SCOPE(h)                                    \
  swh::DeviceScope _device_scope((h)->device);                \
  if (_device_scope.status != cudaSuccess) return (h)->cuda_fail(_device_scope.status, "select device")

sw_status create_fail(sw_status st, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_create_error = buf;
  return st;
}

bool directions_for(int num, std::vector<double>& out) {
  const double(*tab)[3] = nullptr;
  static const double one[1][3] = {{1.0, 0.0, 0.0}};
  switch (num) {  // Directions::from_num, src/sweep/direction/mod.rs:58-75
    case 1: tab = one; break;
    case 16: tab = kDirectionBins16; break;
    case 21: tab = kDirectionBins21; break;
    case 32: tab = kDirectionBins32; break;
    case 64: tab = kDirectionBins64; break;
    case 84: tab = kDirectionBins84; break;
    default: return false;
  }
  out.assign(&tab[0][0], &tab[0][0] + 3 * num);
  return true;
}

// Each LOCAL / LOCAL_PERIODIC face c -> n needs a face n -> c with the bitwise negated
// normal: the reference counts upwind faces from c's side and delivers fluxes from
// n's side, so without it a level sweep could never finish.
bool check_reciprocal_faces(const sw_grid_csr* g, std::string& why) {
  std::atomic<int64_t> bad{-1};
  int nt = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  std::vector<std::thread> th;
  for (int t = 0; t < nt; ++t)
    th.emplace_back([&, t]() {
      for (int64_t c = t; c < g->num_cells; c += nt) {
        if (bad.load(std::memory_order_relaxed) >= 0) return;
        for (int64_t f = g->row_ptr[c]; f < g->row_ptr[c + 1]; ++f) {
          if (g->kind[f] == SW_FACE_BOUNDARY) continue;
          int64_t n = g->nbr[f];
          bool found = false;
          for (int64_t q = g->row_ptr[n]; q < g->row_ptr[n + 1] && !found; ++q)
            found = g->kind[q] != SW_FACE_BOUNDARY && g->nbr[q] == c &&
                    g->normal[3 * q] == -g->normal[3 * f] && g->normal[3 * q + 1] == -g->normal[3 * f + 1] &&
                    g->normal[3 * q + 2] == -g->normal[3 * f + 2];
          if (!found) {
            int64_t expected = -1;
            bad.compare_exchange_strong(expected, f);
            return;
          }
        }
      }
    });
  for (auto& x : th) x.join();
  if (bad.load() >= 0) {
    char buf[200];
    snprintf(buf, sizeof(buf), "face %lld has no reciprocal face with a negated normal",
             (long long)bad.load());
    why = buf;
    return false;
  }
  return true;
}

// check_deadlock analogue (src/sweep/deadlock_detection.rs): with every cell active,
// each direction's dependency graph must be acyclic (Kahn's algorithm on the host).
bool check_acyclic(const sw_grid_csr* g, const std::vector<double>& dirs, int D, std::string& why) {
  int64_t n = g->num_cells;
  std::vector<uint32_t> cnt(n);
  std::vector<int64_t> queue(n);
  for (int d = 0; d < D; ++d) {
    const double* dv = &dirs[3 * d];
    auto dotf = [&](int64_t f) {
      return g->normal[3 * f] * dv[0] + g->normal[3 * f + 1] * dv[1] + g->normal[3 * f + 2] * dv[2];
    };
    int64_t qh = 0, qt = 0;
    for (int64_t c = 0; c < n; ++c) {
      uint32_t k = 0;
      for (int64_t f = g->row_ptr[c]; f < g->row_ptr[c + 1]; ++f)
        if (g->kind[f] == SW_FACE_LOCAL && dotf(f) < 0.0) ++k;
      cnt[c] = k;
      if (k == 0) queue[qt++] = c;
    }
    while (qh < qt) {
      int64_t c = queue[qh++];
      for (int64_t f = g->row_ptr[c]; f < g->row_ptr[c + 1]; ++f)
        if (g->kind[f] == SW_FACE_LOCAL && dotf(f) > 0.0)
          if (--cnt[g->nbr[f]] == 0) queue[qt++] = g->nbr[f];
    }
    if (qt != n) {
      char buf[200];
      snprintf(buf, sizeof(buf), "direction %d: %lld cells lie on dependency cycles", d, (long long)(n - qt));
      why = buf;
      return false;
    }
  }
  return true;
}

sw_status sync_ctl(sw_handle* h) {
  if (!h->pinned) {
    void* ptr = nullptr;
    SW_CUDA(h, cudaMallocHost(&ptr, sizeof(sw_handle::Pinned)), "pinned control block");
    h->pinned = static_cast<sw_handle::Pinned*>(ptr);
  }
  SW_CUDA(h, cudaMemcpyAsync(&h->pinned->ctl, h->p.ctl, sizeof(swk::SweepCtl), cudaMemcpyDeviceToHost, h->stream),
          "read control block");
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  h->ctl_host = h->pinned->ctl;
  h->n_ge_host.assign(h->ctl_host.n_ge, h->ctl_host.n_ge + h->L);
  return SW_OK;
}

// Tasks t in [t0, t1) with t % Np < N listed by level from order[base] on, in id order
// within a level (so each level lists one direction's cells after another in increasing
// order along the space-filling curve, and consecutive tasks touch neighbouring 32-byte
// sectors): each thread counts its contiguous share of the range per level, an
// exclusive scan over (level, thread) gives every share its first slot in each level,
// and the shares are written in parallel.  Returns the tasks per level ([L]).
static std::vector<uint64_t> stable_level_order(const uint16_t* level, uint32_t Np, uint32_t N, uint64_t t0,
                                                uint64_t t1, size_t L, uint64_t base, uint32_t* order) {
  const int nt = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  std::vector<std::vector<uint64_t>> cnt(nt, std::vector<uint64_t>(L, 0u));
  auto range = [&](int t, uint64_t& b, uint64_t& e) {
    b = t0 + (t1 - t0) * t / nt;
    e = t0 + (t1 - t0) * (t + 1) / nt;
  };
  std::vector<std::thread> th;
  for (int t = 0; t < nt; ++t)
    th.emplace_back([&, t]() {
      uint64_t b, e;
      range(t, b, e);
      for (uint64_t i = b; i < e; ++i)
        if (i % Np < N) ++cnt[t][level[i]];
    });
  for (auto& x : th) x.join();
  th.clear();
  std::vector<uint64_t> per_level(L, 0u);
  uint64_t at = base;
  for (size_t l = 0; l < L; ++l) {
    for (int t = 0; t < nt; ++t) {
      const uint64_t n = cnt[t][l];
      cnt[t][l] = at;
      at += n;
      per_level[l] += n;
    }
  }
  for (int t = 0; t < nt; ++t)
    th.emplace_back([&, t]() {
      uint64_t b, e;
      range(t, b, e);
      std::vector<uint64_t>& cur = cnt[t];
      for (uint64_t i = b; i < e; ++i)
        if (i % Np < N) order[cur[level[i]]++] = (uint32_t)i;
    });
  for (auto& x : th) x.join();
  return per_level;
}

// The positions of one task space: its D directions cut into `groups` contiguous
// groups, each group's tasks after the previous group's, by Kahn level (`level`, L
// levels), in task-id order within a level.  Writes order[N * D] and appends the end of
// every non-empty (group, level) segment to seg (which starts with 0); returns the
// number of positions written.
static uint64_t grouped_level_order(const uint16_t* level, uint32_t Np, uint32_t N, uint32_t D, size_t L,
                                    int groups, uint32_t* order, std::vector<uint32_t>& seg) {
  uint64_t base = 0;
  for (int g = 0; g < groups; ++g) {
    const uint64_t d0 = (uint64_t)D * g / groups, d1 = (uint64_t)D * (g + 1) / groups;
    const std::vector<uint64_t> n = stable_level_order(level, Np, N, d0 * Np, d1 * Np, L, base, order);
    for (size_t l = 0; l < L; ++l)
      if (n[l]) {
        base += n[l];
        seg.push_back((uint32_t)base);
      }
  }
  return base;
}

// Closed parts of a grid: contiguous cell ranges that no LOCAL face leaves (the boxes of
// a batch; the whole grid otherwise), at least `min_cells` each.  Returns their offsets.
static std::vector<uint32_t> closed_parts(const sw_grid_csr* g, int64_t min_cells) {
  std::vector<int32_t> farthest(g->num_cells);  // LOCAL neighbour of every cell
  {
    const int nt = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    std::vector<std::thread> th;
    for (int t = 0; t < nt; ++t)
      th.emplace_back([&, t]() {
        for (int64_t c = g->num_cells * t / nt; c < g->num_cells * (t + 1) / nt; ++c) {
          int32_t n = 0;
          for (int64_t f = g->row_ptr[c]; f < g->row_ptr[c + 1]; ++f)
            if (g->kind[f] == SW_FACE_LOCAL) n = std::max(n, (int32_t)g->nbr[f]);
          farthest[c] = n;
        }
      });
    for (auto& x : th) x.join();
  }
  std::vector<uint32_t> parts = {0};
  int64_t reach = 0;
  for (int64_t c = 0; c < g->num_cells; ++c) {
    reach = std::max<int64_t>(reach, farthest[c]);
    if (reach <= c && c + 1 - parts.back() >= min_cells && g->num_cells - (c + 1) >= min_cells)
      parts.push_back((uint32_t)(c + 1));
  }
  parts.push_back((uint32_t)g->num_cells);
  return parts;
}

// The positions in direction streams: direction by direction, part by part, each stream's
// tasks by Kahn level, within a level by number of upwind LOCAL faces (`up`), then by id.
// Writes order[N * D]; the streams' descriptors (base, count, dir, seg0, segs) and the
// level segments' offsets (seg[0] = 0, the end of every segment) are appended; gmax: the
// largest count of every group of kStreamGroup tasks of a level, per stream.  A stream's
// levels are contiguous from 0: every level has a task whose upwind neighbour lies one
// level below, in the same stream.
static void stream_order(const uint16_t* level, const uint8_t* up, uint32_t Np, uint32_t N, uint32_t D,
                         const std::vector<uint32_t>& parts, uint32_t* order, std::vector<uint32_t>& seg,
                         std::vector<swk::StreamDesc>& streams, std::vector<std::vector<uint8_t>>& gmax) {
  const uint32_t np = (uint32_t)parts.size() - 1, ns = D * np;
  std::vector<std::vector<uint32_t>> ends(ns);
  gmax.assign(ns, {});
  std::atomic<uint32_t> next{0};
  const int nt = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  std::vector<std::thread> th;
  for (int t = 0; t < nt; ++t)
    th.emplace_back([&]() {
      std::vector<uint32_t> tmp, at;
      for (uint32_t s; (s = next.fetch_add(1)) < ns;) {
        const uint32_t d = s / np, c0 = parts[s % np], n = parts[s % np + 1] - c0;
        const uint32_t t0 = d * Np + c0;
        tmp.resize(n);
        uint32_t by_count[257] = {0};
        uint32_t depth = 0;
        for (uint32_t i = 0; i < n; ++i) {
          ++by_count[up[t0 + i] + 1u];
          depth = std::max<uint32_t>(depth, level[t0 + i] + 1u);
        }
        for (int k = 0; k < 256; ++k) by_count[k + 1] += by_count[k];
        for (uint32_t i = 0; i < n; ++i) tmp[by_count[up[t0 + i]]++] = t0 + i;
        at.assign(depth + 1, 0u);
        for (uint32_t i = 0; i < n; ++i) ++at[level[t0 + i] + 1u];
        for (uint32_t l = 0; l < depth; ++l) at[l + 1] += at[l];
        const uint32_t base = d * N + c0;
        for (uint32_t l = 1; l <= depth; ++l) ends[s].push_back(base + at[l]);
        for (uint32_t i = 0; i < n; ++i) order[base + at[level[tmp[i]]]++] = tmp[i];
        // the last task of a group has its largest count
        uint32_t p = base;
        for (uint32_t e : ends[s])
          while (p < e) {
            p = std::min(p + swk::kStreamGroup, e);
            gmax[s].push_back(up[order[p - 1]]);
          }
      }
    });
  for (auto& x : th) x.join();
  seg.assign(1, 0u);
  streams.clear();
  for (uint32_t s = 0; s < ns; ++s) {
    swk::StreamDesc x{};
    x.dir = s / np;
    x.base = x.dir * N + parts[s % np];
    x.count = parts[s % np + 1] - parts[s % np];
    x.seg0 = (uint32_t)seg.size() - 1;
    x.segs = (uint32_t)ends[s].size();
    seg.insert(seg.end(), ends[s].begin(), ends[s].end());
    streams.push_back(x);
  }
}

// Whether pairs of blocks walk the streams faster than single blocks: cycles of a level with g
// groups, times the levels of the longest stream, times the rounds (there are half as many
// pairs).  Lines through the measured times of uniform boxes, ms per sweep of 84 directions with
// single blocks and pairs: mixed path 96^3 (18 groups a level) 3.06 and 3.77, 128^3 (31) 7.68 and
// 7.24; FP64 64^3 (8) 2.14 and 2.68, 72^3 3.12 and 3.35, 80^3 4.51 and 4.14, 96^3 8.48 and 7.42; 16
// directions FP64 64^3 1.94 and 2.19, 80^3 3.98 and 3.24, 101^3 (19) 8.02 and 6.56.
static bool pairs_pay(double levels, double groups, double total, int sms, bool mixed) {
  const double g = groups / levels;
  const double one = mixed ? 500.0 + 176.0 * g : std::max(670.0, 580.0 * g - 1300.0);
  const double two = mixed ? 1850.0 + 103.0 * g : 1540.0 + 295.0 * g;
  const auto rounds = [&](int blocks) { return std::max(1.0, total / (groups * blocks)); };
  return two * rounds(sms / 2) < 0.95 * one * rounds(sms);
}

// Whether direction streams are faster than the kernels over the levelled schedule: the longest
// stream, at 3.6 ns a task of its block (FP64 8.1, of a pair of blocks 6.4 where pairs_pay takes them,
// times the streams that a pair has), against the time of a level, from word to word 0.85 us (FP64
// push form, from atomic to atomic: 4), times the levels, plus the tasks at 17 per ns (12).
// Measured on uniform boxes, ms per sweep, levelled and streams.  Mixed path: 84 directions 24^3 0.32
// and 0.15, 48^3 0.97 and 0.50, 64^3 1.67 and 1.04, 128^3 10.6 and 7.3; 16 directions 64^3 0.99 and
// 0.87, but 101^3 2.0 and 3.0: sixteen blocks cannot keep up with the whole device where levels are
// wide.  FP64: 84 directions 16^3 0.95 and 0.18, 24^3 1.60 and 0.32, 32^3 2.08 and 0.47, 64^3 5.4 and
// 2.1, 96^3 13.8 and 7.4, 128^3 34 and 19.5, 160^3 66 and 38; 16 directions 64^3 4.8 and 1.9, 101^3
// 7.8 and 6.6.  Where a level is wide, the ring holds few levels and many words come from memory:
// mixed path 160^3 (1800 tasks a level) 20.8 and 16.1, 192^3 (2200) 35 and 34, 256^3 (3400) 83 and
// 114; hence the limit on the width.
static bool streams_pay(const std::vector<uint32_t>& parts, uint64_t tasks, size_t levels, int sms, bool mixed) {
  uint32_t longest = 0;
  for (size_t k = 1; k < parts.size(); ++k) longest = std::max(longest, parts[k] - parts[k - 1]);
  if (!mixed) {
    double task = 8.1;
    if (pairs_pay((double)levels, longest / (double)swk::kStreamGroup, (double)tasks / swk::kStreamGroup, sms, false))
      task = 6.4 * std::max(1.0, 2.0 * (double)tasks / ((double)longest * sms));
    return task * longest < 4000.0 * (double)levels + (double)tasks / 12.0;
  }
  return longest < 2600.0 * (double)levels && 3.6 * longest < 850.0 * (double)levels + (double)tasks / 17.0;
}

// Compact state (mixed path): task spaces hold fewer than kSpaceTasks tasks each.  The
// fewest spaces of evenly split directions that do, 0 when kMaxSpaces are not enough.
constexpr uint64_t kSpaceTasks = 1ull << 31;
static int min_task_spaces(uint32_t Np, int D) {
  for (int s = 1; s <= std::min(D, swh::kMaxSpaces); ++s)
    if ((uint64_t)Np * (uint64_t)((D + s - 1) / s) < kSpaceTasks) return s;
  return 0;
}

// Number of direction groups of the schedule: SUBSWEEP_DIR_GROUPS, else as many as keep
// a group's levels about 40 K tasks wide on average (one per 40 K tasks of the average
// level, rounded).  That is about the number of tasks the lockstep kernels hold in
// flight (152 SMs x 32 warps x 8 tasks), so a task seldom waits for an upwind word, and
// a level's records, slots and words (~100 bytes a task) stay a small part of L2.
// Measured on the C4 generator at 256^3 x 84 (4,927 levels, 286 K tasks per level):
// 1, 4, 7 and 12 groups move 367, 169, 121 and 106 B of DRAM traffic per task in a
// level-0 sweep of 105, 94, 91 and 93 ms.
static int schedule_dir_groups(int D, uint64_t tasks, size_t levels) {
  constexpr uint64_t kGroupWidth = 40960;
  int g = (int)std::min<uint64_t>((tasks / std::max<size_t>(levels, 1) + kGroupWidth / 2) / kGroupWidth, (uint64_t)D);
  if (const char* env = std::getenv("SUBSWEEP_DIR_GROUPS")) g = std::atoi(env);
  return std::max(1, std::min(g, D));
}

// Fingerprint of a schedule: FNV-1a over the state kind, spaces, groups and offsets.
struct ScheduleHash {
  uint64_t value = 0xcbf29ce484222325ull;
  void mix(uint32_t v) {
    for (int k = 0; k < 4; ++k) value = (value ^ ((v >> (8 * k)) & 0xffu)) * 0x100000001b3ull;
  }
};

// The Kahn levels of a space's tasks (all cells active), on the host: levels[t], their number, and
// for streams the upwind LOCAL faces of every task.  cyclic: some task has no level.
static sw_status kahn_levels(sw_handle* h, const swh::DevicePtrs& q, std::vector<uint16_t>& levels, size_t& depth,
                             std::vector<uint8_t>& up, bool& cyclic) {
  const swh::DevicePtrs& p = h->p;
  const uint64_t total = (uint64_t)h->N * (uint64_t)q.D;
  struct DeviceScratch {
    void* ptr = nullptr;
    ~DeviceScratch() {
      if (ptr) cudaFree(ptr);
    }
  } level_scratch, bounds_scratch;
  SW_CUDA(h, cudaMalloc(&level_scratch.ptr, (size_t)h->Np * q.D * sizeof(uint16_t)), "schedule scratch");
  uint16_t* task_level = static_cast<uint16_t*>(level_scratch.ptr);
  SW_CUDA(h, cudaMemsetAsync(p.ctl, 0, offsetof(swk::SweepCtl, tasks), h->stream), "reset control");
  SW_CUDA(h, cudaMemsetAsync(task_level, 0, (size_t)h->Np * q.D * sizeof(uint16_t), h->stream), "schedule scratch");
  SW_CUDA(h, h->ops->schedule_seed(q, h->stream), "schedule seed kernel");
  std::vector<uint32_t> lvl = {0};
  unsigned long long tail = 0;
  SW_CUDA(h, cudaMemcpyAsync(&tail, &p.ctl->tail, sizeof(tail), cudaMemcpyDeviceToHost, h->stream), "read tail");
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "schedule seed");
  if (h->want_streams) {  // (the rounds count them down)
    up.resize((size_t)h->Np * q.D);
    SW_CUDA(h, h->copy(up.data(), p.counters, up.size(), cudaMemcpyDeviceToHost), "read upwind counts");
  }
  // the rounds, kRounds at a time (those after the last one find nothing to do)
  constexpr uint32_t kRounds = 32, kMaxRounds = 0xffffu;
  SW_CUDA(h, cudaMalloc(&bounds_scratch.ptr, (kMaxRounds + kRounds + 2) * sizeof(uint32_t)), "schedule scratch");
  uint32_t* bounds = static_cast<uint32_t*>(bounds_scratch.ptr) + 1;  // behind the blocks' count
  const uint32_t first[3] = {0u, 0u, (uint32_t)tail};
  SW_CUDA(h, h->copy(bounds - 1, first, sizeof(first), cudaMemcpyHostToDevice), "schedule scratch");
  uint32_t end = (uint32_t)tail;
  if (end > 0) lvl.push_back(end);
  for (uint32_t round = 0; end > 0;) {
    uint32_t ends[kRounds];
    SW_CUDA(h, h->ops->kahn_rounds(q, bounds, bounds - 1, task_level, round, kRounds, h->stream),
            "schedule round kernel");
    SW_CUDA(h, cudaMemcpyAsync(ends, bounds + round + 2, sizeof(ends), cudaMemcpyDeviceToHost, h->stream),
            "read bounds");
    SW_CUDA(h, cudaStreamSynchronize(h->stream), "schedule round");
    bool more = true;
    for (uint32_t k = 0; k < kRounds && more; ++k) {
      more = ends[k] > end;
      if (more) lvl.push_back(end = ends[k]);
    }
    if (!more) break;
    round += kRounds;
    if (round >= kMaxRounds) return h->fail(SW_ERR_UNSUPPORTED, "dependency graph deeper than 65534 levels");
  }
  tail = end;
  if (lvl.size() - 1 >= kMaxRounds) return h->fail(SW_ERR_UNSUPPORTED, "dependency graph deeper than 65534 levels");
  uint32_t err = 0;
  SW_CUDA(h, h->copy(&err, &p.ctl->error, sizeof(err), cudaMemcpyDeviceToHost), "read error flag");
  cyclic = tail != total || err != 0;
  if (cyclic) return SW_OK;
  depth = lvl.size() - 1;
  levels.resize((size_t)h->Np * q.D);
  SW_CUDA(h, h->copy(levels.data(), task_level, levels.size() * sizeof(uint16_t), cudaMemcpyDeviceToHost),
          "read task levels");
  return SW_OK;
}

// Levelled schedule (Kahn levels of all N*D tasks with every cell active), built once
// per grid on the device, per task space (one space unless the compact state splits the
// directions; task ids and positions are local to a space).  A dependency cycle leaves
// tasks unscheduled; such a grid keeps only the dependency-driven path, whose sweep then
// reports the stall as the reference would deadlock (the compact state, which has no
// such path, refuses the grid).
sw_status build_schedule(sw_handle* h) {
  swh::DevicePtrs& p = h->p;
  ScheduleHash hash;
  hash.mix((uint32_t)p.geo_mode);
  hash.mix((uint32_t)p.num_spaces);
  uint32_t depth = 0;
  for (int sp = 0; sp < p.num_spaces; ++sp) {
    const swh::DevicePtrs q = swh::space_view(p, sp);
    const uint64_t total = (uint64_t)h->N * (uint64_t)q.D;
    // (of a grid whose streams were given up, the levels are known)
    std::vector<uint16_t> tl = std::move(h->kept_levels);
    size_t L = h->stats_schedule_levels;
    std::vector<uint8_t> up;
    bool cyclic = false;
    if (tl.empty()) {
      const sw_status st = kahn_levels(h, q, tl, L, up, cyclic);
      if (st != SW_OK) return st;
    }
    if (cyclic) {
      if (p.geo_mode) return h->fail(SW_ERR_STALLED, "the dependency graph has a cycle (compact state)");
      // cyclic dependency graph: no schedule.  The push path falls back to the
      // dependency-driven queue; the pull path visits tasks in id order and its waits run
      // out, so either reports the stall at the first sweep, where the reference deadlocks.
      p.num_sched_levels = 0;
      h->want_streams = false;
      if (h->ops->pull) {
        std::vector<uint32_t> ids;
        ids.reserve(total);
        for (uint32_t d = 0; d < (uint32_t)h->D; ++d)
          for (uint32_t c = 0; c < (uint32_t)h->N; ++c) ids.push_back(d * h->Np + c);
        SW_CUDA(h, h->copy(p.order, ids.data(), ids.size() * sizeof(uint32_t), cudaMemcpyHostToDevice), "order");
      }
      SW_CUDA(h, cudaMemsetAsync(p.ctl, 0, offsetof(swk::SweepCtl, tasks), h->stream), "reset control");
      return SW_OK;
    }
    // The positions: the space's directions are cut into `groups` contiguous groups,
    // each group's tasks listed after the previous group's, by Kahn level, in task-id
    // order within a level.  Directions never depend on one another, so this is a
    // topological order, and its segments (one per non-empty (group, level)) are levels
    // of a valid levelled schedule.  Fewer directions per level keep the words a level
    // reads (written one or a few levels before) in L2 on large grids; the compact
    // state's geometry kernel pays a grid barrier per segment and keeps one group.  The
    // order is a stable counting sort on the host, so every handle on the same grid
    // gets the same schedule: the pull path's words are indexed by schedule position,
    // and checkpoints hold them in that order.
    depth = std::max(depth, (uint32_t)L);
    if (h->want_streams) h->want_streams = h->force_streams || streams_pay(h->parts, total, L, p.num_sms, h->ops->pull);
    int groups = schedule_dir_groups(q.D, total, L);
    if (p.geo_mode && !std::getenv("SUBSWEEP_DIR_GROUPS")) groups = 1;
    std::vector<uint32_t> seg = {0};
    {
      std::vector<uint32_t> order(total);
      if (h->want_streams) {
        stream_order(tl.data(), up.data(), h->Np, (uint32_t)h->N, (uint32_t)q.D, h->parts, order.data(), seg,
                     h->streams, h->stream_gmax);
        h->stream_seg = seg;
        h->kept_levels = std::move(tl);
      } else if (grouped_level_order(tl.data(), h->Np, (uint32_t)h->N, (uint32_t)q.D, L, groups, order.data(), seg) !=
                 total) {
        return h->fail(SW_ERR_CUDA, "schedule order incomplete");
      }
      SW_CUDA(h, h->copy(q.order, order.data(), order.size() * sizeof(uint32_t), cudaMemcpyHostToDevice),
              "upload order");
    }
    uint32_t* d_lvl;
    // padded to a multiple of four entries: the staged wavefront kernel copies them whole
    const size_t lvl_words = (seg.size() + 3) & ~(size_t)3;
    if (!h->alloc(&d_lvl, lvl_words)) return h->fail(SW_ERR_OOM, "device allocation of the schedule failed");
    SW_CUDA(h, cudaMemsetAsync(d_lvl, 0, lvl_words * sizeof(uint32_t), h->stream), "schedule");
    SW_CUDA(h, h->copy(d_lvl, seg.data(), seg.size() * sizeof(uint32_t), cudaMemcpyHostToDevice),
            "upload schedule");
    p.space_lvl[sp] = d_lvl;
    p.space_segments[sp] = (uint32_t)(seg.size() - 1);
    p.space_lvl_words[sp] = (uint32_t)lvl_words;
    hash.mix((uint32_t)groups);
    for (uint32_t o : seg) hash.mix(o);
  }
  SW_CUDA(h, cudaMemsetAsync(p.ctl, 0, offsetof(swk::SweepCtl, tasks), h->stream), "reset control");
  p.lvl = p.space_lvl[0];
  p.num_sched_levels = p.space_segments[0];
  p.lvl_words = p.space_lvl_words[0];
  h->stats_schedule_levels = depth;  // the dependency depth
  h->schedule_hash = hash.value;
  return SW_OK;
}

// Push path: precomputed downwind fractions of every schedule position, when they fit
// in the free device memory less a reserve of 1/16 of the device (at least 4 GiB) for
// later allocations (SUBSWEEP_FP64_RECORDS=0 never builds them, =1 always tries).
// Without them the transport computes the geometry on the fly.
sw_status build_push_records(sw_handle* h) {
  swh::DevicePtrs& p = h->p;
  if (!h->ops->push_records || p.num_sched_levels == 0 || p.stream_mode) return SW_OK;
  int mode = -1;
  if (const char* env = std::getenv("SUBSWEEP_FP64_RECORDS")) mode = std::atoi(env) != 0 ? 1 : 0;
  if (mode == 0) return SW_OK;
  const int64_t positions = h->N * (int64_t)h->D;
  const size_t nc = (size_t)((positions + swk::kCompactChunk - 1) / swk::kCompactChunk);
  const size_t rec_bytes = (size_t)positions * sizeof(uint4);
  size_t free_b = 0, total_b = 0;
  SW_CUDA(h, cudaMemGetInfo(&free_b, &total_b), "memory info");
  const size_t reserve = std::max(total_b / 16, (size_t)4 << 30);
  const size_t room = free_b > reserve ? free_b - reserve : 0;
  if (mode < 0 && rec_bytes > room) return SW_OK;
  struct DeviceScratch {
    void* ptr = nullptr;
    ~DeviceScratch() {
      if (ptr) cudaFree(ptr);
    }
  } rec_mem, off_mem;
  if (cudaMalloc(&rec_mem.ptr, rec_bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    return SW_OK;  // no room: the geometry path
  }
  SW_CUDA(h, cudaMalloc(&off_mem.ptr, (nc + 1) * sizeof(unsigned long long)), "record scratch");
  auto* chunk_off = static_cast<unsigned long long*>(off_mem.ptr);
  p.push_rec = rec_mem.ptr;
  cudaError_t ce = h->ops->push_records(p, 0, chunk_off, h->stream);
  unsigned long long total = 0;
  if (ce == cudaSuccess)
    ce = cudaMemcpyAsync(&total, chunk_off + nc, sizeof(total), cudaMemcpyDeviceToHost, h->stream);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(h->stream);
  p.push_rec = nullptr;
  if (ce != cudaSuccess) return h->cuda_fail(ce, "downwind fraction count kernels");
  const size_t slot_bytes = (size_t)total * (sizeof(uint32_t) + sizeof(double));
  if (mode < 0 && rec_bytes + slot_bytes > room) return SW_OK;
  uint32_t* tgt = nullptr;
  double* frac = nullptr;
  if (!h->alloc(&tgt, std::max<unsigned long long>(total, 1)) || !h->alloc(&frac, std::max<unsigned long long>(total, 1))) {
    (void)cudaGetLastError();
    return SW_OK;
  }
  p.push_rec = rec_mem.ptr;
  p.push_tgt = tgt;
  p.push_frac = frac;
  ce = h->ops->push_records(p, 1, chunk_off, h->stream);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(h->stream);
  uint32_t err = 0;
  if (ce == cudaSuccess) ce = h->copy(&err, &p.ctl->error, sizeof(err), cudaMemcpyDeviceToHost);
  if (ce != cudaSuccess) {
    p.push_rec = nullptr;
    return h->cuda_fail(ce, "downwind fraction kernel");
  }
  if (err & swk::kErrRecords) {
    p.push_rec = nullptr;
    return h->fail(SW_ERR_CUDA, "downwind classification disagrees with its count");
  }
  h->allocations.push_back(rec_mem.ptr);  // kept for the handle's lifetime
  rec_mem.ptr = nullptr;
  h->stats_upwind_slots = (int64_t)total;
  return SW_OK;
}

// The groups of one stream, in order (data and the flags of the shape follow later).
static void plan_stream(const swk::StreamDesc& sd, const uint32_t* seg, const std::vector<uint8_t>& gmax,
                        swk::StreamGroup* out) {
  uint32_t g = 0;
  for (uint32_t k = sd.seg0; k < sd.seg0 + sd.segs; ++k) {
    const uint32_t need = g;
    for (uint32_t p = seg[k]; p < seg[k + 1]; p += swk::kStreamGroup, ++g) {
      const uint32_t n = std::min(swk::kStreamGroup, seg[k + 1] - p), slots = (gmax[g] + 3u) & ~3u;
      out[g] = {need, 0u, p, (n - 1) | (slots << 5)};
    }
  }
}

// The parts of `pairs` pairs of blocks: the streams' groups end to end, cut into equal shares at
// the nearest level.  A stream that is cut has its beginning in front of the next pair's share and
// the rest at the end of this one's, so the beginning is solved by the time the rest is due (no
// stream is longer than a share).  Returns the number of cuts (flags).
static uint32_t plan_parts(const std::vector<swk::StreamDesc>& streams, const std::vector<uint32_t>& seg_group,
                           uint32_t pairs, std::vector<swk::StreamPart>& parts, std::vector<uint32_t>& part0) {
  uint64_t total = 0, longest = 0;
  for (const swk::StreamDesc& s : streams) {
    total += s.groups;
    longest = std::max<uint64_t>(longest, s.groups);
  }
  const uint64_t share = std::max(longest, (total + pairs - 1) / pairs);
  uint32_t flags = 0;
  uint64_t room = share;
  parts.clear();
  part0 = {0};
  for (uint32_t i = 0; i < streams.size(); ++i) {
    const swk::StreamDesc& s = streams[i];
    uint32_t cut = 0;  // groups in front of the next pair's share
    if (s.groups > room) {
      const uint32_t want = (uint32_t)(s.groups - room), last = (uint32_t)(part0.size());
      if (last < pairs) {
        const uint32_t* lo = seg_group.data() + s.seg0;
        const uint32_t* at = std::lower_bound(lo, lo + s.segs, s.group0 + want);
        cut = (at == lo + s.segs ? s.group0 + s.groups : *at) - s.group0;
      }
    }
    if (cut == 0) {
      parts.push_back({i, 0, s.groups, 0, 0});
      room -= std::min<uint64_t>(room, s.groups);
      continue;
    }
    if (cut < s.groups) parts.push_back({i, cut, s.groups, flags + 1, 0});
    part0.push_back((uint32_t)parts.size());
    parts.push_back({i, 0, cut, 0, cut < s.groups ? ++flags : 0});
    room = share - std::min<uint64_t>(share, cut);
  }
  part0.push_back((uint32_t)parts.size());
  return flags;
}

// bytes of a group's piece (StreamPiece), rb bytes a rate
static uint32_t piece_bytes(uint32_t shape, uint32_t rb) {
  const uint32_t slots = (shape >> 5) & 0x7fu, far = shape >> 17;
  return (uint32_t)sizeof(swk::StreamGroup) + (rb == 8 ? 16u : 0u) +
         32u * (rb + (rb == 4 ? 4u : 0u) + slots * (rb + 2u) + ((shape & swk::kGroupExt) ? 2u * rb : 0u) + far * 4u);
}

// Direction streams: groups and their pieces, and the launch shape (after the schedule is in
// place).
sw_status build_streams(sw_handle* h) {
  swh::DevicePtrs& p = h->p;
  const std::vector<uint32_t>& seg = h->stream_seg;
  const uint32_t segs = (uint32_t)seg.size() - 1;
  const uint32_t rb = (uint32_t)h->ops->rate_bytes;
  // no room, at any point: the levelled schedule (build_records frees what was allocated)
  const auto give_up = [h]() {
    (void)cudaGetLastError();
    h->want_streams = false;
    return SW_OK;
  };
#define SW_ROOM(h, call, where)                                  \
  do {                                                           \
    const cudaError_t _r = (call);                               \
    if (_r == cudaErrorMemoryAllocation) return give_up();       \
    if (_r != cudaSuccess) return (h)->cuda_fail(_r, where);     \
  } while (0)
  const double width = (double)h->N * h->D / segs;  // of a level, on average
  // warps of a block: as many as find a group of a level to work on.  Mixed path, 84 directions,
  // ms per sweep with 4, 8 and 16: 24^3 (35 tasks a level) 0.159, 0.152, 0.185; 32^3 (62) 0.289,
  // 0.235, 0.274; 48^3 (138) 0.80, 0.57, 0.52; 64^3 (250) 2.5, 1.55, 1.01.  FP64, whose warps also
  // sum ahead: 24^3 0.36, 0.31, 0.31; 32^3 0.69, 0.48, 0.46; 48^3 2.2, 1.38, 1.02 (sums made anew; of
  // changes with 16 warps 0.32, 0.47, 1.07).
  uint32_t warps = width <= 32 ? 4 : (width <= (rb == 4 ? 96 : 48) ? 8 : 16);
  if (const char* env = std::getenv("SUBSWEEP_STREAM_WARPS")) {
    const int v = std::atoi(env);
    if (v == 4 || v == 8 || v == 16) warps = (uint32_t)v;
  }
  bool pairs = false;
  {
    const double total = (double)h->N * h->D / swk::kStreamGroup;
    double longest = 0, levels = 0;
    for (const swk::StreamDesc& s : h->streams)
      if (s.count > longest) {
        longest = s.count;
        levels = s.segs;
      }
    pairs = pairs_pay(levels, longest / swk::kStreamGroup, total, p.num_sms, rb == 4);
    if (const char* env = std::getenv("SUBSWEEP_STREAM_PAIRS")) pairs = std::atoi(env) != 0;
  }
  uint32_t slots = 0;  // per task of the largest group
  for (const auto& m : h->stream_gmax)
    for (uint8_t v : m) slots = std::max<uint32_t>(slots, (v + 3u) & ~3u);
  std::vector<uint32_t> seg_group(segs + 1), sbase(segs), sgroup(segs);
  uint32_t longest = 0, widest = 0;
  for (swk::StreamDesc& s : h->streams) {
    s.group0 = seg_group[s.seg0];
    for (uint32_t k = s.seg0; k < s.seg0 + s.segs; ++k) {
      widest = std::max(widest, seg[k + 1] - seg[k]);
      seg_group[k + 1] = seg_group[k] + (seg[k + 1] - seg[k] + swk::kStreamGroup - 1) / swk::kStreamGroup;
      sbase[k] = s.base;
      sgroup[k] = s.group0;
    }
    s.groups = seg_group[s.seg0 + s.segs] - s.group0;
    longest = std::max(longest, s.count);
  }
  // Shared memory of a block: its share of the SM's (several blocks share an SM when there are
  // more streams than SMs); the warps' buffers, the rest words: ring, unless that leaves far
  // words, for which the warps then get room.
  int optin = 0, per_sm = 0;
  SW_CUDA(h, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device), "attribute");
  SW_CUDA(h, cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, h->device), "attribute");
  const uint32_t buffer = piece_bytes(31u | (slots << 5) | swk::kGroupExt, rb);
  auto words_for = [&](size_t room, uint32_t far) -> int64_t {
    return std::min<int64_t>(((int64_t)room - 288 - 4 * rb - (int64_t)warps * buffer) / rb - (int64_t)warps * far * 32,
                             60000 - (int64_t)warps * far * 32);
  };
  size_t room = 0;
  uint32_t* shape = p.stream_shape;
  int resident = 0;  // pairs at once
  const uint32_t single = warps;
  for (;; pairs = false) {
    warps = pairs ? swk::kPairWarps : single;
    const int most = pairs ? 1 : std::max(1, std::min(8, (int)(48 / warps)));  // blocks per SM that registers allow
    for (int k = std::max(1, std::min(most, (int)((h->streams.size() + p.num_sms - 1) / p.num_sms))); k >= 1; --k) {
      room = std::min((size_t)optin, (size_t)per_sm / k - 1024);
      if (words_for(room, swk::kStreamFar) >= (int64_t)std::min(longest, 8192u)) break;
    }
    const int64_t ring = words_for(room, swk::kStreamFar);
    // a ring must not wrap inside a level: with a wider one the grid keeps the levelled schedule
    if (ring < (int64_t)std::min(longest, widest)) {
      if (pairs) continue;
      return give_up();
    }
    if (!pairs) break;
    // with the most shared memory that the layout may ask for; none: single blocks
    const uint32_t largest[6] = {(uint32_t)ring, 0u, swk::kStreamFar, warps, buffer, 2u};
    std::copy(largest, largest + 6, shape);
    if (h->ops->stream_pairs(p, &resident) != cudaSuccess) {
      (void)cudaGetLastError();
      resident = 0;
    }
    if (const char* env = std::getenv("SUBSWEEP_STREAM_PAIRS")) {  // at most so many, or (-1) none
      const int v = std::atoi(env);
      if (v > 1 || v < 0) resident = std::min(resident, std::max(v, 0));
    }
    if (resident >= 1) break;
  }
  std::vector<swk::StreamGroup> groups(seg_group[segs]);
  {
    std::atomic<size_t> next{0};
    const int nt = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    std::vector<std::thread> th;
    for (int t = 0; t < nt; ++t)
      th.emplace_back([&]() {
        for (size_t s; (s = next.fetch_add(1)) < h->streams.size();)
          plan_stream(h->streams[s], seg.data(), h->stream_gmax[s], groups.data() + h->streams[s].group0);
      });
    for (auto& x : th) x.join();
  }
  h->stream_gmax.clear();
  // No room: the levelled schedule.  FP64: as for the push form's records, room is what leaves a
  // reserve of 1/16 of the device (at least 4 GiB) for later allocations.
  size_t free_b = 0, total_b = 0;
  SW_CUDA(h, cudaMemGetInfo(&free_b, &total_b), "memory info");
  const size_t reserve = rb == 8 ? std::max(total_b / 16, (size_t)4 << 30) : 0;
  uint64_t least = 0;
  for (const swk::StreamGroup& g : groups) least += piece_bytes(g.shape, rb);
  if (least + reserve > free_b || least > h->stream_limit) {
    return give_up();
  }
  struct Scratch {
    sw_handle* h;
    std::vector<void*> mem;
    ~Scratch() {
      for (void* m : mem) cudaFree(m);
    }
    cudaError_t get(void** out, size_t bytes, const void* src) {
      cudaError_t e = cudaMalloc(out, std::max<size_t>(bytes, 4));
      if (e != cudaSuccess) return e;
      mem.push_back(*out);
      return src ? h->copy(*out, src, bytes, cudaMemcpyHostToDevice) : cudaSuccess;
    }
  } scratch{h, {}};
  swh::StreamScratch b{};
  SW_ROOM(h, scratch.get((void**)&b.gseg, groups.size() * 4, nullptr), "stream scratch");
  SW_ROOM(h, scratch.get((void**)&b.sbase, sbase.size() * 4, sbase.data()), "stream scratch");
  SW_ROOM(h, scratch.get((void**)&b.sgroup, sgroup.size() * 4, sgroup.data()), "stream scratch");
  if (rb == 8) SW_ROOM(h, scratch.get((void**)&b.recip, (size_t)h->E * 4, nullptr), "stream scratch");
  swk::StreamDesc* d_streams = nullptr;
  swk::StreamGroup* d_groups = nullptr;
  if (!h->stream_alloc(&d_streams, h->streams.size()) || !h->stream_alloc(&d_groups, groups.size() + 1) ||
      !h->stream_alloc(&p.seg_group, seg_group.size()))
    return give_up();
  if (rb == 8) {  // what the push form does without
    uint32_t *pos = nullptr, *counts = nullptr;
    if (!h->stream_alloc(&pos, (size_t)h->Np * h->D) || !h->stream_alloc(&counts, 32) ||
        !h->stream_alloc(&p.fold_changed, p.n_periodic_cells) ||
        !h->stream_alloc(&p.fold_off, (size_t)p.n_periodic_cells * h->D + 1))
      return give_up();
    p.pos_of_task = pos;
    p.act_counts = counts;
  }
  p.streams = d_streams;
  p.stream_groups = d_groups;
  p.num_streams = (uint32_t)h->streams.size();
  p.num_groups = (uint32_t)groups.size();
  const size_t group_bytes = groups.size() * sizeof(groups[0]);
  std::stable_sort(h->streams.begin(), h->streams.end(),  // launch order: the longest first
                   [](const swk::StreamDesc& x, const swk::StreamDesc& y) { return x.count > y.count; });
  SW_CUDA(h, h->copy(d_streams, h->streams.data(), h->streams.size() * sizeof(h->streams[0]), cudaMemcpyHostToDevice),
          "streams");
  SW_CUDA(h, h->copy(p.seg_group, seg_group.data(), seg_group.size() * 4, cudaMemcpyHostToDevice), "streams");
  SW_CUDA(h, h->ops->stream_build(p, 0, b, h->stream), "stream position kernels");
  shape[3] = warps;
  shape[5] = pairs ? 2u : 1u;
  bool far = false;
  int64_t late = 0, slow = 0;
  // room for far words is taken from the ring only if there are any: looked for with it where the
  // ring is shorter than the longest stream, and without it again if there are none
  const bool whole = words_for(room, 0) >= (int64_t)longest;
  for (int pass = 0; pass < 2; ++pass) {
    shape[2] = (pass == 0) == whole ? 0u : swk::kStreamFar;
    shape[4] = buffer;
    shape[0] = (uint32_t)std::min<int64_t>(words_for(room, shape[2]), longest);
    shape[1] = (uint32_t)((1ull << 32) / shape[0]) + 1u;
    for (swk::StreamGroup& g : groups) g.shape &= 0xfffu;
    SW_CUDA(h, h->copy(d_groups, groups.data(), group_bytes, cudaMemcpyHostToDevice), "groups");
    SW_CUDA(h, h->ops->stream_build(p, 1, b, h->stream), "stream flag kernel");
    SW_CUDA(h, cudaStreamSynchronize(h->stream), "stream flags");
    SW_CUDA(h, h->copy(groups.data(), d_groups, group_bytes, cudaMemcpyDeviceToHost), "groups");
    far = false;
    late = slow = 0;
    for (const swk::StreamGroup& g : groups) {
      far = far || (g.shape >> 17) != 0;
      late += (g.shape & swk::kGroupLate) != 0;
      slow += (g.shape & swk::kGroupSlow) != 0;
    }
    if (far == (shape[2] != 0u)) break;
  }
  if (pairs) {
    std::vector<swk::StreamPart> parts;
    std::vector<uint32_t> part0;
    plan_parts(h->streams, seg_group, (uint32_t)resident, parts, part0);
    swk::StreamPart* d_parts = nullptr;
    if (!h->stream_alloc(&d_parts, parts.size()) || !h->stream_alloc(&p.stream_part0, part0.size()) ||
        !h->stream_alloc(&p.stream_flags, part0.size()))
      return give_up();
    SW_CUDA(h, h->copy(d_parts, parts.data(), parts.size() * sizeof(parts[0]), cudaMemcpyHostToDevice), "streams");
    SW_CUDA(h, h->copy(p.stream_part0, part0.data(), part0.size() * 4, cudaMemcpyHostToDevice), "streams");
    SW_CUDA(h, cudaMemsetAsync(p.stream_flags, 0xff, part0.size() * 4, h->stream), "streams");
    p.stream_parts = d_parts;
    p.num_pairs = (uint32_t)part0.size() - 1;
  }
  uint64_t at = 0;
  for (swk::StreamGroup& g : groups) {
    g.data = (uint32_t)(at / swk::kStreamUnit);
    at += (piece_bytes(g.shape, rb) + swk::kStreamUnit - 1) / swk::kStreamUnit * swk::kStreamUnit;
  }
  groups.push_back({0u, (uint32_t)(at / swk::kStreamUnit), 0u, 0u});  // where the last piece ends
  if (at / swk::kStreamUnit > 0xffffffffull) {  // past the pieces' 32-bit offsets: the levelled schedule
    return give_up();
  }
  SW_CUDA(h, h->copy(d_groups, groups.data(), groups.size() * sizeof(groups[0]), cudaMemcpyHostToDevice), "groups");
  groups.pop_back();
  SW_CUDA(h, cudaMemGetInfo(&free_b, &total_b), "memory info");
  if (at + reserve > free_b || at > h->stream_limit || !h->stream_alloc(&p.stream_data, at)) return give_up();
  char* cell_att = nullptr;
  std::vector<uint32_t> pcells(p.n_periodic_cells);
  std::vector<uint8_t> has_periodic(h->N, 0);
  SW_CUDA(h, h->copy(pcells.data(), p.periodic_cells, pcells.size() * 4, cudaMemcpyDeviceToHost), "periodic cells");
  for (uint32_t c : pcells) has_periodic[c] = 1;
  if (!h->stream_alloc(&cell_att, (size_t)h->N * rb) || !h->stream_alloc(&p.cell_rate, h->N) ||
      !h->stream_alloc(&p.cell_periodic, h->N) || !h->stream_alloc(&p.stale, h->N))
    return give_up();
  p.stream_bytes = at;
  p.cell_att = cell_att;
  SW_CUDA(h, h->copy(p.cell_periodic, has_periodic.data(), h->N, cudaMemcpyHostToDevice), "periodic cells");
  SW_CUDA(h, cudaMemsetAsync(p.ctl, 0, offsetof(swk::SweepCtl, tasks), h->stream), "reset control");
  SW_CUDA(h, h->ops->stream_build(p, 2, b, h->stream), "upwind slot kernel");
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "upwind slots");
  if (rb == 8 && p.n_periodic_cells > 0) {  // the periodic fold's slots
    const size_t entries = (size_t)p.n_periodic_cells * h->D;
    void* cnt = nullptr;
    SW_ROOM(h, scratch.get(&cnt, entries, nullptr), "fold scratch");
    p.fold_cnt = static_cast<uint8_t*>(cnt);
    SW_CUDA(h, h->ops->stream_build(p, 3, b, h->stream), "periodic fold entries");
    SW_CUDA(h, cudaStreamSynchronize(h->stream), "periodic fold entries");
    p.fold_cnt = nullptr;
    std::vector<uint8_t> n(entries);
    SW_CUDA(h, h->copy(n.data(), cnt, entries, cudaMemcpyDeviceToHost), "periodic fold entries");
    std::vector<uint32_t> off(entries + 1, 0u);
    for (size_t e = 0; e < entries; ++e) off[e + 1] = off[e] + n[e];
    SW_CUDA(h, h->copy(p.fold_off, off.data(), off.size() * 4, cudaMemcpyHostToDevice), "periodic fold entries");
    uint4* fslots = nullptr;
    if (!h->stream_alloc(&fslots, off[entries])) return give_up();
    p.fold_slots = fslots;
    SW_CUDA(h, h->ops->stream_build(p, 4, b, h->stream), "periodic fold entries");
    SW_CUDA(h, cudaStreamSynchronize(h->stream), "periodic fold entries");
  }
  if (rb == 8) {
    unsigned long long faces[2] = {0, 0};  // handed out, found
    SW_CUDA(h, h->copy(&faces[0], &p.ctl->head, 8, cudaMemcpyDeviceToHost), "upwind slots");
    SW_CUDA(h, h->copy(&faces[1], &p.ctl->tail, 8, cudaMemcpyDeviceToHost), "upwind slots");
    const size_t nd = (size_t)h->Np * h->D;
    SW_CUDA(h, cudaMemsetAsync(p.pending, 0, nd * 8, h->stream), "pending rates");
    SW_CUDA(h, cudaMemsetAsync(p.ctl, 0, offsetof(swk::SweepCtl, error), h->stream), "reset control");
    // faces without a partner of their own: only the push form tells them apart
    if (faces[0] != faces[1]) return give_up();
  }
  uint32_t err = 0;
  SW_CUDA(h, h->copy(&err, &p.ctl->error, sizeof(err), cudaMemcpyDeviceToHost), "read error flag");
  if (err & swk::kErrRecords) return h->fail(SW_ERR_CUDA, "upwind slot classification disagrees with its count");
  int64_t all_slots = 0;
  for (const swk::StreamGroup& g : groups) all_slots += (int64_t)((g.shape & 31u) + 1u) * ((g.shape >> 5) & 0x7fu);
  h->stats_upwind_slots = all_slots;
  if (h->trace)
    std::fprintf(stderr, "subsweep streams: %u (%u pairs) of %u warps, buffer %u, ring %u, far %u, %zu groups (%lld late, %lld slow), %llu bytes\n",
                 p.num_streams, p.num_pairs, warps, shape[4], shape[0], shape[2], groups.size(), (long long)late, (long long)slow,
                 (unsigned long long)at);
  p.stream_mode = 1;
  return SW_OK;
}
#undef SW_ROOM

// Pull path: task records and upwind slots of every schedule position (after the
// schedule, or the id order of a cyclic grid, is in place).
sw_status build_records(sw_handle* h) {
  if (h->want_streams) {
    const swh::DevicePtrs before = h->p;
    const size_t allocations = h->allocations.size();
    const int64_t device_bytes = h->device_bytes;
    sw_status st = build_streams(h);
    if (st != SW_OK || h->want_streams) {
      h->kept_levels = {};
      return st;
    }
    // a level too wide for a ring, or no room: the levelled schedule
    for (size_t k = allocations; k < h->allocations.size(); ++k) cudaFree(h->allocations[k]);
    h->allocations.resize(allocations);
    h->device_bytes = device_bytes;
    h->p = before;
    // (the push form adds what `pending` holds to the periodic sources: the tasks' totals were there)
    if (h->p.pending)
      SW_CUDA(h, cudaMemsetAsync(h->p.pending, 0, (size_t)h->Np * h->D * (size_t)h->ops->rate_bytes, h->stream),
              "pending rates");
    SW_CUDA(h, cudaMemsetAsync(h->p.ctl, 0, offsetof(swk::SweepCtl, tasks), h->stream), "reset control");
    SW_CUDA(h, cudaStreamSynchronize(h->stream), "levelled schedule");
    h->streams.clear();
    h->stream_seg.clear();
    h->stream_gmax.clear();
    st = build_schedule(h);
    if (st != SW_OK) return st;
  }
  if (!h->ops->records) return SW_OK;
  swh::DevicePtrs& p = h->p;
  if (p.geo_mode) {  // compact state: only the periodic fold's entries
    SW_CUDA(h, h->ops->records(p, 1, nullptr, h->stream), "periodic fold entries");
    SW_CUDA(h, cudaStreamSynchronize(h->stream), "periodic fold entries");
    return SW_OK;
  }
  const size_t nc = (size_t)((h->N * (int64_t)h->D + swk::kCompactChunk - 1) / swk::kCompactChunk);
  struct DeviceScratch {
    void* ptr = nullptr;
    ~DeviceScratch() {
      if (ptr) cudaFree(ptr);
    }
  } off_scratch;
  SW_CUDA(h, cudaMalloc(&off_scratch.ptr, (nc + 1) * sizeof(unsigned long long)), "record scratch");
  auto* chunk_off = static_cast<unsigned long long*>(off_scratch.ptr);
  if (!p.pull_rec) {  // a cyclic grid that was to be laid out in streams
    uint4* rec = nullptr;
    if (!h->alloc(&rec, (size_t)h->Np * h->D)) return h->fail(SW_ERR_OOM, "device allocation of the task records failed");
    p.pull_rec = rec;
  }
  SW_CUDA(h, h->ops->records(p, 0, chunk_off, h->stream), "task record kernels");
  unsigned long long total = 0;
  SW_CUDA(h, cudaMemcpyAsync(&total, chunk_off + nc, sizeof(total), cudaMemcpyDeviceToHost, h->stream),
          "read slot total");
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "task records");
  uint2* slots = nullptr;
  // two slots of padding: the staged wavefront kernel copies 16-byte aligned ranges
  if (!h->alloc(&slots, total + 2))
    return h->fail(SW_ERR_OOM, "device allocation of the upwind slots (%llu MB) failed", (total * 8) >> 20);
  p.pull_slots = slots;
  SW_CUDA(h, h->ops->records(p, 1, chunk_off, h->stream), "upwind slot kernel");
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "upwind slots");
  uint32_t err = 0;
  SW_CUDA(h, h->copy(&err, &p.ctl->error, sizeof(err), cudaMemcpyDeviceToHost), "read error flag");
  if (err & swk::kErrRecords) return h->fail(SW_ERR_CUDA, "upwind slot classification disagrees with its count");
  h->stats_upwind_slots = (int64_t)total;
  return SW_OK;
}

}  // namespace


namespace swh {

bool handle_view(sw_handle* h, HandleView* out) {
  if (!h || !out) return false;
  out->p = &h->p;
  out->ops = h->ops;
  out->stream = h->stream;
  out->device = h->device;
  out->num_cells = h->N;
  out->num_directions = h->D;
  out->num_levels = h->L;
  return true;
}

sw_status handle_fail(sw_handle* h, sw_status st, const char* message) {
  if (h) h->last_error = message;
  return st;
}

void handle_clear_error(sw_handle* h) {
  if (h) h->last_error.clear();
}

}  // namespace swh

extern "C" {

sw_status sw_default_params(sw_params* p) {
  if (!p) return SW_ERR_INVALID_ARG;
  std::memset(p, 0, sizeof(*p));
  p->num_directions = 84;
  p->explicit_directions = nullptr;
  p->num_timestep_levels = 1;
  p->periodic = 0;
  p->max_timestep = 1e6 * 3.15576e7;  // 1 Myr
  p->rotate_directions = 0;               // parameters.rs:64-78
  p->significant_rate_threshold = 0.0;
  p->timestep_safety_factor = 0.01 * 10.0;  // Dimensionless::percent(10.0)
  p->chemistry_timestep_safety_factor = 0.01 * 10.0;
  p->check_deadlock = 0;
  p->prevent_cooling = 1;
  p->num_tasks_to_solve_before_send_receive = 10000;
  p->scale_factor = 1.0;
  p->precision = SW_PRECISION_FP64;
  p->device = -1;
  p->use_graphs = 0;
  p->autotune = 1;
  return SW_OK;
}

sw_status sw_directions_from_num(int32_t num, double* out) {
  std::vector<double> d;
  if (!out || !directions_for(num, d)) return SW_ERR_INVALID_ARG;
  std::memcpy(out, d.data(), d.size() * sizeof(double));
  return SW_OK;
}

sw_status sw_create(const sw_params* params, const sw_grid_csr* grid, const sw_cell_init* init,
                    sw_handle** out) {
  g_create_error.clear();
  if (!out) return create_fail(SW_ERR_INVALID_ARG, "out is NULL");
  *out = nullptr;
  if (!params || !grid || !init) return create_fail(SW_ERR_INVALID_ARG, "NULL argument");
  const sw_params& P = *params;
  if (P.rotate_directions)
    return create_fail(SW_ERR_UNSUPPORTED, "rotate_directions is not supported by the GPU sweep");
  if (P.num_timestep_levels < 1 || P.num_timestep_levels > 16)
    return create_fail(SW_ERR_INVALID_ARG, "num_timestep_levels must be in 1..16");
  if (!(P.max_timestep > 0.0) || !std::isfinite(P.max_timestep))
    return create_fail(SW_ERR_INVALID_ARG, "max_timestep must be positive");
  if (P.precision != SW_PRECISION_FP64 && P.precision != SW_PRECISION_MIXED)
    return create_fail(SW_ERR_INVALID_ARG, "unknown precision");
  std::vector<double> dirs;
  int D = P.num_directions;
  if (P.explicit_directions) {
    if (D < 1) return create_fail(SW_ERR_INVALID_ARG, "num_directions must be >= 1");
    dirs.assign(P.explicit_directions, P.explicit_directions + 3 * D);
    for (int d = 0; d < D; ++d) {  // glam normalize: v * (1 / |v|)
      double* v = &dirs[3 * d];
      double inv = 1.0 / std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
      if (!std::isfinite(inv)) return create_fail(SW_ERR_INVALID_ARG, "direction %d has zero length", d);
      v[0] *= inv;
      v[1] *= inv;
      v[2] *= inv;
    }
  } else if (!directions_for(D, dirs)) {
    return create_fail(SW_ERR_INVALID_ARG, "num_directions %d has no direction table (1,16,21,32,64,84)", D);
  }
  if (D > swk::kMaxDirections) return create_fail(SW_ERR_UNSUPPORTED, "at most 128 directions");

  const int64_t N = grid->num_cells;
  if (N < 1 || N >= (int64_t)1 << 30) return create_fail(SW_ERR_INVALID_ARG, "num_cells must be in 1..2^30-1");
  const uint32_t Np = (uint32_t)((N + 31) / 32 * 32);
  // The FP64 path keeps 32-bit task ids; the mixed path splits larger grids into task
  // spaces of fewer than 2^31 tasks each (compact state).
  const uint64_t task_ids = (uint64_t)Np * (uint64_t)D;
  if (P.precision == SW_PRECISION_FP64 && task_ids >= 0xffffffffull)
    return create_fail(SW_ERR_UNSUPPORTED, "num_cells * directions must stay below 2^32 task ids (FP64 path)");
  if (min_task_spaces(Np, D) == 0)
    return create_fail(SW_ERR_UNSUPPORTED, "num_cells * directions needs more than %d task spaces of 2^31 tasks",
                       swh::kMaxSpaces);
  if (!grid->row_ptr || !grid->nbr || !grid->kind || !grid->area || !grid->normal || !grid->volume || !grid->size)
    return create_fail(SW_ERR_INVALID_ARG, "grid array is NULL");
  if (!init->density || !init->ionized_hydrogen_fraction || !init->temperature || !init->source)
    return create_fail(SW_ERR_INVALID_ARG, "cell init array is NULL");
  if (grid->row_ptr[0] != 0) return create_fail(SW_ERR_INVALID_ARG, "row_ptr[0] must be 0");
  double max_normal = 0.0;
  for (int64_t c = 0; c < N; ++c) {
    int64_t nf = grid->row_ptr[c + 1] - grid->row_ptr[c];
    if (nf < 0) return create_fail(SW_ERR_INVALID_ARG, "row_ptr not monotone at cell %lld", (long long)c);
    if (nf > swk::kMaxFaces)
      return create_fail(SW_ERR_UNSUPPORTED, "cell %lld has %lld faces (max %d)", (long long)c, (long long)nf,
                         swk::kMaxFaces);
  }
  const int64_t E = grid->row_ptr[N];
  if (E >= 0xffffffffll) return create_fail(SW_ERR_UNSUPPORTED, "at most 2^32-1 faces");
  for (int64_t f = 0; f < E; ++f) {
    uint8_t k = grid->kind[f];
    if (k > SW_FACE_BOUNDARY) return create_fail(SW_ERR_INVALID_ARG, "face %lld has invalid kind", (long long)f);
    if (k != SW_FACE_BOUNDARY && (grid->nbr[f] < 0 || grid->nbr[f] >= N))
      return create_fail(SW_ERR_INVALID_ARG, "face %lld neighbour out of range", (long long)f);
    const double* nv = &grid->normal[3 * f];
    double l = std::sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
    if (!std::isfinite(l) || !std::isfinite(grid->area[f]))
      return create_fail(SW_ERR_INVALID_ARG, "face %lld has non-finite geometry", (long long)f);
    max_normal = std::max(max_normal, l);
  }
  std::string why;
  if (!check_reciprocal_faces(grid, why)) return create_fail(SW_ERR_INVALID_ARG, "%s", why.c_str());
  if (P.check_deadlock && !check_acyclic(grid, dirs, D, why)) return create_fail(SW_ERR_STALLED, "%s", why.c_str());
  if (P.prevent_cooling) {
    // HydrogenOnly clamps x_HII into [x_floor, 1 - 1e-10] and f64::clamp panics when
    // the floor (the current x_HII) is above that range.
    for (int64_t c = 0; c < N; ++c)
      if (init->ionized_hydrogen_fraction[c] > 1.0 - 1e-10)
        return create_fail(SW_ERR_INVALID_ARG,
                           "cell %lld: x_HII above 1 - 1e-10 with prevent_cooling (reference panics)",
                           (long long)c);
  }

  sw_handle* h = new sw_handle();
  h->params = P;
  h->params.explicit_directions = nullptr;
  h->ops = (P.precision == SW_PRECISION_MIXED) ? &swh::kOpsMixed : &swh::kOpsFP64;
  h->dirs = dirs;
  h->D = D;
  h->Np = Np;
  h->L = P.num_timestep_levels;
  h->N = N;
  h->E = E;
  h->ts.init(P.max_timestep, P.num_timestep_levels);
  h->look_at_floors(init->ionized_hydrogen_fraction);

  auto bail = [&](sw_status st) {
    g_create_error = h->last_error;
    delete h;
    return st;
  };
  cudaError_t ce = cudaSuccess;
  if (P.device >= 0)
    h->device = P.device;
  else
    ce = cudaGetDevice(&h->device);
  if (ce != cudaSuccess) {
    h->cuda_fail(ce, "select device");
    return bail(SW_ERR_CUDA);
  }
  // the handle's device is current while the handle is built (and freed on failure)
  swh::DeviceScope device_scope(h->device);
  if (device_scope.status != cudaSuccess) {
    h->cuda_fail(device_scope.status, "select device");
    return bail(SW_ERR_CUDA);
  }
  int coop = 0, sms = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
  if (!coop) {
    h->fail(SW_ERR_CUDA, "device does not support cooperative launches");
    return bail(SW_ERR_CUDA);
  }
  int bps = 0;
  ce = h->ops->occupancy(&bps);
  if (ce != cudaSuccess || bps < 1) {
    h->cuda_fail(ce == cudaSuccess ? cudaErrorInvalidConfiguration : ce, "occupancy");
    return bail(SW_ERR_CUDA);
  }
  if ((ce = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking)) != cudaSuccess) {
    h->cuda_fail(ce, "stream");
    return bail(SW_ERR_CUDA);
  }
  for (auto& e : h->ev) cudaEventCreate(&e);

  swh::DevicePtrs& p = h->p;
  p.num_cells = N;
  p.D = D;
  p.Np = Np;
  p.num_levels = h->L;
  for (int i = 0; i < 3 * D; ++i) p.dir32_host[i] = (float)dirs[i];
  p.threshold = P.significant_rate_threshold;
  p.max_timestep = P.max_timestep;
  p.timestep_safety = P.timestep_safety_factor;
  p.chem_safety = P.chemistry_timestep_safety_factor;
  p.scale_factor = P.scale_factor;
  p.prevent_cooling = P.prevent_cooling;
  // Resident blocks of the persistent transport kernel: at most the occupancy limit;
  // SUBSWEEP_SWEEP_BLOCKS_PER_SM lowers it (launch-shape tuning).
  // The dependency-driven kernel is bound by contention on its queue counters, not by
  // occupancy: one resident block per SM measured fastest.
  int want = 1;
  if (const char* env = std::getenv("SUBSWEEP_SWEEP_BLOCKS_PER_SM")) want = std::atoi(env);
  if (want >= 1 && want < bps) bps = want;
  p.coop_blocks = bps * sms;
  int lbps = 0;
  ce = h->ops->occupancy_levels(&lbps);
  if (ce != cudaSuccess || lbps < 1) {
    h->cuda_fail(ce == cudaSuccess ? cudaErrorInvalidConfiguration : ce, "occupancy");
    return bail(SW_ERR_CUDA);
  }
  if (const char* env = std::getenv("SUBSWEEP_LEVEL_BLOCKS_PER_SM")) {
    int v = std::atoi(env);
    if (v >= 1 && v < lbps) lbps = v;
  }
  p.level_blocks = lbps * sms;
  // SUBSWEEP_TRANSPORT=levels|queue pins the transport kernel (tests and tuning).
  if (const char* env = std::getenv("SUBSWEEP_TRANSPORT")) {
    if (std::strcmp(env, "levels") == 0) h->force_path = 1;
    if (std::strcmp(env, "queue") == 0) h->force_path = 2;
  }
  // transport kernel variant: SUBSWEEP_PULL_VARIANT fixes it, else the autotuner picks
  // it (sw_params.autotune; SUBSWEEP_AUTOTUNE=0|1 overrides)
  p.num_sms = sms;
  if (const char* env = std::getenv("SUBSWEEP_LEVEL_BLOCKS_PER_SM")) p.level_bps_cap = std::atoi(env);
  h->autotune = P.autotune != 0;
  if (const char* env = std::getenv("SUBSWEEP_AUTOTUNE")) h->autotune = std::atoi(env) != 0;
  if (const char* env = std::getenv("SUBSWEEP_PULL_VARIANT")) {
    p.pull_variant = std::atoi(env);
    h->autotune = false;
  }
  if (h->ops->num_tune_variants == 0) h->autotune = false;
  // graph replay of steps (SUBSWEEP_GRAPH=0|1 overrides the parameter)
  h->graph_mode = P.use_graphs != 0;
  if (const char* env = std::getenv("SUBSWEEP_GRAPH")) h->graph_mode = std::atoi(env) != 0;
  // SUBSWEEP_COMPACT=always|never overrides the mixed path's choice between compacting
  // the active positions and stamping inactive tasks in the sweep (tests and tuning).
  if (const char* env = std::getenv("SUBSWEEP_COMPACT")) {
    if (std::strcmp(env, "always") == 0) p.compact_mode = 1;
    if (std::strcmp(env, "never") == 0) p.compact_mode = 2;
  }
  // SUBSWEEP_TRACE=1 prints one line per level sweep to stderr (level, active tasks,
  // transport kernel / transport / chemistry milliseconds, transport attempts).
  if (const char* env = std::getenv("SUBSWEEP_TRACE")) h->trace = env[0] != '\0' && env[0] != '0';
  p.timeout_ns = 2ull * 1000 * 1000 * 1000;  // a lane waits at most 2 s for its queue slot
  double max_dir = 0.0;
  for (int d = 0; d < D; ++d)
    max_dir = std::max(max_dir, std::sqrt(dirs[3 * d] * dirs[3 * d] + dirs[3 * d + 1] * dirs[3 * d + 1] +
                                          dirs[3 * d + 2] * dirs[3 * d + 2]));
  // FP32 dot of FP32-rounded vectors: |error| <= ~5 * 2^-24 * |n| |d|; 4x margin.
  p.guard = (float)(20.0 * std::ldexp(1.0, -24) * std::max(1.0, max_normal) * std::max(1.0, max_dir));
  // Stored rate unit: photons/s in the FP64 drop-in; a power of two in the mixed path,
  // so that rates up to the total source (times 2^32 headroom) stay finite in FP32 and
  // the smallest normal float is ~2^-126 of the largest source.
  double total_source = 0.0;
  for (int64_t c = 0; c < N; ++c) total_source += std::fabs(init->source[c]);
  p.rate_scale = 1.0;
  if (P.precision == SW_PRECISION_MIXED && total_source > 0.0) {
    int e = 0;
    std::frexp(total_source, &e);
    p.rate_scale = std::ldexp(1.0, e - 96);
  }

  // geometry upload in kernel layout.  FP32 areas carry a power-of-two scale that maps
  // the largest face area to ~1 (areas of ~1e42 m^2 overflow FP32); the FP32 transport
  // only uses ratios of areas within a cell, which the scale leaves exact.
  double max_area = 0.0;
  for (int64_t f = 0; f < E; ++f) max_area = std::max(max_area, std::fabs(grid->area[f]));
  int area_exp = 0;
  if (max_area > 0.0) std::frexp(max_area, &area_exp);
  {
    std::vector<double> geo64(4 * (size_t)E);
    std::vector<float> geo32(4 * (size_t)E);
    std::vector<uint32_t> geo16(h->ops->pull ? 4 * (size_t)E : 0);
    std::vector<uint32_t> nbr(E);
    std::vector<uint32_t> row(N + 1);
    for (int64_t i = 0; i <= N; ++i) row[i] = (uint32_t)grid->row_ptr[i];
    for (int64_t f = 0; f < E; ++f) {
      for (int a = 0; a < 3; ++a) {
        geo64[4 * f + a] = grid->normal[3 * f + a];
        geo32[4 * f + a] = (float)grid->normal[3 * f + a];
      }
      geo64[4 * f + 3] = grid->area[f];
      geo32[4 * f + 3] = (float)std::ldexp(grid->area[f], -area_exp);
      uint32_t kind = grid->kind[f];
      uint32_t nb = (kind == SW_FACE_BOUNDARY) ? 0u : (uint32_t)grid->nbr[f];
      nbr[f] = nb | (kind << swk::kKindShift);
      if (h->ops->pull) {  // {area * n in the scaled FP32 area unit, neighbour | kind}
        const double a = std::ldexp(grid->area[f], -area_exp);
        for (int c3 = 0; c3 < 3; ++c3) {
          const float v = (float)(a * grid->normal[3 * f + c3]);
          std::memcpy(&geo16[4 * f + c3], &v, sizeof(float));
        }
        geo16[4 * f + 3] = nbr[f];
      }
    }
    uint32_t* d_row;
    double* d_geo64;
    float* d_geo32;
    uint32_t* d_nbr;
    if (!h->alloc(&d_row, N + 1) || !h->alloc(&d_geo64, 4 * (size_t)E) || !h->alloc(&d_geo32, 4 * (size_t)E) ||
        !h->alloc(&d_nbr, E)) {
      h->fail(SW_ERR_OOM, "device allocation of the grid failed");
      return bail(SW_ERR_OOM);
    }
    cudaMemcpy(d_row, row.data(), (N + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice);
    cudaMemcpy(d_geo64, geo64.data(), geo64.size() * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_geo32, geo32.data(), geo32.size() * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(d_nbr, nbr.data(), E * sizeof(uint32_t), cudaMemcpyHostToDevice);
    if (h->ops->pull) {
      uint32_t* d_geo16;
      if (!h->alloc(&d_geo16, geo16.size())) {
        h->fail(SW_ERR_OOM, "device allocation of the grid failed");
        return bail(SW_ERR_OOM);
      }
      cudaMemcpy(d_geo16, geo16.data(), geo16.size() * sizeof(uint32_t), cudaMemcpyHostToDevice);
      p.geo16 = d_geo16;
    }
    p.off = d_row;
    p.geo64 = d_geo64;
    p.geo32 = d_geo32;
    p.nbr = d_nbr;
    // cells that receive periodic contributions
    std::vector<uint32_t> pcells;
    for (int64_t c = 0; c < N; ++c)
      for (int64_t f = grid->row_ptr[c]; f < grid->row_ptr[c + 1]; ++f)
        if (grid->kind[f] == SW_FACE_LOCAL_PERIODIC) {
          pcells.push_back((uint32_t)c);
          break;
        }
    uint32_t* d_pc;
    if (!h->alloc(&d_pc, pcells.size())) {
      h->fail(SW_ERR_OOM, "device allocation failed");
      return bail(SW_ERR_OOM);
    }
    if (!pcells.empty()) cudaMemcpy(d_pc, pcells.data(), pcells.size() * sizeof(uint32_t), cudaMemcpyHostToDevice);
    p.periodic_cells = d_pc;
    p.n_periodic_cells = (uint32_t)pcells.size();
    if (h->ops->pull && !pcells.empty()) {  // the fold's precomputed upwind periodic faces
      uint8_t *fcnt = nullptr, *fchanged = nullptr;
      uint2* fslots = nullptr;
      const size_t entries = pcells.size() * (size_t)D;
      if (!h->alloc(&fcnt, entries) || !h->alloc(&fslots, entries * 4) || !h->alloc(&fchanged, pcells.size())) {
        h->fail(SW_ERR_OOM, "device allocation of the periodic fold slots failed");
        return bail(SW_ERR_OOM);
      }
      p.fold_cnt = fcnt;
      p.fold_slots = fslots;
      p.fold_changed = fchanged;
    }
  }
  // directions
  {
    std::vector<float> d32(dirs.begin(), dirs.end());
    double* d_dir64;
    float* d_dir32;
    if (!h->alloc(&d_dir64, dirs.size()) || !h->alloc(&d_dir32, dirs.size())) {
      h->fail(SW_ERR_OOM, "device allocation failed");
      return bail(SW_ERR_OOM);
    }
    cudaMemcpy(d_dir64, dirs.data(), dirs.size() * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_dir32, d32.data(), d32.size() * sizeof(float), cudaMemcpyHostToDevice);
    p.dir64 = d_dir64;
    p.dir32 = d_dir32;
  }
  // cells
  {
    double *d_size, *d_volume, *d_density, *d_source, *d_x, *d_y, *d_T, *d_att, *d_prev, *d_cts, *d_sdt, *d_ion;
    uint8_t* d_level;
    char* d_src_dir;
    const size_t rb = (size_t)h->ops->rate_bytes;
    bool ok = h->alloc(&d_size, N) && h->alloc(&d_volume, N) && h->alloc(&d_density, N) && h->alloc(&d_source, N) &&
              h->alloc(&d_x, N) && h->alloc(&d_y, N) && h->alloc(&d_T, N) && h->alloc(&d_att, N) &&
              h->alloc(&d_prev, N) && h->alloc(&d_cts, N) && h->alloc(&d_sdt, N) && h->alloc(&d_ion, N) &&
              h->alloc(&d_level, N) && h->alloc(&d_src_dir, N * rb) && h->alloc(&h->scratch, N);
    if (!ok) {
      h->fail(SW_ERR_OOM, "device allocation of cell state failed");
      return bail(SW_ERR_OOM);
    }
    std::vector<double> y(N), inf(N, INFINITY);
    for (int64_t c = 0; c < N; ++c) y[c] = 1.0 - init->ionized_hydrogen_fraction[c];
    // Site::source_per_direction_bin (site.rs:49-51), in stored rate units
    if (rb == 8) {
      std::vector<double> sd(N);
      for (int64_t c = 0; c < N; ++c) sd[c] = init->source[c] / (double)D;
      cudaMemcpy(d_src_dir, sd.data(), N * sizeof(double), cudaMemcpyHostToDevice);
    } else {
      std::vector<float> sd(N);
      for (int64_t c = 0; c < N; ++c) sd[c] = (float)(init->source[c] / (double)D / p.rate_scale);
      cudaMemcpy(d_src_dir, sd.data(), N * sizeof(float), cudaMemcpyHostToDevice);
    }
    cudaMemcpy(d_size, grid->size, N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_volume, grid->volume, N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_density, init->density, N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_source, init->source, N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_x, init->ionized_hydrogen_fraction, N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_y, y.data(), N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_T, init->temperature, N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d_ion, inf.data(), N * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemset(d_att, 0, N * sizeof(double));
    cudaMemset(d_prev, 0, N * sizeof(double));  // Site::new: zero previous rate
    cudaMemset(d_cts, 0, N * sizeof(double));   // change_timescale = 0
    cudaMemset(d_sdt, 0, N * sizeof(double));   // species timestep = 0
    cudaMemset(d_level, h->L - 1, N);           // Sweep::new: all cells at level n-1
    p.size = d_size;
    p.volume = d_volume;
    p.density = d_density;
    p.source = d_source;
    p.xhii = d_x;
    p.yneu = d_y;
    p.temperature = d_T;
    p.att = d_att;
    p.previous_rate = d_prev;
    p.change_timescale = d_cts;
    p.species_timestep = d_sdt;
    p.ionization_time = d_ion;
    p.level = d_level;
    p.src_dir = d_src_dir;
  }
  // per-(cell, direction) state, [dir][cell]
  // Compact state of the mixed path (no task records, upwind slots or inverse order;
  // words by task; the geometry kernel): for grids of 2^31 tasks or more, for grids whose
  // full state would not fit in the free device memory (records, slots, schedule, words,
  // rates and the active lists of the levels: ~44 + 4 * faces per cell + 4 * (levels - 1)
  // bytes per task), and on request (SUBSWEEP_COMPACT_STATE=1; SUBSWEEP_TASK_SPACES asks
  // for more task spaces than the grid needs).
  p.num_spaces = 1;
  p.space_d0[0] = 0;
  p.space_d0[1] = D;
  if (h->ops->pull) {
    const uint64_t tasks = (uint64_t)Np * (uint64_t)D;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) (void)cudaGetLastError();
    const double full = (44.0 + 4.0 * (double)E / (double)N + 4.0 * (h->L - 1)) * (double)tasks;
    bool geo = tasks >= kSpaceTasks || (free_b > 0 && full > 0.92 * (double)free_b);
    if (const char* env = std::getenv("SUBSWEEP_COMPACT_STATE")) geo = geo || std::atoi(env) != 0;
    if (geo) {
      int spaces = min_task_spaces(Np, D);
      if (const char* env = std::getenv("SUBSWEEP_TASK_SPACES"))
        spaces = std::max(spaces, std::min(std::atoi(env), std::min(D, swh::kMaxSpaces)));
      p.geo_mode = 1;
      p.num_spaces = spaces;
      for (int sp = 0; sp <= spaces; ++sp) p.space_d0[sp] = D * sp / spaces;
      p.compact_mode = 2;  // every sweep visits every position
      p.pull_variant = 0;
      h->autotune = false;
    }
  }
  // Direction streams (SUBSWEEP_STREAMS=0 turns them off; so does pinning a transport
  // kernel variant, the direction groups of the levelled schedule, the FP64 path's push form
  // or its records).
  if (h->ops->stream_build && !p.geo_mode) {
    h->want_streams = !std::getenv("SUBSWEEP_PULL_VARIANT") && !std::getenv("SUBSWEEP_DIR_GROUPS") &&
                      !std::getenv("SUBSWEEP_FP64_RECORDS") && h->force_path == 0;
    if (const char* env = std::getenv("SUBSWEEP_STREAMS")) {
      h->want_streams = h->want_streams && std::atoi(env) != 0;
      h->force_streams = h->want_streams;
    }
    if (const char* env = std::getenv("SUBSWEEP_STREAM_BYTES")) h->stream_limit = std::strtoull(env, nullptr, 10);
    if (const char* env = std::getenv("SUBSWEEP_STREAM_ARRAYS")) h->stream_allocs_left = std::strtoll(env, nullptr, 10);
    if (h->want_streams) h->parts = closed_parts(grid, 256);
  }
  {
    const size_t nd = (size_t)Np * D;
    const size_t rb = (size_t)h->ops->rate_bytes;
    // push path (FP64): incoming, outgoing, periodic, pending rates and the ready queue;
    // pull path (mixed): incoming and periodic rates and the {q, sweep} words (words
    // indexed by schedule position).
    const bool pull = h->ops->pull;
    char *inc = nullptr, *outg = nullptr, *per = nullptr, *pend = nullptr;
    uint32_t *cnt = nullptr, *queue = nullptr, *order = nullptr;
    unsigned long long* qe = nullptr;
    swk::SweepCtl* ctl = nullptr;
    bool ok = h->alloc(&inc, nd * rb) && h->alloc(&per, nd * rb) && h->alloc(&cnt, nd / 4) &&
              h->alloc(&order, nd) && h->alloc(&ctl, 1);
    uint4* rec = nullptr;
    uint32_t *act_counts = nullptr, *chunk = nullptr, *pos_of_task = nullptr, *act_bits = nullptr;
    uint32_t* cell_sweep = nullptr;
    uint2* cellpack = nullptr;
    float* per_pos = nullptr;
    const size_t chunks = (nd + swk::kCompactChunk - 1) / swk::kCompactChunk + 1;
    if (ok) ok = h->alloc(&chunk, chunks);
    if (ok && pull && p.geo_mode)  // compact state: words by task, no records or inverse order
      ok = h->alloc(&qe, nd) && h->alloc(&act_counts, 32) && h->alloc(&cell_sweep, (size_t)h->Np) &&
           h->alloc(&cellpack, (size_t)h->Np);
    else if (ok && pull)
      ok = h->alloc(&qe, nd) && (h->want_streams || h->alloc(&rec, nd)) && h->alloc(&act_counts, 32) && h->alloc(&pos_of_task, nd) &&
           h->alloc(&act_bits, (nd + 31) / 32) && h->alloc(&cell_sweep, (size_t)h->Np) &&
           h->alloc(&cellpack, (size_t)h->Np) &&
           // per-position periodic sources: only for the staged wavefront kernel (78)
           (p.pull_variant != 78 || h->alloc(&per_pos, (size_t)h->N * h->D + 4));
    if (ok && !pull) ok = h->alloc(&outg, nd * rb) && h->alloc(&pend, nd * rb) && h->alloc(&queue, nd);
    if (!ok) {
      h->fail(SW_ERR_OOM, "device allocation of the transport state (%zu MB) failed",
              (pull ? (p.geo_mode ? 2 * rb + 13 : 2 * rb + 41) : 4 * rb + 9) * nd >> 20);
      return bail(SW_ERR_OOM);
    }
    cudaMemset(inc, 0, nd * rb);
    cudaMemset(per, 0, nd * rb);
    cudaMemset(cnt, 0, nd);
    if (pull) {
      cudaMemset(qe, 0, nd * sizeof(unsigned long long));
      cudaMemset(cell_sweep, 0, (size_t)h->Np * sizeof(uint32_t));
      if (per_pos) cudaMemset(per_pos, 0, ((size_t)h->N * h->D + 4) * sizeof(float));
    } else {
      cudaMemset(outg, 0, nd * rb);
      cudaMemset(pend, 0, nd * rb);
      cudaMemset(queue, 0xff, nd * sizeof(uint32_t));  // every slot empty
    }
    cudaMemset(ctl, 0, sizeof(swk::SweepCtl));
    p.qe = qe;
    p.pull_rec = rec;
    p.act_counts = act_counts;
    p.pos_of_task = pos_of_task;
    p.act_bits = act_bits;
    p.cell_sweep = cell_sweep;
    p.cellpack = cellpack;
    p.per_pos = per_pos;
    p.chunk = chunk;
    p.incoming = inc;
    p.outgoing = outg;
    p.periodic = per;
    p.pending = pend;
    p.counters = cnt;
    p.queue = queue;
    p.order = order;
    p.ctl = ctl;
  }
  ce = cudaDeviceSynchronize();
  if (ce != cudaSuccess) {
    h->cuda_fail(ce, "upload");
    return bail(ce == cudaErrorMemoryAllocation ? SW_ERR_OOM : SW_ERR_CUDA);
  }
  if (swh::launch_level_hist(p, h->stream) != cudaSuccess || sync_ctl(h) != SW_OK) {
    if (h->last_error.empty()) h->fail(SW_ERR_CUDA, "level ordering failed");
    return bail(SW_ERR_CUDA);
  }
  {
    sw_status st = build_schedule(h);
    if (st == SW_OK) st = build_records(h);
    if (st == SW_OK) st = build_push_records(h);
    if (st != SW_OK) return bail(st);
  }
  *out = h;
  return SW_OK;
}

// One step replayed as a CUDA graph: the same launches as sw_step (per sweep: control
// reset, attenuation, dependency counts on the push path, transport, periodic fold,
// chemistry; then the level update and the ionization times), captured once per step
// shape (lowest allowed level before and after, and each sweep's level and kernel
// choice, and with streams whether it takes every cell).  The sweep
// numbers and the end time live in the control block, copied from pinned host memory by
// the graph's first node; the error flag stays set across the step's sweeps, so a stall
// ends the remaining sweeps at once, and is read when the step has finished.  Event
// nodes around each sweep's transport give the transport kernel time.
// Pull path: whether the sweep of `level` runs over the compacted list of its active
// positions (above level 0 with fewer than half of the cells active; SUBSWEEP_COMPACT
// overrides), and that list's buffer, allocated on first use.
static bool pull_sparse(sw_handle* h, int level) {
  const swh::DevicePtrs& p = h->p;
  if (level <= 0 || ((h->no_act_list >> level) & 1u)) return false;
  if (p.compact_mode == 1) return true;
  if (p.compact_mode == 2) return false;
  // Streams: a dense sweep takes the time of all tasks, 23 per ns, a sparse one ~5 per ns of
  // the active ones (128^3 x 84: 7.9 ms dense; sparse 14 ms with 39% of the cells active, the
  // crossing near 20%; 64^3 x 84: 1.03 ms dense, 0.13 ms with 0.2% active).  FP64, whose
  // sparse sweeps pass their changes on to the cells beside: six boxes x 84 0.54 ms dense, 0.45 with
  // 6% active, 0.56 with 9%, 0.88 with 24%; 64^3 x 84 2.2 dense, 3.0 with a third.
  if (p.stream_mode) return (int64_t)h->n_ge_host[level] * (h->ops->pull ? 5 : 10) < h->N;
  return h->n_ge_host[level] * 2 < h->N;
}

// The buffer of the list, allocated on first use (outside of a capture).  Streams: without room for
// it `sparse` becomes false, and the level's sweeps visit every position, now and later; the
// lockstep kernels have no such form.
static sw_status ensure_act_list(sw_handle* h, int level, bool& sparse) {
  if (h->p.act_lv[level]) return SW_OK;
  const size_t tasks = (size_t)h->Np * h->D;
  uint32_t* list = nullptr;
  if (h->p.stream_mode) {
    const size_t allocations = h->allocations.size();
    const int64_t device_bytes = h->device_bytes;
    uint32_t *bits = nullptr, *range = nullptr;
    if (h->stream_alloc(&bits, (tasks + 31) / 32) &&
        h->stream_alloc(&range, 2 * (size_t)h->p.num_streams) && h->stream_alloc(&list, tasks)) {
      h->p.act_bits_lv[level] = bits;
      h->p.act_range[level] = range;
      h->p.act_lv[level] = list;
      return SW_OK;
    }
    (void)cudaGetLastError();
    for (size_t k = allocations; k < h->allocations.size(); ++k) cudaFree(h->allocations[k]);
    h->allocations.resize(allocations);
    h->device_bytes = device_bytes;
    h->no_act_list |= 1u << level;
    sparse = false;
    return SW_OK;
  }
  if (!h->alloc(&list, tasks))
    return h->fail(SW_ERR_OOM, "device allocation of the active positions of level %d failed", level);
  h->p.act_lv[level] = list;
  return SW_OK;
}

static sw_status step_graph(sw_handle* h, double* time_elapsed_out) {
  const swh::PrecisionOps& ops = *h->ops;
  swh::DevicePtrs& p = h->p;
  std::vector<int> levels;
  std::vector<bool> variants;
  uint64_t expected = 0;
  TimestepState after = h->ts;
  after.advance();
  std::vector<int64_t> key = {h->ts.lowest, after.lowest, p.pull_variant};
  for (int level : h->ts.sweep_order()) {
    if (h->n_ge_host[level] == 0) continue;  // Sweep::run_sweeps skips empty levels (mod.rs:262)
    levels.push_back(level);
    expected += (uint64_t)h->n_ge_host[level] * (uint64_t)h->D;
    // pull path: compaction or not; push path: levelled schedule or ready queue
    bool variant;
    if (h->pulls()) {
      variant = pull_sparse(h, level);
      if (variant) {
        sw_status st = ensure_act_list(h, level, variant);  // allocations stay outside the capture
        if (st != SW_OK) return st;
      }
    } else {
      variant = p.num_sched_levels > 0 && (uint64_t)h->n_ge_host[level] * 16 >= (uint64_t)h->N;
      if (h->force_path == 1) variant = p.num_sched_levels > 0;
      if (h->force_path == 2) variant = false;
    }
    variants.push_back(variant);
    // (a sweep of every cell runs another kernel of the streams than one that leaves some out)
    const bool all = (int64_t)h->n_ge_host[level] >= h->N;
    key.push_back(level * 4 + (variant ? 2 : 0) + (p.stream_mode && all ? 1 : 0));
  }
  if (!h->graph_scalars) {
    void* ptr = nullptr;
    SW_CUDA(h, cudaMallocHost(&ptr, sizeof(sw_handle::GraphScalars)), "pinned graph scalars");
    h->graph_scalars = static_cast<sw_handle::GraphScalars*>(ptr);
  }
  if (!h->graph_exec || key != h->graph_key) {
    if (h->graph_exec) {
      cudaGraphExecDestroy(h->graph_exec);
      h->graph_exec = nullptr;
    }
    while (h->graph_ev.size() < 2 * levels.size()) {
      cudaEvent_t e;
      SW_CUDA(h, cudaEventCreate(&e), "event");
      h->graph_ev.push_back(e);
    }
    SW_CUDA(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal), "begin graph capture");
    cudaError_t ce = cudaMemcpyAsync(&p.ctl->epoch_base, h->graph_scalars, sizeof(sw_handle::GraphScalars),
                                     cudaMemcpyHostToDevice, h->stream);
    if (ce == cudaSuccess) ce = cudaMemsetAsync(&p.ctl->error, 0, sizeof(uint32_t), h->stream);
    swh::DevicePtrs q = p;
    q.epoch_base = &p.ctl->epoch_base;
    int64_t kernels = 3;  // level update (two kernels) and ionization times
    uint32_t compacted = 0;  // pull path: levels whose list the step has built so far
    std::vector<int> compact_now(levels.size(), 0);
    for (size_t k = 0; k < levels.size(); ++k) {
      // attenuation, transport, chemistry, the periodic fold, and the counts (push) or
      // the compaction at a sparse level's first sweep (pull)
      kernels += 3 + (p.n_periodic_cells > 0 ? 1 : 0);
      // rates of the cells, gather of a dense sweep, the changes beside a sparse one (FP64)
      if (p.stream_mode) kernels += variants[k] ? (ops.pull ? 1 : 3) : 2;
      // the fold's mark pass after a sweep that leaves cells inactive (pull path)
      if (h->pulls() && p.n_periodic_cells > 0 && h->n_ge_host[levels[k]] < h->N) kernels += 1;
      if (!h->pulls()) {
        kernels += 1;
      } else if (variants[k] && !((compacted >> levels[k]) & 1u)) {
        compact_now[k] = 1;
        compacted |= 1u << levels[k];
        kernels += p.stream_mode ? 5 : 4;
      }
    }
    for (size_t k = 0; k < levels.size() && ce == cudaSuccess; ++k) {
      const int level = levels[k];
      q.epoch = (uint32_t)(k + 1);
      q.active_cells = h->n_ge_host[level];
      q.sweep_level = level;
      q.sparse_sweep = (h->pulls() && variants[k]) ? 1 : 0;
      q.compact_now = compact_now[k];
      ce = cudaMemsetAsync(p.ctl, 0, offsetof(swk::SweepCtl, error), h->stream);
      if (ce == cudaSuccess) ce = ops.attenuation(q, level, h->stream);
      if (ce == cudaSuccess && !h->pulls()) ce = ops.init_counts(q, level, nullptr, !variants[k], h->stream);
      // external records: event nodes that are recorded when the graph runs
      if (ce == cudaSuccess) ce = cudaEventRecordWithFlags(h->graph_ev[2 * k], h->stream, cudaEventRecordExternal);
      if (ce == cudaSuccess) ce = (h->pulls() || variants[k]) ? ops.sweep_levels(q, level, h->stream)
                                                            : ops.sweep(q, level, h->stream);
      if (ce == cudaSuccess) ce = cudaEventRecordWithFlags(h->graph_ev[2 * k + 1], h->stream, cudaEventRecordExternal);
      if (ce == cudaSuccess) ce = ops.fold_periodic(q, h->stream);
      if (ce == cudaSuccess) ce = ops.chemistry(q, level, h->stream);
    }
    if (ce == cudaSuccess) ce = swh::launch_update_levels(p, after.lowest, h->stream);
    if (ce == cudaSuccess) ce = swh::launch_ionization_time(p, 0.0, h->stream, &p.ctl->time);
    cudaGraph_t graph = nullptr;
    const cudaError_t end = cudaStreamEndCapture(h->stream, &graph);
    if (ce == cudaSuccess) ce = end;
    if (ce == cudaSuccess) ce = cudaGraphInstantiate(&h->graph_exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (ce != cudaSuccess) {
      h->graph_exec = nullptr;
      return h->cuda_fail(ce, "graph capture of a step");
    }
    h->graph_key = key;
    h->graph_captures += 1;
    h->graph_kernels = kernels;
  }
  const double elapsed = h->ts.current_max_timestep();
  h->graph_scalars->epoch_base = p.epoch;
  h->graph_scalars->time = h->sim_time + elapsed;
  const unsigned long long tasks_before = h->ctl_host.tasks;
  if (!levels.empty()) p.active_cells = h->n_ge_host[levels.back()];  // of the step's last sweep
  SW_CUDA(h, cudaEventRecord(h->ev[5], h->stream), "event");
  SW_CUDA(h, cudaGraphLaunch(h->graph_exec, h->stream), "graph launch");
  SW_CUDA(h, cudaEventRecord(h->ev[1], h->stream), "event");
  sw_status st = sync_ctl(h);
  if (st != SW_OK) return st;
  p.epoch += (uint32_t)levels.size();
  h->last_epoch = p.epoch;
  const uint32_t err = h->ctl_host.error;
  if (err & (swk::kErrStall | swk::kErrQueue)) {
    // leave the queue empty so the handle stays usable for inspection
    if (p.queue) cudaMemsetAsync(p.queue, 0xff, (size_t)h->Np * h->D * sizeof(uint32_t), h->stream);
    cudaStreamSynchronize(h->stream);
    return h->fail(SW_ERR_STALLED, "a sweep of the step stalled: tasks left unsolved after a %.1f s wait "
                   "(dependency cycle; flags 0x%x)", p.timeout_ns * 1e-9, err);
  }
  if (err & swk::kErrClamp)
    return h->fail(SW_ERR_INVALID_ARG, "x_HII floor above 1 - 1e-10 in the chemistry clamp (reference panics)");
  h->ts = after;
  h->sim_time += elapsed;
  h->act_valid = 0;  // the step's level update changed the active sets
  float step_ms = 0.f;
  cudaEventElapsedTime(&step_ms, h->ev[5], h->ev[1]);
  const int64_t n = (int64_t)levels.size();
  for (int64_t k = 0; k < n; ++k) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, h->graph_ev[2 * k], h->graph_ev[2 * k + 1]) == cudaSuccess)
      h->stats.transport_kernel_ms += ms;
  }
  (void)cudaGetLastError();  // a failed timing query must not surface at the next launch
  h->stats.step_ms += step_ms;
  h->stats.steps += 1;
  h->stats.level_sweeps += n;
  for (bool v : variants) h->stats.levelled_sweeps += (h->pulls() || v) ? 1 : 0;
  h->stats.transport_launches += n;
  h->stats.graph_launches += 1;
  h->stats.kernel_launches += h->graph_kernels;
  h->stats.tasks = (int64_t)h->ctl_host.tasks;
  h->stats.chem_cells = (int64_t)h->ctl_host.chem_cells;
  h->stats.chem_attempts = (int64_t)h->ctl_host.chem_attempts;
  h->stats.chem_failures = (int64_t)h->ctl_host.chem_failures;
  h->stats.transport_attempts = (int64_t)h->ctl_host.attempts;
  h->stats.simulation_time = h->sim_time;
  if (time_elapsed_out) *time_elapsed_out = elapsed;
  const uint64_t solved = h->ctl_host.tasks - tasks_before;
  if (solved != expected)
    return h->fail(SW_ERR_STALLED, "sweep solved %llu of %llu tasks: the dependency graph has a cycle",
                   (unsigned long long)solved, (unsigned long long)expected);
  return SW_OK;
}

sw_status sw_create_batch(const sw_params* params, int32_t n_boxes, const sw_grid_csr* grids,
                          const sw_cell_init* inits, sw_handle** out) {
  if (!out) return create_fail(SW_ERR_INVALID_ARG, "out is NULL");
  *out = nullptr;
  if (!params || !grids || !inits || n_boxes < 1) return create_fail(SW_ERR_INVALID_ARG, "invalid batch arguments");
  int64_t n = 0, e = 0;
  for (int32_t b = 0; b < n_boxes; ++b) {
    const sw_grid_csr& g = grids[b];
    const sw_cell_init& in = inits[b];
    if (g.num_cells < 1 || !g.row_ptr || !g.nbr || !g.kind || !g.area || !g.normal || !g.volume || !g.size ||
        !in.density || !in.ionized_hydrogen_fraction || !in.temperature || !in.source)
      return create_fail(SW_ERR_INVALID_ARG, "box %d: missing array", b);
    if (g.row_ptr[0] != 0 || g.row_ptr[g.num_cells] < 0) return create_fail(SW_ERR_INVALID_ARG, "box %d: bad row_ptr", b);
    // neighbour indices must stay inside the box before they are offset into the union
    for (int64_t f = 0; f < g.row_ptr[g.num_cells]; ++f)
      if (g.kind[f] != SW_FACE_BOUNDARY && (g.nbr[f] < 0 || g.nbr[f] >= g.num_cells))
        return create_fail(SW_ERR_INVALID_ARG, "box %d: face %lld has neighbour %d outside the box", b,
                           (long long)f, g.nbr[f]);
    n += g.num_cells;
    e += g.row_ptr[g.num_cells];
  }
  if (n > (int64_t)INT32_MAX) return create_fail(SW_ERR_UNSUPPORTED, "batch of %lld cells", (long long)n);
  std::vector<int64_t> row_ptr(n + 1);
  std::vector<int32_t> nbr(e);
  std::vector<uint8_t> kind(e);
  std::vector<double> area(e), normal(3 * e), volume(n), size(n), density(n), x(n), t(n), src(n);
  int64_t c0 = 0, f0 = 0;
  for (int32_t b = 0; b < n_boxes; ++b) {
    const sw_grid_csr& g = grids[b];
    const sw_cell_init& in = inits[b];
    const int64_t nb = g.num_cells, eb = g.row_ptr[nb];
    for (int64_t c = 0; c < nb; ++c) row_ptr[c0 + c] = f0 + g.row_ptr[c];
    for (int64_t f = 0; f < eb; ++f) {
      kind[f0 + f] = g.kind[f];
      nbr[f0 + f] = g.kind[f] == SW_FACE_BOUNDARY ? g.nbr[f] : (int32_t)(g.nbr[f] + c0);
    }
    std::copy(g.area, g.area + eb, area.begin() + f0);
    std::copy(g.normal, g.normal + 3 * eb, normal.begin() + 3 * f0);
    std::copy(g.volume, g.volume + nb, volume.begin() + c0);
    std::copy(g.size, g.size + nb, size.begin() + c0);
    std::copy(in.density, in.density + nb, density.begin() + c0);
    std::copy(in.ionized_hydrogen_fraction, in.ionized_hydrogen_fraction + nb, x.begin() + c0);
    std::copy(in.temperature, in.temperature + nb, t.begin() + c0);
    std::copy(in.source, in.source + nb, src.begin() + c0);
    c0 += nb;
    f0 += eb;
  }
  row_ptr[n] = e;
  const sw_grid_csr u = {n, row_ptr.data(), nbr.data(), kind.data(), area.data(), normal.data(), volume.data(),
                         size.data()};
  const sw_cell_init ui = {density.data(), x.data(), t.data(), src.data()};
  return sw_create(params, &u, &ui, out);
}

sw_status sw_step(sw_handle* h, double* time_elapsed_out) {
  if (!h) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  const swh::PrecisionOps& ops = *h->ops;
  SW_DEVICE_SCOPE(h);
  if (h->graph_mode && (h->tuned || !h->autotune)) return step_graph(h, time_elapsed_out);
  uint64_t expected = 0;
  std::vector<int> order = h->ts.sweep_order();
  unsigned long long tasks_before = h->ctl_host.tasks;
  float sweep_ms = 0.f, chem_ms = 0.f, level_ms = 0.f, kernel_ms = 0.f;
  int64_t launches = 0;
  SW_CUDA(h, cudaEventRecord(h->ev[5], h->stream), "event");
  // The sweeps are launched one behind another and looked at when the host waits for them, at
  // the step's end (or after kMaxInFlight, or one by one while variants are tried or traced).
  // A failure that can be foreseen is looked for sweep by sweep, and the first one ends the step:
  // the stall of a grid without a schedule, and a floor that the chemistry refuses.  Otherwise the
  // error flag stays set across the sweeps: after a stall no stream waits any longer, and no kernel
  // changes a cell, its level or its ionization time.
  const bool may_fail = h->p.num_sched_levels == 0 || (h->params.prevent_cooling && h->floor_unsafe);
  SW_CUDA(h, cudaMemsetAsync(&h->p.ctl->error, 0, sizeof(uint32_t), h->stream), "reset error flag");
  struct InFlight {
    int level;
    bool trial;  // of a transport variant
  };
  std::vector<InFlight> in_flight;
  auto look = [&]() -> sw_status {  // the stream has been synchronized
    for (size_t k = 0; k < in_flight.size(); ++k) {
      const auto& ev = h->sweep_ev[k];
      const int level = in_flight[k].level;
      const bool trial = in_flight[k].trial;
      float a = 0.f, b = 0.f, t = 0.f;
      cudaEventElapsedTime(&a, ev[0], ev[3]);
      cudaEventElapsedTime(&b, ev[3], ev[4]);
      cudaEventElapsedTime(&t, ev[1], ev[2]);
      (void)cudaGetLastError();  // timing queries are best effort
      sweep_ms += a;
      chem_ms += b;
      kernel_ms += t;
      if (trial && h->p.stream_mode) {  // the streams have one shape: nothing to choose
        h->tuned = true;
      } else if (trial) {  // one autotuning trial per sweep; the fastest variant per task is kept
        h->tune_ns.push_back(1e6 * t / std::max(1.0, (double)h->n_ge_host[level] * h->D));
        if (++h->tune_index == ops.num_tune_variants) {
          int best = 0;
          for (int i = 1; i < ops.num_tune_variants; ++i)
            if (h->tune_ns[i] < h->tune_ns[best]) best = i;
          h->p.pull_variant = ops.tune_variants[best];
          h->tuned = true;
        }
      }
      if (h->trace) {
        swk::SweepCtl c{};
        h->copy(&c, h->p.ctl, sizeof(c), cudaMemcpyDeviceToHost);
        std::fprintf(stderr,
                     "subsweep sweep level=%d active_tasks=%llu kernel_ms=%.3f transport_ms=%.3f chem_ms=%.3f "
                     "attempts=%llu chem_cells=%llu chem_attempts=%llu\n",
                     level, (unsigned long long)h->n_ge_host[level] * (unsigned long long)h->D, t, a, b,
                     (unsigned long long)c.attempts, (unsigned long long)c.chem_cells,
                     (unsigned long long)c.chem_attempts);
      }
      h->stats.level_sweeps += 1;
      const uint32_t err = h->pinned->error[k];
      if (err & (swk::kErrStall | swk::kErrQueue)) {
        // leave the queue empty so the handle stays usable for inspection
        if (h->p.queue) cudaMemsetAsync(h->p.queue, 0xff, (size_t)h->Np * h->D * sizeof(uint32_t), h->stream);
        cudaStreamSynchronize(h->stream);
        return h->fail(SW_ERR_STALLED,
                       "level %d sweep stalled: tasks left unsolved after a %.1f s wait (dependency cycle; flags 0x%x)",
                       level, h->p.timeout_ns * 1e-9, err);
      }
      if (err & swk::kErrClamp)
        return h->fail(SW_ERR_INVALID_ARG, "x_HII floor above 1 - 1e-10 in the chemistry clamp (reference panics)");
    }
    in_flight.clear();
    return SW_OK;
  };
  for (int level : order) {
    // Sweep::run_sweeps skips levels without active cells (mod.rs:262)
    if (h->n_ge_host[level] == 0) continue;
    expected += (uint64_t)h->n_ge_host[level] * (uint64_t)h->D;
    const size_t slot = in_flight.size();
    if (slot == h->sweep_ev.size()) {
      h->sweep_ev.push_back({});
      for (cudaEvent_t& e : h->sweep_ev.back()) SW_CUDA(h, cudaEventCreate(&e), "event");
    }
    const std::array<cudaEvent_t, 5> ev = h->sweep_ev[slot];
    SW_CUDA(h, cudaMemsetAsync(h->p.ctl, 0, offsetof(swk::SweepCtl, error), h->stream), "reset queue");
    SW_CUDA(h, cudaEventRecord(ev[0], h->stream), "event");
    // Sweeps with at least 1/16 of the cells active walk the precomputed schedule;
    // sparser ones use the dependency-driven queue, which touches only active tasks.
    bool levelled = h->p.num_sched_levels > 0 && (uint64_t)h->n_ge_host[level] * 16 >= (uint64_t)h->N;
    if (h->force_path == 1) levelled = h->p.num_sched_levels > 0;
    if (h->force_path == 2) levelled = false;
    // autotuning trials on dense sweeps only: sparse ones always run the lockstep kernel
    const bool trial = ops.pull && h->autotune && !h->tuned && !pull_sparse(h, level);
    if (trial && !h->p.stream_mode) h->p.pull_variant = ops.tune_variants[h->tune_index];
    if (h->pulls()) {
      levelled = true;  // the pull path always walks the schedule (or the id order)
      h->p.epoch += 1;
      h->last_epoch = h->p.epoch;
      h->p.active_cells = h->n_ge_host[level];
      h->p.sweep_level = level;
      bool sparse = pull_sparse(h, level);
      if (sparse) {
        sw_status st = ensure_act_list(h, level, sparse);
        if (st != SW_OK) return st;
      }
      h->p.sparse_sweep = sparse ? 1 : 0;
      h->p.compact_now = 0;
      if (sparse) {
        if (!((h->act_valid >> level) & 1u)) {  // first sweep of this level in the step
          h->p.compact_now = 1;
          h->act_valid |= 1u << level;
          launches += h->p.stream_mode ? 5 : 4;  // compaction of the active positions
        }
      }
    }
    // after the pull path's sweep number advanced: attenuation records it per solved cell
    SW_CUDA(h, ops.attenuation(h->p, level, h->stream), "attenuation kernel");
    if (!h->pulls()) {
      SW_CUDA(h, ops.init_counts(h->p, level, nullptr, !levelled, h->stream), "init_counts kernel");
      launches += 1;
    }
    SW_CUDA(h, cudaEventRecord(ev[1], h->stream), "event");
    if (levelled) {
      SW_CUDA(h, ops.sweep_levels(h->p, level, h->stream), "levelled sweep kernel");
      h->stats.levelled_sweeps += 1;
    } else {
      SW_CUDA(h, ops.sweep(h->p, level, h->stream), "sweep kernel");
    }
    SW_CUDA(h, cudaEventRecord(ev[2], h->stream), "event");
    SW_CUDA(h, ops.fold_periodic(h->p, h->stream), "periodic fold kernel");
    launches += 3 + (h->p.n_periodic_cells > 0 ? 1 : 0);
    // rates of the cells, gather of a dense sweep, the changes beside a sparse one (FP64)
    if (h->p.stream_mode) launches += h->p.sparse_sweep ? (ops.pull ? 1 : 3) : 2;
    if (h->pulls() && h->p.n_periodic_cells > 0 && h->p.active_cells < h->N) launches += 1;  // fold marks
    SW_CUDA(h, cudaEventRecord(ev[3], h->stream), "event");
    SW_CUDA(h, ops.chemistry(h->p, level, h->stream), "chemistry kernel");
    SW_CUDA(h, cudaEventRecord(ev[4], h->stream), "event");
    SW_CUDA(h, cudaMemcpyAsync(&h->pinned->error[slot], &h->p.ctl->error, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                               h->stream), "read error flag");
    in_flight.push_back({level, trial});
    h->stats.transport_launches += 1;
    if (trial || h->trace || may_fail || (int)in_flight.size() == sw_handle::kMaxInFlight) {
      SW_CUDA(h, cudaStreamSynchronize(h->stream), "level sweep");
      const sw_status st = look();
      if (st != SW_OK) return st;
    }
  }
  // TimestepState bookkeeping and level reassignment (mod.rs:268-270)
  double elapsed = h->ts.current_max_timestep();
  TimestepState after = h->ts;
  after.advance();
  SW_CUDA(h, cudaEventRecord(h->ev[3], h->stream), "event");
  SW_CUDA(h, swh::launch_update_levels(h->p, after.lowest, h->stream), "level kernels");
  h->act_valid = 0;  // levels change: the compacted lists are rebuilt next step
  SW_CUDA(h, cudaEventRecord(h->ev[4], h->stream), "event");
  SW_CUDA(h, swh::launch_ionization_time(h->p, h->sim_time + elapsed, h->stream), "ionization time kernel");
  launches += 3;
  SW_CUDA(h, cudaEventRecord(h->ev[1], h->stream), "event");
  sw_status st = sync_ctl(h);
  if (st != SW_OK) return st;
  st = look();
  if (st != SW_OK) return st;
  h->ts = after;
  h->sim_time += elapsed;
  cudaEventElapsedTime(&level_ms, h->ev[3], h->ev[4]);
  float step_ms = 0.f;
  cudaEventElapsedTime(&step_ms, h->ev[5], h->ev[1]);
  (void)cudaGetLastError();
  h->stats.step_ms += step_ms;
  h->stats.transport_kernel_ms += kernel_ms;
  h->stats.kernel_launches += launches;
  uint64_t solved = h->ctl_host.tasks - tasks_before;
  h->stats.steps += 1;
  h->stats.tasks = (int64_t)h->ctl_host.tasks;
  h->stats.chem_cells = (int64_t)h->ctl_host.chem_cells;
  h->stats.chem_attempts = (int64_t)h->ctl_host.chem_attempts;
  h->stats.chem_failures = (int64_t)h->ctl_host.chem_failures;
  h->stats.transport_attempts = (int64_t)h->ctl_host.attempts;
  h->stats.sweep_ms += sweep_ms;
  h->stats.chem_ms += chem_ms;
  h->stats.level_ms += level_ms;
  h->stats.simulation_time = h->sim_time;
  if (time_elapsed_out) *time_elapsed_out = elapsed;
  if (solved != expected)
    return h->fail(SW_ERR_STALLED, "sweep solved %llu of %llu tasks: the dependency graph has a cycle",
                   (unsigned long long)solved, (unsigned long long)expected);
  return SW_OK;
}

sw_status sw_get_fields(sw_handle* h, double* x, double* T, double* dt, double* rate) {
  if (!h) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  SW_DEVICE_SCOPE(h);
  size_t nb = (size_t)h->N * sizeof(double);
  if (x) SW_CUDA(h, cudaMemcpyAsync(x, h->p.xhii, nb, cudaMemcpyDeviceToHost, h->stream), "copy x");
  if (T) SW_CUDA(h, cudaMemcpyAsync(T, h->p.temperature, nb, cudaMemcpyDeviceToHost, h->stream), "copy T");
  if (dt) SW_CUDA(h, cudaMemcpyAsync(dt, h->p.species_timestep, nb, cudaMemcpyDeviceToHost, h->stream), "copy dt");
  if (rate) {
    SW_CUDA(h, h->ops->photon_rate(h->p, h->last_epoch, h->scratch, h->stream), "photon rate kernel");
    SW_CUDA(h, cudaMemcpyAsync(rate, h->scratch, nb, cudaMemcpyDeviceToHost, h->stream), "copy rate");
  }
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return SW_OK;
}

sw_status sw_get_cell_state(sw_handle* h, double* change_timescale, uint8_t* level, double* ionization_time) {
  if (!h) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  SW_DEVICE_SCOPE(h);
  size_t nb = (size_t)h->N * sizeof(double);
  if (change_timescale)
    SW_CUDA(h, cudaMemcpyAsync(change_timescale, h->p.change_timescale, nb, cudaMemcpyDeviceToHost, h->stream), "copy");
  if (level) SW_CUDA(h, cudaMemcpyAsync(level, h->p.level, h->N, cudaMemcpyDeviceToHost, h->stream), "copy");
  if (ionization_time)
    SW_CUDA(h, cudaMemcpyAsync(ionization_time, h->p.ionization_time, nb, cudaMemcpyDeviceToHost, h->stream), "copy");
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "synchronize");
  return SW_OK;
}

sw_status sw_set_fields(sw_handle* h, const double* x, const double* T) {
  if (!h) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  SW_DEVICE_SCOPE(h);
  size_t nb = (size_t)h->N * sizeof(double);
  if (x) {
    std::vector<double> y(h->N);
    for (int64_t c = 0; c < h->N; ++c) y[c] = 1.0 - x[c];
    h->look_at_floors(x);
    SW_CUDA(h, h->copy(h->p.xhii, x, nb, cudaMemcpyHostToDevice), "copy x");
    SW_CUDA(h, h->copy(h->p.yneu, y.data(), nb, cudaMemcpyHostToDevice), "copy y");
  }
  if (T) SW_CUDA(h, h->copy(h->p.temperature, T, nb, cudaMemcpyHostToDevice), "copy T");
  return SW_OK;
}

sw_status sw_get_level_counts(sw_handle* h, int64_t* per_level) {
  if (!h || !per_level) return SW_ERR_INVALID_ARG;
  for (int l = 0; l < h->L; ++l) per_level[l] = h->n_ge_host[l];
  return SW_OK;
}

sw_status sw_get_dependency_counts(sw_handle* h, int32_t level, uint8_t* counts) {
  if (!h || !counts || level < 0 || level >= h->L) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  SW_DEVICE_SCOPE(h);
  uint8_t* d_counts = nullptr;
  size_t nb = (size_t)h->N * h->D;
  SW_CUDA(h, cudaMalloc(&d_counts, nb), "alloc");
  cudaError_t e = cudaSuccess;
  if (h->p.num_spaces <= 1) {
    // inactive cells' entries are not written by the counting kernel: start from zero
    e = cudaMemsetAsync(d_counts, 0, nb, h->stream);
    if (e == cudaSuccess) e = h->ops->init_counts(h->p, level, d_counts, false, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(counts, d_counts, nb, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  } else {  // task spaces: each space's [cell][its directions] block, interleaved on the host
    std::vector<uint8_t> part;
    for (int sp = 0; sp < h->p.num_spaces && e == cudaSuccess; ++sp) {
      const swh::DevicePtrs v = swh::space_view(h->p, sp);
      const size_t ns = (size_t)h->N * v.D;
      part.resize(ns);
      e = cudaMemsetAsync(d_counts, 0, ns, h->stream);
      if (e == cudaSuccess) e = h->ops->init_counts(v, level, d_counts, false, h->stream);
      if (e == cudaSuccess) e = cudaMemcpyAsync(part.data(), d_counts, ns, cudaMemcpyDeviceToHost, h->stream);
      if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
      const int d0 = h->p.space_d0[sp];
      for (int64_t c = 0; c < h->N && e == cudaSuccess; ++c)
        std::memcpy(counts + (size_t)c * h->D + d0, part.data() + (size_t)c * v.D, v.D);
    }
  }
  cudaFree(d_counts);
  if (e != cudaSuccess) return h->cuda_fail(e, "dependency counts");
  return SW_OK;
}

sw_status sw_get_rates(sw_handle* h, double* incoming, double* outgoing, double* periodic) {
  if (!h) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  SW_DEVICE_SCOPE(h);
  size_t nb = (size_t)h->N * h->D * sizeof(double);
  double* d_out = nullptr;
  SW_CUDA(h, cudaMalloc(&d_out, nb), "alloc");
  double* dsts[3] = {incoming, outgoing, periodic};
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < 3 && e == cudaSuccess; ++i) {
    if (!dsts[i]) continue;
    e = h->ops->export_rates(h->p, i, h->last_epoch, d_out, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dsts[i], d_out, nb, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  }
  cudaFree(d_out);
  if (e != cudaSuccess) return h->cuda_fail(e, "export rates");
  return SW_OK;
}

// Checkpoint layout: a header, then the device arrays of checkpoint_sections in order.
struct CheckpointHeader {
  uint64_t magic;
  uint32_t version, precision;
  int64_t num_cells, num_faces;
  int32_t num_directions, num_levels;
  uint32_t np, rate_bytes;
  double sim_time;
  int32_t ts_lowest, ts_first_done;
  uint32_t epoch, last_epoch;
  uint64_t schedule_hash;  // pull path: fingerprint of the schedule the words are ordered by
};
constexpr uint64_t kCheckpointMagic = 0x3154504357535553ull;  // "SUSWCPT1"
// 2: the mixed path's words (8 bytes, by schedule position) and incoming rates (4 bytes,
// by task) in two sections
constexpr uint32_t kCheckpointVersion = 2;

struct CheckpointSection {
  void* dev;
  size_t bytes;
};

static std::vector<CheckpointSection> checkpoint_sections(sw_handle* h) {
  const swh::DevicePtrs& p = h->p;
  const size_t n = (size_t)h->N, nd = (size_t)h->Np * h->D, rb = (size_t)h->ops->rate_bytes;
  std::vector<CheckpointSection> v = {
      {p.xhii, n * 8},           {p.yneu, n * 8},          {p.temperature, n * 8}, {p.previous_rate, n * 8},
      {p.change_timescale, n * 8}, {p.species_timestep, n * 8}, {p.ionization_time, n * 8}, {p.level, n},
      {p.periodic, nd * rb},
  };
  if (h->ops->pull) {
    v.push_back({p.qe, nd * 8});  // words, by schedule position
    v.push_back({p.incoming, nd * 4});
    v.push_back({p.cell_sweep, n * 4});
  } else {
    v.push_back({p.incoming, nd * rb});
    v.push_back({p.outgoing, nd * rb});
    v.push_back({p.pending, nd * rb});
  }
  return v;
}

// Checkpoints hold the words by position of the levelled schedule and the incoming rates by
// task, whatever the handle's own layout.  Direction streams: the levelled order, from the
// streams' (a stream's segments are its levels), and its fingerprint.
static sw_status levelled_schedule(sw_handle* h, std::vector<uint32_t>& own, std::vector<uint32_t>& order,
                                   uint64_t& fingerprint) {
  const swh::DevicePtrs& p = h->p;
  const uint32_t total = (uint32_t)(h->N * (int64_t)h->D);
  own.resize(total);
  SW_CUDA(h, h->copy(own.data(), p.order, (size_t)total * 4, cudaMemcpyDeviceToHost), "read order");
  std::vector<uint16_t> level((size_t)h->Np * h->D, 0);
  uint32_t depth = 0;
  for (const swk::StreamDesc& s : h->streams) {
    for (uint32_t k = 0; k < s.segs; ++k)
      for (uint32_t i = h->stream_seg[s.seg0 + k]; i < h->stream_seg[s.seg0 + k + 1]; ++i) level[own[i]] = (uint16_t)k;
    depth = std::max(depth, s.segs);
  }
  const int groups = schedule_dir_groups(h->D, total, depth);
  order.resize(total);
  std::vector<uint32_t> seg = {0};
  grouped_level_order(level.data(), h->Np, (uint32_t)h->N, (uint32_t)h->D, depth, groups, order.data(), seg);
  ScheduleHash hash;
  hash.mix(0u);
  hash.mix(1u);
  hash.mix((uint32_t)groups);
  for (uint32_t o : seg) hash.mix(o);
  fingerprint = hash.value;
  return SW_OK;
}

// The rates of a checkpoint, from the streams' layout (by position) or back to it: mixed path
// words by position of the levelled schedule and incoming rates by task, FP64 incoming and
// outgoing rates by task.
static void reorder(char* at, size_t nd, size_t elem, const std::vector<uint32_t>& own,
                    const std::vector<uint32_t>* order, bool save) {
  std::vector<uint32_t> to(own);  // index in the checkpoint of every position
  if (order) {
    std::vector<uint32_t> rank(nd, 0);
    for (size_t i = 0; i < order->size(); ++i) rank[(*order)[i]] = (uint32_t)i;
    for (uint32_t& t : to) t = rank[t];
  }
  const std::vector<char> in(at, at + nd * elem);
  std::memset(at, 0, nd * elem);
  for (size_t i = 0; i < to.size(); ++i)
    std::memcpy(at + (save ? to[i] : i) * elem, in.data() + (save ? i : to[i]) * elem, elem);
}
static void reorder_rates(sw_handle* h, char* end, const std::vector<uint32_t>& own, const std::vector<uint32_t>& order,
                          bool save) {
  const size_t nd = (size_t)h->Np * h->D;
  if (h->ops->pull) {  // the sections before the last
    char* words = end - (size_t)h->N * 4 - nd * 12;
    reorder(words, nd, 8, own, &order, save);
    reorder(words + nd * 8, nd, 4, own, nullptr, save);
  } else {
    reorder(end - 3 * nd * 8, nd, 8, own, nullptr, save);
    reorder(end - 2 * nd * 8, nd, 8, own, nullptr, save);
    std::memset(end - nd * 8, 0, nd * 8);  // no pending rates: the last sweep's changes are there
  }
}

static size_t checkpoint_bytes(sw_handle* h) {
  size_t total = sizeof(CheckpointHeader);
  for (const CheckpointSection& s : checkpoint_sections(h)) total += s.bytes;
  return total;
}

// The per-cell level bytes follow seven per-cell double arrays (checkpoint_sections).
static size_t checkpoint_level_offset(int64_t num_cells) {
  return sizeof(CheckpointHeader) + 7 * (size_t)num_cells * sizeof(double);
}

// Checkpoint length implied by a header's counts, in the order of checkpoint_sections;
// 0 for counts no handle can have.
static size_t checkpoint_bytes_for(const CheckpointHeader& hd) {
  if (hd.num_cells < 1 || hd.num_cells >= ((int64_t)1 << 30) || hd.num_directions < 1 ||
      hd.num_directions > swk::kMaxDirections || hd.num_levels < 1 || hd.num_levels > 16 ||
      (int64_t)hd.np < hd.num_cells || (hd.rate_bytes != 4 && hd.rate_bytes != 8) ||
      (hd.precision != SW_PRECISION_FP64 && hd.precision != SW_PRECISION_MIXED))
    return 0;
  const size_t n = (size_t)hd.num_cells, nd = (size_t)hd.np * (size_t)hd.num_directions, rb = hd.rate_bytes;
  size_t total = checkpoint_level_offset(hd.num_cells) + n + nd * rb;
  total += hd.precision == SW_PRECISION_MIXED ? nd * 12 + n * 4 : 3 * nd * rb;
  return total;
}

// Header, length and level checks of a checkpoint buffer, before any byte of it reaches
// the device: a level >= num_levels would index past the per-level histograms.
static int32_t check_checkpoint(const void* buffer, size_t bytes, CheckpointHeader* hd_out) {
  if (bytes < sizeof(CheckpointHeader)) return 2;
  CheckpointHeader hd;
  std::memcpy(&hd, buffer, sizeof(hd));
  if (hd_out) *hd_out = hd;
  if (hd.magic != kCheckpointMagic || hd.version != kCheckpointVersion) return 1;
  const size_t need = checkpoint_bytes_for(hd);
  if (need == 0 || hd.ts_lowest < 0 || hd.ts_lowest >= hd.num_levels) return 1;
  if (bytes < need) return 2;
  const uint8_t* level = static_cast<const uint8_t*>(buffer) + checkpoint_level_offset(hd.num_cells);
  for (int64_t c = 0; c < hd.num_cells; ++c)
    if (level[c] >= hd.num_levels) return 3;
  return 0;
}

int64_t sw_host_schedule_order(const uint16_t* task_level, uint32_t np, uint32_t n, uint32_t d, int32_t levels,
                                int32_t groups, uint32_t* order, uint32_t* seg, int64_t seg_cap) {
  if (!task_level || !order || !seg || n == 0 || np < n || d == 0 || levels < 1 || groups < 1 ||
      groups > (int32_t)d || (uint64_t)np * d >= (1ull << 32))
    return -1;
  for (uint64_t t = 0; t < (uint64_t)np * d; ++t)
    if (t % np < n && task_level[t] >= levels) return -1;
  std::vector<uint32_t> s = {0};
  grouped_level_order(task_level, np, n, d, (size_t)levels, groups, order, s);
  for (size_t i = 0; i < s.size() && (int64_t)i < seg_cap; ++i) seg[i] = s[i];
  return (int64_t)s.size() - 1;
}

int64_t sw_host_stream_plan(const uint16_t* task_level, const uint8_t* up, uint32_t np, uint32_t n, uint32_t d,
                            const uint32_t* parts, uint32_t num_parts, uint32_t* order, int64_t* plan, int64_t plan_cap) {
  if (!task_level || !up || !parts || !order || !plan || n == 0 || np < n || d == 0 || num_parts == 0 ||
      parts[0] != 0 || parts[num_parts] != n || (uint64_t)np * d >= (1ull << 32))
    return -1;
  std::vector<uint32_t> seg;
  std::vector<swk::StreamDesc> streams;
  std::vector<std::vector<uint8_t>> gmax;
  stream_order(task_level, up, np, n, d, std::vector<uint32_t>(parts, parts + num_parts + 1), order, seg, streams, gmax);
  int64_t rows = 0;
  for (size_t s = 0; s < streams.size(); ++s) {
    std::vector<swk::StreamGroup> groups(gmax[s].size());
    plan_stream(streams[s], seg.data(), gmax[s], groups.data());
    for (const swk::StreamGroup& g : groups) {
      if (rows < plan_cap) {
        const int64_t row[5] = {(int64_t)s, g.pos, g.need, (g.shape & 31u) + 1, g.shape >> 5};
        std::copy(row, row + 5, plan + 5 * rows);
      }
      ++rows;
    }
  }
  return rows;
}

int32_t sw_host_task_spaces(uint32_t np, int32_t d) {
  if (np == 0 || d < 1) return -1;
  return min_task_spaces(np, d);
}

int32_t sw_host_dir_groups(int32_t d, uint64_t tasks, int64_t levels) {
  if (d < 1 || levels < 1) return -1;
  return schedule_dir_groups(d, tasks, (size_t)levels);
}

int32_t sw_host_check_checkpoint(const void* buffer, size_t bytes) {
  if (!buffer) return 1;
  return check_checkpoint(buffer, bytes, nullptr);
}

sw_status sw_checkpoint_size(sw_handle* h, size_t* bytes) {
  if (!h || !bytes) return SW_ERR_INVALID_ARG;
  *bytes = checkpoint_bytes(h);
  return SW_OK;
}

sw_status sw_save_state(sw_handle* h, void* buffer, size_t bytes) try {
  if (!h || !buffer) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  if (bytes < checkpoint_bytes(h)) return h->fail(SW_ERR_INVALID_ARG, "checkpoint buffer too small");
  SW_DEVICE_SCOPE(h);
  CheckpointHeader hd{};
  hd.magic = kCheckpointMagic;
  hd.version = kCheckpointVersion;
  hd.precision = (uint32_t)h->params.precision;
  hd.num_cells = h->N;
  hd.num_faces = h->E;
  hd.num_directions = h->D;
  hd.num_levels = h->L;
  hd.np = h->Np;
  hd.rate_bytes = (uint32_t)h->ops->rate_bytes;
  hd.sim_time = h->sim_time;
  hd.ts_lowest = h->ts.lowest;
  hd.ts_first_done = h->ts.first_done ? 1 : 0;
  hd.epoch = h->ops->pull ? h->p.epoch : 0u;
  hd.last_epoch = h->ops->pull ? h->last_epoch : 0u;
  hd.schedule_hash = h->ops->pull ? h->schedule_hash : 0;
  std::vector<uint32_t> own, order;
  if (h->p.stream_mode) {
    uint64_t schedule = 0;
    const sw_status st = levelled_schedule(h, own, order, schedule);
    if (st != SW_OK) return st;
    if (h->ops->pull) hd.schedule_hash = schedule;
  }
  char* out = static_cast<char*>(buffer);
  std::memcpy(out, &hd, sizeof(hd));
  size_t off = sizeof(hd);
  for (const CheckpointSection& s : checkpoint_sections(h)) {
    SW_CUDA(h, cudaMemcpyAsync(out + off, s.dev, s.bytes, cudaMemcpyDeviceToHost, h->stream), "save state");
    off += s.bytes;
  }
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "save state");
  if (h->p.stream_mode) reorder_rates(h, out + off, own, order, true);
  return SW_OK;
} catch (const std::bad_alloc&) {  // the streams' rates are reordered on the host
  return h->fail(SW_ERR_OOM, "no host memory to reorder the checkpoint's rates");
}

sw_status sw_load_state(sw_handle* h, const void* buffer, size_t bytes) try {
  if (!h || !buffer) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  CheckpointHeader hd{};
  const int32_t check = check_checkpoint(buffer, bytes, &hd);
  if (check == 2 && bytes < sizeof(CheckpointHeader))
    return h->fail(SW_ERR_INVALID_ARG, "checkpoint buffer too small");
  if (hd.magic != kCheckpointMagic || hd.version != kCheckpointVersion) return h->fail(SW_ERR_INVALID_ARG, "not a checkpoint");
  if (hd.precision != (uint32_t)h->params.precision || hd.num_cells != h->N || hd.num_faces != h->E ||
      hd.num_directions != h->D || hd.num_levels != h->L || hd.np != h->Np ||
      hd.rate_bytes != (uint32_t)h->ops->rate_bytes)
    return h->fail(SW_ERR_INVALID_ARG, "checkpoint was written by a handle with another grid, parameters or precision");
  if (checkpoint_bytes_for(hd) != checkpoint_bytes(h))
    return h->fail(SW_ERR_INVALID_ARG, "checkpoint layout does not match this handle");
  std::vector<uint32_t> own, order;
  uint64_t schedule = h->schedule_hash;
  if (h->p.stream_mode) {
    SW_DEVICE_SCOPE(h);
    const sw_status st = levelled_schedule(h, own, order, schedule);
    if (st != SW_OK) return st;
  }
  if (h->ops->pull && hd.schedule_hash != schedule)
    return h->fail(SW_ERR_INVALID_ARG, "checkpoint was written with another transport schedule (direction groups)");
  if (check == 1) return h->fail(SW_ERR_INVALID_ARG, "corrupt checkpoint header");
  if (check == 2) return h->fail(SW_ERR_INVALID_ARG, "checkpoint buffer too small");
  if (check == 3) return h->fail(SW_ERR_INVALID_ARG, "corrupt checkpoint: a cell's timestep level is out of range");
  SW_DEVICE_SCOPE(h);
  const char* in = static_cast<const char*>(buffer);
  std::vector<char> reordered;
  if (h->p.stream_mode) {
    reordered.assign(in, in + checkpoint_bytes(h));
    in = reordered.data();
    reorder_rates(h, reordered.data() + reordered.size(), own, order, false);
  }
  size_t off = sizeof(hd);
  for (const CheckpointSection& s : checkpoint_sections(h)) {
    if (s.dev == h->p.xhii) {
      std::vector<double> x(h->N);
      std::memcpy(x.data(), in + off, s.bytes);
      h->look_at_floors(x.data());
    }
    SW_CUDA(h, cudaMemcpyAsync(s.dev, in + off, s.bytes, cudaMemcpyHostToDevice, h->stream), "load state");
    off += s.bytes;
  }
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "load state");
  if (h->p.num_pairs)
    SW_CUDA(h, cudaMemsetAsync(h->p.stream_flags, 0xff, (size_t)h->p.num_pairs * 4, h->stream), "load state");
  h->p.active_cells = 0;  // incoming rates of some cells may be out of date (mixed path)
  if (h->p.stream_mode && !h->ops->pull)  // no sweep is stamped
    SW_CUDA(h, cudaMemsetAsync(h->p.queue, 0xff, (size_t)h->Np * h->D * 4, h->stream), "load state");
  h->sim_time = hd.sim_time;
  h->ts.lowest = hd.ts_lowest;
  h->ts.first_done = hd.ts_first_done != 0;
  h->p.epoch = hd.epoch;
  h->last_epoch = hd.last_epoch;
  // pull path: the periodic sources by schedule position follow from the restored words
  // (between steps the periodic array is the fold of the current words, so this
  // rewrites it unchanged)
  if (h->ops->pull) {
    swh::DevicePtrs q = h->p;
    q.active_cells = h->N;  // every entry
    SW_CUDA(h, h->ops->fold_periodic(q, h->stream), "periodic fold kernel");
  }
  // cells per level for the next step (an earlier step's failure is over)
  h->act_valid = 0;
  SW_CUDA(h, cudaMemsetAsync(&h->p.ctl->error, 0, sizeof(uint32_t), h->stream), "reset error flag");
  SW_CUDA(h, swh::launch_level_hist(h->p, h->stream), "level histogram");
  return sync_ctl(h);
} catch (const std::bad_alloc&) {  // the streams' rates are reordered on the host
  return h->fail(SW_ERR_OOM, "no host memory to reorder the checkpoint's rates");
}

sw_status sw_get_time_series(sw_handle* h, sw_time_series* out) {
  if (!h || !out) return SW_ERR_INVALID_ARG;
  h->last_error.clear();
  SW_DEVICE_SCOPE(h);
  if (!h->series_dev && !h->alloc(&h->series_dev, swh::kTimeSeriesPartials + 8))
    return h->fail(SW_ERR_OOM, "device allocation of the time-series buffer failed");
  double* partial = h->series_dev;
  double* out6 = h->series_dev + swh::kTimeSeriesPartials;
  SW_CUDA(h, h->ops->cell_rates(h->p, h->last_epoch, h->scratch, h->stream), "cell rate kernel");
  SW_CUDA(h, swh::launch_time_series(h->p, h->scratch, h->ops->carry_neutral, partial, out6, h->stream),
          "time series kernels");
  double v[6];
  SW_CUDA(h, cudaMemcpyAsync(v, out6, sizeof(v), cudaMemcpyDeviceToHost, h->stream), "read time series");
  SW_CUDA(h, cudaStreamSynchronize(h->stream), "time series");
  out->hydrogen_ionization_mass_average = v[0];
  out->hydrogen_ionization_volume_average = v[1];
  out->temperature_mass_average = v[2];
  out->temperature_volume_average = v[3];
  out->photoionization_rate_volume_average = v[4];
  out->weighted_photoionization_rate_volume_average = v[5];
  return SW_OK;
}

sw_status sw_get_stats(sw_handle* h, sw_stats* out) {
  if (!h || !out) return SW_ERR_INVALID_ARG;
  h->stats.schedule_levels = h->stats_schedule_levels;
  h->stats.upwind_slots = h->stats_upwind_slots;
  h->stats.pull_variant =
      h->ops->pull && !h->p.geo_mode ? (h->p.pull_variant > 0 ? h->p.pull_variant : swh::kDefaultPullVariant) : 0;
  h->stats.task_spaces = h->p.geo_mode ? h->p.num_spaces : 0;
  h->stats.device_bytes = h->device_bytes;
  *out = h->stats;
  return SW_OK;
}

const char* sw_last_error(const sw_handle* h) {
  if (!h) return g_create_error.c_str();
  return h->last_error.c_str();
}

void sw_destroy(sw_handle* h) {
  if (!h) return;
  swh::DeviceScope device_scope(h->device);  // frees on the handle's device
  cudaStreamSynchronize(h->stream);
  delete h;
}

}  // extern "C"

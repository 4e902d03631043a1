// Launchers of the precision-dependent kernels.  Included once by sweep_fp64.cu
// (R = double, reference-exact neutral fraction) and once by sweep_mixed.cu
// (R = float, carried neutral fraction); each defines SWK_R, SWK_CARRY and SWK_OPS.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "launch.h"
#include "sweep_compact.cuh"
#include "sweep_device.cuh"
#include "sweep_stream.cuh"
#if SWK_PULL
#include "sweep_pull.cuh"
#include "sweep_pull_setup.cuh"
#include "sweep_pull_lockstep.cuh"
#include "sweep_pull_wavefront.cuh"
#include "sweep_pull_geometry.cuh"
#include "sweep_pull_fold.cuh"
#else
#include "sweep_push_records.cuh"
#include "sweep_stream_fp64.cuh"
#endif

namespace swh {
namespace {

using R = SWK_R;
constexpr bool kCarry = SWK_CARRY;

swk::SweepArgs<R> sweep_args(const DevicePtrs& p, int level) {
  swk::SweepArgs<R> a;
  a.off = p.off;
  a.geo32 = static_cast<const float4*>(p.geo32);
  a.geo64 = static_cast<const swk::Geo64*>(p.geo64);
  a.nbr = p.nbr;
  a.dir64 = p.dir64;
  a.dir32 = p.dir32;
  a.D = p.D;
  a.Np = p.Np;
  a.N = (uint32_t)p.num_cells;
  a.guard = p.guard;
  a.level = p.level;
  a.src_dir = static_cast<const R*>(p.src_dir);
  a.att = p.att;
  a.threshold = (R)(p.threshold / p.rate_scale);
  a.incoming = static_cast<R*>(p.incoming);
  a.outgoing = static_cast<R*>(p.outgoing);
  a.periodic = static_cast<R*>(p.periodic);
  a.pending = static_cast<R*>(p.pending);
  a.counters = p.counters;
  a.queue = p.queue;
  a.ctl = p.ctl;
  a.current_level = level;
  a.timeout_ns = p.timeout_ns;
  return a;
}

int grid_for(int64_t work, int block) {
  int64_t g = (work + block - 1) / block;
  if (g < 1) g = 1;
  if (g > 152 * 32) g = 152 * 32;
  return (int)g;
}

// The compacted list of the level's active positions: mark the active cells' positions,
// then compact the bitmap.
cudaError_t compact_active(const DevicePtrs& p, int level, cudaStream_t s) {
  uint32_t* act = p.act_lv[level];
  uint32_t* cnt = p.act_counts + level;
  if (!act) return cudaErrorInvalidValue;
  if (!p.compact_now) return cudaSuccess;
  const uint32_t words = (uint32_t)((p.num_cells * p.D + 31) / 32);
  const uint32_t nb = (words + swk::kBitsThreads - 1) / swk::kBitsThreads;
  uint32_t* bits = p.stream_mode ? p.act_bits_lv[level] : p.act_bits;
  cudaError_t e = cudaMemsetAsync(bits, 0, (size_t)words * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  swk::k_mark_active<<<grid_for(p.num_cells, 256), 256, 0, s>>>(p.level, level, (uint32_t)p.num_cells, p.D, p.Np,
                                                                  p.pos_of_task, bits);
  swk::k_bits_count<<<nb, swk::kBitsThreads, 0, s>>>(bits, words, p.chunk);
  swk::k_compact_scan<<<1, swk::kScanThreads, 0, s>>>(p.chunk, nb, cnt);
  swk::k_bits_scatter<<<nb, swk::kBitsThreads, 0, s>>>(bits, words, p.chunk, act);
  if (p.stream_mode)
    swk::k_stream_act_range<<<grid_for((int64_t)p.num_streams * 64, 256), 256, 0, s>>>(
        bits, p.chunk, static_cast<const swk::StreamDesc*>(p.streams), p.num_streams, (uint32_t)(p.num_cells * p.D),
        cnt, p.act_range[level]);
  return cudaGetLastError();
}

swk::StreamShape stream_shape(const DevicePtrs& p) {
  return {p.stream_shape[0], p.stream_shape[1], p.stream_shape[2],
          p.stream_shape[3], p.stream_shape[4], p.stream_shape[5]};
}

swk::StreamArgs<R> stream_args(const DevicePtrs& p) {
  swk::StreamArgs<R> a{};
  a.streams = static_cast<const swk::StreamDesc*>(p.streams);
  a.groups = static_cast<const swk::StreamGroup*>(p.stream_groups);
  a.data = p.stream_data;
  a.bytes = p.stream_bytes;
  a.evict_first = p.stream_bytes > (64ull << 20);
  a.seg_group = p.seg_group;
#if SWK_PULL
  a.word = p.qe;
#else
  a.word = static_cast<double*>(p.pending);
  a.out = static_cast<double*>(p.outgoing);
  a.stamp = p.queue;
#endif
  a.inc = static_cast<R*>(p.incoming);
  a.threshold = (R)(p.threshold / p.rate_scale);
  a.ctl = p.ctl;
  a.timeout_ns = p.timeout_ns;
  a.epoch = p.epoch;
  a.epoch_base = p.epoch_base;
  a.shape = stream_shape(p);
  a.seg = p.lvl;
  a.order = p.order;
  a.cell_att = static_cast<const R*>(p.cell_att);
  a.periodic = static_cast<const R*>(p.periodic);
  a.Np = p.Np;
  a.parts = static_cast<const swk::StreamPart*>(p.stream_parts);
  a.part0 = p.stream_part0;
  a.flags = p.stream_flags;
  return a;
}

template <int W>
cudaError_t launch_stream(const DevicePtrs& p, bool all, cudaStream_t s) {
  const swk::StreamArgs<R> a = stream_args(p);
  const size_t smem = swk::stream_smem_bytes<R>(a.shape);
  auto fn = a.shape.far ? (all ? swk::k_sweep_stream<R, W, true, true> : swk::k_sweep_stream<R, W, true, false>)
                        : (all ? swk::k_sweep_stream<R, W, false, true> : swk::k_sweep_stream<R, W, false, false>);
  cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  fn<<<p.num_streams, 32 * W, smem, s>>>(a);
  return cudaGetLastError();
}

// Pairs of blocks: clusters of two, no more than can be resident at once.
using PairKernel = void (*)(const swk::StreamArgs<R>);
PairKernel pair_kernel(bool far, bool all) {
  constexpr int W = swk::kPairWarps;
  return far ? (all ? swk::k_sweep_stream<R, W, true, true, true> : swk::k_sweep_stream<R, W, true, false, true>)
             : (all ? swk::k_sweep_stream<R, W, false, true, true> : swk::k_sweep_stream<R, W, false, false, true>);
}
cudaError_t pair_config(const DevicePtrs& p, PairKernel fn, cudaLaunchConfig_t* c, cudaLaunchAttribute* at) {
  const size_t smem = swk::stream_smem_bytes<R>(stream_shape(p));
  c->blockDim = dim3(32 * (swk::kPairWarps + 1));
  c->dynamicSmemBytes = smem;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {2, 1, 1};
  c->attrs = at;
  c->numAttrs = 1;
  return cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}
cudaError_t stream_pairs(const DevicePtrs& p, int* pairs) {
  cudaLaunchConfig_t c{};
  cudaLaunchAttribute at[1];
  const PairKernel fn = pair_kernel(true, true);
  cudaError_t e = pair_config(p, fn, &c, at);
  if (e != cudaSuccess) return e;
  c.gridDim = dim3(2);
  return cudaOccupancyMaxActiveClusters(pairs, (const void*)fn, &c);
}
cudaError_t launch_pairs(const DevicePtrs& p, bool all, cudaStream_t s) {
  cudaLaunchConfig_t c{};
  cudaLaunchAttribute at[1];
  const swk::StreamArgs<R> a = stream_args(p);
  const PairKernel fn = pair_kernel(a.shape.far != 0, all);
  cudaError_t e = pair_config(p, fn, &c, at);
  if (e != cudaSuccess) return e;
  c.gridDim = dim3(2 * p.num_pairs);
  c.stream = s;
  return cudaLaunchKernelEx(&c, fn, a);
}

cudaError_t sweep_stream(const DevicePtrs& p, int level, cudaStream_t s) {
  if (p.sparse_sweep) {
    cudaError_t e = compact_active(p, level, s);
    if (e != cudaSuccess) return e;
    swk::StreamArgs<R> a = stream_args(p);
    a.act = p.act_lv[level];
    a.act_range = p.act_range[level];
    a.act_bits = p.act_bits_lv[level];
    swk::k_sweep_stream_sparse<R><<<p.num_streams, swk::kStreamSparseThreads, 0, s>>>(a);
#if !SWK_PULL
    swk::k_cells_near64<<<grid_for(p.num_cells, 256), 256, 0, s>>>((uint32_t)p.num_cells, p.level, level, p.off, p.nbr,
                                                                    p.stale);
    const int y = std::max(8, (int)(16 * p.num_sms / std::max(1u, p.num_streams)));
    swk::k_stream_take64<<<dim3(p.num_streams, y), 256, 0, s>>>(a, p.stale);
#endif
    return cudaGetLastError();
  }
  swk::k_stream_gather<R><<<grid_for((int64_t)p.num_groups * 32, 256), 256, 0, s>>>(
      static_cast<const swk::StreamGroup*>(p.stream_groups), p.num_groups, p.stream_data, p.order, p.Np,
      static_cast<const R*>(p.cell_att), static_cast<const R*>(p.periodic));
  const bool all = p.active_cells >= p.num_cells;
  if (p.stream_shape[5] == 2) return launch_pairs(p, all, s);
  switch (p.stream_shape[3]) {
    case 4: return launch_stream<4>(p, all, s);
    case 8: return launch_stream<8>(p, all, s);
    case 16: return launch_stream<16>(p, all, s);
    default: return cudaErrorInvalidValue;  // (the layout goes by the number of warps)
  }
}

// Incoming rates of every cell as after the last sweep, before they are exported: a sweep of the
// mixed path leaves those of its inactive cells as they were.
cudaError_t refresh(const DevicePtrs& p, cudaStream_t s) {
#if SWK_PULL
  if (!p.stream_mode || p.active_cells >= p.num_cells) return cudaSuccess;
  swk::k_stream_stale<<<grid_for(p.num_cells, 256), 256, 0, s>>>((uint32_t)p.num_cells, p.off, p.nbr, p.cell_sweep,
                                                                  p.stale);
  const int y = std::max(8, (int)(8 * p.num_sms / std::max(1u, p.num_streams)));
  swk::k_stream_refresh<<<dim3(p.num_streams, y), 256, 0, s>>>(stream_args(p), p.stale);
#endif
  return cudaGetLastError();
}

// positions of the tasks' rates, or null where they lie by task
const uint32_t* rate_pos(const DevicePtrs& p) { return p.stream_mode ? p.pos_of_task : nullptr; }

// exports of the rates as they are stored (the push form's, and the streams' once brought up to date)
cudaError_t photon_rate_stored(const DevicePtrs& p, double* out, cudaStream_t s) {
  const cudaError_t e = refresh(p, s);
  if (e != cudaSuccess) return e;
  swk::k_photon_rate<R><<<grid_for(p.num_cells, 128), 128, 0, s>>>(
      (uint32_t)p.num_cells, static_cast<const R*>(p.incoming), rate_pos(p), p.D, p.Np, p.rate_scale, out);
  return cudaGetLastError();
}

cudaError_t cell_rates_stored(const DevicePtrs& p, double* out, cudaStream_t s) {
  const cudaError_t e = refresh(p, s);
  if (e != cudaSuccess) return e;
  swk::k_cell_rates<R><<<grid_for(p.num_cells, 256), 256, 0, s>>>(
      (uint32_t)p.num_cells, static_cast<const R*>(p.incoming), rate_pos(p), static_cast<const R*>(p.periodic),
      static_cast<const R*>(p.src_dir), p.D, p.Np, p.rate_scale, out);
  return cudaGetLastError();
}

cudaError_t export_rates_stored(const DevicePtrs& p, int which, double* out, cudaStream_t s) {
  const cudaError_t e = which == 0 ? refresh(p, s) : cudaSuccess;
  if (e != cudaSuccess) return e;
  const void* src = which == 0 ? p.incoming : (which == 1 ? p.outgoing : p.periodic);
  swk::k_export_rates<R><<<grid_for(p.num_cells * p.D, 256), 256, 0, s>>>(
      (uint32_t)p.num_cells, static_cast<const R*>(src), which == 2 ? nullptr : rate_pos(p), p.D, p.Np, p.rate_scale,
      out);
  return cudaGetLastError();
}

cudaError_t occupancy(int* blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, swk::k_sweep<R>, swk::kSweepThreads, 0);
}

// Whether the handle runs the staged wavefront kernel (pull variant 78), whose
// per-position periodic sources the fold then maintains.  The variant of a handle is
// fixed at creation (the autotuner's candidates do not include it).
bool staged_inputs(const DevicePtrs& p) {
  if (!p.per_pos) return false;
  int v = p.pull_variant;
  if (v <= 0)
    if (const char* env = std::getenv("SUBSWEEP_PULL_VARIANT")) v = std::atoi(env);
  return v == 78;
}

cudaError_t attenuation(const DevicePtrs& p, int level, cudaStream_t s) {
  swk::k_attenuation<kCarry, R><<<grid_for(p.num_cells, 256), 256, 0, s>>>(
      (uint32_t)p.num_cells, p.level, level, p.density, p.xhii, p.yneu, p.size, p.att, p.cell_sweep,
      p.epoch_base, p.epoch, static_cast<uint2*>(p.cellpack), static_cast<const float*>(p.src_dir),
      static_cast<R*>(p.cell_att));
  return cudaGetLastError();
}

cudaError_t init_counts(const DevicePtrs& p, int level, uint8_t* debug_counts, bool enqueue, cudaStream_t s) {
  swk::SweepArgs<R> a = sweep_args(p, level);
  swk::DirParam dirs;
  for (int i = 0; i < 3 * p.D; ++i) dirs.v[i] = p.dir32_host[i];
  const unsigned long long capacity = enqueue ? (unsigned long long)p.D * p.Np : 0ull;
  const int blocks = (int)((p.num_cells + swk::kCountThreads - 1) / swk::kCountThreads);
  swk::k_init_counts<R><<<blocks, swk::kCountThreads, 0, s>>>(a, dirs, capacity, debug_counts);
  return cudaGetLastError();
}

cudaError_t sweep(const DevicePtrs& p, int level, cudaStream_t s) {
  swk::SweepArgs<R> a = sweep_args(p, level);
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel((const void*)swk::k_sweep<R>, dim3(p.coop_blocks), dim3(swk::kSweepThreads),
                                     args, 0, s);
}

cudaError_t occupancy_levels(int* blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, swk::k_sweep_sched<R>, swk::kLevelThreads, 0);
}

// The levelled push transport: over the precomputed downwind fractions when the grid
// has them, else computing the geometry on the fly.
cudaError_t sweep_levels(const DevicePtrs& p, int level, cudaStream_t s) {
  swk::SweepArgs<R> a = sweep_args(p, level);
  uint32_t total = (uint32_t)(p.num_cells * p.D);
#if !SWK_PULL
  if (p.stream_mode) return sweep_stream(p, level, s);
  if (p.push_rec) {
    const uint4* rec = static_cast<const uint4*>(p.push_rec);
    const uint32_t* tgt = p.push_tgt;
    const double* frac = p.push_frac;
    int bps = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, swk::k_sweep_sched_rec<R>,
                                                                  swk::kLevelThreads, 0);
    if (e != cudaSuccess) return e;
    if (p.level_bps_cap >= 1 && p.level_bps_cap < bps) bps = p.level_bps_cap;
    void* args[] = {&a, &rec, &total, &tgt, &frac};
    return cudaLaunchCooperativeKernel((const void*)swk::k_sweep_sched_rec<R>, dim3(bps * p.num_sms),
                                       dim3(swk::kLevelThreads), args, 0, s);
  }
#endif
  const uint32_t* order = p.order;
  void* args[] = {&a, &order, &total};
  return cudaLaunchCooperativeKernel((const void*)swk::k_sweep_sched<R>, dim3(p.level_blocks),
                                     dim3(swk::kLevelThreads), args, 0, s);
}

#if !SWK_PULL
// push path, once per grid: phase 0 writes the records' counts and the 64-bit scan of
// the chunk totals into `scratch` (total at scratch[num_chunks]); phase 1, with
// push_tgt / push_frac allocated, the offsets and the slots.
cudaError_t push_records(const DevicePtrs& p, int phase, unsigned long long* scratch, cudaStream_t s) {
  swk::SweepArgs<R> a = sweep_args(p, 0);
  uint4* rec = static_cast<uint4*>(p.push_rec);
  const uint32_t total = (uint32_t)(p.num_cells * p.D);
  const uint32_t nc = (total + swk::kCompactChunk - 1) / swk::kCompactChunk;
  if (phase == 0) {
    swk::k_push_rec_count<R><<<grid_for(p.num_cells * p.D, 256), 256, 0, s>>>(a, p.order, total, rec);
    swk::k_push_chunk_sums<R><<<nc, swk::kCompactThreads, 0, s>>>(rec, total, p.chunk);
    swk::k_push_scan64<R><<<1, 1024, 0, s>>>(p.chunk, nc, scratch);
  } else {
    swk::k_push_slots<R><<<nc, swk::kCompactThreads, 0, s>>>(a, rec, total, scratch, p.push_tgt, p.push_frac);
  }
  return cudaGetLastError();
}
#endif

#if !SWK_PULL
swk::FacePull face_pull(const DevicePtrs& p, const double* total, uint32_t* recip) {
  return {sweep_args(p, 0), p.order, p.pos_of_task, total, recip};
}

// FP64 direction streams (the tasks' totals in `pending` until the pieces are written)
cudaError_t stream_build64(const DevicePtrs& p, int phase, const StreamScratch& b, cudaStream_t s) {
  const uint32_t total = (uint32_t)(p.num_cells * p.D);
  double* totals = static_cast<double*>(p.pending);
  const swk::FacePull f = face_pull(p, totals, b.recip);
  if (phase == 0) {
    swk::k_invert_order<<<grid_for(total, 256), 256, 0, s>>>(p.order, total, p.pos_of_task);
    swk::k_stream_group_segs<<<grid_for((int64_t)p.num_sched_levels * 32, 256), 256, 0, s>>>(
        p.seg_group, p.num_sched_levels, b.gseg);
    swk::k_task_totals<<<grid_for(total, 256), 256, 0, s>>>(f, totals);
    swk::k_reciprocal_faces<<<grid_for(p.num_cells, 256), 256, 0, s>>>(f, b.recip);
    return cudaGetLastError();
  }
  if (phase >= 3) {
    if (p.n_periodic_cells > 0)
      swk::k_fold_build64<<<grid_for((int64_t)p.n_periodic_cells * p.D, 256), 256, 0, s>>>(
          f, p.periodic_cells, p.n_periodic_cells, p.fold_cnt, p.fold_off,
          phase == 3 ? nullptr : static_cast<swk::FoldSlot64*>(p.fold_slots));
    return cudaGetLastError();
  }
  const swk::StreamBuild sb{static_cast<swk::StreamGroup*>(p.stream_groups), p.num_groups, b.gseg, p.lvl, p.seg_group,
                            b.sbase, b.sgroup, p.num_sched_levels, phase == 2 ? p.stream_data : nullptr, stream_shape(p)};
  swk::k_stream_slots64<<<grid_for((int64_t)p.num_groups * 32, 256), 256, 0, s>>>(f, sb);
  return cudaGetLastError();
}

#endif

// Seed of the schedule: dependency counts with every cell active (the caller has set
// all levels >= 0), tasks without dependencies appended to `order`.
cudaError_t schedule_seed(const DevicePtrs& p, cudaStream_t s) {
  swk::SweepArgs<R> a = sweep_args(p, 0);
  a.queue = p.order;
  swk::DirParam dirs;
  for (int i = 0; i < 3 * p.D; ++i) dirs.v[i] = p.dir32_host[i];
  const unsigned long long capacity = (unsigned long long)p.D * p.Np;
  const int blocks = (int)((p.num_cells + swk::kCountThreads - 1) / swk::kCountThreads);
  swk::k_init_counts<R><<<blocks, swk::kCountThreads, 0, s>>>(a, dirs, capacity, nullptr);
  return cudaGetLastError();
}

cudaError_t kahn_rounds(const DevicePtrs& p, uint32_t* bounds, uint32_t* done, uint16_t* task_level, uint32_t round,
                        uint32_t rounds, cudaStream_t s) {
  swk::SweepArgs<R> a = sweep_args(p, 0);
  const unsigned long long capacity = (unsigned long long)p.D * p.Np;
  const int grid = std::min(2 * p.num_sms, grid_for(p.num_cells * p.D / 16, 256));
  for (uint32_t r = round; r < round + rounds; ++r)
    swk::k_kahn_round<R><<<grid, 256, 0, s>>>(a, p.order, bounds, done, capacity, task_level, r);
  return cudaGetLastError();
}

cudaError_t fold_periodic(const DevicePtrs& p, cudaStream_t s) {
  if (p.n_periodic_cells == 0) return cudaSuccess;
#if !SWK_PULL
  if (p.stream_mode) {
    uint8_t* changed = nullptr;
    if (p.active_cells < p.num_cells) {  // only entries next to an active cell
      changed = p.fold_changed;
      swk::k_fold_mark64<<<grid_for(p.n_periodic_cells, 256), 256, 0, s>>>(
          sweep_args(p, 0), static_cast<const double*>(p.cell_att), p.periodic_cells, p.n_periodic_cells, changed);
    }
    swk::k_fold64<<<dim3((p.n_periodic_cells + 255) / 256, p.D), 256, 0, s>>>(
        static_cast<const double*>(p.pending), static_cast<double*>(p.periodic), p.Np, p.periodic_cells,
        p.n_periodic_cells, p.fold_off, static_cast<const swk::FoldSlot64*>(p.fold_slots), changed,
        p.sparse_sweep ? p.act_bits_lv[p.sweep_level] : nullptr);
    return cudaGetLastError();
  }
#endif
  swk::k_fold_periodic<R><<<grid_for((int64_t)p.n_periodic_cells * p.D, 256), 256, 0, s>>>(
      static_cast<R*>(p.periodic), static_cast<R*>(p.pending), p.periodic_cells, p.n_periodic_cells, p.D, p.Np);
  return cudaGetLastError();
}

cudaError_t chemistry(const DevicePtrs& p, int level, cudaStream_t s) {
  swk::ChemArgs<R> a;
  a.cell_rate = nullptr;
  if (p.stream_mode) {
    swk::k_cell_sums<R><<<grid_for(p.num_cells, 128), 128, 0, s>>>(
        (uint32_t)p.num_cells, p.level, level, static_cast<const R*>(p.incoming), p.pos_of_task,
        static_cast<const R*>(p.periodic), p.cell_periodic, p.source, p.D, p.Np, p.rate_scale, p.cell_rate);
    a.cell_rate = p.cell_rate;
  }
  a.n = (uint32_t)p.num_cells;
  a.ctl = p.ctl;
  a.current_level = level;
  a.D = p.D;
  a.Np = p.Np;
  a.incoming = static_cast<const R*>(p.incoming);
  a.periodic = static_cast<const R*>(p.periodic);
  a.rate_scale = p.rate_scale;
  a.source = p.source;
  a.density = p.density;
  a.volume = p.volume;
  a.size = p.size;
  a.level = p.level;
  a.xhii = p.xhii;
  a.yneu = p.yneu;
  a.temperature = p.temperature;
  a.previous_rate = p.previous_rate;
  a.change_timescale = p.change_timescale;
  a.species_timestep = p.species_timestep;
  a.max_timestep = p.max_timestep;
  a.threshold = p.threshold;
  // FP32 transport: 2^-120 of the stored rate unit (normal FP32, full 24-bit precision,
  // 6 binary orders above the subnormal range; the unit is 2^(e - 96) of the total
  // source, so the floor is ~1e-65 of the total luminosity)
  a.rate_floor = sizeof(R) == 4 ? std::ldexp(1.0, -120) * p.rate_scale : 0.0;
  a.safety = p.chem_safety;
  a.scale_factor = p.scale_factor;
  a.prevent_cooling = p.prevent_cooling;
  swk::k_chemistry<R, kCarry><<<grid_for(p.num_cells, 128), 128, 0, s>>>(a);
  return cudaGetLastError();
}

#if SWK_PULL
swk::PullArgs pull_args(const DevicePtrs& p, int level) {
  swk::PullArgs a;
  a.off = p.off;
  a.geo16 = static_cast<const uint4*>(p.geo16);
  a.geo64 = static_cast<const swk::Geo64*>(p.geo64);
  a.dir64 = p.dir64;
  a.dir32 = p.dir32;
  a.D = p.D;
  a.Np = p.Np;
  a.N = (uint32_t)p.num_cells;
  a.level = p.level;
  a.src_dir = static_cast<const float*>(p.src_dir);
  a.att = p.att;
  a.threshold = (float)(p.threshold / p.rate_scale);
  a.periodic = static_cast<const float*>(p.periodic);
  a.qe = p.qe;
  a.inc = static_cast<float*>(p.incoming);
  a.ctl = p.ctl;
  a.current_level = level;
  a.epoch = p.epoch;
  a.epoch_base = p.epoch_base;
  a.cell_sweep = p.cell_sweep;
  a.timeout_ns = p.timeout_ns;
  a.rec = static_cast<const uint4*>(p.pull_rec);
  a.slots = static_cast<const uint2*>(p.pull_slots);
  a.act = nullptr;
  a.act_count = nullptr;
  a.count = (uint32_t)(p.num_cells * p.D);
  a.lvl = p.lvl;
  a.num_sched = p.num_sched_levels;
  a.cellpack = static_cast<const uint2*>(p.cellpack);
  a.per_pos = p.per_pos;
  a.pos_of_task = p.pos_of_task;
  a.inc_pos = p.stream_mode ? p.pos_of_task : nullptr;
  a.order = p.order;
  return a;
}

uint32_t num_chunks(const DevicePtrs& p) {
  return (uint32_t)((p.num_cells * p.D + swk::kCompactChunk - 1) / swk::kCompactChunk);
}

cudaError_t records(const DevicePtrs& p, int phase, unsigned long long* chunk_off, cudaStream_t s) {
  if (p.geo_mode) {  // compact state: no records or slots; the fold's periodic entries, space by space
    if (phase != 1 || p.n_periodic_cells == 0) return cudaSuccess;
    for (int sp = 0; sp < p.num_spaces; ++sp) {
      const DevicePtrs v = space_view(p, sp);
      swk::k_fold_build<<<grid_for((int64_t)v.n_periodic_cells * v.D, 256), 256, 0, s>>>(
          pull_args(v, 0), v.periodic_cells, v.n_periodic_cells, v.fold_cnt, static_cast<uint2*>(v.fold_slots));
    }
    return cudaGetLastError();
  }
  swk::PullArgs a = pull_args(p, 0);
  uint4* rec = static_cast<uint4*>(p.pull_rec);
  const uint32_t nc = num_chunks(p);
  if (phase == 0) {
    swk::k_invert_order<<<grid_for(p.num_cells * p.D, 256), 256, 0, s>>>(p.order, a.count, p.pos_of_task);
    swk::k_pull_rec_count<<<grid_for(p.num_cells * p.D, 256), 256, 0, s>>>(a, p.order, a.count, rec);
    swk::k_pull_slot_chunks<<<nc, swk::kCompactThreads, 0, s>>>(rec, a.count, p.chunk);
    swk::k_scan_chunks64<<<1, swk::kScanThreads, 0, s>>>(p.chunk, nc, chunk_off);
  } else {
    swk::k_pull_slots<<<nc, swk::kCompactThreads, 0, s>>>(a, rec, a.count, chunk_off,
                                                          static_cast<uint2*>(p.pull_slots));
    if (p.n_periodic_cells > 0)
      swk::k_fold_build<<<grid_for((int64_t)p.n_periodic_cells * p.D, 256), 256, 0, s>>>(
          a, p.periodic_cells, p.n_periodic_cells, p.fold_cnt, static_cast<uint2*>(p.fold_slots));
  }
  return cudaGetLastError();
}

// Variants of the pull kernel: the warp-lockstep kernel with its shape as parameters
// (100 * prefetch depth (3: the next slots into L1 only) + 10 * lanes per task (2, 4, 8,
// or 6 for 16) + blocks per SM, + 1000 with streaming loads of records and slots, + 2000
// with the next block's words loaded one block ahead (prefetch depth 2); 83 and 84 name
// 183 and 184) and the level-synchronous wavefronts (72: registers, 78: TMA-staged).  SUBSWEEP_PULL_VARIANT picks one.

const void* pull_kernel(int variant) {
  switch (variant) {
    case 83:
    case 183: return (const void*)swk::k_sweep_pull_lockg<3, 8, 1>;
    case 84:
    case 184: return (const void*)swk::k_sweep_pull_lockg<4, 8, 1>;
    case 122: return (const void*)swk::k_sweep_pull_lockg<2, 2, 1>;
    case 123: return (const void*)swk::k_sweep_pull_lockg<3, 2, 1>;
    case 322: return (const void*)swk::k_sweep_pull_lockg<2, 2, 3>;
    case 323: return (const void*)swk::k_sweep_pull_lockg<3, 2, 3>;
    case 143: return (const void*)swk::k_sweep_pull_lockg<3, 4, 1>;
    case 144: return (const void*)swk::k_sweep_pull_lockg<4, 4, 1>;
    case 164: return (const void*)swk::k_sweep_pull_lockg<4, 16, 1>;
    case 242: return (const void*)swk::k_sweep_pull_lockg<2, 4, 2>;
    case 264: return (const void*)swk::k_sweep_pull_lockg<4, 16, 2>;
    case 283: return (const void*)swk::k_sweep_pull_lockg<3, 8, 2>;
    case 343: return (const void*)swk::k_sweep_pull_lockg<3, 4, 3>;
    case 344: return (const void*)swk::k_sweep_pull_lockg<4, 4, 3>;
    case 384: return (const void*)swk::k_sweep_pull_lockg<4, 8, 3>;
    case 1084: return (const void*)swk::k_sweep_pull_lockg<4, 8, 1, true>;
    case 1143: return (const void*)swk::k_sweep_pull_lockg<3, 4, 1, true>;
    case 1242: return (const void*)swk::k_sweep_pull_lockg<2, 4, 2, true>;
    case 1344: return (const void*)swk::k_sweep_pull_lockg<4, 4, 3, true>;
    case 2242: return (const void*)swk::k_sweep_pull_lockg<2, 4, 2, false, true>;
    case 2283: return (const void*)swk::k_sweep_pull_lockg<3, 8, 2, false, true>;
    case 72: return (const void*)swk::k_sweep_pull_wave<2>;
    case 78: return (const void*)swk::k_sweep_pull_staged;
    default: return nullptr;
  }
}

// the variant in use: set on the handle (autotuner or SUBSWEEP_PULL_VARIANT), else the
// default; an unknown number selects the default
int pull_variant(const DevicePtrs* p = nullptr) {
  int v = kDefaultPullVariant;
  if (p && p->pull_variant > 0) {
    v = p->pull_variant;
  } else if (const char* env = std::getenv("SUBSWEEP_PULL_VARIANT")) {
    v = std::atoi(env);
  }
  return pull_kernel(v) ? v : kDefaultPullVariant;
}

// candidates of the autotuner: the lockstep kernel with 2 lanes per task at 2 target
// blocks per SM, with 4 lanes per task at 3, and at 4 with the next block's slots
// brought into L1 only.  Measured on the C4 generator (transport G tasks/s over whole
// steps, direction-grouped schedule): at 256^3 122 18.6, 323 17.6, 344 16.7, 322 16.3,
// 143 16.1, 1344 15.9, 84 10.3, 242 10.2; at 128^3 143 14.3, 122 14.0, 344 13.6, 1344
// 13.1, 323 12.6.  Only dense sweeps are trials and a step may offer a single one (its
// first), so three candidates finish within three steps.
constexpr int kTuneVariants[] = {122, 143, 344};

// cooperative grid of a kernel: its occupancy limit (capped by
// SUBSWEEP_LEVEL_BLOCKS_PER_SM) on every SM
cudaError_t coop_grid(const DevicePtrs& p, const void* fn, int* grid, int threads = swk::kPullThreads) {
  int bps = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, threads, 0);
  if (e != cudaSuccess) return e;
  if (bps < 1) return cudaErrorInvalidConfiguration;
  if (p.level_bps_cap >= 1 && p.level_bps_cap < bps) bps = p.level_bps_cap;
  *grid = bps * p.num_sms;
  return cudaSuccess;
}

cudaError_t occupancy_pull(int* blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, pull_kernel(pull_variant()),
                                                       swk::kPullThreads, 0);
}

// Sparse sweeps (chosen by the host: above level 0 with fewer than half of the cells
// active) visit only the positions of active cells, from a stable compaction of the
// schedule built at the level's first sweep of a step (three launches; the kernel reads
// the count from the device).  Dense sweeps visit every position; the kernel stamps the
// inactive tasks itself.
// Shared memory of the staged wavefront kernel: the largest slot stages that fit the
// device's per-block limit next to the record, periodic and level-offset buffers;
// cudaErrorInvalidConfiguration when a stage would hold fewer than 9 slots per thread
// (the level offsets of a very deep schedule take the room).
cudaError_t staged_layout(const DevicePtrs& p, uint32_t* cap, size_t* smem) {
  int optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, 0);
  if (e != cudaSuccess) return e;
  const size_t fixed = swk::stg_smem_bytes(0, p.lvl_words) + sizeof(swk::StgShared) + 1024;
  if ((size_t)optin <= fixed) return cudaErrorInvalidConfiguration;
  const uint32_t c = (uint32_t)(((size_t)optin - fixed) / 16) & ~1u;
  if (c < 9u * swk::kStgThreads) return cudaErrorInvalidConfiguration;
  *cap = c;
  *smem = swk::stg_smem_bytes(c, p.lvl_words);
  static size_t attr = 0;
  if (attr != *smem) {
    e = cudaFuncSetAttribute((const void*)swk::k_sweep_pull_staged, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)*smem);
    if (e != cudaSuccess) return e;
    attr = *smem;
  }
  return cudaSuccess;
}

// compact state: the geometry kernel over every position of every task space, one
// launch (segment k of all spaces between two grid barriers)
cudaError_t sweep_pull_geo(const DevicePtrs& p, int level, cudaStream_t s) {
  static_assert(swk::kGeoMaxSpaces >= kMaxSpaces, "a task space per entry");
  const void* fn = (const void*)swk::k_sweep_pull_geo<1>;
  int grid = 0;
  cudaError_t e = coop_grid(p, fn, &grid, swk::kGeoThreads);
  if (e != cudaSuccess) return e;
  swk::GeoArgs g{};
  g.a = pull_args(p, level);
  g.num_spaces = p.num_spaces;
  g.max_levels = 0;
  for (int sp = 0; sp < p.num_spaces; ++sp) {
    const DevicePtrs v = space_view(p, sp);
    swk::GeoSpace& x = g.sp[sp];
    x.order = v.order;
    x.lvl = v.lvl;
    x.num_levels = v.num_sched_levels;
    x.qe = v.qe;
    x.inc = static_cast<float*>(v.incoming);
    x.periodic = static_cast<const float*>(v.periodic);
    x.dir32 = v.dir32;
    x.dir64 = v.dir64;
    g.max_levels = std::max(g.max_levels, x.num_levels);
  }
  if (g.max_levels == 0) return cudaSuccess;
  e = cudaMemsetAsync(&p.ctl->head, 0, sizeof(p.ctl->head), s);  // barrier arrivals
  if (e != cudaSuccess) return e;
  void* args[] = {&g};
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(swk::kGeoThreads), args, 0, s);
}

cudaError_t sweep_pull(const DevicePtrs& p, int level, cudaStream_t s) {
  if (p.geo_mode) return sweep_pull_geo(p, level, s);
  if (p.stream_mode) return sweep_stream(p, level, s);
  swk::PullArgs a = pull_args(p, level);
  const int variant = pull_variant(&p);
  if (p.sparse_sweep) {
    cudaError_t e = compact_active(p, level, s);
    if (e != cudaSuccess) return e;
    a.act = p.act_lv[level];
    a.act_count = p.act_counts + level;
  }
  // the wavefront kernels run dense sweeps over a levelled schedule only; sparse sweeps
  // run the handle's lockstep variant (which tests the upwind cells' levels) or the
  // default one
  const bool wave = variant >= 70 && variant < 80;
  int v = (wave && (p.sparse_sweep || p.num_sched_levels == 0)) ? kDefaultPullVariant : variant;
  const void* fn = pull_kernel(v);
  void* args[] = {&a};
  uint32_t cap = 0;
  size_t smem = 0;
  if (fn == (const void*)swk::k_sweep_pull_staged && (!p.per_pos || staged_layout(p, &cap, &smem) != cudaSuccess)) {
    (void)cudaGetLastError();
    v = kDefaultPullVariant;  // no room for the stages: the lockstep kernel
    fn = pull_kernel(v);
  }
  if (fn == (const void*)swk::k_sweep_pull_staged) {  // one block of 1024 threads per SM
    uint32_t words = p.lvl_words;
    void* sargs[] = {&a, &cap, &words};
    return cudaLaunchCooperativeKernel(fn, dim3(p.num_sms), dim3(swk::kStgThreads), sargs, smem, s);
  }
  int grid = 0;
  cudaError_t e = coop_grid(p, fn, &grid);
  if (e != cudaSuccess) return e;
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(swk::kPullThreads), args, 0, s);
}

cudaError_t stream_build(const DevicePtrs& p, int phase, const StreamScratch& b, cudaStream_t s) {
  const uint32_t total = (uint32_t)(p.num_cells * p.D);
  swk::PullArgs a = pull_args(p, 0);
  if (phase == 0) {
    swk::k_invert_order<<<grid_for(total, 256), 256, 0, s>>>(p.order, total, p.pos_of_task);
    swk::k_stream_group_segs<<<grid_for((int64_t)p.num_sched_levels * 32, 256), 256, 0, s>>>(
        p.seg_group, p.num_sched_levels, b.gseg);
    return cudaGetLastError();
  }
  const swk::StreamBuild sb{static_cast<swk::StreamGroup*>(p.stream_groups), p.num_groups, b.gseg, p.lvl, p.seg_group,
                            b.sbase, b.sgroup, p.num_sched_levels, phase == 2 ? p.stream_data : nullptr, stream_shape(p)};
  swk::k_stream_slots<<<grid_for((int64_t)p.num_groups * 32, 256), 256, 0, s>>>(a, sb);
  if (phase == 2 && p.n_periodic_cells > 0)
    swk::k_fold_build<<<grid_for((int64_t)p.n_periodic_cells * p.D, 256), 256, 0, s>>>(
        a, p.periodic_cells, p.n_periodic_cells, p.fold_cnt, static_cast<uint2*>(p.fold_slots));
  return cudaGetLastError();
}

cudaError_t fold_pull(const DevicePtrs& p, cudaStream_t s) {
  if (p.n_periodic_cells == 0) return cudaSuccess;
  swk::PullArgs a = pull_args(p, 0);
  if (!staged_inputs(p)) a.per_pos = nullptr;
  const dim3 grid((p.n_periodic_cells + 255) / 256, p.D);
  // after a sweep that left cells inactive, only entries next to an active cell
  uint8_t* changed = nullptr;
  if (p.active_cells < p.num_cells && p.fold_changed) {
    changed = p.fold_changed;
    swk::k_fold_mark<<<grid_for(p.n_periodic_cells, 256), 256, 0, s>>>(a, p.periodic_cells, p.n_periodic_cells,
                                                                        changed);
  }
  if (p.geo_mode) {  // compact state: the entries of each task space
    for (int sp = 0; sp < p.num_spaces; ++sp) {
      const DevicePtrs v = space_view(p, sp);
      swk::PullArgs av = pull_args(v, 0);
      av.per_pos = nullptr;
      swk::k_fold_pull<<<dim3(grid.x, v.D), 256, 0, s>>>(av, static_cast<float*>(v.periodic), v.periodic_cells,
                                                         v.n_periodic_cells, v.fold_cnt,
                                                         static_cast<const uint2*>(v.fold_slots), changed);
    }
    return cudaGetLastError();
  }
  swk::k_fold_pull<<<grid, 256, 0, s>>>(a, static_cast<float*>(p.periodic), p.periodic_cells, p.n_periodic_cells,
                                        p.fold_cnt, static_cast<const uint2*>(p.fold_slots), changed);
  return cudaGetLastError();
}

cudaError_t photon_rate(const DevicePtrs& p, uint32_t last_epoch, double* out, cudaStream_t s) {
  if (p.stream_mode) return photon_rate_stored(p, out, s);
  swk::PullArgs a = pull_args(p, 0);
  swk::k_photon_rate_pull<<<grid_for(p.num_cells, 128), 128, 0, s>>>(a, last_epoch, p.rate_scale, out);
  return cudaGetLastError();
}

cudaError_t cell_rates(const DevicePtrs& p, uint32_t last_epoch, double* out, cudaStream_t s) {
  if (p.stream_mode) return cell_rates_stored(p, out, s);
  swk::PullArgs a = pull_args(p, 0);
  swk::k_cell_rates_pull<<<grid_for(p.num_cells, 128), 128, 0, s>>>(a, last_epoch, p.rate_scale, out);
  return cudaGetLastError();
}

cudaError_t export_rates(const DevicePtrs& p, int which, uint32_t last_epoch, double* out, cudaStream_t s) {
  if (p.stream_mode && which == 0) return export_rates_stored(p, which, out, s);
  swk::PullArgs a = pull_args(p, 0);
  swk::k_export_pull<<<grid_for(p.num_cells * p.D, 256), 256, 0, s>>>(a, last_epoch, which, p.rate_scale, out);
  return cudaGetLastError();
}
#else
cudaError_t photon_rate(const DevicePtrs& p, uint32_t, double* out, cudaStream_t s) { return photon_rate_stored(p, out, s); }
cudaError_t cell_rates(const DevicePtrs& p, uint32_t, double* out, cudaStream_t s) { return cell_rates_stored(p, out, s); }
cudaError_t export_rates(const DevicePtrs& p, int which, uint32_t, double* out, cudaStream_t s) {
  return export_rates_stored(p, which, out, s);
}
#endif

}  // namespace

#if SWK_PULL
extern const PrecisionOps SWK_OPS = {
    SWK_NAME,       (int)sizeof(R), true,       occupancy,     attenuation, init_counts, sweep,
    occupancy_pull, sweep_pull,     kahn_rounds, schedule_seed, fold_pull,   chemistry,   photon_rate,
    export_rates,   records,        cell_rates, SWK_CARRY != 0,
    (int)(sizeof(kTuneVariants) / sizeof(int)), kTuneVariants, nullptr, stream_build, stream_pairs,
};
#else
extern const PrecisionOps SWK_OPS = {
    SWK_NAME,         (int)sizeof(R), false,      occupancy,     attenuation,   init_counts, sweep,
    occupancy_levels, sweep_levels,   kahn_rounds, schedule_seed, fold_periodic, chemistry,   photon_rate,
    export_rates,     nullptr,        cell_rates, SWK_CARRY != 0,
    0, nullptr,       push_records, stream_build64, stream_pairs,
};
#endif

}  // namespace swh

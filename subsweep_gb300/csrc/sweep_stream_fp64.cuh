// Direction streams of the FP64 path: the pull form of Sweep::solve_task (src/sweep/mod.rs:423-485).
//
// The reference hands every downwind face the share (eff_f / total) of the change of a task's
// outgoing rate, with eff_f = area_f (n_f . d) and total the sum over the task's downwind faces in
// face order, and the receiving task adds it to its incoming rate.  Here the receiving task adds
// the shares of its upwind tasks' changes itself, with the same fractions, computed once per grid
// with the roundings of push_eff.  The share of face f of cell c comes from the upwind cell's own
// face towards c (the reciprocal face, with the negated normal).  The changes are summed, and not
// the outgoing rates anew: near equilibrium the timescale of a cell shows the last bits of its rate,
// those that a history of changes left in it among them.
//
// The outgoing and incoming rates and the changes lie by schedule position.
#pragma once

#include "sweep_push_records.cuh"
#include "sweep_stream.cuh"

namespace swk {

struct FacePull {
  SweepArgs<double> a;
  const uint32_t* order;
  const uint32_t* pos_of_task;
  const double* total;    // per task
  const uint32_t* recip;  // per face (k_reciprocal_faces)
};

__device__ __forceinline__ double task_total(const SweepArgs<double>& a, uint32_t c, uint32_t d) {
  const double dx = a.dir64[3 * d], dy = a.dir64[3 * d + 1], dz = a.dir64[3 * d + 2];
  const float fx = a.dir32[3 * d], fy = a.dir32[3 * d + 1], fz = a.dir32[3 * d + 2];
  double tot = 0.0;  // face order, zeros for the other faces (solve_group)
  for (uint32_t f = a.off[c]; f < a.off[c + 1]; ++f) tot += push_eff(a, f, dx, dy, dz, fx, fy, fz);
  return tot;
}

static __global__ void k_task_totals(FacePull p, double* total) {
  const size_t n = (size_t)p.a.N * p.a.D;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t d = (uint32_t)(i / p.a.N), c = (uint32_t)(i % p.a.N);
    total[(size_t)d * p.a.Np + c] = task_total(p.a, c, d);
  }
}

// Sign of face f against direction d (+1 downwind, -1 upwind).
__device__ __forceinline__ int pull_sign(const SweepArgs<double>& a, uint32_t f, uint32_t d) {
  const float4 g = a.geo32[f];
  const float s = g.x * a.dir32[3 * d] + g.y * a.dir32[3 * d + 1] + g.z * a.dir32[3 * d + 2];
  return face_sign(s, a.geo64 + f, a.dir64[3 * d], a.dir64[3 * d + 1], a.dir64[3 * d + 2], a.guard);
}

// Of every face of a cell c towards a cell n: the face of n towards c of the same kind with the
// negated normal (the k-th of equal ones, as the face is the k-th of its equals), or kNbrMask.
static __global__ void k_reciprocal_faces(FacePull p, uint32_t* recip) {
  const SweepArgs<double>& a = p.a;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < a.N; c += gridDim.x * blockDim.x) {
    for (uint32_t f = a.off[c]; f < a.off[c + 1]; ++f) {
      const uint32_t nb = a.nbr[f], n = nb & kNbrMask, back = c | (nb & ~kNbrMask);
      uint32_t found = kNbrMask;
      if ((nb >> kKindShift) != kKindBoundary) {
        const Geo64 g = a.geo64[f];
        int k = 0;
        for (uint32_t e = a.off[c]; e < f; ++e)
          if (a.nbr[e] == nb && a.geo64[e].x == g.x && a.geo64[e].y == g.y && a.geo64[e].z == g.z) ++k;
        for (uint32_t q = a.off[n]; q < a.off[n + 1] && found == kNbrMask; ++q)
          if (a.nbr[q] == back && a.geo64[q].x == -g.x && a.geo64[q].y == -g.y && a.geo64[q].z == -g.z && k-- == 0)
            found = q;
      }
      recip[f] = found;
    }
  }
}

// The fraction that the cell across upwind face f hands on through it in direction d; negative if
// its reciprocal face is not downwind or there is none.
__device__ __forceinline__ double pull_fraction(const FacePull& p, uint32_t f, uint32_t d) {
  const SweepArgs<double>& a = p.a;
  const uint32_t q = p.recip[f];
  if (q == kNbrMask) return -1.0;
  const double eff = push_eff(a, q, a.dir64[3 * d], a.dir64[3 * d + 1], a.dir64[3 * d + 2], a.dir32[3 * d],
                              a.dir32[3 * d + 1], a.dir32[3 * d + 2]);
  return eff > 0.0 ? eff / p.total[(size_t)d * a.Np + (a.nbr[f] & kNbrMask)] : -1.0;
}

// Finds the flags and far words of every group (b.data null), or writes the groups' pieces, one
// warp each (k_stream_slots of the mixed path).  The faces handed out and the faces found are
// counted in ctl->head and ctl->tail: a grid where they differ keeps the push form.  An upwind face
// without a partner counts as handed out and not found.
static __global__ void k_stream_slots64(FacePull p, StreamBuild b) {
  const SweepArgs<double>& a = p.a;
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long given = 0, found = 0;
  for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / 32; g < b.num_groups; g += gridDim.x * blockDim.x / 32) {
    const StreamGroup gr = b.groups[g];
    const StreamPiece<double> piece(b.data + kStreamUnit * gr.data, gr);
    const uint32_t n = group_tasks(gr.shape), padded = group_slots(gr.shape);
    StreamSlot s = stream_slots(b, g);
    bool ext = false;
    uint32_t* far = const_cast<uint32_t*>(piece.far()) + lane;
    uint16_t* idx = const_cast<uint16_t*>(piece.idx());
    double* w = const_cast<double*>(piece.w());
    // upwind positions and faces, by position
    uint32_t up[kMaxFaces];
    uint8_t face[kMaxFaces];
    uint32_t ups = 0, c = 0, d = 0;
    double source = 0.0;
    if (lane < n) {
      const uint32_t t = p.order[gr.pos + lane];
      d = t / a.Np;
      c = t - d * a.Np;
      source = a.src_dir[c];
      ext = source != 0.0;
      for (uint32_t f = a.off[c]; f < a.off[c + 1]; ++f) {
        const uint32_t nb = a.nbr[f], kind = nb >> kKindShift;
        if (kind == kKindBoundary) continue;
        const int sign = pull_sign(a, f, d);
        if (sign > 0) ++given;
        if (sign >= 0) continue;
        if (kind == kKindPeriodic) {
          ext = true;
          if (!b.data || pull_fraction(p, f, d) >= 0.0) ++found;
          else ++given;  // nothing is handed out through it: no face may be taken for its partner
          continue;
        }
        const uint32_t u = p.pos_of_task[d * a.Np + (nb & kNbrMask)] - s.base;
        uint32_t i = ups++;
        for (; i > 0 && up[i - 1] > u; --i) {
          up[i] = up[i - 1];
          face[i] = face[i - 1];
        }
        up[i] = u;
        face[i] = (uint8_t)(f - a.off[c]);
      }
    }
    if (ups > padded) {
      atomicOr(&a.ctl->error, kErrRecords);
      ups = padded;
    }
    const uint32_t k = b.gseg[g];
    const uint32_t previous = s.number ? b.seg[k - (b.seg[k] > s.base ? 1 : 0)] - s.base : 0u;  // of the level before
    uint32_t late = 0;
    for (uint32_t i = 0; i < ups; ++i) {
      const uint32_t f0 = s.far, x = stream_slot(b, s, gr.shape, lane, up[i]), j = padded - ups + i;
      if (up[i] >= previous) ++late;
      if (b.data) {
        const double frac = pull_fraction(p, a.off[c] + face[i], d);
        if (frac >= 0.0) ++found;
        else ++given;
        idx[piece.slot(j, lane)] = (uint16_t)x;
        w[piece.wslot(j, lane)] = frac;
        if (s.far > f0) far[f0 * 32] = up[i];
      }
    }
    if (b.data) {
      for (uint32_t j = 0; j < padded - ups; ++j) {
        idx[piece.slot(j, lane)] = (uint16_t)b.shape.ring;  // the zero word
        w[piece.wslot(j, lane)] = 0.0;
      }
      for (uint32_t f = s.far; f < group_far(gr.shape); ++f) far[f * 32] = 0xffffffffu;
      const_cast<double*>(piece.att())[lane] = 0.0;
      if (gr.shape & kGroupExt) {
        const_cast<double*>(piece.per())[lane] = 0.0;
        const_cast<double*>(piece.src())[lane] = source;
      }
      const uint32_t most = __reduce_max_sync(0xffffffffu, ups);
      late = __reduce_max_sync(0xffffffffu, late);
      if (lane == 0) {
        unsigned char* at = b.data + kStreamUnit * gr.data;
        *reinterpret_cast<uint4*>(at) = reinterpret_cast<const uint4*>(b.groups)[g];
        const uint32_t need = previous ? b.seg_group[k - 1] - b.sgroup[k] : 0u;
        *reinterpret_cast<StreamEarly*>(at + sizeof(StreamGroup)) = {need, padded - most, late, 0u};
      }
    }
    const uint32_t flags = stream_flags(ext, s, b.shape.far);
    if (!b.data) {
      if (lane == 0) atomicOr(&b.groups[g].shape, flags);
    } else if (((gr.shape ^ flags) & ~(0xfffu | kGroupKeep)) != 0u) {
      if (lane == 0) atomicOr(&a.ctl->error, kErrRecords);
    }
  }
  if (!b.data) return;
  for (int o = 16; o > 0; o >>= 1) {
    given += __shfl_xor_sync(0xffffffffu, given, o);
    found += __shfl_xor_sync(0xffffffffu, found, o);
  }
  if (lane == 0) {
    atomicAdd(&a.ctl->head, given);
    atomicAdd(&a.ctl->tail, found);
  }
}

// Periodic sources after a sweep (snapshot semantics, k_fold_pull of the mixed path): entry
// d * n_cells + (index of the cell in `cells`) has the slots [off[e], off[e + 1]), {upwind
// position, fraction} in face order.  (Computing the fractions of wide entries here, a division
// each, took 3.6 ms of a 64^3 sweep with 84 directions.)
struct alignas(16) FoldSlot64 {
  uint32_t pos, pad;
  double frac;
};

// counts the entries' slots (slots null), or writes them
static __global__ void k_fold_build64(FacePull p, const uint32_t* cells, uint32_t n_cells, uint8_t* cnt,
                                      const uint32_t* off, FoldSlot64* slots) {
  const SweepArgs<double>& a = p.a;
  const size_t total = (size_t)n_cells * a.D;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const uint32_t d = (uint32_t)(e / n_cells), c = cells[e % n_cells];
    uint32_t n = 0;
    for (uint32_t f = a.off[c]; f < a.off[c + 1]; ++f) {
      const uint32_t nb = a.nbr[f];
      if ((nb >> kKindShift) != kKindPeriodic || pull_sign(a, f, d) >= 0) continue;
      if (slots)
        slots[off[e] + n] = {p.pos_of_task[(size_t)d * a.Np + (nb & kNbrMask)], 0u, pull_fraction(p, f, d)};
      ++n;
    }
    if (!slots) cnt[e] = (uint8_t)n;
  }
}

// After a sweep that left cells inactive: the periodic cells with a periodic neighbour that was
// active; the entries of the others stay as they are.
static __global__ void k_fold_mark64(SweepArgs<double> a, const double* cell_att, const uint32_t* cells,
                                     uint32_t n_cells, uint8_t* changed) {
  for (uint32_t pc = blockIdx.x * blockDim.x + threadIdx.x; pc < n_cells; pc += gridDim.x * blockDim.x) {
    const uint32_t c = cells[pc];
    uint8_t ch = 0;
    for (uint32_t f = a.off[c]; f < a.off[c + 1] && !ch; ++f) {
      const uint32_t nb = a.nbr[f];
      if ((nb >> kKindShift) == kKindPeriodic && st_live(cell_att[nb & kNbrMask])) ch = 1;
    }
    changed[pc] = ch;
  }
}

// grid: (periodic cells / blockDim.x, D).  active: bitmap of the positions that a sparse sweep has
// solved (the changes of the others are of an earlier sweep), or null
static __global__ void k_fold64(const double* change, double* periodic, uint32_t Np, const uint32_t* cells,
                                uint32_t n_cells, const uint32_t* off, const FoldSlot64* slots, const uint8_t* changed,
                                const uint32_t* active) {
  const uint32_t d = blockIdx.y, pc = blockIdx.x * blockDim.x + threadIdx.x;
  if (pc >= n_cells || (changed && !changed[pc])) return;
  const size_t e = (size_t)d * n_cells + pc;
  double in = 0.0;
  for (uint32_t k = off[e]; k < off[e + 1]; ++k) {
    const FoldSlot64 s = slots[k];
    if (active && !(active[s.pos >> 5] >> (s.pos & 31u) & 1u)) continue;
    in = fma(s.frac, change[s.pos], in);
  }
  if (in != 0.0) periodic[(size_t)d * Np + cells[pc]] += in;
}

// After a sparse sweep: its changes reach the tasks of inactive cells as well.
// The inactive cells beside an active one.
static __global__ void k_cells_near64(uint32_t n, const uint8_t* level, int cur, const uint32_t* off,
                                      const uint32_t* nbr, uint8_t* near) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    uint8_t s = 0;
    if (level[c] < cur)
      for (uint32_t f = off[c]; f < off[c + 1] && !s; ++f)
        s = (nbr[f] >> kKindShift) == kKindLocal && level[nbr[f] & kNbrMask] >= cur;
    near[c] = s;
  }
}

// Adds the changes upwind to their incoming rates, in the order of the dense sweep.  grid: (streams,
// any).  A pass over the whole device and not part of the streams' walk, where such tasks would
// be waited for like those that others depend on.
static __global__ void k_stream_take64(StreamArgs<double> a, const uint8_t* near) {
  const StreamDesc sd = a.streams[blockIdx.x];
  const uint32_t lane = threadIdx.x & 31, warps = gridDim.y * (blockDim.x / 32);
  const double* word = a.word + sd.base;
  for (uint32_t number = blockIdx.y * (blockDim.x / 32) + threadIdx.x / 32; number < sd.groups; number += warps) {
    const StreamGroup gr = a.groups[sd.group0 + number];
    if (lane >= group_tasks(gr.shape) || near[a.order[gr.pos + lane] % a.Np] == 0) continue;
    const StreamPiece<double> s(a.data + kStreamUnit * gr.data, gr);
    const uint32_t rel = gr.pos - sd.base + lane;
    double sum = 0.0;
    bool any = false;
    for (uint32_t j = 0; j < s.quads; ++j) {
      const uint2 v = reinterpret_cast<const uint2*>(s.idx())[j * 32 + lane];
      const uint32_t x[4] = {v.x & 0xffffu, v.x >> 16, v.y & 0xffffu, v.y >> 16};
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        if (x[k] == a.shape.ring) continue;
        const uint32_t u = stream_slot_position(a.shape, s, number, lane, rel, x[k]), q = sd.base + u;
        if (!(a.act_bits[q >> 5] >> (q & 31u) & 1u)) continue;
        if (!any) sum = a.inc[sd.base + rel];
        any = true;
        sum = fma(s.w()[StreamPiece<double>::wslot(4 * j + k, lane)], st_ldq(word + u), sum);
      }
    }
    if (any) a.inc[sd.base + rel] = sum;
  }
}

}  // namespace swk

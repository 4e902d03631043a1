// Direction streams: the levelled pull sweep with one thread block per direction.
//
// Directions never depend on one another, and neither do the closed parts of a grid (the
// boxes of a batch), so a (direction, part) pair is a stream of tasks whose whole
// dependency chain one block can walk by itself.  The sweep then needs no word of another
// block, so there is no readiness test, no retry and no round trip through L2 per level:
// the upwind words of the last `ring` positions lie in shared memory.  The warps of the
// block take its groups of 32 tasks in turn, each as soon as the groups of the earlier
// levels are counted as solved (a counter in shared memory).  Everything a sweep does not
// write comes by TMA into the warp's buffer while it solves its previous group, and is in
// registers before the wait, so a narrow level costs one count, one gather from shared
// memory and one sum.
//
// Positions.  The schedule lists the streams one after another, each by level and within
// a level by number of upwind faces, so that the 32 tasks of a warp (a group: up to 32
// consecutive positions of a level) have about the same number of slots, and each task is
// padded with slots of weight 0 to the group's largest count, rounded up to four.
//
// A slot is a weight and a 16-bit index into the block's words in shared memory:
//   the ring slot of the upwind word (its position in the stream modulo the ring) when the
//   word is still there at the end of the consumer's level;
//   the zero word (padding);
//   else a far word: the group lists its position, and the warp that solves the group reads
//   it from memory into its own buffer.
//
// What bounds it: the SM's load/store pipe and the warps' instructions.  A group of 32 tasks
// with 12 slots takes ~90 cycles of the pipe (12 gathers from shared memory at ~3.5 bank
// conflicts each, 20 to fill the buffer and 18 to read the slots, the rest small), 84 SMs for
// 84 directions; hence the slots in quads of 16-byte loads at fixed strides, and everything that
// would touch a memory line per task is done elsewhere: the attenuations are gathered into the groups' pieces before the
// sweep (k_stream_gather, the whole device), the incoming rates are stored by position and
// gathered by the sums over directions (k_cell_sums).
//
// Measured, ms per sweep of 84 directions, lockstep kernels and streams (mixed path): 24^3 0.32
// and 0.15, 32^3 0.45 and 0.24, 64^3 1.56 and 1.01, 96^3 4.2 and 3.0, 128^3 10.3 and 7.6 (23
// tasks per ns).  A block barrier or an mbarrier per level instead of the counter: 64^3 1.2,
// 24^3 0.20.
//
// FP64 is bound by its unit instead: a warp's instruction takes 64 cycles of a quarter of the SM,
// so a group of ~10 slots takes a warp 640 cycles for the products alone.  Its slots lie by upwind
// position and all but those of the previous level are summed before that level is done: 64^3
// 2.85 -> 2.0 ms per sweep, 24^3 0.40 -> 0.31 (push form with atomics 5.4 and 1.6).  Its words are
// the changes of the outgoing rates, added to the incoming rates of before, as the push form adds
// them: with gather and fold 2.24 ms, where sums of the outgoing rates themselves took 2.12, but
// left other last bits in the rates; with the products rounded as well 30% more.
//
// FP32 (mixed path): the incoming rate is the sum of the pull kernels over the slots in face
// order, as eight partial sums combined pairwise, with the same roundings as the lockstep
// kernels, so both give the same bits.  FP64: fused multiply-adds one by one.
#pragma once

#include "sweep_device.cuh"

namespace swk {

__host__ __device__ inline uint32_t group_tasks(uint32_t shape) { return (shape & 31u) + 1u; }
__host__ __device__ inline uint32_t group_slots(uint32_t shape) { return (shape >> 5) & 0x7fu; }
__host__ __device__ inline uint32_t group_far(uint32_t shape) { return shape >> 17; }

template <typename R>
struct StreamTraits;
template <>
struct StreamTraits<float> {
  using Word = unsigned long long;  // {q, sweep << 1}
};
template <>
struct StreamTraits<double> {
  using Word = double;  // what the sweep changes the outgoing rate by (0: the cell is not active)
};

// FP64: the slots of a task lie by upwind position, padding first, so that all but the last
// `late` of them are words of levels before the previous one: they are summed while the previous
// level is solved.
struct alignas(16) StreamEarly {
  uint32_t need;  // groups of the stream before the previous level
  uint32_t skip;  // leading slots that are padding in every task
  uint32_t late;  // trailing slots with words of the previous level in any task
  uint32_t pad;
};

// A group's piece of data, 32 tasks (those past the group's read as padding): the group (16
// bytes; FP64: and its StreamEarly), attenuations [32], 1 / A_down [32] (FP32 rates only), weights [quad][32][4]
// (FP64: [pair][32][2]), 16-bit slot indices [quad][32][4], periodic sources and cell sources / D [2][32] (kGroupExt),
// positions of the far words [far][32].  Slot k of task i is number 4 * (k / 4 * 32 + i) + k % 4.
template <typename R>
struct StreamPiece {
  static constexpr uint32_t kAtt = sizeof(StreamGroup) + (sizeof(R) == 8 ? sizeof(StreamEarly) : 0u), kInv = kAtt + 32 * sizeof(R),
                            kW = kInv + (sizeof(R) == 4 ? 128u : 0u);
  const unsigned char* p;
  uint32_t quads, shape;
  __host__ __device__ StreamPiece(const unsigned char* at, const StreamGroup& g)
      : p(at), quads(group_slots(g.shape) / 4), shape(g.shape) {}
  __host__ __device__ const R* att() const { return reinterpret_cast<const R*>(p + kAtt); }
  __host__ __device__ const float* inv() const { return reinterpret_cast<const float*>(p + kInv); }
  __host__ __device__ const R* w() const { return reinterpret_cast<const R*>(p + kW); }
  __host__ __device__ const uint16_t* idx() const { return reinterpret_cast<const uint16_t*>(w() + 128 * quads); }
  __host__ __device__ const R* per() const { return reinterpret_cast<const R*>(idx() + 128 * quads); }
  __host__ __device__ const R* src() const { return per() + 32; }
  __host__ __device__ const uint32_t* far() const {
    return reinterpret_cast<const uint32_t*>(per() + ((shape & kGroupExt) ? 64 : 0));
  }
  __host__ __device__ static uint32_t slot(uint32_t k, uint32_t i) { return 4 * (k / 4 * 32 + i) + k % 4; }
  // of its weight: in 16-byte loads
  static constexpr uint32_t kVec = 16 / sizeof(R);
  __host__ __device__ static uint32_t wslot(uint32_t k, uint32_t i) { return kVec * (k / kVec * 32 + i) + k % kVec; }
};

// The block's words: ring | zero word | far buffers of the warps [W][far][32].
struct StreamShape {
  uint32_t ring;    // ring entries
  uint32_t magic;   // 2^32 / ring, rounded up: positions modulo the ring
  uint32_t far;     // far words of a task in a warp's buffer
  uint32_t warps;   // solving warps
  uint32_t buffer;  // bytes of a warp's buffer: the largest piece without its far list
  uint32_t blocks;  // blocks of a stream: 1, or the 2 of a cluster
};
constexpr uint32_t kStreamZero = 4;  // words between the ring and the far buffers: the zero word

__device__ __forceinline__ uint32_t ring_slot(const StreamShape& s, uint32_t rel) {
  const uint32_t r = rel - __umulhi(rel, s.magic) * s.ring;
  return (int)r < 0 ? r + s.ring : r;
}

template <typename R>
struct StreamArgs {
  using Word = typename StreamTraits<R>::Word;
  const StreamDesc* streams;
  const StreamGroup* groups;
  const unsigned char* data;   // the groups' pieces
  unsigned long long bytes;    // of them
  Word* word;                  // per position
  R* inc;                      // per position: the incoming rate
  R* out;                      // FP64, per position: the outgoing rate
  R threshold;
  SweepCtl* ctl;
  unsigned long long timeout_ns;
  uint32_t epoch;
  const uint32_t* epoch_base;
  StreamShape shape;
  int evict_first;             // the pieces exceed L2: load them evict-first
  const uint32_t* seg_group;   // first group of every level segment (sparse sweeps)
  // sparse sweeps: the active positions in order, their range in each stream and their bitmap,
  // and the segments' first positions
  const uint32_t *act, *act_range, *act_bits;
  const uint32_t* seg;
  // (their attenuations and periodic sources come straight from the cells' and tasks')
  const uint32_t* order;
  const R *cell_att, *periodic;
  uint32_t Np;
  uint32_t* stamp;  // FP64: per position, the last sparse sweep that solved it
  // pairs of blocks: the parts of pair i are parts[part0[i]], ... up to part0[i + 1]; flags[i]: the
  // last sweep in which the first part of a cut stream was solved
  const StreamPart* parts;
  const uint32_t* part0;
  uint32_t* flags;
};

__device__ __forceinline__ uint32_t st_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t st_count(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(st_smem(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_count_up(uint32_t* p) {
  asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;" ::"r"(st_smem(p)) : "memory");
}
// whether a sweep of the step has stalled
__device__ __forceinline__ bool st_stalled(const SweepCtl* ctl) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&ctl->error) : "memory");
  return (v & kErrStall) != 0;
}
// bounded wait of a warp; on a timeout sets kErrStall and returns false, and the caller goes
// on without waiting or solving (it still counts its groups, so no other warp waits for them)
template <typename Test>
__device__ __forceinline__ bool st_wait(Test test, SweepCtl* ctl, unsigned long long limit) {
  bool ok = test();
  if (!ok) {
    unsigned long long w0 = 0;
    for (uint32_t k = 1; !(ok = test()); ++k) {
      if ((k & 255u) == 0) {
        const unsigned long long now = globaltimer_ns();
        if (w0 == 0) w0 = now;
        if (now - w0 > limit || st_stalled(ctl)) break;
      }
    }
    if (!ok) atomicOr(&ctl->error, kErrStall);
  }
  return __all_sync(0xffffffffu, ok);
}

// Pairs of blocks (a cluster): the peer's words and count by their addresses in its shared memory.
__device__ __forceinline__ uint32_t st_peer(uint32_t address, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(address), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_peer_word(uint32_t address, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(address), "f"(v) : "memory");
}
__device__ __forceinline__ void st_peer_word(uint32_t address, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(address), "d"(v) : "memory");
}
// A pair's counts: groups solved by this block, and by the other as far as it has told.  A group of
// a level is solved only when all earlier levels are, so their sum reaches the groups before a
// level exactly when those are solved.
__device__ __forceinline__ uint32_t st_count_pair(const uint32_t* p) {
  uint32_t own, other;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(own) : "r"(st_smem(p)) : "memory");
  asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(other) : "r"(st_smem(p + 1)) : "memory");
  return own + other;
}
// the words counted so far are in the peer's ring: a fence for many groups, by a warp of its own
__device__ __forceinline__ void st_tell_peer(uint32_t peer_other, uint32_t count) {
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(peer_other), "r"(count) : "memory");
}
__device__ __forceinline__ void st_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// whether an attenuation is one, not the mark of a cell that is not active in the sweep
__device__ __forceinline__ bool st_live(float att) { return __float_as_uint(att) != 0xffffffffu; }
__device__ __forceinline__ bool st_live(double att) { return __double_as_longlong(att) != -1ll; }
// the q of a word in memory, the word of a q
__device__ __forceinline__ double st_ldq(const double* w) { return __ldcg(w); }
__device__ __forceinline__ double st_word(double q, uint32_t) { return q; }
__device__ __forceinline__ float st_ldq(const unsigned long long* w) {
  return __uint_as_float(__ldcg(reinterpret_cast<const uint32_t*>(w)));
}
__device__ __forceinline__ unsigned long long st_word(float q, uint32_t sweep) {
  return ((unsigned long long)(sweep << 1) << 32) | (unsigned long long)__float_as_uint(q);
}

// Incoming rate of a task, fed its slots in order.  FP32: eight partial sums, partial k over
// the slots k, k + 8, ... by fused multiply-adds in slot order, combined pairwise as the
// lockstep kernels do (a padding slot adds 0 * 0, which changes no bit).
template <typename R>
struct StreamSum;
template <>
struct StreamSum<float> {
  float part[8];
  __device__ __forceinline__ explicit StreamSum(float) {
#pragma unroll
    for (int k = 0; k < 8; ++k) part[k] = 0.f;
  }
  __device__ __forceinline__ void add(int k, float w, float q) { part[k & 7] = fmaf(w, q, part[k & 7]); }
  __device__ __forceinline__ float total() const {
    return ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
  }
};

// FP64: the incoming rate of before and, one by one, the shares of the upwind tasks' changes, which
// the push form adds in any order (the product is not rounded: half the instructions).
template <>
struct StreamSum<double> {
  double sum;
  __device__ __forceinline__ explicit StreamSum(double before) : sum(before) {}
  __device__ __forceinline__ void add(int, double w, double q) { sum = fma(w, q, sum); }
  __device__ __forceinline__ double total() const { return sum; }
};

// outgoing rate of the task (get_outgoing_rate of Site::get_rate), as the word's q
__device__ __forceinline__ float st_solve(float in, float src, float per, float att, float threshold, float inv) {
  const float rt = (in + src) + per;                    // Site::get_rate, site.rs:53-56
  const float out = (rt < threshold) ? 0.f : rt * att;  // get_outgoing_rate
  return out * inv;
}
// Photons::make_positive (chemistry/mod.rs:61-65), on the bits: a number below 0 becomes 0
__device__ __forceinline__ double st_positive(double in) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(in);
  return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull ? 0.0 : in;
}
// FP64: the comparison on the bits, which order as the numbers do from the threshold up
__device__ __forceinline__ double st_solve(double rt, double att, double threshold) {
  const long long b = __double_as_longlong(rt), t = __double_as_longlong(threshold);
  const bool below = t >= 0 ? b < t && (b & 0x7fffffffffffffffll) <= 0x7ff0000000000000ll : rt < threshold;
  return below ? 0.0 : rt * att;
}
__device__ __forceinline__ double st_solve(double in, double src, double per, double att, double threshold, float) {
  return st_solve((in + src) + per, att, threshold);
}

// Shared memory of a block: a barrier per warp, the counts and parts, the warps' buffers, the words.
constexpr uint32_t kStreamHead = 8 * 36;
template <typename R>
constexpr size_t stream_smem_bytes(const StreamShape& s) {
  return kStreamHead + (size_t)s.warps * s.buffer +
         ((size_t)s.ring + kStreamZero + (size_t)s.warps * s.far * 32) * sizeof(R);
}

__device__ __forceinline__ bool st_bar_test(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(st_smem(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

constexpr uint32_t kStreamQuads = 4;      // quads of slots that are in registers before the wait
constexpr uint32_t kStreamAhead = 98304;  // bytes between a group's piece and what is brought to L2

// four weights and their slot indices
template <typename R>
struct StreamWeights;
template <>
struct StreamWeights<float> {
  float4 v;
  __device__ __forceinline__ void load(const StreamPiece<float>& s, uint32_t k, uint32_t lane) {
    v = reinterpret_cast<const float4*>(s.w())[k * 32 + lane];
  }
  __device__ __forceinline__ float get(int c) const { return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w; }
};
template <>
struct StreamWeights<double> {
  double2 a, b;
  __device__ __forceinline__ void load(const StreamPiece<double>& s, uint32_t k, uint32_t lane) {
    a = reinterpret_cast<const double2*>(s.w())[2 * k * 32 + lane];
    b = reinterpret_cast<const double2*>(s.w())[(2 * k + 1) * 32 + lane];
  }
  __device__ __forceinline__ double get(int c) const { return c == 0 ? a.x : c == 1 ? a.y : c == 2 ? b.x : b.y; }
};
template <typename R>
struct StreamQuad {
  StreamWeights<R> w;
  uint2 x;
  __device__ __forceinline__ void load(const StreamPiece<R>& s, uint32_t k, uint32_t lane) {
    w.load(s, k, lane);
    x = reinterpret_cast<const uint2*>(s.idx())[k * 32 + lane];
  }
};
template <typename R>
__device__ __forceinline__ void st_words(const StreamQuad<R>& t, const R* words, R (&q)[4]) {
  q[0] = words[t.x.x & 0xffffu];
  q[1] = words[t.x.x >> 16];
  q[2] = words[t.x.y & 0xffffu];
  q[3] = words[t.x.y >> 16];
}
template <typename R>
__device__ __forceinline__ void st_add(StreamSum<R>& sum, bool odd, const StreamWeights<R>& w, const R (&q)[4]) {
  if (odd) {
#pragma unroll
    for (int c = 0; c < 4; ++c) sum.add(4 + c, w.get(c), q[c]);
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) sum.add(c, w.get(c), q[c]);
  }
}

// FP64: adds the slots [lo, hi) of a group, in order
__device__ __forceinline__ void st_sum(StreamSum<double>& sum, const StreamQuad<double> (&quad)[kStreamQuads],
                                       const double* words, const StreamPiece<double>& s, uint32_t lane, uint32_t lo,
                                       uint32_t hi) {
  auto add = [&](const StreamQuad<double>& t, uint32_t k) {
    double q[4];
    st_words(t, words, q);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (k + c >= lo && k + c < hi) sum.add(0, t.w.get(c), q[c]);
  };
#pragma unroll
  for (uint32_t c = 0; c < kStreamQuads; ++c)
    if (4 * c + 4 > lo && 4 * c < hi) add(quad[c], 4 * c);
  for (uint32_t c = max(kStreamQuads, lo / 4); 4 * c < hi; ++c) {
    StreamQuad<double> t;
    t.load(s, c, lane);
    add(t, 4 * c);
  }
}

// The dense sweep: every position of every stream, one stream per block.  Warp w solves the
// groups w, w + W, ...; lanes past a group's tasks compute with padding.  kFar: some groups
// have far words.  kAll: every cell is active; otherwise the tasks of inactive cells hand their
// kept word on through the ring.
//
// kPair: a stream is walked by the two blocks of a cluster, with the warps of both taking its
// groups in turn, where levels are wide (96^3 x 84 in FP64 8.5 -> 7.4 ms, 128^3 x 84 in the mixed
// path 7.8 -> 7.3; at 64^3 slower).  Either block holds the whole ring and a word is stored into
// both.  A warp of its own fences the words of all groups solved so far and tells the peer their
// number: with a fence for every group 96^3 took 7.9 ms, since it waits for the stores of the SM.
// There are fewer pairs of SMs than streams (76 for 84 directions), so the streams are laid end to
// end and cut into equal shares: where a share ends inside a stream, the next pair starts with
// that stream's beginning, and this one ends with the rest of it, once the beginning is solved
// (flags), its ring filled from memory.  The clusters take the pairs in the order in which they
// start, the last pair first, so one waits only for another that runs already, in whatever order
// and however many at a time the device starts them.
template <typename R, int W, bool kFar, bool kAll, bool kPair = false>
__global__ void __launch_bounds__(32 * (kPair ? W + 1 : W)) k_sweep_stream(const __grid_constant__ StreamArgs<R> a) {
  constexpr uint32_t S = kPair ? 2 * W : W;  // warps that take the groups in turn
  constexpr bool kAddress = sizeof(R) == 4 && !kFar && !kPair;  // slots' addresses ahead of the wait
  constexpr bool kChange = sizeof(R) == 8;  // words are changes, added to the incoming rate of before
  using Word = typename StreamTraits<R>::Word;
  extern __shared__ __align__(16) unsigned char st_shared[];
  const StreamShape& shape = a.shape;
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(st_shared) + warp;
  uint32_t* count = reinterpret_cast<uint32_t*>(st_shared + 8 * 32);  // solved groups of the stream
  // kPair: the parts of the pair [first, end) (read where they are needed: registers)
  volatile uint32_t* parts_of = count + 4;
  unsigned char* buffer = st_shared + kStreamHead + warp * shape.buffer;
  R* words = reinterpret_cast<R*>(st_shared + kStreamHead + W * shape.buffer);
  StreamDesc sd = a.streams[kPair ? 0 : blockIdx.x];
  uint32_t me = warp, peer_words = 0, peer_count = 0;
  if constexpr (kPair) {
    uint32_t rank, size;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    if (size != 2) {  // launched without its peer
      if (threadIdx.x == 0) atomicOr(&a.ctl->error, kErrStall);
      return;
    }
    // the last pair goes to the cluster that starts first (ctl->head is 0 before every sweep)
    if (rank == 0 && threadIdx.x == 0) count[2] = (uint32_t)atomicAdd(&a.ctl->head, 1ull);
    st_cluster_sync();
    if (threadIdx.x == 0) {
      uint32_t started;
      asm volatile("ld.shared::cluster.u32 %0, [%1];"
                   : "=r"(started)
                   : "r"(st_peer(st_smem(count + 2), 0u))
                   : "memory");
      const bool spare = started >= gridDim.x / 2;  // more clusters than pairs: none
      if (spare) atomicOr(&a.ctl->error, kErrStall);
      const uint32_t* at = a.part0 + (gridDim.x / 2 - 1 - started);
      parts_of[0] = spare ? 0u : at[0];
      parts_of[1] = spare ? 0u : at[1];
    }
    st_cluster_sync();
    me = rank * W + warp;  // (the warp that tells the peer: (rank + 1) * W)
    peer_words = st_peer(st_smem(words), rank ^ 1u);
    peer_count = st_peer(st_smem(count + 1), rank ^ 1u);
  }
  if (threadIdx.x < 2) count[threadIdx.x] = 0;
  if (threadIdx.x < kStreamZero) words[shape.ring + threadIdx.x] = R(0);
  if (lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(st_smem(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  const uint32_t sweep = a.epoch_base ? *a.epoch_base + a.epoch : a.epoch;
  const StreamGroup* groups = a.groups + sd.group0;
  Word* word = a.word + sd.base + lane;
  R* inc = a.inc + sd.base + lane;
  R* outgoing = a.out + sd.base + lane;
  uint32_t begin = 0, stop = sd.groups;  // groups of the part
  auto counted = [&](uint32_t need) { return (kPair ? st_count_pair(count) : st_count(count)) >= need; };
  R* far_words = words + shape.ring + kStreamZero + warp * shape.far * 32u + lane;
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  // the next group of the warp, and where its piece ends (pieces follow one another)
  StreamGroup next{};
  uint32_t end = 0;
  auto locate = [&](uint32_t g) {
    if (g < stop) {
      next = groups[g];
      end = groups[g + 1].data;
    }
  };
  // the warp's reads of its buffer are done: the next piece may overwrite it
  auto copy = [&]() {
    __syncwarp();
    if (lane == 0) {
      // the far list, a piece's last part, need not fit
      const uint32_t bytes = min((end - next.data) * (uint32_t)kStreamUnit, shape.buffer);
      const unsigned char* src = a.data + kStreamUnit * next.data;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(st_smem(bar)), "r"(bytes) : "memory");
      if (a.evict_first)
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
            ::"r"(st_smem(buffer)), "l"(src), "r"(bytes), "r"(st_smem(bar)), "l"(policy)
            : "memory");
      else
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         st_smem(buffer)),
                     "l"(src), "r"(bytes), "r"(st_smem(bar))
                     : "memory");
      if (kStreamUnit * end + kStreamAhead <= a.bytes)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src + kStreamAhead), "r"(bytes) : "memory");
    }
  };
  bool dead = false;
  uint32_t solved = 0, parity = 0, g = me;
  // the group that the warp solves next, in registers
  StreamGroup gr{};
  StreamEarly early{};
  StreamQuad<R> quad[kStreamQuads];
  R att = R(0), per = R(0), src = R(0);
  R own = R(0);  // the word kept by an inactive task; FP64: the outgoing rate of before
  R before = R(0), before_next = R(0);  // FP64: the incoming rate of before, and that of the group `next`
  auto ask = [&]() {
    if constexpr (kChange) before_next = lane < group_tasks(next.shape) ? __ldcg(inc + (next.pos - sd.base)) : R(0);
  };
  float inv = 0.f;
  uint32_t up[kFar ? kStreamFar : 1], up_far = 0;
  // kPair: the far words on their way (the other block wrote some of them, so they come from L2,
  // not by the copies through L1)
  R held[kFar && kPair ? kStreamFar : 1];
  uint32_t held_far = 0;
  bool staged = false;  // its piece is still in the buffer: slots beyond the registers
  // loads group g and starts the copy of the one after it
  auto load = [&]() {
    if (g >= stop) return;
    // (a dead block's copies still land before their buffer is used again or left)
    dead = !st_wait([&]() { return st_bar_test(bar, parity); }, a.ctl, a.timeout_ns) || dead;
    parity ^= 1;
    gr = *reinterpret_cast<const StreamGroup*>(buffer);
    if constexpr (sizeof(R) == 8) early = *reinterpret_cast<const StreamEarly*>(buffer + sizeof(StreamGroup));
    const StreamPiece<R> s(buffer, gr);
    att = s.att()[lane];
    if (sizeof(R) == 4) inv = s.inv()[lane];
#pragma unroll
    for (uint32_t k = 0; k < kStreamQuads; ++k)
      if (k < s.quads) quad[k].load(s, k, lane);
    per = src = R(0);
    if (gr.shape & kGroupExt) {
      per = s.per()[lane];
      src = s.src()[lane];
    }
    if constexpr (kChange) {
      before = before_next;
      if (lane < group_tasks(gr.shape)) own = __ldcg(outgoing + (gr.pos - sd.base));
    } else if (!kAll && lane < group_tasks(gr.shape)) {
      own = st_ldq(word + (gr.pos - sd.base));
    }
    staged = s.quads > kStreamQuads;
    if (g + S < stop) {
      ask();
      if (kFar) {  // the positions of the next group's far words
        up_far = (next.shape & (kGroupLate | kGroupSlow)) ? 0u : group_far(next.shape);
        if (up_far) {
          const StreamPiece<R> t(a.data + kStreamUnit * next.data, next);
#pragma unroll
          for (int f = 0; f < (int)kStreamFar; ++f)
            up[f] = (uint32_t)f < up_far ? __ldcs(t.far() + f * 32 + lane) : 0xffffffffu;
        }
      }
      if (!staged) {
        copy();
        locate(g + 2 * S);
      }
    } else {
      up_far = 0;
    }
    if (kFar && !kPair) asm volatile("cp.async.wait_all;" ::: "memory");  // this group's far words
    if (kFar && kPair) {
#pragma unroll
      for (int f = 0; f < (int)kStreamFar; ++f)
        if ((uint32_t)f < held_far) far_words[f * 32] = held[f];
      held_far = 0;
    }
  };
  // what is left to store of the group solved: behind the count, off the levels' chain
  R in = R(0), out = R(0), q = R(0);
  uint32_t rel = 0;
  bool mine = false, other = false;  // other: FP64, of an inactive cell, which takes the changes upwind
  auto store = [&]() {
    if (mine || other) {
      word[rel] = st_word(q, sweep);
      inc[rel] = in;
    }
    if (mine) {
      if constexpr (kChange) outgoing[rel] = out;
      ++solved;
    }
    mine = other = false;
  };
  for (uint32_t part = kPair ? parts_of[0] : 0u; part < (kPair ? parts_of[1] : 1u); ++part) {
    uint32_t post = 0;
    bool fresh = false;  // the part's first groups: their far words have not been fetched ahead
    if constexpr (kPair) {
      const StreamPart pt = a.parts[part];
      sd = a.streams[pt.stream];
      groups = a.groups + sd.group0;
      word = a.word + sd.base + lane;
      inc = a.inc + sd.base + lane;
      outgoing = a.out + sd.base + lane;
      begin = pt.begin;
      stop = pt.end;
      post = pt.post;
      if (pt.wait) {  // the pair that has the stream's beginning
        const uint32_t* flag = a.flags + pt.wait - 1;
        dead = !st_wait([&]() {
          uint32_t v;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
          return v == sweep;
        }, a.ctl, a.timeout_ns) || dead;
      }
      if (begin > 0) {
        const uint32_t from = groups[begin].pos - sd.base;
        for (uint32_t i = threadIdx.x; i < min(from, shape.ring); i += blockDim.x) {
          const uint32_t at = from - 1 - i;
          words[ring_slot(shape, at)] = st_ldq(a.word + sd.base + at);
        }
        fresh = true;
      }
      // (the groups in front of the part count as this block's)
      if (threadIdx.x < 2) count[threadIdx.x] = threadIdx.x == 0 ? begin : 0u;
      st_cluster_sync();
      g = begin - begin % S + me;
      if (g < begin) g += S;
      if (warp == W) {  // tells the peer of the groups that this block has solved, until all are
        const uint32_t rank = me / W - 1;
        uint32_t mine = 0;  // this block's groups of the part
        for (uint32_t w = rank * W; w < (rank + 1) * W; ++w) {
          const uint32_t f = begin - begin % S + w, from = f < begin ? f + S : f;
          if (from < stop) mine += (stop - from + S - 1) / S;
        }
        uint32_t told = 0, now = 0;
        bool ok = true;
        while (told < mine && ok) {
          ok = st_wait([&]() { return (now = st_count(count) - begin) > told; }, a.ctl, a.timeout_ns);
          now = __shfl_sync(0xffffffffu, now, 0);
          if (lane == 0) st_tell_peer(peer_count, now);
          told = now;
        }
        g = stop;
      }
    }
    locate(g);
    if (g < stop) {
      ask();
      copy();
    }
    locate(g + S);
    load();
    while (g < stop) {
      StreamSum<R> sum(before);
      const uint32_t quads = group_slots(gr.shape) / 4;
      uint32_t first = 0;  // slot that the sum goes on with
      if constexpr (sizeof(R) == 8) {
        const bool ahead = !kFar || (!fresh && !(gr.shape & (kGroupLate | kGroupSlow)));
        if (ahead && !dead) {
          dead = !st_wait([&]() { return counted(early.need); }, a.ctl, a.timeout_ns);
          first = 4 * quads - early.late;
          if (!dead) st_sum(sum, quad, words, StreamPiece<R>(buffer, gr), lane, early.skip, first);
        }
      }
      // (all that needs no word of this level, ahead of the wait)
      const uint32_t n = group_tasks(gr.shape);
      rel = gr.pos - sd.base;
      uint32_t slot = ring_slot(shape, rel) + lane;
      if (slot >= shape.ring) slot -= shape.ring;
      uint32_t at[kAddress ? kStreamQuads : 1][4];
      if constexpr (kAddress) {
#pragma unroll
        for (uint32_t c = 0; c < kStreamQuads; ++c) {
          at[c][0] = st_smem(words) + (quad[c].x.x & 0xffffu) * (uint32_t)sizeof(R);
          at[c][1] = st_smem(words) + (quad[c].x.x >> 16) * (uint32_t)sizeof(R);
          at[c][2] = st_smem(words) + (quad[c].x.y & 0xffffu) * (uint32_t)sizeof(R);
          at[c][3] = st_smem(words) + (quad[c].x.y >> 16) * (uint32_t)sizeof(R);
        }
      }
      // the levels before this group's
      dead = dead || !st_wait([&]() { return counted(gr.need); }, a.ctl, a.timeout_ns);
      if (!dead) {
        if (kFar && (fresh || (gr.shape & (kGroupLate | kGroupSlow)))) {
          const StreamPiece<R> all(a.data + kStreamUnit * gr.data, gr);
          const Word* base = a.word + sd.base;
          if (gr.shape & kGroupSlow) {  // more far words than the buffer holds: index far + number
            const uint32_t far = shape.ring + kStreamZero;
            for (uint32_t j = 0; j < quads; ++j) {
              R q[4];
              StreamQuad<R> t;
              t.load(all, j, lane);
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const uint32_t x = all.idx()[StreamPiece<R>::slot(4 * j + c, lane)];
                q[c] = x >= far ? st_ldq(base + all.far()[(x - far) * 32 + lane]) : words[x];
              }
              st_add(sum, j & 1u, t.w, q);
            }
          } else {
            for (uint32_t f = 0; f < group_far(gr.shape); ++f) {
              const uint32_t at = all.far()[f * 32 + lane];
              far_words[f * 32u] = at != 0xffffffffu ? st_ldq(base + at) : R(0);
            }
          }
        }
        if (!kFar || !(gr.shape & kGroupSlow)) {
          const StreamPiece<R> s(buffer, gr);
          if constexpr (sizeof(R) == 8) {
            st_sum(sum, quad, words, s, lane, max(first, early.skip), 4 * quads);
          } else {
            R q[kStreamQuads][4];
#pragma unroll
            for (uint32_t c = 0; c < kStreamQuads; ++c)
              if (c < quads) {
                if constexpr (kAddress) {
#pragma unroll
                  for (int k = 0; k < 4; ++k)
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(q[c][k]) : "r"(at[c][k]) : "memory");
                } else {
                  st_words(quad[c], words, q[c]);
                }
              }
#pragma unroll
            for (uint32_t c = 0; c < kStreamQuads; ++c)
              if (c < quads) st_add(sum, c & 1u, quad[c].w, q[c]);
            for (uint32_t c = kStreamQuads; c < quads; ++c) {
              StreamQuad<R> t;
              t.load(s, c, lane);
              R qc[4];
              st_words(t, words, qc);
              st_add(sum, c & 1u, t.w, qc);
            }
          }
        }
        in = sum.total();
        mine = lane < n && (kAll || st_live(att));
        if constexpr (kChange) {
          if (mine) in = st_positive(in);
          out = (gr.shape & kGroupExt) ? st_solve(in, src, per, att, a.threshold, inv) : st_solve(in, att, a.threshold);
          other = lane < n && !mine;
          q = mine ? out - own : R(0);
        } else {
          out = st_solve(in, src, per, att, a.threshold, inv);
          q = mine ? out : own;
        }
        if (lane < n) {
          words[slot] = q;
          if constexpr (kPair) st_peer_word(peer_words + slot * (uint32_t)sizeof(R), q);
        }
        // a word that another group reads from memory is there before the barrier
        if (kFar && (gr.shape & kGroupKeep)) store();
      }
      __syncwarp();
      if (lane == 0) st_count_up(count);
      fresh = false;
      if (kFar && up_far) {  // solved by now: their levels lie before this group's
        const Word* base = a.word + sd.base;
#pragma unroll
        for (int f = 0; f < (int)kStreamFar; ++f)
          if constexpr (kPair) {
            held[f] = up[f] != 0xffffffffu ? st_ldq(base + up[f]) : R(0);
          } else if (up[f] != 0xffffffffu)
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(st_smem(far_words + f * 32)),
                         "l"(base + up[f]), "n"(sizeof(R))
                         : "memory");  // the q leads a word
        if constexpr (kPair) held_far = up_far;
        up_far = 0;
      }
      if (staged && g + S < stop) {
        copy();
        locate(g + 2 * S);
      }
      store();
      g += S;
      load();
    }
    if constexpr (kPair) {
      st_cluster_sync();  // both blocks are done with the ring, and have stored all words
      if (post && me == 0 && threadIdx.x == 0)
        asm volatile("fence.acq_rel.gpu;\n\tst.relaxed.gpu.global.u32 [%0], %1;" ::"l"(a.flags + post - 1), "r"(sweep)
                     : "memory");
    }
  }
  for (int o = 16; o > 0; o >>= 1) solved += __shfl_xor_sync(0xffffffffu, solved, o);
  if (lane == 0 && solved) {
    atomicAdd(&a.ctl->tasks, (unsigned long long)solved);
    atomicAdd(&a.ctl->attempts, (unsigned long long)solved);
  }
}

// Position in its stream of the upwind task of slot index x, of task i of group g (number
// `number` of its stream) at position rel in the stream; not of the zero word.
template <typename R>
__device__ __forceinline__ uint32_t stream_slot_position(const StreamShape& shape, const StreamPiece<R>& s,
                                                         uint32_t number, uint32_t i, uint32_t rel, uint32_t x) {
  if (x < shape.ring) {  // the last position before this one that is congruent to it
    const uint32_t rs = ring_slot(shape, rel);
    return rel - (rs > x ? rs - x : rs + shape.ring - x);
  }
  x -= shape.ring + kStreamZero;
  const uint32_t f = (s.shape & kGroupSlow) ? x : (x - number % shape.warps * shape.far * 32u) / 32u;
  return s.far()[f * 32u + i];
}

// The sparse sweep: the active positions only, a thread per task, in the order of the stream.
// A level has few tasks or none, so there is nothing to gain from the ring or from waiting
// level by level: the upwind words are read from memory, an active one until it carries the
// sweep's number.  A warp's tasks may depend on one another, so its lanes try again together;
// all others they wait for come earlier in the list, in warps at work or done.
constexpr int kStreamSparseThreads = 512;
constexpr uint32_t kSparseNone = 0x7fffffffu, kSparseActive = 0x80000000u;

// The upwind words of four slots, and whether those that the sweep solves are there.  FP32: a
// word carries the number of the sweep that wrote it; FP64: the stamp beside it, in the order of
// the block (a stream is one block).
__device__ __forceinline__ void st_try(const StreamArgs<float>&, const unsigned long long* word, uint32_t,
                                       const uint32_t (&up)[4], uint32_t sweep, bool& ready, float (&q)[4]) {
  unsigned long long v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = up[k] != kSparseNone ? ld_relaxed64(word + (up[k] & kSparseNone)) : 0ull;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    ready = ready && (!(up[k] & kSparseActive) || (uint32_t)(v[k] >> 32) == sweep << 1);
    q[k] = __uint_as_float((uint32_t)v[k]);
  }
}
// (FP64: the word of a cell that is not active is 0)
__device__ __forceinline__ void st_try(const StreamArgs<double>& a, const double* word, uint32_t base,
                                       const uint32_t (&up)[4], uint32_t sweep, bool& ready, double (&q)[4]) {
  uint32_t v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = sweep;
    if (up[k] & kSparseActive)
      asm volatile("ld.acquire.cta.global.u32 %0, [%1];"
                   : "=r"(v[k])
                   : "l"(a.stamp + base + (up[k] & kSparseNone))
                   : "memory");
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    ready = ready && v[k] == sweep;
    q[k] = (up[k] & kSparseActive) ? st_ldq(word + (up[k] & kSparseNone)) : 0.0;
  }
}
__device__ __forceinline__ void st_publish(const StreamArgs<float>&, unsigned long long* word, uint32_t, uint32_t rel,
                                           float q, uint32_t sweep) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(word + rel), "l"(st_word(q, sweep)) : "memory");
}
__device__ __forceinline__ void st_publish(const StreamArgs<double>& a, double* word, uint32_t base, uint32_t rel,
                                           double q, uint32_t sweep) {
  word[rel] = q;
  asm volatile("st.release.cta.global.u32 [%0], %1;" ::"l"(a.stamp + base + rel), "r"(sweep) : "memory");
}

template <typename R>
__global__ void __launch_bounds__(kStreamSparseThreads) k_sweep_stream_sparse(const __grid_constant__ StreamArgs<R> a) {
  using Word = typename StreamTraits<R>::Word;
  constexpr uint32_t T = kStreamSparseThreads;
  constexpr bool kChange = sizeof(R) == 8;
  const StreamDesc sd = a.streams[blockIdx.x];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t sweep = a.epoch_base ? *a.epoch_base + a.epoch : a.epoch;
  R* inc = a.inc + sd.base;
  Word* word = a.word + sd.base;
  const uint32_t end = a.act_range[2 * blockIdx.x + 1];
  uint32_t solved = 0;
  for (uint32_t j0 = a.act_range[2 * blockIdx.x] + (threadIdx.x & ~31u); j0 < end; j0 += T) {
    bool todo = j0 + lane < end;
    R before = R(0), own = R(0);
    StreamGroup gr{};
    uint32_t number = 0, i = 0, rel = 0, quads = 0;
    R att = R(0), per = R(0), src = R(0);
    float inv = 0.f;
    StreamWeights<R> w[kStreamQuads];
    uint32_t up[kStreamQuads][4];  // positions of the upwind words, kSparseActive: solved in this sweep
    auto quad = [&](const StreamPiece<R>& s, uint32_t c, StreamWeights<R>& w4, uint32_t (&up4)[4]) {
      StreamQuad<R> v;
      v.load(s, c, i);
      w4 = v.w;
      const uint32_t x[4] = {v.x.x & 0xffffu, v.x.x >> 16, v.x.y & 0xffffu, v.x.y >> 16};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t u = kSparseNone;
        if (x[k] != a.shape.ring) {
          u = stream_slot_position(a.shape, s, number, i, rel, x[k]);
          const uint32_t q = sd.base + u;
          if (a.act_bits[q >> 5] >> (q & 31u) & 1u) u |= kSparseActive;
        }
        up4[k] = u;
      }
    };
    if (todo) {
      const uint32_t p = a.act[j0 + lane];
      uint32_t lo = sd.seg0, hi = sd.seg0 + sd.segs;  // the segment of p
      while (hi - lo > 1) {
        const uint32_t m = (lo + hi) / 2;
        if (a.seg[m] <= p) lo = m;
        else hi = m;
      }
      const uint32_t in_seg = p - a.seg[lo], g = a.seg_group[lo] + in_seg / kStreamGroup;
      i = in_seg % kStreamGroup;
      rel = p - sd.base;
      number = g - sd.group0;
      gr = a.groups[g];
      const uint32_t id = a.order[p];
      att = a.cell_att[id % a.Np];
      if constexpr (kChange) {
        before = __ldcg(inc + rel);
        own = __ldcg(a.out + p);
      }
      const StreamPiece<R> s(a.data + kStreamUnit * gr.data, gr);
      quads = s.quads;
      if (gr.shape & kGroupExt) {
        per = a.periodic[id];
        src = s.src()[i];
      }
      if (sizeof(R) == 4) inv = s.inv()[i];
#pragma unroll
      for (uint32_t c = 0; c < kStreamQuads; ++c)
        if (c < quads) quad(s, c, w[c], up[c]);
    }
    auto attempt = [&]() {
      bool ready = true;
      StreamSum<R> sum(before);
      auto add = [&](bool odd, const StreamWeights<R>& w4, const uint32_t (&up4)[4]) {
        R q[4];
        st_try(a, word, sd.base, up4, sweep, ready, q);
        st_add(sum, odd, w4, q);
      };
#pragma unroll
      for (uint32_t c = 0; c < kStreamQuads; ++c)
        if (c < quads) add(c & 1u, w[c], up[c]);
      if (quads > kStreamQuads) {
        const StreamPiece<R> s(a.data + kStreamUnit * gr.data, gr);
        for (uint32_t c = kStreamQuads; c < quads; ++c) {
          StreamWeights<R> w4;
          uint32_t up4[4];
          quad(s, c, w4, up4);
          add(c & 1u, w4, up4);
        }
      }
      if (ready) {
        R in = sum.total();
        if constexpr (kChange) {
          in = st_positive(in);
          const R out = st_solve(in, src, per, att, a.threshold, inv);
          st_publish(a, word, sd.base, rel, out - own, sweep);
          a.out[sd.base + rel] = out;
        } else {
          st_publish(a, word, sd.base, rel, st_solve(in, src, per, att, a.threshold, inv), sweep);
        }
        inc[rel] = in;
        ++solved;
        todo = false;
      }
    };
    unsigned long long w0 = 0;
    for (uint32_t k = 1; __any_sync(0xffffffffu, todo); ++k) {
      if (todo) attempt();
      if ((k & 255u) == 0) {
        const unsigned long long now = __shfl_sync(0xffffffffu, globaltimer_ns(), 0);
        if (w0 == 0) w0 = now;
        if (now - w0 > a.timeout_ns || __any_sync(0xffffffffu, st_stalled(a.ctl))) break;
      }
    }
    if (__any_sync(0xffffffffu, todo)) {  // stalled: those that wait for this warp's tasks run out as well
      if (lane == 0) atomicOr(&a.ctl->error, kErrStall);
      break;
    }
  }
  for (int o = 16; o > 0; o >>= 1) solved += __shfl_xor_sync(0xffffffffu, solved, o);
  if (lane == 0 && solved) {
    atomicAdd(&a.ctl->tasks, (unsigned long long)solved);
    atomicAdd(&a.ctl->attempts, (unsigned long long)solved);
  }
}

// Before a sweep: the attenuations (or the inactive mark) of the groups' tasks from their
// cells, and the periodic sources of the groups that have any; one group per warp.
template <typename R>
__global__ void k_stream_gather(const StreamGroup* groups, uint32_t ngroups, unsigned char* data, const uint32_t* order,
                                uint32_t Np, const R* cell_att, const R* periodic) {
  const uint32_t lane = threadIdx.x & 31;
  const float inv_np = 1.0f / (float)Np;
  for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / 32; g < ngroups; g += gridDim.x * blockDim.x / 32) {
    const StreamGroup gr = groups[g];
    const StreamPiece<R> s(data + kStreamUnit * gr.data, gr);
    if (lane >= group_tasks(gr.shape)) continue;
    const uint32_t t = order[gr.pos + lane];
    // the cell: t modulo Np (the FP32 quotient is off by one at most)
    long long c = (long long)t - (long long)(int)(__uint2float_rn(t) * inv_np) * Np;
    if (c < 0) c += Np;
    if (c >= (long long)Np) c -= Np;
    const_cast<R*>(s.att())[lane] = cell_att[c];
    if (gr.shape & kGroupExt) const_cast<R*>(s.per())[lane] = periodic[t];
  }
}

// Mixed path: a sweep writes the incoming rates of the active cells only; those of the others are brought up
// to date when something asks for them, as the reference keeps adding corrections to inactive
// cells.  Out of date: a LOCAL neighbour was solved in a later sweep.
static __global__ void k_stream_stale(uint32_t n, const uint32_t* off, const uint32_t* nbr, const uint32_t* cell_sweep,
                                      uint8_t* stale) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    const uint32_t mine = cell_sweep[c];
    uint8_t s = 0;
    for (uint32_t f = off[c]; f < off[c + 1] && !s; ++f) {
      const uint32_t nb = nbr[f];
      if ((nb >> kKindShift) == kKindLocal && cell_sweep[nb & kNbrMask] > mine) s = 1;
    }
    stale[c] = s;
  }
}

// From the words in memory, one fused multiply-add per slot in order (in face order, as gather_in
// sums them).  grid: (streams, any).  Bound by the pieces' bytes: 64^3 x 84 in the mixed
// path 1.5 ms per export from the geometry, 0.4 ms so.
static __global__ void k_stream_refresh(StreamArgs<float> a, const uint8_t* stale) {
  const StreamDesc sd = a.streams[blockIdx.x];
  const uint32_t lane = threadIdx.x & 31, warps = gridDim.y * (blockDim.x / 32);
  const auto* word = a.word + sd.base;
  for (uint32_t number = blockIdx.y * (blockDim.x / 32) + threadIdx.x / 32; number < sd.groups; number += warps) {
    const StreamGroup gr = a.groups[sd.group0 + number];
    if (lane >= group_tasks(gr.shape) || stale[a.order[gr.pos + lane] % a.Np] == 0) continue;
    const StreamPiece<float> s(a.data + kStreamUnit * gr.data, gr);
    const uint32_t rel = gr.pos - sd.base + lane;
    float sum = 0.f;
    for (uint32_t j = 0; j < s.quads; ++j) {
      StreamQuad<float> t;
      t.load(s, j, lane);
      const uint32_t x[4] = {t.x.x & 0xffffu, t.x.x >> 16, t.x.y & 0xffffu, t.x.y >> 16};
      float q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        q[k] = x[k] == a.shape.ring ? 0.f : st_ldq(word + stream_slot_position(a.shape, s, number, lane, rel, x[k]));
#pragma unroll
      for (int k = 0; k < 4; ++k) sum = fma(t.w.get(k), q[k], sum);
    }
    a.inc[sd.base + rel] = sum;
  }
}

// The active positions of every stream: ranks of its first position and its end in the bitmap
// of active positions (chunk: the scanned counts of every 256 words).
static __global__ void k_stream_act_range(const uint32_t* bitmap, const uint32_t* chunk, const StreamDesc* streams,
                                          uint32_t n, uint32_t total, const uint32_t* count, uint32_t* range) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
  for (uint32_t s = warp; s < 2 * n; s += gridDim.x * blockDim.x / 32) {
    const StreamDesc& d = streams[s / 2];
    const uint32_t p = d.base + (s & 1u ? d.count : 0u), w = p >> 5, w0 = w & ~255u;
    if (p == total) {
      if (lane == 0) range[s] = *count;
      continue;
    }
    uint32_t m = 0;
    for (uint32_t i = w0 + lane; i < w; i += 32) m += __popc(bitmap[i]);
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    if (lane == 0) range[s] = chunk[w >> 8] + m + __popc(bitmap[w] & ((1u << (p & 31u)) - 1u));
  }
}

// ---------------------------------------------------------------------------------------
// Build, once per grid.  gseg[G]: the groups' level segments; seg, sbase, sgroup: the
// segments' first positions and the first position and group of their streams.
struct StreamBuild {
  StreamGroup* groups;
  uint32_t num_groups;
  const uint32_t *gseg, *seg, *seg_group, *sbase, *sgroup;
  uint32_t segs;
  unsigned char* data;  // null: only the groups' flags and far words per task are found
  StreamShape shape;
};

// One upwind word of a task: its slot index, or the number of the far word it becomes.
struct StreamSlot {
  uint32_t number;   // of the group in its stream
  uint32_t base, end, early;  // first position; relative: end of the level, end of what is solved early
  uint32_t far;      // far words so far
  bool late;
};
__device__ __forceinline__ StreamSlot stream_slots(const StreamBuild& b, uint32_t g) {
  StreamSlot s;
  const uint32_t k = b.gseg[g];
  s.base = b.sbase[k];
  s.number = g - b.sgroup[k];
  s.end = b.seg[k + 1] - s.base;
  // when a warp takes this group up it has waited for the levels before its previous group's
  const uint32_t turn = b.shape.warps * b.shape.blocks;
  s.early = s.number >= turn ? b.seg[b.gseg[g - turn]] - s.base : 0u;
  s.far = 0;
  s.late = false;
  return s;
}
// the level segment of a position
__device__ __forceinline__ uint32_t segment_of(const StreamBuild& b, uint32_t p) {
  uint32_t lo = 0, hi = b.segs;
  while (hi - lo > 1) {
    const uint32_t m = (lo + hi) / 2;
    if (b.seg[m] <= p) lo = m;
    else hi = m;
  }
  return lo;
}
__device__ __forceinline__ uint32_t stream_slot(const StreamBuild& b, StreamSlot& s, uint32_t shape, uint32_t lane,
                                                uint32_t up) {
  if (b.shape.ring && up + b.shape.ring >= s.end) return up % b.shape.ring;
  const uint32_t f = s.far++;
  s.late = s.late || up >= s.early;
  if (!b.data) {  // the group that holds the word keeps it in memory for this one
    const uint32_t p = s.base + up, k = segment_of(b, p);
    atomicOr(&b.groups[b.seg_group[k] + (p - b.seg[k]) / kStreamGroup].shape, kGroupKeep);
  }
  return b.shape.ring + kStreamZero +
         ((shape & kGroupSlow) ? f : (s.number % b.shape.warps * b.shape.far + f) * 32u + lane);
}
// flags and far words of a group from those of its tasks (all lanes)
__device__ __forceinline__ uint32_t stream_flags(bool ext, const StreamSlot& s, uint32_t max_far) {
  uint32_t far = s.far;
  for (int o = 16; o > 0; o >>= 1) far = max(far, __shfl_xor_sync(0xffffffffu, far, o));
  uint32_t f = far << 17;
  if (__any_sync(0xffffffffu, ext)) f |= kGroupExt;
  if (__any_sync(0xffffffffu, s.late)) f |= kGroupLate;
  if (far > max_far) f |= kGroupSlow;
  return f;
}

static __global__ void k_stream_group_segs(const uint32_t* seg_group, uint32_t segs, uint32_t* gseg) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
  for (uint32_t s = warp; s < segs; s += gridDim.x * blockDim.x / 32)
    for (uint32_t g = seg_group[s] + lane; g < seg_group[s + 1]; g += 32) gseg[g] = s;
}

}  // namespace swk

// Types and constants shared by the host runtime and the sweep kernels.
#pragma once

#include <cstdint>

namespace swk {

// Face geometry in FP64: normal and area in one 32-byte load.
struct alignas(32) Geo64 {
  double x, y, z, w;
};

constexpr int kMaxFaces = 64;       // per cell (validated at upload)
constexpr int kMaxDirections = 128;
constexpr uint32_t kKindShift = 30;
constexpr uint32_t kNbrMask = (1u << kKindShift) - 1;
constexpr uint32_t kKindLocal = 0, kKindPeriodic = 1, kKindBoundary = 2;
constexpr uint32_t kEmptySlot = 0xffffffffu;
// stable compaction of schedule positions (pull path): threads per block, positions per
// thread, positions per chunk
constexpr int kCompactThreads = 256;
constexpr int kCompactPer = 8;
constexpr uint32_t kCompactChunk = kCompactThreads * kCompactPer;

// Direction streams (sweep_stream.cuh): the tasks of one direction over one closed range
// of cells, positions [base, base + count), in groups of up to kStreamGroup consecutive
// positions of one level (the tasks of a warp).
struct StreamDesc {
  uint32_t base, count;
  uint32_t group0, groups;
  uint32_t dir;
  uint32_t seg0, segs;  // its dependency levels: segments [seg0, seg0 + segs)
  uint32_t pad;
};
struct alignas(16) StreamGroup {
  uint32_t need;   // groups of the stream in earlier levels: solved before this one
  uint32_t data;   // its piece of data, in units of kStreamUnit bytes
  uint32_t pos;    // first position
  uint32_t shape;  // tasks - 1 | slots per task << 5 | kGroup* flags | far words per task << 17
};
// Groups [begin, end) of a stream, walked by a pair of blocks; wait, post: 1 + the flag to wait
// for before them or to set after them, or 0.
struct StreamPart {
  uint32_t stream, begin, end, wait, post;
};
constexpr unsigned long long kStreamUnit = 64;  // pieces of up to 256 GB in 32 bits
constexpr uint32_t kStreamGroup = 32;
constexpr int kPairWarps = 15;             // of each block of a pair that solve, and one more
constexpr uint32_t kGroupExt = 1u << 12;   // a task has a periodic source or a cell with a source
constexpr uint32_t kGroupLate = 1u << 13;  // a far word may be solved after the warp's previous group
constexpr uint32_t kGroupSlow = 1u << 14;  // more far words than the buffer holds
constexpr uint32_t kGroupKeep = 1u << 15;  // a word of it is a far word of another group
constexpr uint32_t kStreamFar = 8;         // far words of a task in the buffer at most

enum : uint32_t { kErrStall = 1u, kErrQueue = 2u, kErrClamp = 8u, kErrRecords = 16u };
constexpr uint32_t kErrFailed = kErrStall | kErrQueue | kErrClamp;  // of a step

// Control block of one handle (device memory).
struct SweepCtl {
  unsigned long long head;  // next ready-queue slot to claim (consumers); pull wavefront: barrier arrivals;
                            // pairs of blocks: clusters that have started
  unsigned long long tail;  // next ready-queue slot to fill (producers)
  uint32_t error;           // kErr* bits
  uint32_t pad;
  unsigned long long tasks;     // solved tasks (cumulative)
  unsigned long long chem_cells;
  unsigned long long chem_attempts;
  unsigned long long chem_failures;
  unsigned long long attempts;  // task attempts of the pull transport (retries included)
  uint32_t n_ge[32];       // number of cells with level >= l (current level assignment)
  uint32_t hist[32];       // scratch level histogram
  // scalars of a step replayed from a CUDA graph, copied in by the graph's first node
  uint32_t epoch_base;     // sweep number before the step's first sweep
  uint32_t pad2;
  double time;             // simulation time at the end of the step
};

}  // namespace swk

// The FFA search kernels (ffa_search.cu): task tables, schedules and launch
// arguments shared with the host side (ffa.cu).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace gf {

// Search CTAs: tasks that fit one 512-thread CTA's tiles (110 KB, two CTAs
// per SM, more items in flight) run there; larger tasks run on one
// 1024-thread CTA per SM (222 KB: larger subtrees and column blocks; 45.9
// against 50.4 ms with two 512-thread CTAs for every task, 32 series of 2^22
// samples on the survey plan).
constexpr int kThreads = 1024;
constexpr int kSmallThreads = 512;
constexpr size_t kSmallSmem = 110 * 1024, kLargeSmem = 222 * 1024;
constexpr int kMaxBins = 512;
constexpr int kMaxWidths = 64;

struct TaskDev {
  uint32_t bins, rows, rows_eval, octave;
  uint64_t prep_offset;   // floats from the series' prepared block
  float inv_stdnoise;
  uint32_t ntrials;
  uint32_t trial_offset;
  uint32_t split_depth;   // depth of the on-chip subtrees (0: whole task in one CTA)
  uint32_t max_width;
  uint32_t pass_begin;    // column passes (split_depth > 0)
  uint32_t npasses;
  uint32_t first_depth;   // depth of the first pass's nodes
  uint32_t member;        // observation of a batched program (0 otherwise)
};

// Batched programs: one observation's prepared series, and a run of items
// (all series of one task of one observation) in a class's item order.
struct MemberDev {
  const float* prepared;
  uint64_t prep_stride;
};

struct UnitDev {
  uint64_t item_begin;
  uint32_t task;
  uint32_t member;
};

struct TrialDev {
  float height, baseline;
  uint32_t width, reserved;
};

// ---------------------------------------------------------------------------
// FFA tree evaluation
// ---------------------------------------------------------------------------
//
// A level of the tree is a list of rows, each produced by one MetaEntry:
//   MERGE  out = prev[a] + roll_left(prev[b], roll mod bins)   (ffa.cpp:110-171)
//   CARRY  out = prev[a]              (a one-row node carried up unchanged)
// Levels are evaluated two at a time: a pass of QuadOps reads the rows two
// levels down and writes groups of up to four consecutive rows, the level
// between kept in registers.  Neighbouring rows of a node share their head
// and tail rows (the shift of row s is split between the children as s/2 each,
// rounded), so a group of four needs two head rows, each once, and two or three
// tail rows, at one or two neighbouring phases each:
//   R  outputs h0 + w0(k), h0 + w0(k+1), h1 + w1(k), h1 + w1(k+1)
//   F  outputs h0 + w0(k), h0 + w1(k),   h1 + w1(k+1), h1 + w2(k)
// with h_i = a_i + roll(b_i) and w_i = roll(c_i + roll(d_i)), every sum in the
// reference's order.  RS and FS are the same with the children's own rows
// shared (a1 = a0, b1 = b0 one phase on; likewise c, d in RS); rows that fit no
// group are pairs (two rows of one head and tail) or single rows.  Bound:
// shared-memory accesses -- 16 per 8 merged elements in R and F, 14 in RS and
// FS, 8 per 4 in pairs, against 24 per 8 one level at a time -- and the warps
// in flight that hide their latency: 1024 threads of 64 registers beat 512 of
// 128 with twice the loads ahead (43.7 against 49.1 ms, 32 series of 2^22
// samples on the survey plan).  Rows hold three wrapped samples past their end
// so that neighbouring phases need no index of their own.  A task of an odd number of levels takes
// one level by itself (MetaEntries).
// Rows of a pass live in one of two shared-memory buffers (pitch =
// (bins + 3) | 1); passes alternate buffers, so each costs one __syncthreads.
// Every loop over the bins of a row is unrolled for NB = ceil(bins / 32) (the
// kernels are instantiated per NB).

enum : uint16_t { kMerge = 0, kCarry = 1 };

struct __align__(8) MetaEntry {
  uint16_t op, a, b, roll;
};

enum : uint16_t { kOpR = 0, kOpRS, kOpF, kOpFS, kOpPair, kOpOne };
constexpr uint32_t kHalo = 3;   // wrapped samples kept past the end of a row

// Group of output rows row, row + 1, ...; rolls are phases relative to the
// output (rd: of d itself, the tail's roll included).
struct __align__(16) QuadOp {
  uint16_t type, row;
  uint16_t a[2], b[2], rb[2];
  uint16_t c[3], d[3], rc[3], rd[3];
  uint16_t flags;               // kOpOne: 1 = b present, 2 = c present, 4 = d present
  uint16_t pad[3];
};
static_assert(sizeof(QuadOp) == 48, "QuadOp is three 16-byte words");

// A pass: bit 15 = two levels (QuadOps) or one (MetaEntries); low bits the count.
constexpr uint16_t kPassTwo = 0x8000;
constexpr int kMaxPasses = 10;
__host__ __device__ __forceinline__ uint32_t pass_bytes(uint16_t pass) {
  const uint32_t n = pass & 0x7fffu;
  return pass & kPassTwo ? n * static_cast<uint32_t>(sizeof(QuadOp))
                         : (n * static_cast<uint32_t>(sizeof(MetaEntry)) + 15u) & ~15u;
}

// Schedule of a whole subtree of n rows: passes from the leaves to the root.
// The head also leads the staged entries.
struct __align__(16) SubHead {
  uint32_t offset16;            // first 16-byte word of the passes' entries
  uint16_t size16;
  uint16_t npasses;
  uint16_t pass[kMaxPasses];
  uint16_t pad[2];
};
static_assert(sizeof(SubHead) == 32, "SubHead is two 16-byte words");

struct Node {
  uint32_t a, n, depth;
};

// The node at depth `depth` containing row r (stops at one-row nodes).
__device__ __forceinline__ Node node_of(uint32_t r, uint32_t n, uint32_t depth) {
  Node nd{0u, n, 0u};
  while (nd.depth < depth && nd.n > 1) {
    const uint32_t h = nd.n >> 1;
    if (r - nd.a < h) {
      nd.n = h;
    } else {
      nd.a += h;
      nd.n -= h;
    }
    ++nd.depth;
  }
  return nd;
}

// Node `index` (bits read MSB first, 0 = head) at depth `depth`.
__host__ __device__ __forceinline__ Node node_at(uint32_t index, uint32_t n, uint32_t depth) {
  Node nd{0u, n, depth};
  for (uint32_t b = depth; b-- > 0;) {
    const uint32_t h = nd.n >> 1;
    if ((index >> b) & 1u) {
      nd.a += h;
      nd.n -= h;
    } else {
      nd.n = h;
    }
  }
  return nd;
}

// ffa.cpp:153-171: hs = (size_t)(float((h-1)/(n-1)) * s + 0.5f), likewise ts
__device__ __forceinline__ float shift_scale(uint32_t part, uint32_t n) {
  return __fdiv_rn(static_cast<float>(part - 1), static_cast<float>(n - 1));
}
__device__ __forceinline__ uint32_t scaled_shift(float scale, uint32_t s) {
  return static_cast<uint32_t>(__fadd_rn(__fmul_rn(scale, static_cast<float>(s)), 0.5f));
}

// A column block of a pass (built on the host): rows [s0, s1) of one node X
// at depth dx, evaluated from the rows of depth dx + levels that they depend
// on.  The bottom level is loaded from the pass's source scratch as up to 8
// runs of consecutive task rows.
struct ColBlock {
  uint32_t meta16;        // first 16-byte word of the passes' entries, bottom pass first
  uint32_t out_row;       // final pass: shift of the first root row; else task row of the first output row
  uint16_t rows;          // output rows
  uint16_t nbottom;       // bottom rows
  uint16_t size16;        // entries in 16-byte words
  uint16_t pass[3];
  uint16_t run_off[8];    // bottom level: buffer row where each run starts
  uint16_t run_row[8];    // bottom level: task row where each run starts
  uint8_t npasses, final_pass, nruns, reserved;
  uint32_t pad[2];
};
static_assert(sizeof(ColBlock) == 64, "ColBlock is 16 words");

struct PassDev {
  uint32_t block_begin, nblocks;
};

struct SearchParams {
  const float* prepared;
  uint64_t prep_stride;
  const TaskDev* tasks;
  const TrialDev* trials;
  const uint4* sub_meta;        // subtree schedules
  const SubHead* sub_head;      // [max_rows + 1] by size
  const uint4* col_meta;        // column-block schedules
  const ColBlock* blocks;       // column blocks, pass by pass
  const PassDev* passes;
  const uint32_t* item_tasks;   // task indices of this launch's class
  uint32_t nitem_tasks;
  uint32_t nseries;
  const UnitDev* units;         // batched programs: item runs of this class (else null)
  const MemberDev* members;
  uint32_t nunits;
  uint64_t nitems;
  float threshold;
  gf_peak_record* peaks;
  uint64_t capacity;
  unsigned long long* counters;
  float* scratch;               // per CTA: scratch_elems0 + scratch_elems1 floats
  uint64_t scratch_elems0, scratch_elems1;
  uint32_t pitch;               // shared-memory row pitch ((max bins + 3) | 1)
  uint32_t max_rows;            // rows per shared-memory buffer
  uint32_t front;               // floats before the first row buffer
  uint32_t block_rows;          // output rows of a column block (passes but the last)
};

using SearchKernel = void (*)(SearchParams);

// ffa_search_kernel<NB, T> for NB = 2 Part + 1 and 2 Part + 2 (bins <= 512), T =
// 512 or 1024.  Each part is an object of its own: the 32 kernels take minutes
// in one compilation.
template <int Part>
SearchKernel search_kernel_part(uint32_t nb, int threads);

}  // namespace gf

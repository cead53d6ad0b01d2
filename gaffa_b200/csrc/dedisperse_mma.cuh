// The tensor-core dedispersion kernels (dedisperse_mma.cu): launch arguments,
// shapes and tables.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace gf {

constexpr int kMmaThreads = 352;        // loader, 2 issuers, 8 scatter / epilogue warps
constexpr int kMmaTile = 2048;          // samples per accumulator tile: 128 lanes x 16 phases
constexpr int kMmaSlots = 16;           // DMs x tiles per CTA (16 TMEM columns each)
constexpr int kMmaColumns = 16 * kMmaSlots;
constexpr int kMmaStages = 8;           // deepest ring
constexpr int kMmaRecord = 96;          // offsets mod 16 [16], slice count, slices [16]
constexpr int kMmaRecordArea = 128;
constexpr int kDenseDms = 8;            // dense form: 8 DMs x 16 phases are the rows of the ones' matrix
constexpr int kDenseRecord = 32;        // offsets (16 bits) [8], steps
constexpr int kDenseMaxSteps = 7;
constexpr size_t kMmaBudget = 110 * 1024;   // two CTAs per SM
constexpr size_t kMmaMinSmem = 80 * 1024;   // never three (TMEM holds two)

// slice word: q (units of 16 samples) in bits [0,12), first DM in [12,16),
// DMs in [18,23) (the place of N / 16 in the instruction descriptor, shifted)
constexpr uint32_t kSliceN = 18;

struct MmaParams {
  const uint8_t* in;
  uint64_t in_row_stride, in_group_stride, in_valid;
  int rows_per_group, total_rows;
  const int32_t* base;        // + group * base_group_stride + block * base_block_stride: window base per row
  uint64_t base_group_stride, base_block_stride;
  const uint8_t* records;     // + group * rec_group_stride + block * rec_block_stride + row * kMmaRecord
  uint64_t rec_group_stride, rec_block_stride;
  int nblocks;                // DM blocks per group in the launch (fastest grid index)
  int dm_skip;                // DMs of the first block before the launch's range
  int dm_count, dm_count_last, ngroups;
  int dms, tiles;             // D, T
  int steps;                  // dense form: K steps of the widest row (0: slices)
  uint32_t row_bytes;         // window bytes per row
  uint64_t whole_end;         // windows of tiles that start below this lie inside the valid samples
  uint32_t stage_bytes;
  int stages;
  void* out;
  uint64_t out_row_stride, out_dm_rows, out_group_rows, nout;
  uint32_t grid_x;
  uint32_t* status;
};

// One launch over `groups` groups (out: 8-bit sums, or 32-bit).
void launch_mma(const MmaParams& p, int groups, size_t smem, bool bytes_out, cudaStream_t stream);
// Many launches of one form as one grid: item tables on the device.
void launch_mma_batch(const MmaParams* items, const uint64_t* block_begin, int nitems, uint64_t blocks, size_t smem,
                      bool dense, cudaStream_t stream);

namespace {

// -- host side -----------------------------------------------------------------

struct MmaShape {
  int dms = 0, tiles = 0;   // dms = 0: not used
  int steps = 0;            // dense form
  uint32_t row_bytes = 0, stage_bytes = 0;
  int stages = 0;
  size_t smem = 0;
  double clocks = 0;        // estimated tensor-core and shared-memory clocks of a CTA's row
};

// Clocks of a dense step (128 x 256 x 32 multiply-adds; measured 128.3), and
// what the slices take over their own clocks (their issue does not keep up).
constexpr double kDenseStepClocks = 128, kSliceOverhead = 1.6;

// Slices of one (block, row): runs of at most 8 consecutive DMs, not across
// DM 8 (the issuers' border), with equal offset / 16.  offs[i] is relative to
// the row's window base; `n` DMs.  Words of DMs 8.. start at words[8]; returns
// the two counts, the second in bits [8,16).
uint32_t mma_slices(const int32_t* offs, int n, uint32_t* words) {
  uint32_t counts = 0;
  for (int half = 0; half < 2; ++half) {
    int ns = 0;
    const int end = std::min(n, 8 * half + 8);
    for (int i = 8 * half; i < end;) {
      int e = i + 1;
      while (e < end && (offs[e] >> 4) == (offs[i] >> 4)) ++e;
      words[8 * half + ns++] = static_cast<uint32_t>(offs[i] >> 4) | (static_cast<uint32_t>(i) << 12) |
                               (static_cast<uint32_t>(e - i) << kSliceN);
      i = e;
    }
    counts |= static_cast<uint32_t>(ns) << (8 * half);
  }
  return counts;
}

// The delays of one (group, DM block, row) relative to its window base (the
// smallest delay rounded down to 16); returns the base.
int32_t mma_offsets(const std::vector<int32_t>& delays, int group, int ndm_group, int rows_per_group, int row, int d0,
                    int n, int32_t* offs) {
  const int32_t* d = delays.data() + (static_cast<size_t>(group) * ndm_group + d0) * rows_per_group + row;
  int32_t lo = *d;
  for (int i = 0; i < n; ++i) lo = std::min(lo, offs[i] = d[static_cast<size_t>(i) * rows_per_group]);
  lo &= ~15;
  for (int i = 0; i < n; ++i) offs[i] -= lo;
  return lo;
}

// The window bases of every row of a (group, DM block), as mma_offsets gives
// them, in passes along the rows; returns the largest offset.
int32_t mma_bases(const std::vector<int32_t>& delays, int group, int ndm_group, int rows_per_group, int rows, int d0,
                  int n, int32_t* base) {
  const int32_t* d = delays.data() + (static_cast<size_t>(group) * ndm_group + d0) * rows_per_group;
  std::copy(d, d + rows, base);
  for (int i = 1; i < n; ++i)
    for (int row = 0; row < rows; ++row) base[row] = std::min(base[row], d[static_cast<size_t>(i) * rows_per_group + row]);
  for (int row = 0; row < rows; ++row) base[row] &= ~15;
  int32_t most = 0;
  for (int i = 0; i < n; ++i)
    for (int row = 0; row < rows; ++row) most = std::max(most, d[static_cast<size_t>(i) * rows_per_group + row] - base[row]);
  return most;
}

// Tensor-core clocks of one (block, row) step list, plus the shared-memory
// clocks of the window's arrival and of writing B.
double mma_row_clocks(const uint32_t* words, uint32_t counts, int D, int tiles) {
  double c = 0;
  int qmax = 0;
  for (int i = 0; i < kMmaSlots; ++i) {
    if (static_cast<uint32_t>(i & 7) >= ((counts >> (i & 8)) & 0xffu)) continue;
    const int n = static_cast<int>(words[i] >> kSliceN);
    c += tiles * std::max(39, std::max(32 + 4 * n, 8 * n));
    qmax = std::max(qmax, static_cast<int>(words[i] & 0xfffu));
  }
  return c + (16 * qmax + 16 + tiles * kMmaTile) / 128.0 + D;
}

MmaShape mma_shape(int D, int max_off) {
  MmaShape m;
  if (max_off >= (1 << 16)) return m;
  const int tiles = kMmaSlots / D;
  const uint32_t row = static_cast<uint32_t>(16 * (max_off >> 4) + 16 + tiles * kMmaTile);
  const uint32_t stage = static_cast<uint32_t>(round_up(row, 128)) + 512u * D + kMmaRecordArea;
  const int stages = std::min<int>(kMmaStages, static_cast<int>(kMmaBudget / stage));
  if (stages < 3) return m;
  m.dms = D;
  m.tiles = tiles;
  m.row_bytes = row;
  m.stage_bytes = stage;
  m.stages = stages;
  m.smem = std::max<size_t>(kMmaMinSmem, static_cast<size_t>(stages) * stage);
  return m;
}

// Steps of a row in the dense form: offsets 0 .. max_off, 16 phases each.
int dense_steps(int max_off) { return (max_off + 15) / 32 + 1; }

MmaShape dense_shape(int max_off) {
  MmaShape m;
  const int steps = dense_steps(max_off);
  if (steps > kDenseMaxSteps) return m;
  const uint32_t row = static_cast<uint32_t>(32 * steps + 2 * kMmaTile - 16);
  const uint32_t stage = static_cast<uint32_t>(round_up(row, 128)) + 4096u * steps + kMmaRecordArea;
  const int stages = std::min<int>(kMmaStages, static_cast<int>(kMmaBudget / stage));
  if (stages < 3) return m;
  m.dms = kDenseDms;
  m.tiles = 2;
  m.steps = steps;
  m.row_bytes = row;
  m.stage_bytes = stage;
  m.stages = stages;
  m.smem = std::max<size_t>(kMmaMinSmem, static_cast<size_t>(stages) * stage);
  return m;
}

// DMs per CTA by the clocks of the steps they need, over a sample of (block,
// row) pairs; shapes whose ring does not fit are passed over.
MmaShape choose_mma_shape(const std::vector<int32_t>& delays, int ngroups, int ndm_group, int rows_per_group,
                          int total_rows) {
  struct Option {
    double clocks;
    int D;
  };
  std::vector<Option> options;
  int32_t offs[kMmaSlots];
  uint32_t words[kMmaSlots];
  for (int D = kMmaSlots; D >= 1; D >>= 1) {
    const int blocks = static_cast<int>(ceil_div(ndm_group, D));
    const uint64_t pairs = static_cast<uint64_t>(ngroups) * blocks * rows_per_group;
    const uint64_t step = std::max<uint64_t>(1, pairs / 256) | 1;
    double clocks = 0;
    uint64_t count = 0;
    for (uint64_t i = 0; i < pairs; i += step) {
      const int row = static_cast<int>(i % rows_per_group), b = static_cast<int>(i / rows_per_group % blocks);
      const int g = static_cast<int>(i / rows_per_group / blocks);
      if (g * rows_per_group + row >= total_rows) continue;
      const int n = std::min(D, ndm_group - b * D);
      mma_offsets(delays, g, ndm_group, rows_per_group, row, b * D, n, offs);
      if (*std::max_element(offs, offs + n) >= (1 << 16)) { clocks = INFINITY; break; }
      const uint32_t counts = mma_slices(offs, n, words);
      clocks += kSliceOverhead * mma_row_clocks(words, counts, D, kMmaSlots / D);
      count += static_cast<uint64_t>(n) * (kMmaSlots / D);
    }
    options.push_back(Option{count ? clocks / static_cast<double>(count) : INFINITY, D});
  }
  // the dense form, as an option of its own (D = 0)
  {
    const int blocks = static_cast<int>(ceil_div(ndm_group, kDenseDms));
    const uint64_t pairs = static_cast<uint64_t>(ngroups) * blocks * rows_per_group;
    const uint64_t step = std::max<uint64_t>(1, pairs / 256) | 1;
    double clocks = 0;
    uint64_t count = 0;
    for (uint64_t i = 0; i < pairs; i += step) {
      const int row = static_cast<int>(i % rows_per_group), b = static_cast<int>(i / rows_per_group % blocks);
      const int g = static_cast<int>(i / rows_per_group / blocks);
      if (g * rows_per_group + row >= total_rows) continue;
      const int n = std::min(kDenseDms, ndm_group - b * kDenseDms);
      mma_offsets(delays, g, ndm_group, rows_per_group, row, b * kDenseDms, n, offs);
      clocks += kDenseStepClocks * dense_steps(*std::max_element(offs, offs + n));
      count += static_cast<uint64_t>(n) * 2;
    }
    options.push_back(Option{count ? clocks / static_cast<double>(count) : INFINITY, 0});
  }
  std::stable_sort(options.begin(), options.end(), [](const Option& x, const Option& y) { return x.clocks < y.clocks; });
  for (const Option& o : options) {
    if (!std::isfinite(o.clocks)) continue;
    int max_off = 0;
    std::vector<int32_t> base(rows_per_group);
    const int D = o.D ? o.D : kDenseDms;
    const int blocks = static_cast<int>(ceil_div(ndm_group, D));
    for (int g = 0; g < ngroups; ++g)
      for (int b = 0; b < blocks; ++b)
        max_off = std::max(max_off, mma_bases(delays, g, ndm_group, rows_per_group,
                                              std::min(rows_per_group, total_rows - g * rows_per_group), b * D,
                                              std::min(D, ndm_group - b * D), base.data()));
    MmaShape m = o.D ? mma_shape(o.D, max_off) : dense_shape(max_off);
    m.clocks = kMmaSlots * o.clocks;
    if (m.dms) return m;
  }
  return MmaShape{};
}

int mma_record_bytes(const MmaShape& m) { return m.steps ? kDenseRecord : kMmaRecord; }

struct MmaTables {
  std::vector<int32_t> base;     // [group][block][base_stride]
  std::vector<uint8_t> records;  // [group][block][rows_per_group][record]
  uint64_t base_stride = 0;
  int blocks = 0;
  int32_t max_base = 0;
};

MmaTables build_mma_tables(const std::vector<int32_t>& delays, int ngroups, int ndm_group, int rows_per_group,
                           int total_rows, const MmaShape& m) {
  MmaTables t;
  t.blocks = static_cast<int>(ceil_div(ndm_group, m.dms));
  t.base_stride = static_cast<uint64_t>(rows_per_group);
  t.base.assign(static_cast<size_t>(ngroups) * t.blocks * t.base_stride, 0);
  const int record = mma_record_bytes(m);
  t.records.assign(static_cast<size_t>(ngroups) * t.blocks * rows_per_group * record, 0);
  int32_t offs[kMmaSlots];
  uint32_t words[kMmaSlots];
  for (int g = 0; g < ngroups; ++g)
    for (int b = 0; b < t.blocks; ++b)
      for (int row = 0; row < std::min(rows_per_group, total_rows - g * rows_per_group); ++row) {
        const int n = std::min(m.dms, ndm_group - b * m.dms);
        const size_t at = (static_cast<size_t>(g) * t.blocks + b) * rows_per_group + row;
        t.base[at] = mma_offsets(delays, g, ndm_group, rows_per_group, row, b * m.dms, n, offs);
        t.max_base = std::max(t.max_base, t.base[at]);
        uint8_t* rec = t.records.data() + at * record;
        if (m.steps) {
          const uint32_t steps = static_cast<uint32_t>(dense_steps(*std::max_element(offs, offs + n)));
          for (int i = 0; i < n; ++i) {
            const uint16_t o = static_cast<uint16_t>(offs[i]);
            std::memcpy(rec + 2 * i, &o, 2);
          }
          std::memcpy(rec + 16, &steps, 4);
          continue;
        }
        for (int i = 0; i < n; ++i) rec[i] = static_cast<uint8_t>(offs[i] & 15);
        std::memset(words, 0, sizeof words);
        const uint32_t counts = mma_slices(offs, n, words);
        std::memcpy(rec + 16, &counts, 4);
        std::memcpy(rec + 32, words, sizeof words);
      }
  return t;
}

}  // namespace
}  // namespace gf

// Dedispersion sums on the tensor cores (tcgen05, 8-bit integer operands,
// 32-bit integer accumulators in TMEM; every product and sum is exact).
//
// The sum of one channel for one DM is a shift: out[t] += row[t + d].  Write
// t = 16 n + r and d = 16 q + o: the samples row[16 n + 16 q + k], k < 32, are
// a matrix with a row per n, and the 16 phases r of a DM are one-hot vectors in
// k (a one at k = o + r).  The sample matrix is the channel's window itself,
// read through a matrix descriptor whose core matrices overlap: 8 rows of 16
// bytes are 128 consecutive samples, and the second half of K starts 16 bytes
// on.  Only the ones are written, one byte per DM and phase and channel.
//
// Dense form.  The ones are the A operand, 128 rows = 8 DMs x 16 phases; the
// samples are B, 256 rows = 4096 samples.  A channel takes one K = 32 step per
// 32 samples of the 8 DMs' delay spread plus 15: few, large steps (128 clk
// each) that one thread issues without effort.  Best while the spread is a few
// steps (DM steps to about 0.8 at 1100-1700 MHz and 64 us).
//
// Slices.  The samples are A (128 rows = 2048 samples), the ones B, 16 columns
// per DM.  A DM needs only the one step at its q, so a step serves the DMs of
// the block that share q, and costs the same multiply-adds per DM whatever the
// spread.  A CTA holds D DMs x T tiles of 2048 samples, D * T = 16.  A step
// reads 4 KB of A and its B from shared memory at 128 B/clk: max(39, 32 + 4 n,
// 8 n) clk for n DMs (measured 39.1, 40.1, 48.2, 64.4, 128.8 for n = 1, 2, 4, 8,
// 16 with constant descriptors; 46-50 for n = 2 with the descriptors formed per
// step, which two issuing warps half hide).
//
// Both: 256 TMEM columns and 110 KB per CTA, two CTAs per SM; a loader warp
// copies a channel's window and record (bulk copies on the stage's mbarrier), a
// warp per stage clears the stage's previous ones and writes the new, the
// issuers' tcgen05.commit frees the stage.
//
// Measured (B200, 1965 MHz), against the byte kernel: 4096 channels over
// 1100-1700 MHz, 2^18 samples, 256 DMs of step 0.4885: 18.0 -> 10.8 ms (51 -> 83
// adds/clk/SM, of 100 at the dense steps' own clocks); 256 channels over
// 1200-1500 MHz, 2^18 samples, 512 DMs of step 0.39: 2.39 -> 1.25 ms (93
// adds/clk/SM); two-stage 2-bit, 4096 channels, 2^19 samples: 2.95 -> 1.47 ms.
#pragma once

namespace gf {
namespace {

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

struct MmaShared {
  uint64_t landed[kMmaStages];  // window and record have arrived
  uint64_t built[kMmaStages];   // the ones are written
  uint64_t done[kMmaStages];    // the tensor core has read the stage (one commit per issuer)
  uint64_t final_bar;           // every step of the CTA has finished
  uint32_t valid[kMmaStages];   // bytes of the stage's window below the row's valid end
  uint32_t tmem;
  uint32_t failed;
};

__device__ __forceinline__ uint32_t elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(p));
  return p;
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
// D[tmem] (+)= A x B for M = 128, N from `idesc`, K = 32
__device__ __forceinline__ void mma_u8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc),
      "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// smem matrix descriptors without swizzle, K-major: start address and the two
// strides in units of 16 bytes (K halves, then groups of 8 rows), version 1
constexpr uint64_t kDescWindow = (1ull << 46) | (static_cast<uint64_t>(128 >> 4) << 32) | (static_cast<uint64_t>(16 >> 4) << 16);
constexpr uint64_t kDescOnes = (1ull << 46) | (static_cast<uint64_t>(256 >> 4) << 32) | (static_cast<uint64_t>(128 >> 4) << 16);
// instruction descriptor: S32 accumulator, unsigned 8-bit A and B, M = 128; N / 8 in bits [17,23)
constexpr uint32_t kIdesc = (2u << 4) | (8u << 24);
constexpr uint32_t kIdescDense = kIdesc | (32u << 17);   // N = 256

// Copies a channel's window and record into stage `s` (whole loader warp).  The
// bulk copy ends on the last 16-byte word with a valid sample (rows are a
// multiple of 16 bytes); the scatter warp clears what lies past the valid end.
__device__ __forceinline__ void mma_load_row(const MmaParams& p, MmaShared& ms, uint8_t* stage, int s, const uint8_t* src,
                                             uint64_t t_row, const uint8_t* rec, uint32_t rec_bytes) {
  if ((threadIdx.x & 31) != 0) return;
  const uint64_t left = t_row < p.in_valid ? p.in_valid - t_row : 0;
  const uint32_t valid = static_cast<uint32_t>(umin64(p.row_bytes, left));
  const uint32_t nbulk = (valid + 15u) & ~15u;   // row_bytes is a multiple of 16
  ms.valid[s] = valid;
  mbar_expect_tx(&ms.landed[s], nbulk + rec_bytes);
  if (nbulk) bulk_copy(stage, src + t_row, nbulk, &ms.landed[s]);
  bulk_copy(stage + p.stage_bytes - kMmaRecordArea, rec, rec_bytes, &ms.landed[s]);
  mbar_arrive(&ms.landed[s]);
}

// Issues the N steps of one channel for tiles [tl0, tl1): straight-line code,
// so that one step's descriptors are formed while the one before is issued.
template <int N>
__device__ __forceinline__ void issue_steps(const uint32_t* words, uint32_t a16, uint32_t b16, uint32_t tmem, int D,
                                            int tl0, int tl1, uint32_t accumulate) {
  uint32_t w[N];
#pragma unroll
  for (int j = 0; j < N; ++j) w[j] = words[j];
  for (int tl = tl0; tl < tl1; ++tl) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const uint32_t f = (w[j] >> 12) & 15u;
      mma_u8(tmem + 16u * (tl * D + f), kDescWindow + (a16 + (w[j] & 0xfffu) + tl * (kMmaTile / 16)), kDescOnes + (b16 + f * 32u),
             kIdesc | (w[j] & (31u << kSliceN)), accumulate);
    }
  }
}

template <typename OutT>
__device__ __forceinline__ void mma_store16(OutT* dst, const uint32_t (&v)[16], uint64_t left) {
  if (left >= 16 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
    if (sizeof(OutT) == 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        reinterpret_cast<uint4*>(dst)[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    } else {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = v[4 * j] | (v[4 * j + 1] << 8) | (v[4 * j + 2] << 16) | (v[4 * j + 3] << 24);
      *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 16; ++j)
    if (static_cast<uint64_t>(j) < left) dst[j] = static_cast<OutT>(v[j]);
}

// One CTA: block bx % nblocks of DMs, time bx / nblocks.
template <typename OutT, bool Dense>
__device__ __forceinline__ void mma_cta(const MmaParams& p, unsigned bx, int group, uint8_t* smem, MmaShared& ms) {
  const int block = static_cast<int>(bx % static_cast<unsigned>(p.nblocks));
  const uint64_t t0 = static_cast<uint64_t>(bx / static_cast<unsigned>(p.nblocks)) * p.tiles * kMmaTile;
  const int warp = __shfl_sync(kFull, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int rows = min(p.rows_per_group, p.total_rows - group * p.rows_per_group);
  const int D = p.dms;
  constexpr uint32_t kRecord = Dense ? kDenseRecord : kMmaRecord;
  const uint32_t rec_off = p.stage_bytes - kMmaRecordArea;
  const uint32_t ones_bytes = Dense ? 4096u * p.steps : 512u * D;
  const uint32_t b_off = rec_off - ones_bytes;  // a stage: window, ones, record

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&ms.landed[s], 1);
      mbar_init(&ms.built[s], 1);
      mbar_init(&ms.done[s], Dense ? 1 : 2);
    }
    mbar_init(&ms.final_bar, Dense ? 1 : 2);
    ms.failed = (*reinterpret_cast<const volatile uint32_t*>(p.status) & GF_STATUS_PIPELINE) ? 1u : 0u;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // the ones' matrix starts as zeros; the scatter warps keep the rest of it so
  for (int s = 0; s < p.stages; ++s)
    for (uint32_t b = 16 * threadIdx.x; b < ones_bytes; b += 16 * kMmaThreads)
      *reinterpret_cast<uint4*>(smem + s * p.stage_bytes + b_off + b) = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  __syncthreads();
  if (ms.failed) return;  // another CTA of the launch gave up
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&ms.tmem)),
                 "r"(kMmaColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ms.tmem;

  if (warp == 0) {
    const int32_t* base = p.base + group * p.base_group_stride + static_cast<uint64_t>(block) * p.base_block_stride;
    const uint8_t* rec = p.records + group * p.rec_group_stride + static_cast<uint64_t>(block) * p.rec_block_stride;
    const uint8_t* src = p.in + group * p.in_group_stride;
    int32_t cur = 0, nxt = lane < rows ? __ldg(base + lane) : 0;
    int s = 0;
    uint32_t parity = 1;
    int k = 0;
    for (; k < rows; ++k) {
      if ((k & 31) == 0) {
        cur = nxt;
        nxt = k + 32 + lane < rows ? __ldg(base + k + 32 + lane) : 0;
      }
      if (k >= p.stages && !wait_warp(&ms.done[s], parity, &ms.failed, p.status)) break;
      const int32_t b = __shfl_sync(kFull, cur, k & 31);
      mma_load_row(p, ms, smem + s * p.stage_bytes, s, src + static_cast<uint64_t>(k) * p.in_row_stride,
                   t0 + static_cast<uint64_t>(b), rec + static_cast<uint64_t>(k) * kRecord, kRecord);
      if (++s == p.stages) { s = 0; parity ^= 1u; }
    }
    if (k < rows) {
      // gave up: the copies in flight land in this CTA's memory, so wait (bounded) for them
      const long long start = clock64();
      for (int j = max(0, k - p.stages); j < k; ++j)
        while (!mbar_try_wait(&ms.landed[j % p.stages], (j / p.stages) & 1) && clock64() - start < kDrainCycles) {
        }
    }
  } else if (Dense && warp == 1) {
    int s = 0;
    uint32_t parity = 0;
    const uint32_t issue = elect_one();
    const uint32_t base16 = smem_u32(smem) >> 4;
    for (int k = 0; k < rows; ++k) {
      // written after the window and record had landed: implies `landed`
      if (!wait_warp(&ms.built[s], parity, &ms.failed, p.status)) break;
      tc_fence_after();
      if (issue) {
        const uint32_t stage16 = base16 + ((s * p.stage_bytes) >> 4);
        const uint32_t steps = *reinterpret_cast<const uint32_t*>(smem + s * p.stage_bytes + rec_off + 16);
        for (uint32_t j = 0; j < steps; ++j)
          mma_u8(tmem, kDescOnes + (stage16 + (b_off >> 4) + j * 256u), kDescWindow + (stage16 + 2u * j), kIdescDense,
                 (k | static_cast<int>(j)) != 0 ? 1u : 0u);
        mma_commit(&ms.done[s]);
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; parity ^= 1u; }
    }
    if (issue) mma_commit(&ms.final_bar);
    __syncwarp();
  } else if (!Dense && warp <= 2) {
    // Two issuers: the first and last 8 DMs of 16, or the first and last half
    // of the tiles, so that an accumulator always has the same one.
    const int half = warp - 1;
    int s = 0;
    uint32_t parity = 0;
    const uint32_t issue = elect_one();
    const uint32_t base16 = smem_u32(smem) >> 4;
    for (int k = 0; k < rows; ++k) {
      // written after the window and record had landed: implies `landed`
      if (!wait_warp(&ms.built[s], parity, &ms.failed, p.status)) break;
      tc_fence_after();
      const uint32_t stage16 = base16 + ((s * p.stage_bytes) >> 4);
      const uint8_t* rec = smem + s * p.stage_bytes + rec_off;
      if (issue) {
        const uint32_t accumulate = k > 0 ? 1u : 0u;
        const uint32_t nsl = *reinterpret_cast<const uint32_t*>(rec + 16);
        const uint32_t* words = reinterpret_cast<const uint32_t*>(rec + 32) + (D == kMmaSlots ? 8 * half : 0);
        const uint32_t b16 = stage16 + (b_off >> 4);
        int tl0 = 0, tl1 = 1;
        if (D < kMmaSlots) {
          tl0 = half * (p.tiles / 2);
          tl1 = tl0 + p.tiles / 2;
        }
        switch ((nsl >> (D == kMmaSlots ? 8 * half : 0)) & 0xffu) {
          case 0: break;
          case 1: issue_steps<1>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
          case 2: issue_steps<2>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
          case 3: issue_steps<3>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
          case 4: issue_steps<4>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
          case 5: issue_steps<5>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
          case 6: issue_steps<6>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
          case 7: issue_steps<7>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
          default: issue_steps<8>(words, stage16, b16, tmem, D, tl0, tl1, accumulate); break;
        }
        mma_commit(&ms.done[s]);
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; parity ^= 1u; }
    }
    if (issue) mma_commit(&ms.final_bar);
    __syncwarp();
  } else if (warp >= 3) {
    // Scatter: a warp per stage, so every stage's ones are written at a time
    // and a stage's phases are waited for one by one (a wait on a barrier two
    // phases on would pass at once).
    // Lane l writes rows l, l + 32, ... of B (row dm * 16 + r; its 32 bytes are
    // two runs of 16, 128 bytes apart).
    const int w = warp - 3;
    const bool ragged = t0 >= p.whole_end;
    bool ok = true;
    const uint32_t row0 = (lane >> 3) * 256 + (lane & 7) * 16;
    const int r = lane & 15;
    const int s = w;
    uint32_t parity = 0;
    uint4 old = make_uint4(0, 0, 0, 0);  // the stage's previous offsets, a byte per DM
    for (int k = w < p.stages ? w : rows; k < rows; k += p.stages, parity ^= 1u) {
      if (!wait_warp(&ms.landed[s], parity, &ms.failed, p.status)) {
        ok = false;
        break;
      }
      uint8_t* stage = smem + s * p.stage_bytes;
      const uint4 rec = *reinterpret_cast<const uint4*>(stage + rec_off);
      // samples past the row's valid end read as zero (the last tiles in time)
      const uint32_t valid = ragged ? ms.valid[s] : p.row_bytes;
      if (valid < p.row_bytes) {
        const uint32_t words = (valid + 15u) & ~15u;
        if (valid + lane < words) stage[valid + lane] = 0;
        for (uint32_t b = words + 16 * lane; b < p.row_bytes; b += 512)
          *reinterpret_cast<uint4*>(stage + b) = make_uint4(0, 0, 0, 0);
      }
      uint8_t* B = stage + b_off + row0;
      if (Dense) {
        // whole offsets, 16 bits per DM: step x / 32, byte x % 32
#pragma unroll
        for (int j = 0; j < kDenseDms / 2; ++j) {
          const uint32_t rw = j == 0 ? rec.x : j == 1 ? rec.y : j == 2 ? rec.z : rec.w;
          const uint32_t ow = j == 0 ? old.x : j == 1 ? old.y : j == 2 ? old.z : old.w;
          const uint32_t shift = lane & 16;
          const uint32_t o = ((ow >> shift) & 0xffffu) + r, x = ((rw >> shift) & 0xffffu) + r;
          B[(o >> 5) * 4096 + j * 1024 + ((o >> 4) & 1u) * 128 + (o & 15u)] = 0;
          B[(x >> 5) * 4096 + j * 1024 + ((x >> 4) & 1u) * 128 + (x & 15u)] = 1;
        }
      }
#pragma unroll
      for (int j = 0; !Dense && j < kMmaSlots / 2; ++j) {
        if (2 * j + (lane >> 4) < D) {
          const uint32_t rw = j < 2 ? rec.x : j < 4 ? rec.y : j < 6 ? rec.z : rec.w;
          const uint32_t ow = j < 2 ? old.x : j < 4 ? old.y : j < 6 ? old.z : old.w;
          const uint32_t shift = 16 * (j & 1) + 8 * (lane >> 4);
          const uint32_t o = ((ow >> shift) & 15u) + r, x = ((rw >> shift) & 15u) + r;
          B[j * 1024 + (o >> 4) * 128 + (o & 15u)] = 0;
          B[j * 1024 + (x >> 4) * 128 + (x & 15u)] = 1;
        }
      }
      old = rec;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ms.built[s]);
    }
    // epilogue: lane n of the accumulator holds samples 16 n .. 16 n + 15, or,
    // dense, lane 16 dm + r samples 16 n + r in columns n
    ok = ok && wait_warp(&ms.final_bar, 0, &ms.failed, p.status);
    if (ok) {
      tc_fence_after();
      const int dm_limit = p.dm_skip + (group + 1 == p.ngroups ? p.dm_count_last : p.dm_count);
      const uint32_t lanes = (warp & 3) * 32;
      if (Dense) {
        const int dm = block * kDenseDms + static_cast<int>((lanes + lane) >> 4);
        const bool mine = dm >= p.dm_skip && dm < dm_limit;
        OutT* out = static_cast<OutT*>(p.out) +
                    (static_cast<uint64_t>(mine ? dm - p.dm_skip : 0) * p.out_dm_rows +
                     static_cast<uint64_t>(group) * p.out_group_rows) * p.out_row_stride;
        for (int slot = w >> 2; slot < kMmaSlots; slot += 2) {
          uint32_t v[16];
          __syncwarp();
          tmem_load16(tmem + 16u * slot + (lanes << 16), v);
          const uint64_t t = t0 + 256ull * slot + (lane & 15);
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (mine && t + 16 * j < p.nout) out[t + 16 * j] = static_cast<OutT>(v[j]);
        }
      }
      for (int slot = w >> 2; !Dense && slot < kMmaSlots; slot += 2) {
        const int tl = slot / D, d = slot % D;
        const uint64_t t = t0 + static_cast<uint64_t>(tl) * kMmaTile + 16ull * (lanes + lane);
        const int dm = block * D + d;
        if (dm < p.dm_skip || dm >= dm_limit) continue;
        uint32_t v[16];
        __syncwarp();
        tmem_load16(tmem + 16u * slot + (lanes << 16), v);
        if (t < p.nout) {
          OutT* out = static_cast<OutT*>(p.out) +
                      (static_cast<uint64_t>(dm - p.dm_skip) * p.out_dm_rows +
                       static_cast<uint64_t>(group) * p.out_group_rows) * p.out_row_stride;
          mma_store16<OutT>(out + t, v, p.nout - t);
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 1) {
    // a CTA that gave up waits (bounded) for its steps before it frees TMEM
    if (ms.failed) {
      const long long start = clock64();
      while (!mbar_try_wait(&ms.final_bar, 0) && clock64() - start < kDrainCycles) {
      }
      __syncwarp();
    }
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kMmaColumns));
  }
}

template <typename OutT, bool Dense>
__global__ void __launch_bounds__(kMmaThreads, 2) dedisperse_mma_kernel(const __grid_constant__ MmaParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ MmaShared ms;
  mma_cta<OutT, Dense>(p, blockIdx.x, static_cast<int>(blockIdx.z), smem, ms);
}

// Many launches as one grid (see dedisperse_bytes_batch_kernel).
template <bool Dense>
__global__ void __launch_bounds__(kMmaThreads, 2) dedisperse_mma_batch_kernel(const MmaParams* __restrict__ items,
                                                                              const uint64_t* __restrict__ block_begin,
                                                                              int nitems) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ MmaParams sp;
  __shared__ uint32_t s_local;
  __shared__ MmaShared ms;
  if (threadIdx.x == 0) {
    const uint64_t b = blockIdx.x;
    int lo = 0, hi = nitems;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (block_begin[mid] <= b) lo = mid; else hi = mid;
    }
    sp = items[lo];
    s_local = static_cast<uint32_t>(b - block_begin[lo]);
  }
  __syncthreads();
  const uint32_t local = s_local;
  mma_cta<uint32_t, Dense>(sp, local % sp.grid_x, static_cast<int>(local / sp.grid_x), smem, ms);
}

// -- host side -----------------------------------------------------------------

struct MmaShape {
  int dms = 0, tiles = 0;   // dms = 0: not used
  int steps = 0;            // dense form
  uint32_t row_bytes = 0, stage_bytes = 0;
  int stages = 0;
  size_t smem = 0;
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
    const uint64_t step = std::max<uint64_t>(1, pairs / 2048) | 1;
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
    const uint64_t step = std::max<uint64_t>(1, pairs / 2048) | 1;
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
    const int D = o.D ? o.D : kDenseDms;
    const int blocks = static_cast<int>(ceil_div(ndm_group, D));
    for (int g = 0; g < ngroups; ++g)
      for (int b = 0; b < blocks; ++b)
        for (int row = 0; row < std::min(rows_per_group, total_rows - g * rows_per_group); ++row) {
          const int n = std::min(D, ndm_group - b * D);
          mma_offsets(delays, g, ndm_group, rows_per_group, row, b * D, n, offs);
          max_off = std::max(max_off, *std::max_element(offs, offs + n));
        }
    const MmaShape m = o.D ? mma_shape(o.D, max_off) : dense_shape(max_off);
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

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
#include "dedisperse_mma.cuh"
#include "mbarrier.cuh"

namespace gf {
// A named namespace: the kernels' names do not depend on the file's text.
namespace mma {

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

void set_smem_limit(const void* kernel) {
  cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMmaBudget)),
             "cudaFuncSetAttribute(dedisperse_mma)");
}

}  // namespace mma

void launch_mma(const MmaParams& p, int groups, size_t smem, bool bytes_out, cudaStream_t stream) {
  using namespace mma;
  const bool dense = p.steps != 0;
  auto kernel = bytes_out ? (dense ? dedisperse_mma_kernel<uint8_t, true> : dedisperse_mma_kernel<uint8_t, false>)
                          : (dense ? dedisperse_mma_kernel<uint32_t, true> : dedisperse_mma_kernel<uint32_t, false>);
  set_smem_limit(reinterpret_cast<const void*>(kernel));
  kernel<<<dim3(p.grid_x, 1u, static_cast<unsigned>(groups)), kMmaThreads, smem, stream>>>(p);
  cuda_check(cudaGetLastError(), "dedisperse_mma_kernel launch");
}

void launch_mma_batch(const MmaParams* items, const uint64_t* block_begin, int nitems, uint64_t blocks, size_t smem,
                      bool dense, cudaStream_t stream) {
  using namespace mma;
  auto kernel = dense ? dedisperse_mma_batch_kernel<true> : dedisperse_mma_batch_kernel<false>;
  set_smem_limit(reinterpret_cast<const void*>(kernel));
  kernel<<<static_cast<unsigned>(blocks), kMmaThreads, smem, stream>>>(items, block_begin, nitems);
  cuda_check(cudaGetLastError(), "dedisperse_mma_batch_kernel launch");
}

}  // namespace gf

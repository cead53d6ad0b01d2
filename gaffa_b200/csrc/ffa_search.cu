// FFA search kernels; the algorithm and its execution are described in ffa.cu.
// Compiled once per part (GF_FFA_PART = 0 .. 7, search_kernel_part).
#include "ffa_search.cuh"

namespace gf {
// A named namespace: the kernels' names do not depend on the file's text.
namespace ffa {

// Search-path device functions take the CTA size T (512 or 1024 threads).  The
// ones that merge or detect are inlined: as calls, their register saves and
// the caller's cost 2 % on the survey plan and 17 % on 48-64 bins.

// Dynamic shared memory of the search kernel: two ColBlock headers, the
// staged schedule, then two row buffers.
extern __shared__ __align__(16) float g_smem[];

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// A row read `roll` phases on, in g_smem indexes: lane j's sample of bins
// j + 32 i is at(i), its neighbours after it (kHalo wrapped samples follow a
// row).  The wrap past the row's end is one select per 32 bins.
struct RolledRow {
  uint32_t p, wrapped;
  int32_t w;
  __device__ __forceinline__ RolledRow(uint32_t row, uint32_t roll, uint32_t bins, uint32_t lane) {
    if (roll >= bins) roll %= bins;
    p = row + lane + roll;
    wrapped = p - bins;
    w = static_cast<int32_t>(lane + roll) - static_cast<int32_t>(bins);
  }
  __device__ __forceinline__ const float* at(int i) const {
    // opaque, or the selects of a whole row are formed ahead and spill
    int32_t v = w;
    asm volatile("" : "+r"(v));
    return g_smem + ((v + 32 * i >= 0 ? wrapped : p) + 32u * static_cast<uint32_t>(i));
  }
};

// Output rows of a group: row j is written when lo <= row + j < hi, at row
// row + j - lo of the output buffer; the first lanes write the wrapped samples.
template <bool Clip>
struct OutRows {
  uint32_t first;         // g_smem index of the lane's first sample of row `row`
  uint32_t pitch, bins, lane;
  int32_t lo, hi;         // rows of the group to write (Clip)
  __device__ __forceinline__ void put(int j, int i, float v) const {
    if (Clip && (j < lo || j >= hi)) return;
    float* o = g_smem + (first + static_cast<uint32_t>(j) * pitch + 32u * static_cast<uint32_t>(i));
    *o = v;
    if (i == 0 && lane < kHalo) {
      o[bins] = v;
      if (bins == 2 && lane == 0) o[4] = v;
    }
  }
};

template <int NB, bool Shared, bool Clip>
__device__ __forceinline__ void quad_r(const QuadOp& m, uint32_t prev, uint32_t pitch, const OutRows<Clip>& out,
                                       bool last_ok) {
  const uint32_t lane = out.lane, bins = out.bins;
  const float* a0 = g_smem + prev + m.a[0] * pitch + lane;
  const float* a1 = g_smem + prev + m.a[1] * pitch + lane;
  const RolledRow b0(prev + m.b[0] * pitch, m.rb[0], bins, lane), c0(prev + m.c[0] * pitch, m.rc[0], bins, lane),
      d0(prev + m.d[0] * pitch, m.rd[0], bins, lane);
  if (Shared) {
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (i < NB - 1 || last_ok) {
        const float a = a0[32 * i];
        const float *b = b0.at(i), *c = c0.at(i), *d = d0.at(i);
        const float h0 = __fadd_rn(a, b[0]), h1 = __fadd_rn(a, b[1]);
        const float c1 = c[1];
        out.put(0, i, __fadd_rn(h0, __fadd_rn(c[0], d[0])));
        out.put(1, i, __fadd_rn(h0, __fadd_rn(c1, d[1])));
        out.put(2, i, __fadd_rn(h1, __fadd_rn(c1, d[2])));
        out.put(3, i, __fadd_rn(h1, __fadd_rn(c[2], d[3])));
      }
  } else {
    const RolledRow b1(prev + m.b[1] * pitch, m.rb[1], bins, lane), c1(prev + m.c[1] * pitch, m.rc[1], bins, lane),
        d1(prev + m.d[1] * pitch, m.rd[1], bins, lane);
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (i < NB - 1 || last_ok) {
        const float h0 = __fadd_rn(a0[32 * i], *b0.at(i)), h1 = __fadd_rn(a1[32 * i], *b1.at(i));
        const float *c = c0.at(i), *d = d0.at(i), *e = c1.at(i), *f = d1.at(i);
        out.put(0, i, __fadd_rn(h0, __fadd_rn(c[0], d[0])));
        out.put(1, i, __fadd_rn(h0, __fadd_rn(c[1], d[1])));
        out.put(2, i, __fadd_rn(h1, __fadd_rn(e[0], f[0])));
        out.put(3, i, __fadd_rn(h1, __fadd_rn(e[1], f[1])));
      }
  }
}

template <int NB, bool Shared, bool Clip>
__device__ __forceinline__ void quad_f(const QuadOp& m, uint32_t prev, uint32_t pitch, const OutRows<Clip>& out,
                                       bool last_ok) {
  const uint32_t lane = out.lane, bins = out.bins;
  const float* a0 = g_smem + prev + m.a[0] * pitch + lane;
  const float* a1 = g_smem + prev + m.a[1] * pitch + lane;
  const RolledRow b0(prev + m.b[0] * pitch, m.rb[0], bins, lane), b1(prev + m.b[1] * pitch, m.rb[1], bins, lane);
  const RolledRow c0(prev + m.c[0] * pitch, m.rc[0], bins, lane), d0(prev + m.d[0] * pitch, m.rd[0], bins, lane);
  const RolledRow c1(prev + m.c[1] * pitch, m.rc[1], bins, lane), d1(prev + m.d[1] * pitch, m.rd[1], bins, lane);
  const RolledRow c2(prev + m.c[2] * pitch, m.rc[2], bins, lane), d2(prev + m.d[2] * pitch, m.rd[2], bins, lane);
#pragma unroll
  for (int i = 0; i < NB; ++i)
    if (i < NB - 1 || last_ok) {
      float h0, h1;
      if (Shared) {
        const float a = a0[32 * i];
        const float* b = b0.at(i);
        h0 = __fadd_rn(a, b[0]);
        h1 = __fadd_rn(a, b[1]);
      } else {
        h0 = __fadd_rn(a0[32 * i], *b0.at(i));
        h1 = __fadd_rn(a1[32 * i], *b1.at(i));
      }
      const float *c = c1.at(i), *d = d1.at(i);
      out.put(0, i, __fadd_rn(h0, __fadd_rn(*c0.at(i), *d0.at(i))));
      out.put(1, i, __fadd_rn(h0, __fadd_rn(c[0], d[0])));
      out.put(2, i, __fadd_rn(h1, __fadd_rn(c[1], d[1])));
      out.put(3, i, __fadd_rn(h1, __fadd_rn(*c2.at(i), *d2.at(i))));
    }
}

// Two rows of one head and one tail row (Pair), or one row, any of whose four
// inputs may be missing (rows carried up unchanged).
template <int NB, bool Pair, bool Clip>
__device__ __forceinline__ void quad_rest(const QuadOp& m, uint32_t prev, uint32_t pitch, const OutRows<Clip>& out,
                                          bool last_ok) {
  const uint32_t lane = out.lane, bins = out.bins;
  const float* a0 = g_smem + prev + m.a[0] * pitch + lane;
  const RolledRow b0(prev + m.b[0] * pitch, m.rb[0], bins, lane), c0(prev + m.c[0] * pitch, m.rc[0], bins, lane),
      d0(prev + m.d[0] * pitch, m.rd[0], bins, lane);
  const bool has_b = Pair || (m.flags & 1), has_c = Pair || (m.flags & 2), has_d = Pair || (m.flags & 4);
#pragma unroll
  for (int i = 0; i < NB; ++i)
    if (i < NB - 1 || last_ok) {
      float h = a0[32 * i];
      if (has_b) h = __fadd_rn(h, *b0.at(i));
      if (Pair) {
        const float *c = c0.at(i), *d = d0.at(i);
        out.put(0, i, __fadd_rn(h, __fadd_rn(c[0], d[0])));
        out.put(1, i, __fadd_rn(h, __fadd_rn(c[1], d[1])));
      } else {
        if (has_c) {
          float w = *c0.at(i);
          if (has_d) w = __fadd_rn(w, *d0.at(i));
          h = __fadd_rn(h, w);
        }
        out.put(0, i, h);
      }
    }
}

__device__ __forceinline__ uint32_t op_rows(uint16_t type) { return type == kOpPair ? 2u : type == kOpOne ? 1u : 4u; }

// Two levels: a warp per group, lane j handles bins j, j + 32, ...  Clip: rows
// [lo, hi) only, written from row 0 of the output buffer.
template <int NB, int T, bool Clip>
__device__ __forceinline__ void merge_two(const QuadOp* ops, uint32_t nops, uint32_t prev, uint32_t out_buf,
                                          uint32_t pitch, uint32_t bins, uint32_t lo, uint32_t hi) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool last_ok = lane + 32u * (NB - 1) < bins;
  for (uint32_t q = warp; q < nops; q += T / 32) {
    const QuadOp& m = ops[q];
    const uint16_t type = m.type;
    const uint32_t row = m.row;
    OutRows<Clip> out;
    out.first = out_buf + (Clip ? row - lo : row) * pitch + lane;
    out.pitch = pitch;
    out.bins = bins;
    out.lane = lane;
    if (Clip) {
      out.lo = static_cast<int32_t>(lo) - static_cast<int32_t>(row);
      out.hi = static_cast<int32_t>(hi) - static_cast<int32_t>(row);
      if (out.hi <= 0 || out.lo >= static_cast<int32_t>(op_rows(type))) continue;
    }
    switch (type) {
      case kOpR: quad_r<NB, false, Clip>(m, prev, pitch, out, last_ok); break;
      case kOpRS: quad_r<NB, true, Clip>(m, prev, pitch, out, last_ok); break;
      case kOpF: quad_f<NB, false, Clip>(m, prev, pitch, out, last_ok); break;
      case kOpFS: quad_f<NB, true, Clip>(m, prev, pitch, out, last_ok); break;
      case kOpPair: quad_rest<NB, true, Clip>(m, prev, pitch, out, last_ok); break;
      default: quad_rest<NB, false, Clip>(m, prev, pitch, out, last_ok); break;
    }
  }
}

// One level: rows [lo, hi) of meta into rows 0, 1, ... of the output buffer.
template <int NB, int T>
__device__ __forceinline__ void merge_one(const MetaEntry* meta, uint32_t prev, uint32_t out_buf, uint32_t pitch,
                                          uint32_t bins, uint32_t lo, uint32_t hi) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool last_ok = lane + 32u * (NB - 1) < bins;
  for (uint32_t q = lo + warp; q < hi; q += T / 32) {
    const MetaEntry m = meta[q];
    OutRows<false> out;
    out.first = out_buf + (q - lo) * pitch + lane;
    out.pitch = pitch;
    out.bins = bins;
    out.lane = lane;
    const float* h = g_smem + prev + m.a * pitch + lane;
    if (m.op == kMerge) {
      const RolledRow t(prev + m.b * pitch, m.roll, bins, lane);
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i < NB - 1 || last_ok) out.put(0, i, __fadd_rn(h[32 * i], *t.at(i)));
    } else {
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i < NB - 1 || last_ok) out.put(0, i, h[32 * i]);
    }
  }
}

// A whole pass (the root pass of an on-chip task goes by merge_rows instead).
template <int NB, int T>
__device__ __forceinline__ void run_pass(uint16_t pass, const char* meta, uint32_t prev, uint32_t out_buf,
                                         uint32_t pitch, uint32_t bins) {
  const uint32_t n = pass & 0x7fffu;
  if (pass & kPassTwo)
    merge_two<NB, T, false>(reinterpret_cast<const QuadOp*>(meta), n, prev, out_buf, pitch, bins, 0u, 0u);
  else
    merge_one<NB, T>(reinterpret_cast<const MetaEntry*>(meta), prev, out_buf, pitch, bins, 0u, n);
}

// Rows [lo, hi) of a pass.
template <int NB, int T>
__device__ __forceinline__ void merge_rows(uint16_t pass, const char* meta, uint32_t prev, uint32_t out_buf,
                                           uint32_t pitch, uint32_t bins, uint32_t lo, uint32_t hi) {
  if (pass & kPassTwo)
    merge_two<NB, T, true>(reinterpret_cast<const QuadOp*>(meta), pass & 0x7fffu, prev, out_buf, pitch, bins, lo, hi);
  else
    merge_one<NB, T>(reinterpret_cast<const MetaEntry*>(meta), prev, out_buf, pitch, bins, lo, hi);
}

template <int NB, int I = 0>
__device__ __forceinline__ void copy_bins_async(uint32_t to, const float* from, bool last_ok) {
  if constexpr (I < NB) {
    if (I < NB - 1 || last_ok)
      asm volatile("cp.async.ca.shared.global [%0+%2], [%1+%2], 4;\n" ::"r"(to), "l"(from), "n"(128 * I) : "memory");
    copy_bins_async<NB, I + 1>(to, from, last_ok);
  }
}

// One row of length `bins` from global memory, wrapped samples included, async.
template <int NB>
__device__ __forceinline__ void load_row_async(const float* src, uint32_t bins, float* row, uint32_t lane,
                                               bool last_ok) {
  const float* g = src + lane;
  const uint32_t o = static_cast<uint32_t>(__cvta_generic_to_shared(row + lane));
  copy_bins_async<NB>(o, g, last_ok);
  if (lane < kHalo)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(o + 4 * bins), "l"(lane < bins ? g : g - bins));
}

// rows [0, n) of read-only global `src` (row length bins) into smem, async
template <int NB, int T>
__device__ __forceinline__ void load_rows_async(const float* src, uint32_t n, uint32_t bins, uint32_t out,
                                                uint32_t pitch) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool last_ok = lane + 32u * (NB - 1) < bins;
  for (uint32_t q = warp; q < n; q += T / 32)
    load_row_async<NB>(src + static_cast<uint64_t>(q) * bins, bins, g_smem + out + q * pitch, lane, last_ok);
}

template <int NB, int T>
__device__ __forceinline__ void store_rows(uint32_t in, uint32_t pitch, uint32_t n, uint32_t bins, float* dst) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool last_ok = lane + 32u * (NB - 1) < bins;
  for (uint32_t q = warp; q < n; q += T / 32) {
    float* g = dst + static_cast<uint64_t>(q) * bins + lane;
    const float* s = g_smem + in + q * pitch + lane;
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (i < NB - 1 || last_ok) __stcg(g + 32 * i, s[32 * i]);
  }
}

// ---------------------------------------------------------------------------
// detection
// ---------------------------------------------------------------------------

struct DetectArgs {
  const TrialDev* trials;    // shared memory
  uint32_t ntrials, max_width, bins;
  float inv_stdnoise, threshold;
  uint32_t series, task;
  gf_peak_record* peaks;
  uint64_t capacity;
  unsigned long long* counters;
};

// order-preserving map of finite floats to unsigned keys (for redux.sync)
__device__ __forceinline__ uint32_t float_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// {x0 - y0, x1 - y1}, each rounded to nearest
__device__ __forceinline__ float2 sub2(float x0, float x1, float y0, float y1) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, d;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "sub.rn.f32x2 d, x, y;\n\tmov.b64 {%0, %1}, d;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(x0), "f"(x1), "f"(y0), "f"(y1));
  return d;
}

// rows[i] (pitch `pitch`) hold root rows shift0 + i, i < count.  Prefix sums
// are sequential per row (one thread per row, ffa_detection.cpp:126-139).
// Then a warp per row: lane j holds c[j + 32i] and, for every width, takes
// the maximum of c[ph + w] - c[ph] over its phases; redux.sync gives the
// row maximum, from which S/N follows (:141-170).  Only when S/N passes the
// threshold is the first phase attaining the maximum looked up (the
// reference's strict '>' scan keeps the first maximum), and a peak appended.
template <int NB, int T>
__device__ __forceinline__ void detect_rows(const float* rows, uint32_t pitch, uint32_t count, uint32_t shift0, float* cp,
                            uint32_t cp_pitch, const DetectArgs& a) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bins = a.bins;
  for (uint32_t row = threadIdx.x; row < count; row += T) {
    const float* prof = rows + row * pitch;
    float* c = cp + row * cp_pitch;
    float acc = 0.0f;
    c[0] = 0.0f;
    // loads of the next 8 samples overlap the current 8-add chain
    float cur[8], nxt[8];
    const uint32_t nfull = bins & ~7u;
#pragma unroll
    for (int j = 0; j < 8; ++j) cur[j] = (static_cast<uint32_t>(j) < nfull) ? prof[j] : 0.0f;
    for (uint32_t i = 0; i < nfull; i += 8) {
#pragma unroll
      for (int j = 0; j < 8; ++j) nxt[j] = (i + 8 + j < nfull) ? prof[i + 8 + j] : 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc = __fadd_rn(acc, cur[j]);
        c[i + j + 1] = acc;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) cur[j] = nxt[j];
    }
    for (uint32_t i = nfull; i < bins; ++i) {
      acc = __fadd_rn(acc, prof[i]);
      c[i + 1] = acc;
    }
    for (uint32_t i = 0; i < a.max_width; ++i) {
      acc = __fadd_rn(acc, prof[i]);
      c[bins + i + 1] = acc;
    }
  }
  __syncthreads();
  const bool last_ok = lane + 32u * (NB - 1) < bins;
  for (uint32_t r = warp; r < count; r += T / 32) {
    const float* c = cp + r * cp_pitch + lane;
    float base[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) base[i] = (i < NB - 1 || last_ok) ? c[32 * i] : 0.0f;
    const float psum = cp[r * cp_pitch + bins];
    for (uint32_t k = 0; k < a.ntrials; ++k) {
      const TrialDev tr = a.trials[k];
      const float* cw = c + tr.width;
      // two phases per packed subtraction and per three-input maximum
      float best = -INFINITY;
#pragma unroll
      for (int i = 0; i + 1 < NB - 1; i += 2) {
        const float2 d = sub2(cw[32 * i], cw[32 * i + 32], base[i], base[i + 1]);
        best = max3(best, d.x, d.y);
      }
      if (NB % 2 == 0) best = fmaxf(best, __fsub_rn(cw[32 * (NB - 2)], base[NB - 2 < 0 ? 0 : NB - 2]));
      if (last_ok) best = fmaxf(best, __fsub_rn(cw[32 * (NB - 1)], base[NB - 1]));
      // S/N is monotone in the boxcar sum, so the row passes the threshold
      // exactly when some lane's own maximum does
      const float lane_snr = __fmul_rn(
          __fsub_rn(__fmul_rn(__fadd_rn(tr.height, tr.baseline), best), __fmul_rn(tr.baseline, psum)),
          a.inv_stdnoise);
      if (__any_sync(0xffffffffu, lane_snr >= a.threshold)) {
        const float maxv = key_float(__reduce_max_sync(0xffffffffu, float_key(best)));
        const float snr = __fmul_rn(
            __fsub_rn(__fmul_rn(__fadd_rn(tr.height, tr.baseline), maxv), __fmul_rn(tr.baseline, psum)),
            a.inv_stdnoise);
        uint32_t first = 0xffffffffu;
#pragma unroll
        for (int i = NB - 1; i >= 0; --i)
          if ((i < NB - 1 || last_ok) && __fsub_rn(cw[32 * i], base[i]) == maxv) first = lane + 32u * i;
        const uint32_t ph = __reduce_min_sync(0xffffffffu, first);
        if (lane == 0) {
          const unsigned long long slot = atomicAdd(a.counters, 1ull);
          if (slot < a.capacity) {
            gf_peak_record rec;
            rec.series = a.series;
            rec.task = a.task;
            rec.shift = shift0 + r;
            rec.phase = static_cast<uint16_t>(ph);
            rec.width_index = static_cast<uint16_t>(k);
            rec.snr = snr;
            rec.reserved = 0u;
            a.peaks[slot] = rec;
          } else {
            atomicOr(reinterpret_cast<unsigned int*>(a.counters + 1), GF_STATUS_PEAK_OVERFLOW);
          }
        }
      }
    }
  }
  __syncthreads();
}

__device__ __forceinline__ DetectArgs make_detect(const SearchParams& p, const TaskDev& t, const TrialDev* trials,
                                                  uint32_t series, uint32_t task) {
  DetectArgs da;
  da.trials = trials;
  da.ntrials = t.ntrials;
  da.max_width = t.max_width;
  da.bins = t.bins;
  da.inv_stdnoise = t.inv_stdnoise;
  da.threshold = p.threshold;
  da.series = series;
  da.task = task;
  da.peaks = p.peaks;
  da.capacity = p.capacity;
  da.counters = p.counters;
  return da;
}

// Brings [p, p + n) floats towards L2 (whole 16-byte words inside the range):
// 43.1 -> 42.6 ms on the survey plan.
__device__ __forceinline__ void prefetch_l2(const float* p, uint64_t n) {
  const uint64_t begin = (reinterpret_cast<uint64_t>(p) + 15) & ~15ull;
  const uint64_t end = reinterpret_cast<uint64_t>(p + n) & ~15ull;
  if (begin < end)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(begin), "r"(static_cast<uint32_t>(end - begin)));
}

// Stages `size16` 16-byte words of a schedule, async.
template <int T>
__device__ __forceinline__ void stage_schedule(char* dst, const uint4* src, uint32_t size16) {
  for (uint32_t e = threadIdx.x; e < size16; e += T) cp_async16(dst + 16 * e, src + e);
}

// Evaluates a subtree of n <= max_rows rows (pointer `src` = its first input
// row) up to its last pass, or up to the pass before it when `root` (then
// *meta is that pass's entries).  Returns the buffer that holds the result.
template <int NB, int T>
__device__ __forceinline__ uint32_t eval_subtree(const SearchParams& p, const float* src, uint32_t n, uint32_t bins, bool root,
                                 uint32_t buf0, uint32_t buf1, char* smeta, const char** meta) {
  const uint2 where = __ldg(reinterpret_cast<const uint2*>(p.sub_head + n));  // offset16, size16
  load_rows_async<NB, T>(src, n, bins, buf0, p.pitch);  // ahead of what waits for `where`
  stage_schedule<T>(smeta, p.sub_meta + where.x, where.y & 0xffffu);
  cp_async_wait_all();
  __syncthreads();
  const SubHead& head = *reinterpret_cast<const SubHead*>(smeta);
  const char* m = smeta + sizeof(SubHead);
  const int last = static_cast<int>(head.npasses) - (root ? 1 : 0);
  for (int k = 0; k < last; ++k) {
    run_pass<NB, T>(head.pass[k], m, buf0, buf1, p.pitch, bins);
    m += pass_bytes(head.pass[k]);
    const uint32_t t = buf0;
    buf0 = buf1;
    buf1 = t;
    __syncthreads();
  }
  *meta = m;
  return buf0;
}

// Column block `hb`: stages its schedule, loads its bottom rows from `src`
// (scratch that this CTA wrote before its last barrier), evaluates its passes.
// The output rows end in buf0.
template <int NB, int T>
__device__ __forceinline__ void eval_block(const SearchParams& p, const ColBlock& hb, const ColBlock* next, const float* src,
                           uint32_t bins, uint32_t buf0, uint32_t buf1, char* smeta) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t pitch = p.pitch;
  stage_schedule<T>(smeta, p.col_meta + hb.meta16, hb.size16);
  const uint32_t np = hb.npasses;
  uint32_t from = (np & 1) ? buf1 : buf0, to = (np & 1) ? buf0 : buf1;
  const uint32_t nb = hb.nbottom;
  const uint32_t nruns = hb.nruns;
  const bool last_ok = lane + 32u * (NB - 1) < bins;
  // Bottom rows: async copies, all in flight at once.
  for (uint32_t q = warp; q < nb; q += T / 32) {
    uint32_t j = 0;  // run holding buffer row q (runs ascend in run_off)
#pragma unroll
    for (uint32_t r = 1; r < 8; ++r) j += (r < nruns && hb.run_off[r] <= q) ? 1u : 0u;
    load_row_async<NB>(src + static_cast<uint64_t>(hb.run_row[j] + (q - hb.run_off[j])) * bins, bins,
                       g_smem + from + q * pitch, lane, last_ok);
  }
  cp_async_wait_all();
  __syncthreads();
  // the next block's rows, from DRAM while this block is evaluated
  if (next && threadIdx.x < next->nruns) {
    const uint32_t j = threadIdx.x;
    const uint32_t n = (j + 1 < next->nruns ? next->run_off[j + 1] : next->nbottom) - next->run_off[j];
    prefetch_l2(src + static_cast<uint64_t>(next->run_row[j]) * bins, static_cast<uint64_t>(n) * bins);
  }
  const char* m = smeta;
  for (uint32_t k = 0; k < np; ++k) {
    run_pass<NB, T>(hb.pass[k], m, from, to, pitch, bins);
    m += pass_bytes(hb.pass[k]);
    const uint32_t t = from;
    from = to;
    to = t;
    __syncthreads();
  }
}

// 64-byte header, async (completes at the next cp_async_wait_all)
__device__ __forceinline__ void load_header(ColBlock* dst, const ColBlock* src) {
  if (threadIdx.x < 4)
    cp_async16(reinterpret_cast<uint4*>(dst) + threadIdx.x, reinterpret_cast<const uint4*>(src) + threadIdx.x);
}

// One (series, task) per CTA; items are task-major so the series of one task
// run together.  NB = ceil(bins/32) of every task of the launch.
template <int NB, int T>
__global__ void __launch_bounds__(T, T == kSmallThreads ? 2 : 1) ffa_search_kernel(SearchParams p) {
  __shared__ __align__(16) TrialDev trials[kMaxWidths];
  const uint32_t pitch = p.pitch;
  ColBlock* hdr = reinterpret_cast<ColBlock*>(g_smem);
  char* smeta = reinterpret_cast<char*>(g_smem + 32);
  const uint32_t buf0 = p.front;
  const uint32_t buf1 = buf0 + p.max_rows * pitch;
  float* q0 = p.scratch ? p.scratch + blockIdx.x * (p.scratch_elems0 + p.scratch_elems1) : nullptr;
  float* q1 = q0 ? q0 + p.scratch_elems0 : nullptr;
  const uint64_t nitems = p.units ? p.nitems : static_cast<uint64_t>(p.nseries) * p.nitem_tasks;
  for (uint64_t item = blockIdx.x; item < nitems; item += gridDim.x) {
    uint32_t task, series;
    const float* base;
    uint64_t stride;
    if (p.units) {
      // last run starting at or before the item (runs in item order)
      uint32_t lo = 0, hi = p.nunits;
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (p.units[mid].item_begin <= item) lo = mid; else hi = mid;
      }
      const UnitDev u = p.units[lo];
      task = u.task;
      series = static_cast<uint32_t>(item - u.item_begin);
      base = p.members[u.member].prepared;
      stride = p.members[u.member].prep_stride;
    } else {
      task = p.item_tasks[item / p.nseries];
      series = static_cast<uint32_t>(item % p.nseries);
      base = p.prepared;
      stride = p.prep_stride;
    }
    const TaskDev t = p.tasks[task];
    const float* input = base + series * stride + t.prep_offset;
    const uint32_t bins = t.bins;
    // the item's width trials; every path to detection passes a barrier, and so
    // does the end of the last item's detection
    for (uint32_t k = threadIdx.x; k < t.ntrials; k += T) cp_async16(trials + k, p.trials + t.trial_offset + k);
    const DetectArgs da = make_detect(p, t, trials, series, task);
    const uint32_t cp_pitch = (bins + t.max_width + 2) | 1u;
    const uint32_t dS = t.split_depth;
    if (dS == 0) {
      // whole task on chip: levels below the root, then root rows in batches
      if (t.rows == 1) {
        load_rows_async<NB, T>(input, 1, bins, buf0, pitch);
        cp_async_wait_all();
        __syncthreads();
        detect_rows<NB, T>(g_smem + buf0, pitch, 1, 0, g_smem + buf1, cp_pitch, da);
        __syncthreads();  // the width scans read buf1 until here; the next item loads into it
        continue;
      }
      const char* root;
      const uint32_t below = eval_subtree<NB, T>(p, input, t.rows, bins, true, buf0, buf1, smeta, &root);
      const uint32_t other = below == buf0 ? buf1 : buf0;
      const SubHead& head = *reinterpret_cast<const SubHead*>(smeta);
      const uint16_t root_pass = head.pass[head.npasses - 1];
      const uint32_t batch = umin32(T, (p.max_rows * pitch) / (pitch + cp_pitch));
      for (uint32_t b0 = 0; b0 < t.rows_eval; b0 += batch) {
        const uint32_t cnt = umin32(batch, t.rows_eval - b0);
        merge_rows<NB, T>(root_pass, root, below, other, pitch, bins, b0, b0 + cnt);
        __syncthreads();
        detect_rows<NB, T>(g_smem + other, pitch, cnt, b0, g_smem + other + batch * pitch, cp_pitch, da);
      }
      __syncthreads();  // the last width scans read `other` until here; the next item loads into it
      continue;
    }
    // Subtrees at depth dS on chip, then column passes up to the root (the last
    // one fused with detection).  The first pass follows the subtrees node by
    // node: a node of depth first_depth is at most 8 subtrees, whose rows (well
    // under 1 MB) it reads back from L2 right after they are written there,
    // into scratch that the next node uses again (all subtrees first: 47.4 ms
    // on the survey plan, 45.9 node by node).
    uint32_t block = 0;  // next block of the pass
    for (uint32_t ps = 0; ps < t.npasses; ++ps) {
      const PassDev pd = p.passes[t.pass_begin + ps];
      const ColBlock* blocks = p.blocks + pd.block_begin;
      const uint32_t nnodes = ps == 0 ? 1u << t.first_depth : 1u;
      const float* src = (ps & 1) ? q1 : q0;
      float* dst = (ps & 1) ? q0 : q1;
      block = 0;
      for (uint32_t node = 0; node < nnodes; ++node) {
        uint32_t end = pd.nblocks;
        if (ps == 0) {
          const Node X = node_at(node, t.rows, t.first_depth);
          const uint32_t per = 1u << (dS - t.first_depth);
          for (uint32_t sub = node * per; sub < (node + 1) * per; ++sub) {
            const Node nd = node_at(sub, t.rows, dS);
            if (threadIdx.x == 0 && nd.a + nd.n < t.rows)
              prefetch_l2(input + static_cast<uint64_t>(nd.a + nd.n) * bins,
                          umin64(nd.n, t.rows - nd.a - nd.n) * bins);
            const char* meta_end;
            const uint32_t res = eval_subtree<NB, T>(p, input + static_cast<uint64_t>(nd.a) * bins, nd.n, bins, false,
                                                     buf0, buf1, smeta, &meta_end);
            store_rows<NB, T>(res, pitch, nd.n, bins, q0 + static_cast<uint64_t>(nd.a - X.a) * bins);
            __syncthreads();
          }
          src = q0 - static_cast<uint64_t>(X.a) * bins;
          if (t.first_depth > 0) end = block + (X.n + p.block_rows - 1) / p.block_rows;
        }
        if (block < end) load_header(&hdr[block & 1], blocks + block);
        cp_async_wait_all();
        __syncthreads();
        for (; block < end; ++block) {
          const ColBlock& hb = hdr[block & 1];
          const ColBlock* next = nullptr;
          if (block + 1 < end) {
            load_header(&hdr[(block + 1) & 1], blocks + block + 1);
            next = &hdr[(block + 1) & 1];
          }
          eval_block<NB, T>(p, hb, next, src, bins, buf0, buf1, smeta);
          if (hb.final_pass) {
            detect_rows<NB, T>(g_smem + buf0, pitch, hb.rows, hb.out_row, g_smem + buf1, cp_pitch, da);
            __syncthreads();  // the width scans read buf1 until here; the next block may load into it
          } else {
            store_rows<NB, T>(buf0, pitch, hb.rows, bins, dst + static_cast<uint64_t>(hb.out_row) * bins);
            __syncthreads();
          }
        }
      }
    }
  }
}

template <int T>
SearchKernel search_kernel(uint32_t nb) {
  return nb % 2 == 1 ? ffa_search_kernel<2 * GF_FFA_PART + 1, T> : ffa_search_kernel<2 * GF_FFA_PART + 2, T>;
}

}  // namespace ffa

template <>
SearchKernel search_kernel_part<GF_FFA_PART>(uint32_t nb, int threads) {
  return threads == kSmallThreads ? ffa::search_kernel<kSmallThreads>(nb) : ffa::search_kernel<kThreads>(nb);
}

}  // namespace gf

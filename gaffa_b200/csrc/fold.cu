// Folding of a dedispersed time series into phase bins on sm_100a.
//
// Reference: fold_time_series_cpu, src/gaffa/folding.cpp:452-502 with
// accumulate_interval :124-158.  Sample i covers the scaled phase interval
// [(start+i)*step, (start+i+1)*step), step = tsamp / period * nbin; each bin
// it overlaps receives value * overlap and overlap of exposure (FP64);
// profile = sums / exposure.  The reference has no CUDA path for this.
//
// Each thread folds a contiguous run of samples, carrying the current bin's
// partial sums in registers and flushing them to shared-memory FP64
// accumulators when the bin changes; CTA partials are reduced in a fixed
// order by a second kernel.  Like the reference's per-thread OpenMP
// histograms, the FP64 summation order differs from a serial loop, so
// results agree to FP64 rounding (the float profile to within an ulp).
#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>

namespace gf {
namespace {

constexpr int kThreads = 256;
constexpr int kSamplesPerThread = 64;
constexpr uint64_t kMaxBins = 8192;

template <bool U32>
__global__ void __launch_bounds__(kThreads) fold_partial_kernel(const void* __restrict__ in, uint64_t n,
                                                                double step, uint64_t start, uint64_t nbin,
                                                                double* __restrict__ partial,
                                                                uint32_t* status) {
  extern __shared__ double acc[];  // [2][nbin]
  double* sums = acc;
  double* expo = acc + nbin;
  for (uint64_t b = threadIdx.x; b < 2 * nbin; b += kThreads) acc[b] = 0.0;
  __syncthreads();
  const uint64_t i0 = (static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x) * kSamplesPerThread;
  const int64_t nb = static_cast<int64_t>(nbin);
  int64_t cur = -1;
  double cs = 0.0, ce = 0.0;
  for (uint64_t i = i0; i < n && i < i0 + kSamplesPerThread; ++i) {
    const double v = U32 ? static_cast<double>(static_cast<const uint32_t*>(in)[i])
                         : static_cast<double>(static_cast<const float*>(in)[i]);
    if (!U32 && !isfinite(v)) atomicOr(status, GF_STATUS_NONFINITE);
    const double lo = __dmul_rn(static_cast<double>(start + i), step);
    const double hi = __dadd_rn(lo, step);
    const int64_t first = static_cast<int64_t>(floor(lo));
    const int64_t last = static_cast<int64_t>(ceil(hi) - 1.0);
    for (int64_t bin = first; bin <= last; ++bin) {
      const double bl = static_cast<double>(bin), br = bl + 1.0;
      const double w = __dsub_rn(hi < br ? hi : br, lo > bl ? lo : bl);
      if (!(w > 0.0)) continue;
      int64_t m = bin % nb;
      if (m < 0) m += nb;
      if (m != cur) {
        if (cur >= 0) {
          atomicAdd(sums + cur, cs);
          atomicAdd(expo + cur, ce);
        }
        cur = m;
        cs = 0.0;
        ce = 0.0;
      }
      cs = __dadd_rn(cs, __dmul_rn(v, w));
      ce = __dadd_rn(ce, w);
    }
  }
  if (cur >= 0) {
    atomicAdd(sums + cur, cs);
    atomicAdd(expo + cur, ce);
  }
  __syncthreads();
  double* out = partial + static_cast<uint64_t>(blockIdx.x) * 2 * nbin;
  for (uint64_t b = threadIdx.x; b < 2 * nbin; b += kThreads) out[b] = acc[b];
}

__global__ void __launch_bounds__(kThreads) fold_reduce_kernel(const double* __restrict__ partial, int nblocks,
                                                               uint64_t nbin, float* __restrict__ profile,
                                                               double* __restrict__ exposure) {
  const uint64_t b = static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x;
  if (b >= nbin) return;
  double s = 0.0, e = 0.0;
  for (int k = 0; k < nblocks; ++k) {
    s = __dadd_rn(s, partial[static_cast<uint64_t>(k) * 2 * nbin + b]);
    e = __dadd_rn(e, partial[static_cast<uint64_t>(k) * 2 * nbin + nbin + b]);
  }
  exposure[b] = e;
  profile[b] = e > 0.0 ? static_cast<float>(__ddiv_rn(s, e)) : 0.0f;
}

uint64_t fold_blocks(uint64_t n) { return ceil_div(n, static_cast<uint64_t>(kThreads) * kSamplesPerThread); }

void launch_fold_partial(const void* dev_input, bool u32, uint64_t n, double step, uint64_t start_sample,
                         uint64_t nbin, unsigned blocks, double* partial, uint32_t* status, cudaStream_t s) {
  auto kernel = u32 ? fold_partial_kernel<true> : fold_partial_kernel<false>;
  // the same limit on every call, whatever its bins (calls from several threads)
  cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(2 * kMaxBins * sizeof(double))),
             "cudaFuncSetAttribute(fold)");
  kernel<<<blocks, kThreads, 2 * nbin * sizeof(double), s>>>(dev_input, n, step, start_sample, nbin, partial, status);
}

}  // namespace
}  // namespace gf

using namespace gf;

extern "C" uint64_t gf_fold_workspace_bytes(uint64_t n, uint64_t nbin) {
  return fold_blocks(n) * 2 * nbin * sizeof(double) + 16;
}

extern "C" int gf_fold_time_series(const void* dev_input, int32_t input_is_u32, uint64_t n, double period,
                                   double tsamp, uint64_t nbin, uint64_t start_sample, float* dev_profile,
                                   double* dev_exposure, void* dev_workspace, void* stream) {
  return guarded([&] {
    // folding.cpp:44-73 validation
    check_arg(std::isfinite(period) && period > 0.0, "fold period must be finite and positive");
    check_arg(std::isfinite(tsamp) && tsamp > 0.0, "fold tsamp must be finite and positive");
    check_arg(nbin > 0, "fold nbin must be positive");
    check_arg(nbin <= kMaxBins, "CUDA fold supports nbin <= 8192");
    check_arg(n > 0, "fold input must not be empty");
    check_arg(dev_input && dev_profile && dev_exposure && dev_workspace, "null argument");
    const double step = tsamp / period * static_cast<double>(nbin);
    const double hi = static_cast<double>(start_sample + n - 1) * step + step;
    check_arg(std::isfinite(hi) && std::ceil(hi) < 9.2e18, "fold phase bin index exceeds int64 range");
    auto s = as_stream(stream);
    const uint64_t blocks = fold_blocks(n);
    check_arg(blocks < (1ull << 31), "fold input too long");
    double* partial = static_cast<double*>(dev_workspace);
    uint32_t* status = reinterpret_cast<uint32_t*>(static_cast<char*>(dev_workspace) + blocks * 2 * nbin * 8);
    cuda_check(cudaMemsetAsync(status, 0, 4, s), "cudaMemsetAsync(fold status)");
    launch_fold_partial(dev_input, input_is_u32 != 0, n, step, start_sample, nbin, static_cast<unsigned>(blocks), partial,
                        status, s);
    fold_reduce_kernel<<<static_cast<unsigned>(ceil_div(nbin, kThreads)), kThreads, 0, s>>>(
        partial, static_cast<int>(blocks), nbin, dev_profile, dev_exposure);
    cuda_check(cudaGetLastError(), "fold launch");
  });
}

// ---------------------------------------------------------------------------
// Fold without any device allocation.
//
// Some callers cannot allocate device memory when they fold: a process whose
// device memory has all been handed to another allocator's pool, or a
// latency-critical loop where cudaMalloc's implicit device synchronisation is
// not acceptable.  gf_fold_time_series_noalloc serves them with a fixed
// scratch area compiled into this library: a file-scope device array that
// every GPU which loads the library holds until the process exits.  Its size
// caps the work: fold_blocks(n) * 2 * nbin doubles must fit in
// kNoAllocScratchBytes (4 MiB: e.g. nbin = 64 up to ~67 million samples).
// All calls share the array and it keeps the last call's contents; the
// partial sums are fully rewritten by every call, so nothing needs clearing,
// but calls that overlap on the GPU (different streams, or different host
// threads) race on it and must be serialised by the caller.
// ---------------------------------------------------------------------------

namespace {

constexpr uint64_t kNoAllocScratchBytes = 4ull << 20;
static __device__ __align__(256) unsigned char g_fold_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_fold_scratch_mutex;
void* g_fold_scratch_address[kMaxDevices] = {};

// Device address of g_fold_scratch on the current device, resolved once per
// device.  In host code the array's name is only a host-side stand-in, so
// the kernels must receive this address, never &g_fold_scratch.  The address
// is kept for the life of the process; a cudaDeviceReset reloads the module
// and makes it stale, so the entry point is not to be used after a reset.
void* fold_scratch_address() {
  int device = -1;
  cuda_check(cudaGetDevice(&device), "cudaGetDevice");
  check_arg(device >= 0 && device < kMaxDevices, "device ordinal out of range for the fixed fold scratch");
  std::lock_guard<std::mutex> lock(g_fold_scratch_mutex);
  if (g_fold_scratch_address[device] == nullptr) {
    void* ptr = nullptr;
    cuda_check(cudaGetSymbolAddress(&ptr, g_fold_scratch), "cudaGetSymbolAddress(fold scratch)");
    g_fold_scratch_address[device] = ptr;
  }
  return g_fold_scratch_address[device];
}

}  // namespace

extern "C" uint64_t gf_fold_noalloc_max_bytes(void) { return kNoAllocScratchBytes; }

extern "C" int gf_fold_time_series_noalloc(const void* dev_input, int32_t input_is_u32, uint64_t n, double period,
                                           double tsamp, uint64_t nbin, uint64_t start_sample, float* dev_profile,
                                           double* dev_exposure, uint32_t* dev_status, void* stream) {
  return guarded([&] {
    check_arg(n > 0, "fold input must not be empty");
    check_arg(nbin > 0, "fold nbin must be positive");
    check_arg(nbin <= kMaxBins, "CUDA fold supports nbin <= 8192");
    const uint64_t nblocks = fold_blocks(n);
    check_arg(nblocks < (1ull << 31), "fold input too long");
    // each block keeps 2 * nbin doubles; compared by division so nothing wraps
    if (nblocks > kNoAllocScratchBytes / (2 * nbin * sizeof(double))) {
      raise(GF_EINVAL, "fold without allocation: " + std::to_string(n) + " samples x " + std::to_string(nbin) +
                           " bins need " + std::to_string(nblocks) + " x " + std::to_string(2 * nbin * 8) +
                           " bytes of scratch, above the fixed " + std::to_string(kNoAllocScratchBytes) +
                           " bytes; use gf_fold_time_series");
    }
    // folding.cpp:44-73 validation, as gf_fold_time_series
    check_arg(std::isfinite(period) && period > 0.0, "fold period must be finite and positive");
    check_arg(std::isfinite(tsamp) && tsamp > 0.0, "fold tsamp must be finite and positive");
    check_arg(dev_input && dev_profile && dev_exposure && dev_status, "null argument");
    const double step = tsamp / period * static_cast<double>(nbin);
    const double hi = static_cast<double>(start_sample + n - 1) * step + step;
    check_arg(std::isfinite(hi) && std::ceil(hi) < 9.2e18, "fold phase bin index exceeds int64 range");
    auto s = as_stream(stream);
    const uint64_t blocks = nblocks;
    double* partial = static_cast<double*>(fold_scratch_address());
    // the status word must start at zero; the partial sums are overwritten
    cuda_check(cudaMemsetAsync(dev_status, 0, 4, s), "cudaMemsetAsync(fold status)");
    launch_fold_partial(dev_input, input_is_u32 != 0, n, step, start_sample, nbin, static_cast<unsigned>(blocks), partial,
                        dev_status, s);
    fold_reduce_kernel<<<static_cast<unsigned>(ceil_div(nbin, kThreads)), kThreads, 0, s>>>(
        partial, static_cast<int>(blocks), nbin, dev_profile, dev_exposure);
    cuda_check(cudaGetLastError(), "fold launch");
  });
}

// ---------------------------------------------------------------------------
// Spectrum folding: subint x channel x phase cubes (folding.cpp:237-438)
// ---------------------------------------------------------------------------
//
// fold_spectrum_cpu: sample t of subint s = t / subint_samples covers the
// scaled phase interval [(start+t)*step, (start+t+1)*step); every output
// channel's value (the mean of `factor` adjacent input channels) is added
// with the overlap weight to cube[s][c][phase], the weight to
// exposure[s][phase]; the cube is sums / exposure.  One CTA per (subint, 32 V
// output channels): a lane per V neighbouring channels, each warp over its own
// run of the subint's samples.  A warp stays in one phase bin for 1 / step
// samples, so sums are kept in registers and flushed to the FP64 sums in shared
// memory when the bin changes; the loads of eight samples go ahead of their
// sums.  Bound: FP64 issue, six operations per sample for the phase and its
// weight, shared by V channels, and three per value.  V = 4 (one word) for
// 8-bit channels where the sums of 128 channels fit (nbin <= 96), else 1.
// Whole fold of a candidate (200,003 samples x 1024 channels, 64 bins, 13
// subints), an atomic per sample and channel and serial projections before:
// 3.14 -> 1.12 ms.

namespace gf {
namespace {

constexpr uint64_t kSpecMaxBins = 256;
constexpr uint64_t kSpecWideBins = 96;   // V = 4: 4 x 32 x 8 bytes of sums per bin
constexpr int kSpecThreads = 512;   // at most (spec_threads)
constexpr int kSpecAhead = 8;

template <typename T>
__device__ __forceinline__ double spec_value(const T* row, uint64_t c, uint64_t factor) {
  double v = 0.0;
  for (uint64_t k = 0; k < factor; ++k) v += static_cast<double>(row[c * factor + k]);
  return factor == 1 ? v : v / static_cast<double>(factor);
}

// Warps by the samples of a subint (a run of at least 16 each) and by the sums to
// clear and to write out, 1 to 16.  100,000 samples x 8 channels in subints of 7:
// 169 us with 16 warps, 65 with one.
unsigned spec_threads(uint64_t subint_samples, uint64_t nbin, uint64_t v) {
  const uint64_t warps = std::max(ceil_div(subint_samples, 16), ceil_div(nbin * v, 32));
  return 32 * static_cast<unsigned>(umin64(warps, kSpecThreads / 32));
}

template <typename T, int V>
__global__ void __launch_bounds__(kSpecThreads) fold_spectrum_kernel(const T* __restrict__ in, uint64_t nsamples,
                                                                     uint64_t nchans, uint64_t nout, uint64_t factor,
                                                                     double step, uint64_t start, uint64_t nbin,
                                                                     uint64_t subint_samples,
                                                                     float* __restrict__ cube,
                                                                     double* __restrict__ exposure,
                                                                     uint32_t* status) {
  extern __shared__ double sacc[];  // sums [nbin][V][32], exposure [nbin]
  double* sums = sacc;
  double* expo = sacc + nbin * 32 * V;
  const uint64_t s = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t c = (static_cast<uint64_t>(blockIdx.y) * 32 + lane) * V;
  const bool valid = c < nout;
  for (uint64_t i = threadIdx.x; i < nbin * (32 * V + 1); i += blockDim.x) sacc[i] = 0.0;
  __syncthreads();
  const uint64_t t0 = s * subint_samples;
  const uint64_t t1 = umin64(nsamples, t0 + subint_samples);
  // this warp's run of the subint
  const uint64_t per = ceil_div(t1 - t0, blockDim.x / 32);
  const uint64_t w0 = t0 + umin64(warp * per, t1 - t0), w1 = umin64(w0 + per, t1);
  const int64_t nb = static_cast<int64_t>(nbin);
  int64_t cur = -1, cur_m = 0;   // the bin at hand, and it modulo nbin
  double bl = 0.0, br = 0.0, cs[V], ce = 0.0;
#pragma unroll
  for (int j = 0; j < V; ++j) cs[j] = 0.0;
  auto flush = [&]() {
    if (cur < 0) return;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if (valid) atomicAdd(sums + (cur_m * V + j) * 32 + lane, cs[j]);
      cs[j] = 0.0;
    }
    if (lane == 0) atomicAdd(expo + cur_m, ce);
    ce = 0.0;
  };
  for (uint64_t base = w0; base < w1; base += kSpecAhead) {
    uint32_t words[kSpecAhead];
    double vals[kSpecAhead];
#pragma unroll
    for (int q = 0; q < kSpecAhead; ++q) {
      if (base + q >= w1 || !valid) {
        words[q] = 0u;
        vals[q] = 0.0;
      } else if (V == 4) {
        words[q] = __ldg(reinterpret_cast<const uint32_t*>(in + (base + q) * nchans + c));
      } else {
        vals[q] = spec_value(in + (base + q) * nchans, c, factor);
      }
    }
#pragma unroll
    for (int q = 0; q < kSpecAhead; ++q) {
      const uint64_t t = base + q;
      if (t >= w1) break;
      if (V == 1 && !isfinite(vals[q])) atomicOr(status, GF_STATUS_NONFINITE);
      const double lo = __dmul_rn(static_cast<double>(start + t), step);
      const double hi = __dadd_rn(lo, step);
      auto add = [&](double w) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
          const double v = V == 4 ? static_cast<double>((words[q] >> (8 * j)) & 0xffu) : vals[q];
          cs[j] = __dadd_rn(cs[j], __dmul_rn(v, w));
        }
        ce = __dadd_rn(ce, w);
      };
      if (cur >= 0 && lo >= bl && hi <= br) {
        const double w = __dsub_rn(hi, lo);
        if (w > 0.0) add(w);
        continue;
      }
      const int64_t first = static_cast<int64_t>(floor(lo));
      const int64_t last = static_cast<int64_t>(ceil(hi) - 1.0);
      for (int64_t bin = first; bin <= last; ++bin) {
        const double l = static_cast<double>(bin), r = l + 1.0;
        const double w = __dsub_rn(hi < r ? hi : r, lo > l ? lo : l);
        if (!(w > 0.0)) continue;
        if (bin != cur) {
          flush();
          cur = bin;
          cur_m = bin % nb;
          bl = l;
          br = r;
        }
        add(w);
      }
    }
  }
  flush();
  __syncthreads();
  // a warp per channel, lanes over the bins
  const uint64_t c0 = static_cast<uint64_t>(blockIdx.y) * 32 * V;
  for (uint64_t k = warp; k < 32 * V && c0 + k < nout; k += blockDim.x / 32) {
    float* out = cube + (s * nout + c0 + k) * nbin;
    for (uint64_t p = lane; p < nbin; p += 32) {
      const double e = expo[p];
      out[p] = e > 0.0 ? static_cast<float>(sums[(p * V + k % V) * 32 + k / V] / e) : 0.0f;
    }
  }
  if (blockIdx.y == 0)
    for (uint64_t p = threadIdx.x; p < nbin; p += blockDim.x) exposure[s * nbin + p] = expo[p];
}

// project_folded_cube (folding.cpp:237-296): time_phase[s][p] = mean over
// channels, freq_phase[c][p] and profile[p] exposure-weighted means, FP64.  A
// CTA per 32 bins (and subint): lanes over bins, 32 warps over interleaved
// terms, whose sums are added in warp order (one thread per bin over all terms
// in the reference's order took 1 ms for 13 x 1024 of them).
constexpr int kProjectWarps = 32;

__device__ __forceinline__ double project_sum(double v, double (*part)[32]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  part[warp][lane] = v;
  __syncthreads();
  double sum = 0.0;
  if (warp == 0)
    for (int w = 0; w < kProjectWarps; ++w) sum = __dadd_rn(sum, part[w][lane]);
  return sum;
}

__global__ void __launch_bounds__(32 * kProjectWarps) project_time_kernel(const float* __restrict__ cube,
                                                                          const double* __restrict__ exposure,
                                                                          uint64_t nchans, uint64_t nbin,
                                                                          float* __restrict__ time_phase) {
  __shared__ double part[kProjectWarps][32];
  const uint32_t bin_ctas = static_cast<uint32_t>(ceil_div(nbin, 32));
  const uint64_t s = blockIdx.x / bin_ctas, p = static_cast<uint64_t>(blockIdx.x % bin_ctas) * 32 + (threadIdx.x & 31);
  double acc = 0.0;
  if (p < nbin)
    for (uint64_t c = threadIdx.x >> 5; c < nchans; c += kProjectWarps)
      acc += static_cast<double>(cube[(s * nchans + c) * nbin + p]);
  acc = project_sum(acc, part);
  if (threadIdx.x < 32 && p < nbin)
    time_phase[s * nbin + p] =
        exposure[s * nbin + p] > 0.0 ? static_cast<float>(acc / static_cast<double>(nchans)) : 0.0f;
}

__global__ void project_freq_kernel(const float* __restrict__ cube, const double* __restrict__ exposure,
                                    uint64_t nsubint, uint64_t nchans, uint64_t nbin, float* __restrict__ freq_phase) {
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (i >= nchans * nbin) return;
  const uint64_t c = i / nbin, p = i % nbin;
  double sum = 0.0, ex = 0.0;
  for (uint64_t s = 0; s < nsubint; ++s) {
    const double e = exposure[s * nbin + p];
    if (!(e > 0.0)) continue;
    sum += static_cast<double>(cube[(s * nchans + c) * nbin + p]) * e;
    ex += e;
  }
  freq_phase[i] = ex > 0.0 ? static_cast<float>(sum / ex) : 0.0f;
}

__global__ void __launch_bounds__(32 * kProjectWarps) project_profile_kernel(const float* __restrict__ cube,
                                                                             const double* __restrict__ exposure,
                                                                             uint64_t nsubint, uint64_t nchans,
                                                                             uint64_t nbin,
                                                                             float* __restrict__ profile) {
  __shared__ double part[kProjectWarps][32];
  const uint64_t p = static_cast<uint64_t>(blockIdx.x) * 32 + (threadIdx.x & 31);
  double sum = 0.0, ex = 0.0;
  for (uint64_t s = 0; s < nsubint; ++s) {
    const double e = p < nbin ? exposure[s * nbin + p] : 0.0;
    if (!(e > 0.0)) continue;
    for (uint64_t c = threadIdx.x >> 5; c < nchans; c += kProjectWarps) {
      sum += static_cast<double>(cube[(s * nchans + c) * nbin + p]) * e;
      ex += e;
    }
  }
  sum = project_sum(sum, part);
  ex = project_sum(ex, part);
  if (threadIdx.x < 32 && p < nbin) profile[p] = ex > 0.0 ? static_cast<float>(sum / ex) : 0.0f;
}

}  // namespace
}  // namespace gf

extern "C" int gf_fold_spectrum(const void* dev_in, int32_t elem_bytes, uint64_t nsamples, uint64_t nchans,
                                double period, double tsamp, uint64_t nbin, uint64_t subint_samples,
                                uint64_t start_sample, uint64_t output_channels, float* dev_cube,
                                double* dev_exposure, uint32_t* dev_status, void* stream) {
  return guarded([&] {
    check_arg(dev_in && dev_cube && dev_exposure && dev_status, "null argument");
    check_arg(elem_bytes == 1 || elem_bytes == 2 || elem_bytes == 4, "elem_bytes must be 1, 2 or 4");
    // folding.cpp:44-104 validate_fold_shape / validate_spectrum_input
    check_arg(std::isfinite(period) && period > 0.0, "fold period must be finite and positive");
    check_arg(std::isfinite(tsamp) && tsamp > 0.0, "fold tsamp must be finite and positive");
    check_arg(nbin > 0, "fold nbin must be positive");
    check_arg(nbin <= kSpecMaxBins, "fold spectrum CUDA path supports nbin <= 256");
    check_arg(nsamples > 0 && nchans > 0, "fold spectrum shape must be non-empty");
    check_arg(subint_samples > 0, "fold subint_samples must be positive");
    check_arg(output_channels <= nchans, "fold output_channels must be <= input channel count");
    check_arg(output_channels == 0 || nchans % output_channels == 0,
              "fold input channel count must be divisible by output_channels");
    const uint64_t nout = output_channels == 0 ? nchans : output_channels;
    const uint64_t factor = nchans / nout;
    const double step = tsamp / period * static_cast<double>(nbin);
    const double hi = static_cast<double>(start_sample + nsamples - 1) * step + step;
    check_arg(std::isfinite(hi), "fold phase interval is invalid");
    const uint64_t nsubint = ceil_div(nsamples, subint_samples);
    check_arg(nsubint < (1ull << 31) && ceil_div(nout, 32) < 65536, "fold spectrum too large");
    auto s = as_stream(stream);
    cuda_check(cudaMemsetAsync(dev_status, 0, sizeof(uint32_t), s), "cudaMemsetAsync(status)");
    auto launch = [&](auto kernel, const auto* in, uint64_t v) {
      const size_t smem = nbin * (32 * v + 1) * sizeof(double);
      // the same limit on every call, whatever its bins (calls from several threads)
      const size_t limit = (v == 4 ? kSpecWideBins : kSpecMaxBins) * (32 * v + 1) * sizeof(double);
      const dim3 grid(static_cast<unsigned>(nsubint), static_cast<unsigned>(ceil_div(nout, 32 * v)));
      cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(limit)),
                 "cudaFuncSetAttribute(fold_spectrum)");
      kernel<<<grid, spec_threads(umin64(subint_samples, nsamples), nbin, v), smem, s>>>(in, nsamples, nchans, nout, factor, step, start_sample, nbin,
                                              subint_samples, dev_cube, dev_exposure, dev_status);
    };
    const auto* bytes = static_cast<const uint8_t*>(dev_in);
    if (elem_bytes == 1 && factor == 1 && nchans % 4 == 0 && nbin <= kSpecWideBins &&
        (reinterpret_cast<uintptr_t>(bytes) & 3u) == 0)
      launch(fold_spectrum_kernel<uint8_t, 4>, bytes, 4);
    else if (elem_bytes == 1)
      launch(fold_spectrum_kernel<uint8_t, 1>, bytes, 1);
    else if (elem_bytes == 2)
      launch(fold_spectrum_kernel<uint16_t, 1>, static_cast<const uint16_t*>(dev_in), 1);
    else
      launch(fold_spectrum_kernel<float, 1>, static_cast<const float*>(dev_in), 1);
    cuda_check(cudaGetLastError(), "fold_spectrum_kernel launch");
  });
}

extern "C" int gf_project_folded_cube(const float* dev_cube, const double* dev_exposure, uint64_t nsubint,
                                      uint64_t nchans, uint64_t nbin, float* dev_profile, float* dev_freq_phase,
                                      float* dev_time_phase, void* stream) {
  return guarded([&] {
    check_arg(dev_cube && dev_exposure && dev_profile && dev_freq_phase && dev_time_phase, "null argument");
    check_arg(nsubint > 0 && nchans > 0 && nbin > 0, "folded cube must be non-empty");
    auto s = as_stream(stream);
    const unsigned bin_ctas = static_cast<unsigned>(ceil_div(nbin, 32));
    project_time_kernel<<<static_cast<unsigned>(nsubint * bin_ctas), 32 * kProjectWarps, 0, s>>>(
        dev_cube, dev_exposure, nchans, nbin, dev_time_phase);
    project_freq_kernel<<<static_cast<unsigned>(ceil_div(nchans * nbin, 256)), 256, 0, s>>>(
        dev_cube, dev_exposure, nsubint, nchans, nbin, dev_freq_phase);
    project_profile_kernel<<<bin_ctas, 32 * kProjectWarps, 0, s>>>(dev_cube, dev_exposure, nsubint, nchans, nbin,
                                                                   dev_profile);
    cuda_check(cudaGetLastError(), "project kernels launch");
  });
}

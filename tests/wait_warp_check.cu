// A bounded wait gives one answer to the whole warp.  Block b's barrier
// completes b steps after the start, or never; the steps span the limit, so
// some blocks wait it out, some do not, and some end near it.  Prints "ok".
#define GF_WAIT_CYCLES 200000  // 0.1 ms
#include <cstdio>

#include <cuda_runtime.h>

#include "mbarrier.cuh"

constexpr int kBlocks = 96, kNever = 80;
constexpr long long kStep = 2 * GF_WAIT_CYCLES / kNever;

__global__ void check(uint32_t* answers, uint32_t* status) {
  __shared__ uint64_t bar;
  __shared__ uint32_t failed;
  if (threadIdx.x == 0) {
    gf::mbar_init(&bar, 1);
    failed = 0;
  }
  __syncthreads();
  const int b = blockIdx.x;
  if (threadIdx.x >= 32) {
    const long long start = clock64();
    while (b < kNever && clock64() - start < b * kStep) {
    }
    if (b < kNever && threadIdx.x == 32) gf::mbar_arrive(&bar);
  } else {
    const bool ok = gf::wait_warp(&bar, 0, &failed, status + b);
    const uint32_t votes = __ballot_sync(0xffffffffu, ok);
    answers[b * 32 + threadIdx.x] = __shfl_sync(0xffffffffu, votes, 31 - threadIdx.x);
  }
  __syncthreads();
  if (threadIdx.x == 0 && failed != (status[b] ? 1u : 0u)) answers[b * 32] = 1u;
}

int main() {
  uint32_t *answers, *status;
  cudaMallocManaged(&answers, kBlocks * 32 * sizeof(uint32_t));
  cudaMallocManaged(&status, kBlocks * sizeof(uint32_t));
  for (int b = 0; b < kBlocks; ++b) status[b] = 0;
  check<<<kBlocks, 64>>>(answers, status);
  if (cudaDeviceSynchronize() != cudaSuccess) return std::printf("%s\n", cudaGetErrorString(cudaGetLastError())), 1;
  int passed = 0, gave_up = 0;
  for (int b = 0; b < kBlocks; ++b) {
    const uint32_t want = status[b] ? 0u : 0xffffffffu;
    if (status[b] != 0 && status[b] != GF_STATUS_PIPELINE) return std::printf("block %d: status %u\n", b, status[b]), 1;
    for (int l = 0; l < 32; ++l)
      if (answers[b * 32 + l] != want) return std::printf("block %d lane %d: %08x\n", b, l, answers[b * 32 + l]), 1;
    (status[b] ? gave_up : passed) += 1;
    if (b < kNever / 4 && status[b]) return std::printf("block %d gave up early\n", b), 1;
    if (b >= kNever && !status[b]) return std::printf("block %d did not give up\n", b), 1;
  }
  std::printf("ok %d passed, %d gave up\n", passed, gave_up);
  return 0;
}

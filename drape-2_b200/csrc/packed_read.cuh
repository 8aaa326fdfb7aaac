// Reads of a float4-per-particle device vector into the caller's three floats per particle. A kernel writes the packed
// floats into page-locked host memory (contiguous 128-byte stores over the bus), from where the host copies them: a
// copy of the padded vector into pageable memory went through the driver's staging buffer and a conversion loop (150k
// particles 0.75-0.95 ms, 60k 0.31-0.36 ms; packed 0.16 ms and 0.07 ms).
#pragma once

#include <cstdint>
#include <cstring>

#include "device_buffer.hpp"

namespace packed {

constexpr uint32_t kChunk = 1u << 14;  // particles a chunk; two chunks, one being copied while the next is packed

static __global__ void k_pack3(uint32_t n, const float4* __restrict__ src, float* __restrict__ dst) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < 3 * n; k += gridDim.x * blockDim.x)
    dst[k] = reinterpret_cast<const float*>(src + k / 3)[k % 3];
}

struct Reader {
  dbuf::HostPinned<float> buf;
  cudaEvent_t done[2] = {};
  Reader() = default;
  Reader(const Reader&) = delete;
  Reader& operator=(const Reader&) = delete;
  ~Reader() {
    for (cudaEvent_t e : done)
      if (e) cudaEventDestroy(e);
  }
  void init() {
    buf.alloc(2 * 3 * static_cast<size_t>(kChunk));
    for (cudaEvent_t& e : done) dbuf::check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
  }
  // out[3 * count] from src[count], after the work queued on `stream`; returns when out is written.
  void read(const float4* src, size_t count, float* out, cudaStream_t stream) {
    auto pack = [&](size_t c) {
      const size_t at = c * kChunk, n = count - at < kChunk ? count - at : kChunk;
      k_pack3<<<static_cast<int>((3 * n + 511) / 512), 512, 0, stream>>>(static_cast<uint32_t>(n), src + at,
                                                                         buf.p + (c & 1) * 3 * kChunk);
      dbuf::check(cudaGetLastError(), "k_pack3");
      dbuf::check(cudaEventRecord(done[c & 1], stream), "cudaEventRecord");
    };
    const size_t chunks = (count + kChunk - 1) / kChunk;
    for (size_t c = 0; c < chunks && c < 2; ++c) pack(c);
    for (size_t c = 0; c < chunks; ++c) {
      for (;;) {
        const cudaError_t e = cudaEventQuery(done[c & 1]);
        if (e == cudaSuccess) break;
        if (e != cudaErrorNotReady) dbuf::check(e, "cudaEventQuery");
      }
      const size_t at = c * kChunk, n = count - at < kChunk ? count - at : kChunk;
      std::memcpy(out + 3 * at, buf.p + (c & 1) * 3 * kChunk, 3 * sizeof(float) * n);
      if (c + 2 < chunks) pack(c + 2);
    }
  }
};

}  // namespace packed

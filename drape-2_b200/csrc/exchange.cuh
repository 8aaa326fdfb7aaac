// Sums across the blocks of a cooperative grid by messages: every block writes its value with a sequence number in the
// same 16-byte word, and reads everybody's words until all carry the number. Value and flag arrive together, so an
// exchange needs neither a release fence nor a second read of the partials, the two round trips to the L2 that a counter
// barrier followed by a load of every block's partial sum adds. It orders nothing but its own values.
//
// What bounds it is the way to the L2 and back (measured on a B200: 0.29 us from a store to the poll that sees it within
// a die, 0.5 us across the dies) and the polls themselves: a poll of a word that has not been written yet takes the line
// into the reader's die, and the write then has to fetch it back. Each block therefore writes its message to
// kMailReplicas copies, each read by a quarter of the blocks, each message has 64 bytes to itself, and a block may let
// `delay` clock cycles pass between its message and its first poll, by when the others' words are there if they all sent
// at about the same time. One sum over 148 blocks of 512 threads, block sums included: 1.3 us (0.97-1.2 us with a delay
// of 400-800 cycles in lockstep), against 2.09 us for a counter barrier followed by a read of every block's partial sum
// and 3.1-4.3 us for one copy without a delay; 2 or 8 copies 1.32-1.42 us, 32-byte slots 1.36-1.50 us; a two-level tree
// of blocks 1.6-1.8 us.
#pragma once

#include <cstdint>

namespace dcu {

struct __align__(16) MailWord {
  double value;
  unsigned long long tag;
};

constexpr uint32_t kMailReplicas = 4;  // copies of each message
constexpr uint32_t kMailWords = 4;     // words of a message's slot (64 bytes): up to this many values a message
// Words of the mailbox of `blocks` blocks: two halves, used by turns (a block sends message k + 2 only after it has
// message k + 1 of every block, and hence after every block has read its message k).
__host__ __device__ constexpr size_t mailWords(size_t blocks) { return 2 * static_cast<size_t>(kMailReplicas) * blocks * kMailWords; }

// 16-byte loads and stores that are one access each.
__device__ __forceinline__ void storeWord(MailWord* p, double value, unsigned long long tag) {
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
               "l"(__double_as_longlong(value)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ void loadWord(const MailWord* p, double& value, unsigned long long& tag) {
  long long v;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(v), "=l"(tag)
               : "l"(p)
               : "memory");
  value = __longlong_as_double(v);
}
// A float4 whose w is a tag, the same way.
__device__ __forceinline__ void storeTagged(float4* p, float3 v, uint32_t tag) {
  const unsigned long long lo = static_cast<unsigned long long>(__float_as_uint(v.y)) << 32 | __float_as_uint(v.x);
  const unsigned long long hi = static_cast<unsigned long long>(tag) << 32 | __float_as_uint(v.z);
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p), "l"(lo), "l"(hi)
               : "memory");
}
__device__ __forceinline__ uint32_t loadTagged(const float4* p, float3& v) {
  unsigned long long lo, hi;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  v.x = __uint_as_float(static_cast<uint32_t>(lo));
  v.y = __uint_as_float(static_cast<uint32_t>(lo >> 32));
  v.z = __uint_as_float(static_cast<uint32_t>(hi));
  return static_cast<uint32_t>(hi >> 32);
}

// The sum of a warp's 32 doubles, in every lane, by two FP64 matrix products with a matrix of ones (column sums, then
// the sum of the four pairs left in a quad): 74 cycles, against 184 for five rounds of shuffles and additions.
__device__ __forceinline__ double warpSum(double v) {
  double a, b;
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %5};"
               : "=d"(a), "=d"(b)
               : "d"(1.0), "d"(v), "d"(0.0), "d"(0.0));
  const double t = a + b;
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %5};"
               : "=d"(a), "=d"(b)
               : "d"(t), "d"(1.0), "d"(0.0), "d"(0.0));
  return a;
}

// Polls of one waiting loop: true once the limit has run out or another block has raised the error flag (looked at every
// 32nd poll only).
struct BoundedWait {
  unsigned int spins = 0;
  unsigned long long start = 0;
  __device__ __forceinline__ bool expired(Control* ctl, unsigned long long limitNs) {
    if ((++spins & 31u) != 0) return false;
    if (*reinterpret_cast<volatile int*>(&ctl->error) != 0) return true;
    const unsigned long long now = globalTimerNs();
    if (start == 0) start = now;
    if (now - start <= limitNs) return false;
    atomicExch(&ctl->error, 1);
    return true;
  }
};

// One exchange, run by one whole warp of every block: `mine` (the same in all lanes) is added over the `size` blocks in
// a fixed order, and every lane of every block gets the same totals. `seq` is the exchange's number, one more than the
// last one's. `delay`: clock cycles before the first poll. Returns false when the wait gave up.
template <int K>
__device__ inline bool mailSum(MailWord* box, Control* ctl, unsigned long long limitNs, uint32_t rank, uint32_t size,
                               unsigned long long seq, const double (&mine)[K], double (&total)[K], int delay = 0) {
  static_assert(K >= 1 && K <= static_cast<int>(kMailWords), "mailSum: a message is one slot");
  constexpr int kLoads = 5;  // slots a lane waits for at a time (160 blocks a round: one round for one block per SM)
  const uint32_t lane = threadIdx.x & 31u;
  MailWord* half = box + (seq & 1ull) * (mailWords(size) / 2);
  if (lane < kMailReplicas)
#pragma unroll
    for (int k = 0; k < K; ++k)
      storeWord(half + (static_cast<size_t>(lane) * size + rank) * kMailWords + k, mine[k], seq);
  const MailWord* copy = half + static_cast<size_t>(rank % kMailReplicas) * size * kMailWords;
  double t[K];
#pragma unroll
  for (int k = 0; k < K; ++k) t[k] = 0.0;
  BoundedWait wait;
  for (const long long start = clock64(); clock64() - start < delay;) {
  }
  for (uint32_t b0 = 0; b0 < size; b0 += 32 * kLoads) {
    double x[kLoads][K];
    bool have[kLoads];
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      have[j] = b0 + 32 * j + lane >= size;
#pragma unroll
      for (int k = 0; k < K; ++k) x[j][k] = 0.0;
    }
    for (;;) {
      unsigned long long tag[kLoads][K];
#pragma unroll
      for (int j = 0; j < kLoads; ++j)
        if (!have[j])
#pragma unroll
          for (int k = 0; k < K; ++k) loadWord(copy + static_cast<size_t>(b0 + 32 * j + lane) * kMailWords + k, x[j][k], tag[j][k]);
      bool all = true;
#pragma unroll
      for (int j = 0; j < kLoads; ++j)
        if (!have[j]) {
          bool h = true;
#pragma unroll
          for (int k = 0; k < K; ++k) h = h && tag[j][k] == seq;
          have[j] = h;
          all = all && h;
        }
      if (__all_sync(0xffffffffu, all)) break;
      if (__any_sync(0xffffffffu, wait.expired(ctl, limitNs))) return false;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] += ((x[0][k] + x[1][k]) + (x[2][k] + x[3][k])) + x[4][k];
  }
#pragma unroll
  for (int k = 0; k < K; ++k) total[k] = warpSum(t[k]);
  return true;
}

// Named block barriers (barrier 0 is __syncthreads): `threads` counts everyone who syncs or arrives.
template <int Id>
__device__ __forceinline__ void namedSync(int threads) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"n"(Id), "r"(threads) : "memory");
}
template <int Id>
__device__ __forceinline__ void namedArrive(int threads) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"n"(Id), "r"(threads) : "memory");
}

}  // namespace dcu

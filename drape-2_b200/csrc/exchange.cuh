// Sums across the blocks of a cooperative grid by messages: every block writes its value with a sequence number in the
// same 16-byte word, and reads everybody's words until all carry the number. Value and flag arrive together, so an
// exchange needs neither a release fence nor a second read of the partials, the two round trips to the L2 that a counter
// barrier followed by a load of every block's partial sum adds. It orders nothing but its own values.
//
// What bounds it is the way to the L2 and back (measured on a B200: 0.29 us from a store to the poll that sees it within
// a die, 0.5 us across the dies) and the polls themselves: a poll of a word that has not been written yet takes the line
// into the reader's die, and the write then has to fetch it back. So a block lets some clock cycles pass between its
// message and its first poll, by when the others' words are usually there, and adapts them: a little less after each
// exchange whose first poll saw everything, more after one that did not. The words of one value lie side by side (a
// warp's poll reads 512 contiguous bytes), all loads are issued before any tag is looked at, and one copy of the messages
// serves all readers. One sum over 148 blocks of 512 threads, block sums included, in lockstep: 0.97-1.1 us, against
// 2.09 us for a counter barrier followed by a read of every block's partial sum; polling at once 1.3-4.3 us depending on
// the copies and their spacing. In the PCG (us per iteration at 1,600, 10k and 60k particles): adapted 2.82, 2.85, 4.25;
// a fixed delay of 500 cycles 2.72, 2.92, 5.40, of 700 2.86, 2.86, 4.74, of 900 3.02, 2.85, 4.41; adapted with two copies
// 3.06, 3.05, 4.21; four copies 64 bytes apart at 700 cycles 2.9-3.4, 3.0-3.4, 4.3. A two-level tree of blocks takes
// 1.6-1.8 us a sum.
#pragma once

#include <cstdint>

namespace dcu {

struct __align__(16) MailWord {
  double value;
  unsigned long long tag;
};

constexpr uint32_t kMailWords = 2;  // a message is up to this many values
// The wait before an exchange's first poll, in clock cycles: its steps down and up, and its range.
constexpr int kDelayDown = 8, kDelayUp = 128, kDelayLeast = 300, kDelayMost = 4000;
// Words of the mailbox of `blocks` blocks: two halves, used by turns (a block sends message k + 2 only after it has
// message k + 1 of every block, and hence after every block has read its message k).
__host__ __device__ constexpr size_t mailWords(size_t blocks) { return 2 * blocks * kMailWords; }

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
// last one's. `delay`: clock cycles before the first poll, adapted. Returns false when the wait gave up.
template <int K>
__device__ inline bool mailSum(MailWord* box, Control* ctl, unsigned long long limitNs, uint32_t rank, uint32_t size,
                               unsigned long long seq, const double (&mine)[K], double (&total)[K], int& delay) {
  static_assert(K >= 1 && K <= static_cast<int>(kMailWords), "mailSum: a message is at most kMailWords values");
  constexpr int kLoads = 5;  // words a lane waits for at a time (160 blocks a round: one round for one block per SM)
  const uint32_t lane = threadIdx.x & 31u;
  MailWord* half = box + (seq & 1ull) * (mailWords(size) / 2);
  double t[K];
#pragma unroll
  for (int k = 0; k < K; ++k) t[k] = 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (lane == 0) storeWord(half + static_cast<size_t>(k) * size + rank, mine[k], seq);
  BoundedWait wait;
  for (const long long start = clock64(); clock64() - start < delay;) {
  }
  bool first = true;
  for (uint32_t b0 = 0; b0 < size; b0 += 32 * kLoads) {
    double x[kLoads][K];
    for (;;) {
      // All loads first (lanes past the end repeat the last block's word), then the tags.
      unsigned long long tag[kLoads][K];
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < kLoads; ++j)
          loadWord(half + static_cast<size_t>(k) * size + min(b0 + 32 * j + lane, size - 1), x[j][k], tag[j][k]);
      unsigned long long differ = 0;
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < kLoads; ++j) differ |= tag[j][k] ^ seq;
      if (__all_sync(0xffffffffu, differ == 0)) break;
      first = false;
      if (__any_sync(0xffffffffu, wait.expired(ctl, limitNs))) return false;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
#pragma unroll
      for (int j = 0; j < kLoads; ++j)
        if (b0 + 32 * j + lane >= size) x[j][k] = 0.0;
      t[k] += ((x[0][k] + x[1][k]) + (x[2][k] + x[3][k])) + x[4][k];
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) total[k] = warpSum(t[k]);
  delay = first ? max(delay - kDelayDown, kDelayLeast) : min(delay + kDelayUp, kDelayMost);
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

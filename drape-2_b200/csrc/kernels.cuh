// Device data layout and kernels of one implicit-Euler substep (predict / contact setup, contact activation,
// term records and slot-parallel assembly, persistent PCG + line search, finish), plus statistics.
//
// Reference algorithm: CpuSolver::Impl::substep (libs/sim/src/cpu_solver.cpp:230-314) in the displacement form of the
// reference's 32-bit GPU path (u = x - xStart, term positions relative to the term's first vertex;
// libs/sim/kernels/kernels.h:30-448). Per Newton iteration this file runs four launches instead of the reference's
// ~40 + 13 per CG iteration dispatches with host round trips (gpu_solver_core.cpp:325-407):
//   k_activate   contact activation (kernels.h:85-99)
//   k_terms      every stretch and hinge term evaluated once into a derivative record (kernels.h:137-176)
//   k_assemble   each 3x3 Hessian block summed by the thread that owns its slot from the records of the row's incident
//                terms; the diagonal slot's thread adds the gradient, block-Jacobi inverse and contact release
//                (replaces the contribution buffers + gather, kernels.h:104-231)
//   k_solve      one cooperative persistent launch: PCG (kernels.h:237-347), contact force, FP64 Newton slope, FP64
//                line search and step application (cpu_solver.cpp:264-283) with device-side decisions.
#pragma once

#include <cuda/atomic>
#include <cstdint>

#include "device_math.cuh"

namespace dcu {

constexpr int kWarp = 32;
constexpr int kAssembleThreads = 256;  // k_assemble block size (one thread per block slot)
constexpr int kRowLanes = 2;        // lanes per block row in the single solver's SpMV
constexpr int kSolveThreads = 1024; // k_solve block size (one block per SM)
constexpr uint32_t kPinnedBit = 0x80000000u;
constexpr uint32_t kSmemSlotBytes = 40;      // one block slot in shared memory: 9 floats + a column index
constexpr int kPartialStride = 4;   // doubles per block in the partials array

struct Particle {
  float mass;
  uint32_t fabric, garment, pinned;
};

struct Fabric {
  float k[3];       // stretch warp, weft, bias
  float limit[2];   // strain limits
  float thickness, friction, damping;
};

struct Stretch {
  uint32_t v[3];
  uint32_t fabric;
  float4 d;  // dmInv (0,0), (1,0), (0,1), (1,1)
  float area;
  float pad[3];
};

struct Hinge {
  uint32_t v[4];
  float K, rest;
  float pad[2];
};

struct Seam {
  uint32_t a, b, garment;
  float startGap;
};

struct Contact {
  float4 normal;  // xyz: plane normal, w: offset = r - phi(xStart)
  float force, frictionLambda;
  uint32_t nearBody, active;
};

struct Garment {
  int32_t phase;  // 0 Assembling, 1 Settling
  int32_t pad;
  double assemblyTime;
};

// Device control block: the PCG / Newton scalars every block of k_solve recomputes identically, plus counters.
struct Control {
  int newtonDone;   // this substep's Newton loop has stopped (slope >= 0 or max move < 1e-9)
  int error;        // 1: a grid barrier or an exchange gave up waiting; 2: a row exceeded the assembly capacity; 4: a
                    // block's rows or halo did not fit what the host sized (the resident-row kernels)
  unsigned long long barrierArrivals;
  long long cgIterations, newtonIterations, lineSearchHalvings, substeps, energyEvaluations;
  double lastAlpha, lastSlope, lastE0, lastMaxMove;
  int lastCg;
  int pad;
  long long learnedSolves, precondFallbacks;  // PCG solves with the learned preconditioner; of those, restarted
  long long pcgNs;  // %globaltimer nanoseconds inside the PCG solves (block 0's view: CG init to the last iteration)
  unsigned long long frameBeginNs;  // %globaltimer at the current frame's first kernel (0: not started)
};

constexpr unsigned int kCgLogCapacity = 1u << 16;  // PCG iterations per Newton iteration, ring buffer

struct Params {
  float h, invH2;
  float gravity[3];
  float limitScale, seamStiffness, closingSpeed, frictionSlip, collisionOffset, dampingScale, assemblyExtraDamping;
  float contactReach, contactSnap;
  double hD, cgTolerance;
  int maxCg;
  uint32_t n, nStretch, nHinge, nSeam, nBlocks, nGarments, slotsPadded;
  uint32_t smemSlots;   // k_solve: block slots a block keeps in shared memory
  int learnedSwitch;    // k_solve<true>: block-Jacobi iterations before the learned preconditioner takes over
  int pcgVariant;       // the block-Jacobi PCG form: 0 reference order (resident rows where the scene fits), 1 pipelined,
                        // 2 Chronopoulos-Gear, 3 reference order on the 1024-thread kernel (kept in the view so that
                        // captured frame graphs are recaptured when it changes)
  uint32_t residentSlots, residentNodes;  // k_solve_rows: a block's padded slots and its rows and halo, in shared memory
  uint32_t factorSlots; // k_solve_rows_learned: a block's padded factor slots
  uint32_t haloStride;  // entries of `halo` per solve block
  // k_solve_rows_multi: slots of each row kept in shared memory (even), a block's rows, and its padded slots in the L2.
  uint32_t multiKept, multiRows, spillSlots;
  unsigned long long barrierLimitNs;
};

struct Dev {
  Params P;
  FieldInfo field;
  double fieldOrigin[3], fieldCell;
  const float* fieldValues;
  const Particle* particle;
  const Fabric* fabric;
  Garment* garment;
  const Stretch* stretch;
  const Hinge* hinge;
  const Seam* seam;
  const uint32_t* rowStart;
  const uint32_t* colIndex;  // bit 31: the column's particle is pinned
  const uint32_t* diagSlot;
  const uint32_t* incStart;
  const uint32_t* incEntry;
  const uint32_t* offSlot;   // the off-diagonal slots in slot order: row << 6 | row-local position
  const uint32_t* offStart;  // per off-diagonal slot: its contributions [offStart[k], offStart[k + 1]) of offCode
  const uint32_t* offCode;     // per contribution, in gather order: kind << 30 | term << 4 | vertex a << 2 | block b
  float4 *x, *v, *xStart, *yRel, *u, *grad, *step, *r, *z, *p0, *p1, *ap, *apFull, *resid;
  float4 *pm0, *pm1, *pz;  // pipelined PCG only: the two m = M w buffers and z = A q (null where not allocated)
  float4* stretchDer;      // per stretch term: its StretchDer record (6 float4), written by termsRows
  float4* hingeDer;        // per hinge term: its HingeDer record (4 float4)
  const float* Lf;         // learned factor L: 9 planes of slotsPadded floats on lower slots (k_solve<true>)
  const uint32_t* tslot;   // slot of (j, i) for slot (i, j)
  const float4* LfRows;    // the factor by rows, three float4 a slot: L_ij at lower slots, L_ji at upper (i, j)
  float4* LfSliced;        // k_solve_rows_learned: 3 * factorSlots per block where the factor does not fit shared memory
  const float4* fExt;
  const float4* pinPos;
  float* blocks;   // 9 planes of slotsPadded floats, component 3*row+col
  float4* precond; // 3 float4 (rows) per particle
  Contact* contact;
  const uint16_t* localCol;   // per slot: its column among its solve block's rows and halo (k_localize)
  const uint32_t *halo, *haloCount;
  double* partials;
  uint8_t* spill;             // k_solve_rows_multi: kResidentSlotBytes * spillSlots per block
  struct MailWord* mail;      // the solve grid's mailbox and the number of the last exchange (exchange.cuh)
  unsigned long long* mailSeq;
  Control* ctl;
  int* cgLog;  // kCgLogCapacity entries
};

// ---------------------------------------------------------------------------------------------------------------
// Synchronisation of a group of co-resident blocks for the cooperative persistent kernels (cooperative launch
// guarantees co-residency). A group is the whole grid for one solver, or the blocks a batched launch gives one
// garment: `rank` is the block's index in its group and `size` the group's block count.
//
// Arrivals only ever increase: a launch's k-th barrier completes when the counter reaches base + k * size, base
// being the counter at the launch's start rounded down to a multiple of size (no barrier can complete before
// every block has arrived, so a block that reads the counter late still rounds to the same base). Thread 0 adds its
// block's arrival with release semantics after publishing the block's partial sums and polls with acquire loads; a
// time limit turns a lost block into an error status and a return instead of a hang.
//
// Reductions alternate between two halves of the group's partials array, so a block that has already passed a
// barrier and publishes its next partial cannot overwrite values a slower block is still summing.

__device__ __forceinline__ unsigned long long globalTimerNs() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

struct GridSync {
  Control* ctl;
  unsigned long long target, limitNs;
  unsigned int parity;
  uint32_t rank, size;

  __device__ void init(Control* c, unsigned long long lim, uint32_t rank_, uint32_t size_) {
    __shared__ unsigned long long base;
    if (threadIdx.x == 0) {
      cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> a(c->barrierArrivals);
      const unsigned long long now = a.load(cuda::memory_order_relaxed);
      base = now - now % size_;
    }
    __syncthreads();
    ctl = c;
    target = base;
    limitNs = lim;
    parity = 0;
    rank = rank_;
    size = size_;
  }
  // The whole grid as one group.
  __device__ void init(Control* c, unsigned long long lim) { init(c, lim, blockIdx.x, gridDim.x); }

  // One thread's arrival for the whole block (release: the block's writes before it, ordered by the caller, become
  // visible) and its bounded wait for the group (acquire). The caller advances `target` first. Returns 0 when the
  // limit ran out or another block raised the error flag.
  __device__ int arriveAndWait() const {
    unsigned long long* counter = &ctl->barrierArrivals;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(counter), "l"(1ull) : "memory");
    unsigned int spins = 0;
    const unsigned long long start = globalTimerNs();
    for (;;) {
      unsigned long long seen;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(counter) : "memory");
      if (seen >= target) return 1;
      if ((++spins & 31u) == 0) {
        if (*reinterpret_cast<volatile int*>(&ctl->error) != 0) return 0;
        if (globalTimerNs() - start > limitNs) {
          atomicExch(&ctl->error, 1);
          return 0;
        }
      }
    }
  }

  // A barrier of the whole group (no data).
  __device__ bool sync() {
    __shared__ int ok;
    target += size;
    __syncthreads();
    if (threadIdx.x == 0) ok = arriveAndWait();
    __syncthreads();
    return ok != 0;
  }
};

}  // namespace dcu

#include "exchange.cuh"

namespace dcu {

// Block-wide FP64 sums (or maxima); thread 0 gets the result in out. Fixed tree shape, so deterministic.
template <int K, bool Max = false>
__device__ inline void blockReduce(double (&v)[K], double* out) {
  __shared__ double red[K][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_down_sync(0xffffffffu, v[k], o);
      v[k] = Max ? fmax(v[k], y) : v[k] + y;
    }
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) red[k][w] = v[k];
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double s = lane < nw ? red[k][lane] : (Max ? -INFINITY : 0.0);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_down_sync(0xffffffffu, s, o);
        s = Max ? fmax(s, y) : s + y;
      }
      if (lane == 0) out[k] = s;
    }
  }
}

template <int K>
__device__ inline void blockSum(double (&v)[K], double* out) {
  blockReduce<K, false>(v, out);
}

// a + b, or the larger of the two.
template <bool Max>
__device__ __forceinline__ double combine(double a, double b) {
  return Max ? fmax(a, b) : a + b;
}

// Grid-wide FP64 sums (or maxima). The warps' sums meet in shared memory; warp 0 combines them, publishes the block
// total, arrives at the group barrier and waits, then reads every block's total (lane l: blocks l, l + 32, ..., all
// loads issued before the first add) and combines them in a fixed order; the other warps wait at one block barrier
// meanwhile. Every block obtains bit-identical results and takes the same branches. Two block barriers per call: `red`
// is rewritten only after the closing barrier, by which warp 0 has read it, and `res` only after the next call's first
// barrier, by which every warp has read it; so every call shares one scratch. Returns false when the barrier gave up.
struct ReduceScratch {
  double red[3][32];  // per-warp sums (at most three values, 32 warps)
  double res[3];
  int ok;
};

__device__ __forceinline__ ReduceScratch& reduceScratch() {
  __shared__ ReduceScratch r;
  return r;
}

// The grid stage: the caller has put nw per-warp sums in red and passed a block barrier.
template <int K, bool Max>
__device__ inline bool gridCombine(const Dev& D, GridSync& gs, int nw, double (&out)[K]) {
  static_assert(K >= 1 && K <= 3, "gridReduce: one to three values");
  constexpr int kLoads = 5;  // partials a lane loads at a time (160 blocks per round: one round for one block per SM)
  constexpr double kIdentity = Max ? -INFINITY : 0.0;
  ReduceScratch& sc = reduceScratch();
  double* half = D.partials + static_cast<size_t>(gs.parity) * gs.size * kPartialStride;
  gs.parity ^= 1u;
  gs.target += gs.size;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w == 0) {
    double s[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      s[k] = lane < nw ? sc.red[k][lane] : kIdentity;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[k] = combine<Max>(s[k], __shfl_down_sync(0xffffffffu, s[k], o));
    }
    int good = 0;
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < K; ++k) half[gs.rank * kPartialStride + k] = s[k];
      good = gs.arriveAndWait();
    }
    good = __shfl_sync(0xffffffffu, good, 0);
    __syncwarp();  // the other lanes' reads below follow lane 0's acquire
    if (good) {
      double t[K];
#pragma unroll
      for (int k = 0; k < K; ++k) t[k] = kIdentity;
      for (unsigned int b0 = 0; b0 < gs.size; b0 += 32 * kLoads) {
        double x[kLoads][K];
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
          const unsigned int b = b0 + 32 * j + lane;
#pragma unroll
          for (int k = 0; k < K; ++k) x[j][k] = b < gs.size ? __ldcg(half + b * kPartialStride + k) : kIdentity;
        }
#pragma unroll
        for (int j = 0; j < kLoads; ++j)
#pragma unroll
          for (int k = 0; k < K; ++k) t[k] = combine<Max>(t[k], x[j][k]);
      }
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t[k] = combine<Max>(t[k], __shfl_down_sync(0xffffffffu, t[k], o));
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) sc.res[k] = t[k];
    }
    if (lane == 0) sc.ok = good;
  }
  __syncthreads();
  if (!sc.ok) return false;
#pragma unroll
  for (int k = 0; k < K; ++k) out[k] = sc.res[k];
  return true;
}

template <int K, bool Max = false>
__device__ inline bool gridReduce(const Dev& D, GridSync& gs, double (&v)[K], double (&out)[K]) {
  ReduceScratch& sc = reduceScratch();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] = combine<Max>(v[k], __shfl_down_sync(0xffffffffu, v[k], o));
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) sc.red[k][w] = v[k];
  __syncthreads();
  return gridCombine<K, Max>(D, gs, nw, out);
}

// Sums for a block that stands for one twice its size (at most 512 threads for 1024): thread t carries virtual
// threads t (lo) and t + blockDim.x (hi), so warp w's lo sums are virtual warp w's and its hi sums virtual warp
// w + nw's, in the order a block of the virtual size adds them.
template <int K>
__device__ inline bool gridReducePairs(const Dev& D, GridSync& gs, double (&lo)[K], double (&hi)[K],
                                       double (&out)[K]) {
  ReduceScratch& sc = reduceScratch();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] += __shfl_down_sync(0xffffffffu, lo[k], o);
      hi[k] += __shfl_down_sync(0xffffffffu, hi[k], o);
    }
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      sc.red[k][w] = lo[k];
      sc.red[k][w + nw] = hi[k];
    }
  __syncthreads();
  return gridCombine<K, false>(D, gs, 2 * nw, out);
}

// Block `rank`'s contiguous share of [0, n) in a group of `size` blocks: the persistent kernels give each block one
// range of rows, so the neighbour gathers of the SpMV mostly hit rows the same block (hence the same SM's L1) just
// touched.
__device__ __forceinline__ void blockRange(uint32_t n, uint32_t rank, uint32_t size, uint32_t& r0, uint32_t& r1) {
  const uint32_t per = (n + size - 1) / size;
  r0 = min(n, rank * per);
  r1 = min(n, r0 + per);
}

__device__ __forceinline__ float3 filterContact(const Contact& c, float3 v) {
  if (c.active == 0u) return v;
  const float3 n = xyz(c.normal);
  return v - n * dot(n, v);
}

// The PCG's FP32 arithmetic with every rounding written out (products and sums fused or rounded explicitly, nothing
// left to the compiler's contraction), so that the reference-order kernels (pcgReferenceOrder over 1024-thread blocks,
// pcgResident, pcgCluster and pcgResidentMulti over 512-thread ones) round alike in whatever code surrounds them.
__device__ __forceinline__ float3 axpyRn(float3 x, float s, float3 y) {  // y + s x, one rounding per component
  return mk(__fmaf_rn(x.x, s, y.x), __fmaf_rn(x.y, s, y.y), __fmaf_rn(x.z, s, y.z));
}
__device__ __forceinline__ float dotRn(float a0, float a1, float a2, float3 b) {
  return __fmaf_rn(a2, b.z, __fmaf_rn(a1, b.y, __fmul_rn(a0, b.x)));
}
// The same three products with the first two's sum fused into the first.
__device__ __forceinline__ float dotYRn(float a0, float a1, float a2, float3 b) {
  return __fmaf_rn(a2, b.z, __fmaf_rn(a0, b.x, __fmul_rn(a1, b.y)));
}
__device__ __forceinline__ float3 mulRn(const M3& a, float3 v) {
  return mk(dotRn(a.m[0], a.m[1], a.m[2], v), dotRn(a.m[3], a.m[4], a.m[5], v), dotRn(a.m[6], a.m[7], a.m[8], v));
}
// v - n (n . v) on active contact rows.
__device__ __forceinline__ float3 filterRn(const Contact& c, float3 v) {
  if (c.active == 0u) return v;
  const float3 n = xyz(c.normal);
  return axpyRn(n, -dotRn(n.x, n.y, n.z, v), v);
}
// acc += a v for a row-major 3x3 block a: each row's three products summed in order, then added to acc.
__device__ __forceinline__ void blockMulAddRn(float3& acc, const float (&a)[9], float3 v) {
  acc.x = __fadd_rn(acc.x, dotRn(a[0], a[1], a[2], v));
  acc.y = __fadd_rn(acc.y, dotRn(a[3], a[4], a[5], v));
  acc.z = __fadd_rn(acc.z, dotRn(a[6], a[7], a[8], v));
}

__device__ __forceinline__ float contactRadius(const Params& P, const Fabric& f) {
  return __fadd_rn(P.collisionOffset, __fmul_rn(0.5f, f.thickness));
}

__device__ __forceinline__ float3 ld3(const float4* p, uint32_t i) { return xyz(p[i]); }

__device__ __forceinline__ float seamTarget(const Dev& D, const Seam& s) {
  const Garment g = D.garment[s.garment];
  if (g.phase != 0) return 0.0f;
  return fmaxf(0.0f, s.startGap - D.P.closingSpeed * static_cast<float>(g.assemblyTime));
}

// ---------------------------------------------------------------------------------------------------------------
// Substep setup: predict (kernels.h:34-51) and contact setup (kernels.h:55-82).

__device__ inline void contactSetupOne(const Dev& D, uint32_t i, float3 xs, Contact& c) {
  const float lastForce = c.force;
  c.nearBody = 0u;
  c.active = 0u;
  c.frictionLambda = 0.0f;
  c.force = 0.0f;
  const Particle pa = D.particle[i];
  if (D.field.present && pa.pinned == 0u) {
    const float radius = contactRadius(D.P, D.fabric[pa.fabric]);
    const float phi = fieldSample(D.fieldValues, D.field, xs);
    if (phi < __fadd_rn(radius, D.P.contactReach)) {
      const float3 normal = fieldGradient(D.fieldValues, D.field, xs);
      if (!isZero(normal)) {
        c.nearBody = 1u;
        c.normal = f4(normal, __fsub_rn(radius, phi));
        c.frictionLambda = lastForce;
      }
    }
  }
}

// The point kernels' bodies take the block's rank in the blocks that cover the solver (the grid, or a garment's
// share of a batched launch) and that share's size.
__device__ inline void beginRows(const Dev& D, uint32_t rank, uint32_t size) {
  if (rank == 0 && threadIdx.x == 0) {
    D.ctl->newtonDone = 0;
    D.ctl->substeps += 1;
  }
  const float h = D.P.h;
  for (uint32_t i = rank * blockDim.x + threadIdx.x; i < D.P.n; i += size * blockDim.x) {
    const float4 x4 = D.x[i];
    D.xStart[i] = x4;
    const Particle pa = D.particle[i];
    if (pa.pinned != 0u) {
      D.yRel[i] = make_float4(0, 0, 0, 0);
      D.u[i] = make_float4(0, 0, 0, 0);
    } else {
      const float3 vel = ld3(D.v, i);
      const float3 g = D.garment[pa.garment].phase == 1 ? mk(D.P.gravity[0], D.P.gravity[1], D.P.gravity[2]) : mk(0, 0, 0);
      const float3 acc = g + div(ld3(D.fExt, i), pa.mass);
      D.yRel[i] = f4(vel * h + acc * (h * h));
      D.u[i] = f4(vel * h);
    }
    Contact c = D.contact[i];
    contactSetupOne(D, i, xyz(x4), c);
    D.contact[i] = c;
  }
}

// Holds near particles on their plane for this Newton iteration, projecting any below it (kernels.h:85-99).
__device__ inline void activateRows(const Dev& D, uint32_t rank, uint32_t size) {
  if (D.ctl->newtonDone) return;
  for (uint32_t i = rank * blockDim.x + threadIdx.x; i < D.P.n; i += size * blockDim.x) {
    Contact c = D.contact[i];
    if (c.nearBody == 0u) continue;
    const float3 n = xyz(c.normal);
    float3 ui = ld3(D.u, i);
    const float gap = c.normal.w - dot(n, ui);
    if (gap > -D.P.contactSnap) c.active = 1u;
    if (c.active != 0u && gap > 0.0f) {
      ui += n * gap;
      D.u[i] = f4(ui);
    }
    D.contact[i].active = c.active;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Assembly in two passes. termsRows evaluates every stretch and hinge term once into a derivative record;
// assembleSlots then gives every block slot (i, j) one thread, which adds block (a, b) of each incident term that
// couples i (its vertex a) with j (its vertex b), formed from the term's record, in row i's incidence order (the
// reference's fixed gather order, gpu_solver_core.cpp:184-224). The diagonal slot walks row i's whole incidence list
// (every entry's block (a, a)) after the particle's own inertia and friction term and also sums the row's gradient;
// an off-diagonal slot walks its own contribution list (the reference's per-slot gather list). Deterministic, no
// atomics, no shared memory.

__device__ inline float3 relPos(const Dev& D, uint32_t v0, uint32_t vk) {
  return (ld3(D.xStart, vk) - ld3(D.xStart, v0)) + ld3(D.u, vk);
}

__device__ inline StretchIn stretchIn(const Dev& D, const Stretch& t) {
  const Fabric f = D.fabric[t.fabric];
  StretchIn s;
  s.d = t.d;
  s.area = t.area;
  s.k[0] = f.k[0];
  s.k[1] = f.k[1];
  s.k[2] = f.k[2];
  s.limit[0] = f.limit[0];
  s.limit[1] = f.limit[1];
  s.limitScale = D.P.limitScale;
  return s;
}

// Per-term derivative records of one Newton iteration (every stretch and hinge term evaluated once, one thread per
// term); the assembly then forms each incident row from them.
__device__ inline void termsRows(const Dev& D, uint32_t rank, uint32_t size) {
  if (D.ctl->newtonDone) return;
  const uint32_t S = D.P.nStretch, total = S + D.P.nHinge;
  for (uint32_t idx = rank * blockDim.x + threadIdx.x; idx < total; idx += size * blockDim.x) {
    if (idx < S) {
      const Stretch t = D.stretch[idx];
      float3 x[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) x[k] = relPos(D, t.v[0], t.v[k]);
      StretchDer o;
      stretchDerivs(stretchIn(D, t), x, o);
#pragma unroll
      for (int k = 0; k < 6; ++k) D.stretchDer[6ull * idx + k] = o.w[k];
    } else {
      const uint32_t h = idx - S;
      const Hinge t = D.hinge[h];
      float3 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = relPos(D, t.v[0], t.v[k]);
      HingeDer o;
      hingeDerivs(t.K, t.rest, x, o);
#pragma unroll
      for (int k = 0; k < 4; ++k) D.hingeDer[4ull * h + k] = o.w[k];
    }
  }
}

// Block (a, b) of the term an incidence entry names, and with Grad the gradient of its vertex a (seam springs, a few
// hundred per garment, are evaluated here; stretch and hinge terms come from their records).
template <bool Grad>
__device__ inline void entryBlock(const Dev& D, uint32_t code, int b, float3& g, M3& H) {
  const uint32_t kind = code >> 30, term = (code >> 2) & 0x0FFFFFFFu;
  const int a = static_cast<int>(code & 3u);
  if (kind == 0) {
    stretchBlockFrom<Grad>(D.stretch[term].d, D.stretchDer + 6ull * term, a, b, g, H);
  } else if (kind == 1) {
    hingeBlockFrom<Grad>(D.hingeDer + 4ull * term, a, b, g, H);
  } else {
    const Seam sp = D.seam[term];
    M3 H2[2];
    seamRow(D.P.seamStiffness, seamTarget(D, sp), ld3(D.u, sp.a), relPos(D, sp.a, sp.b), a, g, H2);
    H = b == 0 ? H2[0] : H2[1];
  }
}

// Diagonal slot of row i: the particle's own inertia and friction term, then block (a, a) of every incident entry
// (vertex a of an entry is i itself); also the row's gradient, the block-Jacobi inverse and the contact release.
__device__ inline void diagonalSlot(const Dev& D, uint32_t i, uint32_t SP) {
  const uint32_t s = D.diagSlot[i];
  const Particle pa = D.particle[i];
  const Contact c = D.contact[i];
  M3 acc;
  zero(acc);
  float3 gAcc = mk(0, 0, 0);
  // The particle's own term: inertia 1/2 (m/h^2)|u - yRel|^2 and friction (kernels.h:104-129).
  if (pa.pinned == 0u) {
    const float k = pa.mass * D.P.invH2;
    gAcc = (ld3(D.u, i) - ld3(D.yRel, i)) * k;
    acc.m[0] = acc.m[4] = acc.m[8] = k;
  }
  if (c.frictionLambda > 0.0f)
    frictionRow(ld3(D.u, i), xyz(c.normal), D.fabric[pa.fabric].friction * c.frictionLambda,
                D.P.frictionSlip * D.P.h, gAcc, acc);
  const uint32_t ee = D.incStart[i + 1];
  for (uint32_t e = D.incStart[i]; e < ee; ++e) {
    const uint32_t code = D.incEntry[e];
    float3 g;
    M3 H;
    entryBlock<true>(D, code, static_cast<int>(code & 3u), g, H);
#pragma unroll
    for (int k = 0; k < 9; ++k) acc.m[k] += H.m[k];
    gAcc += g;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) D.blocks[k * SP + s] = acc.m[k];
  // Block-Jacobi inverse of the diagonal block (kernels.h:237-249); zero for pinned particles.
  M3 inv;
  if (pa.pinned != 0u) {
    zero(inv);
  } else {
    bool ok = false;
    inv = invertSpd(acc, ok);
  }
  D.precond[3 * i + 0] = make_float4(inv.m[0], inv.m[1], inv.m[2], 0.0f);
  D.precond[3 * i + 1] = make_float4(inv.m[3], inv.m[4], inv.m[5], 0.0f);
  D.precond[3 * i + 2] = make_float4(inv.m[6], inv.m[7], inv.m[8], 0.0f);
  // Gradient (pinned rows zero) and contact release (kernels.h:204-231).
  const float3 gi = pa.pinned != 0u ? mk(0, 0, 0) : gAcc;
  D.grad[i] = f4(gi);
  if (c.active != 0u && dot(gi, xyz(c.normal)) < 0.0f) D.contact[i].active = 0u;
}

// Off-diagonal slot k (offSlot[k] = row << 6 | row-local position): its contributions (incidence entry, block b of
// the entry's term) in gather order.
__device__ inline void offDiagonalSlot(const Dev& D, uint32_t k, uint32_t SP) {
  const uint32_t packed = D.offSlot[k];
  const uint32_t s = D.rowStart[packed >> 6] + (packed & 63u);
  M3 acc;
  zero(acc);
  const uint32_t ce = D.offStart[k + 1];
  for (uint32_t c = D.offStart[k]; c < ce; ++c) {
    const uint32_t v = D.offCode[c];
    float3 g;
    M3 H;
    // The incidence-entry code (kind 2 bits, term 28, vertex 2) and the block.
    entryBlock<false>(D, (v & 0xC0000000u) | (((v >> 4) & 0x03FFFFFFu) << 2) | ((v >> 2) & 3u), static_cast<int>(v & 3u),
                      g, H);
#pragma unroll
    for (int q = 0; q < 9; ++q) acc.m[q] += H.m[q];
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) D.blocks[q * SP + s] = acc.m[q];
}

// Thread k of the n + (B - n) assembly threads: the diagonal slot of row k for k < n, else off-diagonal slot k - n, so
// that the diagonal slots (every incident entry) and the off-diagonal ones (a few entries each) fill separate warps.
__device__ inline void assembleSlots(const Dev& D, uint32_t rank, uint32_t size) {
  if (D.ctl->newtonDone) return;
  const uint32_t n = D.P.n, SP = D.P.slotsPadded;
  for (uint32_t k = rank * blockDim.x + threadIdx.x; k < D.P.nBlocks; k += size * blockDim.x) {
    if (k < n)
      diagonalSlot(D, k, SP);
    else
      offDiagonalSlot(D, k - n, SP);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Energy at u + alpha * step, in FP64, summed per thread over particles (inertia + friction) and terms. At alpha = 0 the
// step is not read (u stands for it, so that both take the same code): the solve's other blocks may not have written theirs
// yet, and what an abandoned solve left there need not be finite.

// Virtual thread vt of a block of vdim threads: the elements idx = rank * vdim + vt + k * size * vdim (a kernel whose
// blocks stand for larger ones sums in the larger blocks' order).
__device__ inline double energyPartial(const Dev& D, const GridSync& gs, double alpha, uint32_t vt, uint32_t vdim) {
  double e = 0.0;
  const uint32_t n = D.P.n, S = D.P.nStretch, H = D.P.nHinge, K = D.P.nSeam;
  const uint32_t total = n + S + H + K;
  const uint32_t stride = gs.size * vdim;
  const float4* step = alpha == 0.0 ? D.u : D.step;
  auto pos = [&](uint32_t v0, uint32_t vk) -> d3 {
    const d3 rel = toD(ld3(D.xStart, vk)) - toD(ld3(D.xStart, v0));
    return rel + (toD(ld3(D.u, vk)) + alpha * toD(ld3(step, vk)));
  };
  const double invH2 = 1.0 / (D.P.hD * D.P.hD);
  for (uint32_t idx = gs.rank * vdim + vt; idx < total; idx += stride) {
    if (idx < n) {
      const uint32_t i = idx;
      const Particle pa = D.particle[i];
      const d3 ui = toD(ld3(D.u, i)) + alpha * toD(ld3(step, i));
      if (pa.pinned == 0u) {
        const d3 dd = ui - toD(ld3(D.yRel, i));
        e += 0.5 * static_cast<double>(pa.mass) * invH2 * dotd(dd, dd);
      }
      const Contact c = D.contact[i];
      if (c.frictionLambda > 0.0f)
        e += frictionEnergy(ui, toD(xyz(c.normal)),
                            static_cast<double>(D.fabric[pa.fabric].friction) * static_cast<double>(c.frictionLambda),
                            static_cast<double>(D.P.frictionSlip) * D.P.hD);
    } else if (idx < n + S) {
      const Stretch t = D.stretch[idx - n];
      d3 x[3];
      for (int k = 0; k < 3; ++k) x[k] = pos(t.v[0], t.v[k]);
      e += stretchEnergy(stretchIn(D, t), x);
    } else if (idx < n + S + H) {
      const Hinge t = D.hinge[idx - n - S];
      d3 x[4];
      for (int k = 0; k < 4; ++k) x[k] = pos(t.v[0], t.v[k]);
      e += hingeEnergy(t.K, t.rest, x);
    } else {
      const Seam s = D.seam[idx - n - S - H];
      e += seamEnergy(D.P.seamStiffness, seamTarget(D, s), pos(s.a, s.a), pos(s.a, s.b));
    }
  }
  return e;
}

__device__ inline double energyPartial(const Dev& D, const GridSync& gs, double alpha) {
  return energyPartial(D, gs, alpha, threadIdx.x, blockDim.x);
}

// ---------------------------------------------------------------------------------------------------------------
// Persistent solve: PCG with FP64 dot products, then the Newton line search. Every block computes the same scalars
// from the same partials, so all blocks take the same branches.
//
// Each block owns a contiguous range of rows; at the start of the launch it copies its rows' blocks and column
// indices into shared memory (up to P.smemSlots slots; any excess is read from global memory), and every CG
// iteration's SpMV reads them from there.
//
// The PCG follows the reference's order (cpu_solver.cpp:169-213): two grid reductions per iteration (p.Ap, then
// r.r with r.z); the direction update p = z + beta p is folded into the next SpMV (A p = A z + beta A pPrev).

__device__ __forceinline__ M3 loadPrecond(const Dev& D, uint32_t i) {
  const float4 a = D.precond[3 * i], b = D.precond[3 * i + 1], c = D.precond[3 * i + 2];
  return M3{{a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z}};
}

__device__ __forceinline__ double dotd3(float3 a, float3 b) {
  return static_cast<double>(a.x) * b.x + static_cast<double>(a.y) * b.y + static_cast<double>(a.z) * b.z;
}

struct SmemMatrix {
  const float* planes;  // 9 planes of `stride` floats in shared memory
  const uint32_t* cols;
  uint32_t base, cap, stride, SP;  // slots [base, base + cap) are in shared memory
  const float* gblocks;
  const uint32_t* gcols;
  __device__ __forceinline__ bool local(uint32_t s) const { return s - base < cap; }
  __device__ __forceinline__ uint32_t col(uint32_t s) const {
    return local(s) ? cols[s - base] : __ldg(gcols + s);
  }
  // Row-major block at slot s.
  __device__ __forceinline__ void block(uint32_t s, float a[9]) const {
    if (local(s)) {
      const float* p = planes + (s - base);
#pragma unroll
      for (int k = 0; k < 9; ++k) a[k] = p[k * stride];
    } else {
#pragma unroll
      for (int k = 0; k < 9; ++k) a[k] = __ldg(gblocks + k * SP + s);
    }
  }
};

extern __shared__ float4 solveSmem[];

// Copies this block's slot range into shared memory (all threads; ends with a block barrier).
__device__ inline SmemMatrix stageMatrix(const Dev& D, uint32_t r0, uint32_t r1) {
  SmemMatrix A;
  const uint32_t cap = D.P.smemSlots;
  float* planes = reinterpret_cast<float*>(solveSmem);
  uint32_t* cols = reinterpret_cast<uint32_t*>(planes + 9 * cap);
  A.planes = planes;
  A.cols = cols;
  A.SP = D.P.slotsPadded;
  A.gblocks = D.blocks;
  A.gcols = D.colIndex;
  A.base = r0 < r1 ? __ldg(D.rowStart + r0) : 0;
  const uint32_t end = r0 < r1 ? __ldg(D.rowStart + r1) : 0;
  const uint32_t count = min(end - A.base, cap);
  A.stride = cap;
  A.cap = count;
  for (uint32_t k = threadIdx.x; k < count; k += blockDim.x) {
    const uint32_t s = A.base + k;
#pragma unroll
    for (int c = 0; c < 9; ++c) planes[c * cap + k] = __ldg(D.blocks + c * A.SP + s);
    cols[k] = __ldg(D.colIndex + s);
  }
  __syncthreads();
  return A;
}

// y_i (unfiltered) = sum over unpinned columns j of A_ij x_j for row i, by RL lanes (lane `sub`), reduced over the
// lanes; x_j given by a functor. Each lane takes its slots kGatherDepth at a time: their column indices first, then
// all their x_j loads (predicated, so they are in flight together), then the products in slot order; the sums are the
// same as one slot at a time.
constexpr int kGatherDepth = 4;

template <int RL, class X>
__device__ __forceinline__ float3 rowProduct(const SmemMatrix& A, uint32_t rs, uint32_t re, int sub, unsigned mask,
                                             X&& xj) {
  float3 acc = mk(0, 0, 0);
  for (uint32_t s0 = rs + sub; s0 < re; s0 += kGatherDepth * RL) {
    uint32_t col[kGatherDepth];
#pragma unroll
    for (int k = 0; k < kGatherDepth; ++k) {
      const uint32_t s = s0 + k * RL;
      col[k] = s < re ? A.col(s) : kPinnedBit;
    }
    float3 v[kGatherDepth];
#pragma unroll
    for (int k = 0; k < kGatherDepth; ++k) v[k] = (col[k] & kPinnedBit) ? mk(0, 0, 0) : xj(col[k]);
#pragma unroll
    for (int k = 0; k < kGatherDepth; ++k) {
      if (col[k] & kPinnedBit) continue;
      float a[9];
      A.block(s0 + k * RL, a);
      blockMulAddRn(acc, a, v[k]);
    }
  }
#pragma unroll
  for (int o = RL / 2; o > 0; o >>= 1) {
    acc.x = __fadd_rn(acc.x, __shfl_xor_sync(mask, acc.x, o));
    acc.y = __fadd_rn(acc.y, __shfl_xor_sync(mask, acc.y, o));
    acc.z = __fadd_rn(acc.z, __shfl_xor_sync(mask, acc.z, o));
  }
  return acc;
}

// The PCG's product Ap for the direction p = z + beta * pPrev (p = z on the first iteration) over this block's rows
// [r0, r1). The row's product is handed to `out(i, p_i, Ap_i)` (pinned rows: Ap_i = 0; pinned columns add nothing).
// Two schemes, chosen at compile time:
//   RL > 0  RL lanes per row, the lanes' partial sums reduced by shuffles (the matrix mostly in shared memory or L2:
//           no block barriers);
//   RL = 0  slot-parallel (an HBM-resident matrix): the rows are taken kSpmvRows at a time and their slots in passes
//           of kSpmvChunk, each thread computing the products A_s p_j of consecutive slots (coalesced loads of the
//           block planes and column indices); the products are staged in shared memory and the row's thread adds
//           them in slot order.
constexpr uint32_t kSpmvRows = 128;    // slot-parallel: rows per pass (the block needs more threads than this)
constexpr uint32_t kSpmvChunk = 1024;  // slot-parallel: slot products staged per pass

struct SpmvStage {
  uint32_t rowOff[kSpmvRows + 1];
  float prod[3][kSpmvChunk];
};

// The one staging area of a block (every instantiation of directionProducts shares it; its uses never overlap).
__device__ __forceinline__ SpmvStage& spmvStage() {
  __shared__ SpmvStage st;
  return st;
}

template <int RL, class Dir, class Out>
__device__ inline void directionProducts(const Dev& D, const SmemMatrix& A, uint32_t r0, uint32_t r1, Dir&& dir,
                                         Out&& out) {
  if constexpr (RL > 0) {
    const uint32_t groups = blockDim.x / RL;
    const int sub = threadIdx.x & (RL - 1);
    const unsigned groupMask = ((1u << RL) - 1u) << ((threadIdx.x & 31) & ~(RL - 1));
    for (uint32_t i = r0 + threadIdx.x / RL; i < r1; i += groups) {
      const uint32_t rs = __ldg(D.rowStart + i), re = D.particle[i].pinned == 0u ? __ldg(D.rowStart + i + 1) : rs;
      const float3 acc = rowProduct<RL>(A, rs, re, sub, groupMask, dir);
      if (sub == 0) out(i, dir(i), acc);
    }
  } else {
    SpmvStage& st = spmvStage();
    const uint32_t t = threadIdx.x;
    for (uint32_t rr = r0; rr < r1; rr += kSpmvRows) {
      const uint32_t R = min(kSpmvRows, r1 - rr);
      const uint32_t s0 = __ldg(D.rowStart + rr);
      if (t <= R) st.rowOff[t] = __ldg(D.rowStart + rr + t) - s0;
      __syncthreads();
      const uint32_t S = st.rowOff[R];
      float3 acc = mk(0, 0, 0);
      for (uint32_t c = 0; c < S; c += kSpmvChunk) {
        const uint32_t cn = min(kSpmvChunk, S - c);
        for (uint32_t k = t; k < cn; k += blockDim.x) {
          const uint32_t s = s0 + c + k;
          const uint32_t col = A.col(s);
          float3 v = mk(0, 0, 0);
          if (!(col & kPinnedBit)) {
            float a[9];
            A.block(s, a);
            const float3 x = dir(col);
            v.x = a[0] * x.x + a[1] * x.y + a[2] * x.z;
            v.y = a[3] * x.x + a[4] * x.y + a[5] * x.z;
            v.z = a[6] * x.x + a[7] * x.y + a[8] * x.z;
          }
          st.prod[0][k] = v.x;
          st.prod[1][k] = v.y;
          st.prod[2][k] = v.z;
        }
        __syncthreads();
        if (t < R) {
          const uint32_t lo = max(st.rowOff[t], c), hi = min(st.rowOff[t + 1], c + cn);
          for (uint32_t q = lo; q < hi; ++q) {
            acc.x += st.prod[0][q - c];
            acc.y += st.prod[1][q - c];
            acc.z += st.prod[2][q - c];
          }
        }
        __syncthreads();
      }
      if (t < R) {
        const uint32_t i = rr + t;
        out(i, dir(i), D.particle[i].pinned != 0u ? mk(0, 0, 0) : acc);
      }
      __syncthreads();  // rowOff is rewritten for the next rows
    }
  }
}

// One PCG iteration's product for the direction p = z + beta * pPrev without materialising p first: the rows gather
// only z_j and add beta times their previous product A pPrev (apFull). Writes p_i (pCur), Ap_i (apFull) and the
// contact-filtered Ap_i (ap); returns this thread's share of p . filtered Ap.
template <int RL>
__device__ inline double directionStep(const Dev& D, const SmemMatrix& A, uint32_t r0, uint32_t r1,
                                       const float4* pPrev, float4* pCur, float fb, bool first) {
  double vpap = 0.0;
  directionProducts<RL>(
      D, A, r0, r1, [&](uint32_t j) { return ld3(D.z, j); },
      [&](uint32_t i, float3 zi, float3 az) {
        // A p = A z + beta A pPrev: the previous direction's product is this row's apFull.
        const float3 pi = first ? zi : axpyRn(ld3(pPrev, i), fb, zi);
        const float3 acc = first ? az : axpyRn(ld3(D.apFull, i), fb, az);
        pCur[i] = f4(pi);
        const float3 filtered = filterRn(D.contact[i], acc);
        D.apFull[i] = f4(acc);
        D.ap[i] = f4(filtered);
        vpap += dotd3(pi, filtered);
      });
  return vpap;
}

// Contact-filtered block-Jacobi PCG in the reference's order. Writes step, resid; returns the iteration count, or -1
// when a grid barrier gave up.
// At most `budget` iterations (negative: P.maxCg). *r0out gets |r0|; *finished is false only when the budget, not
// the convergence test or pAp <= 0, ended the loop.
template <int PL>
__device__ inline int pcgReferenceOrder(const Dev& D, GridSync& gs, const SmemMatrix& A, int budget = -1,
                                        double* r0out = nullptr, bool* finished = nullptr) {
  const uint32_t n = D.P.n;
  uint32_t r0i, r1i;
  blockRange(n, gs.rank, gs.size, r0i, r1i);
  // CG init (kernels.h:252-268): step = 0, resid = -grad, r = filter(resid), z = filter(M r).
  double tot[2];
  {
    double v[2] = {0.0, 0.0};
    for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
      const Contact c = D.contact[i];
      const float3 res = -ld3(D.grad, i);
      const float3 ri = filterRn(c, res);
      const float3 zi = filterRn(c, mulRn(loadPrecond(D, i), ri));
      D.step[i] = make_float4(0, 0, 0, 0);
      D.resid[i] = f4(res);
      D.r[i] = f4(ri);
      D.z[i] = f4(zi);
      v[0] += dotd3(ri, zi);
      v[1] += dotd3(ri, ri);
    }
    if (!gridReduce<2>(D, gs, v, tot)) return -1;
  }
  double rz = tot[0];
  const double r0 = sqrt(tot[1]);
  if (r0out) *r0out = r0;
  bool done = !(r0 > 0.0);
  double beta = 0.0;
  float4* pPrev = D.p0;
  float4* pCur = D.p1;
  int it = 0;
  const int maxCg = budget < 0 ? D.P.maxCg : min(budget, D.P.maxCg);
  if (finished) *finished = true;
  while (!done && it < maxCg) {
    // SpMV with the direction update folded in: p_j = z_j + beta * pPrev_j.
    double vpap[1] = {directionStep<PL>(D, A, r0i, r1i, pPrev, pCur, static_cast<float>(beta), it == 0)};
    double pAp[1];
    if (!gridReduce<1>(D, gs, vpap, pAp)) return -1;
    if (!(pAp[0] > 0.0)) return it;
    const double alpha = rz / pAp[0];
    const float fa = static_cast<float>(alpha);
    ++it;
    // Update (kernels.h:304-315) fused with the preconditioner apply (kernels.h:324-332).
    double v[2] = {0.0, 0.0};
    for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
      const Contact c = D.contact[i];
      const float3 pi = ld3(pCur, i);
      D.step[i] = f4(axpyRn(pi, fa, ld3(D.step, i)));
      const float3 ri = axpyRn(ld3(D.ap, i), -fa, ld3(D.r, i));
      D.r[i] = f4(ri);
      D.resid[i] = f4(axpyRn(ld3(D.apFull, i), -fa, ld3(D.resid, i)));
      const float3 zi = filterRn(c, mulRn(loadPrecond(D, i), ri));
      D.z[i] = f4(zi);
      v[0] += dotd3(ri, ri);
      v[1] += dotd3(ri, zi);
    }
    double t2[2];
    if (!gridReduce<2>(D, gs, v, t2)) return -1;
    if (sqrt(t2[0]) <= D.P.cgTolerance * r0) return it;
    beta = t2[1] / rz;
    rz = t2[1];
    float4* tmp = pPrev;
    pPrev = pCur;
    pCur = tmp;
  }
  if (finished && !done) *finished = false;
  return it;
}

// ---------------------------------------------------------------------------------------------------------------
// Reference-order PCG with resident rows (k_solve_rows; the form pcgVariant 0 runs where a scene fits it). One thread
// owns one row of its block for the whole solve and keeps the row's PCG state (p, A p and its filtered copy, r, step,
// resid, z, the contact plane and the preconditioner block) and its first kRegSlots matrix blocks in registers; the
// other blocks sit in shared memory in a sliced layout (the rows in warps of 32, warp w's rows padded to its longest,
// slot k of lane l at base_w + 32 k + l), beside the z of every particle the block's rows couple to (its own rows, then
// its halo: the other blocks' particles, listed once per build by k_localize, which also gives every slot the index of
// its column among them). The row's product keeps the two-lane order of pcgReferenceOrder<2> (the even slots in one
// sum, the odd slots in another, added at the end), so the iterates are that kernel's.
//
// The blocks exchange by messages (exchange.cuh). The new z carries the iteration's tag in its fourth component, so a
// block takes its halo as soon as it is there, with no barrier; and since A p = A z + beta A pPrev, the sums r.r and r.z
// that give beta travel while the rows form A z. Only the sum p.Ap, which gives alpha, is waited for. One warp of the
// block does the sums, the scalars and the stopping tests; the others hold the rows.
//
// Measured (us per PCG iteration, one B200; with a counter barrier for each sum, z gathered from the L2 and the matrix
// read four bytes at a time before): 1,600 particles 2.9 (was 6.9), 10k 3.0 (7.2), 60k 4.3 (8.4). What bounds it now: for
// small scenes the two exchanges one after the other (about 1.1 us each with their block sums) and the FP64 division
// and square root between them; at 60k the way of z to the neighbours (about 0.8 us), then the product (38 bytes of
// shared memory a slot and 16 a gathered z, against 128 bytes a clock: 1.3 us), then one exchange. Fewer blocks than SMs
// for small scenes: 2.7-2.9 us for 8 to 148 blocks at 1,600 particles, slower at 4,000 and 10k. A row's slots four at a
// time with two slots in registers: 4.31 us at 60k; two at a time 4.39, six 4.43; four or six slots in registers spill
// (4.30-4.32).
constexpr int kRowThreads = 512;    // k_solve_rows block size
constexpr int kRowWorkers = 480;    // of these, the threads that own a row each; the last warp does the exchanges
constexpr int kResidentRows = 4;    // the solve templates' Variant value of this form; 4 + m: m rows a thread
constexpr int kRegSlots = 2;        // slots of each row kept in registers (even, so that slot parity is the same)
constexpr int kExchangeDelay = 700; // clock cycles before an exchange's first poll, to begin with
constexpr uint32_t kNoColumn = 0xFFFFu;  // localCol of a pinned column

// Shared memory of one padded slot (nine floats and a 16-bit column) and of one particle's z.
constexpr uint32_t kResidentSlotBytes = 38, kResidentNodeBytes = 16;
// k_solve_rows_learned reads up to this many columns past the last padded slot (factorProduct).
constexpr uint32_t kColumnsRead = 64;

struct ResidentMatrix {
  const float4 *a, *b;     // blocks of the slots in shared memory: components 0-3 and 4-7
  const float* c;          // component 8
  const uint32_t* cols;    // columns of slots 2m and 2m + 1: 16 bits each, at base_w / 2 + 32 m + lane
  float4* z;               // z of the block's rows, then of its halo; the last entry is zero
  uint32_t base, len;      // this thread's warp: its first position and its padded slots (even)
  uint32_t rows, haloSize;
  const uint32_t* halo;    // the halo's particles
  const float4* factor;    // the learned factor's slots (row 0; rows 1 and 2 follow): in shared memory or D.LfSliced
  uint32_t factorBase;     // this thread's warp's first position there
  float reg[kRegSlots][9];
  uint32_t regCols[kRegSlots / 2];
};

// What the exchange warp tells the row warps, and their sums on the way to it.
struct ResidentShared {
  double red[2][kRowWorkers / 32];
  float factor;  // beta, or alpha
  int code;      // 0 go on, 1 stop, 2 an exchange gave up
  int failed;    // a halo wait gave up
  unsigned long long seq;  // the last exchange's number
};

// Copies this block's rows [r0, r1) into registers and the sliced layout (all threads; ends with a block barrier).
// Returns false, after raising error 4, when the block does not fit what the host sized (P.residentSlots,
// P.residentNodes; the host picks k_solve_rows only for scenes whose every block fits, so this is a guard).
// Learned: also a second array for gathered vectors, and the factor by rows in the sliced layout: in shared memory, or
// where it does not fit in the block's part of D.LfSliced (so that a warp's loads of it are contiguous).
template <bool Learned>
__device__ inline bool stageResident(const Dev& D, uint32_t rank, uint32_t r0, uint32_t r1, ResidentMatrix& A) {
  constexpr int kWarps = kRowWorkers / 32;
  // The rows' first slots relative to the block's first, bit 31 set for pinned rows (they take no product).
  __shared__ uint32_t off[kRowWorkers + 1];
  __shared__ uint32_t warpLen[kWarps], warpBase[kWarps + 1];
  const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
  const uint32_t R = r1 - r0;
  A.rows = R;
  A.haloSize = __ldg(D.haloCount + rank);
  A.halo = D.halo + static_cast<size_t>(rank) * D.P.haloStride;
  if (R > static_cast<uint32_t>(kRowWorkers) || blockDim.x != static_cast<unsigned>(kRowThreads) ||
      R + A.haloSize >= D.P.residentNodes) {
    if (t == 0) atomicExch(&D.ctl->error, 4);
    return false;
  }
  const uint32_t first = __ldg(D.rowStart + r0);  // r0 <= n: rowStart has n + 1 entries
  uint32_t count = 0, rs = first;
  if (t < R) {
    rs = __ldg(D.rowStart + r0 + t);
    const bool pinned = D.particle[r0 + t].pinned != 0u;
    off[t] = (rs - first) | (pinned ? kPinnedBit : 0u);
    if (!pinned) count = __ldg(D.rowStart + r0 + t + 1) - rs;
  }
  if (t == 0) off[R] = __ldg(D.rowStart + r1) - first;
  const uint32_t longest = __reduce_max_sync(0xffffffffu, count);
  if (lane == 0 && w < kWarps) warpLen[w] = longest > kRegSlots ? (longest - kRegSlots + 1u) & ~1u : 0u;
  __syncthreads();
  if (t == 0) {
    uint32_t acc = 0;
    for (int k = 0; k < kWarps; ++k) {
      warpBase[k] = acc;
      acc += 32u * warpLen[k];
    }
    warpBase[kWarps] = acc;
  }
  __syncthreads();
  const uint32_t total = warpBase[kWarps], cap = D.P.residentSlots;
  if (total > cap) {
    if (t == 0) atomicExch(&D.ctl->error, 4);
    return false;
  }
  float4* a = solveSmem;
  float4* b = a + cap;
  A.z = b + cap;
  float4* behindZ = A.z + (Learned ? 2 : 1) * D.P.residentNodes;
  const uint32_t factorCap = Learned ? D.P.factorSlots : 0u;
  float4* factor = Learned && D.LfSliced ? D.LfSliced + 3 * static_cast<size_t>(factorCap) * rank : behindZ;
  A.factor = factor;
  A.factorBase = w < kWarps ? warpBase[w] + 32u * kRegSlots * w : 0u;  // every slot has a place here
  if (Learned && total + 32u * kRegSlots * kWarps > factorCap) {
    if (t == 0) atomicExch(&D.ctl->error, 4);
    return false;
  }
  float* c = reinterpret_cast<float*>(Learned && !D.LfSliced ? behindZ + 3 * factorCap : behindZ);
  uint16_t* cols = reinterpret_cast<uint16_t*>(c + cap);
  A.a = a;
  A.b = b;
  A.c = c;
  A.cols = reinterpret_cast<const uint32_t*>(cols);
  A.base = w < kWarps ? warpBase[w] : 0u;
  A.len = w < kWarps ? warpLen[w] : 0u;
  const uint32_t SP = D.P.slotsPadded, zeroNode = D.P.residentNodes - 1;
  if (t < (Learned ? 2u : 1u)) A.z[zeroNode + t * D.P.residentNodes] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  // The row's first slots, and the padding of its lane.
  uint32_t rc[kRegSlots];
#pragma unroll
  for (int k = 0; k < kRegSlots; ++k) {
    const uint32_t col = static_cast<uint32_t>(k) < count ? __ldg(D.localCol + rs + k) : kNoColumn;
    rc[k] = col == kNoColumn ? zeroNode : col;
#pragma unroll
    for (int q = 0; q < 9; ++q) A.reg[k][q] = col == kNoColumn ? 0.0f : __ldg(D.blocks + q * SP + rs + k);
  }
#pragma unroll
  for (int k = 0; k < kRegSlots / 2; ++k) A.regCols[k] = rc[2 * k] | rc[2 * k + 1] << 16;
  // 16-bit column of slot j (of those in shared memory) of the row at lane l of the warp whose slots start at `base`.
  auto colAt = [](uint32_t base, uint32_t j, uint32_t l) { return base + (32u * (j >> 1) + l) * 2u + (j & 1u); };
  for (uint32_t j = count > kRegSlots ? count - kRegSlots : 0u; j < A.len; ++j) {
    const uint32_t pos = A.base + 32u * j + lane;
    a[pos] = b[pos] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    c[pos] = 0.0f;
    cols[colAt(A.base, j, lane)] = static_cast<uint16_t>(zeroNode);
  }
  // The slots, read in slot order (coalesced); each finds its row by bisection over off[].
  const uint32_t S = off[R];
  for (uint32_t k = t; k < S; k += blockDim.x) {
    uint32_t lo = 0, hi = R;  // row lo's first slot <= k < row hi's first slot
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if ((off[mid] & ~kPinnedBit) <= k) lo = mid; else hi = mid;
    }
    if (off[lo] & kPinnedBit) continue;  // a pinned row's slot
    const uint32_t j = k - off[lo];
    if (Learned) {
      const float4* row = D.LfRows + 3 * static_cast<size_t>(first + k);
      float4* f = factor + warpBase[lo >> 5] + 32u * kRegSlots * (lo >> 5) + 32u * j + (lo & 31u);
      f[0] = __ldg(row);
      f[factorCap] = __ldg(row + 1);
      f[2 * factorCap] = __ldg(row + 2);
    }
    if (j < kRegSlots) continue;
    const uint32_t pos = warpBase[lo >> 5] + 32u * (j - kRegSlots) + (lo & 31u);
    const uint32_t s = first + k;
    const uint32_t col = __ldg(D.localCol + s);
    float m[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) m[q] = col == kNoColumn ? 0.0f : __ldg(D.blocks + q * SP + s);
    a[pos] = make_float4(m[0], m[1], m[2], m[3]);
    b[pos] = make_float4(m[4], m[5], m[6], m[7]);
    c[pos] = m[8];
    cols[colAt(warpBase[lo >> 5], j - kRegSlots, lo & 31u)] = static_cast<uint16_t>(col == kNoColumn ? zeroNode : col);
  }
  __syncthreads();
  return true;
}

// U of this thread's slots (U even) from slot k on: all their loads are issued before the first product.
template <int U>
__device__ __forceinline__ void residentSlots(const ResidentMatrix& A, const float4* z, uint32_t k, float3 (&acc)[2]) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t cc[U / 2];
  float4 a[U], b[U], x[U];
  float c[U];
#pragma unroll
  for (int u = 0; u < U / 2; ++u) cc[u] = A.cols[A.base / 2 + 16u * k + 32u * u + lane];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t pos = A.base + 32u * (k + u) + lane;
    a[u] = A.a[pos];
    b[u] = A.b[pos];
    c[u] = A.c[pos];
  }
#pragma unroll
  for (int u = 0; u < U; ++u) x[u] = z[(u & 1) ? cc[u / 2] >> 16 : cc[u / 2] & 0xFFFFu];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const float m[9] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w, c[u]};
    blockMulAddRn(acc[u & 1], m, xyz(x[u]));
  }
}

// y_i (unfiltered) = sum over the row's unpinned columns j of A_ij z_j, for this thread's row, in pcgReferenceOrder<2>'s
// order: slot k of the row into sum k mod 2, each sum in slot order, the odd sum added to the even one last. Pinned
// columns and padding hold zero blocks and name the zero particle: they add +0 to a sum that is never -0.
__device__ __forceinline__ float3 residentProduct(const ResidentMatrix& A, const float4* z) {
  float3 acc[2] = {mk(0, 0, 0), mk(0, 0, 0)};
  {
    float4 x[kRegSlots];
#pragma unroll
    for (int k = 0; k < kRegSlots; ++k) x[k] = z[(k & 1) ? A.regCols[k / 2] >> 16 : A.regCols[k / 2] & 0xFFFFu];
#pragma unroll
    for (int k = 0; k < kRegSlots; ++k) blockMulAddRn(acc[k & 1], A.reg[k], xyz(x[k]));
  }
  uint32_t k = 0;
  for (; k + 4 <= A.len; k += 4) residentSlots<4>(A, z, k, acc);
  if (k < A.len) residentSlots<2>(A, z, k, acc);
  return mk(__fadd_rn(acc[0].x, acc[1].x), __fadd_rn(acc[0].y, acc[1].y), __fadd_rn(acc[0].z, acc[1].z));
}

// The halo's entries of `global` into shared memory (behind the block's own in `z`), each particle's as soon as it carries
// `tag`. Returns false when a wait gave up.
template <class Matrix>
__device__ __forceinline__ bool takeHalo(const Dev& D, const Matrix& A, float4* z, const float4* global,
                                         uint32_t tag) {
  constexpr uint32_t kStep = kRowWorkers;
  bool ok = true;
  BoundedWait wait;
  for (uint32_t h = threadIdx.x; h < A.haloSize && ok; h += 2 * kStep) {
    const bool two = h + kStep < A.haloSize;
    const float4* p0 = global + __ldg(A.halo + h);
    const float4* p1 = global + __ldg(A.halo + (two ? h + kStep : h));
    float3 v0, v1;
    for (;;) {
      const uint32_t t0 = loadTagged(p0, v0), t1 = loadTagged(p1, v1);
      if (t0 == tag && t1 == tag) break;
      if (wait.expired(D.ctl, D.P.barrierLimitNs)) {
        ok = false;
        break;
      }
    }
    z[A.rows + h] = f4(v0);
    if (two) z[A.rows + h + kStep] = f4(v1);
  }
  return ok;
}

// The exchange warp of pcgResident and pcgResidentMulti: every iteration's two sums, the scalars and the stopping tests.
// Returns the iteration count; `code` as in ResidentShared.
__device__ inline int residentExchanges(const Dev& D, const GridSync& gs, ResidentShared& sh, unsigned long long base,
                                        int& code) {
  constexpr int kWarps = kRowWorkers / 32;
  const uint32_t lane = threadIdx.x & 31u;
  const int maxCg = D.P.maxCg;
  int it = 0;
  double rz = 0.0, r0 = 0.0;
  unsigned long long num = base;
  int delayA = kExchangeDelay, delayB = kExchangeDelay;
  while (it < maxCg) {
    namedSync<1>(kRowThreads);
    double part[2], sum[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) part[k] = warpSum(lane < kWarps ? sh.red[k][lane] : 0.0);
    float factor = 0.0f;
    if (!mailSum<2>(D.mail, D.ctl, D.P.barrierLimitNs, gs.rank, gs.size, ++num, part, sum, delayB)) {
      code = 2;
    } else if (it == 0) {
      r0 = sqrt(sum[0]);
      code = r0 > 0.0 ? 0 : 1;
    } else {
      code = sqrt(sum[0]) <= D.P.cgTolerance * r0 ? 1 : 0;
      factor = static_cast<float>(sum[1] / rz);
    }
    rz = sum[1];
    if (lane == 0) {
      sh.code = code;
      sh.factor = factor;
    }
    namedArrive<3>(kRowThreads);
    if (code) break;
    namedSync<1>(kRowThreads);
    double pap[1] = {warpSum(lane < kWarps ? sh.red[0][lane] : 0.0)}, pAp[1];
    if (sh.failed || !mailSum<1>(D.mail, D.ctl, D.P.barrierLimitNs, gs.rank, gs.size, ++num, pap, pAp, delayA))
      code = 2;
    else
      code = pAp[0] > 0.0 ? 0 : 1;
    if (lane == 0) {
      sh.code = code;
      sh.factor = code ? 0.0f : static_cast<float>(rz / pAp[0]);
    }
    namedArrive<3>(kRowThreads);
    if (code) break;
    ++it;
  }
  if (lane == 0) sh.seq = num;
  return it;
}

// The reference-order PCG of pcgReferenceOrder (same recurrences, same stopping tests) over resident rows. Writes
// step and resid of the block's rows; returns the iteration count, or -1 when an exchange gave up. `seq` is the last
// exchange's number, advanced by the exchanges done.
//
// Barriers: 1 hands the row warps' sums to the exchange warp (they only arrive), 3 its scalars to the row warps (it only
// arrives), 2 is the row warps' own, between the z in shared memory and the product. The exchange warp evaluates every
// stopping test, so all warps leave after the same exchange; a row warp whose halo wait gave up says so through `failed`
// and leaves like the others.
__device__ inline int pcgResident(const Dev& D, GridSync& gs, ResidentMatrix& A, unsigned long long& seq) {
  constexpr int kWarps = kRowWorkers / 32;
  __shared__ ResidentShared sh;
  const int maxCg = D.P.maxCg;
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const unsigned long long base = seq;
  if (threadIdx.x == 0) sh.failed = 0;
  __syncthreads();
  int it = 0, code = 0;
  if (w == kWarps) {
    it = residentExchanges(D, gs, sh, base, code);
  } else {
    uint32_t r0i, r1i;
    blockRange(D.P.n, gs.rank, gs.size, r0i, r1i);
    const uint32_t i = r0i + threadIdx.x;
    const bool own = i < r1i, busy = 32u * w < r1i - r0i;  // busy: a row of this warp is owned
    Contact c{};
    M3 M{};
    float3 step = mk(0, 0, 0), resid = mk(0, 0, 0), r = mk(0, 0, 0), z = mk(0, 0, 0);
    float3 p = mk(0, 0, 0), apFull = mk(0, 0, 0), ap = mk(0, 0, 0);
    // CG init (kernels.h:252-268): step = 0, resid = -grad, r = filter(resid), z = filter(M r).
    if (own) {
      c = D.contact[i];
      M = loadPrecond(D, i);
      resid = -ld3(D.grad, i);
      r = filterRn(c, resid);
      z = filterRn(c, mulRn(M, r));
    }
    if (!busy && lane == 0) sh.red[0][w] = sh.red[1][w] = 0.0;
    while (it < maxCg) {
      const uint32_t tag = static_cast<uint32_t>(base + 1 + 2 * static_cast<unsigned long long>(it)) | 0x80000000u;
      if (own) {
        storeTagged(D.z + i, z, tag);
        A.z[threadIdx.x] = f4(z);
      }
      if (busy) {
        const double rr = warpSum(dotd3(r, r)), rz = warpSum(dotd3(r, z));  // zero where no row is owned
        if (lane == 0) {
          sh.red[0][w] = rr;
          sh.red[1][w] = rz;
        }
      }
      namedArrive<1>(kRowThreads);
      if (!takeHalo(D, A, A.z, D.z, tag)) sh.failed = 1;
      namedSync<2>(kRowWorkers);
      const float3 az = busy ? residentProduct(A, A.z) : mk(0, 0, 0);
      namedSync<3>(kRowThreads);
      code = sh.code;
      if (code) break;
      // A p = A z + beta A pPrev, p = z + beta pPrev (the direction update folded into the product).
      const float fb = sh.factor;
      if (busy) {
        p = it == 0 ? z : axpyRn(p, fb, z);
        apFull = it == 0 ? az : axpyRn(apFull, fb, az);
        ap = filterRn(c, apFull);
        const double pap = warpSum(dotd3(p, ap));
        if (lane == 0) sh.red[0][w] = pap;
      }
      namedArrive<1>(kRowThreads);
      namedSync<3>(kRowThreads);
      code = sh.code;
      if (code) break;
      const float fa = sh.factor;
      ++it;
      // Update (kernels.h:304-315) fused with the preconditioner apply (kernels.h:324-332).
      step = axpyRn(p, fa, step);
      r = axpyRn(ap, -fa, r);
      resid = axpyRn(apFull, -fa, resid);
      z = filterRn(c, mulRn(M, r));
    }
    if (own) {
      D.step[i] = f4(step);
      D.resid[i] = f4(resid);
    }
  }
  __syncthreads();
  seq = sh.seq;
  __syncthreads();
  return code == 2 ? -1 : it;
}

// ---------------------------------------------------------------------------------------------------------------
// The same PCG for small scenes in one cluster of kClusterBlocks blocks (k_solve_cluster): pcgResident with its exchanges
// in distributed shared memory. A block's exchange warp writes its sums into every block's shared memory (st.async, which
// completes the bytes on the receiver's mbarrier), and the halo's z is read from its owners' shared memory after a cluster
// barrier. Same rows, products and scalars, so the same iterates.
//
// Why: below a few thousand particles an iteration is two ways through the L2 one after the other, whatever the grid;
// between the SMs of a GPC they are shorter. Measured (us per PCG iteration on one B200,
// k_solve_rows on 148 blocks in brackets): 1,600 particles 2.04 (2.79), 2,600 2.25 (2.8), 4,000 2.59 (2.82), 5,000 3.1
// (2.8); a frame of the 1,600-particle sheet 353 us (421). At 4,000 the passes after the PCG, on 16 SMs instead of 148,
// take what the iterations save, so scenes up to 3,500 particles run it (drape_solver::kClusterParticles).
constexpr int kClusterBlocks = 16;
constexpr int kClusterRows = 8;  // the solve templates' Variant value of this form

__device__ __forceinline__ uint32_t sharedAddress(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// The shared-memory address `local` of block `rank` of the cluster.
__device__ __forceinline__ uint32_t clusterAddress(uint32_t local, uint32_t rank) {
  uint32_t out;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local), "r"(rank));
  return out;
}
__device__ __forceinline__ void clusterArrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void clusterWait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct ClusterMail {
  double value[2][kClusterBlocks][2];  // the two sums of an iteration (r.r and r.z; p.Ap), each block's
  unsigned long long bar[2];
};

// One exchange of K values by the exchange warp; `which` alternates, so a message never meets one not yet read (mailSum's
// argument). `phase` counts this mbarrier's uses.
//
// No block may leave an exchange on its own: its shared memory would go away under messages and halo reads of the others.
// So where the wait's limit runs out, or another block has raised the error flag, `late` is set and the messages are
// awaited all the same (they are on their way: the cluster's blocks run together and each sends before it waits); the next
// exchange of r.r tells every block (kClusterLate), and all leave after it. The second wait has a limit too, in polls, so
// that no pause of the whole GPU can end it. Returns false when it runs out.
constexpr double kClusterLate = -1.0;  // in the place of a block's r.r, which is a sum of squares
constexpr unsigned int kClusterDrainPolls = 1u << 24;

template <int K>
__device__ inline bool clusterSum(const Dev& D, ClusterMail& mail, int which, uint32_t phase, uint32_t rank,
                                  const double (&mine)[K], double (&total)[K], bool& late) {
  const uint32_t lane = threadIdx.x & 31u, bar = sharedAddress(&mail.bar[which]);
  if (lane == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"(static_cast<uint32_t>(kClusterBlocks * 16))
                 : "memory");
  __syncwarp();
  if (lane < static_cast<uint32_t>(kClusterBlocks)) {
    const uint32_t to = clusterAddress(sharedAddress(&mail.value[which][rank][0]), lane);
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(to),
                 "l"(__double_as_longlong(mine[0])), "l"(__double_as_longlong(mine[K - 1])),
                 "r"(clusterAddress(bar, lane))
                 : "memory");
  }
  BoundedWait wait;
  for (unsigned int drain = 0;;) {
    uint32_t done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(bar), "r"(phase & 1u)
        : "memory");
    if (__all_sync(0xffffffffu, done != 0)) break;
    if (late) {
      if (++drain == kClusterDrainPolls) return false;
    } else if (__any_sync(0xffffffffu, wait.expired(D.ctl, D.P.barrierLimitNs))) {
      late = true;
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k)
    total[k] = warpSum(lane < static_cast<uint32_t>(kClusterBlocks) ? mail.value[which][lane][k] : 0.0);
  return true;
}

// As pcgResident, on the blocks of one cluster (gs.size == kClusterBlocks). All threads of the cluster pass the same
// cluster barriers, one in each iteration and one at the end, before which no block leaves its shared memory to others that
// may still read it: every block learns the same sums, so all leave after the same exchange. Returns -1 in a block whose
// wait ran out or that another told so.
__device__ inline int pcgCluster(const Dev& D, GridSync& gs, ResidentMatrix& A, ClusterMail& mail) {
  constexpr int kWarps = kRowWorkers / 32;
  __shared__ ResidentShared sh;
  const int maxCg = D.P.maxCg;
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  int it = 0, code = 0;
  if (w == kWarps) {
    double rz = 0.0, r0 = 0.0;
    uint32_t phase = 0;
    bool late = false;
    while (it < maxCg) {
      clusterArrive();
      namedSync<1>(kRowThreads);
      double part[2], sum[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) part[k] = warpSum(lane < kWarps ? sh.red[k][lane] : 0.0);
      float factor = 0.0f;
      if (late) part[0] = kClusterLate;
      if (!clusterSum<2>(D, mail, 0, phase, gs.rank, part, sum, late) ||
          __any_sync(0xffffffffu, lane < static_cast<uint32_t>(kClusterBlocks) && mail.value[0][lane][0] < 0.0)) {
        code = 2;
      } else if (it == 0) {
        r0 = sqrt(sum[0]);
        code = r0 > 0.0 ? 0 : 1;
      } else {
        code = sqrt(sum[0]) <= D.P.cgTolerance * r0 ? 1 : 0;
        factor = static_cast<float>(sum[1] / rz);
      }
      rz = sum[1];
      if (lane == 0) {
        sh.code = code;
        sh.factor = factor;
      }
      namedArrive<3>(kRowThreads);
      clusterWait();
      if (code) break;
      namedSync<1>(kRowThreads);
      double pap[1] = {warpSum(lane < kWarps ? sh.red[0][lane] : 0.0)}, pAp[1];
      if (!clusterSum<1>(D, mail, 1, phase, gs.rank, pap, pAp, late))
        code = 2;
      else
        code = pAp[0] > 0.0 ? 0 : 1;
      ++phase;
      if (lane == 0) {
        sh.code = code;
        sh.factor = code ? 0.0f : static_cast<float>(rz / pAp[0]);
      }
      namedArrive<3>(kRowThreads);
      if (code) break;
      ++it;
    }
    if (lane == 0) sh.failed = late || code == 2;
  } else {
    uint32_t r0i, r1i;
    blockRange(D.P.n, gs.rank, gs.size, r0i, r1i);
    const uint32_t i = r0i + threadIdx.x, per = (D.P.n + gs.size - 1) / gs.size;
    const bool own = i < r1i, busy = 32u * w < r1i - r0i;  // busy: a row of this warp is owned
    // The halo entries this thread copies each iteration: where they are in the cluster's shared memory.
    constexpr int kMine = 3;
    uint32_t from[kMine];
    const uint32_t zBase = sharedAddress(A.z);
    auto owner = [&](uint32_t h) {
      const uint32_t j = __ldg(A.halo + h);
      return clusterAddress(zBase + 16u * (j % per), j / per);
    };
#pragma unroll
    for (int k = 0; k < kMine; ++k) {
      const uint32_t h = threadIdx.x + k * kRowWorkers;
      from[k] = h < A.haloSize ? owner(h) : 0u;
    }
    auto copyFrom = [&](uint32_t address, uint32_t h) {
      float4 v;
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                   : "r"(address)
                   : "memory");
      A.z[A.rows + h] = v;
    };
    Contact c{};
    M3 M{};
    float3 step = mk(0, 0, 0), resid = mk(0, 0, 0), r = mk(0, 0, 0), z = mk(0, 0, 0);
    float3 p = mk(0, 0, 0), apFull = mk(0, 0, 0), ap = mk(0, 0, 0);
    // CG init (kernels.h:252-268): step = 0, resid = -grad, r = filter(resid), z = filter(M r).
    if (own) {
      c = D.contact[i];
      M = loadPrecond(D, i);
      resid = -ld3(D.grad, i);
      r = filterRn(c, resid);
      z = filterRn(c, mulRn(M, r));
    }
    if (!busy && lane == 0) sh.red[0][w] = sh.red[1][w] = 0.0;
    while (it < maxCg) {
      if (own) A.z[threadIdx.x] = f4(z);
      clusterArrive();
      if (busy) {
        const double rr = warpSum(dotd3(r, r)), rz = warpSum(dotd3(r, z));  // zero where no row is owned
        if (lane == 0) {
          sh.red[0][w] = rr;
          sh.red[1][w] = rz;
        }
      }
      namedArrive<1>(kRowThreads);
      clusterWait();
#pragma unroll
      for (int k = 0; k < kMine; ++k) {
        const uint32_t h = threadIdx.x + k * kRowWorkers;
        if (h < A.haloSize) copyFrom(from[k], h);
      }
      for (uint32_t h = threadIdx.x + kMine * kRowWorkers; h < A.haloSize; h += kRowWorkers) copyFrom(owner(h), h);
      namedSync<2>(kRowWorkers);
      const float3 az = busy ? residentProduct(A, A.z) : mk(0, 0, 0);
      namedSync<3>(kRowThreads);
      code = sh.code;
      if (code) break;
      // A p = A z + beta A pPrev, p = z + beta pPrev (the direction update folded into the product).
      const float fb = sh.factor;
      if (busy) {
        p = it == 0 ? z : axpyRn(p, fb, z);
        apFull = it == 0 ? az : axpyRn(apFull, fb, az);
        ap = filterRn(c, apFull);
        const double pap = warpSum(dotd3(p, ap));
        if (lane == 0) sh.red[0][w] = pap;
      }
      namedArrive<1>(kRowThreads);
      namedSync<3>(kRowThreads);
      code = sh.code;
      if (code) break;
      const float fa = sh.factor;
      ++it;
      // Update (kernels.h:304-315) fused with the preconditioner apply (kernels.h:324-332).
      step = axpyRn(p, fa, step);
      r = axpyRn(ap, -fa, r);
      resid = axpyRn(apFull, -fa, resid);
      z = filterRn(c, mulRn(M, r));
    }
    if (own) {
      D.step[i] = f4(step);
      D.resid[i] = f4(resid);
    }
  }
  clusterArrive();
  clusterWait();
  return sh.failed ? -1 : it;
}

// Index arrays of one solve block (blocks of at most 512 threads): its halo (the particles of other blocks its unpinned rows
// couple to, in particle order) and every slot's column as an index among the block's rows and halo (kNoColumn for pinned
// columns). The particles met are marked in a bitmap in shared memory (`words` words, and their running counts). With
// `halo` null, or a halo of more than `limit`, only the count is written.
__device__ inline void localizeBlock(uint32_t n, uint32_t rank, uint32_t size, const uint32_t* __restrict__ rowStart,
                                     const uint32_t* __restrict__ colIndex, uint32_t words,
                                     uint32_t* __restrict__ haloCount, uint32_t* __restrict__ halo,
                                     uint16_t* __restrict__ localCol, uint32_t limit = UINT32_MAX) {
  uint32_t* bits = reinterpret_cast<uint32_t*>(solveSmem);
  uint32_t* before = bits + words;  // bits set in the words before
  __shared__ uint32_t warpTotal[17];
  const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
  uint32_t r0, r1;
  blockRange(n, rank, size, r0, r1);
  const uint32_t s0 = rowStart[r0], s1 = rowStart[r1];
  for (uint32_t k = t; k < words; k += blockDim.x) bits[k] = 0u;
  __syncthreads();
  for (uint32_t s = s0 + t; s < s1; s += blockDim.x) {
    const uint32_t c = colIndex[s];
    if (!(c & kPinnedBit) && (c < r0 || c >= r1)) atomicOr(bits + (c >> 5), 1u << (c & 31u));
  }
  __syncthreads();
  uint32_t base = 0;
  for (uint32_t k0 = 0; k0 < words; k0 += blockDim.x) {
    const uint32_t k = k0 + t;
    const uint32_t mine = k < words ? __popc(bits[k]) : 0u;
    uint32_t sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= static_cast<uint32_t>(o)) sum += y;
    }
    if (lane == 31) warpTotal[w] = sum;
    __syncthreads();
    if (t == 0) {
      uint32_t acc = 0;
      for (uint32_t q = 0; q < blockDim.x / 32; ++q) {
        const uint32_t x = warpTotal[q];
        warpTotal[q] = acc;
        acc += x;
      }
      warpTotal[16] = acc;
    }
    __syncthreads();
    if (k < words) before[k] = base + warpTotal[w] + sum - mine;
    base += warpTotal[16];
    __syncthreads();
  }
  if (t == 0) *haloCount = base;
  if (!halo || base > limit) return;
  for (uint32_t k = t; k < words; k += blockDim.x) {
    uint32_t at = before[k];
    for (uint32_t m = bits[k]; m; m &= m - 1) halo[at++] = 32 * k + __ffs(m) - 1;
  }
  for (uint32_t s = s0 + t; s < s1; s += blockDim.x) {
    const uint32_t c = colIndex[s];
    uint32_t local = kNoColumn;
    if (!(c & kPinnedBit))
      local = c >= r0 && c < r1 ? c - r0
                                : r1 - r0 + before[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31u)) - 1u));
    localCol[s] = static_cast<uint16_t>(local);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// The same PCG for scenes with more rows than k_solve_rows has threads for, or more matrix than its shared memory holds
// (k_solve_rows_multi): each row thread owns Rows rows of its block (rows 32 (w + 15 m) + lane for m < Rows, so slice
// w + 15 m of 32 rows is warp w's), keeps their p, A p, r, resid and step in registers and the contact planes in shared
// memory. The first P.multiKept slots of each row sit in shared memory; the others are copied at the start of the launch
// into the block's part of D.spill, in the sliced layout, and read from the L2 in every product. The preconditioner
// blocks are read from the L2. Exchanges, tags and stopping tests are pcgResident's; beta arrives during the first
// slice's product, so each row's p and A p are formed as soon as its product is.
//
// What bounds it: the bytes an SM reads from the L2 in an iteration, 38 a slot that is not kept and 48 a row. Measured (us per PCG iteration
// on one B200, against the 1024-thread kernel, which reads every row vector and most of the matrix from the L2 and takes
// two counter barriers): 72k particles 7.1 (11.9), 102k 8.4 (18.4), 141k 9.8 (25.5), 150k 10.7 (27.9), 199k 21.6 (45.5).
// Three rows a thread take the block to 213k particles; the state of a fourth would not fit the registers.
struct MultiMatrix {
  const float4 *a, *b;   // kept slots, as in ResidentMatrix
  const float* c;
  const uint32_t* cols;
  const float4 *sa, *sb;  // slots in the L2
  const float* sc;
  const uint32_t* scols;
  float4* z;
  float4* plane;  // the rows' contact planes: normal, and in w whether the contact is active
  uint32_t rows, haloSize;
  const uint32_t* halo;
};

constexpr int kMultiMost = 3;  // rows a thread may own

struct MultiSlices {  // per slice: its first kept slot, its kept slots, its first slot in the L2, and its slots there
  uint32_t kept[kMultiMost * kRowWorkers / 32 + 1], keptLen[kMultiMost * kRowWorkers / 32];
  uint32_t spill[kMultiMost * kRowWorkers / 32 + 1], spillLen[kMultiMost * kRowWorkers / 32];
};

__device__ __forceinline__ float3 filterRn(float4 plane, float3 v) {
  if (plane.w == 0.0f) return v;
  return axpyRn(xyz(plane), -dotRn(plane.x, plane.y, plane.z, v), v);
}

template <int Rows>
__device__ inline bool stageMulti(const Dev& D, uint32_t rank, uint32_t r0, uint32_t r1, MultiMatrix& A,
                                  MultiSlices& sl) {
  constexpr uint32_t kMost = Rows * kRowWorkers;
  __shared__ uint32_t off[kMost + 1];
  const uint32_t t = threadIdx.x, lane = t & 31u;
  const uint32_t R = r1 - r0, slices = (R + 31u) / 32u, q = D.P.multiKept;
  A.rows = R;
  A.haloSize = __ldg(D.haloCount + rank);
  A.halo = D.halo + static_cast<size_t>(rank) * D.P.haloStride;
  if (R > kMost || blockDim.x != static_cast<unsigned>(kRowThreads) || R + A.haloSize >= D.P.residentNodes) {
    if (t == 0) atomicExch(&D.ctl->error, 4);
    return false;
  }
  const uint32_t first = __ldg(D.rowStart + r0);
  for (uint32_t r = t; r < 32u * slices; r += blockDim.x) {
    uint32_t count = 0;
    if (r < R) {
      const uint32_t rs = __ldg(D.rowStart + r0 + r);
      const bool pinned = D.particle[r0 + r].pinned != 0u;
      off[r] = (rs - first) | (pinned ? kPinnedBit : 0u);
      if (!pinned) count = __ldg(D.rowStart + r0 + r + 1) - rs;
    }
    const uint32_t len = (__reduce_max_sync(0xffffffffu, count) + 1u) & ~1u;
    if (lane == 0) {
      sl.keptLen[r / 32] = min(len, q);
      sl.spillLen[r / 32] = len - min(len, q);
    }
  }
  if (t == 0) off[R] = __ldg(D.rowStart + r1) - first;
  __syncthreads();
  if (t == 0) {
    uint32_t k = 0, x = 0;
    for (uint32_t i = 0; i < slices; ++i) {
      sl.kept[i] = k;
      sl.spill[i] = x;
      k += 32u * sl.keptLen[i];
      x += 32u * sl.spillLen[i];
    }
    sl.kept[slices] = k;
    sl.spill[slices] = x;
  }
  __syncthreads();
  const uint32_t cap = D.P.residentSlots, spillCap = D.P.spillSlots, zeroNode = D.P.residentNodes - 1;
  if (sl.kept[slices] > cap || sl.spill[slices] > spillCap) {
    if (t == 0) atomicExch(&D.ctl->error, 4);
    return false;
  }
  float4* a = solveSmem;
  float4* b = a + cap;
  A.z = b + cap;
  A.plane = A.z + D.P.residentNodes;
  float* c = reinterpret_cast<float*>(A.plane + D.P.multiRows);
  uint16_t* cols = reinterpret_cast<uint16_t*>(c + cap);
  float4* sa = reinterpret_cast<float4*>(D.spill + static_cast<size_t>(rank) * spillCap * kResidentSlotBytes);
  float4* sb = sa + spillCap;
  float* sc = reinterpret_cast<float*>(sb + spillCap);
  uint16_t* scols = reinterpret_cast<uint16_t*>(sc + spillCap);
  A.a = a;
  A.b = b;
  A.c = c;
  A.cols = reinterpret_cast<const uint32_t*>(cols);
  A.sa = sa;
  A.sb = sb;
  A.sc = sc;
  A.scols = reinterpret_cast<const uint32_t*>(scols);
  if (t == 0) A.z[zeroNode] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (uint32_t r = t; r < R; r += blockDim.x) {
    const Contact ct = D.contact[r0 + r];
    A.plane[r] = f4(xyz(ct.normal));
    A.plane[r].w = ct.active != 0u ? 1.0f : 0.0f;
  }
  auto colAt = [](uint32_t base, uint32_t j, uint32_t l) { return base + (32u * (j >> 1) + l) * 2u + (j & 1u); };
  auto put = [&](uint32_t slice, uint32_t j, uint32_t l, const float (&m)[9], uint32_t col) {
    const float4 x = make_float4(m[0], m[1], m[2], m[3]), y = make_float4(m[4], m[5], m[6], m[7]);
    const uint16_t cl = static_cast<uint16_t>(col == kNoColumn ? zeroNode : col);
    if (j < q) {
      const uint32_t pos = sl.kept[slice] + 32u * j + l;
      a[pos] = x;
      b[pos] = y;
      c[pos] = m[8];
      cols[colAt(sl.kept[slice], j, l)] = cl;
    } else {
      const uint32_t pos = sl.spill[slice] + 32u * (j - q) + l;
      sa[pos] = x;
      sb[pos] = y;
      sc[pos] = m[8];
      scols[colAt(sl.spill[slice], j - q, l)] = cl;
    }
  };
  // Padding: each row's positions past its own slots (past its pinned rows' none).
  const float zero[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (uint32_t r = t; r < 32u * slices; r += blockDim.x) {
    const uint32_t count = r < R && !(off[r] & kPinnedBit) ? (off[r + 1] & ~kPinnedBit) - off[r] : 0u;
    for (uint32_t j = count; j < sl.keptLen[r / 32] + sl.spillLen[r / 32]; ++j) put(r / 32, j, r & 31u, zero, kNoColumn);
  }
  const uint32_t S = off[R], SP = D.P.slotsPadded;
  for (uint32_t k = t; k < S; k += blockDim.x) {
    uint32_t lo = 0, hi = R;  // row lo's first slot <= k < row hi's first slot
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if ((off[mid] & ~kPinnedBit) <= k) lo = mid; else hi = mid;
    }
    if (off[lo] & kPinnedBit) continue;  // a pinned row's slot
    const uint32_t s = first + k, col = __ldg(D.localCol + s);
    float m[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) m[e] = col == kNoColumn ? 0.0f : __ldg(D.blocks + e * SP + s);
    put(lo >> 5, k - off[lo], lo & 31u, m, col);
  }
  __syncthreads();
  return true;
}

// U slots (U even) of a slice from slot k on, kept (shared memory) or not (L2): all their loads before the first product.
template <int U, bool Kept, bool Sequential>
__device__ __forceinline__ void multiSlots(const MultiMatrix& A, uint32_t base, uint32_t k, float3 (&acc)[2]) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t cc[U / 2];
  float4 a[U], b[U], x[U];
  float c[U];
#pragma unroll
  for (int u = 0; u < U / 2; ++u) {
    const uint32_t at = base / 2 + 16u * k + 32u * u + lane;
    cc[u] = Kept ? A.cols[at] : __ldcg(A.scols + at);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t pos = base + 32u * (k + u) + lane;
    a[u] = Kept ? A.a[pos] : __ldcg(A.sa + pos);
    b[u] = Kept ? A.b[pos] : __ldcg(A.sb + pos);
    c[u] = Kept ? A.c[pos] : __ldcg(A.sc + pos);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) x[u] = A.z[(u & 1) ? cc[u / 2] >> 16 : cc[u / 2] & 0xFFFFu];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const float m[9] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w, c[u]};
    if (Sequential) {
      acc[0].x = __fadd_rn(acc[0].x, dotYRn(m[0], m[1], m[2], xyz(x[u])));
      acc[0].y = __fadd_rn(acc[0].y, dotYRn(m[3], m[4], m[5], xyz(x[u])));
      acc[0].z = __fadd_rn(acc[0].z, dotYRn(m[6], m[7], m[8], xyz(x[u])));
    } else {
      blockMulAddRn(acc[u & 1], m, xyz(x[u]));
    }
  }
}

// A z for this thread's row of a slice, in residentProduct's order (multiKept is even, so slot parity is kept), or
// Sequential in the slot-parallel scheme's (directionProducts<0>): all slots in one sum.
template <bool Sequential>
__device__ __forceinline__ float3 multiProduct(const MultiMatrix& A, const MultiSlices& sl, uint32_t slice) {
  float3 acc[2] = {mk(0, 0, 0), mk(0, 0, 0)};
  const uint32_t kept = sl.keptLen[slice], spill = sl.spillLen[slice];
  uint32_t k = 0;
  for (; k + 4 <= kept; k += 4) multiSlots<4, true, Sequential>(A, sl.kept[slice], k, acc);
  if (k < kept) multiSlots<2, true, Sequential>(A, sl.kept[slice], k, acc);
  k = 0;
  for (; k + 4 <= spill; k += 4) multiSlots<4, false, Sequential>(A, sl.spill[slice], k, acc);
  if (k < spill) multiSlots<2, false, Sequential>(A, sl.spill[slice], k, acc);
  if (Sequential) return acc[0];
  return mk(__fadd_rn(acc[0].x, acc[1].x), __fadd_rn(acc[0].y, acc[1].y), __fadd_rn(acc[0].z, acc[1].z));
}

template <int Rows, bool Sequential>
__device__ inline int pcgResidentMulti(const Dev& D, GridSync& gs, const MultiMatrix& A, const MultiSlices& sl,
                                       unsigned long long& seq) {
  constexpr int kWarps = kRowWorkers / 32;
  __shared__ ResidentShared sh;
  const int maxCg = D.P.maxCg;
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const unsigned long long base = seq;
  if (threadIdx.x == 0) sh.failed = 0;
  __syncthreads();
  int it = 0, code = 0;
  if (w == kWarps) {
    it = residentExchanges(D, gs, sh, base, code);
  } else {
    uint32_t r0i, r1i;
    blockRange(D.P.n, gs.rank, gs.size, r0i, r1i);
    const uint32_t R = r1i - r0i;
    uint32_t row[Rows];  // in the block
    bool own[Rows];
    float3 step[Rows], resid[Rows], r[Rows], p[Rows], apFull[Rows];
#pragma unroll
    for (int m = 0; m < Rows; ++m) {
      row[m] = 32u * (w + kWarps * m) + lane;
      own[m] = row[m] < R;
      step[m] = resid[m] = r[m] = p[m] = apFull[m] = mk(0, 0, 0);
      if (own[m]) {
        resid[m] = -ld3(D.grad, r0i + row[m]);
        r[m] = filterRn(A.plane[row[m]], resid[m]);
      }
    }
    while (it < maxCg) {
      const uint32_t tag = static_cast<uint32_t>(base + 1 + 2 * static_cast<unsigned long long>(it)) | 0x80000000u;
      double rr = 0.0, rz = 0.0;
#pragma unroll
      for (int m = 0; m < Rows; ++m)
        if (own[m]) {
          const uint32_t i = r0i + row[m];
          const float3 z = filterRn(A.plane[row[m]], mulRn(loadPrecond(D, i), r[m]));
          storeTagged(D.z + i, z, tag);
          A.z[row[m]] = f4(z);
          rr += dotd3(r[m], r[m]);
          rz += dotd3(r[m], z);
        }
      rr = warpSum(rr);
      rz = warpSum(rz);
      if (lane == 0) {
        sh.red[0][w] = rr;
        sh.red[1][w] = rz;
      }
      namedArrive<1>(kRowThreads);
      if (!takeHalo(D, A, A.z, D.z, tag)) sh.failed = 1;
      namedSync<2>(kRowWorkers);
      double pap = 0.0;
      float fb = 0.0f;
#pragma unroll
      for (int m = 0; m < Rows; ++m) {
        const bool busy = 32u * (w + kWarps * m) < R;
        const float3 az = busy ? multiProduct<Sequential>(A, sl, w + kWarps * m) : mk(0, 0, 0);
        if (m == 0) {
          namedSync<3>(kRowThreads);
          code = sh.code;
          if (code) break;
          fb = sh.factor;
        }
        if (own[m]) {
          const float3 z = xyz(A.z[row[m]]);
          p[m] = it == 0 ? z : axpyRn(p[m], fb, z);
          apFull[m] = it == 0 ? az : axpyRn(apFull[m], fb, az);
          pap += dotd3(p[m], filterRn(A.plane[row[m]], apFull[m]));
        }
      }
      if (code) break;
      pap = warpSum(pap);
      if (lane == 0) sh.red[0][w] = pap;
      namedArrive<1>(kRowThreads);
      namedSync<3>(kRowThreads);
      code = sh.code;
      if (code) break;
      const float fa = sh.factor;
      ++it;
#pragma unroll
      for (int m = 0; m < Rows; ++m)
        if (own[m]) {
          step[m] = axpyRn(p[m], fa, step[m]);
          r[m] = axpyRn(filterRn(A.plane[row[m]], apFull[m]), -fa, r[m]);
          resid[m] = axpyRn(apFull[m], -fa, resid[m]);
        }
    }
#pragma unroll
    for (int m = 0; m < Rows; ++m)
      if (own[m]) {
        D.step[r0i + row[m]] = f4(step[m]);
        D.resid[r0i + row[m]] = f4(resid[m]);
      }
  }
  __syncthreads();
  seq = sh.seq;
  __syncthreads();
  return code == 2 ? -1 : it;
}

// ---------------------------------------------------------------------------------------------------------------
// The learned PCG over resident rows (k_solve_rows_learned): pcgLearned's recurrences, stopping tests and breakdown rules
// with the matrix, the rows and the exchanges of pcgResident, and the factor by rows in the sliced layout (three float4 a
// slot): in shared memory where a block has the room (up to about 28k particles), else in the L2.
//
// An iteration is three products, A z, y = L^T r and z = L y, each of which needs its operand from the neighbours, and
// three sums. The operands are published with tags and taken as they come; r.r travels during the two factor products
// and r.z during A z, so only p.Ap is waited for. Two arrays in shared memory hold the operands by turns: an operand is
// written only after the barrier that follows every read of the array's last one.
//
// Measured (us per PCG iteration, one B200, against four counter barriers an iteration and the operands gathered from the
// L2): 10k particles 7.0 (was 13.7), 60k 12.7 (25.1). What bounds it: at 10k the way of r, y and z to the neighbours, one
// after the other, and the exchange of p.Ap (about 4 us); at 60k also the factor's 42 MB from the L2. At 60k the factor
// read by rows (each lane its own row) took 18.7-19.7, since every 16-byte load was its own L2 sector; 2, 3 or 4 slots in
// flight 13.2, 12.7 and 14.0 (four spill).
constexpr int kLearnedDepth = 3;  // slots whose factor blocks a row thread has in flight

// The learned PCG's contact filter, with every rounding written out, so that its iterates do not depend on how the
// compiler contracts the code around it.
__device__ __forceinline__ float3 filterYRn(const Contact& c, float3 v) {
  if (c.active == 0u) return v;
  const float3 n = xyz(c.normal);
  return axpyRn(n, -dotYRn(n.x, n.y, n.z, v), v);
}

// acc += B x (Upper: B^T x) for this thread's row over its slots [kBegin, kEnd) (the columns are sorted, so the lower part
// j <= i is [0, kd] and the upper part j >= i is [kd, end) with kd the diagonal's position). InSmem: the factor is in
// shared memory. kLearnedDepth slots' loads are issued before their first product (past the range's end the last slot's
// again, unused). For a slot in registers the first column in shared memory is read too and dropped: a warp whose rows have
// no slots there reads the next warp's, or what follows the last (kColumnsRead). Reading it under a condition takes 7.64
// us an iteration at 10k particles instead of 6.98, and 13.2 instead of 12.6 at 60k.
template <bool Upper, bool InSmem>
__device__ __forceinline__ float3 factorProduct(const Dev& D, const ResidentMatrix& A, const float4* x,
                                                uint32_t kBegin, uint32_t kEnd) {
  const uint32_t lane = threadIdx.x & 31u, zeroNode = D.P.residentNodes - 1;
  const uint16_t* cols = reinterpret_cast<const uint16_t*>(A.cols);
  float3 acc = mk(0, 0, 0);
  for (uint32_t k0 = kBegin; k0 < kEnd; k0 += kLearnedDepth) {
    uint32_t col[kLearnedDepth];
    float4 m[kLearnedDepth][3], v[kLearnedDepth];
#pragma unroll
    for (int u = 0; u < kLearnedDepth; ++u) {
      const uint32_t k = min(k0 + u, kEnd - 1), j = max(k, static_cast<uint32_t>(kRegSlots)) - kRegSlots;
      static_assert(kRegSlots == 2, "the register slots' columns are one word");
      const uint32_t inRegs = k == 0 ? A.regCols[0] & 0xFFFFu : A.regCols[0] >> 16;
      const uint32_t inSmem = cols[A.base + (32u * (j >> 1) + lane) * 2u + (j & 1u)];
      col[u] = k < static_cast<uint32_t>(kRegSlots) ? inRegs : inSmem;
      if (k0 + u >= kEnd) col[u] = zeroNode;
    }
#pragma unroll
    for (int u = 0; u < kLearnedDepth; ++u) {
      const uint32_t k = min(k0 + u, kEnd - 1);
      const float4* f = A.factor + A.factorBase + 32u * k + lane;
#pragma unroll
      for (int q = 0; q < 3; ++q) m[u][q] = InSmem ? f[q * D.P.factorSlots] : __ldcg(f + q * D.P.factorSlots);
      v[u] = x[col[u]];
    }
#pragma unroll
    for (int u = 0; u < kLearnedDepth; ++u) {
      if (col[u] == zeroNode) continue;  // pinned columns and the end of the range
      const float4 a = m[u][0], b = m[u][1], c = m[u][2];
      const float3 w = xyz(v[u]);
      if (Upper) {  // L_ji^T x_j
        acc.x = __fadd_rn(acc.x, dotYRn(a.x, b.x, c.x, w));
        acc.y = __fadd_rn(acc.y, dotYRn(a.y, b.y, c.y, w));
        acc.z = __fadd_rn(acc.z, dotYRn(a.z, b.z, c.z, w));
      } else {  // L_ij x_j
        acc.x = __fadd_rn(acc.x, dotYRn(a.x, a.y, a.z, w));
        acc.y = __fadd_rn(acc.y, dotYRn(b.x, b.y, b.z, w));
        acc.z = __fadd_rn(acc.z, dotYRn(c.x, c.y, c.z, w));
      }
    }
  }
  return acc;
}

// Returns the iteration count, -1 when a wait gave up, or -2 - iterations on a breakdown (the caller then solves with
// block-Jacobi). `seq` is the last exchange's number, advanced by the exchanges done.
__device__ inline int pcgLearnedResident(const Dev& D, GridSync& gs, ResidentMatrix& A, unsigned long long& seq) {
  constexpr int kWarps = kRowWorkers / 32;
  __shared__ ResidentShared sh;
  const int maxCg = D.P.maxCg;
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const unsigned long long base = seq;
  if (threadIdx.x == 0) sh.failed = 0;
  __syncthreads();
  int it = 0, code = 0;
  if (w == kWarps) {  // the exchange warp
    double rz = 0.0, r0 = 0.0, rr0 = 0.0, total = 0.0;
    unsigned long long num = base;
    // One sum: waits for the row warps' part, adds it up over the blocks; false when a wait gave up.
    int delays[3] = {kExchangeDelay, kExchangeDelay, kExchangeDelay};  // p.Ap, r.r, r.z
    auto sum = [&](int& delay) {
      namedSync<1>(kRowThreads);
      const double part[1] = {warpSum(lane < kWarps ? sh.red[0][lane] : 0.0)};
      double t[1] = {0.0};
      const bool ok = !sh.failed && mailSum<1>(D.mail, D.ctl, D.P.barrierLimitNs, gs.rank, gs.size, ++num, part, t,
                                               delay);
      total = t[0];
      return ok;
    };
    auto tell = [&](float factor) {
      if (lane == 0) {
        sh.code = code;
        sh.factor = factor;
        sh.seq = num;
      }
      namedArrive<3>(kRowThreads);
      return code == 0;
    };
    // |r0|, then r.z.
    if (!sum(delays[1])) {
      code = 2;
    } else {
      rr0 = total;
      r0 = sqrt(rr0);
      code = r0 > 0.0 && rr0 > 0.0 ? 0 : 1;
    }
    if (tell(0.0f)) {
      if (!sum(delays[2])) code = 2;
      else code = isfinite(total) ? 0 : 3;
      rz = total;
      if (tell(0.0f)) {
        while (it < maxCg) {
          if (!sum(delays[0])) code = 2;  // p.Ap
          else code = !isfinite(total) ? 3 : total > 0.0 ? 0 : 1;
          if (!tell(code ? 0.0f : static_cast<float>(rz / total))) break;
          ++it;
          if (!sum(delays[1])) code = 2;  // r.r
          else code = !isfinite(total) ? 3 : sqrt(total) <= D.P.cgTolerance * r0 ? 1 : total > 1e6 * rr0 ? 3 : 0;
          if (!tell(0.0f)) break;
          if (!sum(delays[2])) code = 2;  // r.z
          else code = isfinite(total) ? 0 : 3;
          const float beta = static_cast<float>(total / rz);
          rz = total;
          if (!tell(beta)) break;
        }
      }
    }
  } else {
    uint32_t r0i, r1i;
    blockRange(D.P.n, gs.rank, gs.size, r0i, r1i);
    const uint32_t i = r0i + threadIdx.x;
    const bool own = i < r1i, busy = 32u * w < r1i - r0i;
    // The row's length and its diagonal's position (the factor's lower part is [0, kd], the upper [kd, len)); a pinned
    // row takes none (its L is zero), and no range passes the slots staged.
    const uint32_t rs = own ? __ldg(D.rowStart + i) : 0u;
    const bool live = own && D.particle[i].pinned == 0u;
    const uint32_t len = live ? min(__ldg(D.rowStart + i + 1) - rs, A.len + kRegSlots) : 0u;
    const uint32_t kd = live ? min(__ldg(D.diagSlot + i) - rs, len) : 0u;
    Contact c{};
    float3 step = mk(0, 0, 0), resid = mk(0, 0, 0), r = mk(0, 0, 0), z = mk(0, 0, 0);
    float3 p = mk(0, 0, 0), ap = mk(0, 0, 0), apFull = mk(0, 0, 0);
    if (own) {
      c = D.contact[i];
      resid = -ld3(D.grad, i);
      r = filterRn(c, resid);
    }
    if (!busy && lane == 0) sh.red[0][w] = 0.0;
    float4* cur = A.z;                        // the operand being used
    float4* other = A.z + D.P.residentNodes;  // and the next one's place
    unsigned long long num = base;
    // The row's sum on its way to the exchange warp.
    auto send = [&](float3 x, float3 y) {
      if (busy) {
        const double v = warpSum(dotd3(x, y));  // zero where no row is owned
        if (lane == 0) sh.red[0][w] = v;
      }
      namedArrive<1>(kRowThreads);
    };
    auto hear = [&] {
      namedSync<3>(kRowThreads);
      code = sh.code;
      return code == 0;
    };
    const uint32_t high = 0x80000000u;
    auto publish = [&](float4* global, float3 v, uint32_t tag) {
      if (own) {
        storeTagged(global + i, v, tag);
        cur[threadIdx.x] = f4(v);
      }
    };
    auto take = [&](const float4* global, uint32_t tag) {
      if (!takeHalo(D, A, cur, global, tag)) sh.failed = 1;
      namedSync<2>(kRowWorkers);
    };
    auto turn = [&] {
      float4* t = cur;
      cur = other;
      other = t;
    };
    // z = F(L L^T r), r.r on its way meanwhile; then r.z on its way. Returns false when r.r ends the solve.
    auto apply = [&] {
      const uint32_t tag = static_cast<uint32_t>(++num) | high;
      publish(D.r, r, tag);
      send(r, r);
      take(D.r, tag);
      float3 y = mk(0, 0, 0);
      if (busy) y = D.LfSliced ? factorProduct<true, false>(D, A, cur, kd, len)
                               : factorProduct<true, true>(D, A, cur, kd, len);
      turn();
      publish(D.ap, y, tag);
      take(D.ap, tag);
      if (busy) z = filterYRn(c, D.LfSliced ? factorProduct<false, false>(D, A, cur, 0, min(kd + 1, len))
                                            : factorProduct<false, true>(D, A, cur, 0, min(kd + 1, len)));
      turn();
      if (!hear()) return false;
      const uint32_t tagZ = static_cast<uint32_t>(++num) | high;
      publish(D.z, z, tagZ);
      send(r, z);
      return true;
    };
    // A z, r.z arriving meanwhile. Returns false when r.z ends the solve.
    float3 az = mk(0, 0, 0);
    auto product = [&] {
      take(D.z, static_cast<uint32_t>(num) | high);
      if (busy) az = residentProduct(A, cur);
      turn();
      return hear();
    };
    if (apply() && product()) {
      float fb = 0.0f;
      while (it < maxCg) {
        // A p = A z + beta A pPrev, p = z + beta pPrev.
        if (own) {
          p = it == 0 ? z : axpyRn(p, fb, z);
          apFull = it == 0 ? az : axpyRn(apFull, fb, az);
          ap = filterYRn(c, apFull);
        }
        ++num;
        send(p, ap);
        if (!hear()) break;
        const float fa = sh.factor;
        ++it;
        if (own) {
          step = axpyRn(p, fa, step);
          r = axpyRn(ap, -fa, r);
          resid = axpyRn(apFull, -fa, resid);
        }
        if (!apply() || !product()) break;
        fb = sh.factor;
      }
    }
    if (own) {
      D.step[i] = f4(step);
      D.resid[i] = f4(resid);
    }
  }
  __syncthreads();
  seq = sh.seq;
  __syncthreads();
  return code == 2 ? -1 : code == 3 ? -2 - it : it;
}

// Pipelined contact-filtered block-Jacobi PCG (Ghysels and Vanroose, "Hiding global synchronization latency in the
// preconditioned conjugate gradient algorithm", Parallel Computing 40 (2014) 224-238, Alg. 3). In exact arithmetic
// its iterates, iteration count and stopping tests are those of pcgReferenceOrder (operator F A F, preconditioner
// F M F, the same |r| <= tol |r0| and p.Ap <= 0 tests): besides u = M r and w = A u it carries s = A p, q = M s and
// z = A q by recurrence, so each iteration is one pass over the rows and ONE grid exchange instead of two. The pass
// forms n = F A m for the m = F M w of the previous exchange (the only gather), updates the row's z, q, s, p, x, r,
// u, w and forms the next exchange's FP64 partials (r.u, w.u, r.r) and the next m; the exchange (gridReduce<3>)
// publishes partials and m together. m alternates between two buffers: a block cannot pass the next exchange before
// every block has arrived at it, hence before any block still gathers the m it would overwrite. The unfiltered
// residual for the contact force, resid = -grad - A step, is formed once after the loop. Vectors: x = step, r = r,
// u = z, w = ap, s = apFull, p = p0, q = p1, z = pz, m = pm0 / pm1. Returns the iteration count, or -1 when a grid
// barrier gave up.
template <int PL>
__device__ inline int pcgPipelined(const Dev& D, GridSync& gs, const SmemMatrix& A) {
  uint32_t r0i, r1i;
  blockRange(D.P.n, gs.rank, gs.size, r0i, r1i);
  float4 *x = D.step, *r = D.r, *u = D.z, *w = D.ap, *s = D.apFull, *p = D.p0, *q = D.p1, *zq = D.pz;
  // x = 0, r = F(-grad), u = F(M r); u is gathered next, so a plain barrier publishes it.
  for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
    const Contact c = D.contact[i];
    const float3 ri = filterContact(c, -ld3(D.grad, i));
    x[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    r[i] = f4(ri);
    u[i] = f4(filterContact(c, mul(loadPrecond(D, i), ri)));
  }
  if (!gs.sync()) return -1;
  // w = F A u, the first partials and m.
  double t[3];
  {
    double v[3] = {0.0, 0.0, 0.0};
    directionProducts<PL>(
        D, A, r0i, r1i, [&](uint32_t j) { return ld3(u, j); },
        [&](uint32_t i, float3 ui, float3 au) {
          const Contact c = D.contact[i];
          const float3 wi = filterContact(c, au);
          const float3 ri = ld3(r, i);
          w[i] = f4(wi);
          v[0] += dotd3(ri, ui);
          v[1] += dotd3(wi, ui);
          v[2] += dotd3(ri, ri);
          D.pm0[i] = f4(filterContact(c, mul(loadPrecond(D, i), wi)));
        });
    if (!gridReduce<3>(D, gs, v, t)) return -1;
  }
  const double r0 = sqrt(t[2]);
  double gammaPrev = 0.0, alphaPrev = 0.0;
  int it = 0;
  while (it < D.P.maxCg) {
    if (!(r0 > 0.0)) break;
    if (it > 0 && sqrt(t[2]) <= D.P.cgTolerance * r0) break;
    const double gamma = t[0], delta = t[1];
    const double beta = it == 0 ? 0.0 : gamma / gammaPrev;
    const double pAp = it == 0 ? delta : delta - beta * gamma / alphaPrev;
    if (!(pAp > 0.0)) break;
    const double alpha = gamma / pAp;
    const float fa = static_cast<float>(alpha), fb = static_cast<float>(beta);
    const bool first = it == 0;
    const float4* mCur = (it & 1) ? D.pm1 : D.pm0;
    float4* mNext = (it & 1) ? D.pm0 : D.pm1;
    double v[3] = {0.0, 0.0, 0.0};
    directionProducts<PL>(
        D, A, r0i, r1i, [&](uint32_t j) { return ld3(mCur, j); },
        [&](uint32_t i, float3 mi, float3 am) {
          // Each recurrence is formed and stored in turn (z, w, s, r, q, u, p, x), so that only r, u and w stay live.
          const Contact c = D.contact[i];
          const float3 zi = first ? filterContact(c, am) : filterContact(c, am) + ld3(zq, i) * fb;
          zq[i] = f4(zi);
          const float3 wi0 = ld3(w, i);
          const float3 wi = wi0 - zi * fa;
          w[i] = f4(wi);
          const float3 si = first ? wi0 : wi0 + ld3(s, i) * fb;
          s[i] = f4(si);
          const float3 ri = ld3(r, i) - si * fa;
          r[i] = f4(ri);
          const float3 qi = first ? mi : mi + ld3(q, i) * fb;
          q[i] = f4(qi);
          const float3 ui0 = ld3(u, i);
          const float3 ui = ui0 - qi * fa;
          u[i] = f4(ui);
          const float3 pi = first ? ui0 : ui0 + ld3(p, i) * fb;
          p[i] = f4(pi);
          x[i] = f4(ld3(x, i) + pi * fa);
          v[0] += dotd3(ri, ui);
          v[1] += dotd3(wi, ui);
          v[2] += dotd3(ri, ri);
          mNext[i] = f4(filterContact(c, mul(loadPrecond(D, i), wi)));
        });
    ++it;
    gammaPrev = gamma;
    alphaPrev = alpha;
    if (!gridReduce<3>(D, gs, v, t)) return -1;
  }
  // resid = -grad - A step over unpinned rows and columns (the reference-order PCG's recurrence, formed directly). Every
  // exit of the loop follows a grid exchange, whose barrier has published every block's last x.
  directionProducts<PL>(
      D, A, r0i, r1i, [&](uint32_t j) { return ld3(x, j); },
      [&](uint32_t i, float3, float3 ax) { D.resid[i] = f4(-ld3(D.grad, i) - ax); });
  return it;
}

// Contact-filtered block-Jacobi PCG in the Chronopoulos-Gear form ("s-step iterative methods for symmetric linear
// systems", J. Comput. Appl. Math. 25 (1989) 153-168): the same iterates and stopping tests as pcgReferenceOrder in
// exact arithmetic. Each iteration forms w = F A z exactly (the only gather), reduces r.z, w.z and r.r in one FP64 grid
// reduction, and takes alpha = (r.z) / (w.z - beta (r.z) / alpha_prev) (= r.z / p.Ap) with beta = (r.z) / (r.z)_prev;
// A p is carried as s = w + beta s, as the reference-order form carries it. The exchange that publishes the new z is a
// plain barrier instead of the reference order's second reduction. resid = -grad - A step is formed after the loop.
// Vectors: x = step, r = r, z = z, p = p0, s = ap, w = apFull. Returns the iteration count, or -1 when a grid barrier
// gave up.
template <int PL>
__device__ inline int pcgSingleReduction(const Dev& D, GridSync& gs, const SmemMatrix& A) {
  uint32_t r0i, r1i;
  blockRange(D.P.n, gs.rank, gs.size, r0i, r1i);
  float4 *x = D.step, *r = D.r, *z = D.z, *p = D.p0, *s = D.ap, *w = D.apFull;
  for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
    const Contact c = D.contact[i];
    const float3 ri = filterContact(c, -ld3(D.grad, i));
    x[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    r[i] = f4(ri);
    z[i] = f4(filterContact(c, mul(loadPrecond(D, i), ri)));
  }
  if (!gs.sync()) return -1;
  double r0 = 0.0, gammaPrev = 0.0, alphaPrev = 0.0;
  int it = 0;
  while (true) {
    // w = F A z and the three partials.
    double v[3] = {0.0, 0.0, 0.0};
    directionProducts<PL>(
        D, A, r0i, r1i, [&](uint32_t j) { return ld3(z, j); },
        [&](uint32_t i, float3 zi, float3 az) {
          const float3 wi = filterContact(D.contact[i], az);
          const float3 ri = ld3(r, i);
          w[i] = f4(wi);
          v[0] += dotd3(ri, zi);
          v[1] += dotd3(wi, zi);
          v[2] += dotd3(ri, ri);
        });
    double t[3];
    if (!gridReduce<3>(D, gs, v, t)) return -1;
    if (it == 0) r0 = sqrt(t[2]);
    if (!(r0 > 0.0)) break;
    if (it > 0 && sqrt(t[2]) <= D.P.cgTolerance * r0) break;
    if (it >= D.P.maxCg) break;
    const double gamma = t[0];
    const double beta = it == 0 ? 0.0 : gamma / gammaPrev;
    const double pAp = it == 0 ? t[1] : t[1] - beta * gamma / alphaPrev;
    if (!(pAp > 0.0)) break;
    const double alpha = gamma / pAp;
    const float fa = static_cast<float>(alpha), fb = static_cast<float>(beta);
    const bool first = it == 0;
    for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
      const Contact c = D.contact[i];
      const float3 pi = first ? ld3(z, i) : ld3(z, i) + ld3(p, i) * fb;
      p[i] = f4(pi);
      const float3 si = first ? ld3(w, i) : ld3(w, i) + ld3(s, i) * fb;
      s[i] = f4(si);
      x[i] = f4(ld3(x, i) + pi * fa);
      const float3 ri = ld3(r, i) - si * fa;
      r[i] = f4(ri);
      z[i] = f4(filterContact(c, mul(loadPrecond(D, i), ri)));
    }
    ++it;
    gammaPrev = gamma;
    alphaPrev = alpha;
    if (!gs.sync()) return -1;
  }
  // resid = -grad - A step over unpinned rows and columns; the last exchange has published every block's x.
  directionProducts<PL>(
      D, A, r0i, r1i, [&](uint32_t j) { return ld3(x, j); },
      [&](uint32_t i, float3, float3 ax) { D.resid[i] = f4(-ld3(D.grad, i) - ax); });
  return it;
}

// z = F(L L^T r) over this block's rows, with L the learned factor (planes D.Lf, lower slots) and y = L^T r kept in
// D.ap between the two products; returns false when a grid barrier gave up. Adds r.z of its rows to *rz.
template <int RL>
__device__ inline bool applyLearned(const Dev& D, GridSync& gs, uint32_t r0i, uint32_t r1i, double* rz) {
  const uint32_t groups = blockDim.x / RL;
  const int sub = threadIdx.x & (RL - 1);
  const unsigned groupMask = ((1u << RL) - 1u) << ((threadIdx.x & 31) & ~(RL - 1));
  const uint32_t SP = D.P.slotsPadded;
  // y_j = sum over slots (j, i), i >= j, of L_(i, j)^T r_i.
  for (uint32_t j = r0i + threadIdx.x / RL; j < r1i; j += groups) {
    float3 acc = mk(0, 0, 0);
    for (uint32_t s = __ldg(D.rowStart + j) + sub; s < __ldg(D.rowStart + j + 1); s += RL) {
      const uint32_t col = __ldg(D.colIndex + s);
      if ((col & kPinnedBit) || col < j) continue;
      const uint32_t t = __ldg(D.tslot + s);
      const float3 v = ld3(D.r, col);
      const float* L = D.Lf + t;
      acc.x += L[0] * v.x + L[3 * SP] * v.y + L[6 * SP] * v.z;
      acc.y += L[SP] * v.x + L[4 * SP] * v.y + L[7 * SP] * v.z;
      acc.z += L[2 * SP] * v.x + L[5 * SP] * v.y + L[8 * SP] * v.z;
    }
#pragma unroll
    for (int o = RL / 2; o > 0; o >>= 1) {
      acc.x += __shfl_xor_sync(groupMask, acc.x, o);
      acc.y += __shfl_xor_sync(groupMask, acc.y, o);
      acc.z += __shfl_xor_sync(groupMask, acc.z, o);
    }
    if (sub == 0) D.ap[j] = f4(acc);
  }
  if (!gs.sync()) return false;
  // z_i = F(sum over slots (i, j), j <= i, of L_(i, j) y_j).
  for (uint32_t i = r0i + threadIdx.x / RL; i < r1i; i += groups) {
    float3 acc = mk(0, 0, 0);
    for (uint32_t s = __ldg(D.rowStart + i) + sub; s < __ldg(D.rowStart + i + 1); s += RL) {
      const uint32_t col = __ldg(D.colIndex + s);
      if ((col & kPinnedBit) || col > i) continue;
      const float3 v = ld3(D.ap, col);
      const float* L = D.Lf + s;
      acc.x += L[0] * v.x + L[SP] * v.y + L[2 * SP] * v.z;
      acc.y += L[3 * SP] * v.x + L[4 * SP] * v.y + L[5 * SP] * v.z;
      acc.z += L[6 * SP] * v.x + L[7 * SP] * v.y + L[8 * SP] * v.z;
    }
#pragma unroll
    for (int o = RL / 2; o > 0; o >>= 1) {
      acc.x += __shfl_xor_sync(groupMask, acc.x, o);
      acc.y += __shfl_xor_sync(groupMask, acc.y, o);
      acc.z += __shfl_xor_sync(groupMask, acc.z, o);
    }
    if (sub == 0) {
      const float3 zi = filterContact(D.contact[i], acc);
      D.z[i] = f4(zi);
      *rz += dotd3(ld3(D.r, i), zi);
    }
  }
  return true;
}

// PCG with the learned preconditioner M^-1 = L L^T (contact-filtered), in the reference's order otherwise: four grid
// synchronisations per iteration (p.Ap, r.r, y = L^T r, r.z). The convergence test is the reference's, on the
// unpreconditioned residual. Returns the iteration count, -1 when a barrier gave up, or -2 - iterations when the
// solve broke down (a non-finite scalar, or |r|^2 above 1e6 |r0|^2): the caller then solves again with block-Jacobi.
// M^-1 = L L^T is SPD for any finite L with a positive block diagonal, so a finite solve converges like any PCG; its
// unpreconditioned |r| is not monotone and is no stall signal. With `warm`, step, resid and r hold a partial solve
// (a block-Jacobi phase) and the iteration continues from them, with `r0In` (that solve's initial |r|) in the
// convergence test; `budget` bounds the iterations.
template <int PL>
__device__ inline int pcgLearned(const Dev& D, GridSync& gs, const SmemMatrix& A, bool warm = false,
                                 double r0In = 0.0, int budget = -1) {
  const uint32_t n = D.P.n;
  uint32_t r0i, r1i;
  blockRange(n, gs.rank, gs.size, r0i, r1i);
  double rr0;
  {
    double v[1] = {0.0};
    for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
      if (warm) {
        v[0] += dotd3(ld3(D.r, i), ld3(D.r, i));
        continue;
      }
      const float3 res = -ld3(D.grad, i);
      const float3 ri = filterContact(D.contact[i], res);
      D.step[i] = make_float4(0, 0, 0, 0);
      D.resid[i] = f4(res);
      D.r[i] = f4(ri);
      v[0] += dotd3(ri, ri);
    }
    double t[1];
    if (!gridReduce<1>(D, gs, v, t)) return -1;
    rr0 = t[0];
  }
  const double r0 = warm ? r0In : sqrt(rr0);
  if (!(r0 > 0.0) || !(rr0 > 0.0)) return 0;
  double rz;
  {
    double v[1] = {0.0};
    if (!applyLearned<(PL > 0 ? PL : kRowLanes)>(D, gs, r0i, r1i, &v[0])) return -1;
    double t[1];
    if (!gridReduce<1>(D, gs, v, t)) return -1;
    rz = t[0];
  }
  if (!isfinite(rz)) return -2;
  double beta = 0.0;
  float4* pPrev = D.p0;
  float4* pCur = D.p1;
  int it = 0;
  const int maxCg = budget < 0 ? D.P.maxCg : min(budget, D.P.maxCg);
  while (it < maxCg) {
    // SpMV with the direction update folded in: p_j = z_j + beta * pPrev_j.
    double vpap[1] = {directionStep<PL>(D, A, r0i, r1i, pPrev, pCur, static_cast<float>(beta), it == 0)};
    double pAp[1];
    if (!gridReduce<1>(D, gs, vpap, pAp)) return -1;
    if (!isfinite(pAp[0])) return -2 - it;
    if (!(pAp[0] > 0.0)) break;
    const float fa = static_cast<float>(rz / pAp[0]);
    ++it;
    double v[1] = {0.0};
    for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
      const float3 pi = ld3(pCur, i);
      D.step[i] = f4(ld3(D.step, i) + pi * fa);
      const float3 ri = ld3(D.r, i) - ld3(D.ap, i) * fa;
      D.r[i] = f4(ri);
      D.resid[i] = f4(ld3(D.resid, i) - ld3(D.apFull, i) * fa);
      v[0] += dotd3(ri, ri);
    }
    double rr[1];
    if (!gridReduce<1>(D, gs, v, rr)) return -1;
    if (!isfinite(rr[0])) return -2 - it;
    if (sqrt(rr[0]) <= D.P.cgTolerance * r0) break;
    if (rr[0] > 1e6 * rr0) return -2 - it;
    double vz[1] = {0.0};
    if (!applyLearned<(PL > 0 ? PL : kRowLanes)>(D, gs, r0i, r1i, &vz[0])) return -1;
    double rzNew[1];
    if (!gridReduce<1>(D, gs, vz, rzNew)) return -1;
    if (!isfinite(rzNew[0])) return -2 - it;
    beta = rzNew[0] / rz;
    rz = rzNew[0];
    float4* tmp = pPrev;
    pPrev = pCur;
    pCur = tmp;
  }
  return it;
}

// The solve's PCG: block-Jacobi (reference order), or the learned schedule: P.learnedSwitch block-Jacobi iterations
// first (0: none), then, when the solve has not converged, the learned preconditioner from the current iterate within
// the remaining iteration budget; a learned phase that stalls is followed by a full block-Jacobi solve. Returns the
// total iteration count of all phases, or -1 when a barrier gave up.
// Variant (block-Jacobi only): 0 the reference's order (pcgReferenceOrder), 1 pipelined (pcgPipelined; needs the
// pm0/pm1/pz vectors), 2 Chronopoulos-Gear (pcgSingleReduction). A compile-time choice, so each solve kernel carries
// one PCG's registers.
template <bool Learned, int PL, int Variant>
__device__ inline int pcgSolveStaged(const Dev& D, GridSync& gs, const SmemMatrix& A);

template <bool Learned, int PL, int Variant = 0>
__device__ inline int pcgSolve(const Dev& D, GridSync& gs) {
  uint32_t r0i, r1i;
  blockRange(D.P.n, gs.rank, gs.size, r0i, r1i);
  if constexpr (Variant == kClusterRows) {
    __shared__ ClusterMail mail;
    ResidentMatrix A;
    stageResident<false>(D, gs.rank, r0i, r1i, A);  // raises an error status where it does not fit
    if (threadIdx.x < 2) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sharedAddress(&mail.bar[threadIdx.x])) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __threadfence();
    clusterArrive();
    clusterWait();
    // An error of a kernel before, or of a block that did not fit: the same for every thread of the cluster, since none
    // raises one between the two barriers.
    const int error = *reinterpret_cast<volatile int*>(&D.ctl->error);
    clusterArrive();
    clusterWait();
    if (error != 0) return -1;
    const unsigned long long t0 = globalTimerNs();
    const int it = pcgCluster(D, gs, A, mail);
    if (gs.rank == 0 && threadIdx.x == 0) D.ctl->pcgNs += static_cast<long long>(globalTimerNs() - t0);
    return it;
  } else if constexpr (Variant > kResidentRows) {
    constexpr int kRows = Variant - kResidentRows;
    __shared__ MultiSlices sl;
    MultiMatrix A;
    if (!stageMulti<kRows>(D, gs.rank, r0i, r1i, A, sl)) return -1;
    const unsigned long long t0 = globalTimerNs();
    unsigned long long seq = __ldcg(D.mailSeq);
    const int it = pcgResidentMulti<kRows, PL == 0>(D, gs, A, sl, seq);
    if (gs.rank == 0 && threadIdx.x == 0) {
      *D.mailSeq = seq;
      D.ctl->pcgNs += static_cast<long long>(globalTimerNs() - t0);
    }
    return it;
  } else if constexpr (Variant == kResidentRows) {
    ResidentMatrix A;
    if (!stageResident<Learned>(D, gs.rank, r0i, r1i, A)) return -1;
    const unsigned long long t0 = globalTimerNs();
    unsigned long long seq = __ldcg(D.mailSeq);
    int it;
    if constexpr (Learned) {
      // The learned schedule without block-Jacobi iterations first (the host picks this kernel only then): a learned
      // solve that breaks down is followed by a full block-Jacobi solve, as in pcgSolveStaged.
      it = pcgLearnedResident(D, gs, A, seq);
      if (gs.rank == 0 && threadIdx.x == 0) D.ctl->learnedSolves += 1;
      if (it < -1) {
        if (gs.rank == 0 && threadIdx.x == 0) D.ctl->precondFallbacks += 1;
        // A block sends its r.z before it takes its halo of D.z, so a non-finite r.z ends the solve in a fast block while a
        // slower one still waits for z under the old tag: no new z may be published before every block is out.
        if (!gs.sync()) return -1;
        const int jac = pcgResident(D, gs, A, seq);
        it = jac < 0 ? jac : jac + (-2 - it);
      }
    } else {
      it = pcgResident(D, gs, A, seq);
    }
    // Every block has sent a message by now (or none has), so every block has read the number.
    if (gs.rank == 0 && threadIdx.x == 0) {
      *D.mailSeq = seq;
      D.ctl->pcgNs += static_cast<long long>(globalTimerNs() - t0);
    }
    return it;
  } else {
    const SmemMatrix A = stageMatrix(D, r0i, r1i);
    const unsigned long long t0 = globalTimerNs();
    const int it = pcgSolveStaged<Learned, PL, Variant>(D, gs, A);
    if (gs.rank == 0 && threadIdx.x == 0) D.ctl->pcgNs += static_cast<long long>(globalTimerNs() - t0);
    return it;
  }
}

template <bool Learned, int PL, int Variant>
__device__ inline int pcgSolveStaged(const Dev& D, GridSync& gs, const SmemMatrix& A) {
  if constexpr (!Learned) {
    if constexpr (Variant == 1) {
      return pcgPipelined<PL>(D, gs, A);
    } else if constexpr (Variant == 2) {
      return pcgSingleReduction<PL>(D, gs, A);
    } else {
      return pcgReferenceOrder<PL>(D, gs, A);
    }
  }
  int first = 0;
  double r0 = 0.0;
  const int sw = D.P.learnedSwitch;
  if (sw > 0) {
    bool finished = false;
    first = pcgReferenceOrder<PL>(D, gs, A, sw, &r0, &finished);
    if (first < 0 || finished || first >= D.P.maxCg) return first;
  }
  const int it = pcgLearned<PL>(D, gs, A, sw > 0, r0, D.P.maxCg - first);
  if (gs.rank == 0 && threadIdx.x == 0) D.ctl->learnedSolves += 1;
  if (it >= -1) return it < 0 ? it : first + it;
  if (gs.rank == 0 && threadIdx.x == 0) D.ctl->precondFallbacks += 1;
  const int jac = pcgReferenceOrder<PL>(D, gs, A);
  return jac < 0 ? jac : jac + first + (-2 - it);
}

// One Newton iteration's solve for the blocks of one group (the whole grid for one solver, or a garment's blocks in
// a batched launch); gs is initialised. PL: the scheme of the PCG's product A p (lanes per row, or 0 for
// slot-parallel; see directionProducts), also the lanes of the learned factor's products when positive.
template <bool Learned, int PL, int Variant = 0>
__device__ inline void solveGroup(const Dev& D, GridSync& gs) {
  Control* ctl = D.ctl;
  const uint32_t n = D.P.n;
  uint32_t r0i, r1i;
  blockRange(n, gs.rank, gs.size, r0i, r1i);
  const int it = pcgSolve<Learned, PL, Variant>(D, gs);
  if (it < 0) return;
  if (gs.rank == 0 && threadIdx.x == 0) {
    if (D.cgLog) D.cgLog[static_cast<unsigned long long>(ctl->newtonIterations) % kCgLogCapacity] = it;
    ctl->cgIterations += it;
    ctl->newtonIterations += 1;
    ctl->lastCg = it;
    ctl->energyEvaluations += 1;  // E(0) below
  }

  // The resident-row kernel's 512-thread blocks stand for the reference-order kernel's 1024-thread ones: its energies
  // are summed as two virtual threads per thread, in that kernel's order, so both kernels take the same line-search
  // decisions (its rows, at most 512 per block, already sit on the same threads).
  constexpr bool kVirtual = Variant >= kResidentRows;
  // Contact normal force from the residual (kernels.h:391-396), Newton slope grad . step and E(0), in FP64.
  double se[2];
  {
    double v[2] = {0.0, 0.0};
    for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
      const Contact c = D.contact[i];
      const float3 res = ld3(D.resid, i);
      D.contact[i].force = c.active != 0u ? fmaxf(0.0f, -dot(res, xyz(c.normal))) : 0.0f;
      v[0] += dotd3(ld3(D.grad, i), ld3(D.step, i));
    }
    if constexpr (kVirtual) {
      v[1] = energyPartial(D, gs, 0.0, threadIdx.x, 2 * blockDim.x);
      double hi[2] = {0.0, energyPartial(D, gs, 0.0, threadIdx.x + blockDim.x, 2 * blockDim.x)};
      if (!gridReducePairs<2>(D, gs, v, hi, se)) return;
    } else {
      v[1] = energyPartial(D, gs, 0.0);
      if (!gridReduce<2>(D, gs, v, se)) return;
    }
  }
  const double slope = se[0], e0 = se[1];
  if (!(slope < 0.0)) {
    if (gs.rank == 0 && threadIdx.x == 0) {
      ctl->newtonDone = 1;
      ctl->lastSlope = slope;
    }
    return;
  }
  // Backtracking line search, Armijo c = 1e-4, at most 20 halvings (cpu_solver.cpp:269-274).
  double alpha = 1.0;
  for (int ls = 0; ls < 20; ++ls) {
    if (gs.rank == 0 && threadIdx.x == 0) ctl->energyEvaluations += 1;
    double e[1];
    if constexpr (kVirtual) {
      double lo[1] = {energyPartial(D, gs, alpha, threadIdx.x, 2 * blockDim.x)};
      double hi[1] = {energyPartial(D, gs, alpha, threadIdx.x + blockDim.x, 2 * blockDim.x)};
      if (!gridReducePairs<1>(D, gs, lo, hi, e)) return;
    } else {
      double v[1] = {energyPartial(D, gs, alpha)};
      if (!gridReduce<1>(D, gs, v, e)) return;
    }
    if (e[0] <= e0 + 1e-4 * alpha * slope) break;
    alpha *= 0.5;
    if (gs.rank == 0 && threadIdx.x == 0) ctl->lineSearchHalvings += 1;
  }
  // Apply the step; max move; the next Newton iteration's friction uses this solve's forces (kernels.h:407-414).
  double mv[1] = {0.0};
  const float fa = static_cast<float>(alpha);
  for (uint32_t i = r0i + threadIdx.x; i < r1i; i += blockDim.x) {
    const float3 d = ld3(D.step, i) * fa;
    D.u[i] = f4(ld3(D.u, i) + d);
    mv[0] = fmax(mv[0], static_cast<double>(fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z)))));
    const Contact c = D.contact[i];
    D.contact[i].frictionLambda = c.active != 0u ? c.force : 0.0f;
  }
  double maxMove[1];
  if (!gridReduce<1, true>(D, gs, mv, maxMove)) return;
  if (gs.rank == 0 && threadIdx.x == 0) {
    ctl->lastAlpha = alpha;
    ctl->lastSlope = slope;
    ctl->lastE0 = e0;
    ctl->lastMaxMove = maxMove[0];
    if (maxMove[0] < 1e-9) ctl->newtonDone = 1;
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Finish: x = xStart + u, post-solve push-out below the snap tolerance, pins, damped velocity (kernels.h:419-448,
// cpu_solver.cpp:285-313); the assembly clock of Assembling garments advances by h.

__device__ inline void finishRows(const Dev& D, uint32_t rank, uint32_t size) {
  const float h = D.P.h;
  for (uint32_t i = rank * blockDim.x + threadIdx.x; i < D.P.n; i += size * blockDim.x) {
    const Particle pa = D.particle[i];
    const Fabric fab = D.fabric[pa.fabric];
    const float3 xs = ld3(D.xStart, i);
    float3 xn = xs + ld3(D.u, i);
    if (pa.pinned != 0u) {
      xn = ld3(D.pinPos, i);
    } else if (D.field.present) {
      const float radius = contactRadius(D.P, fab);
      if (fieldSample(D.fieldValues, D.field, xn) < radius - D.P.contactSnap) {
        if (isZero(fieldGradient(D.fieldValues, D.field, xn))) {
          xn = landOnBody(D.fieldValues, D.field, radius, xs, xn);
        } else {
          collideBody(D.fieldValues, D.field, radius, fab.friction, xs, xn);
        }
      }
    }
    float c = D.P.dampingScale * fab.damping;
    if (D.garment[pa.garment].phase == 0) c += D.P.assemblyExtraDamping;
    const float3 vel = div(xn - xs, h) * fmaxf(0.0f, 1.0f - c * h);
    D.x[i] = f4(xn);
    D.v[i] = f4(vel);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Statistics of one solver or one garment (sim_model.cpp:222-241), reduced on the device in FP64.

struct StatsOut {
  double kineticEnergy, sumV2, maxSeamGap, maxPenetration;
  unsigned long long moving;
  int nonFinite;
  int pad;
  unsigned long long beginNs, endNs;  // %globaltimer at the frame's first kernel and at its statistics' end
};

}  // namespace dcu

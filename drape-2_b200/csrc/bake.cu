// Collision-field bake (include/drape_bake.h): bakeCollisionField (libs/avatar/src/collision_bake.cpp:98-208) on the
// GPU. The reference walks triangles serially and keeps per sample the first triangle reaching the smallest squared
// distance; here blocks take chunks of the triangles' sample boxes and the choice is made in two passes with 64-bit atomics
// (the exact FP64 minimum, then the lowest triangle index reaching it), which is the same triangle. All double arithmetic is
// explicitly rounded in the reference's order (Ericson's closest point, RTCD 5.1.5; dot products summed left to
// right), so the field equals the serial algorithm's in FP64 rounded to float. Pseudonormals (face, angle-weighted
// vertex, edge sums) are computed on the host in the same order as the reference. The outside of the band is found
// by line sweeps along the six axis directions, repeated until nothing changes: the same set as the reference's
// breadth-first flood fill from the grid boundary.
//
// Each component works on its box alone, the union of its triangles' sample boxes: every sample out of it is farther than
// the band and joined to the grid's boundary along an axis, hence outside (+band, which the field starts with), and a far
// sample on the box's own faces is outside too. Components run together in one launch per pass, in groups whose boxes hold
// no more samples than the grid. On a five-component body at 4 mm (6,656 triangles, 7.8 M grid samples) the boxes hold
// 2.6 M samples where five passes over the grid visited 39 M; device time 4.93 -> 0.84 ms (three capsules 3.07 -> 0.63 ms,
// a sphere 0.31 -> 0.21 ms).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/drape_bake.h"
#include "../../include/drape_cuda.h"
#include "device_buffer.hpp"

using dbuf::check;
using dbuf::DBuf;
#define KCK(x) check((x), #x)

namespace bake {

struct D3 {
  double x, y, z;
};

// Explicitly rounded double operations (no contraction into fused multiply-adds).
__device__ __forceinline__ D3 sub(D3 a, D3 b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)}; }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

__device__ __forceinline__ double dot(D3 a, D3 b) { return add(add(mul(a.x, b.x), mul(a.y, b.y)), mul(a.z, b.z)); }
// a + s * v per component.
__device__ __forceinline__ D3 axpy(D3 a, double s, D3 v) {
  return {add(a.x, mul(s, v.x)), add(a.y, mul(s, v.y)), add(a.z, mul(s, v.z))};
}

enum Feature : int { kVertexA, kVertexB, kVertexC, kEdgeAB, kEdgeBC, kEdgeCA, kFace };

// Closest point on triangle abc to p and the feature it lies on (collision_bake.cpp:19-55).
__device__ inline D3 closestPoint(D3 p, D3 a, D3 b, D3 c, int& f) {
  const D3 ab = sub(b, a), ac = sub(c, a), ap = sub(p, a);
  const double d1 = dot(ab, ap), d2 = dot(ac, ap);
  if (d1 <= 0 && d2 <= 0) {
    f = kVertexA;
    return a;
  }
  const D3 bp = sub(p, b);
  const double d3 = dot(ab, bp), d4 = dot(ac, bp);
  if (d3 >= 0 && d4 <= d3) {
    f = kVertexB;
    return b;
  }
  const double vc = dsub(mul(d1, d4), mul(d3, d2));
  if (vc <= 0 && d1 >= 0 && d3 <= 0) {
    f = kEdgeAB;
    return axpy(a, ddiv(d1, dsub(d1, d3)), ab);
  }
  const D3 cp = sub(p, c);
  const double d5 = dot(ab, cp), d6 = dot(ac, cp);
  if (d6 >= 0 && d5 <= d6) {
    f = kVertexC;
    return c;
  }
  const double vb = dsub(mul(d5, d2), mul(d1, d6));
  if (vb <= 0 && d2 >= 0 && d6 <= 0) {
    f = kEdgeCA;
    return axpy(a, ddiv(d2, dsub(d2, d6)), ac);
  }
  const double va = dsub(mul(d3, d6), mul(d5, d4));
  const double e43 = dsub(d4, d3), e56 = dsub(d5, d6);
  if (va <= 0 && e43 >= 0 && e56 >= 0) {
    f = kEdgeBC;
    return axpy(b, ddiv(e43, add(e43, e56)), sub(c, b));
  }
  const double denom = ddiv(1.0, add(add(va, vb), vc));
  f = kFace;
  return axpy(axpy(a, mul(vb, denom), ab), mul(vc, denom), ac);
}

struct Grid {
  double ox, oy, oz, cell, band, band2;
  int nx, ny, nz;
};

// One component: its box in the grid (first sample, samples per axis), wx words of 32 samples along x, and where its
// samples and words start in the group's arrays.
struct Part {
  int x0, y0, z0, nx, ny, nz, wx;
  size_t at, word;
  __device__ size_t samples() const { return static_cast<size_t>(nx) * ny * nz; }
  __device__ size_t words() const { return static_cast<size_t>(wx) * ny * nz; }
};

// One block's share of a triangle's sample box: samples [sub * chunk, (sub + 1) * chunk) of it, in x, y, z order.
struct Task {
  uint32_t tri, part, sub;
};

struct Mesh {
  const D3* v;
  const uint3* t;
  const double* tbox;  // per triangle: tmin xyz, tmax xyz
  const double* tboxWide;  // the same, larger by 2^-48 of the largest coordinate (pass 2)
  const int* trange;   // per triangle: x0 x1 y0 y1 z0 z1 (sample box, inclusive)
  const D3* faceN;     // per triangle
  const D3* vertexN;   // per vertex
  const D3* edgeN;     // per triangle: AB, BC, CA
};

__device__ __forceinline__ D3 samplePos(const Grid& g, int x, int y, int z) {
  return {add(g.ox, mul(g.cell, static_cast<double>(x))), add(g.oy, mul(g.cell, static_cast<double>(y))),
          add(g.oz, mul(g.cell, static_cast<double>(z)))};
}

// Squared distance from p to a box, lower corner then upper (the reference's cheap reject, with the triangle's bounding box).
__device__ __forceinline__ double boxGap2(const double* tb, D3 p) {
  const double gx = fmax(fmax(dsub(tb[0], p.x), dsub(p.x, tb[3])), 0.0);
  const double gy = fmax(fmax(dsub(tb[1], p.y), dsub(p.y, tb[4])), 0.0);
  const double gz = fmax(fmax(dsub(tb[2], p.z), dsub(p.z, tb[5])), 0.0);
  return add(add(mul(gx, gx), mul(gy, gy)), mul(gz, gz));
}

constexpr int kBakeThreads = 256;
constexpr uint32_t kNoTriangle = 0xFFFFFFFFu;  // a sample without an owner (yet)

// Pass 1 (Owner = false): the smallest squared distance per sample up to the band's (atomic minimum on the double's bits;
// non-negative doubles order like their bit patterns; it starts at the first double beyond the band's square, which stands
// for every far sample). Pass 2 (Owner = true): the lowest triangle index reaching that minimum.
//
// The bounding box bounds the distance from below only in exact arithmetic: the computed closest point is a sum of two
// rounded products and can lie out of the box by a few roundings of its coordinates (a box at 1 m with the last bits of
// its vertices changed has such samples). Pass 1 rejects by the box as the reference does. Pass 2 has to see again every
// triangle that pass 1 took, so its box is larger by 2^-48 of the largest coordinate, some three times those roundings:
// the closest point lies in it, and rounded differences, squares and sums keep that order. The closest point of a
// triangle without area can lie anywhere; a sample whose owner is not found all the same gets 0 (k_bake_combine).
//
// What bounds it: FP64 issue of the closest points (up to three divides each, seven diverging regions). So a sample
// farther than the band, or than its best so far, is left by its distance from the triangle's bounding box, and a large
// box is shared by many blocks: with one block a triangle the largest boxes (150,000 samples) held up two components'
// passes by themselves. Pass 1 / pass 2 of the five-component body at 4 mm (32 M pairs of sample and triangle): 1,490 /
// 1,360 us in ten launches before, 331 / 325 us in two. Measured and dropped: a second bound from the triangle's plane and
// its reach from the centroid (478 / 402 us: its 15 FP64 operations cost more than the closest points that it saves).
template <bool Owner>
__global__ void __launch_bounds__(kBakeThreads) k_bake_distance(Grid g, Mesh m, const Part* parts, const Task* tasks,
                                                                uint32_t chunk, unsigned long long* dist2, uint32_t* owner) {
  const Task task = tasks[blockIdx.x];
  const Part part = parts[task.part];
  const int* r = m.trange + 6 * static_cast<size_t>(task.tri);
  const int bx = r[1] - r[0] + 1, by = r[3] - r[2] + 1, bz = r[5] - r[4] + 1;
  const uint3 tri = m.t[task.tri];
  const D3 a = m.v[tri.x], b = m.v[tri.y], c = m.v[tri.z];
  const double* tb = (Owner ? m.tboxWide : m.tbox) + 6 * static_cast<size_t>(task.tri);
  const uint32_t first = task.sub * chunk, last = min(first + chunk, static_cast<uint32_t>(bx) * by * bz);
  for (uint32_t s = first + threadIdx.x; s < last; s += kBakeThreads) {
    const uint32_t row = s / bx, slab = row / by;
    const int x = r[0] + static_cast<int>(s - row * bx), y = r[2] + static_cast<int>(row - slab * by),
              z = r[4] + static_cast<int>(slab);
    const size_t i = part.at + (static_cast<size_t>(z - part.z0) * part.ny + (y - part.y0)) * part.nx + (x - part.x0);
    const D3 p = samplePos(g, x, y, z);
    const double best = __longlong_as_double(static_cast<long long>(
        Owner ? dist2[i] : *reinterpret_cast<volatile unsigned long long*>(dist2 + i)));
    const double gap = boxGap2(tb, p);
    // Pass 1: no improvement possible when the box is already as far as the best; pass 2: only an exact tie with
    // the final minimum counts, and d2 >= gap.
    if (Owner ? gap > best : gap >= best) continue;
    int f;
    const D3 q = closestPoint(p, a, b, c, f);
    const D3 d = sub(p, q);
    const double d2 = dot(d, d);
    if (!Owner) {
      if (d2 < best) atomicMin(dist2 + i, static_cast<unsigned long long>(__double_as_longlong(d2)));
    } else if (d2 == best) {
      atomicMin(owner + i, task.tri);
    }
  }
}

// Flood-fill state, one bit a sample: far (farther than the band) and outside (a subset of far). Seeds: far samples on the
// faces of the component's box. One warp per word.
__global__ void k_bake_seed(Grid g, const Part* parts, const unsigned long long* dist2, uint32_t* far,
                            uint32_t* outside) {
  const Part part = parts[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const size_t words = part.words(), warps = static_cast<size_t>(gridDim.x) * (blockDim.x >> 5);
  for (size_t w = blockIdx.x * static_cast<size_t>(blockDim.x >> 5) + (threadIdx.x >> 5); w < words; w += warps) {
    const size_t row = w / part.wx;
    const int x = static_cast<int>(w - row * part.wx) * 32 + lane;
    const int y = static_cast<int>(row % part.ny), z = static_cast<int>(row / part.ny);
    const bool isFar = x < part.nx && __longlong_as_double(static_cast<long long>(
                                          dist2[part.at + row * part.nx + min(x, part.nx - 1)])) > g.band2;
    const bool face = x == 0 || y == 0 || z == 0 || x == part.nx - 1 || y == part.ny - 1 || z == part.nz - 1;
    const uint32_t F = __ballot_sync(0xffffffffu, isFar), O = __ballot_sync(0xffffffffu, isFar && face);
    if (lane == 0) {
      far[part.word + w] = F;
      outside[part.word + w] = O;
    }
  }
}

// Sweeps along one axis, in both directions: every line carries "outside" through consecutive far samples; sets *changed
// when it marks a sample. Along x a thread takes one line, a word at a time, F (far) and O (outside, a subset of F): with
// the carry c_in from the previous word, the sum F + O + c_in carries through exactly the far runs that hold a seed or
// continue the previous run, so the reached set is O | ((F + O + c_in) ^ F ^ O) & F and the carry out of bit 31 goes to
// the next word (backwards the same on reversed words). Along y and z a thread takes 32 lines at once, a word a step.
template <int Axis>
__global__ void k_bake_sweep(const Part* parts, const uint32_t* far, uint32_t* outside, int* changed) {
  const Part part = parts[blockIdx.y];
  constexpr int kDepth = 16;  // words loaded before the first is used
  const int len = Axis == 0 ? part.wx : Axis == 1 ? part.ny : part.nz;
  const size_t plane = static_cast<size_t>(part.wx) * part.ny;
  const size_t step = Axis == 0 ? 1 : Axis == 1 ? part.wx : plane;
  const size_t lines = Axis == 0 ? static_cast<size_t>(part.ny) * part.nz
                                 : Axis == 1 ? static_cast<size_t>(part.wx) * part.nz : plane;
  bool marked = false;
  for (size_t l = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; l < lines;
       l += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t base = part.word + (Axis == 0 ? l * part.wx : Axis == 1 ? l / part.wx * plane + l % part.wx : l);
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      uint32_t carry = 0;
      for (int s0 = 0; s0 < len; s0 += kDepth) {
        uint32_t F[kDepth], O[kDepth];
#pragma unroll
        for (int e = 0; e < kDepth; ++e) {
          const int s = dir ? len - 1 - s0 - e : s0 + e;
          const bool in = s0 + e < len;
          F[e] = in ? far[base + s * step] : 0;
          O[e] = in ? outside[base + s * step] : 0;
        }
#pragma unroll
        for (int e = 0; e < kDepth; ++e) {
          uint32_t reached;
          if (Axis == 0) {
            const uint32_t f = dir ? __brev(F[e]) : F[e], o = dir ? __brev(O[e]) : O[e];
            const unsigned long long sum = static_cast<unsigned long long>(f) + o + carry;
            reached = o | ((static_cast<uint32_t>(sum) ^ f ^ o) & f);
            carry = static_cast<uint32_t>(sum >> 32);
            if (dir) reached = __brev(reached);
          } else {
            reached = carry = O[e] | (carry & F[e]);
          }
          if (reached & ~O[e]) {
            marked = true;
            outside[base + (dir ? len - 1 - s0 - e : s0 + e) * step] = reached;
          }
        }
      }
    }
  }
  if (marked) *changed = 1;
}

// Combine a component into the field (collision_bake.cpp:196-204): the sign of a sample within the band from the
// pseudonormal of the nearest feature of its triangle, -band for the others that the flood did not reach. Samples that it
// reached keep what they have: the field starts at +band.
__global__ void k_bake_combine(Grid g, Mesh m, const Part* parts, int which, const unsigned long long* dist2,
                               const uint32_t* owner, const uint32_t* outside, float* values) {
  const Part part = parts[which];
  const size_t count = part.samples();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t row = i / part.nx;
    const int lx = static_cast<int>(i - row * part.nx);
    const int x = part.x0 + lx, y = part.y0 + static_cast<int>(row % part.ny), z = part.z0 + static_cast<int>(row / part.ny);
    const double d2 = __longlong_as_double(static_cast<long long>(dist2[part.at + i]));
    const bool near = d2 <= g.band2;
    const uint32_t t = near ? owner[part.at + i] : kNoTriangle;
    double v;
    if (t != kNoTriangle) {
      const D3 p = samplePos(g, x, y, z);
      const uint3 tri = m.t[t];
      int f;
      const D3 q = closestPoint(p, m.v[tri.x], m.v[tri.y], m.v[tri.z], f);
      D3 n;
      switch (f) {
        case kVertexA: n = m.vertexN[tri.x]; break;
        case kVertexB: n = m.vertexN[tri.y]; break;
        case kVertexC: n = m.vertexN[tri.z]; break;
        case kEdgeAB: n = m.edgeN[3 * static_cast<size_t>(t)]; break;
        case kEdgeBC: n = m.edgeN[3 * static_cast<size_t>(t) + 1]; break;
        case kEdgeCA: n = m.edgeN[3 * static_cast<size_t>(t) + 2]; break;
        default: n = m.faceN[t]; break;
      }
      v = (dot(sub(p, q), n) >= 0 ? 1.0 : -1.0) * __dsqrt_rn(d2);
    } else if (near) {
      v = 0.0;
    } else {
      if (outside[part.word + row * part.wx + (lx >> 5)] >> (lx & 31) & 1u) continue;
      v = -g.band;
    }
    v = fmin(fmax(v, -g.band), g.band);
    float* at = values + (static_cast<size_t>(z) * g.ny + y) * g.nx + x;
    *at = fminf(*at, __double2float_rn(v));
  }
}

__global__ void k_fill(float* values, size_t count, float v) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    values[i] = v;
}

__global__ void k_reset(Grid g, unsigned long long* dist2, uint32_t* owner, size_t count) {
  // The first double beyond the band's square; where that overflowed nothing lies beyond.
  const unsigned long long start =
      static_cast<unsigned long long>(__double_as_longlong(g.band2)) + (isinf(g.band2) ? 0ull : 1ull);
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    dist2[i] = start;
    owner[i] = kNoTriangle;
  }
}

}  // namespace bake

namespace {

thread_local std::string g_bakeError;
thread_local double g_bakeMs = 0.0;

using bake::D3;

D3 vtx(const drape_mesh_desc& m, uint32_t i) { return {m.vertices[3 * i], m.vertices[3 * i + 1], m.vertices[3 * i + 2]}; }
D3 hsub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
double hdot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
D3 hcross(D3 a, D3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
// Eigen's normalized(): divide by the norm when the squared norm is positive.
D3 hnormalized(D3 a) {
  const double z = hdot(a, a);
  if (!(z > 0)) return a;
  const double s = std::sqrt(z);
  return {a.x / s, a.y / s, a.z / s};
}

// isClosedManifold (libs/core/src/triangle_mesh.cpp:16-28): every directed edge once, and its reverse once.
bool closedManifold(const drape_mesh_desc& m) {
  if (m.triangle_count == 0) return false;
  std::vector<uint64_t> e;
  e.reserve(3ull * m.triangle_count);
  for (uint32_t t = 0; t < m.triangle_count; ++t)
    for (int k = 0; k < 3; ++k)
      e.push_back(static_cast<uint64_t>(m.triangles[3 * t + k]) << 32 | m.triangles[3 * t + (k + 1) % 3]);
  std::sort(e.begin(), e.end());
  for (size_t i = 1; i < e.size(); ++i)
    if (e[i] == e[i - 1]) return false;
  for (uint64_t x : e) {
    const uint64_t rev = (x << 32) | (x >> 32);
    if (!std::binary_search(e.begin(), e.end(), rev)) return false;
  }
  return true;
}

void validate(const drape_mesh_desc* components, uint32_t count, const drape_bake_options* o) {
  if (!components || count == 0) throw std::invalid_argument("no collision components");
  if (!o || !(o->cell_size > 0) || !(o->band > 0) || !(o->padding >= 0))
    throw std::invalid_argument("bake options need cell_size > 0, band > 0, padding >= 0");
  for (uint32_t c = 0; c < count; ++c) {
    const drape_mesh_desc& m = components[c];
    if (!m.vertices || !m.triangles) throw std::invalid_argument("null mesh arrays");
    for (size_t k = 0; k < 3ull * m.triangle_count; ++k)
      if (m.triangles[k] >= m.vertex_count) throw std::invalid_argument("triangle vertex index out of range");
    if (!closedManifold(m))
      throw std::invalid_argument("collision component " + std::to_string(c) + " is not a closed manifold");
  }
}

// Grid of the bake (collision_bake.cpp:99-117).
void gridOf(const drape_mesh_desc* components, uint32_t count, const drape_bake_options& o, double origin[3],
            int dims[3]) {
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t c = 0; c < count; ++c)
    for (uint32_t i = 0; i < components[c].vertex_count; ++i)
      for (int a = 0; a < 3; ++a) {
        lo[a] = std::min(lo[a], components[c].vertices[3 * i + a]);
        hi[a] = std::max(hi[a], components[c].vertices[3 * i + a]);
      }
  for (int a = 0; a < 3; ++a) {
    origin[a] = lo[a] - o.padding;
    const double extent = (hi[a] - lo[a]) + 2 * o.padding;
    dims[a] = static_cast<int>(std::ceil(extent / o.cell_size)) + 1;
  }
}

}  // namespace

extern "C" {

int drape_bake_grid(const drape_mesh_desc* components, uint32_t count, const drape_bake_options* options,
                    double origin[3], int32_t dims[3]) {
  try {
    validate(components, count, options);
    if (!origin || !dims) throw std::invalid_argument("null argument");
    int d[3];
    gridOf(components, count, *options, origin, d);
    for (int a = 0; a < 3; ++a) dims[a] = d[a];
    return DRAPE_OK;
  } catch (const std::invalid_argument& e) {
    g_bakeError = e.what();
    return DRAPE_INVALID;
  } catch (const std::exception& e) {
    g_bakeError = e.what();
    return DRAPE_DEVICE_ERROR;
  }
}

int drape_bake_field(int device, const drape_mesh_desc* components, uint32_t count, const drape_bake_options* options,
                     float* values, size_t value_count) {
  try {
    validate(components, count, options);
    const drape_bake_options& o = *options;
    double origin[3];
    int dims[3];
    gridOf(components, count, o, origin, dims);
    const size_t total = static_cast<size_t>(dims[0]) * dims[1] * dims[2];
    if (!values || value_count != total) throw std::invalid_argument("values must hold dims[0] * dims[1] * dims[2]");
    int devices = 0;
    KCK(cudaGetDeviceCount(&devices));
    if (device < 0 || device >= devices) throw std::runtime_error("cuda: no device " + std::to_string(device));
    KCK(cudaSetDevice(device));
    cudaStream_t st;
    KCK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    cudaEvent_t e0, e1;
    KCK(cudaEventCreate(&e0));
    KCK(cudaEventCreate(&e1));
    struct Cleanup {
      cudaStream_t s;
      cudaEvent_t a, b;
      ~Cleanup() {
        cudaStreamSynchronize(s);
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        cudaStreamDestroy(s);
      }
    } cleanup{st, e0, e1};
    int sms = 0;
    KCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    bake::Grid g{origin[0], origin[1], origin[2], o.cell_size, o.band, o.band * o.band, dims[0], dims[1], dims[2]};
    const int pointGrid = sms * 8;
    // Host preparation of every component first (boxes, sample ranges, pseudonormals), in arrays of all components'
    // vertices and triangles one after another, then the device work.
    size_t allV = 0, allT = 0;
    for (uint32_t c = 0; c < count; ++c) {
      allV += components[c].vertex_count;
      allT += components[c].triangle_count;
    }
    std::vector<D3> v, faceN, vertexN(allV, D3{0, 0, 0}), edgeN(3 * allT);
    std::vector<uint3> tris;
    std::vector<double> tbox(6 * allT), tboxWide(6 * allT);
    std::vector<int> trange(6 * allT);
    v.reserve(allV);
    faceN.reserve(allT);
    tris.reserve(allT);
    for (uint32_t c = 0; c < count; ++c) {
      const drape_mesh_desc& m = components[c];
      // Host: vertices, triangles, boxes and sample ranges, pseudonormals (collision_bake.cpp:57-95).
      const uint32_t nv = m.vertex_count, nt = m.triangle_count;
      const uint32_t v0 = static_cast<uint32_t>(v.size());
      const size_t t0 = tris.size();
      for (uint32_t i = 0; i < nv; ++i) v.push_back(vtx(m, i));
      std::vector<std::pair<uint64_t, D3>> edgeSum;  // (min, max) vertex pair -> sum of face normals
      edgeSum.reserve(3ull * nt);
      auto edgeKey = [](uint32_t a, uint32_t b) {
        return static_cast<uint64_t>(std::min(a, b)) << 32 | std::max(a, b);
      };
      for (uint32_t t = 0; t < nt; ++t) {
        const uint32_t* tr = m.triangles + 3ull * t;
        tris.push_back(make_uint3(v0 + tr[0], v0 + tr[1], v0 + tr[2]));
        const D3 a = v[v0 + tr[0]], b = v[v0 + tr[1]], c3 = v[v0 + tr[2]];
        const D3 fn = hnormalized(hcross(hsub(b, a), hsub(c3, a)));
        faceN.push_back(fn);
        for (int k = 0; k < 3; ++k) {
          const D3 p = v[v0 + tr[k]];
          const D3 e1 = hnormalized(hsub(v[v0 + tr[(k + 1) % 3]], p));
          const D3 e2 = hnormalized(hsub(v[v0 + tr[(k + 2) % 3]], p));
          const double ang = std::acos(std::clamp(hdot(e1, e2), -1.0, 1.0));
          D3& vn = vertexN[v0 + tr[k]];
          vn = {vn.x + ang * fn.x, vn.y + ang * fn.y, vn.z + ang * fn.z};
          edgeSum.push_back({edgeKey(tr[k], tr[(k + 1) % 3]), fn});
        }
        const double mn[3] = {std::min(std::min(a.x, b.x), c3.x), std::min(std::min(a.y, b.y), c3.y),
                              std::min(std::min(a.z, b.z), c3.z)};
        const double mx[3] = {std::max(std::max(a.x, b.x), c3.x), std::max(std::max(a.y, b.y), c3.y),
                              std::max(std::max(a.z, b.z), c3.z)};
        double most = 0.0;
        for (int a3 = 0; a3 < 3; ++a3) most = std::max({most, std::fabs(mn[a3]), std::fabs(mx[a3])});
        for (int a3 = 0; a3 < 3; ++a3) {
          tbox[6 * (t0 + t) + a3] = mn[a3];
          tbox[6 * (t0 + t) + 3 + a3] = mx[a3];
          tboxWide[6 * (t0 + t) + a3] = mn[a3] - 0x1p-48 * most;
          tboxWide[6 * (t0 + t) + 3 + a3] = mx[a3] + 0x1p-48 * most;
          const double oa = origin[a3];
          const double i0 = std::max(0.0, std::ceil(((mn[a3] - o.band) - oa) / o.cell_size));
          const double i1 = std::min<double>(dims[a3] - 1, std::floor(((mx[a3] + o.band) - oa) / o.cell_size));
          trange[6 * (t0 + t) + 2 * a3] = static_cast<int>(i0);
          trange[6 * (t0 + t) + 2 * a3 + 1] = static_cast<int>(i1);
        }
      }
      // Edge pseudonormals: the two faces' normals summed in triangle order (the reference's map accumulation).
      std::stable_sort(edgeSum.begin(), edgeSum.end(),
                       [](const auto& x, const auto& y) { return x.first < y.first; });
      std::vector<uint64_t> keys(edgeSum.size());
      std::vector<D3> sums(edgeSum.size());
      size_t u = 0;
      for (size_t i = 0; i < edgeSum.size(); ++i) {
        if (i > 0 && edgeSum[i].first == edgeSum[i - 1].first) {
          D3& s = sums[u - 1];
          s = {s.x + edgeSum[i].second.x, s.y + edgeSum[i].second.y, s.z + edgeSum[i].second.z};
        } else {
          keys[u] = edgeSum[i].first;
          sums[u] = {0.0 + edgeSum[i].second.x, 0.0 + edgeSum[i].second.y, 0.0 + edgeSum[i].second.z};
          ++u;
        }
      }
      keys.resize(u);
      for (uint32_t t = 0; t < nt; ++t)
        for (int k = 0; k < 3; ++k) {  // edges AB, BC, CA
          const uint64_t key = edgeKey(m.triangles[3ull * t + k], m.triangles[3ull * t + (k + 1) % 3]);
          edgeN[3 * (t0 + t) + k] = sums[std::lower_bound(keys.begin(), keys.end(), key) - keys.begin()];
        }
    }
    // Each component's box, the groups of components that run together (no more samples than the grid has, which one box
    // alone never exceeds), and the groups' tasks: chunks of 2,048 samples, larger where that would make more than 2^18
    // tasks besides one a triangle. The host writes and uploads every task: a sphere of 5,120 triangles with boxes of
    // 500,000 samples took 35-38 ms with 2^20 tasks, 29 with 2^18, 27 with 2^16 (32 with one block a triangle); 200 spheres
    // with as wide a band 52, 48 and 52.
    std::vector<bake::Part> parts;
    std::vector<size_t> partTri;  // parts[k]'s triangles are [partTri[2 k], partTri[2 k + 1])
    size_t pairs = 0;
    auto samplesOf = [&](size_t t) {
      const int* r = &trange[6 * t];
      const int bx = r[1] - r[0] + 1, by = r[3] - r[2] + 1, bz = r[5] - r[4] + 1;
      return bx <= 0 || by <= 0 || bz <= 0 ? size_t{0} : static_cast<size_t>(bx) * by * bz;
    };
    for (size_t c = 0, t0 = 0; c < count; t0 += components[c++].triangle_count) {
      int lo[3] = {dims[0], dims[1], dims[2]}, hi[3] = {-1, -1, -1};
      const size_t t1 = t0 + components[c].triangle_count;
      for (size_t t = t0; t < t1; ++t) {
        if (!samplesOf(t)) continue;
        pairs += samplesOf(t);
        for (int a = 0; a < 3; ++a) {
          lo[a] = std::min(lo[a], trange[6 * t + 2 * a]);
          hi[a] = std::max(hi[a], trange[6 * t + 2 * a + 1]);
        }
      }
      if (hi[0] < 0) continue;  // no sample near it: all of the grid is outside
      const int nx = hi[0] - lo[0] + 1;
      parts.push_back({lo[0], lo[1], lo[2], nx, hi[1] - lo[1] + 1, hi[2] - lo[2] + 1, (nx + 31) / 32, 0, 0});
      partTri.insert(partTri.end(), {t0, t1});
    }
    const size_t chunk = std::max<size_t>(2048, (pairs >> 18) + 1);
    struct Group {
      size_t part0, part1, task0, task1, samples, lines;
    };
    std::vector<Group> groups;
    std::vector<bake::Task> tasks;
    size_t mostSamples = 0, mostWords = 0;
    for (size_t k = 0, words = 0; k < parts.size(); ++k) {
      bake::Part& pt = parts[k];
      const size_t rows = static_cast<size_t>(pt.ny) * pt.nz, own = rows * pt.nx;
      if (groups.empty() || groups.back().samples + own > total || k - groups.back().part0 >= 65535) {
        groups.push_back({k, k, tasks.size(), tasks.size(), 0, 0});
        words = 0;
      }
      Group& gr = groups.back();
      pt.at = gr.samples;
      pt.word = words;
      for (size_t t = partTri[2 * k]; t < partTri[2 * k + 1]; ++t)
        for (size_t n = samplesOf(t), sub = 0; sub * chunk < n; ++sub)
          tasks.push_back({static_cast<uint32_t>(t), static_cast<uint32_t>(k - gr.part0), static_cast<uint32_t>(sub)});
      gr.samples += own;
      words += rows * pt.wx;
      gr.lines = std::max({gr.lines, rows, static_cast<size_t>(pt.wx) * std::max(pt.ny, pt.nz)});
      gr.part1 = k + 1;
      gr.task1 = tasks.size();
      mostSamples = std::max(mostSamples, gr.samples);
      mostWords = std::max(mostWords, words);
    }
    DBuf<D3> dv, dface, dvert, dedge;
    DBuf<uint3> dtri;
    DBuf<double> dbox, dboxWide;
    DBuf<int> drange, changed;
    DBuf<bake::Part> dparts;
    DBuf<bake::Task> dtasks;
    DBuf<unsigned long long> dist2;
    DBuf<uint32_t> owner, far, outside;
    DBuf<float> field;
    field.alloc(total);
    if (!parts.empty()) {
      dv.upload(v, st);
      dface.upload(faceN, st);
      dvert.upload(vertexN, st);
      dedge.upload(edgeN, st);
      dtri.upload(tris, st);
      dbox.upload(tbox, st);
      dboxWide.upload(tboxWide, st);
      drange.upload(trange, st);
      dparts.upload(parts, st);
      dtasks.upload(tasks, st);
      dist2.alloc(mostSamples);
      owner.alloc(mostSamples);
      far.alloc(mostWords);
      outside.alloc(mostWords);
      changed.alloc(2);
    }
    const bake::Mesh dm{dv.p, dtri.p, dbox.p, dboxWide.p, drange.p, dface.p, dvert.p, dedge.p};
    KCK(cudaStreamSynchronize(st));  // the uploads' host arrays may go
    KCK(cudaEventRecord(e0, st));
    bake::k_fill<<<pointGrid, 256, 0, st>>>(field.p, total, static_cast<float>(o.band));
    KCK(cudaGetLastError());
    for (const Group& gr : groups) {
      const bake::Part* gp = dparts.p + gr.part0;
      const bake::Task* gt = dtasks.p + gr.task0;
      const uint32_t np = static_cast<uint32_t>(gr.part1 - gr.part0), nt = static_cast<uint32_t>(gr.task1 - gr.task0);
      const uint32_t step = static_cast<uint32_t>(chunk);
      bake::k_reset<<<pointGrid, 256, 0, st>>>(g, dist2.p, owner.p, gr.samples);
      bake::k_bake_distance<false><<<nt, bake::kBakeThreads, 0, st>>>(g, dm, gp, gt, step, dist2.p, owner.p);
      bake::k_bake_distance<true><<<nt, bake::kBakeThreads, 0, st>>>(g, dm, gp, gt, step, dist2.p, owner.p);
      const uint32_t share = std::max(1u, static_cast<uint32_t>(pointGrid) / np);
      bake::k_bake_seed<<<dim3(share, np), 256, 0, st>>>(g, gp, dist2.p, far.p, outside.p);
      KCK(cudaGetLastError());
      // Rounds of sweeps until one marks nothing (bounded by the number of samples, which is never reached), two a host
      // wait: most bodies are done after the first.
      const uint32_t lines = static_cast<uint32_t>(std::min<size_t>((gr.lines + 63) / 64, static_cast<size_t>(sms) * 8));
      for (size_t round = 0; round < gr.samples; round += 2) {
        KCK(cudaMemsetAsync(changed.p, 0, 2 * sizeof(int), st));
        for (int k = 0; k < 2; ++k) {
          bake::k_bake_sweep<0><<<dim3(lines, np), 64, 0, st>>>(gp, far.p, outside.p, changed.p + k);
          bake::k_bake_sweep<1><<<dim3(lines, np), 64, 0, st>>>(gp, far.p, outside.p, changed.p + k);
          bake::k_bake_sweep<2><<<dim3(lines, np), 64, 0, st>>>(gp, far.p, outside.p, changed.p + k);
        }
        KCK(cudaGetLastError());
        int h[2] = {0, 0};
        KCK(cudaMemcpyAsync(h, changed.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        KCK(cudaStreamSynchronize(st));
        if (!h[1]) break;
      }
      for (uint32_t k = 0; k < np; ++k)
        bake::k_bake_combine<<<pointGrid, 256, 0, st>>>(g, dm, gp, static_cast<int>(k), dist2.p, owner.p, outside.p,
                                                        field.p);
      KCK(cudaGetLastError());
    }
    KCK(cudaEventRecord(e1, st));
    KCK(cudaMemcpyAsync(values, field.p, sizeof(float) * total, cudaMemcpyDeviceToHost, st));
    KCK(cudaStreamSynchronize(st));
    float ms = 0;
    KCK(cudaEventElapsedTime(&ms, e0, e1));
    g_bakeMs = ms;
    return DRAPE_OK;
  } catch (const std::invalid_argument& e) {
    g_bakeError = e.what();
    return DRAPE_INVALID;
  } catch (const std::exception& e) {
    g_bakeError = e.what();
    return DRAPE_DEVICE_ERROR;
  }
}

double drape_bake_last_ms(void) { return g_bakeMs; }

const char* drape_bake_last_error(void) { return g_bakeError.c_str(); }

}  // extern "C"

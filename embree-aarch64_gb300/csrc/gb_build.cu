// gb_build.cu -- GPU BVH builder behind rtcCommitScene.
//
// Replaces the reference's CPU binned-SAH builder (kernels/bvh/bvh_builder_sah.cpp:111-189,
// kernels/builders/bvh_builder_sah.h:222-319) with a GPU pipeline:
//   1. primrefs: per-triangle validity + AABB, scene and centroid bounds
//      (validity rule of kernels/common/scene_triangle_mesh.h:127-147)
//   2. Morton codes of the centroids, 30 bits (10 per axis) or 63
//   3. stable LSD radix sort of (code, primref index), 8-bit digits; passes
//      whose digit is constant over all keys are skipped.  Stable sorting by
//      key with the index as value gives exactly std::stable_sort's order.
//   4. PLOC agglomerative clustering (nearest neighbour by merged-box surface
//      area among the clusters on either side, mutual pairs merge; with
//      gpu.ploc_radius within up to +-16) -> binary tree
//   5. top-down collapse into 8-wide nodes of the least surface-area cost for that
//      binary tree (gpu.collapse=greedy: largest-area child opened first), child
//      boxes quantised to 8 bits per plane, children placed in slots
//      so that the ray's direction octant gives a near-to-far visiting order,
//      leaves of <= 4 triangles written as v0/e1/e2 records.
// Everything is deterministic: the same input gives the same bytes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

#include "gb_build.h"
#include "gb_common.h"
#include "gb_launch.h"

namespace gb {

#define GB_CHECK(x)                                \
  do {                                             \
    cudaError_t e_ = (x);                          \
    if (e_ != cudaSuccess) return e_;              \
  } while (0)

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t f2ord(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float ord2f(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
#else
  uint32_t b = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}

struct BoundsAcc {
  uint32_t glo[3], ghi[3];  // ordered-uint min/max of geometry bounds
  uint32_t clo[3], chi[3];  // of centroids
  uint32_t nvalid;
  uint32_t pad;
  unsigned long long kand, kor;
};

__device__ __forceinline__ float half_area(float3 lo, float3 hi) {
  const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
  return dx * (dy + dz) + dy * dz;
}

__device__ __forceinline__ float3 f3min(float3 a, float3 b) {
  return make_float3(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z));
}
__device__ __forceinline__ float3 f3max(float3 a, float3 b) {
  return make_float3(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z));
}

// ---------------------------------------------------------------------------
// 1. primrefs
// ---------------------------------------------------------------------------

constexpr float kFltLarge = 1.844E18f;  // common/math/constants.h:34

__device__ __forceinline__ bool vtx_ok(float x, float y, float z) {
  return x > -kFltLarge && x < kFltLarge && y > -kFltLarge && y < kFltLarge && z > -kFltLarge && z < kFltLarge;
}

__device__ __forceinline__ float3 load_vtx(const GeomDesc& g, uint32_t i) {
  const float* p = reinterpret_cast<const float*>(g.verts + (uint64_t)i * g.vstride);
  return make_float3(p[0], p[1], p[2]);
}

__device__ __forceinline__ uint3 load_tri(const GeomDesc& g, uint32_t j) {
  const uint32_t* p = reinterpret_cast<const uint32_t*>(g.idx + (uint64_t)j * g.istride);
  return make_uint3(p[0], p[1], p[2]);
}

__device__ __forceinline__ int find_geom(const GeomDesc* geoms, int ngeoms, uint32_t gi) {
  int lo = 0, hi = ngeoms - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (geoms[mid].prim_offset <= gi) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// pbox[2i] = (lo.xyz, geometry slot), pbox[2i + 1] = (hi.xyz, primID); invalid
// triangles get an empty box (+inf,-inf).  prec[i] (when non-null) receives
// primitive i's leaf record -- Triangle4 values v0, e1 = v0 - v1, e2 = v2 - v0
// (triangle.h:40-41), or v0, v1, v2 in robust scenes (trianglev.h:93-115), or
// an instance leaf -- read here in primitive order, where the vertex reads
// coalesce, so that the leaf writer later gathers one 48-byte record per leaf.
// Grid-stride: the bounds and the valid count are reduced per thread, per warp
// and per CTA, so the global atomics are 13 per CTA (a grid of a few CTAs per SM).
__global__ void __launch_bounds__(256) k_primrefs(const GeomDesc* __restrict__ geoms, int ngeoms, uint32_t total,
                                                  float4* __restrict__ pbox, BoundsAcc* acc, TriRecord* __restrict__ prec, int robust) {
  __shared__ uint32_t s_b[12];
  __shared__ uint32_t s_cnt;
  if (threadIdx.x < 12) s_b[threadIdx.x] = (threadIdx.x % 6) < 3 ? 0xFFFFFFFFu : 0u;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  float v[12];
#pragma unroll
  for (int k = 0; k < 12; k++) v[k] = (k % 6) < 3 ? INFINITY : -INFINITY;
  unsigned nok = 0;
  for (uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x; gi < total; gi += gridDim.x * blockDim.x) {
    bool ok = false;
    float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
    {
      const int gs = find_geom(geoms, ngeoms, gi);
      const GeomDesc g = geoms[gs];
      const uint32_t j = gi - g.prim_offset;
      if (g.kind == 1) {
        const InstBox bx = reinterpret_cast<const InstBox*>(g.verts)[j];
        if (vtx_ok(bx.lo[0], bx.lo[1], bx.lo[2]) && vtx_ok(bx.hi[0], bx.hi[1], bx.hi[2]) && bx.lo[0] <= bx.hi[0] &&
            bx.lo[1] <= bx.hi[1] && bx.lo[2] <= bx.hi[2]) {
          ok = true;
          lo = make_float3(bx.lo[0], bx.lo[1], bx.lo[2]);
          hi = make_float3(bx.hi[0], bx.hi[1], bx.hi[2]);
        }
        if (prec)
          prec[gi] = TriRecord{make_float4(0.f, 0.f, 0.f, __uint_as_float(bx.inst)),
                               make_float4(0.f, 0.f, 0.f, __uint_as_float(bx.geomID)),
                               make_float4(0.f, 0.f, 0.f, __uint_as_float(kInstanceLeaf))};
      } else {
      const uint3 t = load_tri(g, j);
      if (t.x < g.nverts && t.y < g.nverts && t.z < g.nverts) {
        const float3 a = load_vtx(g, t.x), b = load_vtx(g, t.y), c = load_vtx(g, t.z);
        if (vtx_ok(a.x, a.y, a.z) && vtx_ok(b.x, b.y, b.z) && vtx_ok(c.x, c.y, c.z)) {
          ok = true;
          lo = f3min(f3min(a, b), c);
          hi = f3max(f3max(a, b), c);
          if (prec) {
            const float3 e1 = robust ? b : make_float3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
            const float3 e2 = robust ? c : make_float3(__fsub_rn(c.x, a.x), __fsub_rn(c.y, a.y), __fsub_rn(c.z, a.z));
            prec[gi] = TriRecord{make_float4(a.x, a.y, a.z, __uint_as_float(j)),
                                 make_float4(e1.x, e1.y, e1.z, __uint_as_float(g.geomID)),
                                 make_float4(e2.x, e2.y, e2.z, 0.f)};
          }
        }
      }
      }
      pbox[2 * (size_t)gi] = make_float4(lo.x, lo.y, lo.z, __uint_as_float((uint32_t)gs));
      pbox[2 * (size_t)gi + 1] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(j));
    }
    v[0] = fminf(v[0], lo.x); v[1] = fminf(v[1], lo.y); v[2] = fminf(v[2], lo.z);
    v[3] = fmaxf(v[3], hi.x); v[4] = fmaxf(v[4], hi.y); v[5] = fmaxf(v[5], hi.z);
    if (ok) {
      const float3 c = make_float3((lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f);
      v[6] = fminf(v[6], c.x); v[7] = fminf(v[7], c.y); v[8] = fminf(v[8], c.z);
      v[9] = fmaxf(v[9], c.x); v[10] = fmaxf(v[10], c.y); v[11] = fmaxf(v[11], c.z);
      nok++;
    }
  }
  // warp-reduce bounds then shared atomics
#pragma unroll
  for (int k = 0; k < 12; k++) {
    float x = v[k];
    const bool isMin = (k % 6) < 3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float y = __shfl_xor_sync(0xFFFFFFFFu, x, o);
      x = isMin ? fminf(x, y) : fmaxf(x, y);
    }
    v[k] = x;
  }
  nok = __reduce_add_sync(0xFFFFFFFFu, nok);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 12; k++) {
      if ((k % 6) < 3) atomicMin(&s_b[k], f2ord(v[k]));
      else atomicMax(&s_b[k], f2ord(v[k]));
    }
    atomicAdd(&s_cnt, nok);
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int k = threadIdx.x;
    uint32_t* dst = (k < 3) ? &acc->glo[k] : (k < 6) ? &acc->ghi[k - 3] : (k < 9) ? &acc->clo[k - 6] : &acc->chi[k - 9];
    if ((k % 6) < 3) atomicMin(dst, s_b[k]); else atomicMax(dst, s_b[k]);
  }
  if (threadIdx.x == 0) atomicAdd(&acc->nvalid, s_cnt);
}

// ---------------------------------------------------------------------------
// 2. Morton codes
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint64_t spread21(uint32_t x) {
  uint64_t v = x & 0x1FFFFFu;
  v = (v | (v << 32)) & 0x1F00000000FFFFull;
  v = (v | (v << 16)) & 0x1F0000FF0000FFull;
  v = (v | (v << 8)) & 0x100F00F00F00F00Full;
  v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}

__device__ __forceinline__ uint32_t spread10(uint32_t x) {
  uint32_t v = x & 0x3FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// Segmented builds put the geometry slot (< kMaxSegments) in the key's top 12
// bits, so the sort groups every geometry's primitives.
// bits30 (gpu.morton_bits=30): 10 bits per axis, the lattice of the reference's
// Morton builder (kernels/builders/bvh_builder_morton.h:62-86, LATTICE_BITS_PER_DIM
// 10), so valid keys fit in 30 bits (42 with the slot) and the sort needs 4 (6)
// digit passes instead of 8; invalid primitives get bit 30 (42) set, above every
// valid key, so they sort after all valid ones.  With at most kFewSegments slots all
// keys fit in 40 bits, the invalid ones as 40 set bits (a slot that none has), and the
// sort needs 5 passes (1.8M triangles of 128 scenes: 139 us, with 6 160).  key32: the
// 30-bit keys of an unsegmented build are written as 32-bit words (the sort then moves
// 4-byte keys).  nseg: geometries of a segmented build, else 0.
constexpr uint32_t kMaxSegments = 4096, kFewSegments = 1023;

// Grid-stride; the AND / OR of all keys (constant digits are not sorted) is
// reduced per thread, per warp and per CTA: two global atomics per CTA.
__global__ void __launch_bounds__(256) k_morton(const float4* __restrict__ pbox,
                                                uint32_t n, BoundsAcc* acc, uint64_t* __restrict__ keys,
                                                uint32_t* __restrict__ vals, int cube, uint32_t nseg, int bits30,
                                                int key32) {
  __shared__ unsigned long long s_and, s_or;
  if (threadIdx.x == 0) {
    s_and = ~0ull;
    s_or = 0ull;
  }
  __syncthreads();
  unsigned long long ka = ~0ull, ko = 0ull;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint64_t key = !bits30 ? ~0ull : nseg == 0 ? 1ull << 30 : nseg <= kFewSegments ? (1ull << 40) - 1ull : 1ull << 42;
    {
      const float4 a = pbox[2 * (size_t)i], b = pbox[2 * (size_t)i + 1];
      if (a.x <= b.x) {
        const float lo[3] = {ord2f(acc->clo[0]), ord2f(acc->clo[1]), ord2f(acc->clo[2])};
        const float hi[3] = {ord2f(acc->chi[0]), ord2f(acc->chi[1]), ord2f(acc->chi[2])};
        const float c[3] = {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
        // one scale for all axes (the centroid box's largest extent) keeps the
        // scene's aspect ratio, so flat scenes (heightfields) are ordered mostly
        // in-plane, which lowers their SAH; per-axis scales trace faster on
        // volumetric scenes.  cube: 0 per-axis, 1 one scale, 2 one scale when
        // the centroid box is flat
        const float emax = fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
        const float emin = fminf(fminf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
        const bool one_scale = cube == 1 || (cube == 2 && emin < 0.5f * emax);
        uint64_t code = 0;
        if (bits30) {
          uint32_t c30 = 0;
#pragma unroll
          for (int d = 0; d < 3; d++) {
            const float ext = one_scale ? emax : hi[d] - lo[d];
            float x = ext > 0.0f ? (c[d] - lo[d]) / ext : 0.0f;
            x = fminf(fmaxf(x * 1024.0f, 0.0f), 1023.0f);
            c30 |= spread10((uint32_t)x) << (2 - d);
          }
          key = nseg ? ((uint64_t)(__float_as_uint(a.w) & (kMaxSegments - 1)) << 30) | c30 : c30;
        } else {
#pragma unroll
          for (int d = 0; d < 3; d++) {
            const float ext = one_scale ? emax : hi[d] - lo[d];
            float x = ext > 0.0f ? (c[d] - lo[d]) / ext : 0.0f;
            x = fminf(fmaxf(x * 2097152.0f, 0.0f), 2097151.0f);
            code |= spread21((uint32_t)x) << (2 - d);
          }
          key = nseg ? ((uint64_t)(__float_as_uint(a.w) & (kMaxSegments - 1)) << 51) | (code >> 12) : code;
        }
      }
      if (key32) reinterpret_cast<uint32_t*>(keys)[i] = (uint32_t)key;
      else keys[i] = key;
      vals[i] = i;
    }
    ka &= key;
    ko |= key;
  }
  // AND / OR over all keys to find constant digits
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ka &= __shfl_xor_sync(0xFFFFFFFFu, ka, o);
    ko |= __shfl_xor_sync(0xFFFFFFFFu, ko, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAnd(&s_and, ka);
    atomicOr(&s_or, ko);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAnd(&acc->kand, s_and);
    atomicOr(&acc->kor, s_or);
  }
}

// ---------------------------------------------------------------------------
// Device-to-device copies on the SMs.  A cudaMemcpyAsync between device buffers
// runs on a copy engine: measured on a GB300, restoring 47.5 GB of ray records
// inside a CUDA graph took 29.8 ms that way against 13.7 ms for this kernel.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_copy16(uint4* __restrict__ dst, const uint4* __restrict__ src, size_t n16) {
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n16; i += (size_t)gridDim.x * 256) dst[i] = src[i];
}

static int num_sms_build();

cudaError_t copy_device(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return cudaSuccess;
  if (((uintptr_t)dst | (uintptr_t)src | bytes) % 16 != 0)
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st);
  const size_t n16 = bytes / 16;
  const size_t grid = std::min<size_t>((n16 + 255) / 256, (size_t)num_sms_build() * 8);
  k_copy16<<<(unsigned)grid, 256, 0, st>>>(static_cast<uint4*>(dst), static_cast<const uint4*>(src), n16);
  note_launches(1);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// 3. stable LSD radix sort (64-bit keys, 32-bit values), onesweep style
// ---------------------------------------------------------------------------
//
// One pass over the keys counts every digit (8 bits each) at once; its last CTA
// turns the counts into each digit's bucket bases.  Then one scatter kernel per
// digit pass: CTAs take tiles of 1,024 or 4,096 keys in ticket order, publish their digit counts
// and find the counts of all tiles before them by decoupled look-back (Merrill &
// Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016), rank
// their keys stably and scatter them.  No scan kernels and no host reads.  The
// reference's CPU sort (common/algorithms/parallel_sort.h:256-449) is the same
// stable 8-bit LSD sort, one histogram + scatter round per digit over task blocks.

constexpr int RS_THREADS = 256;
// Keys per thread: 16 where the tiles fill the chip, else 4, so that more SMs work
// and a tile's rows are ranked in a quarter of the time.  Sort of 8k / 60k / 120k /
// 250k keys of 30 bits with 4: 27 / 34 / 40 / 52 us, with 16: 42 / 48 / 51 / 57 us;
// of 300k 55 / 58, of 600k 78 / 65 us.
constexpr int RS_ITEMS = 16, RS_FEW_ITEMS = 4;
constexpr uint32_t RS_FEW = 1u << 18;
constexpr uint32_t os_tile(uint32_t n) { return RS_THREADS * (n <= RS_FEW ? RS_FEW_ITEMS : RS_ITEMS); }

// look-back status words: flag bits over a 30-bit count
constexpr uint32_t kLbAggregate = 1u << 30;   // the tile's own count is published
constexpr uint32_t kLbPrefix = 2u << 30;      // the inclusive prefix through the tile is published
constexpr uint32_t kLbValue = (1u << 30) - 1u;
constexpr uint32_t kLbSpinLimit = 1u << 22;   // re-reads of an unpublished word before giving up
// onesweep scratch (uint32 words, zeroed before each sort): bucket bases of the 8
// digit passes, tile tickets per pass, the histogram kernel's done counter, an
// error word, then per pass ntiles x 256 look-back status words
constexpr uint32_t kOsBases = 0, kOsTickets = 8 * 256, kOsDone = kOsTickets + 8, kOsErr = kOsDone + 1;
constexpr uint32_t kOsStatus = 2112;  // 16-byte aligned start of the status tables

__device__ __forceinline__ void lb_store(uint32_t* p, uint32_t v) { *reinterpret_cast<volatile uint32_t*>(p) = v; }
__device__ __forceinline__ uint32_t lb_load(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }

// Sum of the counts of the tiles before `tile` (status words status[j * stride],
// j < tile), following the chain back to the nearest published inclusive prefix.
// A word that stays unpublished for kLbSpinLimit re-reads sets kErrBuild in *err
// and counts as zero (the sort's result is then invalid and the host reports it).
__device__ __forceinline__ uint32_t lb_exclusive(const uint32_t* status, uint32_t tile, uint32_t stride,
                                                 unsigned int* err) {
  uint32_t excl = 0;
  for (int64_t j = (int64_t)tile - 1; j >= 0; j--) {
    uint32_t w = lb_load(status + (size_t)j * stride);
    for (uint32_t it = 0; w == 0u && it < kLbSpinLimit; it++) {
      __nanosleep(32);
      w = lb_load(status + (size_t)j * stride);
    }
    if (w == 0u) {
      atomicOr(err, kErrBuild);
      break;
    }
    excl += w & kLbValue;
    if (w & kLbPrefix) break;
  }
  return excl;
}

// Counts of every active digit (digit_mask bit d: digit d, bits 8d..8d+7) over all
// keys (K: 32- or 64-bit); the last CTA writes each digit's exclusive bucket bases.
template <typename K>
__global__ void __launch_bounds__(256) k_os_hist(const K* __restrict__ keys, uint32_t n, uint32_t digit_mask,
                                                 uint32_t* __restrict__ scratch) {
  __shared__ uint32_t s_h[8][256];
  __shared__ bool s_last;
  const int tid = threadIdx.x;
#pragma unroll
  for (int d = 0; d < 8; d++) s_h[d][tid] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * 256u + tid; i < n; i += gridDim.x * 256u) {
    const K k = keys[i];
#pragma unroll
    for (int d = 0; d < (int)sizeof(K); d++)
      if (digit_mask >> d & 1u) atomicAdd(&s_h[d][(uint32_t)(k >> (8 * d)) & 0xFFu], 1u);
  }
  __syncthreads();
#pragma unroll
  for (int d = 0; d < 8; d++)
    if ((digit_mask >> d & 1u) && s_h[d][tid]) atomicAdd(scratch + kOsBases + d * 256 + tid, s_h[d][tid]);
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(scratch + kOsDone, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // exclusive scan of each digit's 256 counts (one bin per thread)
  __shared__ uint32_t s_w[8];
  const int lane = tid & 31, warp = tid >> 5;
  for (int d = 0; d < 8; d++) {
    if (!(digit_mask >> d & 1u)) continue;
    const uint32_t c = lb_load(scratch + kOsBases + d * 256 + tid);
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; w++) before += s_w[w];
    scratch[kOsBases + d * 256 + tid] = before + x - c;
    __syncthreads();
  }
}

// One digit pass: tile `ticket` of kin/vin is ranked by digit (bits shift..shift+7)
// and scattered stably to kout/vout.  status: this pass's ntiles x 256 table.
// Warp w ranks the keys from base + w * 32 * ITEMS on (ITEMS rows of 32) by votes
// into per-warp digit counts; the tile's digit counts are published for the look-back;
// the keys are placed in shared memory in (digit, original order) order and written
// out in runs, consecutive threads to consecutive positions of a digit's bucket.
constexpr int RS_WARPS = RS_THREADS / 32;

// Lanes of the warp whose keys are in and have this lane's digit d (8 bits), for a
// lane whose key is: a vote per bit (with match_any, whose time grows with the number
// of different digits, the sort of 4M keys took 224 us instead of 189).
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool in) {
  uint32_t peers = __ballot_sync(0xFFFFFFFFu, in);
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool one = d >> b & 1u;
    const uint32_t vote = __ballot_sync(0xFFFFFFFFu, one);
    peers &= one ? vote : ~vote;
  }
  return peers;
}

template <typename K, int ITEMS>
constexpr size_t os_scatter_smem() { return (size_t)RS_THREADS * ITEMS * (sizeof(K) + sizeof(uint32_t)); }

template <typename K, int ITEMS>
__global__ void __launch_bounds__(RS_THREADS) k_os_scatter(const K* __restrict__ kin,
                                                           const uint32_t* __restrict__ vin,
                                                           K* __restrict__ kout, uint32_t* __restrict__ vout,
                                                           uint32_t n, int shift, uint32_t* __restrict__ scratch,
                                                           uint32_t pass_slot, uint32_t* __restrict__ status,
                                                           unsigned int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char s_stage[];               // the tile's keys, then its values
  constexpr int RS_TILE = RS_THREADS * ITEMS;
  K* s_keys = reinterpret_cast<K*>(s_stage);
  uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys + RS_TILE);
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_wcnt[RS_WARPS][256];  // per-warp digit counts, then per-warp offsets
  __shared__ uint32_t s_lstart[256];          // tile-local start of each digit
  __shared__ uint32_t s_glob[256];            // global position of local index 0 of each digit
  __shared__ uint32_t s_w[RS_WARPS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) s_tile = atomicAdd(scratch + kOsTickets + pass_slot, 1u);
#pragma unroll
  for (int w = 0; w < RS_WARPS; w++) s_wcnt[w][tid] = 0;
  __syncthreads();
  const uint32_t tile = s_tile, base = tile * RS_TILE;
  if (base >= n) return;  // (the grid has exactly one CTA per tile)
  const uint32_t tile_n = min((uint32_t)RS_TILE, n - base);
  const uint32_t lt = (1u << lane) - 1u;
  // ---- per-warp ranking (warp-synchronous: each warp owns its row of s_wcnt)
  K k[ITEMS];
  uint32_t pos[ITEMS];
  const uint32_t wbase = base + (uint32_t)warp * (ITEMS * 32);
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    const uint32_t i = wbase + r * 32 + lane;
    const bool in = i < n;
    k[r] = in ? kin[i] : (K)0;
    const uint32_t d = (uint32_t)(k[r] >> shift) & 0xFFu;
    const uint32_t peers = digit_peers(d, in);
    const uint32_t rank = __popc(peers & lt);
    pos[r] = (in ? s_wcnt[warp][d] : 0u) + rank;
    __syncwarp();
    if (in && rank == 0) s_wcnt[warp][d] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // ---- digit `tid`: tile count, per-warp offsets, tile-local start
  uint32_t cnt = 0;
#pragma unroll
  for (int w = 0; w < RS_WARPS; w++) {
    const uint32_t c = s_wcnt[w][tid];
    s_wcnt[w][tid] = cnt;
    cnt += c;
  }
  {
    uint32_t x = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; w++) before += s_w[w];
    s_lstart[tid] = before + x - cnt;
  }
  // publish this tile's count of digit `tid`, then add up the tiles before it
  {
    uint32_t excl = 0;
    if (tile == 0) {
      lb_store(status + tid, kLbPrefix | cnt);
    } else {
      lb_store(status + (size_t)tile * 256 + tid, kLbAggregate | cnt);
      excl = lb_exclusive(status + tid, tile, 256, err);
      lb_store(status + (size_t)tile * 256 + tid, kLbPrefix | ((excl + cnt) & kLbValue));
    }
    s_glob[tid] = scratch[kOsBases + (shift >> 3) * 256 + tid] + excl - s_lstart[tid];
  }
  __syncthreads();
  // ---- keys to shared memory in (digit, original order) order
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    const uint32_t i = wbase + r * 32 + lane;
    if (i < n) {
      const uint32_t d = (uint32_t)(k[r] >> shift) & 0xFFu;
      const uint32_t j = s_lstart[d] + s_wcnt[warp][d] + pos[r];
      s_keys[j] = k[r];
      s_vals[j] = vin[i];
    }
  }
  __syncthreads();
  // ---- runs out: local index j of digit d goes to s_glob[d] + j
  for (uint32_t j = tid; j < tile_n; j += RS_THREADS) {
    const K key = s_keys[j];
    const uint32_t out = s_glob[(uint32_t)(key >> shift) & 0xFFu] + j;
    if (out < n) {
      kout[out] = key;
      vout[out] = s_vals[j];
    } else {
      atomicOr(err, kErrBuild);
    }
  }
}

// The same sort of at most kSortOneMax keys by one CTA that keeps keys and values on
// chip over all passes (result in keys / vals).  Each pass ranks the keys as
// k_os_scatter does -- warp w those from w * 32 * ROWS on, row by row -- and places
// them by the digits' starts and the counts of the warps before.  A small build's
// sort is a chain of launches (a memset, the histogram, four scatters): 512 / 2048 /
// 3872 keys of 30 bits take 18 / 23 / 25 us so and 14 / 15 / 16 us in one CTA, 8192
// 27 us so and 29 in one CTA of 8 rows.
constexpr int kSortOneThreads = 1024, kSortOneWarps = kSortOneThreads / 32, kSortOneRows = 4;
constexpr uint32_t kSortOneMax = kSortOneThreads * kSortOneRows;
template <typename K>
constexpr size_t sort_one_smem() {
  return (sizeof(K) + sizeof(uint32_t)) * kSortOneMax + sizeof(uint32_t) * kSortOneWarps * 256;
}

template <typename K>
__global__ void __launch_bounds__(kSortOneThreads, 1) k_sort_one(K* __restrict__ keys, uint32_t* __restrict__ vals,
                                                                 uint32_t n, uint32_t digit_mask) {
  constexpr int ROWS = kSortOneRows;
  extern __shared__ __align__(16) unsigned char s_one[];
  K* s_keys = reinterpret_cast<K*>(s_one);
  uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys + kSortOneMax);
  uint32_t(*s_cnt)[256] = reinterpret_cast<uint32_t(*)[256]>(s_vals + kSortOneMax);  // per warp: its digit counts
  __shared__ uint32_t s_group[4][256];  // per 8 warps: counts of each digit, then where they start
  __shared__ uint32_t s_w[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int digit = tid & 255, group = tid >> 8;
  const uint32_t lt = (1u << lane) - 1u, base = (uint32_t)warp * (32 * ROWS) + lane;
  K k[ROWS];
  uint32_t v[ROWS], pos[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    const uint32_t i = base + 32 * r;
    k[r] = i < n ? keys[i] : (K)0;
    v[r] = i < n ? vals[i] : 0u;
  }
  for (int pass = 0; pass < (int)sizeof(K); pass++) {
    if (!(digit_mask >> pass & 1u)) continue;
    const int shift = 8 * pass;
#pragma unroll
    for (int w = 0; w < 8; w++) s_cnt[8 * group + w][digit] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      const bool in = base + 32 * r < n;
      const uint32_t d = (uint32_t)(k[r] >> shift) & 0xFFu;
      const uint32_t peers = digit_peers(d, in), rank = __popc(peers & lt);
      pos[r] = (in ? s_cnt[warp][d] : 0u) + rank;
      __syncwarp();
      if (in && rank == 0) s_cnt[warp][d] += __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
      const uint32_t c = s_cnt[8 * group + w][digit];
      s_cnt[8 * group + w][digit] = sum;
      sum += c;
    }
    s_group[group][digit] = sum;
    __syncthreads();
    uint32_t g[4] = {0u, 0u, 0u, 0u}, x = 0, total = 0;
    if (tid < 256) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        g[q] = total;
        total += s_group[q][tid];
      }
      x = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) s_w[warp] = x;
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t start = x - total;
      for (int w = 0; w < warp; w++) start += s_w[w];
#pragma unroll
      for (int q = 0; q < 4; q++) s_group[q][tid] = start + g[q];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      if (base + 32 * r < n) {
        const uint32_t d = (uint32_t)(k[r] >> shift) & 0xFFu;
        const uint32_t j = s_group[warp >> 3][d] + s_cnt[warp][d] + pos[r];  // a permutation of 0 .. n - 1
        s_keys[j] = k[r];
        s_vals[j] = v[r];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      const uint32_t i = base + 32 * r;
      if (i < n) {
        k[r] = s_keys[i];
        v[r] = s_vals[i];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    const uint32_t i = base + 32 * r;
    if (i < n) {
      keys[i] = k[r];
      vals[i] = v[r];
    }
  }
}

// Exclusive scans of uint32 arrays.  One tile is 1024 threads x 8 consecutive
// elements.  Small arrays are scanned by one CTA; larger ones by
// reduce-then-scan over many CTAs (tile sums, a one-CTA scan of the sums, then
// each tile scanned again from its offset), which reads the array twice and
// writes it once.
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_PER = 8;
constexpr uint32_t SCAN_TILE = SCAN_THREADS * SCAN_PER;

// Scans a[base, base + SCAN_TILE) in place, offset by carry; every thread gets
// the tile's total.  All threads of the CTA must call it.
__device__ __forceinline__ uint32_t scan_tile(uint32_t* __restrict__ a, uint32_t n, uint32_t base, uint32_t carry,
                                              uint32_t* s_w) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t v[SCAN_PER];
  uint32_t sum = 0;
  const uint32_t i0 = base + threadIdx.x * SCAN_PER;
#pragma unroll
  for (int k = 0; k < SCAN_PER; k++) {
    v[k] = (i0 + k < n) ? a[i0 + k] : 0u;
    sum += v[k];
  }
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = s_w[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    s_w[lane] = w;
  }
  __syncthreads();
  uint32_t excl = carry + (warp ? s_w[warp - 1] : 0u) + (x - sum);
#pragma unroll
  for (int k = 0; k < SCAN_PER; k++) {
    if (i0 + k < n) a[i0 + k] = excl;
    excl += v[k];
  }
  const uint32_t tile_total = s_w[31];
  __syncthreads();  // s_w is reused by the next call
  return tile_total;
}

// Element counts of the scans: n itself, or -- when the count is produced on
// the device (builds that run without host reads) -- ceil(*d_n / div) capped
// at n.  Grids are then sized for the cap and the tile loops are grid-stride.
__device__ __forceinline__ uint32_t scan_count(uint32_t n, const uint32_t* d_n, uint32_t div) {
  return d_n ? min(n, (*d_n + div - 1) / div) : n;
}

// Two arrays scanned by one launch (the survivors and merges of a PLOC round,
// the internal children and triangles of a collapse level): blockIdx.y picks
// the array, its total and (look-back scan) its state.
struct ScanPair {
  uint32_t* a[2];
  uint32_t* total[2];
};

// One CTA of 1024 threads over the whole array; optionally writes the total.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_excl(ScanPair sp, uint32_t n,
                                                            const uint32_t* __restrict__ d_n, uint32_t div) {
  __shared__ uint32_t s_w[32];
  uint32_t* __restrict__ a = sp.a[blockIdx.y];
  uint32_t* total = sp.total[blockIdx.y];
  n = scan_count(n, d_n, div);
  uint32_t carry = 0;
  for (uint32_t base = 0; base < n; base += SCAN_TILE) carry += scan_tile(a, n, base, carry, s_w);
  if (total && threadIdx.x == 0) *total = carry;
}

// Single-pass exclusive scan of larger arrays: CTAs take SCAN_TILE tiles in ticket
// order, publish their tile sums and add up those of the tiles before them by
// decoupled look-back, then scan their tile from that offset.  state (per array,
// state_words apart): [0] ticket, [1] CTAs finished, [2 + t] status word of tile
// t; zero on entry, and the last CTA to finish zeroes it again for the next scan
// (graph replays included).
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_lb(ScanPair sp, uint32_t n,
                                                          const uint32_t* __restrict__ d_n, uint32_t div,
                                                          uint32_t* __restrict__ state_base, uint32_t state_words,
                                                          unsigned int* __restrict__ err) {
  __shared__ uint32_t s_w[32];
  __shared__ uint32_t s_tile, s_excl;
  __shared__ bool s_last;
  uint32_t* __restrict__ a = sp.a[blockIdx.y];
  uint32_t* total = sp.total[blockIdx.y];
  uint32_t* __restrict__ state = state_base + (size_t)blockIdx.y * state_words;
  n = scan_count(n, d_n, div);
  const uint32_t ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (threadIdx.x == 0) s_tile = atomicAdd(state, 1u);
  __syncthreads();
  const uint32_t t = s_tile;
  uint32_t* status = state + 2;
  if (t < ntiles) {
    const uint32_t i0 = t * SCAN_TILE + threadIdx.x * SCAN_PER;
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) sum += (i0 + k < n) ? a[i0 + k] : 0u;
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x < 32) {
      const uint32_t tile_sum = __reduce_add_sync(0xFFFFFFFFu, s_w[threadIdx.x]);
      if (threadIdx.x == 0) {
        uint32_t excl = 0;
        if (t == 0) {
          lb_store(status, kLbPrefix | (tile_sum & kLbValue));
        } else {
          lb_store(status + t, kLbAggregate | (tile_sum & kLbValue));
          excl = lb_exclusive(status, t, 1, err);
          lb_store(status + t, kLbPrefix | ((excl + tile_sum) & kLbValue));
        }
        s_excl = excl;
        if (t == ntiles - 1 && total) *total = excl + tile_sum;
      }
    }
    __syncthreads();
    scan_tile(a, n, t * SCAN_TILE, s_excl, s_w);
  } else if (t == 0 && total && threadIdx.x == 0) {
    *total = 0;  // empty input
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(state + 1, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (s_last) {
    for (uint32_t j = threadIdx.x; j < gridDim.x; j += SCAN_THREADS) status[j] = 0;
    if (threadIdx.x == 0) {
      state[0] = 0;
      state[1] = 0;
    }
  }
}

// ---- SAH-optimal collapse (dynamic programming over the binary tree, after
// Ylitie, Karras and Laine, "Efficient incoherent ray traversal on GPUs
// through compressed wide BVHs", HPG 2017).  cost(n, i) is the least SAH cost
// of the subtree of binary node n when it may take up to i child slots of a
// wide node: i = 1 is n itself as one child (a leaf when it holds at most
// leaf_max triangles -- then its cost is area x Triangle4 blocks -- else a wide
// node of its own: area + D(n, 8)); i > 1 is min(cost(n, i - 1), D(n, i)) with
// D(n, i) = min over k of cost(left, k) + cost(right, i - k).  The costs are
// the SAH statistic's terms (bvh_statistics.cpp:10-160), so the tree minimises
// the reported SAH for the given binary tree and leaf size.
//
// link[n] = (left, right, decisions): one 16-byte read per node for the collapse,
// which follows the decisions from node to node.  Byte 0 of the decisions is the
// split of a wide node made from n, byte i - 1 (i = 2..8) the split of n in i slots:
// the slots of the left child in the low and of the right child in the high four
// bits, 0 where n stays one child (then for all fewer slots too).

__device__ __forceinline__ void dp_store(float4* cost, uint4* link, uint32_t n, const float c[8], uint4 lk) {
  __stcg(cost + 2 * (size_t)n, make_float4(c[0], c[1], c[2], c[3]));
  __stcg(cost + 2 * (size_t)n + 1, make_float4(c[4], c[5], c[6], c[7]));
  __stcg(link + n, lk);
}

// A child's cost(., 1..8): a primitive (one triangle) costs its box area
// whatever the number of slots (one leaf block), so primitives have no table
// entries and the caller passes their areas; internal children's costs are
// stored already.
__device__ __forceinline__ void dp_child_costs(const float4* cost, uint32_t c, uint32_t cnt_c, float Ac, float (&out)[8]) {
  if (cnt_c == 1) {
#pragma unroll
    for (int i = 0; i < 8; i++) out[i] = Ac;
    return;
  }
  const float4 a = __ldcg(cost + 2 * (size_t)c), b = __ldcg(cost + 2 * (size_t)c + 1);
  out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w; out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
}

// cost(n, 1..8) into c and the tables, and the choices of n, from its children's costs.
__device__ __forceinline__ void dp_combine(float4* cost, uint4* link, uint32_t n, uint32_t l, uint32_t r, float A,
                                           uint32_t cnt, const float (&cl)[8], const float (&cr)[8], uint32_t leaf_max,
                                           float (&c)[8]) {
  float D[9];
  uint32_t K[9];
#pragma unroll
  for (int i = 2; i <= 8; i++) {
    D[i] = INFINITY;
    K[i] = 1u | (uint32_t)(i - 1) << 4;
#pragma unroll
    for (int k = 1; k < i; k++) {
      const float v = cl[k - 1] + cr[i - k - 1];
      if (v < D[i]) {
        D[i] = v;
        K[i] = (uint32_t)k | (uint32_t)(i - k) << 4;
      }
    }
  }
  const float c_int = A + D[8];
  const float c_leaf = cnt <= leaf_max ? A * (float)((cnt + 3) / 4) : INFINITY;
  c[0] = fminf(c_leaf, c_int);
  uint32_t b[8];
  b[0] = K[8];
#pragma unroll
  for (int i = 2; i <= 8; i++) {
    const bool split = D[i] < c[i - 2];
    c[i - 1] = split ? D[i] : c[i - 2];
    b[i - 1] = split ? K[i] : i > 2 ? b[i - 2] : 0u;
  }
  dp_store(cost, link, n, c,
           make_uint4(l, r, b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24), b[4] | (b[5] << 8) | (b[6] << 16) | (b[7] << 24)));
}

// cost(n, 1..8) and the choices of binary node n with children l and r (cnt_l,
// cnt_r triangles; a child of one triangle is a primitive, whose area Al / Ar
// the caller passes); A is n's box area.  The PLOC kernels call it as they
// create each node, so the table is complete when the clustering ends
// (children are always created before their parent).
__device__ __forceinline__ void dp_node(float4* cost, uint4* link, uint32_t n, uint32_t l, uint32_t r, float A,
                                        uint32_t cnt_l, uint32_t cnt_r, float Al, float Ar, uint32_t leaf_max) {
  float cl[8], cr[8], c[8];
  dp_child_costs(cost, l, cnt_l, Al, cl);
  dp_child_costs(cost, r, cnt_r, Ar, cr);
  dp_combine(cost, link, n, l, r, A, cnt_l + cnt_r, cl, cr, leaf_max, c);
}

// Grid barrier of the cooperative build kernels (all CTAs resident).
struct GridBarrier {
  unsigned int count;
};

// Barrier over all CTAs of a cooperative launch; every thread calls it.  b->count
// is zero before the launch (a barrier adds gridDim.x to it).  A CTA that waits for
// more than kLbSpinLimit re-reads (a CTA missing) sets kErrBuild in *err; false
// once *err is set, so the grid leaves its loop.  A build waits at about 70 of
// these and a refit at 12, so their latency counts: one
// releasing atomic, plain reads of the same word and one acquiring read at the end.
// (Acquire-release fences around the atomic and the reads cost 0.3 us more per
// barrier, the rounds of the 4M soup 571 us instead of 555; a separate generation
// word, sequentially consistent fences and sleeping between the reads 1.1 us more.)
__device__ __forceinline__ bool grid_sync(GridBarrier* b, unsigned int* err) {
  __shared__ bool s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int ticket;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(&b->count) : "memory");
    const unsigned int target = (ticket / gridDim.x + 1u) * gridDim.x;
    uint32_t it = 0, e = lb_load(err);
    while (lb_load(&b->count) < target && e == 0u && it < kLbSpinLimit) {
      e = lb_load(err);
      it++;
    }
    if (it == kLbSpinLimit) atomicOr(err, kErrBuild);
    unsigned int last;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(last) : "l"(&b->count) : "memory");
    s_ok = e == 0u && it < kLbSpinLimit;
  }
  __syncthreads();
  return s_ok;
}

// ---------------------------------------------------------------------------
// 4. PLOC
// ---------------------------------------------------------------------------

// PLOC's search radius (clusters on each side in Morton order) is a template
// parameter of the nearest-neighbour kernel; gpu.ploc_radius picks 1, 2, 4, 8
// or 16.  Measured on a GB300, radius 1 gave the lowest SAH on heightfields,
// the fastest traversal and the fastest build (a wider window made the
// clusters' merges less local: the 4M soup went from 1033 to 889 Mrays/s
// closest between radius 1 and 16).
constexpr int PLOC_R_MAX = 16;
constexpr int PLOC_BLOCK = 256;
constexpr uint32_t PLOC_SMALL = 4096;   // finish on one CTA below this many clusters
constexpr int PLOC_SMALL_THREADS = 1024;
// k_ploc_small's shared memory: boxes, node ids, nearest neighbours, segments, counts
constexpr size_t kPlocSmallSmem = (size_t)PLOC_SMALL * (2 * sizeof(float3) + 4 * sizeof(uint32_t));

// binary nodes: bnbox[2k] = (lo.xyz, left), bnbox[2k + 1] = (hi.xyz, right), one
// 32-byte sector (they are read one by one, in no order);
// leaves k < N: left = -1, right = primref index
// Cluster boxes carry their segment in clo.w (0 unless the build is segmented)
// and their triangle count in chi.w (so a merge has both children's counts
// with their boxes, without a dependent read of bncnt).
__global__ void __launch_bounds__(256) k_ploc_init(const float4* __restrict__ pbox,
                                                   const uint32_t* __restrict__ sorted, uint32_t n,
                                                   const uint32_t* __restrict__ d_n,
                                                   float4* __restrict__ bnbox, uint32_t* __restrict__ cidx,
                                                   float4* __restrict__ clo, float4* __restrict__ chi, int segmented) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || i >= *d_n) return;  // n bounds the grid, *d_n is the count of valid primitives
  const uint32_t p = sorted[i];
  const float4 a = pbox[2 * (size_t)p], b = pbox[2 * (size_t)p + 1];
  bnbox[2 * (size_t)i] = make_float4(a.x, a.y, a.z, __int_as_float(-1));
  bnbox[2 * (size_t)i + 1] = make_float4(b.x, b.y, b.z, __uint_as_float(p));
  cidx[i] = i;
  clo[i] = make_float4(a.x, a.y, a.z, segmented ? a.w : __uint_as_float(0u));
  chi[i] = make_float4(b.x, b.y, b.z, __uint_as_float(1u));
}

// PLOC rounds run back to back without the host.  ploc_state (device memory):
// [0] cluster count n, [1] next binary node index, [2] rounds that merged,
// [3] 256-cluster tiles of n, [4] done -- set once n <= PLOC_SMALL (the one-CTA
// kernel finishes) or a round merged nothing; every kernel of a later round is
// then a no-op, so a fixed number of rounds can be enqueued (or captured) and
// the tree is the same whatever the number of extra rounds.  The kernels loop
// over the tiles grid-stride, so the grid is any size.
enum : int { kPlocN = 0, kPlocNext = 1, kPlocRounds = 2, kPlocTiles = 3, kPlocDone = 4, kPlocParity = 5,
             kPlocIters = 6, kPlocStateWords = 8 };
// device-decided PLOC loops (the cooperative rounds of captured builds) stop
// after this many rounds
constexpr uint32_t kPlocMaxIters = 1024;

// The two cluster buffers of the PLOC rounds; a round reads set ploc_state[kPlocParity]
// and writes the other one, so every round runs the same kernels with the same
// arguments (a loop body captured once serves every iteration).
struct PlocBufs {
  float4* clo[2];
  float4* chi[2];
  uint32_t* cidx[2];
};


// The clusters alternate between two buffers, one round reading A and writing
// B, the next the reverse; kPlocParity counts (mod 2) the rounds that ran, so
// the current clusters are in B when it is 1 whatever no-op rounds followed.
// bar, the cooperative rounds' barrier (or null), is zeroed too.  expect: the valid
// primitives that every array from here on is sized for.  A replayed build whose
// input has another number of them clusters nothing: without clusters there are no
// roots, no levels and no leaves, no kernel leaves its arrays (with more primitives
// than planned the rounds would index past theirs) or takes a merged node for a
// primitive (ids below `expect`), and k_graph_build_check reports the count.
__global__ void k_ploc_state_init(const BoundsAcc* __restrict__ acc, uint32_t expect, uint32_t* __restrict__ ploc_state,
                                  GridBarrier* bar) {
  if (threadIdx.x == 0) {
    if (bar) bar->count = 0;
    const uint32_t n = acc->nvalid == expect ? expect : 0u;
    ploc_state[kPlocN] = n;
    ploc_state[kPlocNext] = n;  // binary leaves are the primitives 0..n-1
    ploc_state[kPlocRounds] = 0;
    ploc_state[kPlocTiles] = (n + PLOC_BLOCK - 1) / PLOC_BLOCK;
    ploc_state[kPlocDone] = n <= PLOC_SMALL ? 1u : 0u;
    ploc_state[kPlocParity] = 0;
    ploc_state[kPlocIters] = 0;
  }
}

// Nearest neighbour (least merged-box area within PLOC_R clusters on either
// side, same segment) of every cluster of one PLOC_BLOCK tile; the window with
// its halo is staged in shared memory.
template <int PLOC_R>
__device__ __forceinline__ void ploc_nn_tile(const float4* clo, const float4* chi, uint32_t n,
                                             uint32_t tile, uint32_t* __restrict__ nn, float3* s_lo, float3* s_hi,
                                             uint32_t* s_seg) {
  const int base = (int)(tile * PLOC_BLOCK);
  for (int k = threadIdx.x; k < PLOC_BLOCK + 2 * PLOC_R; k += PLOC_BLOCK) {
    const int j = base - PLOC_R + k;
    if (j >= 0 && j < (int)n) {
      const float4 a = clo[j], b = chi[j];
      s_lo[k] = make_float3(a.x, a.y, a.z);
      s_hi[k] = make_float3(b.x, b.y, b.z);
      s_seg[k] = __float_as_uint(a.w);
    }
  }
  __syncthreads();
  const int i = base + threadIdx.x;
  if (i < (int)n) {
    const float3 lo = s_lo[threadIdx.x + PLOC_R], hi = s_hi[threadIdx.x + PLOC_R];
    const uint32_t seg = s_seg[threadIdx.x + PLOC_R];
    unsigned long long best = ~0ull;
#pragma unroll 4
    for (int o = -PLOC_R; o <= PLOC_R; o++) {
      const int j = i + o;
      if (o == 0 || j < 0 || j >= (int)n || s_seg[threadIdx.x + PLOC_R + o] != seg) continue;
      const float a = half_area(f3min(lo, s_lo[threadIdx.x + PLOC_R + o]), f3max(hi, s_hi[threadIdx.x + PLOC_R + o]));
      const unsigned long long key = ((unsigned long long)__float_as_uint(a) << 32) | (uint32_t)j;
      best = key < best ? key : best;
    }
    nn[i] = best != ~0ull ? (uint32_t)best : (uint32_t)i;  // no neighbour in the segment: stays alone
  }
  __syncthreads();  // the window is reloaded for the next tile
}

// The same nearest neighbour for one cluster h, read from global memory (the
// halo clusters just outside a CTA's run of tiles; bit-identical to the tile
// form: same boxes, same area arithmetic, the least (area, index) key).
template <int PLOC_R>
__device__ __forceinline__ uint32_t ploc_nn_one(const float4* clo, const float4* chi,
                                                uint32_t n, int h) {
  const float4 a = clo[h], b = chi[h];
  const float3 lo = make_float3(a.x, a.y, a.z), hi = make_float3(b.x, b.y, b.z);
  const uint32_t seg = __float_as_uint(a.w);
  unsigned long long best = ~0ull;
  for (int o = -PLOC_R; o <= PLOC_R; o++) {
    const int j = h + o;
    if (o == 0 || j < 0 || j >= (int)n) continue;
    const float4 c = clo[j], d = chi[j];
    if (__float_as_uint(c.w) != seg) continue;
    const float ar = half_area(f3min(lo, make_float3(c.x, c.y, c.z)), f3max(hi, make_float3(d.x, d.y, d.z)));
    const unsigned long long key = ((unsigned long long)__float_as_uint(ar) << 32) | (uint32_t)j;
    best = key < best ? key : best;
  }
  return best != ~0ull ? (uint32_t)best : (uint32_t)h;
}

template <int PLOC_R>
__global__ void __launch_bounds__(PLOC_BLOCK) k_ploc_nn(const PlocBufs bufs, const uint32_t* __restrict__ ploc_state,
                                                        uint32_t* __restrict__ nn) {
  __shared__ float3 s_lo[PLOC_BLOCK + 2 * PLOC_R], s_hi[PLOC_BLOCK + 2 * PLOC_R];
  __shared__ uint32_t s_seg[PLOC_BLOCK + 2 * PLOC_R];
  if (ploc_state[kPlocDone]) return;
  const uint32_t n = ploc_state[kPlocN];
  const uint32_t par = ploc_state[kPlocParity] & 1u;
  for (uint32_t tile = blockIdx.x; tile * PLOC_BLOCK < n; tile += gridDim.x)
    ploc_nn_tile<PLOC_R>(bufs.clo[par], bufs.chi[par], n, tile, nn, s_lo, s_hi, s_seg);
}

// Survivor and merge counts of every tile of the round.
__global__ void __launch_bounds__(PLOC_BLOCK) k_ploc_count(const uint32_t* __restrict__ nn,
                                                           const uint32_t* __restrict__ ploc_state,
                                                           uint32_t* __restrict__ bsurv, uint32_t* __restrict__ bmerge) {
  if (ploc_state[kPlocDone]) return;
  const uint32_t n = ploc_state[kPlocN];
  for (uint32_t tile = blockIdx.x; tile * PLOC_BLOCK < n; tile += gridDim.x) {
    const uint32_t i = tile * PLOC_BLOCK + threadIdx.x;
    int surv = 0, merge = 0;
    if (i < n) {
      const uint32_t j = nn[i];
      const bool mutual = (j != i) && nn[j] == i;
      merge = mutual && i < j;
      surv = !(mutual && j < i);
    }
    const int cs = __syncthreads_count(surv);
    const int cm = __syncthreads_count(merge);
    if (threadIdx.x == 0) {
      bsurv[tile] = cs;
      bmerge[tile] = cm;
    }
  }
}

__device__ __forceinline__ uint32_t block_excl_scan_flag(int flag, uint32_t* s_warp) {
  // exclusive rank of this thread among flagged threads of the block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t bal = __ballot_sync(0xFFFFFFFFu, flag);
  if (lane == 0) s_warp[warp] = __popc(bal);
  __syncthreads();
  uint32_t pre = 0;
  for (int w = 0; w < warp; w++) pre += s_warp[w];
  __syncthreads();
  return pre + __popc(bal & ((1u << lane) - 1u));
}

// Output of cluster i at position pos of the next round: itself (j == i), or the
// new node `id` that merges it with cluster j, whose collapse costs are computed
// here.
__device__ __forceinline__ void ploc_emit_one(const PlocBufs& bufs, uint32_t par, uint32_t i, uint32_t j, uint32_t pos,
                                              uint32_t id, uint32_t n, float4* __restrict__ bnbox,
                                              uint32_t* __restrict__ bncnt, uint32_t node_cap, uint32_t* err,
                                              float4* __restrict__ dp_cost, uint4* __restrict__ dp_link,
                                              uint32_t leaf_max) {
  const float4 *clo = bufs.clo[par], *chi = bufs.chi[par];
  const uint32_t* cidx = bufs.cidx[par];
  float4 lo = clo[i], hi = chi[i];
  uint32_t out = cidx[i];
  if (pos >= n) {
    atomicOr(err, kErrBuild);
    return;
  }
  if (j != i) {
    const float4 a = lo, b = hi, c = clo[j], d = chi[j];
    const uint32_t l = out, r = cidx[j];
    if (id >= node_cap) {
      atomicOr(err, kErrBuild);
      return;
    }
    lo = make_float4(fminf(a.x, c.x), fminf(a.y, c.y), fminf(a.z, c.z), a.w);
    const uint32_t cnt_l = __float_as_uint(b.w), cnt_r = __float_as_uint(d.w);
    hi = make_float4(fmaxf(b.x, d.x), fmaxf(b.y, d.y), fmaxf(b.z, d.z), __uint_as_float(cnt_l + cnt_r));
    bnbox[2 * (size_t)id] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(l));
    bnbox[2 * (size_t)id + 1] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(r));
    bncnt[id] = cnt_l + cnt_r;
    if (dp_cost)
      dp_node(dp_cost, dp_link, id, l, r, half_area(make_float3(lo.x, lo.y, lo.z), make_float3(hi.x, hi.y, hi.z)),
              cnt_l, cnt_r, cnt_l == 1 ? half_area(make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z)) : 0.f,
              cnt_r == 1 ? half_area(make_float3(c.x, c.y, c.z), make_float3(d.x, d.y, d.z)) : 0.f, leaf_max);
    out = id;
  }
  bufs.clo[par ^ 1u][pos] = lo;
  bufs.chi[par ^ 1u][pos] = hi;
  bufs.cidx[par ^ 1u][pos] = out;
}

// Survivors and merges of one tile: a cluster whose nearest neighbour is
// mutual merges with it (the lower index creates the node, the higher one is
// dropped), the others survive as they are; outputs go to position
// surv_off + rank among the tile's survivors, new nodes to node_next + merge_off
// + rank among its merges.  Each new node's collapse costs are computed here.
__device__ __forceinline__ void ploc_emit_tile(const PlocBufs& bufs, uint32_t par, const uint32_t* __restrict__ nn,
                                               uint32_t n, uint32_t node_next, uint32_t tile, uint32_t surv_off,
                                               uint32_t merge_off, float4* __restrict__ bnbox,
                                               uint32_t* __restrict__ bncnt,
                                               uint32_t node_cap, uint32_t* err, float4* __restrict__ dp_cost,
                                               uint4* __restrict__ dp_link, uint32_t leaf_max, uint32_t* s_w) {
  const uint32_t i = tile * PLOC_BLOCK + threadIdx.x;
  int surv = 0, merge = 0;
  uint32_t j = 0;
  if (i < n) {
    j = nn[i];
    const bool mutual = (j != i) && nn[j] == i;
    merge = mutual && i < j;
    surv = !(mutual && j < i);
  }
  const uint32_t rs = block_excl_scan_flag(surv, s_w);
  const uint32_t rm = block_excl_scan_flag(merge, s_w);
  if (i >= n || !surv) return;
  ploc_emit_one(bufs, par, i, merge ? j : i, surv_off + rs, node_next + merge_off + rm, n, bnbox, bncnt, node_cap, err,
                dp_cost, dp_link, leaf_max);
}

__global__ void __launch_bounds__(PLOC_BLOCK) k_ploc_emit(const PlocBufs bufs, const uint32_t* __restrict__ nn,
                                                          const uint32_t* __restrict__ ploc_state,
                                                          const uint32_t* __restrict__ bsurv_off,
                                                          const uint32_t* __restrict__ bmerge_off,
                                                          float4* __restrict__ bnbox,
                                                          uint32_t* __restrict__ bncnt, uint32_t node_cap, uint32_t* err,
                                                          float4* __restrict__ dp_cost, uint4* __restrict__ dp_link,
                                                          uint32_t leaf_max) {
  __shared__ uint32_t s_w[PLOC_BLOCK / 32];
  if (ploc_state[kPlocDone]) return;
  const uint32_t n = ploc_state[kPlocN], node_next = ploc_state[kPlocNext];
  const uint32_t par = ploc_state[kPlocParity] & 1u;
  for (uint32_t tile = blockIdx.x; tile * PLOC_BLOCK < n; tile += gridDim.x)
    ploc_emit_tile(bufs, par, nn, n, node_next, tile, bsurv_off[tile], bmerge_off[tile], bnbox, bncnt, node_cap,
                   err, dp_cost, dp_link, leaf_max, s_w);
}

// After a round: the survivors are the new clusters, the merges took the next
// binary node indices; rounds end once n <= PLOC_SMALL or nothing merged.
__global__ void k_ploc_advance(const uint32_t* __restrict__ tot, uint32_t* __restrict__ ploc_state) {
  if (threadIdx.x != 0) return;
  if (!ploc_state[kPlocDone]) {
    const uint32_t n = tot[0], merged = tot[1];
    ploc_state[kPlocN] = n;
    ploc_state[kPlocNext] += merged;
    ploc_state[kPlocRounds] += merged > 0 ? 1u : 0u;
    ploc_state[kPlocTiles] = (n + PLOC_BLOCK - 1) / PLOC_BLOCK;
    ploc_state[kPlocParity] ^= 1u;
    if (n <= PLOC_SMALL || merged == 0) ploc_state[kPlocDone] = 1u;
  }
  ++ploc_state[kPlocIters];
}

// All PLOC rounds above PLOC_SMALL clusters in one cooperative launch (captured
// builds): per round (A) nearest neighbours of the CTA's contiguous run of
// tiles and of the PLOC_R clusters either side of it, (B) survivors and merges
// of each tile (mutual pairs decided from A alone), per-CTA sums, [barrier],
// (C) this CTA's offsets from the sums and its tiles' outputs, [barrier]: two
// grid barriers per round (with a third between A and B the 4M soup rebuilt
// in 2.50 ms, without it 2.46).  Each CTA keeps the round state (the k_ploc_advance
// rules) in registers; CTA 0 writes it back to ploc_state.  cta_sums holds
// 2 * gridDim.x words; *bar is zero on entry.
template <int PLOC_R>
__global__ void __launch_bounds__(PLOC_BLOCK) k_ploc_all(const PlocBufs bufs, uint32_t* __restrict__ ploc_state,
                                                         uint32_t* __restrict__ nn, uint32_t* __restrict__ tile_s,
                                                         uint32_t* __restrict__ tile_m, uint32_t* __restrict__ cta_sums,
                                                         float4* __restrict__ bnbox,
                                                         uint32_t* __restrict__ bncnt, uint32_t node_cap,
                                                         float4* __restrict__ dp_cost, uint4* __restrict__ dp_link,
                                                         uint32_t leaf_max, GridBarrier* bar, unsigned int* err) {
  __shared__ float3 s_lo[PLOC_BLOCK + 2 * PLOC_R], s_hi[PLOC_BLOCK + 2 * PLOC_R];
  __shared__ uint32_t s_seg[PLOC_BLOCK + 2 * PLOC_R];
  __shared__ uint32_t s_w[PLOC_BLOCK / 32];
  __shared__ uint32_t s_red[4][PLOC_BLOCK / 32];
  __shared__ uint32_t s_halo_nn[2 * PLOC_R];  // nearest neighbours of the R clusters either side of the run
  uint32_t n = __ldcg(ploc_state + kPlocN), node_next = __ldcg(ploc_state + kPlocNext);
  uint32_t par = __ldcg(ploc_state + kPlocParity) & 1u, rounds = __ldcg(ploc_state + kPlocRounds);
  uint32_t iters = __ldcg(ploc_state + kPlocIters);
  bool done = __ldcg(ploc_state + kPlocDone) != 0u;
  while (!done && iters < kPlocMaxIters) {
    const uint32_t ntiles = (n + PLOC_BLOCK - 1) / PLOC_BLOCK;
    const uint32_t per = (ntiles + gridDim.x - 1) / gridDim.x;
    const uint32_t t0 = min(blockIdx.x * per, ntiles), t1 = min(t0 + per, ntiles);
    // (A) nearest neighbours of this CTA's run of tiles [r0, r1), and of the R
    // clusters either side of it (computed here as their own CTAs compute
    // them), so that (B) needs no grid barrier before it
    const int r0 = (int)(t0 * PLOC_BLOCK), r1 = (int)min(t1 * PLOC_BLOCK, n);
    for (uint32_t tile = t0; tile < t1; tile++)
      ploc_nn_tile<PLOC_R>(bufs.clo[par], bufs.chi[par], n, tile, nn, s_lo, s_hi, s_seg);
    if (threadIdx.x < 2 * PLOC_R && t0 < t1) {
      const int h = threadIdx.x < PLOC_R ? r0 - PLOC_R + (int)threadIdx.x : r1 + (int)threadIdx.x - PLOC_R;
      if (h >= 0 && h < (int)n) s_halo_nn[threadIdx.x] = ploc_nn_one<PLOC_R>(bufs.clo[par], bufs.chi[par], n, h);
    }
    __syncthreads();
    // (B) survivors and merges per tile (the run's nn written above by this CTA)
    auto nn_of = [&](uint32_t j) -> uint32_t {
      if ((int)j < r0) return s_halo_nn[(int)j - (r0 - PLOC_R)];
      if ((int)j >= r1) return s_halo_nn[PLOC_R + (int)j - r1];
      return nn[j];
    };
    uint32_t cs_sum = 0, cm_sum = 0;
    for (uint32_t tile = t0; tile < t1; tile++) {
      const uint32_t i = tile * PLOC_BLOCK + threadIdx.x;
      int surv = 0, merge = 0;
      if (i < n) {
        const uint32_t j = nn[i];
        const bool mutual = (j != i) && nn_of(j) == i;
        merge = mutual && i < j;
        surv = !(mutual && j < i);
      }
      const uint32_t cs = (uint32_t)__syncthreads_count(surv);
      const uint32_t cm = (uint32_t)__syncthreads_count(merge);
      if (threadIdx.x == 0) {
        tile_s[tile] = cs;
        tile_m[tile] = cm;
      }
      cs_sum += cs;
      cm_sum += cm;
    }
    if (threadIdx.x == 0) {
      __stcg(cta_sums + blockIdx.x, cs_sum);
      __stcg(cta_sums + gridDim.x + blockIdx.x, cm_sum);
    }
    if (!grid_sync(bar, err)) break;
    // (C) this CTA's offsets and the round's totals, then its tiles' outputs
    uint32_t v[4] = {0u, 0u, 0u, 0u};  // prefix survivors, prefix merges, total survivors, total merges
    for (uint32_t c = threadIdx.x; c < gridDim.x; c += blockDim.x) {
      const uint32_t a = __ldcg(cta_sums + c), b = __ldcg(cta_sums + gridDim.x + c);
      v[2] += a;
      v[3] += b;
      if (c < blockIdx.x) {
        v[0] += a;
        v[1] += b;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      v[q] = __reduce_add_sync(0xFFFFFFFFu, v[q]);
      if ((threadIdx.x & 31) == 0) s_red[q][threadIdx.x >> 5] = v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint32_t t = 0;
      for (int w = 0; w < PLOC_BLOCK / 32; w++) t += s_red[q][w];
      v[q] = t;
    }
    __syncthreads();  // s_red is reused next round
    uint32_t ps = v[0], pm = v[1];
    for (uint32_t tile = t0; tile < t1; tile++) {
      ploc_emit_tile(bufs, par, nn, n, node_next, tile, ps, pm, bnbox, bncnt, node_cap, err, dp_cost, dp_link,
                     leaf_max, s_w);
      ps += tile_s[tile];
      pm += tile_m[tile];
    }
    // next round (the k_ploc_advance rules, alike in every CTA)
    const uint32_t merged = v[3];
    n = v[2];
    node_next += merged;
    rounds += merged > 0 ? 1u : 0u;
    par ^= 1u;
    iters++;
    if (n <= PLOC_SMALL || merged == 0) done = true;
    if (!grid_sync(bar, err)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ploc_state[kPlocN] = n;
    ploc_state[kPlocNext] = node_next;
    ploc_state[kPlocRounds] = rounds;
    ploc_state[kPlocTiles] = (n + PLOC_BLOCK - 1) / PLOC_BLOCK;
    ploc_state[kPlocParity] = par;
    ploc_state[kPlocDone] = done ? 1u : 0u;
    ploc_state[kPlocIters] = iters;
  }
}

// The line of p into L2, for a read of the loop's next turn.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Area of the box around clusters j and j + 1; infinite where they are no
// neighbours (the ends, another segment).
__device__ __forceinline__ float ploc_adjacent(const float4* clo, const float4* chi, uint32_t n, int j) {
  if (j < 0 || j + 1 >= (int)n) return INFINITY;
  const float4 a = clo[j], b = chi[j], c = clo[j + 1], d = chi[j + 1];
  if (__float_as_uint(a.w) != __float_as_uint(c.w)) return INFINITY;
  return half_area(f3min(make_float3(a.x, a.y, a.z), make_float3(c.x, c.y, c.z)),
                   f3max(make_float3(b.x, b.y, b.z), make_float3(d.x, d.y, d.z)));
}

// Exclusive block scan of two values (a, b); returns (prefix a, prefix b) and
// the block totals in *ta, *tb.  All THREADS threads call it.
template <int THREADS = 256>
__device__ __forceinline__ uint2 block_excl_scan2(uint32_t a, uint32_t b, uint32_t* ta, uint32_t* tb) {
  constexpr int kWarps = THREADS / 32;
  static_assert(kWarps <= 32, "every warp adds up the warps' sums");
  __shared__ uint2 s_ab[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t xa = a, xb = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t ya = __shfl_up_sync(0xFFFFFFFFu, xa, o), yb = __shfl_up_sync(0xFFFFFFFFu, xb, o);
    if (lane >= o) {
      xa += ya;
      xb += yb;
    }
  }
  if (lane == 31) s_ab[warp] = make_uint2(xa, xb);
  __syncthreads();
  const uint2 w = s_ab[min(lane, kWarps - 1)];
  const bool all = lane < kWarps, before = lane < warp;
  *ta = __reduce_add_sync(0xFFFFFFFFu, all ? w.x : 0u);
  *tb = __reduce_add_sync(0xFFFFFFFFu, all ? w.y : 0u);
  const uint32_t oa = __reduce_add_sync(0xFFFFFFFFu, before ? w.x : 0u), ob = __reduce_add_sync(0xFFFFFFFFu, before ? w.y : 0u);
  __syncthreads();  // s_ab is used again by the next call
  return make_uint2(oa + xa - a, ob + xb - b);
}

// Every CTA of a cooperative launch gives a pair (a, b) of its thread 0; after the
// grid barrier in here it has the sums of the pairs of the CTAs before it (in x and
// y) and of all CTAs (z, w).  All threads call it; words holds gridDim.x pairs, and
// another grid barrier lies between two calls.  False as grid_sync.  Reading tagged
// words in a loop until all have arrived, without the barrier, is slower (152 CTAs
// of 1024 threads: rounds of the 4M soup 580 us against 530, of 300k triangles 151
// against 107; collapse of 8k triangles 50 against 46): the CTAs that wait then
// delay the stores they wait for.
template <int THREADS>
__device__ __forceinline__ bool grid_sums(uint2* __restrict__ words, uint32_t a, uint32_t b, uint4& sums,
                                          GridBarrier* bar, unsigned int* err) {
  __shared__ uint4 s_sums[THREADS / 32];
  if (threadIdx.x == 0) __stcg(words + blockIdx.x, make_uint2(a, b));
  if (!grid_sync(bar, err)) return false;
  uint4 s = make_uint4(0, 0, 0, 0);
  for (uint32_t c = threadIdx.x; c < gridDim.x; c += THREADS) {
    const uint2 v = __ldcg(words + c);
    s.z += v.x;
    s.w += v.y;
    if (c < blockIdx.x) s.x += v.x, s.y += v.y;
  }
  const uint32_t warps = min(THREADS / 32u, (gridDim.x + 31u) / 32u);  // that read a word
  if (threadIdx.x >> 5 < warps) {
    s = make_uint4(__reduce_add_sync(0xFFFFFFFFu, s.x), __reduce_add_sync(0xFFFFFFFFu, s.y),
                   __reduce_add_sync(0xFFFFFFFFu, s.z), __reduce_add_sync(0xFFFFFFFFu, s.w));
    if ((threadIdx.x & 31) == 0) s_sums[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  sums = make_uint4(0, 0, 0, 0);
  for (uint32_t k = 0; k < warps; k++) {
    const uint4 o = s_sums[k];
    sums.x += o.x;
    sums.y += o.y;
    sums.z += o.z;
    sums.w += o.w;
  }
  return true;
}

// k_ploc_all for radius 1.  With one neighbour on either side a cluster's nearest
// neighbour is the side of the smaller adjacent area (the left one in a tie, the
// least (area, index)), so clusters i and i + 1 merge exactly where the adjacent
// areas have a local minimum: a[i - 1] > a[i] <= a[i + 1].  That needs no window in
// shared memory: the warps of a CTA take the 32-cluster tiles of its run in turn,
// (1) the merges of a tile as a bit mask from shuffles and a ballot, the run's
// offsets by one block scan over the tiles, [barrier], (2) the tiles' outputs,
// [barrier].  The tile-per-CTA form waits at six CTA barriers per 256 clusters,
// which the threads that compute collapse costs reach last (17 of its 29 stall
// cycles per issue).  tile_m, tile_s, tile_p: one word per tile.  One CTA per SM: a
// round ends at two grid barriers, and 152 CTAs arrive sooner and read fewer sums
// than 608 of 256 threads.  Rounds of 8k / 300k / 1M / 4M triangles: 23 / 105 / 190 /
// 527 us, with 4 x 256 threads per SM 27 / 129 / 216 / 563, with 2 x 512 23 / 110 /
// 196 / 534 (tile per CTA: 732 us at 4M).  What does not fit L2 waits for memory with
// 32 warps per SM: prefetching each warp's next tile makes it 501 us at 4M (two tiles
// ahead 508, four 517; collapse costs by full warps of merges 576).
constexpr int PLOC1_THREADS = 1024, PLOC1_CTAS = 1;
__global__ void __launch_bounds__(PLOC1_THREADS, PLOC1_CTAS)
    k_ploc_rounds1(const PlocBufs bufs, uint32_t* __restrict__ ploc_state, uint32_t* tile_m, uint32_t* tile_s,
                   uint32_t* tile_p, uint2* cta_sums, float4* __restrict__ bnbox, uint32_t* __restrict__ bncnt,
                   uint32_t node_cap, float4* __restrict__ dp_cost, uint4* __restrict__ dp_link, uint32_t leaf_max,
                   GridBarrier* bar, unsigned int* err) {
  constexpr uint32_t kWarps = PLOC1_THREADS / 32;
  __shared__ uint32_t s_before;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  uint32_t n = __ldcg(ploc_state + kPlocN), node_next = __ldcg(ploc_state + kPlocNext);
  uint32_t par = __ldcg(ploc_state + kPlocParity) & 1u, rounds = __ldcg(ploc_state + kPlocRounds);
  uint32_t iters = __ldcg(ploc_state + kPlocIters);
  bool done = __ldcg(ploc_state + kPlocDone) != 0u;
  while (!done && iters < kPlocMaxIters) {
    const float4 *clo = bufs.clo[par], *chi = bufs.chi[par];
    const uint32_t ntiles = (n + 31u) / 32u;
    const uint32_t per = (ntiles + gridDim.x - 1) / gridDim.x;
    const uint32_t t0 = min(blockIdx.x * per, ntiles), t1 = min(t0 + per, ntiles);
    // (1) merges of the run's tiles
    for (uint32_t t = t0 + warp; t < t1; t += kWarps) {
      const int i = (int)(32u * t + lane);
      if (const uint32_t p = 32u * (t + kWarps) + lane; t + kWarps < t1 && p < n) {  // the next tile's
        prefetch_l2(clo + p);
        prefetch_l2(chi + p);
      }
      const float a = ploc_adjacent(clo, chi, n, i);
      const float edge = lane < 2u ? ploc_adjacent(clo, chi, n, lane ? (int)(32u * t) + 32 : (int)(32u * t) - 1) : 0.f;
      float left = __shfl_up_sync(0xFFFFFFFFu, a, 1), right = __shfl_down_sync(0xFFFFFFFFu, a, 1);
      const float e0 = __shfl_sync(0xFFFFFFFFu, edge, 0), e1 = __shfl_sync(0xFFFFFFFFu, edge, 1);
      if (lane == 0) left = e0;
      if (lane == 31) right = e1;
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, a != INFINITY && a < left && a <= right);
      if (lane == 0) tile_m[t] = m;
    }
    if (warp == 0 && t0 < t1) {  // whether the pair across the run's start merges
      const float a = lane < 3u ? ploc_adjacent(clo, chi, n, (int)(32u * t0) - 2 + (int)lane) : 0.f;
      const float b = __shfl_sync(0xFFFFFFFFu, a, 0), c = __shfl_sync(0xFFFFFFFFu, a, 1), d = __shfl_sync(0xFFFFFFFFu, a, 2);
      if (lane == 0) s_before = c != INFINITY && c < b && c <= d ? 1u : 0u;
    }
    __syncthreads();
    const uint32_t before = s_before;
    uint32_t ps = 0, pm = 0;
    for (uint32_t k0 = t0; k0 < t1; k0 += PLOC1_THREADS) {
      const uint32_t t = k0 + threadIdx.x;
      uint32_t a = 0, b = 0;
      if (t < t1) {
        const uint32_t m = tile_m[t], carry = t > t0 ? tile_m[t - 1] >> 31 : before;
        a = min(n - 32u * t, 32u) - __popc(m << 1) - carry;
        b = __popc(m);
      }
      uint32_t ta, tb;
      const uint2 e = block_excl_scan2<PLOC1_THREADS>(a, b, &ta, &tb);
      if (t < t1) {
        tile_s[t] = ps + e.x;
        tile_p[t] = pm + e.y;
      }
      ps += ta;
      pm += tb;
    }
    // (2) this CTA's offsets and the round's totals (survivors, merges), then its
    // tiles' outputs
    uint4 v;
    if (!grid_sums<PLOC1_THREADS>(cta_sums, ps, pm, v, bar, err)) break;
    for (uint32_t t = t0 + warp; t < t1; t += kWarps) {
      if (const uint32_t p = 32u * (t + kWarps) + lane; t + kWarps < t1 && p < n) {
        prefetch_l2(clo + p);
        prefetch_l2(chi + p);
        prefetch_l2(bufs.cidx[par] + p);
      }
      const uint32_t m = tile_m[t], i = 32u * t + lane, carry = t > t0 ? tile_m[t - 1] >> 31 : before;
      const uint32_t s0 = tile_s[t], m0 = tile_p[t];
      const uint32_t in = min(n - 32u * t, 32u), absorbed = (m << 1) | carry;
      const uint32_t alive = (in == 32u ? 0xFFFFFFFFu : (1u << in) - 1u) & ~absorbed;
      if (alive >> lane & 1u)
        ploc_emit_one(bufs, par, i, m >> lane & 1u ? i + 1u : i, v.x + s0 + __popc(alive & lt),
                      node_next + v.y + m0 + __popc(m & lt), n, bnbox, bncnt, node_cap, err, dp_cost, dp_link, leaf_max);
    }
    // next round (the k_ploc_advance rules, alike in every CTA)
    const uint32_t merged = v.w;
    n = v.z;
    node_next += merged;
    rounds += merged > 0 ? 1u : 0u;
    par ^= 1u;
    iters++;
    if (n <= PLOC_SMALL || merged == 0) done = true;
    if (!grid_sync(bar, err)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ploc_state[kPlocN] = n;
    ploc_state[kPlocNext] = node_next;
    ploc_state[kPlocRounds] = rounds;
    ploc_state[kPlocTiles] = (n + PLOC_BLOCK - 1) / PLOC_BLOCK;
    ploc_state[kPlocParity] = par;
    ploc_state[kPlocDone] = done ? 1u : 0u;
    ploc_state[kPlocIters] = iters;
  }
}

// Finishes clustering of the n <= PLOC_SMALL clusters left by the rounds
// inside one CTA (n and the next node index from ploc_state, where the final
// node count is written back).
__global__ void __launch_bounds__(PLOC_SMALL_THREADS) k_ploc_small(const float4* __restrict__ clo_a,
                                                                  const float4* __restrict__ chi_a,
                                                                  const uint32_t* __restrict__ cidx_a,
                                                                  const float4* __restrict__ clo_b,
                                                                  const float4* __restrict__ chi_b,
                                                                  const uint32_t* __restrict__ cidx_b,
                                                                  uint32_t* __restrict__ ploc_state,
                                                                  float4* __restrict__ bnbox,
                                                                  uint32_t* __restrict__ bncnt, uint32_t* root_out,
                                                                  uint32_t* iters_out, uint32_t node_cap,
                                                                  uint32_t* err, uint32_t nseg, int radius,
                                                                  float4* __restrict__ dp_cost,
                                                                  uint4* __restrict__ dp_link, uint32_t leaf_max) {
  extern __shared__ unsigned char smem[];
  float3* s_lo = reinterpret_cast<float3*>(smem);
  float3* s_hi = s_lo + PLOC_SMALL;
  uint32_t* s_idx = reinterpret_cast<uint32_t*>(s_hi + PLOC_SMALL);
  uint32_t* s_nn = s_idx + PLOC_SMALL;
  uint32_t* s_seg = s_nn + PLOC_SMALL;
  uint32_t* s_cnt = s_seg + PLOC_SMALL;
  __shared__ uint32_t s_w[32];
  __shared__ uint32_t s_tot[2];
  constexpr int EPT = PLOC_SMALL / PLOC_SMALL_THREADS;  // elements per thread (contiguous)
  const uint32_t n0 = ploc_state[kPlocN], node_next0 = ploc_state[kPlocNext];
  const bool in_b = ploc_state[kPlocParity] != 0;
  const float4* __restrict__ clo = in_b ? clo_b : clo_a;
  const float4* __restrict__ chi = in_b ? chi_b : chi_a;
  const uint32_t* __restrict__ cidx = in_b ? cidx_b : cidx_a;
  if (n0 > PLOC_SMALL) {  // the rounds did not get below the threshold (too few enqueued)
    if (threadIdx.x == 0) atomicOr(err, kErrBuild);
    return;
  }
  for (uint32_t k = threadIdx.x; k < n0; k += blockDim.x) {
    const float4 a = clo[k], b = chi[k];
    s_lo[k] = make_float3(a.x, a.y, a.z);
    s_hi[k] = make_float3(b.x, b.y, b.z);
    s_idx[k] = cidx[k];
    s_seg[k] = __float_as_uint(a.w);
    s_cnt[k] = __float_as_uint(b.w);
  }
  uint32_t n = n0, node_next = node_next0, iters = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // every round merges at least the closest pair of each segment that still
  // has two clusters, so n0 - 1 rounds always suffice; the bound only guards
  // against a logic error.  A round without merges ends the clustering.
  while (n > 1) {
    if (iters >= PLOC_SMALL) {
      if (threadIdx.x == 0) atomicOr(err, kErrBuild);
      break;
    }
    iters++;
    // nearest neighbours
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      const float3 lo = s_lo[i], hi = s_hi[i];
      const uint32_t seg = s_seg[i];
      unsigned long long best = ~0ull;
      for (int o = -radius; o <= radius; o++) {
        const int j = (int)i + o;
        if (o == 0 || j < 0 || j >= (int)n || s_seg[j] != seg) continue;
        const float a = half_area(f3min(lo, s_lo[j]), f3max(hi, s_hi[j]));
        const unsigned long long key = ((unsigned long long)__float_as_uint(a) << 32) | (uint32_t)j;
        best = key < best ? key : best;
      }
      s_nn[i] = best != ~0ull ? (uint32_t)best : i;
    }
    __syncthreads();
    // flags for this thread's contiguous chunk
    uint32_t cs = 0, cm = 0;
    int fs[EPT], fm[EPT];
    const uint32_t i0 = threadIdx.x * EPT;
#pragma unroll
    for (int e = 0; e < EPT; e++) {
      const uint32_t i = i0 + e;
      fs[e] = fm[e] = 0;
      if (i < n) {
        const uint32_t j = s_nn[i];
        const bool mutual = j != i && s_nn[j] == i;
        fm[e] = mutual && i < j;
        fs[e] = !(mutual && j < i);
      }
      cs += fs[e];
      cm += fm[e];
    }
    // block exclusive scan of (cs, cm) packed into one 32-bit word (both < 2^16)
    uint32_t x = cs | (cm << 16);
    const uint32_t mine = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = s_w[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
        if (lane >= o) w += y;
      }
      s_w[lane] = w;
      if (lane == 31) { s_tot[0] = w & 0xFFFFu; s_tot[1] = w >> 16; }
    }
    __syncthreads();
    const uint32_t excl = (warp ? s_w[warp - 1] : 0u) + (x - mine);
    uint32_t ps = excl & 0xFFFFu, pm = excl >> 16;
    // gather outputs into registers
    float3 olo[EPT], ohi[EPT];
    uint32_t oidx[EPT], opos[EPT], oseg[EPT], ocnt[EPT];
#pragma unroll
    for (int e = 0; e < EPT; e++) {
      const uint32_t i = i0 + e;
      opos[e] = 0xFFFFFFFFu;
      if (i < n && fs[e]) {
        float3 lo = s_lo[i], hi = s_hi[i];
        uint32_t id = s_idx[i], cnt = s_cnt[i];
        if (fm[e]) {
          const uint32_t j = s_nn[i];
          const uint32_t nid = node_next + pm;
          const uint32_t l = id, r = s_idx[j];
          if (nid >= node_cap) {
            atomicOr(err, kErrBuild);
            break;
          }
          const uint32_t cnt_l = cnt, cnt_r = s_cnt[j];
          const float Al = cnt_l == 1 ? half_area(lo, hi) : 0.f;
          const float Ar = cnt_r == 1 ? half_area(s_lo[j], s_hi[j]) : 0.f;
          lo = f3min(lo, s_lo[j]);
          hi = f3max(hi, s_hi[j]);
          bnbox[2 * (size_t)nid] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(l));
          bnbox[2 * (size_t)nid + 1] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(r));
          cnt = cnt_l + cnt_r;
          bncnt[nid] = cnt;
          // children come from earlier rounds: their costs were stored before
          // this round's barriers
          if (dp_cost) dp_node(dp_cost, dp_link, nid, l, r, half_area(lo, hi), cnt_l, cnt_r, Al, Ar, leaf_max);
          id = nid;
          pm++;
        }
        olo[e] = lo;
        ohi[e] = hi;
        oidx[e] = id;
        oseg[e] = s_seg[i];
        ocnt[e] = cnt;
        opos[e] = ps++;
      }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < EPT; e++) {
      if (opos[e] != 0xFFFFFFFFu) {
        s_lo[opos[e]] = olo[e];
        s_hi[opos[e]] = ohi[e];
        s_idx[opos[e]] = oidx[e];
        s_seg[opos[e]] = oseg[e];
        s_cnt[opos[e]] = ocnt[e];
      }
    }
    const uint32_t merged = s_tot[1];
    node_next += merged;
    n = s_tot[0];
    __syncthreads();
    if (merged == 0) break;
  }
  // one root per segment (nseg == 1: the single tree's root)
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
    const uint32_t seg = nseg > 1 ? s_seg[k] : 0u;
    if (seg < nseg) root_out[seg] = s_idx[k];
  }
  if (threadIdx.x == 0) {
    *iters_out += iters;
    ploc_state[kPlocNext] = node_next;  // binary nodes in use: [0, node_next)
  }
}

// k_ploc_small for radius 1, where clusters merge at the local minima of the
// adjacent areas (k_ploc_rounds1).  A round of one CTA is a chain of steps between
// barriers, so the new nodes' collapse costs -- two dependent L2 reads and 28
// sums, the longest step -- are left to the next round, which reads them while it
// works on its own areas and merges, and the last 32 clusters to one warp
// (ploc_last).  The last 4,096 clusters of the 4M soup: 174 us with the costs inside
// the round, 96 us so, 88 us with the last warp; 4,096 of 8k triangles 44 and 35 us.
struct PlocTask {       // costs to compute: node task_base + index
  uint32_t l, r;        // children
  float A, Al, Ar;      // areas (Al, Ar: of primitive children)
  uint32_t cnt;         // triangles of the children, 255 at most, 8 bits each
};
constexpr size_t kPlocFinishSmem = (size_t)PLOC_SMALL * (2 * sizeof(float3) + 3 * sizeof(uint32_t)) +
                                   (PLOC_SMALL + 2) * sizeof(float) + (PLOC_SMALL / 2) * sizeof(PlocTask);

// The last 32 clusters, by one warp: a cluster per lane with its collapse costs, a
// round in registers and shuffles instead of four CTA barriers (8 us less for the ten
// rounds or so).
struct PlocLast {
  uint32_t n, node_next, iters;
  uint8_t src[32];  // lane of each survivor
};
__device__ __noinline__ void ploc_last(float3* s_lo, float3* s_hi, uint32_t* s_idx, uint32_t* s_seg, uint32_t* s_cnt,
                                       PlocLast& st, float4* __restrict__ bnbox, uint32_t* __restrict__ bncnt,
                                       uint32_t node_cap, uint32_t* err, float4* __restrict__ dp_cost,
                                       uint4* __restrict__ dp_link, uint32_t leaf_max) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  uint32_t n = st.n, node_next = st.node_next, iters = st.iters;
  float3 lo = s_lo[lane], hi = s_hi[lane];  // of lanes past n: not used
  uint32_t id = s_idx[lane], seg = s_seg[lane], cnt = s_cnt[lane];
  float c[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (dp_cost && lane < n) dp_child_costs(dp_cost, id, cnt, half_area(lo, hi), c);
  while (n > 1) {
    iters++;
    const float3 rlo = make_float3(__shfl_down_sync(0xFFFFFFFFu, lo.x, 1), __shfl_down_sync(0xFFFFFFFFu, lo.y, 1),
                                   __shfl_down_sync(0xFFFFFFFFu, lo.z, 1));
    const float3 rhi = make_float3(__shfl_down_sync(0xFFFFFFFFu, hi.x, 1), __shfl_down_sync(0xFFFFFFFFu, hi.y, 1),
                                   __shfl_down_sync(0xFFFFFFFFu, hi.z, 1));
    const uint32_t rid = __shfl_down_sync(0xFFFFFFFFu, id, 1), rcnt = __shfl_down_sync(0xFFFFFFFFu, cnt, 1);
    const uint32_t rseg = __shfl_down_sync(0xFFFFFFFFu, seg, 1);
    const float3 ulo = f3min(lo, rlo), uhi = f3max(hi, rhi);
    const float a = lane + 1u < n && seg == rseg ? half_area(ulo, uhi) : INFINITY;
    float left = __shfl_up_sync(0xFFFFFFFFu, a, 1), right = __shfl_down_sync(0xFFFFFFFFu, a, 1);
    if (lane == 0u) left = INFINITY;
    if (lane == 31u) right = INFINITY;
    const bool merge = a != INFINITY && a < left && a <= right;
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, merge);
    if (m == 0u) break;
    if (node_next + __popc(m) > node_cap) {
      if (lane == 0u) atomicOr(err, kErrBuild);
      break;
    }
    float cr[8];
#pragma unroll
    for (int i = 0; i < 8; i++) cr[i] = __shfl_down_sync(0xFFFFFFFFu, c[i], 1);
    if (merge) {
      const uint32_t nid = node_next + __popc(m & lt);
      bnbox[2 * (size_t)nid] = make_float4(ulo.x, ulo.y, ulo.z, __uint_as_float(id));
      bnbox[2 * (size_t)nid + 1] = make_float4(uhi.x, uhi.y, uhi.z, __uint_as_float(rid));
      lo = ulo;
      hi = uhi;
      cnt += rcnt;
      bncnt[nid] = cnt;
      if (dp_cost) {
        float cn[8];
        dp_combine(dp_cost, dp_link, nid, id, rid, a, cnt, c, cr, leaf_max, cn);
#pragma unroll
        for (int i = 0; i < 8; i++) c[i] = cn[i];
      }
      id = nid;
    }
    // the survivors move up
    const uint32_t alive = (n == 32u ? 0xFFFFFFFFu : (1u << n) - 1u) & ~(m << 1);
    if (alive >> lane & 1u) st.src[__popc(alive & lt)] = (uint8_t)lane;
    __syncwarp();
    node_next += __popc(m);
    n = __popc(alive);
    const int src = lane < n ? st.src[lane] : 31;
    lo = make_float3(__shfl_sync(0xFFFFFFFFu, lo.x, src), __shfl_sync(0xFFFFFFFFu, lo.y, src), __shfl_sync(0xFFFFFFFFu, lo.z, src));
    hi = make_float3(__shfl_sync(0xFFFFFFFFu, hi.x, src), __shfl_sync(0xFFFFFFFFu, hi.y, src), __shfl_sync(0xFFFFFFFFu, hi.z, src));
    id = __shfl_sync(0xFFFFFFFFu, id, src);
    seg = __shfl_sync(0xFFFFFFFFu, seg, src);
    cnt = __shfl_sync(0xFFFFFFFFu, cnt, src);
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = __shfl_sync(0xFFFFFFFFu, c[i], src);
    __syncwarp();  // st.src is written again
  }
  if (lane < n) {
    s_idx[lane] = id;
    s_seg[lane] = seg;
  }
  if (lane == 0u) st.n = n, st.node_next = node_next, st.iters = iters;
}

__global__ void __launch_bounds__(PLOC_SMALL_THREADS) k_ploc_finish1(const PlocBufs bufs, uint32_t* __restrict__ ploc_state,
                                                                     float4* __restrict__ bnbox,
                                                                     uint32_t* __restrict__ bncnt, uint32_t* root_out,
                                                                     uint32_t* iters_out, uint32_t node_cap,
                                                                     uint32_t* err, uint32_t nseg,
                                                                     float4* __restrict__ dp_cost,
                                                                     uint4* __restrict__ dp_link, uint32_t leaf_max) {
  extern __shared__ unsigned char smem[];
  float3* s_lo = reinterpret_cast<float3*>(smem);
  float3* s_hi = s_lo + PLOC_SMALL;
  uint32_t* s_idx = reinterpret_cast<uint32_t*>(s_hi + PLOC_SMALL);
  uint32_t* s_seg = s_idx + PLOC_SMALL;
  uint32_t* s_cnt = s_seg + PLOC_SMALL;
  float* s_area = reinterpret_cast<float*>(s_cnt + PLOC_SMALL) + 1;  // s_area[-1 .. n]: box of clusters i, i + 1
  PlocTask* s_task = reinterpret_cast<PlocTask*>(s_area + PLOC_SMALL + 1);
  __shared__ uint32_t s_w[32];
  constexpr int EPT = PLOC_SMALL / PLOC_SMALL_THREADS;
  const uint32_t n0 = ploc_state[kPlocN], node_next0 = ploc_state[kPlocNext], par = ploc_state[kPlocParity] & 1u;
  if (n0 > PLOC_SMALL) {  // the rounds did not get below the threshold (too few enqueued)
    if (threadIdx.x == 0) atomicOr(err, kErrBuild);
    return;
  }
  for (uint32_t k = threadIdx.x; k < n0; k += blockDim.x) {
    const float4 a = bufs.clo[par][k], b = bufs.chi[par][k];
    s_lo[k] = make_float3(a.x, a.y, a.z);
    s_hi[k] = make_float3(b.x, b.y, b.z);
    s_idx[k] = bufs.cidx[par][k];
    s_seg[k] = __float_as_uint(a.w);
    s_cnt[k] = __float_as_uint(b.w);
  }
  if (threadIdx.x == 0) s_area[-1] = INFINITY;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  uint32_t n = n0, node_next = node_next0, iters = 0, tasks = 0;  // tasks: nodes of the last round
  bool failed = false;
  auto pay = [&](uint32_t k) {  // the collapse costs of task k
    const PlocTask t = s_task[k];
    dp_node(dp_cost, dp_link, node_next - tasks + k, t.l, t.r, t.A, t.cnt & 0xFFu, t.cnt >> 8, t.Al, t.Ar, leaf_max);
  };
  __syncthreads();
  // every round merges at least the closest pair of each segment that still
  // has two clusters, so n0 - 1 rounds always suffice; the bound only guards
  // against a logic error.  A round without merges ends the clustering.
  bool stalled = false;  // a round merged nothing
  while (n > 32 && !failed) {
    if (iters >= PLOC_SMALL) {
      if (threadIdx.x == 0) atomicOr(err, kErrBuild);
      break;
    }
    iters++;
    // adjacent areas, and the costs of the last round's nodes
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
      s_area[i] = i + 1 < n && s_seg[i] == s_seg[i + 1]
                      ? half_area(f3min(s_lo[i], s_lo[i + 1]), f3max(s_hi[i], s_hi[i + 1]))
                      : INFINITY;
    for (uint32_t k = threadIdx.x; k < tasks; k += blockDim.x) pay(k);
    __syncthreads();
    // the warp's tiles of 32 clusters: merges as bit masks
    const uint32_t per = (n + PLOC_SMALL_THREADS - 1) / PLOC_SMALL_THREADS, w0 = warp * 32u * per;
    uint32_t mask[EPT], alive[EPT], survivors = 0, merges = 0, carry = 0;
    if (w0 > 0 && w0 < n) {
      const float a = s_area[w0 - 1];
      carry = a != INFINITY && a < s_area[(int)w0 - 2] && a <= s_area[w0] ? 1u : 0u;
    }
#pragma unroll
    for (int e = 0; e < EPT; e++) {
      const uint32_t i = w0 + 32u * e + lane;
      bool m = false;
      if ((uint32_t)e < per && i < n) {
        const float a = s_area[i];
        m = a != INFINITY && a < s_area[(int)i - 1] && a <= s_area[i + 1];
      }
      mask[e] = __ballot_sync(0xFFFFFFFFu, m);
      alive[e] = __ballot_sync(0xFFFFFFFFu, (uint32_t)e < per && i < n) & ~((mask[e] << 1) | carry);
      carry = mask[e] >> 31;
      survivors += __popc(alive[e]);
      merges += __popc(mask[e]);
    }
    if (lane == 0) s_w[warp] = survivors | (merges << 16);  // both below 2^16
    __syncthreads();
    uint32_t x = s_w[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, x, 31);
    const uint32_t before = __shfl_sync(0xFFFFFFFFu, x, warp ? warp - 1 : 0);
    uint32_t ps = warp ? before & 0xFFFFu : 0u, pm = warp ? before >> 16 : 0u;
    failed = node_next + (total >> 16) > node_cap;
    // outputs into registers, the new nodes and their tasks
    float3 olo[EPT], ohi[EPT];
    uint32_t oidx[EPT], oseg[EPT], ocnt[EPT], opos[EPT];
#pragma unroll
    for (int e = 0; e < EPT; e++) {
      opos[e] = 0xFFFFFFFFu;
      if ((alive[e] >> lane & 1u) && !failed) {
        const uint32_t i = w0 + 32u * e + lane;
        float3 lo = s_lo[i], hi = s_hi[i];
        uint32_t id = s_idx[i], cnt = s_cnt[i];
        if (mask[e] >> lane & 1u) {
          const uint32_t q = pm + __popc(mask[e] & lt), nid = node_next + q;
          const uint32_t l = id, r = s_idx[i + 1], cnt_l = cnt, cnt_r = s_cnt[i + 1];
          const float3 rlo = s_lo[i + 1], rhi = s_hi[i + 1];
          PlocTask t;
          t.l = l;
          t.r = r;
          t.Al = cnt_l == 1 ? half_area(lo, hi) : 0.f;
          t.Ar = cnt_r == 1 ? half_area(rlo, rhi) : 0.f;
          t.cnt = min(cnt_l, 255u) | (min(cnt_r, 255u) << 8);
          lo = f3min(lo, rlo);
          hi = f3max(hi, rhi);
          t.A = half_area(lo, hi);
          s_task[q] = t;
          bnbox[2 * (size_t)nid] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(l));
          bnbox[2 * (size_t)nid + 1] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(r));
          cnt = cnt_l + cnt_r;
          bncnt[nid] = cnt;
          id = nid;
        }
        olo[e] = lo;
        ohi[e] = hi;
        oidx[e] = id;
        oseg[e] = s_seg[i];
        ocnt[e] = cnt;
        opos[e] = ps + __popc(alive[e] & lt);
      }
      ps += __popc(alive[e]);
      pm += __popc(mask[e]);
    }
    __syncthreads();
    if (failed) {
      if (threadIdx.x == 0) atomicOr(err, kErrBuild);
      tasks = 0;
      break;
    }
#pragma unroll
    for (int e = 0; e < EPT; e++) {
      if (opos[e] != 0xFFFFFFFFu) {
        s_lo[opos[e]] = olo[e];
        s_hi[opos[e]] = ohi[e];
        s_idx[opos[e]] = oidx[e];
        s_seg[opos[e]] = oseg[e];
        s_cnt[opos[e]] = ocnt[e];
      }
    }
    tasks = total >> 16;
    node_next += tasks;
    n = total & 0xFFFFu;
    if (!dp_cost) tasks = 0;
    __syncthreads();
    if ((total >> 16) == 0) {
      stalled = true;
      break;
    }
  }
  for (uint32_t k = threadIdx.x; k < tasks; k += blockDim.x) pay(k);
  __shared__ PlocLast s_last;
  if (threadIdx.x == 0) s_last.n = n, s_last.node_next = node_next, s_last.iters = iters;
  __syncthreads();
  if (n > 1 && n <= 32 && !failed && !stalled) {
    if (warp == 0) ploc_last(s_lo, s_hi, s_idx, s_seg, s_cnt, s_last, bnbox, bncnt, node_cap, err, dp_cost, dp_link, leaf_max);
    __syncthreads();
    n = s_last.n;
    node_next = s_last.node_next;
    iters = s_last.iters;
  }
  // one root per segment (nseg == 1: the single tree's root)
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
    const uint32_t seg = nseg > 1 ? s_seg[k] : 0u;
    if (seg < nseg) root_out[seg] = s_idx[k];
  }
  if (threadIdx.x == 0) {
    *iters_out += iters;
    ploc_state[kPlocNext] = node_next;  // binary nodes in use: [0, node_next)
  }
}

// ---------------------------------------------------------------------------
// 5. collapse to 8-wide quantised nodes
// ---------------------------------------------------------------------------

// Adds the per-thread values a, b to acc[0], acc[1] with one atomic each per
// CTA; every thread of the CTA calls it (blockDim.x a multiple of 32).
__device__ __forceinline__ void block_add2(double a, double b, double* acc) {
  __shared__ double s_a[32], s_b[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xFFFFFFFFu, a, o);
    b += __shfl_down_sync(0xFFFFFFFFu, b, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) {
    s_a[warp] = a;
    s_b[warp] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tb = 0.0;
    for (int w = 0; w < nw; w++) {
      ta += s_a[w];
      tb += s_b[w];
    }
    if (ta != 0.0) atomicAdd(acc + 0, ta);
    if (tb != 0.0) atomicAdd(acc + 1, tb);
  }
}

struct BinTree {
  const float4* box;  // two per node: (lo.xyz, left), (hi.xyz, right)
  const uint32_t* cnt;
  uint32_t nleaves;
  uint32_t leaf_max;  // subtrees of at most this many triangles may become leaves
  uint32_t robust;    // write raw vertices into triangle records
  const uint4* link;  // (left, right, SAH-optimal collapse decisions); null: greedy collapse
};

__device__ __forceinline__ bool bt_leaf(const BinTree& t, uint32_t k) { return k < t.nleaves; }
// Triangles of binary node k as the collapse needs them: with one-triangle
// leaves only "one (a primitive) or more" matters, so no count is read (2
// stands for any internal node).
__device__ __forceinline__ uint32_t bt_cnt(const BinTree& t, uint32_t k) {
  if (t.leaf_max == 1) return bt_leaf(t, k) ? 1u : 2u;
  return bt_leaf(t, k) ? 1u : t.cnt[k];
}
__device__ __forceinline__ uint32_t bt_left(const BinTree& t, uint32_t k) { return __float_as_uint(t.box[2 * (size_t)k].w); }
__device__ __forceinline__ uint32_t bt_right(const BinTree& t, uint32_t k) { return __float_as_uint(t.box[2 * (size_t)k + 1].w); }
__device__ __forceinline__ float3 bt_lo(const BinTree& t, uint32_t k) {
  const float4 a = t.box[2 * (size_t)k];
  return make_float3(a.x, a.y, a.z);
}
__device__ __forceinline__ float3 bt_hi(const BinTree& t, uint32_t k) {
  const float4 a = t.box[2 * (size_t)k + 1];
  return make_float3(a.x, a.y, a.z);
}


// Chooses up to 8 children for the wide node that replaces binary node b, greedily
// (gpu.collapse=greedy).
__device__ int gather_children(const BinTree& t, uint32_t b, uint32_t kids[8]) {
  if (bt_leaf(t, b)) {
    kids[0] = b;
    return 1;
  }
  kids[0] = bt_left(t, b);
  kids[1] = bt_right(t, b);
  int nk = 2;
  while (nk < 8) {
    int best = -1;
    bool bestMand = false;
    float bestA = -1.0f;
    for (int i = 0; i < nk; i++) {
      const uint32_t c = kids[i];
      if (bt_leaf(t, c)) continue;
      const bool mand = bt_cnt(t, c) > t.leaf_max;
      const float A = half_area(bt_lo(t, c), bt_hi(t, c));
      if (!mand) {
        // opening a small subtree pays off only if its children's boxes
        // cover less area than its own box
        const uint32_t l = bt_left(t, c), r = bt_right(t, c);
        const float Al = half_area(bt_lo(t, l), bt_hi(t, l)), Ar = half_area(bt_lo(t, r), bt_hi(t, r));
        if (!(Al + Ar < A)) continue;
      }
      if ((mand && !bestMand) || (mand == bestMand && A > bestA)) {
        best = i;
        bestMand = mand;
        bestA = A;
      }
    }
    if (best < 0) break;
    const uint32_t c = kids[best];
    kids[best] = bt_left(t, c);
    kids[nk++] = bt_right(t, c);
  }
  return nk;
}

// The children of the wide node made from binary node b by the recorded decisions,
// gathered by the 8 lanes of a lane group (all 32 lanes call it; `have` is the
// group's).  An entry (n, i) -- node n may take up to i slots -- lives in the lane
// where its slots begin; a split keeps the right child there and sends the left
// child to the lane behind the right child's slots, so the children come out with
// the right subtrees first, and a wide node takes as many dependent reads as its
// binary subtree is deep, not as it has nodes.  A live lane returns its child in
// `kid`; live: the group's live lanes.
__device__ __forceinline__ void gather_group(const BinTree& t, uint32_t b, bool have, uint32_t& kid, uint32_t& live) {
  const uint32_t s = threadIdx.x & 7u, gshift = threadIdx.x & 24u;
  uint32_t n = kInvalidID, i = 0;
  if (have) {
    if (bt_leaf(t, b)) {
      if (s == 0) n = b, i = 1;
    } else {
      const uint4 lk = t.link[b];
      const uint32_t k = lk.z & 15u, rem = lk.z >> 4 & 15u;
      if (s == 0) n = lk.y, i = rem;
      if (s == rem) n = lk.x, i = k;
    }
  }
  for (;;) {
    bool split = false;
    uint32_t k = 0, left = 0, right = 0;
    if (i > 1u) {
      if (bt_leaf(t, n)) {
        i = 1;
      } else {
        const uint4 lk = t.link[n];
        left = lk.x;
        right = lk.y;
        const uint32_t d = (i < 5u ? lk.z >> (8u * (i - 1u)) : lk.w >> (8u * (i - 5u))) & 0xFFu;
        split = d != 0u;
        k = d & 15u;
        i = split ? d >> 4 : 1u;
      }
    }
    live = __ballot_sync(0xFFFFFFFFu, i > 0u) >> gshift & 0xFFu;
    if (!__any_sync(0xFFFFFFFFu, split)) break;
    const uint32_t dst = split ? s + i : 8u;
    const uint32_t below = live & ((1u << s) - 1u);
    const int src = below ? 31 - __clz(below) : 0;  // the entry whose slots this lane may lie in
    const uint32_t d2 = __shfl_sync(0xFFFFFFFFu, dst, src, 8), k2 = __shfl_sync(0xFFFFFFFFu, k, src, 8);
    const uint32_t l2 = __shfl_sync(0xFFFFFFFFu, left, src, 8);
    if (split) {
      n = right;
    } else if (i == 0u && below && d2 == s) {
      n = l2;
      i = k2;
    }
  }
  kid = n;
}

// Children and counts of item k of a level (all 32 lanes call it): kids[8k ..] =
// its children, *ni internal ones, *nt triangles in leaf children.
__device__ __forceinline__ void collapse_count_group(const BinTree& t, const uint32_t* __restrict__ items, uint32_t k,
                                                     bool have, uint32_t* __restrict__ kids, uint32_t* ni,
                                                     uint32_t* nt) {
  const uint32_t s = threadIdx.x & 7u, gshift = threadIdx.x & 24u;
  uint32_t kid = kInvalidID, live = 0;
  if (t.link) {
    gather_group(t, have ? __ldcg(items + k) : 0u, have, kid, live);
  } else {  // greedy: one lane gathers
    uint32_t kk[8];
    const int nk = have && s == 0u ? gather_children(t, items[k], kk) : 0;
    live = (1u << __shfl_sync(0xFFFFFFFFu, nk, 0, 8)) - 1u;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t c = __shfl_sync(0xFFFFFFFFu, j < nk ? kk[j] : kInvalidID, 0, 8);
      if ((uint32_t)j == s) kid = c;
    }
  }
  const uint32_t nk = __popc(live);
  const bool mine = live >> s & 1u;
  uint32_t cnt = mine ? bt_cnt(t, kid) : 0u;
  const bool inner = cnt > t.leaf_max;
  *ni = __popc(__ballot_sync(0xFFFFFFFFu, inner) >> gshift & 0xFFu);
  if (inner) cnt = 0;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o, 8);
  *nt = cnt;
  if (have) {
    if (mine) kids[8 * (size_t)k + __popc(live & ((1u << s) - 1u))] = kid;
    if (s >= nk) kids[8 * (size_t)k + s] = 0xFFFFFFFFu;
  }
}

// The collapse runs level by level from a state in device memory, so levels
// can be enqueued (or captured) before their sizes are known: [kColN] items of
// the current level, [kColBase] its first wide node, [kColTri] its first
// triangle record, [kColDepth] levels done, [kColErr] overflow, and from
// [kColLevels] the first node of every level (plus the end).  Kernels loop
// grid-stride over the level's items; a level with no items is a no-op.
enum : int { kColN = 0, kColBase = 1, kColTri = 2, kColDepth = 3, kColErr = 4, kColLevels = 8, kColMaxLevels = 64,
             kColStateWords = kColLevels + kColMaxLevels + 1 };

// Exclusive scan of one value per thread over a CTA of 1024 threads.
__device__ __forceinline__ uint32_t cta_excl_scan_1024(uint32_t v, uint32_t* s_w, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = s_w[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    s_w[lane] = w;
  }
  __syncthreads();
  const uint32_t excl = (warp ? s_w[warp - 1] : 0u) + x - v;
  total = s_w[31];
  __syncthreads();
  return excl;
}

// First level: the roots of the non-empty segments in segment order (one CTA
// of 1024 threads, nseg <= 4 x 1024); seg_index[s] = position of segment s's
// root (kInvalidID for an empty segment).  It also zeroes what the collapse adds
// to (cstate, the SAH sums, the leaf count, the barrier of k_collapse_all): as
// memsets these were four launches of a captured build.
__global__ void __launch_bounds__(1024) k_collapse_roots(const uint32_t* __restrict__ d_root, uint32_t nseg,
                                                         uint32_t nbin, uint32_t* __restrict__ items,
                                                         uint32_t* __restrict__ seg_index,
                                                         uint32_t* __restrict__ cstate, double* __restrict__ sah_acc,
                                                         uint32_t* __restrict__ leaf_count,
                                                         GridBarrier* __restrict__ bar) {
  __shared__ uint32_t s_w[32];
  for (uint32_t k = threadIdx.x; k < (uint32_t)kColStateWords; k += 1024) cstate[k] = 0;
  if (threadIdx.x < 2) sah_acc[threadIdx.x] = 0.0;
  if (threadIdx.x == 0) {
    *leaf_count = 0;
    if (bar) bar->count = 0;
  }
  __syncthreads();
  uint32_t r[4], cnt = 0;
  const uint32_t s0 = threadIdx.x * 4;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    r[q] = s0 + q < nseg ? d_root[s0 + q] : kInvalidID;
    if (r[q] != kInvalidID && r[q] >= nbin) r[q] = kInvalidID, cstate[kColErr] = 1u;
    cnt += r[q] != kInvalidID;
  }
  uint32_t total = 0;
  uint32_t pos = cta_excl_scan_1024(cnt, s_w, total);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (s0 + q >= nseg) break;
    if (r[q] != kInvalidID) items[pos] = r[q];
    seg_index[s0 + q] = r[q] != kInvalidID ? pos++ : kInvalidID;
  }
  if (threadIdx.x == 0) {
    cstate[kColN] = total;
    cstate[kColBase] = 0;
    cstate[kColTri] = 0;
    cstate[kColDepth] = 0;
  }
}

// leaf_root entry of a one-triangle leaf: the primitive index with this bit set
// (primitive indices and binary node ids are below 2^31)
constexpr uint32_t kLeafPrim = 0x80000000u;

// The two item buffers of the collapse levels: level d reads items[d & 1] and writes
// items[(d & 1) ^ 1] (d = cstate[kColDepth]), so every level runs the same kernels
// with the same arguments.
struct ColItems {
  uint32_t* items[2];
};

__global__ void __launch_bounds__(128) k_collapse_count(BinTree t, const ColItems ci,
                                                        const uint32_t* __restrict__ cstate,
                                                        uint32_t* __restrict__ kids_out, uint32_t* __restrict__ nint,
                                                        uint32_t* __restrict__ ntri) {
  const uint32_t nitems = cstate[kColN];
  const uint32_t* __restrict__ items = ci.items[cstate[kColDepth] & 1u];
  for (uint32_t k0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) >> 3; k0 < nitems; k0 += (gridDim.x * blockDim.x) >> 3) {
    const uint32_t k = k0 + ((threadIdx.x & 31u) >> 3);
    uint32_t ni, nt;
    collapse_count_group(t, items, k, k < nitems, kids_out, &ni, &nt);
    if (k < nitems && (threadIdx.x & 7u) == 0u) {
      nint[k] = ni;
      ntri[k] = nt;
    }
  }
}

// After a level: its wide nodes are written; the next level's items are its
// internal children (tot[0]), their triangles follow (tot[1]).  Level starts
// are kept for the first kColMaxLevels levels; max_levels bounds the depth of
// builds that need them all on the device (the host-driven build records
// them itself and has no bound: a chain-like binary tree, e.g. thousands of
// identical triangles, collapses into thousands of levels).
__global__ void k_collapse_advance(const uint32_t* __restrict__ tot, uint32_t* __restrict__ cstate, uint32_t node_cap,
                                   uint32_t max_levels) {
  if (threadIdx.x != 0) return;
  const uint32_t n = cstate[kColN];
  if (n == 0) {
    return;
  }
  const uint32_t d = cstate[kColDepth];
  if (d < (uint32_t)kColMaxLevels) cstate[kColLevels + d] = cstate[kColBase];
  const uint32_t base = cstate[kColBase] + n;
  cstate[kColBase] = base;
  cstate[kColTri] += tot[1];
  cstate[kColDepth] = d + 1;
  uint32_t next = tot[0];
  if ((next > 0 && d + 1 >= max_levels) || base + next > node_cap) {
    cstate[kColErr] = 1u;
    next = 0;
  }
  cstate[kColN] = next;
  if (next == 0 && d + 1 <= (uint32_t)kColMaxLevels) cstate[kColLevels + d + 1] = base;  // end of the last level
}

// A plane byte as a float, without a conversion: in the mantissa of 2^23.
__device__ __forceinline__ float byte_f(uint32_t q) { return __uint_as_float(0x4B000000u | q) - 8388608.0f; }

__device__ __forceinline__ uint32_t exp_for(float ext) {
  // smallest power of two 2^(E-127) with 255 * 2^(E-127) >= ext: with ext = m 2^e,
  // 1 <= m < 2, that is e - 7 while m <= 255 / 128 and e - 6 above
  const uint32_t bits = __float_as_uint(ext), e = bits >> 23 & 0xFFu;
  if (e == 255u) return 253u;
  return min(max(e + ((bits & 0x7FFFFFu) > 0x7F0000u ? 1u : 0u), 8u) - 7u, 253u);
}

__device__ __forceinline__ void write_tri(const GeomDesc* __restrict__ geoms, const float4* __restrict__ pbox,
                                          uint32_t prim, TriRecord* dst, bool robust) {
  const uint32_t gs = __float_as_uint(pbox[2 * (size_t)prim].w);
  const uint32_t j = __float_as_uint(pbox[2 * (size_t)prim + 1].w);
  const GeomDesc g = geoms[gs];
  if (g.kind == 1) {  // instance leaf
    const InstBox bx = reinterpret_cast<const InstBox*>(g.verts)[j];
    dst->a = make_float4(0.f, 0.f, 0.f, __uint_as_float(bx.inst));
    dst->b = make_float4(0.f, 0.f, 0.f, __uint_as_float(bx.geomID));
    dst->c = make_float4(0.f, 0.f, 0.f, __uint_as_float(kInstanceLeaf));
    return;
  }
  const uint3 t = load_tri(g, j);
  const float3 p0 = load_vtx(g, t.x), p1 = load_vtx(g, t.y), p2 = load_vtx(g, t.z);
  // Triangle4: e1 = v0 - v1, e2 = v2 - v0 (triangle.h:40-41); Triangle4v of
  // robust scenes keeps v1 and v2 themselves (trianglev.h:93-115)
  const float3 e1 = robust ? p1 : make_float3(__fsub_rn(p0.x, p1.x), __fsub_rn(p0.y, p1.y), __fsub_rn(p0.z, p1.z));
  const float3 e2 = robust ? p2 : make_float3(__fsub_rn(p2.x, p0.x), __fsub_rn(p2.y, p0.y), __fsub_rn(p2.z, p0.z));
  dst->a = make_float4(p0.x, p0.y, p0.z, __uint_as_float(j));
  dst->b = make_float4(e1.x, e1.y, e1.z, __uint_as_float(g.geomID));
  dst->c = make_float4(e2.x, e2.y, e2.z, 0.f);
}

// Shared memory of the lane groups that emit wide nodes: the node's words.
template <int GROUPS>
struct EmitSmem {
  alignas(16) uint32_t node[GROUPS][sizeof(WideNode) / 4];
};

// The wide node of item k, built by the 8 lanes of a lane group (lane & 7 is the
// child index; all 32 lanes call it, `have` is the group's; g: the group's index in
// the CTA; k_next: the item the group takes next, or 0xFFFFFFFF: its children's boxes
// are prefetched, 13 of 578 us at 4M triangles).  Children are placed in slots greedily, the cheapest (child, free slot)
// pair first with ties to the lower child and then the lower slot, the cost being
// the child's offset from the node centre along the slot's octant direction (slot s
// prefers children far along the direction with sign bits s), so that visiting
// slots in ascending order of (slot ^ ray octant) is roughly near-to-far.  One
// order of all pairs ranks the slots for every child and the children for every
// slot, so the greedy choice is the stable assignment, which rounds of offers
// find: every child stands at its next slot, and of the children at one slot all
// but the first move on to theirs.  Opposite slots have opposite costs, so 16
// comparisons rank a child's slots and 56 tell which children come before it at
// each; a round is then four votes.  (With every child scanning the free slots and
// 64-bit shared atomics for the offers, a level waited up to 4,300 cycles for the
// slots of its slowest node; so, 700.)  Planes are quantised outward, internal children are numbered and
// leaf triangles laid out in slot order.
template <int GROUPS>
__device__ __forceinline__ void collapse_emit_group(
    const BinTree& t, const uint32_t* __restrict__ kids_in, uint32_t k, bool have, uint32_t g, EmitSmem<GROUPS>& sm,
    const uint32_t* __restrict__ off_int, const uint32_t* __restrict__ off_tri, uint2 off, uint32_t k_next, uint32_t level_base,
    uint32_t next_base, uint32_t tri_next, WideNode* __restrict__ nodes, uint32_t* __restrict__ leaf_root,
    uint32_t* __restrict__ next_items, uint32_t node_cap, uint32_t tri_cap, uint32_t* err, double& sah_out,
    double& sahx_out, uint32_t& nleaf_out) {
  const uint32_t i = threadIdx.x & 7u;
  const uint32_t kid = have ? kids_in[8 * (size_t)k + i] : 0xFFFFFFFFu;
  const bool valid = kid != 0xFFFFFFFFu;
  float3 lo = make_float3(0.f, 0.f, 0.f), hi = lo;
  uint32_t prim = 0;  // a leaf node's primitive
  if (valid) {
    const float4 a = t.box[2 * (size_t)kid], b = t.box[2 * (size_t)kid + 1];
    lo = make_float3(a.x, a.y, a.z);
    hi = make_float3(b.x, b.y, b.z);
    prim = __float_as_uint(b.w);
  }
  uint32_t cnt = valid ? bt_cnt(t, kid) : 0u;
  const uint32_t oi = have ? off.x + off_int[k] : 0u, ot = have ? off.y + off_tri[k] : 0u;
  const uint32_t kid_next = k_next != 0xFFFFFFFFu ? kids_in[8 * (size_t)k_next + i] : 0xFFFFFFFFu;
  // union box and quantisation frame
  float3 ulo = valid ? lo : make_float3(INFINITY, INFINITY, INFINITY);
  float3 uhi = valid ? hi : make_float3(-INFINITY, -INFINITY, -INFINITY);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    ulo.x = fminf(ulo.x, __shfl_xor_sync(0xFFFFFFFFu, ulo.x, o));
    ulo.y = fminf(ulo.y, __shfl_xor_sync(0xFFFFFFFFu, ulo.y, o));
    ulo.z = fminf(ulo.z, __shfl_xor_sync(0xFFFFFFFFu, ulo.z, o));
    uhi.x = fmaxf(uhi.x, __shfl_xor_sync(0xFFFFFFFFu, uhi.x, o));
    uhi.y = fmaxf(uhi.y, __shfl_xor_sync(0xFFFFFFFFu, uhi.y, o));
    uhi.z = fmaxf(uhi.z, __shfl_xor_sync(0xFFFFFFFFu, uhi.z, o));
  }
  // one axis' exponent per lane
  const uint32_t Ea = exp_for(i == 0u ? __fsub_ru(uhi.x, ulo.x) : i == 1u ? __fsub_ru(uhi.y, ulo.y) : __fsub_ru(uhi.z, ulo.z));
  const uint32_t Ex = __shfl_sync(0xFFFFFFFFu, Ea, 0, 8), Ey = __shfl_sync(0xFFFFFFFFu, Ea, 1, 8),
                 Ez = __shfl_sync(0xFFFFFFFFu, Ea, 2, 8);
  const float sx = __uint_as_float(Ex << 23), sy = __uint_as_float(Ey << 23), sz = __uint_as_float(Ez << 23);
  const float ix = __uint_as_float((254u - Ex) << 23), iy = __uint_as_float((254u - Ey) << 23),
              iz = __uint_as_float((254u - Ez) << 23);
  // slot costs of this lane's child
  const float3 pc = make_float3((ulo.x + uhi.x) * 0.5f, (ulo.y + uhi.y) * 0.5f, (ulo.z + uhi.z) * 0.5f);
  const float dx = (lo.x + hi.x) * 0.5f - pc.x, dy = (lo.y + hi.y) * 0.5f - pc.y, dz = (lo.z + hi.z) * 0.5f - pc.z;
  // cost of slot q < 4 as an integer of the same order (zeros of both signs equal);
  // slot 7 - q costs -c[q]
  auto ordered = [](float x) {
    const int b = __float_as_int(x);
    return b < 0 ? -(b & 0x7FFFFFFF) : b;
  };
  const int c[4] = {ordered((dx + dy) + dz), ordered((-dx + dy) + dz), ordered((dx - dy) + dz), ordered((-dx - dy) + dz)};
  // ranks of slots 0..3 (4 bits each): slots before them, equal costs in slot order
  uint32_t ranks = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
#pragma unroll
    for (int w = q; w < 4; w++) {
      if (w > q) ranks += c[w] < c[q] ? 1u << (4 * q) : 1u << (4 * w);
      // slot 7 - w before slot q, and 7 - q before w
      if (-c[w] < c[q]) ranks += w > q ? (1u << (4 * q)) + (1u << (4 * w)) : 1u << (4 * q);
    }
  }
  uint32_t order = 0;  // the slots, cheapest first, 4 bits each
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t r4 = (ranks >> (4 * q) & 7u) * 4u;
    order |= ((uint32_t)q << r4) | ((7u - q) << (28u - r4));
  }
  // the children that come before this one at slot q (byte q of w03) and at slot
  // 7 - q (byte q of w74)
  uint32_t w03 = 0, w74 = 0;
#pragma unroll
  for (uint32_t d = 1; d < 8; d++) {
    const uint32_t bit = 1u << (i ^ d);
    const int lower = i >> (d < 2u ? 0 : d < 4u ? 1 : 2) & 1u;  // child i ^ d is the lower one: it wins a tie
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int o = __shfl_xor_sync(0xFFFFFFFFu, c[q], d);
      if (o < c[q] + lower) w03 |= bit << (8 * q);
      if (o > c[q] - lower) w74 |= bit << (8 * q);
    }
  }
  uint32_t* words = sm.node[g];
  // empty slots: meta 0, lower planes 255, upper planes 0
  if (i < 7u) *reinterpret_cast<uint2*>(words + 6 + 2 * i) = i >= 1u && i <= 3u ? make_uint2(~0u, ~0u) : make_uint2(0u, 0u);
  __syncwarp();
  const uint32_t gshift = threadIdx.x & 24u, kids8 = __ballot_sync(0xFFFFFFFFu, valid) >> gshift & 0xFFu;
  for (bool lost = true; __any_sync(0xFFFFFFFFu, lost);) {
#pragma unroll
    for (int r = 0; r < 2; r++) {  // two rounds per vote on going on: one too many changes nothing
      const uint32_t q = order & 7u;
      const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, q & 1u), b1 = __ballot_sync(0xFFFFFFFFu, q & 2u),
                     b2 = __ballot_sync(0xFFFFFFFFu, q & 4u);
      const uint32_t same = ((q & 1u ? b0 : ~b0) & (q & 2u ? b1 : ~b1) & (q & 4u ? b2 : ~b2)) >> gshift & kids8;
      lost = (same & __funnelshift_r(q < 4u ? w03 : w74, 0u, 8u * (q < 4u ? q : 7u - q))) != 0u && valid;
      if (lost) order >>= 4;
    }
  }
  const uint32_t slot = valid ? order & 7u : 8u;
  if (kid_next != 0xFFFFFFFFu) prefetch_l2(t.box + 2 * (size_t)kid_next);
  // this child's planes, its part of the SAH, its place among the slots
  const bool inner = cnt > t.leaf_max;
  uint32_t places = valid ? (inner ? 8u : cnt) << (4u * slot) : 0u;  // 4 bits per slot: triangles, bit 3 an internal child
  uint32_t int_slots = inner ? 1u << slot : 0u;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    places |= __shfl_xor_sync(0xFFFFFFFFu, places, o);
    int_slots |= __shfl_xor_sync(0xFFFFFFFFu, int_slots, o);
  }
  const uint32_t child_base = next_base + oi, tri_base = tri_next + ot;
  float A = 0.f, Ax = 0.f;
  if (valid) {
    const uint32_t qlx = min(__float2uint_rd(__fsub_rd(lo.x, ulo.x) * ix), 255u);
    const uint32_t qly = min(__float2uint_rd(__fsub_rd(lo.y, ulo.y) * iy), 255u);
    const uint32_t qlz = min(__float2uint_rd(__fsub_rd(lo.z, ulo.z) * iz), 255u);
    const uint32_t qhx = min(__float2uint_ru(__fsub_ru(hi.x, ulo.x) * ix), 255u);
    const uint32_t qhy = min(__float2uint_ru(__fsub_ru(hi.y, ulo.y) * iy), 255u);
    const uint32_t qhz = min(__float2uint_ru(__fsub_ru(hi.z, ulo.z) * iz), 255u);
    const float flx = byte_f(qlx), fly = byte_f(qly), flz = byte_f(qlz), fhx = byte_f(qhx), fhy = byte_f(qhy),
                fhz = byte_f(qhz);
    // decoded (outward-rounded) box, as traversal sees it
    const float3 dlo = make_float3(__fmaf_rd(flx, sx, ulo.x), __fmaf_rd(fly, sy, ulo.y), __fmaf_rd(flz, sz, ulo.z));
    const float3 dhi = make_float3(__fmaf_ru(fhx, sx, ulo.x), __fmaf_ru(fhy, sy, ulo.y), __fmaf_ru(fhz, sz, ulo.z));
    A = fmaxf(0.f, half_area(dlo, dhi));
    Ax = fmaxf(0.f, half_area(lo, hi));
    // an inner child's place among the next level's items; a leaf's triangles behind
    // those of the leaves in lower slots (the sum of their 3-bit counts)
    const uint32_t below = places & ((1u << (4u * slot)) - 1u), c = below & 0x77777777u;
    const uint32_t tri_off = (((c & 0x0F0F0F0Fu) + (c >> 4 & 0x0F0F0F0Fu)) * 0x01010101u) >> 24;
    const uint32_t rank = __popc(below & 0x88888888u);
    const uint32_t meta = inner ? 0x80u | slot : 0x80u | ((cnt - 1u) << 5) | tri_off;
    // a leaf's triangle records are written after the last level by k_write_leaves,
    // one thread per leaf: here only its binary subtree is recorded at the slot of
    // its first triangle
    const uint32_t at = inner ? oi + rank : tri_base + tri_off;
    const bool fits = inner ? at < node_cap && child_base + rank < node_cap : at + cnt <= tri_cap;
    if (fits) (inner ? next_items : leaf_root)[at] = inner || cnt > 1u ? kid : prim | kLeafPrim;
    else atomicOr(err, kErrBuild);
    uint8_t* bytes = reinterpret_cast<uint8_t*>(words);
    bytes[24 + slot] = (uint8_t)meta;
    bytes[32 + slot] = (uint8_t)qlx;
    bytes[40 + slot] = (uint8_t)qly;
    bytes[48 + slot] = (uint8_t)qlz;
    bytes[56 + slot] = (uint8_t)qhx;
    bytes[64 + slot] = (uint8_t)qhy;
    bytes[72 + slot] = (uint8_t)qhz;
  }
  if (i == 0u)
    *reinterpret_cast<uint4*>(words) = make_uint4(__float_as_uint(ulo.x), __float_as_uint(ulo.y), __float_as_uint(ulo.z),
                                                  Ex | (Ey << 8) | (Ez << 16) | ((int_slots & 0xFFu) << 24));
  else if (i == 1u)
    *reinterpret_cast<uint2*>(words + 4) = make_uint2(child_base, tri_base);
  else if (i == 2u)
    *reinterpret_cast<uint4*>(words + 20) = make_uint4(__float_as_uint(sx * 32768.0f), __float_as_uint(sy * 32768.0f),
                                                       __float_as_uint(sz * 32768.0f), 0u);
  __syncwarp();
  if (have) {
    if (level_base + k >= node_cap) {
      if (i == 0u) atomicOr(err, kErrBuild);
    } else if (i < 6u) {
      reinterpret_cast<uint4*>(nodes + level_base + k)[i] = reinterpret_cast<const uint4*>(words)[i];
    }
  }
  if (valid) {  // the SAH's terms: area for an inner node, area x Triangle4 blocks for a leaf
    sah_out += (double)A;
    sahx_out += (double)Ax;
    if (!inner) nleaf_out++;
  }
  __syncwarp();  // the words are built again for the next node
}

constexpr int COLLAPSE_THREADS = 128;
// One wide node per 8-lane group; the SAH sums and the leaf count are reduced
// per CTA first (one atomic per CTA instead of one per node).
__global__ void __launch_bounds__(COLLAPSE_THREADS) k_collapse_emit(
    BinTree t, const uint32_t* __restrict__ kids_in, const uint32_t* __restrict__ cstate,
    const uint32_t* __restrict__ off_int, const uint32_t* __restrict__ off_tri, WideNode* __restrict__ nodes,
    uint32_t* __restrict__ leaf_root, const ColItems ci, double* sah_acc, uint32_t* leaf_count,
    uint32_t node_cap, uint32_t tri_cap, uint32_t* err) {
  const uint32_t nitems = cstate[kColN], level_base = cstate[kColBase], tri_next = cstate[kColTri];
  uint32_t* __restrict__ next_items = ci.items[(cstate[kColDepth] & 1u) ^ 1u];
  const uint32_t next_base = level_base + nitems;
  double sah = 0.0, sahx = 0.0;
  uint32_t nleaf = 0;
  __shared__ EmitSmem<COLLAPSE_THREADS / 8> sm;
  for (uint32_t k0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) >> 3; k0 < nitems; k0 += (gridDim.x * blockDim.x) >> 3) {
    const uint32_t k = k0 + ((threadIdx.x & 31u) >> 3);
    collapse_emit_group(t, kids_in, k, k < nitems, threadIdx.x >> 3, sm, off_int, off_tri, make_uint2(0u, 0u), 0xFFFFFFFFu, level_base, next_base, tri_next,
                        nodes, leaf_root, next_items, node_cap, tri_cap, err, sah, sahx, nleaf);
  }
  nleaf = __reduce_add_sync(0xFFFFFFFFu, nleaf);
  if ((threadIdx.x & 31) == 0 && nleaf) atomicAdd(leaf_count, nleaf);
  block_add2(sah, sahx, sah_acc);
}

// ---- all collapse levels in one cooperative launch (captured builds)
//
// A grid barrier between the phases of a level replaces the kernel boundaries
// of the level-by-level form (count, scan, emit, advance: four launches per
// level).  Every CTA keeps the level state in registers and advances it alike;
// CTA 0 writes it back to cstate at the end.


// Threads of a CTA of k_collapse_all, one CTA per SM: 512 threads have registers for
// two node's reads in flight and wait less at each other (a level of few nodes takes
// 13,000 cycles against 16,000), 1024 threads have the warps that a wide level needs.
// The levels of a tree of 8k / 300k / 1M / 4M triangles take 44 / 137 / 269 / 744 us
// with 512 threads and 53 / 144 / 244 / 573 with 1024, so the line lies between 300k
// and 1M.  (Four CTAs of 256 threads per SM waited longer at the barriers, where 608
// arrive and read each other's sums instead of 152.)
constexpr int COLLAPSE_NARROW_THREADS = 512, COLLAPSE_WIDE_THREADS = 1024;
constexpr uint32_t COLLAPSE_WIDE_TRIS = 1u << 19;

// Every level of the collapse, from the roots in cstate: each CTA takes a
// contiguous chunk of the level's items, (1) gathers their children and counts
// internal children and leaf triangles, (2) scans the counts within the chunk and
// sums them with the other CTAs (grid_sums), [barrier in there], (3) writes its wide
// nodes and the next level's items, [barrier].  cta_sums holds gridDim.x pairs; *bar
// is zero on entry.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_collapse_all(
    BinTree t, const ColItems ci, uint32_t* __restrict__ cstate, uint32_t* __restrict__ kids,
    uint32_t* __restrict__ nint, uint32_t* __restrict__ ntri, uint2* __restrict__ cta_sums,
    WideNode* __restrict__ nodes, uint32_t* __restrict__ leaf_root, double* sah_acc, uint32_t* leaf_count,
    uint32_t node_cap, uint32_t tri_cap, uint32_t max_levels, GridBarrier* bar, unsigned int* err) {
  uint32_t nitems = __ldcg(cstate + kColN), base = __ldcg(cstate + kColBase), tri_next = __ldcg(cstate + kColTri),
           depth = __ldcg(cstate + kColDepth);
  bool failed = __ldcg(cstate + kColErr) != 0u;
  __shared__ EmitSmem<THREADS / 8> sm;
  double sah = 0.0, sahx = 0.0;
  uint32_t nleaf = 0;
  while (nitems > 0 && !failed) {
    const uint32_t* __restrict__ items = ci.items[depth & 1u];
    uint32_t* __restrict__ next_items = ci.items[(depth & 1u) ^ 1u];
    const uint32_t per = (nitems + gridDim.x - 1) / gridDim.x;
    const uint32_t first = min(blockIdx.x * per, nitems), last = min(first + per, nitems);
    // (1) children and counts
    for (uint32_t k0 = first + ((threadIdx.x & ~31u) >> 3); k0 < last; k0 += blockDim.x >> 3) {
      const uint32_t k = k0 + ((threadIdx.x & 31u) >> 3);
      uint32_t ni, nt;
      collapse_count_group(t, items, k, k < last, kids, &ni, &nt);
      if (k < last && (threadIdx.x & 7u) == 0u) {
        nint[k] = ni;
        ntri[k] = nt;
      }
    }
    __syncthreads();
    // (2) offsets within the chunk; the chunk's place and the level's totals
    uint32_t ci_sum = 0, ct_sum = 0;
    if (last - first <= 32u) {  // one warp
      if (threadIdx.x < 32u) {
        const uint32_t k = first + threadIdx.x;
        const uint32_t a = k < last ? nint[k] : 0u, b = k < last ? ntri[k] : 0u;
        uint32_t xa = a, xb = b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t ya = __shfl_up_sync(0xFFFFFFFFu, xa, o), yb = __shfl_up_sync(0xFFFFFFFFu, xb, o);
          if (threadIdx.x >= o) xa += ya, xb += yb;
        }
        if (k < last) {
          nint[k] = xa - a;
          ntri[k] = xb - b;
        }
        ci_sum = __shfl_sync(0xFFFFFFFFu, xa, 31);
        ct_sum = __shfl_sync(0xFFFFFFFFu, xb, 31);
      }
    } else for (uint32_t k0 = first; k0 < last; k0 += blockDim.x) {
      const uint32_t k = k0 + threadIdx.x;
      uint32_t ta, tb;
      const uint2 e = block_excl_scan2<THREADS>(k < last ? nint[k] : 0u, k < last ? ntri[k] : 0u, &ta, &tb);
      if (k < last) {
        nint[k] = ci_sum + e.x;
        ntri[k] = ct_sum + e.y;
      }
      ci_sum += ta;
      ct_sum += tb;
    }
    uint4 sums;
    if (!grid_sums<THREADS>(cta_sums, ci_sum, ct_sum, sums, bar, err)) break;
    // (3) the wide nodes of this CTA's items, one per 8-lane group
    for (uint32_t k0 = first + ((threadIdx.x & ~31u) >> 3); k0 < last; k0 += blockDim.x >> 3) {
      const uint32_t k = k0 + ((threadIdx.x & 31u) >> 3);
      const uint32_t k_next = k + (blockDim.x >> 3);
      collapse_emit_group(t, kids, k, k < last, threadIdx.x >> 3, sm, nint, ntri, make_uint2(sums.x, sums.y),
                          k_next < last ? k_next : 0xFFFFFFFFu, base, base + nitems, tri_next, nodes, leaf_root,
                          next_items, node_cap, tri_cap, err, sah, sahx, nleaf);
    }
    // (4) the next level, alike in every CTA
    if (blockIdx.x == 0 && threadIdx.x == 0 && depth < (uint32_t)kColMaxLevels) cstate[kColLevels + depth] = base;
    base += nitems;
    tri_next += sums.w;
    depth++;
    uint32_t next = sums.z;
    if ((next > 0 && depth >= max_levels) || base + next > node_cap) {
      failed = true;
      next = 0;
      if (blockIdx.x == 0 && threadIdx.x == 0) cstate[kColErr] = 1u;
    }
    nitems = next;
    if (!grid_sync(bar, err)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cstate[kColN] = 0;
    cstate[kColBase] = base;
    cstate[kColTri] = tri_next;
    cstate[kColDepth] = depth;
    if (depth <= (uint32_t)kColMaxLevels) cstate[kColLevels + depth] = base;  // end of the last level
    if (lb_load(err) != 0u) cstate[kColErr] = 1u;
  }
  nleaf = __reduce_add_sync(0xFFFFFFFFu, nleaf);
  if ((threadIdx.x & 31) == 0 && nleaf) atomicAdd(leaf_count, nleaf);
  block_add2(sah, sahx, sah_acc);
}

// Writes the triangle records of every leaf: slot t holds the binary subtree of
// the leaf whose first triangle goes to t, or for a one-triangle leaf its
// primitive with kLeafPrim set (kInvalidID elsewhere); a subtree's primitives
// (at most 4) are written in depth-first order, left first.
__global__ void __launch_bounds__(256) k_write_leaves(BinTree t, const GeomDesc* __restrict__ geoms,
                                                      const float4* __restrict__ pbox,
                                                      const uint32_t* __restrict__ leaf_root, uint32_t ntris,
                                                      TriRecord* __restrict__ tris, uint32_t* err,
                                                      const TriRecord* __restrict__ prec) {
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
  if (first >= ntris) return;
  const uint32_t c = leaf_root[first];
  if (c == kInvalidID) return;
  if (c & kLeafPrim) {  // one triangle: its primitive, no subtree to walk
    const uint32_t prim = c & ~kLeafPrim;
    if (prec) tris[first] = prec[prim];
    else write_tri(geoms, pbox, prim, &tris[first], t.robust != 0);
    return;
  }
  uint32_t st[8];
  int sp = 0;
  st[sp++] = c;
  uint32_t w = 0;
  while (sp > 0) {
    const uint32_t x = st[--sp];
    if (bt_leaf(t, x)) {
      if (first + w >= ntris || w >= (uint32_t)kLeafMaxLimit) {
        atomicOr(err, kErrBuild);
        return;
      }
      if (prec) tris[first + w] = prec[bt_right(t, x)];
      else write_tri(geoms, pbox, bt_right(t, x), &tris[first + w], t.robust != 0);
      w++;
    } else {
      if (sp + 2 > 8) {
        atomicOr(err, kErrBuild);
        return;
      }
      st[sp++] = bt_right(t, x);
      st[sp++] = bt_left(t, x);
    }
  }
}

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------

template <typename T>
static cudaError_t dalloc(T** p, size_t count, cudaStream_t st) {
  return cudaMallocAsync((void**)p, std::max<size_t>(count, 1) * sizeof(T), st);
}

static inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

static int num_sms_build() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n < 1) n = 1;
  }
  return n;
}

// Blocks of 256 threads for a grid-stride kernel over n items: up to 8 per SM.
static unsigned grid_stride_blocks(uint64_t n) {
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)num_sms_build() * 8));
}

// Words of look-back state that scan_excl needs for n elements (ticket, done
// counter, one status word per tile); zero when allocated, and every scan leaves
// it zero again.
static inline uint32_t scan_scratch(uint32_t n) { return cdiv(n, SCAN_TILE) + 2; }

// Exclusive scans of a[0, n) and b[0, n) in place, by one launch (totals to
// *ta / *tb); sums holds 2 * scan_scratch(n) zeroed words.  With d_n the count
// is *d_n (at most n), read on the device, so the scans can be enqueued before
// the count is known.  One CTA per array for short arrays, else the look-back
// scan.
static void scan_excl2(uint32_t* a, uint32_t* b, uint32_t n, uint32_t* ta, uint32_t* tb, uint32_t* sums,
                       cudaStream_t st, unsigned int* err, const uint32_t* d_n = nullptr) {
  const ScanPair sp{{a, b}, {ta, tb}};
  if (n <= 2 * SCAN_TILE) {
    k_scan_excl<<<dim3(1, 2), SCAN_THREADS, 0, st>>>(sp, n, d_n, 1);
  } else {
    k_scan_lb<<<dim3(cdiv(n, SCAN_TILE), 2), SCAN_THREADS, 0, st>>>(sp, n, d_n, 1, sums, scan_scratch(n), err);
  }
  note_launches(1);
}

// Scratch words of onesweep_sort for exactly n keys and `passes` digit passes.
static inline size_t onesweep_scratch_words(uint32_t n, int passes) {
  return kOsStatus + (size_t)passes * cdiv(n, os_tile(n)) * 256u;
}

// Stable LSD sort of (ka, va) by the digits set in digit_mask (bit d: key bits
// 8d..8d+7), least significant first, ping-ponging with (kb, vb): on return
// (ka, va) name the buffers that hold the result.  scratch: at least
// onesweep_scratch_words(n, passes) words, zeroed here.  A look-back that gives up
// sets kErrBuild in *err (or in the scratch's error word when err is null).
template <typename K>
static cudaError_t onesweep_sort(K*& ka, uint32_t*& va, K*& kb, uint32_t*& vb, uint32_t n, uint32_t digit_mask,
                                 uint32_t* scratch, unsigned int* err, cudaStream_t st) {
  digit_mask &= (1u << sizeof(K)) - 1u;
  const int passes = __builtin_popcount(digit_mask);
  if (n == 0 || passes == 0) return cudaSuccess;
  if (n >= kLbValue) return cudaErrorInvalidValue;  // look-back counts are 30-bit
  if (n <= kSortOneMax) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GB_CHECK(cudaStreamIsCapturing(st, &cap));
    if (cap == cudaStreamCaptureStatusNone)
      GB_CHECK(cudaFuncSetAttribute(k_sort_one<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_one_smem<K>()));
    if (!err) GB_CHECK(cudaMemsetAsync(scratch + kOsErr, 0, sizeof(uint32_t), st));
    k_sort_one<K><<<1, kSortOneThreads, sort_one_smem<K>(), st>>>(ka, va, n, digit_mask);
    note_launches(1);
    return cudaGetLastError();
  }
  const uint32_t ntiles = cdiv(n, os_tile(n));
  GB_CHECK(cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * onesweep_scratch_words(n, passes), st));
  const uint32_t hgrid = std::min<uint32_t>(ntiles, 4u * (uint32_t)num_sms_build());
  // up to 48 KB of staged keys and values beyond the static shared memory (per
  // device; a captured build sets it in graph_build_prepare)
  const bool few = n <= RS_FEW;
  const auto scatter = few ? k_os_scatter<K, RS_FEW_ITEMS> : k_os_scatter<K, RS_ITEMS>;
  const size_t smem = few ? os_scatter_smem<K, RS_FEW_ITEMS>() : os_scatter_smem<K, RS_ITEMS>();
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  GB_CHECK(cudaStreamIsCapturing(st, &cap));
  if (cap == cudaStreamCaptureStatusNone)
    GB_CHECK(cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_os_hist<K><<<hgrid, 256, 0, st>>>(ka, n, digit_mask & ((1u << sizeof(K)) - 1u), scratch);
  uint32_t slot = 0;
  for (int d = 0; d < (int)sizeof(K); d++) {
    if (!(digit_mask >> d & 1u)) continue;
    scatter<<<ntiles, RS_THREADS, smem, st>>>(ka, va, kb, vb, n, 8 * d, scratch, slot,
                                              scratch + kOsStatus + (size_t)slot * ntiles * 256u,
                                              err ? err : scratch + kOsErr);
    std::swap(ka, kb);
    std::swap(va, vb);
    slot++;
  }
  note_launches(1 + passes);
  return cudaGetLastError();
}

// The one-CTA finish of the clustering, by search radius.
static cudaError_t ploc_finish_prepare() {
  GB_CHECK(cudaFuncSetAttribute(k_ploc_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlocSmallSmem));
  return cudaFuncSetAttribute(k_ploc_finish1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlocFinishSmem);
}
static cudaError_t ploc_finish(const PlocBufs& pb, uint32_t* ploc_state, float4* bnbox, uint32_t* bncnt,
                               uint32_t* root_out, uint32_t* iters_out, uint32_t node_cap, uint32_t* err,
                               uint32_t nseg, int radius, float4* dp_cost, uint4* dp_link, uint32_t leaf_max,
                               cudaStream_t st) {
  if (radius == 1)
    k_ploc_finish1<<<1, PLOC_SMALL_THREADS, kPlocFinishSmem, st>>>(pb, ploc_state, bnbox, bncnt, root_out, iters_out,
                                                                   node_cap, err, nseg, dp_cost, dp_link, leaf_max);
  else
    k_ploc_small<<<1, PLOC_SMALL_THREADS, kPlocSmallSmem, st>>>(pb.clo[0], pb.chi[0], pb.cidx[0], pb.clo[1], pb.chi[1],
                                                                pb.cidx[1], ploc_state, bnbox, bncnt, root_out,
                                                                iters_out, node_cap, err, nseg, radius, dp_cost,
                                                                dp_link, leaf_max);
  note_launches(1);
  return cudaGetLastError();
}

// Stream-ordered scratch of one build: device allocations, pinned host
// buffers and events are released when the arena goes out of scope, on every
// return path (free() releases a buffer early to lower the peak).
struct BuildArena {
  cudaStream_t st;
  std::vector<void*> dev, pinned;
  std::vector<cudaEvent_t> events;
  explicit BuildArena(cudaStream_t s) : st(s) {}
  BuildArena(const BuildArena&) = delete;
  BuildArena& operator=(const BuildArena&) = delete;
  template <typename T>
  cudaError_t alloc(T** p, size_t count) {
    const cudaError_t e = cudaMallocAsync((void**)p, std::max<size_t>(count, 1) * sizeof(T), st);
    if (e == cudaSuccess) dev.push_back(*p);
    return e;
  }
  template <typename T>
  cudaError_t host(T** p, size_t count) {
    const cudaError_t e = cudaMallocHost((void**)p, std::max<size_t>(count, 1) * sizeof(T));
    if (e == cudaSuccess) pinned.push_back(*p);
    return e;
  }
  cudaError_t event(cudaEvent_t* e) {
    const cudaError_t r = cudaEventCreate(e);
    if (r == cudaSuccess) events.push_back(*e);
    return r;
  }
  void free(void* p) {
    for (size_t i = 0; i < dev.size(); i++)
      if (dev[i] == p) {
        cudaFreeAsync(p, st);
        dev.erase(dev.begin() + (long)i);
        return;
      }
  }
  ~BuildArena() {
    for (void* p : dev) cudaFreeAsync(p, st);
    if (!pinned.empty()) cudaStreamSynchronize(st);  // copies into them may still be in flight
    for (void* p : pinned) cudaFreeHost(p);
    for (cudaEvent_t e : events) cudaEventDestroy(e);
  }
};

cudaError_t build_bvh(const GeomDesc* h_geoms, int ngeoms, cudaStream_t st, const BuildOptions& opt, DeviceBVH* out,
                      BuildStats* stats) {
  *out = DeviceBVH();
  *stats = BuildStats();
  for (int d = 0; d < 3; d++) { out->lo[d] = INFINITY; out->hi[d] = -INFINITY; }
  uint64_t total64 = 0;
  for (int g = 0; g < ngeoms; g++) total64 += h_geoms[g].ntris;
  if (total64 == 0) return cudaSuccess;
  if (total64 >= 0x7FFFFFFFull) return cudaErrorInvalidValue;
  const uint32_t total = (uint32_t)total64;

  BuildArena arena(st);  // scratch and events of this build, released on every return
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  GB_CHECK(arena.event(&ev0));
  GB_CHECK(arena.event(&ev1));
  GB_CHECK(cudaEventRecord(ev0, st));

  GeomDesc* d_geoms = nullptr;
  GB_CHECK(arena.alloc(&d_geoms, ngeoms));
  GB_CHECK(cudaMemcpyAsync(d_geoms, h_geoms, sizeof(GeomDesc) * ngeoms, cudaMemcpyHostToDevice, st));

  float4* pbox = nullptr;
  BoundsAcc* acc = nullptr;
  GB_CHECK(arena.alloc(&pbox, 2 * (size_t)total));
  GB_CHECK(arena.alloc(&acc, 1));
  BoundsAcc h_acc;
  for (int d = 0; d < 3; d++) { h_acc.glo[d] = h_acc.clo[d] = 0xFFFFFFFFu; h_acc.ghi[d] = h_acc.chi[d] = 0u; }
  h_acc.nvalid = 0;
  h_acc.pad = 0;
  h_acc.kand = ~0ull;
  h_acc.kor = 0ull;
  GB_CHECK(cudaMemcpyAsync(acc, &h_acc, sizeof(BoundsAcc), cudaMemcpyHostToDevice, st));
  // leaf records in primitive order (read back by k_write_leaves)
  TriRecord* prec = nullptr;
  GB_CHECK(arena.alloc(&prec, total));
  k_primrefs<<<grid_stride_blocks(total), 256, 0, st>>>(d_geoms, ngeoms, total, pbox, acc, prec,
                                                        opt.robust ? 1 : 0);
  note_launches(1);

  uint64_t *keys_a = nullptr, *keys_b = nullptr;
  uint32_t *vals_a = nullptr, *vals_b = nullptr;
  GB_CHECK(arena.alloc(&keys_a, total));
  GB_CHECK(arena.alloc(&keys_b, total));
  GB_CHECK(arena.alloc(&vals_a, total));
  GB_CHECK(arena.alloc(&vals_b, total));
  const bool segmented = opt.segmented != 0;
  const uint32_t nseg = segmented ? (uint32_t)ngeoms : 1u;
  if (segmented && (uint32_t)ngeoms > kMaxSegments) return cudaErrorInvalidValue;
  const bool key32 = opt.morton_bits == 30 && !segmented;  // 30-bit keys sorted as 32-bit words
  k_morton<<<grid_stride_blocks(total), 256, 0, st>>>(pbox, total, acc, keys_a, vals_a, opt.morton_cube,
                                                      segmented ? nseg : 0u, opt.morton_bits == 30 ? 1 : 0,
                                                      key32 ? 1 : 0);
  note_launches(1);
  GB_CHECK(cudaGetLastError());
  GB_CHECK(cudaMemcpyAsync(&h_acc, acc, sizeof(BoundsAcc), cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaStreamSynchronize(st));
  const uint32_t N = h_acc.nvalid;
  for (int d = 0; d < 3; d++) { out->lo[d] = ord2f(h_acc.glo[d]); out->hi[d] = ord2f(h_acc.ghi[d]); }
  if (N == 0) {
    for (int d = 0; d < 3; d++) { out->lo[d] = INFINITY; out->hi[d] = -INFINITY; }
    arena.free(d_geoms); arena.free(pbox); arena.free(acc); arena.free(prec);
    arena.free(keys_a); arena.free(keys_b); arena.free(vals_a); arena.free(vals_b);
    return cudaStreamSynchronize(st);
  }

  // ---- radix sort (all `total` keys; invalid ones carry a key above every valid
  // one and sort last), the digits that are constant over all keys skipped
  {
    uint32_t digit_mask = 0;
    for (int d = 0; d < 8; d++)
      if (((h_acc.kand >> (8 * d)) & 0xFF) != ((h_acc.kor >> (8 * d)) & 0xFF)) digit_mask |= 1u << d;
    uint32_t* hist = nullptr;
    GB_CHECK(arena.alloc(&hist, onesweep_scratch_words(total, __builtin_popcount(digit_mask))));
    if (key32) {
      uint32_t *ka32 = reinterpret_cast<uint32_t*>(keys_a), *kb32 = reinterpret_cast<uint32_t*>(keys_b);
      GB_CHECK(onesweep_sort(ka32, vals_a, kb32, vals_b, total, digit_mask, hist, &acc->pad, st));
    } else {
      GB_CHECK(onesweep_sort(keys_a, vals_a, keys_b, vals_b, total, digit_mask, hist, &acc->pad, st));
    }
    arena.free(hist);
  }

  // ---- PLOC over the N valid primitives (sorted positions 0..N-1)
  float4* bnbox = nullptr;
  uint32_t* bncnt = nullptr;
  // leaf size: explicit, or by the scene -- flat scenes (centroid box's
  // smallest extent below half the largest: heightfields, terrain) and scenes
  // that will be refitted every frame take 2 triangles per leaf, the rest 1
  // (measured on a GB300: the 4M soup traces 5 % faster with 1; a 724^2
  // heightfield 8 % faster with 2, and its SAH is 1.12x the reference
  // builder's with 2, 1.31x with 1; the animated 4M soup, refitted per frame,
  // renders 4 % faster with 2, whose tree has 40 % fewer nodes to refit)
  int leaf_max = opt.leaf_max;
  if (leaf_max <= 0) {
    float emin = INFINITY, emax = 0.f;
    for (int d = 0; d < 3; d++) {
      const float e = ord2f(h_acc.chi[d]) - ord2f(h_acc.clo[d]);
      emin = std::min(emin, e);
      emax = std::max(emax, e);
    }
    leaf_max = (emin < 0.5f * emax || opt.refit_target) ? 2 : 1;
  }
  stats->leaf_max = (uint32_t)std::min(leaf_max, kLeafMaxLimit);
  const uint32_t nnodes_bin = 2 * N - 1;
  // SAH-optimal collapse: the cost table is filled as PLOC creates the nodes
  float4* dp_cost = nullptr;
  uint4* d_link = nullptr;
  if (opt.collapse == 1) {
    GB_CHECK(arena.alloc(&dp_cost, 2 * (size_t)nnodes_bin));
    GB_CHECK(arena.alloc(&d_link, nnodes_bin));
  }
  GB_CHECK(arena.alloc(&bnbox, 2 * (size_t)nnodes_bin));
  GB_CHECK(arena.alloc(&bncnt, nnodes_bin));
  float4 *clo_a, *chi_a, *clo_b, *chi_b;
  uint32_t *cidx_a, *cidx_b, *nn;
  GB_CHECK(arena.alloc(&clo_a, N));
  GB_CHECK(arena.alloc(&chi_a, N));
  GB_CHECK(arena.alloc(&clo_b, N));
  GB_CHECK(arena.alloc(&chi_b, N));
  GB_CHECK(arena.alloc(&cidx_a, N));
  GB_CHECK(arena.alloc(&cidx_b, N));
  GB_CHECK(arena.alloc(&nn, N));
  const uint32_t leaf_max_used = (uint32_t)std::min(std::max(leaf_max, 1), kLeafMaxLimit);
  k_ploc_init<<<cdiv(N, 256), 256, 0, st>>>(pbox, vals_a, N, &acc->nvalid, bnbox, cidx_a, clo_a,
                                            chi_a, segmented ? 1 : 0);
  note_launches(1);
  uint32_t *bsurv, *bmerge, *d_tot, *d_root, *d_iters;
  const uint32_t maxb = cdiv(N, PLOC_BLOCK);
  GB_CHECK(arena.alloc(&bsurv, maxb));
  GB_CHECK(arena.alloc(&bmerge, maxb));
  uint32_t* scan_sums = nullptr;  // look-back state of the PLOC and collapse scans (zero between scans)
  GB_CHECK(arena.alloc(&scan_sums, 2 * (size_t)scan_scratch(std::max(maxb, N))));
  GB_CHECK(cudaMemsetAsync(scan_sums, 0, sizeof(uint32_t) * 2 * scan_scratch(std::max(maxb, N)), st));
  GB_CHECK(arena.alloc(&d_tot, 4));
  GB_CHECK(arena.alloc(&d_root, nseg));
  GB_CHECK(cudaMemsetAsync(d_root, 0xFF, sizeof(uint32_t) * nseg, st));
  GB_CHECK(arena.alloc(&d_iters, 1));
  GB_CHECK(cudaMemsetAsync(d_iters, 0, sizeof(uint32_t), st));
  // PLOC rounds in batches of kPlocBatch between host reads of the state; the
  // count only shrinks, so the count read last bounds the grids of a batch,
  // and rounds after the last real one are no-ops (the done flag)
  constexpr int kPlocBatch = 4;
  uint32_t* ploc_state = nullptr;
  GB_CHECK(arena.alloc(&ploc_state, kPlocStateWords));
  uint32_t* h_tot = nullptr;
  GB_CHECK(arena.host(&h_tot, kPlocStateWords));
  k_ploc_state_init<<<1, 32, 0, st>>>(acc, N, ploc_state, nullptr);
  note_launches(1);
  const int radius = opt.ploc_radius == 1 || opt.ploc_radius == 2 || opt.ploc_radius == 4 || opt.ploc_radius == 8
                         ? opt.ploc_radius
                         : PLOC_R_MAX;
  const PlocBufs pb{{clo_a, clo_b}, {chi_a, chi_b}, {cidx_a, cidx_b}};
  uint32_t round = 0;
  auto enqueue_round = [&](uint32_t grid) {
    switch (radius) {
      case 1: k_ploc_nn<1><<<grid, PLOC_BLOCK, 0, st>>>(pb, ploc_state, nn); break;
      case 2: k_ploc_nn<2><<<grid, PLOC_BLOCK, 0, st>>>(pb, ploc_state, nn); break;
      case 4: k_ploc_nn<4><<<grid, PLOC_BLOCK, 0, st>>>(pb, ploc_state, nn); break;
      case 8: k_ploc_nn<8><<<grid, PLOC_BLOCK, 0, st>>>(pb, ploc_state, nn); break;
      default: k_ploc_nn<PLOC_R_MAX><<<grid, PLOC_BLOCK, 0, st>>>(pb, ploc_state, nn); break;
    }
    k_ploc_count<<<grid, PLOC_BLOCK, 0, st>>>(nn, ploc_state, bsurv, bmerge);
    note_launches(2);
    scan_excl2(bsurv, bmerge, maxb, d_tot + 0, d_tot + 1, scan_sums, st, &acc->pad, ploc_state + kPlocTiles);
    k_ploc_emit<<<grid, PLOC_BLOCK, 0, st>>>(pb, nn, ploc_state, bsurv, bmerge, bnbox, bncnt, nnodes_bin,
                                             &acc->pad, dp_cost, d_link, leaf_max_used);
    k_ploc_advance<<<1, 32, 0, st>>>(d_tot, ploc_state);
    note_launches(2);
    round++;
  };
  uint32_t n = N;
  while (n > PLOC_SMALL) {
    const uint32_t nb = cdiv(n, PLOC_BLOCK);
    for (int b = 0; b < kPlocBatch; b++) enqueue_round(nb);
    GB_CHECK(cudaGetLastError());
    GB_CHECK(cudaMemcpyAsync(h_tot, ploc_state, kPlocStateWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    GB_CHECK(cudaStreamSynchronize(st));
    n = h_tot[kPlocN];
    if (h_tot[kPlocDone]) break;
  }
  // a round without merges while more than PLOC_SMALL clusters remain cannot
  // happen without segments (the globally closest pair is mutual); with
  // segments it means every segment is down to one cluster (<= kMaxSegments)
  const uint32_t iters = round > 0 ? h_tot[kPlocRounds] : 0u;
  {
    GB_CHECK(ploc_finish_prepare());
    GB_CHECK(ploc_finish(pb, ploc_state, bnbox, bncnt, d_root, d_iters, nnodes_bin, &acc->pad, nseg, radius, dp_cost,
                         d_link, leaf_max_used, st));
  }
  uint32_t small_iters = 0, berr = 0;
  std::vector<uint32_t> seg_root(nseg, kInvalidID);
  GB_CHECK(cudaMemcpyAsync(seg_root.data(), d_root, sizeof(uint32_t) * nseg, cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaMemcpyAsync(&small_iters, d_iters, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaMemcpyAsync(&berr, &acc->pad, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaStreamSynchronize(st));
  // the first collapse level holds one wide root per non-empty segment, in segment order
  std::vector<uint32_t> root_items;
  if (segmented) out->roots.assign(nseg, kInvalidID);
  for (uint32_t s = 0; s < nseg; s++) {
    if (seg_root[s] == kInvalidID) continue;
    if (seg_root[s] >= nnodes_bin) berr = 1;
    if (segmented) out->roots[s] = (uint32_t)root_items.size();
    root_items.push_back(seg_root[s]);
  }
  if (berr || root_items.empty() || (!segmented && root_items.size() != 1)) {
    return cudaErrorUnknown;
  }
  stats->ploc_iterations = iters + small_iters;
  stats->ploc_rounds = iters;
  arena.free(clo_b); arena.free(chi_b); arena.free(cidx_b);
  arena.free(clo_a); arena.free(chi_a); arena.free(cidx_a);
  arena.free(nn); arena.free(bsurv); arena.free(bmerge); arena.free(ploc_state);

  // ---- collapse, level by level (breadth-first node order)
  BinTree bt{bnbox, bncnt, N, leaf_max_used, (uint32_t)(opt.robust != 0), d_link};
  if (dp_cost) arena.free(dp_cost);
  WideNode* wnodes = nullptr;
  TriRecord* wtris = nullptr;
  const uint32_t maxw = N;  // wide internal nodes <= binary internal nodes + 1
  GB_CHECK(arena.alloc(&wnodes, maxw));
  GB_CHECK(arena.alloc(&wtris, N));
  uint32_t *items_a, *items_b, *kids, *nint, *ntri;
  GB_CHECK(arena.alloc(&items_a, maxw));
  GB_CHECK(arena.alloc(&items_b, maxw));
  GB_CHECK(arena.alloc(&kids, (size_t)8 * maxw));
  GB_CHECK(arena.alloc(&nint, maxw));
  GB_CHECK(arena.alloc(&ntri, maxw));
  uint32_t* leaf_root = nullptr;  // binary subtree of each leaf, at its first triangle's slot
  GB_CHECK(arena.alloc(&leaf_root, N));
  GB_CHECK(cudaMemsetAsync(leaf_root, 0xFF, sizeof(uint32_t) * N, st));
  double* d_sah = nullptr;
  uint32_t* d_leaves = nullptr;
  GB_CHECK(arena.alloc(&d_sah, 2));  // quantised, exact
  GB_CHECK(arena.alloc(&d_leaves, 1));
  uint32_t *cstate = nullptr, *seg_index = nullptr, *h_col = nullptr;
  GB_CHECK(arena.alloc(&cstate, kColStateWords));
  GB_CHECK(arena.alloc(&seg_index, nseg));
  GB_CHECK(arena.host(&h_col, kColStateWords));
  k_collapse_roots<<<1, 1024, 0, st>>>(d_root, nseg, nnodes_bin, items_a, seg_index, cstate, d_sah, d_leaves, nullptr);
  note_launches(1);
  const ColItems citems{{items_a, items_b}};
  uint32_t level = 0;
  const uint32_t max_levels = 0xFFFFFFFFu;  // host-driven: level starts recorded here, no bound
  auto enqueue_level = [&](uint32_t nitems_known) {  // the level's size, read by the host
    const uint32_t grid = cdiv(8ull * nitems_known, 128);
    k_collapse_count<<<grid, 128, 0, st>>>(bt, citems, cstate, kids, nint, ntri);
    note_launches(1);
    scan_excl2(nint, ntri, nitems_known, d_tot + 0, d_tot + 1, scan_sums, st, &acc->pad);
    k_collapse_emit<<<cdiv(8ull * nitems_known, COLLAPSE_THREADS),
                      COLLAPSE_THREADS, 0, st>>>(
        bt, kids, cstate, nint, ntri, wnodes, leaf_root, citems, d_sah, d_leaves, maxw, N, &acc->pad);
    k_collapse_advance<<<1, 32, 0, st>>>(d_tot, cstate, maxw, max_levels);
    note_launches(2);
    level++;
  };
  // one level per host read of the state: the grid fits the level
  uint32_t nitems = (uint32_t)root_items.size();
  std::vector<uint32_t> level_start;
  uint32_t level_base = 0;
  while (nitems > 0) {
    level_start.push_back(level_base);
    enqueue_level(nitems);
    GB_CHECK(cudaGetLastError());
    GB_CHECK(cudaMemcpyAsync(h_col, cstate, sizeof(uint32_t) * kColLevels, cudaMemcpyDeviceToHost, st));
    GB_CHECK(cudaStreamSynchronize(st));
    if (h_col[kColErr]) return cudaErrorUnknown;
    nitems = h_col[kColN];
    level_base = h_col[kColBase];
  }
  const uint32_t num_nodes = level_base, depth = (uint32_t)level_start.size();
  const uint32_t tri_next = level < 1 ? 0u : h_col[kColTri];
  k_write_leaves<<<cdiv(N, 256), 256, 0, st>>>(bt, d_geoms, pbox, leaf_root, N, wtris, &acc->pad, prec);
  note_launches(1);
  GB_CHECK(cudaGetLastError());
  arena.free(leaf_root);
  GB_CHECK(cudaMemcpyAsync(&berr, &acc->pad, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaStreamSynchronize(st));
  if (berr || tri_next != N) {
    return cudaErrorUnknown;
  }
  double sah_sum[2] = {0.0, 0.0};
  uint32_t nleaves = 0;
  GB_CHECK(cudaMemcpyAsync(sah_sum, d_sah, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaMemcpyAsync(&nleaves, d_leaves, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));

  // exact-size outputs
  GB_CHECK(cudaMalloc((void**)&out->nodes, (size_t)num_nodes * sizeof(WideNode)));
  GB_CHECK(cudaMalloc((void**)&out->tris, (size_t)N * sizeof(TriRecord)));
  GB_CHECK(copy_device(out->nodes, wnodes, (size_t)num_nodes * sizeof(WideNode), st));
  GB_CHECK(copy_device(out->tris, wtris, (size_t)N * sizeof(TriRecord), st));
  out->num_nodes = num_nodes;
  out->num_tris = N;
  out->depth = depth;
  out->robust = opt.robust != 0;
  level_start.push_back(num_nodes);
  out->level_start = level_start;

  arena.free(wnodes); arena.free(wtris);
  arena.free(items_a); arena.free(items_b); arena.free(kids);
  arena.free(nint); arena.free(ntri); arena.free(d_sah); arena.free(d_leaves);
  if (d_link) arena.free(d_link);
  arena.free(d_tot); arena.free(d_root); arena.free(d_iters); arena.free(scan_sums);
  arena.free(bnbox); arena.free(bncnt);
  arena.free(pbox); arena.free(acc); arena.free(d_geoms); arena.free(prec);
  arena.free(keys_a); arena.free(keys_b); arena.free(vals_a); arena.free(vals_b);
  GB_CHECK(cudaEventRecord(ev1, st));
  GB_CHECK(cudaStreamSynchronize(st));
  float ms = 0;
  cudaEventElapsedTime(&ms, ev0, ev1);

  // SAH relative to the root box (bvh_statistics.cpp: root node counts once)
  const float gx = out->hi[0] - out->lo[0], gy = out->hi[1] - out->lo[1], gz = out->hi[2] - out->lo[2];
  const double Aroot = std::max(0.0, (double)(gx * (gy + gz) + gy * gz));
  stats->sah = Aroot > 0 ? (Aroot + sah_sum[0]) / Aroot : 0.0;
  stats->sah_exact = Aroot > 0 ? (Aroot + sah_sum[1]) / Aroot : 0.0;
  stats->build_ms = ms;
  stats->num_nodes = num_nodes;
  stats->num_leaves = nleaves;
  stats->num_prims = N;
  stats->depth = depth;
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// builds without host reads (captured into CUDA graphs)
// ---------------------------------------------------------------------------

__global__ void k_acc_init(BoundsAcc* __restrict__ acc) {
  if (threadIdx.x == 0) {
    for (int d = 0; d < 3; d++) {
      acc->glo[d] = acc->clo[d] = 0xFFFFFFFFu;
      acc->ghi[d] = acc->chi[d] = 0u;
    }
    acc->nvalid = 0;
    acc->pad = 0;
    acc->kand = ~0ull;
    acc->kor = 0ull;
  }
}

// What the host reads of a replayed build, in page-locked host memory that the
// last kernel writes: one wait instead of a copy per value.
struct GraphBuildOut {
  double sah[2];
  uint32_t status, leaves, ploc_iters;
  uint32_t glo[3], ghi[3];  // ordered keys of the geometry bounds
  uint32_t cstate[kColStateWords];
  uint32_t roots[1];        // nseg entries
};

// Status of a replayed build: the plan's counts still hold, the rounds and
// levels sufficed, and no kernel flagged an error.
__global__ void k_graph_build_check(const BoundsAcc* __restrict__ acc, const uint32_t* __restrict__ ploc_state,
                                    const uint32_t* __restrict__ cstate, uint32_t valid_tris,
                                    const double* __restrict__ sah, const uint32_t* __restrict__ leaves,
                                    const uint32_t* __restrict__ seg_index, uint32_t nseg,
                                    GraphBuildOut* __restrict__ out) {
  for (uint32_t i = threadIdx.x; i < (uint32_t)kColStateWords; i += blockDim.x) out->cstate[i] = cstate[i];
  for (uint32_t i = threadIdx.x; i < nseg; i += blockDim.x) out->roots[i] = seg_index[i];
  if (threadIdx.x != 0) return;
  out->sah[0] = sah[0];
  out->sah[1] = sah[1];
  out->leaves = *leaves;
  out->ploc_iters = ploc_state[kPlocIters];
  for (int d = 0; d < 3; d++) {
    out->glo[d] = acc->glo[d];
    out->ghi[d] = acc->ghi[d];
  }
  uint32_t s = 0;
  if (acc->nvalid != valid_tris) s |= kGraphBuildCount;
  if (!ploc_state[kPlocDone] || ploc_state[kPlocN] > PLOC_SMALL) s |= kGraphBuildRounds;
  if (cstate[kColN] != 0 || cstate[kColTri] != valid_tris) s |= kGraphBuildLevels;
  if (acc->pad || cstate[kColErr]) s |= kGraphBuildError;
  out->status = s;
}

// Device time (globaltimer, ns) into stamps[k]: one thread, enqueued between the
// phases of a captured build when BuildOptions::phase_stamps is set.
__global__ void k_phase_stamp(unsigned long long* stamps, int k) {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  stamps[k] = t;
}

cudaError_t graph_build_prepare(const GeomDesc* h_geoms, int ngeoms, const BuildOptions& opt,
                                const GraphBuildPlan& plan, GraphBuild* g) {
  *g = GraphBuild{};
  g->plan = plan;
  g->opt = opt;
  g->ngeoms = ngeoms;
  uint64_t total64 = 0;
  for (int k = 0; k < ngeoms; k++) total64 += h_geoms[k].ntris;
  const uint32_t N = plan.valid_tris;
  if (total64 == 0 || total64 >= 0x7FFFFFFFull || N == 0 || N > total64 || plan.roots == 0 || plan.roots > N ||
      plan.levels == 0 || plan.levels > (uint32_t)kColMaxLevels)
    return cudaErrorInvalidValue;
  if (opt.segmented && (uint32_t)ngeoms > kMaxSegments) return cudaErrorInvalidValue;
  g->total = (uint32_t)total64;
  g->nseg = opt.segmented ? (uint32_t)ngeoms : 1u;
  g->nbin = 2 * N - plan.roots;
  g->maxw = N;
  g->radius = (opt.ploc_radius == 1 || opt.ploc_radius == 2 || opt.ploc_radius == 4 || opt.ploc_radius == 8)
                  ? (uint32_t)opt.ploc_radius
                  : (uint32_t)PLOC_R_MAX;
  auto alloc = [&](auto** p, size_t count) -> cudaError_t {
    using T = std::remove_pointer_t<std::remove_reference_t<decltype(*p)>>;
    const cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T));
    if (e == cudaSuccess) g->allocs.push_back((void*)*p);
    return e;
  };
  const uint32_t T = g->total, maxw = g->maxw;
  BoundsAcc* acc = nullptr;
  cudaError_t e = cudaSuccess;
  // the cooperative collapse: as many CTAs as can be resident at once
  {
    int per_sm = 0;
    g->col_threads = N > COLLAPSE_WIDE_TRIS ? COLLAPSE_WIDE_THREADS : COLLAPSE_NARROW_THREADS;
    const void* collapse = g->col_threads == COLLAPSE_WIDE_THREADS ? (const void*)k_collapse_all<COLLAPSE_WIDE_THREADS>
                                                                   : (const void*)k_collapse_all<COLLAPSE_NARROW_THREADS>;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, collapse, g->col_threads, 0)) != cudaSuccess) return e;
    g->col_grid = (uint32_t)std::max(1, std::min(per_sm, 1)) * (uint32_t)num_sms_build();
    // and the cooperative PLOC rounds (of the chosen search radius)
    const void* pk = g->radius == 1   ? (const void*)k_ploc_rounds1
                     : g->radius == 2 ? (const void*)k_ploc_all<2>
                     : g->radius == 4 ? (const void*)k_ploc_all<4>
                     : g->radius == 8 ? (const void*)k_ploc_all<8>
                                      : (const void*)k_ploc_all<PLOC_R_MAX>;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pk, g->radius == 1 ? PLOC1_THREADS : PLOC_BLOCK, 0)) !=
        cudaSuccess)
      return e;
    g->ploc_grid = (uint32_t)std::max(1, std::min(per_sm, g->radius == 1 ? PLOC1_CTAS : 8)) * (uint32_t)num_sms_build();
  }
  if ((e = alloc(&g->d_geoms, ngeoms)) || (e = alloc(&g->pbox, 2 * (size_t)T)) ||
      (e = alloc(&acc, 1)) || (e = alloc(&g->keys_a, T)) || (e = alloc(&g->keys_b, T)) ||
      (e = alloc(&g->vals_a, T)) || (e = alloc(&g->vals_b, T)) || (e = alloc(&g->hist, sort_hist_entries(T))) ||
      (e = alloc(&g->bnbox, 4 * (size_t)N)) ||
      (e = alloc(&g->bncnt, 2 * (size_t)N)) || (e = alloc(&g->clo[0], N)) || (e = alloc(&g->clo[1], N)) ||
      (e = alloc(&g->chi[0], N)) || (e = alloc(&g->chi[1], N)) || (e = alloc(&g->cidx[0], N)) ||
      (e = alloc(&g->cidx[1], N)) || (e = alloc(&g->nn, N)) || (e = alloc(&g->bsurv, cdiv(N, 32))) ||
      (e = alloc(&g->bmerge, cdiv(N, 32))) ||
      (e = alloc(&g->d_root, g->nseg)) || (e = alloc(&g->d_iters, 1)) ||
      (e = alloc(&g->ploc_state, kPlocStateWords)) || (e = alloc(&g->cost, 2 * (size_t)(2 * N))) ||
      (e = alloc(&g->link, 2 * (size_t)N)) || (e = alloc(&g->nodes, maxw)) || (e = alloc(&g->tris, N)) ||
      (e = alloc(&g->items[0], maxw)) || (e = alloc(&g->items[1], maxw)) || (e = alloc(&g->kids, 8 * (size_t)maxw)) ||
      (e = alloc(&g->nint, maxw)) || (e = alloc(&g->ntri, maxw)) || (e = alloc(&g->leaf_root, N)) ||
      (e = alloc(&g->d_sah, 2)) || (e = alloc(&g->d_leaves, 1)) || (e = alloc(&g->cstate, kColStateWords)) ||
      (e = alloc(&g->seg_index, g->nseg)) ||
      (e = cudaMallocHost((void**)&g->out, sizeof(GraphBuildOut) + sizeof(uint32_t) * g->nseg)) ||
      (e = alloc(&g->col_sums, g->col_grid)) || (e = alloc(&g->col_bar, 2)) ||
      (e = alloc(&g->prec, T)) || (e = alloc(&g->ploc_sums, 2 * (size_t)g->ploc_grid)) ||
      (e = alloc(&g->ploc_bar, 2)) || (opt.phase_stamps && (e = alloc(&g->stamps, kBuildPhases + 1)))) {
    graph_build_release(g);
    return e;
  }
  g->acc = acc;
  e = cudaMemcpy(g->d_geoms, h_geoms, sizeof(GeomDesc) * ngeoms, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_os_scatter<uint64_t, RS_ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)os_scatter_smem<uint64_t, RS_ITEMS>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_os_scatter<uint32_t, RS_ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)os_scatter_smem<uint32_t, RS_ITEMS>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sort_one<uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sort_one_smem<uint64_t>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sort_one<uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sort_one_smem<uint32_t>());
  if (e == cudaSuccess) e = ploc_finish_prepare();
  if (e != cudaSuccess) graph_build_release(g);
  return e;
}


cudaError_t graph_build_enqueue(const GraphBuild& g, cudaStream_t st) {
  const uint32_t T = g.total, N = g.plan.valid_tris, maxw = g.maxw;
  BoundsAcc* acc = reinterpret_cast<BoundsAcc*>(g.acc);
  auto stamp = [&](int k) {
    if (g.stamps) k_phase_stamp<<<1, 1, 0, st>>>(g.stamps, k);
  };
  stamp(0);
  k_acc_init<<<1, 32, 0, st>>>(acc);
  k_primrefs<<<grid_stride_blocks(T), 256, 0, st>>>(g.d_geoms, g.ngeoms, T, g.pbox, acc, g.prec,
                                                    g.opt.robust ? 1 : 0);
  const bool key32 = g.opt.morton_bits == 30 && !g.opt.segmented;  // 30-bit keys sorted as 32-bit words
  k_morton<<<grid_stride_blocks(T), 256, 0, st>>>(g.pbox, T, acc, g.keys_a, g.vals_a, g.opt.morton_cube,
                                                  g.opt.segmented ? g.nseg : 0u, g.opt.morton_bits == 30 ? 1 : 0,
                                                  key32 ? 1 : 0);
  note_launches(3);
  stamp(1);
  // all digits of the key width (the ordinary build skips constant ones: the same order)
  uint64_t *ka = g.keys_a, *kb = g.keys_b;
  uint32_t *va = g.vals_a, *vb = g.vals_b;
  // the digits the key width can use: 63-bit keys 8, 30-bit keys 4 (5 or 6 with the slot)
  const uint32_t digits = g.opt.morton_bits != 30 ? 0xFFu
                          : !g.opt.segmented    ? 0x0Fu
                          : g.nseg <= kFewSegments ? 0x1Fu
                                                   : 0x3Fu;
  if (key32) {
    uint32_t *ka32 = reinterpret_cast<uint32_t*>(ka), *kb32 = reinterpret_cast<uint32_t*>(kb);
    GB_CHECK(onesweep_sort(ka32, va, kb32, vb, T, digits, g.hist, &acc->pad, st));
  } else {
    GB_CHECK(onesweep_sort(ka, va, kb, vb, T, digits, g.hist, &acc->pad, st));
  }
  stamp(2);
  // PLOC: the rounds in one cooperative launch that ends them itself, then the
  // one-CTA finish
  GB_CHECK(cudaMemsetAsync(g.d_root, 0xFF, sizeof(uint32_t) * g.nseg, st));
  GB_CHECK(cudaMemsetAsync(g.d_iters, 0, sizeof(uint32_t), st));
  const uint32_t leaf_max = (uint32_t)std::min(std::max(g.plan.leaf_max, 1), kLeafMaxLimit);
  float4* dp_cost = g.opt.collapse == 1 ? g.cost : nullptr;
  uint4* dp_link = g.opt.collapse == 1 ? g.link : nullptr;
  k_ploc_init<<<cdiv(N, 256), 256, 0, st>>>(g.pbox, va, N, &acc->nvalid, g.bnbox, g.cidx[0],
                                            g.clo[0], g.chi[0], g.opt.segmented ? 1 : 0);
  stamp(3);
  k_ploc_state_init<<<1, 32, 0, st>>>(acc, N, g.ploc_state, reinterpret_cast<GridBarrier*>(g.ploc_bar));
  note_launches(2);
  const uint32_t nbin_cap = 2 * N;
  const PlocBufs pb{{g.clo[0], g.clo[1]}, {g.chi[0], g.chi[1]}, {g.cidx[0], g.cidx[1]}};
  // the rounds above PLOC_SMALL clusters in one cooperative launch, then the one-CTA finish
  {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.ploc_grid);
    cfg.blockDim = dim3(g.radius == 1 ? PLOC1_THREADS : PLOC_BLOCK);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GridBarrier* bar = reinterpret_cast<GridBarrier*>(g.ploc_bar);
    switch (g.radius) {
      case 1: GB_CHECK(cudaLaunchKernelEx(&cfg, k_ploc_rounds1, pb, g.ploc_state, g.nn, g.bsurv, g.bmerge,
                                          reinterpret_cast<uint2*>(g.ploc_sums),
                                          g.bnbox, g.bncnt, nbin_cap, dp_cost, dp_link, leaf_max, bar, &acc->pad)); break;
      case 2: GB_CHECK(cudaLaunchKernelEx(&cfg, k_ploc_all<2>, pb, g.ploc_state, g.nn, g.bsurv, g.bmerge, g.ploc_sums,
                                          g.bnbox, g.bncnt, nbin_cap, dp_cost, dp_link, leaf_max, bar,
                                          &acc->pad)); break;
      case 4: GB_CHECK(cudaLaunchKernelEx(&cfg, k_ploc_all<4>, pb, g.ploc_state, g.nn, g.bsurv, g.bmerge, g.ploc_sums,
                                          g.bnbox, g.bncnt, nbin_cap, dp_cost, dp_link, leaf_max, bar,
                                          &acc->pad)); break;
      case 8: GB_CHECK(cudaLaunchKernelEx(&cfg, k_ploc_all<8>, pb, g.ploc_state, g.nn, g.bsurv, g.bmerge, g.ploc_sums,
                                          g.bnbox, g.bncnt, nbin_cap, dp_cost, dp_link, leaf_max, bar,
                                          &acc->pad)); break;
      default: GB_CHECK(cudaLaunchKernelEx(&cfg, k_ploc_all<PLOC_R_MAX>, pb, g.ploc_state, g.nn, g.bsurv, g.bmerge,
                                           g.ploc_sums, g.bnbox, g.bncnt, nbin_cap, dp_cost, dp_link,
                                           leaf_max, bar, &acc->pad)); break;
    }
    note_launches(2);
  }
  stamp(4);
  {
    GB_CHECK(ploc_finish(pb, g.ploc_state, g.bnbox, g.bncnt, g.d_root, g.d_iters, nbin_cap, &acc->pad, g.nseg,
                         (int)g.radius, dp_cost, dp_link, leaf_max, st));
  }
  stamp(5);
  // all collapse levels in one cooperative launch
  BinTree bt{g.bnbox, g.bncnt, N, leaf_max, (uint32_t)(g.opt.robust != 0), dp_link};
  GB_CHECK(cudaMemsetAsync(g.leaf_root, 0xFF, sizeof(uint32_t) * N, st));
  stamp(6);
  k_collapse_roots<<<1, 1024, 0, st>>>(g.d_root, g.nseg, g.nbin, g.items[0], g.seg_index, g.cstate, g.d_sah, g.d_leaves,
                                       reinterpret_cast<GridBarrier*>(g.col_bar));
  {
    const ColItems ci{{g.items[0], g.items[1]}};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.col_grid);
    cfg.blockDim = dim3(g.col_threads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const auto collapse = g.col_threads == COLLAPSE_WIDE_THREADS ? k_collapse_all<COLLAPSE_WIDE_THREADS>
                                                                 : k_collapse_all<COLLAPSE_NARROW_THREADS>;
    GB_CHECK(cudaLaunchKernelEx(&cfg, collapse, bt, ci, g.cstate, g.kids, g.nint, g.ntri, g.col_sums, g.nodes,
                                g.leaf_root, g.d_sah, g.d_leaves, maxw, N, (uint32_t)kColMaxLevels,
                                reinterpret_cast<GridBarrier*>(g.col_bar), &acc->pad));
  }
  note_launches(2);
  stamp(7);
  k_write_leaves<<<cdiv(N, 256), 256, 0, st>>>(bt, g.d_geoms, g.pbox, g.leaf_root, N, g.tris, &acc->pad,
                                                g.prec);
  stamp(8);
  k_graph_build_check<<<1, 128, 0, st>>>(acc, g.ploc_state, g.cstate, N, g.d_sah, g.d_leaves, g.seg_index, g.nseg,
                                         g.out);
  note_launches(2);
  return cudaGetLastError();
}

cudaError_t graph_build_result(const GraphBuild& g, const float scene_lo[3], const float scene_hi[3],
                               GraphBuildResult* out, cudaStream_t st) {
  *out = GraphBuildResult{};
  unsigned long long ts[kBuildPhases + 1] = {};
  if (g.stamps) GB_CHECK(cudaMemcpyAsync(ts, g.stamps, sizeof(ts), cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaStreamSynchronize(st));
  const GraphBuildOut& r = *g.out;
  const uint32_t* col = r.cstate;
  out->status = r.status;
  out->num_leaves = r.leaves;
  out->ploc_rounds = r.ploc_iters;
  if (g.opt.segmented) out->roots.assign(r.roots, r.roots + g.nseg);
  if (g.stamps) {
    out->nphases = kBuildPhases;
    for (int k = 0; k < kBuildPhases; k++) out->phase_us[k] = (double)(ts[k + 1] - ts[k]) * 1e-3;
  }
  out->num_nodes = col[kColBase];
  out->depth = std::min<uint32_t>(col[kColDepth], (uint32_t)kColMaxLevels);
  out->level_start.assign(col + kColLevels, col + kColLevels + out->depth + 1);
  // the replayed build's own geometry bounds, unless the caller passes the scene's
  for (int d = 0; d < 3; d++) {
    out->lo[d] = scene_lo ? scene_lo[d] : ord2f(r.glo[d]);
    out->hi[d] = scene_hi ? scene_hi[d] : ord2f(r.ghi[d]);
  }
  if (!g.opt.segmented) out->roots.assign(1, 0u);
  const float gx = out->hi[0] - out->lo[0], gy = out->hi[1] - out->lo[1], gz = out->hi[2] - out->lo[2];
  const double Aroot = std::max(0.0, (double)(gx * (gy + gz) + gy * gz));
  out->sah = Aroot > 0 ? (Aroot + r.sah[0]) / Aroot : 0.0;
  out->sah_exact = Aroot > 0 ? (Aroot + r.sah[1]) / Aroot : 0.0;
  return cudaSuccess;
}

void graph_build_release(GraphBuild* g) {
  for (void* p : g->allocs) cudaFree(p);
  if (g->out) cudaFreeHost(g->out);
  *g = GraphBuild{};
}

void cached_build_release(CachedBuild* c) {
  if (!c) return;
  if (c->exec) cudaGraphExecDestroy(c->exec);
  if (c->graph) cudaGraphDestroy(c->graph);
  if (c->e0) cudaEventDestroy(c->e0);
  if (c->e1) cudaEventDestroy(c->e1);
  graph_build_release(&c->g);
  delete c;
}

cudaError_t cached_build_create(const GeomDesc* h_geoms, int ngeoms, const BuildOptions& opt,
                                const GraphBuildPlan& plan, cudaStream_t st, CachedBuild** out) {
  *out = nullptr;
  CachedBuild* c = new CachedBuild;
  cudaError_t e = graph_build_prepare(h_geoms, ngeoms, opt, plan, &c->g);
  if (e == cudaSuccess) e = cudaEventCreate(&c->e0);
  if (e == cudaSuccess) e = cudaEventCreate(&c->e1);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    const cudaError_t e1 = graph_build_enqueue(c->g, st);
    const cudaError_t e2 = cudaStreamEndCapture(st, &c->graph);
    e = e1 != cudaSuccess ? e1 : e2;
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&c->exec, c->graph, 0);
  if (e != cudaSuccess) {
    cudaGetLastError();
    cached_build_release(c);
    return e;
  }
  *out = c;
  return cudaSuccess;
}

cudaError_t cached_build_run(CachedBuild* c, const GeomDesc* h_geoms, int ngeoms, cudaStream_t st, DeviceBVH* out,
                             BuildStats* stats) {
  if (!c || ngeoms != c->g.ngeoms) return cudaErrorNotReady;
  // the geometry table is read by the graph's kernels: buffers may have moved
  GB_CHECK(cudaMemcpyAsync(c->g.d_geoms, h_geoms, sizeof(GeomDesc) * ngeoms, cudaMemcpyHostToDevice, st));
  GB_CHECK(cudaEventRecord(c->e0, st));
  GB_CHECK(cudaGraphLaunch(c->exec, st));
  GB_CHECK(cudaEventRecord(c->e1, st));
  GraphBuildResult r;
  GB_CHECK(graph_build_result(c->g, nullptr, nullptr, &r, st));
  if (r.status != 0) return cudaErrorNotReady;
  const uint32_t N = c->g.plan.valid_tris;
  // the BVH stays where the build wrote it: a copy of its own cost two allocations,
  // two releases and 0.1 ms of copying per commit of a 4M-triangle scene
  out->nodes = c->g.nodes;
  out->tris = c->g.tris;
  out->borrowed = true;
  out->num_nodes = r.num_nodes;
  out->num_tris = N;
  out->depth = r.depth;
  out->robust = c->g.opt.robust != 0;
  for (int d = 0; d < 3; d++) { out->lo[d] = r.lo[d]; out->hi[d] = r.hi[d]; }
  out->level_start = r.level_start;
  out->roots = r.roots;
  float ms = 0;
  cudaEventElapsedTime(&ms, c->e0, c->e1);
  *stats = BuildStats{};
  stats->sah = r.sah;
  stats->sah_exact = r.sah_exact;
  stats->leaf_max = (uint32_t)c->g.plan.leaf_max;
  stats->build_ms = ms;
  stats->num_nodes = r.num_nodes;
  stats->num_leaves = r.num_leaves;
  stats->num_prims = N;
  stats->depth = r.depth;
  stats->ploc_iterations = r.ploc_rounds;
  stats->nphases = r.nphases;
  for (int k = 0; k < kBuildPhases; k++) stats->phase_us[k] = r.phase_us[k];
  return cudaSuccess;
}

// Sorts (key, value) pairs by their low `passes` digits with the builder's
// radix sort.  Device pointers; results in keys/vals (even pass counts).
cudaError_t sort_pairs_passes(uint64_t* keys, uint32_t* vals, uint64_t* kb, uint32_t* vb, uint32_t* hist, uint32_t n,
                              int passes, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (passes < 0 || passes > 8 || (passes & 1)) return cudaErrorInvalidValue;
  uint64_t* ka = keys;
  uint32_t* va = vals;
  return onesweep_sort(ka, va, kb, vb, n, (1u << passes) - 1u, hist, nullptr, st);
}

// onesweep scratch for all 8 digits of exactly n keys (fewer keys in smaller tiles can
// need more)
uint32_t sort_hist_entries(uint32_t n) { return (uint32_t)onesweep_scratch_words(n, 8); }

cudaError_t sort_pairs(uint64_t* keys, uint32_t* vals, uint32_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  uint64_t* kb = nullptr;
  uint32_t* vb = nullptr;
  uint32_t* hist = nullptr;
  GB_CHECK(dalloc(&kb, n, st));
  GB_CHECK(dalloc(&vb, n, st));
  GB_CHECK(dalloc(&hist, (size_t)sort_hist_entries(n), st));
  uint64_t* ka = keys;
  uint32_t* va = vals;
  cudaError_t e = onesweep_sort(ka, va, kb, vb, n, 0xFFu, hist, nullptr, st);  // 8 passes: back in keys/vals
  uint32_t serr = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&serr, hist + kOsErr, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(kb, st);
  cudaFreeAsync(vb, st);
  cudaFreeAsync(hist, st);
  const cudaError_t s2 = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  if (s2 != cudaSuccess) return s2;
  return serr ? cudaErrorUnknown : cudaSuccess;
}


// ---------------------------------------------------------------------------
// 6. refit: same topology, new vertex positions
//
// Replaces the reference's BVH refitter (kernels/bvh/bvh_refit.cpp:30-247),
// which recomputes node bounds bottom-up for meshes whose topology did not
// change.  Triangle records are re-gathered from the updated vertex buffers,
// then every breadth-first level, deepest first, recomputes its children's
// boxes (leaves from their triangles' vertices, inner children from the box
// the deeper level stored) and requantises them in the node's new frame.
// Slot order and leaf grouping stay as built.
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool refit_tri_vertices(const GeomDesc* __restrict__ geoms,
                                                   const uint32_t* __restrict__ slot_of, uint32_t nslots,
                                                   const TriRecord& rec, float3& p0, float3& p1, float3& p2) {
  const uint32_t primID = __float_as_uint(rec.a.w), geomID = __float_as_uint(rec.b.w);
  if (geomID >= nslots) return false;
  const uint32_t slot = slot_of[geomID];
  if (slot == kInvalidID) return false;
  const GeomDesc g = geoms[slot];
  if (primID >= g.ntris) return false;
  const uint3 t = load_tri(g, primID);
  if (t.x >= g.nverts || t.y >= g.nverts || t.z >= g.nverts) return false;
  p0 = load_vtx(g, t.x);
  p1 = load_vtx(g, t.y);
  p2 = load_vtx(g, t.z);
  return vtx_ok(p0.x, p0.y, p0.z) && vtx_ok(p1.x, p1.y, p1.z) && vtx_ok(p2.x, p2.y, p2.z);
}

// Rewrites triangle record i from the current vertices and stores the triangle's
// box (tri_box[2i] = lo, [2i + 1] = hi) for the node levels.
__device__ __forceinline__ void refit_tri(const GeomDesc* __restrict__ geoms, const uint32_t* __restrict__ slot_of,
                                          uint32_t nslots, TriRecord* __restrict__ tris, uint32_t i, int robust,
                                          float4* __restrict__ tri_box, uint32_t* err) {
  TriRecord rec = tris[i];
  float3 p0, p1, p2;
  if (!refit_tri_vertices(geoms, slot_of, nslots, rec, p0, p1, p2)) {
    atomicOr(err, kErrBuild);  // the host falls back to a full build
    return;
  }
  const float3 e1 = robust ? p1 : make_float3(__fsub_rn(p0.x, p1.x), __fsub_rn(p0.y, p1.y), __fsub_rn(p0.z, p1.z));
  const float3 e2 = robust ? p2 : make_float3(__fsub_rn(p2.x, p0.x), __fsub_rn(p2.y, p0.y), __fsub_rn(p2.z, p0.z));
  rec.a = make_float4(p0.x, p0.y, p0.z, rec.a.w);
  rec.b = make_float4(e1.x, e1.y, e1.z, rec.b.w);
  rec.c = make_float4(e2.x, e2.y, e2.z, 0.f);
  tris[i] = rec;
  const float3 lo = f3min(f3min(p0, p1), p2), hi = f3max(f3max(p0, p1), p2);
  tri_box[2 * (size_t)i] = make_float4(lo.x, lo.y, lo.z, 0.f);
  tri_box[2 * (size_t)i + 1] = make_float4(hi.x, hi.y, hi.z, 0.f);
}

// Refits wide node k from its children's boxes (inner children: node_box of the
// level below; leaf children: the boxes refit_tri stored for their triangles) and
// adds the node's SAH terms on the decoded and on the exact boxes.  The 8 lanes of
// a lane group share the node, lane i its slot i (all 32 lanes of the warp call it,
// `have` is the group's): the children's loads are one dependent step instead of eight,
// and a level takes as long as its widest lane.  Boxes are read past L1, where
// another CTA of the same launch may have written them.
__device__ __forceinline__ void refit_node_group(const float4* tri_box, uint32_t num_tris,
                                                 WideNode* __restrict__ nodes, uint32_t num_nodes, float* node_box,
                                                 uint32_t k, bool have, uint32_t* err, double& sah_out,
                                                 double& sahx_out) {
  const uint32_t s = threadIdx.x & 7u;
  WideNode* node = nodes + (have ? k : 0u);
  const uint32_t m = have ? node->meta[s] : 0u, imask = node->imask;
  float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
  bool ok = true;
  if (m != 0) {
    if (imask >> s & 1u) {
      const uint32_t c = node->child_base + __popc(imask & ((1u << s) - 1u));
      if (c >= num_nodes || c <= k) {
        ok = false;
      } else {
        const float* bx = node_box + 6 * (size_t)c;
        lo = make_float3(__ldcg(bx + 0), __ldcg(bx + 1), __ldcg(bx + 2));
        hi = make_float3(__ldcg(bx + 3), __ldcg(bx + 4), __ldcg(bx + 5));
      }
    } else {
      const uint32_t cnt = ((m >> 5) & 3u) + 1u, first = node->tri_base + (m & 31u);
      if (first + cnt > num_tris) {
        ok = false;
      } else {
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) {
          if (q < cnt) {
            const float4 a = __ldcg(tri_box + 2 * (size_t)(first + q)), b = __ldcg(tri_box + 2 * (size_t)(first + q) + 1);
            lo = f3min(lo, make_float3(a.x, a.y, a.z));
            hi = f3max(hi, make_float3(b.x, b.y, b.z));
          }
        }
      }
    }
  }
  const uint32_t bad = __ballot_sync(0xFFFFFFFFu, !ok) >> (threadIdx.x & 24u) & 0xFFu;
  if (bad && s == 0) atomicOr(err, kErrBuild);
  have = have && bad == 0u;
  float3 ulo = lo, uhi = hi;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    ulo.x = fminf(ulo.x, __shfl_xor_sync(0xFFFFFFFFu, ulo.x, o));
    ulo.y = fminf(ulo.y, __shfl_xor_sync(0xFFFFFFFFu, ulo.y, o));
    ulo.z = fminf(ulo.z, __shfl_xor_sync(0xFFFFFFFFu, ulo.z, o));
    uhi.x = fmaxf(uhi.x, __shfl_xor_sync(0xFFFFFFFFu, uhi.x, o));
    uhi.y = fmaxf(uhi.y, __shfl_xor_sync(0xFFFFFFFFu, uhi.y, o));
    uhi.z = fmaxf(uhi.z, __shfl_xor_sync(0xFFFFFFFFu, uhi.z, o));
  }
  const uint32_t Ex = exp_for(__fsub_ru(uhi.x, ulo.x));
  const uint32_t Ey = exp_for(__fsub_ru(uhi.y, ulo.y));
  const uint32_t Ez = exp_for(__fsub_ru(uhi.z, ulo.z));
  const float sx = __uint_as_float(Ex << 23), sy = __uint_as_float(Ey << 23), sz = __uint_as_float(Ez << 23);
  if (!have) return;
  if (m != 0) {
    const float ix = __uint_as_float((254u - Ex) << 23), iy = __uint_as_float((254u - Ey) << 23),
                iz = __uint_as_float((254u - Ez) << 23);
    const uint32_t qlx = min(__float2uint_rd(__fsub_rd(lo.x, ulo.x) * ix), 255u);
    const uint32_t qly = min(__float2uint_rd(__fsub_rd(lo.y, ulo.y) * iy), 255u);
    const uint32_t qlz = min(__float2uint_rd(__fsub_rd(lo.z, ulo.z) * iz), 255u);
    const uint32_t qhx = min(__float2uint_ru(__fsub_ru(hi.x, ulo.x) * ix), 255u);
    const uint32_t qhy = min(__float2uint_ru(__fsub_ru(hi.y, ulo.y) * iy), 255u);
    const uint32_t qhz = min(__float2uint_ru(__fsub_ru(hi.z, ulo.z) * iz), 255u);
    node->qlo_x[s] = (uint8_t)qlx; node->qlo_y[s] = (uint8_t)qly; node->qlo_z[s] = (uint8_t)qlz;
    node->qhi_x[s] = (uint8_t)qhx; node->qhi_y[s] = (uint8_t)qhy; node->qhi_z[s] = (uint8_t)qhz;
    const float3 dlo = make_float3(__fmaf_rd(byte_f(qlx), sx, ulo.x), __fmaf_rd(byte_f(qly), sy, ulo.y), __fmaf_rd(byte_f(qlz), sz, ulo.z));
    const float3 dhi = make_float3(__fmaf_ru(byte_f(qhx), sx, ulo.x), __fmaf_ru(byte_f(qhy), sy, ulo.y), __fmaf_ru(byte_f(qhz), sz, ulo.z));
    sah_out += (double)fmaxf(0.f, half_area(dlo, dhi));  // leaves of <= 4 triangles: one block each
    sahx_out += (double)fmaxf(0.f, half_area(lo, hi));
  }
  // frame and scales (16-byte words 0 and 5), then the node's box
  if (s == 0)
    reinterpret_cast<uint4*>(node)[0] = make_uint4(__float_as_uint(ulo.x), __float_as_uint(ulo.y), __float_as_uint(ulo.z),
                                                   Ex | (Ey << 8) | (Ez << 16) | (imask << 24));
  else if (s == 1)
    reinterpret_cast<uint4*>(node)[5] = make_uint4(__float_as_uint(sx * 32768.0f), __float_as_uint(sy * 32768.0f),
                                                   __float_as_uint(sz * 32768.0f), 0u);
  else
    node_box[6 * (size_t)k + s - 2] = s == 2 ? ulo.x : s == 3 ? ulo.y : s == 4 ? ulo.z : s == 5 ? uhi.x : s == 6 ? uhi.y : uhi.z;
}

// The breadth-first levels of a BVH whose levels fit (deeper ones are refitted by
// one launch per level).
struct RefitLevels {
  uint32_t n;
  uint32_t start[kColMaxLevels + 1];
};

// Two CTAs of 256 threads per SM: the refit of a soup of 8k / 60k / 200k / 500k / 1M
// triangles takes 25 / 36 / 48 / 71 / 117 us, with 2 x 512 28 / 36 / 55 / 75 / 109, with
// 3 x 256 25 / 36 / 55 / 78 / 115, with 4 x 256 25 / 36 / 64 / 87 / 123, with 1 x 512
// 28 / 36 / 48 / 72 / 117 and with 1 x 1024 36 / 47 / 58 / 79 / 113 us: a chain of levels
// waits for all CTAs and warps at each barrier, and only the largest trees have work
// for more of them.  Levels of at most kRefitNarrow nodes are refitted by the first CTA
// alone, without a grid barrier between two of them (64 or 128: 1 to 2 us more).
constexpr int kRefitThreads = 256, kRefitCtas = 2;
constexpr uint32_t kRefitNarrow = 32;

// The whole refit in one cooperative launch: the triangles, then the levels,
// deepest first, a grid barrier between two levels.  A refit is a chain of about 14
// levels that each take a few microseconds at most: as one launch per level with
// one thread per node, its eight children's loads in sequence, the chain took
// 0.44 ms on a 1M-triangle soup whatever the bandwidth (the whole refit 0.61 ms;
// here 0.12 ms, of which the 176 MB of the triangle pass need 0.03).  *bar and *bar_err are
// zero before the first launch and left ready for the next one (an error of the
// triangles or nodes does not stop the refit, a barrier that fails does).
__global__ void __launch_bounds__(kRefitThreads, kRefitCtas) k_refit_all(const GeomDesc* __restrict__ geoms,
                                                   const uint32_t* __restrict__ slot_of, uint32_t nslots,
                                                   TriRecord* __restrict__ tris, uint32_t num_tris, int robust,
                                                   float4* tri_box, WideNode* __restrict__ nodes, uint32_t num_nodes,
                                                   float* node_box, const RefitLevels lv, double* sah_acc,
                                                   GridBarrier* bar, unsigned int* bar_err, uint32_t* err) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < num_tris; i += gridDim.x * blockDim.x)
    refit_tri(geoms, slot_of, nslots, tris, i, robust, tri_box, err);
  double sah = 0.0, sahx = 0.0;
  bool wide_below = true;
  for (uint32_t l = lv.n; l-- > 0;) {
    const uint32_t begin = lv.start[l], end = min(lv.start[l + 1], num_nodes);
    const bool wide = end - begin > kRefitNarrow;
    if (wide || wide_below) {
      if (!grid_sync(bar, bar_err)) {
        if (threadIdx.x == 0) atomicOr(err, kErrBuild);
        break;
      }
    } else {
      __syncthreads();
    }
    wide_below = wide;
    if (!wide && blockIdx.x != 0) continue;
    const uint32_t stride = (wide ? gridDim.x * blockDim.x : blockDim.x) >> 3;
    const uint32_t warp0 = (wide ? blockIdx.x * blockDim.x : 0u) + (threadIdx.x & ~31u);
    for (uint32_t k0 = begin + (warp0 >> 3); k0 < end; k0 += stride) {
      const uint32_t k = k0 + ((threadIdx.x & 31u) >> 3);
      refit_node_group(tri_box, num_tris, nodes, num_nodes, node_box, k, k < end, err, sah, sahx);
    }
  }
  block_add2(sah, sahx, sah_acc);
}

// The same as separate launches, for BVHs of more levels than RefitLevels holds.
__global__ void __launch_bounds__(256) k_refit_tris(const GeomDesc* __restrict__ geoms,
                                                    const uint32_t* __restrict__ slot_of, uint32_t nslots,
                                                    TriRecord* __restrict__ tris, uint32_t n, int robust,
                                                    float4* __restrict__ tri_box, uint32_t* err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) refit_tri(geoms, slot_of, nslots, tris, i, robust, tri_box, err);
}
__global__ void __launch_bounds__(128) k_refit_level(const float4* tri_box, uint32_t num_tris,
                                                     WideNode* __restrict__ nodes, uint32_t num_nodes,
                                                     float* node_box, uint32_t begin, uint32_t end, double* sah_acc,
                                                     uint32_t* err) {
  const uint32_t k = begin + ((blockIdx.x * blockDim.x + threadIdx.x) >> 3);
  double sah = 0.0, sahx = 0.0;
  refit_node_group(tri_box, num_tris, nodes, num_nodes, node_box, k, k < end && k < num_nodes, err, sah, sahx);
  block_add2(sah, sahx, sah_acc);
}

cudaError_t refit_prepare(const GeomDesc* h_geoms, int ngeoms, const DeviceBVH& bvh, RefitScratch* out,
                          cudaStream_t st) {
  *out = RefitScratch{};
  if (bvh.num_nodes == 0 || bvh.level_start.size() < 2) return cudaErrorInvalidValue;
  uint32_t nslots = 0;
  for (int g = 0; g < ngeoms; g++) nslots = std::max(nslots, h_geoms[g].geomID + 1);
  std::vector<uint32_t> slot_of(std::max(nslots, 1u), kInvalidID);
  for (int g = 0; g < ngeoms; g++) slot_of[h_geoms[g].geomID] = (uint32_t)g;
  out->nslots = (uint32_t)slot_of.size();
  out->ngeoms = ngeoms;
  int per_sm = 0;
  GB_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_refit_all, kRefitThreads, 0));
  // enough CTAs for the triangles and the widest level, at most kRefitCtas per SM (a
  // grid barrier costs more with every CTA)
  uint64_t work = bvh.num_tris;
  for (size_t l = 0; l + 1 < bvh.level_start.size(); l++)
    work = std::max<uint64_t>(work, 8ull * (bvh.level_start[l + 1] - bvh.level_start[l]));
  out->grid = std::min<uint32_t>(cdiv(work, kRefitThreads),
                                 (uint32_t)std::max(1, std::min(per_sm, kRefitCtas)) * (uint32_t)num_sms_build());
  cudaError_t e = cudaMalloc(&out->d_geoms, sizeof(GeomDesc) * std::max(ngeoms, 1));
  if (e == cudaSuccess) e = cudaMalloc(&out->d_slot, sizeof(uint32_t) * slot_of.size());
  if (e == cudaSuccess) e = cudaMalloc(&out->result, sizeof(RefitResult) + sizeof(float) * 6 * (size_t)bvh.num_nodes);
  if (e == cudaSuccess) e = cudaMalloc(&out->tri_box, sizeof(float4) * 2 * std::max<size_t>(bvh.num_tris, 1));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(out->d_geoms, h_geoms, sizeof(GeomDesc) * ngeoms, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(out->d_slot, slot_of.data(), sizeof(uint32_t) * slot_of.size(), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(out->result, 0, sizeof(RefitResult), st);
  if (e == cudaSuccess) e = cudaEventCreate(&out->e0);
  if (e == cudaSuccess) e = cudaEventCreate(&out->e1);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) refit_release(out);
  return e;
}

cudaError_t refit_enqueue(const DeviceBVH& bvh, const RefitScratch& s, cudaStream_t st) {
  RefitResult* r = s.result;
  float* node_box = reinterpret_cast<float*>(r + 1);
  GB_CHECK(cudaMemsetAsync(r, 0, offsetof(RefitResult, err), st));  // sums and barrier
  const size_t nlevels = bvh.level_start.size() - 1;
  if (nlevels <= (size_t)kColMaxLevels) {
    RefitLevels lv{};
    lv.n = (uint32_t)nlevels;
    std::copy(bvh.level_start.begin(), bvh.level_start.end(), lv.start);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s.grid);
    cfg.blockDim = dim3(kRefitThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GB_CHECK(cudaLaunchKernelEx(&cfg, k_refit_all, (const GeomDesc*)s.d_geoms, (const uint32_t*)s.d_slot, s.nslots,
                                bvh.tris, bvh.num_tris, bvh.robust, s.tri_box, bvh.nodes, bvh.num_nodes, node_box, lv,
                                r->sah, reinterpret_cast<GridBarrier*>(&r->bar), &r->bar_err, &r->err));
    note_launches(1);
    return cudaGetLastError();
  }
  k_refit_tris<<<cdiv(bvh.num_tris, 256), 256, 0, st>>>(s.d_geoms, s.d_slot, s.nslots, bvh.tris, bvh.num_tris,
                                                        bvh.robust, s.tri_box, &r->err);
  note_launches(1);
  for (size_t l = nlevels; l-- > 0;) {
    const uint32_t b = bvh.level_start[l], e = bvh.level_start[l + 1];
    if (e <= b) continue;
    k_refit_level<<<cdiv(8ull * (e - b), 128), 128, 0, st>>>(s.tri_box, bvh.num_tris, bvh.nodes, bvh.num_nodes,
                                                             node_box, b, e, r->sah, &r->err);
    note_launches(1);
  }
  return cudaGetLastError();
}

// The scratch of a scene's refits is kept in *s between commits: it is made for the
// BVH of the last build (released when the scene is built again).
cudaError_t refit_bvh(const GeomDesc* h_geoms, int ngeoms, cudaStream_t st, DeviceBVH* bvh, BuildStats* stats,
                      bool* fallback, RefitScratch* s) {
  *fallback = false;
  if (bvh->num_nodes == 0 || bvh->level_start.size() < 2) {
    *fallback = true;
    return cudaSuccess;
  }
  if (!s->result) GB_CHECK(refit_prepare(h_geoms, ngeoms, *bvh, s, st));
  if (s->ngeoms != ngeoms) return cudaErrorInvalidValue;
  // buffers may have moved since the last commit
  GB_CHECK(cudaMemcpyAsync(s->d_geoms, h_geoms, sizeof(GeomDesc) * ngeoms, cudaMemcpyHostToDevice, st));
  GB_CHECK(cudaMemsetAsync(&s->result->err, 0, sizeof(uint32_t), st));
  GB_CHECK(cudaEventRecord(s->e0, st));
  GB_CHECK(refit_enqueue(*bvh, *s, st));
  GB_CHECK(cudaEventRecord(s->e1, st));
  struct {
    RefitResult r;
    float root[6];
  } out;
  static_assert(sizeof(out.r) + sizeof(out.root) <= sizeof(out), "result and root box in one copy");
  GB_CHECK(cudaMemcpyAsync(&out, s->result, sizeof(out.r) + sizeof(out.root), cudaMemcpyDeviceToHost, st));
  GB_CHECK(cudaStreamSynchronize(st));
  float ms = 0;
  cudaEventElapsedTime(&ms, s->e0, s->e1);
  if (out.r.err) {  // a vertex became invalid or the records are inconsistent: rebuild
    *fallback = true;
    return cudaSuccess;
  }
  for (int d = 0; d < 3; d++) {
    bvh->lo[d] = out.root[d];
    bvh->hi[d] = out.root[3 + d];
  }
  const float gx = bvh->hi[0] - bvh->lo[0], gy = bvh->hi[1] - bvh->lo[1], gz = bvh->hi[2] - bvh->lo[2];
  const double Aroot = std::max(0.0, (double)(gx * (gy + gz) + gy * gz));
  stats->sah = Aroot > 0 ? (Aroot + out.r.sah[0]) / Aroot : 0.0;
  stats->sah_exact = Aroot > 0 ? (Aroot + out.r.sah[1]) / Aroot : 0.0;
  stats->build_ms = ms;
  stats->num_nodes = bvh->num_nodes;
  stats->num_prims = bvh->num_tris;
  stats->depth = bvh->depth;
  stats->refit = 1;
  return cudaSuccess;
}

void refit_release(RefitScratch* s) {
  void* ptrs[] = {s->d_geoms, s->d_slot, s->result, s->tri_box};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  if (s->e0) cudaEventDestroy(s->e0);
  if (s->e1) cudaEventDestroy(s->e1);
  *s = RefitScratch{};
}

void free_bvh(DeviceBVH* b) {
  if (b->nodes && !b->borrowed) cudaFree(b->nodes);
  if (b->tris && !b->borrowed) cudaFree(b->tris);
  b->nodes = nullptr;
  b->tris = nullptr;
  b->borrowed = false;
  b->num_nodes = b->num_tris = 0;
}

}  // namespace gb

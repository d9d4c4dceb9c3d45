// gb_trace_kernel.cuh -- the persistent traversal kernel k_trace and the
// device arithmetic it uses, shared by the translation unit of the default
// launch shape (gb_trace.cu) and the one of the tuned shapes (gb_trace_shapes.cu).
//
// Replaces the reference's single-ray / hybrid traversal
// (kernels/bvh/bvh_intersector1.cpp:30-195, bvh_intersector_hybrid.cpp:36-375)
// with persistent CTAs: warps refill idle lanes with rays fetched by one
// atomic, every lane walks the 8-wide quantised BVH with a short stack of node
// groups (child base + hit bits), visiting children in the order given by the
// ray's direction octant, and the triangles of the leaves that a warp's rays
// reach are tested in batches over all its lanes.
//
// Arithmetic that decides hits is the reference's, bit for bit:
//   Moeller-Trumbore  kernels/geometry/triangle_intersector_moeller.h:62-104
//   dot / cross FMA placement  common/math/vec3.h:204-209, math.h:367-373
//   epilog t = T * rcp(absDen)  triangle_intersector_moeller.h:29-35
// with rcp the correctly rounded reciprocal.  Files including this one are
// compiled with --fmad=false and every rounding step is spelled out with
// intrinsics.
//
// The node test only prunes: its slab distances are widened by a bound on
// their rounding error, so a box that contains an accepted intersection is
// never culled.
#pragma once
#include <cuda_runtime.h>

#include "gb_build.h"
#include "gb_common.h"
#include "gb_trace.h"

namespace gb {

constexpr float kMinRcpInput = 1E-18f;  // common/math/constants.h:31

__device__ __forceinline__ float dot3(const float3 a, const float3 b) {
  return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, __fmul_rn(a.z, b.z)));
}
__device__ __forceinline__ float3 cross3(const float3 a, const float3 b) {
  return make_float3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
                     __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}

// Returns true when the triangle is hit inside (absDen*tnear, absDen*tfar].
__device__ __forceinline__ bool moeller(const float3 v0, const float3 e1, const float3 e2, const float3 O,
                                        const float3 D, const float tnear, const float tfar, float& U, float& V,
                                        float& T, float& absDen) {
  const float3 C = make_float3(__fsub_rn(v0.x, O.x), __fsub_rn(v0.y, O.y), __fsub_rn(v0.z, O.z));
  const float3 R = cross3(C, D);
  const float3 Ng = cross3(e2, e1);
  const float den = dot3(Ng, D);
  absDen = fabsf(den);
  const uint32_t sgn = __float_as_uint(den) & 0x80000000u;
  U = __uint_as_float(__float_as_uint(dot3(R, e2)) ^ sgn);
  V = __uint_as_float(__float_as_uint(dot3(R, e1)) ^ sgn);
  if (!((den != 0.0f) & (U >= 0.0f) & (V >= 0.0f) & (__fadd_rn(U, V) <= absDen))) return false;
  T = __uint_as_float(__float_as_uint(dot3(Ng, C)) ^ sgn);
  return (__fmul_rn(absDen, tnear) < T) & (T <= __fmul_rn(absDen, tfar));
}

// stable_triangle_normal (common/math/vec3.h:210-222): per component the
// cross product of (a,b) or (b,c) whose cancelling product is smaller.
__device__ __forceinline__ float3 stable_normal(const float3 a, const float3 b, const float3 c) {
  const float ab_x = __fmul_rn(a.z, b.y), ab_y = __fmul_rn(a.x, b.z), ab_z = __fmul_rn(a.y, b.x);
  const float bc_x = __fmul_rn(b.z, c.y), bc_y = __fmul_rn(b.x, c.z), bc_z = __fmul_rn(b.y, c.x);
  const float3 cab = make_float3(__fmaf_rn(a.y, b.z, -ab_x), __fmaf_rn(a.z, b.x, -ab_y), __fmaf_rn(a.x, b.y, -ab_z));
  const float3 cbc = make_float3(__fmaf_rn(b.y, c.z, -bc_x), __fmaf_rn(b.z, c.x, -bc_y), __fmaf_rn(b.x, c.y, -bc_z));
  return make_float3(fabsf(ab_x) < fabsf(bc_x) ? cab.x : cbc.x, fabsf(ab_y) < fabsf(bc_y) ? cab.y : cbc.y,
                     fabsf(ab_z) < fabsf(bc_z) ? cab.z : cbc.z);
}

__device__ __forceinline__ float3 f3sub(const float3 a, const float3 b) {
  return make_float3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float3 f3add(const float3 a, const float3 b) {
  return make_float3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z));
}

// Pluecker test of robust scenes (triangle_intersector_pluecker.h:60-111):
// vertices relative to the origin, edge functions U,V,W accepted within
// ulp*|U+V+W| of zero, t = rcp(2 Ng.D) * 2 v0.Ng inside [tnear, tfar].
__device__ __forceinline__ bool pluecker(const float3 tv0, const float3 tv1, const float3 tv2, const float3 O,
                                         const float3 D, const float tnear, const float tfar, float& U, float& V,
                                         float& UVW, float& t) {
  const float3 v0 = f3sub(tv0, O), v1 = f3sub(tv1, O), v2 = f3sub(tv2, O);
  const float3 e0 = f3sub(v2, v0), e1 = f3sub(v0, v1), e2 = f3sub(v1, v2);
  U = dot3(cross3(e0, f3add(v2, v0)), D);
  V = dot3(cross3(e1, f3add(v0, v1)), D);
  const float W = dot3(cross3(e2, f3add(v1, v2)), D);
  UVW = __fadd_rn(__fadd_rn(U, V), W);
  const float eps = __fmul_rn(1.1920928955078125e-07f, fabsf(UVW));
  if (!((fminf(fminf(U, V), W) >= -eps) | (fmaxf(fmaxf(U, V), W) <= eps))) return false;
  const float3 Ng = stable_normal(e0, e1, e2);
  const float dd = dot3(Ng, D), den = __fadd_rn(dd, dd);
  const float tt = dot3(v0, Ng), T = __fadd_rn(tt, tt);
  t = __fmul_rn(__frcp_rn(den), T);
  return (tnear <= t) & (t <= tfar) & (den != 0.0f);
}

// Geometric normal of a robust-scene hit, as the test computed it.
__device__ __forceinline__ float3 pluecker_normal(const float3 tv0, const float3 tv1, const float3 tv2, const float3 O) {
  const float3 v0 = f3sub(tv0, O), v1 = f3sub(tv1, O), v2 = f3sub(tv2, O);
  return stable_normal(f3sub(v2, v0), f3sub(v0, v1), f3sub(v1, v2));
}

struct TRay {
  float3 org, dir, rdir;
  float tnear;     // raw ray tnear (triangle test)
  float tnear_c;   // max(tnear, 0) (node test)
  uint32_t oct;    // bit a set when rdir_a < 0
};

__device__ __forceinline__ float rcp_safe(float d) {
  // zero_fix: |d| < 1e-18 -> +1e-18  (common/math/vec3fa.h:172-177)
  if (fabsf(d) < kMinRcpInput) d = kMinRcpInput;
  return __frcp_rn(d);
}

__device__ __forceinline__ void init_ray(TRay& r) {
  r.rdir = make_float3(rcp_safe(r.dir.x), rcp_safe(r.dir.y), rcp_safe(r.dir.z));
  r.oct = (r.rdir.x < 0.0f ? 1u : 0u) | (r.rdir.y < 0.0f ? 2u : 0u) | (r.rdir.z < 0.0f ? 4u : 0u);
  r.tnear_c = fmaxf(r.tnear, 0.0f);
}

// Three-input minimum / maximum (PTX ISA 8.8, sm_100 and later).
__device__ __forceinline__ float fmax3(const float a, const float b, const float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float fmin3(const float a, const float b, const float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// 32-byte word k of a node, in one load (sm_100 and later).  The divergent node
// loads are the L1 data pipe's main work, and it takes as long for 32 bytes of a
// line as for 16: three such loads instead of five of 16 bytes, from a node padded
// to 96 bytes (the pad holds the scales as floats, six operations less per visit).
// GB300, traversal kernel alone: 16M closest-hit rays on the 4M soup 9.79 -> 9.33 ms,
// 16M shadow rays 5.88 -> 5.58 ms, 14.6M batched rays 1.98 -> 1.92 ms.
__device__ __forceinline__ void ldg256(const WideNode* __restrict__ p, const int k, uint4& a, uint4& b) {
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
      : "l"(reinterpret_cast<const char*>(p) + 32 * k));
}

// Byte k of w as the float 1 + bb * 2^-15 (exact): one byte permute puts bb
// in mantissa bits 8..15 under the exponent of 1.0 (0x3F80bb00).
__device__ __forceinline__ float ubyte_f(uint32_t w, uint32_t k) {
  return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u | (k << 4)));
}

// Rounding slack of the slab test, relative to (|p - o| + 2^15 s) |1/d|: the
// computed slab distances carry at most ~6 unit roundoffs of that magnitude
// (one each from p - o, the product with 1/d, 1/d itself, the offset a - 2^15 b,
// the FMA and the subtraction of the slack); 8u = 2^-21 covers them with
// margin.  The 2^15 s term widens a box by 2^15 * 8u = 1.6 % of one
// quantisation step.  It is formed from the products the test needs anyway:
// |a| + |B| with a = fl((p - o) / d) >= |p - o| |1/d| (1 - u) and B = 2^15 s / d
// exact, so (|a| + |B|) * 2^-21 (1 + 2^-21), all rounded up, is at least
// (|p - o| + 2^15 s) |1/d| 8u; the floor 2^-144 (32 ulps of the smallest
// subnormal) covers the absolute rounding errors where the products underflow.
constexpr float kSlabEps = 0x1.000008p-21f;  // 2^-21 (1 + 2^-21)
constexpr float kSlabFloor = 0x1p-144f;      // 2^-144

// Intersects the 8 children of `np`.  Child box planes are p + q * 2^e; with
// B = 2^15 * 2^e / d and A = (p - o) / d - B precomputed per node and axis, a
// plane distance is one FMA (1 + q * 2^-15) * B + A = (p - o) / d + q * 2^e / d,
// whose first factor is the plane byte placed in a float's mantissa (no
// integer-to-float conversion or subtraction per plane), widened by the
// rounding slack (near planes down, far planes up) so a box that contains an
// accepted intersection is never culled.  Where B overflows (a 2^55 scale and
// |1/d| near 1e18) the products are NaN and fminf/fmaxf drop that plane, so
// the box only grows.  Returns the node group of hit internal children (bit
// 31 - j set when slot j ^ oct was hit, so the next child to visit is the
// leading one; imask in bits 0..7), the slots of the hit leaves, and the node's
// triangle base and meta bytes, which say where those leaves' triangles are.
// perm: the row of the ray's octant in the slot permutation table (perm[m] has
// bit 7 - j set when m has bit j ^ oct).
__device__ __forceinline__ void intersect_node(const WideNode* __restrict__ np, const TRay& r, const float tfar,
                                               uint32_t& g_base, uint32_t& g_bits, uint32_t& t_base, uint32_t& leaf,
                                               uint2& meta, const uint8_t* __restrict__ perm, const uint32_t row) {
  uint4 n0, n1, n2, n3, n4, n5;
  ldg256(np, 0, n0, n1);
  ldg256(np, 1, n2, n3);
  ldg256(np, 2, n4, n5);
  const uint32_t imask = n0.w >> 24;
  float bx, by, bz, anx, afx, any_, afy, anz, afz;
  {
    const float xo = __fsub_rn(__uint_as_float(n0.x), r.org.x);
    const float yo = __fsub_rn(__uint_as_float(n0.y), r.org.y);
    const float zo = __fsub_rn(__uint_as_float(n0.z), r.org.z);
    const float ax = __fmul_rn(xo, r.rdir.x), ay = __fmul_rn(yo, r.rdir.y), az = __fmul_rn(zo, r.rdir.z);
    // B = 2^15 s / d (exact scaling of s / d by a power of two), A = a - B
    bx = __fmul_rn(__uint_as_float(n5.x), r.rdir.x);
    by = __fmul_rn(__uint_as_float(n5.y), r.rdir.y);
    bz = __fmul_rn(__uint_as_float(n5.z), r.rdir.z);
    const float ax2 = __fsub_rn(ax, bx), ay2 = __fsub_rn(ay, by), az2 = __fsub_rn(az, bz);
    const float ex = __fmaf_ru(__fadd_ru(fabsf(ax), fabsf(bx)), kSlabEps, kSlabFloor);
    const float ey = __fmaf_ru(__fadd_ru(fabsf(ay), fabsf(by)), kSlabEps, kSlabFloor);
    const float ez = __fmaf_ru(__fadd_ru(fabsf(az), fabsf(bz)), kSlabEps, kSlabFloor);
    anx = __fsub_rd(ax2, ex); afx = __fadd_ru(ax2, ex);
    any_ = __fsub_rd(ay2, ey); afy = __fadd_ru(ay2, ey);
    anz = __fsub_rd(az2, ez); afz = __fadd_ru(az2, ez);
  }
  // near / far quantised planes by the ray direction's sign per axis
  const bool px = r.rdir.x >= 0.0f, py = r.rdir.y >= 0.0f, pz = r.rdir.z >= 0.0f;
  const uint32_t nx0 = px ? n2.x : n3.z, nx1 = px ? n2.y : n3.w, fx0 = px ? n3.z : n2.x, fx1 = px ? n3.w : n2.y;
  const uint32_t ny0 = py ? n2.z : n4.x, ny1 = py ? n2.w : n4.y, fy0 = py ? n4.x : n2.z, fy1 = py ? n4.y : n2.w;
  const uint32_t nz0 = pz ? n3.x : n4.z, nz1 = pz ? n3.y : n4.w, fz0 = pz ? n4.z : n3.x, fz1 = pz ? n4.w : n3.y;
  // + 0.0f turns a -0 into +0: the sign test below reads tmax - tmin, which
  // must not be -0 for the equal interval [+0, +0]
  const float tfar_c = fmaxf(tfar, 0.0f) + 0.0f;
  // the per-child work is only the slab test; the masks are built once per
  // node (ALU is the kernel's busiest pipe: this form measured 6-8 % faster
  // than testing validity and expanding leaves per child).  A child is missed
  // when tmax - tmin is negative: its sign bit is shifted into miss8 by one
  // funnel shift (children 7..0, so child s lands in bit s); an overflowed
  // plane pair (inf - inf = NaN, positive) counts as a hit, as tmin <= tmax did.
  // The six plane FMAs of a child run as three packed f32x2 FMAs (x and y near
  // planes, x and y far planes, z near and far), each half rounded exactly as
  // the scalar FMA (1.2 % faster than six scalar FMAs).
  const float2 b_xy = make_float2(bx, by), an_xy = make_float2(anx, any_), af_xy = make_float2(afx, afy);
  const float2 b_zz = make_float2(bz, bz), a_z = make_float2(anz, afz);
  uint32_t miss8 = 0;
#pragma unroll
  for (int s = 7; s >= 0; s--) {
    const uint32_t k = s & 3;
    const float2 tn = __ffma2_rn(make_float2(ubyte_f(s < 4 ? nx0 : nx1, k), ubyte_f(s < 4 ? ny0 : ny1, k)), b_xy, an_xy);
    const float2 tf = __ffma2_rn(make_float2(ubyte_f(s < 4 ? fx0 : fx1, k), ubyte_f(s < 4 ? fy0 : fy1, k)), b_xy, af_xy);
    const float2 tz = __ffma2_rn(make_float2(ubyte_f(s < 4 ? nz0 : nz1, k), ubyte_f(s < 4 ? fz0 : fz1, k)), b_zz, a_z);
    const float tmin = fmax3(tn.x, tn.y, fmaxf(tz.x, r.tnear_c));
    const float tmax = fmin3(tf.x, tf.y, fminf(tz.y, tfar_c));
    miss8 = __funnelshift_l(__float_as_uint(__fsub_rn(tmax, tmin)), miss8, 1);
  }
  // Empty slots hold inverted boxes (lower planes 255, upper planes 0), so they
  // miss without a validity mask (dropping the per-node gather of the meta
  // bytes' valid bits measured 1.6 % faster on the 4M soup, 2 % on the
  // heightfield).  Where overflowed planes make an empty slot count as hit, it
  // is a leaf slot (its imask bit is clear) whose meta byte lacks bit 7, and
  // it adds no triangles.
  const uint32_t hit8 = ~miss8 & 0xFFu;
  // internal children: bit 31 - j of the group is slot j ^ oct (near to far),
  // one lookup in the octant's row of the permutation table
  const uint32_t inner = perm[hit8 & imask];
  leaf = hit8 & ~imask & 0xFFu;
  meta = make_uint2(n1.z, n1.w);
  g_base = n1.x;
  g_bits = (inner << 24) | imask | row;
  t_base = n1.y;
}

// Meta byte of slot s (0..7): triangle offset in bits 0..4, triangle count - 1
// in bits 5..6, bit 7 clear for an empty slot.
__device__ __forceinline__ uint32_t meta_of(const uint2 meta, const uint32_t s) {
  return __byte_perm(meta.x, meta.y, s) & 0xFFu;
}

struct Ctx {
  const WideNode* __restrict__ nodes;
  const TriRecord* __restrict__ tris;
  unsigned int* err;
  uint32_t max_iters;
  uint32_t num_nodes;
  uint32_t num_tris;
};

// A refill runs with the idle lanes alone, so it weighs more the fewer nodes a ray
// visits: where the rays that a warp last ended visited fewer than kShortVisits nodes
// each, it waits for kShortRefill times the idle lanes of the launch shape.  Kernel
// time without / with: 1M primary rays on the 131k heightfield (3.5 nodes a ray)
// 92.8 / 84.6 us, 1M rays in a robust scene (3.2) 181 / 171 us, 14.6M batched rays
// (8) 2.08 / 1.92 ms, 16M rays on the 4M soup (34) 9.32 / 9.25 ms; waiting for three
// times the lanes always costs the soup's shadow rays 9 %.  Twice 91 and 174 us, four
// times 88 and 166 us but 1 % on the batched rays.  Scenes with instances, whose rays
// that miss all instances are short, lose 1.5 % and do without.
constexpr uint32_t kShortVisits = 12;
constexpr int kShortRefill = 3;

// Leaves wait for their triangle tests in a ring per warp (k_trace below): up
// to 31 waiting + 32 new.
constexpr int kQueue = 64;

constexpr uint32_t kTriGroup = 0x80000000u;  // stack entry flag: triangle group

template <bool ALIGNED>
__device__ __forceinline__ void load_ray(const char* p, TRay& r, float& tfar) {
  if (ALIGNED) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    const float4 b = *reinterpret_cast<const float4*>(p + 16);
    tfar = *reinterpret_cast<const float*>(p + 32);
    r.org = make_float3(a.x, a.y, a.z);
    r.tnear = a.w;
    r.dir = make_float3(b.x, b.y, b.z);
  } else {
    const float* f = reinterpret_cast<const float*>(p);
    r.org = make_float3(f[0], f[1], f[2]);
    r.tnear = f[3];
    r.dir = make_float3(f[4], f[5], f[6]);
    tfar = f[8];
  }
}

// Persistent traversal.  Every lane owns one ray at a time; a warp refills
// its idle lanes with one atomic once SH::kRefillIdle of them are idle (three times
// as many where rays are short).  Each
// loop iteration an active lane (1) visits one node of its current group,
// (2) queues the triangles of the leaves it hit, and (3) pops the stack when
// its group is exhausted.
//
// Triangle tests are not done by the lane that found the leaf: a node visit
// yields a triangle on only a few lanes of a warp (4 tests per 37 node visits
// on an incoherent soup), so testing them in place ran the test with 2-3 of 32
// lanes.  Instead the warp's lanes append (triangle, owner lane) to a ring in
// shared memory, and a batch of up to 32 entries is tested by all lanes at
// once, each reading its entry's ray from the owner lane by shuffles.  A ray's
// entries are tested in the order in which it found them, and two hits of one
// ray in a batch are committed in that order, the later one checked again
// against the lowered tfar, so the accepted hit is the one that testing in
// place accepts, except among triangles whose distances differ by no more than
// their rounding: there a triangle can be accepted whose box testing in place had
// culled by then, and of a leaf of several triangles a later one is tested against
// the distance of the first, also where that one then loses to an earlier entry.
// Between finding a triangle and its batch a ray visits nodes with an older,
// larger tfar: 1.5 % more visits on the soup, none fewer.  A lane whose traversal is over waits for its last entry's batch before
// it takes another ray.  The finished rays' results are written when the warp
// refills (several lanes at a time), from the per-lane result words in shared
// memory.  The ray's octant travels in the node group (bits 8..10), its direction
// and tnear in shared memory: 56 registers hold the rest without spills (16 bytes
// of spills cost 10 % on the soup).
// Measured on a GB300 (whole calls, in place -> batched): 16M closest-hit rays on
// the 4M soup 12.02 -> 11.54 ms, 16M shadow rays 7.73 -> 7.26 ms, 1M primary rays
// on the 131k heightfield 161 -> 153 us, 1M rays in a robust scene 253 -> 242 us.
//
// SEEDED: the ray's stack starts as [root, seed3, seed2, seed1] with seed0 as
// the current group, so the proposed subtrees are searched first and the whole
// tree afterwards.  The answer is the plain traversal's: an any-hit ray that
// hits inside a proposed subtree is occluded in the whole tree, and a closest
// hit found there only lowers tfar before the full search, which still tests
// every triangle whose distance can be the minimum.  `seeding` stays set until
// the root group is popped; a ray whose final hit was found while it was set
// counts as a proposal hit.
//
// INST: the scene holds instance leaves (kInstanceLeaf records).  Reaching one,
// the lane pushes the rest of its triangle group and a marker, switches to the
// instanced scene's BVH and transforms its ray into the instance's space the
// way the reference does (kernels/geometry/instance_intersector.cpp:56-69,
// xfmPoint / xfmVector of common/math/affinespace.h:102-103).  The ray
// parameter t is the same in both spaces (affine map, direction not
// renormalised), so tfar carries over.  Popping the marker reloads the world
// ray from its record.  Instances inside instances are skipped (one instance
// level, RTC_MAX_INSTANCE_LEVEL_COUNT = 1).
constexpr uint32_t kInstMarker = 0xFFFFFFFFu;  // stack entry (kInstMarker, 0)

__device__ __forceinline__ void to_instance(const float* __restrict__ m, TRay& r) {
  const float3 o = r.org, d = r.dir;
  r.org = make_float3(__fmaf_rn(o.x, m[0], __fmaf_rn(o.y, m[3], __fmaf_rn(o.z, m[6], m[9]))),
                      __fmaf_rn(o.x, m[1], __fmaf_rn(o.y, m[4], __fmaf_rn(o.z, m[7], m[10]))),
                      __fmaf_rn(o.x, m[2], __fmaf_rn(o.y, m[5], __fmaf_rn(o.z, m[8], m[11]))));
  r.dir = make_float3(__fmaf_rn(d.x, m[0], __fmaf_rn(d.y, m[3], __fmul_rn(d.z, m[6]))),
                      __fmaf_rn(d.x, m[1], __fmaf_rn(d.y, m[4], __fmul_rn(d.z, m[7]))),
                      __fmaf_rn(d.x, m[2], __fmaf_rn(d.y, m[5], __fmul_rn(d.z, m[8]))));
}

// Launch shape (SH, one of kTraceShapes): threads per CTA, the resident CTAs
// per SM whose register budget the plain variants are compiled for (9 x 128
// threads: at most 56 registers a thread, which they meet without spills),
// traversal stack entries kept in shared memory, and the number of idle lanes at
// which a warp fetches new rays.  The variants that would spill 20-50 bytes under
// that budget (proposals, instances, exclusion lists, closest hit in robust
// scenes) are compiled for 1,024 resident threads, 64 registers, at most: with
// the 100 registers they take unbounded, 4 CTAs fit an SM (1M primary rays on 125
// instances: 1005 us so, 861 us with 64 registers and batched writes).
template <int THREADS, int CTAS, int SHARED_STACK, int REFILL>
struct Shape {
  static constexpr int kThreads = THREADS, kCtas = CTAS, kSharedStack = SHARED_STACK, kRefillIdle = REFILL;
  static_assert(SHARED_STACK >= 1 && SHARED_STACK <= kStackSize, "shared stack entries");
  static_assert(THREADS % 32 == 0 && REFILL >= 1 && REFILL <= 32, "launch shape");
};
using DefaultShape = Shape<kTraceShapes[0].threads, kTraceShapes[0].ctas, kTraceShapes[0].shared_stack,
                           kTraceShapes[0].refill>;

template <bool ANYHIT, bool COUNT, bool ROBUST, bool SEEDED, bool INST, bool EXCL, class SH>
constexpr int min_ctas() {
  if (COUNT) return 1;
  const bool wide = SEEDED || INST || EXCL || (ROBUST && !ANYHIT);
  return wide && SH::kCtas * SH::kThreads > 1024 ? 1024 / SH::kThreads : SH::kCtas;
}

template <bool ANYHIT, bool COUNT, bool ALIGNED, bool ROBUST, bool SEEDED, bool INST = false, bool EXCL = false,
          class SH = DefaultShape>
__global__ void __launch_bounds__(SH::kThreads, min_ctas<ANYHIT, COUNT, ROBUST, SEEDED, INST, EXCL, SH>())
    k_trace(TraceParams P) {
  constexpr int kSharedStack = SH::kSharedStack;
  constexpr int kWarps = SH::kThreads / 32;
  Ctx c{P.nodes, P.tris, P.err, P.max_iters, P.num_nodes, P.num_tris};
  uint32_t cur_inst = kInvalidID, hit_inst = kInvalidID;  // INST: instance being traversed / of the hit
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t nrays = P.nrays_ptr ? *P.nrays_ptr : P.nrays;
  // stack of node groups (and, in scenes with instances, triangle groups): the
  // first kSharedStack entries live in shared memory ([entry][thread]: a warp's
  // accesses are conflict-free), the deeper ones in local memory.  16M closest-hit
  // rays on the 4M soup with 8 entries 9.27 ms, with 4 9.85, with 12 9.37, with 16
  // 17.6 (the results and the ring take shared memory too: 28 KB of L1 are left).
  uint2 stack[kStackSize];
  int sp = 0;
  __shared__ uint2 s_stack[kSharedStack][SH::kThreads];
  // per lane: distance, u, v and triangle of its ray's nearest hit so far
  // (any hit: the distance becomes -inf at a hit); SEEDED: the triangle of the
  // last hit found in a proposed subtree (any hit: 0 once there is one)
  __shared__ float s_t[SH::kThreads], s_u[ANYHIT ? 1 : SH::kThreads], s_v[ANYHIT ? 1 : SH::kThreads];
  __shared__ uint32_t s_tri[SH::kThreads], s_seed[SEEDED ? SH::kThreads : 1];
  // per lane: ray direction and tnear, which only triangle tests read
  __shared__ float4 s_dir[INST ? 1 : SH::kThreads];
  // per warp: ring of leaves to test, as (first triangle, owner lane | bits 5..7
  // of the leaf's meta byte | bit 8: found while seeding)
  __shared__ uint2 s_queue[INST ? 1 : kWarps][kQueue];
  // slot permutation by octant: s_perm[o][m] has bit 7 - j set when m has bit
  // j ^ o (one shared-memory byte load per node instead of a three-stage swap
  // network: 1.4 % faster; the reversed order lets one count of leading zeros
  // find the next child: 0.5 %)
  alignas(4) __shared__ uint8_t s_perm[8][256];
  // four entries at a time (one by one, the filling took 1.5 us of a 1,000-ray query's 28)
  for (int i = threadIdx.x; i < 8 * 64; i += SH::kThreads) {
    const uint32_t o = i >> 6;
    // bit j ^ o of the slot mask moves to bit j: swaps of 1, 2 and 4 bits of each byte
    uint32_t v = 0x03020100u + 0x04040404u * (i & 63u);
    if (o & 1u) v = ((v & 0x55555555u) << 1) | ((v >> 1) & 0x55555555u);
    if (o & 2u) v = ((v & 0x33333333u) << 2) | ((v >> 2) & 0x33333333u);
    if (o & 4u) v = ((v & 0x0F0F0F0Fu) << 4) | ((v >> 4) & 0x0F0F0F0Fu);
    reinterpret_cast<uint32_t*>(s_perm)[i] = __byte_perm(__brev(v), 0u, 0x0123u);
  }
  s_tri[threadIdx.x] = kInvalidID;  // no result to write yet
  __shared__ uint32_t s_batch[kWarps];  // batched queries: a batch that a ray of this warp was in
  if (lane == 0) s_batch[warp] = 0;
  __syncthreads();
  const int stk_tid = threadIdx.x, w0 = threadIdx.x & ~31;
  auto push = [&](uint2 e) {
    if (sp < kSharedStack) s_stack[sp][stk_tid] = e; else stack[sp] = e;
    sp++;
  };
  auto pop = [&]() -> uint2 {
    --sp;
    return sp < kSharedStack ? s_stack[sp][stk_tid] : stack[sp];
  };
  // idle lanes to wait for before a refill; 33: no ray is left (one register for both:
  // two spill; INST, which waits for the same number always, is 2.7 % faster with the flag)
  int wait = SH::kRefillIdle;
  bool active = false, exhausted = false, seeding = false;
  uint32_t rid = 0;
  TRay r;
  r.org = r.dir = r.rdir = make_float3(0.f, 0.f, 0.f);
  r.tnear = r.tnear_c = 0.f;
  r.oct = 0;
  float t_best = 0.f;
  uint32_t g_base = 0, g_bits = 0, iters = 0;
  uint32_t ex_lo = 0, ex_hi = 0;  // EXCL: this ray's range of excluded triangles
  uint32_t qhead = 0, qtail = 0;  // ring positions (uniform in the warp): tested up to qhead, queued up to qtail
  unsigned long long n_nodes = 0, n_tris = 0, n_rays = 0, n_prop = 0;

  // one ray against triangle ti (record a, b, d); true when it is hit in range.
  // Moeller: (A, B, C, D) = (U, V, T, |den|); Pluecker: (U, V, UVW, t).
  auto test = [&](const float4 a, const float4 b, const float4 d, const float3 org, const float3 dir,
                  const float tnear, const float tfar, float& A, float& B, float& C, float& D) -> bool {
    const float3 p = make_float3(a.x, a.y, a.z), q = make_float3(b.x, b.y, b.z), s = make_float3(d.x, d.y, d.z);
    return ROBUST ? pluecker(p, q, s, org, dir, tnear, tfar, A, B, C, D)
                  : moeller(p, q, s, org, dir, tnear, tfar, A, B, C, D);
  };
  // records a hit of the ray of the thread `o` of this CTA
  auto commit = [&](const int o, const uint32_t ti, const float A, const float B, const float C, const float D) {
    if (ANYHIT) {
      s_t[o] = -INFINITY;
      s_tri[o] = ti;
      return;
    }
    if (ROBUST) {
      // PlueckerHitM::finalize: u,v = U,V * rcp(UVW), 0 when |UVW| < 1e-18
      const float rcp = fabsf(C) < kMinRcpInput ? 0.0f : __frcp_rn(C);
      s_t[o] = D;
      s_u[o] = __fmul_rn(A, rcp);
      s_v[o] = __fmul_rn(B, rcp);
    } else {
      const float rcp = __frcp_rn(D);
      s_t[o] = __fmul_rn(C, rcp);
      s_u[o] = __fmul_rn(A, rcp);
      s_v[o] = __fmul_rn(B, rcp);
    }
    s_tri[o] = ti;
  };
  // tests the first 32 (or all) entries of the ring; the whole warp calls it.
  // A lane tests its entry's triangles in order against the entry's own running
  // distance; the nearest of them is then committed in queue order.
  auto flush = [&]() {
    __syncwarp();
    const uint32_t n = min(qtail - qhead, 32u);
    uint2 e = make_uint2(0u, (uint32_t)lane);
    if ((uint32_t)lane < n) e = s_queue[warp][(qhead + lane) & (kQueue - 1)];
    // the meta byte of an empty slot (bit 7 clear) holds no triangle: overflowed
    // planes can make one count as hit
    const bool have = (e.y & 128u) != 0u;
    const int own = (int)(e.y & 31u);
    const float3 org = make_float3(__shfl_sync(0xFFFFFFFFu, r.org.x, own), __shfl_sync(0xFFFFFFFFu, r.org.y, own),
                                   __shfl_sync(0xFFFFFFFFu, r.org.z, own));
    float tfar = __shfl_sync(0xFFFFFFFFu, t_best, own);
    uint32_t xl = 0, xh = 0;
    if (EXCL) {
      xl = __shfl_sync(0xFFFFFFFFu, ex_lo, own);
      xh = __shfl_sync(0xFFFFFFFFu, ex_hi, own);
    }
    bool hit = false;
    uint32_t hit_ti = 0;
    float A = 0.f, B = 0.f, C = 0.f, D = 0.f;
    if (have) {
      const float4 dn = s_dir[w0 + own];
      const uint32_t end = e.x + ((e.y >> 5) & 3u);
      if (end >= c.num_tris) {
        atomicOr(c.err, kErrBuild);
      } else {
        for (uint32_t ti = e.x;; ti++) {
          const float4* tp = reinterpret_cast<const float4*>(c.tris + ti);
          const float4 a = __ldg(tp + 0), b = __ldg(tp + 1), d = __ldg(tp + 2);
          bool skip = false;
          if (EXCL) {  // a triangle whose hit a filter callback rejected
            for (uint32_t x = xl; x < xh && !skip; x++) {
              const uint2 y = __ldg(P.excl + x);
              skip = y.x == __float_as_uint(a.w) && y.y == __float_as_uint(b.w);
            }
          }
          if (!skip) {
            if (COUNT) n_tris++;
            float A1, B1, C1, D1;
            if (test(a, b, d, org, make_float3(dn.x, dn.y, dn.z), dn.w, tfar, A1, B1, C1, D1)) {
              hit = true;
              hit_ti = ti;
              A = A1; B = B1; C = C1; D = D1;
              if (ANYHIT) break;
              if (ti != end) tfar = ROBUST ? D : __fmul_rn(C, __frcp_rn(D));
            }
          }
          if (ti == end) break;
        }
      }
    }
    if (ANYHIT) {
      // Lanes with hits of one ray write in no order.  All of a ray's proposed subtrees
      // come before the rest, so its first hit is a proposal's if any of them is: a word
      // for that, which all its writers set alike, counts as testing in place would.
      if (hit) {
        commit(w0 + own, hit_ti, A, B, C, D);
        if (SEEDED && (e.y & 256u)) s_seed[w0 + own] = 0u;
      }
      __syncwarp();
    } else {
      // a ray's hits are committed in queue order, each tested again against the
      // distance that the ones before it left
      uint32_t pend = __ballot_sync(0xFFFFFFFFu, hit);
      while (pend) {
        if (hit && lane == __ffs(__match_any_sync(pend, own)) - 1) {
          commit(w0 + own, hit_ti, A, B, C, D);
          if (SEEDED && (e.y & 256u)) s_seed[w0 + own] = hit_ti;
          hit = false;
        }
        __syncwarp();
        if (hit) {
          const float tf = s_t[w0 + own];
          hit = ROBUST ? D <= tf : C <= __fmul_rn(D, tf);
        }
        pend = __ballot_sync(0xFFFFFFFFu, hit);
      }
    }
    qhead += n;
    t_best = s_t[threadIdx.x];
    if (ANYHIT && t_best == -INFINITY) {  // occluded: nothing left to search
      active = false;
      g_bits = 0;
    }
    __syncwarp();
  };
  for (;;) {
    // ---- write finished rays, refill idle lanes
    uint32_t idle = __ballot_sync(0xFFFFFFFFu, !active);
    const bool refill = idle == 0xFFFFFFFFu || (INST ? !exhausted && __popc(idle) >= SH::kRefillIdle : __popc(idle) >= wait);
    // waiting leaves (at most 31: one batch empties the ring) are tested before a
    // refill and once there is one per active lane
    if (!INST && qtail != qhead && (refill || qtail - qhead + __popc(idle) >= 32u)) {
      flush();
      if (ANYHIT) idle = __ballot_sync(0xFFFFFFFFu, !active);
    }
    if (refill) {
      if (!active) {
        const uint32_t hit_tri = s_tri[threadIdx.x];
        if (hit_tri != kInvalidID) {
          s_tri[threadIdx.x] = kInvalidID;
          if (SEEDED && (ANYHIT ? s_seed[threadIdx.x] == 0u : hit_tri == s_seed[threadIdx.x])) n_prop++;
          char* rec = P.rays + (uint64_t)rid * P.stride;
          if (ANYHIT) {
            *reinterpret_cast<float*>(rec + 32) = -INFINITY;
          } else {
            const TriRecord* htris = (INST && hit_inst != kInvalidID) ? P.insts[hit_inst].tris : P.tris;
            const uint32_t inst_id = (INST && hit_inst != kInvalidID) ? P.insts[hit_inst].geomID : kInvalidID;
            const float4* tp = reinterpret_cast<const float4*>(htris + hit_tri);
            const float4 a = __ldg(tp + 0), b = __ldg(tp + 1), d = __ldg(tp + 2);
            const float3 Ng = ROBUST ? pluecker_normal(make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z),
                                                       make_float3(d.x, d.y, d.z), r.org)
                                     : cross3(make_float3(d.x, d.y, d.z), make_float3(b.x, b.y, b.z));
            const float hu = s_u[threadIdx.x], hv = s_v[threadIdx.x];
            *reinterpret_cast<float*>(rec + 32) = s_t[threadIdx.x];
            if (ALIGNED) {
              *reinterpret_cast<float4*>(rec + 48) = make_float4(Ng.x, Ng.y, Ng.z, hu);
              *reinterpret_cast<uint4*>(rec + 64) =
                  make_uint4(__float_as_uint(hv), __float_as_uint(a.w), __float_as_uint(b.w), inst_id);
            } else {
              float* f = reinterpret_cast<float*>(rec + 48);
              f[0] = Ng.x; f[1] = Ng.y; f[2] = Ng.z; f[3] = hu; f[4] = hv;
              uint32_t* w = reinterpret_cast<uint32_t*>(rec + 68);
              w[0] = __float_as_uint(a.w); w[1] = __float_as_uint(b.w); w[2] = inst_id;
            }
          }
        }
      }
      if (INST ? exhausted : wait > 32) break;  // no ray left, no lane active
      const uint32_t visits = INST ? 0u : __reduce_add_sync(0xFFFFFFFFu, active ? 0u : iters);  // of the rays that ended
      wait = !INST && visits < kShortVisits * __popc(idle) ? min(SH::kRefillIdle * kShortRefill, 32) : SH::kRefillIdle;
      const int leader = __ffs(idle) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(P.ray_counter, (unsigned)__popc(idle));
      base = __shfl_sync(0xFFFFFFFFu, base, leader);
      if (base + __popc(idle) >= nrays) {
        if (INST) exhausted = true;
        else wait = 33;
      }
      if (!active) {
        rid = base + __popc(idle & lt_mask);
        if (rid < nrays) {
          if (P.order) rid = __ldg(P.order + rid);  // the record this fetch slot traces
          if (EXCL) {
            ex_lo = __ldg(P.excl_off + rid);
            ex_hi = __ldg(P.excl_off + rid + 1);
          }
          float tfar;
          load_ray<ALIGNED>(P.rays + (uint64_t)rid * P.stride, r, tfar);
          // stream semantics: only tnear <= tfar rays are traced; any-hit also
          // skips already occluded rays (bvh_intersector_stream_filters.cpp:75)
          const bool valid = ANYHIT ? ((r.tnear <= tfar) && !(tfar < 0.0f)) : (r.tnear <= tfar);
          // batched queries: the ray's batch (binary search) gives its tree's root
          uint32_t root = 0;
          if (P.batch_root) {
            // rays are fetched in order: most are in the batch of the last one
            uint32_t lo = s_batch[warp], hi = P.nbatches;
            if (__ldg(P.batch_start + lo) > rid) lo = 0;
            else if (__ldg(P.batch_start + lo + 1) > rid) hi = lo + 1;
            while (hi - lo > 1) {
              const uint32_t mid = (lo + hi) >> 1;
              if (__ldg(P.batch_start + mid) <= rid) lo = mid; else hi = mid;
            }
            s_batch[warp] = lo;
            root = __ldg(P.batch_root + lo);
          }
          if (INST) {  // a ray that ended inside an instance left the lane in its space
            c.nodes = P.nodes;
            c.tris = P.tris;
            c.num_nodes = P.num_nodes;
            c.num_tris = P.num_tris;
            cur_inst = kInvalidID;
            hit_inst = kInvalidID;
          }
          if (valid && root < c.num_nodes) {
            init_ray(r);
            if (!INST) s_dir[threadIdx.x] = make_float4(r.dir.x, r.dir.y, r.dir.z, r.tnear);
            t_best = tfar;
            s_t[threadIdx.x] = tfar;
            s_tri[threadIdx.x] = kInvalidID;
            g_base = root;
            g_bits = (0x80000000u >> r.oct) | (r.oct << 8) | 1u;  // virtual group: the root as internal slot 0
            sp = 0;
            iters = 0;
            active = true;
            if (SEEDED) {
              // a virtual group (n, root bits) visits node n alone
              const uint4 s4 = P.seeds[rid];
              const uint32_t sd[4] = {s4.x, s4.y, s4.z, s4.w};
              push(make_uint2(g_base, g_bits));
              s_seed[threadIdx.x] = kInvalidID;
              seeding = false;
              for (int q = 3; q >= 0; q--) {
                if (sd[q] == 0u || sd[q] >= c.num_nodes) continue;
                if (seeding) push(make_uint2(g_base, g_bits));
                g_base = sd[q];
                seeding = true;
              }
              if (!seeding) sp = 0;  // no proposal: plain traversal from the root
            }
            if (COUNT) n_rays++;
          }
        }
      }
    }
    // ---- (1) one node of the current group
    uint32_t leaf = 0, t_base = 0;
    uint2 meta = make_uint2(0u, 0u);
    if (active && (g_bits & 0xFF000000u) && !(INST && (g_base & kTriGroup))) {
      const uint32_t k = __clz(g_bits);  // visiting position of the next child (bit 31 - k)
      g_bits &= ~(0x80000000u >> k);
      const uint32_t row = g_bits & 0x700u;  // the ray's octant << 8
      const uint32_t slot = k ^ (row >> 8);
      const uint32_t child = g_base + __popc(g_bits & ((1u << slot) - 1u) & 0xFFu);
      const bool rest = (g_bits & 0xFF000000u) != 0u, room = !rest || sp < kStackSize;
      if (room && child < c.num_nodes && ++iters <= c.max_iters) {
        if (rest) push(make_uint2(g_base, g_bits));
        if (COUNT) n_nodes++;
        intersect_node(c.nodes + child, r, t_best, g_base, g_bits, t_base, leaf, meta, &s_perm[0][0] + row, row);
      } else {
        atomicOr(c.err, !room ? kErrStackOverflow : child >= c.num_nodes ? kErrBuild : kErrIterationLimit);
        active = false;
        g_bits = 0;
      }
    }
    if constexpr (!INST) {
      // ---- (2) queue the leaves that were hit; a full batch is tested
      for (uint32_t bal; (bal = __ballot_sync(0xFFFFFFFFu, leaf != 0u)) != 0u;) {
        if (leaf) {
          const uint32_t m = meta_of(meta, __ffs(leaf) - 1);
          leaf &= leaf - 1u;
          const uint32_t at = (qtail + __popc(bal & lt_mask)) & (kQueue - 1);
          s_queue[warp][at] = make_uint2(t_base + (m & 31u), (uint32_t)lane | (m & 0xE0u) | (SEEDED && seeding ? 256u : 0u));
        }
        qtail += __popc(bal);
        if (qtail - qhead >= 32u) {
          flush();
          if (ANYHIT && !active) leaf = 0;
        }
      }
    } else {
      // ---- (2) scenes with instances: each lane tests its own triangles, since
      // entering an instance changes the lane's ray and BVH.  A leaf group that an
      // instance interrupted comes back from the stack as the current group (kTriGroup
      // in g_base) and is tested in the next turn, beside the other lanes' nodes: with
      // a loop here that took it from the stack and tested it at once, the warp waited
      // for its slowest lane (kernel, 30k / 100k / 300k / 1M rays on 125 instances 107 /
      // 121 / 364 / 725 us so, 87 / 102 / 321 / 670 now).
      uint32_t t_bits = 0;
      if (active && (g_base & kTriGroup)) {  // the rest of a leaf group, from the stack
        t_base = g_base & ~kTriGroup;
        t_bits = g_bits;
        g_base = g_bits = 0;
      }
      while (leaf) {  // the triangle bits of the leaves that were hit
        const uint32_t m = meta_of(meta, __ffs(leaf) - 1);
        leaf &= leaf - 1u;
        if (m & 0x80u) t_bits |= ((2u << ((m >> 5) & 3u)) - 1u) << (m & 31u);
      }
      while (active && t_bits) {
        const uint32_t idx = __ffs(t_bits) - 1;
        t_bits &= t_bits - 1;
        const uint32_t ti = t_base + idx;
        if (ti >= c.num_tris) { atomicOr(c.err, kErrBuild); active = false; break; }
        const float4* tp = reinterpret_cast<const float4*>(c.tris + ti);
        const float4 a = __ldg(tp + 0), b = __ldg(tp + 1), d = __ldg(tp + 2);
        if (__float_as_uint(d.w) == kInstanceLeaf) {
          const uint32_t ii = __float_as_uint(a.w);
          if (cur_inst != kInvalidID) continue;  // nested instance: not traversed
          if (ii >= P.ninsts) { atomicOr(c.err, kErrBuild); active = false; break; }
          const InstDesc* in = P.insts + ii;
          const uint32_t bn = in->num_nodes;
          if (bn == 0) continue;  // empty instanced scene
          if (sp + 3 > kStackSize) { atomicOr(c.err, kErrStackOverflow); active = false; break; }
          // the node group of this visit (its hit internal children) and the rest of this
          // leaf group resume after the instance
          if (g_bits & 0xFF000000u) push(make_uint2(g_base, g_bits));
          if (t_bits) push(make_uint2(t_base | kTriGroup, t_bits));
          push(make_uint2(kInstMarker, 0u));
          t_bits = 0;
          cur_inst = ii;
          c.nodes = in->nodes;
          c.tris = in->tris;
          c.num_nodes = bn;
          c.num_tris = in->num_tris;
          to_instance(in->w2l, r);
          init_ray(r);
          g_base = 0;
          g_bits = (0x80000000u >> r.oct) | (r.oct << 8) | 1u;
          break;
        }
        if (COUNT) n_tris++;
        float A, B, C, D;
        if (test(a, b, d, r.org, r.dir, r.tnear, t_best, A, B, C, D)) {
          commit(threadIdx.x, ti, A, B, C, D);
          t_best = s_t[threadIdx.x];
          hit_inst = cur_inst;
          if (ANYHIT) {
            t_bits = 0;
            g_bits = 0;
            sp = 0;
            break;
          }
        }
      }
    }
    // ---- (3) next group from the stack, or finish
    if (active && !(g_bits & 0xFF000000u)) {
      if (sp > 0) {
        uint2 e = pop();
        if (INST && e.x == kInstMarker && e.y == 0u) {
          // leaving the instance: world ray and top-level BVH again
          float unused_tfar;
          load_ray<ALIGNED>(P.rays + (uint64_t)rid * P.stride, r, unused_tfar);
          init_ray(r);
          c.nodes = P.nodes;
          c.tris = P.tris;
          c.num_nodes = P.num_nodes;
          c.num_tris = P.num_tris;
          cur_inst = kInvalidID;
          if (sp > 0) {
            e = pop();
          } else {
            e = make_uint2(0u, 0u);
            active = false;
          }
        }
        g_base = e.x;
        g_bits = e.y;
        if (SEEDED && sp == 0) seeding = false;  // the root group: proposals are done
      } else {
        active = false;
      }
    }
  }
  if (SEEDED) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_prop += __shfl_xor_sync(0xFFFFFFFFu, n_prop, o);
    if (lane == 0 && n_prop) atomicAdd(&P.counters->proposal_hits, n_prop);
  }
  if (COUNT) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      n_nodes += __shfl_xor_sync(0xFFFFFFFFu, n_nodes, o);
      n_tris += __shfl_xor_sync(0xFFFFFFFFu, n_tris, o);
      n_rays += __shfl_xor_sync(0xFFFFFFFFu, n_rays, o);
    }
    if (lane == 0) {
      atomicAdd(&P.counters->nodes, n_nodes);
      atomicAdd(&P.counters->tris, n_tris);
      atomicAdd(&P.counters->rays, n_rays);
    }
  }
  // The CTA that ends last reports the state and zeroes it.  A CTA's ticket releases what
  // its threads added to the state; only the last one acquires, and its lanes take one
  // word each.  (Two full fences in every CTA and ten exchanges one after the other made
  // queries of 20k to 300k rays 3 to 9 us longer: 150k shadow rays on a 36k / 300k soup
  // 80 / 195 us of kernel time so, 75 / 188 now.)
  if (P.done) {
    __syncthreads();
    if (warp == 0) {
      uint32_t last = 0;
      if (lane == 0) {
        uint32_t ticket;
        asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(P.done) : "memory");
        last = ticket == gridDim.x - 1 ? 1u : 0u;
        if (last) __threadfence();
      }
      if (__shfl_sync(0xFFFFFFFFu, last, 0)) {
        __syncwarp();
        if (lane < kStateWords) P.host_state[lane] = atomicExch(P.ray_counter + lane, 0u);
        if (lane == 0) *P.done = 0u;
      }
    }
  }
}


// One launch of k_trace in shape SH: a persistent grid of (SMs x resident CTAs)
// blocks, or fewer when the rays do not fill it.  The occupancy is looked up
// once per instantiation.
template <bool ANYHIT, bool COUNT, bool ALIGNED, bool ROBUST, bool SEEDED, bool INST, bool EXCL, class SH>
static cudaError_t launch_shaped(const TraceParams& P, cudaStream_t st) {
  static int blocks_per_sm = -1, num_sms = 0;
  if (blocks_per_sm < 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, k_trace<ANYHIT, COUNT, ALIGNED, ROBUST, SEEDED, INST, EXCL, SH>,
                                                  SH::kThreads, 0);
    if (blocks_per_sm < 1) blocks_per_sm = 1;
  }
  uint64_t want = ((uint64_t)P.nrays + SH::kThreads - 1) / SH::kThreads;
  uint64_t grid = (uint64_t)num_sms * blocks_per_sm;
  if (want < grid) grid = want;
  if (grid < 1) grid = 1;
  k_trace<ANYHIT, COUNT, ALIGNED, ROBUST, SEEDED, INST, EXCL, SH><<<(unsigned)grid, SH::kThreads, 0, st>>>(P);
  return cudaGetLastError();
}

}  // namespace gb

// Device ray queries over the wide BVH (bvh_build.h): closest hit and any
// hit.  Shared by the ray-cast kernels and the path tracers.
//
// Replaces Bvh::traverse_elems (src/dort/bvh.cpp:418-469) with the callbacks
// of MeshBvhPrimitive::intersect / intersect_p (mesh_bvh_primitive.cpp:13-45)
// and the triangle tests TriangleUv::hit / Triangle::hit_p
// (triangle.cpp:14-46, 102-134).
//
// Traversal: node groups (base index, internal-slot mask << 8 | child-hit
// bits) on a per-thread stack; child slots are visited in an order fixed by
// the ray octant (slot bit index XOR octant), so no per-node sort is needed.
// Child boxes are tested with fused multiply-adds on the quantized planes.  The
// quantization's 1/32 step covers the rounding of the planes' decoding, a
// relative widening (DORT_SLAB_FAR_WIDEN) that of the distances, and a margin
// that grows with the distance from the ray's origin to the node
// (DORT_RAY_MARGIN) that of the triangle test.  That margin is wide enough for
// triangles of ordinary shape; a sliver's test may be off by more, so that a
// hit that it reports beside its box may be culled.
//
// Triangle test: the reference's Moller-Trumbore operations in the
// reference's order with explicit round-to-nearest intrinsics (no fused
// multiply-add, IEEE reciprocal), so (t, b1, b2) are bit-identical to the
// reference computed on the same triangle.
#pragma once
#include <cstdint>
#include <cstring>

#include "common.h"

// The traversal is compiled for the device and, with plain IEEE float
// arithmetic (no contraction), for the host, so that the host can check the
// tree and the traversal without a GPU.
#ifdef __CUDA_ARCH__
#define DG_MUL(a, b) __fmul_rn(a, b)
#define DG_ADD(a, b) __fadd_rn(a, b)
#define DG_SUB(a, b) __fsub_rn(a, b)
#define DG_RCP(a) __frcp_rn(a)
#define DG_POPC(x) __popc(x)
#define DG_LDG(p) __ldg(p)
#define DG_AS_FLOAT(u) __uint_as_float(u)
#define DG_AS_UINT(f) __float_as_uint(f)
#define DG_FMA(a, b, c) fmaf(a, b, c)
#define DG_RCP_FAST(a) __frcp_rn(a)
// three-input float max / min (one instruction on sm_100a; exact, like two
// fmaxf / fminf)
__device__ __forceinline__ float dg_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float dg_min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// reciprocal to one unit in the last place (the box test's, see
// DORT_SLAB_FAR_WIDEN)
__device__ __forceinline__ float dg_rcp_approx(float a) {
  float d;
  asm("rcp.approx.f32 %0, %1;" : "=f"(d) : "f"(a));
  return d;
}
#define DG_RCP_APPROX(a) dg_rcp_approx(a)
#define DG_MAX3(a, b, c) dg_max3(a, b, c)
#define DG_MIN3(a, b, c) dg_min3(a, b, c)
// the sign bit of `f` shifted into the low end of `m` (one funnel shift)
#define DG_PUSH_SIGN(m, f) __funnelshift_l(__float_as_uint(f), m, 1)
// byte j of `w` as the float 32768 + byte, `one` = the bits of 32768.f: one
// byte permutation.  (`one` comes from the node: as a constant the compiler
// moves it into a register before every one of a node's 48 permutations.)
#define DG_BYTE_FLOAT(w, one, j) \
  __uint_as_float(__byte_perm(w, one, 0x7404u | (uint32_t(j) << 4)))
// byte j of `w` as the float 65536 + byte: one dot product of bytes (128 steps
// of 2^-7 added to the bits of 65536.f), on another pipe than the permutations
#define DG_BYTE_FLOAT_DP(w, j) __uint_as_float(__dp4a(w, 0x80u << (8 * (j)), 0x47800000u))
#else
namespace dort_gpu {
inline float host_as_float(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
inline uint32_t host_as_uint(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
}
#define DG_MUL(a, b) ((a) * (b))
#define DG_ADD(a, b) ((a) + (b))
#define DG_SUB(a, b) ((a) - (b))
#define DG_RCP(a) (1.f / (a))
#define DG_POPC(x) __builtin_popcount(x)
#define DG_LDG(p) (*(p))
#define DG_AS_FLOAT(u) ::dort_gpu::host_as_float(u)
#define DG_AS_UINT(f) ::dort_gpu::host_as_uint(f)
#define DG_FMA(a, b, c) std::fma(a, b, c)
#define DG_RCP_FAST(a) (1.f / (a))
#define DG_RCP_APPROX(a) (1.f / (a))
#define DG_MAX3(a, b, c) fmaxf(fmaxf(a, b), c)
#define DG_MIN3(a, b, c) fminf(fminf(a, b), c)
#define DG_PUSH_SIGN(m, f) (((m) << 1) | (DG_AS_UINT(f) >> 31))
#define DG_BYTE_FLOAT(w, one, j) (32768.f + float(((w) >> (8 * (j))) & 0xffu))
#define DG_BYTE_FLOAT_DP(w, j) (65536.f + float(((w) >> (8 * (j))) & 0xffu))
#endif
#define DG_HD __host__ __device__ __forceinline__

namespace dort_gpu {

constexpr uint32_t kMiss = 0xffffffffu;
constexpr int kTraceStack = 64;   // == kMaxWideDepth (bvh_build.h)

struct Hit {
  float t, b1, b2;
  uint32_t prim;   // original triangle index, kMiss if none
};

DG_HD float dot_rn(float ax, float ay, float az,
                                        float bx, float by, float bz) {
  // (a.x*b.x + a.y*b.y) + a.z*b.z, each product and sum rounded separately
  return DG_ADD(DG_ADD(DG_MUL(ax, bx), DG_MUL(ay, by)), DG_MUL(az, bz));
}

// Moller-Trumbore as triangle.cpp:109-134 (also 18-42).
DG_HD bool mt_exact(float4 a, float4 e1, float4 e2,
                                         float ox, float oy, float oz,
                                         float dx, float dy, float dz,
                                         float t_min, float t_max,
                                         float& out_t, float& out_b1, float& out_b2) {
  // s1 = cross(dir, e2)
  float s1x = DG_SUB(DG_MUL(dy, e2.z), DG_MUL(dz, e2.y));
  float s1y = DG_SUB(DG_MUL(dz, e2.x), DG_MUL(dx, e2.z));
  float s1z = DG_SUB(DG_MUL(dx, e2.y), DG_MUL(dy, e2.x));
  float det = dot_rn(s1x, s1y, s1z, e1.x, e1.y, e1.z);
  if(det == 0.f) { return false; }
  float inv_det = DG_RCP(det);
  // s = orig - p0
  float sx = DG_SUB(ox, a.x), sy = DG_SUB(oy, a.y), sz = DG_SUB(oz, a.z);
  float b1 = DG_MUL(inv_det, dot_rn(s1x, s1y, s1z, sx, sy, sz));
  if(b1 < 0.f || b1 > 1.f) { return false; }
  // s2 = cross(s, e1)
  float s2x = DG_SUB(DG_MUL(sy, e1.z), DG_MUL(sz, e1.y));
  float s2y = DG_SUB(DG_MUL(sz, e1.x), DG_MUL(sx, e1.z));
  float s2z = DG_SUB(DG_MUL(sx, e1.y), DG_MUL(sy, e1.x));
  float b2 = DG_MUL(inv_det, dot_rn(s2x, s2y, s2z, dx, dy, dz));
  if(b2 < 0.f || DG_ADD(b1, b2) > 1.f) { return false; }
  float t = DG_MUL(inv_det, dot_rn(s2x, s2y, s2z, e2.x, e2.y, e2.z));
  if(t < t_min || t > t_max) { return false; }
  out_t = t;
  out_b1 = b1;
  out_b2 = b2;
  return true;
}

// Moller-Trumbore with fused multiply-adds, for the path tracers (which need
// the reference's estimator, not its rounding).
DG_HD bool mt_fast(float4 a, float4 e1, float4 e2, float ox, float oy, float oz,
                   float dx, float dy, float dz, float t_min, float t_max,
                   float& out_t, float& out_b1, float& out_b2) {
  float s1x = DG_FMA(dy, e2.z, -dz * e2.y);
  float s1y = DG_FMA(dz, e2.x, -dx * e2.z);
  float s1z = DG_FMA(dx, e2.y, -dy * e2.x);
  float det = DG_FMA(s1x, e1.x, DG_FMA(s1y, e1.y, s1z * e1.z));
  if(det == 0.f) { return false; }
  float inv_det = DG_RCP_FAST(det);
  float sx = ox - a.x, sy = oy - a.y, sz = oz - a.z;
  float b1 = inv_det * DG_FMA(s1x, sx, DG_FMA(s1y, sy, s1z * sz));
  if(b1 < 0.f || b1 > 1.f) { return false; }
  float s2x = DG_FMA(sy, e1.z, -sz * e1.y);
  float s2y = DG_FMA(sz, e1.x, -sx * e1.z);
  float s2z = DG_FMA(sx, e1.y, -sy * e1.x);
  float b2 = inv_det * DG_FMA(s2x, dx, DG_FMA(s2y, dy, s2z * dz));
  if(b2 < 0.f || b1 + b2 > 1.f) { return false; }
  float t = inv_det * DG_FMA(s2x, e2.x, DG_FMA(s2y, e2.y, s2z * e2.z));
  if(t < t_min || t > t_max) { return false; }
  out_t = t;
  out_b1 = b1;
  out_b2 = b2;
  return true;
}

// Watertight ray/triangle test: Woop, Benthin and Wald, "Watertight
// Ray/Triangle Intersection", JCGT 2(1), 2013.  The ray's dominant axis
// becomes z and a shear maps the ray onto the z axis; the triangle's edge
// functions U, V, W are then 2-D cross products of the sheared vertices.  An
// edge shared by two triangles gets the same operands in both, so its
// function is computed identically (exactly negated) in both and a ray can
// pass through neither: no leak at edges or vertices.  Products and
// differences are rounded separately (no contraction) so that the negation
// is exact; an edge function that comes out exactly zero is recomputed in
// double.  Barycentrics: b1 = V / det (weight of p1), b2 = W / det (p2).
struct WtRay {
  uint32_t kx, ky, kz;   // dominant axis kz; kx, ky keep the winding
  float sx, sy, sz;      // shear: d[kx] / d[kz], d[ky] / d[kz], 1 / d[kz]
};

DG_HD float wt_sel(float x, float y, float z, uint32_t k) {
  return k == 0 ? x : (k == 1 ? y : z);
}

DG_HD WtRay wt_setup(float dx, float dy, float dz) {
  WtRay r;
  float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
  r.kz = ax > ay ? (ax > az ? 0u : 2u) : (ay > az ? 1u : 2u);
  r.kx = r.kz == 2u ? 0u : r.kz + 1u;
  r.ky = r.kx == 2u ? 0u : r.kx + 1u;
  float dk = wt_sel(dx, dy, dz, r.kz);
  if(dk < 0.f) { uint32_t t = r.kx; r.kx = r.ky; r.ky = t; }
  r.sx = wt_sel(dx, dy, dz, r.kx) / dk;
  r.sy = wt_sel(dx, dy, dz, r.ky) / dk;
  r.sz = 1.f / dk;
  return r;
}

DG_HD bool wt_hit(const WtRay& r, float4 p0, float4 p1, float4 p2, float ox, float oy, float oz,
                  float t_min, float t_max, float& out_t, float& out_b1, float& out_b2) {
  // vertices relative to the origin, permuted (kx, ky, kz)
  float ax = DG_SUB(wt_sel(p0.x, p0.y, p0.z, r.kx), wt_sel(ox, oy, oz, r.kx));
  float ay = DG_SUB(wt_sel(p0.x, p0.y, p0.z, r.ky), wt_sel(ox, oy, oz, r.ky));
  float az = DG_SUB(wt_sel(p0.x, p0.y, p0.z, r.kz), wt_sel(ox, oy, oz, r.kz));
  float bx = DG_SUB(wt_sel(p1.x, p1.y, p1.z, r.kx), wt_sel(ox, oy, oz, r.kx));
  float by = DG_SUB(wt_sel(p1.x, p1.y, p1.z, r.ky), wt_sel(ox, oy, oz, r.ky));
  float bz = DG_SUB(wt_sel(p1.x, p1.y, p1.z, r.kz), wt_sel(ox, oy, oz, r.kz));
  float cx = DG_SUB(wt_sel(p2.x, p2.y, p2.z, r.kx), wt_sel(ox, oy, oz, r.kx));
  float cy = DG_SUB(wt_sel(p2.x, p2.y, p2.z, r.ky), wt_sel(ox, oy, oz, r.ky));
  float cz = DG_SUB(wt_sel(p2.x, p2.y, p2.z, r.kz), wt_sel(ox, oy, oz, r.kz));
  // shear into the ray's frame
  float Ax = DG_SUB(ax, DG_MUL(r.sx, az)), Ay = DG_SUB(ay, DG_MUL(r.sy, az));
  float Bx = DG_SUB(bx, DG_MUL(r.sx, bz)), By = DG_SUB(by, DG_MUL(r.sy, bz));
  float Cx = DG_SUB(cx, DG_MUL(r.sx, cz)), Cy = DG_SUB(cy, DG_MUL(r.sy, cz));
  float U = DG_SUB(DG_MUL(Cx, By), DG_MUL(Cy, Bx));
  float V = DG_SUB(DG_MUL(Ax, Cy), DG_MUL(Ay, Cx));
  float W = DG_SUB(DG_MUL(Bx, Ay), DG_MUL(By, Ax));
  if(U == 0.f || V == 0.f || W == 0.f) {
    U = float(double(Cx) * double(By) - double(Cy) * double(Bx));
    V = float(double(Ax) * double(Cy) - double(Ay) * double(Cx));
    W = float(double(Bx) * double(Ay) - double(By) * double(Ax));
  }
  if((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) { return false; }
  float det = DG_ADD(DG_ADD(U, V), W);
  if(det == 0.f) { return false; }
  float T = DG_ADD(DG_ADD(DG_MUL(U, DG_MUL(r.sz, az)), DG_MUL(V, DG_MUL(r.sz, bz))),
                   DG_MUL(W, DG_MUL(r.sz, cz)));
  float inv = DG_RCP(det);
  float t = DG_MUL(T, inv);
  if(!(t >= t_min && t <= t_max)) { return false; }
  out_t = t;
  out_b1 = DG_MUL(V, inv);
  out_b2 = DG_MUL(W, inv);
  return true;
}

// Widening of the slab test.  The plane distances t carry a relative
// rounding error below 2^-20 of |t| (> 8 ulp).  Widening both ends by that,
// tnear - |tnear| 2^-20 <= tfar + |tfar| 2^-20, takes two fused multiply-adds
// per child; the test used, tnear <= tfar + |tfar| 2^-18, takes one and
// accepts every box the two-sided form accepts, for every sign of tnear and
// tfar (the widening only decides where tnear > tfar: with both >= 0 the
// two-sided form needs tnear <= tfar (1 + 2^-20) / (1 - 2^-20) < tfar (1 +
// 2^-18); with both < 0, |tfar| > |tnear| and 2^-18 |tfar| exceeds the two
// margins together; with tnear >= 0 > tfar both forms reject).
#define DORT_SLAB_FAR_WIDEN 3.814697265625e-6f

// 32 bytes of a node with one load (32-byte aligned).
DG_HD void load_32(const uint4* p, uint32_t v[8]) {
#ifdef __CUDA_ARCH__
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7])
      : "l"(p));
#else
  std::memcpy(v, p, 32);
#endif
}

constexpr uint32_t kNodeWords = 6;   // uint4 words per TraceNode

// The box test's margin for the triangle test's rounding.  A triangle test sees
// a triangle at distance D through coordinates rounded to about 2^-24 D, so it
// may report a hit where the ray passes the triangle, and with it its box, by a
// small multiple of that: at most some 20 units for a triangle about as high as
// wide, times its aspect and the ray's slant to it.  The margin is 2^-16 (256
// units) of the largest coordinate difference between the ray's origin and the
// node, but at most four of the node's largest grid steps (TraceNode::
// margin_max).  Without that limit rays from far away visit whole trees: a grid
// of 500 x 500 quads took 162 node visits a ray from 1,000 of its widths away
// and 5,700 from 10,000, against 14 and 72 with it (2 steps: 12 and 69; 8: 18
// and 80).  It only counts where 2^-24 D nears the size of a triangle.
// The margin is the ray's and not the boxes', since the error is: a margin in
// the boxes of 2^-14 of the node's largest coordinate lost hits of meshes at the
// coordinate origin (a 0.04 wide one seen from 10 and more of its widths away)
// and made the nodes of small meshes far from it overlap (the same mesh at
// (100, 0, 50): 129 node visits a ray instead of 7).
#define DORT_RAY_MARGIN 1.52587890625e-5f

// A ray's view of a node's quantization grid.  The distance of plane q on an
// axis is t = (p + s q - o) i; a near plane's, less the margin, is
// (32768 + q) a + b, a far plane's, plus the margin, (65536 + q) a + c.  (The
// rounding of b and c is below a / 100, of the 1/32 step's a / 32.)
struct NodeSlabs {
  float ax, ay, az, bx, by, bz, cx, cy, cz;
};
DG_HD NodeSlabs node_slabs(const uint32_t n0[8], float margin_max, float ox, float oy, float oz,
                           float ix, float iy, float iz) {
  NodeSlabs f;
  const float px = DG_AS_FLOAT(n0[0]) - ox, py = DG_AS_FLOAT(n0[1]) - oy,
              pz = DG_AS_FLOAT(n0[2]) - oz;
  const float m = fminf(DORT_RAY_MARGIN * DG_MAX3(fabsf(px), fabsf(py), fabsf(pz)), margin_max);
  f.ax = DG_AS_FLOAT(n0[3]) * ix;
  f.ay = DG_AS_FLOAT(n0[4]) * iy;
  f.az = DG_AS_FLOAT(n0[5]) * iz;
  // the margin comes last: a lone ray waits for the chain that leads to it
  f.bx = DG_FMA(-32768.f, f.ax, px * ix);
  f.by = DG_FMA(-32768.f, f.ay, py * iy);
  f.bz = DG_FMA(-32768.f, f.az, pz * iz);
  f.cx = DG_FMA(m, fabsf(ix), DG_FMA(-32768.f, f.ax, f.bx));
  f.cy = DG_FMA(m, fabsf(iy), DG_FMA(-32768.f, f.ay, f.by));
  f.cz = DG_FMA(m, fabsf(iz), DG_FMA(-32768.f, f.az, f.bz));
  f.bx = DG_FMA(-m, fabsf(ix), f.bx);
  f.by = DG_FMA(-m, fabsf(iy), f.by);
  f.bz = DG_FMA(-m, fabsf(iz), f.bz);
  return f;
}

// Whether a ray's [t_min, t_max] meets a box of near distance tn and far
// distance tf, as a sign bit (set: it does not).  t_far_max = t_max widened.
DG_HD float slab_sign(float tn, float tf, float t_min, float t_far_max) {
  tf = DG_FMA(fabsf(tf), DORT_SLAB_FAR_WIDEN, tf);
  // tn <= tf, t_min <= tf and tn <= t_far_max: no difference is negative
  return DG_MIN3(tf - tn, tf - t_min, t_far_max - tn);
}

// Tests the 8 child boxes of one node (TraceNode, as three 32-byte loads):
// bit s of the result is set when the ray's [t_min, t_max] meets slot s's
// box (t_far_max = t_max widened).  Empty slots have no bit in either mask of
// the node, so their result does not matter.
//
// What bounds it: a node of 8 byte-quantized boxes fetched as three 32-byte
// loads costs the L1 data pipe a third of the same node with float planes in
// fourteen 16-byte loads (a warp of 13 divergent lanes: 40 against 123 cycles
// per node step on one SM; the pipe was 82 % busy), and then the instructions
// count: half-rate integer and min / max operations (the ALU pipe) first.
// Hence one operation per plane byte, near planes on the ALU pipe and far
// planes on the FMA pipe (all 48 on the ALU pipe: +2 % on the camera rays),
// and one funnel shift per child to collect the results as sign bits.
DG_HD uint32_t node_hits(const uint32_t n0[8], const uint32_t n1[8], const uint32_t n2[8],
                         float ox, float oy, float oz, float ix, float iy, float iz,
                         float t_min, float t_far_max) {
  const NodeSlabs f = node_slabs(n0, DG_AS_FLOAT(n2[6]), ox, oy, oz, ix, iy, iz);
  // near / far plane bytes per axis, by direction sign
  const bool nx = ix < 0.f, ny = iy < 0.f, nz = iz < 0.f;
  const uint32_t near_x[2] = { nx ? n1[4] : n1[2], nx ? n1[5] : n1[3] };
  const uint32_t far_x[2]  = { nx ? n1[2] : n1[4], nx ? n1[3] : n1[5] };
  const uint32_t near_y[2] = { ny ? n2[0] : n1[6], ny ? n2[1] : n1[7] };
  const uint32_t far_y[2]  = { ny ? n1[6] : n2[0], ny ? n1[7] : n2[1] };
  const uint32_t near_z[2] = { nz ? n2[4] : n2[2], nz ? n2[5] : n2[3] };
  const uint32_t far_z[2]  = { nz ? n2[2] : n2[4], nz ? n2[3] : n2[5] };
  const uint32_t one = n1[1];
  uint32_t miss = 0;
#pragma unroll
  for(int s = 7; s >= 0; --s) {
    const int h = s >> 2, j = s & 3;
    const float tn = DG_MAX3(DG_FMA(DG_BYTE_FLOAT(near_x[h], one, j), f.ax, f.bx),
                             DG_FMA(DG_BYTE_FLOAT(near_y[h], one, j), f.ay, f.by),
                             DG_FMA(DG_BYTE_FLOAT(near_z[h], one, j), f.az, f.bz));
    const float tf = DG_MIN3(DG_FMA(DG_BYTE_FLOAT_DP(far_x[h], j), f.ax, f.cx),
                             DG_FMA(DG_BYTE_FLOAT_DP(far_y[h], j), f.ay, f.cy),
                             DG_FMA(DG_BYTE_FLOAT_DP(far_z[h], j), f.az, f.cz));
    miss = DG_PUSH_SIGN(miss, slab_sign(tn, tf, t_min, t_far_max));
  }
  return ~miss & 0xffu;
}

// The same test, operation for operation, for slot `slot` alone (a lane per
// slot, trace_wide).
DG_HD bool slot_hit(const uint32_t n0[8], const uint32_t n1[8], const uint32_t n2[8],
                    uint32_t slot, float ox, float oy, float oz, float ix, float iy, float iz,
                    float t_min, float t_far_max) {
  const NodeSlabs f = node_slabs(n0, DG_AS_FLOAT(n2[6]), ox, oy, oz, ix, iy, iz);
  const bool h = slot >= 4u, nx = ix < 0.f, ny = iy < 0.f, nz = iz < 0.f;
  const uint32_t lo_x = h ? n1[3] : n1[2], hi_x = h ? n1[5] : n1[4];
  const uint32_t lo_y = h ? n1[7] : n1[6], hi_y = h ? n2[1] : n2[0];
  const uint32_t lo_z = h ? n2[3] : n2[2], hi_z = h ? n2[5] : n2[4];
  const uint32_t one = n1[1], j = slot & 3u;
  const float tn = DG_MAX3(DG_FMA(DG_BYTE_FLOAT(nx ? hi_x : lo_x, one, j), f.ax, f.bx),
                           DG_FMA(DG_BYTE_FLOAT(ny ? hi_y : lo_y, one, j), f.ay, f.by),
                           DG_FMA(DG_BYTE_FLOAT(nz ? hi_z : lo_z, one, j), f.az, f.bz));
  const float tf = DG_MIN3(DG_FMA(DG_BYTE_FLOAT_DP(nx ? lo_x : hi_x, j), f.ax, f.cx),
                           DG_FMA(DG_BYTE_FLOAT_DP(ny ? lo_y : hi_y, j), f.ay, f.cy),
                           DG_FMA(DG_BYTE_FLOAT_DP(nz ? lo_z : hi_z, j), f.az, f.cz));
  return (DG_AS_UINT(slab_sign(tn, tf, t_min, t_far_max)) >> 31) == 0u;
}

// Traversal state of one ray.  trav_node visits one node, trav_tri tests one
// triangle, trav_step does a node and its triangles; trace_ray runs the steps
// of one ray to the end, trace_queue (trace_queue.cuh) those of a whole queue.
struct TravState {
  float ox, oy, oz, dx, dy, dz, t_min;
  float ix, iy, iz;
  uint32_t near4, near2, near1;   // slots on the ray's near side, by slot bit 2, 1, 0
  WtRay wt;              // the watertight test's ray frame (WT traversals)
  uint2 group;           // current node group: (base, internal mask << 8 | child-hit bits)
  int sp;                // entries on the caller's stack
  Hit best;              // closest hit so far (best.t = t_max while none)
};

DG_HD void trav_init(TravState& s, const TraceScene& sc, float ox, float oy, float oz,
                     float t_min, float dx, float dy, float dz, float t_max) {
  s.ox = ox; s.oy = oy; s.oz = oz; s.dx = dx; s.dy = dy; s.dz = dz; s.t_min = t_min;
  s.best.t = t_max;
  s.best.b1 = 0.f;
  s.best.b2 = 0.f;
  s.best.prim = kMiss;
  // Box-test reciprocals; zero components become tiny so no NaN appears.
  const float tiny = 1e-20f;
  s.ix = DG_RCP_APPROX(fabsf(dx) < tiny ? copysignf(tiny, dx) : dx);
  s.iy = DG_RCP_APPROX(fabsf(dy) < tiny ? copysignf(tiny, dy) : dy);
  s.iz = DG_RCP_APPROX(fabsf(dz) < tiny ? copysignf(tiny, dz) : dz);
  s.near4 = s.iz < 0.f ? 0xf0u : 0x0fu;
  s.near2 = s.iy < 0.f ? 0xccu : 0x33u;
  s.near1 = s.ix < 0.f ? 0xaau : 0x55u;
  s.wt = wt_setup(dx, dy, dz);
  s.sp = 0;
  // root group: one child with an empty internal-slot mask -> node 0.  An empty
  // tree or interval starts finished.  So does a ray that leaves its origin away
  // from every box on some axis, from so far off that its distances overflow: the
  // box test would subtract infinite distances and let every box pass.  A ray
  // without a position on any axis (a NaN origin or direction) would pass every
  // box too; the triangle test reports NaN distances as hits, and those of the
  // last node (leaves only) do as well as any.
  const float out = DG_MAX3(ox * s.ix, oy * s.iy, oz * s.iz);
  const bool undefined = out != out;
  const bool open = undefined ? t_min <= t_max : out <= 2e38f && !(t_max < t_min);
  s.group = make_uint2(undefined ? sc.node_count - 1u : 0u, sc.node_count && open ? 1u : 0u);
}

// Traversal stacks.  A node group is pushed per level descended, so a ray's
// stack holds at most the tree's depth (<= kTraceStack) entries; the trees
// of the benchmark scenes are 8 levels deep.
//
// LocalStack (the default): the stack in per-thread local memory.  Only the
// first few entries are ever touched, and local memory is interleaved so a
// warp's accesses to one depth are coalesced; they stay in the L1 cache.
//
// ShortStack (built with DORT_SHORT_STACK): the first kShortStack entries of
// every thread in shared memory, one column per thread (entry k of thread t
// at k * kShortStackThreads + t: a warp's 8-byte accesses fall in distinct
// banks whatever depth each lane is at), deeper entries in local memory.  It
// measured slower on B200: 598 against 618 M samples/s on the 1080p frame,
// 2,315 against 2,457 Mrays/s on the ray cast, as the shared array takes
// its share of the SM's L1 from the node and triangle fetches.  Blocks wider
// than kShortStackThreads keep the whole stack in local memory.
struct LocalStack {
  uint2 e[kTraceStack];
  DG_HD void init() {}
  DG_HD void push(int sp, uint2 v) { e[sp] = v; }
  DG_HD uint2 pop(int sp) { return e[sp]; }
};

#if defined(__CUDA_ARCH__) && defined(DORT_SHORT_STACK)
constexpr int kShortStack = 8;
constexpr int kShortStackThreads = 128;

// One array per block for every traversal of the kernel (a thread runs one
// traversal at a time).
__device__ __forceinline__ uint2* short_stack_block() {
  __shared__ uint2 s[kShortStack * kShortStackThreads];
  return s;
}

struct ShortStack {
  uint32_t col;        // this thread's column in the block's array
  int lim;             // entries below lim live in shared memory (0: none)
  uint2 deep[kTraceStack];
  __device__ __forceinline__ void init() {
    const uint32_t nt = blockDim.x * blockDim.y * blockDim.z;
    col = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    lim = nt <= kShortStackThreads ? kShortStack : 0;
  }
  __device__ __forceinline__ void push(int sp, uint2 v) {
    if(sp < lim) { short_stack_block()[sp * kShortStackThreads + col] = v; } else { deep[sp] = v; }
  }
  __device__ __forceinline__ uint2 pop(int sp) {
    return sp < lim ? short_stack_block()[sp * kShortStackThreads + col] : deep[sp];
  }
};
using TraceStack = ShortStack;
#else
using TraceStack = LocalStack;
#endif

// Triangle tests of a traversal (WT): kTriMt = Moller-Trumbore on the leaf
// layout (p0, e1, e2), kTriWatertight = wt_hit on the layout (p0, p1, p2) of
// scenes built watertight, kTriByScene = whichever the scene was built for
// (TraceScene::watertight).
enum : int { kTriMt = 0, kTriWatertight = 1, kTriByScene = 2 };

// A node's leaf triangles that a ray still has to test: x = index of the
// node's first triangle, y = their bits (low half, bit 8 k + s: triangle k of
// slot s) under the bits of all its triangles (high half).
DG_HD bool leaf_empty(uint2 leaf) { return (leaf.y & 0xffffu) == 0u; }

// Whether the ray has nodes left (the current group is refilled from the
// stack as soon as it is empty).
DG_HD bool group_left(const TravState& s) { return (s.group.y & 0xffu) != 0u; }

// Takes the next node off the current group (there must be one, group_left):
// the hit child nearest in octant order, that is, the near half by slot bit 2,
// then bit 1, then bit 0.
DG_HD const uint4* trav_next(TravState& s, const TraceScene& sc) {
  uint32_t pick = s.group.y & 0xffu;
  pick = (pick & s.near4) ? pick & s.near4 : pick;
  pick = (pick & s.near2) ? pick & s.near2 : pick;
  pick = (pick & s.near1) ? pick & s.near1 : pick;
  s.group.y ^= pick;
  const uint32_t node = s.group.x + DG_POPC((s.group.y >> 8) & (pick - 1u));
  return sc.nodes + kNodeWords * size_t(node);
}

// Goes on from a node with the slots `hits`: its internal ones become the
// current group, its leaf ones are returned.
template<class Stack>
DG_HD uint2 trav_enter(TravState& s, Stack& stack, uint32_t hits, uint32_t child_base,
                       uint32_t tri_base, uint32_t masks) {
  // written as selects: as nested branches it cost 1.5 % of the ray cast
  const uint32_t inner = hits & masks & 0xffu;
  const bool left = group_left(s);
  // sp < kTraceStack: each push descends one level and the builder bounds the
  // depth by kMaxWideDepth.
  if(inner && left) { stack.push(s.sp, s.group); }
  s.sp += (inner && left) ? 1 : 0;
  const bool pop = !inner && !left && s.sp > 0;
  s.sp -= pop ? 1 : 0;
  if(inner) { s.group = make_uint2(child_base, (masks << 8) | inner); }
  if(pop) { s.group = stack.pop(s.sp); }
  return make_uint2(tri_base, (masks & 0xffff0000u) | ((hits * 0x101u) & (masks >> 16)));
}

// Visits the next node: its hit children become the current group, its hit
// leaf slots are returned.
template<class Stack>
DG_HD uint2 trav_node(TravState& s, const TraceScene& sc, Stack& stack) {
  const uint4* np = trav_next(s, sc);
  uint32_t n0[8], n1[8], n2[8];
  load_32(np, n0);
  load_32(np + 2, n1);
  load_32(np + 4, n2);
  const uint32_t hits = node_hits(n0, n1, n2, s.ox, s.oy, s.oz, s.ix, s.iy, s.iz, s.t_min,
                                  DG_FMA(fabsf(s.best.t), DORT_SLAB_FAR_WIDEN, s.best.t));
  return trav_enter(s, stack, hits, n0[6], n0[7], n1[0]);
}

// Tests the next triangle of a non-empty `leaf`; true when it was hit (and
// is the closest hit so far, or for ANY_HIT ends the ray).
template<bool ANY_HIT, bool EXACT_MT, int WT>
DG_HD bool trav_tri(TravState& s, const TraceScene& sc, uint2& leaf) {
  const uint32_t below = (leaf.y & (0u - leaf.y)) - 1u;
  const uint32_t index = leaf.x + DG_POPC((leaf.y >> 16) & below);
  leaf.y &= leaf.y - 1u;
  const float4* tp = sc.tris + 3 * size_t(index);
  float4 a = DG_LDG(tp), e1 = DG_LDG(tp + 1), e2 = DG_LDG(tp + 2);
  float t, b1, b2;
  bool h;
  if(WT == kTriWatertight || (WT == kTriByScene && sc.watertight)) {
    h = wt_hit(s.wt, a, e1, e2, s.ox, s.oy, s.oz, s.t_min, s.best.t, t, b1, b2);
  } else {
    h = EXACT_MT
        ? mt_exact(a, e1, e2, s.ox, s.oy, s.oz, s.dx, s.dy, s.dz, s.t_min, s.best.t, t, b1, b2)
        : mt_fast(a, e1, e2, s.ox, s.oy, s.oz, s.dx, s.dy, s.dz, s.t_min, s.best.t, t, b1, b2);
  }
  if(h) {
    uint32_t id = DG_AS_UINT(a.w);
    if(ANY_HIT || s.best.prim == kMiss || t < s.best.t || id > s.best.prim) {
      s.best.t = t; s.best.b1 = b1; s.best.b2 = b2; s.best.prim = id;
      return true;
    }
  }
  return false;
}

// One traversal step; returns true when the ray is finished (s.best holds
// the closest hit, or for ANY_HIT the first hit found, or prim = kMiss).
template<bool ANY_HIT, bool EXACT_MT, class Stack, int WT = kTriMt>
DG_HD bool trav_step(TravState& s, const TraceScene& sc, Stack& stack) {
  if(!group_left(s)) { return true; }   // an empty tree or interval
  uint2 leaf = trav_node(s, sc, stack);
  while(!leaf_empty(leaf)) {
    if(trav_tri<ANY_HIT, EXACT_MT, WT>(s, sc, leaf) && ANY_HIT) { return true; }
  }
  return !group_left(s);
}

// Closest hit (ANY_HIT = false) or any hit (ANY_HIT = true) of one ray.
// Returns the hit with prim = kMiss on a miss.  For any hit, prim = the first
// triangle found to intersect.
template<bool ANY_HIT, bool EXACT_MT = true, int WT = kTriMt>
DG_HD Hit trace_ray(const TraceScene& sc, float ox, float oy, float oz, float t_min,
                    float dx, float dy, float dz, float t_max) {
  TravState s;
  trav_init(s, sc, ox, oy, oz, t_min, dx, dy, dz, t_max);
  TraceStack stack;
  stack.init();
  while(!trav_step<ANY_HIT, EXACT_MT, TraceStack, WT>(s, sc, stack)) {}
  return s.best;
}

}  // namespace dort_gpu

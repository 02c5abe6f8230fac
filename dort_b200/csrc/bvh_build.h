// Host-side BVH construction for the device scene.
//
// The reference builds a binary BVH per mesh with middle or SAH splits
// (src/dort/bvh.cpp:9-416) and traverses it with a 64-entry stack of 32-byte
// nodes (bvh.cpp:418-469).  The device scene instead uses a wide BVH (up to 8
// children per node) with 8-bit quantized child boxes and octant-ordered
// child slots:
//
//   WideNode: the builders' form of a node
//     float    p[3], s[3]  origin and steps of the quantization grid
//     uint8_t  imask       bit s set: slot s is an internal child
//     uint32_t child_base  node index of the first internal child; internal
//                          children are contiguous, ordered by slot
//     uint32_t tri_base    index of the node's first triangle
//     uint8_t  meta[8]     triangles of slot s when it is a leaf, else 0; a
//                          node's triangles are its leaf slots' first ones in
//                          slot order, then their second ones
//     uint8_t  qlo[3][8], qhi[3][8]   quantized child boxes
//   TraceNode: the same as the device traverses it (three 32-byte loads)
//
// Child boxes are quantized outward with 1/32 of a grid step to spare, which
// covers the rounding of the device slab test's decoding; the triangle test's
// own rounding grows with the distance from the ray and is covered there
// (trace.cuh, DORT_RAY_MARGIN).  (A whole step of margin on this grid, beside
// the ray's: 16.8M rays on the 1M-triangle soup 7.56 against 7.33 ms, 3M shadow
// rays on a 250k-triangle sphere 0.86 against 0.83 ms.)
//
//   Triangle (48 bytes = 3 x float4, leaf order):
//     (p0.xyz, original triangle index as bits), (e1.xyz, 0), (e2.xyz, 0)
//   with e1 = p1 - p0 and e2 = p2 - p0 rounded exactly as the reference does
//   inside Triangle::hit_p (triangle.cpp:18-19).
#pragma once
#include <cstdint>
#include <string>
#include <vector>

namespace dort_gpu {

// Throws std::bad_alloc when a test's injected allocation failure is due
// (dort_gpu_debug_fail_alloc); called before the builders' large allocations.
void alloc_checkpoint();


struct WideNode {
  float p[3];
  float s[3];
  uint8_t imask;
  uint32_t child_base;
  uint32_t tri_base;
  uint8_t meta[8];
  uint8_t qlo[3][8];
  uint8_t qhi[3][8];
};

// Limit of the box test's margin in the largest of a node's steps.
constexpr float kMarginSteps = 4.f;

// The same node as the device traverses it.  96 bytes = three 32-byte loads.
struct alignas(32) TraceNode {
  float p[3];            // origin of the quantization grid
  float s[3];            // its steps
  uint32_t child_base;
  uint32_t tri_base;
  uint32_t masks;        // bits 0..7: imask; bit 16 + 8 k + s: slot s is a leaf of more than k triangles
  uint32_t byte_one;     // 32768.f: a plane byte in its second byte makes the float 32768 + byte
  uint32_t q[3][2][2];   // [axis][0: lo, 1: hi][slots 0..3, 4..7]: child planes, a byte per slot
  float margin_max;      // upper limit of the box test's margin (trace.cuh): kMarginSteps steps
  uint32_t pad;
};
static_assert(sizeof(TraceNode) == 96, "TraceNode must be 96 bytes");

// Quantized nodes as TraceNodes.
void pack_trace_nodes(const std::vector<WideNode>& in, std::vector<TraceNode>& out);

struct alignas(16) LeafTri {
  float p0[3];
  uint32_t id;
  float e1[3];
  float pad1;
  float e2[3];
  float pad2;
};
static_assert(sizeof(LeafTri) == 48, "LeafTri must be 48 bytes");

// Cost of a traversal step relative to a triangle test in the binary SAH of
// both builders (host and device build the same tree).
constexpr double kSahTraversal = 0.5;

struct BuildOptions {
  uint32_t width = 8;          // children per node, 2..8
  uint32_t max_leaf_tris = 2;  // triangles per leaf slot, 1..2 (2: +2.7 % on the ray cast over 3)
  uint32_t bins = 32;          // SAH bins per axis
  uint32_t threads = 0;        // 0: hardware concurrency
};

struct WideBvh {
  std::vector<WideNode> nodes;
  std::vector<TraceNode> trace;    // the nodes as traversed
  std::vector<LeafTri> tris;
  uint32_t depth = 0;          // levels of wide nodes
  double root_lo[3] = {0, 0, 0};
  double root_hi[3] = {0, 0, 0};
};

// The node array the device traversal reads, and its size in bytes.
inline const void* traversal_nodes(const WideBvh& b) { return b.trace.data(); }
inline size_t traversal_node_bytes(const WideBvh& b) {
  return b.trace.size() * sizeof(TraceNode);
}

// Maximum stack depth the device traversal supports; the builder guarantees
// that no root-to-leaf path of the wide tree is deeper.
constexpr uint32_t kMaxWideDepth = 64;

// The binary tree the device made, for checks.  A leaf has bit 31 set in
// `left`, the rest of `left` is its first position in leaf_idx and `right`
// its triangle count; an internal node has its children in left / right.
// count = triangles below each node.
struct BinaryDump {
  std::vector<float> lo, hi;      // 3 per node
  std::vector<uint32_t> left, right, count;
  std::vector<uint32_t> leaf_idx;    // triangle indices in leaf order
  uint32_t root = 0;
};

// Collapses a binary tree made elsewhere (the device builder's) with the
// host's collapse, for checking the device collapse byte for byte.
bool collapse_binary_dump(const BinaryDump& tree, const float* verts, const uint32_t* tris,
                          uint32_t tri_count, const BuildOptions& opts, WideBvh& out,
                          std::string& err);

// Surface-area cost of a wide BVH from its child planes, relative to the
// root box: sum over visited child nodes of area, plus sum over leaf slots of
// area x triangle count (traversal and intersection cost 1 each).
double wide_sah_cost(const TraceNode* nodes, size_t node_count);

// The input checks of build_wide_bvh, with the same messages (indices in
// range, finite coordinates of magnitude at most 1e15).
bool validate_mesh(const float* verts, uint32_t vert_count, const uint32_t* tris,
                   uint32_t tri_count, std::string& err);

// validate_mesh and the bounds of the vertices that triangles use, in one pass
// over the mesh on several threads (a 500k-triangle scene spent 8 of its 17 ms
// of creation on two passes of one thread).  lo / hi are only written for a
// valid mesh with triangles.
bool scan_mesh(const float* verts, uint32_t vert_count, const uint32_t* tris, uint32_t tri_count,
               float lo[3], float hi[3], std::string& err);

// Builds the wide BVH; returns false (with a message) on invalid input.
bool build_wide_bvh(const float* verts, uint32_t vert_count,
                    const uint32_t* tris, uint32_t tri_count,
                    const BuildOptions& opts, WideBvh& out, std::string& err);

}  // namespace dort_gpu

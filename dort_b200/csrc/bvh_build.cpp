// Host-side wide BVH construction: binned SAH binary build, greedy collapse
// to up to 8 children, octant slot assignment and conservative 8-bit
// quantization.  See bvh_build.h for the node format.
//
// The reference's own build (src/dort/bvh.cpp:98-383) differs on purpose:
// it defaults to middle splits, its SAH uses 12 buckets on one axis with an
// area formula missing the x*y term (include/dort/box.hpp:29) and integer
// costs.  Hit results do not depend on the tree shape (closest hit is a
// property of the triangle set), so the device tree is free to be a better
// one.
#include "bvh_build.h"
#include "bvh_wide.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <future>
#include <limits>
#include <thread>

namespace dort_gpu {
namespace {

struct Aabb {
  float lo[3] = {INFINITY, INFINITY, INFINITY};
  float hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  void grow(const Aabb& b) {
    for(int a = 0; a < 3; ++a) {
      lo[a] = std::min(lo[a], b.lo[a]);
      hi[a] = std::max(hi[a], b.hi[a]);
    }
  }
  void grow(const float* p) {
    for(int a = 0; a < 3; ++a) {
      lo[a] = std::min(lo[a], p[a]);
      hi[a] = std::max(hi[a], p[a]);
    }
  }
  bool empty() const { return !(lo[0] <= hi[0]); }
  double area() const {
    if(empty()) { return 0.0; }
    double x = double(hi[0]) - lo[0], y = double(hi[1]) - lo[1], z = double(hi[2]) - lo[2];
    return 2.0 * (x * y + y * z + z * x);
  }
};

struct BinNode {
  Aabb box;
  uint32_t left = 0, right = 0;   // internal: children
  uint32_t first = 0, count = 0;  // leaf: range in the primitive order
  uint32_t tri_total = 0;         // triangles below this node
};

struct Prim {
  Aabb box;
  float c[3];
};

class BinaryBuilder {
 public:
  BinaryBuilder(std::vector<Prim>& prims, const BuildOptions& o)
      : prims_(prims), opts_(o) {
    order_.resize(prims.size());
    for(uint32_t i = 0; i < order_.size(); ++i) { order_[i] = i; }
  }

  std::vector<BinNode> nodes;
  std::vector<uint32_t> order_;

  void build() {
    nodes.reserve(prims_.size() * 2 / std::max(1u, opts_.max_leaf_tris) + 16);
    nodes.emplace_back();
    build_rec(0, 0, uint32_t(prims_.size()), 0);
  }

 private:
  std::vector<Prim>& prims_;
  const BuildOptions& opts_;

  // Splits are SAH-binned on all three axes; a degenerate or over-deep node
  // falls back to an object-median split so that the depth stays bounded.
  void build_rec(uint32_t node_idx, uint32_t begin, uint32_t end, uint32_t depth) {
    uint32_t n = end - begin;
    Aabb box, cbox;
    for(uint32_t i = begin; i < end; ++i) {
      const Prim& p = prims_[order_[i]];
      box.grow(p.box);
      cbox.grow(p.c);
    }
    nodes[node_idx].box = box;
    nodes[node_idx].tri_total = n;

    // Binary SAH costs (relative): a traversal step at half a triangle test.
    // The wide collapse then packs more single-triangle leaves; measured +3 %
    // on the ray cast and the 1080p frame against equal costs (and -5 % at
    // 2 or 4).  The device builder uses the same constant (kSahTraversal).
    const double c_trav = kSahTraversal, c_isect = 1.0;
    if(n <= 1) { make_leaf(node_idx, begin, n); return; }

    int best_axis = -1;
    uint32_t best_bin = 0;
    double best_cost = std::numeric_limits<double>::infinity();
    uint32_t nb = std::max(2u, std::min(opts_.bins, 64u));
    bool force_median = depth >= 36;

    if(!force_median) {
      for(int a = 0; a < 3; ++a) {
        double ext = double(cbox.hi[a]) - cbox.lo[a];
        if(!(ext > 0.0)) { continue; }
        Aabb bins[64];
        uint32_t counts[64] = {0};
        double k = nb / ext;
        for(uint32_t i = begin; i < end; ++i) {
          const Prim& p = prims_[order_[i]];
          int b = int((double(p.c[a]) - cbox.lo[a]) * k);
          b = std::min(std::max(b, 0), int(nb) - 1);
          bins[b].grow(p.box);
          counts[b] += 1;
        }
        double right_area[64];
        uint32_t right_count[64];
        Aabb acc;
        uint32_t cnt = 0;
        for(int b = int(nb) - 1; b > 0; --b) {
          acc.grow(bins[b]);
          cnt += counts[b];
          right_area[b] = acc.area();
          right_count[b] = cnt;
        }
        Aabb lacc;
        uint32_t lcnt = 0;
        for(uint32_t b = 0; b + 1 < nb; ++b) {
          lacc.grow(bins[b]);
          lcnt += counts[b];
          uint32_t rc = right_count[b + 1];
          if(lcnt == 0 || rc == 0) { continue; }
          double cost = lacc.area() * lcnt + right_area[b + 1] * rc;
          if(cost < best_cost) { best_cost = cost; best_axis = a; best_bin = b; }
        }
      }
    }

    double parent_area = std::max(box.area(), 1e-300);
    double split_cost = c_trav + c_isect * best_cost / parent_area;
    double leaf_cost = c_isect * n;
    if(n <= opts_.max_leaf_tris && (best_axis < 0 || leaf_cost <= split_cost)) {
      make_leaf(node_idx, begin, n);
      return;
    }

    uint32_t mid;
    if(best_axis >= 0) {
      int a = best_axis;
      double ext = double(cbox.hi[a]) - cbox.lo[a];
      double k = nb / ext;
      auto it = std::partition(order_.begin() + begin, order_.begin() + end,
          [&](uint32_t idx) {
            int b = int((double(prims_[idx].c[a]) - cbox.lo[a]) * k);
            b = std::min(std::max(b, 0), int(nb) - 1);
            return uint32_t(b) <= best_bin;
          });
      mid = uint32_t(it - order_.begin());
    } else {
      mid = begin;  // fall through to the median split below
    }
    if(mid == begin || mid == end) {
      int a = 0;
      for(int k = 1; k < 3; ++k) {
        if(cbox.hi[k] - cbox.lo[k] > cbox.hi[a] - cbox.lo[a]) { a = k; }
      }
      mid = begin + n / 2;
      std::nth_element(order_.begin() + begin, order_.begin() + mid,
          order_.begin() + end, [&](uint32_t x, uint32_t y) {
            return prims_[x].c[a] < prims_[y].c[a];
          });
    }

    uint32_t l = uint32_t(nodes.size());
    nodes.emplace_back();
    nodes.emplace_back();
    nodes[node_idx].left = l;
    nodes[node_idx].right = l + 1;
    nodes[node_idx].count = 0;
    build_rec(l, begin, mid, depth + 1);
    build_rec(l + 1, mid, end, depth + 1);
  }

  void make_leaf(uint32_t node_idx, uint32_t begin, uint32_t n) {
    nodes[node_idx].first = begin;
    nodes[node_idx].count = n;
    nodes[node_idx].left = nodes[node_idx].right = 0;
  }
};

struct Collapser {
  const std::vector<BinNode>& bn;
  const std::vector<uint32_t>& order;
  const float* verts;
  const uint32_t* tris;
  const BuildOptions& opts;
  WideBvh& out;
  std::string& err;

  struct Pending {
    uint32_t bin;       // binary node to expand into a wide node
    uint32_t wide;      // its index in out.nodes
    uint32_t depth;
  };

  void collect_tris(uint32_t b, std::vector<uint32_t>& dst) const {
    if(bn[b].count > 0 || (bn[b].left == 0 && bn[b].right == 0)) {
      for(uint32_t i = 0; i < bn[b].count; ++i) { dst.push_back(order[bn[b].first + i]); }
      return;
    }
    collect_tris(bn[b].left, dst);
    collect_tris(bn[b].right, dst);
  }

  bool is_leaf(uint32_t b) const { return bn[b].left == 0 && bn[b].right == 0; }

  struct Acc {
    const std::vector<BinNode>& bn;
    bool leaf(uint32_t b) const { return bn[b].left == 0 && bn[b].right == 0; }
    uint32_t left(uint32_t b) const { return bn[b].left; }
    uint32_t right(uint32_t b) const { return bn[b].right; }
    const float* lo(uint32_t b) const { return bn[b].box.lo; }
    const float* hi(uint32_t b) const { return bn[b].box.hi; }
  };

  bool run() {
    out.nodes.clear();
    out.tris.clear();
    if(bn.empty() || bn[0].tri_total == 0) { out.depth = 0; return true; }
    out.nodes.emplace_back();
    std::vector<Pending> queue;
    queue.push_back({0, 0, 1});
    uint32_t max_depth = 1;
    size_t head = 0;
    uint32_t width = std::min(8u, std::max(2u, opts.width));
    Acc acc{bn};
    while(head < queue.size()) {
      Pending cur = queue[head++];
      max_depth = std::max(max_depth, cur.depth);
      uint32_t cands[8];
      uint32_t n = open_candidates(acc, cur.bin, width, cands);
      float nlo[3], nhi[3];
      int cand_in_slot[8];
      assign_slots(acc, cands, n, nlo, nhi, cand_in_slot);
      WideNode node;
      std::memset(&node, 0, sizeof(node));
      if(!quantize_node(acc, cands, cand_in_slot, nlo, nhi, node)) {
        err = "BVH quantization failed (scene coordinates out of range)";
        return false;
      }

      // Internal children first (contiguous, slot order), then leaf triangles.
      uint32_t child_base = uint32_t(out.nodes.size());
      uint32_t tri_base = uint32_t(out.tris.size());
      node.child_base = child_base;
      node.tri_base = tri_base;
      std::vector<uint32_t> leaf_tris;
      std::vector<uint32_t> layer[2];   // the slots' first and second triangles
      for(int s = 0; s < 8; ++s) {
        int c = cand_in_slot[s];
        if(c < 0) { continue; }   // an empty slot (inverted box)
        uint32_t b = cands[c];
        bool leaf = is_leaf(b) || bn[b].tri_total <= opts.max_leaf_tris;
        if(!leaf) {
          node.imask |= uint8_t(1u << s);
          uint32_t wi = uint32_t(out.nodes.size());
          out.nodes.emplace_back();
          queue.push_back({b, wi, cur.depth + 1});
        } else {
          leaf_tris.clear();
          collect_tris(b, leaf_tris);
          uint32_t cnt = uint32_t(leaf_tris.size());
          if(cnt == 0) {
            for(int a = 0; a < 3; ++a) { node.qlo[a][s] = 255; node.qhi[a][s] = 0; }
            continue;
          }
          if(cnt > 2) {
            err = "internal error: wide BVH leaf overflow";
            return false;
          }
          node.meta[s] = uint8_t(cnt);
          for(uint32_t k = 0; k < cnt; ++k) { layer[k].push_back(leaf_tris[k]); }
        }
      }
      for(const std::vector<uint32_t>& one : layer) {
        for(uint32_t t : one) {
          LeafTri lt;
          std::memset(&lt, 0, sizeof(lt));
          const float* p0 = verts + 3 * size_t(tris[3 * size_t(t)]);
          const float* p1 = verts + 3 * size_t(tris[3 * size_t(t) + 1]);
          const float* p2 = verts + 3 * size_t(tris[3 * size_t(t) + 2]);
          for(int a = 0; a < 3; ++a) {
            lt.p0[a] = p0[a];
            lt.e1[a] = p1[a] - p0[a];
            lt.e2[a] = p2[a] - p0[a];
          }
          lt.id = t;
          out.tris.push_back(lt);
        }
      }
      out.nodes[cur.wide] = node;
      if(cur.depth > kMaxWideDepth) {
        err = "BVH too deep for the device traversal stack";
        return false;
      }
    }
    out.depth = max_depth;
    for(int a = 0; a < 3; ++a) {
      out.root_lo[a] = bn[0].box.lo[a];
      out.root_hi[a] = bn[0].box.hi[a];
    }
    return true;
  }
};

}  // namespace

void pack_trace_nodes(const std::vector<WideNode>& in, std::vector<TraceNode>& out) {
  out.resize(in.size());
  for(size_t i = 0; i < in.size(); ++i) { pack_trace_node(in[i], out[i]); }
}

bool collapse_binary_dump(const BinaryDump& tree, const float* verts, const uint32_t* tris,
                          uint32_t tri_count, const BuildOptions& opts, WideBvh& out,
                          std::string& err) {
  const uint32_t kLeaf = 0x80000000u;
  size_t count = tree.left.size();
  // the host collapse starts at node 0: swap the root into place
  auto map = [&](uint32_t i) -> uint32_t {
    return i == tree.root ? 0u : (i == 0 ? tree.root : i);
  };
  std::vector<BinNode> bn(count);
  const std::vector<uint32_t>& order = tree.leaf_idx;
  for(size_t i = 0; i < count; ++i) {
    BinNode& b = bn[map(uint32_t(i))];
    for(int a = 0; a < 3; ++a) {
      b.box.lo[a] = tree.lo[3 * i + a];
      b.box.hi[a] = tree.hi[3 * i + a];
    }
    b.tri_total = tree.count[i];
    if(tree.left[i] & kLeaf) {
      b.left = b.right = 0;
      b.first = tree.left[i] & ~kLeaf;
      b.count = tree.right[i];
      if(size_t(b.first) + b.count > order.size()) {
        err = "binary tree leaf out of range";
        return false;
      }
    } else {
      b.left = map(tree.left[i]);
      b.right = map(tree.right[i]);
      b.count = 0;
    }
  }
  Collapser col{bn, order, verts, tris, opts, out, err};
  if(tri_count > 0 && !col.run()) { return false; }
  pack_trace_nodes(out.nodes, out.trace);
  return true;
}

double wide_sah_cost(const TraceNode* nodes, size_t node_count) {
  if(node_count == 0) { return 0.0; }
  auto slot_box = [](const TraceNode& n, int s, float lo[3], float hi[3]) {
    for(int a = 0; a < 3; ++a) {
      auto plane = [&](int side) {
        const uint32_t q = (n.q[a][side][s >> 2] >> (8 * (s & 3))) & 0xffu;
        return float(double(n.p[a]) + double(q) * double(n.s[a]));
      };
      lo[a] = plane(0);
      hi[a] = plane(1);
    }
  };
  auto tris_of = [](const TraceNode& n, int s) {
    return ((n.masks >> (16 + s)) & 1u) + ((n.masks >> (24 + s)) & 1u);
  };
  float lo[3], hi[3];
  float rlo[3] = {INFINITY, INFINITY, INFINITY}, rhi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for(int s = 0; s < 8; ++s) {
    if(!(nodes[0].masks & (1u << s)) && !tris_of(nodes[0], s)) { continue; }
    slot_box(nodes[0], s, lo, hi);
    for(int a = 0; a < 3; ++a) {
      rlo[a] = std::min(rlo[a], lo[a]);
      rhi[a] = std::max(rhi[a], hi[a]);
    }
  }
  double root = std::max(bw_area(rlo, rhi), 1e-300);
  double cost = 1.0;   // the root itself
  for(size_t i = 0; i < node_count; ++i) {
    const TraceNode& n = nodes[i];
    for(int s = 0; s < 8; ++s) {
      const bool internal = n.masks & (1u << s);
      if(!internal && !tris_of(n, s)) { continue; }
      slot_box(n, s, lo, hi);
      double a = bw_area(lo, hi) / root;
      cost += internal ? a : a * double(tris_of(n, s));
    }
  }
  return cost;
}

bool validate_mesh(const float* verts, uint32_t vert_count, const uint32_t* tris,
                   uint32_t tri_count, std::string& err) {
  for(uint32_t t = 0; t < tri_count; ++t) {
    for(int k = 0; k < 3; ++k) {
      uint32_t vi = tris[3 * size_t(t) + k];
      if(vi >= vert_count) {
        err = "triangle " + std::to_string(t) + " references vertex " + std::to_string(vi) +
              " >= vert_count";
        return false;
      }
      const float* v = verts + 3 * size_t(vi);
      if(!std::isfinite(v[0]) || !std::isfinite(v[1]) || !std::isfinite(v[2])) {
        err = "vertex " + std::to_string(vi) + " is not finite";
        return false;
      }
      if(std::fabs(v[0]) > 1e15f || std::fabs(v[1]) > 1e15f || std::fabs(v[2]) > 1e15f) {
        err = "vertex " + std::to_string(vi) + " is out of range (|coord| > 1e15)";
        return false;
      }
    }
  }
  return true;
}

bool scan_mesh(const float* verts, uint32_t vert_count, const uint32_t* tris, uint32_t tri_count,
               float lo[3], float hi[3], std::string& err) {
  struct Part {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool ok = true;
  };
  auto scan = [&](uint32_t begin, uint32_t end, Part& part) {
    for(uint32_t i = begin; i < end; ++i) {
      for(int k = 0; k < 3; ++k) {
        const uint32_t vi = tris[3 * size_t(i) + k];
        if(vi >= vert_count) { part.ok = false; return; }
        const float* v = verts + 3 * size_t(vi);
        for(int a = 0; a < 3; ++a) {
          // also false for NaN
          if(!(std::fabs(v[a]) <= 1e15f)) { part.ok = false; return; }
          part.lo[a] = std::min(part.lo[a], v[a]);
          part.hi[a] = std::max(part.hi[a], v[a]);
        }
      }
    }
  };
  constexpr uint32_t kPerThread = 32768;
  const uint32_t threads = std::max(1u, std::min({tri_count / kPerThread, 8u,
                                                  std::thread::hardware_concurrency()}));
  std::vector<Part> parts(threads);
  std::vector<std::thread> pool;
  auto begin_of = [&](uint32_t k) { return uint32_t(uint64_t(tri_count) * k / threads); };
  uint32_t started = 1;   // part 0 runs here
  pool.reserve(threads);
  try {
    for(; started < threads; ++started) {
      pool.emplace_back(scan, begin_of(started), begin_of(started + 1), std::ref(parts[started]));
    }
  } catch(...) {}         // no more threads: the rest runs here too
  scan(0, begin_of(1), parts[0]);
  for(uint32_t k = started; k < threads; ++k) { scan(begin_of(k), begin_of(k + 1), parts[k]); }
  for(std::thread& t : pool) { t.join(); }
  for(const Part& part : parts) {
    // the first fault's message is the one-pass check's
    if(!part.ok) { return validate_mesh(verts, vert_count, tris, tri_count, err); }
  }
  if(tri_count > 0) {
    for(int a = 0; a < 3; ++a) {
      lo[a] = INFINITY;
      hi[a] = -INFINITY;
      for(const Part& part : parts) {
        lo[a] = std::min(lo[a], part.lo[a]);
        hi[a] = std::max(hi[a], part.hi[a]);
      }
    }
  }
  return true;
}

bool build_wide_bvh(const float* verts, uint32_t vert_count,
                    const uint32_t* tris, uint32_t tri_count,
                    const BuildOptions& opts, WideBvh& out, std::string& err) {
  if(opts.max_leaf_tris < 1 || opts.max_leaf_tris > 2) {
    err = "max_leaf_tris must be 1..2";
    return false;
  }
  if(opts.width < 2 || opts.width > 8) {
    err = "bvh_width must be 2..8";
    return false;
  }
  alloc_checkpoint();
  std::vector<Prim> prims(tri_count);
  for(uint32_t t = 0; t < tri_count; ++t) {
    Prim& p = prims[t];
    for(int k = 0; k < 3; ++k) {
      uint32_t vi = tris[3 * size_t(t) + k];
      if(vi >= vert_count) {
        err = "triangle " + std::to_string(t) + " references vertex " +
              std::to_string(vi) + " >= vert_count";
        return false;
      }
      const float* v = verts + 3 * size_t(vi);
      if(!std::isfinite(v[0]) || !std::isfinite(v[1]) || !std::isfinite(v[2])) {
        err = "vertex " + std::to_string(vi) + " is not finite";
        return false;
      }
      // keeps every quantization step and slab product finite on the device
      if(std::fabs(v[0]) > 1e15f || std::fabs(v[1]) > 1e15f || std::fabs(v[2]) > 1e15f) {
        err = "vertex " + std::to_string(vi) + " is out of range (|coord| > 1e15)";
        return false;
      }
      p.box.grow(v);
    }
    for(int a = 0; a < 3; ++a) { p.c[a] = 0.5f * (p.box.lo[a] + p.box.hi[a]); }
  }
  alloc_checkpoint();
  BinaryBuilder bb(prims, opts);
  if(tri_count > 0) { bb.build(); }
  alloc_checkpoint();
  Collapser col{bb.nodes, bb.order_, verts, tris, opts, out, err};
  if(!col.run()) { return false; }
  pack_trace_nodes(out.nodes, out.trace);
  return true;
}

}  // namespace dort_gpu

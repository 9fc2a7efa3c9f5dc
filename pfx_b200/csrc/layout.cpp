// Reference node array (bvh.rs Node, 48 B) -> B200 traversal layout.
//
// Every inner node X of the reference BVH2 becomes one 64-byte WideNode that
// holds the fp32 boxes of both children (X+1 and X.first).  The box arithmetic
// that the reference runs when it pops a child (trace.wgsl:453-468 box_hit) is
// run on the same fp32 numbers when the parent is opened, so one 4 x 16 B load
// feeds two box tests.  The visiting order stays the reference's left-first
// depth-first order, and the part of box_hit that depends on the current hit
// distance (near <= hit.t) is re-checked when an entry is popped, so the set and
// the order of triangle tests equal the reference's.
//
// The scene root and every bottom-level root get a "pseudo-parent" wide node
// whose child 0 is the root, so that the root box is tested exactly as the
// reference tests it after popping index 0 (or after entering an instance).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <unordered_map>

#include "pfxt_internal.h"

namespace pfxt {

namespace {

struct Builder {
  const GpuNode* nodes;
  size_t node_count;
  const GpuSurface* surfaces;
  size_t surface_count;
  uint64_t tri_count;
  TraversalLayout out;
  std::unordered_map<uint32_t, uint32_t> pseudo_of;  // reference root -> pseudo-parent wide index

  void set_box(WideNode& w, int child, const GpuNode& n) {
    float* f = &w.b0[0];  // b0, b1, b2 are contiguous: 12 floats
    for (int k = 0; k < 3; ++k) {
      f[child * 6 + k] = n.lo[k];
      f[child * 6 + 3 + k] = n.hi[k];
    }
  }

  // Largest leaf end (first + count) under each pseudo-parent, so that every
  // slot a kernel can reach is checked against the triangle count.
  std::unordered_map<uint32_t, uint64_t> reach_of;
  uint64_t reach = 0;  // running maximum while one subtree is laid out

  // The slot base of the subtree being laid out (0: the top level's own
  // leaves) and the base each pseudo-parent's subtree was laid out with.  Scene
  // builds put a slot in one leaf; buffers that do not are walked with the
  // two-box nodes alone (`unboxed`).
  uint32_t base = 0;
  std::unordered_map<uint32_t, uint32_t> base_of;
  bool unboxed = false;
  bool uncontained = false;  // a box does not hold a child's
  // Entries the four-box walk's stack can come to hold, whichever of a node's
  // children it enters first (any hits go to the nearest one; the buffers' own
  // max_depth is the caller's word, and the two-box walk's): below the child
  // laid out last as one entry, and below its own two children when it is an
  // inner node; below each pseudo-parent's root as a node of its own.
  struct Need {
    uint32_t whole = 0, child[2] = {0, 0};
    bool inner = false;
  } need;
  std::unordered_map<uint32_t, uint32_t> need_of;

  // Of a node whose children need l and r: inside any entry of its up to four,
  // all the others may wait.
  static uint32_t quad_need(const Need& l, const Need& r) {
    uint32_t list[4], n = 0, most = 0;
    for (const Need* c : {&l, &r}) {
      if (c->inner) {
        list[n++] = c->child[0];
        list[n++] = c->child[1];
      } else {
        list[n++] = c->whole;
      }
    }
    for (uint32_t i = 0; i < n; ++i) most = std::max(most, list[i]);
    return n - 1u + most;
  }

  // The leaf `at` (wide node << 1 | child, whose box the wide node has already).
  void box_leaf(const GpuNode& n, uint32_t at) {
    const uint64_t first = (uint64_t)base + n.first;
    if (first + n.count > tri_count) return;  // refused by the reach check
    for (uint64_t i = first; i < first + n.count; ++i) {
      const uint32_t earlier = out.leaf_of[i];
      if (earlier != REF_NONE) {
        const float* f = &out.wide[earlier >> 1].b0[0] + 6u * (earlier & 1u);
        if (memcmp(f, n.lo, 12) != 0 || memcmp(f + 3, n.hi, 12) != 0) unboxed = true;
      }
      out.leaf_of[i] = at;
    }
  }

  uint32_t leaf_ref(const GpuNode& n, uint32_t at) {
    if (n.count == 0 || n.count > 16) throw Invalid("BVH leaf holds more than 16 triangles");
    if (n.first > LEAF_FIRST_MASK) throw Invalid("BVH leaf offset exceeds the traversal encoding");
    reach = std::max<uint64_t>(reach, (uint64_t)n.first + n.count);
    box_leaf(n, at);
    return REF_LEAF | ((n.count - 1u) << LEAF_FIRST_BITS) | n.first;
  }

  uint32_t inst_ref(const GpuNode& n) {
    InstRec r{};
    uint32_t record = f2bits(n.lo[3]);
    if (record >= surface_count) throw Invalid("instance record out of range");
    const GpuSurface& s = surfaces[record];
    r.record = record;
    r.base = n.count;
    r.word = s.info[0];
    r.inv_det = bits2f(s.info[3]);
    r.transformed = n.pad[1] > 0 ? 1u : 0u;
    if (r.transformed) {
      if (n.pad[1] >= node_count) throw Invalid("instance rows out of range");
      const GpuNode& m = nodes[n.pad[1]];
      for (int k = 0; k < 4; ++k) {
        r.inv[0][k] = m.lo[k];
        r.inv[1][k] = m.hi[k];
      }
      r.inv[2][0] = bits2f(m.first);
      r.inv[2][1] = bits2f(m.count);
      r.inv[2][2] = bits2f(m.pad[0]);
      r.inv[2][3] = bits2f(m.pad[1]);
    }
    if (n.first >= node_count) throw Invalid("instance root out of range");
    memcpy(r.lo, n.lo, 12);
    memcpy(r.hi, n.hi, 12);
    uint64_t outer = reach;
    uint32_t outer_base = base;
    reach = 0;
    base = r.base;
    r.root = pseudo(n.first);
    uint64_t inner = reach_of[r.root];
    if (base_of[r.root] != r.base) unboxed = true;
    need = Need{};
    need.whole = 1u + need_of[r.root];  // the sentinel that ends the instance
    reach = outer;
    base = outer_base;
    if ((uint64_t)r.base + inner > tri_count) throw Invalid("an instance leaf reaches past the triangles");
    uint32_t index = (uint32_t)out.insts.size();
    if (index >= (1u << 30)) throw Invalid("too many instances");
    out.insts.push_back(r);
    return REF_INST | index;
  }

  // Reference of child node `i` as seen from its parent, which holds it at `at`.
  uint32_t child_ref(uint32_t i, uint32_t at) {
    const GpuNode& n = nodes[i];
    if (n.pad[0] == INSTANCE_LEAF) return inst_ref(n);
    if (n.count == 0) return wide_of(i);
    need = Need{};
    return leaf_ref(n, at);
  }

  uint32_t pseudo(uint32_t root) {
    auto it = pseudo_of.find(root);
    if (it != pseudo_of.end()) return it->second;
    uint32_t w = (uint32_t)out.wide.size();
    out.wide.push_back(WideNode{});
    pseudo_of[root] = w;
    base_of[w] = base;
    uint64_t outer = reach;
    reach = 0;
    WideNode node{};
    set_box(node, 0, nodes[root]);
    out.wide[w] = node;
    node.child[0] = child_ref(root, w << 1);
    node.child[1] = REF_NONE;
    out.wide[w] = node;
    need_of[w] = need.whole;
    reach_of[w] = reach;
    reach = outer;
    return w;
  }

  // Wide node of inner node `i`; children are laid out depth first, left first.
  uint32_t wide_of(uint32_t i) {
    const GpuNode& n = nodes[i];
    uint32_t left = i + 1, right = n.first;
    if (left >= node_count || right >= node_count) throw Invalid("BVH child out of range");
    uint32_t w = (uint32_t)out.wide.size();
    out.wide.push_back(WideNode{});
    WideNode node{};
    set_box(node, 0, nodes[left]);
    set_box(node, 1, nodes[right]);
    for (const GpuNode* c : {&nodes[left], &nodes[right]})
      for (int k = 0; k < 3; ++k)
        if (!(c->lo[k] >= n.lo[k]) || !(c->hi[k] <= n.hi[k])) uncontained = true;
    out.wide[w] = node;
    node.child[0] = child_ref(left, w << 1);
    const Need l = need;
    node.child[1] = child_ref(right, w << 1 | 1u);
    const Need r = need;
    need.whole = quad_need(l, r);
    need.child[0] = l.whole;
    need.child[1] = r.whole;
    need.inner = true;
    out.wide[w] = node;
    return w;
  }
};

}  // namespace

TraversalLayout make_layout(const pfxt_buffers& b) {
  Builder builder;
  builder.nodes = (const GpuNode*)b.nodes;
  builder.node_count = b.nodes_bytes / sizeof(GpuNode);
  builder.surfaces = (const GpuSurface*)b.surfaces;
  builder.surface_count = b.surfaces_bytes / sizeof(GpuSurface);
  builder.tri_count = b.triangles_bytes / sizeof(GpuTriangle);
  if (b.triangle_count != builder.tri_count) throw Invalid("triangle count does not match the triangle buffer");
  builder.out.leaf_of.assign(builder.tri_count, REF_NONE);
  if (builder.node_count > 0 && b.triangle_count > 0) {
    builder.out.wide.reserve(builder.node_count / 2 + 16);
    builder.out.root = builder.pseudo(0);
    // the top level itself: world leaves (base 0) must stay inside the triangles
    if (builder.reach_of[builder.out.root] > builder.tri_count)
      throw Invalid("a BVH leaf reaches past the triangles");
    builder.out.stack_need = builder.need_of[builder.out.root];
  }
  // The box test needs no range check on its quotients when every box
  // coordinate is 0 or of magnitude in [2^-70, 2^79] (traverse.cuh,
  // BOUNDED_TINY and BOUNDED_COORD); NaN coordinates fail this too.  The
  // four-box walk also passes over the boxes between a leaf and the root, which a
  // leaf that passes implies only where lo <= hi and every box holds its
  // children's, and needs leaves whose triangles know their box.
  builder.out.small = !builder.unboxed && !builder.uncontained;
  for (const WideNode& w : builder.out.wide) {
    const float* f = &w.b0[0];
    for (int k = 0; k < 12; ++k) {
      float a = std::fabs(f[k]);
      if (!(a == 0.0f || (a >= 0x1p-70f && a <= 0x1p+79f))) builder.out.small = false;
    }
    for (int k = 0; k < 3; ++k)
      if (!(f[k] <= f[3 + k]) || !(f[6 + k] <= f[9 + k])) builder.out.small = false;
  }
  return std::move(builder.out);
}

}  // namespace pfxt

// treelet.cu -- LBVH+ treelet restructuring passes.
//
// Reference: kRefitAndOptimize(doOptimize=true) with optimizeTreeletSerial,
// src/cuda/lbvh_plus_builder.cu:71-247 and :341-366.  There one pass climbs from every leaf; the
// second child to arrive at a node refits its box and restructures the treelet rooted there
// (up to 7 treelet leaves, grown by expanding the largest-area internal leaf; subset DP with
// cost = min split + area; internal node ids reused in DFS order).
//
// A treelet at X only reads and writes nodes of X's subtree, all of which are final when the
// second child arrives, so the result is independent of scheduling and equal to any
// children-before-parent order (the oracle uses post-order).
//
// The pass goes height by height (a node's height is known from the emission or from the last rebuild): growth
// writes a descriptor per treelet, the DP kernels read it, one lane per treelet; narrow heights take one
// warp per treelet in one cooperative launch.  Trees higher than 254 take the climb-ordered fallback, whose
// warps keep looping while any lane still climbs and do each treelet's DP with all 32 lanes.
#include <algorithm>

#include "emit.cuh"
#include "lbvh.cuh"

namespace bvhgb {

constexpr int kTlMax = 7;
constexpr float kTlInf = 1e30f;
// Minimum of three; as fminf, a NaN operand never wins.
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
}  // namespace bvhgb
#include "treelet_dp_unrolled.cuh"
namespace bvhgb {

__device__ __forceinline__ Box ldcg_box(const Node* nodes, int32_t idx) {
  const float4* p = reinterpret_cast<const float4*>(nodes + idx);
  Box b;
  b.lo = __ldcg(p);
  b.hi = __ldcg(p + 1);
  return b;
}
__device__ __forceinline__ int2 ldcg_children(const Node* nodes, int32_t idx) {
  return __ldcg(reinterpret_cast<const int2*>(&nodes[idx].left));
}

// What a treelet's growth reads of an inner node: its children and their areas.  Every inner node carries the
// areas of its children's boxes as they are (see write_internal; the passes below keep them so), so a
// treelet grows through one 16-byte load per expanded node instead of two 48-byte children.
struct Links {
  int32_t l, r;
  float al, ar;
};
__device__ __forceinline__ Links ldcg_links(const Node* nodes, int32_t idx) {
  const int4 v = __ldcg(reinterpret_cast<const int4*>(&nodes[idx].left));
  return Links{v.x, v.y, __int_as_float(v.z), __int_as_float(v.w)};
}
__device__ __forceinline__ void stcg_links(Node* nodes, int32_t idx, const Links& k) {
  __stcg(reinterpret_cast<int4*>(&nodes[idx].left), make_int4(k.l, k.r, __float_as_int(k.al), __float_as_int(k.ar)));
}
// Height of node idx (leaves, from first_leaf on: 0).
__device__ __forceinline__ uint32_t node_height(const uint8_t* hgt, int32_t first_leaf, int32_t idx) {
  return idx < first_leaf ? (uint32_t)__ldcg(hgt + idx) : 0u;
}

// Subsets of {0..6} with 2..7 members, by size, increasing within a size.  For a treelet of
// n < 7 leaves the subsets of its full mask are the entries <= (1 << n) - 1, in the same order.
__constant__ uint8_t c_subsets[120] = {
    3, 5, 6, 9, 10, 12, 17, 18, 20, 24, 33, 34, 36, 40, 48, 65, 66, 68, 72, 80, 96,
    7, 11, 13, 14, 19, 21, 22, 25, 26, 28, 35, 37, 38, 41, 42, 44, 49, 50, 52, 56, 67, 69, 70, 73, 74, 76, 81,
    82, 84, 88, 97, 98, 100, 104, 112,
    15, 23, 27, 29, 30, 39, 43, 45, 46, 51, 53, 54, 57, 58, 60, 71, 75, 77, 78, 83, 85, 86, 89, 90, 92, 99,
    101, 102, 105, 106, 108, 113, 114, 116, 120,
    31, 47, 55, 59, 61, 62, 79, 87, 91, 93, 94, 103, 107, 109, 110, 115, 117, 118, 121, 122, 124,
    63, 95, 111, 119, 123, 125, 126,
    127};
__constant__ uint8_t c_sub_off[9] = {0, 0, 0, 21, 56, 91, 112, 119, 120};  // first entry of size k

// One lane's treelet: its leaves (node ids, boxes, cached children), the expansions that grew
// it (which the id reuse walks instead of reloading nodes) and the DP's best partitions.
struct LaneTreelet {
  float box[6][kTlMax];  // lo.x lo.y lo.z hi.x hi.y hi.z of each leaf
  int32_t act[kTlMax];
  int32_t chl[kTlMax], chr[kTlMax];  // children of each leaf node (left has kLeafBit for a BVH leaf)
  int32_t exp_node[kTlMax - 1], exp_l[kTlMax - 1], exp_r[kTlMax - 1];
  uint8_t part[1 << kTlMax];
  int32_t n;
};

__device__ __forceinline__ Box leaf_box(const LaneTreelet& T, int i) {
  Box b;
  b.lo = make_float4(T.box[0][i], T.box[1][i], T.box[2][i], 0.f);
  b.hi = make_float4(T.box[3][i], T.box[4][i], T.box[5][i], 0.f);
  return b;
}
__device__ __forceinline__ void set_leaf(LaneTreelet& T, int i, int32_t id, const Box& b, int2 ch) {
  T.act[i] = id;
  T.box[0][i] = b.lo.x; T.box[1][i] = b.lo.y; T.box[2][i] = b.lo.z;
  T.box[3][i] = b.hi.x; T.box[4][i] = b.hi.y; T.box[5][i] = b.hi.z;
  T.chl[i] = ch.x;
  T.chr[i] = ch.y;
}

// 1. Grow the treelet at `root` (lbvh_plus_builder.cu:73-114): up to 6 times, expand the leaf
//    with the largest area among those that are internal nodes (first such on ties).  Run by
//    one lane; the lanes of a warp grow their own treelets side by side.
__device__ void treelet_grow(const Node* nodes, int32_t root, LaneTreelet& T) {
  set_leaf(T, 0, root, ldcg_box(nodes, root), ldcg_children(nodes, root));
  int cnt = 1;
  for (int step = 0; step < kTlMax - 1; ++step) {
    int best = -1;
    float max_area = -1.0f;
#pragma unroll
    for (int i = 0; i < kTlMax; ++i) {
      if (i < cnt && !((uint32_t)T.chl[i] & kLeafBit)) {
        const float a = box_area(leaf_box(T, i));
        if (a > max_area) { max_area = a; best = i; }
      }
    }
    if (best < 0) break;
    const int32_t l = T.chl[best], r = T.chr[best];
    T.exp_node[step] = T.act[best];
    T.exp_l[step] = l;
    T.exp_r[step] = r;
    const Box bl = ldcg_box(nodes, l), br = ldcg_box(nodes, r);
    const int2 cl = ldcg_children(nodes, l), cr = ldcg_children(nodes, r);
    set_leaf(T, best, l, bl, cl);
    set_leaf(T, cnt, r, br, cr);
    ++cnt;
  }
  T.n = cnt;
}

// The split p of s with the smallest cost among `count` from the (first+1)-th of its enumeration on (p =
// the nonempty subsets of s without its lowest member, increasing); the first of equals; 0 where none is
// below INF.  Unrolled, so that all cost loads are in flight together.
template <int COUNT>
__device__ __forceinline__ float scan_splits(const float* cost, uint32_t s, uint32_t first, uint32_t end, uint32_t& bp) {
  const uint32_t delta = s & (s - 1u);
  // the (first+1)-th nonempty subset of delta: the bits of first + 1 spread over delta's members
  uint32_t p = 0, rest = delta;
#pragma unroll
  for (int i = 0; i < kTlMax - 1; ++i) {
    const uint32_t low = rest & (0u - rest);
    p |= ((first + 1u) >> i) & 1u ? low : 0u;
    rest ^= low;
  }
  float v[COUNT];
  uint32_t q[COUNT];
#pragma unroll
  for (int k = 0; k < COUNT; ++k) {
    q[k] = p;
    v[k] = first + (uint32_t)k < end ? __fadd_rn(cost[p], cost[s ^ p]) : kTlInf;
    p = (p - delta) & delta;
  }
  float best = kTlInf;
  bp = 0;
#pragma unroll
  for (int k = 0; k < COUNT; ++k)
    if (v[k] < best) {
      best = v[k];
      bp = q[k];
    }
  return best;
}

// One size K of the DP: COUNT subsets from c_subsets[c_sub_off[K]], two per lane side by side.
template <int K>
__device__ __forceinline__ void warp_dp_size(LaneTreelet& T, float* cost, const float* area, uint32_t full) {
  constexpr uint32_t kParts = (1u << (K - 1)) - 1u;
  const uint32_t lane = threadIdx.x & 31, base = c_sub_off[K], count = c_sub_off[K + 1] - base;
  uint32_t s[2], bp[2];
  float best[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t e = lane + 32u * i;
    s[i] = e < count ? c_subsets[base + e] : 0u;
    if (s[i] > full) s[i] = 0;
    best[i] = s[i] ? scan_splits<(int)kParts>(cost, s[i], 0, kParts, bp[i]) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (s[i]) {
      cost[s[i]] = __fadd_rn(best[i], area[s[i]]);  // (no split below INF: INF plus the area, and split 0)
      T.part[s[i]] = (uint8_t)bp[i];
    }
  __syncwarp();
}

// A float's bits as an unsigned number of the same order (no NaN).
__device__ __forceinline__ uint32_t ordered_bits(float v) {
  const uint32_t u = __float_as_uint(v);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}

// 2+3. Subset areas and the DP over subsets by size (:119-165), by the whole warp for one
//    treelet.  cost[s] = min over splits (cost[p] + cost[s^p]) + area[s], leaves cost 0;
//    the best split is the first minimum in the enumeration p = increasing nonempty subsets of
//    s without its lowest member.  Sizes 3 to 5 take one lane per subset, size 6 four lanes and
//    size 7 the whole warp.  A chain of five sizes: bound by latency, so each size's loads are issued
//    together (one node of k_tl_narrow: see there).
__device__ void treelet_dp(LaneTreelet& T, float* cost, float* area) {
  const uint32_t lane = threadIdx.x & 31;
  const int n = T.n;
  const uint32_t full = (1u << n) - 1u;
  // lane's subsets lane + 32 {0..3}: the members among leaves 0..4 once, then with leaves 5, 6, both
  Box low = box_empty();
#pragma unroll
  for (int i = 0; i < 5; ++i)
    if ((lane >> i) & 1u) low = box_union(low, leaf_box(T, i));
  const Box b5 = leaf_box(T, 5), b6 = leaf_box(T, 6);
#pragma unroll
  for (uint32_t hi = 0; hi < 4; ++hi) {
    const uint32_t s = lane + 32u * hi;
    Box b = low;
    if (hi & 1u) b = box_union(b, b5);
    if (hi & 2u) b = box_union(b, b6);
    if (s >= 1 && s <= full) {
      const float a = box_area(b);
      const int members = __popc(s);
      area[s] = a;
      // one member: 0; two: the only split costs 0 + 0
      cost[s] = members == 1 ? 0.0f : members == 2 ? __fadd_rn(0.0f, a) : kTlInf;
      if (members == 2) T.part[s] = (uint8_t)(s & (s - 1u));
    }
  }
  __syncwarp();
  warp_dp_size<3>(T, cost, area, full);
  if (n >= 4) warp_dp_size<4>(T, cost, area, full);
  if (n >= 5) warp_dp_size<5>(T, cost, area, full);
  if (n >= 6) {  // 7 subsets of 31 splits, four lanes each
    const uint32_t e = lane >> 2, j = lane & 3u;
    uint32_t s = e < 7 ? c_subsets[c_sub_off[6] + e] : 0u, bp = 0;
    if (s > full) s = 0;
    float best = s ? scan_splits<8>(cost, s, 8u * j, 31u, bp) : kTlInf;
    uint32_t ord = best < kTlInf ? j : 4u;
#pragma unroll
    for (uint32_t o = 1; o < 4; o <<= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const uint32_t oo = __shfl_xor_sync(0xffffffffu, ord, o), op = __shfl_xor_sync(0xffffffffu, bp, o);
      if (ob < best || (ob == best && oo < ord)) {
        best = ob;
        ord = oo;
        bp = op;
      }
    }
    if (s && j == 0) {
      cost[s] = __fadd_rn(best, area[s]);
      T.part[s] = (uint8_t)bp;
    }
    __syncwarp();
  }
  if (n == 7) {  // the full set's 63 splits, two per lane; only its split is asked for
    uint32_t bp = 0;
    const float best = scan_splits<2>(cost, 127u, 2u * lane, 63u, bp);
    const uint32_t key = ordered_bits(best), least = __reduce_min_sync(0xffffffffu, key);
    const uint32_t first = __ffs(__ballot_sync(0xffffffffu, key == least)) - 1;
    bp = __shfl_sync(0xffffffffu, bp, first);
    if (lane == 0) T.part[127] = (uint8_t)bp;
    __syncwarp();
  }
}

// 4. Reuse the treelet's internal ids (DFS from the root, right child popped first,
//    :167-191) and rebuild it breadth-first from the partitions (:194-246).  One lane.
__device__ void treelet_rebuild(Node* nodes, int32_t* parents, int32_t root, LaneTreelet& T) {
  const int n = T.n;
  if (n < 2) return;
  const uint32_t full = (1u << n) - 1u;
  int avail[kTlMax];
  int n_avail = 0;
  int stack[kTlMax + 8];
  int top = 0;
  stack[top++] = root;
  while (top > 0) {
    const int cur = stack[--top];
    bool in_leaves = false;
    for (int i = 0; i < n; ++i)
      if (T.act[i] == cur) { in_leaves = true; break; }
    if (!in_leaves && n_avail < kTlMax && top + 2 <= kTlMax + 8) {
      avail[n_avail++] = cur;
      int2 ch = make_int2(0, 0);
      bool known = false;
      for (int e = 0; e < n - 1; ++e)
        if (T.exp_node[e] == cur) { ch = make_int2(T.exp_l[e], T.exp_r[e]); known = true; break; }
      if (!known) ch = ldcg_children(nodes, cur);
      stack[top++] = ch.x;
      stack[top++] = ch.y;
    }
  }
  // A subset whose partitions all cost >= INF (NaN areas) has no valid split; the reference
  // would index out of bounds there, this leaves the treelet unchanged.
  {
    int vm[kTlMax], vh = 0, vt = 0;
    bool ok = true;
    vm[vt++] = (int)full;
    while (vh < vt && ok) {
      const int mask = vm[vh++];
      const int lm = T.part[mask], rm = mask ^ lm;
      if (lm == 0 || rm == 0 || (lm & ~mask)) { ok = false; break; }
      if (__popc(lm) > 1) { if (vt >= kTlMax) { ok = false; break; } vm[vt++] = lm; }
      if (__popc(rm) > 1) { if (vt >= kTlMax) { ok = false; break; } vm[vt++] = rm; }
    }
    if (!ok || n_avail != n - 1) return;
  }
  int qm[kTlMax], qn[kTlMax];
  int qh = 0, qt = 0, used = 1;
  qm[qt] = (int)full;
  qn[qt++] = avail[0];
  while (qh < qt) {
    const int mask = qm[qh], cur = qn[qh];
    qh++;
    const int lm = T.part[mask], rm = mask ^ lm;
    int li, ri;
    if (__popc(lm) == 1) li = T.act[__ffs(lm) - 1];
    else { li = avail[used++]; qm[qt] = lm; qn[qt++] = li; }
    if (__popc(rm) == 1) ri = T.act[__ffs(rm) - 1];
    else { ri = avail[used++]; qm[qt] = rm; qn[qt++] = ri; }
    Box b = box_empty();
    for (int i = 0; i < n; ++i)
      if ((mask >> i) & 1) b = box_union(b, leaf_box(T, i));
    float4* p = reinterpret_cast<float4*>(nodes + cur);
    __stcg(p, b.lo);
    __stcg(p + 1, b.hi);
    __stcg(reinterpret_cast<int2*>(&nodes[cur].left), make_int2(li, ri));
    __stcg(parents + li, cur);
    __stcg(parents + ri, cur);
  }
}

// ---------------------------------------------------------------------------------------
// Level-synchronous pass.  Any children-before-parent order gives the same tree, and nodes of
// equal height have disjoint subtrees (neither is an ancestor of the other), so each height
// is one parallel step: every lane owns one treelet and does its refit, growth, DP and rebuild
// alone, so the 32 lanes of a warp run the same 7-leaf work in step.  Heights come from the emission
// and, for a further pass, from the rebuilds of the one before; node ids are then grouped by height.
// Trees higher than kTlMaxHeight (not reachable by a Karras tree: its depth is at most the
// key bits plus 32; many passes might) fall back to the climb-ordered kernel below for the rest.
//
// A pass is bound by its scattered 32-byte sectors, so what a node carries is laid out for it: the children's
// areas lie beside their ids (a treelet grows through one sector per expansion instead of two nodes of two
// sectors), tame boxes are not refitted or rewritten at the root, and there are no parent links.  10M
// triangles, one pass, before -> with that: growth 1.60 -> 0.63 ms, heights by a climb over parent links
// 0.31 ms -> none, DP and rebuild of heights 2, 3 and 4 on 0.35, 0.55 and 1.99 -> 0.21, 0.39 and 1.50 ms;
// three passes 19.0 -> 12.1 ms, one pass at 200k 880 -> 542 us.
// ---------------------------------------------------------------------------------------
constexpr int kTlMaxHeight = 254;
constexpr uint32_t kTlTooHigh = 1u, kTlStop = 2u;  // flags of the first control word
constexpr int kLvThreads = 32;  // one warp per block; its DP table is 16 KB of shared memory

// A lane's treelet in registers (all indexing below is unrolled to constant indices).
struct RegTreelet {
  Box b[kTlMax];
  int32_t id[kTlMax];
  int n;
};

__device__ __forceinline__ int32_t reg_id(const RegTreelet& T, int i) {
  int32_t v = 0;
#pragma unroll
  for (int k = 0; k < kTlMax; ++k)
    if (k == i) v = T.id[k];
  return v;
}
__device__ __forceinline__ Box reg_union(const RegTreelet& T, uint32_t mask) {
  Box b = box_empty();
#pragma unroll
  for (int k = 0; k < kTlMax; ++k)
    if ((mask >> k) & 1u) b = box_union(b, T.b[k]);
  return b;
}

// Growth state: the leaves (ids and areas), the links of those that are inner nodes, and the expanded
// nodes in order.  Expansion s replaces leaf `slot s` by the left child and appends the right child
// as leaf s + 1; the slots, 3 bits each, say what the treelet looks like.
struct GrowTreelet {
  int32_t id[kTlMax];
  float area[kTlMax];
  Links k[kTlMax];
  int32_t en[kTlMax - 1];
  uint32_t slots;
  int n;
};

// Growth (lbvh_plus_builder.cu:73-114) from the root's links: the leaf with the largest area among the
// inner ones is expanded, the first such on ties.
__device__ __forceinline__ void reg_grow(const Node* nodes, int32_t first_leaf, int32_t root, const Links& rl,
                                         GrowTreelet& T) {
#pragma unroll
  for (int i = 0; i < kTlMax; ++i) {
    T.id[i] = first_leaf;
    T.area[i] = 0.f;
    T.k[i] = Links{0, 0, 0.f, 0.f};
  }
  T.id[0] = rl.l;
  T.id[1] = rl.r;
  T.area[0] = rl.al;
  T.area[1] = rl.ar;
  if (rl.l < first_leaf) T.k[0] = ldcg_links(nodes, rl.l);
  if (rl.r < first_leaf) T.k[1] = ldcg_links(nodes, rl.r);
  T.en[0] = root;
  T.slots = 0;
  T.n = 2;
#pragma unroll
  for (int step = 1; step < kTlMax - 1; ++step) {
    int best = -1;
    float max_area = -1.0f;
    Links x{0, 0, 0.f, 0.f};
    int32_t xid = 0;
#pragma unroll
    for (int i = 0; i <= step; ++i)
      if (T.id[i] < first_leaf && T.area[i] > max_area) {
        max_area = T.area[i];
        best = i;
        x = T.k[i];
        xid = T.id[i];
      }
    if (best < 0) break;
    T.en[step] = xid;
    T.slots |= (uint32_t)best << (3 * step);
    Links kl{0, 0, 0.f, 0.f};
    if (x.l < first_leaf) kl = ldcg_links(nodes, x.l);
    if (x.r < first_leaf) T.k[step + 1] = ldcg_links(nodes, x.r);
    T.id[step + 1] = x.r;
    T.area[step + 1] = x.ar;
#pragma unroll
    for (int i = 0; i <= step; ++i)
      if (i == best) {
        T.id[i] = x.l;
        T.area[i] = x.al;
        T.k[i] = kl;
      }
    T.n = step + 2;
  }
}

// The order in which a rebuild reuses the treelet's inner ids (:167-191): depth first from the root, the
// right child first.  Four bits each, the expansions' numbers.
__device__ __forceinline__ uint32_t reuse_order(uint32_t slots, int m) {
  uint32_t order = 0, stack = 0;  // stack: four bits per entry, the top lowest; 0 (the root) is never pushed
  int s = 0;
#pragma unroll
  for (int k = 0; k < kTlMax - 1; ++k) {
    if (k >= m) break;
    order |= (uint32_t)s << (4 * k);
    const uint32_t left = (slots >> (3 * s)) & 7u, right = (uint32_t)s + 1u;
    int l = 0, r = 0;  // the first later expansion of either child
#pragma unroll
    for (int e = kTlMax - 2; e >= 1; --e) {
      const uint32_t x = (slots >> (3 * e)) & 7u;
      if (e > s && e < m && x == left) l = e;
      if (e > s && e < m && x == right) r = e;
    }
    if (l) stack = stack << 4 | (uint32_t)l;
    if (r) stack = stack << 4 | (uint32_t)r;
    s = (int)(stack & 15u);
    stack >>= 4;
  }
  return order;
}

// The root's links for its treelet, and whether it grows at all (not where its area is NaN).  Tame boxes
// are final as they are; others are refitted (box and areas) from the children, as the reference does.
__device__ __forceinline__ Links refit_root(Node* nodes, int32_t x, bool wild, bool& expand) {
  Links k = ldcg_links(nodes, x);
  expand = true;
  if (wild) {
    const Box lb = ldcg_box(nodes, k.l), rb = ldcg_box(nodes, k.r);
    const Box box = box_union(lb, rb);
    float4* p = reinterpret_cast<float4*>(nodes + x);
    __stcg(p, box.lo);
    __stcg(p + 1, box.hi);
    k.al = box_area(lb);
    k.ar = box_area(rb);
    stcg_links(nodes, x, k);
    expand = box_area(box) > -1.0f;
  }
  return k;
}

// A root whose treelet is not rebuilt by the DP (n = 1 or 2 leaves): two leaves change places, since the
// DP's only split puts the second left.  Its height follows its children's.
__device__ __forceinline__ void finish_short(Node* nodes, uint8_t* hgt, int32_t first_leaf, int32_t x, const Links& k,
                                             bool two) {
  if (two) stcg_links(nodes, x, Links{k.r, k.l, k.ar, k.al});
  if (hgt)
    __stcg(hgt + x, (uint8_t)min(1u + max(node_height(hgt, first_leaf, k.l), node_height(hgt, first_leaf, k.r)), 255u));
}

// Areas of the subsets s < 2^nv with two or more leaves into this lane's column A (stride 32):
// the box of s is (its leaves among 3..6) U (its leaves among 0..2).  NVMAX: nv's bound.
template <int NVMAX = kTlMax>
__device__ __forceinline__ void reg_areas(const RegTreelet& T, int nv, float* A) {
  const uint32_t full = (1u << nv) - 1u;
  Box lo8[8];
  lo8[0] = box_empty();
  lo8[1] = box_union(lo8[0], T.b[0]);
  lo8[2] = box_union(lo8[0], T.b[1]);
  lo8[3] = box_union(lo8[1], T.b[1]);
  lo8[4] = box_union(lo8[0], T.b[2]);
  lo8[5] = box_union(lo8[1], T.b[2]);
  lo8[6] = box_union(lo8[2], T.b[2]);
  lo8[7] = box_union(lo8[3], T.b[2]);
  for (uint32_t hi = 0; hi * 8u <= full; ++hi) {
    Box bh = box_empty();
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (3 + j < NVMAX && ((hi >> j) & 1u)) bh = box_union(bh, T.b[3 + j]);
#pragma unroll
    for (int lo = 0; lo < 8; ++lo) {
      const uint32_t s = hi * 8u + (uint32_t)lo;
      if (s <= full && __popc(s) > 1) A[s * 32u] = box_area(box_union(bh, lo8[lo]));
    }
  }
}

// Subset DP (:119-165) by one lane for up to nv leaves, straight-line code with the costs in
// registers (treelet_dp_unrolled.cuh); this lane's column C holds the areas and receives the costs.
// Costs only, the splits looked up afterwards for the subsets that the rebuild visits: the 10M pass's
// heights from 4 on 2.53 -> 1.99 ms, three passes 21.1 -> 19.0 ms (carrying every subset's split
// took 4 operations per split in a serial chain and a store per subset).
// *of: the leaf count whose full set's best split is returned.
template <int NVMAX = kTlMax>
__device__ __forceinline__ uint32_t reg_dp(int nv, float* C, int* of) {
  *of = std::min(NVMAX, std::max(nv, 4));
  if (NVMAX <= 4 || nv <= 4) return dp_unrolled_4(C);
  if (NVMAX <= 5 || nv == 5) return dp_unrolled_5(C);
  if (NVMAX <= 6 || nv == 6) return dp_unrolled_6(C);
  return dp_unrolled_7(C);
}

// The best split of `mask` from the costs in this lane's column: the first minimum over the nonempty
// subsets of mask without its lowest member in increasing order; 0 where no split is finite.
__device__ __forceinline__ uint32_t best_split(const float* C, uint32_t mask) {
  const uint32_t delta = mask & (mask - 1u);
  uint32_t p = delta & (0u - delta), bp = 0u;
  float b = kTlInf;
  do {
    const float v = __fadd_rn(C[p * 32u], C[(mask ^ p) * 32u]);
    if (v < b) { b = v; bp = p; }
    p = (p - delta) & delta;
  } while (p);
  return bp;
}

// The subsets of a rebuilt treelet, breadth-first (:194-246): byte j of masks is the j-th subset, of lefts
// its left part; nibble j of lpos / rpos the place of that part in the queue (0: a single leaf).
struct Splits {
  unsigned long long masks, lefts;
  uint32_t lpos, rpos;
};
// split(mask): the best split of a subset.  False where one has no finite split (NaN areas).
template <typename Split>
__device__ __forceinline__ bool reg_splits(int n, Split split, Splits& Q) {
  Q.masks = (1u << n) - 1u;
  Q.lefts = 0;
  Q.lpos = Q.rpos = 0;
  uint32_t qt = 1;
#pragma unroll
  for (int j = 0; j < kTlMax - 1; ++j) {
    if (j >= n - 1) break;
    const uint32_t mask = (uint32_t)(Q.masks >> (8 * j)) & 255u;
    const uint32_t lm = split(mask), rm = mask ^ lm;
    if (lm == 0 || rm == 0 || (lm & ~mask)) return false;
    Q.lefts |= (unsigned long long)lm << (8 * j);
    if (__popc(lm) > 1) {
      Q.masks |= (unsigned long long)lm << (8 * qt);
      Q.lpos |= qt++ << (4 * j);
    }
    if (__popc(rm) > 1) {
      Q.masks |= (unsigned long long)rm << (8 * qt);
      Q.rpos |= qt++ << (4 * j);
    }
  }
  return true;
}

// Rebuild by one lane: the j-th subset of the queue gets the j-th reused id.  Children come later in the
// queue than their parents, so the nodes are written from the last: a node's areas and height then have
// its children's at hand.  root_box: the root's box is written too (a tame one is what it was).
__device__ __forceinline__ void reg_build(Node* nodes, uint8_t* hgt, int32_t first_leaf, const RegTreelet& T,
                                          const Splits& Q, const int* avail, bool root_box) {
  float area[kTlMax], narea[kTlMax - 1];
  uint32_t h[kTlMax], nh[kTlMax - 1];
#pragma unroll
  for (int i = 0; i < kTlMax; ++i) {
    area[i] = box_area(T.b[i]);
    h[i] = hgt && i < T.n ? node_height(hgt, first_leaf, T.id[i]) : 0u;
  }
#pragma unroll
  for (int j = kTlMax - 2; j >= 0; --j) {
    narea[j] = 0.f;
    nh[j] = 0;
    if (j >= T.n - 1) continue;
    const uint32_t mask = (uint32_t)(Q.masks >> (8 * j)) & 255u, lm = (uint32_t)(Q.lefts >> (8 * j)) & 255u;
    int child[2];
    float ca[2];
    uint32_t hm = 0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const uint32_t cm = s ? mask ^ lm : lm;
      const int pos = (int)(((s ? Q.rpos : Q.lpos) >> (4 * j)) & 15u), leaf = __ffs(cm) - 1;
      uint32_t ch = 0;
      child[s] = 0;
      ca[s] = 0.f;
#pragma unroll
      for (int k = 0; k < kTlMax; ++k)
        if (k == leaf) {
          child[s] = T.id[k];
          ca[s] = area[k];
          ch = h[k];
        }
#pragma unroll
      for (int k = 1; k < kTlMax - 1; ++k)
        if (k > j && k == pos) {
          child[s] = avail[k];
          ca[s] = narea[k];
          ch = nh[k];
        }
      hm = max(hm, ch);
    }
    const Box b = reg_union(T, mask);
    narea[j] = box_area(b);
    nh[j] = hm + 1u;
    if (j > 0 || root_box) {
      float4* p = reinterpret_cast<float4*>(nodes + avail[j]);
      __stcg(p, b.lo);
      __stcg(p + 1, b.hi);
    }
    stcg_links(nodes, avail[j], Links{child[0], child[1], ca[0], ca[1]});
    if (hgt) __stcg(hgt + avail[j], (uint8_t)min(nh[j], 255u));
  }
}

// Nodes per height (block histograms in shared memory, one global add per nonzero bin).
// A height past kTlMaxHeight hands this pass and the following ones to the fallback (kTlTooHigh in flags[0]).
__global__ void __launch_bounds__(256) k_tl_count(const uint8_t* __restrict__ hgt, uint32_t m, uint32_t* __restrict__ cnt,
                                                  uint32_t* __restrict__ flags) {
  after_previous();
  __shared__ uint32_t s_cnt[256];
  s_cnt[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    atomicAdd(&s_cnt[hgt[i]], 1u);
  __syncthreads();
  const uint32_t c = s_cnt[threadIdx.x];
  if (c) atomicAdd(cnt + threadIdx.x, c);
  if (c && threadIdx.x > kTlMaxHeight) atomicOr(flags, kTlTooHigh);
}

// off[h] = first list position of height h (exclusive scan of cnt over 256 heights), cursor
// copy for the scatter, off[256] = total, flags[1] = the largest height.  A build that has given up
// (any status bit: its tree may be unfinished, and growth would follow whatever its nodes hold) stops
// here: this pass and the following ones, the fallback too, leave the tree alone (kTlStop in flags[0]).
__global__ void __launch_bounds__(256) k_tl_offsets(const uint32_t* __restrict__ cnt, const uint32_t* __restrict__ status,
                                                    uint32_t* __restrict__ off, uint32_t* __restrict__ cursor,
                                                    uint32_t* __restrict__ flags) {
  after_previous();
  __shared__ uint32_t s_w[8];
  __shared__ uint32_t s_maxh;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) s_maxh = 0;
  const uint32_t v = cnt[t];
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[w] = x;
  __syncthreads();
  if (v) atomicMax(&s_maxh, (uint32_t)t);
  uint32_t before = 0;
  for (int k = 0; k < w; ++k) before += s_w[k];
  off[t] = before + x - v;
  cursor[t] = before + x - v;
  if (t == 255) off[256] = before + x;
  if (t == 0 && __ldcg(status) != 0u) atomicOr(flags, kTlStop);
  __syncthreads();
  if (t == 0) {
    flags[1] = s_maxh;
    flags[2] = 4;  // the first height of the loop (heights 1 to 3 have launches of their own)
  }
}

// Internal node ids grouped by height (order within a height is irrelevant).
__global__ void __launch_bounds__(256) k_tl_scatter(const uint8_t* __restrict__ hgt, uint32_t m,
                                                    uint32_t* __restrict__ cursor, uint32_t* __restrict__ list) {
  after_previous();
  __shared__ uint32_t s_cnt[256], s_base[256];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t h = i < m ? hgt[i] : 0u;
  const uint32_t rank = i < m ? atomicAdd(&s_cnt[h], 1u) : 0u;
  __syncthreads();
  const uint32_t c = s_cnt[threadIdx.x];
  if (c) s_base[threadIdx.x] = atomicAdd(cursor + threadIdx.x, c);
  __syncthreads();
  if (i < m) {
    const uint32_t pos = s_base[h] + rank;
    if (pos < m) list[pos] = i;
  }
}

// Per height, two kernels: k_tl_grow (latency-bound: many warps, few registers) grows each node's
// treelet and writes a descriptor; k_tl_dp (compute-bound) loads the leaf boxes, runs the DP and
// rebuilds.  Descriptors are structure-of-arrays, kTlDescWords words per
// node at stride `stride` (>= the largest height's node count): [0] n | n_avail << 8,
// [1..7] leaf ids, [8..13] reused internal ids in order.  ctl: [0] flags, [1] largest
// height, [2] current height.  at: the height, 0 for the current one.
constexpr int kGrowThreads = 128;

struct TlArgs {
  Node* nodes;
  uint8_t* hgt;  // heights, kept up to date where another pass follows (else NULL)
  int32_t first_leaf;
  const uint32_t* wild;
  const uint32_t* off;
  uint32_t* desc;
  uint32_t stride;
};

__global__ void __launch_bounds__(kGrowThreads, 8) k_tl_grow(TlArgs A, const uint32_t* __restrict__ list,
                                                             const uint32_t* __restrict__ ctl, uint32_t at) {
  after_previous();
  if (__ldcg(ctl) != 0u) return;  // too high (the fallback pass does the work) or stopped
  const uint32_t h = at ? at : __ldcg(ctl + 2);
  const uint32_t b = __ldcg(A.off + h), e = __ldcg(A.off + h + 1);
  const bool wild = __ldcg(A.wild) != 0u;
  for (uint32_t k = b + blockIdx.x * blockDim.x + threadIdx.x; k < e; k += gridDim.x * blockDim.x) {
    const int32_t x = (int32_t)__ldcg(list + k);
    bool expand;
    const Links rl = refit_root(A.nodes, x, wild, expand);
    const uint32_t q = k - b;
    if (h == 1) {  // both children are BVH leaves
      if (expand) stcg_links(A.nodes, x, Links{rl.r, rl.l, rl.ar, rl.al});
      continue;  // (no DP is launched for height 1)
    }
    GrowTreelet T;
    T.n = 1;
    if (expand) reg_grow(A.nodes, A.first_leaf, x, rl, T);
    if (T.n <= 2) {
      finish_short(A.nodes, A.hgt, A.first_leaf, x, rl, T.n == 2);
      A.desc[q] = 0u;  // nothing left for k_tl_dp
      continue;
    }
    const int m = T.n - 1;
    const uint32_t order = reuse_order(T.slots, m);
    A.desc[q] = (uint32_t)T.n | ((uint32_t)m << 8);
#pragma unroll
    for (int i = 0; i < kTlMax; ++i)
      if (i < T.n) A.desc[(size_t)(1 + i) * A.stride + q] = (uint32_t)T.id[i];
#pragma unroll
    for (int i = 0; i < kTlMax - 1; ++i) {
      if (i >= m) break;
      const int s = (int)((order >> (4 * i)) & 15u);
      int32_t id = 0;
#pragma unroll
      for (int c = 0; c < kTlMax - 1; ++c)
        if (c == s) id = T.en[c];
      A.desc[(size_t)(8 + i) * A.stride + q] = (uint32_t)id;
    }
  }
}

// A box through L1, whose line serves the second half: for kernels that write no box that they read (the treelets
// of a height are disjoint).
__device__ __forceinline__ Box ldca_box(const Node* nodes, int32_t idx) {
  const float4* p = reinterpret_cast<const float4*>(nodes + idx);
  Box b;
  b.lo = __ldca(p);
  b.hi = __ldca(p + 1);
  return b;
}

// One lane's treelet q of the current height (act: a real one): leaf ids and boxes from its
// descriptor and the nodes, subset areas and the DP in this lane's shared-memory column C
// (stride 32), then the rebuild.  The warp runs the DP variant of its largest treelet, at most
// NVMAX leaves.  Called by all 32 lanes together.
template <int NVMAX>
__device__ __forceinline__ void lane_dp(const TlArgs& A, bool wild, uint32_t q, bool act, float* C) {
  const uint32_t w0 = act ? __ldcg(A.desc + q) : 0u;
  RegTreelet T;
  T.n = (int)(w0 & 255u);
#pragma unroll
  for (int i = 0; i < kTlMax; ++i) {
    T.id[i] = i < NVMAX && i < T.n ? (int32_t)__ldcg(A.desc + (size_t)(1 + i) * A.stride + q) : 0;
    T.b[i] = i < NVMAX && i < T.n ? ldca_box(A.nodes, T.id[i]) : box_empty();
  }
  const int nv = (int)__reduce_max_sync(0xffffffffu, (uint32_t)T.n);
  if (nv < 2) return;
  reg_areas<NVMAX>(T, nv, C);
  int of;
  const uint32_t top = reg_dp<NVMAX>(nv, C, &of);
  if (T.n >= 2) {
    int avail[kTlMax];
#pragma unroll
    for (int i = 0; i < kTlMax - 1; ++i)
      avail[i] = i < NVMAX - 1 && i < T.n - 1 ? (int)__ldcg(A.desc + (size_t)(8 + i) * A.stride + q) : 0;
    const uint32_t full = (1u << of) - 1u;
    Splits Q;
    if (reg_splits(T.n, [&](uint32_t mask) { return mask == full ? top : best_split(C, mask); }, Q))
      reg_build(A.nodes, A.hgt, A.first_leaf, T, Q, avail, wild);
    else
      finish_short(A.nodes, A.hgt, A.first_leaf, avail[0], ldcg_links(A.nodes, avail[0]), false);
  }
}

// NVMAX < kTlMax: a DP for treelets of at most NVMAX leaves (heights where no more fit: height 2
// holds at most 4), compiled for fewer registers, so more warps share an SM.
template <int NVMAX>
__global__ void __launch_bounds__(kLvThreads) k_tl_dp(TlArgs A, const uint32_t* __restrict__ ctl, uint32_t at) {
  after_previous();
  __shared__ float s_cost[(1 << NVMAX) * 32];  // per-lane columns of 2^NVMAX areas, then costs
  if (__ldcg(ctl) != 0u) return;
  const uint32_t h = at ? at : __ldcg(ctl + 2);
  const uint32_t b = __ldcg(A.off + h), e = __ldcg(A.off + h + 1);
  const bool wild = __ldcg(A.wild) != 0u;
  const int lane = threadIdx.x & 31;
  // warp-uniform loop: the warp runs the DP variant of its largest treelet
  for (uint32_t kb = b + blockIdx.x * kLvThreads; kb < e; kb += gridDim.x * kLvThreads) {
    const uint32_t k = kb + lane;
    lane_dp<NVMAX>(A, wild, k - b, k < e, s_cost + lane);
  }
}

// A height where treelet sizes are mixed (height 3: most treelets have 4 or 5 leaves, few 7):
// one kernel per size class, NV = 4 (3 or 4 leaves), 5, 6, 7, each running only the
// height's treelets of its class, so a warp runs the DP its own treelets need.  Each warp scans
// R rounds of 32 nodes, packs those of its class into a shared list (ballots) and runs them 32
// at a time; R shrinks with the height's node count so that every block gets a chunk.
template <int NV>
__global__ void __launch_bounds__(kLvThreads) k_tl_dpc(TlArgs A, const uint32_t* __restrict__ ctl, uint32_t at) {
  after_previous();
  constexpr int R = 8;
  __shared__ float s_cost[(1 << NV) * 32];
  __shared__ uint32_t s_list[32 * R];
  if (__ldcg(ctl) != 0u) return;
  const uint32_t b = __ldcg(A.off + at), e = __ldcg(A.off + at + 1);
  const bool wild = __ldcg(A.wild) != 0u;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  float* C = s_cost + lane;
  const uint32_t rounds = max(1u, min((uint32_t)R, div_up(e - b, 32u * gridDim.x)));
  for (uint32_t chunk = b + blockIdx.x * (32u * rounds); chunk < e; chunk += gridDim.x * (32u * rounds)) {
    uint32_t cnt = 0;
    for (uint32_t r = 0; r < rounds; ++r) {
      const uint32_t k = chunk + r * 32u + (uint32_t)lane;
      const int n = k < e ? (int)(__ldcg(A.desc + (k - b)) & 255u) : 0;
      const bool match = n >= 2 && (n <= 4 ? 4 : n) == NV;
      const uint32_t bal = __ballot_sync(0xffffffffu, match);
      if (match) s_list[cnt + __popc(bal & lt)] = k - b;
      cnt += (uint32_t)__popc(bal);
    }
    __syncwarp();
    for (uint32_t i = 0; i < cnt; i += 32) {
      const bool act = i + (uint32_t)lane < cnt;
      lane_dp<NV>(A, wild, act ? s_list[i + lane] : 0u, act, C);
    }
    __syncwarp();  // the list is refilled by the next chunk
  }
}

// The narrow heights in one cooperative launch.  Once a height has few nodes, its launches (growth, DP) cost
// mostly their latency; k_tl_narrow runs the remaining heights, from the current one (ctl[2]) to the
// largest (ctl[1]), with a grid barrier between heights (nodes of one height have disjoint subtrees, a
// height needs all lower ones done).  Per node, one warp: lane 0 grows the treelet, seven lanes load the
// leaf boxes, the warp runs the cooperative DP, all lanes follow the splits and each writes one of the
// rebuilt nodes.  Same work and result as the per-height kernels.  A height is a chain of some ten L2
// round trips and a barrier: about 8 us (17 us with a DP whose cost loads waited for one another).
constexpr int kNarrowThreads = 256;

struct NarrowWarp {
  LaneTreelet S;
  float cost[1 << kTlMax];
  float area[1 << kTlMax];
  int32_t avail[kTlMax];
  uint8_t h[kTlMax + 1];
};

__global__ void __launch_bounds__(kNarrowThreads) k_tl_narrow(TlArgs A, const uint32_t* __restrict__ list,
                                                              uint32_t* __restrict__ ctl,
                                                              uint32_t* __restrict__ status) {
  __shared__ NarrowWarp s_warp[kNarrowThreads / 32];
  __shared__ uint32_t s_ok;
  // every block reads the same words (nothing writes them in this kernel)
  if (__ldcg(ctl) != 0u) return;  // too high (the fallback pass does the work) or stopped
  const uint32_t h0 = __ldcg(ctl + 2), h1 = __ldcg(ctl + 1);
  const bool wild = __ldcg(A.wild) != 0u;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  NarrowWarp& W = s_warp[w];
  const uint32_t gw = blockIdx.x * (kNarrowThreads / 32) + (uint32_t)w, nw = gridDim.x * (kNarrowThreads / 32);
  uint32_t nbar = 0;
  bool alone = false;
  for (uint32_t h = h0; h <= h1; ++h) {
    const uint32_t b = __ldcg(A.off + h), e = __ldcg(A.off + h + 1);
    // A height has no more nodes than the one below it: from the first that one block's warps hold on,
    // block 0 goes on alone, with block barriers.
    alone = alone || e - b <= kNarrowThreads / 32;
    if (alone && blockIdx.x != 0) return;
    for (uint32_t k = b + gw; k < e; k += alone ? kNarrowThreads / 32 : nw) {
      if (lane == 0) {
        const int32_t x = (int32_t)__ldcg(list + k);
        bool expand;
        const Links rl = refit_root(A.nodes, x, wild, expand);
        GrowTreelet T;
        T.n = 1;
        if (expand) reg_grow(A.nodes, A.first_leaf, x, rl, T);
        if (T.n <= 2) {
          finish_short(A.nodes, A.hgt, A.first_leaf, x, rl, T.n == 2);
        } else {
          const uint32_t order = reuse_order(T.slots, T.n - 1);
#pragma unroll
          for (int i = 0; i < kTlMax; ++i) W.S.act[i] = T.id[i];
#pragma unroll
          for (int i = 0; i < kTlMax - 1; ++i) W.S.exp_node[i] = T.en[i];
#pragma unroll
          for (int i = 0; i < kTlMax - 1; ++i)
            if (i < T.n - 1) W.avail[i] = W.S.exp_node[(order >> (4 * i)) & 15u];
        }
        W.S.n = T.n;
      }
      __syncwarp();
      const int n = W.S.n;
      if (n > 2) {  // uniform over the warp
        if (lane < kTlMax) {
          const Box bx = lane < n ? ldcg_box(A.nodes, W.S.act[lane]) : box_empty();
          W.S.box[0][lane] = bx.lo.x; W.S.box[1][lane] = bx.lo.y; W.S.box[2][lane] = bx.lo.z;
          W.S.box[3][lane] = bx.hi.x; W.S.box[4][lane] = bx.hi.y; W.S.box[5][lane] = bx.hi.z;
          W.h[lane] = A.hgt && lane < n ? (uint8_t)node_height(A.hgt, A.first_leaf, W.S.act[lane]) : 0;
        }
        __syncwarp();
        treelet_dp(W.S, W.cost, W.area);
        Splits Q;
        if (!reg_splits(n, [&](uint32_t mask) { return (uint32_t)W.S.part[mask]; }, Q)) {
          if (lane == 0) finish_short(A.nodes, A.hgt, A.first_leaf, W.avail[0], ldcg_links(A.nodes, W.avail[0]), false);
        } else {
          // every lane walks the queue for the heights (last first); lane j keeps node j
          uint32_t mine = 0;
          unsigned long long hq = 0;  // byte j: node j's height
          for (int j = n - 2; j >= 0; --j) {
            const uint32_t mask = (uint32_t)(Q.masks >> (8 * j)) & 255u, lm = (uint32_t)(Q.lefts >> (8 * j)) & 255u;
            const uint32_t lp = (Q.lpos >> (4 * j)) & 15u, rp = (Q.rpos >> (4 * j)) & 15u;
            const uint32_t hl = lp ? (uint32_t)(hq >> (8 * lp)) & 255u : W.h[__ffs(lm) - 1];
            const uint32_t hr = rp ? (uint32_t)(hq >> (8 * rp)) & 255u : W.h[__ffs(mask ^ lm) - 1];
            const uint32_t nh = min(1u + max(hl, hr), 255u);
            hq |= (unsigned long long)nh << (8 * j);
            if (j == lane) mine = nh;
          }
          if (lane < n - 1) {
            const uint32_t mask = (uint32_t)(Q.masks >> (8 * lane)) & 255u, lm = (uint32_t)(Q.lefts >> (8 * lane)) & 255u;
            const uint32_t rm = mask ^ lm, lp = (Q.lpos >> (4 * lane)) & 15u, rp = (Q.rpos >> (4 * lane)) & 15u;
            const int32_t cur = W.avail[lane];
            const int li = __ffs(lm) - 1, ri = __ffs(rm) - 1;
            Links out;
            out.l = lp ? W.avail[lp] : W.S.act[li];
            out.r = rp ? W.avail[rp] : W.S.act[ri];
            out.al = lp ? W.area[lm] : box_area(leaf_box(W.S, li));
            out.ar = rp ? W.area[rm] : box_area(leaf_box(W.S, ri));
            Box bx = box_empty();
            for (int i = 0; i < n; ++i)
              if ((mask >> i) & 1u) bx = box_union(bx, leaf_box(W.S, i));
            if (lane > 0 || wild) {
              float4* p = reinterpret_cast<float4*>(A.nodes + cur);
              __stcg(p, bx.lo);
              __stcg(p + 1, bx.hi);
            }
            stcg_links(A.nodes, cur, out);
            if (A.hgt) __stcg(A.hgt + cur, (uint8_t)mine);
          }
        }
      }
      __syncwarp();
    }
    if (alone) {
      __threadfence_block();
      __syncthreads();
    } else if (h < h1 && !grid_sync(ctl + 4, ++nbar * gridDim.x, status, &s_ok)) {
      return;
    }
  }
}

// End of a height: the next one, and whether the loop goes on (the graph's WHILE condition;
// the host-driven loop only advances the height).  The loop also stops at the first height of
// at most `narrow` nodes (0: never), from which k_tl_narrow goes on.
template <bool GRAPH>
__global__ void k_tl_step(uint32_t* __restrict__ ctl, const uint32_t* __restrict__ off, uint32_t narrow,
                          cudaGraphConditionalHandle handle) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const uint32_t h = ctl[2] + 1;
  ctl[2] = h;
  bool go = ctl[0] == 0u && h <= ctl[1];
  if (go && narrow && off[h + 1] - off[h] <= narrow) go = false;
  if constexpr (GRAPH) cudaGraphSetConditional(handle, go ? 1u : 0u);
}

// Parent links for the fallback; returns at once unless flags[0] is kTlTooHigh.
__global__ void __launch_bounds__(256) k_tl_parents(const Node* __restrict__ nodes, uint32_t m,
                                                    int32_t* __restrict__ parents, const uint32_t* __restrict__ flags) {
  after_previous();
  if (__ldcg(flags) != kTlTooHigh) return;
  for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < m; x += gridDim.x * blockDim.x) {
    const int2 ch = ldcg_children(nodes, (int32_t)x);
    parents[ch.x] = (int32_t)x;
    parents[ch.y] = (int32_t)x;
  }
}

// The climb-ordered pass as a fallback for trees higher than kTlMaxHeight: persistent warps
// take groups of 32 leaves.  Launched every pass; returns at once unless flags[0] is kTlTooHigh, which it
// stays for the following passes (this kernel keeps neither heights nor areas).
__global__ void __launch_bounds__(64) k_treelet_fallback(Node* __restrict__ nodes, int32_t* __restrict__ parents,
                                                         unsigned long long* __restrict__ slots,
                                                         const uint32_t* epoch_word, uint32_t round, uint32_t n,
                                                         const uint32_t* __restrict__ flags) {
  after_previous();
  __shared__ LaneTreelet S[64];
  __shared__ float s_cost[2][1 << kTlMax], s_area[2][1 << kTlMax];
  if (__ldcg(flags) != kTlTooHigh) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned long long tag = (unsigned long long)(__ldcg(epoch_word) + 0x20u + round) << 32;
  LaneTreelet& mine = S[threadIdx.x];
  for (uint32_t base = (blockIdx.x * 2 + w) * 32u; base < n; base += gridDim.x * 64u) {
    const uint32_t i = base + lane;
    bool active = i < n;
    int32_t idx = (int32_t)(n - 1 + i);
    while (__any_sync(0xffffffffu, active)) {
      bool work = false;
      if (active) {
        if (idx == 0) {
          active = false;
        } else {
          int32_t parent = __ldcg(parents + idx);
          __threadfence();
          unsigned long long old = atomicExch(slots + parent, tag | 1u);
          if ((old & 0xffffffff00000000ull) != tag) {
            active = false;
          } else {
            __threadfence();
            int2 ch = ldcg_children(nodes, parent);
            Box b = box_union(ldcg_box(nodes, ch.x), ldcg_box(nodes, ch.y));
            float4* p = reinterpret_cast<float4*>(nodes + parent);
            __stcg(p, b.lo);
            __stcg(p + 1, b.hi);
            idx = parent;
            work = true;
          }
        }
      }
      if (work) treelet_grow(nodes, idx, mine);
      __syncwarp();
      uint32_t ballot = __ballot_sync(0xffffffffu, work && mine.n >= 2);
      while (ballot) {
        const int src = __ffs(ballot) - 1;
        ballot &= ballot - 1;
        treelet_dp(S[w * 32 + src], s_cost[w], s_area[w]);
      }
      __syncwarp();
      if (work) treelet_rebuild(nodes, parents, idx, mine);
      __threadfence();
    }
  }
}

static int g_dp_grid[64] = {};      // resident blocks of k_tl_dp per device
static int g_dp4_grid[64] = {};     // resident blocks of k_tl_dp<4> per device
static int g_dpc_grid[64][4] = {};  // resident blocks of k_tl_dpc<4..7> per device
static int g_narrow_grid[64] = {};  // resident blocks of k_tl_narrow per device (-1: no cooperative launch)

// The loop over heights as a graph: WHILE(cond) { grow; dp; step }.
static cudaError_t make_height_graph(const TlArgs& A, const uint32_t* list, uint32_t* ctl, uint32_t grow_grid,
                                     uint32_t dp_grid, uint32_t narrow, cudaGraphExec_t* out) {
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaGraphCreate(&g, 0);
  if (e != cudaSuccess) return e;
  cudaStream_t cs = nullptr;
  do {
    cudaGraphConditionalHandle handle;
    if ((e = cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault)) != cudaSuccess) break;
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    if ((e = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &cp)) != cudaSuccess) break;
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    if ((e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) != cudaSuccess) break;
    if ((e = cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
      break;
    k_tl_grow<<<grow_grid, kGrowThreads, 0, cs>>>(A, list, ctl, 0u);
    k_tl_dp<kTlMax><<<dp_grid, kLvThreads, 0, cs>>>(A, ctl, 0u);
    k_tl_step<true><<<1, 32, 0, cs>>>(ctl, A.off, narrow, handle);
    cudaGraph_t captured = nullptr;
    const cudaError_t e2 = cudaGetLastError();
    e = cudaStreamEndCapture(cs, &captured);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) break;
    e = cudaGraphInstantiate(out, g, 0);
  } while (false);
  if (cs) cudaStreamDestroy(cs);
  cudaGraphDestroy(g);
  return e;
}

cudaError_t treelet_rounds_run(Workspace& ws, uint32_t n, int rounds, cudaStream_t st, int fb, bool host_loop) {
  if (n < 2) return cudaSuccess;
  ScratchLayout L = scratch_layout(ws.cap_n);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  int sms = 0;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if (!g_dp_grid[dev]) {
    int per_sm = 0;
    // Registers (241) leave k_tl_dp<7> eight blocks per SM; the carve-out that comes with them is 164 KB and leaves L1
    // the rest for the lines of the boxes' loads.  132 KB, seven blocks, take longer (one pass over 10M 3,836 ->
    // 3,913 us); all memory shared, or twelve blocks in fewer registers, longer still.
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tl_dp<kTlMax>, kLvThreads, 0)) != cudaSuccess)
      return e;
    g_dp_grid[dev] = std::max(1, per_sm * sms);
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tl_dp<4>, kLvThreads, 0)) != cudaSuccess) return e;
    g_dp4_grid[dev] = std::max(1, per_sm * sms);
    const void* dpc[4] = {reinterpret_cast<const void*>(k_tl_dpc<4>), reinterpret_cast<const void*>(k_tl_dpc<5>),
                          reinterpret_cast<const void*>(k_tl_dpc<6>), reinterpret_cast<const void*>(k_tl_dpc<7>)};
    for (int c = 0; c < 4; ++c) {
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dpc[c], kLvThreads, 0)) != cudaSuccess) return e;
      g_dpc_grid[dev][c] = std::max(1, per_sm * sms);
    }
  }
  if (!g_narrow_grid[dev]) {
    int coop = 0, per_sm = 0;
    if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tl_narrow, kNarrowThreads, 0)) != cudaSuccess)
      return e;
    g_narrow_grid[dev] = coop && per_sm > 0 ? per_sm * sms : -1;
  }
  // heights of at most `narrow` nodes (two per warp of the cooperative grid) run in k_tl_narrow
  const uint32_t narrow =
      !host_loop && g_narrow_grid[dev] > 0 ? 2u * (uint32_t)g_narrow_grid[dev] * (kNarrowThreads / 32) : 0u;
  // scratch: the id list in the idle value buffer, descriptors in the triangle boxes (32 B per triangle; a
  // height has at most n/2 nodes), the fallback's parent links in the idle key buffer, counters / offsets /
  // control words in the sort histogram words
  uint32_t* list = ws.vals[fb ^ 1];
  int32_t* parents = static_cast<int32_t*>(ws.keys[fb ^ 1]);
  const uint32_t stride = std::max<uint32_t>(n / 2, 1);
  uint32_t* cnt = ws.scratch + L.hist;       // 256
  uint32_t* off = cnt + 256;                 // 257
  uint32_t* cursor = off + 264;              // 256
  uint32_t* ctl = cursor + 256;              // [0] flags, [1] largest height, [2] current height
  static_assert(kTlCtlWord == 256 + 264 + 256, "control words of the treelet pass");
  static_assert(kTlCtlWord + 8 <= (size_t)kMaxPasses * 256, "treelet words fit the histogram area");
  TlArgs A;
  A.nodes = ws.nodes;
  A.first_leaf = (int32_t)(n - 1);
  A.wild = ws.scratch + L.wild;
  A.off = off;
  A.desc = reinterpret_cast<uint32_t*>(ws.boxes);
  A.stride = stride;
  const uint32_t* epoch = ws.scratch + L.epoch;
  const uint32_t grow_grid = std::max<uint32_t>(1, std::min<uint32_t>(div_up(stride, kGrowThreads), sms * 16));
  if (host_loop && !ws.ploc_host && (e = cudaMallocHost(&ws.ploc_host, 64)) != cudaSuccess) return e;
  const auto kept = [&](int round) { return round + 1 < rounds ? ws.heights : nullptr; };
  // one loop graph per choice of keeping the heights: [1] for a pass that another follows
  for (int keep = rounds > 1 ? 1 : 0; keep >= 0 && !host_loop; --keep) {
    if (ws.tl_exec[keep] && ws.tl_key_n == n && ws.tl_key_list == list) continue;
    for (cudaGraphExec_t& x : ws.tl_exec) {
      if (x) cudaGraphExecDestroy(x);
      x = nullptr;
    }
    for (int k = 0; k <= (rounds > 1 ? 1 : 0); ++k) {
      A.hgt = k ? ws.heights : nullptr;
      if ((e = make_height_graph(A, list, ctl, grow_grid, (uint32_t)g_dp_grid[dev], narrow, &ws.tl_exec[k])) != cudaSuccess)
        return e;
    }
    ws.tl_key_n = n;
    ws.tl_key_list = list;
  }
  ws.tl_narrow = narrow != 0;
  for (int r = 0; r < rounds && r + 1 < 0x20; ++r) {
    A.hgt = kept(r);
    if (r == 0) {  // the counts, the offsets and the control words ([0] stays for all passes)
      if ((e = cudaMemsetAsync(cnt, 0, (kTlCtlWord + 8) * 4, st)) != cudaSuccess) return e;
    } else {
      if ((e = cudaMemsetAsync(cnt, 0, 256 * 4, st)) != cudaSuccess) return e;
      if ((e = cudaMemsetAsync(ctl + 1, 0, 7 * 4, st)) != cudaSuccess) return e;  // [4]: k_tl_narrow's barrier
    }
    k_tl_count<<<std::max<uint32_t>(1, std::min<uint32_t>(div_up(n - 1, 256), sms * 8)), 256, 0, st>>>(ws.heights, n - 1,
                                                                                                      cnt, ctl);
    const uint32_t* clist = list;
    const uint32_t* cctl = ctl;
    // early starts save each launch's latency; the grids of large builds take room that the one before still
    // has use for (one pass: 200,000 triangles 411 us against 427, 1M 747 / 770, 10M 3,817 / 3,806)
    const auto launch = [&](auto kernel, uint32_t grid, uint32_t block, size_t smem, cudaStream_t s, auto... args) {
      return launch_after(ws.alone && n < 2000000u, kernel, grid, block, smem, s, args...);
    };
    e = launch(k_tl_offsets, 1, 256, 0, st, cnt, ws.scratch + L.status, off, cursor, ctl);
    if (e == cudaSuccess) e = launch(k_tl_scatter, div_up(n - 1, 256), 256, 0, st, ws.heights, n - 1, cursor, list);
    // heights 1 to 3 first: every height-1 treelet has two leaves and is finished by the growth
    // kernel (in the first pass by the emission); height 2 holds at most 4 leaves and takes the smaller
    // DP; height 3 mixes treelet sizes (mostly 4 and 5 leaves, few 7) and runs one DP per size class, where
    // there are more of them than one round of the general DP's blocks holds (200,000 triangles: four
    // launches 47 us, one of the general DP 19)
    if (e == cudaSuccess && r > 0) e = launch(k_tl_grow, grow_grid, kGrowThreads, 0, st, A, clist, cctl, 1u);
    if (e == cudaSuccess) e = launch(k_tl_grow, grow_grid, kGrowThreads, 0, st, A, clist, cctl, 2u);
    if (e == cudaSuccess) e = launch(k_tl_dp<4>, g_dp4_grid[dev], kLvThreads, 0, st, A, cctl, 2u);
    if (e == cudaSuccess) e = launch(k_tl_grow, grow_grid, kGrowThreads, 0, st, A, clist, cctl, 3u);
    if (e != cudaSuccess) return e;
    ws.tl_dp3 = n / 8 <= (uint32_t)g_dp_grid[dev] * kLvThreads ? 1 : 4;
    if (ws.tl_dp3 == 1) {
      e = launch(k_tl_dp<kTlMax>, g_dp_grid[dev], kLvThreads, 0, st, A, cctl, 3u);
    } else {
      e = launch(k_tl_dpc<4>, g_dpc_grid[dev][0], kLvThreads, 0, st, A, cctl, 3u);
      if (e == cudaSuccess) e = launch(k_tl_dpc<5>, g_dpc_grid[dev][1], kLvThreads, 0, st, A, cctl, 3u);
      if (e == cudaSuccess) e = launch(k_tl_dpc<6>, g_dpc_grid[dev][2], kLvThreads, 0, st, A, cctl, 3u);
      if (e == cudaSuccess) e = launch(k_tl_dpc<7>, g_dpc_grid[dev][3], kLvThreads, 0, st, A, cctl, 3u);
    }
    if (e != cudaSuccess) return e;
    if (host_loop) {
      // read the largest height (and the too-high flag) once, then one grow + dp per height
      if ((e = cudaMemcpyAsync(ws.ploc_host, ctl, 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
          (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return e;
      const uint32_t maxh = ws.ploc_host[0] ? 0u : ws.ploc_host[1];
      for (uint32_t h = 4; h <= maxh; ++h) {
        k_tl_grow<<<grow_grid, kGrowThreads, 0, st>>>(A, list, ctl, 0u);
        k_tl_dp<kTlMax><<<g_dp_grid[dev], kLvThreads, 0, st>>>(A, ctl, 0u);
        k_tl_step<false><<<1, 32, 0, st>>>(ctl, off, 0u, cudaGraphConditionalHandle{});
      }
    } else {
      if ((e = cudaGraphLaunch(ws.tl_exec[A.hgt ? 1 : 0], st)) != cudaSuccess) return e;
      if (narrow) {  // the remaining heights, from where the graph's loop stopped
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((uint32_t)g_narrow_grid[dev]);
        cfg.blockDim = dim3(kNarrowThreads);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = ws.no_cooperative ? cudaErrorNotSupported
                              : cudaLaunchKernelEx(&cfg, k_tl_narrow, A, (const uint32_t*)list, ctl,
                                                   ws.scratch + L.status);
        if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
          // no co-resident grid (a client limited to part of the GPU, or asked for): the
          // remaining heights as one grow + dp launch each, driven from the host
          (void)cudaGetLastError();
          ws.tl_narrow = false;
          if (!ws.ploc_host && (e = cudaMallocHost(&ws.ploc_host, 64)) != cudaSuccess) return e;
          if ((e = cudaMemcpyAsync(ws.ploc_host, ctl, 12, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
              (e = cudaStreamSynchronize(st)) != cudaSuccess)
            return e;
          if (!ws.ploc_host[0])
            for (uint32_t h = ws.ploc_host[2]; h <= ws.ploc_host[1]; ++h) {
              k_tl_grow<<<grow_grid, kGrowThreads, 0, st>>>(A, list, ctl, 0u);
              k_tl_dp<kTlMax><<<g_dp_grid[dev], kLvThreads, 0, st>>>(A, ctl, 0u);
              k_tl_step<false><<<1, 32, 0, st>>>(ctl, off, 0u, cudaGraphConditionalHandle{});
            }
        } else if (e != cudaSuccess) {
          return e;
        }
      }
    }
    e = launch(k_tl_parents, sms * 8, 256, 0, st, ws.nodes, n - 1, parents, cctl);
    if (e == cudaSuccess)
      e = launch(k_treelet_fallback, sms * 8, 64, 0, st, ws.nodes, parents, ws.slots, epoch, (uint32_t)r, n, cctl);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

// k_tl_offsets over counts of zero and the given status word.
__device__ uint32_t g_tl_selftest[256 + 264 + 256 + 8 + 8];

cudaError_t treelet_stop_selftest(uint32_t status, bool* stops) {
  *stops = false;
  void* p = nullptr;
  cudaStream_t st = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_tl_selftest);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  uint32_t *cnt = static_cast<uint32_t*>(p), *off = cnt + 256, *cursor = off + 264, *ctl = cursor + 256, *word = ctl + 8;
  uint32_t flags = 0;
  e = cudaMemsetAsync(p, 0, sizeof(g_tl_selftest), st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(word, &status, 4, cudaMemcpyHostToDevice, st);
  k_tl_offsets<<<1, 256, 0, st>>>(cnt, word, off, cursor, ctl);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&flags, ctl, 4, cudaMemcpyDeviceToHost, st);
  const cudaError_t e2 = cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  *stops = (flags & kTlStop) != 0;
  return e != cudaSuccess ? e : e2;
}

}  // namespace bvhgb

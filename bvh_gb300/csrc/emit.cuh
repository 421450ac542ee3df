// emit.cuh -- bottom-up Karras hierarchy + refit, shared by single-mesh and batched builds.
//
// Reference: kBuildInternalNodes_nt (src/cuda/lbvh_builder.cu:183-229), kInitLeafNodes_nt
// (:231-241) and kRefitHierarchy_nt (:243-274); same node ids, children and boxes.
//
// Step 1: D[k] = delta(k, k+1) + 1 for adjacent sorted positions, one byte each (delta_nt,
// lbvh_builder.cu:33-43: common-prefix length of the codes, or 32/64 + clz(origIdx_k ^
// origIdx_k+1) when the codes are equal; 0 marks a segment boundary).  30-bit codes: k_emit
// computes them for its tile; 60/63-bit codes: the run fix-up writes them; batched keys:
// k_delta_seg_split.
// Step 2 (k_emit): one thread per sorted position climbs; merges whose two children belong to
// threads of one block happen in shared memory.  Nodes whose sibling is built by another block,
// and nodes still climbing after kEmitMaxSteps levels, are listed as a frontier, from which
// k_emit_climb continues through global rendezvous words.  A node with range [f, l] has its
// parent's split on the side whose adjacent delta is larger (Apetrei 2014): gamma = l when
// D[l] > D[f-1], else gamma = f-1.  The second child to reach gamma's rendezvous word completes
// the parent.  Karras ids: leaf i -> n-1+i, a left child's id is its last index, a right
// child's its first, the root is 0.  Segments (batched meshes) number their nodes from their
// own base and see delta = -1 across their boundaries.
#pragma once
#include "climb_message.h"
#include "common.cuh"

namespace bvhgb {

// Single mesh: one segment [0, n) with node base 0; original indices are global.
struct SegSingle {
  uint32_t n;
  __device__ __forceinline__ void get(uint32_t /*i*/, uint32_t& off, uint32_t& cnt, uint32_t& nbase) const {
    off = 0;
    cnt = n;
    nbase = 0;
  }
  __device__ __forceinline__ uint32_t mesh_of_key(unsigned long long) const { return 0; }
};

// Batched meshes: key = mesh << 30 | code30; mesh m owns sorted positions
// [offsets[m], offsets[m+1]) and node ids [2*offsets[m] - m, ...).
// hkeys = (mesh << 30 | code30) >> shift0, so the mesh is hkeys >> (30 - shift0).
struct SegBatch {
  const uint32_t* hkeys;
  const uint32_t* offsets;
  int mshift;  // 30 - shift0
  __device__ __forceinline__ void get(uint32_t i, uint32_t& off, uint32_t& cnt, uint32_t& nbase) const {
    const uint32_t m = __ldg(hkeys + i) >> mshift;
    off = __ldg(offsets + m);
    cnt = __ldg(offsets + m + 1) - off;
    nbase = 2 * off - m;
  }
};

// In-tile climbs stop after this many levels and continue in k_emit_climb (k_emit's max_steps): the longest
// chain of a block no longer holds its 512 threads.  Fewer levels leave more to k_emit_climb, which pays
// while its chains' latency is what a build waits for (100,000 triangles: 4 levels 59.3 us, 5 59.7, 8 63.9; 1M
// 155 / 154 / 160; 3M 5 345, 8 342; 10M 1,152 / 1,096 / 1,029).
constexpr uint32_t kEmitMaxSteps = 8;
inline uint32_t emit_max_steps(uint32_t n) { return n < 2000000u ? 5u : kEmitMaxSteps; }
constexpr uint32_t kEmitTile = 512;  // sorted positions (threads) per k_emit block

__device__ __forceinline__ void store_node(Node* nodes, uint32_t idx, const Box& b, int32_t l, int32_t r, int32_t aux0) {
  float4* p = reinterpret_cast<float4*>(nodes + idx);
  __stcg(p, b.lo);
  __stcg(p + 1, b.hi);
  __stcg(reinterpret_cast<int4*>(p + 2), make_int4(l, r, aux0, 0));
}
__device__ __forceinline__ Box load_node_box(const Node* nodes, uint32_t idx) {
  const float4* p = reinterpret_cast<const float4*>(nodes + idx);
  Box b;
  b.lo = __ldcg(p);
  b.hi = __ldcg(p + 1);
  return b;
}

__device__ __forceinline__ uint32_t atom_or_acq_rel_cta(uint32_t* p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.acq_rel.cta.shared::cta.or.b32 %0, [%1], %2;"
               : "=r"(old)
               : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v)
               : "memory");
  return old;
}

__device__ __forceinline__ unsigned long long atom_exch_relaxed(unsigned long long* p, unsigned long long v) {
  unsigned long long old;
  asm volatile("atom.relaxed.gpu.global.exch.b64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
  return old;
}

// Batched meshes: keys mesh << 30 | code30 held split as hk = key >> shift0 (sorted) and lows =
// key & (2^shift0 - 1) by original index.  delta = -1 across meshes, the clz of the 30-bit code
// XOR within a mesh, 32 + clz of the in-mesh indices' XOR for equal codes.
static __global__ void __launch_bounds__(256)
    k_delta_seg_split(const uint32_t* __restrict__ hk, const uint32_t* __restrict__ vals,
                      const uint32_t* __restrict__ lows, const uint32_t* __restrict__ offsets, int shift0,
                      uint8_t* __restrict__ D, uint32_t n) {
  after_previous();
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k + 1 >= n) return;
  const uint32_t a = __ldg(hk + k), b = __ldg(hk + k + 1);
  const uint32_t ma = a >> (30 - shift0), mb = b >> (30 - shift0);
  int d;
  if (ma != mb) {
    d = -1;
  } else if (a != b) {
    d = __clz((uint32_t)((unsigned long long)(a ^ b) << shift0));
  } else {
    const uint32_t va = __ldg(vals + k), vb = __ldg(vals + k + 1);
    const uint32_t la = shift0 ? __ldg(lows + va) : 0u, lb = shift0 ? __ldg(lows + vb) : 0u;
    const uint32_t off = __ldg(offsets + ma);
    d = la != lb ? __clz(la ^ lb) : 32 + __clz((va - off) ^ (vb - off));
  }
  D[k] = (uint8_t)(d + 1);
}

// Delta bytes increase strictly from a node to its inner children and take at most 63 values from the code (one
// per bit) and 32 from the index that ties are broken by, so no node of an emitted tree is higher than
// this: it fits the byte that carries it.
constexpr uint32_t kMaxTreeHeight = 63 + 32;
static_assert(kMaxTreeHeight < 255, "a height takes one byte, 255 means higher");

// Climb state of one lane: the node it currently owns covers sorted positions [f, l].  al, ar (its
// children's areas) and h (its height) are kept for LBVH+ alone.
struct Climb {
  uint32_t f, l;
  Box box;
  int32_t lc, rc, my;
  float al, ar;
  uint32_t h;
  bool internal;
};

// 16 bytes read or written as one (b128 accesses are single-copy atomic).
__device__ __forceinline__ float4 ld_relaxed16(const float4* p) {
  unsigned long long x, y;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(x), "=l"(y)
               : "l"(p)
               : "memory");
  return make_float4(__uint_as_float((uint32_t)x), __uint_as_float((uint32_t)(x >> 32)), __uint_as_float((uint32_t)y),
                     __uint_as_float((uint32_t)(y >> 32)));
}
__device__ __forceinline__ void st_relaxed16(float4* p, float4 v) {
  const unsigned long long x = (unsigned long long)__float_as_uint(v.y) << 32 | __float_as_uint(v.x),
                           y = (unsigned long long)__float_as_uint(v.w) << 32 | __float_as_uint(v.z);
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
               "l"(x), "l"(y)
               : "memory");
}

// PLUS: what the treelet passes read of a node besides its box -- the children's areas beside their ids
// (one 16-byte load when a treelet grows through the node) and its height.
template <bool PLUS>
__device__ __forceinline__ void write_internal(Node* nodes, uint8_t* hgt, uint32_t nb, int32_t my, const Climb& c) {
  if (!PLUS) {
    store_node(nodes, nb + (uint32_t)my, c.box, c.lc, c.rc, -1);
    return;
  }
  float4* p = reinterpret_cast<float4*>(nodes + nb + (uint32_t)my);
  __stcg(p, c.box.lo);
  __stcg(p + 1, c.box.hi);
  __stcg(reinterpret_cast<int4*>(p + 2), make_int4(c.lc, c.rc, __float_as_int(c.al), __float_as_int(c.ar)));
  __stcg(hgt + nb + (uint32_t)my, (uint8_t)min(c.h, 255u));
}

// The lane's node becomes the parent of itself and its sibling `sib` (height hs), the right one when is_left.
// PLUS: the first treelet pass turns the children of a node of height 1 round (its two-leaf treelet's
// only split puts the second leaf left; not where the area is NaN); here they are written that way at once.
template <bool PLUS>
__device__ __forceinline__ void climb_merge(Climb& c, bool is_left, int32_t sib_id, const Box& sib, uint32_t hs) {
  if (PLUS) {
    const float mine = box_area(c.box), other = box_area(sib);
    c.al = is_left ? mine : other;
    c.ar = is_left ? other : mine;
  }
  if (is_left) {
    c.lc = c.my;
    c.rc = sib_id;
    c.box = box_union(c.box, sib);
  } else {
    c.lc = sib_id;
    c.rc = c.my;
    c.box = box_union(sib, c.box);
  }
  if (PLUS) {
    c.h = 1u + max(c.h, hs);
    if (c.h == 1u && box_area(c.box) > -1.0f) {
      const int32_t t = c.lc;
      c.lc = c.rc;
      c.rc = t;
      const float u = c.al;
      c.al = c.ar;
      c.ar = u;
    }
  }
}

__device__ __forceinline__ void clear_padding(Node* nodes, uint32_t idx) {
  __stcg(&nodes[idx].lo.w, 0.f);
  __stcg(&nodes[idx].hi.w, 0.f);
}

// T sorted positions per block, one thread each (a larger block leaves fewer nodes whose sibling
// lies in another block to the frontier pass).
// KEYS30: the tile's delta bytes are computed here from the sorted 30-bit keys (the delta_nt
// rule, as k_delta) and written to D for k_emit_climb; otherwise they are read from D.
// CLEAR: the node memory is a caller's and may hold anything; the padding of the nodes that no climb in the
// tile writes is cleared, since k_emit_climb reads it (100,000 triangles 0.4 us; 10M 24, 29M in 1,024 meshes
// 104, which is why a workspace's memory is cleared when it is allocated and kept so).
template <typename Seg, bool PLUS, uint32_t T = 256, bool KEYS30 = false, bool CLEAR = false>
__global__ void __launch_bounds__(T, 2048 / T) k_emit(uint8_t* __restrict__ D, const uint32_t* __restrict__ keys30,
                                            const uint32_t* __restrict__ vals,
                                            const Box* __restrict__ tri_boxes, Node* __restrict__ nodes,
                                            uint32_t n, Seg seg, uint32_t* __restrict__ out_idx,
                                            uint2* __restrict__ frontier, uint32_t* __restrict__ frontier_count,
                                            uint32_t max_steps, unsigned long long* __restrict__ stamps,
                                            uint8_t* __restrict__ hgt) {
  // D of positions bbase-1 .. bbase+T-1 (0 outside [0, n-1) : a segment boundary)
  __shared__ uint8_t s_D[T + 1];
  // KEYS30: keys and values of positions bbase-1 .. bbase+T
  __shared__ uint32_t s_k[KEYS30 ? T + 2 : 1], s_v[KEYS30 ? T + 2 : 1];
  // rendezvous slot k <-> split gamma = bbase + k: one side per child (0 left, 1 right); the
  // child's box with its id in lo.w and its far end (f of a left child, l of a right child) in hi.w
  __shared__ uint32_t s_flag[T];
  __shared__ float4 s_lo[2][T];
  __shared__ float4 s_hi[2][T];
  __shared__ uint8_t s_h[2][PLUS ? T : 1];  // the child's height
  __shared__ uint8_t s_written[CLEAR ? T : 1];  // the inner node of position bbase + k was written here
  const uint32_t tid = threadIdx.x;
  const uint32_t i = blockIdx.x * T + tid;
  const uint32_t bbase = blockIdx.x * T;  // sorted position of thread 0
  s_flag[tid] = 0;
  if (CLEAR) s_written[tid] = 0;
  after_previous();
  stage_stamp(stamps, 3);
  bool active = i < n;
  uint32_t off = 0, cnt = 1, nb = 0;
  Climb c;
  c.f = c.l = i;
  c.lc = c.rc = -1;
  c.internal = false;
  c.my = 0;
  c.h = 0;
  if (active) {
    seg.get(i, off, cnt, nb);
    const uint32_t prim_g = __ldcg(vals + i);
    const uint32_t prim = prim_g - off;  // original index within the mesh
    if (out_idx) out_idx[i] = prim;
    c.box = ld_box_cg(tri_boxes + prim_g);
    c.my = (int32_t)(cnt - 1) + (int32_t)(i - off);
    store_node(nodes, nb + (uint32_t)c.my, c.box, (int32_t)(prim | kLeafBit), -1, -1);
    if (cnt == 1) active = false;  // a one-triangle mesh: the leaf is the root
    if (KEYS30) {
      s_k[tid + 1] = __ldcg(keys30 + i);
      s_v[tid + 1] = prim_g;
    }
  }
  if (KEYS30) {
    if (tid == 0 && bbase > 0) {
      s_k[0] = __ldcg(keys30 + bbase - 1);
      s_v[0] = __ldcg(vals + bbase - 1);
    }
    if (tid == T - 1 && bbase + T < n) {
      s_k[T + 1] = __ldcg(keys30 + bbase + T);
      s_v[T + 1] = __ldcg(vals + bbase + T);
    }
    __syncthreads();
    // s_D[k] = D[bbase - 1 + k]; position j and j + 1 sit at s_k[k], s_k[k + 1]
    for (uint32_t k = tid; k <= T; k += T) {
      const int64_t j = (int64_t)bbase - 1 + k;
      uint8_t d = 0;
      if (j >= 0 && j + 1 < (int64_t)n) {
        const uint32_t a = s_k[k], b = s_k[k + 1];
        d = (uint8_t)((a == b ? 32 + __clz(s_v[k] ^ s_v[k + 1]) : __clz(a ^ b)) + 1);
        if (k >= 1) D[j] = d;  // the tile's own positions bbase .. bbase + T - 1
      }
      s_D[k] = d;
    }
  } else {
    const int64_t j = (int64_t)bbase - 1 + tid;
    s_D[tid] = (j >= 0 && j + 1 < (int64_t)n) ? __ldg(D + j) : (uint8_t)0;
    if (tid == 0) {
      const uint64_t jl = (uint64_t)bbase + T - 1;
      s_D[T] = jl + 1 < n ? __ldg(D + jl) : (uint8_t)0;
    }
  }
  __syncthreads();
  // ---- climb inside the block: the second child to reach a split completes the parent ----
  // A node [f, l] with both ends in this block reads D[f-1] and D[l] from s_D; its parent's
  // split is gamma = l (it is the left child) when D[l] > D[f-1], else gamma = f-1.
  bool to_frontier = false;
  for (uint32_t step = 0; active; ++step) {
    const int dl = (int)s_D[c.f - bbase] - 1;
    const int dr = (int)s_D[c.l - bbase + 1] - 1;
    if (dl < 0 && dr < 0) {  // segment root
      write_internal<PLUS>(nodes, hgt, nb, 0, c);
      break;
    }
    const bool is_left = dr > dl;
    const uint32_t gamma = is_left ? c.l : c.f - 1;
    const bool pending = c.internal;  // complete; its id is known now: a left child is named by its last index
    if (pending) c.my = (int32_t)((is_left ? c.l : c.f) - off);
    if (CLEAR && pending) s_written[(is_left ? c.l : c.f) - bbase] = 1;  // (below, on either way)
    // sibling starts outside the block, or the climb has gone max_steps levels: the node
    // continues in k_emit_climb, so that one long chain does not hold the block
    if (step >= max_steps || (is_left ? gamma + 1 >= bbase + T : gamma < bbase)) {
      if (pending) write_internal<PLUS>(nodes, hgt, nb, c.my, c);
      to_frontier = true;
      break;
    }
    const uint32_t k = gamma - bbase;
    const int side = is_left ? 0 : 1;
    s_lo[side][k] = make_float4(c.box.lo.x, c.box.lo.y, c.box.lo.z, __int_as_float(c.my));
    s_hi[side][k] = make_float4(c.box.hi.x, c.box.hi.y, c.box.hi.z, __uint_as_float(is_left ? c.f : c.l));
    if (PLUS) s_h[side][k] = (uint8_t)c.h;  // (at most kMaxTreeHeight)
    // release: the slot is visible before the flag bit; acquire: the sibling's slot is read after
    const uint32_t prev = atom_or_acq_rel_cta(&s_flag[k], 1u << side);
    if (pending) write_internal<PLUS>(nodes, hgt, nb, c.my, c);
    if (prev == 0u) break;  // first to arrive
    const float4 a = s_lo[side ^ 1][k], b = s_hi[side ^ 1][k];
    Box sb;
    sb.lo = make_float4(a.x, a.y, a.z, 0.f);
    sb.hi = make_float4(b.x, b.y, b.z, 0.f);
    const uint32_t hs = PLUS ? s_h[side ^ 1][k] : 0u;
    if (is_left) {
      c.l = __float_as_uint(b.w);
      climb_merge<PLUS>(c, true, __float_as_int(a.w), sb, hs);
    } else {
      c.f = __float_as_uint(b.w);
      climb_merge<PLUS>(c, false, __float_as_int(a.w), sb, hs);
    }
    c.internal = true;
  }
  __syncthreads();
  if (CLEAR && i < n && i - off + 1 < cnt && !s_written[tid]) clear_padding(nodes, nb + (i - off));
  // ---- finished nodes whose parent needs a sibling built elsewhere continue in k_emit_climb:
  // those stopped at the block edge and those whose in-block sibling never completed ----
  uint2 fr0 = make_uint2(c.f, c.l), fr1 = make_uint2(0u, 0u);
  uint32_t nf = to_frontier ? 1u : 0u;
  if (tid < T - 1) {
    const uint32_t fl = s_flag[tid];
    const uint32_t g = bbase + tid;
    uint2 e = fl == 1u ? make_uint2(__float_as_uint(s_hi[0][tid].w), g)
                       : make_uint2(g + 1, __float_as_uint(s_hi[1][tid].w));
    if (fl == 1u || fl == 2u) {
      if (nf) fr1 = e;
      else fr0 = e;
      ++nf;
    }
  }
  __shared__ uint32_t s_count, s_base;
  if (tid == 0) s_count = 0;
  __syncthreads();
  uint32_t slot_in_block = 0;
  if (nf) slot_in_block = atomicAdd(&s_count, nf);
  __syncthreads();
  if (tid == 0 && s_count) s_base = atomicAdd(frontier_count, s_count);
  __syncthreads();
  if (nf) frontier[s_base + slot_in_block] = fr0;
  if (nf > 1) frontier[s_base + slot_in_block + 1] = fr1;
}

constexpr uint32_t kClimbSpins = 1u << 22;  // re-reads of a node whose writer has announced it

// The node c, a left child (LEFT) or a right one, and its sibling, announced by `old`, become their parent; dfar
// becomes the delta byte past the sibling's far end.  slo, shi: the sibling's corners as read last, if it is
// the internal node `sib`.  False where they did not arrive.  (One body per side: with selects in place of
// branches, the loads wait for each other.)
template <bool PLUS, bool LEFT>
__device__ __forceinline__ bool climb_join(Climb& c, uint32_t& dfar, unsigned long long old, uint32_t sib, float4 slo,
                                           float4 shi, uint32_t here, uint32_t g, uint32_t off, uint32_t cnt,
                                           uint32_t nb, uint32_t n, uint32_t epoch, uint32_t mark, uint32_t limit,
                                           const uint8_t* __restrict__ D, Node* nodes, const uint8_t* hgt) {
  const uint32_t other = (uint32_t)old;
  if (here) clear_padding(nodes, nb + (uint32_t)c.my);
  if (LEFT) c.l = other;
  else c.f = other;
  if ((old >> 32) & 1u) {
    const float4* sp = reinterpret_cast<const float4*>(nodes + nb + sib);
    for (uint32_t spins = 0; !climb_whole(__float_as_uint(slo.w), __float_as_uint(shi.w), epoch, mark); ++spins) {
      if (spins >= limit) return false;
      slo = ld_relaxed16(sp);
      shi = ld_relaxed16(sp + 1);
    }
    clear_padding(nodes, nb + sib);
    const uint32_t w = __float_as_uint(shi.w);
    dfar = climb_delta(w);
    Box sb;
    sb.lo = make_float4(slo.x, slo.y, slo.z, 0.f);
    sb.hi = make_float4(shi.x, shi.y, shi.z, 0.f);
    climb_merge<PLUS>(c, LEFT, (int32_t)sib, sb, climb_height(w));
    return true;
  }
  const bool leaf = other == g + off + (LEFT ? 1u : 0u);
  if (leaf) sib = LEFT ? cnt + g : cnt - 1 + g;
  if (LEFT) dfar = other + 1 >= n ? 0u : __ldg(D + other);
  else dfar = other == 0 ? 0u : __ldg(D + other - 1);
  const uint32_t hs = PLUS && !leaf ? __ldcg(hgt + nb + sib) : 0u;
  climb_merge<PLUS>(c, LEFT, (int32_t)sib, load_node_box(nodes, nb + sib), hs);
  return true;
}

// Climb from every frontier node (a finished node whose parent needs a sibling built by another block)
// through the rendezvous words; the second child to arrive completes the parent.
//
// What bounds it is the chain of one round trip after another, a dozen or more levels from the tiles to
// the root.  A node is therefore its own message: while its parent is missing, the padding of its two
// corners (each written and read as 16 bytes at once) holds the build's epoch and a mark of it and, beside
// that, the delta byte past its far end and its height (climb_message.h).  No fence orders the node's
// stores before its announcement: the sibling, which reads the node while its own announcement is under way,
// sees by epoch and mark whether it has it, and otherwise reads again.  Both paddings are 0 before (see
// Workspace::nodes, and k_emit's CLEAR) and again once the parent is complete.  A rendezvous word is
// (epoch | written in this kernel) << 32 | far end; a node written by k_emit (bit 0 clear) carries
// no epoch and needs none.
// With a fence before the exchange, and the sibling's box and delta byte read after it, emission took 43 us of
// 100,000 triangles (30 now), 98 of 1M (77), 523 of 10M (496), 1,400 of 29M in 1,024 meshes (1,357).
template <typename Seg, bool PLUS>
__global__ void __launch_bounds__(256) k_emit_climb(const uint8_t* __restrict__ D, Node* __restrict__ nodes,
                                                    unsigned long long* __restrict__ slots,
                                                    const uint32_t* epoch_word, uint32_t n, Seg seg,
                                                    const uint2* __restrict__ frontier,
                                                    const uint32_t* __restrict__ frontier_count,
                                                    uint8_t* __restrict__ hgt, uint32_t* __restrict__ status,
                                                    uint32_t limit) {
  after_previous();
  const uint32_t count = __ldcg(frontier_count);
  const uint32_t epoch = __ldcg(epoch_word);  // (a multiple of kEpochStride)
  const uint32_t mark = climb_mark(epoch);
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < count; e += gridDim.x * blockDim.x) {
    const uint2 fl = __ldcg(frontier + e);
    Climb c;
    c.f = fl.x;
    c.l = fl.y;
    uint32_t off, cnt, nb;
    seg.get(c.f, off, cnt, nb);
    // delta bytes beside the node's ends (0 at the ends of the mesh)
    uint32_t dl = c.f == 0 ? 0u : __ldg(D + c.f - 1), dr = c.l + 1 >= n ? 0u : __ldg(D + c.l);
    bool is_left = dr > dl;
    c.my = c.f == c.l ? (int32_t)(cnt - 1 + (c.f - off)) : (int32_t)((is_left ? c.l : c.f) - off);
    c.box = load_node_box(nodes, nb + (uint32_t)c.my);
    c.h = PLUS && c.f != c.l ? __ldcg(hgt + nb + (uint32_t)c.my) : 0u;
    uint32_t here = 0;  // 1: the node was written in this kernel
    while (true) {
      const uint32_t gamma = is_left ? c.l : c.f - 1, g = gamma - off;
      // the sibling, if it is an internal node: a right child is named by its first position, a left by its last
      uint32_t sib = is_left ? g + 1 : g;
      const float4* sp = reinterpret_cast<const float4*>(nodes + nb + sib);
      float4 slo = make_float4(0.f, 0.f, 0.f, 0.f), shi = slo;
      if (here) {
        slo = ld_relaxed16(sp);
        shi = ld_relaxed16(sp + 1);
      }
      const unsigned long long old =
          atom_exch_relaxed(slots + gamma, (unsigned long long)(epoch | here) << 32 | (is_left ? c.f : c.l));
      if ((uint32_t)(old >> 33) != epoch >> 1) break;  // first child to arrive
      const bool ok =
          is_left ? climb_join<PLUS, true>(c, dr, old, sib, slo, shi, here, g, off, cnt, nb, n, epoch, mark, limit, D, nodes, hgt)
                  : climb_join<PLUS, false>(c, dl, old, sib, slo, shi, here, g, off, cnt, nb, n, epoch, mark, limit, D, nodes, hgt);
      if (!ok) {  // nothing above is completed by anyone: the root becomes a leaf, so that no walk meets what is missing
        atomicOr(status, kStatusClimbTimeout);
        store_node(nodes, nb, c.box, (int32_t)kLeafBit, -1, -1);
        break;
      }
      if (dl == 0 && dr == 0) {
        write_internal<PLUS>(nodes, hgt, nb, 0, c);
        break;
      }
      is_left = dr > dl;
      c.my = (int32_t)((is_left ? c.l : c.f) - off);
      here = 1;
      // (each corner, with its padding, may be read while it is written)
      float4* np = reinterpret_cast<float4*>(nodes + nb + (uint32_t)c.my);
      st_relaxed16(np, make_float4(c.box.lo.x, c.box.lo.y, c.box.lo.z, __uint_as_float(epoch)));
      st_relaxed16(np + 1, make_float4(c.box.hi.x, c.box.hi.y, c.box.hi.z,
                                       __uint_as_float(climb_hi_word(mark, is_left ? dl : dr, c.h))));
      __stcg(reinterpret_cast<int4*>(np + 2), PLUS ? make_int4(c.lc, c.rc, __float_as_int(c.al), __float_as_int(c.ar))
                                                   : make_int4(c.lc, c.rc, -1, 0));
      if (PLUS) __stcg(hgt + nb + (uint32_t)c.my, (uint8_t)min(c.h, 255u));
    }
  }
}

}  // namespace bvhgb

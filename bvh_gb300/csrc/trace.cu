// trace.cu -- closest-hit ray traversal used to measure tree quality.
//
// Reference: traverseBVH (src/render_engine.cu:289-356) with intersectAABB (:194-214),
// intersectTriangle (:220-273) and generateRay (:155-188).  Same visiting order (left child
// first, 128-entry stack that silently drops pushes when full), same counters (a node counts as
// visited before its box test), same closest-hit rule (strict <).
//
// Rounding: every float operation is an explicitly rounded intrinsic, in the form nvcc gives the
// reference's expressions under its default -fmad=true.  A two-product difference a*b - c*d is
// fma(a, b, -(c*d)); a three-term dot product (a.x*b.x + a.y*b.y) + a.z*b.z is
// fma(a.z, b.z, fma(a.x, b.x, a.y*b.y)); x + a*b is fma(a, b, x).  (The left product of a sum is
// fused first, and a sum whose left operand is already fused takes the right product into a second
// fma.)  Expressions with a division or subtraction between the multiply and the add
// ((lo - o) * inv, (2(x + 0.5)/w - 1) * half_w) have nothing to contract.  The forms are pinned
// against the reference's own traverseBVH and generateRay on the same rays.  The CPU oracle uses
// the same forms (C fmaf), so it reproduces t, hit ids and counters bit for bit.
#include <algorithm>

#include "lbvh.cuh"
#include "trace.cuh"

namespace bvhgb {

constexpr int kStack = 128;
constexpr float kEps = 1e-6f;

// The slab test without its upper bound; tenter comes back for `tenter < tmax`.
__device__ __forceinline__ bool hit_slabs(const float3 o, const float3 inv, float lx, float ly, float lz, float hx,
                                          float hy, float hz, float& tenter) {
  float ax = __fmul_rn(__fsub_rn(lx, o.x), inv.x), bx = __fmul_rn(__fsub_rn(hx, o.x), inv.x);
  float ay = __fmul_rn(__fsub_rn(ly, o.y), inv.y), by = __fmul_rn(__fsub_rn(hy, o.y), inv.y);
  float az = __fmul_rn(__fsub_rn(lz, o.z), inv.z), bz = __fmul_rn(__fsub_rn(hz, o.z), inv.z);
  tenter = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz));
  float texit = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz));
  return texit >= fmaxf(tenter, 0.0f);
}

__device__ __forceinline__ bool hit_box(const float3 o, const float3 inv, const float4 lo, const float4 hi, float tmax) {
  float tenter;
  return hit_slabs(o, inv, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, tenter) && tenter < tmax;
}

// d_dot (:122-124): (a*x + b*y) + c*z, contracted.
__device__ __forceinline__ float dot3(float a, float b, float c, float x, float y, float z) {
  return __fmaf_rn(c, z, __fmaf_rn(a, x, __fmul_rn(b, y)));
}
// a*b - c*d, contracted (d_cross :114-120 and the edge products of intersectTriangle).
__device__ __forceinline__ float cross_c(float a, float b, float c, float d) {
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}

// intersectTriangle from the vertex and the two edges (v1 - v0, v2 - v0, each rounded).
__device__ __forceinline__ bool hit_edges(const float3 o, const float3 d, float v0x, float v0y, float v0z, float e1x,
                                          float e1y, float e1z, float e2x, float e2y, float e2z, float& t_out) {
  const float px = cross_c(d.y, e2z, d.z, e2y), py = cross_c(d.z, e2x, d.x, e2z), pz = cross_c(d.x, e2y, d.y, e2x);
  const float det = dot3(e1x, e1y, e1z, px, py, pz);
  if (fabsf(det) < kEps) return false;
  const float inv_det = __fdiv_rn(1.0f, det);
  const float tx = __fsub_rn(o.x, v0x), ty = __fsub_rn(o.y, v0y), tz = __fsub_rn(o.z, v0z);
  const float u = __fmul_rn(dot3(tx, ty, tz, px, py, pz), inv_det);
  if (u < -1e-5f || u > 1.00001f) return false;
  const float qx = cross_c(ty, e1z, tz, e1y), qy = cross_c(tz, e1x, tx, e1z), qz = cross_c(tx, e1y, ty, e1x);
  const float v = __fmul_rn(dot3(d.x, d.y, d.z, qx, qy, qz), inv_det);
  if (v < -1e-5f || __fadd_rn(u, v) > 1.00001f) return false;
  const float t = __fmul_rn(dot3(e2x, e2y, e2z, qx, qy, qz), inv_det);
  if (t < kEps) return false;
  t_out = t;
  return true;
}

__device__ __forceinline__ bool hit_tri(const float3 o, const float3 d, const MeshPtrs& m, uint32_t p, float& t_out) {
  const float v0x = __ldg(m.v[0] + p), v0y = __ldg(m.v[1] + p), v0z = __ldg(m.v[2] + p);
  const float e1x = __fsub_rn(__ldg(m.v[3] + p), v0x), e1y = __fsub_rn(__ldg(m.v[4] + p), v0y),
              e1z = __fsub_rn(__ldg(m.v[5] + p), v0z);
  const float e2x = __fsub_rn(__ldg(m.v[6] + p), v0x), e2y = __fsub_rn(__ldg(m.v[7] + p), v0y),
              e2z = __fsub_rn(__ldg(m.v[8] + p), v0z);
  return hit_edges(o, d, v0x, v0y, v0z, e1x, e1y, e1z, e2x, e2y, e2z, t_out);
}

__device__ __forceinline__ float inv_dir(float d) {
  return fabsf(d) > kEps ? __fdiv_rn(1.0f, d) : (d >= 0.0f ? 1e30f : -1e30f);
}

__device__ void trace_one(const float3 o, const float3 d, const Node* __restrict__ nodes, int n_nodes,
                          const MeshPtrs& m, uint32_t n_tris, uint32_t r, const HitOut& out) {
  const float3 inv = make_float3(inv_dir(d.x), inv_dir(d.y), inv_dir(d.z));
  float best = 1e30f;
  int32_t prim = -1, vis = 0, at = 0, tt = 0;
  int stack[kStack];
  int sp = 0;
  if (n_nodes > 0) stack[sp++] = 0;
  while (sp > 0) {
    const int x = stack[--sp];
    if (x < 0 || x >= n_nodes) continue;
    const float4* np = reinterpret_cast<const float4*>(nodes + x);
    const float4 lo = __ldg(np), hi = __ldg(np + 1);
    vis++;
    at++;
    if (!hit_box(o, inv, lo, hi, best)) continue;
    const int2 ch = __ldg(reinterpret_cast<const int2*>(np + 2));
    if (ch.x < 0) {
      const uint32_t p = (uint32_t)ch.x & 0x7FFFFFFFu;
      tt++;
      float t;
      if (p < n_tris && hit_tri(o, d, m, p, t)) {
        if (t < best) {
          best = t;
          prim = (int32_t)p;
        }
      }
    } else {
      if (ch.y >= 0 && ch.y < n_nodes && sp < kStack) stack[sp++] = ch.y;
      if (ch.x >= 0 && ch.x < n_nodes && sp < kStack) stack[sp++] = ch.x;
    }
  }
  out.t[r] = best;
  out.prim[r] = prim;
  out.vis[r] = vis;
  out.aabb[r] = at;
  out.tri[r] = tt;
}

__global__ void __launch_bounds__(128) k_trace(const Node* __restrict__ nodes, int n_nodes, MeshPtrs m, uint32_t n_tris,
                                               RayPtrs rays, uint32_t nr, HitOut out) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nr) return;
  const float3 o = make_float3(__ldg(rays.o[0] + r), __ldg(rays.o[1] + r), __ldg(rays.o[2] + r));
  const float3 d = make_float3(__ldg(rays.d[0] + r), __ldg(rays.d[1] + r), __ldg(rays.d[2] + r));
  trace_one(o, d, nodes, n_nodes, m, n_tris, r, out);
}

// d_normalize (:130-135): zero below length 1e-12, else each component times 1 / length.
__device__ __forceinline__ float3 normalize3(float x, float y, float z) {
  const float len = __fsqrt_rn(dot3(x, y, z, x, y, z));
  if (len < 1e-12f) return make_float3(0.f, 0.f, 0.f);
  const float inv = __fdiv_rn(1.0f, len);
  return make_float3(__fmul_rn(x, inv), __fmul_rn(y, inv), __fmul_rn(z, inv));
}

// generateRay (:155-188) for pixel (x, y): the camera basis and tan(fov/2) are computed per ray,
// as the reference does, with the device's own tanf.
__device__ __forceinline__ float3 pinhole_dir(const PinholeCam& c, int x, int y) {
  const float3 f = normalize3(__fsub_rn(c.look[0], c.eye[0]), __fsub_rn(c.look[1], c.eye[1]),
                              __fsub_rn(c.look[2], c.eye[2]));
  const float3 rt = normalize3(cross_c(f.y, c.up[2], f.z, c.up[1]), cross_c(f.z, c.up[0], f.x, c.up[2]),
                               cross_c(f.x, c.up[1], f.y, c.up[0]));
  const float3 up = make_float3(cross_c(rt.y, f.z, rt.z, f.y), cross_c(rt.z, f.x, rt.x, f.z),
                                cross_c(rt.x, f.y, rt.y, f.x));
  const float fov = __fdiv_rn(__fmul_rn(c.fov_deg, 3.14159265358979f), 180.0f);
  const float half_h = tanf(__fmul_rn(fov, 0.5f));
  const float half_w = __fmul_rn(half_h, __fdiv_rn((float)c.width, (float)c.height));
  const float uu = __fmul_rn(__fsub_rn(__fdiv_rn(__fmul_rn(2.0f, __fadd_rn((float)x, 0.5f)), (float)c.width), 1.0f), half_w);
  const float vv = __fmul_rn(__fsub_rn(__fdiv_rn(__fmul_rn(2.0f, __fadd_rn((float)y, 0.5f)), (float)c.height), 1.0f), half_h);
  // forward + u*right - v*up, contracted: fma(-v, up, fma(u, right, forward))
  return normalize3(__fmaf_rn(-vv, up.x, __fmaf_rn(uu, rt.x, f.x)), __fmaf_rn(-vv, up.y, __fmaf_rn(uu, rt.y, f.y)),
                    __fmaf_rn(-vv, up.z, __fmaf_rn(uu, rt.z, f.z)));
}

__global__ void __launch_bounds__(128) k_trace_pinhole(const Node* __restrict__ nodes, int n_nodes, MeshPtrs m,
                                                       uint32_t n_tris, PinholeCam cam, HitOut out) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t total = (uint32_t)cam.width * (uint32_t)cam.height;
  if (r >= total) return;
  const int x = (int)(r % (uint32_t)cam.width), y = (int)(r / (uint32_t)cam.width);
  const float3 o = make_float3(cam.eye[0], cam.eye[1], cam.eye[2]);
  trace_one(o, pinhole_dir(cam, x, y), nodes, n_nodes, m, n_tris, r, out);
}

// ---------------------------------------------------------------------------------------
// Packed traversal.  A ray's loop is a chain of dependent loads, and a warp's 32 rays load from 32
// places: k_trace above fetches a 48-byte node per visit (two sectors each, then its children's
// indices, then nine separate triangle arrays) and spends most of its time waiting for them.  For
// a trace of many rays, a kernel first rewrites tree and mesh as 64-byte records -- per inner node
// both children's boxes and references, per triangle its vertex and edges -- so that
//   - one 64-byte load decides both children: half the steps and half the bytes per visited node,
//     a child that misses is counted without being fetched or pushed;
//   - an inner node and a leaf load alike, so lanes at leaves wait together with lanes at inner nodes.
// Order, counters and hits are the reference's: a node counts as visited when its parent was entered
// (it would be popped later whatever the hits before it), a box is tested against the best hit at
// the time of its visit (its entry distance is kept on the stack and compared again when it is taken
// off), and `vs` is the height that the reference's 128-entry stack would have at this node, so
// pushes are dropped exactly where it drops them.  Stack entries live in shared memory (the first
// kPackStack) and in local memory beyond.
// Measured (GB300): 1M sphere rays on a 2M-strand LBVH+ tree 22.1 -> 7.6 ms, 1M on a 1.3M icosphere
// PLOC tree 1.84 -> 0.98 ms, 65,536 on a 50k LBVH 0.19 -> 0.12 ms; full-HD primary rays and shading
// on a 10M LBVH-63 20.4 -> 7.8 ms, on a 330k icosphere 0.35 -> 0.27 ms; all with the repacking
// (0.50 ms at 10M triangles, 0.11 ms at 2M).  What is left on the dense scene is the longest ray: 13,321
// visits, 7,800 steps of about 0.5 us alone and 0.9 us among its warp's other rays.
// ---------------------------------------------------------------------------------------
struct __align__(64) PackNode {
  float lo_l[3], hi_l[3], lo_r[3], hi_r[3];
  int32_t left, right;  // >= 0: an inner node's record, < 0: kLeafBit | triangle, kPackNone: no child
  int32_t pad[2];
};
struct __align__(64) PackTri {
  float v0[3], e1[3], e2[3], pad[7];
};
static_assert(sizeof(PackNode) == 64 && sizeof(PackTri) == 64, "one record is half a 128-byte line");
constexpr int32_t kPackNone = 0x7fffffff;  // never an index: n_nodes <= 2^31 - 1
constexpr int kPackThreads = 64;
constexpr int kPackStack = 12;  // stack entries per thread in shared memory: 8 -> 12 took 2% off, 16 cost L1
constexpr uint64_t kPackMaxBytes = 16ull << 30;

__device__ __forceinline__ void ld_record(const void* p, float (&w)[16]) {  // two 32-byte loads
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(w[8 * h]), "=f"(w[8 * h + 1]), "=f"(w[8 * h + 2]), "=f"(w[8 * h + 3]), "=f"(w[8 * h + 4]),
                   "=f"(w[8 * h + 5]), "=f"(w[8 * h + 6]), "=f"(w[8 * h + 7])
                 : "l"(reinterpret_cast<const char*>(p) + 32 * h));
}

// The record of inner node i, whose children are ch.
__device__ __forceinline__ void node_record(const Node* __restrict__ nodes, int n_nodes, int2 ch, float (&w)[16]) {
  float4 b[2][2];
  int32_t ref[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int c = s ? ch.y : ch.x;
    ref[s] = kPackNone;
    b[s][0] = b[s][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c >= 0 && c < n_nodes) {
      const float4* p = reinterpret_cast<const float4*>(nodes + c);
      b[s][0] = __ldg(p);
      b[s][1] = __ldg(p + 1);
      const int32_t l = __ldg(reinterpret_cast<const int32_t*>(p + 2));
      ref[s] = l < 0 ? l : c;
    }
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    w[6 * s] = b[s][0].x; w[6 * s + 1] = b[s][0].y; w[6 * s + 2] = b[s][0].z;
    w[6 * s + 3] = b[s][1].x; w[6 * s + 4] = b[s][1].y; w[6 * s + 5] = b[s][1].z;
    w[12 + s] = __int_as_float(ref[s]);
  }
  w[14] = w[15] = 0.f;
}
__device__ __forceinline__ int2 node_children(const Node* __restrict__ nodes, int64_t i) {
  return __ldg(reinterpret_cast<const int2*>(reinterpret_cast<const float4*>(nodes + i) + 2));
}

// The first nine words of triangle p's record.
__device__ __forceinline__ void tri_record(const MeshPtrs& m, uint64_t p, float (&w)[16]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    w[k] = __ldg(m.v[k] + p);
    w[3 + k] = __fsub_rn(__ldg(m.v[3 + k] + p), w[k]);
    w[6 + k] = __fsub_rn(__ldg(m.v[6 + k] + p), w[k]);
  }
}

// The rays of a trace: given ones, or the pixels of an image.
struct GivenRays {
  RayPtrs p;
  __device__ __forceinline__ void get(uint32_t r, float3& o, float3& d) const {
    o = make_float3(__ldg(p.o[0] + r), __ldg(p.o[1] + r), __ldg(p.o[2] + r));
    d = make_float3(__ldg(p.d[0] + r), __ldg(p.d[1] + r), __ldg(p.d[2] + r));
  }
};
struct PixelRays {
  PinholeCam cam;
  __device__ __forceinline__ void get(uint32_t r, float3& o, float3& d) const {
    o = make_float3(cam.eye[0], cam.eye[1], cam.eye[2]);
    d = pinhole_dir(cam, (int)(r % (uint32_t)cam.width), (int)(r / (uint32_t)cam.width));
  }
};

// Whether one of 256 rays spread over the nr, one per thread of the block, enters the root's box.  Each is taken
// at an odd place of its own 256th, so that the pixels of an image are not all of one column.
template <typename Rays>
__device__ __forceinline__ bool some_ray_enters(const Rays& rays, uint32_t nr, const Node* __restrict__ nodes) {
  const uint32_t k = threadIdx.x, width = nr >> 8;
  float3 o, d;
  rays.get((uint32_t)(((uint64_t)k * nr) >> 8) + (k * 0x9e3779b1u >> 8) % width, o, d);
  const float4* np = reinterpret_cast<const float4*>(nodes);
  return __syncthreads_or(hit_box(o, make_float3(inv_dir(d.x), inv_dir(d.y), inv_dir(d.z)), __ldg(np), __ldg(np + 1), 1e30f));
}

// One record per inner node, read by two gathers of its children (neighbours in Karras numbering), and
// one per triangle; bound by DRAM traffic (20M nodes and 10M triangles: 2.6 GB in 0.50 ms).
// Where rays enter the scene at all, a trace waits for its longest chains and the records pay from the first few on:
// with 2 in 100 entering, 16,384 rays over 16,000 nodes take 50 us packed and 82 plain, 262,144 over 4M 1,161
// and 1,580.  A trace of which no ray enters is over in 5 us, which the records made 17 to 146.  So every block
// looks at the same 256 rays first; where none of them enters, nothing is packed and *packed is 0 (12 to 21
// us then, most of it the call's; with one ray in 2,000 entering 4M nodes 577 -> 323).
template <typename Rays>
__global__ void __launch_bounds__(256, 5) k_pack(const Node* __restrict__ nodes, int n_nodes, MeshPtrs m, uint32_t n_tris,
                                              Rays rays, uint32_t nr, PackNode* __restrict__ rec,
                                              PackTri* __restrict__ tris, uint32_t* __restrict__ packed) {
  const bool enters = some_ray_enters(rays, nr, nodes);
  if (blockIdx.x == 0 && threadIdx.x == 0) *packed = enters ? 1u : 0u;
  if (!enters) return;
  const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 1
  for (int64_t i = first; i < n_nodes; i += step) {
    const int2 ch = node_children(nodes, i);
    if (ch.x < 0) continue;  // a leaf has no record
    float w[16];
    node_record(nodes, n_nodes, ch, w);
    float4* o = reinterpret_cast<float4*>(rec + i);
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = make_float4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
  }
#pragma unroll 1
  for (int64_t p = first; p < n_tris; p += step) {
    float w[16];
    tri_record(m, (uint64_t)p, w);
    float4* o = reinterpret_cast<float4*>(tris + p);
    o[0] = make_float4(w[0], w[1], w[2], w[3]);
    o[1] = make_float4(w[4], w[5], w[6], w[7]);
    o[2] = make_float4(w[8], 0.f, 0.f, 0.f);
  }
}

// The tree and its records, and whether these were made.
struct PackedTree {
  const Node* nodes;
  int n_nodes;
  MeshPtrs m;
  uint32_t n_tris;
  const PackNode* rec;
  const PackTri* tris;
  const uint32_t* packed;
};

struct RayStack {  // what lies above the shared part
  int2 entry[kStack - kPackStack];
  uint8_t vs[kStack - kPackStack];
};

// PACKED: from the records; otherwise each is put together from the tree and the mesh when it is met.
template <bool PACKED>
__device__ __forceinline__ void trace_records(bool live, const float3 o, const float3 d, const PackedTree& T, uint32_t r,
                                              const HitOut& out, int2 (*s_entry)[kPackThreads],
                                              uint8_t (*s_vs)[kPackThreads], RayStack& local) {
  const int tid = threadIdx.x;
  const uint32_t n_tris = T.n_tris;
  const float3 inv = make_float3(inv_dir(d.x), inv_dir(d.y), inv_dir(d.z));
  float best = 1e30f;
  int32_t prim = -1, vis = 0, tt = 0;
  int vs = 0, sp = 0;
  int32_t cur = kPackNone;
  if (live) {
    const float4* np = reinterpret_cast<const float4*>(T.nodes);
    vis = 1;
    if (hit_box(o, inv, __ldg(np), __ldg(np + 1), best)) {
      const int32_t x = __ldg(reinterpret_cast<const int32_t*>(np + 2));
      cur = x < 0 ? x : 0;
    }
  }
  while (cur != kPackNone) {
    const bool leaf = cur < 0;
    const uint32_t id = (uint32_t)cur & ~kLeafBit;
    float w[16];
    if (PACKED)
      ld_record(leaf ? static_cast<const void*>(T.tris + min(id, n_tris - 1)) : static_cast<const void*>(T.rec + id), w);
    else if (leaf)
      tri_record(T.m, min(id, n_tris - 1), w);
    else
      node_record(T.nodes, T.n_nodes, node_children(T.nodes, id), w);
    bool pop;
    if (leaf) {
      tt++;
      float t;
      if (id < n_tris && hit_edges(o, d, w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], t) && t < best) {
        best = t;
        prim = (int32_t)id;
      }
      pop = true;
    } else {
      const int32_t left = __float_as_int(w[12]), right = __float_as_int(w[13]);
      // the reference pushes the right child, then the left, while its stack has room
      const bool has_r = right != kPackNone && vs < kStack;
      const bool has_l = left != kPackNone && vs + (has_r ? 1 : 0) < kStack;
      float tl, tr;
      const bool hl = hit_slabs(o, inv, w[0], w[1], w[2], w[3], w[4], w[5], tl) && tl < best && has_l;
      const bool hr = hit_slabs(o, inv, w[6], w[7], w[8], w[9], w[10], w[11], tr) && tr < best && has_r;
      vis += (has_l ? 1 : 0) + (has_r ? 1 : 0);
      if (hl && hr) {
        const int2 e = make_int2(right, __float_as_int(tr));
        if (sp < kPackStack) {
          s_entry[sp][tid] = e;
          s_vs[sp][tid] = (uint8_t)vs;
        } else {
          local.entry[sp - kPackStack] = e;
          local.vs[sp - kPackStack] = (uint8_t)vs;
        }
        sp++;
      }
      if (hl && has_r) vs++;  // the right child lies below the left one on the reference's stack
      cur = hl ? left : right;
      pop = !(hl || hr);
    }
    while (pop) {
      if (sp == 0) {
        cur = kPackNone;
        break;
      }
      sp--;
      int2 e;
      if (sp < kPackStack) {
        e = s_entry[sp][tid];
        vs = s_vs[sp][tid];
      } else {
        e = local.entry[sp - kPackStack];
        vs = local.vs[sp - kPackStack];
      }
      cur = e.x;
      pop = !(__int_as_float(e.y) < best);
    }
  }
  if (live) {
    out.t[r] = best;
    out.prim[r] = prim;
    out.vis[r] = vis;
    out.aabb[r] = vis;
    out.tri[r] = tt;
  }
}

__device__ __forceinline__ void trace_packed(bool live, const float3 o, const float3 d, const PackedTree& T, uint32_t r,
                                             const HitOut& out) {
  __shared__ int2 s_entry[kPackStack][kPackThreads];  // reference, entry distance
  __shared__ uint8_t s_vs[kPackStack][kPackThreads];
  RayStack local;
  if (__ldcg(T.packed)) trace_records<true>(live, o, d, T, r, out, s_entry, s_vs, local);
  else trace_records<false>(live, o, d, T, r, out, s_entry, s_vs, local);
}

// 20 blocks of 64 threads per SM (48 registers): smaller blocks end as soon as their own rays do.
__global__ void __launch_bounds__(kPackThreads, 20)
    k_trace_packed(PackedTree T, GivenRays rays, uint32_t nr, HitOut out) {
  const uint32_t r = blockIdx.x * kPackThreads + threadIdx.x;
  const bool live = r < nr;
  float3 o, d;
  rays.get(live ? r : nr - 1, o, d);
  trace_packed(live, o, d, T, r, out);
}

// A warp takes two 4x4 pixel tiles from opposite halves of the image: coherent within a tile, and
// the pixels that need thousands of steps (a dense part of the scene) spread over twice the warps.
// One 8x4 tile: 8.0 -> 7.0 ms on the dense 10M scene and 0.26 -> 0.28 ms on the icosphere; four
// tiles of 4x2: 6.8 and 0.35 ms.
__host__ __device__ inline uint32_t pinhole_tiles(int w, int h) { return div_up((uint32_t)w, 4) * div_up((uint32_t)h, 4); }
__global__ void __launch_bounds__(kPackThreads, 20)
    k_trace_pinhole_packed(PackedTree T, PinholeCam cam, HitOut out) {
  const uint32_t warp = (blockIdx.x * kPackThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const uint32_t tiles = pinhole_tiles(cam.width, cam.height), half = div_up(tiles, 2);
  const uint32_t tile = warp + (lane >> 4) * half, across = div_up((uint32_t)cam.width, 4);
  const uint32_t x = (tile % across) * 4 + (lane & 3), y = (tile / across) * 4 + ((lane >> 2) & 3);
  const bool live = warp < half && tile < tiles && x < (uint32_t)cam.width && y < (uint32_t)cam.height;
  const float3 o = make_float3(cam.eye[0], cam.eye[1], cam.eye[2]);
  trace_packed(live, o, pinhole_dir(cam, (int)x, (int)y), T, y * (uint32_t)cam.width + x, out);
}

void trace_pool_free(TracePool& p) {
  if (p.pool) cudaMemPoolDestroy(p.pool);
  p = TracePool{p.device};
}

uint64_t trace_pool_bytes(const TracePool& p) {
  uint64_t bytes = 0;
  if (p.pool && cudaMemPoolGetAttribute(p.pool, cudaMemPoolAttrReservedMemCurrent, &bytes) != cudaSuccess) bytes = 0;
  return bytes;
}

// The pool's memory comes in pieces of 32 MiB; a threshold in the midst of one gives that piece back at every
// synchronisation.
constexpr uint64_t kPoolPiece = 32ull << 20;
static cudaError_t trace_pool_keep(TracePool& p, uint64_t bytes) {
  p.keep = bytes;
  uint64_t threshold = (bytes + kPoolPiece - 1) / kPoolPiece * kPoolPiece;
  return cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &threshold);
}

bool trace_pool_trim(TracePool& p) {
  if (trace_pool_bytes(p) == 0) return false;
  p.recent = p.traces = 0;
  return trace_pool_keep(p, 0) == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess &&
         cudaMemPoolTrimTo(p.pool, 0) == cudaSuccess;
}

// Whether a trace repacks (if its rays enter the scene: k_pack): repacking costs ~0.025 ns per node and ~10 us of
// launches; it gains 0.85 ns per ray on the cheapest tree measured (100 visits per ray, 1.3M triangles)
// and 7 to 14 ns on deep ones.  At 16 nodes per ray and 16,384 rays the least gain is about twice the
// cost.  Not while the stream is being captured (a graph of the trace stays free of allocations), and
// where the pool has no room the trace runs on the tree as it is.  T: its records, allocated on the stream,
// filled there, and given back by unpack().
template <typename Rays>
static bool pack(TracePool* tp, const Node* nodes, int n_nodes, const MeshPtrs& m, uint32_t n_tris, const Rays& rays,
                 uint32_t nr, cudaStream_t st, PackedTree* T) {
  if (!tp || nr < 16384u || n_nodes < 3 || n_tris == 0 || (uint64_t)n_nodes > 16ull * nr) return false;
  const uint64_t node_bytes = (uint64_t)n_nodes * sizeof(PackNode);
  const uint64_t bytes = sizeof(PackNode) + node_bytes + (uint64_t)n_tris * sizeof(PackTri);  // *packed first
  if (bytes > kPackMaxBytes) return false;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  bool ok = cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone;
  if (ok && !tp->pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = tp->device;
    ok = cudaMemPoolCreate(&tp->pool, &props) == cudaSuccess;
    if (!ok) tp->pool = nullptr;
  }
  if (ok) {
    tp->recent = std::max(tp->recent, bytes);
    if (tp->keep < bytes) ok = trace_pool_keep(*tp, bytes) == cudaSuccess;
    if (ok && ++tp->traces == kTraceWindow) {
      if (tp->recent < tp->keep) ok = trace_pool_keep(*tp, tp->recent) == cudaSuccess && cudaMemPoolTrimTo(tp->pool, tp->recent) == cudaSuccess;
      tp->recent = tp->traces = 0;
    }
  }
  void* buf = nullptr;
  if (!ok || cudaMallocFromPoolAsync(&buf, bytes, tp->pool, st) != cudaSuccess) {
    cudaGetLastError();  // not the caller's error: the trace still runs
    return false;
  }
  PackNode* rec = static_cast<PackNode*>(buf) + 1;
  PackTri* tris = reinterpret_cast<PackTri*>(rec + n_nodes);
  *T = PackedTree{nodes, n_nodes, m, n_tris, rec, tris, static_cast<uint32_t*>(buf)};
  k_pack<<<std::min<uint32_t>(div_up(std::max((uint32_t)n_nodes, n_tris), 256), 152 * 8), 256, 0, st>>>(
      nodes, n_nodes, m, n_tris, rays, nr, rec, tris, static_cast<uint32_t*>(buf));
  return true;
}
static cudaError_t unpack(const PackedTree& T, cudaStream_t st) {
  const cudaError_t e = cudaGetLastError();
  const cudaError_t f = cudaFreeAsync(const_cast<uint32_t*>(T.packed), st);
  return e != cudaSuccess ? e : f;
}

__global__ void k_pinhole_rays(PinholeCam cam, float* ox, float* oy, float* oz, float* dx, float* dy, float* dz) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t total = (uint32_t)cam.width * (uint32_t)cam.height;
  if (r >= total) return;
  const float3 d = pinhole_dir(cam, (int)(r % (uint32_t)cam.width), (int)(r / (uint32_t)cam.width));
  ox[r] = cam.eye[0]; oy[r] = cam.eye[1]; oz[r] = cam.eye[2];
  dx[r] = d.x; dy[r] = d.y; dz[r] = d.z;
}

// ---------------------------------------------------------------------------------------
// Shading and the traversal-cost heatmap: kRenderKernel's shading (src/render_engine.cu:395-446)
// and the host post-processing of renderImage -- applyHeatmapColormap (:541-595) with
// getTurboColor (:519-535), and savePPM's float-to-byte conversion (:502-507) -- on the device,
// with the same explicitly rounded operations as the traversal above.
// ---------------------------------------------------------------------------------------
constexpr float kBgR = 0.15f, kBgG = 0.15f, kBgB = 0.18f;  // a pixel without a hit (BG_R/G/B)

// Geometric normal of triangle p (intersectTriangle, :267-271): normalise(e1 x e2).
__device__ __forceinline__ float3 tri_normal(const MeshPtrs& m, uint32_t p) {
  const float v0x = __ldg(m.v[0] + p), v0y = __ldg(m.v[1] + p), v0z = __ldg(m.v[2] + p);
  const float e1x = __fsub_rn(__ldg(m.v[3] + p), v0x), e1y = __fsub_rn(__ldg(m.v[4] + p), v0y),
              e1z = __fsub_rn(__ldg(m.v[5] + p), v0z);
  const float e2x = __fsub_rn(__ldg(m.v[6] + p), v0x), e2y = __fsub_rn(__ldg(m.v[7] + p), v0y),
              e2z = __fsub_rn(__ldg(m.v[8] + p), v0z);
  return normalize3(cross_c(e1y, e2z, e1z, e2y), cross_c(e1z, e2x, e1x, e2z), cross_c(e1x, e2y, e1y, e2x));
}

__global__ void __launch_bounds__(256) k_shade(PinholeCam cam, MeshPtrs m, uint32_t n_tris, ShadeIn in, int mode,
                                               float diag, float3 light, float* __restrict__ rgb) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t total = (uint32_t)cam.width * (uint32_t)cam.height;
  if (r >= total) return;
  const int32_t p = in.prim[r];
  float cr, cg, cb;
  if (p < 0 || (uint32_t)p >= n_tris) {
    cr = kBgR; cg = kBgG; cb = kBgB;
  } else if (mode == 0) {  // normal mapped to RGB
    const float3 n = tri_normal(m, (uint32_t)p);
    cr = __fmul_rn(__fadd_rn(n.x, 1.0f), 0.5f);
    cg = __fmul_rn(__fadd_rn(n.y, 1.0f), 0.5f);
    cb = __fmul_rn(__fadd_rn(n.z, 1.0f), 0.5f);
  } else if (mode == 1) {  // depth: closer is brighter
    const float depth = fmaxf(0.0f, fminf(1.0f, __fdiv_rn(in.t[r], diag)));
    cr = cg = cb = __fsub_rn(1.0f, depth);
  } else if (mode == 2) {  // diffuse: directional light + ambient, normal facing the camera
    float3 n = tri_normal(m, (uint32_t)p);
    const float3 d = pinhole_dir(cam, (int)(r % (uint32_t)cam.width), (int)(r / (uint32_t)cam.width));
    if (dot3(n.x, n.y, n.z, d.x, d.y, d.z) > 0.0f) n = make_float3(-n.x, -n.y, -n.z);
    const float diffuse = fmaxf(0.0f, dot3(n.x, n.y, n.z, light.x, light.y, light.z));
    // ambient + diffuse*0.85 and 0.7 + 0.3*|n|, contracted
    const float shade = fminf(1.0f, __fmaf_rn(diffuse, 0.85f, 0.15f));
    cr = __fmul_rn(shade, __fmaf_rn(0.3f, fabsf(n.x), 0.7f));
    cg = __fmul_rn(shade, __fmaf_rn(0.3f, fabsf(n.y), 0.7f));
    cb = __fmul_rn(shade, __fmaf_rn(0.3f, fabsf(n.z), 0.7f));
  } else if (mode == 3) {  // raw node visits (the heatmap colours them afterwards)
    cr = cg = cb = (float)in.vis[r];
  } else {  // unknown mode: magenta
    cr = 1.0f; cg = 0.0f; cb = 1.0f;
  }
  rgb[3 * (size_t)r + 0] = cr;
  rgb[3 * (size_t)r + 1] = cg;
  rgb[3 * (size_t)r + 2] = cb;
}

// The heatmap's normalisation (applyHeatmapColormap, :547-572): the value at index
// min(k - 1, floor(k * 0.999)) of the k nonzero visit counts in ascending order (128 when k = 0),
// at least 1.  Found by a two-level select on the counts' high and low 16 bits: histogram the
// high halves, find the bin holding that rank, histogram the low halves inside it.
// ctl: [0] k, [1] high half of the value, [2] rank inside that bin, [3] value.
__global__ void __launch_bounds__(256) k_heat_hist(const int32_t* __restrict__ vis, uint32_t np, int level,
                                                   uint32_t* __restrict__ hist, const uint32_t* __restrict__ ctl) {
  const uint32_t hi = level == 0 ? 0u : __ldcg(ctl + 1);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
    const int32_t c = vis[i];
    if (c <= 0) continue;
    const uint32_t u = (uint32_t)c;
    if (level == 0) atomicAdd(hist + (u >> 16), 1u);
    else if ((u >> 16) == hi) atomicAdd(hist + (u & 0xffffu), 1u);
  }
}

// One block of 1024 threads: level 0 counts k, picks the rank and finds its high-half bin;
// level 1 finds the rank inside the low-half histogram.
__global__ void __launch_bounds__(1024) k_heat_find(const uint32_t* __restrict__ hist, int level,
                                                    uint32_t* __restrict__ ctl) {
  constexpr int kBins = 65536, kPer = kBins / 1024;
  __shared__ uint32_t s_sum[1024];
  const int t = threadIdx.x;
  uint32_t sum = 0;
  for (int j = 0; j < kPer; ++j) sum += hist[t * kPer + j];
  s_sum[t] = sum;
  __syncthreads();
  // inclusive scan of the 1024 partial sums (Hillis-Steele)
  for (int o = 1; o < 1024; o <<= 1) {
    const uint32_t v = t >= o ? s_sum[t - o] : 0u;
    __syncthreads();
    s_sum[t] += v;
    __syncthreads();
  }
  const uint32_t total = s_sum[1023];
  uint32_t rank;
  if (level == 0) {
    if (total == 0) {
      if (t == 0) ctl[0] = 0;
      return;
    }
    const unsigned long long k = total;
    const unsigned long long q = (unsigned long long)((double)k * 0.999);
    rank = (uint32_t)(q < k - 1 ? q : k - 1);
  } else {
    rank = __ldcg(ctl + 2);
  }
  const uint32_t before = t ? s_sum[t - 1] : 0u;
  if (rank >= before && rank < s_sum[t]) {  // exactly one thread holds the rank
    uint32_t cum = before;
    for (int j = 0; j < kPer; ++j) {
      const uint32_t h = hist[t * kPer + j];
      if (rank < cum + h) {
        const uint32_t bin = (uint32_t)(t * kPer + j);
        if (level == 0) {
          ctl[0] = total;
          ctl[1] = bin;
          ctl[2] = rank - cum;
        } else {
          ctl[3] = (__ldcg(ctl + 1) << 16) | bin;
        }
        break;
      }
      cum += h;
    }
  }
}

// getTurboColor + the per-pixel loop of applyHeatmapColormap (:519-535, 574-594): t = count /
// max clamped to [0, 1], linear interpolation between the two nearest of 256 colormap entries;
// a count of 0 gets the background.
__global__ void __launch_bounds__(256) k_heat_color(const int32_t* __restrict__ vis, uint32_t np,
                                                    const float* __restrict__ lut, float fixed_max,
                                                    const uint32_t* __restrict__ ctl, float* __restrict__ rgb,
                                                    float* __restrict__ used_max) {
  float mx = fixed_max;
  if (!(mx > 0.0f)) {
    const uint32_t k = __ldcg(ctl + 0);
    mx = k == 0 ? 128.0f : fmaxf(1.0f, (float)__ldcg(ctl + 3));
  }
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && used_max) *used_max = mx;
  if (i >= np) return;
  const int32_t c = vis[i];
  float cr, cg, cb;
  if (c == 0) {
    cr = kBgR; cg = kBgG; cb = kBgB;
  } else {
    float t = fmaxf(0.0f, fminf(1.0f, __fdiv_rn((float)c, mx)));
    t = fmaxf(0.0f, fminf(1.0f, t));
    const float scaled = __fmul_rn(t, 255.0f);
    const int i0 = (int)scaled;
    const int i1 = min(i0 + 1, 255);
    const float frac = __fsub_rn(scaled, (float)i0);
    const float w0 = __fsub_rn(1.0f, frac);
    cr = __fadd_rn(__fmul_rn(__ldg(lut + 3 * i0 + 0), w0), __fmul_rn(__ldg(lut + 3 * i1 + 0), frac));
    cg = __fadd_rn(__fmul_rn(__ldg(lut + 3 * i0 + 1), w0), __fmul_rn(__ldg(lut + 3 * i1 + 1), frac));
    cb = __fadd_rn(__fmul_rn(__ldg(lut + 3 * i0 + 2), w0), __fmul_rn(__ldg(lut + 3 * i1 + 2), frac));
  }
  rgb[3 * (size_t)i + 0] = cr;
  rgb[3 * (size_t)i + 1] = cg;
  rgb[3 * (size_t)i + 2] = cb;
}

// savePPM's conversion (:502-507): clamp to [0, 1], v * 255 + 0.5, truncated to a byte.
__global__ void __launch_bounds__(256) k_rgb8(const float* __restrict__ rgb, uint32_t nv, uint8_t* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
    const float v = fmaxf(0.0f, fminf(1.0f, rgb[i]));
    out[i] = (uint8_t)__fadd_rn(__fmul_rn(v, 255.0f), 0.5f);
  }
}

cudaError_t shade_pixels(const PinholeCam& cam, const MeshPtrs& m, uint32_t n_tris, const ShadeIn& in, int mode,
                         float diag, float3 light, float* rgb, cudaStream_t st) {
  const uint32_t total = (uint32_t)cam.width * (uint32_t)cam.height;
  if (total == 0) return cudaSuccess;
  k_shade<<<div_up(total, 256), 256, 0, st>>>(cam, m, n_tris, in, mode, diag, light, rgb);
  return cudaGetLastError();
}

size_t heatmap_scratch_bytes() { return (size_t)2 * 65536 * 4 + 16 * 4; }

cudaError_t heatmap(const int32_t* vis, uint32_t np, const float* lut, float fixed_max, void* scratch, float* rgb,
                    float* used_max, cudaStream_t st) {
  if (np == 0) return cudaSuccess;
  uint32_t* h1 = static_cast<uint32_t*>(scratch);
  uint32_t* h2 = h1 + 65536;
  uint32_t* ctl = h2 + 65536;
  cudaError_t e;
  if (!(fixed_max > 0.0f)) {
    if ((e = cudaMemsetAsync(scratch, 0, heatmap_scratch_bytes(), st)) != cudaSuccess) return e;
    const uint32_t grid = std::min<uint32_t>(div_up(np, 256), 152 * 8);
    k_heat_hist<<<grid, 256, 0, st>>>(vis, np, 0, h1, ctl);
    k_heat_find<<<1, 1024, 0, st>>>(h1, 0, ctl);
    k_heat_hist<<<grid, 256, 0, st>>>(vis, np, 1, h2, ctl);
    k_heat_find<<<1, 1024, 0, st>>>(h2, 1, ctl);
  }
  k_heat_color<<<div_up(np, 256), 256, 0, st>>>(vis, np, lut, fixed_max, ctl, rgb, used_max);
  return cudaGetLastError();
}

cudaError_t rgb_to_bytes(const float* rgb, uint32_t nv, uint8_t* out, cudaStream_t st) {
  if (nv == 0) return cudaSuccess;
  k_rgb8<<<std::min<uint32_t>(div_up(nv, 256), 152 * 16), 256, 0, st>>>(rgb, nv, out);
  return cudaGetLastError();
}

cudaError_t trace_rays(const Node* nodes, int n_nodes, const MeshPtrs& m, uint32_t n_tris, const RayPtrs& rays,
                       uint32_t nr, const HitOut& out, TracePool* pool, cudaStream_t st) {
  if (nr == 0) return cudaSuccess;
  PackedTree T;
  const GivenRays given{rays};
  if (pack(pool, nodes, n_nodes, m, n_tris, given, nr, st, &T)) {
    // (launched plainly: started early, its blocks crowd the first SMs that k_pack leaves, 65,536 rays 448 -> 665 us)
    k_trace_packed<<<div_up(nr, kPackThreads), kPackThreads, 0, st>>>(T, given, nr, out);
    return unpack(T, st);
  }
  k_trace<<<div_up(nr, 128), 128, 0, st>>>(nodes, n_nodes, m, n_tris, rays, nr, out);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(128) k_trace_seg(const Node* __restrict__ nodes, MeshPtrs m, RayPtrs rays,
                                                   uint32_t nr, const RaySeg* __restrict__ segs, uint32_t count,
                                                   HitOut out) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nr) return;
  uint32_t lo = 0, hi = count;  // the last segment whose first ray is <= r
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&segs[mid].ray_begin) <= r) lo = mid;
    else hi = mid;
  }
  const RaySeg g = segs[lo];
  MeshPtrs mm;
#pragma unroll
  for (int k = 0; k < 9; ++k) mm.v[k] = m.v[k] + g.tri_base;
  const float3 o = make_float3(__ldg(rays.o[0] + r), __ldg(rays.o[1] + r), __ldg(rays.o[2] + r));
  const float3 d = make_float3(__ldg(rays.d[0] + r), __ldg(rays.d[1] + r), __ldg(rays.d[2] + r));
  trace_one(o, d, nodes + g.node_base, g.n_tris ? (int)(2 * g.n_tris - 1) : 0, mm, g.n_tris, r, out);
}

cudaError_t trace_rays_batched(const Node* nodes, const MeshPtrs& m, const RayPtrs& rays, uint32_t nr,
                               const RaySeg* segs, uint32_t count, const HitOut& out, cudaStream_t st) {
  if (nr == 0 || count == 0) return cudaSuccess;
  k_trace_seg<<<div_up(nr, 128), 128, 0, st>>>(nodes, m, rays, nr, segs, count, out);
  return cudaGetLastError();
}

// One piece (64 KB) per block iteration; 16-byte accesses where both sides allow.
__global__ void __launch_bounds__(256) k_copy_many(const CopyDesc* __restrict__ descs, uint32_t count,
                                                   uint32_t total_pieces) {
  for (uint32_t q = blockIdx.x; q < total_pieces; q += gridDim.x) {
    uint32_t lo = 0, hi = count;  // the last descriptor whose first piece is <= q
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__ldg(&descs[mid].first_piece) <= q) lo = mid;
      else hi = mid;
    }
    const CopyDesc c = descs[lo];
    const uint32_t b = (q - c.first_piece) * kCopyPiece;
    if (b >= c.n) continue;
    const uint32_t len = min(c.n - b, kCopyPiece);
    const float* src = c.src + b;
    float* dst = c.dst + b;
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
      const uint32_t n4 = len >> 2;
      for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x)
        reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
      for (uint32_t i = (n4 << 2) + threadIdx.x; i < len; i += blockDim.x) dst[i] = src[i];
    } else {
      for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) dst[i] = src[i];
    }
  }
}

cudaError_t copy_many(const CopyDesc* d_descs, uint32_t count, uint32_t total_pieces, cudaStream_t st) {
  if (count == 0 || total_pieces == 0) return cudaSuccess;
  k_copy_many<<<std::min<uint32_t>(total_pieces, 152 * 8), 256, 0, st>>>(d_descs, count, total_pieces);
  return cudaGetLastError();
}

cudaError_t trace_pinhole(const Node* nodes, int n_nodes, const MeshPtrs& m, uint32_t n_tris, const PinholeCam& cam,
                          const HitOut& out, TracePool* pool, cudaStream_t st) {
  uint32_t total = (uint32_t)cam.width * (uint32_t)cam.height;
  if (total == 0) return cudaSuccess;
  PackedTree T;
  if (pack(pool, nodes, n_nodes, m, n_tris, PixelRays{cam}, total, st, &T)) {
    const uint32_t warps = div_up(pinhole_tiles(cam.width, cam.height), 2);
    k_trace_pinhole_packed<<<div_up(warps, kPackThreads / 32), kPackThreads, 0, st>>>(T, cam, out);
    return unpack(T, st);
  }
  k_trace_pinhole<<<div_up(total, 128), 128, 0, st>>>(nodes, n_nodes, m, n_tris, cam, out);
  return cudaGetLastError();
}

cudaError_t pinhole_rays(const PinholeCam& cam, float* ox, float* oy, float* oz, float* dx, float* dy, float* dz,
                         cudaStream_t st) {
  uint32_t total = (uint32_t)cam.width * (uint32_t)cam.height;
  if (total == 0) return cudaSuccess;
  k_pinhole_rays<<<div_up(total, 256), 256, 0, st>>>(cam, ox, oy, oz, dx, dy, dz);
  return cudaGetLastError();
}

}  // namespace bvhgb

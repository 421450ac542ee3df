// ploc.cu -- PLOC (parallel locally-ordered clustering) on sm_103a.
//
// Reference: PLOCBuilderCUDA::build, src/cuda/ploc_builder.cu:403-586.  Same Morton-30 order,
// same leaves (node i = sorted triangle i), same nearest-neighbour rule (smallest union area in
// the window [i-r, i+r], first j on ties, :173-209), same mutual-pair merge (:211-264) and
// order-preserving compaction (:267-293), same root move to index 0 (:563-582).
//
// Differences by design: new node ids are handed out in ascending cluster order through a
// scan (the reference uses atomicAdd, so its ids vary run to run); merge and compaction share
// one reduce-then-scan over 2048-cluster tiles; and the iteration loop runs on the device as a CUDA
// graph WHILE node (the reference synchronises with the host five times per iteration,
// :489-548): a one-thread step kernel swaps the cluster buffers, stops on convergence, on an
// iteration that merges nothing (NaN/Inf areas, where the reference loops forever) or at the
// iteration cap, and sets the loop condition.
#include <algorithm>

#include "lbvh.cuh"

namespace bvhgb {

constexpr int kPlocThreads = 256;
constexpr int kPlocIpt = 8;
constexpr int kPlocTile = kPlocThreads * kPlocIpt;

// control words (scratch + L.ploc):
//   [0] live clusters  [1] next node id  [2] count ticket  [3] buffer parity
//   [4] survivors (next iteration)  [5] next node id (next iteration)  [6] iterations  [7] cap
//   [8..9] sum of live clusters over iterations (64-bit)  [10] go on (host-driven loop)
//   [11] meshes (1 for a single build): the loop ends at one cluster per mesh
//   [12] hand-over size: the loop stops at this many live clusters and k_ploc_tail finishes
//        (0: no hand-over)
//   [13] single builds: the node that took node 0 (sorted triangle 0's leaf) as its left child,
//        for the root fix (cluster 0 stays at position 0 until it merges, always as the left)
//   [14] single builds: the loop also stops at this many live clusters and k_ploc_grid goes on
//        (0: no hand-over)  [15] k_ploc_grid's barrier counter
//   [16] iterations run by k_ploc_grid  [17] iterations run by k_ploc_tail
//   [18] k_ploc_grid was launched  [19] k_ploc_tail was launched (launch accounting)
struct PlocBufs {
  Box* cbox[2];
  int32_t* cid[2];
  int32_t* nbr;
  uint2* flags;  // per (tile, warp, round): the merge and survivor ballots of 32 clusters
  unsigned long long* desc;
  Node* nodes;
  uint32_t* ctrl;
  uint32_t* status;
};

// Batched builds: per-mesh loop state.  seg[par * count + m] = position of mesh m's first live
// cluster (a mesh's first cluster always survives: it is never the larger index of a pair);
// id_base[m] = the mesh-local id of this iteration's first new node minus the global merge
// rank of the mesh's first cluster, so a merge's local id is id_base[m] + its global rank.
struct PlocSeg {
  const uint32_t* offsets;  // count + 1 triangle offsets
  uint32_t* seg;            // 2 * count (ping-pong with the cluster buffers' parity)
  uint32_t* id_base;        // count
  uint32_t count;
};

__global__ void k_ploc_init(const uint32_t* __restrict__ sidx, const Box* __restrict__ tri_boxes, PlocBufs B, uint32_t n,
                            uint32_t cap, uint32_t tail, uint32_t grid_at,
                            unsigned long long* __restrict__ stamps) {
  after_previous();
  stage_stamp(stamps, 3);
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    B.ctrl[0] = n;
    B.ctrl[1] = n;
    B.ctrl[2] = 0;
    B.ctrl[3] = 0;
    B.ctrl[6] = 0;
    B.ctrl[7] = cap;
    B.ctrl[8] = 0;
    B.ctrl[9] = 0;
    B.ctrl[11] = 1;
    B.ctrl[12] = tail;
    B.ctrl[13] = 0xffffffffu;
    B.ctrl[14] = grid_at;
#pragma unroll
    for (int k = 15; k < 20; ++k) B.ctrl[k] = 0;
  }
  if (i >= n) return;
  uint32_t prim = __ldg(sidx + i);
  const Box box = ld_box_cg(tri_boxes + prim);
  st_box(B.cbox[0] + i, box);
  B.cid[0][i] = (int32_t)i;
  float4* np = reinterpret_cast<float4*>(B.nodes + i);
  np[0] = box.lo;
  np[1] = box.hi;
  reinterpret_cast<int4*>(np + 2)[0] = make_int4((int32_t)(prim | kLeafBit), -1, 0, 0);
}

// Nearest neighbour in the +-r window (:173-209): the smallest union area, the smallest j on
// ties; areas that are NaN or infinite never win.  The area of a pair is symmetric (fminf/fmaxf
// commute), so each pair is evaluated once, by the thread of its earlier cluster x: it keeps x's
// forward best in registers and writes the area into a per-offset table D[k][j] for the later
// cluster j = x + k, which after a barrier reads its backward candidates from its column (the
// later offset, i.e. the smaller index, wins ties).  Offsets go in chunks of kNnKc to bound the
// table.  The r clusters before a tile ("halo") only fill the table; their pairs are spread over
// all warps.  Tiles of kNnTile clusters (kNnPer per thread, strided so lanes are consecutive),
// the window staged in shared memory.
constexpr int kNnPer = 4;
constexpr int kNnTile = kPlocThreads * kNnPer;
constexpr int kNnKc = 5;

__device__ __forceinline__ float pair_area(float4 xa, float4 xb, float4 ja, float4 jb) {
  return sa_xyz(__fsub_rn(fmaxf(xb.x, jb.x), fminf(xa.x, ja.x)), __fsub_rn(fmaxf(xb.y, jb.y), fminf(xa.y, ja.y)),
                __fsub_rn(fmaxf(xb.z, jb.z), fminf(xa.z, ja.z)));
}

// Batched builds keep each cluster's mesh in the w lane of its lo corner: a pair from two meshes
// has no area (+inf never wins), which clips every window at its mesh's boundary exactly as a
// single build's window ends at the ends of its cluster array.
template <bool SEG>
__device__ __forceinline__ float pair_d(float4 xa, float4 xb, float4 ja, float4 jb) {
  if (SEG && __float_as_int(xa.w) != __float_as_int(ja.w)) return __int_as_float(0x7f800000);
  return pair_area(xa, xb, ja, jb);
}

template <int PER, bool SEG>
__device__ __forceinline__ void nn_tiles(const PlocBufs& B, int r, uint32_t c, const Box* __restrict__ cbox,
                                         float4* sw) {
  constexpr int TILE = kPlocThreads * PER;
  // (TILE + 2r) boxes: all lo corners, then all hi corners (lanes read consecutive 16 bytes)
  float* sD = reinterpret_cast<float*>(sw + 2 * (TILE + 2 * r));  // [kNnKc][TILE]
  const int span = TILE + 2 * r;
  float4* s_lo = sw;
  float4* s_hi = sw + span;
  const int t = threadIdx.x;
  const float kInf = __int_as_float(0x7f800000);
  for (uint32_t base = blockIdx.x * (uint32_t)TILE; base < c; base += gridDim.x * (uint32_t)TILE) {
    const int lo = (int)base - r;  // window position 0; may be negative
    const int tile_n = (int)min((uint32_t)TILE, c - base);
    __syncthreads();  // previous tile's window no longer read
    for (int k = t; k < span; k += kPlocThreads) {
      const int j = lo + k;
      if (j >= 0 && j < (int)c) {
        const Box box = ld_box_cg(cbox + j);
        s_lo[k] = box.lo;
        s_hi[k] = box.hi;
      }
    }
    __syncthreads();
    float fd[PER], ed[PER];  // forward / backward best areas (+inf: none yet)
    int fj[PER], ej[PER];
    float4 xa[PER], xb[PER];
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      fd[m] = ed[m] = kInf;
      fj[m] = ej[m] = -1;
      const int xi = t + m * kPlocThreads;
      xa[m] = s_lo[min(xi + r, span - 1)];
      xb[m] = s_hi[min(xi + r, span - 1)];
    }
    // interior tile: every cluster has all r neighbours on both sides, so full offset chunks
    // take a path without bounds checks (fully unrolled)
    const bool interior = (int)base >= r && base + (uint32_t)TILE + (uint32_t)r <= c;
    for (int k0 = 1; k0 <= r; k0 += kNnKc) {
      const int kc = min(kNnKc, r - k0 + 1);
      const bool full = interior && kc == kNnKc;
      // pairs (x, x + k), k in [k0, k0 + kc): forward candidates of x, table entries for x + k
      if (full) {
#pragma unroll
        for (int m = 0; m < PER; ++m) {
          const int xi = t + m * kPlocThreads;
#pragma unroll
          for (int kk = 0; kk < kNnKc; ++kk) {
            const int jw = xi + r + k0 + kk;
            const float d = pair_d<SEG>(xa[m], xb[m], s_lo[jw], s_hi[jw]);
            if (d < fd[m]) {
              fd[m] = d;
              fj[m] = (int)base + xi + k0 + kk;
            }
            if (xi + k0 + kk < TILE) sD[kk * TILE + xi + k0 + kk] = d;
          }
        }
      } else {
#pragma unroll
        for (int m = 0; m < PER; ++m) {
          const int xi = t + m * kPlocThreads;
          if (xi < tile_n) {
            const int kmax = min(kc, (int)c - 1 - ((int)base + xi) - k0 + 1);  // j = base + xi + k < c
            for (int kk = 0; kk < kmax; ++kk) {
              const int jw = xi + r + k0 + kk;
              const float d = pair_d<SEG>(xa[m], xb[m], s_lo[jw], s_hi[jw]);
              if (d < fd[m]) {  // increasing j: the first of equal areas stays
                fd[m] = d;
                fj[m] = (int)base + xi + k0 + kk;
              }
              if (xi + k0 + kk < tile_n) sD[kk * TILE + xi + k0 + kk] = d;
            }
          }
        }
      }
      // halo pairs (h, jj) with jj < k: the table entries of the tile's first clusters
      for (int kk = 0; kk < kc; ++kk) {
        const int k = k0 + kk;
        const int rot = (k * 37) & (kPlocThreads - 1);  // spread each offset's pairs over the block
        for (int p = (t - rot) & (kPlocThreads - 1); p < k && p < tile_n; p += kPlocThreads) {
          const int h = (int)base + p - k;  // the halo cluster; p is the tile-relative target
          if (h >= 0) {
            const int hw = p - k + r;
            sD[kk * TILE + p] = pair_d<SEG>(s_lo[hw], s_hi[hw], s_lo[p + r], s_hi[p + r]);
          }
        }
      }
      __syncthreads();
      // backward candidates j - k of this thread's clusters
      if (full) {
#pragma unroll
        for (int m = 0; m < PER; ++m) {
          const int xi = t + m * kPlocThreads;
#pragma unroll
          for (int kk = 0; kk < kNnKc; ++kk) {
            const float d = sD[kk * TILE + xi];
            if (d < kInf && d <= ed[m]) {
              ed[m] = d;
              ej[m] = (int)base + xi - k0 - kk;
            }
          }
        }
      } else {
#pragma unroll
        for (int m = 0; m < PER; ++m) {
          const int xi = t + m * kPlocThreads;
          if (xi < tile_n) {
            for (int kk = 0; kk < kc; ++kk) {
              const int src = (int)base + xi - k0 - kk;
              if (src < 0) break;
              const float d = sD[kk * TILE + xi];
              if (d < kInf && d <= ed[m]) {  // later offset = smaller index: wins ties
                ed[m] = d;
                ej[m] = src;
              }
            }
          }
        }
      }
      __syncthreads();  // the table is refilled by the next chunk
    }
#pragma unroll
    for (int m = 0; m < PER; ++m) {
      const int xi = t + m * kPlocThreads;
      if (xi < tile_n) B.nbr[base + xi] = (ej[m] >= 0 && ed[m] <= fd[m]) ? ej[m] : fj[m];  // earlier index wins ties
    }
  }
}

// Searches that keep no areas compare halves: doubling is exact, so the order is the same, and a half below
// 2^127 is an area below infinity.
constexpr float kHalfInf = 0x1p127f;
__device__ __forceinline__ float pair_half(float4 xa, float4 xb, float4 ja, float4 jb) {
  const float dx = __fsub_rn(fmaxf(xb.x, jb.x), fminf(xa.x, ja.x)), dy = __fsub_rn(fmaxf(xb.y, jb.y), fminf(xa.y, ja.y)),
              dz = __fsub_rn(fmaxf(xb.z, jb.z), fminf(xa.z, ja.z));
  return __fmaf_rn(dz, dx, __fmaf_rn(dx, dy, __fmul_rn(dy, dz)));
}

// The large iterations take a second form of the same search (ploc_builder.cu:173-209): thread t owns kNcP
// consecutive clusters x0 .. x0 + 3, so each window box it loads serves all four (r + 3 loads for 4r pairs),
// and the backward candidates it produces for one later cluster are reduced to one before they go
// through the shared-memory table, a distance q of threads at a time.  The first h = ceil(r / kNcP)
// threads of a tile hold the r clusters before it: they only feed backward candidates.  One box in nine
// of the window's storage is unused, which puts the 16-byte boxes that 8 lanes read -- every fourth
// box, or 8 consecutive ones -- in distinct bank groups at constant offsets from a thread's first.
// What bounds it is instructions (the six min/max of a pair on the half-rate pipe, three blocks per SM
// by registers), and what it loads waits on L1, whose lines loads in flight need and the window takes:
// pairs past the last distances' ends only are checked against r, areas are halves, and the table
// holds one distance.  First iteration on 10M: r = 25
// 319 -> 275 us, r = 100 (nc_tile_min) 1,071 -> 826.
// Two pairs per packed add or multiply took longer than two single ones (its operands are moved into place).
constexpr int kNcP = 4;      // consecutive clusters per thread
constexpr int kNcMaxR = 128;  // larger radii keep the strided form (a halo of 32 threads at 128)
// From here on nc_tile_min: settling indexes at the end costs as much as 30 radii of keeping them (4M, whole loop:
// r = 10 1,674 against 1,566 us, 25 2,363 / 2,325, 32 2,595 / 2,629, 64 3,818 / 4,045).
constexpr int kNcMinR = 32;
__host__ __device__ constexpr int nc_at(int w) { return w + (w >> 3); }
// boxes staged: the halo, the tile, r past it, + kNcP read past the last pair; rounded to 8
__host__ __device__ constexpr int nc_span(int r) { return nc_at((kPlocThreads * kNcP + r + kNcP + 7) & ~7); }
// per thread, the table holds a distance's four (area, index) twice, or its four areas once
__host__ __device__ constexpr int nc_table(int r) { return (r < kNcMinR ? 4 : 1) * (kPlocThreads + (r + kNcP - 1) / kNcP); }
static size_t nc_smem(int r) { return 16 * (2 * (size_t)nc_span(r) + nc_table(r)); }

template <bool SEG>
__device__ __forceinline__ float nc_half(float4 xa, float4 xb, float4 ja, float4 jb) {
  if (SEG && __float_as_int(xa.w) != __float_as_int(ja.w)) return kHalfInf;  // (two meshes: no area)
  return pair_half(xa, xb, ja, jb);
}

// The thread's clusters against box j = x0 + o (those with m < o <= m + r): fd, fj and the smallest of the four,
// with its index.
template <bool SEG, bool CHECK, bool EDGE>
__device__ __forceinline__ float2 nc_four(int r, int c, int x0, int o, const float4 (&a)[kNcP],
                                          const float4 (&b)[kNcP], float4 jl, float4 jh, float (&fd)[kNcP],
                                          int (&fj)[kNcP]) {
  static_assert(kNcP == 4, "two halves");
  float t[2];
  int i[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    t[k] = kHalfInf;
    i[k] = 2 * k;
    if (EDGE && (o <= 2 * k || o - 2 * k - 1 > r)) continue;  // (the same for every thread)
    float d[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int m = 2 * k + e;
      d[e] = nc_half<SEG>(a[m], b[m], jl, jh);
      if (EDGE && (o <= m || o - m > r)) d[e] = kHalfInf;
      if (CHECK && !(x0 + m >= 0 && x0 + o < c)) d[e] = kHalfInf;
      if (d[e] < fd[m]) {  // increasing o: the first of equal areas stays
        fd[m] = d[e];
        fj[m] = o;
      }
    }
    t[k] = fminf(d[0], d[1]);  // (NaN only where both are)
    if (t[k] != d[0]) i[k] = 2 * k + 1;
  }
  const float m = fminf(t[0], t[1]);
  return make_float2(m, __int_as_float(x0 + (m == t[0] ? i[0] : i[1])));
}

// Group q, the clusters of thread t + q, whose table entry is col.
template <bool SEG, bool CHECK, bool EDGE>
__device__ __forceinline__ void nc_group(int r, int c, int x0, int q, const float4 (&a)[kNcP], const float4 (&b)[kNcP],
                                         const float4* s_lo, const float4* s_hi, float4* col, int tw,
                                         float (&fd)[kNcP], int (&fj)[kNcP]) {
  const int w = nc_at(kNcP * ((int)threadIdx.x + q));  // (four boxes from a multiple of four on are adjacent)
  const float4* lo = s_lo + w;
  const float4* hi = s_hi + w;
#pragma unroll
  for (int mp = 0; mp < kNcP; mp += 2) {
    const float2 e = nc_four<SEG, CHECK, EDGE>(r, c, x0, kNcP * q + mp, a, b, lo[mp], hi[mp], fd, fj);
    const float2 f = nc_four<SEG, CHECK, EDGE>(r, c, x0, kNcP * q + mp + 1, a, b, lo[mp + 1], hi[mp + 1], fd, fj);
    col[mp / 2 * tw] = make_float4(e.x, e.y, f.x, f.y);
  }
}

template <bool SEG, bool CHECK>
__device__ __forceinline__ void nc_tile(const PlocBufs& B, int r, int c, int lo, int h, const float4* s_lo,
                                        const float4* s_hi, float4* sT) {
  constexpr int P = kNcP;
  const int t = threadIdx.x, tw = kPlocThreads + h;
  const int x0 = lo + P * t;
  float4 a[P], b[P];
  float fd[P], ed[P];
  int fj[P], ej[P];  // fj: relative to x0
#pragma unroll
  for (int m = 0; m < P; ++m) {
    a[m] = s_lo[nc_at(P * t) + m];
    b[m] = s_hi[nc_at(P * t) + m];
    fd[m] = ed[m] = kHalfInf;
    fj[m] = 0;
    ej[m] = -1;
  }
  // pairs among the thread's own clusters
#pragma unroll
  for (int o = 1; o < P; ++o) {
    const float2 e = nc_four<SEG, CHECK, true>(r, c, x0, o, a, b, a[o], b[o], fd, fj);
    if (e.x < kHalfInf) {
      ed[o] = e.x;
      ej[o] = __float_as_int(e.y);
    }
  }
  // pairs with the clusters of the threads q = 1 .. h further on; every pair up to distance qf is within r
  const int qf = r >= P - 1 ? (r - (P - 1)) / P : 0;
  for (int q = 1, buf = 0; q <= h; ++q, buf ^= P / 2 * tw) {
    if (q <= qf) nc_group<SEG, CHECK, false>(r, c, x0, q, a, b, s_lo, s_hi, sT + buf + t + q, tw, fd, fj);
    else nc_group<SEG, CHECK, true>(r, c, x0, q, a, b, s_lo, s_hi, sT + buf + t + q, tw, fd, fj);
    __syncthreads();
#pragma unroll
    for (int mp = 0; mp < P; mp += 2) {
      const float4 e = sT[buf + mp / 2 * tw + t];
      if (e.x <= ed[mp]) {  // a larger distance has the smaller indices: it wins ties
        ed[mp] = e.x;
        ej[mp] = __float_as_int(e.y);
      }
      if (e.z <= ed[mp + 1]) {
        ed[mp + 1] = e.z;
        ej[mp + 1] = __float_as_int(e.w);
      }
    }
  }
  if (t >= h) {
#pragma unroll
    for (int m = 0; m < P; ++m) {
      const int x = x0 + m;
      // the earlier index wins ties
      if (x < c) B.nbr[x] = ed[m] < kHalfInf && ed[m] <= fd[m] ? ej[m] : fd[m] < kHalfInf ? x0 + fj[m] : -1;
    }
  }
}

// The thread's four clusters against box j = x0 + o: d[m], kHalfInf where not m < o <= m + r.
template <bool SEG, bool CHECK, bool EDGE>
__device__ __forceinline__ void nc_areas(int r, int c, int x0, int o, const float4 (&a)[kNcP], const float4 (&b)[kNcP],
                                        float4 jl, float4 jh, float (&d)[kNcP]) {
#pragma unroll
  for (int m = 0; m < kNcP; ++m) {
    d[m] = kHalfInf;
    if (EDGE && (o <= m || o - m > r)) continue;  // (the same for every thread)
    d[m] = nc_half<SEG>(a[m], b[m], jl, jh);
    if (CHECK && !(x0 + m >= 0 && x0 + o < c)) d[m] = kHalfInf;
  }
}
template <bool SEG, bool CHECK, bool EDGE>
__device__ __forceinline__ void nc_group_min(int r, int c, int x0, int q, const float4 (&a)[kNcP], const float4 (&b)[kNcP],
                                         const float4* s_lo, const float4* s_hi, float4* col, float (&fm)[kNcP]) {
  static_assert(kNcP == 4, "one float4 of the table");
  const int w = nc_at(kNcP * ((int)threadIdx.x + q));
  const float4* lo = s_lo + w;
  const float4* hi = s_hi + w;
  float e[kNcP];
#pragma unroll
  for (int mp = 0; mp < kNcP; ++mp) {
    float d[kNcP];
    nc_areas<SEG, CHECK, EDGE>(r, c, x0, kNcP * q + mp, a, b, lo[mp], hi[mp], d);
#pragma unroll
    for (int m = 0; m < kNcP; ++m) fm[m] = mp == 0 ? d[m] : fminf(fm[m], d[m]);
    e[mp] = fminf(fminf(d[0], d[1]), fminf(d[2], d[3]));
  }
  *col = make_float4(e[0], e[1], e[2], e[3]);
}

// The form of radii from kNcMinR on keeps only smallest areas, with the group q of four clusters -- thread t + q's
// or t - q's -- that they were seen in, and settles the index at the end, once per cluster: the winning
// group's four areas are computed again (the same bits) and the first that equals the minimum is the
// neighbour.
template <bool SEG, bool CHECK>
__device__ __forceinline__ void nc_tile_min(const PlocBufs& B, int r, int c, int lo, int h, const float4* s_lo,
                                        const float4* s_hi, float4* sT) {
  constexpr int P = kNcP;
  const int t = threadIdx.x;
  const int x0 = lo + P * t;
  float4 a[P], b[P];
  float fd[P], ed[P];
  uint32_t fe[P];  // the groups of fd (low half) and ed
#pragma unroll
  for (int m = 0; m < P; ++m) {
    a[m] = s_lo[nc_at(P * t) + m];
    b[m] = s_hi[nc_at(P * t) + m];
    fd[m] = ed[m] = kHalfInf;
    fe[m] = 0;
  }
  // group 0, the thread's own clusters
#pragma unroll
  for (int o = 1; o < P; ++o) {
    float d[P];
    nc_areas<SEG, CHECK, true>(r, c, x0, o, a, b, a[o], b[o], d);
#pragma unroll
    for (int m = 0; m < P; ++m)
      if (m < o) {
        fd[m] = fminf(fd[m], d[m]);
        ed[o] = fminf(ed[o], d[m]);
      }
  }
  // groups 1 .. h; every pair of groups up to qf is within r
  const int qf = r >= P - 1 ? (r - (P - 1)) / P : 0;
  for (int q = 1; q <= h; ++q) {
    float fm[P];
    if (q <= qf) nc_group_min<SEG, CHECK, false>(r, c, x0, q, a, b, s_lo, s_hi, sT + t + q, fm);
    else nc_group_min<SEG, CHECK, true>(r, c, x0, q, a, b, s_lo, s_hi, sT + t + q, fm);
#pragma unroll
    for (int m = 0; m < P; ++m)
      if (fm[m] < fd[m]) {  // increasing distance: the first of equal areas stays
        fd[m] = fm[m];
        fe[m] = __byte_perm(fe[m], q, 0x3254);
      }
    __syncthreads();
    const float4 e4 = sT[t];
    const float e[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
    for (int mp = 0; mp < P; ++mp)
      if (e[mp] <= ed[mp]) {  // a larger distance has the smaller indices: it wins ties
        ed[mp] = e[mp];
        fe[mp] = __byte_perm(fe[mp], q, 0x5410);
      }
    __syncthreads();  // the table is refilled by the next distance
  }
  if (t < h) return;
#pragma unroll
  for (int m = 0; m < P; ++m) {
    const int x = x0 + m;
    if (x >= c) break;
    const bool back = ed[m] <= fd[m];  // the earlier index wins ties
    const float best = back ? ed[m] : fd[m];
    int nb = -1;
    if (best < kHalfInf) {
      const int g = back ? t - (int)(fe[m] >> 16) : t + (int)(fe[m] & 0xffffu), y0 = lo + P * g;
      const int lim0 = back ? max(x - r, 0) : x + 1, lim1 = back ? x - 1 : min(x + r, c - 1);
      const float4* gl = s_lo + nc_at(P * g);
      const float4* gh = s_hi + nc_at(P * g);
#pragma unroll
      for (int mp = P - 1; mp >= 0; --mp)  // descending: the smallest index stays
        if (nc_half<SEG>(gl[mp], gh[mp], a[m], b[m]) == best && y0 + mp >= lim0 && y0 + mp <= lim1) nb = y0 + mp;
    }
    B.nbr[x] = nb;
  }
}

template <bool SEG, bool MIN>
__device__ __forceinline__ void nn_tiles_consec(const PlocBufs& B, int r, uint32_t c, const Box* __restrict__ cbox,
                                                float4* sw) {
  const int h = (r + kNcP - 1) / kNcP;            // halo threads = the largest thread distance of a pair
  const int out = (kPlocThreads - h) * kNcP;      // clusters a tile decides
  const int span = kPlocThreads * kNcP + r;       // boxes staged: the halo, the tile, r past it
  float4* s_lo = sw;
  float4* s_hi = sw + nc_span(r);
  float4* sT = s_hi + nc_span(r);
  const int t = threadIdx.x;
  for (uint32_t tb = blockIdx.x * (uint32_t)out; tb < c; tb += gridDim.x * (uint32_t)out) {
    const int lo = (int)tb - kNcP * h;  // window position 0; may be negative
    __syncthreads();                    // previous tile's window no longer read
    for (int k = t; k < span; k += kPlocThreads) {
      const int j = lo + k;
      if (j >= 0 && j < (int)c) {
        const Box box = ld_box_cg(cbox + j);
        s_lo[nc_at(k)] = box.lo;
        s_hi[nc_at(k)] = box.hi;
      }
    }
    __syncthreads();
    const bool inside = lo >= 0 && lo + span <= (int)c;
    if constexpr (MIN) {
      if (inside) nc_tile_min<SEG, false>(B, r, (int)c, lo, h, s_lo, s_hi, sT);
      else nc_tile_min<SEG, true>(B, r, (int)c, lo, h, s_lo, s_hi, sT);
    } else {
      if (inside) nc_tile<SEG, false>(B, r, (int)c, lo, h, s_lo, s_hi, sT);
      else nc_tile<SEG, true>(B, r, (int)c, lo, h, s_lo, s_hi, sT);
    }
  }
}

template <bool SEG, bool MIN>  // (MIN: r >= kNcMinR; both forms in one kernel cost each 2%)
__global__ void __launch_bounds__(kPlocThreads, 3) k_ploc_nn(PlocBufs B, int r) {
  extern __shared__ float4 sw[];
  const uint32_t c = __ldcg(B.ctrl + 0);
  const Box* __restrict__ cbox = (__ldcg(B.ctrl + 3) & 1u) ? B.cbox[1] : B.cbox[0];  // no stack copy of B
  // Once the live clusters no longer fill the grid with 4-per-thread tiles, an iteration lasts
  // one tile's latency: smaller tiles (2 or 1 clusters per thread) then spread it over more
  // blocks.  The result does not depend on the tiling.
  const uint32_t g = gridDim.x * (uint32_t)kPlocThreads;
  if (c > 2u * g && r <= kNcMaxR) nn_tiles_consec<SEG, MIN>(B, r, c, cbox, sw);
  else if (c > 2u * g) nn_tiles<kNnPer, SEG>(B, r, c, cbox, sw);
  else if (c > g) nn_tiles<2, SEG>(B, r, c, cbox, sw);
  else nn_tiles<1, SEG>(B, r, c, cbox, sw);
}

// Merge mutual pairs (i < j keeps position i, :211-264) and compact the survivors (:267-293),
// as reduce-then-scan: k_ploc_count totals each tile of 256 R clusters (R <= 8 rounds per warp)
// and stores its ballots, its last block scans the tile totals, k_ploc_scatter reads the ballots
// and writes, k_ploc_step ends the iteration.  Warp w of a tile takes its items w*32R + r*32 +
// lane in R rounds r of 32 consecutive clusters, so positions within the warp come from ballots
// and new node ids follow the cluster order whatever R is.  Counts are packed as
// merges << 31 | survivors.
constexpr int kPlocRounds = kPlocTile / kPlocThreads;  // 8

// Item i merges here (as the smaller index of a mutual pair) / survives, from its neighbour j
// and j's neighbour `back` (-1 where not loaded).
__device__ __forceinline__ void item_flags(uint32_t c, uint32_t i, int32_t j, int32_t back, bool& m, bool& v) {
  const bool mutual = i < c && j >= 0 && (uint32_t)j < c && back == (int32_t)i;
  m = mutual && (int32_t)i < j;
  v = i < c && !(mutual && j < (int32_t)i);
}

// End of one iteration: publish the survivors, swap buffers, decide whether to go on (the
// graph's WHILE condition, or ctrl[10] for the host-driven loop).
template <bool GRAPH>
__device__ __forceinline__ void ploc_step(PlocBufs B, cudaGraphConditionalHandle handle) {
  const uint32_t c = B.ctrl[0], nc = B.ctrl[4], it = B.ctrl[6] + 1, cap = B.ctrl[7];
  unsigned long long sum = ((unsigned long long)B.ctrl[9] << 32 | B.ctrl[8]) + c;
  B.ctrl[8] = (uint32_t)sum;
  B.ctrl[9] = (uint32_t)(sum >> 32);
  B.ctrl[6] = it;
  B.ctrl[0] = nc;
  B.ctrl[1] = B.ctrl[5];
  B.ctrl[3] ^= 1u;
  bool go = nc > B.ctrl[11];
  if (go && (nc >= c || it >= cap)) {  // no mutual pair anywhere, or the cap: stop and report
    atomicOr(B.status, kStatusNoProgress);
    go = false;
  } else if (go && (nc <= B.ctrl[12] || nc <= B.ctrl[14])) {  // k_ploc_grid / k_ploc_tail go on
    go = false;
  }
  if constexpr (GRAPH) cudaGraphSetConditional(handle, go ? 1u : 0u);
  else B.ctrl[10] = go ? 1u : 0u;
}

// Exclusive prefix of the tile totals (in place), the survivors and the next node id; run by
// the last block of k_ploc_count.
__device__ __forceinline__ void ploc_scan_tiles(PlocBufs B, uint32_t tiles, unsigned long long* s_w) {
  const uint32_t per = div_up(tiles, (uint32_t)kPlocThreads);
  const uint32_t t0 = threadIdx.x * per, t1 = min(t0 + per, tiles);
  unsigned long long sum = 0;
  for (uint32_t t = t0; t < t1; ++t) sum += __ldcg(B.desc + t);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[w] = x;
  __syncthreads();
  unsigned long long run = x - sum, total = 0;
#pragma unroll
  for (int k = 0; k < kPlocThreads / 32; ++k) {
    if (k < w) run += s_w[k];
    total += s_w[k];
  }
  for (uint32_t t = t0; t < t1; ++t) {
    const unsigned long long v = __ldcg(B.desc + t);
    B.desc[t] = run;
    run += v;
  }
  if (threadIdx.x == 0) {
    B.ctrl[4] = (uint32_t)(total & 0x7fffffffull);             // survivors
    B.ctrl[5] = __ldcg(B.ctrl + 1) + (uint32_t)(total >> 31);  // next node id
  }
}

// Rounds of 32 clusters per warp in a merge tile (8 at most, 2048 clusters per tile): the fewest
// whose tiles still fill the grid, so that late iterations (few clusters) spread over all blocks.
// k_ploc_count and k_ploc_scatter run on the same grid and agree on it.
__device__ __forceinline__ int ploc_rounds(uint32_t c, uint32_t grid) {
#pragma unroll
  for (int r = 1; r < kPlocRounds; r <<= 1)
    if (div_up(c, (uint32_t)(kPlocThreads * r)) <= grid) return r;
  return kPlocRounds;
}
__device__ __forceinline__ int ploc_rounds(uint32_t c) { return ploc_rounds(c, gridDim.x); }

template <int R>
__device__ __forceinline__ void count_tiles(const PlocBufs& B, uint32_t c, uint32_t tiles, unsigned long long* s_w) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t base = tile * (uint32_t)(kPlocThreads * R) + w * (32u * R);
    // all rounds' neighbours, then their neighbours, so that each load batch is in flight at once
    int32_t j[R], back[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t i = base + r * 32 + lane;
      j[r] = i < c ? __ldcg(B.nbr + i) : -1;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) back[r] = (j[r] >= 0 && (uint32_t)j[r] < c) ? __ldcg(B.nbr + j[r]) : -1;
    uint32_t tm = 0, tv = 0;
    uint2 mine = make_uint2(0u, 0u);  // lane r keeps round r's ballots
#pragma unroll
    for (int r = 0; r < R; ++r) {
      bool m, v;
      item_flags(c, base + r * 32 + lane, j[r], back[r], m, v);
      const uint32_t mb = __ballot_sync(0xffffffffu, m), vb = __ballot_sync(0xffffffffu, v);
      if (lane == r) mine = make_uint2(mb, vb);
      tm += __popc(mb);
      tv += __popc(vb);
    }
    if (lane < R) B.flags[((size_t)tile * (kPlocThreads / 32) + w) * R + lane] = mine;
    if (lane == 0) s_w[w] = ((unsigned long long)tm << 31) | tv;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t = 0;
#pragma unroll
      for (int k = 0; k < kPlocThreads / 32; ++k) t += s_w[k];
      B.desc[tile] = t;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kPlocThreads) k_ploc_count(PlocBufs B) {
  __shared__ unsigned long long s_w[kPlocThreads / 32];
  const uint32_t c = __ldcg(B.ctrl + 0);
  const int R = ploc_rounds(c);
  const uint32_t tiles = div_up(c, (uint32_t)(kPlocThreads * R));
  switch (R) {
    case 1: count_tiles<1>(B, c, tiles, s_w); break;
    case 2: count_tiles<2>(B, c, tiles, s_w); break;
    case 4: count_tiles<4>(B, c, tiles, s_w); break;
    default: count_tiles<kPlocRounds>(B, c, tiles, s_w); break;
  }
  // the last block to finish scans the tile totals (ticket in ctrl[2])
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(B.ctrl + 2, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  ploc_scan_tiles(B, tiles, s_w);
  if (threadIdx.x == 0) B.ctrl[2] = 0;
}

template <int R, bool SEG>
__device__ __forceinline__ void scatter_tiles(const PlocBufs& B, uint32_t c, uint32_t next, uint32_t tiles,
                                              const Box* __restrict__ cin, const int32_t* __restrict__ idin,
                                              Box* __restrict__ cout, int32_t* __restrict__ idout,
                                              Node* __restrict__ nodes, unsigned long long* s_w,
                                              const PlocSeg& S) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t base = tile * (uint32_t)(kPlocThreads * R) + w * (32u * R);
    uint32_t mb[R], vb[R];
    int32_t nj[R];
    uint32_t tm = 0, tv = 0;
    // the ballots k_ploc_count stored; the partner of each merging cluster
    const uint2* fl = B.flags + ((size_t)tile * (kPlocThreads / 32) + w) * R;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint2 f = __ldcg(fl + r);
      mb[r] = f.x;
      vb[r] = f.y;
      nj[r] = ((f.x >> lane) & 1u) ? __ldcg(B.nbr + base + r * 32 + lane) : -1;
      tm += __popc(mb[r]);
      tv += __popc(vb[r]);
    }
    if (lane == 0) s_w[w] = ((unsigned long long)tm << 31) | tv;
    __syncthreads();
    unsigned long long before = __ldcg(B.desc + tile);
#pragma unroll
    for (int k = 0; k < kPlocThreads / 32; ++k)
      if (k < w) before += s_w[k];
    __syncthreads();  // s_w is rewritten by the next tile
    uint32_t mpos = (uint32_t)(before >> 31), vpos = (uint32_t)(before & 0x7fffffffull);
    // two rounds at a time: both rounds' boxes and ids are loaded before either round stores
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += 2) {
      float4 lo[2], hi[2], jlo[2], jhi[2];
      int32_t id[2], jid[2];
#pragma unroll
      for (int g = 0; g < 2 && r0 + g < R; ++g) {
        const int r = r0 + g;
        const uint32_t i = base + r * 32 + lane;
        const bool m = (mb[r] >> lane) & 1u, v = (vb[r] >> lane) & 1u;
        lo[g] = hi[g] = jlo[g] = jhi[g] = make_float4(0.f, 0.f, 0.f, 0.f);
        id[g] = jid[g] = 0;
        if (m || v) {
          const Box x = ld_box_cg(cin + i);
          lo[g] = x.lo;
          hi[g] = x.hi;
          id[g] = __ldcg(idin + i);
        }
        if (m) {
          const Box y = ld_box_cg(cin + nj[r]);
          jlo[g] = y.lo;
          jhi[g] = y.hi;
          jid[g] = __ldcg(idin + nj[r]);
        }
      }
#pragma unroll
      for (int g = 0; g < 2 && r0 + g < R; ++g) {
        const int r = r0 + g;
        const bool m = (mb[r] >> lane) & 1u, v = (vb[r] >> lane) & 1u;
        float4 a = lo[g], b = hi[g];
        int32_t nid = id[g];
        if (m) {
          // a batched cluster keeps its mesh in lo.w; nodes get 0 there
          a = make_float4(fminf(a.x, jlo[g].x), fminf(a.y, jlo[g].y), fminf(a.z, jlo[g].z), SEG ? a.w : 0.f);
          b = make_float4(fmaxf(b.x, jhi[g].x), fmaxf(b.y, jhi[g].y), fmaxf(b.z, jhi[g].z), 0.f);
          float4* np;
          np = nullptr;
          if constexpr (SEG) {
            const uint32_t mesh = (uint32_t)__float_as_int(a.w);
            const uint32_t local = mesh < S.count ? __ldcg(S.id_base + mesh) + mpos + __popc(mb[r] & lt) : ~0u;
            nid = (int32_t)local;  // children and cluster ids are mesh-local
            if (mesh < S.count) {
              const uint32_t off = __ldg(S.offsets + mesh), nm = __ldg(S.offsets + mesh + 1) - off;
              if (local < 2 * nm - 1) np = reinterpret_cast<float4*>(nodes + (2 * (size_t)off - mesh) + local);
            }
            if (!np) atomicOr(B.status, kStatusBadInput);  // outside its mesh's range: skipped
          } else {
            nid = (int32_t)(next + mpos + __popc(mb[r] & lt));
            np = reinterpret_cast<float4*>(nodes + nid);
            if (id[g] == 0) B.ctrl[13] = (uint32_t)nid;  // node 0's parent, for the root fix
          }
          if (np) {
            np[0] = make_float4(a.x, a.y, a.z, 0.f);
            np[1] = b;
            reinterpret_cast<int4*>(np + 2)[0] = make_int4(id[g], jid[g], 0, 0);
          }
        }
        if (v) {
          const uint32_t o = vpos + __popc(vb[r] & lt);
          st_box(cout + o, Box{a, b});
          idout[o] = nid;
        }
        mpos += __popc(mb[r]);
        vpos += __popc(vb[r]);
      }
    }
  }
}

template <bool SEG>
__global__ void __launch_bounds__(kPlocThreads, 3) k_ploc_scatter(PlocBufs B, PlocSeg S) {
  __shared__ unsigned long long s_w[kPlocThreads / 32];
  const uint32_t c = __ldcg(B.ctrl + 0);
  const uint32_t next = __ldcg(B.ctrl + 1);
  const uint32_t par = __ldcg(B.ctrl + 3) & 1u;
  // selects, not an indexed parameter array (which would be copied to the stack)
  const Box* __restrict__ cin = par ? B.cbox[1] : B.cbox[0];
  const int32_t* __restrict__ idin = par ? B.cid[1] : B.cid[0];
  Box* __restrict__ cout = par ? B.cbox[0] : B.cbox[1];
  int32_t* __restrict__ idout = par ? B.cid[0] : B.cid[1];
  Node* __restrict__ nodes = B.nodes;
  const int R = ploc_rounds(c);
  const uint32_t tiles = div_up(c, (uint32_t)(kPlocThreads * R));
  switch (R) {
    case 1: scatter_tiles<1, SEG>(B, c, next, tiles, cin, idin, cout, idout, nodes, s_w, S); break;
    case 2: scatter_tiles<2, SEG>(B, c, next, tiles, cin, idin, cout, idout, nodes, s_w, S); break;
    case 4: scatter_tiles<4, SEG>(B, c, next, tiles, cin, idin, cout, idout, nodes, s_w, S); break;
    default: scatter_tiles<kPlocRounds, SEG>(B, c, next, tiles, cin, idin, cout, idout, nodes, s_w, S); break;
  }
}

// Batched builds, between k_ploc_count (whose last block has scanned the tile totals) and
// k_ploc_scatter: per mesh, the global merge and survivor ranks of its first live cluster, from
// its tile's prefix and the stored ballots before it in the tile (at most 64 words).  From them
// the mesh's id base (a merge's local id = id_base + its global rank) and the position of its
// first cluster after the compaction.  mg_grid = the grid of k_ploc_count / k_ploc_scatter,
// which fixes their tiling.
__global__ void __launch_bounds__(256) k_ploc_seg(PlocBufs B, PlocSeg S, uint32_t mg_grid) {
  const uint32_t c = __ldcg(B.ctrl + 0);
  const uint32_t par = __ldcg(B.ctrl + 3) & 1u;
  const int R = ploc_rounds(c, mg_grid);
  const uint32_t per_tile = (uint32_t)kPlocThreads * (uint32_t)R, per_warp = 32u * (uint32_t)R;
  const uint32_t* seg_in = S.seg + (size_t)par * S.count;
  uint32_t* seg_out = S.seg + (size_t)(par ^ 1u) * S.count;
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < S.count; m += gridDim.x * blockDim.x) {
    const uint32_t p = seg_in[m];
    const uint32_t pe = m + 1 < S.count ? seg_in[m + 1] : c;
    if (p >= c || pe > c || pe <= p) {  // inconsistent loop state: no ranks for this mesh
      atomicOr(B.status, kStatusBadInput);
      S.id_base[m] = ~0u;
      seg_out[m] = p;
      continue;
    }
    const uint32_t nm = __ldg(S.offsets + m + 1) - __ldg(S.offsets + m);
    const uint32_t tile = p / per_tile, o = p - tile * per_tile;
    const uint32_t w = o / per_warp, rr = (o % per_warp) >> 5, lane = o & 31u;
    const uint2* fl = B.flags + (size_t)tile * (kPlocThreads / 32) * R;
    uint32_t mc = 0, vc = 0;
    for (uint32_t k = 0; k < w * (uint32_t)R + rr; ++k) {  // whole rounds before p's round
      const uint2 f = __ldcg(fl + k);
      mc += __popc(f.x);
      vc += __popc(f.y);
    }
    const uint2 f = __ldcg(fl + w * (uint32_t)R + rr);
    const uint32_t below = (1u << lane) - 1u;
    mc += __popc(f.x & below);
    vc += __popc(f.y & below);
    const unsigned long long pre = __ldcg(B.desc + tile);
    const uint32_t G = (uint32_t)(pre >> 31) + mc, V = (uint32_t)(pre & 0x7fffffffull) + vc;
    // local id of the next new node = n_m + merges so far = 2 n_m - live clusters
    S.id_base[m] = 2u * nm - (pe - p) - G;
    seg_out[m] = V;
  }
}

// Batched builds: leaves and clusters from the sorted order of all meshes (positions
// [offsets[m], offsets[m+1]) hold mesh m's triangles in its own Morton order).  Mesh m's tree
// starts at node 2 offsets[m] - m; its leaves are nodes 0 .. n_m - 1 of that range (mesh-local
// ids, as a single build numbers them); indices get mesh-local triangle numbers.
__global__ void __launch_bounds__(256) k_ploc_init_seg(const uint32_t* __restrict__ sidx,
                                                       const Box* __restrict__ tri_boxes, PlocBufs B, PlocSeg S,
                                                       const SegItem* __restrict__ items, uint32_t n_items,
                                                       uint32_t n, uint32_t cap, uint32_t* __restrict__ d_indices,
                                                       unsigned long long* __restrict__ stamps) {
  stage_stamp(stamps, 3);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    B.ctrl[0] = n;
    B.ctrl[1] = n;
    B.ctrl[2] = 0;
    B.ctrl[3] = 0;
    B.ctrl[6] = 0;
    B.ctrl[7] = cap;
    B.ctrl[8] = 0;
    B.ctrl[9] = 0;
    B.ctrl[11] = S.count;
    B.ctrl[12] = 0;
#pragma unroll
    for (int k = 14; k < 20; ++k) B.ctrl[k] = 0;
  }
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const SegItem w = items[it];
    const uint32_t off = __ldg(S.offsets + w.mesh);
    const size_t base = 2 * (size_t)off - w.mesh;
    if (w.begin == off && threadIdx.x == 0) S.seg[w.mesh] = off;
    for (uint32_t p = w.begin + threadIdx.x; p < w.end; p += blockDim.x) {
      const uint32_t prim = __ldg(sidx + p);
      Box box = ld_box_cg(tri_boxes + prim);
      const float4 lo = box.lo, hi = box.hi;
      box.lo.w = __int_as_float((int)w.mesh);
      st_box(B.cbox[0] + p, box);
      B.cid[0][p] = (int32_t)(p - off);
      float4* np = reinterpret_cast<float4*>(B.nodes + base + (p - off));
      np[0] = make_float4(lo.x, lo.y, lo.z, 0.f);
      np[1] = hi;
      reinterpret_cast<int4*>(np + 2)[0] = make_int4((int32_t)((prim - off) | kLeafBit), -1, 0, 0);
      d_indices[p] = prim - off;
    }
  }
}

// End of an iteration, one thread.
template <bool GRAPH>
__global__ void k_ploc_step(PlocBufs B, cudaGraphConditionalHandle handle) {
  if (threadIdx.x == 0 && blockIdx.x == 0) ploc_step<GRAPH>(B, handle);
}

// The last iterations in one block.  Once the live clusters fit in shared memory (at most
// kTailMax, and few enough that their 2r pairs per cluster are cheap), an iteration over many
// blocks costs mostly launch latency; this kernel runs the remaining iterations in one block of
// kTailThreads, with the same rules and results as the kernels above: neighbour = smallest union
// area in [x-r, x+r], smallest j on ties, +inf and NaN never winning; mutual pairs merge into
// the smaller index, new node ids in ascending cluster order, survivors compacted in order; the
// same stop (one cluster), no-progress and cap rules, iteration count and live-cluster sum.
constexpr int kTailThreads = 1024;
constexpr uint32_t kTailMax = 2048;

// log2 of the lanes that share one cluster's search of 2r pairs when a block of kTailThreads searches for
// cnt clusters: as many as the block has to spare, but no more than have four pairs each.
__device__ __forceinline__ int search_lanes(uint32_t cnt, int r) {
  int lg = 0;
  while (lg < 5 && (cnt << (lg + 1)) <= (uint32_t)kTailThreads && (4 << lg) < 2 * r) ++lg;
  return lg;
}

// The nearest of the clusters j0..j1 (staged boxes) to cluster x of that range: the smallest area, the smallest
// j on ties, -1 where none is below infinity.  Alone (lg = 0), a thread scans both sides of x without
// checks; otherwise lane g of 2^lg takes every 2^lg-th j, four at a time, so that a search is not one
// chain of shared-memory loads, and the lanes' bests are compared.  Every lane of the warp takes part.
__device__ __forceinline__ int32_t group_nearest(const float4* lo, const float4* hi, int x, int j0, int j1, int g,
                                                 int lg) {
  const float4 xa = lo[x], xb = hi[x];
  float best = kHalfInf;
  int32_t bj = -1;
  if (lg == 0) {
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int e = side ? j1 + 1 : x;
      int j = side ? x + 1 : j0;
#pragma unroll 1
      for (; j + 4 <= e; j += 4) {
        float d[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] = pair_half(xa, xb, lo[j + q], hi[j + q]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (d[q] < best) {  // ascending j: the first of equal areas stays
            best = d[q];
            bj = j + q;
          }
      }
      for (; j < e; ++j) {
        const float d = pair_half(xa, xb, lo[j], hi[j]);
        if (d < best) {
          best = d;
          bj = j;
        }
      }
    }
    return bj;
  }
  for (int j = j0 + g; j <= j1; j += 4 << lg) {
    float d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = j + (q << lg);
      d[q] = pair_half(xa, xb, lo[min(k, j1)], hi[min(k, j1)]);
      if (k > j1 || k == x) d[q] = kHalfInf;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (d[q] < best) {
        best = d[q];
        bj = j + (q << lg);
      }
  }
  for (int o = 0; o < lg; ++o) {
    const float od = __shfl_xor_sync(0xffffffffu, best, 1 << o);
    const int32_t oj = __shfl_xor_sync(0xffffffffu, bj, 1 << o);
    if (od < best || (od == best && oj < bj)) {  // (two without a candidate both have j = -1)
      best = od;
      bj = oj;
    }
  }
  return bj;
}

uint32_t ploc_tail_threshold(int radius, uint32_t pairs) {
  if (pairs == 0) return 0;
  const uint32_t t = pairs / (2u * (uint32_t)std::max(radius, 1));
  return std::min<uint32_t>(kTailMax, std::max<uint32_t>(t, 64));
}
static size_t tail_smem() { return (size_t)kTailMax * (4 * 16 + 3 * 4) + 2 * 32 * 4; }

__global__ void __launch_bounds__(kTailThreads, 1) k_ploc_tail(PlocBufs B, int r) {
  after_previous();
  extern __shared__ float4 tsm[];
  float4* s_lo[2] = {tsm, tsm + 2 * kTailMax};
  float4* s_hi[2] = {tsm + kTailMax, tsm + 3 * kTailMax};
  int32_t* s_id[2] = {reinterpret_cast<int32_t*>(tsm + 4 * kTailMax),
                      reinterpret_cast<int32_t*>(tsm + 4 * kTailMax) + kTailMax};
  int32_t* s_nbr = s_id[1] + kTailMax;
  uint32_t* s_w = reinterpret_cast<uint32_t*>(s_nbr + kTailMax);  // 2 x 32 warp sums
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) B.ctrl[19] = 1;
  uint32_t c = __ldcg(B.ctrl + 0);
  // nothing left, or the loop stopped without handing over (too many clusters, an error)
  if (c <= 1 || c > kTailMax || (__ldcg(B.status) & kStatusNoProgress)) return;
  const uint32_t par = __ldcg(B.ctrl + 3) & 1u;
  const Box* cin = par ? B.cbox[1] : B.cbox[0];
  const int32_t* idin = par ? B.cid[1] : B.cid[0];
  for (uint32_t x = tid; x < c; x += kTailThreads) {
    const float4* bp = reinterpret_cast<const float4*>(cin + x);
    s_lo[0][x] = __ldcg(bp);
    s_hi[0][x] = __ldcg(bp + 1);
    s_id[0][x] = __ldcg(idin + x);
  }
  uint32_t next = __ldcg(B.ctrl + 1), it = __ldcg(B.ctrl + 6);
  const uint32_t it0 = it;
  const uint32_t cap = __ldcg(B.ctrl + 7);
  unsigned long long sum = (unsigned long long)__ldcg(B.ctrl + 9) << 32 | __ldcg(B.ctrl + 8);
  int cur = 0;
  bool no_progress = false;
  __syncthreads();
  while (c > 32) {
    sum += c;
    ++it;
    const float4* lo = s_lo[cur];
    const float4* hi = s_hi[cur];
    {
      const int lg = search_lanes(c, r), g = tid & ((1 << lg) - 1);
      for (uint32_t base = (uint32_t)(wid * 32) >> lg; base < c; base += (uint32_t)kTailThreads >> lg) {
        const uint32_t x = base + (uint32_t)(lane >> lg);  // (a warp without clusters skips the search)
        const int xi = (int)min(x, c - 1);
        const int32_t j = group_nearest(lo, hi, xi, max(0, xi - r), min((int)c - 1, xi + r), g, lg);
        if (x < c && g == 0) s_nbr[x] = j;
      }
    }
    __syncthreads();
    // merge and survivor flags of this thread's clusters x = 2 tid, 2 tid + 1 (ascending)
    const bool busy = 64u * (uint32_t)wid < c;  // the warp has clusters
    uint32_t mk = 0, vk = 0;
    bool m2[2], v2[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t x = 2u * (uint32_t)tid + (uint32_t)q;
      bool mm = false, vv = false;
      if (x < c) {
        const int32_t j = s_nbr[x];
        const bool mutual = j >= 0 && s_nbr[j] == (int32_t)x;
        mm = mutual && (int32_t)x < j;
        vv = !(mutual && j < (int32_t)x);
      }
      m2[q] = mm;
      v2[q] = vv;
      mk += mm;
      vk += vv;
    }
    // block exclusive scan of (merges, survivors), packed 16 + 16 bits (c <= 2048); every busy warp adds
    // up the totals before it
    uint32_t packed = mk << 16 | vk, x = packed;
    if (busy) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
    }
    if (lane == 31) s_w[wid] = x;
    __syncthreads();
    const uint32_t wt = s_w[lane];
    const uint32_t total = __reduce_add_sync(0xffffffffu, wt);
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < wid ? wt : 0u) + x - packed;
    uint32_t mpos = before >> 16, vpos = before & 0xffffu;
    const int nb = cur ^ 1;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t xi = 2u * (uint32_t)tid + (uint32_t)q;
      if (xi >= c) continue;
      float4 a = lo[xi], b = hi[xi];
      int32_t nid = s_id[cur][xi];
      if (m2[q]) {
        const int32_t j = s_nbr[xi];
        const float4 ja = lo[j], jb = hi[j];
        a = make_float4(fminf(a.x, ja.x), fminf(a.y, ja.y), fminf(a.z, ja.z), 0.f);
        b = make_float4(fmaxf(b.x, jb.x), fmaxf(b.y, jb.y), fmaxf(b.z, jb.z), 0.f);
        const int32_t id_new = (int32_t)(next + mpos);
        float4* np = reinterpret_cast<float4*>(B.nodes + id_new);
        np[0] = a;
        np[1] = b;
        reinterpret_cast<int4*>(np + 2)[0] = make_int4(nid, s_id[cur][j], 0, 0);
        if (nid == 0) B.ctrl[13] = (uint32_t)id_new;  // node 0's parent, for the root fix
        nid = id_new;
        ++mpos;
      }
      if (v2[q]) {
        s_lo[nb][vpos] = a;
        s_hi[nb][vpos] = b;
        s_id[nb][vpos] = nid;
        ++vpos;
      }
    }
    const uint32_t nc = total & 0xffffu, merges = total >> 16;
    next += merges;
    __syncthreads();  // the next buffer is complete; this iteration's buffers are free
    cur = nb;
    const uint32_t prev = c;
    c = nc;
    if (c <= 1) break;
    if (c >= prev || it >= cap) {  // no mutual pair anywhere, or the cap
      no_progress = true;
      break;
    }
  }
  // The last 32 clusters: one warp, a cluster per lane, flags and positions from ballots, no barriers.
  if (wid == 0 && !no_progress) {
    const uint32_t lt = (1u << lane) - 1u;
    while (c > 1) {
      sum += c;
      ++it;
      const float4* lo = s_lo[cur];
      const float4* hi = s_hi[cur];
      const int x = min(lane, (int)c - 1);
      float4 a = lo[x], b = hi[x];
      float best = kHalfInf;
      int32_t nbr = -1;
      for (int j = 0; j < (int)c; j += 4) {
        float d[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int k = min(j + q, (int)c - 1), away = j + q - x;
          d[q] = pair_half(a, b, lo[k], hi[k]);
          if (j + q >= (int)c || away == 0 || away > r || away < -r) d[q] = kHalfInf;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (d[q] < best) {
            best = d[q];
            nbr = j + q;
          }
      }
      const bool in = lane < (int)c;
      const int32_t back = __shfl_sync(0xffffffffu, nbr, nbr < 0 ? lane : nbr);
      const bool mutual = in && nbr >= 0 && back == lane;
      const uint32_t merges = __ballot_sync(0xffffffffu, mutual && lane < nbr);
      const uint32_t lives = __ballot_sync(0xffffffffu, in && !(mutual && nbr < lane));
      int32_t nid = s_id[cur][x];
      if ((merges >> lane) & 1u) {
        const float4 ja = lo[nbr], jb = hi[nbr];
        a = make_float4(fminf(a.x, ja.x), fminf(a.y, ja.y), fminf(a.z, ja.z), 0.f);
        b = make_float4(fmaxf(b.x, jb.x), fmaxf(b.y, jb.y), fmaxf(b.z, jb.z), 0.f);
        const int32_t id_new = (int32_t)(next + __popc(merges & lt));
        float4* np = reinterpret_cast<float4*>(B.nodes + id_new);
        np[0] = a;
        np[1] = b;
        reinterpret_cast<int4*>(np + 2)[0] = make_int4(nid, s_id[cur][nbr], 0, 0);
        if (nid == 0) B.ctrl[13] = (uint32_t)id_new;
        nid = id_new;
      }
      if ((lives >> lane) & 1u) {
        const uint32_t p = __popc(lives & lt);
        s_lo[cur ^ 1][p] = a;
        s_hi[cur ^ 1][p] = b;
        s_id[cur ^ 1][p] = nid;
      }
      __syncwarp();
      next += __popc(merges);
      cur ^= 1;
      const uint32_t prev = c;
      c = __popc(lives);
      if (c > 1 && (c >= prev || it >= cap)) {
        no_progress = true;
        break;
      }
    }
  }
  if (tid == 0) {
    B.ctrl[0] = c;
    B.ctrl[1] = next;
    B.ctrl[6] = it;
    B.ctrl[8] = (uint32_t)sum;
    B.ctrl[9] = (uint32_t)(sum >> 32);
    B.ctrl[17] = it - it0;
    if (no_progress) atomicOr(B.status, kStatusNoProgress);
  }
}

// The middle iterations in one cooperative kernel.  Between the iterations over many clusters
// (one launch per phase over persistent grids) and k_ploc_tail (one block), an iteration costs
// mostly the latency of its four launches.  k_ploc_grid runs those iterations in one cooperative
// launch (every block resident): block b owns the contiguous chunk [b*ch, (b+1)*ch) of at most
// kGridPerBlock clusters and stages its window (the chunk and r clusters either side) in shared
// memory; grid barriers separate the neighbour search, the flag count and the merge + compaction.
// Same rules and results as the kernels above and k_ploc_tail (neighbour = smallest union area in
// [x-r, x+r], smallest j on ties, +inf and NaN never winning; mutual pairs merge into the smaller
// index; new ids in ascending cluster order; survivors compacted in order; the same stop rules,
// iteration count and live-cluster sum).  It runs while the live clusters number more than the
// tail hand-over (ctrl[12]) and at most kGridPerBlock per block.
constexpr int kGridThreads = 1024;
constexpr uint32_t kGridPerBlock = 2048;
constexpr int kGridPer = (int)kGridPerBlock / kGridThreads;  // consecutive clusters per thread
constexpr int kGridMaxR = 128;
// the window: the chunk and 2r clusters either side (the neighbours of the chunk and of r
// clusters either side of it, so the flag count needs no other block's neighbours)
constexpr uint32_t kGridWin = kGridPerBlock + 4 * kGridMaxR;
constexpr uint32_t kGridNbr = kGridPerBlock + 2 * kGridMaxR;
constexpr uint32_t kGridMaxBlocks = 1024;
static size_t grid_smem() { return (size_t)kGridWin * (2 * 16 + 4) + (size_t)kGridNbr * 4 + 64 * 8; }

// Exclusive block scan of one 64-bit value per thread (kGridThreads); *total gets the sum.
__device__ __forceinline__ unsigned long long grid_block_scan(unsigned long long v, unsigned long long* s_w,
                                                              unsigned long long* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_w[wid] = x;
  __syncthreads();
  if (wid == 0) {
    unsigned long long t = s_w[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    s_w[32 + lane] = t;  // inclusive warp totals
  }
  __syncthreads();
  const unsigned long long before = (wid ? s_w[32 + wid - 1] : 0ull) + x - v;
  *total = s_w[32 + 31];
  __syncthreads();  // s_w is reused by the next scan
  return before;
}

__global__ void __launch_bounds__(kGridThreads, 1) k_ploc_grid(PlocBufs B, int r) {
  extern __shared__ float4 gsm[];
  float4* s_lo = gsm;
  float4* s_hi = gsm + kGridWin;
  int32_t* s_id = reinterpret_cast<int32_t*>(gsm + 2 * kGridWin);
  int32_t* s_nbr = s_id + kGridWin;  // neighbours of [h0, h1)
  unsigned long long* s_w = reinterpret_cast<unsigned long long*>(s_nbr + kGridNbr);
  __shared__ uint32_t s_ok, s_asked;
  __shared__ uint32_t s_ask[2 * kGridMaxR];  // clusters outside the chunk whose neighbour is asked for
  const uint32_t G = gridDim.x, b = blockIdx.x;
  const int tid = threadIdx.x;
  if (b == 0 && tid == 0) B.ctrl[18] = 1;  // (no block reads it)
  // every block reads the same words (nothing writes them before the first barrier)
  uint32_t c = __ldcg(B.ctrl + 0);
  const uint32_t tail = __ldcg(B.ctrl + 12), cap = __ldcg(B.ctrl + 7);
  if (c <= 1 || c <= tail || c > G * kGridPerBlock || r > kGridMaxR || r < 1 ||
      (__ldcg(B.status) & kStatusNoProgress))
    return;
  uint32_t next = __ldcg(B.ctrl + 1), par = __ldcg(B.ctrl + 3) & 1u, it = __ldcg(B.ctrl + 6);
  const uint32_t it0 = it;
  unsigned long long sum = (unsigned long long)__ldcg(B.ctrl + 9) << 32 | __ldcg(B.ctrl + 8);
  uint32_t* bar = B.ctrl + 15;
  unsigned long long* totals = reinterpret_cast<unsigned long long*>(B.flags);  // one per block
  uint32_t nbar = 0;
  bool no_progress = false, ok = true;
  while (true) {
    const Box* cin = par ? B.cbox[1] : B.cbox[0];
    const int32_t* idin = par ? B.cid[1] : B.cid[0];
    Box* cout = par ? B.cbox[0] : B.cbox[1];
    int32_t* idout = par ? B.cid[0] : B.cid[1];
    const uint32_t ch = div_up(c, G);
    const uint32_t x0 = min(c, b * ch), x1 = min(c, x0 + ch);
    const uint32_t h0 = x0 > (uint32_t)r ? x0 - (uint32_t)r : 0u, h1 = min(c, x1 + (uint32_t)r);
    const uint32_t w0 = h0 > (uint32_t)r ? h0 - (uint32_t)r : 0u, w1 = min(c, h1 + (uint32_t)r);
    for (uint32_t x = w0 + tid; x < w1; x += kGridThreads) {
      const Box box = ld_box_cg(cin + x);
      s_lo[x - w0] = box.lo;
      s_hi[x - w0] = box.hi;
      s_id[x - w0] = __ldcg(idin + x);
    }
    __syncthreads();
    // Neighbours of the chunk's clusters, then of those outside it (within r) that some of them point to: a
    // mutual pair may cross the chunk's ends.  They are few, where all 2r of them were as many as the
    // chunk itself.
    const auto search = [&](uint32_t cnt, const auto& cluster) {
      static_assert(kGridThreads == kTailThreads, "search_lanes");
      const int lg = search_lanes(cnt, r), g = tid & ((1 << lg) - 1);
      for (uint32_t base = (uint32_t)((tid >> 5) * 32) >> lg; base < cnt; base += (uint32_t)kGridThreads >> lg) {
        const uint32_t k = base + (uint32_t)((tid & 31) >> lg);
        const uint32_t x = cluster(min(k, cnt - 1));
        const uint32_t j0 = x > (uint32_t)r ? x - (uint32_t)r : 0u, j1 = min(c - 1, x + (uint32_t)r);
        const int32_t j = group_nearest(s_lo, s_hi, (int)(x - w0), (int)(j0 - w0), (int)(j1 - w0), g, lg);
        if (k < cnt && g == 0) s_nbr[x - h0] = j < 0 ? -1 : j + (int32_t)w0;
      }
    };
    if (tid == 0) s_asked = 0;
    for (uint32_t x = h0 + tid; x < h1; x += kGridThreads)
      if (x < x0 || x >= x1) s_nbr[x - h0] = -2;  // not asked for
    search(x1 - x0, [&](uint32_t k) { return x0 + k; });
    __syncthreads();
    for (uint32_t x = x0 + tid; x < x1; x += kGridThreads) {
      const int32_t j = s_nbr[x - h0];
      if (j >= 0 && ((uint32_t)j < x0 || (uint32_t)j >= x1) && atomicCAS(&s_nbr[(uint32_t)j - h0], -2, -3) == -2)
        s_ask[atomicAdd(&s_asked, 1u)] = (uint32_t)j;
    }
    __syncthreads();
    search(s_asked, [&](uint32_t k) { return s_ask[k]; });
    __syncthreads();
    // merge / survivor flags of this thread's clusters x0 + kGridPer tid + q (ascending); a
    // neighbour j lies within r of x, so both j and its neighbour are in s_nbr
    bool m2[kGridPer], v2[kGridPer];
    int32_t nj[kGridPer];
    uint32_t mk = 0, vk = 0;
#pragma unroll
    for (int q = 0; q < kGridPer; ++q) {
      const uint32_t x = x0 + (uint32_t)kGridPer * (uint32_t)tid + (uint32_t)q;
      m2[q] = v2[q] = false;
      nj[q] = -1;
      if (x < x1) {  // (a chunk may be empty)
        const int32_t j = s_nbr[x - h0];
        const int32_t back = j >= 0 ? s_nbr[(uint32_t)j - h0] : -1;
        const bool mutual = j >= 0 && back == (int32_t)x;
        m2[q] = mutual && (int32_t)x < j;
        v2[q] = !(mutual && j < (int32_t)x);
        nj[q] = j;
      }
      mk += m2[q];
      vk += v2[q];
    }
    unsigned long long btot;
    const unsigned long long before = grid_block_scan((unsigned long long)mk << 32 | vk, s_w, &btot);
    if (tid == 0) __stcg(totals + b, btot);
    if (!(ok = grid_sync(bar, ++nbar * G, B.status, &s_ok))) break;
    // this block's offset and the totals over all blocks, added up by one warp
    if (tid < 32) {
      unsigned long long mine = 0, all = 0;
      for (uint32_t k = (uint32_t)tid; k < G; k += 32) {
        const unsigned long long t = __ldcg(totals + k);
        all += t;
        if (k < b) mine += t;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        mine += __shfl_xor_sync(0xffffffffu, mine, o);
        all += __shfl_xor_sync(0xffffffffu, all, o);
      }
      if (tid == 0) {
        s_w[0] = mine;
        s_w[1] = all;
      }
    }
    __syncthreads();
    const unsigned long long offs_b = s_w[0], grand_b = s_w[1];
    uint32_t mpos = (uint32_t)(offs_b >> 32) + (uint32_t)(before >> 32);
    uint32_t vpos = (uint32_t)offs_b + (uint32_t)before;
    const uint32_t M = (uint32_t)(grand_b >> 32), V = (uint32_t)grand_b;
#pragma unroll
    for (int q = 0; q < kGridPer; ++q) {
      const uint32_t xi = x0 + (uint32_t)kGridPer * (uint32_t)tid + (uint32_t)q;
      if (xi >= x1) continue;
      float4 a = s_lo[xi - w0], bb = s_hi[xi - w0];
      int32_t nid = s_id[xi - w0];
      if (m2[q]) {
        const uint32_t j = (uint32_t)nj[q];  // within [xi - r, xi + r], so inside the staged window
        const float4 ja = s_lo[j - w0], jb = s_hi[j - w0];
        a = make_float4(fminf(a.x, ja.x), fminf(a.y, ja.y), fminf(a.z, ja.z), 0.f);
        bb = make_float4(fmaxf(bb.x, jb.x), fmaxf(bb.y, jb.y), fmaxf(bb.z, jb.z), 0.f);
        const int32_t id_new = (int32_t)(next + mpos);
        float4* np = reinterpret_cast<float4*>(B.nodes + id_new);
        np[0] = a;
        np[1] = bb;
        reinterpret_cast<int4*>(np + 2)[0] = make_int4(nid, s_id[j - w0], 0, 0);
        if (nid == 0) B.ctrl[13] = (uint32_t)id_new;  // node 0's parent, for the root fix
        nid = id_new;
        ++mpos;
      }
      if (v2[q]) {
        st_box(cout + vpos, Box{a, bb});
        idout[vpos] = nid;
        ++vpos;
      }
    }
    sum += c;
    ++it;
    next += M;
    const uint32_t prev = c;
    c = V;
    par ^= 1u;
    if (c <= 1) break;
    if (c >= prev || it >= cap) {  // no mutual pair anywhere, or the cap
      no_progress = true;
      break;
    }
    if (c <= tail) break;
    if (!(ok = grid_sync(bar, ++nbar * G, B.status, &s_ok))) break;  // the next window reads the compacted buffer
  }
  if (ok && b == 0 && tid == 0) {
    B.ctrl[0] = c;
    B.ctrl[1] = next;
    B.ctrl[3] = par;
    B.ctrl[6] = it;
    B.ctrl[8] = (uint32_t)sum;
    B.ctrl[9] = (uint32_t)(sum >> 32);
    B.ctrl[16] = it - it0;
    if (no_progress) atomicOr(B.status, kStatusNoProgress);
  }
}

// Self-test of the grid barrier's bound: a cooperative launch whose blocks wait for one arrival
// more than there are blocks (a block that never comes), giving up after `limit` polls each.
// Words: [0] arrival counter, [1] status.
__device__ uint32_t g_grid_selftest[2];

__global__ void k_grid_selftest(uint32_t limit) {
  __shared__ uint32_t s_ok;
  grid_sync(g_grid_selftest, gridDim.x + 1, g_grid_selftest + 1, &s_ok, limit);
}

cudaError_t grid_wait_selftest(uint32_t limit, uint32_t* status_out) {
  int dev = 0, coop = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (e != cudaSuccess) return e;
  if (!coop) return cudaErrorNotSupported;
  cudaStream_t st = nullptr;
  if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) return e;
  const uint32_t zero[2] = {0u, 0u};
  e = cudaMemcpyToSymbolAsync(g_grid_selftest, zero, sizeof(zero), 0, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(4);
    cfg.blockDim = dim3(64);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, k_grid_selftest, limit);
  }
  if (e == cudaSuccess) e = cudaMemcpyFromSymbolAsync(status_out, g_grid_selftest, 4, 4, cudaMemcpyDeviceToHost, st);
  const cudaError_t e2 = cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return e != cudaSuccess ? e : e2;
}

// Move the root (last node) to index 0 and swap every reference to 0 and the root
// (ploc_builder.cu:563-582); skipped when the loop did not converge.  The root has no parent and
// node 0 (a leaf) has one, recorded by the merge that made it (ctrl[13]), so three nodes change:
// 0, R and that parent.  Without a recorded parent every node is checked (one block).
__global__ void k_ploc_root(Node* __restrict__ nodes, uint32_t total, const uint32_t* __restrict__ ctrl) {
  after_previous();
  if (__ldcg(ctrl + 0) != 1 || total < 2) return;
  const uint32_t R = total - 1;
  auto fix = [&](int32_t c) -> int32_t {
    if (c < 0) return c;
    if (c == 0) return (int32_t)R;
    if (c == (int32_t)R) return 0;
    return c;
  };
  const uint32_t p = __ldcg(ctrl + 13);
  const bool known = p > 0 && p < total;
  for (uint32_t k = threadIdx.x; k < total; k += blockDim.x) {
    if (known && k != 0) {  // only node 0's parent refers to 0 or R (R itself moves with k == 0)
      if (k == 1 && p != R) {
        int2 ch = *reinterpret_cast<int2*>(&nodes[p].left);
        *reinterpret_cast<int2*>(&nodes[p].left) = make_int2(fix(ch.x), fix(ch.y));
      }
      break;
    }
    if (k == 0) {
      Node a = nodes[0], b = nodes[R];
      if (b.left >= 0) { b.left = fix(b.left); b.right = fix(b.right); }
      if (a.left >= 0) { a.left = fix(a.left); a.right = fix(a.right); }
      nodes[0] = b;
      nodes[R] = a;
    } else if (k != R) {
      int2 ch = *reinterpret_cast<int2*>(&nodes[k].left);
      if (ch.x >= 0) {
        int2 nc = make_int2(fix(ch.x), fix(ch.y));
        if (nc.x != ch.x || nc.y != ch.y) *reinterpret_cast<int2*>(&nodes[k].left) = nc;
      }
    }
  }
}

// Batched builds: each mesh's root (its last node) moves to the start of its range, as in
// k_ploc_root; work items split the node ranges evenly.
__global__ void __launch_bounds__(256) k_ploc_root_seg(Node* __restrict__ nodes, const SegItem* __restrict__ items,
                                                       uint32_t n_items, PlocSeg S, const uint32_t* __restrict__ ctrl) {
  if (__ldcg(ctrl + 0) != S.count) return;
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const SegItem w = items[it];
    const uint32_t off = __ldg(S.offsets + w.mesh), nm = __ldg(S.offsets + w.mesh + 1) - off;
    Node* mn = nodes + (2 * (size_t)off - w.mesh);
    const uint32_t R = 2 * nm - 2;
    auto fix = [&](int32_t c) -> int32_t {
      if (c < 0) return c;
      if (c == 0) return (int32_t)R;
      if (c == (int32_t)R) return 0;
      return c;
    };
    const uint32_t k0 = 2 * (w.begin - off), k1 = min(2 * (w.end - off), 2 * nm - 1);
    for (uint32_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
      if (k == 0) {
        Node a = mn[0], b = mn[R];
        if (b.left >= 0) { b.left = fix(b.left); b.right = fix(b.right); }
        if (a.left >= 0) { a.left = fix(a.left); a.right = fix(a.right); }
        mn[0] = b;
        mn[R] = a;
      } else if (k != R) {
        int2 ch = *reinterpret_cast<int2*>(&mn[k].left);
        if (ch.x >= 0) {
          int2 nc = make_int2(fix(ch.x), fix(ch.y));
          if (nc.x != ch.x || nc.y != ch.y) *reinterpret_cast<int2*>(&mn[k].left) = nc;
        }
      }
    }
  }
}

cudaError_t workspace_reserve_ploc(Workspace& ws, uint32_t n) {
  if (!ws.aux_stream) {  // captures the batched loop body while a batch is being captured
    cudaError_t e = cudaStreamCreateWithFlags(&ws.aux_stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
  }
  if (n <= ws.ploc_cap && ws.nbr) return cudaSuccess;
  uint32_t cap = std::max<uint32_t>(n, 1024);
  workspace_moves(ws);
  cudaFree(ws.cbox[0]); cudaFree(ws.cbox[1]); cudaFree(ws.cid[0]); cudaFree(ws.cid[1]); cudaFree(ws.nbr);
  ws.cbox[0] = ws.cbox[1] = nullptr; ws.cid[0] = ws.cid[1] = nullptr; ws.nbr = nullptr; ws.ploc_cap = 0;
  cudaError_t e;
  if ((e = cudaMalloc(&ws.cbox[0], (size_t)cap * sizeof(Box))) != cudaSuccess) return e;
  if ((e = cudaMalloc(&ws.cbox[1], (size_t)cap * sizeof(Box))) != cudaSuccess) return e;
  if ((e = cudaMalloc(&ws.cid[0], (size_t)cap * 4)) != cudaSuccess) return e;
  if ((e = cudaMalloc(&ws.cid[1], (size_t)cap * 4)) != cudaSuccess) return e;
  // neighbours (cap) + per-tile merge totals / prefixes (64-bit) share one allocation
  // ... and the per-round ballots (8 B per 32 clusters)
  size_t desc_words = div_up(cap, kPlocTile) + 8;
  // (smaller tiles in late iterations: at most one partial tile's worth more; never more tiles
  // than the grid, so desc_words holds their totals)
  size_t flag_words = (size_t)div_up(cap, kPlocTile) * (kPlocThreads / 32) * kPlocRounds +
                      (kPlocThreads / 32) * kPlocRounds + kGridMaxBlocks;  // (k_ploc_grid: one total per block)
  if ((e = cudaMalloc(&ws.nbr, (size_t)cap * 4 + desc_words * 8 + flag_words * 8 + 64)) != cudaSuccess) return e;
  ws.ploc_cap = cap;
  return cudaSuccess;
}

static size_t nn_smem(int radius) {
  const size_t tile = radius <= kNcMaxR ? 2 * kPlocThreads : kNnTile;  // the largest strided tile that is taken
  const size_t strided = 32 * (tile + 2 * (size_t)radius) + 4 * (size_t)kNnKc * tile;
  return radius <= kNcMaxR ? std::max(strided, nc_smem(radius)) : strided;
}

// Persistent grids sized for n, capped at `bps` blocks per SM (the workspace's launch shapes).
struct PlocShape {
  int nn_bps, mg_bps;
  uint32_t key() const { return (uint32_t)nn_bps << 16 | (uint32_t)mg_bps; }
};
static PlocShape ploc_shape(const Workspace& ws) {
  return PlocShape{std::max(1, std::min(ws.ploc_nn_bps, 16)), std::max(1, std::min(ws.ploc_mg_bps, 32))};
}
static uint32_t nn_grid_for(uint32_t n, const PlocShape& sh) {
  return std::max<uint32_t>(1, std::min<uint32_t>(div_up(n, kNnTile), 152u * (uint32_t)sh.nn_bps));
}
static uint32_t mg_grid_for(uint32_t n, const PlocShape& sh) {
  return std::max<uint32_t>(1, std::min<uint32_t>(div_up(n, kPlocTile), 152u * (uint32_t)sh.mg_bps));
}

// One clustering iteration: neighbours, tile counts + scan, (batched: per-mesh ranks), merge +
// compaction, loop control.  Grids are persistent (sized for n); the kernels read the live
// cluster count from the control words.
template <bool SEG, bool GRAPH>
static void enqueue_iteration(const PlocBufs& B, const PlocSeg& S, uint32_t n, int radius, const PlocShape& sh,
                              cudaStream_t st, cudaGraphConditionalHandle handle) {
  const uint32_t mg_grid = mg_grid_for(n, sh);
  const auto nn = radius < kNcMinR ? k_ploc_nn<SEG, false> : k_ploc_nn<SEG, true>;
  nn<<<nn_grid_for(n, sh), kPlocThreads, nn_smem(radius), st>>>(B, radius);
  k_ploc_count<<<mg_grid, kPlocThreads, 0, st>>>(B);
  if constexpr (SEG) k_ploc_seg<<<std::max<uint32_t>(1, std::min<uint32_t>(div_up(S.count, 256), 152 * 4)), 256, 0,
                                  st>>>(B, S, mg_grid);
  k_ploc_scatter<SEG><<<mg_grid, kPlocThreads, 0, st>>>(B, S);
  k_ploc_step<GRAPH><<<1, 32, 0, st>>>(B, handle);
}

// The loop as a graph: WHILE(cond) { one iteration }.
template <bool SEG>
static cudaError_t make_loop_graph(const PlocBufs& B, const PlocSeg& S, uint32_t n, int radius, const PlocShape& sh,
                                   cudaGraphExec_t* out) {
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaGraphCreate(&g, 0);
  if (e != cudaSuccess) return e;
  cudaGraphConditionalHandle handle;
  cudaStream_t cs = nullptr;
  cudaGraphNode_t node;
  cudaGraphNodeParams cp = {};
  do {
    if ((e = cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault)) != cudaSuccess) break;
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    if ((e = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &cp)) != cudaSuccess) break;
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    if ((e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) != cudaSuccess) break;
    if ((e = cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
      break;
    enqueue_iteration<SEG, true>(B, S, n, radius, sh, cs, handle);
    cudaGraph_t captured = nullptr;
    cudaError_t e2 = cudaGetLastError();
    e = cudaStreamEndCapture(cs, &captured);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) break;
    e = cudaGraphInstantiate(out, g, 0);
  } while (false);
  if (cs) cudaStreamDestroy(cs);
  cudaGraphDestroy(g);
  return e;
}

static PlocBufs ploc_bufs(Workspace& ws, const ScratchLayout& L) {
  PlocBufs B;
  B.cbox[0] = ws.cbox[0];
  B.cbox[1] = ws.cbox[1];
  B.cid[0] = ws.cid[0];
  B.cid[1] = ws.cid[1];
  B.nbr = ws.nbr;
  B.desc = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(ws.nbr) +
                                                  (((size_t)ws.ploc_cap * 4 + 15) & ~size_t(15)));
  B.flags = reinterpret_cast<uint2*>(B.desc + div_up(ws.ploc_cap, kPlocTile) + 8);
  B.nodes = ws.nodes;
  B.ctrl = ws.scratch + L.ploc;
  B.status = ws.scratch + L.status;
  return B;
}

template <bool SEG>
static cudaError_t set_nn_smem(int radius) {
  if (nn_smem(radius) <= 48 * 1024) return cudaSuccess;
  const auto nn = radius < kNcMinR ? k_ploc_nn<SEG, false> : k_ploc_nn<SEG, true>;
  return cudaFuncSetAttribute(nn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nn_smem(radius));
}

static cudaError_t set_tail_smem() {
  return cudaFuncSetAttribute(k_ploc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tail_smem());
}

// Blocks of a k_ploc_grid launch on the current device: SMs x resident blocks per SM, or 0 where
// cooperative launches are not available.  Sets the kernel's shared-memory limit (so it is called
// before any capture, from ploc_prepare, and again by builds).
static uint32_t ploc_grid_blocks() {
  int dev = 0, coop = 0, sms = 0, occ = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaFuncSetAttribute(k_ploc_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grid_smem()) != cudaSuccess)
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_ploc_grid, kGridThreads, grid_smem()) != cudaSuccess)
    return 0;
  return (uint32_t)std::min<long long>((long long)sms * occ, kGridMaxBlocks);
}

constexpr uint32_t kHostGridMin = 65536;
constexpr uint32_t kLoopTailPairs = 100000;

// The blocks that a build of n triangles takes of the `all` that fit the GPU.  A cooperative grid starts when all of its
// blocks have room, so builds in several streams take turns unless their grids fit side by side; and a
// block has no use for less than 512 clusters or 25,600 pairs to search (20,000 triangles, r = 25: 40 blocks
// take 204 us where 152 take 202; four streams 63 us per build, where they took 180).  Between a half and
// four fifths of the GPU, a half: two builds then run at once.
static uint32_t ploc_grid_share(uint32_t all, uint32_t n, int radius) {
  const uint32_t per = std::max<uint32_t>(1, std::min<uint32_t>(512, 12800u / (uint32_t)std::max(radius, 1)));
  const uint32_t want = std::max<uint32_t>(16, div_up(n, per)), half = all / 2;
  return want > half && (unsigned long long)want * 5 <= (unsigned long long)all * 4 ? half : std::min(all, want);
}

cudaError_t ploc_prepare(int radius) {
  cudaError_t e = set_nn_smem<false>(radius);
  if (e == cudaSuccess) e = set_nn_smem<true>(radius);
  if (e == cudaSuccess) e = set_tail_smem();
  if (e == cudaSuccess) ploc_grid_blocks();
  return e;
}

cudaError_t ploc_build(Workspace& ws, const MeshPtrs& m, uint32_t n, int radius, int max_iter, cudaStream_t st,
                       StageEvents* evs, uint32_t** out_indices, bool host_loop) {
  cudaError_t e = workspace_reserve(ws, n, st);
  if (e != cudaSuccess) return e;
  if ((e = workspace_reserve_ploc(ws, n)) != cudaSuccess) return e;
  ScratchLayout L = scratch_layout(ws.cap_n);
  const PlocBufs B = ploc_bufs(ws, L);
  const PlocSeg none{};
  if ((e = set_nn_smem<false>(radius)) != cudaSuccess) return e;
  if ((e = set_tail_smem()) != cudaSuccess) return e;
  // every iteration that makes progress removes at least one cluster, so n bounds the loop
  const uint32_t cap = max_iter > 0 ? (uint32_t)max_iter : n;
  // k_ploc_grid: from grid_at live clusters down to the tail hand-over (its per-block totals
  // live in the ballot words).  Where no cooperative kernel runs, its iterations would be driven from the host
  // (20,000 triangles 890 us); below kHostGridMin the loop graph runs them all (552 us, and a build that only
  // has the tail can be captured), and the tail takes over earlier, since an iteration of the loop
  // costs four launches: so it does for radii that k_ploc_grid does not take.
  const bool cooperative = !ws.no_cooperative && !ws.cooperative_refused;
  const uint32_t grid_blocks = ploc_grid_share(ploc_grid_blocks(), n, radius);
  uint32_t grid_at = 0;
  if (grid_blocks && radius <= kGridMaxR && (cooperative || n >= kHostGridMin))
    grid_at = std::min<uint32_t>(ws.ploc_grid_max, grid_blocks * kGridPerBlock);
  uint32_t pairs = ws.ploc_tail_pairs;
  if (pairs && (!grid_at || !cooperative)) pairs = std::max(pairs, kLoopTailPairs);
  const uint32_t tail = ploc_tail_threshold(radius, pairs);
  if (grid_at <= tail || n <= tail) grid_at = 0;
  const bool loop = n > 1 && n > std::max(tail, grid_at);  // else the one-launch kernels do every iteration
  const PlocShape sh = ploc_shape(ws);
  if (host_loop && !ws.ploc_host && (e = cudaMallocHost(&ws.ploc_host, 64)) != cudaSuccess) return e;
  if (loop && !host_loop) {
    const bool same = ws.ploc_exec && ws.ploc_key_n == n && ws.ploc_key_r == radius && ws.ploc_key_shape == sh.key();
    if (!same) {
      if (ws.ploc_exec) cudaGraphExecDestroy(ws.ploc_exec);
      ws.ploc_exec = nullptr;
      if ((e = make_loop_graph<false>(B, none, n, radius, sh, &ws.ploc_exec)) != cudaSuccess) return e;
      ws.ploc_key_n = n;
      ws.ploc_key_r = radius;
      ws.ploc_key_shape = sh.key();
    }
  }
  if (evs && evs->use) cudaEventRecord(evs->ev[0], st);
  uint32_t* sidx = nullptr;
  if ((e = prefix_sort30(ws, m, n, st, &sidx)) != cudaSuccess) return e;
  *out_indices = sidx;
  if ((e = launch_after(ws.alone, k_ploc_init, div_up(n, 256), 256, 0, st, sidx, ws.boxes, B, n, cap, tail, grid_at,
                        reinterpret_cast<unsigned long long*>(ws.scratch + L.stamps))) != cudaSuccess)
    return e;
  if (evs && evs->use) {
    cudaEventRecord(evs->ev[4], st);
    evs->split = true;
  }
  if (loop && host_loop) {
    for (uint32_t it = 0; it < cap; ++it) {
      enqueue_iteration<false, false>(B, none, n, radius, sh, st, cudaGraphConditionalHandle{});
      if ((e = cudaMemcpyAsync(ws.ploc_host, B.ctrl + 10, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
          (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return e;
      if (!*ws.ploc_host) break;
    }
  } else if (loop) {
    if ((e = cudaGraphLaunch(ws.ploc_exec, st)) != cudaSuccess) return e;
  }
  if (n > 1) {
    if (grid_at) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(grid_blocks);
      cfg.blockDim = dim3(kGridThreads);
      cfg.dynamicSmemBytes = grid_smem();
      cfg.stream = st;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeCooperative;
      attr[0].val.cooperative = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      e = cooperative ? cudaLaunchKernelEx(&cfg, k_ploc_grid, B, radius) : cudaErrorNotSupported;
      if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        // no co-resident grid (a client limited to part of the GPU, or asked for): the same
        // iterations as one launch per kernel each, driven from the host, down to the tail
        // hand-over; the loop above stopped at grid_at live clusters or for good
        (void)cudaGetLastError();
        if (cooperative) ws.cooperative_refused = true;
        if (!ws.ploc_host && (e = cudaMallocHost(&ws.ploc_host, 64)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(B.ctrl + 14, 0, 4, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(ws.ploc_host, B.ctrl, 8 * 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
            (e = cudaStreamSynchronize(st)) != cudaSuccess)
          return e;
        bool go = ws.ploc_host[0] > std::max<uint32_t>(tail, 1u) && ws.ploc_host[6] < ws.ploc_host[7];
        while (go) {
          enqueue_iteration<false, false>(B, none, n, radius, sh, st, cudaGraphConditionalHandle{});
          if ((e = cudaMemcpyAsync(ws.ploc_host, B.ctrl + 10, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
              (e = cudaStreamSynchronize(st)) != cudaSuccess)
            return e;
          go = *ws.ploc_host != 0;
        }
      } else if (e != cudaSuccess) {
        return e;
      }
    }
    if (tail && (e = launch_after(ws.alone, k_ploc_tail, 1, kTailThreads, tail_smem(), st, B, radius)) != cudaSuccess) return e;
    if ((e = launch_after(ws.alone, k_ploc_root, 1, 256, 0, st, ws.nodes, 2 * n - 1, B.ctrl)) != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

// Batched PLOC: the batched prefix (per-mesh boxes and keys, one sort), then every mesh's
// clustering in the same iterations -- windows clipped at mesh boundaries, merges numbered per
// mesh -- until each mesh has one cluster, then each mesh's root fix.  Mesh m's result equals its
// single build: the same leaves, the same neighbours in every iteration, the same node ids
// relative to its range [2 offsets[m] - m, 2 offsets[m+1] - m - 1).  A mesh that has finished
// keeps its one cluster, which has no neighbour.  The loop is a CUDA graph WHILE node (or a
// host loop); the iteration count is the largest of the meshes' own.
cudaError_t batched_ploc_build(Workspace& ws, const MeshPtrs& m, uint32_t n, const uint32_t* d_offsets,
                               uint32_t count, const SegItem* d_items, uint32_t n_items, float* d_mbox,
                               uint32_t* d_indices, int radius, uint32_t max_iter, cudaStream_t st,
                               StageEvents* evs, bool host_loop) {
  cudaError_t e = workspace_reserve(ws, n, st);
  if (e != cudaSuccess) return e;
  if ((e = workspace_reserve_ploc(ws, n)) != cudaSuccess) return e;
  ScratchLayout L = scratch_layout(ws.cap_n);
  const PlocBufs B = ploc_bufs(ws, L);
  PlocSeg S;
  S.offsets = d_offsets;
  S.seg = reinterpret_cast<uint32_t*>(d_mbox);  // the mesh boxes are dead once the keys are made
  S.id_base = S.seg + 2 * (size_t)count;
  S.count = count;
  if ((e = set_nn_smem<true>(radius)) != cudaSuccess) return e;
  const uint32_t cap = max_iter > 0 ? max_iter : n;
  if (host_loop && !ws.ploc_host && (e = cudaMallocHost(&ws.ploc_host, 64)) != cudaSuccess) return e;
  const bool loop = n > count;  // some mesh has two or more triangles
  const PlocShape sh = ploc_shape(ws);
  cudaStreamCaptureStatus cst0 = cudaStreamCaptureStatusNone;
  if ((e = cudaStreamIsCapturing(st, &cst0)) != cudaSuccess) return e;
  if (loop && !host_loop && cst0 == cudaStreamCaptureStatusNone) {
    const bool same = ws.ploc_seg_exec && ws.ploc_seg_key_n == n && ws.ploc_seg_key_count == count &&
                      ws.ploc_seg_key_r == radius && ws.ploc_seg_key[0] == d_offsets &&
                      ws.ploc_seg_key[1] == d_mbox && ws.ploc_seg_key_shape == sh.key();
    if (!same) {
      if (ws.ploc_seg_exec) cudaGraphExecDestroy(ws.ploc_seg_exec);
      ws.ploc_seg_exec = nullptr;
      if ((e = make_loop_graph<true>(B, S, n, radius, sh, &ws.ploc_seg_exec)) != cudaSuccess) return e;
      ws.ploc_seg_key_shape = sh.key();
      ws.ploc_seg_key_n = n;
      ws.ploc_seg_key_count = count;
      ws.ploc_seg_key_r = radius;
      ws.ploc_seg_key[0] = d_offsets;
      ws.ploc_seg_key[1] = d_mbox;
    }
  }
  BatchedSort bs;
  if ((e = batched_prefix(ws, m, n, count, d_items, n_items, d_mbox, d_indices, st, evs, &bs)) != cudaSuccess) return e;
  const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>(n_items, 152 * 8));
  k_ploc_init_seg<<<grid, 256, 0, st>>>(ws.vals[bs.fb], ws.boxes, B, S, d_items, n_items, n, cap, d_indices,
                                       reinterpret_cast<unsigned long long*>(ws.scratch + L.stamps));
  if (evs && evs->use) {
    cudaEventRecord(evs->ev[4], st);
    evs->split = true;
  }
  if (loop && host_loop) {
    for (uint32_t it = 0; it < cap; ++it) {
      enqueue_iteration<true, false>(B, S, n, radius, sh, st, cudaGraphConditionalHandle{});
      if ((e = cudaMemcpyAsync(ws.ploc_host, B.ctrl + 10, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
          (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return e;
      if (!*ws.ploc_host) break;
    }
  } else if (loop) {
    cudaStreamCaptureStatus cst = cudaStreamCaptureStatusNone;
    cudaGraph_t cg = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    const cudaGraphEdgeData* edata = nullptr;
    size_t nd = 0;
    if ((e = cudaStreamGetCaptureInfo(st, &cst, nullptr, &cg, &deps, &edata, &nd)) != cudaSuccess) return e;
    if (cst == cudaStreamCaptureStatusActive) {
      // the batch is being captured into one graph: the loop becomes a conditional node of it
      cudaGraphConditionalHandle h;
      if ((e = cudaGraphConditionalHandleCreate(&h, cg, 1, cudaGraphCondAssignDefault)) != cudaSuccess) return e;
      cudaGraphNodeParams cp = {};
      cp.type = cudaGraphNodeTypeConditional;
      cp.conditional.handle = h;
      cp.conditional.type = cudaGraphCondTypeWhile;
      cp.conditional.size = 1;
      cudaGraphNode_t node;
      if ((e = cudaGraphAddNode(&node, cg, deps, edata, nd, &cp)) != cudaSuccess) return e;
      cudaStream_t aux = ws.aux_stream;
      if (!aux) return cudaErrorInvalidResourceHandle;  // made by workspace_reserve_ploc, before any capture
      if ((e = cudaStreamBeginCaptureToGraph(aux, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                             cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
        return e;
      enqueue_iteration<true, true>(B, S, n, radius, sh, aux, h);
      cudaGraph_t body = nullptr;
      const cudaError_t e2 = cudaGetLastError();
      if ((e = cudaStreamEndCapture(aux, &body)) != cudaSuccess) return e;
      if (e2 != cudaSuccess) return e2;
      if ((e = cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies)) !=
          cudaSuccess)
        return e;
    } else if ((e = cudaGraphLaunch(ws.ploc_seg_exec, st)) != cudaSuccess) {
      return e;
    }
  }
  if (loop) k_ploc_root_seg<<<grid, 256, 0, st>>>(ws.nodes, d_items, n_items, S, B.ctrl);
  return cudaGetLastError();
}

// Order-independent hash of a tree's node fields: each node's (index, min, max, left, right)
// mixed to 64 bits (splitmix64 finaliser), XOR-combined per warp and then atomically.
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__global__ void __launch_bounds__(256) k_tree_hash(const Node* __restrict__ nodes, uint32_t n_nodes,
                                                   unsigned long long* __restrict__ out) {
  unsigned long long h = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_nodes; i += gridDim.x * blockDim.x) {
    const float4* p = reinterpret_cast<const float4*>(nodes + i);
    const float4 lo = __ldg(p), hi = __ldg(p + 1);
    const int2 ch = __ldg(reinterpret_cast<const int2*>(p + 2));
    unsigned long long z = mix64(i + 0x9e3779b97f4a7c15ull);
    z = mix64(z ^ ((unsigned long long)__float_as_uint(lo.x) << 32 | __float_as_uint(lo.y)));
    z = mix64(z ^ ((unsigned long long)__float_as_uint(lo.z) << 32 | __float_as_uint(hi.x)));
    z = mix64(z ^ ((unsigned long long)__float_as_uint(hi.y) << 32 | __float_as_uint(hi.z)));
    z = mix64(z ^ ((unsigned long long)(uint32_t)ch.x << 32 | (uint32_t)ch.y));
    h ^= z;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) h ^= __shfl_xor_sync(0xffffffffu, h, o);
  if ((threadIdx.x & 31) == 0 && h) atomicXor(out, h);
}

cudaError_t tree_hash(const Node* nodes, uint32_t n_nodes, unsigned long long* out, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(out, 0, 8, st);
  if (e != cudaSuccess || n_nodes == 0) return e;
  k_tree_hash<<<std::min<uint32_t>(div_up(n_nodes, 256), 152 * 8), 256, 0, st>>>(nodes, n_nodes, out);
  return cudaGetLastError();
}

}  // namespace bvhgb

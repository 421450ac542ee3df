// small.cuh -- a whole LBVH (or PLOC's sorted order) of a small mesh in one block; part of lbvh.cu.
//
// At a thousand triangles the general path's ten kernels take 51 us per build, nearly all of it launch
// latency and the chains of L2 round trips between blocks (look-back, rendezvous words).  One block keeps
// everything between the input and the nodes in shared memory and registers: scene box, codes, an LSD
// radix sort over the whole code (so 60/63-bit codes need no run fix-up), delta bytes and the Karras
// climb, whose rendezvous all lie inside the block.  Same arithmetic, order and node ids as the
// general kernels.
//
// kSmallMax: two triangles per thread is what the climb's records leave room for (64 bytes per position,
// 215 KB of shared memory in all).
#pragma once

namespace bvhgb {

constexpr int kSmallThreads = 1024;
constexpr uint32_t kSmallMax = 2048;

enum SmallMode { kSmallLbvh, kSmallLbvhPlus, kSmallSort };

template <typename K, int IPT>
struct SmallShared {
  static constexpr int CAP = kSmallThreads * IPT, NW = kSmallThreads / 32;
  float box[6][CAP];  // by original index: lo.xyz, hi.xyz
  K key[CAP];
  uint32_t val[CAP];
  float red[NW][6];
  float scene[6];
  uint8_t D[CAP + 16];  // D[k]: between sorted positions k - 1 and k
  union {
    struct {
      uint32_t whist[NW * 256];
      uint32_t match[NW * kMatchWords];
      uint32_t part[4 * 256];
      uint32_t start[256];
      uint32_t wsum[8];
    } sort;
    struct {
      float4 lo[2][CAP], hi[2][CAP];  // a child's box with its id (lo.w) and far end (hi.w), by side and split
      uint32_t flag[CAP];
      uint8_t h[2][CAP];  // the child's height (LBVH+)
    } climb;
  };
};

// One stable pass over the 8-bit digit at `shift`; key and val are warp-striped (see warp_rank).
template <typename K, int IPT>
__device__ __forceinline__ void small_pass(SmallShared<K, IPT>& S, K (&key)[IPT], uint32_t (&val)[IPT], int shift,
                                           uint32_t n) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint32_t wbase = (uint32_t)w * 32u * IPT;
  for (int b = t; b < 32 * 256; b += kSmallThreads) S.sort.whist[b] = 0;
  __syncthreads();
  uint32_t rnk[IPT];
  uint32_t* wh = S.sort.whist + w * 256;
  warp_rank<true>(key, rnk, shift, wbase, n, wh, S.sort.match + w * kMatchWords, (uint32_t)lane);
  __syncthreads();
  // bin b's counts of 8 warps per thread, the bin totals' exclusive scan, then every warp's offset
  const int b = t & 255, q = t >> 8;
  uint32_t c[8], sum = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    c[j] = S.sort.whist[(8 * q + j) * 256 + b];
    sum += c[j];
  }
  S.sort.part[q * 256 + b] = sum;
  __syncthreads();
  uint32_t x = 0, total = 0;
  if (t < 256) {
    total = S.sort.part[t] + S.sort.part[256 + t] + S.sort.part[512 + t] + S.sort.part[768 + t];
    x = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) S.sort.wsum[w] = x;
  }
  __syncthreads();
  if (t < 256) {
    uint32_t before = 0;
    for (int k = 0; k < w; ++k) before += S.sort.wsum[k];
    S.sort.start[t] = before + x - total;
  }
  __syncthreads();
  uint32_t run = S.sort.start[b];
  for (int k = 0; k < q; ++k) run += S.sort.part[k * 256 + b];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    S.sort.whist[(8 * q + j) * 256 + b] = run;
    run += c[j];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    if (wbase + (uint32_t)k * 32u + lane < n) {
      const uint32_t pos = wh[(uint32_t)(key[k] >> shift) & 255u] + rnk[k];
      S.key[pos] = key[k];
      S.val[pos] = val[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t i = wbase + (uint32_t)k * 32u + lane;
    key[k] = i < n ? S.key[i] : K(0);
    val[k] = i < n ? S.val[i] : 0u;
  }
}

// vals: the sorted original indices; boxes: triangle boxes by original index (kSmallSort only); host:
// where not null, the build's report (as k_finish writes it).
template <int BITS, int MODE, int IPT>
__global__ void __launch_bounds__(kSmallThreads, 1)
    k_small(MeshPtrs m, uint32_t n, uint32_t* __restrict__ vals, Box* __restrict__ boxes, Node* __restrict__ nodes,
            uint32_t* __restrict__ scratch, ScratchLayout L, uint32_t* __restrict__ host, uint8_t* __restrict__ hgt) {
  using K = typename std::conditional<BITS == 30, uint32_t, unsigned long long>::type;
  using Shared = SmallShared<K, IPT>;
  extern __shared__ __align__(16) unsigned char smem[];
  Shared& S = *reinterpret_cast<Shared*>(smem);
  unsigned long long* stamps = reinterpret_cast<unsigned long long*>(scratch + L.stamps);
  stage_stamp(stamps, 0);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) {
    scratch[L.status] = 0;
    const uint32_t e = scratch[L.epoch] + kEpochStride;
    scratch[L.epoch] = e < kEpochStride ? kEpochStride : e;
  }
  // ---- scene box ----
  float v[IPT][9];
  float sb[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t i = (uint32_t)w * 32u * IPT + (uint32_t)k * 32u + lane;
#pragma unroll
    for (int a = 0; a < 9; ++a) v[k][a] = i < n ? __ldcs(m.v[a] + i) : 0.f;
    if (i < n)
#pragma unroll
      for (int a = 0; a < 3; ++a) tri_box_acc(v[k][a], v[k][3 + a], v[k][6 + a], sb[a], sb[3 + a]);
  }
  warp_reduce_box(sb[0], sb[1], sb[2], sb[3], sb[4], sb[5]);
  if (lane == 0)
#pragma unroll
    for (int a = 0; a < 6; ++a) S.red[w][a] = sb[a];
  for (int b = t; b < Shared::NW * kMatchWords; b += kSmallThreads) S.sort.match[b] = 0;
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int a = 0; a < 6; ++a) sb[a] = S.red[lane][a];
    warp_reduce_box(sb[0], sb[1], sb[2], sb[3], sb[4], sb[5]);
    if (lane == 0)
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float e = sb[3 + a] - sb[a];
        S.scene[a] = sb[a];
        S.scene[3 + a] = (e > 1e-6f) ? e : 1.0f;
      }
  }
  __syncthreads();
  // ---- codes and boxes ----
  stage_stamp(stamps, 1);
  K key[IPT];
  uint32_t val[IPT];
  bool wild = false;
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t i = (uint32_t)w * 32u * IPT + (uint32_t)k * 32u + lane;
    key[k] = K(0);
    val[k] = i;
    if (i < n) {
      Box b;
      key[k] = tri_code<BITS, K>(v[k][0], v[k][1], v[k][2], v[k][3], v[k][4], v[k][5], v[k][6], v[k][7], v[k][8], S.scene,
                                 S.scene + 3, b);
      if (MODE == kSmallLbvhPlus) wild |= !tame_box(b);
      if (MODE == kSmallSort) {
        boxes[i] = b;
      } else {
        S.box[0][i] = b.lo.x; S.box[1][i] = b.lo.y; S.box[2][i] = b.lo.z;
        S.box[3][i] = b.hi.x; S.box[4][i] = b.hi.y; S.box[5][i] = b.hi.z;
      }
    }
  }
  if (MODE == kSmallLbvhPlus) {
    wild = __syncthreads_or(wild);
    if (t == 0) scratch[L.wild] = wild ? 1u : 0u;
  }
  // ---- sort ----
  stage_stamp(stamps, 2);
  for (int shift = 0; shift < BITS; shift += 8) small_pass<K, IPT>(S, key, val, shift, n);
#pragma unroll
  for (int k = 0; k < IPT; ++k) {
    const uint32_t i = (uint32_t)w * 32u * IPT + (uint32_t)k * 32u + lane;
    if (i < n) vals[i] = val[k];
  }
  if (MODE == kSmallSort) return;
  // ---- delta bytes (delta_nt, lbvh_builder.cu:33-43) ----
  stage_stamp(stamps, 3);
  for (uint32_t k = t; k <= n; k += kSmallThreads) {
    uint8_t d = 0;
    if (k > 0 && k < n) {
      const K x = S.key[k - 1] ^ S.key[k];
      const uint32_t tie = (BITS == 30 ? 32u : 64u) + (uint32_t)__clz(S.val[k - 1] ^ S.val[k]);
      d = (uint8_t)((x == 0 ? tie : BITS == 30 ? (uint32_t)__clz((uint32_t)x) : (uint32_t)__clzll((long long)x)) + 1u);
    }
    S.D[k] = d;
  }
  __syncthreads();  // the sort's tables are dead: the climb's records take their place
  for (uint32_t k = t; k < n; k += kSmallThreads) S.climb.flag[k] = 0;
  __syncthreads();
  // ---- climb: as k_emit, every rendezvous inside the block ----
  constexpr bool PLUS = MODE == kSmallLbvhPlus;
  for (uint32_t i = t; i < n; i += kSmallThreads) {
    const uint32_t prim = S.val[i];
    Climb c;
    c.f = c.l = i;
    c.lc = c.rc = -1;
    c.internal = false;
    c.h = 0;
    c.box.lo = make_float4(S.box[0][prim], S.box[1][prim], S.box[2][prim], 0.f);
    c.box.hi = make_float4(S.box[3][prim], S.box[4][prim], S.box[5][prim], 0.f);
    c.my = (int32_t)(n - 1 + i);
    store_node(nodes, (uint32_t)c.my, c.box, (int32_t)(prim | kLeafBit), -1, -1);
    while (true) {
      const int dl = (int)S.D[c.f] - 1, dr = (int)S.D[c.l + 1] - 1;
      if (dl < 0 && dr < 0) {  // the root (a one-triangle mesh: its leaf)
        if (c.internal) write_internal<PLUS>(nodes, hgt, 0, 0, c);
        break;
      }
      const bool is_left = dr > dl, pending = c.internal;
      const uint32_t gamma = is_left ? c.l : c.f - 1;
      if (pending) c.my = (int32_t)(is_left ? c.l : c.f);
      const int side = is_left ? 0 : 1;
      S.climb.lo[side][gamma] = make_float4(c.box.lo.x, c.box.lo.y, c.box.lo.z, __int_as_float(c.my));
      S.climb.hi[side][gamma] = make_float4(c.box.hi.x, c.box.hi.y, c.box.hi.z, __uint_as_float(is_left ? c.f : c.l));
      if (PLUS) S.climb.h[side][gamma] = (uint8_t)c.h;  // (at most kMaxTreeHeight)
      const uint32_t prev = atom_or_acq_rel_cta(&S.climb.flag[gamma], 1u << side);
      if (pending) write_internal<PLUS>(nodes, hgt, 0, c.my, c);
      if (prev == 0u) break;  // first to arrive
      const float4 a = S.climb.lo[side ^ 1][gamma], b = S.climb.hi[side ^ 1][gamma];
      Box sib;
      sib.lo = make_float4(a.x, a.y, a.z, 0.f);
      sib.hi = make_float4(b.x, b.y, b.z, 0.f);
      climb_merge<PLUS>(c, is_left, __float_as_int(a.w), sib, PLUS ? S.climb.h[side ^ 1][gamma] : 0u);
      if (is_left) c.l = __float_as_uint(b.w);
      else c.f = __float_as_uint(b.w);
      c.internal = true;
    }
  }
  if (host && w == 0) {  // (no wait in here can give up: the status is 0)
    if (lane == 0) host[0] = 0;
    if (lane >= 24) host[lane] = __ldcg(scratch + L.stamps + (lane - 24));
  }
}

template <int BITS, int MODE>
static const void* small_kernel(uint32_t n, size_t* smem) {
  using K = typename std::conditional<BITS == 30, uint32_t, unsigned long long>::type;
  const bool one = n <= (uint32_t)kSmallThreads;
  *smem = one ? sizeof(SmallShared<K, 1>) : sizeof(SmallShared<K, 2>);
  return one ? reinterpret_cast<const void*>(&k_small<BITS, MODE, 1>) : reinterpret_cast<const void*>(&k_small<BITS, MODE, 2>);
}
static const void* small_kernel(int bits, int mode, uint32_t n, size_t* smem) {
  if (mode == kSmallSort) return small_kernel<30, kSmallSort>(n, smem);
  if (mode == kSmallLbvhPlus)
    return bits == 30   ? small_kernel<30, kSmallLbvhPlus>(n, smem)
           : bits == 60 ? small_kernel<60, kSmallLbvhPlus>(n, smem)
                        : small_kernel<63, kSmallLbvhPlus>(n, smem);
  return bits == 30   ? small_kernel<30, kSmallLbvh>(n, smem)
         : bits == 60 ? small_kernel<60, kSmallLbvh>(n, smem)
                      : small_kernel<63, kSmallLbvh>(n, smem);
}

// Builds (or sorts) a mesh of at most kSmallMax triangles; the sorted indices land in ws.vals[0].
static cudaError_t small_build(Workspace& ws, const MeshPtrs& m, uint32_t n, int bits, int mode, cudaStream_t st,
                               const ScratchLayout& L, uint32_t* host) {
  cudaError_t e = epoch_tick(ws, st);
  if (e != cudaSuccess) return e;
  size_t smem = 0;
  const void* fn = small_kernel(bits, mode, n, &smem);
  const uint32_t bit = 1u << ((mode * 3 + (bits == 60) + 2 * (bits == 63)) * 2 + (n > (uint32_t)kSmallThreads));
  if (!(ws.small_ready & bit)) {
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
    ws.small_ready |= bit;
  }
  MeshPtrs mp = m;
  ScratchLayout Lc = L;
  void* args[] = {&mp, &n, &ws.vals[0], &ws.boxes, &ws.nodes, &ws.scratch, &Lc, &host, &ws.heights};
  return cudaLaunchKernel(fn, dim3(1), dim3(kSmallThreads), args, smem, st);
}

// Shared memory of every variant (once per device, outside any stream capture).
static cudaError_t prepare_small() {
  for (int mode : {(int)kSmallLbvh, (int)kSmallLbvhPlus, (int)kSmallSort})
    for (int bits : {30, 60, 63})
      for (uint32_t n : {1u, kSmallMax}) {
        size_t smem = 0;
        const void* fn = small_kernel(bits, mode, n, &smem);
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
      }
  return cudaSuccess;
}

}  // namespace bvhgb

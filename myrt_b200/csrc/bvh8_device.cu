// Device BVH build: linear BVH (Morton order + radix tree) collapsed into the
// 80-byte 8-wide quantised nodes of bvh8.hpp, entirely on the GPU.
//
// The host builder (bvh8.cpp) makes better trees (binned SAH, SAH-optimal
// 8-wide collapse) but takes O(n log n) host time per upload; this builder
// rebuilds a 2 M-triangle scene in milliseconds, which is what dynamic scenes
// need (the reference rebuilds its TLAS on the host whenever an instance
// moves, src/pathtracer/scene.cpp:336-344). Answers of the ray queries do not
// depend on the tree (ties go to the smaller prim id), only their speed.
//
//   k_prim_boxes   padded triangle boxes (+1e-5, as generate_triangle_bounds,
//                  bvh.cpp:136-152) and the bounds of their centres
//   k_morton       63-bit Morton codes of the centres (21 bits per axis)
//   (CUB)          radix sort of (code, prim) pairs
//   k_radix_tree   binary radix tree over the sorted codes (Karras, "Maximizing
//                  parallelism in the construction of BVHs, octrees and k-d
//                  trees", HPG 2012); equal codes are ordered by position
//   k_boxes_block, k_boxes_cross  internal boxes, as ranges of leaf boxes
//   k_collapse     one wide node per 8 lanes, level by level: expand the
//                  largest-area child with more than 4 triangles until 8
//                  children, then quantise, assign slots by octant and emit
//                  the node, its triangles' prims and its internal children
//   k_emit_tris    the leaf-ordered triangles
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <vector>

#include "bvh8.hpp"
#include "bvh8_device.hpp"

namespace myrt_b200 {
namespace {

constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kNone = 0xffffffffu;  // no node
constexpr int kMaxLeaf = 4;
constexpr int kMaxLevels = 4096;
constexpr uint32_t kColGrid = 2368;   // collapse blocks of a large level: 16 for each of 148 SMs
constexpr uint32_t kCrossGrid = 592;  // blocks of k_boxes_cross: 4 for each of 148 SMs

struct ibox {
  float4 lo, hi;  // w unused
};

__device__ __forceinline__ uint32_t f2ord(float f) {  // order-preserving float -> uint
  uint32_t const u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__global__ void k_prim_boxes(float const* __restrict__ pos, uint32_t n, float pad, ibox* __restrict__ boxes,
    uint32_t* __restrict__ cbounds) {
  uint32_t const i = blockIdx.x * blockDim.x + threadIdx.x;
  float c[3] = {0.f, 0.f, 0.f};
  bool const ok = i < n;
  if (ok) {
    float const* v = pos + 9 * size_t(i);
    float lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
      lo[a] = fminf(fminf(v[a], v[3 + a]), v[6 + a]) - pad;
      hi[a] = fmaxf(fmaxf(v[a], v[3 + a]), v[6 + a]) + pad;
      c[a] = 0.5f * (lo[a] + hi[a]);
    }
    boxes[i] = ibox{make_float4(lo[0], lo[1], lo[2], 0.f), make_float4(hi[0], hi[1], hi[2], 0.f)};
  }
  // block-wide min / max of the centres, then one atomic per block and bound
  __shared__ uint32_t s[6];
  if (threadIdx.x < 6) s[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
  __syncthreads();
  if (ok)
    for (int a = 0; a < 3; ++a) {
      atomicMin(&s[a], f2ord(c[a]));
      atomicMax(&s[3 + a], f2ord(c[a]));
    }
  __syncthreads();
  if (threadIdx.x < 3) atomicMin(&cbounds[threadIdx.x], s[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(&cbounds[threadIdx.x], s[threadIdx.x]);
}

__device__ __forceinline__ uint64_t spread21(uint32_t v) {
  uint64_t x = v & 0x1fffffu;
  x = (x | (x << 32)) & 0x1f00000000ffffull;
  x = (x | (x << 16)) & 0x1f0000ff0000ffull;
  x = (x | (x << 8)) & 0x100f00f00f00f00full;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

__global__ void k_morton(ibox const* __restrict__ boxes, uint32_t n, uint32_t const* __restrict__ cbounds,
    uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  uint32_t const i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ibox const b = boxes[i];
  float const c[3] = {0.5f * (b.lo.x + b.hi.x), 0.5f * (b.lo.y + b.hi.y), 0.5f * (b.lo.z + b.hi.z)};
  uint64_t code = 0;
  for (int a = 0; a < 3; ++a) {
    float const lo = ord2f(cbounds[a]), hi = ord2f(cbounds[3 + a]);
    float const ext = hi - lo;
    float const t = ext > 0.f ? (c[a] - lo) / ext : 0.f;
    uint32_t const q = uint32_t(fminf(fmaxf(t * 2097152.f, 0.f), 2097151.f));
    code |= spread21(q) << a;
  }
  keys[i] = code;
  vals[i] = i;
}

__device__ __forceinline__ int delta(uint64_t const* k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  uint64_t const a = k[i], b = k[j];
  if (a == b) return 64 + __clz(uint32_t(i) ^ uint32_t(j));
  return __clzll(a ^ b);
}

// internal node i: children (leaf bit | index), prim range
__global__ void k_radix_tree(uint64_t const* __restrict__ keys, int n, uint2* __restrict__ child,
    uint2* __restrict__ range) {
  int const i = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n - 1) return;
  int const d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  int const dmin = delta(keys, n, i, i - d);
  int lmax = 2;
  while (delta(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
  int l = 0;
  for (int t = lmax / 2; t >= 1; t /= 2)
    if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int const j = i + l * d;
  int const dnode = delta(keys, n, i, j);
  int s = 0;
  int t = l;
  do {
    t = (t + 1) / 2;
    if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  int const gamma = i + s * d + min(d, 0);
  int const first = min(i, j), last = max(i, j);
  uint32_t const left = first == gamma ? (kLeafBit | uint32_t(gamma)) : uint32_t(gamma);
  uint32_t const right = last == gamma + 1 ? (kLeafBit | uint32_t(gamma + 1)) : uint32_t(gamma + 1);
  child[i] = make_uint2(left, right);
  range[i] = make_uint2(uint32_t(first), uint32_t(last));
}

__device__ __forceinline__ ibox load_box(uint32_t ref, ibox const* leaf_boxes, uint32_t const* order,
    ibox const* inner) {
  if (ref & kLeafBit) return leaf_boxes[order[ref & ~kLeafBit]];
  ibox b;
  b.lo = inner[ref].lo;
  b.hi = inner[ref].hi;
  return b;
}
__device__ __forceinline__ ibox merge(ibox a, ibox b) {
  return ibox{make_float4(fminf(a.lo.x, b.lo.x), fminf(a.lo.y, b.lo.y), fminf(a.lo.z, b.lo.z), 0.f),
      make_float4(fmaxf(a.hi.x, b.hi.x), fmaxf(a.hi.y, b.hi.y), fmaxf(a.hi.z, b.hi.z), 0.f)};
}

// Boxes of the internal nodes. A node covers a range of the sorted leaves, so
// its box is a range minimum / maximum over leaf boxes: no order among nodes,
// where a bottom-up pass is a chain of global arrivals, fences and loads as
// long as the tree is deep (655,872 triangles: 81 us; 96 us with the lower
// levels' arrivals in shared memory). k_boxes_block keeps the boxes of every
// run of 2^j leaves of its 256 (eight levels, 48 KB) and answers each node
// within them from two runs; it also writes the 256 leaves' own box and lists
// the nodes that reach past them. k_boxes_cross gives each of those a warp:
// the leaves at both ends and the whole blocks between. Together 50 us.
constexpr int kBoxBlock = 256, kBoxRuns = 8;
__global__ void __launch_bounds__(kBoxBlock) k_boxes_block(ibox const* __restrict__ leaf_boxes,
    uint32_t const* __restrict__ order, int n, uint2 const* __restrict__ range, ibox* __restrict__ inner,
    ibox* __restrict__ block_box, uint32_t* __restrict__ cross, uint32_t* __restrict__ n_cross) {
  __shared__ float s_run[kBoxRuns][6][kBoxBlock];
  uint32_t const b0 = blockIdx.x * kBoxBlock, t = threadIdx.x;
  bool const leaf = b0 + t < uint32_t(n);
  float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (leaf) {
    ibox const b = leaf_boxes[order[b0 + t]];
    v[0] = b.lo.x, v[1] = b.lo.y, v[2] = b.lo.z, v[3] = b.hi.x, v[4] = b.hi.y, v[5] = b.hi.z;
  }
#pragma unroll
  for (int j = 0; j < kBoxRuns; ++j) {  // s_run[j][.][t]: leaves t .. t + 2^j - 1 (those of the block)
    if (j > 0) {
      uint32_t const o = t + (1u << (j - 1));
      if (o < kBoxBlock)
        for (int c = 0; c < 6; ++c)
          v[c] = c < 3 ? fminf(v[c], s_run[j - 1][c][o]) : fmaxf(v[c], s_run[j - 1][c][o]);
    }
    for (int c = 0; c < 6; ++c) s_run[j][c][t] = v[c];
    __syncthreads();
  }
  auto runs = [&](uint32_t lo, uint32_t hi) {  // leaves lo .. hi of the block
    int const j = min(31 - __clz(hi - lo + 1u), kBoxRuns - 1);
    uint32_t const o = hi + 1u - (1u << j);
    float w[6];
    for (int c = 0; c < 6; ++c)
      w[c] = c < 3 ? fminf(s_run[j][c][lo], s_run[j][c][o]) : fmaxf(s_run[j][c][lo], s_run[j][c][o]);
    return ibox{make_float4(w[0], w[1], w[2], 0.f), make_float4(w[3], w[4], w[5], 0.f)};
  };
  if (t == 0) block_box[blockIdx.x] = runs(0u, kBoxBlock - 1u);
  if (b0 + t >= uint32_t(n) - 1u) return;  // n - 1 internal nodes
  uint2 const r = range[b0 + t];
  if (r.x >= b0 && r.y < b0 + kBoxBlock) inner[b0 + t] = runs(r.x - b0, r.y - b0);
  else cross[atomicAdd(n_cross, 1u)] = b0 + t;
}

__global__ void __launch_bounds__(256) k_boxes_cross(ibox const* __restrict__ leaf_boxes,
    uint32_t const* __restrict__ order, uint2 const* __restrict__ range, ibox const* __restrict__ block_box,
    uint32_t const* __restrict__ cross, uint32_t const* __restrict__ n_cross, ibox* __restrict__ inner) {
  uint32_t const lane = threadIdx.x & 31u, n = *n_cross;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    uint32_t const node = cross[i];
    uint2 const r = range[node];
    uint32_t const bx = r.x / kBoxBlock, by = r.y / kBoxBlock;  // bx < by
    ibox b{make_float4(INFINITY, INFINITY, INFINITY, 0.f), make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f)};
    for (uint32_t l = r.x + lane; l < (bx + 1u) * kBoxBlock; l += 32u) b = merge(b, leaf_boxes[order[l]]);
    for (uint32_t l = by * kBoxBlock + lane; l <= r.y; l += 32u) b = merge(b, leaf_boxes[order[l]]);
    for (uint32_t k = bx + 1u + lane; k < by; k += 32u) b = merge(b, block_box[k]);
    float* const f[6] = {&b.lo.x, &b.lo.y, &b.lo.z, &b.hi.x, &b.hi.y, &b.hi.z};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        float const v = __shfl_xor_sync(0xffffffffu, *f[c], o);
        *f[c] = c < 3 ? fminf(*f[c], v) : fmaxf(*f[c], v);
      }
    if (lane == 0) inner[node] = b;
  }
}

struct collapse_item {
  uint32_t ref;   // binary node (leaf bit | index)
  uint32_t wide;  // wide node index to write
  uint32_t depth;
};

struct collapse_args {
  ibox const* leaf_boxes;  // per prim (input order)
  uint32_t const* order;   // sorted position -> prim
  uint2 const* child;
  uint2 const* range;
  ibox const* inner;
  bvh8_node* nodes;
  uint32_t* tri_prim;      // leaf-ordered triangle -> prim
  uint32_t* counters;      // [0] wide nodes, [1] triangles, [3] max depth, [4] leaf slots
  collapse_item const* in;
  uint32_t const* n_in;    // this level's queue length (device)
  collapse_item* out;
  uint32_t* n_out;         // the next level's (zeroed before the build)
};

__device__ __forceinline__ uint32_t prim_count(collapse_args const& a, uint32_t ref) {
  if (ref & kLeafBit) return 1u;
  uint2 const r = a.range[ref];
  return r.y - r.x + 1u;
}
__device__ __forceinline__ float area(ibox const& b) {
  float const dx = b.hi.x - b.lo.x, dy = b.hi.y - b.lo.y, dz = b.hi.z - b.lo.z;
  return ((dx + dy) * dz + dx * dy) * 2.f;
}

// 2^e as a double, -1022 <= e <= 1023
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double(static_cast<long long>(1023 + e) << 52); }

// Smallest e with extent / 2^e <= 255 (the host builder's biased_exponent_for).
__device__ __forceinline__ uint8_t biased_exponent(float extent) {
  if (!(extent > 0.f)) return uint8_t(127 - 100);
  // extent / 255 in [2^(e-1), 2^e); its rounding can put it one binade off
  int e = int((__double_as_longlong(double(extent) / 255.0) >> 52) & 0x7ff) - 1022;
  while (e > -126 && 255.0 * pow2(e - 1) >= double(extent)) --e;
  while (255.0 * pow2(e) < double(extent)) ++e;
  e = max(-126, min(127, e));
  return uint8_t(e + 127);
}

// One wide node per 8 lanes of a warp, lane k holding child k while the node
// is opened and slot k once the slots are assigned. A level of the tree is one
// launch and its time was the serial work of one thread -- 7 dependent
// expansions, a 64-entry cost search per slot, 24 double divisions, calls of
// frexp and ldexp -- on arrays in local memory; spread over 8 lanes the search
// and the quantisation run side by side, a block takes its queue and output
// space with one atomic per counter, and the triangles are copied by their own
// kernel (k_emit_tris), coalesced. 655,872 triangles: 1,313 -> 194 us in eleven launches and 15 for the triangles.
constexpr int kColBlock = 128, kColNodes = kColBlock / 8;
__global__ void __launch_bounds__(kColBlock) k_collapse(collapse_args a) {
  __shared__ uint32_t s_int[kColNodes], s_tri[kColNodes], s_slots[kColNodes], s_base[3];
  __shared__ __align__(16) uint8_t s_node[kColNodes][sizeof(bvh8_node)];
  constexpr uint32_t kAll = 0xffffffffu;
  uint32_t const lane = threadIdx.x & 31u, sub = lane & 7u, base8 = lane & ~7u, oct = threadIdx.x >> 3;
  uint32_t const n_in = *a.n_in;
  for (uint32_t first = blockIdx.x * kColNodes; first < n_in; first += gridDim.x * kColNodes) {
    uint32_t const it = first + oct;
    bool const live = it < n_in;
    collapse_item item{kLeafBit, 0u, 0u};
    if (live) item = a.in[it];
    // open the node: the child with the largest area among those of more than
    // kMaxLeaf triangles (ties: the first) is replaced by its two children
    uint32_t ref = kNone, cnt = 0;
    uint2 kids = make_uint2(0u, 0u);  // ref's own children, loaded with its box
    ibox kb{make_float4(INFINITY, INFINITY, INFINITY, 0.f), make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f)};
    uint32_t nk = 0;
    auto fetch = [&](uint32_t r) {
      ref = r;
      if (!(r & kLeafBit)) kids = a.child[r];
      cnt = prim_count(a, r);
      kb = load_box(r, a.leaf_boxes, a.order, a.inner);
    };
    if (live) {
      if ((item.ref & kLeafBit) || prim_count(a, item.ref) <= uint32_t(kMaxLeaf)) {
        nk = 1;  // the whole (small) tree is one leaf slot
        if (sub == 0) fetch(item.ref);
      } else {
        uint2 const c = a.child[item.ref];
        nk = 2;
        if (sub < 2) fetch(sub == 0 ? c.x : c.y);
      }
    }
#pragma unroll 1
    for (int r = 0; r < 6; ++r) {
      float ar = -1.f;
      if (cnt > uint32_t(kMaxLeaf)) {
        float const v = area(kb);
        if (v > -1.f) ar = v;
      }
      uint32_t who = sub;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        float const oa = __shfl_xor_sync(kAll, ar, o);
        uint32_t const ow = __shfl_xor_sync(kAll, who, o);
        if (oa > ar || (oa == ar && ow < who)) ar = oa, who = ow;
      }
      bool const open = ar > -1.f;
      if (!__any_sync(kAll, open)) break;
      uint2 const c = make_uint2(__shfl_sync(kAll, kids.x, int(base8 + who)),
          __shfl_sync(kAll, kids.y, int(base8 + who)));
      if (open) {
        if (sub == who || sub == nk) fetch(sub == who ? c.x : c.y);
        ++nk;
      }
    }
    // the node's box
    ibox nb = kb;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      nb.lo.x = fminf(nb.lo.x, __shfl_xor_sync(kAll, nb.lo.x, o));
      nb.lo.y = fminf(nb.lo.y, __shfl_xor_sync(kAll, nb.lo.y, o));
      nb.lo.z = fminf(nb.lo.z, __shfl_xor_sync(kAll, nb.lo.z, o));
      nb.hi.x = fmaxf(nb.hi.x, __shfl_xor_sync(kAll, nb.hi.x, o));
      nb.hi.y = fmaxf(nb.hi.y, __shfl_xor_sync(kAll, nb.hi.y, o));
      nb.hi.z = fmaxf(nb.hi.z, __shfl_xor_sync(kAll, nb.hi.z, o));
    }
    // octant slot assignment (the host builder's rule): slot s faces (+-1, +-1,
    // +-1), bit a of s set meaning +; repeatedly the (child, slot) pair with the
    // largest projection takes the slot (ties: the first child, its first slot)
    uint32_t slot = 8u, free_slots = 0xffu;
    {
      float const dx = 0.5f * (kb.lo.x + kb.hi.x) - 0.5f * (nb.lo.x + nb.hi.x);
      float const dy = 0.5f * (kb.lo.y + kb.hi.y) - 0.5f * (nb.lo.y + nb.hi.y);
      float const dz = 0.5f * (kb.lo.z + kb.hi.z) - 0.5f * (nb.lo.z + nb.hi.z);
      bool todo = sub < nk;
#pragma unroll 1
      for (uint32_t r = 0; r < 8u; ++r) {
        float bc = -3.402823466e38f;
        uint32_t pick = 0x800u | (sub << 4);  // 0x800: no slot above the floor (NaN boxes)
        if (todo) {
#pragma unroll
          for (uint32_t s = 0; s < 8u; ++s) {
            float const v = ((s & 1) ? dx : -dx) + ((s & 2) ? dy : -dy) + ((s & 4) ? dz : -dz);
            if (((free_slots >> s) & 1u) && v > bc) bc = v, pick = (sub << 4) | s;
          }
        } else {
          pick = 0x1000u;
        }
        // largest projection; without one, the first child still to place
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          float const oc = __shfl_xor_sync(kAll, bc, o);
          uint32_t const op = __shfl_xor_sync(kAll, pick, o);
          bool const mine = pick < 0x800u, theirs = op < 0x800u;
          if (theirs != mine ? theirs : (theirs && oc != bc ? oc > bc : op < pick)) bc = oc, pick = op;
        }
        if (!__any_sync(kAll, pick < 0x1000u)) break;
        if (pick < 0x1000u) {
          uint32_t const s = pick < 0x800u ? pick & 15u : uint32_t(__ffs(free_slots) - 1);
          if (((pick >> 4) & 7u) == sub) {
            slot = s;
            todo = false;
          }
          free_slots &= ~(1u << s);
        }
      }
    }
    // lane = slot from here on
    uint32_t from = 8u;
#pragma unroll
    for (uint32_t k = 0; k < 8u; ++k)
      if (__shfl_sync(kAll, slot, int(base8 + k)) == sub) from = k;
    {
      int const src = int(base8 + (from & 7u));
      ref = __shfl_sync(kAll, ref, src);
      cnt = __shfl_sync(kAll, cnt, src);
      kb.lo.x = __shfl_sync(kAll, kb.lo.x, src), kb.lo.y = __shfl_sync(kAll, kb.lo.y, src);
      kb.lo.z = __shfl_sync(kAll, kb.lo.z, src), kb.hi.x = __shfl_sync(kAll, kb.hi.x, src);
      kb.hi.y = __shfl_sync(kAll, kb.hi.y, src), kb.hi.z = __shfl_sync(kAll, kb.hi.z, src);
      if (from == 8u) cnt = 0;
    }
    bool const internal = cnt > uint32_t(kMaxLeaf);
    uint32_t const tris = internal ? 0u : cnt;
    uint32_t const imask = (__ballot_sync(kAll, internal) >> base8) & 0xffu;
    uint32_t const leaves = (__ballot_sync(kAll, tris > 0u) >> base8) & 0xffu;
    uint32_t const rank = uint32_t(__popc(imask & ((1u << sub) - 1u)));
    uint32_t tri_end = tris;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      uint32_t const v = __shfl_up_sync(kAll, tri_end, o, 8);
      if (sub >= uint32_t(o)) tri_end += v;
    }
    uint32_t const tri_off = tri_end - tris;
    // queue, node and triangle space of the block's nodes
    if (sub == 7u) {
      s_int[oct] = uint32_t(__popc(imask));
      s_tri[oct] = tri_end;
      s_slots[oct] = uint32_t(__popc(leaves));
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      uint32_t const i0 = lane < kColNodes ? s_int[lane] : 0u, t0 = lane < kColNodes ? s_tri[lane] : 0u;
      uint32_t i1 = i0, t1 = t0, sl = lane < kColNodes ? s_slots[lane] : 0u;
#pragma unroll
      for (int o = 1; o < kColNodes; o <<= 1) {
        uint32_t const vi = __shfl_up_sync(kAll, i1, o), vt = __shfl_up_sync(kAll, t1, o);
        if (lane >= uint32_t(o)) i1 += vi, t1 += vt;
      }
      sl = __reduce_add_sync(kAll, sl);
      if (lane < kColNodes) s_int[lane] = i1 - i0, s_tri[lane] = t1 - t0;
      if (lane == kColNodes - 1) {
        s_base[0] = i1 ? atomicAdd(&a.counters[0], i1) : 0u;
        s_base[1] = t1 ? atomicAdd(&a.counters[1], t1) : 0u;
        s_base[2] = i1 ? atomicAdd(a.n_out, i1) : 0u;
      } else if (lane == 0) {
        if (sl) atomicAdd(&a.counters[4], sl);
        atomicMax(&a.counters[3], item.depth);
      }
    }
    __syncthreads();
    uint32_t const child_base = s_base[0] + s_int[oct], tri_base = s_base[1] + s_tri[oct],
                   out_base = s_base[2] + s_int[oct];
    // quantise the slot's box outwards
    float const p[3] = {nb.lo.x, nb.lo.y, nb.lo.z};
    float const ext[3] = {nb.hi.x - nb.lo.x, nb.hi.y - nb.lo.y, nb.hi.z - nb.lo.z};
    float const blo[3] = {kb.lo.x, kb.lo.y, kb.lo.z}, bhi[3] = {kb.hi.x, kb.hi.y, kb.hi.z};
    uint8_t* const img = s_node[oct];
    uint32_t exps = imask << 24;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      uint32_t const e = biased_exponent(ext[ax]);
      exps |= e << (8 * ax);
      double const inv = pow2(127 - int(e));
      double const lo = floor((double(blo[ax]) - double(p[ax])) * inv);
      double const hi = ceil((double(bhi[ax]) - double(p[ax])) * inv);
      img[32 + 8 * ax + sub] = cnt ? uint8_t(fmin(fmax(lo, 0.0), 255.0)) : uint8_t(1);
      img[56 + 8 * ax + sub] = cnt ? uint8_t(fmin(fmax(hi, 0.0), 255.0)) : uint8_t(0);
    }
    img[24 + sub] = internal ? uint8_t(0x20u | sub) : (cnt ? uint8_t(tri_off | (cnt << 5)) : uint8_t(0));
    if (sub == 0) {
      uint32_t* const h = reinterpret_cast<uint32_t*>(img);
      h[0] = __float_as_uint(p[0]), h[1] = __float_as_uint(p[1]), h[2] = __float_as_uint(p[2]);
      h[3] = exps;
      h[4] = __popc(imask) ? child_base : 0u;
      h[5] = leaves ? tri_base : 0u;
    }
    __syncwarp();
    if (live) {
      if (sub < 5u) reinterpret_cast<uint4*>(a.nodes + item.wide)[sub] = reinterpret_cast<uint4 const*>(img)[sub];
      if (internal) {
        a.out[out_base + rank] = collapse_item{ref, child_base + rank, item.depth + 1u};
      } else if (cnt) {
        uint32_t const q = (ref & kLeafBit) ? (ref & ~kLeafBit) : a.range[ref].x;
        for (uint32_t i = 0; i < cnt; ++i) a.tri_prim[tri_base + tri_off + i] = a.order[q + i];
      }
    }
    __syncthreads();  // the shared arrays are reused
  }
}

// Leaf-ordered triangles from their prims.
__global__ void k_emit_tris(float const* __restrict__ pos, uint32_t const* __restrict__ tri_prim, uint32_t n,
    float4* __restrict__ tris) {
  uint32_t const t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  uint32_t const prim = tri_prim[t];
  float const* v = pos + 9 * size_t(prim);
  float4* o = tris + 3 * size_t(t);
  o[0] = make_float4(v[0], v[1], v[2], __uint_as_float(prim));
  o[1] = make_float4(v[3], v[4], v[5], 0.f);
  o[2] = make_float4(v[6], v[7], v[8], 0.f);
}

template <typename T> int dalloc(T** p, size_t count, std::vector<void*>& owned) {
  cudaError_t const e = cudaMalloc(reinterpret_cast<void**>(p), std::max<size_t>(count, 1) * sizeof(T));
  if (e != cudaSuccess) return int(e);
  owned.push_back(*p);
  return 0;
}

// Sub-allocation of the scratch block: 256-byte aligned slices.
struct carve {
  size_t total = 0;
  template <typename T> size_t take(size_t count) {
    size_t const at = total;
    total += (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
    return at;
  }
};

}  // namespace

int build_bvh8_device(float const* d_pos, size_t n_tris, cudaStream_t st, device_build_scratch& scratch,
    device_bvh8 const* reuse, device_bvh8& out, char const** what) {
  out = device_bvh8{};
  *what = nullptr;
  if (n_tris == 0) return 0;
  if (n_tris >= (size_t(1) << 30)) {
    *what = "too many triangles for the device builder";
    return -1;
  }
  auto const t0 = std::chrono::steady_clock::now();
  int const n = int(n_tris);
  int e = 0;
  size_t tb = 0;
  if ((e = int(cub::DeviceRadixSort::SortPairs(nullptr, tb, static_cast<uint64_t const*>(nullptr),
           static_cast<uint64_t*>(nullptr), static_cast<uint32_t const*>(nullptr), static_cast<uint32_t*>(nullptr), n,
           0, 63, st)))) {
    *what = "device BVH sort size";
    return e;
  }
  carve c;
  size_t const o_boxes = c.take<ibox>(n), o_cb = c.take<uint32_t>(6), o_k0 = c.take<uint64_t>(n),
               o_k1 = c.take<uint64_t>(n), o_v0 = c.take<uint32_t>(n), o_v1 = c.take<uint32_t>(n),
               o_child = c.take<uint2>(n), o_range = c.take<uint2>(n), o_cross = c.take<uint32_t>(n),
               o_blocks = c.take<ibox>(size_t(n) / kBoxBlock + 1), o_counters = c.take<uint32_t>(8 + kMaxLevels + 1),
               o_inner = c.take<ibox>(n), o_q0 = c.take<collapse_item>(n), o_q1 = c.take<collapse_item>(n),
               o_temp = c.take<char>(tb);
  if (scratch.bytes < c.total) {
    scratch.release();
    if ((e = int(cudaMalloc(&scratch.base, c.total)))) {
      scratch.base = nullptr;
      *what = "device BVH scratch";
      return e;
    }
    scratch.bytes = c.total;
  }
  char* const B = static_cast<char*>(scratch.base);
  auto* const boxes = reinterpret_cast<ibox*>(B + o_boxes);
  auto* const cb = reinterpret_cast<uint32_t*>(B + o_cb);
  auto* const k0 = reinterpret_cast<uint64_t*>(B + o_k0);
  auto* const k1 = reinterpret_cast<uint64_t*>(B + o_k1);
  auto* const v0 = reinterpret_cast<uint32_t*>(B + o_v0);
  auto* const v1 = reinterpret_cast<uint32_t*>(B + o_v1);
  auto* const child = reinterpret_cast<uint2*>(B + o_child);
  auto* const range = reinterpret_cast<uint2*>(B + o_range);
  auto* const cross = reinterpret_cast<uint32_t*>(B + o_cross);
  auto* const block_box = reinterpret_cast<ibox*>(B + o_blocks);
  auto* const counters = reinterpret_cast<uint32_t*>(B + o_counters);
  auto* const inner = reinterpret_cast<ibox*>(B + o_inner);
  collapse_item* const q[2] = {reinterpret_cast<collapse_item*>(B + o_q0), reinterpret_cast<collapse_item*>(B + o_q1)};
  void* const temp = B + o_temp;
  // wide nodes: at most one per 2 triangles (every wide node but the root holds > 4) + 1
  size_t const max_nodes = n_tris / 2 + 2;
  bvh8_node* nodes;
  float4* tris;
  bool const reused = reuse && reuse->nodes && reuse->tris && reuse->node_capacity >= max_nodes &&
                      reuse->tri_capacity >= 3 * n_tris;
  if (reused) {
    nodes = reuse->nodes;
    tris = reuse->tris;
  } else {
    std::vector<void*> keep;
    if ((e = dalloc(&nodes, max_nodes, keep)) || (e = dalloc(&tris, 3 * n_tris, keep))) {
      for (void* p : keep) cudaFree(p);
      *what = "device BVH output";
      return e;
    }
  }
  auto fail = [&](int err, char const* w) {
    if (!reused) {
      cudaFree(nodes);
      cudaFree(tris);
    }
    *what = w;
    return err;
  };
  // counters: [0] wide nodes (the root); lens[l]: level l's queue length (level 0: the root item)
  static uint32_t const init_cb[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
  static uint32_t const init_counters[9] = {1u, 0u, 0u, 0u, 0u, 0u, 0u, 0u, 1u};
  uint32_t* const lens = counters + 8;
  collapse_item const root{n >= 2 ? 0u : kLeafBit, 0u, 1u};
  cudaMemcpyAsync(cb, init_cb, sizeof init_cb, cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(counters, 0, (8 + kMaxLevels + 1) * sizeof(uint32_t), st);
  cudaMemcpyAsync(counters, init_counters, sizeof init_counters, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(q[0], &root, sizeof root, cudaMemcpyHostToDevice, st);
  uint32_t const blocks = uint32_t((n + 255) / 256);
  k_prim_boxes<<<blocks, 256, 0, st>>>(d_pos, uint32_t(n), 1e-5f, boxes, cb);
  k_morton<<<blocks, 256, 0, st>>>(boxes, uint32_t(n), cb, k0, v0);
  if ((e = int(cub::DeviceRadixSort::SortPairs(temp, tb, k0, k1, v0, v1, n, 0, 63, st))))
    return fail(e, "device BVH sort");
  if (n >= 2) {
    k_radix_tree<<<uint32_t((n - 1 + 255) / 256), 256, 0, st>>>(k1, n, child, range);
    k_boxes_block<<<uint32_t((n + kBoxBlock - 1) / kBoxBlock), kBoxBlock, 0, st>>>(boxes, v1, n, range, inner,
        block_box, cross, counters + 2);
    k_boxes_cross<<<kCrossGrid, 256, 0, st>>>(boxes, v1, range, block_box, cross, counters + 2, inner);
  }
  collapse_args ca{};
  ca.leaf_boxes = boxes;
  ca.order = v1;
  ca.child = child;
  ca.range = range;
  ca.inner = inner;
  ca.nodes = nodes;
  ca.tri_prim = v0;  // the sort's input order, no longer needed
  ca.counters = counters;
  // Level l reads queue l & 1, lens[l] items long, and appends to the other.
  // Levels are launched in batches without reading their lengths back: a
  // level holds at most 8^l items (and at most n), which sizes its grid, up to
  // a fixed number of blocks that then loop. The first batch is what a tree of
  // n triangles usually has (an eighth per level down to 2 triangles, and 4
  // more); one read-back per batch finds the end.
  uint32_t hc[8], len = 1;
  uint32_t bound = 1;
  int batch = 4;
  for (size_t m = n_tris / 2; m > 0; m /= 8) ++batch;
  for (int level = 0; len;) {
    if (level + batch > kMaxLevels) return fail(-1, "device BVH collapse did not finish");
    for (int b = 0; b < batch; ++b, ++level) {
      int const in = level & 1;
      ca.in = q[in];
      ca.n_in = lens + level;
      ca.out = q[in ^ 1];
      ca.n_out = lens + level + 1;
      k_collapse<<<std::min<uint32_t>((bound + kColNodes - 1) / kColNodes, kColGrid), kColBlock, 0, st>>>(ca);
      bound = uint32_t(std::min<uint64_t>(uint64_t(bound) * 8u, uint64_t(n)));
    }
    // complete once no level is left; until then v0 holds valid prims
    k_emit_tris<<<blocks, 256, 0, st>>>(d_pos, v0, uint32_t(n), tris);
    cudaMemcpyAsync(hc, counters, sizeof hc, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&len, lens + level, sizeof len, cudaMemcpyDeviceToHost, st);
    if ((e = int(cudaStreamSynchronize(st)))) return fail(e, "device BVH collapse");
    batch = 4;
  }
  if ((e = int(cudaGetLastError()))) return fail(e, "device BVH launch");
  out.nodes = nodes;
  out.tris = tris;
  out.node_capacity = reused ? reuse->node_capacity : max_nodes;
  out.tri_capacity = reused ? reuse->tri_capacity : 3 * n_tris;
  out.n_nodes = hc[0];
  out.n_tris = hc[1];
  out.wide_depth = int(hc[3]);
  out.leaf_slots = hc[4];
  out.binary_nodes = n >= 2 ? size_t(2 * n - 1) : 1;
  out.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  return 0;
}

}  // namespace myrt_b200

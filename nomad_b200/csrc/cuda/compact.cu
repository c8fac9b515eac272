// Residency compaction of the SceneBVH arrays on the device.
//
// Produces, from the full SceneBVH arrays and a per-primitive active mask, exactly the compacted
// arrays the reference's rebuildResidentResources builds on the host when residency compaction
// is on (Nomad Path Tracer/Renderer/Renderer.cpp:5359-5560, the cached-BLAS path): active
// primitives in object order and, within an object, in BLAS leaf order; each object's BLAS
// pruned of leaves without active primitives, inner nodes with one surviving child replaced by
// that child, surviving nodes numbered in post-order (children before parents) with unchanged
// bounds; instance records pointing at the compact ranges; the TLAS unchanged.
//
// The reference walks each object's tree recursively. Here every primitive and every node is
// one thread, with two exclusive scans:
//   * cpos = exclusive scan of the active flags in leaf order. A primitive's compact index is
//     cpos at its leaf position; a leaf keeps cpos[first] and cpos[end] - cpos[first] primitives.
//     Because a SceneBVH subtree covers a contiguous leaf range (left subtree first), a subtree
//     survives iff its range holds an active primitive, and an inner node is emitted iff both
//     children survive (otherwise it is dropped or replaced by its surviving child).
//   * epos = exclusive scan of the emitted flags in node (pre-)order. A node's post-order index
//     among emitted nodes is epos[end of its subtree] - 1 - (emitted strict ancestors), its right
//     child's representative is the node just before it, and its left child's representative
//     precedes the right subtree's emitted nodes.
// Every pointer walk is bounded by the traversal stack limit and every index is range-checked;
// a violation sets a bit in counts[2] instead of faulting.
//
// Five launches. The primitive copy is bound by HBM, the node walks by the latency of dependent
// loads; they share a launch, their blocks alternating, so one hides the other. Flags are bits, and
// a scan is a launch that writes them with their tiles' sums and one that adds up the sums before
// its tile. City of 2.48M triangles at 40 % of objects:
// 142 us (418 MB in all: 64 us at the copy rate, 53 for the 343 MB that are copied); 209 us as 14 launches
// one after the other.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../../include/nomad_scene.h"

namespace {

constexpr int kT = 256;           // threads per block of the per-item kernels
constexpr int kScanT = 1024;      // threads of the block that scans the sums of large inputs
constexpr uint32_t kTile = 4096;  // items per scan tile
constexpr uint32_t kTileWords = kTile / 32;
constexpr uint32_t kDirect = 16384;  // sums up to which every tile adds up those before it itself
constexpr int kMaxWalk = 128;     // longest root-to-leaf walk accepted

enum : uint32_t { kErrIndex = 1u, kErrDepth = 2u, kErrLayout = 4u };

__device__ __forceinline__ int32_t left_first(const float4 *bvh, int32_t i) {
  return __float_as_int(__ldg(&bvh[2 * (size_t)i].w));
}
__device__ __forceinline__ int32_t count_of(const float4 *bvh, int32_t i) {
  return __float_as_int(__ldg(&bvh[2 * (size_t)i + 1].w));
}

__device__ __forceinline__ void flag(uint32_t *err, uint32_t bit) { atomicOr(err, bit); }

// ---- exclusive scan of bits (sums by the kernels that set them, then one pass) ----

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}

// Exclusive prefix of v over the block; *total receives the block sum.
__device__ uint32_t block_exclusive(uint32_t v, uint32_t *sh, uint32_t *total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t inc = warp_inclusive(v);
  if (lane == 31) sh[w] = inc;
  __syncthreads();
  if (w == 0) {
    const uint32_t s = lane < nw ? sh[lane] : 0u;
    const uint32_t si = warp_inclusive(s);
    if (lane < nw) sh[lane] = si;
  }
  __syncthreads();
  const uint32_t off = w ? sh[w - 1] : 0u;
  *total = sh[nw - 1];
  __syncthreads();
  return off + inc - v;
}

// One block: exclusive scan of the tile sums in place; pos[m] = total.
__global__ void __launch_bounds__(kScanT) k_scan_top(uint32_t *__restrict__ sums, uint32_t tiles,
                                                     uint32_t *__restrict__ pos, uint32_t m) {
  __shared__ uint32_t sh[32];
  uint32_t carry = 0;
  for (uint32_t b = 0; b < tiles; b += kScanT) {
    const uint32_t i = b + threadIdx.x;
    const uint32_t v = i < tiles ? sums[i] : 0u;
    uint32_t tot;
    const uint32_t ex = block_exclusive(v, sh, &tot);
    if (i < tiles) sums[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) pos[m] = carry;
}

// The set bits before tile `tile` (sums: set bits per tile, or per 1 / `per` of one; scanned: already
// prefix sums). Called by a whole block.
__device__ __forceinline__ uint32_t bits_before(const uint32_t *__restrict__ sums, uint32_t tile, uint32_t per, bool scanned,
                                                uint32_t *sh) {
  if (scanned) return sums[tile * per];
  uint32_t v = 0;
  for (uint32_t i = threadIdx.x; i < tile * per; i += blockDim.x) v += sums[i];
  uint32_t total;
  block_exclusive(v, sh, &total);
  return total;
}

// The tile's words and the set bits before each of them, in shared memory; returns those up to the
// tile's end.
__device__ __forceinline__ uint32_t tile_words(const uint32_t *__restrict__ bits, uint32_t tile, uint32_t before, uint32_t *sh,
                                               uint32_t *word, uint32_t *pos) {
  const uint32_t w = threadIdx.x < kTileWords ? bits[(size_t)tile * kTileWords + threadIdx.x] : 0u;
  uint32_t total;
  const uint32_t ex = block_exclusive(__popc(w), sh, &total);
  if (threadIdx.x < kTileWords) {
    word[threadIdx.x] = w;
    pos[threadIdx.x] = before + ex;
  }
  __syncthreads();
  return before + total;
}

// ---- compaction ----

// Last node (a leaf, in pre-order) of the subtree of node u; its index + 1 ends the subtree.
__device__ __forceinline__ bool rightmost_leaf(const float4 *bvh, uint32_t N, int32_t u, int32_t &leaf,
                                               uint32_t *err) {
  for (int s = 0; s < kMaxWalk; ++s) {
    if (u < 0 || (uint32_t)u >= N) {
      flag(err, kErrIndex);
      return false;
    }
    const int32_t c = count_of(bvh, u);
    if (c > 0) {
      leaf = u;
      return true;
    }
    u = -c;
  }
  flag(err, kErrDepth);
  return false;
}

// Leaf-order activity bits (bit j: active[primIdx[j]]) with the tiles' sums, a block per tile; then a
// thread per object for the end of its node range, which needs nothing of it.
__global__ void __launch_bounds__(kT) k_prim_bits(const int32_t *__restrict__ primIdx, const uint8_t *__restrict__ active,
                                                  uint32_t n, uint32_t tiles, uint32_t *__restrict__ bits,
                                                  uint32_t *__restrict__ sums, const float4 *__restrict__ bvh, uint32_t N,
                                                  const nomad_instance_record *__restrict__ inst, uint32_t nobj,
                                                  int32_t *__restrict__ objEnd, uint32_t *__restrict__ err) {
  const uint32_t tile = blockIdx.x;
  if (tile >= tiles) {
    const uint32_t o = (tile - tiles) * kT + threadIdx.x;
    if (o >= nobj) return;
    const int32_t r = inst[o].blas_root_index;
    int32_t leaf = -1;
    objEnd[o] = (r >= 0 && rightmost_leaf(bvh, N, r, leaf, err)) ? leaf + 1 : -1;
    return;
  }
  __shared__ uint32_t sh[32];
  uint32_t sum = 0;
  const uint32_t first = tile * kTile + threadIdx.x;
#pragma unroll 4
  for (uint32_t k = 0; k < kTile / kT; ++k) {
    const uint64_t j = (uint64_t)first + k * kT;
    bool on = false;
    if (j < n) {
      const int32_t g = primIdx[j];
      if (g < 0 || (uint32_t)g >= n) flag(err, kErrIndex);
      else on = active[g] != 0;
    }
    const uint32_t w = __ballot_sync(0xffffffffu, on);
    if ((threadIdx.x & 31) == 0) {
      bits[(size_t)tile * kTileWords + k * (kT / 32) + (threadIdx.x >> 5)] = w;
      sum += __popc(w);
    }
  }
  uint32_t total;
  block_exclusive(sum, sh, &total);
  if (threadIdx.x == 0) sums[tile] = total;
}

// Compact slots: cpos (exclusive scan of the bits), remap (compact -> global), compact primitive index
// (its own slot), global -> compact map; then a block per object for its nodes' root (rootOf).
__global__ void __launch_bounds__(kT) k_prim_slots(const int32_t *__restrict__ primIdx, const uint32_t *__restrict__ bits,
                                                   const uint32_t *__restrict__ sums, bool scanned, uint32_t n,
                                                   uint32_t tiles, uint32_t *__restrict__ cpos,
                                                   uint32_t *__restrict__ oRemap, int32_t *__restrict__ oIdx,
                                                   int32_t *__restrict__ oPrimToRes,
                                                   const nomad_instance_record *__restrict__ inst,
                                                   const int32_t *__restrict__ objEnd, int32_t *__restrict__ rootOf) {
  if (blockIdx.x >= tiles) {
    const uint32_t o = blockIdx.x - tiles;
    const int32_t r = inst[o].blas_root_index, end = objEnd[o];
    for (int32_t v = r + (int32_t)threadIdx.x; v < end; v += (int32_t)kT) rootOf[v] = r;  // end is -1 without a BLAS
    return;
  }
  __shared__ uint32_t sh[32], word[kTileWords], pos[kTileWords];
  const uint32_t before = bits_before(sums, blockIdx.x, 1, scanned, sh);
  const uint32_t end = tile_words(bits, blockIdx.x, before, sh, word, pos);
  if (blockIdx.x + 1 == tiles && threadIdx.x == 0) cpos[n] = end;
  const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll 4
  for (uint32_t k = 0; k < kTile / kT; ++k) {
    const uint64_t j = (uint64_t)blockIdx.x * kTile + k * kT + threadIdx.x;
    if (j >= n) break;
    const uint32_t i = k * (kT / 32) + (threadIdx.x >> 5), w = word[i];
    const uint32_t slot = pos[i] + __popc(w & lt);
    const bool on = w & (lt + 1u);  // only valid indices are flagged
    const int32_t g = primIdx[j];
    cpos[j] = slot;
    if (g >= 0 && (uint32_t)g < n) oPrimToRes[g] = on ? (int32_t)slot : -1;
    if (on) {
      oRemap[slot] = (uint32_t)g;
      oIdx[slot] = (int32_t)slot;
    }
  }
}

// The active primitives' packed primitive (7 float4) and material (5 float4), one float4 per
// thread and step in compact order: reads follow the remap, writes are contiguous; four steps'
// loads are in flight at once. Block `block` of `blocks`.
__device__ __forceinline__ void copy_prims(const uint32_t *__restrict__ remap, uint64_t items, uint32_t block, uint32_t blocks,
                                           const float4 *__restrict__ prims, const float4 *__restrict__ mats,
                                           float4 *__restrict__ oPrims, float4 *__restrict__ oMats) {
  for (uint64_t t0 = (uint64_t)block * 4 * kT + threadIdx.x; t0 < items; t0 += (uint64_t)blocks * 4 * kT) {
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint64_t t = t0 + k * kT;
      if (t < items) {
        const uint64_t slot = t / 12ull;
        const uint32_t part = (uint32_t)(t - slot * 12ull), g = __ldg(&remap[slot]);
        v[k] = __ldg(part < 7u ? &prims[(size_t)g * 7 + part] : &mats[(size_t)g * 5 + (part - 7u)]);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint64_t t = t0 + k * kT;
      if (t < items) {
        const uint64_t slot = t / 12ull;
        const uint32_t part = (uint32_t)(t - slot * 12ull);
        if (part < 7u) oPrims[slot * 7 + part] = v[k];
        else oMats[slot * 5 + (part - 7u)] = v[k];
      }
    }
  }
}

// Whether node v is emitted: its range holds an active primitive (leaf), or both of its children's
// do.
__device__ __forceinline__ bool node_emitted(const float4 *__restrict__ bvh, uint32_t N, uint32_t v,
                                             const uint32_t *__restrict__ cpos, uint32_t n, uint32_t *__restrict__ err) {
  const int32_t c = count_of(bvh, v), lf = left_first(bvh, v);
  if (c > 0) {
    if (lf < 0 || (int64_t)lf + c > (int64_t)n) {
      flag(err, kErrIndex);
      return false;
    }
    return cpos[lf + c] != cpos[lf];
  }
  // First leaf of the left and of the right subtree (walking left children), last leaf of the right one
  // (walking right children, in pre-order the subtree's last node): three walks of dependent loads,
  // taken side by side.
  int32_t at[3] = {lf, -c, -c}, cnt[3] = {0, 0, 0}, first[3] = {0, 0, 0};
  for (int step = 0; step < kMaxWalk && !(cnt[0] > 0 && cnt[1] > 0 && cnt[2] > 0); ++step) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (cnt[k] > 0) continue;
      if (at[k] < 0 || (uint32_t)at[k] >= N) {
        flag(err, kErrIndex);
        return false;
      }
      cnt[k] = count_of(bvh, at[k]);
      first[k] = left_first(bvh, at[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (cnt[k] <= 0) at[k] = k < 2 ? first[k] : -cnt[k];
  }
  if (!(cnt[0] > 0 && cnt[1] > 0 && cnt[2] > 0)) {
    flag(err, kErrDepth);
    return false;
  }
  const int32_t s = first[0], mid = first[1];
  const int64_t end = (int64_t)first[2] + cnt[2];
  if (s < 0 || mid < s || end < mid || end > (int64_t)n) {
    flag(err, kErrLayout);
    return false;
  }
  return cpos[mid] != cpos[s] && cpos[end] != cpos[mid];
}

// Emitted bits of the nodes (a thread a node, a sum per block) and the primitive copy, in alternating
// blocks. The copy's blocks stay until it is done and take 6 of the 8 an SM holds (4 of 8: 11 % slower per
// compaction of the city, 5: 3 %, all 8: 16 %); the node blocks pass through the others.
__global__ void __launch_bounds__(kT, 8) k_copy_nodes(const uint32_t *__restrict__ remap, const uint32_t *__restrict__ cpos,
                                                   uint32_t n, const float4 *__restrict__ prims,
                                                   const float4 *__restrict__ mats, float4 *__restrict__ oPrims,
                                                   float4 *__restrict__ oMats, uint32_t copyBlocks,
                                                   const float4 *__restrict__ bvh, uint32_t N, uint32_t nodeBlocks,
                                                   uint32_t *__restrict__ bits, uint32_t *__restrict__ sums,
                                                   uint32_t *__restrict__ err) {
  const uint32_t both = 2 * min(copyBlocks, nodeBlocks), b = blockIdx.x;
  const bool copies = b < both ? !(b & 1u) : copyBlocks > nodeBlocks;
  const uint32_t at = b < both ? b / 2 : b - both / 2;
  if (copies) {
    copy_prims(remap, (uint64_t)cpos[n] * 12ull, at, copyBlocks, prims, mats, oPrims, oMats);
    return;
  }
  __shared__ uint32_t sh[32];
  const uint32_t v = at * kT + threadIdx.x;
  const uint32_t w = __ballot_sync(0xffffffffu, v < N && node_emitted(bvh, N, v, cpos, n, err));
  const bool head = (threadIdx.x & 31) == 0;
  if (head) bits[v >> 5] = w;
  uint32_t total;
  block_exclusive(head ? __popc(w) : 0u, sh, &total);
  if (threadIdx.x == 0) sums[at] = total;
}

// epos: exclusive scan of the emitted bits.
__global__ void __launch_bounds__(kT) k_node_slots(const uint32_t *__restrict__ bits, const uint32_t *__restrict__ sums,
                                                   bool scanned, uint32_t N, uint32_t *__restrict__ epos) {
  __shared__ uint32_t sh[32], word[kTileWords], pos[kTileWords];
  const uint32_t before = bits_before(sums, blockIdx.x, kTile / kT, scanned, sh);
  const uint32_t end = tile_words(bits, blockIdx.x, before, sh, word, pos);
  if (blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) epos[N] = end;
  const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll 4
  for (uint32_t k = 0; k < kTile / kT; ++k) {
    const uint64_t v = (uint64_t)blockIdx.x * kTile + k * kT + threadIdx.x;
    if (v >= N) break;
    const uint32_t i = k * (kT / 32) + (threadIdx.x >> 5);
    epos[v] = pos[i] + __popc(word[i] & lt);
  }
}

// Emitted nodes to their post-order slots.
__device__ __forceinline__ bool bit(const uint32_t *__restrict__ bits, int32_t i) { return (bits[i >> 5] >> (i & 31)) & 1u; }

__device__ __forceinline__ void emit_node(int32_t v, const float4 *__restrict__ bvh, uint32_t N,
                                          const uint32_t *__restrict__ cpos, const uint32_t *__restrict__ bits,
                                          const uint32_t *__restrict__ epos, const int32_t *__restrict__ rootOf,
                                          float4 *__restrict__ oBvh, uint32_t *__restrict__ err) {
  if ((uint32_t)v >= N || !bit(bits, v)) return;
  // emitted strict ancestors (walking down from the object's root) and the end of the node's subtree
  // (walking its right children), side by side
  const int32_t c = count_of(bvh, v), lf = left_first(bvh, v);
  int32_t u = rootOf[v], last = c > 0 ? v : -c;
  bool ended = c > 0;
  uint32_t anc = 0;
  for (int s = 0; s < kMaxWalk && (u != v || !ended); ++s) {
    if (u != v) {
      if (u < 0 || (uint32_t)u >= N || u > v) {
        flag(err, kErrLayout);
        return;
      }
    }
    if (!ended && (last < 0 || (uint32_t)last >= N)) {
      flag(err, kErrIndex);
      return;
    }
    const int32_t cu = u != v ? count_of(bvh, u) : 0, cl = ended ? 0 : count_of(bvh, last);
    if (u != v) {
      if (bit(bits, u)) ++anc;
      if (cu > 0) {
        flag(err, kErrLayout);
        return;
      }
      u = v < -cu ? left_first(bvh, u) : -cu;
    }
    if (!ended) {
      if (cl > 0) ended = true;
      else last = -cl;
    }
  }
  if (u != v || !ended) {
    flag(err, kErrDepth);
    return;
  }
  const int32_t end = last + 1;
  const int32_t P = (int32_t)(epos[end] - 1u - anc);
  float4 lo = __ldg(&bvh[2 * (size_t)v]), hi = __ldg(&bvh[2 * (size_t)v + 1]);
  if (c > 0) {
    lo.w = __int_as_float((int32_t)cpos[lf]);
    hi.w = __int_as_float((int32_t)(cpos[lf + c] - cpos[lf]));
  } else {
    const int32_t rightRep = P - 1;
    const int32_t leftRep = rightRep - (int32_t)(epos[end] - epos[-c]);
    lo.w = __int_as_float(leftRep);
    hi.w = __int_as_float(-rightRep);
  }
  oBvh[2 * (size_t)P] = lo;
  oBvh[2 * (size_t)P + 1] = hi;
}

__device__ __forceinline__ void object_record(uint32_t o, const nomad_instance_record *__restrict__ inst, uint32_t nobj,
                                              uint32_t n, const uint32_t *__restrict__ cpos,
                                              const uint32_t *__restrict__ epos, uint32_t N,
                                              const int32_t *__restrict__ objEnd,
                                              nomad_instance_record *__restrict__ oInst, uint32_t *__restrict__ counts,
                                              uint32_t *__restrict__ err) {
  if (o == 0) {
    counts[0] = cpos[n];
    counts[1] = epos[N];
  }
  if (o >= nobj) return;
  const nomad_instance_record r = inst[o];
  const uint64_t first = r.primitive_index_base, end = first + r.primitive_count;
  nomad_instance_record w;
  w.blas_root_index = -1;
  if (end > n || r.primitive_base != r.primitive_index_base) {
    flag(err, kErrIndex);
    w.primitive_base = w.primitive_index_base = 0;
    w.primitive_count = 0;
    oInst[o] = w;
    return;
  }
  const uint32_t base = cpos[first], cnt = cpos[end] - base;
  w.primitive_base = base;
  w.primitive_index_base = base;
  w.primitive_count = cnt;
  if (cnt > 0) {
    const int32_t root = r.blas_root_index, oe = root >= 0 ? objEnd[o] : -1;
    if (root < 0 || oe <= root || epos[oe] == epos[root])
      flag(err, kErrLayout);  // active primitives without a BLAS over them
    else
      w.blas_root_index = (int32_t)(epos[oe] - 1u);  // the pruned root is last in post-order
  }
  oInst[o] = w;
}

// The emitted nodes, then the instance records.
__global__ void __launch_bounds__(kT) k_emit(const float4 *__restrict__ bvh, uint32_t N, uint32_t nodeBlocks,
                                             const uint32_t *__restrict__ cpos, uint32_t n,
                                             const uint32_t *__restrict__ bits, const uint32_t *__restrict__ epos,
                                             const int32_t *__restrict__ rootOf, float4 *__restrict__ oBvh,
                                             const nomad_instance_record *__restrict__ inst, uint32_t nobj,
                                             const int32_t *__restrict__ objEnd,
                                             nomad_instance_record *__restrict__ oInst, uint32_t *__restrict__ counts,
                                             uint32_t *__restrict__ err) {
  if (blockIdx.x < nodeBlocks)
    emit_node((int32_t)(blockIdx.x * kT + threadIdx.x), bvh, N, cpos, bits, epos, rootOf, oBvh, err);
  else
    object_record((blockIdx.x - nodeBlocks) * kT + threadIdx.x, inst, nobj, n, cpos, epos, N, objEnd, oInst, counts, err);
}

size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

uint32_t tiles_of(uint32_t m) { return (uint32_t)(((uint64_t)m + kTile - 1) / kTile); }

struct Work {
  uint32_t *pbits, *psums, *cpos, *nbits, *nsums, *epos, *err;
  int32_t *rootOf, *objEnd;
};

size_t layout(uint32_t n, uint32_t N, uint32_t nobj, char *base, Work *w) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += align_up(bytes);
    return p;
  };
  const size_t pt = tiles_of(n), nt = tiles_of(N);
  char *pbits = take(pt * kTileWords * 4), *psums = take(pt * 4), *cpos = take(((size_t)n + 1) * 4),
       *nbits = take(nt * kTileWords * 4), *nsums = take(nt * (kTile / kT) * 4), *epos = take(((size_t)N + 1) * 4),
       *err = take(4), *rootOf = take((size_t)N * 4), *objEnd = take((size_t)nobj * 4);
  if (w) {
    w->pbits = (uint32_t *)pbits;
    w->psums = (uint32_t *)psums;
    w->cpos = (uint32_t *)cpos;
    w->nbits = (uint32_t *)nbits;
    w->nsums = (uint32_t *)nsums;
    w->epos = (uint32_t *)epos;
    w->err = (uint32_t *)err;
    w->rootOf = (int32_t *)rootOf;
    w->objEnd = (int32_t *)objEnd;
  }
  return off;
}

}  // namespace

extern "C" size_t nomad_compact_workspace_bytes(uint32_t prim_count, uint32_t bvh_node_count,
                                                uint32_t object_count) {
  return layout(prim_count, bvh_node_count, object_count, nullptr, nullptr);
}

extern "C" nomad_status nomad_scenebvh_compact_gpu(const nomad_scenebvh_device *in, const uint8_t *prim_active,
                                                   void *workspace, size_t workspace_bytes,
                                                   const nomad_compact_out *out, void *stream) {
  if (!in || !out || !prim_active || !workspace) return NOMAD_ERR_INVALID_ARGUMENT;
  const uint32_t n = in->prim_count, N = in->bvh_node_count, nobj = in->object_count;
  if (n == 0 || nobj == 0 || !in->bvh_nodes || !in->prims || !in->materials || !in->prim_indices ||
      !in->instances || !out->bvh_nodes || !out->prims || !out->materials || !out->prim_indices ||
      !out->remap || !out->prim_to_resident || !out->instances || !out->counts)
    return NOMAD_ERR_INVALID_ARGUMENT;
  if (n > 0x7fffffffu || N > 0x7fffffffu) return NOMAD_ERR_LIMIT;
  Work w;
  if (workspace_bytes < layout(n, N, nobj, static_cast<char *>(workspace), &w)) return NOMAD_ERR_INVALID_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float4 *bvh = reinterpret_cast<const float4 *>(in->bvh_nodes);
  // node blocks: whole tiles, so that every word and sum of the last one is written
  const uint32_t pt = tiles_of(n), nt = tiles_of(N), gn = nt * (kTile / kT);
  if (cudaMemsetAsync(w.err, 0, 4, s) != cudaSuccess) return NOMAD_ERR_CUDA;
  if (N && cudaMemsetAsync(w.rootOf, 0xff, (size_t)N * 4, s) != cudaSuccess) return NOMAD_ERR_CUDA;
  if (!N && cudaMemsetAsync(w.objEnd, 0xff, (size_t)nobj * 4, s) != cudaSuccess) return NOMAD_ERR_CUDA;
  k_prim_bits<<<pt + (N ? (nobj + kT - 1) / kT : 0u), kT, 0, s>>>(in->prim_indices, prim_active, n, pt, w.pbits, w.psums,
                                                                  bvh, N, in->instances, nobj, w.objEnd, w.err);
  if (pt > kDirect) k_scan_top<<<1, kScanT, 0, s>>>(w.psums, pt, w.cpos, n);
  k_prim_slots<<<pt + (N ? nobj : 0u), kT, 0, s>>>(in->prim_indices, w.pbits, w.psums, pt > kDirect, n, pt, w.cpos,
                                                   out->remap, out->prim_indices, out->prim_to_resident, in->instances,
                                                   w.objEnd, w.rootOf);
  {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t gc = (uint32_t)std::min<uint64_t>((uint64_t)sms * 6, ((uint64_t)n * 12 + 4 * kT - 1) / (4 * kT));
    k_copy_nodes<<<gc + gn, kT, 0, s>>>(out->remap, w.cpos, n, reinterpret_cast<const float4 *>(in->prims),
                                        reinterpret_cast<const float4 *>(in->materials),
                                        reinterpret_cast<float4 *>(out->prims),
                                        reinterpret_cast<float4 *>(out->materials), gc, bvh, N, gn, w.nbits, w.nsums,
                                        w.err);
  }
  if (N) {
    if (gn > kDirect) k_scan_top<<<1, kScanT, 0, s>>>(w.nsums, gn, w.epos, N);
    k_node_slots<<<nt, kT, 0, s>>>(w.nbits, w.nsums, gn > kDirect, N, w.epos);
  } else if (cudaMemsetAsync(w.epos, 0, 4, s) != cudaSuccess) {
    return NOMAD_ERR_CUDA;
  }
  k_emit<<<gn + (nobj + kT - 1) / kT, kT, 0, s>>>(bvh, N, gn, w.cpos, n, w.nbits, w.epos, w.rootOf,
                                                  reinterpret_cast<float4 *>(out->bvh_nodes), in->instances, nobj,
                                                  w.objEnd, out->instances, out->counts, w.err);
  if (cudaMemcpyAsync(out->counts + 2, w.err, 4, cudaMemcpyDeviceToDevice, s) != cudaSuccess) return NOMAD_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? NOMAD_OK : NOMAD_ERR_CUDA;
}

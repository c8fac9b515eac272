// Persistent warps with cooperative leaf tests.
//
// A warp keeps one ray per lane. Lanes walk nodes on their own until enough of them hold a leaf
// (kCoopLeaves) or none has a node left; then the whole warp tests the pending leaves together:
// eight lanes per leaf, four leaves at a time, each lane one (ray, record) pair. A leaf of the
// SceneBVH builder has at most eight records (six on average on the city); a longer one stays
// pending for another pass. Rays and their closest hits live in shared memory, where the lane that
// finds a hit keeps the lexicographically smallest (t, primitive). The hits are the per-lane
// walk's bit for bit: every record of a leaf is tested against the same ray in the same
// arithmetic, and the order of the tests does not matter.
// Scenes and batches that gain nothing by it keep a per-lane walk (coop_pays).
//
// What bounds it: instruction issue on coherent rays (75 % of active cycles, the half-rate pipe of
// min, max, compare and select at 56 %), the L1's load-store wavefronts on diffuse bounces (77 % of its
// peak: each lane reads seven rows of another node). Whole nodes in four 32-byte loads, with near and
// far planes chosen in registers, took 1.54 ms for the bounces instead of 1.46. A per-lane walk
// spends most of its issue slots on leaves: lanes reach them at different steps, and a loop over
// six records runs at 4 to 9 of 32 lanes. Measured on the 2.48M-triangle city, 4-wide nodes, the
// per-lane persistent walk before and this one: 8.29M primary rays 1.19 -> 1.06 ms, 4.98M diffuse
// bounces 2.18 -> 1.46 ms, 4.98M shadow any-hits 1.85 -> 1.21 ms.
//
// Any-hit walks take the nearest child first too (in slot order the shadows took 1.72 ms, the longest
// overlap first 1.80, from the far end 2.25), but leave the other children unsorted and stack their refs
// alone, as no distance is compared again: 1.24 -> 1.21 ms.
//
// The constants, each the fastest of those tried on the same rays:
//   kCoopLeaves 8   leaf tests wait for eight leaves: 1.46 ms for the bounces; 4: 1.52, 12: 1.50.
//   kCoopOwn    13  from this many leaves on each lane walks its own records (six steps for up to
//                   32 leaves against one pass per four): primary 1.06 ms; never: 1.07, 9: 1.08.
//   kCoopRefill 16  rays of mixed octants: idle lanes store their results and take the next rays
//                   when fewer than 16 are busy (bounces 1.46; 12: 1.55, 8: 1.61, only when all
//                   are idle: 1.53; shadows 1.24, 1.31, 1.44, 1.56). Rays of one octant, such as a
//                   camera's, stay together until the warp is idle: primary 1.06 against 1.23.
//   kCoopMinBlocks 9  56 registers, 36 warps per SM: bounces 1.46; 8 blocks (64 registers) 1.48,
//                   10 blocks (48, spilling) 1.58.
#pragma once
#include <cfloat>

#include "rt_wide.cuh"

namespace nomad_dev {

constexpr int kCoopLeaves = 8;
constexpr int kCoopOwn = 13;
constexpr int kCoopRefill = 16;
constexpr int kCoopMinBlocks = 9;
constexpr int kCoopBlock = 128;
constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kNoRay = 0xffffffffu;

struct CoopShared {
  float4 o[kCoopBlock];   // origin; distance of the closest hit so far (tmax before)
  float4 d[kCoopBlock];   // direction; bits of the closest hit's primitive (INT32_MIN before)
  float4 hit[kCoopBlock]; // its u, v and the bits of its instance
  uint32_t next[kCoopBlock / 32], end[kCoopBlock / 32];  // a warp's rays of the batch not handed out yet
  int2 leaf[kCoopBlock];  // pending leaves of a warp: first record, lane of the ray
  int win[kCoopBlock];    // per ray: the lane whose hit is taken in this round
};

// What waits on a lane's stack: a ref and, for closest hits, the bits of its entry distance.
template <bool ANY>
struct alignas(ANY ? 4 : 8) StackEntry {
  int32_t ref, t;
};
template <>
struct StackEntry<true> {
  int32_t ref;
};

// A ray as the node tests use it: origin, reciprocal direction and the rows of a wide node that hold
// the planes it meets first. Along an axis the reference treats as parallel (|d| < kRayEps) the
// reciprocal is +infinity: (plane - o) * inf is -inf for the minimum and +inf for the maximum of a
// slab that contains the origin (NaN, which min and max skip, when it lies on the plane), and
// leaves an empty interval otherwise, which is the slab test's containment rule.
struct CoopRay {
  float ox, oy, oz, ix, iy, iz;
  int nX, nY, nZ;  // near-plane rows (see traverse_wide)
};

// Box tests of one node's children, unsorted: entry distance (INFINITY when missed) and ref. The
// bound is finite, so a hit's entry distance is. A ref may be kEmptyRef (a non-resident instance).
template <int W>
__device__ __forceinline__ void coop_children(const DevScene &S, const WideScene &WS, const CoopRay &r, int32_t ref,
                                              float bound, float (&t)[W], int32_t (&c)[W]) {
  if constexpr (W == 2) {
    const float4 *n = S.pn + 4ll * ref;
    const float4 p[4] = {ldg4(n), ldg4(n + 1), ldg4(n + 2), ldg4(n + 3)};
    c[0] = __float_as_int(p[0].w);
    c[1] = __float_as_int(p[1].w);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float4 mn = p[2 * k], mx = p[2 * k + 1];
      const bool px = r.nX == 0, py = r.nY == 1, pz = r.nZ == 2;
      const float tnx = ((px ? mn.x : mx.x) - r.ox) * r.ix, tfx = ((px ? mx.x : mn.x) - r.ox) * r.ix;
      const float tny = ((py ? mn.y : mx.y) - r.oy) * r.iy, tfy = ((py ? mx.y : mn.y) - r.oy) * r.iy;
      const float tnz = ((pz ? mn.z : mx.z) - r.oz) * r.iz, tfz = ((pz ? mx.z : mn.z) - r.oz) * r.iz;
      const float tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, kRayEps));
      const float tf = fminf(fminf(tfx, tfy), fminf(tfz, bound));
      t[k] = tf < tn ? INFINITY : tn;
    }
  } else {
    constexpr int Q = W / 4;
    const float4 *n = WS.wn + (long long)(W == 4 ? 8 : 16) * ref;
    const float4 *nx = n + r.nX * Q, *ny = n + r.nY * Q, *nz = n + r.nZ * Q;
    const float4 *fx = n + (3 - r.nX) * Q, *fy = n + (5 - r.nY) * Q, *fz = n + (7 - r.nZ) * Q;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float4 px = ldg4(nx + q), py = ldg4(ny + q), pz = ldg4(nz + q);
      const float4 gx = ldg4(fx + q), gy = ldg4(fy + q), gz = ldg4(fz + q), rf = ldg4(n + 6 * Q + q);
      const float ax[4] = {px.x, px.y, px.z, px.w}, ay[4] = {py.x, py.y, py.z, py.w};
      const float az[4] = {pz.x, pz.y, pz.z, pz.w}, bx[4] = {gx.x, gx.y, gx.z, gx.w};
      const float by[4] = {gy.x, gy.y, gy.z, gy.w}, bz[4] = {gz.x, gz.y, gz.z, gz.w};
      const float rr[4] = {rf.x, rf.y, rf.z, rf.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float tnx = (ax[k] - r.ox) * r.ix, tny = (ay[k] - r.oy) * r.iy, tnz = (az[k] - r.oz) * r.iz;
        const float tfx = (bx[k] - r.ox) * r.ix, tfy = (by[k] - r.oy) * r.iy, tfz = (bz[k] - r.oz) * r.iz;
        const float tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, kRayEps));
        const float tf = fminf(fminf(tfx, tfy), fminf(tfz, bound));
        t[q * 4 + k] = tf < tn ? INFINITY : tn;
        c[q * 4 + k] = __float_as_int(rr[k]);
      }
    }
  }
}

// intersect_prim of a triangle record without early exits (the lanes of a warp test 32 records at
// once, and some lane nearly always needs the last step): the same values by the same operations.
__device__ __forceinline__ bool intersect_tri(float4 o, float4 d, float4 A, float4 B, float4 C, float &tt, float &u,
                                              float &v) {
  const float hx = d.y * C.z - d.z * C.y, hy = d.z * C.x - d.x * C.z, hz = d.x * C.y - d.y * C.x;
  const float a = dot3(B.x, B.y, B.z, hx, hy, hz);
  const float f = __frcp_rn(a);
  const float sx = o.x - A.x, sy = o.y - A.y, sz = o.z - A.z;
  u = f * dot3(sx, sy, sz, hx, hy, hz);
  const float qx = sy * B.z - sz * B.y, qy = sz * B.x - sx * B.z, qz = sx * B.y - sy * B.x;
  v = f * dot3(d.x, d.y, d.z, qx, qy, qz);
  tt = f * dot3(C.x, C.y, C.z, qx, qy, qz);
  return (fabsf(a) > 1e-5f) & (u >= 0.0f) & (u <= 1.0f) & (v >= 0.0f) & (u + v <= 1.0f) & (tt > kRayEps);
}

// One pair of ray and record. With OTHER a record runs its own type's test alone; without, every lane
// runs the triangles' and the few other records add theirs. Spheres and rectangles pay for the triangle
// test that way (500 spheres, 1M coherent rays: 156 us, 119 with OTHER; a 1080p frame of 1,000 spheres
// 5,189, 4,492), triangles for the branch the other way (city bounces 3 to 8 %).
template <bool OTHER>
__device__ __forceinline__ bool coop_intersect(const DevScene &S, float4 o, float4 d, float4 A, float4 B, float4 C,
                                               int32_t pid, int type, float best, float &tt, float &u, float &v) {
  if constexpr (!OTHER) {
    bool hit = intersect_tri(o, d, A, B, C, tt, u, v) & (type == 1);
    if (type != 1 && pid >= 0)
      hit = intersect_prim(S, o.x, o.y, o.z, d.x, d.y, d.z, A, B, C, pid, type, best, tt, u, v);
    return hit;
  } else {
    tt = u = v = 0.0f;
    if (type == 1) return intersect_tri(o, d, A, B, C, tt, u, v);
    return pid >= 0 && intersect_prim(S, o.x, o.y, o.z, d.x, d.y, d.z, A, B, C, pid, type, best, tt, u, v);
  }
}

// Rays of a warp's share where n rays are dealt out in shares, on `sms` SMs. Up to 32 rays for each of 28
// warps per SM: equal shares, down to 8 rays, as the chip has lanes to spare and a warp waits for
// its slowest lane (1,000 rays of a lone call: 18.5 us in 32s, 14.4 in 8s; a 58k-ray two-bounce frame 342
// against 288 us). Above that up to 128: coherent rays want less (1M into the 117k-triangle city: 237 us,
// 220 in 32s), incoherent ones more, from which idle lanes are refilled (1M shadow rays there: 177 us, 204
// in 96s).
__host__ __device__ constexpr uint32_t coop_share(uint32_t n, uint32_t sms) {
  const uint32_t share = n / (sms * 28) + (n % (sms * 28) != 0);
  return share <= 8 ? 8u : share <= 32 ? (share + 3u) & ~3u : share < 128 ? (share + 31u) & ~31u : 128u;
}

// The same for a path tracer's queue, n the length that it has: its capacity says little, as later bounces
// are a fraction of it (1280x720, one sample, six bounces of an untuned context in the 117k-triangle
// city: 1,838 us with shares of the capacity, 915 now).
__host__ __device__ constexpr uint32_t coop_queue_share(uint32_t n, uint32_t sms) {
  return n <= sms * 896 ? coop_share(n, sms) : 32u;
}

// Walks the rays of the batch (N < 2^32): the warp's own share of `chunk` rays, or, with a cursor, 32
// rays at a time from it; DONE(i, h) stores the result of ray i (called by the lanes
// that finished one, warp-divergent). OTHER: most records are no triangles.
template <int W, int STACK, bool ANY, bool OTHER, typename DONE>
__device__ __forceinline__ void coop_trace(const DevScene &S, const WideScene &WS, CoopShared &sh,
                                           const float4 *__restrict__ rays, uint32_t N, uint32_t chunk,
                                           unsigned long long *__restrict__ cursor, DONE done) {
  const int tid = threadIdx.x, lane = tid & 31, wb = tid & ~31;
  const unsigned lt = (1u << lane) - 1u;
  CoopRay r{};
  // Where boxes are cut off: tmax for any-hit, the closest hit's distance with the pruning margin
  // otherwise; kept finite, so that INFINITY marks a missed box.
  float bound = 0.0f;
  StackEntry<ANY> stk[STACK];
  int sp = 0;
  int32_t ref = kEmptyRef;
  uint32_t ray = kNoRay;  // the lane's ray, until its result is stored
  bool more = true, mixed = false;
  // The share is kept as its two ends: with its length, min(chunk, N - first), one build of this kernel took
  // the whole chunk of the last share (CUDA 12.9), 7 rays beyond the batch.
  const uint64_t first = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (wb >> 5)) * chunk;
  if (!cursor && first >= N) return;
  if (lane == 0) {
    sh.next[wb >> 5] = cursor ? N : (uint32_t)first;
    sh.end[wb >> 5] = (uint32_t)min(first + chunk, (uint64_t)N);
  }
  for (;;) {
    while (ref == kEmptyRef && sp > 0) {  // the newest entry that still starts before the bound
      const StackEntry<ANY> e = stk[--sp];
      ref = e.ref;
      if constexpr (!ANY) ref = __int_as_float(e.t) > bound ? kEmptyRef : ref;
    }
    if (ref >= 0) {
      float t[W];
      int32_t c[W];
      coop_children<W>(S, WS, r, ref, bound, t, c);
      if constexpr (ANY && W == 4) {
        cswap(t[0], c[0], t[1], c[1]);
        cswap(t[2], c[2], t[3], c[3]);
        cswap(t[0], c[0], t[2], c[2]);
      } else {
        sort_children<W>(t, c);
      }
      // The upload sized the stack for W - 1 entries per level; the guard reports, not overruns.
      if (sp + W - 1 <= STACK) {
#pragma unroll
        for (int k = W - 1; k >= 1; --k) {
          if (t[k] < INFINITY) {
            stk[sp].ref = c[k];
            if constexpr (!ANY) stk[sp].t = __float_as_int(t[k]);
            ++sp;
          }
        }
      } else {
        atomicOr(S.status, kStatusStackOverflow);
      }
      ref = t[0] < INFINITY ? c[0] : kEmptyRef;
    }
    const unsigned leaves = __ballot_sync(kFull, (uint32_t)ref > (uint32_t)kEmptyRef);
    const unsigned busy = __ballot_sync(kFull, ref != kEmptyRef || sp > 0);
    const bool low = more && __popc(busy) < (mixed ? kCoopRefill : 1);
    if (__popc(leaves) < kCoopLeaves && leaves != busy && !low) continue;
    if (low || busy == 0) {
      const bool idle = !((busy >> lane) & 1u);
      if (ray != kNoRay && idle) {
        const float4 o = sh.o[tid], d = sh.d[tid];
        HitRec h{o.w, 0.0f, 0.0f, __float_as_int(d.w), -1};
        if (h.prim == INT32_MIN) {
          h.prim = -1;
        } else if (!ANY) {
          const float4 f = sh.hit[tid];
          h.u = f.x;
          h.v = f.y;
          h.inst = __float_as_int(f.z);
        }
        done(ray, h);
        ray = kNoRay;
      }
      __syncwarp();
      if (!more) break;  // nothing busy and nothing left
      uint32_t next = sh.next[wb >> 5], end = sh.end[wb >> 5];
      if (next >= end) {
        unsigned long long base = N;
        if (cursor) {
          if (lane == 0) base = atomicAdd(cursor, 32ull);
          base = __shfl_sync(kFull, base, 0);
        }
        if (base >= N) {
          more = false;
          continue;
        }
        next = (uint32_t)base;
        end = N - next < 32u ? N : next + 32u;
      }
      const uint32_t rank = __popc(~busy & lt);
      if (idle && rank < end - next) {
        ray = next + rank;
        const float4 a = __ldg(rays + 2ull * ray), b = __ldg(rays + 2ull * ray + 1);
        const RayP p = prep_ray(a, b);
        r = CoopRay{p.ox, p.oy, p.oz, p.ix, p.iy, p.iz, p.ix > 0.0f ? 0 : 3, p.iy > 0.0f ? 1 : 4, p.iz > 0.0f ? 2 : 5};
        if (p.par & 1) r.ix = INFINITY, r.nX = 0;
        if (p.par & 2) r.iy = INFINITY, r.nY = 1;
        if (p.par & 4) r.iz = INFINITY, r.nZ = 2;
        bound = fminf(ANY ? b.w : b.w * kPruneScale, FLT_MAX);
        if (b.w > kRayEps) {
          float tn0;
          if (slab(p, S.rmin[0], S.rmin[1], S.rmin[2], S.rmax[0], S.rmax[1], S.rmax[2], bound, tn0))
            ref = W == 2 ? S.rootRef : WS.root;
        }
        sh.o[tid] = make_float4(a.x, a.y, a.z, b.w);
        sh.d[tid] = make_float4(b.x, b.y, b.z, __int_as_float(INT32_MIN));
      }
      __syncwarp();
      if (lane == 0) {
        sh.next[wb >> 5] = min(next + __popc(~busy), end);
        sh.end[wb >> 5] = end;
      }
      // rays of one octant stay together well; mixed ones are worth refilling lane by lane
      const bool on = ray != kNoRay;
      const unsigned all = __ballot_sync(kFull, on), sx = __ballot_sync(kFull, on && r.nX == 0),
                     sy = __ballot_sync(kFull, on && r.nY == 1), sz = __ballot_sync(kFull, on && r.nZ == 2);
      mixed = !((sx == 0 || sx == all) && (sy == 0 || sy == all) && (sz == 0 || sz == all));
      continue;
    }
    const bool mine = (leaves >> lane) & 1u;
    const int total = __popc(leaves);
    if (total >= kCoopOwn) {
      // most lanes hold a leaf: each walks its own, record by record
      if (mine) {
        const float4 o = make_float4(r.ox, r.oy, r.oz, 0.0f), d = sh.d[tid];
        float ht = sh.o[tid].w, hu = 0.0f, hv = 0.0f;
        int32_t hp = __float_as_int(d.w), hi = 0;
        const int32_t p0 = hp;
        bool stop = false;
        for (const float4 *q = S.tri + 3ll * (int64_t)~ref;; q += 3) {
          const float4 A = ldg4(q), B = ldg4(q + 1), C = ldg4(q + 2);
          const int32_t pid = __float_as_int(A.w), meta = __float_as_int(C.w);
          float tt, u, v;
          const bool hit = coop_intersect<OTHER>(S, o, d, A, B, C, pid, meta & 0xff, ht, tt, u, v);
          if (hit & (pid >= 0) & ((tt < ht) | ((tt == ht) & (pid < hp)))) {
            ht = tt;
            hp = pid;
            hu = u;
            hv = v;
            hi = __float_as_int(B.w);
            stop = ANY;
          }
          if ((meta & kLastInLeaf) || stop) break;
        }
        ref = kEmptyRef;
        if (hp != p0) {
          sh.o[tid].w = ht;
          sh.d[tid].w = __int_as_float(hp);
          if (ANY)
            sp = 0;
          else
            sh.hit[tid] = make_float4(hu, hv, __int_as_float(hi), 0.0f);
        }
      }
    } else {
      // every pending leaf of the warp, four at a time
      const int rank = __popc(leaves & lt);
      if (mine) sh.leaf[wb + rank] = make_int2(~ref, lane);
      __syncwarp();
      bool occluded = false;
      for (int b = 0; b < total; b += 4) {
        const int g = b + (lane >> 3), k = lane & 7;
        const int2 e = sh.leaf[wb + min(g, total - 1)];
        const float4 *q = S.tri + 3ll * min(e.x + k, S.triCount - 1);
        const float4 A = ldg4(q), B = ldg4(q + 1), C = ldg4(q + 2);
        const int to = wb + e.y;
        const float4 o = sh.o[to], d = sh.d[to];
        const int32_t pid = __float_as_int(A.w), meta = __float_as_int(C.w);
        const unsigned last = __ballot_sync(kFull, (meta & kLastInLeaf) != 0);
        const unsigned before = ((last >> (lane & 24)) & 0xffu) & ((1u << k) - 1u);  // the leaf ended earlier
        float tt, u, v;
        bool hit = coop_intersect<OTHER>(S, o, d, A, B, C, pid, meta & 0xff, o.w, tt, u, v);
        hit = hit & (g < total) & (before == 0) & (pid >= 0) & (tt <= o.w);
        if (ANY) {
          const unsigned occ = __reduce_or_sync(kFull, hit && tt < o.w ? 1u << e.y : 0u);
          occluded = occluded || ((occ >> lane) & 1u);
        } else {
          // one hit per ray and round: a lane whose mark stands compares with the ray's closest
          while (__any_sync(kFull, hit)) {
            if (hit) sh.win[to] = lane;
            __syncwarp();
            if (hit && sh.win[to] == lane) {
              const float ht = sh.o[to].w;
              if (tt < ht || (tt == ht && pid < __float_as_int(sh.d[to].w))) {
                sh.o[to].w = tt;
                sh.d[to].w = __int_as_float(pid);
                sh.hit[to] = make_float4(u, v, B.w, 0.0f);
              }
              hit = false;
            }
            __syncwarp();
          }
        }
        if (mine && rank >= b && rank < b + 4)
          ref = ((last >> ((rank - b) * 8)) & 0xffu) ? kEmptyRef : ref - 8;  // a longer leaf goes on
      }
      if (ANY && occluded) {
        sh.d[tid].w = __int_as_float(0);
        sp = 0;
        ref = kEmptyRef;
      }
      __syncwarp();
    }
    if constexpr (!ANY) {
      if (mine) {
        bound = fminf(sh.o[tid].w * kPruneScale, FLT_MAX);
        // entries that now start beyond the bound
        while (sp > 0 && __int_as_float(stk[sp - 1].t) > bound) --sp;
      }
    }
  }
}

}  // namespace nomad_dev

// Learned residency scorer: MLP 24 -> 128 -> 128 -> 1 (ReLU), BF16 weights and activations,
// FP32 accumulation on the tensor cores, trained on the device with AdamW. Every matrix product
// runs on tcgen05 with tensor-memory accumulators: inference (every residency step) and the
// training forward pass in one fused kernel (both hidden layers and the output dot product, the
// weights staged by one bulk copy), the backward products in two kernels whose operands arrive by
// bulk copies of images that the kernel before laid out for them.
//
// The GEMMs are tiny (2,048 objects x 128 x 128 per frame; a 4,096-row training batch), so the
// kernels are built for latency; the backward products use split-K partial sums reduced in a
// fixed order, and bias gradients are summed row by row, so training is bit-reproducible for a
// given seed.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <numeric>
#include <random>
#include <vector>

#include "bulk_ring.h"
#include "residency_features.cuh"
#include "rt_context.h"

namespace {

constexpr int kIn = NOMAD_FEATURES;  // 24
constexpr int kInPad = 32;
constexpr int kHid = 128;
// offsets in the fp32 parameter blob
constexpr int oW1 = 0;
constexpr int oB1 = oW1 + kHid * kInPad;
constexpr int oW2 = oB1 + kHid;
constexpr int oB2 = oW2 + kHid * kHid;
constexpr int oW3 = oB2 + kHid;
constexpr int oB3 = oW3 + kHid;
constexpr int oMean = oB3 + 1;
constexpr int oIstd = oMean + kIn;
constexpr int kParams = oIstd + kIn;
static_assert(kParams == NOMAD_MLP_PARAMS, "parameter blob layout");

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);  // a -> low half
  return *reinterpret_cast<uint32_t *>(&h);
}

// ---- inference on the 5th-generation tensor cores (tcgen05) ---------------------------------
// One CTA of 128 threads scores 128 rows. Both layers run as tcgen05.mma (kind::f16, BF16 inputs,
// FP32 accumulators in tensor memory, M = 128, N = 128, K = 16 per instruction) issued by one
// thread, with the operands in shared memory in the canonical K-major layout without swizzle:
// 8 x 8 core matrices of 128 contiguous bytes, row groups 128 B apart (stride byte offset) and
// 8-element K chunks (rows / 8) * 128 B apart (leading byte offset). Each thread then owns one
// accumulator row (its tensor-memory lane) for the bias / ReLU epilogue and the final dot product.
constexpr int kTcRows = 128;
constexpr uint32_t kTcCols = 256;                   // tensor-memory columns: D1 [0,128), D2 [128,256)
constexpr uint32_t kTcX = 0;                        // X tile, 128 x 32 bf16
constexpr uint32_t kTcW1 = kTcX + 128 * kInPad * 2; // W1, 128 x 32, then W2 right after it:
constexpr uint32_t kTcW2 = kTcW1 + 128 * kInPad * 2; // both arrive pre-packed in one bulk copy
constexpr uint32_t kTcWBytes = 128 * kInPad * 2 + 128 * kHid * 2;  // 40 KB
constexpr uint32_t kTcH1 = kTcW2 + 128 * kHid * 2;
constexpr uint32_t kTcF = kTcH1 + 128 * kHid * 2;   // fp32: b1, b2, w3, b3, mean, istd
constexpr uint32_t kTcBar = kTcF + 4 * (3 * kHid + 1 + 2 * kIn + 7);  // copy barrier, MMA barrier, TMEM slot
constexpr size_t kTcSmem = kTcBar + 24;
constexpr uint32_t kTcIdx = kTcBar + 24;            // training: the tile's sample indices
constexpr size_t kTcSmemTrain = kTcIdx + 4 * kTcRows;
constexpr uint32_t kStatusWaitExpired = 1u << 1;
constexpr long long kTcWaitPolls = 1ll << 22;

// Byte offset of element (r, k) of a 128-row K-major operand in the canonical layout.
__device__ __forceinline__ uint32_t canon_off(int r, int k) {
  return (uint32_t)((((k >> 3) * 16 + (r >> 3)) << 7) + ((r & 7) << 4) + ((k & 7) << 1));
}

// Shared-memory matrix descriptor: start, leading byte offset (next K chunk: 16 row groups of
// 128 B), stride byte offset (next row group: 128 B), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t canon_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)(2048u >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) |
         (1ull << 46);
}

// kind::f16 instruction descriptor: FP32 accumulator, BF16 A and B, both K-major, N = 128, M = 128.
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void tc_mma(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(kTcIdesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity) {
  for (long long i = 0; i < kTcWaitPolls; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// 32 consecutive accumulator columns of this thread's lane.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// Wc holds W1 and W2 (bf16) already in the canonical shared-memory layout (k_refresh_bf16 packs
// them whenever the weights change), so one bulk asynchronous copy stages both.
// FEAT: the rows are the residency step's objects; each thread computes its object's features
// (nomad_res::object_features, the same code as the feature kernel) instead of reading X.
// TRAIN: the rows are a batch, row r the sample perm[(cursor + r) % n] (or r itself without perm);
// besides the outputs' errors the kernel stores what the backward pass needs, per 128-row tile:
//   ximg, h1img, z2img  X, H1 and dZ2 as operand images (canon_off). One image serves both as a
//          K-major operand (rows against columns: dH1) and, rows being the K of the weight
//          gradients, as an MN-major one (dW1, dW2), so nothing is transposed.
//   g2c, g3c  dZ2 and ReLU(Z2) dy column by column (fp32, col_off), whose row-ordered sums are db2
//          and dw3; mask: Z1 > 0, 128 bits a row.
struct TrainBufs {
  unsigned char *ximg, *h1img, *z2img, *z1img;
  float *g1c, *g2c, *g3c, *dy, *se;
  uint32_t *mask;
  float *part1, *part2;
};
struct TrainRows {
  const float *T;
  const uint32_t *perm;
  uint64_t cursor, n;
};
constexpr uint32_t kTileBytes = 128 * kHid * 2;    // a 128-row tile of 128 columns
constexpr uint32_t kXTileBytes = 128 * kInPad * 2;  // and of X

// Float offset of (column c, row r) in the fp32 columns: tiles of 128 rows, a column's 128 rows
// together, their 16-byte groups permuted by the column so that 32 lanes reading the same group of
// 32 columns meet different banks.
__device__ __forceinline__ size_t col_off(int c, int r) {
  return (size_t)(r >> 7) * (128 * kHid) + c * 128 + (((((r & 127) >> 2) ^ (c & 31)) << 2) | (r & 3));
}

__device__ __forceinline__ void bulk_store(void *dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}

template <bool FEAT, bool TRAIN>
__global__ void __launch_bounds__(128) k_mlp_forward_tc(const float *__restrict__ X, uint64_t n,
                                                        const float *__restrict__ P,
                                                        const unsigned char *__restrict__ Wc, float *__restrict__ y,
                                                        uint32_t *__restrict__ status, nomad_res::FeatArgs fa,
                                                        TrainRows rows, TrainBufs tb) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  float *sB1 = reinterpret_cast<float *>(smem + kTcF);
  float *sB2 = sB1 + kHid;
  float *sW3 = sB2 + kHid;
  float *sB3 = sW3 + kHid;
  float *sMean = sB3 + 1;
  float *sIstd = sMean + kIn;
  const uint32_t barCopy = sbase + kTcBar, bar = sbase + kTcBar + 8;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + kTcBar + 16);
  const int tid = threadIdx.x, warp = tid >> 5;

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barCopy) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // weights: one bulk copy (no multicast) of the pre-packed W1 | W2 block
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barCopy), "r"(kTcWBytes) : "memory");
    for (uint32_t off = 0; off < kTcWBytes; off += 16384u) {
      const uint32_t sz = min(16384u, kTcWBytes - off);
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              sbase + kTcW1 + off),
          "l"(Wc + off), "r"(sz), "r"(barCopy)
          : "memory");
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kTcBar + 16),
                 "r"(kTcCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // the standardised X tile and the fp32 vectors while the weights are in flight
  for (int i = tid; i < kHid; i += 128) {
    sB1[i] = P[oB1 + i];
    sB2[i] = P[oB2 + i];
    sW3[i] = P[oW3 + i];
  }
  if (tid == 0) sB3[0] = P[oB3];
  if (tid < kIn) {
    sMean[tid] = P[oMean + tid];
    sIstd[tid] = P[oIstd + tid];
  }
  __syncthreads();
  const uint64_t row0 = (uint64_t)blockIdx.x * kTcRows;
  uint32_t *sIdx = reinterpret_cast<uint32_t *>(smem + kTcIdx);  // TRAIN: the tile's samples
  float target = 0.0f;
  if constexpr (TRAIN) {
    uint32_t s = 0;
    if (row0 + tid < n) {
      s = rows.perm ? rows.perm[(rows.cursor + row0 + tid) % rows.n] : (uint32_t)(row0 + tid);
      target = rows.T[s];
    }
    sIdx[tid] = s;
    __syncthreads();
  }
  if constexpr (FEAT) {
    float f[NOMAD_FEATURES];
    const bool live = row0 + tid < n;
    if (live) nomad_res::object_features(fa, (uint32_t)(row0 + tid), f);
#pragma unroll
    for (int k = 0; k < kInPad; ++k) {
      const float v = (live && k < kIn) ? (f[k < kIn ? k : 0] - sMean[k < kIn ? k : 0]) * sIstd[k < kIn ? k : 0] : 0.0f;
      *reinterpret_cast<__nv_bfloat16 *>(smem + kTcX + canon_off(tid, k)) = __float2bfloat16_rn(v);
    }
  } else {
#pragma unroll
    for (int i0 = 0; i0 < kTcRows * kInPad; i0 += 128) {  // all of a thread's loads in flight at once
      const int i = i0 + tid;
      const int r = i / kInPad, f = i % kInPad;
      float v = 0.0f;
      if (f < kIn && row0 + r < n) v = (X[(TRAIN ? (uint64_t)sIdx[r] : row0 + r) * kIn + f] - sMean[f]) * sIstd[f];
      const __nv_bfloat16 b = __float2bfloat16_rn(v);
      *reinterpret_cast<__nv_bfloat16 *>(smem + kTcX + canon_off(r, f)) = b;
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
  bool ok = tc_wait(barCopy, 0);  // weights landed

  // layer 1: D1 = X . W1^T, K = 32 in two steps
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < kInPad / 16; ++s)
      tc_mma(tmem, canon_desc(sbase + kTcX + s * 2 * 2048), canon_desc(sbase + kTcW1 + s * 2 * 2048), s > 0);
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
  }
  ok = tc_wait(bar, 0) && ok;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // epilogue 1: bias, ReLU, BF16 into the layer-2 operand (row = this thread's lane)
  const int r = tid;
  const bool rowLive = row0 + r < n;
  // The 32-column steps of the epilogues stay loops: unrolled, each instruction runs once per
  // block, and fetching 100 KB of code took longer (45 us a training launch) than the work.
#pragma unroll 1
  for (int c0 = 0; c0 < kHid; c0 += 32) {
    float v[32];
    tc_ld32(lane_base + c0, v);
    uint32_t mask = 0u;
    uint32_t h[16];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float za = v[j] + sB1[c0 + j], zb = v[j + 1] + sB1[c0 + j + 1];
      h[j / 2] = pack_bf16(fmaxf(za, 0.0f), fmaxf(zb, 0.0f));
      if (TRAIN) mask |= (za > 0.0f ? 1u << j : 0u) | (zb > 0.0f ? 2u << j : 0u);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4 *>(smem + kTcH1 + canon_off(r, c0 + 8 * q)) =
          make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
    if (TRAIN && rowLive) tb.mask[(row0 + r) * 4 + c0 / 32] = mask;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // layer 2: D2 = H1 . W2^T, K = 128 in eight steps
  if (TRAIN && tid == 0) {  // the operand images of X and H1 go out while it runs
    bulk_store(tb.ximg + (uint64_t)blockIdx.x * kXTileBytes, sbase + kTcX, kXTileBytes);
    bulk_store(tb.h1img + (uint64_t)blockIdx.x * kTileBytes, sbase + kTcH1, kTileBytes);
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < kHid / 16; ++s)
      tc_mma(tmem + 128, canon_desc(sbase + kTcH1 + s * 2 * 2048), canon_desc(sbase + kTcW2 + s * 2 * 2048), s > 0);
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
  }
  ok = tc_wait(bar, 1) && ok;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // epilogue 2: ReLU(D2 + b2) . w3 + b3 for this thread's row
  float acc = 0.0f;
#pragma unroll 1
  for (int c0 = 0; c0 < kHid; c0 += 32) {
    float v[32];
    tc_ld32(lane_base + 128 + c0, v);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float z = v[j] + sB2[c0 + j];
      acc += fmaxf(z, 0.0f) * sW3[c0 + j];
    }
  }
  if constexpr (TRAIN) {
    // the error of this row, its output gradient 2 (y - t) / n, and dZ2 = dy w3 (Z2 > 0)
    const float d = (ok ? acc + sB3[0] : 0.0f) - target;
    const float dy = 2.0f * d / (float)(int)n;
    if (rowLive) {
      tb.dy[row0 + r] = dy;
      tb.se[row0 + r] = d * d;
    }
    unsigned char *img = tb.z2img + (uint64_t)blockIdx.x * kTileBytes;
#pragma unroll 1
    for (int c0 = 0; c0 < kHid; c0 += 32) {
      float v[32];
      tc_ld32(lane_base + 128 + c0, v);
      uint32_t h[16];
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float za = v[j] + sB2[c0 + j], zb = v[j + 1] + sB2[c0 + j + 1];
        const float ga = za > 0.0f ? dy * sW3[c0 + j] : 0.0f, gb = zb > 0.0f ? dy * sW3[c0 + j + 1] : 0.0f;
        const size_t oa = col_off(c0 + j, (int)row0 + r), ob = col_off(c0 + j + 1, (int)row0 + r);
        tb.g2c[oa] = ga;
        tb.g2c[ob] = gb;
        tb.g3c[oa] = (za > 0.0f ? za : 0.0f) * dy;
        tb.g3c[ob] = (zb > 0.0f ? zb : 0.0f) * dy;
        h[j / 2] = rowLive ? pack_bf16(ga, gb) : 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4 *>(img + canon_off(r, c0 + 8 * q)) =
            make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
    }
    if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  } else {
    if (row0 + r < n) y[row0 + r] = ok ? acc + sB3[0] : 0.0f;
  }
  if (!ok && tid == 0) atomicOr(status, kStatusWaitExpired);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols) : "memory");
  }
}

// ---- backward pass on the 5th-generation tensor cores (tcgen05) -----------------------------
// Descriptor of an operand image read with its rows as K (MN-major): 8 x 8 core matrices, the next
// eight rows 128 B on (leading offset), the next eight columns 2,048 B on (stride offset).
__device__ __forceinline__ uint64_t rows_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(2048u >> 4) << 32) |
         (1ull << 46);
}

// D[128][NT] += A B with both operands MN-major.
template <int NT>
__device__ __forceinline__ void tc_mma_rows(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(NT >> 3) << 17) |
                             ((128u >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void bar_init(uint32_t bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One bulk copy (no multicast) of this GPU's own memory.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
      "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Tensor memory of the block (cols columns) and its barriers, before and after the products.
__device__ __forceinline__ uint32_t tc_begin(uint32_t slot, const uint32_t *slotPtr, uint32_t bar0, int bars, uint32_t cols) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < bars; ++i) bar_init(bar0 + 8 * i);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return *slotPtr;
}
__device__ __forceinline__ void tc_end(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
  }
}

// One split of a weight gradient: D[128][NT] = sum of A^T B over the 64-row blocks [b0, b0 + nb) of two
// images (A 128 columns, B NT columns), 16 rows an instruction. One thread runs a ring of kRing
// tiles of bulk copies ahead of the MMAs; the others wait for the last commit. The partial goes
// out row-major.
constexpr int kRing = 3;
template <int NT>
__device__ __forceinline__ void split_product(unsigned char *smem, const unsigned char *A, const unsigned char *B, int b0,
                                              int nb, float *__restrict__ out, uint32_t *__restrict__ status) {
  constexpr uint32_t bBytes = NT * 128 * 2, stage = kTileBytes + bBytes;
  const int tid = threadIdx.x;
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const uint32_t bars = base + kRing * stage;  // full[kRing], free[kRing], done
  const uint32_t fin = bars + 16 * kRing;
  uint32_t *slot = reinterpret_cast<uint32_t *>(smem + kRing * stage + 16 * kRing + 8);
  const uint32_t tmem = tc_begin(fin + 8, slot, bars, 2 * kRing + 1, NT);
  if (tid == 0) {
    const int t0 = b0 / 2, nt = (b0 + nb - 1) / 2 - t0 + 1;
    auto load = [&](int i) {
      const uint32_t s = base + (i % kRing) * stage, bar = bars + 8 * (i % kRing);
      bar_expect(bar, stage);
      bulk_load(s, A + (size_t)(t0 + i) * kTileBytes, kTileBytes, bar);
      bulk_load(s + kTileBytes, B + (size_t)(t0 + i) * bBytes, bBytes, bar);
    };
    int loaded = 0;
    for (; loaded < kRing && loaded < nt; ++loaded) load(loaded);
    bool ok = true, first = true;
    for (int i = 0; i < nt && ok; ++i) {
      const uint32_t s = base + (i % kRing) * stage;
      ok = tc_wait(bars + 8 * (i % kRing), (i / kRing) & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // the split may begin or end in the middle of a tile
      const int k0 = max(0, (b0 - 2 * (t0 + i)) * 4), k1 = min(8, (b0 + nb - 2 * (t0 + i)) * 4);
      for (int k = k0; k < k1; ++k) {
        tc_mma_rows<NT>(tmem, rows_desc(s + k * 256), rows_desc(s + kTileBytes + k * 256), first ? 0u : 1u);
        first = false;
      }
      if (loaded < nt) {  // refill this stage once its products are done
        tc_commit(bars + 8 * (kRing + i % kRing));
        ok = tc_wait(bars + 8 * (kRing + i % kRing), (i / kRing) & 1) && ok;
        if (ok) load(loaded++);
      }
    }
    // a wait that ran out: let the copies in flight land before the block ends
    if (!ok)
      for (int i = max(0, loaded - kRing); i < loaded; ++i) tc_wait(bars + 8 * (i % kRing), (i / kRing) & 1);
    tc_commit(fin);
    if (!ok) atomicOr(status, kStatusWaitExpired);
  }
  const bool ok = __syncthreads_and(tc_wait(fin, 0) ? 1 : 0) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok && tid == 0) atomicOr(status, kStatusWaitExpired);
  const uint32_t lane_base = tmem + ((uint32_t)((tid >> 5) * 32) << 16);
  float4 *row = reinterpret_cast<float4 *>(out + (size_t)tid * NT);
#pragma unroll 1
  for (int c0 = 0; c0 < NT; c0 += 32) {
    float v[32];
    tc_ld32(lane_base + c0, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) row[c0 / 4 + j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  }
  tc_end(tmem, NT);
}
constexpr size_t split_smem(int nt) { return kRing * (kTileBytes + (size_t)nt * 256) + 16 * kRing + 16; }

// The hidden layers' backward products. Blocks [0, tiles): dH1 = dZ2 W2 of one 128-row tile and
// dZ1 = dH1 (Z1 > 0), stored as a bf16 operand image and as fp32 columns. Blocks from tiles on: one
// split of dW2 = dZ2^T H1.
__global__ void __launch_bounds__(128) k_train_hidden(int n, int tiles, int blocksPerSplit,
                                                      const unsigned char *__restrict__ W2t, TrainBufs tb,
                                                      uint32_t *__restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x;
  if ((int)blockIdx.x >= tiles) {
    const int z = blockIdx.x - tiles, b0 = z * blocksPerSplit;
    split_product<kHid>(smem, tb.z2img, tb.h1img, b0, min(blocksPerSplit, n / 64 - b0),
                        tb.part2 + (size_t)z * kHid * kHid, status);
    return;
  }
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const uint32_t bar = base + 2 * kTileBytes, fin = bar + 8;
  const uint32_t tmem = tc_begin(fin + 8, reinterpret_cast<uint32_t *>(smem + 2 * kTileBytes + 16), bar, 2, kHid);
  if (tid == 0) {
    bar_expect(bar, 2 * kTileBytes);
    bulk_load(base, tb.z2img + (size_t)blockIdx.x * kTileBytes, kTileBytes, bar);
    bulk_load(base + kTileBytes, W2t, kTileBytes, bar);
  }
  bool ok = tc_wait(bar, 0);
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < kHid / 16; ++s)
      tc_mma(tmem, canon_desc(base + s * 2 * 2048), canon_desc(base + kTileBytes + s * 2 * 2048), s > 0);
    tc_commit(fin);
  }
  ok = tc_wait(fin, 0) && ok;
  if (!ok) {
    tc_wait(bar, 0);
    atomicOr(status, kStatusWaitExpired);
  }
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t lane_base = tmem + ((uint32_t)((tid >> 5) * 32) << 16);
  const int r = blockIdx.x * kTcRows + tid;
  const bool live = r < n;
  unsigned char *img = tb.z1img + (size_t)blockIdx.x * kTileBytes;
#pragma unroll 1
  for (int c0 = 0; c0 < kHid; c0 += 32) {
    float v[32];
    tc_ld32(lane_base + c0, v);
    const uint32_t mask = live ? tb.mask[(size_t)r * 4 + c0 / 32] : 0u;
    uint32_t h[16];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float ga = (mask >> j) & 1u ? v[j] : 0.0f, gb = (mask >> (j + 1)) & 1u ? v[j + 1] : 0.0f;
      h[j / 2] = pack_bf16(ga, gb);
      tb.g1c[col_off(c0 + j, r)] = ga;
      tb.g1c[col_off(c0 + j + 1, r)] = gb;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4 *>(img + canon_off(tid, c0 + 8 * q)) =
          make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
  }
  tc_end(tmem, kHid);
}
constexpr size_t kHiddenSmem = std::max<size_t>(split_smem(kHid), 2 * kTileBytes + 32);

// Row-ordered column sums: out[c] = sum over rows r, in order, of col[c][r], 32 columns (from c0, laid
// out by col_off) a block and a lane a column, or of one plain column (PLAIN). The chain of
// dependent additions sets the time (4 cycles a row: 8.7 us for 4,096 rows at 1.9 GHz), so one warp
// does nothing but wait, load four rows at a time from shared memory and add, while another
// thread keeps a ring of bulk copies (128 rows each) ahead of it.
constexpr int kSumRing = 8;
constexpr uint32_t kSumStage = 32 * 128 * 4;
template <bool PLAIN>
__device__ __forceinline__ void ordered_sums(unsigned char *smem, int n, int c0, const float *__restrict__ col,
                                             float *__restrict__ out, uint32_t *__restrict__ status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem)), bars = base + kSumRing * kSumStage;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * kSumRing; ++i) bar_init(bars + 8 * i);  // full, free
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  const int tiles = (n + 127) / 128;
  bool ok = true;
  using Ring = BulkRing<kSumRing>;
  if (warp == 1 && lane == 0) {
    int issued = 0;
    for (; issued < tiles; ++issued) {
      const int t = issued, s = Ring::stage(t);
      if (t >= kSumRing && !tc_wait(bars + 8 * (kSumRing + s), Ring::parity(t - kSumRing))) {
        ok = false;
        break;
      }
      const uint32_t bytes = PLAIN ? min(128, n - t * 128) * 4 : kSumStage;
      bar_expect(bars + 8 * s, bytes);
      bulk_load(base + s * kSumStage, col + (PLAIN ? (size_t)t * 128 : (size_t)t * (128 * kHid) + c0 * 128), bytes,
                bars + 8 * s);
    }
    // every copy has landed before the block ends, also when a wait of either warp ran out
    for (int t = Ring::first_open(issued); t < issued; ++t) ok = tc_wait(bars + 8 * Ring::stage(t), Ring::parity(t)) && ok;
  } else if (warp == 0) {
    // chunks of 32 rows, the next one loading while one is added
    float sum = 0.0f;
    const int chunks = n / 32, x = PLAIN ? 0 : lane;  // n is a multiple of 64: an even number
    float4 p[8], q[8];
    auto at = [&](int i) {
      return reinterpret_cast<const float4 *>(smem + (size_t)((i >> 2) % kSumRing) * kSumStage) + (PLAIN ? 0 : lane * 32);
    };
    // one load between every four additions: the loads fill the chain's idle issue slots
    auto step = [&](const float4 (&v)[8], float4 (&w)[8], const float4 *src, int g) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        w[k] = src[(g + k) ^ x];
        sum += v[k].x;
        sum += v[k].y;
        sum += v[k].z;
        sum += v[k].w;
      }
    };
    ok = __all_sync(0xffffffffu, tc_wait(bars, 0));
#pragma unroll
    for (int k = 0; k < 8; ++k) p[k] = at(0)[k ^ x];
#pragma unroll 1
    for (int i = 0; i < chunks && ok; i += 2) {
      step(p, q, at(i), ((i + 1) & 3) * 8);
      int next = i + 2;
      if (next < chunks) {
        if ((next & 3) == 0) {  // the tile is in registers: free it, wait for the next
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bars + 8 * (kSumRing + (i >> 2) % kSumRing))
                         : "memory");
          const int t = next >> 2;
          ok = __all_sync(0xffffffffu, tc_wait(bars + 8 * Ring::stage(t), Ring::parity(t)));
        }
      } else {
        next = i;  // nothing follows: what is loaded is not used
      }
      step(q, p, at(next), (next & 3) * 8);
    }
    if (!PLAIN || lane == 0) out[lane] = sum;
  }
  if (!ok && lane == 0) atomicOr(status, kStatusWaitExpired);
  __syncthreads();
}

// The input layer's weight gradient and the vectors' gradients. Blocks [0, splits): one split of
// dW1 = dZ1^T X. Then four blocks of 32 columns each for db1 = sum dZ1, db2 = sum dZ2 and
// dw3 = sum ReLU(Z2) dy, and one for db3 = sum dy.
__global__ void __launch_bounds__(128) k_train_input(int n, int splits, int blocksPerSplit, float *__restrict__ G,
                                                     TrainBufs tb, uint32_t *__restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if ((int)blockIdx.x < splits) {
    const int z = blockIdx.x, b0 = z * blocksPerSplit;
    split_product<kInPad>(smem, tb.z1img, tb.ximg, b0, min(blocksPerSplit, n / 64 - b0),
                          tb.part1 + (size_t)z * kHid * kInPad, status);
    return;
  }
  const int q = blockIdx.x - splits, c0 = (q & 3) * 32;
  if (q < 12) {
    const float *col = q < 4 ? tb.g1c : q < 8 ? tb.g2c : tb.g3c;
    ordered_sums<false>(smem, n, c0, col, G + (q < 4 ? oB1 : q < 8 ? oB2 : oW3) + c0, status);
  } else {
    ordered_sums<true>(smem, n, 0, tb.dy, G + oB3, status);
  }
}
constexpr size_t kInputSmem = std::max<size_t>(split_smem(kInPad), kSumRing * kSumStage + 16 * kSumRing);

// The bf16 weights of the tensor-core kernels: W1 then W2 in the canonical operand layout (one
// block), and W2 transposed for dH1. W1's padded input columns stay zero.
__device__ __forceinline__ void store_weight(int i, float p, unsigned char *__restrict__ Wc, unsigned char *__restrict__ W2t) {
  if (i < oB1) {
    const int c = i % kInPad;
    *reinterpret_cast<__nv_bfloat16 *>(Wc + canon_off(i / kInPad, c)) = __float2bfloat16_rn(c < kIn ? p : 0.0f);
  } else if (i >= oW2 && i < oB2) {
    const int r = (i - oW2) / kHid, c = (i - oW2) % kHid;
    const __nv_bfloat16 w = __float2bfloat16_rn(p);
    *reinterpret_cast<__nv_bfloat16 *>(Wc + (kTcW2 - kTcW1) + canon_off(r, c)) = w;
    *reinterpret_cast<__nv_bfloat16 *>(W2t + canon_off(c, r)) = w;
  }
}

// Completes the gradient (split-K partials summed in split order) and, with update, takes the AdamW
// step over the trainable part of the blob (everything before the feature statistics) and
// refreshes the bf16 weights. Without update the gradient goes to G.
__global__ void __launch_bounds__(128) k_adamw(float *__restrict__ P, float *__restrict__ G, float *__restrict__ m,
                                               float *__restrict__ v, int splits, TrainBufs tb, bool update, float lr,
                                               float b1, float b2, float eps, float wd, float bc1, float bc2,
                                               unsigned char *__restrict__ Wc, unsigned char *__restrict__ W2t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= oMean) return;
  const bool w1 = i < oB1, w2 = i >= oW2 && i < oB2;
  float g;
  if (w1 || w2) {
    const size_t count = w1 ? kHid * kInPad : kHid * kHid;
    const float *part = w1 ? tb.part1 + i : tb.part2 + (i - oW2);
    g = 0.0f;
#pragma unroll 8
    for (int z = 0; z < splits; ++z) g += part[(size_t)z * count];
  } else {
    g = G[i];
  }
  if (!update) {
    G[i] = g;
    return;
  }
  const float mi = b1 * m[i] + (1.0f - b1) * g;
  const float vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float mh = mi / bc1, vh = vi / bc2;
  float p = P[i];
  if (w1 || w2 || (i >= oW3 && i < oB3)) p = p - lr * wd * p;
  p = p - lr * mh / (sqrtf(vh) + eps);
  P[i] = p;
  store_weight(i, p, Wc, W2t);
}

__global__ void k_refresh_bf16(const float *__restrict__ P, unsigned char *__restrict__ Wc,
                               unsigned char *__restrict__ W2t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < oMean) store_weight(i, P[i], Wc, W2t);
}

// Mean squared error of each step's batch, the rows added in order in double.
__global__ void __launch_bounds__(128) k_loss(const float *__restrict__ se, int n, float *__restrict__ loss) {
  __shared__ float tile[2048];
  const float *row = se + (size_t)blockIdx.x * n;
  double acc = 0.0;
  for (int r0 = 0; r0 < n; r0 += 2048) {
    const int m = min(2048, n - r0);
    for (int i = threadIdx.x; i < m; i += 128) tile[i] = row[r0 + i];
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 0; i < m; ++i) acc += tile[i];
    __syncthreads();
  }
  if (threadIdx.x == 0) loss[blockIdx.x] = (float)(acc / n);
}

}  // namespace

// ---- host side ------------------------------------------------------------------------------

struct MlpState {
  bool ready = false;
  bool smemSet = false;  // the kernels opted in to their shared memory on this context's device
  DeviceBuf P, Wc, W2t, M, V, G;
  DeviceBuf X, T, perm[2], ximg, h1img, z2img, z1img, g1c, g2c, g3c, dy, se, mask, part1, part2, loss;
  DeviceBuf inX, inY;
};

namespace {
MlpState &mlp(nomad_ctx *ctx) {
  static_assert(sizeof(MlpState) > 0, "");
  if (!ctx->mlp) ctx->mlp = new MlpState();
  return *static_cast<MlpState *>(ctx->mlp);
}

nomad_status refresh(nomad_ctx *ctx, MlpState &S) {
  k_refresh_bf16<<<(oMean + 255) / 256, 256, 0, ctx->stream>>>(S.P.as<const float>(), S.Wc.as<unsigned char>(),
                                                               S.W2t.as<unsigned char>());
  NOMAD_CUDA(ctx, cudaGetLastError());
  return NOMAD_OK;
}

nomad_status ensure(nomad_ctx *ctx, MlpState &S) {
  NOMAD_CUDA(ctx, S.P.reserve(kParams * 4));
  NOMAD_CUDA(ctx, S.W2t.reserve(kTileBytes));
  NOMAD_CUDA(ctx, S.Wc.reserve(kTcWBytes));
  NOMAD_CUDA(ctx, S.M.reserve(kParams * 4));
  NOMAD_CUDA(ctx, S.V.reserve(kParams * 4));
  NOMAD_CUDA(ctx, S.G.reserve(kParams * 4));
  if (!S.smemSet) {
    NOMAD_CUDA(ctx, cudaFuncSetAttribute(k_mlp_forward_tc<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kTcSmem));
    NOMAD_CUDA(ctx, cudaFuncSetAttribute(k_mlp_forward_tc<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kTcSmem));
    NOMAD_CUDA(ctx, cudaFuncSetAttribute(k_mlp_forward_tc<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kTcSmemTrain));
    NOMAD_CUDA(ctx, cudaFuncSetAttribute(k_train_hidden, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHiddenSmem));
    NOMAD_CUDA(ctx, cudaFuncSetAttribute(k_train_input, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInputSmem));
    S.smemSet = true;
  }
  return NOMAD_OK;
}
}  // namespace

void nomad_mlp_free(void *p) { delete static_cast<MlpState *>(p); }

// Inference on device features (n x 24 fp32) into y (n fp32), on the context stream.
nomad_status nomad_mlp_infer_device(nomad_ctx *ctx, const float *X, uint64_t n, float *y) {
  MlpState &S = mlp(ctx);
  if (!S.ready) return nomad_fail(ctx, NOMAD_ERR_NOT_READY, "MLP not initialised or trained");
  if (n == 0) return NOMAD_OK;
  const unsigned blocks = (unsigned)((n + kTcRows - 1) / kTcRows);
  k_mlp_forward_tc<false, false><<<blocks, 128, kTcSmem, ctx->stream>>>(X, n, S.P.as<const float>(),
                                                                        S.Wc.as<const unsigned char>(), y,
                                                                        ctx->status.as<uint32_t>(),
                                                                        nomad_res::FeatArgs{}, TrainRows{}, TrainBufs{});
  NOMAD_CUDA(ctx, cudaGetLastError());
  return NOMAD_OK;
}

nomad_status nomad_mlp_score_objects(nomad_ctx *ctx, const nomad_res::FeatArgs *fa, float *keys) {
  MlpState &S = mlp(ctx);
  if (!S.ready) return nomad_fail(ctx, NOMAD_ERR_NOT_READY, "MLP not initialised or trained");
  if (fa->n == 0) return NOMAD_OK;
  const unsigned blocks = (fa->n + kTcRows - 1) / kTcRows;
  k_mlp_forward_tc<true, false><<<blocks, 128, kTcSmem, ctx->stream>>>(nullptr, fa->n, S.P.as<const float>(),
                                                                       S.Wc.as<const unsigned char>(), keys,
                                                                       ctx->status.as<uint32_t>(), *fa, TrainRows{}, TrainBufs{});
  NOMAD_CUDA(ctx, cudaGetLastError());
  return NOMAD_OK;
}

extern "C" nomad_status nomad_mlp_init(nomad_ctx *ctx, uint64_t seed) {
  if (!ctx) return NOMAD_ERR_INVALID_ARGUMENT;
  NOMAD_DEVICE_SCOPE(ctx);
  MlpState &S = mlp(ctx);
  nomad_status st = ensure(ctx, S);
  if (st != NOMAD_OK) return st;
  std::vector<float> p(kParams, 0.0f);
  std::mt19937_64 rng(seed);
  auto uni = [&](float lim) { return (float)(((rng() >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0) * lim; };
  float l1 = std::sqrt(6.0f / kIn), l2 = std::sqrt(6.0f / kHid), l3 = std::sqrt(3.0f / kHid);
  for (int o = 0; o < kHid; ++o)
    for (int i = 0; i < kIn; ++i) p[oW1 + o * kInPad + i] = uni(l1);
  for (int i = 0; i < kHid * kHid; ++i) p[oW2 + i] = uni(l2);
  for (int i = 0; i < kHid; ++i) p[oW3 + i] = uni(l3);
  for (int i = 0; i < kIn; ++i) p[oIstd + i] = 1.0f;
  NOMAD_CUDA(ctx, cudaMemcpy(S.P.p, p.data(), kParams * 4, cudaMemcpyHostToDevice));
  NOMAD_CUDA(ctx, cudaMemset(S.M.p, 0, kParams * 4));
  NOMAD_CUDA(ctx, cudaMemset(S.V.p, 0, kParams * 4));
  st = refresh(ctx, S);
  if (st != NOMAD_OK) return st;
  S.ready = true;
  NOMAD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return NOMAD_OK;
}

extern "C" nomad_status nomad_mlp_get(nomad_ctx *ctx, float *out) {
  if (!ctx || !out) return NOMAD_ERR_INVALID_ARGUMENT;
  MlpState &S = mlp(ctx);
  if (!S.ready) return nomad_fail(ctx, NOMAD_ERR_NOT_READY, "MLP not initialised");
  NOMAD_CUDA(ctx, cudaMemcpyAsync(out, S.P.p, kParams * 4, cudaMemcpyDeviceToHost, ctx->stream));
  NOMAD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return NOMAD_OK;
}

bool nomad_mlp_ready(nomad_ctx *ctx) { return ctx->mlp && static_cast<MlpState *>(ctx->mlp)->ready; }

extern "C" nomad_status nomad_mlp_set(nomad_ctx *ctx, const float *in) {
  if (!ctx || !in) return NOMAD_ERR_INVALID_ARGUMENT;
  NOMAD_DEVICE_SCOPE(ctx);
  MlpState &S = mlp(ctx);
  for (int i = 0; i < kParams; ++i)
    if (!std::isfinite(in[i])) {
      S.ready = false;
      return nomad_fail(ctx, NOMAD_ERR_INVALID_ARGUMENT,
                        "model parameter " + std::to_string(i) +
                            " is not finite; learned steps fall back to the ray-hit budget");
    }
  nomad_status st = ensure(ctx, S);
  if (st != NOMAD_OK) return st;
  NOMAD_CUDA(ctx, cudaMemcpy(S.P.p, in, kParams * 4, cudaMemcpyHostToDevice));
  NOMAD_CUDA(ctx, cudaMemset(S.M.p, 0, kParams * 4));
  NOMAD_CUDA(ctx, cudaMemset(S.V.p, 0, kParams * 4));
  st = refresh(ctx, S);
  if (st != NOMAD_OK) return st;
  S.ready = true;
  NOMAD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return NOMAD_OK;
}

namespace {
constexpr uint32_t kModelVersion = 1;
constexpr size_t kModelHeader = 16;  // magic, version, parameter count, feature count

uint64_t fnv1a(const unsigned char *p, size_t n) {
  uint64_t h = 1469598103934665603ull;
  for (size_t i = 0; i < n; ++i) {
    h ^= p[i];
    h *= 1099511628211ull;
  }
  return h;
}

void put_u32(unsigned char *p, uint32_t v) {
  for (int k = 0; k < 4; ++k) p[k] = static_cast<unsigned char>(v >> (8 * k));
}

uint32_t get_u32(const unsigned char *p) {
  return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
}
}  // namespace

extern "C" nomad_status nomad_mlp_save(nomad_ctx *ctx, const char *path) {
  if (!ctx || !path) return NOMAD_ERR_INVALID_ARGUMENT;
  std::vector<float> p(kParams);
  nomad_status st = nomad_mlp_get(ctx, p.data());
  if (st != NOMAD_OK) return st;
  std::vector<unsigned char> buf(kModelHeader + (size_t)kParams * 4 + 8);
  std::memcpy(buf.data(), "NMLP", 4);
  put_u32(buf.data() + 4, kModelVersion);
  put_u32(buf.data() + 8, (uint32_t)kParams);
  put_u32(buf.data() + 12, (uint32_t)kIn);
  for (int i = 0; i < kParams; ++i) {
    uint32_t bits;
    std::memcpy(&bits, &p[i], 4);
    put_u32(buf.data() + kModelHeader + 4 * (size_t)i, bits);
  }
  const size_t body = kModelHeader + (size_t)kParams * 4;
  const uint64_t h = fnv1a(buf.data(), body);
  put_u32(buf.data() + body, (uint32_t)h);
  put_u32(buf.data() + body + 4, (uint32_t)(h >> 32));
  FILE *f = std::fopen(path, "wb");
  if (!f) return nomad_fail(ctx, NOMAD_ERR_INVALID_ARGUMENT, std::string("cannot write ") + path);
  const bool ok = std::fwrite(buf.data(), 1, buf.size(), f) == buf.size();
  const bool closed = std::fclose(f) == 0;
  if (!ok || !closed) return nomad_fail(ctx, NOMAD_ERR_INVALID_ARGUMENT, std::string("cannot write ") + path);
  return NOMAD_OK;
}

extern "C" nomad_status nomad_mlp_load(nomad_ctx *ctx, const char *path) {
  if (!ctx || !path) return NOMAD_ERR_INVALID_ARGUMENT;
  NOMAD_DEVICE_SCOPE(ctx);
  MlpState &S = mlp(ctx);
  auto reject = [&](const std::string &why) {
    S.ready = false;
    return nomad_fail(ctx, NOMAD_ERR_INVALID_ARGUMENT,
                      std::string("model file ") + path + ": " + why +
                          "; learned steps fall back to the ray-hit budget");
  };
  const size_t body = kModelHeader + (size_t)kParams * 4;
  std::vector<unsigned char> buf;
  {
    FILE *f = std::fopen(path, "rb");
    if (!f) return reject("cannot be opened");
    unsigned char tmp[65536];
    size_t got;
    while ((got = std::fread(tmp, 1, sizeof(tmp), f)) > 0 && buf.size() <= body + 8)
      buf.insert(buf.end(), tmp, tmp + got);
    std::fclose(f);
  }
  if (buf.size() < kModelHeader || std::memcmp(buf.data(), "NMLP", 4) != 0) return reject("not a model file");
  if (get_u32(buf.data() + 4) != kModelVersion)
    return reject("format version " + std::to_string(get_u32(buf.data() + 4)) + ", expected " +
                  std::to_string(kModelVersion));
  if (get_u32(buf.data() + 8) != (uint32_t)kParams || get_u32(buf.data() + 12) != (uint32_t)kIn)
    return reject("shape differs from this library's model");
  if (buf.size() != body + 8) return reject("size " + std::to_string(buf.size()) + " bytes, expected " +
                                            std::to_string(body + 8));
  const uint64_t want = (uint64_t)get_u32(buf.data() + body) | ((uint64_t)get_u32(buf.data() + body + 4) << 32);
  if (fnv1a(buf.data(), body) != want) return reject("checksum mismatch");
  std::vector<float> p(kParams);
  for (int i = 0; i < kParams; ++i) {
    const uint32_t bits = get_u32(buf.data() + kModelHeader + 4 * (size_t)i);
    std::memcpy(&p[i], &bits, 4);
    if (!std::isfinite(p[i])) return reject("parameter " + std::to_string(i) + " is not finite");
  }
  return nomad_mlp_set(ctx, p.data());
}

extern "C" nomad_status nomad_mlp_infer(nomad_ctx *ctx, const float *features, uint64_t n, float *out,
                                        uint32_t flags) {
  if (!ctx || (!features && n) || (!out && n)) return NOMAD_ERR_INVALID_ARGUMENT;
  NOMAD_DEVICE_SCOPE(ctx);
  MlpState &S = mlp(ctx);
  if (flags & NOMAD_TRACE_DEVICE_POINTERS) return nomad_mlp_infer_device(ctx, features, n, out);
  NOMAD_CUDA(ctx, S.inX.reserve(std::max<uint64_t>(1, n) * kIn * 4));
  NOMAD_CUDA(ctx, S.inY.reserve(std::max<uint64_t>(1, n) * 4));
  NOMAD_CUDA(ctx, cudaMemcpyAsync(S.inX.p, features, n * kIn * 4, cudaMemcpyHostToDevice, ctx->stream));
  nomad_status st = nomad_mlp_infer_device(ctx, S.inX.as<const float>(), n, S.inY.as<float>());
  if (st != NOMAD_OK) return st;
  NOMAD_CUDA(ctx, cudaMemcpyAsync(out, S.inY.p, n * 4, cudaMemcpyDeviceToHost, ctx->stream));
  NOMAD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return NOMAD_OK;
}

namespace {

// Split-K of the weight gradients: a split takes a whole number of 64-row blocks.
struct Splits {
  int blocks, count;
};
Splits batch_splits(int B) {
  const int want = std::max(1, std::min(32, B / 256));
  const int per = (B / want + 63) / 64;
  return {per, (B / 64 + per - 1) / per};
}

nomad_status ensure_batch(nomad_ctx *ctx, MlpState &S, int B, uint64_t losses) {
  const size_t tiles = ((size_t)B + 127) / 128, splits = batch_splits(B).count;
  NOMAD_CUDA(ctx, S.ximg.reserve(tiles * kXTileBytes));
  for (DeviceBuf *b : {&S.h1img, &S.z2img, &S.z1img}) NOMAD_CUDA(ctx, b->reserve(tiles * kTileBytes));
  for (DeviceBuf *b : {&S.g1c, &S.g2c, &S.g3c}) NOMAD_CUDA(ctx, b->reserve(tiles * 128 * kHid * 4));
  NOMAD_CUDA(ctx, S.dy.reserve((size_t)B * 4));
  NOMAD_CUDA(ctx, S.se.reserve((size_t)B * 4 * losses));
  NOMAD_CUDA(ctx, S.loss.reserve(4 * losses));
  NOMAD_CUDA(ctx, S.mask.reserve((size_t)B * 16));
  NOMAD_CUDA(ctx, S.part1.reserve(splits * kHid * kInPad * 4));
  NOMAD_CUDA(ctx, S.part2.reserve(splits * kHid * kHid * 4));
  return NOMAD_OK;
}

// Forward and backward of a batch of B samples of X and rows.T (B a multiple of 64): the gradient
// of the mean squared error with respect to every trainable parameter, as split-K partials and in
// S.G (k_adamw completes it; W1's padded input columns get 0), the per-row squared errors into se.
// Mixed precision as in the forward pass: BF16 operands of every product (standardised inputs,
// weights, hidden activations, the gradients that flow into a product), FP32 accumulation, FP32
// biases and output layer.
//
// Three launches a step and one for the update: a step of 4,096 rows takes 48 us (forward 19,
// hidden 7, input 17, update 4). It took 757 us as 17 launches whose column sums added 4,096 rows
// straight from memory, a thread a column, three times about 200 us. The chain of those additions is
// what bounds a step now (17.2k cycles of dependent additions): their order is the result's, so the
// sums of both layers run side by side, after the one that ends last.
nomad_status batch_gradient(nomad_ctx *ctx, MlpState &S, int B, const float *X, const TrainRows &rows, float *se,
                            TrainBufs &tb) {
  cudaStream_t s = ctx->stream;
  const Splits sp = batch_splits(B);
  const int tiles = (B + kTcRows - 1) / kTcRows;
  uint32_t *status = ctx->status.as<uint32_t>();
  tb = TrainBufs{S.ximg.as<unsigned char>(), S.h1img.as<unsigned char>(), S.z2img.as<unsigned char>(),
                 S.z1img.as<unsigned char>(), S.g1c.as<float>(), S.g2c.as<float>(), S.g3c.as<float>(),
                 S.dy.as<float>(), se,
                 S.mask.as<uint32_t>(), S.part1.as<float>(), S.part2.as<float>()};
  k_mlp_forward_tc<false, true><<<tiles, 128, kTcSmemTrain, s>>>(X, B, S.P.as<const float>(),
                                                                 S.Wc.as<const unsigned char>(), nullptr, status,
                                                                 nomad_res::FeatArgs{}, rows, tb);
  k_train_hidden<<<tiles + sp.count, 128, kHiddenSmem, s>>>(B, tiles, sp.blocks, S.W2t.as<const unsigned char>(), tb,
                                                            status);
  k_train_input<<<sp.count + 13, 128, kInputSmem, s>>>(B, sp.count, sp.blocks, S.G.as<float>(), tb, status);
  NOMAD_CUDA(ctx, cudaGetLastError());
  return NOMAD_OK;
}

}  // namespace

extern "C" nomad_status nomad_mlp_train(nomad_ctx *ctx, const float *features, const float *targets, uint64_t n,
                                        uint32_t steps, uint32_t batch, float lr, float wd, uint64_t seed,
                                        float *loss_out) {
  if (!ctx || !features || !targets || n == 0 || batch == 0 || batch % 64 != 0 || batch > 65536)
    return nomad_fail(ctx, NOMAD_ERR_INVALID_ARGUMENT, "training needs samples and a batch that is a multiple of 64");
  if (n > 0xffffffffull) return nomad_fail(ctx, NOMAD_ERR_LIMIT, "too many samples");
  NOMAD_DEVICE_SCOPE(ctx);
  MlpState &S = mlp(ctx);
  if (!S.ready) {
    nomad_status st = nomad_mlp_init(ctx, seed);
    if (st != NOMAD_OK) return st;
  }
  cudaStream_t s = ctx->stream;
  // Feature statistics (double accumulation on the host, each feature in sample order), stored in
  // the blob.
  double mean[kIn] = {}, sq[kIn] = {};
  for (uint64_t i = 0; i < n; ++i)
    for (int f = 0; f < kIn; ++f) {
      const double v = features[i * kIn + f];
      mean[f] += v;
      sq[f] += v * v;
    }
  float stats[2 * kIn];
  for (int f = 0; f < kIn; ++f) {
    double m = mean[f] / n;
    double var = std::max(0.0, sq[f] / n - m * m);
    stats[f] = (float)m;
    stats[kIn + f] = (float)(1.0 / std::max(std::sqrt(var), 1e-6));
  }
  NOMAD_CUDA(ctx, cudaMemcpyAsync(S.P.as<float>() + oMean, stats, sizeof(stats), cudaMemcpyHostToDevice, s));
  // Every call is a fresh AdamW run from the current weights: the moments start at zero, as the
  // bias correction (from step 1) assumes.
  NOMAD_CUDA(ctx, cudaMemsetAsync(S.M.p, 0, kParams * 4, s));
  NOMAD_CUDA(ctx, cudaMemsetAsync(S.V.p, 0, kParams * 4, s));
  const int B = (int)batch;
  // The squared errors of up to this many steps wait on the device for k_loss (at most 64 MB).
  const uint32_t keep = loss_out ? std::max(1u, std::min<uint32_t>(steps, (16u << 20) / batch)) : 1u;
  NOMAD_CUDA(ctx, S.X.reserve(n * kIn * 4));
  NOMAD_CUDA(ctx, S.T.reserve(n * 4));
  for (auto &p : S.perm) NOMAD_CUDA(ctx, p.reserve(n * 4));
  {
    nomad_status st = ensure_batch(ctx, S, B, keep);
    if (st != NOMAD_OK) return st;
  }
  NOMAD_CUDA(ctx, cudaMemcpyAsync(S.X.p, features, n * kIn * 4, cudaMemcpyHostToDevice, s));
  NOMAD_CUDA(ctx, cudaMemcpyAsync(S.T.p, targets, n * 4, cudaMemcpyHostToDevice, s));
  // Each epoch's permutation goes up on a copy stream into one of two buffers, so the host shuffles
  // and sends the next one while the steps of this one run. used[k]: the steps that read buffer k;
  // sent[k]: the copy into it, which the next steps wait for, and the host before it writes that copy's
  // source again.
  struct Events {
    cudaEvent_t used[2] = {nullptr, nullptr}, sent[2] = {nullptr, nullptr};
    cudaStream_t copy = nullptr, compute = nullptr;
    ~Events() {  // also after an error: nothing of this call may still be in flight
      cudaStreamSynchronize(copy);
      cudaStreamSynchronize(compute);
      for (cudaEvent_t e : {used[0], used[1], sent[0], sent[1]})
        if (e) cudaEventDestroy(e);
    }
  };
  std::mt19937_64 rng(seed ^ 0x5EEDull);
  std::vector<uint32_t> perm(n), source[2];
  std::iota(perm.begin(), perm.end(), 0u);
  Events ev;
  ev.copy = ctx->copyStreams[0];
  ev.compute = s;
  for (cudaEvent_t *e : {&ev.used[0], &ev.used[1], &ev.sent[0], &ev.sent[1]})
    NOMAD_CUDA(ctx, cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  uint64_t cursor = n;
  int buf = 1;
  bool first = true;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (uint32_t step = 0; step < steps; ++step) {
    if (cursor + B > n) {
      std::shuffle(perm.begin(), perm.end(), rng);
      if (!first) NOMAD_CUDA(ctx, cudaEventRecord(ev.used[buf], s));
      first = false;
      buf ^= 1;
      NOMAD_CUDA(ctx, cudaEventSynchronize(ev.sent[buf]));  // at once if nothing was sent from it yet
      source[buf] = perm;
      NOMAD_CUDA(ctx, cudaStreamWaitEvent(ev.copy, ev.used[buf], 0));
      NOMAD_CUDA(ctx, cudaMemcpyAsync(S.perm[buf].p, source[buf].data(), n * 4, cudaMemcpyHostToDevice, ev.copy));
      NOMAD_CUDA(ctx, cudaEventRecord(ev.sent[buf], ev.copy));
      NOMAD_CUDA(ctx, cudaStreamWaitEvent(s, ev.sent[buf], 0));
      cursor = 0;
    }
    TrainBufs tb;
    float *se = S.se.as<float>() + (size_t)(loss_out ? step % keep : 0) * B;
    nomad_status st = batch_gradient(ctx, S, B, S.X.as<const float>(),
                                     TrainRows{S.T.as<const float>(), S.perm[buf].as<const uint32_t>(), cursor, n}, se, tb);
    if (st != NOMAD_OK) return st;
    cursor += B;
    const float bc1 = 1.0f - std::pow(b1, (float)(step + 1)), bc2 = 1.0f - std::pow(b2, (float)(step + 1));
    k_adamw<<<(oMean + 127) / 128, 128, 0, s>>>(S.P.as<float>(), S.G.as<float>(), S.M.as<float>(), S.V.as<float>(),
                                                batch_splits(B).count, tb, true, lr, b1, b2, eps, wd, bc1, bc2,
                                                S.Wc.as<unsigned char>(), S.W2t.as<unsigned char>());
    NOMAD_CUDA(ctx, cudaGetLastError());
    if (loss_out && (step + 1 == steps || (step + 1) % keep == 0)) {
      const uint32_t done = step % keep + 1;
      k_loss<<<done, 128, 0, s>>>(S.se.as<const float>(), B, S.loss.as<float>());
      NOMAD_CUDA(ctx, cudaGetLastError());
      NOMAD_CUDA(ctx, cudaMemcpyAsync(loss_out + (step + 1 - done), S.loss.p, (size_t)done * 4, cudaMemcpyDeviceToHost, s));
    }
  }
  NOMAD_CUDA(ctx, cudaStreamSynchronize(s));
  return NOMAD_OK;
}

extern "C" nomad_status nomad_mlp_gradient(nomad_ctx *ctx, const float *features, const float *targets, uint64_t n,
                                           float *grad, float *loss) {
  if (!ctx) return NOMAD_ERR_INVALID_ARGUMENT;
  if (!features || !targets || !grad || n == 0 || n % 64 != 0 || n > 65536)
    return nomad_fail(ctx, NOMAD_ERR_INVALID_ARGUMENT, "the gradient needs 64 to 65,536 samples, a multiple of 64");
  NOMAD_DEVICE_SCOPE(ctx);
  MlpState &S = mlp(ctx);
  if (!S.ready) return nomad_fail(ctx, NOMAD_ERR_NOT_READY, "MLP not initialised or trained");
  const int B = (int)n;
  nomad_status st = ensure_batch(ctx, S, B, 1);
  if (st != NOMAD_OK) return st;
  cudaStream_t s = ctx->stream;
  NOMAD_CUDA(ctx, S.X.reserve(n * kIn * 4));
  NOMAD_CUDA(ctx, S.T.reserve(n * 4));
  NOMAD_CUDA(ctx, cudaMemcpyAsync(S.X.p, features, n * kIn * 4, cudaMemcpyHostToDevice, s));
  NOMAD_CUDA(ctx, cudaMemcpyAsync(S.T.p, targets, n * 4, cudaMemcpyHostToDevice, s));
  NOMAD_CUDA(ctx, cudaMemsetAsync(S.G.p, 0, kParams * 4, s));
  TrainBufs tb;
  st = batch_gradient(ctx, S, B, S.X.as<const float>(), TrainRows{S.T.as<const float>(), nullptr, 0, n}, S.se.as<float>(),
                      tb);
  if (st != NOMAD_OK) return st;
  k_adamw<<<(oMean + 127) / 128, 128, 0, s>>>(S.P.as<float>(), S.G.as<float>(), nullptr, nullptr, batch_splits(B).count,
                                              tb, false, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f, 1.0f, nullptr, nullptr);
  NOMAD_CUDA(ctx, cudaGetLastError());
  NOMAD_CUDA(ctx, cudaMemcpyAsync(grad, S.G.p, kParams * 4, cudaMemcpyDeviceToHost, s));
  std::vector<float> se(B);
  NOMAD_CUDA(ctx, cudaMemcpyAsync(se.data(), S.se.p, (size_t)B * 4, cudaMemcpyDeviceToHost, s));
  NOMAD_CUDA(ctx, cudaStreamSynchronize(s));
  if (loss) {
    double acc = 0.0;
    for (int i = 0; i < B; ++i) acc += se[i];
    *loss = (float)(acc / B);
  }
  return NOMAD_OK;
}

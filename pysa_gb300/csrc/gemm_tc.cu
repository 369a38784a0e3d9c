// gemm_tc.cu -- batched BF16 GEMM on the 5th-generation tensor cores for the
// learned flip proposal (MLP forward, backward and weight gradients).
//
//   C[b] (+)= A[b] * B[b]^T (+ bias[b], optionally ReLU), FP32 accumulation
//
// A is M x K and B is N x K, both BF16 and pre-packed by k_pack_kmajor into
// the canonical no-swizzle K-major core-matrix layout: tiles of 128 (A) or
// 256 (B) rows by 64 K, 16 KB / 32 KB each, so one 1-D bulk copy (TMA
// engine) moves a whole MMA operand tile.  One CTA computes a 128 x 256
// output tile in tensor memory: warp 5 streams the A/B tiles through a ring of
// shared-memory stages, one thread of warp 4 issues the tcgen05.mma
// instructions (four K=16 steps per 64-wide K tile) and warps 0-3 (thread =
// TMEM lane = output row) read the accumulator back with tcgen05.ld, add the
// bias and apply the ReLU.  M must be a multiple of 128, N of 256 and K of 64.
// Every wait is bounded.
//
// At the sizes of the proposal network (K 128 .. 1024) the epilogue is what
// takes the time, so it is kept to full lines: 32 x 32 blocks turn in the
// shared memory of the finished stages, from thread = row to eight lanes a
// row.  A row a thread and 4 bytes a store took 54 us a launch (mean over the
// learned-proposal loop at 32 networks of 512 - 1024 - 512), this 23 us.  The
// next layer's operand (BF16, packed) and the ReLU's mask of
// the backward pass are taken along, which saves a pass over C each.
#include "aux.cuh"
#include "gemm_api.h"
#include "tc_ptx.cuh"

namespace pysa_gb {

namespace {
constexpr int kStages = 4;  // at most
constexpr uint32_t kATile = 16384, kBTile = 32768;
constexpr uint32_t kStage = kATile + kBTile;
constexpr size_t kBarBytes = (2 * kStages + 1) * 8 + 16;

__device__ __forceinline__ bool gwait(uint64_t* bar, uint32_t parity,
                                      int32_t* status) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (globaltimer_ns() - t0 > 1000000000ull) {
      set_status(status, PYSA_GB_ERR_TIMEOUT);
      return false;
    }
  }
}
}  // namespace

__global__ void __launch_bounds__(192, 2) k_gemm_tc(const GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int stages = g.stages;
  uint64_t* full =
      reinterpret_cast<uint64_t*>(smem + (size_t)stages * kStage);
  uint64_t* empty = full + kStages;
  uint64_t* done = empty + kStages;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mt = blockIdx.x, nt = blockIdx.y, b = blockIdx.z;
  const int kt_n = g.K / 64;
  const uint16_t* A = g.A + (size_t)b * g.strideA +
                      (size_t)mt * kt_n * (kATile / 2);
  const uint16_t* B = g.B + (size_t)b * g.strideB +
                      (size_t)nt * kt_n * (kBTile / 2);

  if (warp == 0) {
    tc::tmem_alloc(tslot, 256);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  const uint32_t sbase = smem_addr(smem);

  if (warp == 5 && lane == 0) {
    int issued = 0;
    for (int kt = 0; kt < kt_n; ++kt) {
      const int s = kt % stages;
      if (kt >= stages &&
          !gwait(&empty[s], ((kt / stages) - 1) & 1, g.status))
        break;
      mbar_expect_tx_arrive(&full[s], kStage);
      bulk_g2s(smem + s * kStage, A + (size_t)kt * (kATile / 2), kATile,
               &full[s]);
      bulk_g2s(smem + s * kStage + kATile, B + (size_t)kt * (kBTile / 2),
               kBTile, &full[s]);
      issued = kt + 1;
    }
    // the CTA stays until its last copies have landed (bounded)
    for (int kt = issued > stages ? issued - stages : 0; kt < issued; ++kt)
      gwait(&full[kt % stages], (kt / stages) & 1, g.status);
  } else if (warp == 4 && lane == 0) {
    const uint32_t idesc = tc::idesc_bf16(128, 256);
    bool ok = true;
    for (int kt = 0; kt < kt_n; ++kt) {
      const int s = kt % stages;
      if (!gwait(&full[s], (kt / stages) & 1, g.status)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      const uint32_t a0 = sbase + s * kStage, b0 = a0 + kATile;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        tc::mma_bf16(taddr, tc::smem_desc(a0 + 256 * ks, 128, 1024),
                     tc::smem_desc(b0 + 256 * ks, 128, 1024), idesc,
                     (kt | ks) ? 1u : 0u);
      tc::commit(&empty[s]);
    }
    if (ok) tc::commit(done);
  } else if (warp < 4) {
    const bool ok = gwait(done, 0, g.status);
    tc::fence_after_sync();
    if (__all_sync(0xffffffffu, ok)) {
      // every copy has landed and every MMA has read its stage: the first
      // 16 KB are the epilogue's, 4 KB a warp
      float4* sq = reinterpret_cast<float4*>(smem) + warp * 256;
      const int row0 = mt * 128 + warp * 32;
      const size_t base =
          (size_t)b * g.strideC + (size_t)row0 * g.ldc + nt * 256;
      const float* bias =
          g.bias ? g.bias + (size_t)b * g.strideBias + nt * 256 : nullptr;
      uint4* packed =
          g.packed ? reinterpret_cast<uint4*>(
                         g.packed + (size_t)b * g.stridePacked)
                   : nullptr;
      for (int c0 = 0; c0 < 256; c0 += 32) {
        float v[32];
        const float bl = bias ? bias[c0 + lane] : 0.0f;
        tc::tmem_ld32(taddr + ((uint32_t)(warp * 32) << 16) + c0, v);
        if (bias) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            v[i] += __shfl_sync(0xffffffffu, bl, i);
        }
        if (g.relu && !g.accumulate) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.0f);
        }
        if (packed) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            packed[packed_unit(row0 + lane, (nt * 256 + c0) / 8 + q, g.N,
                               128)] = pack8(v + 8 * q);
        }
        __syncwarp();  // the last block has been read
#pragma unroll
        for (int q = 0; q < 8; ++q)
          sq[lane * 8 + (q ^ (lane & 7))] = make_float4(
              v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        __syncwarp();
        const int q = lane & 7;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = 4 * i + (lane >> 3);
          const float4 x = sq[r * 8 + (q ^ (r & 7))];
          const size_t o = base + (size_t)r * g.ldc + c0 + 4 * q;
          float y[4] = {x.x, x.y, x.z, x.w};
          if (g.vec) {
            if (g.accumulate) {
              const float4 c = *reinterpret_cast<const float4*>(g.C + o);
              y[0] += c.x; y[1] += c.y; y[2] += c.z; y[3] += c.w;
            }
            if (g.mask) {
              const float4 c = *reinterpret_cast<const float4*>(g.mask + o);
              if (c.x <= 0.0f) y[0] = 0.0f;
              if (c.y <= 0.0f) y[1] = 0.0f;
              if (c.z <= 0.0f) y[2] = 0.0f;
              if (c.w <= 0.0f) y[3] = 0.0f;
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (g.accumulate) y[k] += g.C[o + k];
              if (g.mask && g.mask[o + k] <= 0.0f) y[k] = 0.0f;
            }
          }
          if (g.relu && g.accumulate) {
#pragma unroll
            for (int k = 0; k < 4; ++k) y[k] = fmaxf(y[k], 0.0f);
          }
          if (g.vec) {
            *reinterpret_cast<float4*>(g.C + o) =
                make_float4(y[0], y[1], y[2], y[3]);
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) g.C[o + k] = y[k];
          }
        }
      }
    }
  }
  __syncwarp();
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(taddr, 256);
  }
}

// Pack rows x K of an FP32 matrix into BF16 K-major core-matrix tiles of
// `tile_rows` rows (128 or 256) by 64.  src(r, k) = src[r * ld + k], or
// src[k * ld + r] when TRANSPOSE.  Batched over blockIdx.y.  Bound by its
// bytes: a thread makes the 16 bytes of one core-matrix row, and a warp reads
// and writes whole 128-byte lines (8 rows x 32 columns, or 32 rows of a
// transposed source).  Launches of 2 to 4 M elements:
// 39 us with a thread per element, 4.7 us so.
template <bool TRANSPOSE, bool VEC>
__global__ void k_pack_kmajor(const float* src, int ld, int64_t src_stride,
                              int rows, int K, int tile_rows, uint16_t* dst,
                              int64_t dst_stride) {
  const int64_t units = (int64_t)rows * (K / 8);
  const float* s = src + (size_t)blockIdx.y * src_stride;
  uint4* d = reinterpret_cast<uint4*>(dst + (size_t)blockIdx.y * dst_stride);
  const int kt_n = K / 64, per = tile_rows * 8;  // units of a tile
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < units;
       u += (int64_t)gridDim.x * blockDim.x) {
    const int t = (int)(u / per), w = (int)(u - (int64_t)t * per);
    const int rt = t / kt_n, kt = t - rt * kt_n;
    float v[8];
    int64_t out = u;
    if (TRANSPOSE) {
      const int k8 = w / tile_rows, r = w - k8 * tile_rows;
      const float* p = s + (int64_t)(kt * 64 + 8 * k8) * ld +
                       (int64_t)rt * tile_rows + r;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = p[(int64_t)i * ld];
      out = (int64_t)t * per + (r >> 3) * 64 + k8 * 8 + (r & 7);
    } else {
      const int r = (w >> 6) * 8 + (w & 7), k8 = (w >> 3) & 7;
      const float* p =
          s + ((int64_t)rt * tile_rows + r) * ld + kt * 64 + 8 * k8;
      if (VEC) {
        const float4 x = reinterpret_cast<const float4*>(p)[0];
        const float4 y = reinterpret_cast<const float4*>(p)[1];
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[i];
      }
    }
    d[out] = pack8(v);
  }
}

cudaError_t launch_gemm_tc(const GemmArgs& args, int batch,
                           cudaStream_t st) {
  GemmArgs g = args;
  // two tiles per SM when K is short (two stages): the second one's loads
  // and products run under the first one's epilogue
  g.stages = g.K / 64 <= 2 ? 2 : kStages;
  const auto aligned = [](const void* p) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0;
  };
  g.vec = aligned(g.C) && g.ldc % 4 == 0 && g.strideC % 4 == 0 &&
          (!g.mask || aligned(g.mask));
  const size_t smem = (size_t)g.stages * kStage + kBarBytes;
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !attr[dev]) {
    cudaError_t e = cudaFuncSetAttribute(
        k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
        (int)(kStages * kStage + kBarBytes));
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  dim3 grid(g.M / 128, g.N / 256, batch);
  k_gemm_tc<<<grid, 192, smem, st>>>(g);
  return cudaGetLastError();
}

cudaError_t launch_pack_kmajor(const float* src, int ld, int64_t src_stride,
                               int rows, int K, int transpose, int tile_rows,
                               uint16_t* dst, int64_t dst_stride, int batch,
                               cudaStream_t st) {
  const int64_t units = (int64_t)rows * (K / 8);
  int blocks = (int)((units + 255) / 256 < 4096 ? (units + 255) / 256 : 4096);
  dim3 grid(blocks, batch);
  const bool vec = ld % 4 == 0 && src_stride % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(src) % 16 == 0;
  auto k = transpose ? k_pack_kmajor<true, false>
           : vec     ? k_pack_kmajor<false, true>
                     : k_pack_kmajor<false, false>;
  k<<<grid, 256, 0, st>>>(src, ld, src_stride, rows, K, tile_rows, dst,
                          dst_stride);
  return cudaGetLastError();
}

}  // namespace pysa_gb

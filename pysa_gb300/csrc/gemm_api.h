// gemm_api.h -- batched BF16 tcgen05 GEMM and operand packing.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace pysa_gb {

struct GemmArgs {
  const uint16_t* A;  // packed [batch][M/128][K/64] tiles of 128 x 64
  const uint16_t* B;  // packed [batch][N/256][K/64] tiles of 256 x 64
  float* C;           // [batch][M][ldc]
  const float* bias;  // [batch][N] or null
  int32_t* status;
  int64_t strideA, strideB, strideC, strideBias;  // elements per batch item
  int32_t M, N, K, ldc;
  int32_t accumulate;  // C += A B^T
  int32_t relu;        // ReLU after bias
  const float* mask;   // as C, or null: C is 0 where mask <= 0
  uint16_t* packed;    // or null (not with accumulate or mask): C as an A
  int64_t stridePacked;  // operand, [batch][M/128][N/64] tiles of 128 x 64
  int32_t stages, vec;   // set by launch_gemm_tc
};

// (tile, core row) order of a packed operand: where the 16 bytes of row r,
// columns 8 k8 .. 8 k8 + 7 start (in 8-element units).
__host__ __device__ inline int64_t packed_unit(int64_t r, int k8, int K,
                                               int tile_rows) {
  const int64_t rt = r / tile_rows;
  const int rr = (int)(r - rt * tile_rows);
  const int64_t tile = rt * (K / 64) + (k8 >> 3);
  return tile * (tile_rows * 8) + (rr >> 3) * 64 + (k8 & 7) * 8 + (rr & 7);
}

// Eight f32 as BF16 (nearest), in order.
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

cudaError_t launch_gemm_tc(const GemmArgs& g, int batch, cudaStream_t st);
cudaError_t launch_pack_kmajor(const float* src, int ld, int64_t src_stride,
                               int rows, int K, int transpose, int tile_rows,
                               uint16_t* dst, int64_t dst_stride, int batch,
                               cudaStream_t st);

}  // namespace pysa_gb

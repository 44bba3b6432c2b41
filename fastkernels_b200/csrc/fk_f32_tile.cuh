// True fp32 products of a tile on the FMA pipes, for fk_gemm_f32 and the fp32 form of
// fk_group_gemm.
//
// Bound by the fp32 rate.  A warp computes 32 rows x 64 weight rows, a lane 8 x 8 of them, with
// the packed fma.rn.f32x2: both halves of an accumulator are the same output, over the even and
// over the odd k's, so operands come as they lie in memory (k runs along both rows) and nothing
// is packed or transposed.  Per 4 k's a lane reads 16 float4 for 256 multiply-adds; rows are
// padded to 36 floats, so the 8 rows that a quarter of a warp reads start in different banks.
// WR x WC warps make the CTA's tile; loads run kStages - 1 blocks of 32 k's ahead (cp.async).
#pragma once

#include "fk_common.cuh"

namespace fk {

template <int WR, int WC>
struct F32Tile {
  static constexpr int kRows = 32 * WR, kCols = 64 * WC, kThreads = 32 * WR * WC;
  static constexpr int kBK = 32, kPitch = kBK + 4;
  static constexpr int kStages = 3;
  static constexpr int kStageFloats = (kRows + kCols) * kPitch;
  static constexpr int kSmem = kStages * kStageFloats * 4;

  struct Acc {
    float2 v[8][8];
  };

  // xrow(r) / wrow(c): pointer to the k's of row r < kRows of x or c < kCols of the weights, or
  // null for a row of zeros.  Rows are 16-byte aligned, k a multiple of 4.
  template <typename XRow, typename WRow>
  static __device__ __forceinline__ void run(float* smem, int k, XRow xrow, WRow wrow, Acc& acc) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kLoads = (kRows + kCols) * (kBK / 4) / kThreads;   // float4 per thread
    static_assert((kRows + kCols) * (kBK / 4) % kThreads == 0, "whole rounds of loads");
    const int c4 = (tid & 7) * 4;                 // 8 threads a row
    const float* src[kLoads];
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int r = (tid >> 3) + i * (kThreads / 8);
      src[i] = r < kRows ? xrow(r) : wrow(r - kRows);
    }
    auto load = [&](int stage, int k0) {
#pragma unroll
      for (int i = 0; i < kLoads; ++i) {
        const int r = (tid >> 3) + i * (kThreads / 8);
        float* dst = smem + stage * kStageFloats + r * kPitch + c4;
        const bool on = src[i] != nullptr && k0 + c4 < k;
        const uint32_t bytes = on ? 16u : 0u;     // the rest is filled with zeros
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)),
                     "l"(on ? src[i] + k0 + c4 : smem_any(smem)), "r"(bytes)
                     : "memory");
      }
    };
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc.v[i][j] = make_float2(0.f, 0.f);
    const int blocks = (k + kBK - 1) / kBK;
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
      if (s < blocks) load(s, s * kBK);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int ty = lane >> 3, tx = lane & 7;
    const int wr = warp / WC, wc = warp % WC;
    int stage = 0;
    for (int b = 0; b < blocks; ++b) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncthreads();
      const int ahead = b + kStages - 1;
      if (ahead < blocks) load(stage == 0 ? kStages - 1 : stage - 1, ahead * kBK);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const float* xs = smem + stage * kStageFloats + (wr * 32 + ty) * kPitch;
      const float* ws = smem + stage * kStageFloats + (kRows + wc * 64 + tx) * kPitch;
#pragma unroll
      for (int kk = 0; kk < kBK; kk += 4) {
        float4 a[8], w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          a[i] = *reinterpret_cast<const float4*>(xs + i * 4 * kPitch + kk);
          w[i] = *reinterpret_cast<const float4*>(ws + i * 8 * kPitch + kk);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            fma2(acc.v[i][j], a[i].x, a[i].y, w[j].x, w[j].y);
            fma2(acc.v[i][j], a[i].z, a[i].w, w[j].z, w[j].w);
          }
      }
      if (++stage == kStages) stage = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  // row and weight row of acc.v[i][j] within the CTA's tile
  static __device__ __forceinline__ int row(int i) {
    return (threadIdx.x >> 5) / WC * 32 + i * 4 + ((threadIdx.x & 31) >> 3);
  }
  static __device__ __forceinline__ int col(int j) {
    return (threadIdx.x >> 5) % WC * 64 + j * 8 + (threadIdx.x & 7);
  }
  static __device__ __forceinline__ float value(const Acc& acc, int i, int j) {
    return acc.v[i][j].x + acc.v[i][j].y;
  }

 private:
  // a source for copies of no bytes: any address of global memory would do, and none is read
  static __device__ __forceinline__ const float* smem_any(float* smem) { return smem; }
  static __device__ __forceinline__ void fma2(float2& c, float ax, float ay, float bx, float by) {
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "mov.b64 c, {%0, %1};\n\tfma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(c.x), "+f"(c.y)
        : "f"(ax), "f"(ay), "f"(bx), "f"(by));
  }
};

}  // namespace fk

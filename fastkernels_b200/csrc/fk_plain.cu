// Kernels without shape restrictions, for the number format and the head sizes the
// tensor-core kernels do not take:
//
//   fk_gemm_f32         y = x w^T (+ bias) in true fp32, any m, n
//   fk_paged_attn_any   causal attention over the paged NHD pool, bf16 or fp32, any
//                       head size up to 1152 and any query / KV head ratio; prompt
//                       portions and single decoded tokens alike
#include "fk_f32_tile.cuh"
#include "fk_gemm_shared.cuh"
#include "fk_types.cuh"

#include <mutex>

namespace fk {

// ------------------------------------------------------------------- fp32 products
// True fp32 products on the tensor cores.  An fp32 number is the sum of three bf16 numbers (each
// the rest rounded to 8 bits, so nothing is left over), and a product of two of them is six
// products of parts; the three that are left out are below 2^-26 of it.  Products of parts are
// exact in fp32, and sums are kept in fp32: 32 k's in tensor memory (whose adder cuts off instead
// of rounding, so chains there are kept short), smallest parts first, and the blocks of 32 in
// registers, rounded to nearest.  Off from 64 bits by 1.2 to 1.9e-7 (2-norm; k 2048 to 12288,
// normal operands), where chains of fp32 multiply-adds are by 2.1 to 5.0e-7.  bf16 goes down to
// 2^-133 and fp32 to 2^-149, so both operands are taken apart times 2^16, and the sums multiplied by
// 2^-32 when all are added up: exact, and every fp32 number keeps all of its bits (operands of 1e-36
// as they are were off by 2.6e-5).  It takes 1 to 2 % of the time.
//
// A CTA computes 128 weight rows (the M operand) x up to 128 rows of x.  Two teams of eight warps
// take every other block of k each: they read it ahead, take the numbers apart, and lay the parts
// out, the weights' in tensor memory, x's in shared memory, in a ring of four blocks.  One warp
// issues the 12 instructions of a block, four add up its sums.  Two teams, because the stretches of
// a block (waits, conversions, loads) follow one another in a warp: sixteen warps on one block go
// through them in step and take 1800 cycles for it, the teams 1350, the tensor cores alone 770.
//
// us, 1 / 100 / 1000 rows (fp32 multiply-adds in register tiles), calls apart: 24576 x 4096 136 186
// 1295 (217 644 4542), 155 TFLOP/s at 1000 rows; 2048 x 2048 14 23 98 (36 60 243); 4096 x 12288 69
// 90 700 (267 317 2540).  Back to back the power limit has 24576 x 4096, 1000 rows at 1455.
//
// A cluster of CTAs shares one tile: each takes a part of k, leaves its sums in its shared
// memory, and adds up its share of the rows over all parts in their order (f32_parts).  Where a
// sum is not finite, an operand may not have been either (the parts of an infinity are no
// numbers), or operands or products may have been too large (from 2^111 and 2^95 on): that output is
// computed again from the operands, in 64 bits (a matrix full of them: 40 to 70 times as long).
struct F32Tile {
  static constexpr int kRows = 128, kCols = 128;       // rows of x, weight rows
  static constexpr int kBK = 32, kStages = 4, kSums = 2;
  // two teams of warps that lay out operands, every other block each; warps that add up sums; a
  // warpgroup of which one issues the products
  static constexpr int kTeams = 2, kTeam = 8, kWarps = kTeams * kTeam, kAdders = 4;
  static constexpr int kIssuer = kWarps + kAdders;
  static constexpr int kThreads = 32 * (kIssuer + 4);
  // registers a thread of the three (setmaxnreg); what the warpgroup that adds up takes must come
  // from what the CTA was launched with: the host refuses a build that has fewer
  static constexpr int kRegsTeam = 72, kRegsAdder = 152, kRegsIssuer = 40;
  static constexpr int kRegsNeeded =
      32 * (kWarps * kRegsTeam + kAdders * kRegsAdder + 4 * kRegsIssuer);
  static_assert(kRegsNeeded <= 80 * kThreads, "register split exceeds the CTA's pool");
  static constexpr int kPlane = kRows * kBK * 2;       // one part of the rows of x
  static constexpr int kStageBytes = 3 * kPlane;
  // tensor memory: two blocks' sums, then the weights' parts, two numbers a cell
  static constexpr int kSumCols = kSums * kRows, kPartCols = kBK / 2, kTmemCols = 512;
  static constexpr int kOutPitch = kCols + 8;
  static constexpr float kScale = 65536.f;   // of either operand
  static constexpr int kSmem = 128 * 1024;
  static_assert(kSumCols + kStages * 3 * kPartCols <= kTmemCols, "tensor memory");
  static_assert(kStages * kStageBytes + 1024 <= kSmem && kRows * kOutPitch * 4 + 1024 <= kSmem,
                "operands, and the sums in their place");
  static_assert(tmem_alone(kSmem), "two CTAs could wait for one another's tensor memory");
};

// 16 rows x 8 cells: lane l has cells 2 (l & 3), + 1 of rows l / 4 and l / 4 + 8
__device__ __forceinline__ void tc_st_16x256(uint32_t taddr, uint2 a, uint2 b) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr),
               "r"(a.x), "r"(a.y), "r"(b.x), "r"(b.y)
               : "memory");
}
// K-major operand in rows of 64 bytes, 64-byte swizzle: 16-byte piece c of row r lies at
// c ^ (r >> 1 & 3); groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3fff) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
__device__ __forceinline__ float2 add_f32x2(float2 a, float2 b) {
  float2 c;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "add.rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "=f"(c.x), "=f"(c.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return c;
}
__device__ __forceinline__ float2 mul_f32x2(float2 a, float b) {
  float2 c;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\t"
      "mul.rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "=f"(c.x), "=f"(c.y) : "f"(a.x), "f"(a.y), "f"(b));
  return c;
}
// One part of two numbers, and what is left of them
__device__ __forceinline__ uint32_t f32_part(float2& a) {
  const uint32_t p = pack_bf16(a.x, a.y);
  const uint32_t n = p ^ 0x80008000u;
  a = add_f32x2(a, make_float2(bf16lo(n), bf16hi(n)));
  return p;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, int rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
// One output from the operands, in 64 bits
__device__ __noinline__ float f32_dot(const float* x, const float* w, int k) {
  double s[2] = {0., 0.};
  for (int i = 0; i < k; i += 4) {
    const float4 a = *reinterpret_cast<const float4*>(x + i);
    const float4 b = *reinterpret_cast<const float4*>(w + i);
    s[0] = fma((double)a.x, (double)b.x, s[0]);
    s[1] = fma((double)a.y, (double)b.y, s[1]);
    s[0] = fma((double)a.z, (double)b.z, s[0]);
    s[1] = fma((double)a.w, (double)b.w, s[1]);
  }
  return (float)(s[0] + s[1]);
}

// Row tile `t` of a product with row groups: its group and first row (of the group).
// Uniform over the block; every warp finds it by itself.
__device__ __forceinline__ bool f32_row_tile(const F32Product& p, int tile_rows, int64_t t,
                                             int* group, int64_t* m0) {
  const int lane = threadIdx.x & 31;
  for (int g0 = 0; g0 < p.groups; g0 += 32) {
    const int g = g0 + lane;
    int64_t tiles = 0;
    if (g < p.groups) {
      const int64_t a = p.offsets[g], b = p.offsets[g + 1];
      if (a < 0 || b < a || b > p.rows) {
        if (p.status) atomicOr(p.status, FK_DEV_BAD_SLOT);
      } else {
        tiles = (b - a + tile_rows - 1) / tile_rows;
      }
    }
    int64_t upto = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const uint32_t hit = __ballot_sync(0xffffffffu, t < upto);
    if (hit) {
      const int l = __ffs(hit) - 1;
      *group = g0 + l;
      *m0 = __shfl_sync(0xffffffffu, t - (upto - tiles), l) * tile_rows;
      return true;
    }
    t -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

template <bool ACT>
__global__ void __launch_bounds__(F32Tile::kThreads, 1)
    f32_product_kernel(const F32Product p, int parts, int64_t row_tiles) {
  using Tile = F32Tile;
  extern __shared__ uint8_t f32_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(f32_raw) + 1023) &
                                             ~uintptr_t(1023));
  __shared__ const float* f32_rows[Tile::kCols + Tile::kRows];   // weight rows, rows of x
  __shared__ uint64_t full[Tile::kStages], done[Tile::kStages],
      taken[Tile::kSums];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  constexpr int kOut = ACT ? Tile::kCols / 2 : Tile::kCols;     // outputs a row
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int i = 0; i < Tile::kStages; ++i) {
      mbar_init(&full[i], Tile::kTeam);
      mbar_init(&done[i], 1);
    }
    for (int i = 0; i < Tile::kSums; ++i) mbar_init(&taken[i], Tile::kAdders);
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == Tile::kIssuer) tmem_alloc(&tmem_slot, Tile::kTmemCols);
  pdl_wait();
  const int part = (int)(blockIdx.x % parts);
  const int64_t tile = blockIdx.x / parts, t = tile % row_tiles;
  const int n0 = (int)(tile / row_tiles) * kOut;
  const int blocks_all = (p.k + Tile::kBK - 1) / Tile::kBK;
  const int first_block = (int)((int64_t)blocks_all * part / parts);
  const int blocks = (int)((int64_t)blocks_all * (part + 1) / parts) - first_block;
  int g = blockIdx.z;
  int64_t m0 = t * Tile::kRows, first = 0, count = p.rows;
  bool there = true;                               // uniform over the cluster
  if (p.offsets) {
    there = f32_row_tile(p, Tile::kRows, t, &g, &m0);
    if (there) {
      first = p.offsets[g];
      count = p.offsets[g + 1] - first;
    }
  }
  const int live = there ? (int)(count - m0 < Tile::kRows ? count - m0 : Tile::kRows) : 0;
  const int width = (live + 15) & ~15;             // rows of x that are multiplied
  // addresses of the tile's rows; where there is none the last one, whose products are not kept
  if (there && tid < Tile::kCols + Tile::kRows) {
    const float* src;
    if (tid < Tile::kCols) {
      // with an activation 64 gate rows and the 64 up rows of the same outputs
      const int wrow = min(n0 + (ACT ? tid & 63 : tid), p.n - 1);
      src = p.w + ((int64_t)g * p.w_rows + wrow + (ACT && tid >= 64 ? p.n : 0)) * p.k;
    } else {
      int64_t xr = first + m0 + min(tid - Tile::kCols, live - 1);
      if (p.gather) {
        xr = p.gather[xr];
        if (xr < 0 || xr >= p.x_rows) {
          if (p.status) atomicOr(p.status, FK_DEV_BAD_SLOT);
          xr = 0;
        }
      }
      src = p.x + (p.offsets ? 0 : g * p.x_group) + xr * p.x_stride;
    }
    f32_rows[tid] = src;
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  auto cluster_sync = [] {
    __syncwarp();                      // lanes may have stored different numbers of outputs
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  // a wait of all of the warp's lanes; false in all of them when it ran out
  auto wait = [&](uint64_t* bar, int use) {
    const bool ok = gemm_wait(bar, (uint32_t)use & 1u, abort_flag, p.status);
    return __all_sync(0xffffffffu, ok) != 0;
  };
  float* const out = reinterpret_cast<float*>(smem);
  if (warp >= Tile::kIssuer) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Tile::kRegsIssuer));
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(width >> 3) << 17) |
                           ((uint32_t)(Tile::kCols >> 4) << 24);
    // the products of a block, smallest first, when all of its parts are laid out and the sums
    // that were in their place are taken
    for (int b = 0; there && warp == Tile::kIssuer && b < blocks; ++b) {
      const int stage = b % Tile::kStages, sum = b % Tile::kSums;
      if (b >= Tile::kSums && !wait(&taken[sum], b / Tile::kSums - 1)) break;
      if (!wait(&full[stage], b / Tile::kStages)) break;
      tc_fence_after();
      const uint32_t w = tmem + Tile::kSumCols + stage * 3 * Tile::kPartCols;
      constexpr int kW[6] = {2, 0, 1, 1, 0, 0}, kX[6] = {0, 2, 1, 0, 1, 0};
      // one branch for all: an instruction every 64 cycles, 130 where each has its own
      if (elect_one()) {
        const uint64_t x = smem_desc_sw64(smem_u32(smem + stage * Tile::kStageBytes));
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int kk = 0; kk < Tile::kBK / 16; ++kk)
            tc_mma_bf16_ts(tmem + sum * Tile::kRows, w + kW[i] * Tile::kPartCols + kk * 8,
                           x + ((kX[i] * Tile::kPlane + kk * 32) >> 4), idesc,
                           i > 0 || kk > 0 ? 1u : 0u);
        tc_commit(&done[stage]);
      }
      __syncwarp();
    }
    cluster_sync();                    // sums are laid out
    cluster_sync();                    // and read
    if (warp == Tile::kIssuer) tmem_dealloc(tmem, Tile::kTmemCols);
    return;
  }
  if (warp >= Tile::kWarps) {
    // a lane has one weight row and all rows of x
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Tile::kRegsAdder));
    const int q = warp & 3;
    float2 acc[Tile::kRows / 2];
#pragma unroll
    for (int i = 0; i < Tile::kRows / 2; ++i) acc[i] = make_float2(0.f, 0.f);
    bool ok = true;
    for (int b = 0; there && b < blocks; ++b) {
      const int sum = b % Tile::kSums;
      ok = wait(&done[b % Tile::kStages], b / Tile::kStages);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < Tile::kRows; h += 16) {
        if (h >= width) break;
        uint32_t v[16];
        tc_ld16(tmem + sum * Tile::kRows + h + ((uint32_t)(q * 32) << 16), v);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i)
          acc[h / 2 + i] = add_f32x2(acc[h / 2 + i], make_float2(__uint_as_float(v[2 * i]),
                                                                 __uint_as_float(v[2 * i + 1])));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&taken[sum]);
    }
    // a wait ran out: no number, so that the outputs are computed from the operands
    float* to = out + q * 32 + lane;
#pragma unroll
    for (int i = 0; i < Tile::kRows; ++i)
      if (i < live)
        to[i * Tile::kOutPitch] = ok ? (i & 1 ? acc[i / 2].y : acc[i / 2].x) : __int_as_float(0x7fffffff);
    cluster_sync();
    cluster_sync();
    return;
  }
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Tile::kRegsTeam));
  if (there) {
    const int team = warp / Tile::kTeam, half = warp >> 2 & 1;
    // weights: 16-byte pieces lane & 3 and 4 further of rows w0 and w0 + 8, as tc_st_16x256 wants
    // them; x: piece `c` of rows r, r + 32, ...
    const int w0 = (warp & 3) * 32 + half * 16;
    const uint32_t wdst = tmem + Tile::kSumCols + ((uint32_t)w0 << 16);
    const float* ws[2] = {f32_rows[w0 + (lane >> 2)], f32_rows[w0 + (lane >> 2) + 8]};
    const int c = tid & 7, r = (tid & 255) >> 3;
    const int xdst = r * 64 + (((c >> 1) ^ ((r >> 1) & 3)) << 4) + (c & 1) * 8;   // rows + 32 too
    const float* const* xs = f32_rows + Tile::kCols + r;
    float4 wv[4], xv[4];
    auto load = [&](int b) {
      if (b >= blocks) return;
      const int k0 = (first_block + b) * Tile::kBK;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k1 = k0 + (i >> 1) * 16 + (lane & 3) * 4;
        wv[i] = k1 < p.k ? __ldg(reinterpret_cast<const float4*>(ws[i & 1] + k1)) : zero;
      }
      const bool in = k0 + c * 4 < p.k;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (r + 32 * i < width)
          xv[i] = in ? __ldg(reinterpret_cast<const float4*>(xs[32 * i] + k0 + c * 4)) : zero;
    };
    load(team);
    for (int b = team; b < blocks; b += Tile::kTeams) {
      const int stage = b % Tile::kStages;
      if (b >= Tile::kStages && !wait(&done[stage], b / Tile::kStages - 1)) break;
      tc_fence_after();
      const uint32_t wto = wdst + stage * 3 * Tile::kPartCols;
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        float2 lo0 = mul_f32x2(make_float2(wv[i].x, wv[i].y), Tile::kScale);
        float2 hi0 = mul_f32x2(make_float2(wv[i].z, wv[i].w), Tile::kScale);
        float2 lo1 = mul_f32x2(make_float2(wv[i + 1].x, wv[i + 1].y), Tile::kScale);
        float2 hi1 = mul_f32x2(make_float2(wv[i + 1].z, wv[i + 1].w), Tile::kScale);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const uint2 a = make_uint2(f32_part(lo0), f32_part(hi0));
          const uint2 e = make_uint2(f32_part(lo1), f32_part(hi1));
          tc_st_16x256(wto + j * Tile::kPartCols + i * 4, a, e);
        }
      }
      uint8_t* xto = smem + stage * Tile::kStageBytes + xdst;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (r + 32 * i >= width) continue;
        float2 lo = mul_f32x2(make_float2(xv[i].x, xv[i].y), Tile::kScale);
        float2 hi = mul_f32x2(make_float2(xv[i].z, xv[i].w), Tile::kScale);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const uint32_t pl = f32_part(lo), ph = f32_part(hi);
          *reinterpret_cast<uint2*>(xto + j * Tile::kPlane + i * 32 * 64) = make_uint2(pl, ph);
        }
      }
      load(b + Tile::kTeams);
      tc_wait_st();
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[stage]);
    }
  }
  cluster_sync();
  const int r0 = live * part / parts, r1 = live * (part + 1) / parts;
  float* y = p.y + (p.offsets ? 0 : g * p.y_group);
  auto sum = [&](int r, int c) {
    const uint32_t addr = smem_u32(out + r * Tile::kOutPitch + c);
    float v = ld_cluster_f32(addr, 0);
    for (int q = 1; q < parts; ++q) v += ld_cluster_f32(addr, q);
    if (!(fabsf(v) <= 3.402823466e38f))
      return f32_dot(f32_rows[Tile::kCols + r], f32_rows[c], p.k);
    return v * (1.f / (Tile::kScale * Tile::kScale));
  };
  for (int i = r0 * kOut + tid; i < r1 * kOut; i += 32 * Tile::kWarps) {
    const int r = i / kOut, c = i % kOut;
    if (n0 + c >= p.n) continue;
    float v;
    if (ACT) {
      const float gate = sum(r, c) + (p.bias ? p.bias[n0 + c] : 0.f);
      const float up = sum(r, c + 64) + (p.bias ? p.bias[p.n + n0 + c] : 0.f);
      v = (p.act == FK_ACT_SILU ? gate * sigmoid_f32(gate) : gelu_tanh_f32(gate)) * up;
    } else {
      v = sum(r, c) + (p.bias ? p.bias[n0 + c] : 0.f);
    }
    y[(first + m0 + r) * p.y_stride + n0 + c] = v;
  }
  cluster_sync();                      // peers may still read this CTA's sums
}

// Short k: the tiles above spend their time filling the ring and handing sums on, and half of a
// tile's weight rows may be missing.  fp32 multiply-adds, 64 x 64
// outputs, 4 x 4 a thread, k in one order.  us, 60 / 200 / 1000 rows, here and in the tiles above:
// 16 heads of 96 -> 512 7 21 54 (11 28 98), 40 of 256 -> 64 15 35 50 (13 28 76), 40 of 64 -> 256
// 10 15 48 (20 34 116).
constexpr int FS_M = 64, FS_N = 64, FS_K = 16, FS_MAX_K = 511;

template <bool ACT>
__global__ void __launch_bounds__(256) f32_short_kernel(const F32Product p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int NB = ACT ? 2 : 1;
  __shared__ float xs[FS_K][FS_M + 4], ws[NB][FS_K][FS_N + 4];
  const int g = blockIdx.z;
  int64_t first = 0, count = p.rows;
  if (p.offsets) {
    const int64_t a = p.offsets[g], b = p.offsets[g + 1];
    if (a < 0 || b < a || b > p.rows) {
      if (p.status && threadIdx.x == 0) atomicOr(p.status, FK_DEV_BAD_SLOT);
      return;
    }
    first = a;
    count = b - a;
  }
  const int n0 = blockIdx.x * FS_N;
  const int64_t m0 = (int64_t)blockIdx.y * FS_M;
  if (m0 >= count) return;
  const float* x = p.x + (p.offsets ? 0 : g * p.x_group);
  const float* w = p.w + (int64_t)g * p.w_rows * p.k;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int lr = threadIdx.x >> 2, lc = (threadIdx.x & 3) * 4;
  const bool x_on = m0 + lr < count, w_on = n0 + lr < p.n;
  int64_t row = 0;
  if (x_on) {
    row = first + m0 + lr;
    if (p.gather) {
      row = p.gather[row];
      if (row < 0 || row >= p.x_rows) {
        if (p.status) atomicOr(p.status, FK_DEV_BAD_SLOT);
        row = 0;
      }
    }
  }
  const float* xr = x + row * p.x_stride;
  float acc[NB][4][4] = {};
  for (int k0 = 0; k0 < p.k; k0 += FS_K) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b[NB];
#pragma unroll
    for (int e = 0; e < NB; ++e) b[e] = a;
    if (k0 + lc < p.k) {                        // k is a multiple of 4
      if (x_on) a = *reinterpret_cast<const float4*>(xr + k0 + lc);
#pragma unroll
      for (int e = 0; e < NB; ++e)
        if (w_on)
          b[e] = *reinterpret_cast<const float4*>(w + ((int64_t)e * p.n + n0 + lr) * p.k + k0 + lc);
    }
    __syncthreads();
    xs[lc][lr] = a.x; xs[lc + 1][lr] = a.y; xs[lc + 2][lr] = a.z; xs[lc + 3][lr] = a.w;
#pragma unroll
    for (int e = 0; e < NB; ++e) {
      ws[e][lc][lr] = b[e].x; ws[e][lc + 1][lr] = b[e].y;
      ws[e][lc + 2][lr] = b[e].z; ws[e][lc + 3][lr] = b[e].w;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < FS_K; ++kk) {
      const float4 av = *reinterpret_cast<const float4*>(&xs[kk][ty * 4]);
      const float aa[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int e = 0; e < NB; ++e) {
        const float4 bv = *reinterpret_cast<const float4*>(&ws[e][kk][tx * 4]);
        const float bb[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[e][i][j] = fmaf(aa[i], bb[j], acc[e][i][j]);
      }
    }
  }
  float* y = p.y + (p.offsets ? 0 : g * p.y_group);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t r = m0 + ty * 4 + i;
    if (r >= count) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tx * 4 + j;
      if (c >= p.n) continue;
      float v = acc[0][i][j] + (p.bias ? p.bias[c] : 0.f);
      if (ACT) {
        const float up = acc[NB - 1][i][j] + (p.bias ? p.bias[p.n + c] : 0.f);
        v = (p.act == FK_ACT_SILU ? v * sigmoid_f32(v) : gelu_tanh_f32(v)) * up;
      }
      y[(first + r) * p.y_stride + c] = v;
    }
  }
}

template <bool ACT>
static int launch_f32_short(const F32Product& p, cudaStream_t s) {
  const dim3 grid((unsigned)((p.n + FS_N - 1) / FS_N), (unsigned)((p.rows + FS_M - 1) / FS_M),
                  (unsigned)p.groups);
  FK_CUDA_OK(launch_kernel(f32_short_kernel<ACT>, grid, dim3(256), 0, s, p));
  count_launch();
  return FK_OK;
}

// Parts of k, by the weights' sizes alone: a row's sums are taken in the same order whatever other
// rows are in the call.  Few weight tiles get more parts, so that few rows find SMs; many rows
// would have them anyway and pay for the exchange.  us, rows 1 / 100 / 500 / 1000 in 1, 2, 4, 8 parts:
//   n 544, k 2048     36 55 60 61     21 34 38 38     14 22 25 46      11 17 35 51
//   n 2048, k 2048    36 55 61 64     21 34 39 75     14 23 49 95      20 32 86 152
//   n 4096, k 4096    70 101 117 223  39 58 124 243   23 35 145 288    41 65 211 416
//   n 7680, k 2560    48 71 149 292   28 43 173 300   33 51 216 402    47 72 308 607
//   n 24576, k 4096   163 222 682 1231  135 184 677 1279  154 215 858 1662  210 303 1213 2382
//   n 32768, k 2048   91 125 438 853  101 146 526 1032  126 188 754 1458  198 303 1189 2332
// 32 experts, 2 x 1024 x 2048, 4 / 60 / 400 / 3100 rows in all: 38 180 187 264, 26 185 199 297,
// 34 256 283 437, 52 424 473 743; 64 of 4096 x 1408: 37 285 485 595, 43 354 573 751.
static int f32_parts(const F32Product& p) {
  const int64_t tiles = (p.w_rows + 127) / 128 * p.groups;
  return tiles <= 12 && p.k >= 2048 ? 8 : tiles <= 32 && p.k >= 1024 ? 4 : tiles < 256 ? 2 : 1;
}

template <bool ACT>
static int launch_f32_tile(const F32Product& p, cudaStream_t s) {
  using Tile = F32Tile;
  constexpr int kOut = ACT ? Tile::kCols / 2 : Tile::kCols;
  const int64_t n_tiles = (p.n + kOut - 1) / kOut;
  const int64_t upto = (p.rows + Tile::kRows - 1) / Tile::kRows;
  // row groups: at most one part-filled tile a group
  const int64_t used = p.rows < p.groups ? p.rows : p.groups;
  const int64_t row_tiles = p.offsets ? upto + used : upto;
  const int parts = f32_parts(p);
  FK_REQUIRE(n_tiles * row_tiles * parts <= 0x7fffffff, FK_ERR_UNSUPPORTED,
             "fp32 product: too many tiles");
  // registers a thread of the compiled kernel: the same on every device
  static std::once_flag regs_once;
  static cudaError_t regs_err = cudaSuccess;
  static int launch_regs = 0;
  std::call_once(regs_once, [] {
    cudaFuncAttributes f;
    regs_err = cudaFuncGetAttributes(&f, f32_product_kernel<ACT>);
    if (regs_err == cudaSuccess) launch_regs = f.numRegs;
  });
  FK_CUDA_OK(regs_err);
  FK_REQUIRE(launch_regs * Tile::kThreads >= Tile::kRegsNeeded, FK_ERR_UNSUPPORTED,
             "fp32 product: this build of the kernel holds %d registers per thread, fewer than its "
             "register split needs", launch_regs);
  static PerDeviceOnce once;
  FK_CUDA_OK(set_max_dynamic_smem(once, f32_product_kernel<ACT>, Tile::kSmem));
  cudaLaunchConfig_t cfg{};
  // rows fastest: the tiles of a weight tile find it in L2
  cfg.gridDim = dim3((unsigned)(n_tiles * row_tiles * parts), 1u,
                     p.offsets ? 1u : (unsigned)p.groups);
  cfg.blockDim = dim3(Tile::kThreads);
  cfg.dynamicSmemBytes = Tile::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  attr[na].id = cudaLaunchAttributeClusterDimension;
  attr[na].val.clusterDim.x = (unsigned)parts;
  attr[na].val.clusterDim.y = 1;
  attr[na++].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = na;
  FK_CUDA_OK(cudaLaunchKernelEx(&cfg, f32_product_kernel<ACT>, p, parts, row_tiles));
  count_launch();
  return FK_OK;
}

template <bool ACT>
static int launch_f32(const F32Product& p, cudaStream_t s) {
  return p.k <= FS_MAX_K ? launch_f32_short<ACT>(p, s) : launch_f32_tile<ACT>(p, s);
}
int launch_f32_product(const F32Product& p, cudaStream_t s) {
  return p.act >= 0 ? launch_f32<true>(p, s) : launch_f32<false>(p, s);
}

// ----------------------------------------------------------------------- attention
struct AnyAttnParams {
  const void* q; int64_t q_stride; void* out; int64_t out_stride;
  const void* k_cache; const void* v_cache;
  const int32_t* cu_q; const int32_t* kv_lens;
  const int32_t* block_tables; int64_t bt_stride;
  int num_seqs, hq, hkv, d, block_size, num_blocks;
  int64_t rows;
  int64_t least, below;             // sequences of least .. below - 1 queries a KV head are taken
  float scale;
  int32_t* status;
};

// Bound by shared-memory reads and the fp32 rate.  A CTA takes 8 R queries of one sequence and
// KV head (rows x the heads that share it) through runs of 32 keys, which it lays out in shared
// memory once for all of them: lane j of a warp scores key j for its R queries, then the lanes
// own the value channels lane, lane + 32, ...; few queries per sequence (single tokens) are spread
// over all warps.  R changes no sum's order.
constexpr int AA_WARPS = 8, AA_THREADS = 32 * AA_WARPS, AA_KEYS = 32;
constexpr int AA_MAX_SMEM = 227 * 1024 - 1024;

__host__ __device__ inline int aa_pitch(int d) { return (d + 31) / 32 * 32 + 4; }

// The sequence whose queries blk (then within it) QB at a time are, its rows, -1: none; every warp
// finds it by itself.
template <int QB>
__device__ __forceinline__ int aa_find(const AnyAttnParams& p, int grp, int64_t& blk, int64_t& row0,
                                       int64_t& row1) {
  const int lane = threadIdx.x & 31;
  int seq = -1;
  row0 = row1 = 0;
  for (int s0 = 0; s0 < p.num_seqs && seq < 0; s0 += 32) {
    const int sq = s0 + lane;
    int64_t a = 0, b = 0;
    if (sq < p.num_seqs) {
      a = sq == 0 ? 0 : p.cu_q[sq];
      b = sq == p.num_seqs - 1 ? p.rows : p.cu_q[sq + 1];
      a = a < 0 ? 0 : a;
      b = b > p.rows ? p.rows : b;
    }
    const int64_t n = (b - a) * grp;
    const int64_t mine = n > 0 && n >= p.least && n < p.below ? (n + QB - 1) / QB : 0;
    int64_t upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const uint32_t hit = __ballot_sync(0xffffffffu, blk < upto);
    if (hit) {
      const int l = __ffs(hit) - 1;
      seq = s0 + l;
      blk -= __shfl_sync(0xffffffffu, upto - mine, l);
      row0 = __shfl_sync(0xffffffffu, a, l);
      row1 = __shfl_sync(0xffffffffu, b, l);
    } else {
      blk -= __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  return seq;
}

// Rows of one run of keys to shared memory; keys that are not there are rows of zeros.  All pieces
// of a thread are under way at once: in a loop, each waited for the one before it (fp32, 576
// channels, 16 heads on one KV head, 20 tokens on 700 keys 313 -> 231 us, 4 heads, 5 on 300
// 151 -> 116; 128 channels, 16 heads on 4, 900 tokens 371 -> 313; bf16 368 -> 328).
template <typename T, int CH, int WARPS>
__device__ __forceinline__ void aa_stage(const AnyAttnParams& p, const void* cache,
                                         const int64_t* key_off, float* ks, int pitch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quads = p.d >> 2;
  if constexpr (sizeof(T) == 4) {
    for (int j = warp; j < AA_KEYS; j += WARPS) {
      const int64_t off = key_off[j];
      const float* src = static_cast<const float*>(cache) + (off < 0 ? 0 : off);
      const uint32_t dst = smem_u32(ks + j * pitch), bytes = off < 0 ? 0 : 16;
#pragma unroll
      for (int i = 0; i < (CH + 3) / 4; ++i) {
        const int c = lane + i * 32;
        if (c < quads)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + c * 16),
                       "l"(src + c * 4), "r"(bytes) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    for (int j = warp; j < AA_KEYS; j += WARPS) {
      const int64_t off = key_off[j];
      const T* src = static_cast<const T*>(cache) + off;
      float4 v[(CH + 3) / 4];
#pragma unroll
      for (int i = 0; i < (CH + 3) / 4; ++i) {
        const int c = lane + i * 32;
        v[i] = off < 0 || c >= quads ? make_float4(0.f, 0.f, 0.f, 0.f)
                                     : Elem<T>::load4(src + c * 4);
      }
#pragma unroll
      for (int i = 0; i < (CH + 3) / 4; ++i) {
        const int c = lane + i * 32;
        if (c < quads) *reinterpret_cast<float4*>(ks + j * pitch + c * 4) = v[i];
      }
    }
  }
}

template <typename T, int CH, int R>
__global__ void __launch_bounds__(AA_THREADS) paged_attn_any_kernel(const AnyAttnParams p,
                                                                    int64_t blocks) {
  extern __shared__ __align__(16) float aa_smem[];
  __shared__ int64_t key_off[AA_KEYS];
  constexpr int QB = AA_WARPS * R;
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = p.hq / p.hkv, pitch = aa_pitch(p.d);
  float* qs = aa_smem;                          // [QB][d], scaled
  float* ks = aa_smem + QB * p.d;               // [32][pitch]; d is a multiple of 4
  const bool shared_rows = p.k_cache == p.v_cache;
  for (int64_t it = blockIdx.x; it < blocks * p.hkv; it += gridDim.x) {
    const int kvh = (int)(it % p.hkv);
    int64_t blk = it / p.hkv;
    int64_t row0, row1;
    const int seq = aa_find<QB>(p, grp, blk, row0, row1);
    if (seq < 0) continue;                      // uniform over the block
    const int64_t queries = (row1 - row0) * grp, q0 = blk * QB;
    const int live = (int)(queries - q0 < QB ? queries - q0 : QB);
    const int kv_len = p.kv_lens[seq];
    // keys that row `row` sees
    const int64_t seen0 = (int64_t)kv_len - (p.cu_q[seq + 1] - p.cu_q[seq]) + 1 - p.cu_q[seq];
    auto visible = [&](int64_t row) {
      const int64_t v = seen0 + row;
      return (int)(v < kv_len ? v : kv_len);
    };
    const int keys = visible(row0 + (q0 + live - 1) / grp);
    __syncthreads();                            // the queries before are done with
    for (int i = tid; i < live * p.d; i += AA_THREADS) {
      const int j = i / p.d, c = i - j * p.d;
      const int64_t row = row0 + (q0 + j) / grp;
      const int head = kvh * grp + (int)((q0 + j) % grp);
      qs[j * p.d + c] = Elem<T>::load(static_cast<const T*>(p.q) + row * p.q_stride +
                                      (int64_t)head * p.d + c) * p.scale;
    }
    // a warp's queries: warp, warp + 8, ...
    const float* q[R];
    int vis[R], vis_min = 0x7fffffff;
    float m[R], l[R], acc[R][CH];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = warp + r * AA_WARPS;
      const bool on = j < live;
      q[r] = qs + (on ? j : 0) * p.d;
      vis[r] = on ? visible(row0 + (q0 + j) / grp) : 0;
      vis_min = min(vis_min, vis[r]);
      m[r] = -INFINITY;
      l[r] = 0.f;
#pragma unroll
      for (int i = 0; i < CH; ++i) acc[r][i] = 0.f;
    }
    const bool idle = warp >= live;
    const int32_t* bt = p.block_tables + (int64_t)seq * p.bt_stride;
    auto stage = [&](const void* cache) { aa_stage<T, CH, AA_WARPS>(p, cache, key_off, ks, pitch); };
    for (int k0 = 0; k0 < keys; k0 += AA_KEYS) {
      __syncthreads();
      if (tid < AA_KEYS) {
        const int kk = k0 + tid;
        int64_t off = -1;
        if (kk < keys) {
          const int page = bt[kk / p.block_size];
          if (page < 0 || page >= p.num_blocks) {
            if (p.status) atomicOr(p.status, FK_DEV_BAD_PAGE);
          } else {
            off = (((int64_t)page * p.block_size + kk % p.block_size) * p.hkv + kvh) * p.d;
          }
        }
        key_off[tid] = off;
      }
      __syncthreads();
      stage(p.k_cache);
      __syncthreads();
      float pr[R];
      if (!idle) {
        float s4[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) s4[r][e] = 0.f;
        const float* kr = ks + lane * pitch;
#pragma unroll 2
        for (int c = 0; c < p.d; c += 4) {
          const float4 kv = *reinterpret_cast<const float4*>(kr + c);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float4 qv = *reinterpret_cast<const float4*>(q[r] + c);
            s4[r][0] = fmaf(kv.x, qv.x, s4[r][0]);
            s4[r][1] = fmaf(kv.y, qv.y, s4[r][1]);
            s4[r][2] = fmaf(kv.z, qv.z, s4[r][2]);
            s4[r][3] = fmaf(kv.w, qv.w, s4[r][3]);
          }
        }
        const bool there = key_off[lane] >= 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float s = there && k0 + lane < vis[r]
                              ? (s4[r][0] + s4[r][1]) + (s4[r][2] + s4[r][3]) : -INFINITY;
          float mx = s;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
          const float m_new = fmaxf(m[r], mx);
          pr[r] = 0.f;
          if (m_new == -INFINITY) continue;     // uniform over the warp
          const float alpha = expf(m[r] - m_new);
          m[r] = m_new;
          pr[r] = expf(s - m_new);
          l[r] = l[r] * alpha + warp_sum(pr[r]);
#pragma unroll
          for (int i = 0; i < CH; ++i) acc[r][i] *= alpha;
        }
      }
      if (!shared_rows) {
        __syncthreads();
        stage(p.v_cache);
        __syncthreads();
      }
      if (idle) continue;
      const int cnt = min(AA_KEYS, keys - k0);
      if (k0 + cnt <= vis_min) {
        for (int j = 0; j < cnt; ++j) {
          float pj[R];
#pragma unroll
          for (int r = 0; r < R; ++r) pj[r] = __shfl_sync(0xffffffffu, pr[r], j);
#pragma unroll
          for (int i = 0; i < CH; ++i) {
            if (lane + i * 32 < p.d) {
              const float v = ks[j * pitch + lane + i * 32];
#pragma unroll
              for (int r = 0; r < R; ++r) acc[r][i] = fmaf(pj[r], v, acc[r][i]);
            }
          }
        }
      } else {
        // some query does not see all of them: what it does not see is not multiplied by a
        // weight of zero, it may be anything
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int n = min(cnt, vis[r] - k0);
          for (int j = 0; j < n; ++j) {
            const float pj = __shfl_sync(0xffffffffu, pr[r], j);
#pragma unroll
            for (int i = 0; i < CH; ++i)
              if (lane + i * 32 < p.d)
                acc[r][i] = fmaf(pj, ks[j * pitch + lane + i * 32], acc[r][i]);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = warp + r * AA_WARPS;
      if (j >= live) break;
      const float inv = l[r] > 0.f ? 1.0f / l[r] : 0.f;
      T* o = static_cast<T*>(p.out) + (row0 + (q0 + j) / grp) * p.out_stride +
             (kvh * grp + (q0 + j) % grp) * p.d;
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int c = lane + i * 32;
        if (c < p.d) Elem<T>::store(o + c, acc[r][i] * inv);
      }
    }
  }
}

// Many queries a sequence: 32 of them (rows x the heads that share a KV head) through runs of 32
// keys.  What bounds it is the latency and the bytes of shared-memory reads, so that both products
// are tiles in registers: a warp makes the scores of 16 queries from an eighth of the channels, a
// thread 4 x 4 of them, and the parts are added; then a warp has 8 queries and a quarter of the
// channels.  16 warps an SM are what fits (8, with twice the tile each: 864 us where these take
// 680, one portion of 900 tokens, 16 heads of 576 channels).  The longest queries come first.
constexpr int AT_WARPS = 16, AT_THREADS = 32 * AT_WARPS, AT_SLICES = 8;
constexpr int AT_QUERIES = 32, AT_PPITCH = AT_QUERIES + 4, AT_SPITCH = AA_KEYS + 8;
__host__ __device__ inline int at_smem(int d) {
  return ((AT_QUERIES + AA_KEYS) * aa_pitch(d) + AT_SLICES * AT_QUERIES * AT_SPITCH +
          AA_KEYS * AT_PPITCH) * 4;
}
__device__ __forceinline__ uint64_t at_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t at_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 at_unpack(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

template <typename T, int CH>
__global__ void __launch_bounds__(AT_THREADS, 1)
paged_attn_tile_kernel(const AnyAttnParams p, int64_t blocks) {
  extern __shared__ __align__(16) float aa_smem[];
  __shared__ int64_t key_off[AA_KEYS];
  __shared__ int vis_s[AT_QUERIES];
  __shared__ __align__(16) float alpha_s[AT_QUERIES], inv_s[AT_QUERIES];
  constexpr int HC = (CH + 3) / 4;              // chunks of 32 channels a warp owns
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grp = p.hq / p.hkv, pitch = aa_pitch(p.d);
  float* qs = aa_smem;                          // [32][pitch], scaled
  float* ks = qs + AT_QUERIES * pitch;          // [32][pitch]
  float* part = ks + AA_KEYS * pitch;           // [8 slices][32 queries][40]: scores
  float* pt = part + AT_SLICES * AT_QUERIES * AT_SPITCH;    // [32 keys][36]: weights
  const bool shared_rows = p.k_cache == p.v_cache;
  const int quads = p.d >> 2, per = (quads + AT_SLICES - 1) / AT_SLICES * 4;
  const int slice = warp & 7, half = warp >> 3;
  const int c_begin = min(p.d, slice * per), c_end = min(p.d, c_begin + per);
  const int hc = ((p.d + 31) / 32 + 3) / 4;     // of them in use
  const int group = warp >> 2, ch0 = (warp & 3) * hc * 32 + lane;
  const int ch1 = min(p.d, ch0 - lane + hc * 32);
  const bool wide_q = sizeof(T) == 4 && ((uintptr_t)p.q | (uintptr_t)(p.q_stride * 4)) % 16 == 0;
  for (int64_t it = blocks * p.hkv - 1 - blockIdx.x; it >= 0; it -= gridDim.x) {
    const int kvh = (int)(it % p.hkv);
    int64_t blk = it / p.hkv, row0, row1;
    const int seq = aa_find<AT_QUERIES>(p, grp, blk, row0, row1);
    if (seq < 0) continue;                      // uniform over the block
    const int64_t queries = (row1 - row0) * grp, q0 = blk * AT_QUERIES;
    const int live = (int)(queries - q0 < AT_QUERIES ? queries - q0 : AT_QUERIES);
    const int kv_len = p.kv_lens[seq];
    const int64_t seen0 = (int64_t)kv_len - (p.cu_q[seq + 1] - p.cu_q[seq]) + 1 - p.cu_q[seq];
    auto visible = [&](int64_t row) {
      const int64_t v = seen0 + row;
      return (int)(v < kv_len ? v : kv_len);
    };
    const int keys = visible(row0 + (q0 + live - 1) / grp);
    __syncthreads();                            // the queries before are done with
    for (int j = warp; j < AT_QUERIES; j += AT_WARPS) {
      const int64_t row = row0 + (q0 + j) / grp;
      const T* src = static_cast<const T*>(p.q) + row * p.q_stride +
                     (int64_t)(kvh * grp + (int)((q0 + j) % grp)) * p.d;
      if (lane == 0) vis_s[j] = j < live ? visible(row) : 0;
      for (int c = lane * 4; c < p.d; c += 128) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < live) {
          if (wide_q) v = Elem<T>::load4(src + c);
          else v = make_float4(Elem<T>::load(src + c), Elem<T>::load(src + c + 1),
                               Elem<T>::load(src + c + 2), Elem<T>::load(src + c + 3));
        }
        *reinterpret_cast<float4*>(qs + j * pitch + c) = v * p.scale;
      }
    }
    float m[2], l[2];                           // of queries 2 warp, 2 warp + 1
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      m[r] = -INFINITY;
      l[r] = 0.f;
    }
    uint64_t acc[4][HC];                        // pairs of queries 8 group ..
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < HC; ++i) acc[r][i] = 0ull;
    const int32_t* bt = p.block_tables + (int64_t)seq * p.bt_stride;
    auto stage = [&](const void* cache) { aa_stage<T, CH, AT_WARPS>(p, cache, key_off, ks, pitch); };
    for (int k0 = 0; k0 < keys; k0 += AA_KEYS) {
      __syncthreads();
      if (tid < AA_KEYS) {
        const int kk = k0 + tid;
        int64_t off = -1;
        if (kk < keys) {
          const int page = bt[kk / p.block_size];
          if (page < 0 || page >= p.num_blocks) {
            if (p.status) atomicOr(p.status, FK_DEV_BAD_PAGE);
          } else {
            off = (((int64_t)page * p.block_size + kk % p.block_size) * p.hkv + kvh) * p.d;
          }
        }
        key_off[tid] = off;
      }
      __syncthreads();
      stage(p.k_cache);
      __syncthreads();
      {
        // queries qg, qg + 4, ..; keys kg, kg + 8, ..
        const int qg = half * 16 + (lane >> 3), kg = lane & 7;
        uint64_t s2[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int k = 0; k < 4; ++k) s2[q][k] = 0ull;
        const float* kr = ks + kg * pitch;
        const float* qr = qs + qg * pitch;
        for (int c = c_begin; c < c_end; c += 4) {
          ulonglong2 kv[4];
#pragma unroll
          for (int k = 0; k < 4; ++k)
            kv[k] = *reinterpret_cast<const ulonglong2*>(kr + k * 8 * pitch + c);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qr + q * 4 * pitch + c);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              s2[q][k] = at_fma(kv[k].y, qv.y, at_fma(kv[k].x, qv.x, s2[q][k]));
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 v = at_unpack(s2[q][k]);
            part[(slice * AT_QUERIES + qg + q * 4) * AT_SPITCH + kg + k * 8] = v.x + v.y;
          }
      }
      __syncthreads();
      if (!shared_rows) stage(p.v_cache);
      {
        const bool there = key_off[lane] >= 0;
        float pr[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int q = warp * 2 + r;
          float s = 0.f;
#pragma unroll
          for (int w = 0; w < AT_SLICES; ++w) s += part[(w * AT_QUERIES + q) * AT_SPITCH + lane];
          if (!there || k0 + lane >= vis_s[q]) s = -INFINITY;
          float mx = s;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
          const float m_new = fmaxf(m[r], mx);
          float alpha = 1.f;
          pr[r] = 0.f;
          if (m_new != -INFINITY) {             // uniform over the warp
            alpha = expf(m[r] - m_new);
            m[r] = m_new;
            pr[r] = expf(s - m_new);
            l[r] = l[r] * alpha + warp_sum(pr[r]);
          }
          if (lane == 0) alpha_s[q] = alpha;
        }
        *reinterpret_cast<float2*>(pt + lane * AT_PPITCH + warp * 2) = make_float2(pr[0], pr[1]);
      }
      __syncthreads();
      const int first = group * 8;
      if (first >= live) continue;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 a = *reinterpret_cast<const float2*>(alpha_s + first + r * 2);
        if (a.x != 1.f || a.y != 1.f) {
#pragma unroll
          for (int i = 0; i < HC; ++i) {
            const float2 v = at_unpack(acc[r][i]);
            acc[r][i] = at_pack(v.x * a.x, v.y * a.y);
          }
        }
      }
      const int cnt = min(AA_KEYS, keys - k0);
      const int all = max(0, min(cnt, vis_s[first] - k0));      // keys that all eight see
#pragma unroll 4
      for (int j = 0; j < all; ++j) {
        const ulonglong2 pa = *reinterpret_cast<const ulonglong2*>(pt + j * AT_PPITCH + first);
        const ulonglong2 pb = *reinterpret_cast<const ulonglong2*>(pt + j * AT_PPITCH + first + 4);
#pragma unroll
        for (int i = 0; i < HC; ++i) {
          if (ch0 + i * 32 < ch1) {
            const float v = ks[j * pitch + ch0 + i * 32];
            const uint64_t vv = at_pack(v, v);
            acc[0][i] = at_fma(pa.x, vv, acc[0][i]);
            acc[1][i] = at_fma(pa.y, vv, acc[1][i]);
            acc[2][i] = at_fma(pb.x, vv, acc[2][i]);
            acc[3][i] = at_fma(pb.y, vv, acc[3][i]);
          }
        }
      }
      // what a query does not see is not multiplied by a weight of zero, it may be anything
      if (all < cnt) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int n = min(cnt, vis_s[first + r] - k0);
          for (int j = all; j < n; ++j) {
            const float pj = pt[j * AT_PPITCH + first + r];
#pragma unroll
            for (int i = 0; i < HC; ++i)
              if (ch0 + i * 32 < ch1) {
                float2 v = at_unpack(acc[r / 2][i]);
                float& x = r % 2 ? v.y : v.x;
                x = fmaf(pj, ks[j * pitch + ch0 + i * 32], x);
                acc[r / 2][i] = at_pack(v.x, v.y);
              }
          }
        }
      }
    }
    if (lane < 2) {
      const float s = lane == 0 ? l[0] : l[1];
      inv_s[warp * 2 + lane] = s > 0.f ? 1.0f / s : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int j = group * 8 + r;
      if (j >= live) break;
      const float inv = inv_s[j];
      T* o = static_cast<T*>(p.out) + (row0 + (q0 + j) / grp) * p.out_stride +
             (kvh * grp + (q0 + j) % grp) * p.d;
#pragma unroll
      for (int i = 0; i < HC; ++i) {
        const int c = ch0 + i * 32;
        const float2 v = at_unpack(acc[r / 2][i]);
        if (c < ch1) Elem<T>::store(o + c, (r % 2 ? v.y : v.x) * inv);
      }
    }
  }
}

// Blocks of qb queries at most, over all sequences of a launch
static int64_t any_blocks(const AnyAttnParams& p, int qb) {
  const int64_t queries = p.rows * (p.hq / p.hkv), most = (p.below - 1 + qb - 1) / qb;
  const int64_t all = (queries + qb - 1) / qb + p.num_seqs;
  return most < all / p.num_seqs ? most * p.num_seqs : all;
}
template <typename T, int CH>
static int launch_attn_tile(const AnyAttnParams& p, cudaStream_t s) {
  const int64_t blocks = any_blocks(p, AT_QUERIES);
  const int64_t cap = (int64_t)sm_count() * 32, want = blocks * p.hkv;
  static PerDeviceOnce once;
  FK_CUDA_OK(set_max_dynamic_smem(once, paged_attn_tile_kernel<T, CH>, AA_MAX_SMEM));
  FK_CUDA_OK(launch_kernel(paged_attn_tile_kernel<T, CH>,
                           dim3((unsigned)(want < cap ? want : cap)), dim3(AT_THREADS),
                           (size_t)at_smem(p.d), s, p, blocks));
  count_launch();
  return FK_OK;
}
template <typename T, int CH, int R>
static int launch_any_r(const AnyAttnParams& p, cudaStream_t s) {
  const int64_t blocks = any_blocks(p, AA_WARPS * R);
  const int64_t cap = (int64_t)sm_count() * 32, want = blocks * p.hkv;
  const size_t smem = ((size_t)AA_WARPS * R * p.d + AA_KEYS * aa_pitch(p.d)) * sizeof(float);
  static PerDeviceOnce once;
  FK_CUDA_OK(set_max_dynamic_smem(once, paged_attn_any_kernel<T, CH, R>, AA_MAX_SMEM));
  FK_CUDA_OK(launch_kernel(paged_attn_any_kernel<T, CH, R>,
                           dim3((unsigned)(want < cap ? want : cap)), dim3(AA_THREADS), smem, s,
                           p, blocks));
  count_launch();
  return FK_OK;
}
// Tiles or warps is chosen for each sequence by its own portion, so that a row comes out with the
// same bits whatever else is in the batch: tiles from 512 rows x query heads on, and two full ones
// a KV head, beyond 128 channels (up to there the two are too close for a second form).  Alone that
// is where they meet on short contexts; on long ones the warps, which spread over more SMs, stay
// ahead to three times as much, and in a batch the tiles are ahead from the first full one.  us,
// warps / tiles: fp32, 576 channels, 16 heads on one KV head, one portion of 32 tokens 22 / 22, 64
// 36 / 36, 128 73 / 64, 333 228 / 161; of 32 behind 300 keys 109 / 157, 128 214 / 200, 333 505 / 326;
// portions of 40, 120 and 333 271 / 160, 8 of 60 97 / 55, 16 of 20 62 / 34; 256 channels, 8 heads on
// 2, one of 64 tokens 22 / 26, 192 69 / 63, 900 436 / 267, 8 of 60 39 / 25; 192 channels, 16 KV heads,
// one of 32 15 / 16, 96 40 / 33, 900 631 / 442.
//
// Queries per warp, which change no sum's order: one while all CTAs are in the first round (or
// there are no more than eight queries to share a run of keys), then two, which halve the CTAs.
// us, one / two: 576 channels, 4 heads on one KV head, a portion of 5 tokens on 300 keys 108 / 153;
// 16 heads, 40 of them 322 / 218, one of 20 on 700 231 / 319, 8 of 31 49 / 40; 128 channels, 16 heads
// on 4, 900 tokens 394 / 299, 8 portions of 30 on 200 keys 60 / 65, 64 single tokens on 500 95 / 99;
// 64 channels, 16 KV heads, 40 portions of two tokens 53 / 89.
template <typename T, int CH>
static int launch_any_ch(AnyAttnParams p, int64_t shortest, int64_t longest, cudaStream_t s) {
  const int64_t grp = p.hq / p.hkv;
  int64_t rest = p.rows * grp;                  // queries that are left for the warps
  if constexpr (CH == 18) {
    const int64_t full = (512 + p.hkv - 1) / p.hkv;
    const int64_t least = full > 2 * AT_QUERIES ? full : 2 * AT_QUERIES;
    if (longest * grp >= least) {
      p.least = least;
      const int rc = launch_attn_tile<T, CH>(p, s);
      if (rc != FK_OK || shortest * grp >= least) return rc;
      p.least = 0;
      p.below = least;
      rest = rest < least * p.num_seqs ? rest : least * p.num_seqs;
    }
  }
  const int64_t ctas = ((rest + AA_WARPS - 1) / AA_WARPS) * p.hkv;
  if (rest <= (int64_t)AA_WARPS * p.num_seqs || ctas <= sm_count())
    return launch_any_r<T, CH, 1>(p, s);
  return launch_any_r<T, CH, 2>(p, s);
}
template <typename T>
static int launch_any(const AnyAttnParams& p, int64_t shortest, int64_t longest, cudaStream_t s) {
  if (p.d <= 64) return launch_any_ch<T, 2>(p, shortest, longest, s);
  if (p.d <= 128) return launch_any_ch<T, 4>(p, shortest, longest, s);
  if (p.d <= 576) return launch_any_ch<T, 18>(p, shortest, longest, s);
  return launch_any_r<T, 36, 1>(p, s);
}

}  // namespace fk

using namespace fk;

extern "C" {

int fk_gemm_f32(const float* x, int64_t x_stride, const float* w, const float* bias, float* y,
                int64_t y_stride, int64_t m, int64_t n, int64_t k, fk_stream_t stream) {
  FK_REQUIRE(m >= 0 && n >= 0 && k > 0, FK_ERR_INVALID_ARG, "fk_gemm_f32: bad sizes");
  if (m == 0 || n == 0) return FK_OK;
  FK_REQUIRE(x && w && y, FK_ERR_INVALID_ARG, "fk_gemm_f32: null pointer");
  FK_REQUIRE(x_stride >= k && y_stride >= n, FK_ERR_INVALID_ARG,
             "fk_gemm_f32: row stride smaller than the row");
  FK_REQUIRE(k % 4 == 0 && x_stride % 4 == 0 && aligned16(x) && aligned16(w), FK_ERR_ALIGNMENT,
             "fk_gemm_f32: x and w need 16-byte aligned rows");
  FK_REQUIRE(n < (1ll << 31) && k < (1ll << 31) && (m + 63) / 64 <= 65535,
             FK_ERR_UNSUPPORTED, "fk_gemm_f32: dimension too large");
  F32Product p{};
  p.x = x; p.x_stride = x_stride; p.w = w; p.w_rows = n; p.bias = bias; p.y = y;
  p.y_stride = y_stride; p.rows = p.x_rows = m; p.groups = 1; p.n = (int)n; p.k = (int)k;
  p.act = -1;
  return launch_f32_product(p, static_cast<cudaStream_t>(stream));
}

int fk_paged_attn_any_of(const void* q, int64_t q_stride, void* out, int64_t out_stride,
                      const void* k_cache, const void* v_cache, int is_f32, int64_t num_blocks,
                      int block_size, const int32_t* cu_seqlens_q, const int32_t* kv_lens,
                      const int32_t* block_tables, int64_t block_table_stride, int num_seqs,
                      int64_t rows, int num_q_heads, int num_kv_heads, int head_dim,
                      float softmax_scale, int64_t shortest, int64_t longest, int32_t* status,
                      fk_stream_t stream) {
  FK_REQUIRE(rows >= 0 && num_seqs >= 0 && head_dim > 0 && num_q_heads > 0 && num_kv_heads > 0,
             FK_ERR_INVALID_ARG, "fk_paged_attn_any: bad sizes");
  if (rows == 0 || num_seqs == 0) return FK_OK;
  FK_REQUIRE(q && out && k_cache && v_cache && cu_seqlens_q && kv_lens && block_tables,
             FK_ERR_INVALID_ARG, "fk_paged_attn_any: null pointer");
  FK_REQUIRE(num_q_heads % num_kv_heads == 0 && block_size > 0 && num_blocks > 0 &&
                 num_blocks < (1ll << 31) && block_table_stride > 0,
             FK_ERR_INVALID_ARG, "fk_paged_attn_any: bad sizes");
  FK_REQUIRE(head_dim % 4 == 0 && head_dim <= 1152, FK_ERR_UNSUPPORTED,
             "fk_paged_attn_any: head_dim %d must be a multiple of 4, at most 1152", head_dim);
  FK_REQUIRE(aligned16(k_cache) && aligned16(v_cache), FK_ERR_ALIGNMENT,
             "fk_paged_attn_any: caches must be 16-byte aligned");
  FK_REQUIRE(q_stride >= (int64_t)num_q_heads * head_dim &&
                 out_stride >= (int64_t)num_q_heads * head_dim,
             FK_ERR_INVALID_ARG, "fk_paged_attn_any: token stride too small");
  AnyAttnParams p{};
  p.q = q; p.q_stride = q_stride; p.out = out; p.out_stride = out_stride; p.k_cache = k_cache;
  p.v_cache = v_cache; p.cu_q = cu_seqlens_q; p.kv_lens = kv_lens; p.block_tables = block_tables;
  p.bt_stride = block_table_stride; p.num_seqs = num_seqs; p.hq = num_q_heads;
  p.hkv = num_kv_heads; p.d = head_dim; p.block_size = block_size; p.num_blocks = (int)num_blocks;
  p.rows = rows; p.scale = softmax_scale; p.status = status;
  p.below = p.rows * (num_q_heads / num_kv_heads) + 1;
  if (num_seqs == 1) shortest = longest = rows;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return is_f32 ? launch_any<float>(p, shortest, longest, s)
                : launch_any<uint16_t>(p, shortest, longest, s);
}

int fk_paged_attn_any(const void* q, int64_t q_stride, void* out, int64_t out_stride,
                      const void* k_cache, const void* v_cache, int is_f32, int64_t num_blocks,
                      int block_size, const int32_t* cu_seqlens_q, const int32_t* kv_lens,
                      const int32_t* block_tables, int64_t block_table_stride, int num_seqs,
                      int64_t rows, int num_q_heads, int num_kv_heads, int head_dim,
                      float softmax_scale, int32_t* status, fk_stream_t stream) {
  return fk_paged_attn_any_of(q, q_stride, out, out_stride, k_cache, v_cache, is_f32, num_blocks,
                              block_size, cu_seqlens_q, kv_lens, block_tables, block_table_stride,
                              num_seqs, rows, num_q_heads, num_kv_heads, head_dim, softmax_scale,
                              0, rows, status, stream);
}

}  // extern "C"

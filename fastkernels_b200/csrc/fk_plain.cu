// Kernels without shape restrictions, for the number format and the head sizes the
// tensor-core kernels do not take:
//
//   fk_gemm_f32         y = x w^T (+ bias) in true fp32 (no tensor cores, so no reduced
//                       precision), any m, n
//   fk_paged_attn_any   causal attention over the paged NHD pool, bf16 or fp32, any
//                       head size up to 1152 and any query / KV head ratio; prompt
//                       portions and single decoded tokens alike
#include "fk_f32_tile.cuh"
#include "fk_types.cuh"


namespace fk {

// ------------------------------------------------------------------- fp32 products
// Bound by the fp32 rate.  A warp computes 32 rows x 64 weight rows, a lane 8 x 8 of them, with
// the packed fma.rn.f32x2: both halves of an accumulator are the same output, over the even and
// over the odd k's, so operands come as they lie in memory (k runs along both rows) and nothing
// is packed or transposed.  Per 4 k's a lane reads 16 float4 for 256 multiply-adds; rows are
// padded to 36 floats, so the 8 rows that a quarter of a warp reads start in different banks.
// WR x WC warps make the CTA's tile; loads run kStages - 1 blocks of 32 k's ahead (cp.async).
//
// A cluster of 2 to 8 CTAs shares one tile: each takes a part of k, leaves its sums in its shared
// memory, and adds up its share of the rows over all parts in their order (f32_parts).
// 1000 rows, 24576 x 4096: 44 TFLOP/s of 72 (scalar 64 x 64 tiles 33).
template <int WR, int WC>
struct F32Tile {
  static constexpr int kRows = 32 * WR, kCols = 64 * WC, kThreads = 32 * WR * WC;
  static constexpr int kBK = 32, kPitch = kBK + 4;
  static constexpr int kStages = 3;
  static constexpr int kStageFloats = (kRows + kCols) * kPitch;
  static constexpr int kOutPitch = kCols + 8;  // lanes of a store: 4 rows x 8 columns
  static constexpr int kSmem = kStages * kStageFloats * 4;
  static_assert(kSmem % 8 == 0 && kRows * kOutPitch * 4 <= kSmem, "sums take the place of the operands");
};

__device__ __forceinline__ void fma_f32x2(float2& c, float ax, float ay, float bx, float by) {
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "mov.b64 c, {%0, %1};\n\tfma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "+f"(c.x), "+f"(c.y)
      : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, int rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
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

template <int WR, int WC, bool ACT>
__global__ void __launch_bounds__(32 * WR * WC, WR * WC == 8 ? 1 : 2)
    f32_product_kernel(const F32Product p, int parts, int64_t row_tiles) {
  using Tile = F32Tile<WR, WC>;
  extern __shared__ __align__(16) float f32_smem[];
  constexpr int kLoads = (Tile::kRows + Tile::kCols) * (Tile::kBK / 4) / Tile::kThreads;
  __shared__ const float* f32_rows[Tile::kRows + Tile::kCols];
  constexpr int kOut = ACT ? Tile::kCols / 2 : Tile::kCols;     // outputs a row
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = lane >> 3, tx = lane & 7, wr = warp / WC, wc = warp % WC;
  const int part = (int)(blockIdx.x % parts);
  const int n0 = (int)(blockIdx.x / parts) * kOut;
  const int blocks_all = (p.k + Tile::kBK - 1) / Tile::kBK;
  const int first_block = (int)((int64_t)blocks_all * part / parts);
  const int blocks = (int)((int64_t)blocks_all * (part + 1) / parts) - first_block;
  const int c4 = (tid & 7) * 4;                 // 8 threads a row of a block
  for (int64_t t = blockIdx.y; t < row_tiles; t += gridDim.y) {
    int g = blockIdx.z;
    int64_t m0 = t * Tile::kRows, first = 0, count = p.rows;
    if (p.offsets) {
      if (!f32_row_tile(p, Tile::kRows, t, &g, &m0)) return;    // uniform over the cluster
      first = p.offsets[g];
      count = p.offsets[g + 1] - first;
    }
    const float* x = p.x + (p.offsets ? 0 : g * p.x_group);
    const float* w = p.w + (int64_t)g * p.w_rows * p.k;
    // addresses of the tile's rows, null where there is none (in registers they would spill)
    for (int r = tid; r < Tile::kRows + Tile::kCols; r += Tile::kThreads) {
      const float* src = nullptr;
      if (r < Tile::kRows) {
        if (m0 + r < count) {
          int64_t xr = first + m0 + r;
          if (p.gather) {
            xr = p.gather[xr];
            if (xr < 0 || xr >= p.x_rows) {
              if (p.status) atomicOr(p.status, FK_DEV_BAD_SLOT);
              xr = 0;
            }
          }
          src = x + xr * p.x_stride;
        }
      } else {
        // with an activation 32 of a warp's 64 columns are gate rows, 32 the up rows of the
        // same outputs
        const int c = r - Tile::kRows;
        const int wrow = n0 + (ACT ? (c >> 6) * 32 + (c & 31) : c);
        if (wrow < p.n) src = w + (int64_t)(wrow + (ACT && (c & 32) ? p.n : 0)) * p.k;
      }
      f32_rows[r] = src;
    }
    __syncthreads();
    auto load = [&](int stage, int block) {
      const int k0 = (first_block + block) * Tile::kBK + c4;
      float* dst = f32_smem + stage * Tile::kStageFloats + (tid >> 3) * Tile::kPitch + c4;
#pragma unroll
      for (int i = 0; i < kLoads; ++i) {
        const float* src = f32_rows[(tid >> 3) + i * (Tile::kThreads / 8)];
        const bool ok = src != nullptr && k0 < p.k;
        const uint32_t bytes = ok ? 16u : 0u;   // the rest is filled with zeros
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         smem_u32(dst + i * (Tile::kThreads / 8) * Tile::kPitch)),
                     "l"(ok ? src + k0 : p.w), "r"(bytes)
                     : "memory");
      }
    };
    float2 acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < Tile::kStages - 1; ++s) {
      if (s < blocks) load(s, s);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0;
    for (int b = 0; b < blocks; ++b) {
      asm volatile("cp.async.wait_group %0;" ::"n"(Tile::kStages - 2) : "memory");
      __syncthreads();
      const int ahead = b + Tile::kStages - 1;
      if (ahead < blocks) load(stage == 0 ? Tile::kStages - 1 : stage - 1, ahead);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const float* xs = f32_smem + stage * Tile::kStageFloats + (wr * 32 + ty) * Tile::kPitch;
      const float* ws = f32_smem + stage * Tile::kStageFloats +
                        (Tile::kRows + wc * 64 + tx) * Tile::kPitch;
#pragma unroll
      for (int kk = 0; kk < Tile::kBK; kk += 4) {
        float4 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          a[i] = *reinterpret_cast<const float4*>(xs + i * 4 * Tile::kPitch + kk);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(ws + j * 8 * Tile::kPitch + kk);
#pragma unroll
          for (int i = 0; i < 8; ++i) fma_f32x2(acc[i][j], a[i].x, a[i].y, v.x, v.y);
#pragma unroll
          for (int i = 0; i < 8; ++i) fma_f32x2(acc[i][j], a[i].z, a[i].w, v.z, v.w);
        }
      }
      if (++stage == Tile::kStages) stage = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        f32_smem[(wr * 32 + i * 4 + ty) * Tile::kOutPitch + wc * 64 + j * 8 + tx] =
            acc[i][j].x + acc[i][j].y;
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int live = (int)(count - m0 < Tile::kRows ? count - m0 : Tile::kRows);
    const int r0 = live * part / parts, r1 = live * (part + 1) / parts;
    float* y = p.y + (p.offsets ? 0 : g * p.y_group);
    auto sum = [&](int r, int c) {
      const int at = r * Tile::kOutPitch + c;
      const uint32_t addr = smem_u32(f32_smem + at);
      float v = ld_cluster_f32(addr, 0);
      for (int q = 1; q < parts; ++q) v += ld_cluster_f32(addr, q);
      return v;
    };
    for (int i = r0 * kOut + tid; i < r1 * kOut; i += Tile::kThreads) {
      const int r = i / kOut, c = i % kOut;
      if (n0 + c >= p.n) continue;
      float v;
      if (ACT) {
        const int col = (c >> 5) * 64 + (c & 31);
        const float gate = sum(r, col) + (p.bias ? p.bias[n0 + c] : 0.f);
        const float up = sum(r, col + 32) + (p.bias ? p.bias[p.n + n0 + c] : 0.f);
        v = (p.act == FK_ACT_SILU ? gate * sigmoid_f32(gate) : gelu_tanh_f32(gate)) * up;
      } else {
        v = sum(r, c) + (p.bias ? p.bias[n0 + c] : 0.f);
      }
      y[(first + m0 + r) * p.y_stride + n0 + c] = v;
    }
    // peers may still read this CTA's sums; the next tile overwrites them
    __syncwarp();                      // lanes stored different numbers of outputs
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// Short k: the tiles above spend their time filling the ring and handing sums on.  64 x 64
// outputs, 4 x 4 a thread, k in one order.  us, 60 / 200 / 1000 rows, here and in the tiles above:
// 16 heads of 96 -> 512 8 21 55 (18 21 80), 40 of 256 -> 64 15 35 50 (17 38 108 in one part),
// 12288 x 256 34 58 196 (35 65 213; one row 31 and 21).
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
// rows are in the call (tiles of every height add up k alike).  Few weight tiles get more parts, so
// that few rows find SMs; many rows would have them anyway and pay for the exchange.  us, rows 1 /
// 100 / 500 / 1000, k 2048 unless said, in 2, 4 and 8 parts (scalar 64 x 64 tiles):
//   n 544            67 115 118 120     36 61 64 123       21 34 68 102       (94 98 99 193)
//   n 2048           67 113 118 231     36 61 123 244      21 66 168 302      (94 99 278 297)
//   n 4096, k 4096   131 216 436 869    93 112 451 898     58 175 534 1063    (213 353 604 1043)
//   n 6144           78 116 347 685     54 120 366 729     32 131 437 871     (126 198 441 797)
//   n 4352           68 114 230 458     40 119 303 544     32 99 333 633      (95 199 297 580)
// 32 experts, 2 x 1024 x 2048, 4 / 60 / 400 / 3100 rows in all: 70 201 239 753, 59 207 257 808,
// 51 234 299 936 (243 364 632 999).
static int f32_parts(const F32Product& p) {
  const int64_t tiles = (p.w_rows + 127) / 128 * p.groups;
  return tiles <= 12 && p.k >= 2048 ? 8 : tiles <= 32 && p.k >= 1024 ? 4 : 2;
}

template <int WR, int WC, bool ACT>
static int launch_f32_tile(const F32Product& p, cudaStream_t s) {
  using Tile = F32Tile<WR, WC>;
  constexpr int kOut = ACT ? Tile::kCols / 2 : Tile::kCols;
  const int64_t n_tiles = (p.n + kOut - 1) / kOut;
  const int64_t upto = (p.rows + Tile::kRows - 1) / Tile::kRows;
  // row groups: at most one part-filled tile a group
  const int64_t used = p.rows < p.groups ? p.rows : p.groups;
  const int64_t row_tiles = p.offsets ? upto + used : upto;
  const int parts = f32_parts(p);
  static PerDeviceOnce once;
  FK_CUDA_OK(set_max_dynamic_smem(once, f32_product_kernel<WR, WC, ACT>, Tile::kSmem));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n_tiles * parts), (unsigned)(row_tiles < 65535 ? row_tiles : 65535),
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
  FK_CUDA_OK(cudaLaunchKernelEx(&cfg, f32_product_kernel<WR, WC, ACT>, p, parts, row_tiles));
  count_launch();
  return FK_OK;
}

// Row tiles of 32, 64 or 128: the smallest that holds the rows; row groups take 64 up to three
// tiles on average, since their last tile is half empty.
template <bool ACT>
static int launch_f32(const F32Product& p, int64_t expect, cudaStream_t s) {
  if (p.k <= FS_MAX_K) return launch_f32_short<ACT>(p, s);
  if (expect <= 32) return launch_f32_tile<1, 2, ACT>(p, s);
  if (expect <= 64 || (p.offsets && expect <= 192)) return launch_f32_tile<2, 2, ACT>(p, s);
  return launch_f32_tile<4, 2, ACT>(p, s);
}
int launch_f32_product(const F32Product& p, int64_t expect, cudaStream_t s) {
  return p.act >= 0 ? launch_f32<true>(p, expect, s) : launch_f32<false>(p, expect, s);
}

// ----------------------------------------------------------------------- attention
struct AnyAttnParams {
  const void* q; int64_t q_stride; void* out; int64_t out_stride;
  const void* k_cache; const void* v_cache;
  const int32_t* cu_q; const int32_t* kv_lens;
  const int32_t* block_tables; int64_t bt_stride;
  int num_seqs, hq, hkv, d, block_size, num_blocks;
  int64_t rows;
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
    // the sequence of block `blk`; every warp finds it by itself
    int seq = -1;
    int64_t row0 = 0, row1 = 0;
    for (int s0 = 0; s0 < p.num_seqs && seq < 0; s0 += 32) {
      const int sq = s0 + lane;
      int64_t a = 0, b = 0;
      if (sq < p.num_seqs) {
        a = sq == 0 ? 0 : p.cu_q[sq];
        b = sq == p.num_seqs - 1 ? p.rows : p.cu_q[sq + 1];
        a = a < 0 ? 0 : a;
        b = b > p.rows ? p.rows : b;
      }
      const int64_t mine = b > a ? ((b - a) * grp + QB - 1) / QB : 0;
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
    // rows of one run of keys; keys that are not there are rows of zeros
    auto stage = [&](const void* cache) {
      const int quads = p.d >> 2;
      for (int j = warp; j < AA_KEYS; j += AA_WARPS) {
        const int64_t off = key_off[j];
        const T* src = static_cast<const T*>(cache) + off;
        for (int c = lane; c < quads; c += 32)
          *reinterpret_cast<float4*>(ks + j * pitch + c * 4) =
              off < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : Elem<T>::load4(src + c * 4);
      }
    };
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

template <typename T, int CH, int R>
static int launch_any_r(const AnyAttnParams& p, cudaStream_t s) {
  const int64_t queries = p.rows * (p.hq / p.hkv);
  const int64_t blocks = (queries + AA_WARPS * R - 1) / (AA_WARPS * R) + p.num_seqs;
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
// Queries per warp: one while all CTAs are in the first round (or there are no more than eight
// queries to share a run of keys), then two, which halve the CTAs for 5 to 10 % more time each.
// Four, in keys of 576 channels, leave one CTA an SM and were behind at every size.  us, one / two /
// four a warp (and a warp per query that reads its keys from L2): fp32, 576 channels, 4 heads on one
// KV head, a portion of 5 tokens on 300 keys 131 / 135 / 252 (196); 16 heads, 40 portions of 5
// 342 / 203 / 232 (1143); one of 900 tokens 1633 / 1031 / 1306 (5827); 128 channels, 16 heads on 4,
// 64 single tokens on 500 keys 142 / 141 / 145 (346); 64 channels, 16 KV heads, 40 portions of two
// tokens 72 / 134 / 204 (156).
template <typename T, int CH>
static int launch_any_ch(const AnyAttnParams& p, cudaStream_t s) {
  const int64_t queries = p.rows * (p.hq / p.hkv);
  const int64_t ctas = ((queries + AA_WARPS - 1) / AA_WARPS) * p.hkv;
  if (queries <= (int64_t)AA_WARPS * p.num_seqs || ctas <= sm_count())
    return launch_any_r<T, CH, 1>(p, s);
  return launch_any_r<T, CH, 2>(p, s);
}
template <typename T>
static int launch_any(const AnyAttnParams& p, cudaStream_t s) {
  if (p.d <= 64) return launch_any_ch<T, 2>(p, s);
  if (p.d <= 128) return launch_any_ch<T, 4>(p, s);
  if (p.d <= 576) return launch_any_ch<T, 18>(p, s);
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
  return launch_f32_product(p, m, static_cast<cudaStream_t>(stream));
}

int fk_paged_attn_any(const void* q, int64_t q_stride, void* out, int64_t out_stride,
                      const void* k_cache, const void* v_cache, int is_f32, int64_t num_blocks,
                      int block_size, const int32_t* cu_seqlens_q, const int32_t* kv_lens,
                      const int32_t* block_tables, int64_t block_table_stride, int num_seqs,
                      int64_t rows, int num_q_heads, int num_kv_heads, int head_dim,
                      float softmax_scale, int32_t* status, fk_stream_t stream) {
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
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return is_f32 ? launch_any<float>(p, s) : launch_any<uint16_t>(p, s);
}

}  // extern "C"

// Generalized delta rule with a decay per key channel (linear attention with a
// matrix state per head), fp32 throughout:
//
//   S_t = diag(w_t) S_{t-1} - (a_t * u_t) (u_t^T S_{t-1}) + k_t v_t^T,   o_t = S_t^T r_t
//
//   w_t = exp(-c sigmoid(W2 tanh(y1) + w0)),  a_t = sigmoid(y_a + b_a),
//   u_t = k_t / sqrt(sum k_t^2 + eps_u)       (per head)
//
// Kernels:
//   delta_prepare_kernel        everything of a token that does not depend on the state:
//                               w, u, b = a * u, k, r, v as fp32, packed per (head, token);
//                               for portions in blocks of 4 or chunks of 16 tokens, with
//                               what their tokens do to one another worked out (below)
//   delta_scan_kernel           the recurrence, token by token: single tokens, bound by
//                               the state's bytes
//   delta_scan_blocked_kernel   the recurrence over blocks, for portions
//   delta_scan_chunk_kernel     the recurrence over chunks, for portions in bf16 with heads
//                               of 33 to 128 channels
//
// The columns of S (value channels) are independent, so a column lives in the registers
// of LANES threads; a CTA owns some columns of one head of one sequence.  The state comes
// from and returns to HBM once per call, as [slot][head][value channel][key channel
// (padded)], so that the threads of a column read 16-byte pieces adjacent across lanes.
//
// Blocks.  With S the state ahead of a block, its tokens 1..4 and w_{j..i} = w_j ... w_i
// (elementwise):
//
//   p_i = u_i^T S_{i-1} = (u_i w_{1..i-1})^T S + sum_{j<i} A_ij v_j - C_ij p_j
//   o_i = S_i^T r_i     = (r_i w_{1..i})^T S   + sum_{j<=i} E_ij v_j - F_ij p_j
//   S_4 = w_{1..4} S + sum_j (k_j w_{j+1..4}) v_j^T - (b_j w_{j+1..4}) p_j^T
//   A_ij = u_i . (k_j w_{j+1..i-1}),  C: b for k,   E_ij = r_i . (k_j w_{j+1..i}),  F: b for k
//
// so a block has ONE reduction over a column's lanes on its critical path instead of
// four, and nothing is divided by a decay.  Missing tokens of a portion's last block are
// w = 1 and zeros.  A block is 21 dp + 48 floats:
//   u_i w_{1..i-1} [4][dp] | k_j w_{j+1..4} | -b_j w_{j+1..4} | r_i w_{1..i} | v_i |
//   w_{1..4} [dp] | A (6) C (6) pad (4) | E [4][4] | F [4][4]
// Blocks come in units of 16 tokens; portion i owns the units from cu[i] / 16 + i on.
//
// Chunks.  The same over 16 tokens, where every sum over channels or tokens is a 16 x 16 x n
// product for mma; that leaves the state's multiply-adds (four a channel, value channel and token)
// to the tensor cores.  Five portions of 700 to 2400 tokens, us of prepare / scan, blocks and then
// chunks: 64 heads of 64 370 / 1174 and 538 / 388, 24 heads of 128 275 / 1311 and 470 / 520; one of
// 1500, 32 heads of 64 59 / 280 and 79 / 167; 60 of 24 77 / 73 and 101 / 68, of 3 46 / 27 and
// 60 / 51, so that portions below 32 tokens stay with blocks, each by its own length: a row comes out
// with the same bits whatever else is in the batch.  Error of o against 64
// bits, of the norm: 2.0 to 2.6e-7 (5.4e-7 with decays that forget nothing in 1500 tokens), blocks
// 2.7e-7 to 1.6e-6, most of it the decays' (decay_of).
#include "fk_types.cuh"

#include <cmath>

namespace fk {

constexpr int DL_FIELDS = 6;      // w, u, a * u, k, r, v
constexpr int DL_UNIT = 16;       // tokens per CTA of the prepare kernel
constexpr int DL_BLK = 4;         // tokens per block
constexpr int DL_STAGES = 3;
constexpr int DL_STAGE_BLOCKS = 2;
constexpr int DL_MAX_DIM = 256;
constexpr int DL_THREADS = 128;
constexpr int DL_CHUNKS_FROM = 32;   // tokens of a portion that goes in chunks
constexpr uint32_t DL_WAIT_LIMIT = 1u << 20;
__host__ __device__ constexpr int dl_block_floats(int dp) { return 21 * dp + 48; }

// A chunk's record, in bytes: four operands of [16 tokens][dp], four of [16][16], each in three
// bf16 parts and the order of mma fragments; v in one part; w_{1..16} in fp32; a flag.
constexpr int DL_FRAG = 512;      // a 16 x 16 piece of one part: 16 bytes a lane
__host__ __device__ constexpr int dl_chunk_mats(int dp) { return 4 * (dp / 16) * 3 * DL_FRAG; }
__host__ __device__ constexpr int dl_chunk_v(int dp) { return dl_chunk_mats(dp) + 4 * 3 * DL_FRAG; }
__host__ __device__ constexpr int dl_chunk_decay(int dp) { return dl_chunk_v(dp) + dp / 16 * DL_FRAG; }
__host__ __device__ constexpr int dl_chunk_flag(int dp) { return dl_chunk_decay(dp) + dp * 4; }
__host__ __device__ constexpr int dl_chunk_bytes(int dp) { return dl_chunk_flag(dp) + 16; }
__host__ __device__ constexpr int dl_chunk_stages(int dp) { return dp == 64 ? 3 : 2; }
static_assert(dl_chunk_flag(64) >= DL_FIELDS * DL_UNIT * 64 * 4 &&
              dl_chunk_flag(128) >= DL_FIELDS * DL_UNIT * 128 * 4, "a plain record fits");

// Packed pairs of fp32: one instruction, two IEEE multiply-adds.
__device__ __forceinline__ uint64_t dl_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void dl_unpack(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t dl_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t dl_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Two fp32 as three packed bf16 pairs: x = hi + mid + lo up to 2^-25 |x|.
__device__ __forceinline__ void dl_split(float a, float b, uint32_t& hi, uint32_t& mid,
                                         uint32_t& lo) {
  auto pack = [](float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
  };
  const uint64_t minus = dl_pack(-1.f, -1.f);
  hi = pack(a, b);
  dl_unpack(dl_fma(dl_pack(bf16lo(hi), bf16hi(hi)), minus, dl_pack(a, b)), a, b);
  mid = pack(a, b);
  dl_unpack(dl_fma(dl_pack(bf16lo(mid), bf16hi(mid)), minus, dl_pack(a, b)), a, b);
  lo = pack(a, b);
}

struct DeltaPrepParams {
  const void* r; const void* k; const void* v; const void* a; const void* y1;
  int64_t in_stride;                    // packed projection rows
  const void* w2; int64_t w2_stride;    // [heads * d, rank]
  const float* w0; const float* a_bias; // [heads * d]
  float* packed;
  const int32_t* cu; int num_portions;  // blocks only
  int least, below;                     // portions of least .. below - 1 tokens are taken
  int64_t rows, units; int heads, d, rank, rank_p, heads_per_cta;
  float decay_scale, unit_eps;
};

// fp32 exponential and sigmoid: the hardware approximations (relative error around
// 1e-6) beside bf16 operands, the accurate functions beside fp32 ones.
template <typename T>
struct Gate {
  static __device__ __forceinline__ float exp(float x) { return sizeof(T) == 2 ? __expf(x) : expf(x); }
  static __device__ __forceinline__ float sigmoid(float z) {
    return sizeof(T) == 2 ? __fdividef(1.0f, 1.0f + __expf(-z)) : sigmoid_f32(z);
  }
};

// A decay's error is that of every later token.  Chunks: e^x as 1 + x (1 + x/2 (1 + x/3 ...)),
// Taylor's series up to x^10, rounded once at the end (0.7^11 / 11! < 2^-30), where the hardware's
// approximation is off by 2 units in the last place.
template <typename T, bool CHUNK>
__device__ __forceinline__ float decay_of(float x) {
  if (!CHUNK) return Gate<T>::exp(x);
  if (!(fabsf(x) <= 0.7f)) return expf(x);
  float y = fmaf(x, 1.f / 10, 1.f);
#pragma unroll
  for (int i = 9; i > 1; --i) y = fmaf(x * (1.f / i), y, 1.f);
  return fmaf(x, y, 1.f);
}

// The record of one chunk from its operands vec [6][16][DP + 4] (w, u, b, k, r, v; overwritten),
// by all threads of a CTA.  mats [4][16][16] is zero on entry.
//
// A warp first takes the 4 tokens of a block as for blocks (the sums over the channels of what its
// tokens do to one another); then a thread takes the four sums of one pair of tokens of different
// blocks, whose operands carry the decays inside their blocks and are a product of whole blocks'
// decays apart.  (I + C)^-1 is a product of contractions: no entry exceeds 1.
template <int DP>
__device__ void delta_chunk_record(float* vec, float* mats, uint8_t* rec) {
  constexpr int VP = DP + 4, F = DL_UNIT * VP, KT = DP / 16;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* ma = mats;              // A [i][j]
  float* mc = mats + 256;        // C [j][i], then (I + C)^-1 [i][j]
  float* me = mats + 512;        // E [i][j]
  float* mf = mats + 768;        // F [i][j]
  {
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
#pragma unroll
    for (int c0 = 0; c0 < DP; c0 += 32) {
      float* src = vec + warp * DL_BLK * VP + c0 + lane;
      float kk[DL_BLK], bb[DL_BLK], gam = 1.f;
#pragma unroll
      for (int i = 0; i < DL_BLK; ++i) {
        const int ia = i * (i - 1) / 2, ie = 12 + i * (i + 1) / 2;
        float* s = src + i * VP;
        const float w = s[0], u = s[F], r = s[4 * F];
#pragma unroll
        for (int j = 0; j < i; ++j) {
          acc[ia + j] = fmaf(u, kk[j], acc[ia + j]);
          acc[6 + ia + j] = fmaf(u, bb[j], acc[6 + ia + j]);
          kk[j] *= w;
          bb[j] *= w;
        }
        bb[i] = s[2 * F];
        kk[i] = s[3 * F];
#pragma unroll
        for (int j = 0; j <= i; ++j) {
          acc[ie + j] = fmaf(r, kk[j], acc[ie + j]);
          acc[10 + ie + j] = fmaf(r, bb[j], acc[10 + ie + j]);
        }
        s[F] = u * gam;
        gam *= w;
        s[4 * F] = r * gam;
      }
      src[0] = gam;              // of the whole block; the row behind it: one
      src[VP] = 1.f;
#pragma unroll
      for (int j = 0; j < DL_BLK; ++j) {
        src[j * VP + 3 * F] = kk[j];
        src[j * VP + 2 * F] = bb[j];
      }
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
      const bool up = (lane & w) != 0;
#pragma unroll
      for (int i = 0; i < w; ++i) {
        const float keep = up ? acc[i + w] : acc[i];
        const float give = up ? acc[i] : acc[i + w];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, w);
      }
    }
    const int t = lane < 12 ? lane % 6 : (lane - 12) % 10;
    const int tri = t < 1 ? 0 : t < 3 ? 1 : t < 6 ? 2 : 3;
    const int j = t - tri * (tri + 1) / 2 + warp * DL_BLK;
    const int i = warp * DL_BLK + tri + (lane < 12 ? 1 : 0);
    if (lane < 6) ma[i * 16 + j] = acc[0];
    else if (lane < 12) mc[j * 16 + i] = acc[0];
    else if (lane < 22) me[i * 16 + j] = acc[0];
    else mf[i * 16 + j] = -acc[0];
  }
  __syncthreads();
  if (threadIdx.x < 96) {
    const int pair = threadIdx.x >> 4;                 // (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
    const int bi = pair < 1 ? 1 : pair < 3 ? 2 : 3, bj = pair - bi * (bi - 1) / 2;
    const int i = bi * DL_BLK + ((threadIdx.x >> 2) & 3), j = bj * DL_BLK + (threadIdx.x & 3);
    const float* g1 = vec + (bi > 1 && bj < 1 ? DL_BLK : 1) * VP;        // blocks between
    const float* g2 = vec + (bi > 2 && bj < 2 ? 2 * DL_BLK : 1) * VP;
    const float* u = vec + F + i * VP;
    const float* r = vec + 4 * F + i * VP;
    const float* k = vec + 3 * F + j * VP;
    const float* b = vec + 2 * F + j * VP;
    uint64_t sum[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 4
    for (int x = 0; x < DP / 4; ++x) {
      const int at = x * 4;
      const ulonglong2 uu = *reinterpret_cast<const ulonglong2*>(u + at);
      const ulonglong2 rr = *reinterpret_cast<const ulonglong2*>(r + at);
      ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(k + at);
      ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(b + at);
      ulonglong2 gg = *reinterpret_cast<const ulonglong2*>(g1 + at);
      const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(g2 + at);
      gg.x = dl_mul(gg.x, x2.x);
      gg.y = dl_mul(gg.y, x2.y);
      kk.x = dl_mul(kk.x, gg.x);
      kk.y = dl_mul(kk.y, gg.y);
      bb.x = dl_mul(bb.x, gg.x);
      bb.y = dl_mul(bb.y, gg.y);
      sum[0] = dl_fma(uu.y, kk.y, dl_fma(uu.x, kk.x, sum[0]));
      sum[1] = dl_fma(uu.y, bb.y, dl_fma(uu.x, bb.x, sum[1]));
      sum[2] = dl_fma(rr.y, kk.y, dl_fma(rr.x, kk.x, sum[2]));
      sum[3] = dl_fma(rr.y, bb.y, dl_fma(rr.x, bb.x, sum[3]));
    }
    auto both = [](uint64_t v) {
      float x, y;
      dl_unpack(v, x, y);
      return x + y;
    };
    ma[i * 16 + j] = both(sum[0]);
    mc[j * 16 + i] = both(sum[1]);
    me[i * 16 + j] = both(sum[2]);
    mf[i * 16 + j] = -both(sum[3]);
  }
  __syncthreads();
  const int g = lane >> 2, q2 = (lane & 3) * 2;
  auto put = [&](int at, float2 x0, float2 x1, float2 x2, float2 x3, float sign) {
    uint4 hi, mid, lo;
    dl_split(x0.x * sign, x0.y * sign, hi.x, mid.x, lo.x);
    dl_split(x1.x * sign, x1.y * sign, hi.y, mid.y, lo.y);
    dl_split(x2.x * sign, x2.y * sign, hi.z, mid.z, lo.z);
    dl_split(x3.x * sign, x3.y * sign, hi.w, mid.w, lo.w);
    uint4* dst = reinterpret_cast<uint4*>(rec + at) + lane;
    dst[0] = hi;
    dst[DL_FRAG / 16] = mid;
    dst[2 * (DL_FRAG / 16)] = lo;
  };
  auto decay = [&](int blk, int c) { return vec[blk * DL_BLK * VP + c]; };
  // u and r: a lane's channels of tokens g and g + 8, decayed from the chunk's start
  for (int kt = warp; kt < KT; kt += DL_THREADS / 32) {
    float2 f0[2], f1[2];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      float lo[2], hi[2];
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int c = kt * 16 + hf * 8 + q2 + y;
        const float d0 = decay(0, c), d1 = decay(1, c), d2 = decay(2, c);
        lo[y] = g < DL_BLK ? 1.f : d0;
        hi[y] = g < DL_BLK ? d0 * d1 : d0 * d1 * d2;
      }
      f0[hf] = make_float2(lo[0], lo[1]);
      f1[hf] = make_float2(hi[0], hi[1]);
    }
#pragma unroll
    for (int op = 0; op < 2; ++op) {
      const float* src = vec + (op == 0 ? 1 : 4) * F + kt * 16 + q2;
      float2 x[4];
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const float2 z = *reinterpret_cast<const float2*>(src + (g + y / 2 * 8) * VP + y % 2 * 8);
        const float2 f = y < 2 ? f0[y] : f1[y - 2];
        x[y] = make_float2(z.x * f.x, z.y * f.y);
      }
      put((op * KT + kt) * 3 * DL_FRAG, x[0], x[1], x[2], x[3], 1.f);
    }
  }
  // k and -b: a lane's tokens of channels g and g + 8, decayed to the chunk's end; v as it is
  for (int kt = warp; kt < KT; kt += DL_THREADS / 32) {
    const int c = kt * 16 + g;
    float f[2][2];                       // [channel][tokens 2 q2 .. / 8 + 2 q2 ..]
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const float d1 = decay(1, c + y * 8), d2 = decay(2, c + y * 8), d3 = decay(3, c + y * 8);
      f[y][0] = q2 < DL_BLK ? d1 * d2 * d3 : d2 * d3;
      f[y][1] = q2 < DL_BLK ? d3 : 1.f;
    }
#pragma unroll
    for (int op = 0; op < 2; ++op) {
      const float* src = vec + (op == 0 ? 3 : 2) * F + c;
      float2 x[4];
#pragma unroll
      for (int y = 0; y < 4; ++y) {      // channel y / 2, token half y % 2
        const float* at = src + (q2 + y % 2 * 8) * VP + y / 2 * 8;
        x[y] = make_float2(at[0] * f[y / 2][y % 2], at[VP] * f[y / 2][y % 2]);
      }
      put(((2 + op) * KT + kt) * 3 * DL_FRAG, x[0], x[1], x[2], x[3], op == 0 ? 1.f : -1.f);
    }
    const float* sv = vec + 5 * F + c;
    uint32_t vv[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) {        // rows g, g + 8; then tokens from 8 on
      const float* at = sv + (q2 + y / 2 * 8) * VP + y % 2 * 8;
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(vv[y]) : "f"(at[VP]), "f"(at[0]));
    }
    reinterpret_cast<uint4*>(rec + dl_chunk_v(DP))[kt * 32 + lane] =
        make_uint4(vv[0], vv[1], vv[2], vv[3]);
  }
  for (int c = threadIdx.x; c < DP; c += DL_THREADS)
    reinterpret_cast<float*>(rec + dl_chunk_decay(DP))[c] =
        decay(0, c) * decay(1, c) * (decay(2, c) * decay(3, c));
  if (warp == 3) {
    // (I + C)^-1, a column a lane: what is known of it goes into all rows below at once
    float x[16];
    const int col = lane & 15;
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = i == col ? 1.f : 0.f;
#pragma unroll
    for (int k = 0; k < 15; ++k) {
      float row[16];
#pragma unroll
      for (int y = k / 4 * 4; y < 16; y += 4) {
        const float4 z = *reinterpret_cast<const float4*>(mc + k * 16 + y);
        row[y] = z.x;
        row[y + 1] = z.y;
        row[y + 2] = z.z;
        row[y + 3] = z.w;
      }
#pragma unroll
      for (int i = k + 1; i < 16; ++i) x[i] = fmaf(-row[i], x[k], x[i]);
    }
    __syncwarp();
    if (lane < 16)
#pragma unroll
      for (int i = 0; i < 16; ++i) mc[i * 16 + col] = x[i];
  }
  __syncthreads();
  {
    const float* m = mats + warp * 256;
    float2 x[4];
#pragma unroll
    for (int y = 0; y < 4; ++y)
      x[y] = *reinterpret_cast<const float2*>(m + (g + y / 2 * 8) * 16 + q2 + y % 2 * 8);
    put(dl_chunk_mats(DP) + warp * 3 * DL_FRAG, x[0], x[1], x[2], x[3], 1.f);
  }
}

// CTA = 16 tokens, some heads in turn.  VEC (bf16, rows of whole 16-byte pieces): a thread takes
// 8 channels of a token, one 16-byte load per input, all requested before the decay projection
// (the first head's before the tanh too); the sum of k^2 stays within the lanes of the token.
template <typename T, int DP, bool BLOCKED, bool VEC, bool CHUNK>
__global__ void __launch_bounds__(DL_THREADS, !CHUNK ? 0 : DP == 64 ? 6 : 4)
delta_prepare_kernel(const DeltaPrepParams p) {
  extern __shared__ __align__(16) uint8_t dl_prep_smem[];
  pdl_launch_dependents();
  if (VEC && !BLOCKED) {
    // a decode step finds the decay projection's weights in HBM: towards L2 while the kernel
    // in front still runs
    const char* w2 = reinterpret_cast<const char*>(
        static_cast<const T*>(p.w2) + (int64_t)blockIdx.y * p.heads_per_cta * p.d * p.w2_stride);
    const int heads = min(p.heads_per_cta, p.heads - (int)blockIdx.y * p.heads_per_cta);
    const int64_t bytes = (int64_t)heads * p.d * p.w2_stride * (int64_t)sizeof(T);
    for (int64_t i = (int64_t)threadIdx.x * 128; i < bytes; i += DL_THREADS * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(w2 + i));
  }
  pdl_wait();
  constexpr bool MMA = sizeof(T) == 2;
  constexpr int VP = CHUNK ? DP + 4 : DP;      // fragments read 8 rows at a time
  constexpr int NW = DL_THREADS / 32;
  int64_t t0 = (int64_t)blockIdx.x * DL_UNIT;
  int nt = (int)min((int64_t)DL_UNIT, p.rows - t0);
  if (BLOCKED) {
    int lo_i = 0, hi_i = p.num_portions;
    while (hi_i - lo_i > 1) {
      const int mid = (lo_i + hi_i) >> 1;
      if (p.cu[mid] / DL_UNIT + mid <= (int)blockIdx.x) lo_i = mid; else hi_i = mid;
    }
    t0 = p.cu[lo_i] + (int64_t)((int)blockIdx.x - (p.cu[lo_i] / DL_UNIT + lo_i)) * DL_UNIT;
    const int n = p.cu[lo_i + 1] - p.cu[lo_i];
    nt = n < p.least || n >= p.below ? 0
                                     : (int)min((int64_t)DL_UNIT, (int64_t)p.cu[lo_i + 1] - t0);
  }
  if (nt <= 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // tanh(y1): bf16 in two parts (w2 is bf16 to begin with, so the tensor cores keep 16
  // bits of the fp32 value and accumulate in fp32), fp32 as it is.  Rows of 16-bit
  // elements are padded by 8 so that fragment loads hit different banks.
  const int rank_p = p.rank_p, ld = rank_p + 8;
  uint16_t* hi = reinterpret_cast<uint16_t*>(dl_prep_smem);      // [16][ld] each
  uint16_t* lo = hi + DL_UNIT * ld;
  float* th = reinterpret_cast<float*>(dl_prep_smem);            // fp32: [16][rank_p]
  float* vec = reinterpret_cast<float*>(dl_prep_smem) + DL_UNIT * ld;   // [6][16][VP]
  float* part = vec + DL_FIELDS * DL_UNIT * VP;                  // [16][DP / 32]
  float* unit = part + DL_UNIT * (DP / 32);                      // [16]
  float* mats = unit + DL_UNIT;                                  // chunks: [4][16][16]
  constexpr int TPT = DP / 8, TOKS = DL_THREADS / TPT;    // VEC: threads a token, tokens a pass
  constexpr int NP8 = VEC ? (DL_UNIT + TOKS - 1) / TOKS : 1;
  const int c8 = (int)(threadIdx.x % TPT) * 8;
  uint4 k8[NP8], a8[NP8], r8[NP8], v8[NP8];
  auto fetch8 = [&](int head) {
#pragma unroll
    for (int x = 0; x < NP8; ++x) {
      const int t = (int)threadIdx.x / TPT + x * TOKS;
      k8[x] = a8[x] = r8[x] = v8[x] = make_uint4(0u, 0u, 0u, 0u);
      if (t < nt && c8 < p.d) {
        const int64_t o = (t0 + t) * p.in_stride + (int64_t)head * p.d + c8;
        k8[x] = __ldg(reinterpret_cast<const uint4*>(static_cast<const T*>(p.k) + o));
        a8[x] = __ldg(reinterpret_cast<const uint4*>(static_cast<const T*>(p.a) + o));
        r8[x] = __ldg(reinterpret_cast<const uint4*>(static_cast<const T*>(p.r) + o));
        v8[x] = __ldg(reinterpret_cast<const uint4*>(static_cast<const T*>(p.v) + o));
      }
    }
  };
  const int h0 = blockIdx.y * p.heads_per_cta;
  if (VEC) fetch8(h0);
  for (int i = threadIdx.x; i < DL_UNIT * rank_p; i += DL_THREADS) {
    const int t = i / rank_p, r = i - t * rank_p;
    float z = 0.f;
    if (t < nt && r < p.rank)
      z = tanhf(Elem<T>::load(static_cast<const T*>(p.y1) + (t0 + t) * p.in_stride + r));
    if (MMA) {
      const float zh = round_bf16(z);
      hi[t * ld + r] = __bfloat16_as_ushort(__float2bfloat16_rn(zh));
      lo[t * ld + r] = __bfloat16_as_ushort(__float2bfloat16_rn(z - zh));
    } else {
      th[i] = z;
    }
  }
  // where the sum that this lane ends up with goes inside a block's scalars
  int scal_off = lane;
  if (lane >= 12) {
    const int e = lane - 12, f = e >= 10 ? 1 : 0, t = e - f * 10;
    const int row = t < 1 ? 0 : t < 3 ? 1 : t < 6 ? 2 : 3;
    scal_off = 16 + f * 16 + row * 4 + (t - row * (row + 1) / 2);
  }
  const int h1 = min((int)(blockIdx.y + 1) * p.heads_per_cta, p.heads);
  for (int h = h0; h < h1; ++h) {
    __syncthreads();       // tanh written; vec and unit of the last head consumed
    const int64_t ch0 = (int64_t)h * p.d;
    float seen = 0.f;      // becomes NaN where anything is not finite
    // this thread's elements of the head's [16][DP] tile.  Single tokens: requested before
    // the decay projection so that their latency passes behind it; blocks: as they are
    // needed, many CTAs share an SM
    constexpr int F = DL_UNIT * VP;                      // floats of one field
    constexpr int NIT = DL_UNIT * DP / DL_THREADS;
    constexpr int PASS = BLOCKED ? 4 : NIT < 16 ? NIT : 16;
    constexpr int SL = DP / 32;                          // warps that hold one token
    // element x: token tok(x), channel chan(x); one channel per thread up to DP = 128
    constexpr int TSTEP = DP <= DL_THREADS ? DL_THREADS / DP : 1;
    constexpr int CPT = DP <= DL_THREADS ? 1 : DP / DL_THREADS;
    const int c_first = DP <= DL_THREADS ? (int)(threadIdx.x % DP) : (int)threadIdx.x;
    const int t_first = DP <= DL_THREADS ? (int)(threadIdx.x / DP) : 0;
    auto tok = [&](int x) { return t_first + x / CPT * TSTEP; };
    auto chan = [&](int x) { return c_first + x % CPT * DL_THREADS; };
    const int64_t base = (t0 + t_first) * p.in_stride + ch0 + c_first;
    const T* pk = static_cast<const T*>(p.k) + base;
    const T* pa = static_cast<const T*>(p.a) + base;
    const T* pr = static_cast<const T*>(p.r) + base;
    const T* pv = static_cast<const T*>(p.v) + base;
    auto offset = [&](int x) {
      return (int64_t)(x / CPT * TSTEP) * p.in_stride + x % CPT * DL_THREADS;
    };
    float w0c[CPT], abc[CPT];
#pragma unroll
    for (int x = 0; x < CPT; ++x) {
      const bool on = !VEC && chan(x) < p.d;
      w0c[x] = on ? __ldg(p.w0 + ch0 + chan(x)) : 0.f;
      abc[x] = on ? __ldg(p.a_bias + ch0 + chan(x)) : 0.f;
    }
    if (VEC && h != h0) fetch8(h);
    T kx[PASS], ax[PASS], rx[PASS], vx[PASS];
    auto fetch = [&](int x0) {
#pragma unroll
      for (int x = 0; x < PASS; ++x) {
        kx[x] = ax[x] = rx[x] = vx[x] = T(0);
        if (tok(x0 + x) < nt && chan(x0 + x) < p.d) {
          const int64_t o = offset(x0 + x);
          kx[x] = __ldg(pk + o);
          ax[x] = __ldg(pa + o);
          rx[x] = __ldg(pr + o);
          vx[x] = __ldg(pv + o);
        }
      }
    };
    if (!BLOCKED && !VEC) fetch(0);
    // decay projection into field 0
    if (MMA) {
      const int kq = (lane & 3) * 2, r0 = lane >> 2;
      for (int n0 = warp * 8; n0 < p.d; n0 += NW * 8) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        const int ch = n0 + r0;
        const bool on = ch < p.d;
        const uint16_t* w2 = static_cast<const uint16_t*>(p.w2) + (ch0 + (on ? ch : 0)) * p.w2_stride;
        for (int k1 = 0; k1 < rank_p; k1 += 128) {
          uint32_t b0[8], b1[8];
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            const int k0 = k1 + x * 16 + kq;
            b0[x] = b1[x] = 0u;
            if (on && k0 < p.w2_stride) b0[x] = __ldg(reinterpret_cast<const uint32_t*>(w2 + k0));
            if (on && k0 + 8 < p.w2_stride)
              b1[x] = __ldg(reinterpret_cast<const uint32_t*>(w2 + k0 + 8));
          }
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            const int k0 = k1 + x * 16;
            if (k0 >= rank_p) break;
            const uint16_t* ah = hi + r0 * ld + k0 + kq;
            const uint16_t* al = lo + r0 * ld + k0 + kq;
            const uint32_t fh[4] = {*reinterpret_cast<const uint32_t*>(ah),
                                    *reinterpret_cast<const uint32_t*>(ah + 8 * ld),
                                    *reinterpret_cast<const uint32_t*>(ah + 8),
                                    *reinterpret_cast<const uint32_t*>(ah + 8 * ld + 8)};
            const uint32_t fl[4] = {*reinterpret_cast<const uint32_t*>(al),
                                    *reinterpret_cast<const uint32_t*>(al + 8 * ld),
                                    *reinterpret_cast<const uint32_t*>(al + 8),
                                    *reinterpret_cast<const uint32_t*>(al + 8 * ld + 8)};
            mma_bf16_16816(c, fl, b0[x], b1[x]);
            mma_bf16_16816(c, fh, b0[x], b1[x]);
          }
        }
        *reinterpret_cast<float2*>(vec + r0 * VP + n0 + kq) = make_float2(c[0], c[1]);
        *reinterpret_cast<float2*>(vec + (r0 + 8) * VP + n0 + kq) = make_float2(c[2], c[3]);
      }
    } else {
      for (int i = threadIdx.x; i < nt * DP; i += DL_THREADS) {
        const int t = i / DP, c = i % DP;
        float z = 0.f;
        if (c < p.d) {
          const float* w2 = reinterpret_cast<const float*>(p.w2) + (ch0 + c) * p.w2_stride;
          for (int r = 0; r < p.rank; ++r) z = fmaf(w2[r], th[t * rank_p + r], z);
        }
        vec[i] = z;
      }
    }
    if (VEC) {
      __syncthreads();
      const int swap = (lane >> 2) & 1;        // of a row's 32 bytes, so that 8 lanes' halves
                                               // fall into different banks
#pragma unroll
      for (int x = 0; x < NP8; ++x) {
        const int t = (int)threadIdx.x / TPT + x * TOKS;
        const uint32_t kw[4] = {k8[x].x, k8[x].y, k8[x].z, k8[x].w};
        const uint32_t aw[4] = {a8[x].x, a8[x].y, a8[x].z, a8[x].w};
        const uint32_t rw[4] = {r8[x].x, r8[x].y, r8[x].z, r8[x].w};
        const uint32_t vw[4] = {v8[x].x, v8[x].y, v8[x].z, v8[x].w};
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) ss += bf16lo(kw[i]) * bf16lo(kw[i]) + bf16hi(kw[i]) * bf16hi(kw[i]);
#pragma unroll
        for (int o = TPT / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float un = 1.0f / sqrtf(ss + p.unit_eps);
        if (t >= DL_UNIT) continue;
        const bool on = t < nt && c8 < p.d;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int half = hh ^ swap, i = t * VP + c8 + half * 4;
          float w[4], u[4], b[4], k[4], r[4], v[4];
          const float4 z = *reinterpret_cast<const float4*>(vec + i);
          const float zz[4] = {z.x, z.y, z.z, z.w};
          float4 w0 = make_float4(0.f, 0.f, 0.f, 0.f), ab = w0;
          if (on) {
            w0 = __ldg(reinterpret_cast<const float4*>(p.w0 + ch0 + c8 + half * 4));
            ab = __ldg(reinterpret_cast<const float4*>(p.a_bias + ch0 + c8 + half * 4));
          }
          const float w0v[4] = {w0.x, w0.y, w0.z, w0.w}, abv[4] = {ab.x, ab.y, ab.z, ab.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            auto pick = [&](const uint32_t (&q)[4]) {
              const uint32_t lo = half ? q[2 + (e >> 1)] : q[e >> 1];
              return (e & 1) ? bf16hi(lo) : bf16lo(lo);
            };
            k[e] = pick(kw);
            r[e] = pick(rw);
            v[e] = pick(vw);
            w[e] = 1.f;
            u[e] = b[e] = 0.f;
            if (on) {
              w[e] = decay_of<T, CHUNK>(-p.decay_scale * Gate<T>::sigmoid(zz[e] + w0v[e]));
              u[e] = k[e] * un;
              b[e] = u[e] * Gate<T>::sigmoid(pick(aw) + abv[e]);
            }
            if (CHUNK) seen = fmaf(w[e] + u[e] + b[e] + k[e] + r[e] + v[e], 0.f, seen);
          }
          // blocks: into the tile; single tokens: straight to the token's fields
          if (!BLOCKED && t >= nt) continue;
          float* dst = BLOCKED ? vec + i
                               : p.packed + (((int64_t)h * p.rows + t0 + t) * DL_FIELDS) * DP + c8 +
                                     half * 4;
          constexpr int S = BLOCKED ? F : DP;
          *reinterpret_cast<float4*>(dst) = make_float4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<float4*>(dst + S) = make_float4(u[0], u[1], u[2], u[3]);
          *reinterpret_cast<float4*>(dst + 2 * S) = make_float4(b[0], b[1], b[2], b[3]);
          *reinterpret_cast<float4*>(dst + 3 * S) = make_float4(k[0], k[1], k[2], k[3]);
          *reinterpret_cast<float4*>(dst + 4 * S) = make_float4(r[0], r[1], r[2], r[3]);
          *reinterpret_cast<float4*>(dst + 5 * S) = make_float4(v[0], v[1], v[2], v[3]);
        }
      }
    } else {
    // sums of k^2 per token: [16][SL] partial sums, one per warp that holds some of it
#pragma unroll(BLOCKED ? 4 : NIT)
    for (int x = 0; x < NIT; ++x) {
      float k = 0.f;
      if (!BLOCKED && NIT <= PASS)
        k = Elem<T>::load(&kx[x < PASS ? x : 0]);
      else if (tok(x) < nt && chan(x) < p.d)
        k = Elem<T>::load(pk + offset(x));
      const float ss = warp_sum(k * k);
      if (lane == 0) part[tok(x) * SL + chan(x) / 32] = ss;
    }
    __syncthreads();
    if (threadIdx.x < DL_UNIT) {
      float ss = 0.f;
#pragma unroll
      for (int y = 0; y < SL; ++y) ss += part[threadIdx.x * SL + y];
      unit[threadIdx.x] = 1.0f / sqrtf(ss + p.unit_eps);
    }
    __syncthreads();
#pragma unroll(BLOCKED ? 1 : NIT / PASS)
    for (int x0 = 0; x0 < NIT; x0 += PASS) {
      if (BLOCKED || x0 > 0) fetch(x0);
#pragma unroll
      for (int x = 0; x < PASS; ++x) {
        const int t = tok(x0 + x), c = chan(x0 + x), i = t * VP + c;
        const bool on = t < nt && c < p.d;
        float w = 1.f, u = 0.f, b = 0.f;
        const float k = Elem<T>::load(&kx[x]), r = Elem<T>::load(&rx[x]);
        const float v = Elem<T>::load(&vx[x]);
        if (on) {
          w = decay_of<T, CHUNK>(-p.decay_scale * Gate<T>::sigmoid(vec[i] + w0c[x % CPT]));
          u = k * unit[t];
          b = u * Gate<T>::sigmoid(Elem<T>::load(&ax[x]) + abc[x % CPT]);
        }
        if (CHUNK) seen = fmaf(w + u + b + k + r + v, 0.f, seen);
        if (BLOCKED) {
          vec[i] = w;
          vec[F + i] = u;
          vec[2 * F + i] = b;
          vec[3 * F + i] = k;
          vec[4 * F + i] = r;
          vec[5 * F + i] = v;
        } else if (t < nt) {
          float* dst = p.packed + (((int64_t)h * p.rows + t0 + t) * DL_FIELDS) * DP + c;
          dst[0] = w;
          dst[DP] = u;
          dst[2 * DP] = b;
          dst[3 * DP] = k;
          dst[4 * DP] = r;
          dst[5 * DP] = v;
        }
      }
    }
    }
    if (!BLOCKED) continue;
    if constexpr (CHUNK) {
      uint8_t* rec = reinterpret_cast<uint8_t*>(p.packed) +
                     ((int64_t)h * p.units + blockIdx.x) * dl_chunk_bytes(DP);
      for (int i = threadIdx.x; i < 1024; i += DL_THREADS) mats[i] = 0.f;
      const bool plain = __syncthreads_or(seen != 0.f);
      if (threadIdx.x == 0) *reinterpret_cast<int*>(rec + dl_chunk_flag(DP)) = plain;
      if (plain) {
        for (int i = threadIdx.x; i < DL_FIELDS * DL_UNIT * DP; i += DL_THREADS)
          reinterpret_cast<float*>(rec)[i] = vec[i / DP * VP + i % DP];
      } else {
        delta_chunk_record<DP>(vec, mats, rec);
      }
      continue;
    }
    __syncthreads();
    // a warp per block, lane = channel
    for (int blk = warp; blk * DL_BLK < nt; blk += NW) {
      float* dst = p.packed + (((int64_t)h * p.units + blockIdx.x) * (DL_UNIT / DL_BLK) + blk) *
                                  dl_block_floats(DP);
      float acc[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = 0.f;
#pragma unroll
      for (int c0 = 0; c0 < DP; c0 += 32) {
        const int c = c0 + lane;
        const float* src = vec + blk * DL_BLK * DP + c;
        float kk[DL_BLK], bb[DL_BLK], gam = 1.f;
#pragma unroll
        for (int i = 0; i < DL_BLK; ++i) {
          const int ia = i * (i - 1) / 2, ie = 12 + i * (i + 1) / 2;
          const float* s = src + i * DP;
          const float w = s[0], u = s[F], r = s[4 * F];
#pragma unroll
          for (int j = 0; j < i; ++j) {
            acc[ia + j] = fmaf(u, kk[j], acc[ia + j]);
            acc[6 + ia + j] = fmaf(u, bb[j], acc[6 + ia + j]);
            kk[j] *= w;
            bb[j] *= w;
          }
          bb[i] = s[2 * F];
          kk[i] = s[3 * F];
#pragma unroll
          for (int j = 0; j <= i; ++j) {
            acc[ie + j] = fmaf(r, kk[j], acc[ie + j]);
            acc[10 + ie + j] = fmaf(r, bb[j], acc[10 + ie + j]);
          }
          dst[i * DP + c] = u * gam;
          gam *= w;
          dst[(12 + i) * DP + c] = r * gam;
          dst[(16 + i) * DP + c] = s[5 * F];
        }
        dst[20 * DP + c] = gam;
#pragma unroll
        for (int j = 0; j < DL_BLK; ++j) {
          dst[(4 + j) * DP + c] = kk[j];
          dst[(8 + j) * DP + c] = -bb[j];
        }
      }
      // 32 sums over the warp in 31 exchanges: lane l ends with sum number l
#pragma unroll
      for (int w = 16; w > 0; w >>= 1) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; ++i) {
          const float keep = up ? acc[i + w] : acc[i];
          const float give = up ? acc[i] : acc[i + w];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, w);
        }
      }
      float* scal = dst + 21 * DP;
      scal[16 + lane] = 0.f;           // E and F above their diagonals
      __syncwarp();
      scal[scal_off] = acc[0];
    }
  }
}

struct DeltaScanParams {
  const float* packed;                 // per token or blocks (see above)
  float* o;                            // [rows][heads * d]
  float* state;                        // [slots][heads][d][dp]
  const int32_t* cu; const int32_t* slots; const int64_t* positions;
  int64_t rows, units; int heads, d, num_slots, num_portions;
  int least, below;                    // portions of least .. below - 1 tokens are taken
  int32_t* status;
};

// The CPL key channels of lane q: 4 q .., 4 (LANES + q) .., ...
template <int LANES, int CPL>
__device__ __forceinline__ void dl_load(const float* row, int q, uint64_t (&x)[CPL / 2]) {
#pragma unroll
  for (int g = 0; g < CPL / 4; ++g) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(row + (g * LANES + q) * 4);
    x[2 * g] = a.x;
    x[2 * g + 1] = a.y;
  }
}
template <int LANES, int CPL>
__device__ __forceinline__ void dl_store(float* row, int q, const uint64_t (&x)[CPL / 2]) {
#pragma unroll
  for (int g = 0; g < CPL / 4; ++g)
    *reinterpret_cast<ulonglong2*>(row + (g * LANES + q) * 4) =
        make_ulonglong2(x[2 * g], x[2 * g + 1]);
}
__device__ __forceinline__ uint64_t dl_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
template <int N>
__device__ __forceinline__ float dl_dot(const uint64_t (&a)[N], const uint64_t (&b)[N]) {
  uint64_t x = dl_mul(a[0], b[0]);
  if (N > 2) {
    uint64_t y = dl_mul(a[1], b[1]);
#pragma unroll
    for (int i = 2; i < N; i += 2) {
      x = dl_fma(a[i], b[i], x);
      y = dl_fma(a[i + 1], b[i + 1], y);
    }
    x = dl_add(x, y);
  } else {
    x = dl_fma(a[N - 1], b[N - 1], x);
  }
  float a0, a1;
  dl_unpack(x, a0, a1);
  return a0 + a1;
}

// Token by token.  Thread = (column group, lane); NC columns per thread.
template <int LANES, int CPL, int NC>
__global__ void __launch_bounds__(DL_THREADS) delta_scan_kernel(const DeltaScanParams p) {
  constexpr int GROUPS = DL_THREADS / LANES;
  constexpr int COLS = GROUPS * NC;
  constexpr int DP = LANES * CPL, NP = CPL / 2;
  constexpr int REC = DL_FIELDS * DP;         // floats per token
  const int h = blockIdx.y, seq = blockIdx.z;
  const int q = threadIdx.x % LANES, col0 = blockIdx.x * COLS + threadIdx.x / LANES;
  pdl_launch_dependents();
  pdl_wait();
  const int64_t begin = p.cu[seq], end = p.cu[seq + 1];
  if (end - begin < p.least || end - begin >= p.below) return;
  const int slot = begin < end ? p.slots[begin] : -1;
  if (slot >= p.num_slots) {
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, FK_DEV_BAD_SLOT);
    return;
  }
  if (slot < 0) return;
  uint64_t s[NC][NP];
  float* st[NC];
  bool col_on[NC];
  const bool fresh = p.positions[begin] == 0;
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const int col = col0 + j * GROUPS;
    col_on[j] = col < p.d;
    st[j] = p.state + (((int64_t)slot * p.heads + h) * p.d + (col_on[j] ? col : 0)) * DP;
#pragma unroll
    for (int i = 0; i < NP; ++i) s[j][i] = 0ull;
    if (col_on[j] && !fresh) dl_load<LANES, CPL>(st[j], q, s[j]);
  }
  for (int64_t t = begin; t < end; ++t) {
    const float* rec = p.packed + ((int64_t)h * p.rows + t) * REC;
    uint64_t w[NP], u[NP], b[NP], k[NP], r[NP];
    dl_load<LANES, CPL>(rec + DP, q, u);
    dl_load<LANES, CPL>(rec, q, w);
    dl_load<LANES, CPL>(rec + 3 * DP, q, k);
    dl_load<LANES, CPL>(rec + 2 * DP, q, b);
    dl_load<LANES, CPL>(rec + 4 * DP, q, r);
    float dot[NC], out[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) dot[j] = dl_dot<NP>(u, s[j]);
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < NC; ++j) dot[j] += __shfl_xor_sync(0xffffffffu, dot[j], o);
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const int col = col0 + j * GROUPS;
      const float v = col < DP ? rec[5 * DP + col] : 0.f;
      const uint64_t vv = dl_pack(v, v), nd = dl_pack(-dot[j], -dot[j]);
#pragma unroll
      for (int i = 0; i < NP; ++i)
        s[j][i] = dl_fma(b[i], nd, dl_fma(k[i], vv, dl_mul(w[i], s[j][i])));
      out[j] = dl_dot<NP>(r, s[j]);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < NC; ++j) out[j] += __shfl_xor_sync(0xffffffffu, out[j], o);
    if (q == 0) {
#pragma unroll
      for (int j = 0; j < NC; ++j)
        if (col_on[j])
          p.o[t * ((int64_t)p.heads * p.d) + (int64_t)h * p.d + col0 + j * GROUPS] = out[j];
    }
  }
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (col_on[j]) dl_store<LANES, CPL>(st[j], q, s[j]);
}

// Blocks of a portion.  They stream through a ring of shared-memory stages (bulk
// copies); what limits the kernel is reading the blocks' vectors out of shared memory,
// which NC columns per thread share.
template <int LANES, int CPL, int NC>
__global__ void __launch_bounds__(DL_THREADS) delta_scan_blocked_kernel(const DeltaScanParams p) {
  extern __shared__ __align__(128) uint8_t dl_smem[];
  constexpr int GROUPS = DL_THREADS / LANES;
  constexpr int COLS = GROUPS * NC;
  constexpr int DP = LANES * CPL, NP = CPL / 2;
  constexpr int BLK = DL_BLK, SB = DL_STAGE_BLOCKS;
  constexpr int REC = dl_block_floats(DP);    // floats per block
  float* stages = reinterpret_cast<float*>(dl_smem);
  float* outs = stages + DL_STAGES * SB * REC;                     // [2][SB * 4][COLS]
  uint64_t* full = reinterpret_cast<uint64_t*>(outs + 2 * SB * BLK * COLS);
  __shared__ int failed;

  const int h = blockIdx.y, seq = blockIdx.z;
  const int col0 = blockIdx.x * COLS;
  const int q = threadIdx.x % LANES, grp = threadIdx.x / LANES;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < DL_STAGES; ++i) mbar_init(&full[i], 1);
    mbar_fence_init();
    failed = 0;
  }
  pdl_wait();
  const int64_t begin = p.cu[seq], end = p.cu[seq + 1];
  const int slot = begin < end ? p.slots[begin] : -1;
  const int64_t n = end - begin;
  if (n < p.least || n >= p.below) return;
  if (slot >= p.num_slots) {
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, FK_DEV_BAD_SLOT);
    return;
  }
  if (slot < 0 || n <= 0) return;
  __syncthreads();
  const int nblk = (int)((n + BLK - 1) / BLK);
  const int nst = (nblk + SB - 1) / SB;
  const float* src = p.packed + ((int64_t)h * p.units + begin / DL_UNIT + seq) *
                                    ((DL_UNIT / BLK) * (int64_t)REC);
  auto issue = [&](int si) {
    const int s = si % DL_STAGES;
    const uint32_t bytes = (uint32_t)(min(SB, nblk - si * SB) * REC * sizeof(float));
    mbar_arrive_expect_tx(&full[s], bytes);
    bulk_load(stages + s * SB * REC, src + (int64_t)si * SB * REC, bytes, &full[s]);
  };
  if (threadIdx.x == 0)
    for (int i = 0; i < DL_STAGES - 1 && i < nst; ++i) issue(i);

  uint64_t s[NC][NP];
  float* st[NC];
  bool col_on[NC];
  const bool fresh = p.positions[begin] == 0;
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const int col = col0 + grp + j * GROUPS;
    col_on[j] = col < p.d;
    st[j] = p.state + (((int64_t)slot * p.heads + h) * p.d + (col_on[j] ? col : 0)) * DP;
#pragma unroll
    for (int i = 0; i < NP; ++i) s[j][i] = 0ull;
    if (col_on[j] && !fresh) dl_load<LANES, CPL>(st[j], q, s[j]);
  }

  int si = 0;
  for (; si < nst; ++si) {
    const int sg = si % DL_STAGES;
    if (!mbar_wait_warp(&full[sg], (uint32_t)(si / DL_STAGES) & 1u, DL_WAIT_LIMIT)) {
      if (p.status) atomicOr(p.status, FK_DEV_WAIT_TIMEOUT);
      failed = 1;
    }
    const int blocks = min(SB, nblk - si * SB);
    float* ot = outs + (si & 1) * SB * BLK * COLS;
    for (int b = 0; b < blocks; ++b) {
      const float* rec = stages + (sg * SB + b) * REC;
      const float* sc = rec + 21 * DP;
      float v[BLK][NC], d[BLK][NC], o[BLK][NC];
#pragma unroll
      for (int i = 0; i < BLK; ++i) {
        uint64_t u[NP];
        dl_load<LANES, CPL>(rec + i * DP, q, u);
#pragma unroll
        for (int j = 0; j < NC; ++j) d[i][j] = dl_dot<NP>(u, s[j]);
      }
#pragma unroll
      for (int w = LANES / 2; w > 0; w >>= 1)
#pragma unroll
        for (int i = 0; i < BLK; i += 2)
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            const float x0 = __shfl_xor_sync(0xffffffffu, d[i][j], w);
            const float x1 = __shfl_xor_sync(0xffffffffu, d[i + 1][j], w);
            dl_unpack(dl_add(dl_pack(d[i][j], d[i + 1][j]), dl_pack(x0, x1)), d[i][j],
                      d[i + 1][j]);
          }
      // off the critical path: output shares of the old state, decayed state, keys
#pragma unroll
      for (int i = 0; i < BLK; ++i) {
        uint64_t r[NP];
        dl_load<LANES, CPL>(rec + (12 + i) * DP, q, r);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          o[i][j] = dl_dot<NP>(r, s[j]);
          const int col = col0 + grp + j * GROUPS;
          v[i][j] = col < DP ? rec[(16 + i) * DP + col] : 0.f;
        }
      }
      {
        uint64_t g[NP];
        dl_load<LANES, CPL>(rec + 20 * DP, q, g);
#pragma unroll
        for (int j = 0; j < NC; ++j)
#pragma unroll
          for (int x = 0; x < NP; ++x) s[j][x] = dl_mul(g[x], s[j][x]);
      }
#pragma unroll
      for (int i = 0; i < BLK; ++i) {
        uint64_t k[NP];
        dl_load<LANES, CPL>(rec + (4 + i) * DP, q, k);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const uint64_t vv = dl_pack(v[i][j], v[i][j]);
#pragma unroll
          for (int x = 0; x < NP; ++x) s[j][x] = dl_fma(k[x], vv, s[j][x]);
        }
      }
      // p_1 .. p_4 (kept in d)
      const float4 sa = *reinterpret_cast<const float4*>(sc);
      const float4 sb = *reinterpret_cast<const float4*>(sc + 4);
      const float4 sd = *reinterpret_cast<const float4*>(sc + 8);
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        d[1][j] += sa.x * v[0][j];
        d[2][j] += sa.y * v[0][j] + sa.z * v[1][j];
        d[3][j] += sa.w * v[0][j] + sb.x * v[1][j] + sb.y * v[2][j];
        d[1][j] -= sb.z * d[0][j];
        d[2][j] -= sb.w * d[0][j] + sd.x * d[1][j];
        d[3][j] -= sd.y * d[0][j] + sd.z * d[1][j] + sd.w * d[2][j];
      }
#pragma unroll
      for (int i = 0; i < BLK; ++i) {
        uint64_t bv[NP];
        dl_load<LANES, CPL>(rec + (8 + i) * DP, q, bv);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const uint64_t np = dl_pack(d[i][j], d[i][j]);
#pragma unroll
          for (int x = 0; x < NP; ++x) s[j][x] = dl_fma(bv[x], np, s[j][x]);
        }
      }
      // outputs: halving exchanges over the low two lane bits leave token q & 3 in o[0],
      // then the sum over the other lanes and what the block's own tokens add
#pragma unroll
      for (int w = 2; w > 0; w >>= 1) {
        const bool up = (q & w) != 0;
#pragma unroll
        for (int i = 0; i < w; ++i)
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            const float keep = up ? o[i + w][j] : o[i][j];
            const float give = up ? o[i][j] : o[i + w][j];
            o[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, w);
          }
      }
#pragma unroll
      for (int w = LANES / 2; w >= BLK; w >>= 1)
#pragma unroll
        for (int j = 0; j < NC; ++j) o[0][j] += __shfl_xor_sync(0xffffffffu, o[0][j], w);
      if (q < BLK) {
        const float4 er = *reinterpret_cast<const float4*>(sc + 16 + q * 4);
        const float4 fr = *reinterpret_cast<const float4*>(sc + 32 + q * 4);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const float x0 = er.x * v[0][j] + er.y * v[1][j] + er.z * v[2][j] + er.w * v[3][j];
          const float x1 = fr.x * d[0][j] + fr.y * d[1][j] + fr.z * d[2][j] + fr.w * d[3][j];
          ot[(b * BLK + q) * COLS + grp + j * GROUPS] = o[0][j] + (x0 - x1);
        }
      }
    }
    __syncthreads();            // stage sg is free, its outputs are complete
    if (failed) break;
    if (threadIdx.x == 0 && si + DL_STAGES - 1 < nst) issue(si + DL_STAGES - 1);
    const int64_t row0 = begin + (int64_t)si * SB * BLK;
    const int cnt = (int)min((int64_t)SB * BLK, end - row0);
    for (int i = threadIdx.x; i < cnt * COLS; i += DL_THREADS) {
      const int t2 = i / COLS, c = i - t2 * COLS;
      if (col0 + c < p.d)
        p.o[(row0 + t2) * ((int64_t)p.heads * p.d) + (int64_t)h * p.d + col0 + c] = ot[i];
    }
  }
  if (failed) {
    // copies that were requested must land before the shared memory goes away
    for (int i = si; i < nst && i < si + DL_STAGES - 1; ++i)
      (void)mbar_wait_warp(&full[i % DL_STAGES], (uint32_t)(i / DL_STAGES) & 1u, DL_WAIT_LIMIT);
    return;
  }
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (col_on[j]) dl_store<LANES, CPL>(st[j], q, s[j]);
}

// Chunks of a portion, on the tensor cores: S^T, 16 value channels a warp, stays in the registers
// of its mma accumulators, which are also the layout of an A operand.  With S ahead of a chunk
// (operands as in its record, tokens 1..16)
//
//   P = (I + C)^-1 (U S + A V)      O = R S + E V - F P      S' = diag(w_{1..16}) S + K^T V - B^T P
//
// Bound by the tensor cores where the SMs have two CTAs (8 cycles an mma, 204 a chunk and warp at 64
// channels), else by a chunk's chain of products: 3500 cycles, 6000 at 128 channels.
//
// Every product is of three bf16 parts a number (v has one), the six of them that reach 2^-24.
// The largest of them, hi hi, has an accumulator of its own for each 16 k's, which it fills almost
// exactly, and those are added in fp32; the others share one, whose rounding is 2^-8 of that.
struct DlParts { uint32_t hi[4], mid[4], lo[4]; };
struct DlFrag { uint4 hi, mid, lo; };
__device__ __forceinline__ void dl_mma1(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                        uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c[0], c[1] += a times the two halves of b
__device__ __forceinline__ void dl_mma(float (&c)[2][4], const uint32_t (&a)[4], const uint4& b) {
  dl_mma1(c[0], a, b.x, b.y);
  dl_mma1(c[1], a, b.z, b.w);
}
__device__ __forceinline__ void dl_add(float (&c)[2][4], const float (&t)[2][4]) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[i][e] += t[i][e];
}
// two 16 x 8 accumulator tiles as one 16 x 16 A operand
__device__ __forceinline__ void dl_parts(const float (&x)[4], const float (&y)[4], DlParts& a) {
  dl_split(x[0], x[1], a.hi[0], a.mid[0], a.lo[0]);
  dl_split(x[2], x[3], a.hi[1], a.mid[1], a.lo[1]);
  dl_split(y[0], y[1], a.hi[2], a.mid[2], a.lo[2]);
  dl_split(y[2], y[3], a.hi[3], a.mid[3], a.lo[3]);
}
__device__ __forceinline__ DlFrag dl_frag(const uint8_t* at, int lane) {
  const uint4* x = reinterpret_cast<const uint4*>(at) + lane;
  return {x[0], x[DL_FRAG / 16], x[2 * (DL_FRAG / 16)]};
}
// the five smaller products of two operands at once, so that four chains run side by side
__device__ __forceinline__ void dl_five(float (&c)[2][4], const DlParts& a, const DlFrag& x,
                                        float (&d)[2][4], const DlParts& b, const DlFrag& y) {
  dl_mma(c, a.lo, x.hi);
  dl_mma(d, b.lo, y.hi);
  dl_mma(c, a.hi, x.lo);
  dl_mma(d, b.hi, y.lo);
  dl_mma(c, a.mid, x.mid);
  dl_mma(d, b.mid, y.mid);
  dl_mma(c, a.mid, x.hi);
  dl_mma(d, b.mid, y.hi);
  dl_mma(c, a.hi, x.mid);
  dl_mma(d, b.hi, y.mid);
}

// The longest portions come first, so that their CTAs start one an SM; two CTAs an SM, as a third
// one slows those that the kernel waits for (five portions of 700 to 2400 tokens, 64 heads: 577 us
// in the order of the batch, 448 longest first, 388 and no more than two an SM).
constexpr int DL_RANKED = 128;    // portions that are put in order; more even themselves out
template <int DP, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, DP == 64 ? 2 : 1)
delta_scan_chunk_kernel(const DeltaScanParams p) {
  extern __shared__ __align__(128) uint8_t dl_smem[];
  constexpr int KT = DP / 16, BYTES = dl_chunk_bytes(DP), ST = dl_chunk_stages(DP);
  uint64_t* full = reinterpret_cast<uint64_t*>(dl_smem + ST * BYTES);
  __shared__ int failed;
  __shared__ int ranked;
  const int h = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = (int)(blockIdx.z * WARPS + (threadIdx.x >> 5));
  const int g = lane >> 2, q2 = (lane & 3) * 2;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < ST; ++i) mbar_init(&full[i], 1);
    mbar_fence_init();
    failed = 0;
    ranked = blockIdx.y;
  }
  pdl_wait();
  __syncthreads();
  for (int j = threadIdx.x; j < p.num_portions && p.num_portions <= DL_RANKED; j += 32 * WARPS) {
    // portion j is this CTA's, if blockIdx.y are ahead of it
    const int len = p.cu[j + 1] - p.cu[j];
    int ahead = 0;
    for (int i = 0; i < p.num_portions; ++i) {
      const int other = p.cu[i + 1] - p.cu[i];
      ahead += other > len || (other == len && i < j) ? 1 : 0;
    }
    if (ahead == (int)blockIdx.y) ranked = j;
  }
  __syncthreads();
  const int seq = ranked;
  const int64_t begin = p.cu[seq], end = p.cu[seq + 1];
  if (end - begin < p.least || end - begin >= p.below) return;
  const int slot = begin < end ? p.slots[begin] : -1;
  if (slot >= p.num_slots) {
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, FK_DEV_BAD_SLOT);
    return;
  }
  if (slot < 0) return;
  const int chunks = (int)((end - begin + DL_UNIT - 1) / DL_UNIT);
  const uint8_t* src = reinterpret_cast<const uint8_t*>(p.packed) +
                       ((int64_t)h * p.units + begin / DL_UNIT + seq) * BYTES;
  auto issue = [&](int n) {
    mbar_arrive_expect_tx(&full[n % ST], BYTES);
    bulk_load(dl_smem + n % ST * BYTES, src + (int64_t)n * BYTES, BYTES, &full[n % ST]);
  };
  if (threadIdx.x == 0)
    for (int n = 0; n < ST && n < chunks; ++n) issue(n);

  // rows (value channels) v0 and v0 + 8 of S^T; columns 8 n + q2, + 1
  const int v0 = warp * 16 + g;
  const bool on0 = v0 < p.d, on1 = v0 + 8 < p.d;
  float s[2 * KT][4];
  float* st = p.state + ((int64_t)slot * p.heads + h) * p.d * DP + q2;
  const bool fresh = p.positions[begin] == 0;
#pragma unroll
  for (int n = 0; n < 2 * KT; ++n) {
    float2 a = make_float2(0.f, 0.f), b = a;
    if (on0 && !fresh) a = *reinterpret_cast<const float2*>(st + (int64_t)v0 * DP + n * 8);
    if (on1 && !fresh) b = *reinterpret_cast<const float2*>(st + (int64_t)(v0 + 8) * DP + n * 8);
    s[n][0] = a.x;
    s[n][1] = a.y;
    s[n][2] = b.x;
    s[n][3] = b.y;
  }
  const bool live = warp * 16 < p.d;
  float* out = p.o + (int64_t)h * p.d + v0;
  const int64_t o_stride = (int64_t)p.heads * p.d;
  int n = 0;
  for (; n < chunks; ++n) {
    if (!mbar_wait_warp(&full[n % ST], (uint32_t)(n / ST) & 1u, DL_WAIT_LIMIT)) {
      if (p.status) atomicOr(p.status, FK_DEV_WAIT_TIMEOUT);
      failed = 1;
    }
    const uint8_t* rec = dl_smem + n % ST * BYTES;
    const int64_t row0 = begin + (int64_t)n * DL_UNIT;
    const int cnt = (int)min((int64_t)DL_UNIT, end - row0);
    if (live && *reinterpret_cast<const int*>(rec + dl_chunk_flag(DP)) != 0) {
      // something is not finite: token by token, so that no token before it sees it
      const float* f = reinterpret_cast<const float*>(rec);
      constexpr int F = DL_UNIT * DP;
      for (int t = 0; t < cnt; ++t) {
        const float* x = f + t * DP + q2;
        float d0 = 0.f, d1 = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int i = 0; i < 2 * KT; ++i) {
          const float2 u = *reinterpret_cast<const float2*>(x + F + i * 8);
          d0 = fmaf(u.y, s[i][1], fmaf(u.x, s[i][0], d0));
          d1 = fmaf(u.y, s[i][3], fmaf(u.x, s[i][2], d1));
        }
#pragma unroll
        for (int w = 1; w < 4; w <<= 1) {
          d0 += __shfl_xor_sync(0xffffffffu, d0, w);
          d1 += __shfl_xor_sync(0xffffffffu, d1, w);
        }
        const float va = f[5 * F + t * DP + v0], vb = f[5 * F + t * DP + v0 + 8];
#pragma unroll
        for (int i = 0; i < 2 * KT; ++i) {
          const float2 w = *reinterpret_cast<const float2*>(x + i * 8);
          const float2 b = *reinterpret_cast<const float2*>(x + 2 * F + i * 8);
          const float2 k = *reinterpret_cast<const float2*>(x + 3 * F + i * 8);
          const float2 r = *reinterpret_cast<const float2*>(x + 4 * F + i * 8);
          s[i][0] = fmaf(b.x, -d0, fmaf(k.x, va, w.x * s[i][0]));
          s[i][1] = fmaf(b.y, -d0, fmaf(k.y, va, w.y * s[i][1]));
          s[i][2] = fmaf(b.x, -d1, fmaf(k.x, vb, w.x * s[i][2]));
          s[i][3] = fmaf(b.y, -d1, fmaf(k.y, vb, w.y * s[i][3]));
          o0 = fmaf(r.y, s[i][1], fmaf(r.x, s[i][0], o0));
          o1 = fmaf(r.y, s[i][3], fmaf(r.x, s[i][2], o1));
        }
#pragma unroll
        for (int w = 1; w < 4; w <<= 1) {
          o0 += __shfl_xor_sync(0xffffffffu, o0, w);
          o1 += __shfl_xor_sync(0xffffffffu, o1, w);
        }
        if (q2 == 0) {
          if (on0) out[(row0 + t) * o_stride] = o0;
          if (on1) out[(row0 + t) * o_stride + 8] = o1;
        }
      }
    } else if (live) {
      float pp[2][4] = {}, oo[2][4] = {}, ps[2][4] = {}, os[2][4] = {};
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        DlParts a;
        dl_parts(s[2 * kt], s[2 * kt + 1], a);
        const DlFrag u = dl_frag(rec + kt * 3 * DL_FRAG, lane);
        const DlFrag r = dl_frag(rec + (KT + kt) * 3 * DL_FRAG, lane);
        float t[2][4] = {}, z[2][4] = {};
        dl_mma(t, a.hi, u.hi);
        dl_mma(z, a.hi, r.hi);
        dl_five(ps, a, u, os, a, r);
        dl_add(pp, t);
        dl_add(oo, z);
      }
      const uint4 v4 = reinterpret_cast<const uint4*>(rec + dl_chunk_v(DP))[warp * 32 + lane];
      const uint32_t v[4] = {v4.x, v4.y, v4.z, v4.w};
      const uint8_t* mats = rec + dl_chunk_mats(DP);
      DlParts a;
      {
        const DlFrag x = dl_frag(mats, lane);
        float t[2][4] = {};
        dl_mma(t, v, x.hi);
        dl_mma(ps, v, x.lo);
        dl_mma(ps, v, x.mid);
        dl_add(pp, t);
        dl_add(pp, ps);
        dl_parts(pp[0], pp[1], a);
        const DlFrag m = dl_frag(mats + 3 * DL_FRAG, lane);
        float z[2][4] = {}, y0[2][4] = {}, y1[2][4] = {};
        dl_mma(z, a.hi, m.hi);
        dl_mma(y0, a.lo, m.hi);
        dl_mma(y1, a.mid, m.hi);
        dl_mma(y0, a.hi, m.lo);
        dl_mma(y1, a.hi, m.mid);
        dl_mma(y0, a.mid, m.mid);
        dl_add(y1, y0);
        dl_add(z, y1);
        dl_parts(z[0], z[1], a);
      }
      const float* gam = reinterpret_cast<const float*>(rec + dl_chunk_decay(DP)) + q2;
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        const DlFrag x = dl_frag(rec + (2 * KT + kt) * 3 * DL_FRAG, lane);
        const DlFrag y = dl_frag(rec + (3 * KT + kt) * 3 * DL_FRAG, lane);
        float t[2][4] = {}, z[2][4] = {}, y0[2][4] = {}, y1[2][4] = {};
        dl_mma(t, v, x.hi);
        dl_mma(z, a.hi, y.hi);
        dl_mma(y0, v, x.lo);
        dl_mma(y1, a.lo, y.hi);
        dl_mma(y0, v, x.mid);
        dl_mma(y1, a.hi, y.lo);
        dl_mma(y0, a.mid, y.hi);
        dl_mma(y1, a.mid, y.mid);
        dl_mma(y0, a.hi, y.mid);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 w = *reinterpret_cast<const float2*>(gam + (2 * kt + i) * 8);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float& x1 = s[2 * kt + i][e];
            x1 = fmaf(e & 1 ? w.y : w.x, x1, t[i][e] + z[i][e]) + (y0[i][e] + y1[i][e]);
          }
        }
      }
      {
        const DlFrag x = dl_frag(mats + 6 * DL_FRAG, lane), y = dl_frag(mats + 9 * DL_FRAG, lane);
        float t[2][4] = {}, z[2][4] = {}, y1[2][4] = {};
        dl_mma(t, v, x.hi);
        dl_mma(z, a.hi, y.hi);
        dl_mma(os, v, x.lo);
        dl_mma(y1, a.lo, y.hi);
        dl_mma(os, v, x.mid);
        dl_mma(y1, a.hi, y.lo);
        dl_mma(os, a.mid, y.hi);
        dl_mma(y1, a.mid, y.mid);
        dl_mma(os, a.hi, y.mid);
        dl_add(os, y1);
        dl_add(oo, t);
        dl_add(oo, z);
        dl_add(oo, os);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int tok = i * 8 + q2 + (e & 1);
            if (tok < cnt && (e < 2 ? on0 : on1))
              out[(row0 + tok) * o_stride + (e < 2 ? 0 : 8)] = oo[i][e];
          }
      }
    }
    __syncthreads();             // the record has been read
    if (failed) break;
    if (threadIdx.x == 0 && n + ST < chunks) issue(n + ST);
  }
  if (failed) {
    // copies that were requested must land before the shared memory goes away
    for (int i = n; i < chunks && i < n + ST; ++i)
      (void)mbar_wait_warp(&full[i % ST], (uint32_t)(i / ST) & 1u, DL_WAIT_LIMIT);
    return;
  }
#pragma unroll
  for (int i = 0; i < 2 * KT; ++i) {
    if (on0)
      *reinterpret_cast<float2*>(st + (int64_t)v0 * DP + i * 8) = make_float2(s[i][0], s[i][1]);
    if (on1)
      *reinterpret_cast<float2*>(st + (int64_t)(v0 + 8) * DP + i * 8) =
          make_float2(s[i][2], s[i][3]);
  }
}

static int delta_padded(int d) { return d <= 32 ? 32 : d <= 64 ? 64 : d <= 128 ? 128 : 256; }

template <typename T, int DP, bool BLOCKED, bool VEC, bool CHUNK = false>
static int launch_prepare_one(const DeltaPrepParams& p, unsigned gx, cudaStream_t s) {
  constexpr int kFixed = DL_FIELDS * DL_UNIT * (CHUNK ? DP + 4 : DP) * 4 +
                         DL_UNIT * (DP / 32 + 1) * 4 + (CHUNK ? 4 * 256 * 4 : 0);
  const size_t smem = (size_t)DL_UNIT * (p.rank_p + 8) * 4 + kFixed;
  static PerDeviceOnce once;
  constexpr int kMaxSmem = DL_UNIT * 520 * 4 + kFixed;
  FK_CUDA_OK(set_max_dynamic_smem(once, delta_prepare_kernel<T, DP, BLOCKED, VEC, CHUNK>,
                                  kMaxSmem));
  const dim3 grid(gx, (unsigned)((p.heads + p.heads_per_cta - 1) / p.heads_per_cta));
  FK_CUDA_OK(launch_kernel(delta_prepare_kernel<T, DP, BLOCKED, VEC, CHUNK>, grid,
                           dim3(DL_THREADS), smem, s, p));
  count_launch();
  return FK_OK;
}
template <typename T, int DP>
static int launch_prepare_dp(const DeltaPrepParams& p, int blocked, cudaStream_t s) {
  const unsigned single = (unsigned)((p.rows + DL_UNIT - 1) / DL_UNIT);
  // rows of whole 16-byte pieces, where 2-byte loads waited for one another: five prompts of
  // 700 to 2500 tokens, 64 heads of 64 687 -> 436 us, 24 heads of 128 765 -> 335;
  // a decode step of 16 rows, 32 heads of 64, 10.9 -> 8.2
  if constexpr (sizeof(T) == 2) {
    const bool pieces = p.d % 8 == 0 && p.in_stride % 8 == 0 && aligned16(p.r) &&
                        aligned16(p.k) && aligned16(p.v) && aligned16(p.a) && aligned16(p.w0) &&
                        aligned16(p.a_bias);
    if constexpr (DP == 64 || DP == 128) {
      if (blocked == 2)
        return pieces ? launch_prepare_one<T, DP, true, true, true>(p, (unsigned)p.units, s)
                      : launch_prepare_one<T, DP, true, false, true>(p, (unsigned)p.units, s);
    }
    if (pieces)
      return blocked ? launch_prepare_one<T, DP, true, true>(p, (unsigned)p.units, s)
                     : launch_prepare_one<T, DP, false, true>(p, single, s);
  }
  return blocked ? launch_prepare_one<T, DP, true, false>(p, (unsigned)p.units, s)
                 : launch_prepare_one<T, DP, false, false>(p, single, s);
}
template <typename T>
static int launch_prepare(const DeltaPrepParams& p, int blocked, cudaStream_t s) {
  switch (delta_padded(p.d)) {
    case 32: return launch_prepare_dp<T, 32>(p, blocked, s);
    case 64: return launch_prepare_dp<T, 64>(p, blocked, s);
    case 128: return launch_prepare_dp<T, 128>(p, blocked, s);
    default: return launch_prepare_dp<T, 256>(p, blocked, s);
  }
}

template <int LANES, int CPL, int NC>
static int launch_scan_blocked(DeltaScanParams& p, cudaStream_t s) {
  constexpr int COLS = DL_THREADS / LANES * NC;
  constexpr size_t kSmem = ((size_t)DL_STAGES * DL_STAGE_BLOCKS * dl_block_floats(LANES * CPL) +
                            2 * DL_STAGE_BLOCKS * DL_BLK * COLS) * 4 +
                           DL_STAGES * sizeof(uint64_t);
  static PerDeviceOnce once;
  FK_CUDA_OK(set_max_dynamic_smem(once, delta_scan_blocked_kernel<LANES, CPL, NC>, (int)kSmem));
  const dim3 grid((unsigned)((p.d + COLS - 1) / COLS), (unsigned)p.heads,
                  (unsigned)p.num_portions);
  // not ahead of its predecessor's end: CTAs that squeeze in beside the last ones of it
  // pile up on a few SMs and stay there
  FK_CUDA_OK(launch_kernel_after(delta_scan_blocked_kernel<LANES, CPL, NC>, grid,
                                 dim3(DL_THREADS), kSmem, s, p));
  count_launch();
  return FK_OK;
}
template <int DP, int WARPS>
static int launch_scan_chunks(const DeltaScanParams& p, cudaStream_t s) {
  constexpr int kSmem = dl_chunk_stages(DP) * (dl_chunk_bytes(DP) + (int)sizeof(uint64_t));
  static PerDeviceOnce once;
  FK_CUDA_OK(set_max_dynamic_smem(once, delta_scan_chunk_kernel<DP, WARPS>, kSmem));
  const dim3 grid((unsigned)p.heads, (unsigned)p.num_portions,
                  (unsigned)((p.d + 16 * WARPS - 1) / (16 * WARPS)));
  FK_CUDA_OK(launch_kernel_after(delta_scan_chunk_kernel<DP, WARPS>, grid, dim3(32 * WARPS), kSmem,
                                 s, p));
  count_launch();
  return FK_OK;
}
static int launch_scan_chunks(const DeltaScanParams& p, int dp, cudaStream_t s) {
  // heads of 128 channels: as two CTAs while every head of every portion has an SM to itself (24
  // heads: one portion of 1500 tokens 471 -> 290 us, five of 700 to 2400 749 -> 520); more of them
  // share a record's copy between all columns
  if (dp == 64) return launch_scan_chunks<64, 4>(p, s);
  return p.heads * (int64_t)p.num_portions <= sm_count() ? launch_scan_chunks<128, 4>(p, s)
                                                             : launch_scan_chunks<128, 8>(p, s);
}
// LANES x CPL for single tokens, BL x BC for blocks
template <int LANES, int CPL, int BL, int BC>
static int launch_scan(DeltaScanParams& p, int blocked, cudaStream_t s) {
  if constexpr (LANES * CPL == 64 || LANES * CPL == 128) {
    if (blocked == 2) return launch_scan_chunks(p, LANES * CPL, s);
  }
  if (!blocked) {
    constexpr int COLS = DL_THREADS / LANES * 2;
    const dim3 grid((unsigned)((p.d + COLS - 1) / COLS), (unsigned)p.heads,
                    (unsigned)p.num_portions);
    FK_CUDA_OK(launch_kernel(delta_scan_kernel<LANES, CPL, 2>, grid, dim3(DL_THREADS), 0, s, p));
    count_launch();
    return FK_OK;
  }
  // four columns per thread read a stage's vectors half as often as two; two make a
  // block's instructions fewer where small heads and few sequences do not fill the SMs
  constexpr int COLS4 = DL_THREADS / BL * 4;
  if (p.d > 64 || (p.d > COLS4 / 2 && (int64_t)p.heads * p.num_portions *
                                              ((p.d + COLS4 - 1) / COLS4) >= 2 * sm_count()))
    return launch_scan_blocked<BL, BC, 4>(p, s);
  return launch_scan_blocked<BL, BC, 2>(p, s);
}

}  // namespace fk

using namespace fk;

extern "C" {

// Portions that a form takes: blocks and chunks take all, 3 the ones below, 4 those from 32 tokens on
static int delta_form(int blocked, int* least, int* below) {
  *least = blocked == 4 ? DL_CHUNKS_FROM : 0;
  *below = blocked == 3 ? DL_CHUNKS_FROM : 0x7fffffff;
  return blocked == 3 ? 1 : blocked == 4 ? 2 : blocked;
}

int fk_delta_padded_dim(int dim) {
  return dim <= 0 || dim > DL_MAX_DIM ? 0 : delta_padded(dim);
}

int fk_delta_chunked(int dim) {
  const int dp = fk_delta_padded_dim(dim);
  return dp == 64 || dp == 128;
}

int64_t fk_delta_packed_floats(int64_t rows, int num_portions, int heads, int dim, int blocked) {
  const int dp = fk_delta_padded_dim(dim);
  if (dp == 0 || rows < 0 || num_portions < 0 || heads <= 0) return 0;
  if (blocked == 2 || blocked == 4)
    return fk_delta_chunked(dim) ? heads * (rows / DL_UNIT + num_portions) *
                                       (int64_t)(dl_chunk_bytes(dp) / 4) : 0;
  return blocked ? heads * (rows / DL_UNIT + num_portions) * (DL_UNIT / DL_BLK) *
                       (int64_t)dl_block_floats(dp)
                 : heads * rows * (int64_t)DL_FIELDS * dp;
}

int fk_delta_prepare(const void* r, const void* k, const void* v, const void* a, const void* y1,
                     int64_t in_stride, int is_f32, const void* w2, int64_t w2_stride,
                     const float* w0, const float* a_bias, float* packed, int blocked,
                     const int32_t* cu_portions, int num_portions, int64_t rows,
                     int heads, int dim, int rank, float decay_scale, float unit_eps,
                     fk_stream_t stream) {
  FK_REQUIRE(rows >= 0 && heads > 0 && dim > 0 && rank > 0, FK_ERR_INVALID_ARG,
             "fk_delta_prepare: bad sizes");
  if (rows == 0) return FK_OK;
  FK_REQUIRE(r && k && v && a && y1 && w2 && w0 && a_bias && packed, FK_ERR_INVALID_ARG,
             "fk_delta_prepare: null pointer");
  DeltaPrepParams p{};
  blocked = delta_form(blocked, &p.least, &p.below);
  FK_REQUIRE(!blocked || (cu_portions && num_portions > 0), FK_ERR_INVALID_ARG,
             "fk_delta_prepare: blocks need the portions");
  FK_REQUIRE(blocked != 2 || (fk_delta_chunked(dim) && !is_f32), FK_ERR_UNSUPPORTED,
             "fk_delta_prepare: chunks need bf16 and heads of 33 to 128 channels");
  FK_REQUIRE(dim <= DL_MAX_DIM && rank <= 512 && heads <= 65535 && rows < (1ll << 31),
             FK_ERR_UNSUPPORTED, "fk_delta_prepare: head size %d or rank %d too large", dim, rank);
  FK_REQUIRE(w2_stride % 4 == 0 && w2_stride >= rank && aligned16(w2) && aligned16(packed),
             FK_ERR_ALIGNMENT, "fk_delta_prepare: w2 rows must be padded to 4 elements");
  p.r = r; p.k = k; p.v = v; p.a = a; p.y1 = y1; p.in_stride = in_stride;
  p.w2 = w2; p.w2_stride = w2_stride; p.w0 = w0; p.a_bias = a_bias; p.packed = packed;
  p.cu = cu_portions; p.num_portions = num_portions;
  p.rows = rows; p.units = rows / DL_UNIT + num_portions;
  p.heads = heads; p.d = dim; p.rank = rank; p.rank_p = (rank + 15) / 16 * 16;
  p.decay_scale = decay_scale; p.unit_eps = unit_eps;
  // heads per CTA: the tanh tile is shared by them, as long as the SMs stay busy
  int hpc = 1;
  // (chunks, at most six CTAs an SM: more of them leave a shorter last wave)
  const int least = (blocked == 2 ? 32 : 16) * sm_count();
  while (hpc < 8 && (rows / DL_UNIT + 1) * heads / (hpc * 2) >= least) hpc *= 2;
  p.heads_per_cta = hpc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return is_f32 ? launch_prepare<float>(p, blocked, s) : launch_prepare<uint16_t>(p, blocked, s);
}

int fk_delta_scan(const float* packed, int blocked, float* o, float* state, int num_slots,
                  const int32_t* cu_portions, int num_portions, const int32_t* slots,
                  const int64_t* positions, int64_t rows, int heads, int dim, int32_t* status,
                  fk_stream_t stream) {
  FK_REQUIRE(rows >= 0 && heads > 0 && dim > 0 && num_portions >= 0, FK_ERR_INVALID_ARG,
             "fk_delta_scan: bad sizes");
  if (rows == 0 || num_portions == 0) return FK_OK;
  FK_REQUIRE(packed && o && state && cu_portions && slots && positions && num_slots > 0,
             FK_ERR_INVALID_ARG, "fk_delta_scan: null pointer");
  FK_REQUIRE(dim <= DL_MAX_DIM && heads <= 65535 && num_portions <= 65535, FK_ERR_UNSUPPORTED,
             "fk_delta_scan: head size %d or counts too large", dim);
  DeltaScanParams p{};
  blocked = delta_form(blocked, &p.least, &p.below);
  FK_REQUIRE(blocked != 2 || fk_delta_chunked(dim), FK_ERR_UNSUPPORTED,
             "fk_delta_scan: chunks need heads of 33 to 128 channels");
  FK_REQUIRE(aligned16(packed) && aligned16(state), FK_ERR_ALIGNMENT,
             "fk_delta_scan: 16-byte alignment required");
  p.packed = packed; p.o = o; p.state = state; p.cu = cu_portions; p.slots = slots;
  p.positions = positions; p.rows = rows; p.units = rows / DL_UNIT + num_portions;
  p.heads = heads; p.d = dim; p.num_slots = num_slots; p.num_portions = num_portions;
  p.status = status;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (delta_padded(dim)) {
    case 32: return launch_scan<4, 8, 4, 8>(p, blocked, s);
    case 64: return launch_scan<8, 8, 8, 8>(p, blocked, s);
    case 128: return launch_scan<16, 8, 16, 8>(p, blocked, s);
    default: return launch_scan<32, 8, 32, 8>(p, blocked, s);
  }
}

}  // extern "C"

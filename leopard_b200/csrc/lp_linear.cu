// leopard_b200 — general linear layers for the 32-bit residual-stream models (any M, N, K; fp32 or bf16 activations).
//
//   lp_linear          C[M,N] = epi(A[M,K] · W[N,K]^T): A fp32 or bf16, W bf16 (nn.Linear layout), C fp32 or bf16, accumulation in
//                      fp32 (with fp32 A this is a true 32-bit product: the bf16 weight is exact, no operand is rounded).  Epilogues: none, xIELU, squared relu, and the gated units silu, gelu (tanh form)
//                      and the clamped one (W = [gate rows; up rows], C has N/2 columns).  Before the epilogue every accumulator may be multiplied by a
//                      number per output row (row_scale: a router weight that multiplies an expert's INPUT is the same as one
//                      that multiplies its first products) and take a bias per weight row.  With c_accum the result is scaled
//                      and ADDED to C (the residual update of a pre-norm layer); with `gate` it is first multiplied by
//                      sigmoid(gate[m, n]) (a gated residual branch closes in the store of its last product).
//                      seg_cols: groups of output columns that read operands of their own (a mixer whose projections see different
//                      mixes of the stream) in one launch.  `batch` independent problems with element strides (per-head products of latent attention).
//                      Operands whose rows are whole 16-byte pieces run on the matrix instructions, weight-streaming kernels for up to 64
//                      rows (through a TMA ring where rows and sizes allow) and 64 x 128 tiles for more; fp32 rows as three bf16 terms that add up to them exactly.  The others run on
//                      two fp32-FMA kernels: a 64 x 64 x 16 shared-memory tile kernel, and one with one warp
//                      per output column for M <= 8 rows (decode: every weight byte is read once, 16-byte loads).
//   lp_linear_grouped  the same tile kernel over row tiles that each belong to one group (expert): tile t multiplies rows
//                      [64 t, 64 t + 64) of the padded, group-sorted row space by the weight of group tile_group[t] (< 0: skip);
//                      a_rows (optional) gathers the A row of each sorted row (< 0: a padding row, computed as zero).
//
// The tcgen05 GEMM (lp_gemm_bf16) stays the matrix product of large bf16 problems; these kernels cover what it does not take:
// fp32 operands, arbitrary shapes, few rows, and row-indexed groups whose sizes are only known on the device.
#include <cuda_pipeline.h>
#include "lp_common.cuh"
#include "lp_host.h"
#include "../../include/leopard_b200.h"

namespace lp {

typedef __nv_bfloat16 bf16;

constexpr int LIN_BM = 64, LIN_BN = 64, LIN_BK = 16, LIN_THREADS = 256;

struct LinArgs {
  const void* A; long long lda; long long a_batch;
  const bf16* W; long long ldw; long long w_batch;
  void* C; long long ldc; long long c_batch;
  int M, N, K;            // N = rows of W that are used (gated: 2 x output columns)
  int epi; float e0, e1;  // lp_linear_epi and its two constants
  int c_accum; float c_scale;   // C <- C + c_scale * epi(A W^T) instead of C <- epi(A W^T)
  const int* a_rows;      // grouped: source row of each sorted row, or NULL
  const int* tile_group;  // grouped: group of each row tile, or NULL
  const int* z_group;     // pairs (rows kernel): weight group of problem z, or NULL; problem z reads A row z / a_div and writes C row z
  int a_div;
  const float* bias;      // [N] added to the accumulators before the epilogue, or NULL
  const float* row_scale; // [rows of C] multiplies the accumulators before the bias, or NULL
  int seg_cols, n_segs; long long a_seg;   // seg_cols > 0: output columns [i seg_cols, (i + 1) seg_cols) read A + i a_seg (the last of n_segs: all that follow)
  int w_constant;         // nothing that may still run writes W (LP_LINEAR_W_CONSTANT): its first pieces are asked for before the launch before has ended
  const float* gate; long long ldg, gate_batch;   // [rows of C, N'] pre-activations: the result is multiplied by sigmoid(gate), or NULL
};

// elements between A and the operand of the columns from n on
__device__ __forceinline__ long long lin_seg(const LinArgs& a, int n) {
  if (a.seg_cols <= 0) return 0;
  const int i = n / a.seg_cols;
  return (long long)(i < a.n_segs ? i : a.n_segs - 1) * a.a_seg;
}

__device__ __forceinline__ float lin_load(const float* p) { return *p; }
__device__ __forceinline__ float lin_load(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void lin_store(float* p, float v) { *p = v; }
__device__ __forceinline__ void lin_store(bf16* p, float v) { *p = __float2bfloat16(v); }

// eight bf16 values of a 16-byte load -> fp32 (a bf16 is the upper half of an fp32)
__device__ __forceinline__ void bf16x8_to_f32(const uint4& u, float* f) {
  f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
  f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
  f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
  f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
}

// xIELU with a = softplus(p), b = 1/2 + softplus(q):  z > 0: a z^2 + z/2;  z <= 0: b (exp(z) - 1 - z) + z/2
__device__ __forceinline__ float xielu_f(float z, float a, float b) {
  return z > 0.f ? a * z * z + 0.5f * z : b * (expm1f(z) - z) + 0.5f * z;
}
__device__ __forceinline__ float silu32_f(float z) { return z / (1.0f + expf(-z)); }

__device__ __forceinline__ float lin_epi(int epi, float v, float e0, float e1) {
  if (epi == LP_EPI_RELU2) {      // the square of relu
    const float r = fmaxf(v, 0.f);
    return r * r;
  }
  return epi == LP_EPI_XIELU ? xielu_f(v, e0, e1) : v;
}

// tanh-form gelu: 1/2 (1 + tanh t) is sigmoid(2 t), so one exponential serves
__device__ __forceinline__ float gelu_tanh32_f(float z) {
  const float t = 0.7978845608028654f * fmaf(0.044715f * z * z, z, z);      // sqrt(2 / pi) (z + 0.044715 z^3)
  return z / (1.0f + expf(-2.0f * t));
}

// the gated units: silu(g) * u, gelu(g) * u, and g' sigmoid(e1 g') (u' + 1) with g' = min(g, e0), u' = clamp(u, -e0, e0)
__device__ __forceinline__ float lin_gate(int epi, float g, float u, float e0, float e1) {
  if (epi == LP_EPI_CLAMP_GLU) {
    g = fminf(g, e0);
    u = fminf(fmaxf(u, -e0), e0);
    return g / (1.0f + expf(-e1 * g)) * (u + 1.0f);
  }
  if (epi == LP_EPI_GELU_GATE) return gelu_tanh32_f(g) * u;
  return silu32_f(g) * u;
}

// 64 x 64 output tile per CTA, 4 x 4 outputs per thread, K in steps of 16 through shared memory.  GATED: two accumulator sets, the
// second one for weight row n + N/2; the output is silu(first) * second.
template <typename AT, typename CT, bool GATED>
__global__ void __launch_bounds__(LIN_THREADS) linear_tile_kernel(LinArgs a) {
  __shared__ float As[LIN_BK][LIN_BM + 4];
  __shared__ float Ws[GATED ? 2 : 1][LIN_BK][LIN_BN + 4];
  const int tid = threadIdx.x;
  const int tile_m = blockIdx.y, tile_n = blockIdx.x, z_id = blockIdx.z;
  int group = 0;
  if (a.tile_group != nullptr) {
    group = a.tile_group[tile_m];
    if (group < 0) return;
  }
  const int n_out = GATED ? a.N / 2 : a.N;
  const AT* A = reinterpret_cast<const AT*>(a.A) + (long long)z_id * a.a_batch + lin_seg(a, tile_n * LIN_BN);
  const bf16* W = a.W + (long long)(z_id + group) * a.w_batch;   // grouped launches have one batch: z_id = 0
  CT* C = reinterpret_cast<CT*>(a.C) + (long long)z_id * a.c_batch;
  const int m0 = tile_m * LIN_BM, n0 = tile_n * LIN_BN;
  // loader mapping: 256 threads x 4 elements = 64 rows x 16 k
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  long long a_row = -1;
  if (m0 + lr < a.M) {
    a_row = m0 + lr;
    if (a.a_rows != nullptr) a_row = a.a_rows[m0 + lr];
  }
  const int w_row = n0 + lr;
  float acc[4][4], acc2[GATED ? 4 : 1][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[i][j] = 0.f;
      if (GATED) acc2[i][j] = 0.f;
    }
  const int tm = (tid >> 4) * 4, tn = (tid & 15) * 4;
  for (int k0 = 0; k0 < a.K; k0 += LIN_BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + lk + i;
      As[lk + i][lr] = (a_row >= 0 && k < a.K) ? lin_load(A + a_row * a.lda + k) : 0.f;
      Ws[0][lk + i][lr] = (w_row < n_out && k < a.K) ? __bfloat162float(W[(long long)w_row * a.ldw + k]) : 0.f;
      if (GATED) Ws[1][lk + i][lr] = (w_row < n_out && k < a.K) ? __bfloat162float(W[(long long)(w_row + n_out) * a.ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < LIN_BK; ++kk) {
      float av[4], wv[4], wv2[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        av[i] = As[kk][tm + i];
        wv[i] = Ws[0][kk][tn + i];
        if (GATED) wv2[i] = Ws[1][kk][tn + i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
          if (GATED) acc2[i][j] = fmaf(av[i], wv2[j], acc2[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + tm + i;
    if (m >= a.M) continue;
    const float rs = a.row_scale != nullptr ? a.row_scale[m] : 1.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tn + j;
      if (n >= n_out) continue;
      float z = acc[i][j] * rs, z2 = GATED ? acc2[i][j] * rs : 0.f;
      if (a.bias != nullptr) {
        z += a.bias[n];
        if (GATED) z2 += a.bias[n + n_out];
      }
      float v = GATED ? lin_gate(a.epi, z, z2, a.e0, a.e1) : lin_epi(a.epi, z, a.e0, a.e1);
      if (a.gate != nullptr) v /= 1.0f + expf(-a.gate[(long long)z_id * a.gate_batch + (long long)m * a.ldg + n]);
      if (a.c_accum) v = fmaf(a.c_scale, v, lin_load(C + (long long)m * a.ldc + n));
      lin_store(C + (long long)m * a.ldc + n, v);
    }
  }
}

// Few rows (M <= 8): one warp per output column, the lanes split K; the weight row is read once with 16-byte loads when K allows.
// The rows of A are staged in shared memory K-chunk by K-chunk (fp32, laid out so that the lanes' eight consecutive k of one
// 16-byte weight load fall into different banks) and shared by the CTA's eight columns.
constexpr int ROWS_MAX = 8, ROWS_WARPS = 8, ROWS_KC = 512, ROWS_LD = ROWS_KC / 8 + 1;
__device__ __forceinline__ int rows_slot(int kk) { return (kk & 7) * ROWS_LD + (kk >> 3); }
template <typename AT, typename CT, bool GATED>
__global__ void __launch_bounds__(ROWS_WARPS * 32) linear_rows_kernel(LinArgs a) {
  __shared__ float As[ROWS_MAX][8 * ROWS_LD];
  const int lane = threadIdx.x & 31;
  const int n = blockIdx.x * ROWS_WARPS + (threadIdx.x >> 5);
  const int z = blockIdx.z;
  const int n_out = GATED ? a.N / 2 : a.N;
  const bool active = n < n_out;
  const bool pairs = a.z_group != nullptr;
  const int M = pairs ? 1 : a.M;
  const AT* A = reinterpret_cast<const AT*>(a.A) + (pairs ? (long long)(z / a.a_div) * a.lda : (long long)z * a.a_batch) +
                lin_seg(a, blockIdx.x * ROWS_WARPS);
  const bf16* W = a.W + (long long)(pairs ? a.z_group[z] : z) * a.w_batch;
  CT* C = reinterpret_cast<CT*>(a.C) + (pairs ? (long long)z * a.ldc : (long long)z * a.c_batch);
  const bf16* w1 = W + (long long)(active ? n : 0) * a.ldw;
  const bf16* w2 = W + (long long)(active ? n + n_out : 0) * a.ldw;
  float acc[ROWS_MAX], acc2[GATED ? ROWS_MAX : 1];
#pragma unroll
  for (int m = 0; m < ROWS_MAX; ++m) {
    acc[m] = 0.f;
    if (GATED) acc2[m] = 0.f;
  }
  const bool vec = (a.K % 8 == 0) && (a.ldw % 8 == 0) && ((reinterpret_cast<uintptr_t>(W) & 15) == 0);
  for (int k0 = 0; k0 < a.K; k0 += ROWS_KC) {
    const int kc = min(ROWS_KC, a.K - k0);
    __syncthreads();
    for (int i = threadIdx.x; i < M * kc; i += blockDim.x) {
      const int m = i / kc, kk = i % kc;
      As[m][rows_slot(kk)] = lin_load(A + (long long)m * a.lda + k0 + kk);
    }
    __syncthreads();
    if (!active) continue;
    if (vec) {
      for (int kk = lane * 8; kk < kc; kk += 256) {
        const uint4 u1 = *reinterpret_cast<const uint4*>(w1 + k0 + kk);
        uint4 u2 = u1;
        if (GATED) u2 = *reinterpret_cast<const uint4*>(w2 + k0 + kk);
        float f1[8], f2[8];
        bf16x8_to_f32(u1, f1);
        bf16x8_to_f32(u2, f2);
        const int base = kk >> 3;
#pragma unroll
        for (int m = 0; m < ROWS_MAX; ++m) {
          if (m < M) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float x = As[m][i * ROWS_LD + base];
              acc[m] = fmaf(x, f1[i], acc[m]);
              if (GATED) acc2[m] = fmaf(x, f2[i], acc2[m]);
            }
          }
        }
      }
    } else {
      for (int kk = lane; kk < kc; kk += 32) {
        const float f1 = __bfloat162float(w1[k0 + kk]);
        const float f2 = GATED ? __bfloat162float(w2[k0 + kk]) : 0.f;
#pragma unroll
        for (int m = 0; m < ROWS_MAX; ++m) {
          if (m < M) {
            const float x = As[m][rows_slot(kk)];
            acc[m] = fmaf(x, f1, acc[m]);
            if (GATED) acc2[m] = fmaf(x, f2, acc2[m]);
          }
        }
      }
    }
  }
  if (!active) return;
#pragma unroll
  for (int m = 0; m < ROWS_MAX; ++m) {
    if (m < M) {
      float s = acc[m], s2 = GATED ? acc2[m] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        if (GATED) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      }
      if (lane == 0) {
        if (a.row_scale != nullptr) {
          const float rs = a.row_scale[pairs ? z : m];
          s *= rs;
          s2 *= rs;
        }
        if (a.bias != nullptr) {
          s += a.bias[n];
          if (GATED) s2 += a.bias[n + n_out];
        }
        float v = GATED ? lin_gate(a.epi, s, s2, a.e0, a.e1) : lin_epi(a.epi, s, a.e0, a.e1);
        if (a.gate != nullptr) v /= 1.0f + expf(-a.gate[(pairs ? 0 : (long long)z * a.gate_batch) + (long long)(pairs ? z : m) * a.ldg + n]);
        if (a.c_accum) v = fmaf(a.c_scale, v, lin_load(C + (long long)m * a.ldc + n));
        lin_store(C + (long long)m * a.ldc + n, v);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// Up to 64 rows (decoding): a product is bound by reading its weights once, at every number of rows, when the multiply-adds are
// out of the way.  So the weight tile is the 16-row operand of the warp's matrix instruction and up to MG groups of eight rows of A
// are its other one: a CTA owns 16 NT output columns, its warps share out K in steps of 32 (a lane reads 16 bytes of each weight row and of its
// row of A; the same permutation of k on both sides, which a sum does not see), 4 NT weight loads per lane (2 NT from 17 rows on, where registers
// are short) are in flight before the first product, and the warps' sums meet in shared memory in a fixed order; up to 16 rows, and for pairs,
// what each addition rounds off is kept and added at the end (one-row kernels did these before; with more rows it costs up to 8 % of short
// products).  The gated units take gate row n and up row n + N / 2 as rows g and g + 8 of one tile, so both halves of an output end up in one lane.
// fp32 rows of A are cut into three bf16 terms that add up to them exactly (8 + 8 + 8 bits): every product is still exact.  The
// instruction cuts its running sum off instead of rounding it, a bias that grows with the chain.  So chains are short and added in fp32: 16
// products of bf16 rows, 3 x 16 of fp32 rows (small terms first), 256 of 33 to 64 bf16 rows, whose additions would cost more than the products.
// Measured (B200, graph of launches, weights from HBM, M = 8): N = 8192, K = 2048 10.4 us (3.2 TB/s; a warp per column with fp32 FMAs: 67.6),
// N = 32000, K = 4096 51 us (5.1 TB/s; 350), N = 2048, K = 2048 6.6 us (29.7), fp32 A 6.5 us (66).  Error against 64 bits at N = 2048, K = 2048 /
// 8192, 1e-7 of the result: bf16 rows 0.58 / 0.70 (without what the sums of the warps round off 0.92 / 1.23; FMA chains of a lane, which this
// kernel replaced, 0.80 / 1.24), fp32 rows 0.75 / 1.0 (1.6 / 2.9), 64 bf16 rows 2.3 / 2.4 (FMA chains over K 3.9 / 9.5).
// Pairs (experts): the CTAs of weight group blockIdx.y gather the pairs that chose it and read the group's weights once for all of them.
constexpr int STREAM_MAX_ROWS = 64, STREAM_MAX_PAIRS = 1024;

struct Bf16Terms { uint4 hi, mid, lo; };
__device__ __forceinline__ float4 as_floats(const uint4& u) {
  return make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
}
__device__ __forceinline__ uint32_t pack_upper(float x, float y) { return (__float_as_uint(x) >> 16) | (__float_as_uint(y) & 0xffff0000u); }
__device__ __forceinline__ uint32_t take_upper(float& x, float& y) {      // what is left of x and y stays behind
  const uint32_t r = pack_upper(x, y);
  x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
  y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
  return r;
}
__device__ __forceinline__ Bf16Terms split3(const float4& a, const float4& b) {
  float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  Bf16Terms r;
  bool odd = false;
#pragma unroll
  for (int i = 0; i < 8; ++i) odd |= (__float_as_uint(v[i]) & 0x7f800000u) == 0x7f800000u;
  if (odd) {      // an infinity leaves nothing behind, a NaN stays one without its lower bits
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t u = __float_as_uint(v[i]);
      const bool whole = (u & 0x7f800000u) == 0x7f800000u;
      w[i] = !whole ? v[i] - __uint_as_float(u & 0xffff0000u) : 0.f;
      if (whole && (u & 0x7fffffu)) v[i] = __uint_as_float(u | 0x400000u);
    }
    r.hi = make_uint4(pack_upper(v[0], v[1]), pack_upper(v[2], v[3]), pack_upper(v[4], v[5]), pack_upper(v[6], v[7]));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = w[i];
  } else {
    r.hi.x = take_upper(v[0], v[1]); r.hi.y = take_upper(v[2], v[3]); r.hi.z = take_upper(v[4], v[5]); r.hi.w = take_upper(v[6], v[7]);
  }
  r.mid.x = take_upper(v[0], v[1]); r.mid.y = take_upper(v[2], v[3]); r.mid.z = take_upper(v[4], v[5]); r.mid.w = take_upper(v[6], v[7]);
  r.lo = make_uint4(pack_upper(v[0], v[1]), pack_upper(v[2], v[3]), pack_upper(v[4], v[5]), pack_upper(v[6], v[7]));
  return r;
}
// s <- s + v, rounded; the exact rest of that sum (Knuth's two-sum)
__device__ __forceinline__ float add_exactly(float& s, float v) {
  const float t = s + v, u = t - s;
  const float rest = (s - (t - u)) + (v - u);
  s = t;
  return rest;
}
// An infinite weight times a term that is zero, or of the other sign, is a NaN that the product of the uncut number is not.  So sums of three-term
// rows that are not finite are looked at once more, a CTA at a time: each that is NaN is taken again in fp32 multiply-adds (a NaN ends the
// walk: it stays one).  The walks are functions of their own: in the epilogues their registers made the tile kernel spill (5 to 17 % slower).
template <typename AT>
__device__ float lin_plain_dot(const AT* x, const bf16* w, int K) {
  float s = 0.f;
#pragma unroll 1
  for (int k = 0; k < K && s == s; ++k) s = fmaf(lin_load(x + k), lin_load(w + k), s);
  return s;
}
template <typename AT>
__device__ __noinline__ float lin_plain_sum(const AT* x, const bf16* w, int K) { return lin_plain_dot(x, w, K); }
// linear_stream_kernel: `here` rows from m0 on, the first warp's share takes the new sum
template <typename AT, int NT, int MG>
__device__ __noinline__ void lin_mend_sums(float* sums, const AT* A, long long lda, const int* pair_of, int a_div, const bf16* W, long long ldw, int K,
                                           int m0, int here, int n0, int n_out, int gated) {
  const int n_warps = blockDim.x >> 5, cols = gated ? 8 * NT : 16 * NT;
  for (int e = threadIdx.x; e < cols * here; e += blockDim.x) {
    const int nl = e % cols, ml = e / cols, n = n0 + nl;
    if (n >= n_out) continue;
    const int j = gated ? nl >> 3 : nl >> 4, r = gated ? nl & 7 : nl & 15;
    const int at = (((j * MG + (ml >> 3)) * 4 + (r >> 3) * 2 + (ml & 1)) * 32) + (r & 7) * 4 + ((ml & 7) >> 1);
    const AT* x = A + (long long)(pair_of != nullptr ? pair_of[m0 + ml] / a_div : m0 + ml) * lda;
    for (int half = 0; half < (gated ? 2 : 1); ++half) {
      float* p = sums + at + 64 * half;
      float s = 0.f;
      for (int w = 0; w < n_warps; ++w) s += p[w * NT * MG * 4 * 32];
      if (s == s) continue;
      p[0] = lin_plain_dot(x, W + (long long)(n + half * n_out) * ldw, K);
      for (int w = 1; w < n_warps; ++w) p[w * NT * MG * 4 * 32] = 0.f;
    }
  }
  __syncthreads();
}
// the two halves of a step of 32 products, in chains of their own
__device__ __forceinline__ void mma_step(float* d, float* e, const uint4& w0, const uint4& w1, const uint4& x) {
  mma_bf16(d, w0.x, w1.x, w0.y, w1.y, x.x, x.y);
  mma_bf16(e, w0.z, w1.z, w0.w, w1.w, x.z, x.w);
}

template <typename AT, int NT, int MG>
__global__ void __launch_bounds__(MG * NT == 1 && sizeof(AT) == 2 ? 1024 : 512) linear_stream_kernel(LinArgs a, int gated, int c_fp32, int n_pairs) {
  pdl_wait();
  extern __shared__ float dyn_smem[];      // [warps][NT MG 4][32] partial sums
  __shared__ int pair_of[STREAM_MAX_PAIRS];
  __shared__ int pair_count[STREAM_MAX_PAIRS / 32];
  constexpr int U = MG >= 4 ? 1 : 2;      // k steps whose weights are in flight together
  // a warp's steps are neighbours, whole 128-byte lines of the weight rows (one tile: 14.6 us a launch of ronelorn's one-request steps, 13.7 so), or lie n_warps
  // apart (two tiles)
  constexpr bool NEAR = NT == 1;
  constexpr int SLOTS = NT * MG * 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const bool pairs = a.z_group != nullptr;
  const int z = blockIdx.z;
  const int n_out = gated ? a.N / 2 : a.N;
  const int cols = gated ? 8 * NT : 16 * NT;
  const int n0 = blockIdx.x * cols;
  int rows = a.M;
  if (pairs) {      // the group's pairs, in order: a ballot for every 32 of them, then their places
    const int spans = (n_pairs + 31) / 32;
    for (int q = warp; q < spans; q += n_warps) {
      const unsigned m = __ballot_sync(0xffffffffu, q * 32 + lane < n_pairs && a.z_group[q * 32 + lane] == (int)blockIdx.y);
      if (lane == 0) pair_count[q] = __popc(m);
      pair_of[q * 32 + lane] = (m >> lane & 1u) ? __popc(m & ((1u << lane) - 1u)) : -1;
    }
    __syncthreads();
    int at[STREAM_MAX_PAIRS / (4 * 32)];      // the places of this warp's pairs
    int before = 0, k = 0;
    for (int q = 0; q < spans; ++q) {
      if (q % n_warps == warp) {
        const int r = pair_of[q * 32 + lane];
        at[k++] = r >= 0 ? before + r : -1;
      }
      before += pair_count[q];
    }
    __syncthreads();
    k = 0;
    for (int q = warp; q < spans; q += n_warps, ++k)
      if (at[k] >= 0) pair_of[at[k]] = q * 32 + lane;
    __syncthreads();
    rows = before;
    if (rows == 0) return;
  }
  const AT* A = reinterpret_cast<const AT*>(a.A) + (pairs ? 0 : (long long)z * a.a_batch) + lin_seg(a, n0);
  const bf16* W = a.W + (long long)(pairs ? (int)blockIdx.y : z) * a.w_batch;
  const bf16* w0[NT];
  const bf16* w1[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const int r0 = n0 + j * (gated ? 8 : 16) + g, r1 = gated ? r0 + n_out : r0 + 8;
    w0[j] = r0 < n_out ? W + (long long)r0 * a.ldw : nullptr;
    w1[j] = (gated ? r0 : r1) < n_out ? W + (long long)r1 * a.ldw : nullptr;
  }
  const uint4 none = make_uint4(0, 0, 0, 0);
  for (int m0 = 0; m0 < rows; m0 += 8 * MG) {
    const AT* x[MG];
#pragma unroll
    for (int i = 0; i < MG; ++i) {
      const int m = m0 + 8 * i + g;
      x[i] = m < rows ? A + (long long)(pairs ? pair_of[m] / a.a_div : m) * a.lda : nullptr;
    }
    constexpr bool LONG = MG == 8 && sizeof(AT) == 2;      // many rows: chains of eight steps, the additions would cost more than the products
    float acc[NT][MG][4], run[LONG ? NT : 1][LONG ? MG : 1][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < MG; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[j][i][c] = run[LONG ? j : 0][LONG ? i : 0][c] = 0.f;
    int turn = 0;
    auto fetch = [&](int s, uint4 (&u0)[U][NT], uint4 (&u1)[U][NT]) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = (NEAR ? s * U + u : s + u * n_warps) * 32 + t * 8;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          u0[u][j] = k < a.K && w0[j] != nullptr ? ldg_once(w0[j] + k) : none;
          u1[u][j] = k < a.K && w1[j] != nullptr ? ldg_once(w1[j] + k) : none;
        }
      }
    };
    auto take = [&](int s, const uint4 (&u0)[U][NT], const uint4 (&u1)[U][NT]) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = (NEAR ? s * U + u : s + u * n_warps) * 32 + t * 8;
        if constexpr (sizeof(AT) == 2) {
          uint4 v[MG];
#pragma unroll
          for (int i = 0; i < MG; ++i) v[i] = k < a.K && x[i] != nullptr ? *reinterpret_cast<const uint4*>(x[i] + k) : none;
#pragma unroll
          for (int i = 0; i < MG; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              if constexpr (LONG) {
                mma_step(run[j][i], run[j][i], u0[u][j], u1[u][j], v[i]);
              } else {
                float d[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
                mma_step(d, e, u0[u][j], u1[u][j], v[i]);
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[j][i][c] += d[c] + e[c];
              }
            }
        } else {
#pragma unroll
          for (int i = 0; i < MG; ++i) {
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
            if (k < a.K && x[i] != nullptr) {
              p = *reinterpret_cast<const float4*>(x[i] + k);
              q = *reinterpret_cast<const float4*>(x[i] + k + 4);
            }
            const Bf16Terms v = split3(p, q);
#pragma unroll
            for (int j = 0; j < NT; ++j) {      // the small terms first
              float d[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
              mma_step(d, e, u0[u][j], u1[u][j], v.lo);
              mma_step(d, e, u0[u][j], u1[u][j], v.mid);
              mma_step(d, e, u0[u][j], u1[u][j], v.hi);
#pragma unroll
              for (int c = 0; c < 4; ++c) acc[j][i][c] += d[c] + e[c];
            }
          }
        }
      }
      if constexpr (LONG) {
        if ((++turn & 7) == 0) {
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int i = 0; i < MG; ++i)
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                acc[j][i][c] += run[j][i][c];
                run[j][i][c] = 0.f;
              }
        }
      }
    };
    uint4 a0[U][NT], a1[U][NT];
    // one tile of up to eight bf16 rows leaves registers free: the next steps' weights are asked for before these are used (K = N = 4096, one row: 10.6 us,
    // 8.7 so; fp32 rows 4.6, 5.3: their registers cost CTAs)
    const int stride = NEAR ? n_warps : U * n_warps, steps = NEAR ? (a.K + 32 * U - 1) / (32 * U) : (a.K + 31) / 32;
    if constexpr (MG == 1 && NT == 1 && sizeof(AT) == 2) {
      uint4 b0[U][NT], b1[U][NT];
      fetch(warp, a0, a1);
      for (int s = warp; s < steps; s += 2 * stride) {
        fetch(s + stride, b0, b1);
        take(s, a0, a1);
        if (s + stride >= steps) break;
        fetch(s + 2 * stride, a0, a1);
        take(s + stride, b0, b1);
      }
    } else {
      for (int s = warp; s < steps; s += stride) {
        fetch(s, a0, a1);
        take(s, a0, a1);
      }
    }
    if constexpr (LONG) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < MG; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[j][i][c] += run[j][i][c];
    }
    if (m0 > 0) __syncthreads();      // the sums of the rows before have been read
    bool odd = false;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < MG; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          dyn_smem[(warp * SLOTS + (j * MG + i) * 4 + c) * 32 + lane] = acc[j][i][c];
          if constexpr (sizeof(AT) == 4) odd |= not_finite(acc[j][i][c]);
        }
    const int here = min(8 * MG, rows - m0);
    if constexpr (sizeof(AT) == 4) {
      if (__syncthreads_or(odd))
        lin_mend_sums<AT, NT, MG>(dyn_smem, A, a.lda, pairs ? pair_of : nullptr, a.a_div, W, a.ldw, a.K, m0, here, n0, n_out, gated);
    } else {
      __syncthreads();
    }
    for (int e = threadIdx.x; e < cols * here; e += blockDim.x) {
      const int nl = e % cols, ml = e / cols, n = n0 + nl;
      if (n >= n_out) continue;
      const int j = gated ? nl >> 3 : nl >> 4, r = gated ? nl & 7 : nl & 15;
      const int at = (((j * MG + (ml >> 3)) * 4 + (r >> 3) * 2 + (ml & 1)) * 32) + (r & 7) * 4 + ((ml & 7) >> 1);
      float s = 0.f, s2 = 0.f;
      if (MG <= 2 || pairs) {      // what the additions round off is added at the end
        float lost = 0.f, lost2 = 0.f;
        for (int w = 0; w < n_warps; ++w) {
          lost += add_exactly(s, dyn_smem[w * SLOTS * 32 + at]);
          if (gated) lost2 += add_exactly(s2, dyn_smem[w * SLOTS * 32 + at + 64]);
        }
        if (s + lost == s + lost) s += lost;      // beside an infinity the rest is NaN
        if (s2 + lost2 == s2 + lost2) s2 += lost2;
      } else {
        for (int w = 0; w < n_warps; ++w) {
          s += dyn_smem[w * SLOTS * 32 + at];
          if (gated) s2 += dyn_smem[w * SLOTS * 32 + at + 64];
        }
      }
      const int m = pairs ? pair_of[m0 + ml] : m0 + ml;
      if (a.row_scale != nullptr) {
        s *= a.row_scale[m];
        s2 *= a.row_scale[m];
      }
      if (a.bias != nullptr) {
        s += a.bias[n];
        if (gated) s2 += a.bias[n + n_out];
      }
      float v = gated ? lin_gate(a.epi, s, s2, a.e0, a.e1) : lin_epi(a.epi, s, a.e0, a.e1);
      if (a.gate != nullptr) v /= 1.0f + expf(-a.gate[(pairs ? 0 : (long long)z * a.gate_batch) + (long long)m * a.ldg + n]);
      const long long at_c = (pairs ? 0 : (long long)z * a.c_batch) + (long long)m * a.ldc + n;
      if (c_fp32) {
        float* C = reinterpret_cast<float*>(a.C) + at_c;
        *C = a.c_accum ? fmaf(a.c_scale, v, *C) : v;
      } else {
        bf16* C = reinterpret_cast<bf16*>(a.C) + at_c;
        *C = __float2bfloat16(a.c_accum ? fmaf(a.c_scale, v, __bfloat162float(*C)) : v);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// The same product as one stream of weights: a CTA an SM walks its tiles of 16 or 32 weight rows, and one thread keeps a ring of pieces
// of them full by TMA, so that DRAM sees whole kilobytes and the next pieces are under way while the sums of a tile are
// stored.  Eight warps take the products of a piece, four others add up their sums and store the tile before: nothing in the stream waits for
// an epilogue.  Where no launch before this one writes the weights (w_constant), the ring is filled before that launch has ended.
// What bounds it is DRAM from about 30 MB of weights on (K = 4096, N = 32000: 39 us, 6.7 TB/s; the kernel above 46 at one row and 62 at 16; N = 16384 21.3 and
// 24.7), below that the latency of a launch (K = N = 2048 3.7 us, 4.9).  A piece has to be large: at half of these sizes the waits between
// pieces took the issue slots (39 -> 49 us), and bulk copies of a row each cost 110 cycles of a warp.  192 KB of pieces under way an SM (one to eight bf16 rows: 128 KB of them weights, which
// alone are asked for before the wait): with 96 KB the same took 50 us.
// The weights leave the L2 first: left to its usual order, they threw out the caches and states of the small kernels around them (window attention of one row 13 ->
// 23 us).  Sums: 16 products a chain, which the instruction cuts off, then exactly; error against 64 bits, 1e-7 of the result: 0.5 for bf16 rows, 0.7 for fp32
// rows at every K (above: 0.5 to 1.2 and 0.7 to 1.2); more than 16 rows are added up plainly, 0.6 and 0.75 at K = 1024 (above: 0.9 to 1.3 and 0.9 to 1.0).
constexpr int RING_TAKERS = 8, RING_STORERS = 4, RING_WARPS = 2 + RING_TAKERS + RING_STORERS, RING_MAX_STAGES = 8, RING_MAX_GROUPS = 256;
constexpr int RING_BYTES = 208 * 1024;      // of pieces and sums
// A piece is KC columns of 16 NT weight rows and of the rows of A, boxes of 8 rows x 128 bytes one after another: a warp takes KC / 32 / 8 steps of it between two waits.
// More rows of A take more of the ring: fewer columns of them.
template <typename AT, int MG> constexpr int ring_kc() { return MG == 8 ? 256 : MG == 4 ? (sizeof(AT) == 2 ? 512 : 256) : sizeof(AT) == 2 ? 1024 : 512; }
template <typename AT, int NT, int MG> constexpr int ring_w() { return NT * 16 * ring_kc<AT, MG>() * 2; }
// the rows of pairs lie apart and come by a bulk copy each: bytes from one to the next (four lanes' pieces of two rows are in banks of their own)
template <typename AT, int MG> constexpr int ring_pair_row() { return ring_kc<AT, MG>() * (int)sizeof(AT) + (sizeof(AT) == 2 ? 64 : 16); }
template <typename AT, int NT, int MG, bool PAIRS> constexpr int ring_piece() {
  return ring_w<AT, NT, MG>() + (PAIRS ? (8 * MG * ring_pair_row<AT, MG>() + 1023) / 1024 * 1024 : 8 * MG * ring_kc<AT, MG>() * (int)sizeof(AT));
}
template <int MG> constexpr int ring_bufs() { return MG <= 2 ? 2 : 1; }      // tiles of sums: more rows leave room for one
template <int NT, int MG> constexpr int ring_sums() { return ring_bufs<MG>() * RING_TAKERS * NT * MG * 4 * 32 * (int)sizeof(float); }
template <typename AT, int NT, int MG, bool PAIRS> constexpr int ring_stages() {
  constexpr int n = (RING_BYTES - ring_sums<NT, MG>()) / ring_piece<AT, NT, MG, PAIRS>();
  return n < RING_MAX_STAGES ? n : RING_MAX_STAGES;
}

template <typename AT, int NT, int MG, bool PAIRS>
__global__ void __launch_bounds__(RING_WARPS * 32, 1) linear_ring_kernel(const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap ta, LinArgs a,
                                                                         int gated, int c_fp32, int batch, int n_pairs, int n_groups) {
  extern __shared__ float dyn_smem[];      // (from the next multiple of 1024 bytes) [stages] pieces, then [BUFS][takers][NT MG 4][32] sums
  __shared__ uint64_t full[RING_MAX_STAGES], empty[RING_MAX_STAGES], sums_full[2], sums_empty[2];
  __shared__ int pair_of[PAIRS ? STREAM_MAX_PAIRS : 1];      // the pairs, a group's together
  __shared__ int count[PAIRS ? RING_MAX_GROUPS : 1];
  __shared__ int2 block_of[PAIRS ? RING_MAX_GROUPS + STREAM_MAX_PAIRS / 8 : 1];      // {group, place of its first pair, number of pairs << 16} of up to 8 MG of a group's pairs
  __shared__ int n_blocks;
  constexpr int KC = ring_kc<AT, MG>(), STEPS = KC / 32 / RING_TAKERS, SLOTS = NT * MG * 4, PIECE = ring_piece<AT, NT, MG, PAIRS>(), STAGES = ring_stages<AT, NT, MG, PAIRS>();
  constexpr int HALF = 8 * KC * 2;      // eight weight rows
  constexpr int BUFS = ring_bufs<MG>();
  constexpr bool EXACT = MG <= 2;      // what the additions round off is kept; the kernel above has longer chains with more rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n_out = gated ? a.N / 2 : a.N, cols = gated ? 8 * NT : 16 * NT, tiles = (n_out + cols - 1) / cols;
  uint8_t* const ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~(uintptr_t)1023);
  float* const sums = reinterpret_cast<float*>(ring + STAGES * PIECE);
  const int pieces = (a.K + KC - 1) / KC;
  const bool ahead = !PAIRS && a.w_constant != 0;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], RING_TAKERS);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sums_full[i], RING_TAKERS);
      mbar_init(&sums_empty[i], RING_STORERS);
    }
    fence_barrier_init();
  }
  if constexpr (PAIRS) {      // the pairs of each group, in order: counts, places, blocks of up to 8 MG
    pdl_wait();
    const int spans = (n_pairs + 31) / 32;
    for (int e = warp; e < n_groups; e += RING_WARPS) {
      int c = 0;
      for (int q = 0; q < spans; ++q) c += __popc(__ballot_sync(0xffffffffu, q * 32 + lane < n_pairs && a.z_group[q * 32 + lane] == e));
      if (lane == 0) count[e] = c;
    }
    __syncthreads();
    for (int e = warp; e < n_groups; e += RING_WARPS) {
      if (count[e] == 0) continue;
      int place = 0, block = 0;
      for (int i = 0; i < e; ++i) {
        place += count[i];
        block += (count[i] + 8 * MG - 1) / (8 * MG);
      }
      for (int i = lane; i * 8 * MG < count[e]; i += 32) block_of[block + i] = make_int2(e, (place + i * 8 * MG) | (min(8 * MG, count[e] - i * 8 * MG) << 16));
      for (int q = 0; q < spans; ++q) {
        const bool mine = q * 32 + lane < n_pairs && a.z_group[q * 32 + lane] == e;
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (mine) pair_of[place + __popc(m & ((1u << lane) - 1u))] = q * 32 + lane;
        place += __popc(m);
      }
    }
    if (threadIdx.x == 0) {
      int n = 0;
      for (int i = 0; i < n_groups; ++i) n += (count[i] + 8 * MG - 1) / (8 * MG);
      n_blocks = n;
    }
  }
  __syncthreads();
  const int units = tiles * (PAIRS ? n_blocks : batch);
  struct Unit { int n0, z, first, here; };      // its first output column, its problem or group, its rows (PAIRS: from place `first` on)
  auto unit_at = [&](int u) {
    Unit r;
    const int b = u / tiles;
    r.n0 = (u - b * tiles) * cols;
    if constexpr (PAIRS) {
      const int2 v = block_of[b];
      r.z = v.x;
      r.first = v.y & 0xffff;
      r.here = v.y >> 16;
    } else {
      r.z = b;
      r.first = 0;
      r.here = a.M;
    }
    return r;
  };
  auto row_of = [&](const Unit& u, int m) {      // row m of a unit's operand
    const AT* A = reinterpret_cast<const AT*>(a.A);
    if constexpr (PAIRS) return A + (long long)(pair_of[u.first + m] / a.a_div) * a.lda;
    return A + (long long)u.z * a.a_batch + lin_seg(a, u.n0) + (long long)m * a.lda;
  };
  if (warp == 0) {
    // ---------------------------------------------------------------- copies
    const uint64_t once = read_once_policy();
    struct At { int u, piece; Unit unit; };      // a place in the stream of this CTA's pieces
    auto next = [&](At& p) {
      if (++p.piece < pieces) return;
      p.piece = 0;
      p.u += gridDim.x;
      if (p.u < units) p.unit = unit_at(p.u);
    };
    auto load_w = [&](const At& p, int stage) {
      if (lane != 0) return;
      const int kc = min(KC, a.K - p.piece * KC);
      mbar_arrive_expect_tx(&full[stage], (uint32_t)(ring_w<AT, NT, MG>() + (PAIRS ? p.unit.here * kc : 8 * MG * KC) * (int)sizeof(AT)));
#pragma unroll
      for (int h = 0; h < 2 * NT; ++h) {
        const int n = gated ? p.unit.n0 + (h >> 1) * 8 + (h & 1) * n_out : p.unit.n0 + h * 8;
        tma_load_4d_once(ring + stage * PIECE + h * HALF, &tw, &full[stage], 0, n, p.piece * (KC / 64), p.unit.z, once);
      }
    };
    auto load_a = [&](const At& p, int stage) {
      if (PAIRS || lane != 0) return;
      const int z = a.seg_cols > 0 ? min(p.unit.n0 / a.seg_cols, a.n_segs - 1) : p.unit.z;
#pragma unroll
      for (int i = 0; i < MG; ++i)
        tma_load_4d(ring + stage * PIECE + ring_w<AT, NT, MG>() + i * 8 * KC * (int)sizeof(AT), &ta, &full[stage], 0, 8 * i, p.piece * (KC * (int)sizeof(AT) / 128), z);
    };
    At w{(int)blockIdx.x, 0, {}};
    if (w.u < units) w.unit = unit_at(w.u);
    int stage = 0;
    uint32_t phase = 0;
    if (ahead) {
      At x = w;
      for (; stage < STAGES && w.u < units; ++stage) {
        load_w(w, stage);
        next(w);
      }
      pdl_wait();
      for (int i = 0; i < stage; ++i) {
        load_a(x, i);
        next(x);
      }
      if (stage == STAGES) { stage = 0; phase = 1; }
    } else {
      pdl_wait();
    }
    for (; w.u < units; next(w)) {
      mbar_wait_warp(&empty[stage], phase ^ 1);      // one lane's copies let the ring go on
      load_w(w, stage);
      load_a(w, stage);
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp <= RING_TAKERS) {
    // ---------------------------------------------------------------- products: STEPS steps of 32 columns of every piece are this warp's
    const int cw = warp - 1;
    // row g of a box lies where four lanes' pieces of two rows are in banks of their own
    const int at_row = (g >> 1) | ((g & 1) << 2), x_row = sizeof(AT) == 2 ? at_row : g;
    constexpr int XV = sizeof(AT) == 2 ? 1 : 2;      // 16-byte pieces of eight values of a row
    // this lane's piece of a step in the lower half of a 128-byte line; the upper half's is 64 bytes away, either way
    const int w_at = at_row * 128 + (t ^ at_row) * 16;
    // The columns from K on of a piece are zeros, but for rows of pairs: a bulk copy ends at K and leaves there what was there, maybe a NaN.  K is a multiple of 64, so
    // where a warp takes more columns its last steps are looked at one by one.
    constexpr bool ENDS_WITHIN = PAIRS && STEPS * 32 > 64;
    const int x_at = PAIRS ? g * ring_pair_row<AT, MG>() + t * 8 * (int)sizeof(AT) : sizeof(AT) == 2 ? w_at : x_row * 128;
    int stage = 0, turn = 0;
    uint32_t phase = 0;
    pdl_wait();
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++turn) {
      float acc[NT][MG][4], rest[EXACT ? NT : 1][EXACT ? MG : 1][4];      // rest: what adding the steps' sums rounded off
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < MG; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[j][i][c] = rest[EXACT ? j : 0][EXACT ? i : 0][c] = 0.f;
#pragma unroll 1
      for (int piece = 0; piece < pieces; ++piece) {
        mbar_wait(&full[stage], phase);
        const uint8_t* const base = ring + stage * PIECE;
        uint4 u0[STEPS][NT], u1[STEPS][NT], v[STEPS][MG][XV];
#pragma unroll
        for (int q = 0; q < STEPS; ++q) {
          const int step = STEPS * cw + q, upper = ((STEPS == 1 ? cw : q) & 1) * 64;      // the half of the line
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const uint8_t* const w = base + j * 2 * HALF + (step >> 1) * 1024 + (w_at ^ upper);
            u0[q][j] = *reinterpret_cast<const uint4*>(w);
            u1[q][j] = *reinterpret_cast<const uint4*>(w + HALF);
          }
#pragma unroll
          for (int i = 0; i < MG; ++i)
#pragma unroll
            for (int p = 0; p < XV; ++p) {
              const uint8_t* x = base + ring_w<AT, NT, MG>();
              if constexpr (PAIRS) x += 8 * i * ring_pair_row<AT, MG>() + step * 32 * (int)sizeof(AT) + x_at + 16 * p;
              else if constexpr (sizeof(AT) == 2) x += i * 8 * KC * 2 + (step >> 1) * 1024 + (x_at ^ upper);
              else x += i * 8 * KC * 4 + step * 1024 + x_at + ((2 * t + p) ^ x_row) * 16;
              v[q][i][p] = !ENDS_WITHIN || piece * KC + step * 32 < a.K ? *reinterpret_cast<const uint4*>(x) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        if (piece * KC + STEPS * cw * 32 >= a.K) continue;      // no column of this warp's
#pragma unroll
        for (int i = 0; i < MG; ++i) {
          float sum[NT][STEPS][4];
#pragma unroll
          for (int q = 0; q < STEPS; ++q) {
            Bf16Terms y;
            if constexpr (sizeof(AT) == 4) y = split3(as_floats(v[q][i][0]), as_floats(v[q][i][XV - 1]));
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              float d[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
              if constexpr (sizeof(AT) == 2) {
                mma_step(d, e, u0[q][j], u1[q][j], v[q][i][0]);
              } else {      // the small terms first
                mma_step(d, e, u0[q][j], u1[q][j], y.lo);
                mma_step(d, e, u0[q][j], u1[q][j], y.mid);
                mma_step(d, e, u0[q][j], u1[q][j], y.hi);
              }
#pragma unroll
              for (int c = 0; c < 4; ++c) sum[j][q][c] = d[c] + e[c];
            }
          }
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int q = 0; q < STEPS; ++q) {
                if constexpr (EXACT) rest[j][i][c] += add_exactly(acc[j][i][c], sum[j][q][c]);
                else acc[j][i][c] += sum[j][q][c];
              }
        }
      }
      const int buf = turn % BUFS;
      mbar_wait(&sums_empty[buf], ((turn / BUFS) & 1) ^ 1);
      float* mine = sums + (buf * RING_TAKERS + cw) * SLOTS * 32 + lane;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < MG; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float s = EXACT ? acc[j][i][c] + rest[EXACT ? j : 0][EXACT ? i : 0][c] : acc[j][i][c];
            mine[((j * MG + i) * 4 + c) * 32] = s == s ? s : acc[j][i][c];      // beside an infinity the rest is NaN
          }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sums_full[buf]);
    }
  } else if (warp == RING_WARPS - 1) {
    // ---------------------------------------------------------------- the rows of pairs, which lie apart: a lane each
    if constexpr (PAIRS) {
      int stage = 0;
      uint32_t phase = 0;
      for (int at = blockIdx.x; at < units; at += gridDim.x) {
        const Unit u = unit_at(at);
        const AT* const x = lane < u.here ? row_of(u, lane) : nullptr;
        for (int piece = 0; piece < pieces; ++piece) {
          mbar_wait_warp(&empty[stage], phase ^ 1);      // as many lanes as there are rows let the ring go on
          if (x != nullptr)
            bulk_load(ring + stage * PIECE + ring_w<AT, NT, MG>() + lane * ring_pair_row<AT, MG>(), x + piece * KC,
                      (uint32_t)(min(KC, a.K - piece * KC) * (int)sizeof(AT)), &full[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- the takers' sums in a fixed order, what the additions round off kept; the epilogue
    const int et = threadIdx.x - (1 + RING_TAKERS) * 32;
    int turn = 0;
    pdl_wait();
    for (int at = blockIdx.x; at < units; at += gridDim.x, ++turn) {
      const Unit u = unit_at(at);
      const int buf = turn % BUFS;
      mbar_wait(&sums_full[buf], (turn / BUFS) & 1);
      const float* part = sums + buf * RING_TAKERS * SLOTS * 32;
      for (int e = et; e < cols * u.here; e += RING_STORERS * 32) {
        const int nl = e & (cols - 1), ml = e / cols, n = u.n0 + nl;
        if (n >= n_out) continue;
        const int j = gated ? nl >> 3 : nl >> 4, r = gated ? nl & 7 : nl & 15;
        const int lane_row = ((r & 3) << 1) | ((r & 7) >> 2);      // the lanes' g whose weight row this is
        const int mc = sizeof(AT) == 2 && !PAIRS ? ((ml & 3) << 1) | ((ml & 7) >> 2) : ml & 7;      // and whose row of A
        const int slot = ((j * MG + (ml >> 3)) * 4 + (r >> 3) * 2 + (mc & 1)) * 32 + lane_row * 4 + (mc >> 1);
        float s = 0.f, s2 = 0.f, lost = 0.f, lost2 = 0.f;
#pragma unroll
        for (int w = 0; w < RING_TAKERS; ++w) {
          lost += add_exactly(s, part[w * SLOTS * 32 + slot]);
          if (gated) lost2 += add_exactly(s2, part[w * SLOTS * 32 + slot + 64]);
        }
        if (s + lost == s + lost) s += lost;      // beside an infinity the rest is NaN
        if (s2 + lost2 == s2 + lost2) s2 += lost2;
        if constexpr (sizeof(AT) == 4) {      // terms of what is not finite: the sum in plain multiply-adds
          const bf16* W = a.W + (long long)u.z * a.w_batch;
          if (s != s) s = lin_plain_sum(row_of(u, ml), W + (long long)n * a.ldw, a.K);
          if (s2 != s2) s2 = lin_plain_sum(row_of(u, ml), W + (long long)(n + n_out) * a.ldw, a.K);
        }
        const int m = PAIRS ? pair_of[u.first + ml] : ml;
        if (a.row_scale != nullptr) {
          s *= a.row_scale[m];
          s2 *= a.row_scale[m];
        }
        if (a.bias != nullptr) {
          s += a.bias[n];
          if (gated) s2 += a.bias[n + n_out];
        }
        float v = gated ? lin_gate(a.epi, s, s2, a.e0, a.e1) : lin_epi(a.epi, s, a.e0, a.e1);
        const int z = PAIRS ? 0 : u.z;
        if (a.gate != nullptr) v /= 1.0f + expf(-a.gate[(long long)z * a.gate_batch + (long long)m * a.ldg + n]);
        const long long at_c = (long long)z * a.c_batch + (long long)m * a.ldc + n;
        if (c_fp32) {
          float* C = reinterpret_cast<float*>(a.C) + at_c;
          *C = a.c_accum ? fmaf(a.c_scale, v, *C) : v;
        } else {
          bf16* C = reinterpret_cast<bf16*>(a.C) + at_c;
          *C = __float2bfloat16(a.c_accum ? fmaf(a.c_scale, v, __bfloat162float(*C)) : v);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sums_empty[buf]);
    }
  }
}

static bool gated_epi(int epi) { return epi == LP_EPI_SILU_GATE || epi == LP_EPI_CLAMP_GLU || epi == LP_EPI_GELU_GATE; }

template <typename AT, int NT, int MG>
static int launch_stream(const LinArgs& a, int c_fp32, dim3 grid, int warps, int n_pairs, cudaStream_t stream) {
  const size_t smem = (size_t)warps * NT * MG * 4 * 32 * sizeof(float);
  if (smem > 40 * 1024) LP_CHECK_CUDA(cudaFuncSetAttribute(linear_stream_kernel<AT, NT, MG>, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536));
  LP_CHECK_CUDA((launch_next(linear_stream_kernel<AT, NT, MG>, grid, dim3(warps * 32), smem, stream, a, gated_epi(a.epi), c_fp32, n_pairs)));
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

template <typename AT, int NT, int MG, bool PAIRS>
static int launch_ring(const LinArgs& a, int c_fp32, int batch, int n_pairs, int n_groups, cudaStream_t stream) {
  constexpr int KC = ring_kc<AT, MG>(), halves = sizeof(AT) / 2;
  const int n_out = gated_epi(a.epi) ? a.N / 2 : a.N, per = (gated_epi(a.epi) ? 8 : 16) * NT, problems = PAIRS ? n_groups : batch;
  const long long units = (long long)problems * ((n_out + per - 1) / per);
  // 64 columns of 16 bits, the rows, the blocks of 64, the problems (of A: the segments)
  CUtensorMap tw, ta = {};
  const uint64_t w_dims[4] = {64, (uint64_t)a.N, (uint64_t)(a.K / 64), (uint64_t)problems}, w_strides[3] = {(uint64_t)(a.N > 1 ? a.ldw : 64), 64, (uint64_t)(problems > 1 ? a.w_batch : 64)};
  const uint32_t w_box[4] = {64, 8, KC / 64, 1};
  if (const int rc = make_tmap_bf16_4d(&tw, a.W, w_dims, w_strides, w_box)) return rc;
  if (!PAIRS) {
    const uint64_t many = a.seg_cols > 0 ? a.n_segs : batch, far = a.seg_cols > 0 ? a.a_seg : a.a_batch;
    const uint64_t dims[4] = {64, (uint64_t)a.M, (uint64_t)(a.K * halves / 64), many}, strides[3] = {(uint64_t)(a.M > 1 ? a.lda * halves : 64), 64, many > 1 ? far * halves : 64};
    const uint32_t box[4] = {64, 8, KC * halves / 64, 1};
    if (const int rc = make_tmap_bf16_4d(&ta, a.A, dims, strides, box)) return rc;
  }
  constexpr int smem = 1024 + ring_stages<AT, NT, MG, PAIRS>() * ring_piece<AT, NT, MG, PAIRS>() + ring_sums<NT, MG>();
  LP_CHECK_CUDA((cudaFuncSetAttribute(linear_ring_kernel<AT, NT, MG, PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)));
  LP_CHECK_CUDA((launch_next(linear_ring_kernel<AT, NT, MG, PAIRS>, dim3((unsigned)(units < sm_count() ? units : sm_count())), dim3(RING_WARPS * 32), smem, stream, tw, ta, a,
                             (int)gated_epi(a.epi), c_fp32, batch, n_pairs, n_groups)));
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// rows of whole 16-byte pieces on both sides: what linear_stream_kernel reads
static bool stream_ok(const LinArgs& a, int a_fp32, int batch) {
  const int q = a_fp32 ? 4 : 8;
  return a.K % 8 == 0 && a.ldw % 8 == 0 && a.lda % q == 0 && (batch == 1 || a.a_batch % q == 0) && a.w_batch % 8 == 0 &&
         (a.seg_cols == 0 || a.a_seg % q == 0) && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.W) & 15) == 0;
}

// Where the ring is ahead of the kernel without it (both on 9,000 random sizes, us a launch in a graph, that kernel and the ring).  It brings whole pieces of a tile through one
// CTA an SM, so it wants a K of several pieces, and full rounds of tiles: 8 rows of bf16, K = 512, N = 7168 3.8, 5.3; K = 640, N = 7808 4.6, 5.9; K = 2048, N = 2048
// 5.0, 3.6; K = 4096, N = 6144 12.1, 9.1; 16 rows, K = 4096, N = 32000 62, 44.  A few columns over a very long K: all of it comes through a few CTAs (one row, K = 13312, N = 16 7.1,
// 7.9; fp32 K = 8256, N = 96 10.0, 12.2).
// The lines are those of whole decode steps, where weights that may be read early come while the small kernel before it runs and what others keep in the L2 stays there: after a
// row norm of 2 us, 111 to 148 tiles of K = 512 took 0.89 of that kernel's time (alone 1.05), two rounds of K = 640 to 1024 0.93 (1.0).  Launches alone put K = 12288, N = 3072 (192 tiles
// on 148 SMs; 17.3, 18.9) and K = 1536, N = 6144 (4.7, 4.9) on the other side; steps with these took 221 us so for 203, and 132 for 126.
// fp32 rows are cut into terms for every tile: two tiles a piece where there is more than one a CTA (4 rows, K = 2048, N = 8192 13.0, 10.2 with one and
// two tiles); 9 to 16 of them fill the issue slots up to one tile a CTA (K = N = 2048 7.3, 7.5; but N = 6144, K = 4096 34, 29).
// 17 to 64 rows: A is most of what a CTA brings (64 rows, K = 4096, N = 1024 24.6, 15.4; fp32 K = 1024, N = 2048 14.9, 12.7), and up to 32 its plain sums are the cheaper
// ones at most sizes; more are ahead up to a tile a CTA (a step of 64 requests of width 512 176 us without K = 512, so 172), and in a third round (K = 2048, N = 6144, 33 rows 23.9, 21.1) that is nearly full, not in a
// second or a fourth (35 rows, K = 16192, N = 2752 72, 93; 58 gated rows, K = 5120, N = 2864 28.8, 32.5).
static bool ring_pays_rows(int a_fp32, int mg, long long tiles, int K) {
  const long long sms = sm_count();
  const bool one = tiles <= sms, few = 4 * tiles <= sms;      // one tile a CTA; a quarter of the SMs at most
  if (mg == 8) {
    if (!one) return tiles > 2 * sms && tiles <= 3 * sms && K >= 2048;
    return a_fp32 || tiles > 8 || K <= 2048;
  }
  if (mg == 4) {
    if (one) return !a_fp32 || K < 1024 || (K >= 2048 && !few) || (K > 4096 && tiles > 8);
    return K >= (tiles <= 2 * sms ? 1024 : 2048) && tiles <= 4 * sms;
  }
  if (mg == 2) {
    if (a_fp32) return !one && tiles <= 4 * sms && K >= 2048;
    return K > (one ? 512 : 2047);
  }
  if (a_fp32) {
    if (one) return few ? K <= 1536 : K > 128;
    return K >= 1024 || (K >= 512 && (tiles <= 2 * sms || tiles > 3 * sms));
  }
  if (one) return K > 256 && (tiles > 8 || K <= 8192);
  return K >= 1024 || (K > 512 && tiles <= 2 * sms);
}
// The same for pairs.  Its CTAs sort all pairs, 0.75 ns a group that has some and group (200 groups of 512 x 512, 188 pairs 35.8, 58.4); that kernel has CTAs for the groups
// without pairs too (256 groups of 512 x 512: 18 us for two pairs, 13).  So: few groups to sort, or weights that take eight times as long, and then either many CTAs there, or
// enough weights and tiles (16 groups of 2048 x 1024, 12 pairs 13.4, 11.7; 32 of 2048 x 4096, 32 pairs 67, 59; 8 of 1024 x 1024, 16 pairs 6.1, 7.1).  Two short steps a
// tile, or more than 8 rows a group, are that kernel's (128 x 1544, 4 pairs 3.8, 5.8; 52 pairs in 8 groups of 2048 x 2304 4.9, 12.5).
static bool ring_pays_pairs(const LinArgs& a, int a_fp32, long long tiles, int n_groups, int n_pairs) {
  const long long used = n_pairs < n_groups ? n_pairs : n_groups, weights = used * a.N * a.K, sorting = used * n_groups;
  if (sorting > 4000 && weights < 8000 * sorting) return false;
  if (tiles >= 40LL * sm_count() && a.K >= (n_pairs <= 12 ? 192 : 512)) return true;
  return weights >= (1 << 24) && n_groups * (n_pairs > 32 ? n_pairs : 32) <= 1024 && tiles / n_groups * used >= 4 * sm_count() && a.K >= (a_fp32 ? 512 : 1024);
}

// n_groups > 0: pairs, of which a group has up to about `rows` (more run in further rounds over its weights); else one problem of `rows` rows per batch entry
static int dispatch_stream(const LinArgs& a, int a_fp32, int c_fp32, int batch, int rows, int n_groups, int n_pairs, cudaStream_t stream) {
  const int n_out = gated_epi(a.epi) ? a.N / 2 : a.N, per = gated_epi(a.epi) ? 8 : 16;
  const int mg = rows <= 8 ? 1 : rows <= 16 ? 2 : rows <= 32 ? 4 : 8;
  const long long problems = n_groups > 0 ? n_groups : batch;
  const long long ring_units = problems * ((n_out + per - 1) / per);
  // rows, operands and problems lie at increasing addresses less than 2^40 bytes apart: what a tensor map can say
  auto follows = [](long long count, long long elements) { return count == 1 || (elements > 0 && elements < (1LL << 38)); };
  const bool ring_reads = follows(a.N, a.ldw) && follows(a.M, a.lda) && follows(problems, a.w_batch) && follows(batch, a.a_batch) &&
                          (a.seg_cols == 0 || follows(a.n_segs, a.a_seg));
  // The ring waits while a thread takes sums of fp32 rows again that are not finite: up to 8 of them, 76 ns a product (64 rows, K = 16384, infinite weights: 10 ms for
  // 0.12).  0.6 s at this K; the waits give up after two.
  const bool ring_mends = !a_fp32 || a.K <= (1 << 20);
  const bool ring_pays = n_groups > 0 ? mg == 1 && ring_pays_pairs(a, a_fp32, ring_units, n_groups, n_pairs) : ring_pays_rows(a_fp32, mg, ring_units, a.K);
  if (ring_reads && ring_pays && n_groups <= RING_MAX_GROUPS && a.K % 64 == 0 && ring_units < (1LL << 31) && ring_mends) {
    const bool two = a_fp32 && ring_units > sm_count() && (a.seg_cols == 0 || a.seg_cols % (2 * per) == 0);
#define LP_RING(NT, MG, PAIRS) (a_fp32 ? launch_ring<float, NT, MG, PAIRS>(a, c_fp32, batch, n_pairs, n_groups, stream) : launch_ring<bf16, 1, MG, PAIRS>(a, c_fp32, batch, n_pairs, n_groups, stream))
    if (n_groups > 0) return LP_RING(2, 1, true);
    if (mg == 1) return two ? LP_RING(2, 1, false) : LP_RING(1, 1, false);
    if (mg == 2) return two ? LP_RING(2, 2, false) : LP_RING(1, 2, false);
    return mg == 4 ? LP_RING(1, 4, false) : LP_RING(1, 8, false);
#undef LP_RING
  }
  // fp32 rows: two tiles a CTA read A half as often and cut it into terms once, taken once the grid still has two CTAs for every SM and where segments
  // allow.  bf16 rows take one: its registers leave room for the next steps' weights (one row, us, two tiles and one: K = 4096, N = 16384 28.1, 25.9, N =
  // 32000 49.2, 46.1; eight rows of 14 experts, K = 2048, N = 2048 27.2, 24.1; with 16 rows, N = 12288, K = 4096, 46, 35)
  const long long wide = problems * ((n_out + 2 * per - 1) / (2 * per));
  const int nt = a_fp32 && wide >= 2 * sm_count() && (a.seg_cols == 0 || a.seg_cols % (2 * per) == 0) ? 2 : 1;
  const long long ctas = problems * ((n_out + nt * per - 1) / (nt * per));
  // a short K has no work for more warps (K = 192, one row: 4.0 us with four, 3.2 with eight); a grid of few CTAs wants more loads in flight in each (N = 2048, K = 8192: 15 us with 16 warps, 11 with 32)
  int warps = a.K <= (mg == 1 ? 128 : 256) ? 4 : !a_fp32 && mg * nt == 1 && ctas <= sm_count() && a.K >= 4096 ? 32 : ctas <= 2 * sm_count() && a.K >= 1024 && mg <= 4 ? 16 : 8;
  dim3 grid((n_out + nt * per - 1) / (nt * per), n_groups > 0 ? n_groups : 1, n_groups > 0 ? 1 : batch);
#define LP_STREAM(MG)                                                                                                               \
  (a_fp32 ? (nt == 2 ? launch_stream<float, 2, MG>(a, c_fp32, grid, warps, n_pairs, stream) : launch_stream<float, 1, MG>(a, c_fp32, grid, warps, n_pairs, stream)) \
          : launch_stream<bf16, 1, MG>(a, c_fp32, grid, warps, n_pairs, stream))
  return mg == 1 ? LP_STREAM(1) : mg == 2 ? LP_STREAM(2) : mg == 4 ? LP_STREAM(4) : LP_STREAM(8);
#undef LP_STREAM
}

// ---------------------------------------------------------------------------------------------------------------------------------
// More rows: 64 x 128 output tiles, K in steps of 32 through two shared-memory buffers, two CTAs an SM (one's loads and cuts run beside the
// other's products: 128-row tiles with one CTA of 16 warps were 15 % slower), a warp to 32 x 32 outputs on the same matrix instruction.  fp32 rows are cut into their three bf16 terms once, on the way
// into shared memory (a plane each), so the inner loop is loads and products only; the next step's global loads are in flight meanwhile.
// A lane reads 16 bytes of a row, eight k, the same permutation of k on both sides; rows are 64 bytes apart, so eight lanes read two
// whole rows: no two of them in the same bank.  Chains as above: each step's products form sums of their own, added in fp32.
// The gated units interleave gate and up rows in groups of eight, so both halves of an output are neighbours in one lane.
// Measured (B200, M = 4096, N = 8192, K = 2048): fp32 rows 1.47 ms = 93 TFLOP/s (three products each; 64 x 64 tiles on fp32 FMAs 5.4 ms, 25),
// bf16 rows 0.72 ms; mma.sync alone reaches 520 TFLOP/s of bf16 products here, 450 with a sum of its own every few.  Error against 64 bits at
// K = 1024 / 4096: 1.2e-7 / 2.1e-7 (FMA chains over K: 5.7e-7 / 1.1e-6).
// What a product is added to (c_accum) and its gate are copied in (cp.async) while the products run: read where they are used, a load at a time, they
// took 6 us of every CTA (65 rows, N = 64, K = 16 to 256: 15.0 to 21.4 us instead of 9.1 to 15.8).
constexpr int MT_BM = LIN_BM, MT_BN = 128, MT_BK = 32, MT_LDC = MT_BN + 4, MT_THREADS = 256;
// bytes of shared memory: the stages, then in their place the tile of sums, and after them a tile each of what it is added to and of the gate
template <typename AT> constexpr size_t mt_smem() {
  constexpr size_t stages = 2 * sizeof(uint32_t) * ((sizeof(AT) == 4 ? 3 : 1) * MT_BM * MT_BK / 2 + MT_BN * MT_BK / 2), tile = sizeof(float) * MT_BM * MT_LDC;
  return stages > tile ? stages : tile;
}
constexpr size_t MT_SIDE = sizeof(float) * MT_BM * MT_BN;

// the tile's sums in shared memory (a gated unit's halves eight columns apart), rows from m0 and output columns from n0 on
template <typename AT>
__device__ __noinline__ void lin_mend_tile(float* tile, const AT* A, long long lda, const int* a_rows, const bf16* W, long long ldw, int K, int m0,
                                           int M, int n0, int n_out, int gated) {
  const int cols = gated ? MT_BN / 2 : MT_BN;
  for (int e = threadIdx.x; e < MT_BM * cols; e += MT_THREADS) {
    const int ml = e / cols, nl = e % cols, m = m0 + ml, n = n0 + nl;
    if (m >= M || n >= n_out) continue;
    const long long r = a_rows != nullptr ? a_rows[m] : m;
    for (int half = 0; half < (gated ? 2 : 1); ++half) {
      float* s = tile + ml * MT_LDC + (gated ? (nl >> 3) * 16 + (nl & 7) + 8 * half : nl);
      if (r >= 0 && *s != *s) *s = lin_plain_dot(A + r * lda, W + (long long)(n + half * n_out) * ldw, K);
    }
  }
  __syncthreads();
}

template <typename AT, bool SIDE>
__global__ void __launch_bounds__(MT_THREADS, 2) linear_mma_kernel(LinArgs a, int gated, int c_fp32) {
  extern __shared__ float dyn_smem[];
  constexpr int PLANES = sizeof(AT) == 4 ? 3 : 1;
  constexpr int BM = MT_BM, A_WORDS = BM * MT_BK / 2, W_WORDS = MT_BN * MT_BK / 2, STAGE = PLANES * A_WORDS + W_WORDS;      // 32-bit words
  constexpr int THREADS = MT_THREADS, WARPS_N = 4, NI = MT_BN / WARPS_N / 8;
  constexpr int A_CHUNKS = BM * 4 / THREADS, W_CHUNKS = MT_BN * 4 / THREADS;      // 16-byte (eight k) pieces a thread brings
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int z = blockIdx.z, m0 = blockIdx.y * BM, n_out = gated ? a.N / 2 : a.N;
  const int cols = gated ? MT_BN / 2 : MT_BN, n0 = blockIdx.x * cols;
  int group = 0;
  if (a.tile_group != nullptr) {
    group = a.tile_group[blockIdx.y];
    if (group < 0) return;
  }
  const AT* A = reinterpret_cast<const AT*>(a.A) + (long long)z * a.a_batch + lin_seg(a, n0);
  const bf16* W = a.W + (long long)(z + group) * a.w_batch;
  uint32_t* smem = reinterpret_cast<uint32_t*>(dyn_smem);
  const AT* a_src[A_CHUNKS];
  const bf16* w_src[W_CHUNKS];
#pragma unroll
  for (int i = 0; i < A_CHUNKS; ++i) {
    const int m = m0 + (tid + i * THREADS) / 4;
    const long long r = m >= a.M ? -1 : a.a_rows != nullptr ? a.a_rows[m] : m;
    a_src[i] = r < 0 ? nullptr : A + r * a.lda;
  }
#pragma unroll
  for (int i = 0; i < W_CHUNKS; ++i) {
    const int j = (tid + i * THREADS) / 4;
    const int n = gated ? n0 + (j >> 4) * 8 + (j & 7) : n0 + j;
    w_src[i] = n >= n_out ? nullptr : W + (long long)(gated && (j & 8) ? n + n_out : n) * a.ldw;
  }
  const int kc = (tid & 3) * 8;      // this thread's eight k of a step
  const uint4 none = make_uint4(0, 0, 0, 0);
  uint4 ra[A_CHUNKS][sizeof(AT) / 2], rw[W_CHUNKS];
  auto fetch = [&](int k0) {
    const bool in = k0 + kc < a.K;
#pragma unroll
    for (int i = 0; i < A_CHUNKS; ++i)
#pragma unroll
      for (int h = 0; h < (int)sizeof(AT) / 2; ++h)
        ra[i][h] = in && a_src[i] != nullptr ? *(reinterpret_cast<const uint4*>(a_src[i] + k0 + kc) + h) : none;
#pragma unroll
    for (int i = 0; i < W_CHUNKS; ++i) rw[i] = in && w_src[i] != nullptr ? *reinterpret_cast<const uint4*>(w_src[i] + k0 + kc) : none;
  };
  auto put = [&](int buf) {
    uint32_t* st = smem + buf * STAGE;
#pragma unroll
    for (int i = 0; i < A_CHUNKS; ++i) {
      uint4* dst = reinterpret_cast<uint4*>(st + (tid + i * THREADS) * 4);
      if constexpr (PLANES == 3) {
        const uint4 p = ra[i][0], q = ra[i][1];
        const Bf16Terms v = split3(make_float4(__uint_as_float(p.x), __uint_as_float(p.y), __uint_as_float(p.z), __uint_as_float(p.w)),
                                   make_float4(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z), __uint_as_float(q.w)));
        dst[0] = v.hi;
        dst[A_WORDS / 4] = v.mid;
        dst[2 * (A_WORDS / 4)] = v.lo;
      } else {
        dst[0] = ra[i][0];
      }
    }
#pragma unroll
    for (int i = 0; i < W_CHUNKS; ++i) *reinterpret_cast<uint4*>(st + PLANES * A_WORDS + (tid + i * THREADS) * 4) = rw[i];
  };
  if constexpr (SIDE) {      // each thread fetches what it will use itself: no barrier
    float* side = dyn_smem + mt_smem<AT>() / sizeof(float);
#pragma unroll 1
    for (int e = tid; e < BM * cols; e += THREADS) {
      const int m = m0 + e / cols, n = n0 + e % cols;
      if (m >= a.M || n >= n_out) continue;
      if (a.c_accum && c_fp32)
        __pipeline_memcpy_async(side + e, reinterpret_cast<const float*>(a.C) + (long long)z * a.c_batch + (long long)m * a.ldc + n, 4);
      if (a.gate != nullptr)
        __pipeline_memcpy_async(side + BM * MT_BN + e, a.gate + (long long)z * a.gate_batch + (long long)m * a.ldg + n, 4);
    }
    __pipeline_commit();
  }
  const int wm = (warp / WARPS_N) * 32, wn = (warp % WARPS_N) * NI * 8;
  float acc[2][NI][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;
  fetch(0);
  put(0);
  __syncthreads();
  const int steps = (a.K + MT_BK - 1) / MT_BK;
  for (int s = 0; s < steps; ++s) {
    if (s + 1 < steps) fetch((s + 1) * MT_BK);
    const uint32_t* st = smem + (s & 1) * STAGE;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint4 x0[PLANES], x1[PLANES];
#pragma unroll
      for (int p = 0; p < PLANES; ++p) {
        x0[p] = *reinterpret_cast<const uint4*>(st + p * A_WORDS + (wm + 16 * i + g) * 16 + t * 4);
        x1[p] = *reinterpret_cast<const uint4*>(st + p * A_WORDS + (wm + 16 * i + g + 8) * 16 + t * 4);
      }
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        const uint4 w = *reinterpret_cast<const uint4*>(st + PLANES * A_WORDS + (wn + 8 * j + g) * 16 + t * 4);
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int p = PLANES - 1; p >= 0; --p) {      // the small terms first
          mma_bf16(d, x0[p].x, x1[p].x, x0[p].y, x1[p].y, w.x, w.y);
          mma_bf16(d, x0[p].z, x1[p].z, x0[p].w, x1[p].w, w.z, w.w);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][j][c] += d[c];
      }
    }
    if (s + 1 < steps) put((s + 1) & 1);
    __syncthreads();
  }
  // through shared memory, so that one copy of the epilogue's code serves whole rows (the stages are no longer read)
  bool odd = false;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        dyn_smem[(wm + 16 * i + g + 8 * (c >> 1)) * MT_LDC + wn + 8 * j + 2 * t + (c & 1)] = acc[i][j][c];
        if constexpr (PLANES == 3) odd |= not_finite(acc[i][j][c]);
      }
  if constexpr (PLANES == 3) {
    if (__syncthreads_or(odd)) lin_mend_tile(dyn_smem, A, a.lda, a.a_rows, W, a.ldw, a.K, m0, a.M, n0, n_out, gated);
  } else {
    __syncthreads();
  }
  const float* side = dyn_smem + mt_smem<AT>() / sizeof(float);
  if constexpr (SIDE) __pipeline_wait_prior(0);
#pragma unroll 1
  for (int e = tid; e < BM * cols; e += THREADS) {
    const int ml = e / cols, nl = e % cols, m = m0 + ml, n = n0 + nl;
    if (m >= a.M || n >= n_out) continue;
    const int at = ml * MT_LDC + (gated ? (nl >> 3) * 16 + (nl & 7) : nl);
    float s = dyn_smem[at], s2 = gated ? dyn_smem[at + 8] : 0.f;
    if (a.row_scale != nullptr) {
      s *= a.row_scale[m];
      s2 *= a.row_scale[m];
    }
    if (a.bias != nullptr) {
      s += a.bias[n];
      if (gated) s2 += a.bias[n + n_out];
    }
    float v = gated ? lin_gate(a.epi, s, s2, a.e0, a.e1) : lin_epi(a.epi, s, a.e0, a.e1);
    if (SIDE && a.gate != nullptr) v /= 1.0f + expf(-side[BM * MT_BN + e]);
    const long long at_c = (long long)z * a.c_batch + (long long)m * a.ldc + n;
    if (c_fp32) {
      float* C = reinterpret_cast<float*>(a.C) + at_c;
      *C = SIDE && a.c_accum ? fmaf(a.c_scale, v, side[e]) : v;
    } else {
      bf16* C = reinterpret_cast<bf16*>(a.C) + at_c;
      *C = __float2bfloat16(a.c_accum ? fmaf(a.c_scale, v, __bfloat162float(*C)) : v);
    }
  }
}

template <typename AT, bool SIDE>
static int launch_mma(const LinArgs& a, int c_fp32, int batch, int m_tiles, cudaStream_t stream) {
  constexpr size_t smem = mt_smem<AT>() + (SIDE ? 2 * MT_SIDE : 0);
  const int cols = gated_epi(a.epi) ? MT_BN / 2 : MT_BN, n_out = gated_epi(a.epi) ? a.N / 2 : a.N;
  if (smem > 48 * 1024) LP_CHECK_CUDA(cudaFuncSetAttribute(linear_mma_kernel<AT, SIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((n_out + cols - 1) / cols, m_tiles, batch);
  linear_mma_kernel<AT, SIDE><<<grid, MT_THREADS, smem, stream>>>(a, gated_epi(a.epi), c_fp32);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}
// A K of a few steps does not pay for the terms, the tile in shared memory and a K step of 32; columns for half a tile pay for a whole one.  Measured (us,
// linear_tile_kernel and this one, fp32 rows): K = 16: 65 x 64 5.3, 9.1, 4096 x 8192 84, 133; K = 32: 300 x 512 7.0, 9.3, 4096 x 2048 34, 37; K = 64: 300 x 512
// 9.2, 10.2, 300 x 2048 11.6, 10.3, 4096 x 2048 56, 42; 16 products of 4096 x 64 32, 42; K = 96: 300 x 512 11.0, 11.2, 300 x 2048 13.9, 11.3; K = 128: 65 x 64
// 12.8, 11.8.  Gated: K = 16 300 x 8192 10.1, 13.2; K = 32 65 x 64 8.8, 7.6, 300 x 8192 14.0, 13.2.  Added to a stream: K = 128 300 x 512
// 14.7, 15.7, 300 x 8192 40, 31; behind a gate: 15.2, 17.8, K = 192 19.5, 19.4.  bf16 rows cross at the same places.
static bool mma_pays(const LinArgs& a, int batch, int m_tiles) {
  if (gated_epi(a.epi)) return a.K >= 32;
  const int lo = a.c_accum || a.gate != nullptr ? 96 : 40, hi = a.c_accum || a.gate != nullptr ? 192 : 128;      // two more tiles to bring in
  if (a.K < lo || a.K >= hi) return a.K >= hi;
  return a.N > MT_BN / 2 && 2LL * batch * m_tiles * ((a.N + MT_BN - 1) / MT_BN) > sm_count();
}
// The same for up to 64 rows: 33 x 512 5.4, 6.9 (fp32 rows, K = 8), 6.7, 7.1 (32), 8.5, 7.1 (64); 64 x 512 5.4, 8.7, 6.7, 8.7, 8.7, 8.7; bf16 rows 64 x 512 5.6, 6.9
// (8), 6.4, 6.7 (32), 33 x 512 5.6, 5.2 (8); up to 32 rows the streaming kernel is ahead at every K.
static bool stream_pays(const LinArgs& a, int a_fp32) {
  return a.M <= (a_fp32 ? 32 : 48) || a.K > 32 || (gated_epi(a.epi) && a.K >= 16);
}

static int dispatch_mma(const LinArgs& a, int a_fp32, int c_fp32, int batch, int m_tiles, cudaStream_t stream) {
  if ((a.c_accum && c_fp32) || a.gate != nullptr)
    return a_fp32 ? launch_mma<float, true>(a, c_fp32, batch, m_tiles, stream) : launch_mma<bf16, true>(a, c_fp32, batch, m_tiles, stream);
  return a_fp32 ? launch_mma<float, false>(a, c_fp32, batch, m_tiles, stream) : launch_mma<bf16, false>(a, c_fp32, batch, m_tiles, stream);
}

template <typename AT, typename CT, bool GATED>
static int launch_linear(const LinArgs& a, int batch, int m_tiles, bool allow_rows, cudaStream_t stream) {
  const int n_out = GATED ? a.N / 2 : a.N;
  if (allow_rows && a.M <= ROWS_MAX) {
    dim3 grid((n_out + ROWS_WARPS - 1) / ROWS_WARPS, 1, batch);
    linear_rows_kernel<AT, CT, GATED><<<grid, ROWS_WARPS * 32, 0, stream>>>(a);
  } else {
    dim3 grid((n_out + LIN_BN - 1) / LIN_BN, m_tiles, batch);
    linear_tile_kernel<AT, CT, GATED><<<grid, LIN_THREADS, 0, stream>>>(a);
  }
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

static int dispatch_linear(const LinArgs& a, int a_fp32, int c_fp32, int batch, int m_tiles, bool allow_rows, cudaStream_t stream) {
  const bool gated = gated_epi(a.epi);
  if (a_fp32) {
    if (c_fp32) return gated ? launch_linear<float, float, true>(a, batch, m_tiles, allow_rows, stream)
                             : launch_linear<float, float, false>(a, batch, m_tiles, allow_rows, stream);
    return gated ? launch_linear<float, bf16, true>(a, batch, m_tiles, allow_rows, stream)
                 : launch_linear<float, bf16, false>(a, batch, m_tiles, allow_rows, stream);
  }
  if (c_fp32) return gated ? launch_linear<bf16, float, true>(a, batch, m_tiles, allow_rows, stream)
                           : launch_linear<bf16, float, false>(a, batch, m_tiles, allow_rows, stream);
  return gated ? launch_linear<bf16, bf16, true>(a, batch, m_tiles, allow_rows, stream)
               : launch_linear<bf16, bf16, false>(a, batch, m_tiles, allow_rows, stream);
}

}  // namespace lp

using namespace lp;

extern "C" int lp_linear(const lp_linear_desc* d, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LP_REQUIRE(d != nullptr && d->A != nullptr && d->W != nullptr && d->C != nullptr, "lp_linear: null operand");
  LP_REQUIRE(d->M >= 0 && d->N > 0 && d->K > 0 && d->batch >= 1, "lp_linear: bad problem M=%d N=%d K=%d batch=%d", d->M, d->N, d->K,
             d->batch);
  const int epi = d->epi & ~LP_LINEAR_W_CONSTANT;
  LP_REQUIRE(epi >= LP_EPI_NONE && epi <= LP_EPI_GELU_GATE, "lp_linear: bad epilogue %d", d->epi);
  LP_REQUIRE(!gated_epi(epi) || d->N % 2 == 0, "lp_linear: the gated epilogue needs an even N (gate rows, then up rows)");
  if (d->M == 0) return 0;
  LinArgs a;
  a.A = d->A; a.lda = d->lda; a.a_batch = d->a_batch;
  a.W = reinterpret_cast<const bf16*>(d->W); a.ldw = d->ldw; a.w_batch = d->w_batch;
  a.C = d->C; a.ldc = d->ldc; a.c_batch = d->c_batch;
  a.M = d->M; a.N = d->N; a.K = d->K;
  a.epi = epi; a.e0 = d->epi_a; a.e1 = d->epi_b; a.c_accum = d->c_accum; a.c_scale = d->c_scale;
  a.a_rows = nullptr; a.tile_group = nullptr; a.z_group = nullptr; a.a_div = 1;
  a.bias = d->bias; a.row_scale = d->row_scale; a.gate = d->gate; a.ldg = d->ldg; a.gate_batch = d->gate_batch;
  a.seg_cols = d->seg_cols; a.n_segs = d->n_segs; a.a_seg = d->a_seg;
  a.w_constant = d->epi & LP_LINEAR_W_CONSTANT;
  LP_REQUIRE(d->batch == 1 || (d->bias == nullptr && d->row_scale == nullptr), "lp_linear: bias and row scale are for one problem");
  // a CTA's columns read one operand: 8 columns for few rows, a tile otherwise
  LP_REQUIRE(d->seg_cols == 0 || (d->seg_cols > 0 && d->n_segs >= 1 && d->seg_cols % (d->M <= ROWS_MAX ? ROWS_WARPS : LIN_BN) == 0),
             "lp_linear: column segments of %d do not fit the CTAs of a product of %d rows", d->seg_cols, d->M);
  LP_REQUIRE(d->seg_cols == 0 || !gated_epi(epi), "lp_linear: a gated unit has one operand");
  if (d->M <= STREAM_MAX_ROWS && stream_ok(a, d->a_fp32, d->batch) && (d->seg_cols == 0 || d->seg_cols % 16 == 0) && stream_pays(a, d->a_fp32))
    return dispatch_stream(a, d->a_fp32, d->c_fp32, d->batch, d->M, 0, 0, stream);
  // the tile kernel on the matrix instructions; operands without 16-byte rows stay on fp32 FMAs
  if (stream_ok(a, d->a_fp32, d->batch) && (d->seg_cols == 0 || d->seg_cols % MT_BN == 0) && d->M > STREAM_MAX_ROWS &&
      mma_pays(a, d->batch, (d->M + MT_BM - 1) / MT_BM))
    return dispatch_mma(a, d->a_fp32, d->c_fp32, d->batch, (d->M + MT_BM - 1) / MT_BM, stream);
  return dispatch_linear(a, d->a_fp32, d->c_fp32, d->batch, (d->M + LIN_BM - 1) / LIN_BM, true, stream);
}

static int linear_pairs(const lp_linear_desc* d, const int* pair_group, int n_groups, int a_div, int n_pairs, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LP_REQUIRE(d != nullptr && d->A != nullptr && d->W != nullptr && d->C != nullptr && pair_group != nullptr, "lp_linear_pairs: null operand");
  LP_REQUIRE(d->N > 0 && d->K > 0 && a_div >= 1 && n_pairs >= 0 && n_pairs <= 65535, "lp_linear_pairs: bad problem N=%d K=%d pairs=%d", d->N,
             d->K, n_pairs);
  LP_REQUIRE(d->epi >= LP_EPI_NONE && d->epi <= LP_EPI_GELU_GATE, "lp_linear_pairs: bad epilogue %d", d->epi);
  LP_REQUIRE(!gated_epi(d->epi) || d->N % 2 == 0, "lp_linear_pairs: the gated epilogue needs an even N");
  if (n_pairs == 0) return 0;
  LinArgs a;
  a.A = d->A; a.lda = d->lda; a.a_batch = 0;
  a.W = reinterpret_cast<const bf16*>(d->W); a.ldw = d->ldw; a.w_batch = d->w_batch;
  a.C = d->C; a.ldc = d->ldc; a.c_batch = 0;
  a.M = 1; a.N = d->N; a.K = d->K;
  a.epi = d->epi; a.e0 = d->epi_a; a.e1 = d->epi_b; a.c_accum = d->c_accum; a.c_scale = d->c_scale;
  a.a_rows = nullptr; a.tile_group = nullptr; a.z_group = pair_group; a.a_div = a_div;
  a.bias = d->bias; a.row_scale = d->row_scale; a.gate = d->gate; a.ldg = d->ldg; a.gate_batch = d->gate_batch;
  a.seg_cols = 0; a.n_segs = 0; a.a_seg = 0; a.w_constant = 0;
  // with the number of groups a group's weights are read once for all of its pairs
  if (n_groups > 0 && n_pairs <= STREAM_MAX_PAIRS && stream_ok(a, d->a_fp32, 1))
    return dispatch_stream(a, d->a_fp32, d->c_fp32, 1, 2 * ((n_pairs + n_groups - 1) / n_groups), n_groups, n_pairs, stream);
  return dispatch_linear(a, d->a_fp32, d->c_fp32, n_pairs, 1, true, stream);
}

// n_pairs one-row problems on the weight-streaming kernel: problem z multiplies A row z / a_div by the weight of group pair_group[z]
// (w_batch elements apart) into C row z — the expert products of a decode step, where every (token, choice) pair has its own weight.
extern "C" int lp_linear_pairs(const lp_linear_desc* d, const int* pair_group, int a_div, int n_pairs, void* stream) {
  return linear_pairs(d, pair_group, 0, a_div, n_pairs, stream);
}

// the same for a caller that knows the number of groups (pair_group[z] < n_groups): a CTA a group and column tile reads the weights once
// for all of the group's pairs
extern "C" int lp_linear_group_pairs(const lp_linear_desc* d, const int* pair_group, int n_groups, int a_div, int n_pairs, void* stream) {
  LP_REQUIRE(n_groups >= 1 && n_groups <= 65535, "lp_linear_group_pairs: %d groups", n_groups);
  return linear_pairs(d, pair_group, n_groups, a_div, n_pairs, stream);
}

extern "C" int lp_linear_grouped(const lp_linear_desc* d, const int* tile_group, int n_tiles, const int* a_rows, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LP_REQUIRE(d != nullptr && d->A != nullptr && d->W != nullptr && d->C != nullptr && tile_group != nullptr,
             "lp_linear_grouped: null operand");
  LP_REQUIRE(d->N > 0 && d->K > 0 && n_tiles >= 0, "lp_linear_grouped: bad problem N=%d K=%d tiles=%d", d->N, d->K, n_tiles);
  LP_REQUIRE(d->epi >= LP_EPI_NONE && d->epi <= LP_EPI_GELU_GATE, "lp_linear_grouped: bad epilogue %d", d->epi);
  LP_REQUIRE(!gated_epi(d->epi) || d->N % 2 == 0, "lp_linear_grouped: the gated epilogue needs an even N");
  if (n_tiles == 0) return 0;
  LinArgs a;
  a.A = d->A; a.lda = d->lda; a.a_batch = 0;
  a.W = reinterpret_cast<const bf16*>(d->W); a.ldw = d->ldw; a.w_batch = d->w_batch;   // w_batch = elements between groups
  a.C = d->C; a.ldc = d->ldc; a.c_batch = 0;
  a.M = n_tiles * LIN_BM; a.N = d->N; a.K = d->K;
  a.epi = d->epi; a.e0 = d->epi_a; a.e1 = d->epi_b; a.c_accum = d->c_accum; a.c_scale = d->c_scale;
  a.a_rows = a_rows; a.tile_group = tile_group; a.z_group = nullptr; a.a_div = 1;
  a.bias = d->bias; a.row_scale = d->row_scale; a.gate = d->gate; a.ldg = d->ldg; a.gate_batch = d->gate_batch;
  a.seg_cols = 0; a.n_segs = 0; a.a_seg = 0; a.w_constant = 0;
  if (stream_ok(a, d->a_fp32, 1) && mma_pays(a, 1, n_tiles)) return dispatch_mma(a, d->a_fp32, d->c_fp32, 1, n_tiles, stream);
  return dispatch_linear(a, d->a_fp32, d->c_fp32, 1, n_tiles, false, stream);
}

extern "C" int lp_linear_tile_rows(void) { return LIN_BM; }

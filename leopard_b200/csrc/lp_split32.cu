// leopard_b200 — 32-bit products and attention of prompts on the tcgen05 tensor cores.
//
// An fp32 number is three bf16 terms (its upper 8, middle 8 and lower 8 bits of mantissa: cut off, so they add up to it exactly).  Operands
// lie in memory as three planes of terms, so TMA brings them to shared memory as they are and the tensor cores take them:
//   gemm32_kernel   C[M, N] = A[M, K] W[N, K]^T, A in three planes, W bf16: every product is exact (three MMAs)
//   attn32_kernel   softmax(Q K^T) V, all three in planes, heads of 128 (+ 64 channels whose keys all heads share): the six products of weight
//                   above 2^-26 of what an fp32 product would be
// The tensor cores cut their running sum off instead of rounding it, a bias that grows with the chain.  So chains are short, small terms go
// first, and sums of chains are fp32 additions in registers: 64 of K (four MMAs at full size) in the product, all channels of one
// score (8 or 12) and 128 keys of an output (8) in attention.
#ifdef LP_EMULATE                  // CPU emulation build (tests/test_split32.py)
#include "tc_emu.h"
#include "emu_helpers.inc"
#else
#include "lp_common.cuh"
#include "lp_host.h"
#include "../../include/leopard_b200.h"
#endif

namespace lp {

constexpr int S32_BOX = 128 * 128;      // one TMA box: 128 rows x 64 bf16
// of the 168 registers a thread that 384 threads start with, the warpgroup of TMA and MMA warps gives up 96 and the two others take 48 each
constexpr int S32_FEW = 72, S32_MANY = 216;

#ifdef LP_EMULATE
inline void s32_bar(int id, int n) { named_bar(id, n, true); }
template <int N> inline void s32_more_regs() {}
template <int N> inline void s32_fewer_regs() {}
#else
__device__ __forceinline__ void s32_bar(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
template <int N> __device__ __forceinline__ void s32_more_regs() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void s32_fewer_regs() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
#define LP_TMEM_ST_16(regs, taddr)                                                                                  \
  asm volatile(                                                                                                     \
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, " \
      "%15, %16};" ::"r"(taddr),                                                                                    \
      "r"(regs[0]), "r"(regs[1]), "r"(regs[2]), "r"(regs[3]), "r"(regs[4]), "r"(regs[5]), "r"(regs[6]),             \
      "r"(regs[7]), "r"(regs[8]), "r"(regs[9]), "r"(regs[10]), "r"(regs[11]), "r"(regs[12]), "r"(regs[13]),         \
      "r"(regs[14]), "r"(regs[15])                                                                                  \
      : "memory")
#endif

// the three terms of x and y, packed in pairs: cut off, so that they add up to x and y exactly.  An infinity leaves nothing behind, a NaN
// stays one without its lower bits.
__device__ __forceinline__ void s32_terms(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  uint32_t u = __float_as_uint(x), v = __float_as_uint(y);
  const bool ux = (u & 0x7f800000u) == 0x7f800000u, vx = (v & 0x7f800000u) == 0x7f800000u;
  if (ux || vx) {
    if (ux && (u & 0x7fffffu)) u |= 0x400000u;
    if (vx && (v & 0x7fffffu)) v |= 0x400000u;
  }
  hi = (u >> 16) | (v & 0xffff0000u);
  x = ux ? 0.f : x - __uint_as_float(u & 0xffff0000u);
  y = vx ? 0.f : y - __uint_as_float(v & 0xffff0000u);
  u = __float_as_uint(x);
  v = __float_as_uint(y);
  mid = (u >> 16) | (v & 0xffff0000u);
  x -= __uint_as_float(u & 0xffff0000u);
  y -= __uint_as_float(v & 0xffff0000u);
  lo = (__float_as_uint(x) >> 16) | (__float_as_uint(y) & 0xffff0000u);
}
__device__ __forceinline__ void s32_store_terms(bf16* dst, long long plane, const float* v) {      // eight numbers
  uint4 h, m, l;
  s32_terms(v[0], v[1], h.x, m.x, l.x);
  s32_terms(v[2], v[3], h.y, m.y, l.y);
  s32_terms(v[4], v[5], h.z, m.z, l.z);
  s32_terms(v[6], v[7], h.w, m.w, l.w);
  *reinterpret_cast<uint4*>(dst) = h;
  *reinterpret_cast<uint4*>(dst + plane) = m;
  *reinterpret_cast<uint4*>(dst + 2 * plane) = l;
}
__device__ __forceinline__ float s32_value(const bf16* p, long long plane) {
  const float h = (float)p[0];
  return (__float_as_uint(h) & 0x7f800000u) == 0x7f800000u ? h : h + ((float)p[plane] + (float)p[2 * plane]);
}

// fp32 rows -> planes, eight columns a thread
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ src, long long ld, int M, int K, bf16* __restrict__ dst,
                                                         long long ldd, long long plane) {
  const int per = K >> 3;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)M * per) return;
  const long long r = i / per;
  const int c = (int)(i - r * per) * 8;
  const float* s = src + r * ld + c;
  const float4 a = *reinterpret_cast<const float4*>(s), b = *reinterpret_cast<const float4*>(s + 4);
  const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  s32_store_terms(dst + r * ldd + c, plane, v);
}

// ---------------------------------------------------------------------------------------------------------------------------------
// C[M, N] = A W^T (+ bias).  Persistent CTAs (one an SM) walk 128 x BN tiles; a k block of 64 is W's box(es) and A's three boxes, each with a
// barrier pair of its own so that a term's box is refilled as soon as its product has run.  Every k block is a chain of its own in one of two
// TMEM accumulators; eight warps add the finished one to the fp32 sums in their registers while the other is filled, and write a tile
// out while the next one's first chains run.
// Bound by the operand feed from L2 with BN = 128 (64 KB a k block of 768 tensor clocks) and by the tensor cores with BN = 256 (80 KB, 1,536).
// ---------------------------------------------------------------------------------------------------------------------------------
constexpr int G32_THREADS = 384, G32_EPI = 256;
enum { G32_OUT_BF16 = 0, G32_OUT_F32 = 1, G32_OUT_PLANES = 2 };

struct Gemm32Args {
  int M, N, K, n_tiles_m, n_tiles_n;
  const float* bias;
  void* C;
  long long ldc, c_plane;
  int out;
  const bf16* A;      // as the tensor map sees it: read again only where a sum is NaN
  long long lda, a_plane;
  const bf16* W;
  long long ldw;
};

// An infinite weight times a term that is zero, or of the other sign, is a NaN that the product of the uncut number is not: outputs that came out NaN
// are taken again in fp32 multiply-adds (by the thread that wrote them)
__device__ __noinline__ void gemm32_mend(const Gemm32Args& a, int row, int col0, int cols) {
#pragma unroll 1
  for (int c = col0; c < col0 + cols && c < a.N; ++c) {
    const long long at = (long long)row * a.ldc + c;
    const float was = a.out == G32_OUT_F32 ? reinterpret_cast<const float*>(a.C)[at] : (float)reinterpret_cast<const bf16*>(a.C)[at];
    if (was == was) continue;
    const bf16* x = a.A + (long long)row * a.lda;
    const bf16* w = a.W + (long long)c * a.ldw;
    float s = 0.f;
#pragma unroll 1
    for (int k = 0; k < a.K && s == s; ++k) s = fmaf(s32_value(x + k, a.a_plane), (float)w[k], s);
    if (a.bias != nullptr) s += a.bias[c];
    if (a.out == G32_OUT_F32) {
      reinterpret_cast<float*>(a.C)[at] = s;
    } else if (a.out == G32_OUT_BF16) {
      reinterpret_cast<bf16*>(a.C)[at] = __float2bfloat16(s);
    } else {
      uint32_t h, m, l;
      s32_terms(s, 0.f, h, m, l);
      uint16_t* p = reinterpret_cast<uint16_t*>(a.C) + at;
      p[0] = (uint16_t)h;
      p[a.c_plane] = (uint16_t)m;
      p[2 * a.c_plane] = (uint16_t)l;
    }
  }
}

template <int BN>
struct Gemm32Smem {
  static constexpr int STAGES = BN == 256 ? 2 : 3;
  static constexpr int W_BYTES = BN * 128, STAGE = W_BYTES + 3 * S32_BOX;
  static constexpr int BAR_OFF = STAGES * STAGE, TOTAL = BAR_OFF + 256 + 1024;
};

template <int BN>
__global__ void __launch_bounds__(G32_THREADS, 1)
gemm32_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ Gemm32Args a) {
  using S = Gemm32Smem<BN>;
  constexpr int STAGES = S::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);      // [STAGES][4]: W, lo, mid, hi
  uint64_t* empty = full + STAGES * 4;
  uint64_t* acc_full = empty + STAGES * 4;                               // [2]
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int tiles = a.n_tiles_m * a.n_tiles_n, kb_n = (a.K + 63) / 64;
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < STAGES * 4; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full + i, 1);
      mbar_init(acc_empty + i, G32_EPI);
    }
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_ptr, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = *tmem_ptr;
  // tiles of one column of W run side by side on different SMs, so W's boxes are shared through L2
  if (warp < 4) {
  s32_fewer_regs<S32_FEW>();
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmW);
      int it = 0;
      for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int m0 = (tile % a.n_tiles_m) * 128, n0 = (tile / a.n_tiles_m) * BN;
        for (int kb = 0; kb < kb_n; ++kb, ++it) {
          const int st = it % STAGES;
          const uint32_t ph = (uint32_t)(it / STAGES) & 1;
          uint8_t* base = smem + st * S::STAGE;
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            if (it >= STAGES) mbar_wait(empty + st * 4 + p, ph ^ 1);
            mbar_arrive_expect_tx(full + st * 4 + p, p == 0 ? S::W_BYTES : S32_BOX);
            if (p == 0) tma_load_2d(base, &tmW, full + st * 4, kb * 64, n0);
            else tma_load_3d(base + S::W_BYTES + (p - 1) * S32_BOX, &tmA, full + st * 4 + p, kb * 64, m0, 3 - p);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, BN, 0, 0);
      int it = 0;
      for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        for (int kb = 0; kb < kb_n; ++kb, ++it) {
          const int st = it % STAGES, b = it & 1;
          const uint32_t ph = (uint32_t)(it / STAGES) & 1;
          const uint32_t base = smem_u32(smem + st * S::STAGE);
          if (it >= 2) mbar_wait(acc_empty + b, ((uint32_t)(it >> 1) & 1) ^ 1);
          mbar_wait(full + st * 4, ph);
#pragma unroll
          for (int p = 1; p < 4; ++p) {      // the small terms first
            mbar_wait(full + st * 4 + p, ph);
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_ss(tm + (uint32_t)b * BN, umma_desc_sw128(base + S::W_BYTES + (p - 1) * S32_BOX + ks * 32, 0, 1024),
                      umma_desc_sw128(base + ks * 32, 0, 1024), idesc, (p > 1 || ks > 0) ? 1u : 0u);
            umma_commit(empty + st * 4 + p);
          }
          umma_commit(empty + st * 4);
          umma_commit(acc_full + b);
        }
      }
    }
  }
  } else {
    s32_more_regs<S32_MANY>();
    const int lg = warp & 3, half = (warp - 4) >> 2;
    const uint32_t lane_addr = tm + ((uint32_t)(lg * 32) << 16) + half * (BN / 2);
    int it = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int row = (tile % a.n_tiles_m) * 128 + lg * 32 + lane, n0 = (tile / a.n_tiles_m) * BN + half * (BN / 2);
      float acc[BN / 2];
#pragma unroll
      for (int i = 0; i < BN / 2; ++i) acc[i] = 0.f;
      for (int kb = 0; kb < kb_n; ++kb, ++it) {
        const int b = it & 1;
        mbar_wait(acc_full + b, (uint32_t)(it >> 1) & 1);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < BN / 64; ++c) {
          uint32_t v[32];
          LP_TMEM_LD_32(v, lane_addr + b * BN + c * 32);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[c * 32 + i] += __uint_as_float(v[i]);
        }
        tc_fence_before();
        mbar_arrive(acc_empty + b);
      }
      if (row < a.M) {
        bool odd = false;
#pragma unroll
        for (int g = 0; g < BN / 16; ++g) {
          const int col = n0 + g * 8;
          if (col < a.N) {
            float* v = acc + g * 8;
            if (a.bias != nullptr) {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] += a.bias[col + i];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) odd |= v[i] != v[i];
            const long long at = (long long)row * a.ldc + col;
            if (a.out == G32_OUT_F32) {
              float4* p = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.C) + at);
              p[0] = make_float4(v[0], v[1], v[2], v[3]);
              p[1] = make_float4(v[4], v[5], v[6], v[7]);
            } else if (a.out == G32_OUT_BF16) {
              *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(a.C) + at) =
                  make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
            } else {
              s32_store_terms(reinterpret_cast<bf16*>(a.C) + at, a.c_plane, v);
            }
          }
        }
        if (odd) gemm32_mend(a, row, n0, BN / 2);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tm, 2 * BN);
  }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// Latent attention of prompts, keys and values expanded per head: 192 products a score and 128 a value instead of the 576 and 512 that the
// latents themselves take.  The visible rows of a request's cache become a contiguous run of key rows: request s has the positions from
// max(0, pos0 - window + 1) to its last, one request after the other.
// ---------------------------------------------------------------------------------------------------------------------------------
struct Seqs32 {
  int n, window;
  const int* row0;      // [n + 1]
  const int* pos0;
};
__device__ __forceinline__ int seq_first_key(const Seqs32& q, int pos0) { return q.window > 0 && pos0 - q.window + 1 > 0 ? pos0 - q.window + 1 : 0; }

// cache rows (latent, then the rotated key part) of the visible positions -> planes [3][n_keys][width], eight columns a thread
__global__ void __launch_bounds__(256) latent_gather_kernel(Seqs32 q, int n_keys, const float* __restrict__ cache, int page_size,
                                                            const int* __restrict__ page_table, int max_pages, int width, bf16* __restrict__ dst,
                                                            long long plane) {
  const int per = width >> 3;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)n_keys * per) return;
  const int k = (int)(i / per), c = (int)(i - (long long)k * per) * 8;
  int s = 0, left = k, lo = 0;
  for (; s < q.n; ++s) {
    const int p0 = q.pos0[s];
    lo = seq_first_key(q, p0);
    const int count = p0 + q.row0[s + 1] - q.row0[s] - lo;
    if (left < count) break;
    left -= count;
  }
  if (s >= q.n) return;
  const int pos = lo + left;
  const float* src = cache + ((long long)page_table[(long long)s * max_pages + pos / page_size] * page_size + pos % page_size) * width + c;
  const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + 4);
  const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  s32_store_terms(dst + (long long)k * width + c, plane, v);
}

struct Attn32Args {
  Seqs32 seqs;
  int heads, head0;      // this launch has heads head0 .. head0 + gridDim.x - 1; keys and values lie from head0 on
  float scale;
  const float* sink;
  const float* gate;     // [rows, ldg]: head h's output is multiplied by sigmoid(gate[r, h])
  long long ldg;
  const float* out_gate; // [rows, ldog]: output c of head h is multiplied by sigmoid(out_gate[r, 128 h + c])
  long long ldog;
  void* out;
  long long ldo;
  int out_fp32;
  // as the tensor maps see them: read again only where an output is not finite
  const bf16 *q, *k, *kr, *v;
  long long ldq, ldk, ldkr, q_plane, k_plane, kr_plane;
};

constexpr int A32_THREADS = 384;
template <int NR>
struct Attn32Smem {
  static constexpr int NB = 2 + NR, DQ = 64 * NB;      // 64-channel blocks of a query / key
  static constexpr int SLOTS = NR ? 4 : 6;
  static constexpr int RING = 3 * NB * S32_BOX, BAR_OFF = RING + SLOTS * S32_BOX, TOP_OFF = BAR_OFF + 256, TOTAL = TOP_OFF + 2 * 2 * 128 * 4 + 1024;
};

// the rows of a tile again, each over the keys it sees, in fp32 multiply-adds: a warp a row, a lane a key and four channels
template <int NR>
__device__ __noinline__ void attn32_plain(const Attn32Args& a, int r0, int nrows, int pos0, int kbase, int klo, int hl, float* p_s, int n_warps) {
  constexpr int DQ = Attn32Smem<NR>::DQ;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = a.head0 + hl;
  p_s += warp * 32;
  for (int x = warp; x < nrows; x += n_warps) {
    const int pos = pos0 + x, lo = seq_first_key(a.seqs, pos);
    const bf16* q = a.q + (long long)(r0 + x) * a.ldq + (long long)h * DQ;
    float mx = a.sink != nullptr ? a.sink[h] : -INFINITY, den = a.sink != nullptr ? 1.f : 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int t0 = lo; t0 <= pos; t0 += 32) {
      const int t = t0 + lane;
      float s = -INFINITY;
      if (t <= pos) {
        const long long kr = kbase + (t - klo);
        s = 0.f;
        for (int d = 0; d < DQ; ++d) {
          const float kv = d < 128 ? s32_value(a.k + kr * a.ldk + hl * 128 + d, a.k_plane) : s32_value(a.kr + kr * a.ldkr + (d - 128), a.kr_plane);
          s = fmaf(s32_value(q + d, a.q_plane), kv, s);
        }
        s *= a.scale;
      }
      float top = s;
      for (int m = 16; m > 0; m >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, m));
      const float mn = fmaxf(mx, top), ref = mn == -INFINITY ? 0.f : mn, corr = expf(mx - ref), p = t <= pos ? expf(s - ref) : 0.f;
      float sum = p;
      for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
      den = fmaf(den, corr, sum);
      mx = mn;
      p_s[lane] = p;
      __syncwarp();
      for (int i = 0; i < 4; ++i) o[i] *= corr;
      for (int j = 0; j < 32 && t0 + j <= pos; ++j) {
        const long long kr = kbase + (t0 + j - klo);
        for (int i = 0; i < 4; ++i) o[i] = fmaf(p_s[j], s32_value(a.v + kr * a.ldk + hl * 128 + lane + 32 * i, a.k_plane), o[i]);
      }
      __syncwarp();
    }
    float f = 1.0f / den;
    if (a.gate != nullptr) f *= 1.0f / (1.0f + expf(-a.gate[(long long)(r0 + x) * a.ldg + h]));
    for (int i = 0; i < 4; ++i) {
      const long long at = (long long)(r0 + x) * a.ldo + (long long)h * 128 + lane + 32 * i;
      if (a.out_gate != nullptr) o[i] *= 1.0f / (1.0f + expf(-a.out_gate[(long long)(r0 + x) * a.ldog + h * 128 + lane + 32 * i]));
      if (a.out_fp32) reinterpret_cast<float*>(a.out)[at] = o[i] * f;
      else reinterpret_cast<bf16*>(a.out)[at] = __float2bfloat16(o[i] * f);
    }
  }
}

// One CTA a head and 128 rows of a request, 128 keys at a time.
//   warp 0      TMA: the rows' queries once (3 planes), then keys and values through a ring of 16 KB boxes
//   warp 1      MMA: S(i + 1) = Q K^T is issued before P(i) V, so the tensor cores work while the softmax warps have S(i)
//   warps 4-11  softmax, a thread to one row and half of its keys and output channels: P's terms go back to TMEM over S (upper and middle) and
//               beside it (lower), and the output of the tile before is added to fp32 sums in registers
// TMEM columns: S of even and odd tiles [0, 128) [128, 256), lower terms of P [256, 320), P V of one tile [384, 512).
// The products of a tile, terms (key, query) or (value, weight): (2,0) (1,1) (1,0) (0,2) (0,1) and last (0,0), whose box is brought twice so
// that nothing small is added to a full-size sum.  Tensor time of a tile: 6 (DQ + 128) / 16 MMAs of 64 clocks.
template <int NR>
__global__ void __launch_bounds__(A32_THREADS, 1)
attn32_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmKr,
              const __grid_constant__ CUtensorMap tmV, const __grid_constant__ Attn32Args a) {
  using S = Attn32Smem<NR>;
  constexpr int NB = S::NB, SLOTS = S::SLOTS;
  constexpr uint32_t TM_X = 256, TM_O = 384;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);
  uint64_t* full = q_full + 1;            // [SLOTS]
  uint64_t* empty = full + SLOTS;         // [SLOTS]
  uint64_t* s_full = empty + SLOTS;       // [2]
  uint64_t* p_full = s_full + 2;
  uint64_t* pv_done = p_full + 1;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(pv_done + 1);
  float* top_s = reinterpret_cast<float*>(smem + S::TOP_OFF);      // [2][2][128]
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // this tile's request and rows, and where its keys lie; later tiles see more keys: they start first
  int tile = (int)gridDim.y - 1 - (int)blockIdx.y, s = 0, kbase = 0, r0 = 0, nrows = 0, pos0 = 0, klo = 0;
  for (; s < a.seqs.n; ++s) {
    const int first = a.seqs.row0[s], len = a.seqs.row0[s + 1] - first, p0 = a.seqs.pos0[s], tiles = (len + 127) >> 7;
    klo = seq_first_key(a.seqs, p0);
    if (tile < tiles) {
      r0 = first + tile * 128;
      nrows = min(128, len - tile * 128);
      pos0 = p0 + tile * 128;
      break;
    }
    tile -= tiles;
    kbase += p0 + len - klo;
  }
  if (s >= a.seqs.n) return;
  const int hl = blockIdx.x, h = a.head0 + hl;
  const int key0 = seq_first_key(a.seqs, pos0) - klo, key_end = pos0 + nrows - klo;      // of the request's run
  const int n = (key_end - key0 + 127) >> 7;

  if (warp == 1 && lane == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < SLOTS; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_full + 1, 1);
    mbar_init(p_full, 256);
    mbar_init(pv_done, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = *tmem_ptr;
  bool odd = false;
  if (warp < 4) {
  s32_fewer_regs<S32_FEW>();
  if (warp == 0) {
    if (lane == 0) {
      int u = 0;
      auto slot = [&]() {
        const int st = u % SLOTS;
        if (u >= SLOTS) mbar_wait(empty + st, ((uint32_t)(u / SLOTS) & 1) ^ 1);
        mbar_arrive_expect_tx(full + st, S32_BOX);
        ++u;
        return st;
      };
      auto keys = [&](int i) {
        for (int g = 0; g < 4; ++g)
          for (int b = 0; b < NB; ++b) {
            const int st = slot(), pl = g == 0 ? 2 : g == 1 ? 1 : 0;
            if (b < 2) tma_load_3d(smem + S::RING + st * S32_BOX, &tmK, full + st, hl * 128 + b * 64, kbase + key0 + i * 128, pl);
            else tma_load_3d(smem + S::RING + st * S32_BOX, &tmKr, full + st, 0, kbase + key0 + i * 128, pl);
          }
      };
      auto values = [&](int i) {
        for (int g = 0; g < 4; ++g)
          for (int kh = 0; kh < 2; ++kh) {
            const int st = slot(), pl = g == 0 ? 2 : g == 1 ? 1 : 0;
            for (int d = 0; d < 2; ++d)
              tma_load_3d(smem + S::RING + st * S32_BOX + d * (S32_BOX / 2), &tmV, full + st, hl * 128 + d * 64, kbase + key0 + i * 128 + kh * 64, pl);
          }
      };
      mbar_arrive_expect_tx(q_full, 3 * NB * S32_BOX);
      for (int p = 0; p < 3; ++p)
        for (int b = 0; b < NB; ++b) tma_load_3d(smem + (p * NB + b) * S32_BOX, &tmQ, q_full, h * S::DQ + b * 64, r0, p);
      keys(0);
      for (int i = 0; i < n; ++i) {
        if (i + 1 < n) keys(i + 1);
        values(i);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0), idesc_o = umma_idesc_bf16(128, 128, 0, 1);
      const uint32_t q_addr = smem_u32(smem);
      int u = 0;
      auto box = [&]() {
        const int st = u % SLOTS;
        mbar_wait(full + st, (uint32_t)(u / SLOTS) & 1);
        tc_fence_after();
        ++u;
        return st;
      };
      // boxes of term pl of the second operand and the terms of the first that they meet
      auto scores = [&](int i) {
        const uint32_t d = tm + (uint32_t)(i & 1) * 128;
        uint32_t more = 0;
        for (int g = 0; g < 4; ++g) {
          const int from = g == 0 ? 0 : g == 1 ? 1 : g == 2 ? 2 : 0, to = g == 2 ? 1 : 0;
          for (int b = 0; b < NB; ++b) {
            const int st = box();
            const uint32_t k_addr = smem_u32(smem + S::RING + st * S32_BOX);
            for (int q = from; q >= to; --q)
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                umma_ss(d, umma_desc_sw128(q_addr + (q * NB + b) * S32_BOX + ks * 32, 0, 1024), umma_desc_sw128(k_addr + ks * 32, 0, 1024), idesc_s, more);
                more = 1;
              }
            umma_commit(empty + st);
          }
        }
        umma_commit(s_full + (i & 1));
      };
      auto outputs = [&](int i) {
        const uint32_t p = tm + (uint32_t)(i & 1) * 128;
        uint32_t more = 0;
        for (int g = 0; g < 4; ++g) {
          const int from = g == 0 ? 0 : g == 1 ? 1 : g == 2 ? 2 : 0, to = g == 2 ? 1 : 0;
          for (int kh = 0; kh < 2; ++kh) {
            const int st = box();
            const uint32_t v_addr = smem_u32(smem + S::RING + st * S32_BOX);
            for (int q = from; q >= to; --q)
#pragma unroll
              for (int k4 = 0; k4 < 4; ++k4) {
                const int ks = kh * 4 + k4;      // 16 keys: upper and middle terms lie side by side, 32 keys at a time
                const uint32_t p_addr = q == 2 ? tm + TM_X + ks * 8 : p + (ks >> 1) * 32 + (ks & 1) * 8 + q * 16;
                umma_ts(tm + TM_O, p_addr, umma_desc_sw128(v_addr + k4 * 2048, S32_BOX / 2, 1024), idesc_o, more);
                more = 1;
              }
            umma_commit(empty + st);
          }
        }
        umma_commit(pv_done);
      };
      mbar_wait(q_full, 0);
      scores(0);
      for (int i = 0; i < n; ++i) {
        if (i + 1 < n) scores(i + 1);
        mbar_wait(p_full, i & 1);
        tc_fence_after();
        outputs(i);
      }
    }
  }
  } else {
    s32_more_regs<S32_MANY>();
    const int lg = warp & 3, hh = (warp - 4) >> 2, x = lg * 32 + lane;
    const uint32_t lane_addr = tm + ((uint32_t)(lg * 32) << 16);
    const bool mine = x < nrows;
    const int my_lo = seq_first_key(a.seqs, pos0 + x) - klo, my_hi = mine ? pos0 + x - klo : -1;
    const int all_lo = seq_first_key(a.seqs, pos0 + nrows - 1) - klo, all_hi = pos0 - klo;      // keys that every row sees
    float mx = a.sink != nullptr ? a.sink[h] : -INFINITY, den = a.sink != nullptr && hh == 0 ? 1.f : 0.f, corr_before = 0.f;
    float o[64];
#pragma unroll
    for (int c = 0; c < 64; ++c) o[c] = 0.f;
    auto add_outputs = [&](float corr) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t w[32];
        LP_TMEM_LD_32(w, lane_addr + TM_O + hh * 64 + c * 32);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) o[c * 32 + j] = fmaf(o[c * 32 + j], corr, __uint_as_float(w[j]));
      }
    };
    for (int i = 0; i < n; ++i) {
      uint32_t v[64];
      mbar_wait(s_full + (i & 1), (uint32_t)(i >> 1) & 1);
      tc_fence_after();
      const uint32_t s_addr = lane_addr + (uint32_t)(i & 1) * 128 + hh * 64;
      LP_TMEM_LD_32((v + 0), s_addr);
      LP_TMEM_LD_32((v + 32), s_addr + 32);
      tmem_wait_ld();
      const int k0 = key0 + i * 128;
      const bool whole = nrows == 128 && k0 >= all_lo && k0 + 127 <= all_hi;
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 64; ++j) {
        float sc = __uint_as_float(v[j]) * a.scale;
        if (!whole) {
          const int idx = k0 + hh * 64 + j;
          if (idx < my_lo || idx > my_hi) sc = -INFINITY;
        }
        v[j] = __float_as_uint(sc);
        top = fmaxf(top, sc);
      }
      float* ts = top_s + (i & 1) * 256;
      ts[hh * 128 + x] = top;
      s32_bar(1 + lg, 64);
      const float mn = fmaxf(mx, fmaxf(top, ts[(hh ^ 1) * 128 + x])), ref = mn == -INFINITY ? 0.f : mn;      // -inf: nothing seen so far
      const float corr = expf(mx - ref);
      float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
      for (int j = 0; j < 64; j += 2) {
        const float p0 = expf(__uint_as_float(v[j]) - ref), p1 = expf(__uint_as_float(v[j + 1]) - ref);      // exp(-inf) = 0: not seen
        v[j] = __float_as_uint(p0);
        v[j + 1] = __float_as_uint(p1);
        sum0 += p0;
        sum1 += p1;
      }
      den = fmaf(den, corr, sum0 + sum1);
      mx = mn;
      if (i > 0) {      // P V of the tile before has run: its sums are taken, and its lower terms of P are no longer read
        mbar_wait(pv_done, (uint32_t)(i - 1) & 1);
        tc_fence_after();
        add_outputs(corr_before);
      }
      corr_before = corr;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[16], mid[16], lo[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) s32_terms(__uint_as_float(v[c * 32 + 2 * j]), __uint_as_float(v[c * 32 + 2 * j + 1]), hi[j], mid[j], lo[j]);
        LP_TMEM_ST_16(hi, s_addr + c * 32);
        LP_TMEM_ST_16(mid, s_addr + c * 32 + 16);
        LP_TMEM_ST_16(lo, lane_addr + TM_X + hh * 32 + c * 16);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full);
    }
    mbar_wait(pv_done, (uint32_t)(n - 1) & 1);
    tc_fence_after();
    add_outputs(corr_before);
    float* ds = top_s + (n & 1) * 256;
    ds[hh * 128 + x] = den;
    s32_bar(1 + lg, 64);
    den += ds[(hh ^ 1) * 128 + x];
    if (mine) {
      float f = 1.0f / den;
      if (a.gate != nullptr) f *= 1.0f / (1.0f + expf(-a.gate[(long long)(r0 + x) * a.ldg + h]));
      const long long at = (long long)(r0 + x) * a.ldo + (long long)h * 128 + hh * 64;
#pragma unroll
      for (int c = 0; c < 64; ++c) {
        odd |= !(fabsf(o[c]) <= 3.402823466e38f);
        o[c] *= f;
      }
      if (a.out_gate != nullptr) {
        const float* g = a.out_gate + (long long)(r0 + x) * a.ldog + h * 128 + hh * 64;
#pragma unroll
        for (int c = 0; c < 64; ++c) o[c] *= 1.0f / (1.0f + expf(-g[c]));
      }
      if (a.out_fp32) {
        float4* p = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + at);
#pragma unroll
        for (int c = 0; c < 16; ++c) p[c] = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
      } else {
        uint4* p = reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(a.out) + at);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          p[c] = make_uint4(pack_bf16x2(o[8 * c], o[8 * c + 1]), pack_bf16x2(o[8 * c + 2], o[8 * c + 3]), pack_bf16x2(o[8 * c + 4], o[8 * c + 5]),
                            pack_bf16x2(o[8 * c + 6], o[8 * c + 7]));
      }
    }
  }
  tc_fence_before();
  const int again = __syncthreads_or(odd);
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tm, 512);
  }
  // an infinity or a NaN among the keys or values: weights of zero times it are NaN in every row of the product, seen or not
  if (again) attn32_plain<NR>(a, r0, nrows, pos0, kbase, klo, hl, reinterpret_cast<float*>(smem), A32_THREADS / 32);
}

}  // namespace lp

#ifndef LP_EMULATE
using namespace lp;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

extern "C" int lp_split_rows(const float* src, long long ld, int M, int K, void* planes, long long ldp, long long plane, void* stream_) {
  LP_REQUIRE(src != nullptr && planes != nullptr, "lp_split_rows: null operand");
  LP_REQUIRE(K % 8 == 0 && ld % 4 == 0 && ldp % 8 == 0 && plane % 8 == 0 && aligned16(src) && aligned16(planes), "lp_split_rows: 16-byte rows of whole eights");
  if (M <= 0 || K <= 0) return 0;
  const long long pieces = (long long)M * (K >> 3);
  split_rows_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(src, ld, M, K, reinterpret_cast<bf16*>(planes), ldp, plane);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

template <int BN>
static int launch_gemm32(Gemm32Args a, cudaStream_t stream) {
  using S = Gemm32Smem<BN>;
  static bool configured = false;
  auto kern = gemm32_kernel<BN>;
  if (!configured) {
    LP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    configured = true;
  }
  CUtensorMap ta, tw;
  if (int rc = make_tmap_bf16_3d(&ta, a.A, a.K, a.M, 3, a.lda, a.a_plane, 64, 128, 1)) return rc;
  if (int rc = make_tmap_bf16_2d(&tw, a.W, a.K, a.N, a.ldw, 64, BN)) return rc;
  a.n_tiles_m = (a.M + 127) / 128;
  a.n_tiles_n = (a.N + BN - 1) / BN;
  const int tiles = a.n_tiles_m * a.n_tiles_n;
  kern<<<tiles < sm_count() ? tiles : sm_count(), G32_THREADS, S::TOTAL, stream>>>(ta, tw, a);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}
static int gemm32(const Gemm32Args& a, cudaStream_t stream) {
  if (a.M <= 0 || a.N <= 0) return 0;
  // a k block of a 256-wide tile takes 1,536 tensor clocks, of a 128-wide one 1,090 (its operands come no faster)
  const long long m = (a.M + 127) / 128, sms = sm_count();
  const long long wide = (m * ((a.N + 255) / 256) + sms - 1) / sms * 1536, narrow = (m * ((a.N + 127) / 128) + sms - 1) / sms * 1090;
  return wide < narrow ? launch_gemm32<256>(a, stream) : launch_gemm32<128>(a, stream);
}

extern "C" int lp_gemm_split(const void* A, long long lda, long long a_plane, const void* W, long long ldw, void* C, long long ldc, long long c_plane,
                             int out, int M, int N, int K, const float* bias, void* stream_) {
  LP_REQUIRE(A != nullptr && W != nullptr && C != nullptr, "lp_gemm_split: null operand");
  LP_REQUIRE(out >= G32_OUT_BF16 && out <= G32_OUT_PLANES, "lp_gemm_split: unknown output form %d", out);
  LP_REQUIRE(K >= 8 && K % 8 == 0 && N % 8 == 0 && lda % 8 == 0 && a_plane % 8 == 0 && ldw % 8 == 0 && ldc % (out == G32_OUT_F32 ? 4 : 8) == 0 && c_plane % 8 == 0 &&
                 aligned16(A) && aligned16(W) && aligned16(C),
             "lp_gemm_split: 16-byte rows of whole eights");
  Gemm32Args a = {};
  a.M = M; a.N = N; a.K = K;
  a.bias = bias;
  a.C = C; a.ldc = ldc; a.c_plane = c_plane; a.out = out;
  a.A = reinterpret_cast<const bf16*>(A); a.lda = lda; a.a_plane = a_plane;
  a.W = reinterpret_cast<const bf16*>(W); a.ldw = ldw;
  return gemm32(a, reinterpret_cast<cudaStream_t>(stream_));
}

// ---- latent attention, keys and values expanded
constexpr size_t LX_GROUP_BYTES = (size_t)512 << 20;      // heads whose expanded keys and values are held at a time
static int lx_group(int heads, int n_keys) {
  const long long one = (long long)n_keys * 256 * 6;
  const long long g = (long long)LX_GROUP_BYTES / (one > 0 ? one : 1);
  return g < 1 ? 1 : g < heads ? (int)g : heads;
}
static size_t lx_round(size_t b) { return (b + 255) & ~(size_t)255; }

extern "C" size_t lp_latent_expanded_workspace_bytes(int R, int heads, int dim, int rot_dim, int kv_rank, int n_keys) {
  return lx_round((size_t)6 * R * heads * (dim + rot_dim)) + lx_round((size_t)6 * n_keys * (kv_rank + rot_dim)) +
         lx_round((size_t)6 * n_keys * lx_group(heads, n_keys) * 256);
}

extern "C" int lp_latent_attend_expanded(const lp_latent_desc* d, int R, int n_seqs, const int* seq_row0, const int* seq_pos0, int n_tiles, int n_keys,
                                         const void* w_kv, long long ldw, const float* out_gate, long long ldog, void* out, long long ldo, int out_fp32,
                                         void* ws, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LP_REQUIRE(d != nullptr && d->q != nullptr && d->cache != nullptr && d->page_table != nullptr && seq_row0 != nullptr && seq_pos0 != nullptr &&
                 w_kv != nullptr && out != nullptr && ws != nullptr,
             "lp_latent_attend_expanded: null operand");
  LP_REQUIRE(d->dim == 128 && d->rot_dim == 64, "lp_latent_attend_expanded: heads of 128 + 64 only, not %d + %d", d->dim, d->rot_dim);
  LP_REQUIRE(d->kv_rank >= 8 && d->kv_rank % 8 == 0 && d->ldq % 4 == 0 && ldw % 8 == 0 && ldo % (out_fp32 ? 4 : 8) == 0 && aligned16(d->q) &&
                 aligned16(d->cache) && aligned16(w_kv) && aligned16(out) && aligned16(ws) && d->page_size > 0,
             "lp_latent_attend_expanded: 16-byte rows of whole eights");
  LP_REQUIRE(ws_bytes >= lp_latent_expanded_workspace_bytes(R, d->heads, d->dim, d->rot_dim, d->kv_rank, n_keys), "lp_latent_attend_expanded: workspace");
  if (R <= 0 || n_seqs <= 0 || n_tiles <= 0 || n_keys <= 0) return 0;
  LP_REQUIRE(n_tiles <= 65535, "lp_latent_attend_expanded: %d tiles", n_tiles);
  const int H = d->heads, C = d->kv_rank, width = C + d->rot_dim, G = lx_group(H, n_keys);
  bf16* q_p = reinterpret_cast<bf16*>(ws);
  bf16* c_p = q_p + lx_round((size_t)6 * R * H * 192) / 2;
  bf16* kv_p = c_p + lx_round((size_t)6 * n_keys * width) / 2;
  const long long q_plane = (long long)R * H * 192, c_plane = (long long)n_keys * width;
  if (int rc = lp_split_rows(d->q, d->ldq, R, H * 192, q_p, (long long)H * 192, q_plane, stream_)) return rc;
  Seqs32 seqs = {n_seqs, d->window, seq_row0, seq_pos0};
  const long long pieces = (long long)n_keys * (width >> 3);
  latent_gather_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, stream>>>(seqs, n_keys, d->cache, d->page_size, d->page_table, d->max_pages, width, c_p, c_plane);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  using S = Attn32Smem<1>;
  auto kern = attn32_kernel<1>;
  static bool configured = false;
  if (!configured) {
    LP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    configured = true;
  }
  CUtensorMap tq, tr;
  if (int rc = make_tmap_bf16_3d(&tq, q_p, (uint64_t)H * 192, R, 3, (uint64_t)H * 192, q_plane, 64, 128, 1)) return rc;
  if (int rc = make_tmap_bf16_3d(&tr, c_p + C, 64, n_keys, 3, width, c_plane, 64, 128, 1)) return rc;
  const bf16* W = reinterpret_cast<const bf16*>(w_kv);
  for (int h0 = 0; h0 < H; h0 += G) {
    const int g = H - h0 < G ? H - h0 : G;
    const long long ld = 256LL * g, plane = ld * n_keys;
    Gemm32Args m = {};
    m.M = n_keys; m.K = C;
    m.A = c_p; m.lda = width; m.a_plane = c_plane;
    m.ldw = ldw;
    m.ldc = ld; m.c_plane = plane; m.out = G32_OUT_PLANES;
    if (g == H) {      // both weights in one product
      m.W = W; m.C = kv_p; m.N = 256 * H;
      if (int rc = gemm32(m, stream)) return rc;
    } else {
      m.N = 128 * g;
      m.W = W + (long long)h0 * 128 * ldw; m.C = kv_p;
      if (int rc = gemm32(m, stream)) return rc;
      m.W = W + (long long)(H + h0) * 128 * ldw; m.C = kv_p + 128 * g;
      if (int rc = gemm32(m, stream)) return rc;
    }
    CUtensorMap tk, tv;
    if (int rc = make_tmap_bf16_3d(&tk, kv_p, 128ULL * g, n_keys, 3, ld, plane, 64, 128, 1)) return rc;
    if (int rc = make_tmap_bf16_3d(&tv, kv_p + 128 * g, 128ULL * g, n_keys, 3, ld, plane, 64, 64, 1)) return rc;
    Attn32Args a = {};
    a.seqs = seqs; a.heads = H; a.head0 = h0;
    a.scale = d->scale; a.sink = d->sink; a.gate = d->gate; a.ldg = d->ldg;
    a.out_gate = out_gate; a.ldog = ldog;
    a.out = out; a.ldo = ldo; a.out_fp32 = out_fp32;
    a.q = q_p; a.ldq = H * 192LL; a.q_plane = q_plane;
    a.k = kv_p; a.v = kv_p + 128 * g; a.ldk = ld; a.k_plane = plane;
    a.kr = c_p + C; a.ldkr = width; a.kr_plane = c_plane;
    kern<<<dim3(g, n_tiles), A32_THREADS, S::TOTAL, stream>>>(tq, tk, tr, tv, a);
    note_launch();
    LP_CHECK_CUDA(cudaGetLastError());
  }
  return 0;
}
#endif  // !LP_EMULATE

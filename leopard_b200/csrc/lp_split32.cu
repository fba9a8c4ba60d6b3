// leopard_b200 — 32-bit products and attention of prompts on the tcgen05 tensor cores.
//
// An fp32 number is three bf16 terms that add up to it (rounded to nearest, each takes 8 bits of what the ones before left).  Operands
// lie in memory as three planes of terms, so TMA brings them to shared memory as they are and the tensor cores take them:
//   gemm32_kernel   C[M, N] = A[M, K] W[N, K]^T, A in three planes, W bf16: every product is exact (three MMAs)
//   attn32_kernel   softmax(Q K^T) V, all three in planes, heads of 128 (+ 64 channels whose keys all heads share): the six products of weight
//                   above 2^-25 of a product
// The tensor cores cut their running sum off instead of rounding it, a bias that grows with the chain.  So chains are short, small terms go
// first, and sums of chains are fp32 additions in registers: 64 of K (four MMAs at full size) in the product, all channels of one
// score (8 or 12) and 64 keys of an output (4) in attention.
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
// of the 168 registers a thread that 384 threads start with, the warpgroup of TMA and MMA warps gives up 64 and the two others take 32 each
constexpr int S32_FEW = 104, S32_MANY = 200;

#ifdef LP_EMULATE
inline void s32_wait(uint64_t* bar, uint32_t parity) { mbar_wait(bar, parity); }
inline void s32_wait_warp(uint64_t* bar, uint32_t parity) { mbar_wait_warp(bar, parity); }
inline void s32_bar(int id, int n) { named_bar(id, n, true); }
inline float s32_ex2(float x) { return exp2f(x); }
inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t) { return (a >> 16) | (b & 0xffff0000u); }
template <int N> inline void s32_more_regs() { emu_registers = N; }
template <int N> inline void s32_fewer_regs() { emu_registers = N; }
inline void s32_serial() { emu_serial(); }
#else
__device__ __forceinline__ void s32_serial() {}      // where results are taken again one by one: the emulated build looks at what the CTA is about then
// as mbar_wait, without its message: a call in the loop of the warp that issues the MMAs costs it registers, and its spills the tensor cores' time
__device__ __forceinline__ void s32_wait(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (clock64() - t0 > LP_WATCHDOG_CYCLES) __trap();
}
__device__ __forceinline__ void s32_wait_warp(uint64_t* bar, uint32_t parity) {      // as mbar_wait_warp
  s32_wait(bar, parity);
  __syncwarp();
}
__device__ __forceinline__ float s32_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
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

// umma_desc_sw128 with the parts that do not change folded: `at` = (address >> 4) | (leading byte offset >> 4) << 16, steps are added to it
__device__ __forceinline__ uint64_t s32_desc(uint32_t at) { return umma_desc_sw128(0, 0, 1024) | at; }
// a place in a ring of N boxes and the parity of its round
template <int N>
struct Ring32 {
  int at = 0;
  uint32_t round = 0;
  __device__ __forceinline__ void next() {
    if (++at == N) {
      at = 0;
      round ^= 1;
    }
  }
};

// the upper halves of u and v, packed
__device__ __forceinline__ uint32_t s32_upper(uint32_t u, uint32_t v) { return __byte_perm(u, v, 0x7632); }
// the three terms of finite x and y, rounded to nearest each (what is left of a number after three of 8 bits and their signs is nothing), packed in pairs
__device__ __forceinline__ void s32_weight_terms(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(x, y);
  x -= __uint_as_float(hi << 16);
  y -= __uint_as_float(hi & 0xffff0000u);
  mid = pack_bf16x2(x, y);
  x -= __uint_as_float(mid << 16);
  y -= __uint_as_float(mid & 0xffff0000u);
  lo = pack_bf16x2(x, y);
}
// the same of any x and y: an infinity leaves nothing behind, a NaN stays one, and a number that would round to infinity has its bits cut off instead
__device__ __forceinline__ void s32_terms(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  if (fabsf(x) < 3.38e38f && fabsf(y) < 3.38e38f) return s32_weight_terms(x, y, hi, mid, lo);
  uint32_t u = __float_as_uint(x), v = __float_as_uint(y);
  const bool ux = (u & 0x7f800000u) == 0x7f800000u, vx = (v & 0x7f800000u) == 0x7f800000u;
  if (ux && (u & 0x7fffffu)) u |= 0x400000u;
  if (vx && (v & 0x7fffffu)) v |= 0x400000u;
  hi = s32_upper(u, v);
  x = ux ? 0.f : x - __uint_as_float(u & 0xffff0000u);
  y = vx ? 0.f : y - __uint_as_float(v & 0xffff0000u);
  u = __float_as_uint(x);
  v = __float_as_uint(y);
  mid = s32_upper(u, v);
  x -= __uint_as_float(u & 0xffff0000u);
  y -= __uint_as_float(v & 0xffff0000u);
  lo = s32_upper(__float_as_uint(x), __float_as_uint(y));
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

// a factor in two floats, so that its own rounding does not reach everything that it is applied to
struct Factor32 {
  float hi, lo;
};
inline Factor32 factor32(double f) {
  const float hi = (float)f;
  return {hi, (float)(f - (double)hi)};
}
// x times it; an infinity stays one
__device__ __forceinline__ float times32(float x, const Factor32& f) {
  const float y = x * f.hi;
  return fabsf(y) < INFINITY ? fmaf(x, f.hi, x * f.lo) : y;
}
// fp32 rows (times a factor) -> planes, eight columns a thread
template <bool SCALED>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ src, long long ld, int M, int K, bf16* __restrict__ dst,
                                                         long long ldd, long long plane, Factor32 factor) {
  const int per = K >> 3;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)M * per) return;
  const long long r = i / per;
  const int c = (int)(i - r * per) * 8;
  const float* s = src + r * ld + c;
  const float4 a = *reinterpret_cast<const float4*>(s), b = *reinterpret_cast<const float4*>(s + 4);
  float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (SCALED) v[i] = times32(v[i], factor);
  s32_store_terms(dst + r * ldd + c, plane, v);
}

// rows of src by an index (a negative one: zeros), eight columns a thread: bf16 as they are, or fp32 -> planes
template <bool SPLIT>
__global__ void __launch_bounds__(256) gather_rows_kernel(const void* __restrict__ src, long long ld, const int* __restrict__ row_of, int rows, int K,
                                                          bf16* __restrict__ dst, long long plane) {
  const int per = K >> 3;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)rows * per) return;
  const long long r = i / per;
  const int c = (int)(i - r * per) * 8, from = row_of[r];
  bf16* to = dst + r * K + c;
  if (SPLIT) {
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (from >= 0) {
      const float* s = reinterpret_cast<const float*>(src) + from * ld + c;
      const float4 a = *reinterpret_cast<const float4*>(s), b = *reinterpret_cast<const float4*>(s + 4);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    s32_store_terms(to, plane, v);
  } else {
    *reinterpret_cast<uint4*>(to) = from >= 0 ? *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(src) + from * ld + c) : make_uint4(0u, 0u, 0u, 0u);
  }
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
  long long w_group;          // between the weights of groups
  const int* tile_group;      // [n_tiles_m] weight group of each row tile (< 0: an empty tile), or null
  const float* row_scale;     // [M] multiplies a gated unit's products, or null
};

// An infinite weight times a term that is zero, or of the other sign, is a NaN that the product of the uncut number is not: outputs that came out NaN
// are taken again in fp32 multiply-adds (by the thread that wrote them, once its CTA's products have run: K steps an output are too long for other warps
// to wait on)
__device__ float gemm32_plain(const Gemm32Args& a, int row, const bf16* w) {
  const bf16* x = a.A + (long long)row * a.lda;
  float s = 0.f;
#pragma unroll 1
  for (int k = 0; k < a.K && s == s; ++k) s = fmaf(s32_value(x + k, a.a_plane), (float)w[k], s);
  return s;
}
__device__ __forceinline__ float gemm32_gated(float z, float u, float rs) {
  z *= rs;
  return z / (1.0f + expf(-z)) * (u * rs);
}
// What cutting off takes on average from a gated unit of three-term products: 0.6e-7 from each of its sums at every K from 64 to 8192 (1.29e-7 to 1.40e-7 of
// the result; without it both products of 8 experts, width and inside 512, were 2.42e-7 of the result off, with it 1.90, lp_linear_grouped 2.22; 1024 2.69, 2.19, 2.60)
constexpr float CUT_GATED = 1.3e-7f;
__device__ __noinline__ void gemm32_mend(const Gemm32Args& a, int row, int group, int col0, int cols, int gated) {
  s32_serial();
  const bf16* W = a.W + (long long)group * a.w_group;
#pragma unroll 1
  for (int c = col0; c < col0 + cols && c < (gated ? a.N / 2 : a.N); ++c) {
    const long long at = (long long)row * a.ldc + c;
    const float was = a.out == G32_OUT_F32 ? reinterpret_cast<const float*>(a.C)[at] : (float)reinterpret_cast<const bf16*>(a.C)[at];
    if (was == was) continue;
    float s = gemm32_plain(a, row, W + (long long)c * a.ldw);
    if (gated) s = gemm32_gated(s, gemm32_plain(a, row, W + (long long)(c + a.N / 2) * a.ldw), a.row_scale != nullptr ? a.row_scale[row] : 1.f);
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

template <int BN, int PLANES>
struct Gemm32Smem {
  static constexpr int STAGES = PLANES == 1 ? 4 : BN == 256 ? 2 : 3;
  static constexpr int W_BYTES = BN * 128, STAGE = W_BYTES + PLANES * S32_BOX;
  static constexpr int BAR_OFF = STAGES * STAGE, TOTAL = BAR_OFF + 320 + 1024;
};

// PLANES = 1: bf16 rows, chains of two k blocks (eight MMAs).  GATED: W's boxes are 64 rows of gates, the 64 of the same channels' other factors, 64
// more gates and theirs, so a thread that adds up 128 columns has both halves of 64 outputs.
template <int BN, int PLANES, bool GATED>
__global__ void __launch_bounds__(G32_THREADS, 1)
gemm32_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ Gemm32Args a) {
  using S = Gemm32Smem<BN, PLANES>;
  constexpr int STAGES = S::STAGES, PARTS = PLANES + 1, CHAIN = PLANES == 1 ? 2 : 1, COLS = GATED ? BN / 2 : BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);      // [STAGES][PARTS]: W, then the smallest term to the largest
  uint64_t* empty = full + STAGES * PARTS;
  uint64_t* acc_full = empty + STAGES * PARTS;                           // [2]
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int tiles = a.n_tiles_m * a.n_tiles_n, kb_n = (a.K + 63) / 64;
  if (warp == 1 && lane == 0) {
    for (int i = 0; i < STAGES * PARTS; ++i) {
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
  // one product: tiles of one column of W run side by side on different SMs, so W's boxes are shared through L2; groups: a row tile's columns do
  auto tile_m = [&](int tile) { return a.tile_group == nullptr ? tile % a.n_tiles_m : tile / a.n_tiles_n; };
  auto tile_n = [&](int tile) { return a.tile_group == nullptr ? tile / a.n_tiles_m : tile % a.n_tiles_n; };
  auto group_of = [&](int tile) { return a.tile_group == nullptr ? 0 : a.tile_group[tile_m(tile)]; };      // < 0: nothing there
  if (warp < 4) {
    s32_fewer_regs<S32_FEW>();
    if (warp == 0) {
      if (lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmW);
        Ring32<STAGES> ring;
        int it = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
          const int m0 = tile_m(tile) * 128, n0 = tile_n(tile) * COLS, group = group_of(tile);
          if (group < 0) continue;
          for (int kb = 0; kb < kb_n; ++kb, ++it, ring.next()) {
            const int st = ring.at;
            uint8_t* base = smem + st * S::STAGE;
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
              if (it >= STAGES) s32_wait(empty + st * PARTS + p, ring.round ^ 1);
              mbar_arrive_expect_tx(full + st * PARTS + p, p == 0 ? S::W_BYTES : S32_BOX);
              if (p > 0) {
                tma_load_3d(base + S::W_BYTES + (p - 1) * S32_BOX, &tmA, full + st * PARTS + p, kb * 64, m0, PLANES - p);
              } else if (GATED) {
#pragma unroll
                for (int q = 0; q < BN / 64; ++q)
                  tma_load_3d(base + q * (S32_BOX / 2), &tmW, full + st * PARTS, kb * 64, (q & 1 ? a.N / 2 : 0) + n0 + (q >> 1) * 64, group);
              } else {
                tma_load_3d(base, &tmW, full + st * PARTS, kb * 64, n0, group);
              }
            }
          }
        }
      }
    } else if (warp == 1) {
      {
        const bool issue = elect_one();
        constexpr uint32_t idesc = umma_idesc_bf16(128, BN, 0, 0);
        const uint32_t first = smem_u32(smem) >> 4;
        Ring32<STAGES> ring;
        int chain = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
          if (group_of(tile) < 0) continue;
          for (int kb = 0; kb < kb_n; ++kb, ring.next()) {
            const int st = ring.at, b = chain & 1;
            const uint32_t base = first + st * (S::STAGE >> 4);
            const bool starts = kb % CHAIN == 0;
            if (starts && chain >= 2) s32_wait_warp(acc_empty + b, ((uint32_t)(chain >> 1) & 1) ^ 1);
            s32_wait_warp(full + st * PARTS, ring.round);
#pragma unroll
            for (int p = 1; p < PARTS; ++p) {      // the small terms first
              s32_wait_warp(full + st * PARTS + p, ring.round);
              tc_fence_after();
              if (issue) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                  umma_ss(tm + (uint32_t)b * BN, s32_desc(base + ((S::W_BYTES + (p - 1) * S32_BOX) >> 4) + ks * 2), s32_desc(base + ks * 2), idesc,
                          (p > 1 || ks > 0 || !starts) ? 1u : 0u);
                umma_commit(empty + st * PARTS + p);
              }
            }
            if (issue) umma_commit(empty + st * PARTS);
            if (kb % CHAIN == CHAIN - 1 || kb == kb_n - 1) {
              if (issue) umma_commit(acc_full + b);
              ++chain;
            }
          }
        }
      }
    }
  } else {
    s32_more_regs<S32_MANY>();
    const int lg = warp & 3, half = (warp - 4) >> 2;
    const uint32_t lane_addr = tm + ((uint32_t)(lg * 32) << 16) + half * (BN / 2);
    const int chains = (kb_n + CHAIN - 1) / CHAIN;
    int it = 0;
    uint32_t odd_turns = 0;      // bit t: a tile of turn t, t + 32, .. has a NaN
    for (int tile = blockIdx.x, turn = 0; tile < tiles; tile += gridDim.x, ++turn) {
      if (group_of(tile) < 0) continue;
      const int row = tile_m(tile) * 128 + lg * 32 + lane, n0 = tile_n(tile) * COLS + half * (COLS / 2);
      float acc[BN / 2];
#pragma unroll
      for (int i = 0; i < BN / 2; ++i) acc[i] = 0.f;
      for (int c0 = 0; c0 < chains; ++c0, ++it) {
        const int b = it & 1;
        s32_wait(acc_full + b, (uint32_t)(it >> 1) & 1);
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
        if (GATED) {
          const float rs = a.row_scale != nullptr ? a.row_scale[row] : 1.f;
#pragma unroll
          for (int g = 0; g < COLS / 16; ++g) {
            const int col = n0 + g * 8;
            if (col < a.N / 2) {
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                v[i] = gemm32_gated(acc[g * 8 + i], acc[COLS / 2 + g * 8 + i], rs);
                if (PLANES == 3) {
                  v[i] = fmaf(v[i], CUT_GATED, v[i]);
                  odd |= v[i] != v[i];
                }
              }
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
        } else {
#pragma unroll
          for (int g = 0; g < BN / 16; ++g) {
            const int col = n0 + g * 8;
            if (col < a.N) {
              float* v = acc + g * 8;
              if (a.bias != nullptr) {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] += a.bias[col + i];
              }
              if (PLANES == 3) {
#pragma unroll
                for (int i = 0; i < 8; ++i) odd |= v[i] != v[i];
              }
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
        }
        if (PLANES == 3 && odd) odd_turns |= 1u << (turn & 31);
      }
    }
    for (int tile = blockIdx.x, turn = 0; odd_turns != 0 && tile < tiles; tile += gridDim.x, ++turn)
      if (odd_turns >> (turn & 31) & 1) {
        const int row = tile_m(tile) * 128 + lg * 32 + lane;
        if (group_of(tile) >= 0 && row < a.M) gemm32_mend(a, row, group_of(tile), tile_n(tile) * COLS + half * (COLS / 2), COLS / 2, GATED);
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
// what a query at `pos` sees of its request: the first `keep` tokens, `blocks` means of pooled blocks, and the tokens from `lo` to its own
struct Seqs32 {
  int n, window;
  const int* row0;      // [n + 1]
  const int* pos0;
  int chunk, keep_first, pool;      // 0: no such rule
};
struct Seen32 {
  int keep, blocks, lo;
};
__host__ __device__ __forceinline__ Seen32 seen32(const Seqs32& q, int pos) {
  Seen32 v;
  v.lo = q.window > 0 && pos - q.window + 1 > 0 ? pos - q.window + 1 : 0;
  if (q.chunk > 0 && pos / q.chunk * q.chunk > v.lo) v.lo = pos / q.chunk * q.chunk;
  v.keep = q.keep_first < v.lo ? q.keep_first : v.lo;
  if (v.keep < 0) v.keep = 0;
  v.blocks = q.pool > 0 && q.window > 0 && pos - q.window + 1 > 0 ? (pos - q.window + 1) / q.pool : 0;
  return v;
}
// the key rows of one request: kept tokens and blocks that its last row sees, then the tokens from its first row's `lo` to the last
struct Run32 {
  int keep, blocks, lo, count;
};
__host__ __device__ __forceinline__ Run32 run32(const Seqs32& q, int pos0, int len) {
  const Seen32 last = seen32(q, pos0 + len - 1);
  Run32 r;
  r.keep = last.keep;
  r.blocks = last.blocks;
  r.lo = seen32(q, pos0).lo;
  r.count = r.keep + r.blocks + pos0 + len - r.lo;
  return r;
}

// cache rows of the visible positions (and block means) -> planes [3][n_keys][width], eight columns a thread
__global__ void __launch_bounds__(256) gather_keys_kernel(Seqs32 q, int n_keys, const float* __restrict__ cache, int page_size,
                                                          const int* __restrict__ page_table, int max_pages, const float* __restrict__ blocks,
                                                          const int* __restrict__ block_table, int max_block_pages, int width, bf16* __restrict__ dst,
                                                          long long plane) {
  const int per = width >> 3;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)n_keys * per) return;
  const int k = (int)(i / per), c = (int)(i - (long long)k * per) * 8;
  int s = 0, left = k;
  Run32 run = {};
  for (; s < q.n; ++s) {
    run = run32(q, q.pos0[s], q.row0[s + 1] - q.row0[s]);
    if (left < run.count) break;
    left -= run.count;
  }
  if (s >= q.n) return;
  const bool block = left >= run.keep && left < run.keep + run.blocks;
  const int at = left < run.keep ? left : block ? left - run.keep : run.lo + left - run.keep - run.blocks;
  const int page = block ? block_table[(long long)s * max_block_pages + at / page_size] : page_table[(long long)s * max_pages + at / page_size];
  const float* src = (block ? blocks : cache) + ((long long)page * page_size + at % page_size) * width + c;
  const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + 4);
  const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  s32_store_terms(dst + (long long)k * width + c, plane, v);
}

struct Attn32Args {
  Seqs32 seqs;
  int head0, ratio;      // this launch has heads head0 .. head0 + gridDim.x - 1; `ratio` of them share a key / value head, which lie from head0's on
  float cap;             // scores are cap * tanh(query * key), or 0: query * key.  The queries' planes hold what makes that the score times log2(e): scale32
  const float* sink;     // [heads] or null
  int sink_one;          // 1 joins the denominator
  int zero_empty;        // a row whose scores are all -inf gives zeros (else NaN)
  const float* gate;     // [rows, ldg]: head h's output is multiplied by sigmoid(gate[r, h])
  long long ldg;
  const float* out_gate; // [rows, ldog]: output c of head h is multiplied by sigmoid(out_gate[r, 128 h + c])
  long long ldog;
  const float2* turn;    // [rows][turn_half] (cos, sin): pair i of the first 2 turn_half output channels of every head is turned back by its angle, or null
  int turn_half, turn_interleaved;
  float out_scale;
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

constexpr float LOG2E = 1.4426950408889634f;
// What cutting sums off instead of rounding them takes from a score (eight to twelve full-size steps) and from an output (chains of four), of itself and on
// average: measured as the error's component along the score and along the output, 1.2e-7 to 1.4e-7 and 0.2e-7 to 1.0e-7 over 100 to 4096 rows, 128 and 192
// channels, windows of 100 keys and none, scores of deviation 0.2 and 1, values around 0 and around 1
constexpr double CUT_SCORE = 1.2e-7, CUT_OUT = 0.4e-7, TANH_OVER = 0.5e-7;      // (tanhf of a small number is the last so much too large)
// the factor of the queries and the cap of the scores, both for scores times log2(e)
inline Factor32 scale32(float scale, float softcap, float& cap) {
  constexpr double log2e = 1.4426950408889634;
  cap = softcap > 0.f ? (float)(softcap * log2e) : 0.f;
  // small scores are query * key * cap: what rounding takes from the cap goes to the queries
  return factor32((softcap > 0.f ? scale / (double)softcap * (softcap * log2e / cap) : scale * log2e) * (1.0 + CUT_SCORE - (softcap > 0.f ? TANH_OVER : 0.0)));
}
__device__ __forceinline__ float score32(const Attn32Args& a, float s) { return a.cap > 0.f ? a.cap * tanhf(s) : s; }
__device__ __forceinline__ float out32(const Attn32Args& a, int row, int h, int c, float v) {
  if (a.out_gate != nullptr) v *= 1.0f / (1.0f + expf(-a.out_gate[(long long)row * a.ldog + h * 128 + c]));
  return v * a.out_scale;
}
// channel c of a head's output row `o` (in shared memory), turned back by its row's position: (u, v) -> (u cos + v sin, v cos - u sin)
__device__ __forceinline__ float turned32(const Attn32Args& a, int row, int c, float v, const float* o) {
  if (c >= 2 * a.turn_half) return v;
  const bool first = a.turn_interleaved ? (c & 1) == 0 : c < a.turn_half;
  const int pair = a.turn_interleaved ? c >> 1 : first ? c : c - a.turn_half, partner = a.turn_interleaved ? c ^ 1 : first ? c + a.turn_half : c - a.turn_half;
  const float2 t = a.turn[(long long)row * a.turn_half + pair];
  return first ? v * t.x + o[partner] * t.y : v * t.x - o[partner] * t.y;
}
__global__ void __launch_bounds__(256) turn_table_kernel(Seqs32 q, int R, const float* __restrict__ inv_freq, int half, float2* __restrict__ table) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)R * half) return;
  const int r = (int)(i / half);
  int s = 0;
  while (s + 1 < q.n && r >= q.row0[s + 1]) ++s;
  float sn, cs;
  sincosf((float)(q.pos0[s] + r - q.row0[s]) * inv_freq[i - (long long)r * half], &sn, &cs);
  table[i] = make_float2(cs, sn);
}

// the rows of a tile again, each over the keys it sees, in fp32 multiply-adds: a warp a row, a lane a key and four channels
template <int NR>
__device__ __noinline__ void attn32_plain(const Attn32Args& a, int r0, int nrows, int pos0, int kbase, const Run32& run, int h, int kvl, float* p_s,
                                          int warp, int n_warps) {
  constexpr int DQ = Attn32Smem<NR>::DQ;
  const int lane = threadIdx.x & 31;
  s32_serial();
  p_s += warp * 160;
  for (int x = warp; x < nrows; x += n_warps) {
    const int pos = pos0 + x;
    const Seen32 see = seen32(a.seqs, pos);
    const int count = see.keep + see.blocks + pos - see.lo + 1;
    auto key_row = [&](int t) {
      return (long long)kbase + (t < see.keep ? t : t < see.keep + see.blocks ? run.keep + t - see.keep
                                                                              : run.keep + run.blocks + see.lo - run.lo + t - see.keep - see.blocks);
    };
    const bf16* q = a.q + (long long)(r0 + x) * a.ldq + (long long)h * DQ;
    float mx = a.sink != nullptr ? a.sink[h] * LOG2E : a.sink_one ? 0.f : -INFINITY, den = a.sink != nullptr || a.sink_one ? 1.f : 0.f;
    float o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int t0 = 0; t0 < count; t0 += 32) {
      const int t = t0 + lane;
      float s = -INFINITY;
      if (t < count) {
        const long long kr = key_row(t);
        s = 0.f;
        for (int d = 0; d < DQ; ++d) {
          const float kv = d < 128 ? s32_value(a.k + kr * a.ldk + kvl * 128 + d, a.k_plane) : s32_value(a.kr + kr * a.ldkr + (d - 128), a.kr_plane);
          s = fmaf(s32_value(q + d, a.q_plane), kv, s);
        }
        s = score32(a, s * (float)(1.0 - CUT_SCORE));      // nothing is cut off here
      }
      float top = s;
      for (int m = 16; m > 0; m >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, m));
      const float mn = fmaxf(mx, top), ref = mn == -INFINITY ? 0.f : mn, corr = exp2f(mx - ref), p = t < count ? exp2f(s - ref) : 0.f;
      float sum = p;
      for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
      den = fmaf(den, corr, sum);
      mx = mn;
      p_s[lane] = p;
      __syncwarp();
      for (int i = 0; i < 4; ++i) o[i] *= corr;
      for (int j = 0; j < 32 && t0 + j < count; ++j) {
        const long long kr = key_row(t0 + j);
        for (int i = 0; i < 4; ++i) o[i] = fmaf(p_s[j], s32_value(a.v + kr * a.ldk + kvl * 128 + lane + 32 * i, a.k_plane), o[i]);
      }
      __syncwarp();
    }
    const bool empty = den == 0.f && a.sink == nullptr && a.zero_empty;
    float f = 1.0f / den;
    if (a.gate != nullptr) f *= 1.0f / (1.0f + expf(-a.gate[(long long)(r0 + x) * a.ldg + h]));
    for (int i = 0; i < 4; ++i) p_s[32 + lane + 32 * i] = empty ? 0.f : o[i] * f;
    __syncwarp();
    for (int i = 0; i < 4; ++i) {
      const long long at = (long long)(r0 + x) * a.ldo + (long long)h * 128 + lane + 32 * i;
      float v = p_s[32 + lane + 32 * i];
      if (a.turn != nullptr) v = turned32(a, r0 + x, lane + 32 * i, v, p_s + 32);
      v = out32(a, r0 + x, h, lane + 32 * i, v);
      if (a.out_fp32) reinterpret_cast<float*>(a.out)[at] = v;
      else reinterpret_cast<bf16*>(a.out)[at] = __float2bfloat16(v);
    }
    __syncwarp();
  }
}

// One CTA a head and 128 rows of a request, 128 keys at a time.
//   warp 0      TMA: the rows' queries once (3 planes), then keys and values through a ring of 16 KB boxes
//   warp 1      MMA: S(i + 1) = Q K^T is issued before P(i) V, so the tensor cores work while the softmax warps have S(i)
//   warps 4-11  softmax, a thread to one row and half of its keys and output channels: P's terms go back to TMEM over S (upper and middle) and
//               beside it (lower), and the two sums of the tile before are added to fp32 sums in registers
// TMEM columns: S of even and odd tiles [0, 128) [128, 256), lower terms of P [256, 320), P V of one tile [384, 512).
// The products of a tile's scores, terms (key, query): (2,0) (1,1) (1,0) (0,2) (0,1) and last (0,0), whose box is brought twice so that nothing small is
// added to a full-size sum.  Tensor time of a tile: 6 (DQ + 128) / 16 MMAs of 64 clocks; what bounds it is the chain of scores, softmax (about 800
// instructions a warp and tile, two warps a scheduler) and outputs: tensor pipe 45 % active, the softmax warps mostly waiting for TMEM.
// Measured (B200, 4096 tokens, 16 heads): latent attention over 1024 keys 240 us (fp32 multiply-adds over the latents themselves 6,125), window attention 205 to
// 280 (window_attn_mma_kernel on mma.sync 760 to 930).  The MMA thread's spills and the softmax in expf with truncated terms had cost 100 us.
// Error against 64 bits, 1e-7 of the output (window_attn_mma_kernel; this kernel before its queries carried the scale and what cutting off takes; now): 4096 rows
// of 16 heads, window 1024, 4 kept 1.70, 1.97, 1.45; capped at 30, blocks of 64 1.79, 1.99, 1.56; 500 rows of 32 heads 1.33, 1.65, 1.23; 640 rows after 3000
// 2.11, 2.39, 1.72; 200 rows of 64 heads 1.23, 1.48, 1.16; scores of deviation 3 over values of mean 1, beyond what layers make of normed queries and keys,
// 1.94, 2.68, 2.15.  Latent attention, 4096 rows over 1024 keys (fp32 multiply-adds over the latents; before; now): 3.92, 1.72, 1.36.
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
  uint64_t* pv_done = p_full + 1;         // [2]: the first sum of a tile, the second
  uint64_t* o_taken = pv_done + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(o_taken + 1);
  uint32_t* odd_s = tmem_ptr + 1;         // outputs that are not finite
  float* top_s = reinterpret_cast<float*>(smem + S::TOP_OFF);      // [2][2][128]
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // this tile's request and rows, and where its keys lie; later tiles see more keys: they start first
  int tile = (int)gridDim.y - 1 - (int)blockIdx.y, s = 0, kbase = 0, r0 = 0, nrows = 0, pos0 = 0;
  Run32 run = {};
  for (; s < a.seqs.n; ++s) {
    const int first = a.seqs.row0[s], len = a.seqs.row0[s + 1] - first, p0 = a.seqs.pos0[s], tiles = (len + 127) >> 7;
    run = run32(a.seqs, p0, len);
    if (tile < tiles) {
      r0 = first + tile * 128;
      nrows = min(128, len - tile * 128);
      pos0 = p0 + tile * 128;
      break;
    }
    tile -= tiles;
    kbase += run.count;
  }
  if (s >= a.seqs.n) return;
  const int h = a.head0 + blockIdx.x, kvl = blockIdx.x / a.ratio;
  // the tile walks two pieces of the request's run: kept tokens and blocks up to `end_a`, tokens from `at_b` to `end_b`
  const Seen32 see0 = seen32(a.seqs, pos0), see1 = seen32(a.seqs, pos0 + nrows - 1);
  const int tok = run.keep + run.blocks - run.lo;      // a token's place in the run, less its position
  const int end_a = see1.blocks > 0 ? run.keep + see1.blocks : see1.keep, at_b = tok + see0.lo, end_b = tok + pos0 + nrows;
  const int n_a = (end_a + 127) >> 7, n = n_a + ((end_b - at_b + 127) >> 7);
  auto key_at = [&](int i) { return i < n_a ? i * 128 : at_b + (i - n_a) * 128; };
  auto sixteens = [&](int i) { return min(8, ((i < n_a ? end_a : end_b) - key_at(i) + 15) >> 4); };      // groups of 16 keys that hold any

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
    mbar_init(pv_done + 1, 1);
    mbar_init(o_taken, 256);
    fence_barrier_init();
    *odd_s = 0;
  }
  if (warp == 0) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = *tmem_ptr;
  if (warp < 4) {
    s32_fewer_regs<S32_FEW>();
    if (warp == 0) {
      if (lane == 0) {
        Ring32<SLOTS> ring;
        int filled = 0;
        auto slot = [&]() {
          const int st = ring.at;
          if (filled == SLOTS) s32_wait(empty + st, ring.round ^ 1);
          else ++filled;
          mbar_arrive_expect_tx(full + st, S32_BOX);
          ring.next();
          return st;
        };
        auto keys = [&](int i) {
          const int at = kbase + key_at(i);
#pragma unroll 1
          for (int g = 0; g < 4; ++g) {
            const int pl = g == 0 ? 2 : g == 1 ? 1 : 0;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              const int st = slot();
              if (b < 2) tma_load_3d(smem + S::RING + st * S32_BOX, &tmK, full + st, kvl * 128 + b * 64, at, pl);
              else tma_load_3d(smem + S::RING + st * S32_BOX, &tmKr, full + st, 0, at, pl);
            }
          }
        };
        auto values = [&](int i) {      // as the products take them: see `outputs`
          const int at = kbase + key_at(i), halves = sixteens(i) > 4 ? 2 : 1;
#pragma unroll 1
          for (int g = 0; g < 8; ++g) {
            const int pl = g == 1 || g == 2 ? 2 : g == 3 || g == 4 ? 1 : 0, kh = g == 7 || (g > 0 && (g & 1) == 0);
            if (kh >= halves) continue;
            const int st = slot();
            tma_load_3d(smem + S::RING + st * S32_BOX, &tmV, full + st, kvl * 128, at + kh * 64, pl);
            tma_load_3d(smem + S::RING + st * S32_BOX + S32_BOX / 2, &tmV, full + st, kvl * 128 + 64, at + kh * 64, pl);
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
      {
        const bool issue = elect_one();
        constexpr uint32_t idesc_o = umma_idesc_bf16(128, 128, 0, 1);
        const uint32_t q_at = smem_u32(smem) >> 4, ring_at = smem_u32(smem + S::RING) >> 4;
        constexpr uint32_t BOX = S32_BOX >> 4;
        Ring32<SLOTS> ring;
        auto box = [&]() {
          s32_wait_warp(full + ring.at, ring.round);
          tc_fence_after();
          return ring_at + ring.at * BOX;
        };
        auto done = [&]() {
          if (issue) umma_commit(empty + ring.at);
          ring.next();
        };
        // a box of keys and the terms of the queries that it meets
        auto scores = [&](int i) {
          const uint32_t d = tm + (uint32_t)(i & 1) * 128, idesc_s = umma_idesc_bf16(128, 16 * sixteens(i), 0, 0);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              const uint32_t k_at = box();
              if (issue) {
#pragma unroll
                for (int q = g == 1 ? 1 : g == 2 ? 2 : 0; q >= (g == 2 ? 1 : 0); --q)
#pragma unroll
                  for (int ks = 0; ks < 4; ++ks)
                    umma_ss(d, s32_desc(q_at + (q * NB + b) * BOX + ks * 2), s32_desc(k_at + ks * 2), idesc_s, g + b + ks > 0 ? 1u : 0u);
              }
              done();
            }
          }
          if (issue) umma_commit(s_full + (i & 1));
        };
        // the output of a tile as two sums, one after the other in the same columns: full-size products of the first 64 keys; then all smaller
        // ones and after them the full-size ones of the other keys.  One chain of eight full-size steps lost 1.4e-7 of the output.
        auto outputs = [&](int i) {
          const uint32_t p = tm + (uint32_t)(i & 1) * 128;
          const int steps = sixteens(i);
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const int kh = g == 7 || (g > 0 && (g & 1) == 0);
            if (kh * 4 < steps) {
              const uint32_t v_at = box() | (S32_BOX / 2 >> 4) << 16;
              if (issue) {
#pragma unroll
                for (int q = g == 3 || g == 4 ? 1 : g == 5 || g == 6 ? 2 : 0; q >= (g == 5 || g == 6 ? 1 : 0); --q)
#pragma unroll
                  for (int k4 = 0; k4 < 4; ++k4) {
                    const int ks = kh * 4 + k4;      // 16 keys: upper and middle terms lie side by side, 32 keys at a time
                    if (ks < steps)
                      umma_ts(tm + TM_O, q == 2 ? tm + TM_X + ks * 8 : p + (ks >> 1) * 32 + (ks & 1) * 8 + q * 16, s32_desc(v_at + k4 * 128), idesc_o,
                              g > 1 || k4 > 0 ? 1u : 0u);
                  }
              }
              done();
            }
            if (g == 0) {
              if (issue) umma_commit(pv_done);
              s32_wait_warp(o_taken, i & 1);
              tc_fence_after();
            }
          }
          if (issue) umma_commit(pv_done + 1);
        };
        s32_wait_warp(q_full, 0);
        scores(0);
        for (int i = 0; i < n; ++i) {
          if (i + 1 < n) scores(i + 1);
          s32_wait_warp(p_full, i & 1);
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
    const Seen32 see = seen32(a.seqs, pos0 + x);
    const int my_keep = mine ? see.keep : 0, my_blocks = mine ? run.keep + see.blocks : 0, my_lo = tok + see.lo, my_hi = mine ? tok + pos0 + x : -1;
    const int all_lo = tok + see1.lo, all_hi = tok + pos0;      // tokens that every row sees
    const float cap = a.cap > 0.f ? a.cap : 1.f;
    float mx = a.sink != nullptr ? a.sink[h] * LOG2E : a.sink_one ? 0.f : -INFINITY, den = (a.sink != nullptr || a.sink_one) && hh == 0 ? 1.f : 0.f;
    float corr_before = 0.f;
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
    auto take_first = [&](int i) {
      s32_wait(pv_done, (uint32_t)i & 1);
      tc_fence_after();
      add_outputs(corr_before);
      tc_fence_before();
      mbar_arrive(o_taken);
    };
    for (int i = 0; i < n; ++i) {
      uint32_t v[64];
      s32_wait(s_full + (i & 1), (uint32_t)(i >> 1) & 1);
      tc_fence_after();
      const uint32_t s_addr = lane_addr + (uint32_t)(i & 1) * 128 + hh * 64;
      LP_TMEM_LD_32((v + 0), s_addr);
      LP_TMEM_LD_32((v + 32), s_addr + 32);
      tmem_wait_ld();
      const int k0 = key_at(i) + hh * 64;
      if (a.cap > 0.f) {
#pragma unroll
        for (int j = 0; j < 64; ++j) v[j] = __float_as_uint(tanhf(__uint_as_float(v[j])));
      }
      if (i < n_a) {      // kept tokens, then blocks
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const int idx = k0 + j;
          if (idx >= end_a || (idx < run.keep ? idx >= my_keep : idx >= my_blocks)) v[j] = 0xff800000u;      // -inf
        }
      } else if (nrows < 128 || k0 < all_lo || k0 + 63 > all_hi) {
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (k0 + j < my_lo || k0 + j > my_hi) v[j] = 0xff800000u;
      }
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 64; ++j) top = fmaxf(top, __uint_as_float(v[j]));
      top *= cap;
      float* ts = top_s + (i & 1) * 256;
      ts[hh * 128 + x] = top;
      s32_bar(1 + lg, 64);
      if (i > 0) take_first(i - 1);
      const float mn = fmaxf(mx, fmaxf(top, ts[(hh ^ 1) * 128 + x])), ref = mn == -INFINITY ? 0.f : mn;      // -inf: nothing seen so far
      const float corr = s32_ex2(mx - ref);
      float sums[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 64; j += 2) {
        const float p0 = s32_ex2(fmaf(__uint_as_float(v[j]), cap, -ref)), p1 = s32_ex2(fmaf(__uint_as_float(v[j + 1]), cap, -ref));      // 2^-inf = 0: not seen
        v[j] = __float_as_uint(p0);
        v[j + 1] = __float_as_uint(p1);
        sums[j & 2] += p0;
        sums[(j & 2) + 1] += p1;
      }
      den = fmaf(den, corr, (sums[0] + sums[1]) + (sums[2] + sums[3]));
      mx = mn;
      if (i > 0) {      // all of P V of the tile before has run: its lower terms of P are no longer read
        s32_wait(pv_done + 1, (uint32_t)(i - 1) & 1);
        tc_fence_after();
        add_outputs(1.f);
      }
      corr_before = corr;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[16], mid[16], lo[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) s32_weight_terms(__uint_as_float(v[c * 32 + 2 * j]), __uint_as_float(v[c * 32 + 2 * j + 1]), hi[j], mid[j], lo[j]);
        LP_TMEM_ST_16(hi, s_addr + c * 32);
        LP_TMEM_ST_16(mid, s_addr + c * 32 + 16);
        LP_TMEM_ST_16(lo, lane_addr + TM_X + hh * 32 + c * 16);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full);
    }
    take_first(n - 1);
    s32_wait(pv_done + 1, (uint32_t)(n - 1) & 1);
    tc_fence_after();
    add_outputs(1.f);
    float* ds = top_s + (n & 1) * 256;
    ds[hh * 128 + x] = den;
    s32_bar(1 + lg, 64);
    den += ds[(hh ^ 1) * 128 + x];
    if (mine) {
      bool odd = false;
      const bool empty = den == 0.f && a.sink == nullptr && a.zero_empty;
      Factor32 f = {empty ? 0.f : 1.0f / den, 0.f};
      if (!empty) f.lo = fmaf(fmaf(-f.hi, den, 1.f), f.hi, den > 1.f ? (float)CUT_OUT * f.hi : 0.f);      // (one key: its value as it is)
      if (a.gate != nullptr) {
        const float open = 1.0f / (1.0f + expf(-a.gate[(long long)(r0 + x) * a.ldg + h]));
        f.hi *= open;
        f.lo *= open;
      }
#pragma unroll
      for (int c = 0; c < 64; ++c) {
        odd |= !(fabsf(o[c]) <= 3.402823466e38f);
        o[c] = fmaf(o[c], f.hi, o[c] * f.lo);
      }
      if (odd) *odd_s = 1;
    }
    if (a.turn != nullptr) {      // the two threads of a row exchange their channels where the queries were: all products have run
      float* os = reinterpret_cast<float*>(smem) + x * 129;
#pragma unroll
      for (int c = 0; c < 64; ++c) os[hh * 64 + c] = o[c];
      s32_bar(1 + lg, 64);
      if (mine) {
#pragma unroll
        for (int c = 0; c < 64; ++c) o[c] = turned32(a, r0 + x, hh * 64 + c, o[c], os);
      }
    }
    if (mine) {
      const long long at = (long long)(r0 + x) * a.ldo + (long long)h * 128 + hh * 64;
#pragma unroll
      for (int c = 0; c < 64; ++c) o[c] *= a.out_scale;
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
    // an infinity or a NaN among the keys or values: weights of zero times it are NaN in every row of the product, seen or not.  All products have run.
    // The other warps have given up the registers that this may want: they stay out.
    s32_bar(5, A32_THREADS - 128);
    if (*odd_s != 0) attn32_plain<NR>(a, r0, nrows, pos0, kbase, run, h, kvl, reinterpret_cast<float*>(smem), warp - 4, A32_THREADS / 32 - 4);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tm, 512);
  }
}

}  // namespace lp

#ifndef LP_EMULATE
using namespace lp;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static int split_rows(const float* src, long long ld, int M, int K, void* planes, long long ldp, long long plane, const Factor32* factor, void* stream_) {
  LP_REQUIRE(src != nullptr && planes != nullptr, "lp_split_rows: null operand");
  LP_REQUIRE(K % 8 == 0 && ld % 4 == 0 && ldp % 8 == 0 && plane % 8 == 0 && aligned16(src) && aligned16(planes), "lp_split_rows: 16-byte rows of whole eights");
  if (M <= 0 || K <= 0) return 0;
  const long long pieces = (long long)M * (K >> 3);
  const unsigned grid = (unsigned)((pieces + 255) / 256);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  bf16* dst = reinterpret_cast<bf16*>(planes);
  if (factor != nullptr) split_rows_kernel<true><<<grid, 256, 0, stream>>>(src, ld, M, K, dst, ldp, plane, *factor);
  else split_rows_kernel<false><<<grid, 256, 0, stream>>>(src, ld, M, K, dst, ldp, plane, Factor32{});
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}
extern "C" int lp_split_rows(const float* src, long long ld, int M, int K, void* planes, long long ldp, long long plane, void* stream) {
  return split_rows(src, ld, M, K, planes, ldp, plane, nullptr, stream);
}

extern "C" int lp_gather_rows(const void* src, long long ld, int src_fp32, const int* row_of, int rows, int K, void* dst, long long plane, void* stream_) {
  LP_REQUIRE(src != nullptr && row_of != nullptr && dst != nullptr, "lp_gather_rows: null operand");
  LP_REQUIRE(K % 8 == 0 && ld % (src_fp32 ? 4 : 8) == 0 && plane % 8 == 0 && aligned16(src) && aligned16(dst), "lp_gather_rows: 16-byte rows of whole eights");
  if (rows <= 0 || K <= 0) return 0;
  const unsigned grid = (unsigned)(((long long)rows * (K >> 3) + 255) / 256);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (src_fp32) gather_rows_kernel<true><<<grid, 256, 0, stream>>>(src, ld, row_of, rows, K, reinterpret_cast<bf16*>(dst), plane);
  else gather_rows_kernel<false><<<grid, 256, 0, stream>>>(src, ld, row_of, rows, K, reinterpret_cast<bf16*>(dst), plane);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

template <int BN, int PLANES, bool GATED>
static int launch_gemm32(Gemm32Args a, int groups, long long w_group, cudaStream_t stream) {
  using S = Gemm32Smem<BN, PLANES>;
  static bool configured = false;
  auto kern = gemm32_kernel<BN, PLANES, GATED>;
  if (!configured) {
    LP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    configured = true;
  }
  constexpr int cols = GATED ? BN / 2 : BN;
  CUtensorMap ta, tw;
  if (int rc = make_tmap_bf16_3d(&ta, a.A, a.K, a.M, PLANES, a.lda, PLANES == 1 ? a.lda * a.M : a.a_plane, 64, 128, 1)) return rc;
  if (int rc = make_tmap_bf16_3d(&tw, a.W, a.K, a.N, groups, a.ldw, w_group, 64, GATED ? 64 : BN, 1)) return rc;
  a.n_tiles_m = (a.M + 127) / 128;
  a.n_tiles_n = ((GATED ? a.N / 2 : a.N) + cols - 1) / cols;
  a.w_group = w_group;
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
  return wide < narrow ? launch_gemm32<256, 3, false>(a, 1, a.ldw * a.N, stream) : launch_gemm32<128, 3, false>(a, 1, a.ldw * a.N, stream);
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

extern "C" int lp_linear_split(const float* A, long long lda, const void* W, long long ldw, void* C, long long ldc, int out, int M, int N, int K,
                               const float* bias, void* terms, void* stream) {
  if (int rc = lp_split_rows(A, lda, M, K, terms, K, (long long)M * K, stream)) return rc;
  return lp_gemm_split(terms, K, (long long)M * K, W, ldw, C, ldc, 0, out, M, N, K, bias, stream);
}

template <int NR>
static int launch_attn32(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tr, const CUtensorMap& tv, const Attn32Args& a, int heads,
                         int n_tiles, cudaStream_t stream) {
  using S = Attn32Smem<NR>;
  auto kern = attn32_kernel<NR>;
  static bool configured = false;
  if (!configured) {
    LP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    configured = true;
  }
  kern<<<dim3(heads, n_tiles), A32_THREADS, S::TOTAL, stream>>>(tq, tk, tr, tv, a);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int lp_gemm_grouped(const void* A, long long lda, long long a_plane, const void* W, long long ldw, long long w_group, int groups,
                               const int* tile_group, int n_tiles, int gated, const float* row_scale, void* C, long long ldc, long long c_plane, int out, int N,
                               int K, void* stream_) {
  LP_REQUIRE(A != nullptr && W != nullptr && C != nullptr && tile_group != nullptr, "lp_gemm_grouped: null operand");
  LP_REQUIRE(out >= G32_OUT_BF16 && out <= G32_OUT_PLANES, "lp_gemm_grouped: unknown output form %d", out);
  LP_REQUIRE(K >= 8 && K % 8 == 0 && N % 16 == 0 && groups > 0 && lda % 8 == 0 && a_plane % 8 == 0 && ldw % 8 == 0 && w_group % 8 == 0 &&
                 ldc % (out == G32_OUT_F32 ? 4 : 8) == 0 && c_plane % 8 == 0 && aligned16(A) && aligned16(W) && aligned16(C),
             "lp_gemm_grouped: 16-byte rows of whole eights");
  LP_REQUIRE(gated || row_scale == nullptr, "lp_gemm_grouped: a row scale comes with a gated unit");
  if (n_tiles <= 0 || N <= 0) return 0;
  Gemm32Args a = {};
  a.M = n_tiles * 128; a.N = N; a.K = K;
  a.C = C; a.ldc = ldc; a.c_plane = c_plane; a.out = out;
  a.A = reinterpret_cast<const bf16*>(A); a.lda = lda; a.a_plane = a_plane;
  a.W = reinterpret_cast<const bf16*>(W); a.ldw = ldw;
  a.tile_group = tile_group; a.row_scale = row_scale;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (a_plane > 0) return gated ? launch_gemm32<256, 3, true>(a, groups, w_group, stream) : launch_gemm32<256, 3, false>(a, groups, w_group, stream);
  return gated ? launch_gemm32<256, 1, true>(a, groups, w_group, stream) : launch_gemm32<256, 1, false>(a, groups, w_group, stream);
}

// ---- latent attention, keys and values expanded
constexpr size_t LX_GROUP_BYTES = (size_t)512 << 20;      // heads whose expanded keys and values are held at a time
static int lx_group(int heads, int n_keys) {
  const long long one = (long long)n_keys * 256 * 6;
  const long long g = (long long)LX_GROUP_BYTES / (one > 0 ? one : 1);
  return g < 1 ? 1 : g < heads ? (int)g : heads;
}
static size_t lx_round(size_t b) { return (b + 255) & ~(size_t)255; }

// tiles of 128 rows and key rows of a step, from the requests' tables as they lie on the host
static void count32(const Seqs32& q, int* n_tiles, int* n_keys) {
  int tiles = 0, keys = 0;
  for (int s = 0; s < q.n; ++s) {
    const int len = q.row0[s + 1] - q.row0[s];
    tiles += (len + 127) / 128;
    keys += run32(q, q.pos0[s], len).count;
  }
  *n_tiles = tiles;
  *n_keys = keys;
}
// Whether a step's latents are expected to be attended sooner with every head's keys and values expanded (1) or as they are (0).  Expanding pays 1.4 ns (rank 128)
// to 2 ns (512) for every visible key and head, however few rows see it, and then a tile's chain of 55 ns a key; lp_latent_attend_tiles about 80 GFMA/s a CTA of
// 64 (row, head) pairs of a chunk over keys of 2 rank + 64, one CTA an SM, and its two head products.  The figures (us) are fitted to 366 steps of 4 to 32 heads over
// latents of 128 to 512 (1 to 128 requests of 1 to 4096 rows behind 0 to 64,000 tokens, windows of 100 to 2048 keys and none, both precisions), of which this picks the
// slower way 7 times, by 7 to 23 %.  Some of them (tiles and expanded), 16 heads of rank 512: one request of 17 rows 123, 99, behind 4000 tokens 3,377, 382; a prompt of
// 20 rows beside 7 running requests of 2000 tokens 1,731, 562, beside 31 of 2000 1,744, 2,768, of 8000 6,670, 14,829; of 2000 rows beside 31 of 2000 4,526, 2,891;
// 64 requests of 4 rows behind 4000 tokens 3,422, 11,767, of 48 rows 20,478, 11,934.
extern "C" int lp_latent_route(const int* seq_row0, const int* seq_pos0, int n_seqs, int heads, int kv_rank, int window, int* n_tiles, int* n_keys) {
  const Seqs32 q = {n_seqs, window, seq_row0, seq_pos0, 0, 0, 0};
  count32(q, n_tiles, n_keys);
  const int sms = sm_count();
  double ctas = 0, cta_keys = 0, longest = 0, tile_keys = 0, longest_tile = 0;
  for (int s = 0; s < n_seqs; ++s) {
    const double pos0 = seq_pos0[s];
    const int len = seq_row0[s + 1] - seq_row0[s];
    auto seen = [&](int block, double& last, double& mean) {      // keys of the last and of the average `block` rows
      const int few = len < block ? len : block;
      last = pos0 + len;
      mean = pos0 + (len + few) / 2.0;
      if (window > 0 && last > window + few - 1) last = window + few - 1;
      if (window > 0 && mean > window + few - 1) mean = window + few - 1;
    };
    double last, mean;
    seen(128, last, mean);
    tile_keys += (len + 127) / 128 * mean;
    longest_tile = last > longest_tile ? last : longest_tile;
    seen(LP_RETENTION_CHUNK, last, mean);
    const double c = (double)(len / LP_RETENTION_CHUNK) * ((LP_RETENTION_CHUNK * heads + 63) / 64) + (len % LP_RETENTION_CHUNK * heads + 63) / 64;
    ctas += c;
    cta_keys += c * mean;
    longest = last > longest ? last : longest;
  }
  if (ctas == 0) return 0;
  const double waves = cta_keys / ctas * (double)(((long long)ctas + sms - 1) / sms);
  const double tiles_us = 90 + 64.0 * (2 * kv_rank + 64) * 1.21e-5 * (waves > longest ? waves : longest) + (double)seq_row0[n_seqs] * heads * kv_rank * 2.2e-5;
  const int groups = (heads + lx_group(heads, *n_keys) - 1) / lx_group(heads, *n_keys);      // each walks a request's keys anew
  const double chain = groups * (17 + 0.055 * longest_tile), all = (17.0 * *n_tiles + 0.055 * tile_keys) * heads / sms, a_key = 0.0022 - 0.1 / kv_rank;
  const double expanded_us = 60 + (double)*n_keys * heads * (a_key > 0.0008 ? a_key : 0.0008) + (chain > all ? chain : all);
  return expanded_us <= tiles_us;
}

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
  float cap;
  const Factor32 factor = scale32(d->scale, 0.f, cap);
  if (int rc = split_rows(d->q, d->ldq, R, H * 192, q_p, (long long)H * 192, q_plane, &factor, stream_)) return rc;
  const Seqs32 seqs = {n_seqs, d->window, seq_row0, seq_pos0, 0, 0, 0};
  const long long pieces = (long long)n_keys * (width >> 3);
  gather_keys_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, stream>>>(seqs, n_keys, d->cache, d->page_size, d->page_table, d->max_pages, nullptr, nullptr, 0,
                                                                            width, c_p, c_plane);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
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
    a.seqs = seqs; a.head0 = h0; a.ratio = 1;
    a.out_scale = 1.0f; a.sink = d->sink; a.gate = d->gate; a.ldg = d->ldg;
    a.out_gate = out_gate; a.ldog = ldog;
    a.out = out; a.ldo = ldo; a.out_fp32 = out_fp32;
    a.q = q_p; a.ldq = H * 192LL; a.q_plane = q_plane;
    a.k = kv_p; a.v = kv_p + 128 * g; a.ldk = ld; a.k_plane = plane;
    a.kr = c_p + C; a.ldkr = width; a.kr_plane = c_plane;
    if (int rc = launch_attn32<1>(tq, tk, tr, tv, a, g, n_tiles, stream)) return rc;
  }
  return 0;
}

// ---- window attention of prompts
static int window_row(const lp_window_attn_desc* d) { return d->kv_heads * 128 * (d->v_is_k ? 1 : 2); }
extern "C" int lp_window_prompt_count(const lp_window_attn_desc* d, const int* seq_row0, const int* seq_pos0, int n_seqs, int* n_tiles, int* n_keys) {
  LP_REQUIRE(d != nullptr && seq_row0 != nullptr && seq_pos0 != nullptr && n_tiles != nullptr && n_keys != nullptr, "lp_window_prompt_count: null operand");
  count32({n_seqs, d->window, seq_row0, seq_pos0, d->chunk, d->keep_first, d->pool}, n_tiles, n_keys);
  return 0;
}
extern "C" size_t lp_window_prompt_workspace_bytes(int R, int heads, int row_floats, int n_keys) {
  return lx_round((size_t)6 * R * heads * 128) + lx_round((size_t)6 * n_keys * row_floats) + lx_round((size_t)8 * R * 64);
}

extern "C" int lp_window_attn_prompt(const lp_window_attn_desc* d, int R, int n_seqs, const int* seq_row0, const int* seq_pos0, int n_tiles, int n_keys,
                                     void* out, long long ldo, int out_fp32, void* ws, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LP_REQUIRE(d != nullptr && d->qkv != nullptr && d->cache != nullptr && d->page_table != nullptr && seq_row0 != nullptr && seq_pos0 != nullptr &&
                 out != nullptr && ws != nullptr,
             "lp_window_attn_prompt: null operand");
  LP_REQUIRE(d->dim == 128 && d->vdim == 128 && d->heads > 0 && d->kv_heads > 0 && d->heads % d->kv_heads == 0,
             "lp_window_attn_prompt: heads of 128 only, not %d and %d", d->dim, d->vdim);
  LP_REQUIRE(d->dist_amp == nullptr && d->talk == nullptr, "lp_window_attn_prompt: no distance bias, no mixed heads");
  LP_REQUIRE(d->v_inv_freq == nullptr || (d->v_rot_dims >= 0 && d->v_rot_dims <= 128 && d->v_rot_dims % 2 == 0), "lp_window_attn_prompt: v_rot_dims=%d",
             d->v_rot_dims);
  LP_REQUIRE(d->pool >= 0 && (d->pool == 0 || (d->pooled != nullptr && d->pooled_table != nullptr)) && d->keep_first >= 0 && d->chunk >= 0 && d->page_size > 0,
             "lp_window_attn_prompt: bad visibility");
  LP_REQUIRE(d->ld % 4 == 0 && d->q_off % 4 == 0 && ldo % (out_fp32 ? 4 : 8) == 0 && aligned16(d->qkv) && aligned16(d->cache) &&
                 (d->pool == 0 || aligned16(d->pooled)) && aligned16(out) && aligned16(ws),
             "lp_window_attn_prompt: 16-byte rows");
  const int H = d->heads, row = window_row(d);
  LP_REQUIRE(ws_bytes >= lp_window_prompt_workspace_bytes(R, H, row, n_keys), "lp_window_attn_prompt: workspace");
  if (R <= 0 || n_seqs <= 0 || n_tiles <= 0 || n_keys <= 0) return 0;
  LP_REQUIRE(n_tiles <= 65535, "lp_window_attn_prompt: %d tiles", n_tiles);
  bf16* q_p = reinterpret_cast<bf16*>(ws);
  bf16* kv_p = q_p + lx_round((size_t)6 * R * H * 128) / 2;
  const long long q_plane = (long long)R * H * 128, plane = (long long)n_keys * row;
  float cap;
  const Factor32 factor = scale32(d->scale, d->softcap, cap);
  if (int rc = split_rows(d->qkv + d->q_off, d->ld, R, H * 128, q_p, (long long)H * 128, q_plane, &factor, stream_)) return rc;
  const Seqs32 seqs = {n_seqs, d->window, seq_row0, seq_pos0, d->chunk, d->keep_first, d->pool};
  const long long pieces = (long long)n_keys * (row >> 3);
  gather_keys_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, stream>>>(seqs, n_keys, d->cache, d->page_size, d->page_table, d->max_pages, d->pooled,
                                                                          d->pooled_table, d->max_pooled_pages, row, kv_p, plane);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  const bf16* v_p = kv_p + (d->v_is_k ? 0 : d->kv_heads * 128);
  CUtensorMap tq, tk, tv;
  if (int rc = make_tmap_bf16_3d(&tq, q_p, (uint64_t)H * 128, R, 3, (uint64_t)H * 128, q_plane, 64, 128, 1)) return rc;
  if (int rc = make_tmap_bf16_3d(&tk, kv_p, (uint64_t)d->kv_heads * 128, n_keys, 3, row, plane, 64, 128, 1)) return rc;
  if (int rc = make_tmap_bf16_3d(&tv, v_p, (uint64_t)d->kv_heads * 128, n_keys, 3, row, plane, 64, 64, 1)) return rc;
  Attn32Args a = {};
  a.seqs = seqs; a.ratio = H / d->kv_heads;
  a.cap = cap; a.sink_one = d->sink != 0; a.zero_empty = 1;
  a.out_gate = d->gate; a.ldog = d->ldg; a.out_scale = d->out_scale == 0.f ? 1.f : d->out_scale;
  a.out = out; a.ldo = ldo; a.out_fp32 = out_fp32;
  a.q = q_p; a.ldq = H * 128LL; a.q_plane = q_plane;
  a.k = kv_p; a.v = v_p; a.ldk = row; a.k_plane = plane;
  const int half = d->v_inv_freq != nullptr ? d->v_rot_dims / 2 : 0;
  if (half > 0) {
    float2* table = reinterpret_cast<float2*>(reinterpret_cast<char*>(ws) + lx_round((size_t)6 * R * H * 128) + lx_round((size_t)6 * n_keys * row));
    turn_table_kernel<<<(unsigned)(((long long)R * half + 255) / 256), 256, 0, stream>>>(seqs, R, d->v_inv_freq, half, table);
    note_launch();
    LP_CHECK_CUDA(cudaGetLastError());
    a.turn = table; a.turn_half = half; a.turn_interleaved = d->v_rot_layout == LP_ROT_INTERLEAVED;
  }
  return launch_attn32<0>(tq, tk, tk, tv, a, H, n_tiles, stream);
}
#endif  // !LP_EMULATE

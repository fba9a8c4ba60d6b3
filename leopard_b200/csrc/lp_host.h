// leopard_b200 — host-side helpers shared by the .cu translation units (not part of the public C ABI).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include "lp_pdl.cuh"

namespace lp {

// error plumbing: every entry point returns 0 or a negative lp_status and records a message
void set_error(const char* fmt, ...);
const char* get_error();

#define LP_CHECK_CUDA(expr)                                                                   \
  do {                                                                                        \
    cudaError_t _e = (expr);                                                                  \
    if (_e != cudaSuccess) {                                                                  \
      lp::set_error("%s:%d: %s -> %s", __FILE__, __LINE__, #expr, cudaGetErrorString(_e));    \
      return -2; /* LP_ERR_CUDA */                                                            \
    }                                                                                         \
  } while (0)

#define LP_REQUIRE(cond, ...)           \
  do {                                  \
    if (!(cond)) {                      \
      lp::set_error(__VA_ARGS__);       \
      return -1; /* LP_ERR_ARG */       \
    }                                   \
  } while (0)

int sm_count();

#ifdef __CUDACC__
// two fp32 multiply-adds (products) in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)),
        "l"(reinterpret_cast<const unsigned long long&>(c)));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
  return d;
}
// 16 bytes that this kernel reads once (weights): past the first-level cache, through the read-only path
__device__ __forceinline__ uint4 ldg_once(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// warp-wide 16 x 8 x 16 product of bf16 operands, fp32 sums: d[16, 8] += a[16, 16] b[16, 8].  Lane (g, t) = (lane / 4, lane % 4) brings
// a rows g, g + 8 at columns 2t, 2t + 1 (a0, a1) and 8 + 2t, 9 + 2t (a2, a3), b column g at the same rows (b0, b1), and holds
// d[g, 2t], d[g, 2t + 1], d[g + 8, 2t], d[g + 8, 2t + 1].
__device__ __forceinline__ void mma_bf16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same from zero sums: d = a b
__device__ __forceinline__ void mma_bf16_first(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// fp32 values as three bf16 terms, rounded to nearest each (8 + 8 + 8 bits: what is left is below 2^-26 of the value), packed in pairs
__device__ __forceinline__ void cut3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
  hi = *reinterpret_cast<const uint32_t*>(&p);
  x -= __uint_as_float(hi << 16);
  y -= __uint_as_float(hi & 0xffff0000u);
  p = __floats2bfloat162_rn(x, y);
  mid = *reinterpret_cast<const uint32_t*>(&p);
  x -= __uint_as_float(mid << 16);
  y -= __uint_as_float(mid & 0xffff0000u);
  p = __floats2bfloat162_rn(x, y);
  lo = *reinterpret_cast<const uint32_t*>(&p);
}
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.402823466e38f); }
#endif

// prefill kernels are launched with the programmatic-dependent-launch attribute when this is on (lp_set_prefill_pdl):
// every such kernel calls griddepcontrol.wait before its first dependent global access
bool prefill_pdl();

// kernel launch with optional cluster dimension and optional programmatic dependent launch
template <typename... KArgs, typename... Args>
inline cudaError_t launch_ex(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster_x,
                             bool pdl, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster_x > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// The next kernel of a step: where it is small (decoding), its CTAs may be placed while the kernel before it still drains, when that one has asked for it; it
// waits (pdl_wait) before it touches memory.  Pointers to what earlier kernels wrote are not __restrict__ there: a read-only load could be moved
// before the wait.  Kernels of many CTAs gain nothing (prompts of 4,096 rows: 0.5 % slower with all of them launched so).  For short kernels only: CTAs that are placed early lie
// on the SMs that the launch before leaves empty, where long ones then take longer (attention below; retention's decode step, MinGRU's prompts and the router are launched plainly).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_next(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  return launch_ex(kern, grid, block, smem, stream, 1, (long long)grid.x * grid.y * grid.z <= 4LL * sm_count(), args...);
}

// Attention of a step over the past, `work` = rows x heads x keys at most: where it runs for long, CTAs that were placed beside the launch before, on the SMs that this one left empty,
// make it longer (us a step, early and not: 32 requests of 900 tokens, window 512, 8 heads 287, 275; 48 of 1,400, 8 heads of latents 287, 276, now and then 335; 8 of 1,500, window
// 1024, 16 heads 198, 188; one of 3,000, window 2048, 32 heads 304, 297; but one of 530 283, 284.5).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_attention(long long work, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  return work < 50000 ? launch_next(kern, grid, block, smem, stream, args...) : launch_ex(kern, grid, block, smem, stream, 1, false, args...);
}

// launch accounting + optional per-launch CUDA-event timing (off by default; see lp_profile_* in the public header)
void note_launch(int n = 1);
struct ProfScope {
  int idx;
  cudaStream_t stream;
  ProfScope(int kind, int a, int b, int c, cudaStream_t s);
  ~ProfScope();
};

// RoPE in place on the q|k heads of x [S, ld] fused with the KV-cache append of the same rows (lp_elem.cu)
int rope_kv_append(void* x, long long ld, int S, int n_q, int n_kv, int head_dim, const float* cos_t, const float* sin_t,
                   void* kc, void* vc, long long ld_cache, cudaStream_t stream);

// attention launch arguments (shared by lp_attn.cu and lp_attn2.cu)
struct AttnArgs {
  int T, B, n_heads, group;   // T = query rows per sequence
  int Tk;                     // key/value rows per sequence (== T for self-attention)
  int q_off, k_off, v_off, hs;
  int dh_out;
  __nv_bfloat16* O;
  long long ldo;
  float scale_log2;
  int pingpong;               // lp_attn2: strict A/B alternation of the softmax warpgroups (turn protocol)
};
int launch_attn2(const CUtensorMap& tm, const AttnArgs& a, int head_dim, int causal, int emu, cudaStream_t stream);
int launch_attn3(const CUtensorMap& tm, const AttnArgs& a, int head_dim, int causal, int emu, cudaStream_t stream);
int launch_attn4(const CUtensorMap& tm, const AttnArgs& a, int head_dim, int causal, int emu, cudaStream_t stream);
// persistent v3 for short non-causal sequences (lp_attn5.cu): the ViT tower's T = 676
bool attn5_eligible(const AttnArgs& a, int head_dim, int causal);
int launch_attn5(const CUtensorMap& tm, const AttnArgs& a, cudaStream_t stream);

// 2-D / 3-D bf16 tensor maps with 128B swizzle (inner box = 64 elements = 128 B), zero OOB fill.
// dims/strides are innermost-first; strides are in ELEMENTS for dims >= 1.
int make_tmap_bf16_2d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t ld_elems,
                      uint32_t box_inner, uint32_t box_outer);
// generic 2-D map: elem_bytes 2 (bf16); swizzle_bytes in {0, 32, 64, 128}; inner box bytes must equal the swizzle span
int make_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t inner, uint64_t outer, uint64_t ld_elems,
                 uint32_t box_inner, uint32_t box_outer, int swizzle_bytes);
int make_tmap_bf16_3d(CUtensorMap* map, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t ld1_elems,
                      uint64_t ld2_elems, uint32_t b0, uint32_t b1, uint32_t b2);
int make_tmap_bf16_4d(CUtensorMap* map, const void* base, const uint64_t* dims, const uint64_t* strides_elems, const uint32_t* box);

}  // namespace lp

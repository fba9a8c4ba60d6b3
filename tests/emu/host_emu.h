// Test infrastructure: the handful of CUDA runtime names a kernel file's HOST code uses, so that whole .cu files (kernels + the
// host function that sequences them) can run on the CPU under cuda_emu.h once the test has rewritten every
// `kernel<<<grid, block, smem, stream>>>(args);` into `emu::launch(dim3(grid), dim3(block), [&] { kernel(args); });`.
#pragma once
#include "cuda_emu.h"

#include <cstdarg>
#include <cstdio>

// asynchronous copies into shared memory complete at once
inline void __pipeline_memcpy_async(void* dst, const void* src, size_t n) { std::memcpy(dst, src, n); }
inline void __pipeline_commit() {}
inline void __pipeline_wait_prior(int) {}

typedef void* cudaStream_t;
typedef int cudaError_t;
constexpr cudaError_t cudaSuccess = 0;
constexpr int cudaFuncAttributeMaxDynamicSharedMemorySize = 8;
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline const char* cudaGetErrorString(cudaError_t) { return "emulated"; }
template <typename F> inline cudaError_t cudaFuncSetAttribute(F, int, int) { return cudaSuccess; }
// cudaLaunchKernelEx (programmatic-dependent / cooperative / cluster launch attributes are accepted and ignored: blocks run one
// after another, so a cooperative kernel that needs a grid-wide barrier cannot run here)
enum cudaLaunchAttributeID { cudaLaunchAttributeProgrammaticStreamSerialization = 1, cudaLaunchAttributeCooperative = 2,
                             cudaLaunchAttributeClusterDimension = 3 };
struct cudaLaunchAttribute {
  cudaLaunchAttributeID id;
  struct { int programmaticStreamSerializationAllowed; int cooperative; struct { unsigned x, y, z; } clusterDim; } val;
};
struct cudaLaunchConfig_t {
  dim3 gridDim, blockDim;
  size_t dynamicSmemBytes = 0;
  cudaStream_t stream = nullptr;
  cudaLaunchAttribute* attrs = nullptr;
  unsigned numAttrs = 0;
};
template <typename... KArgs, typename... Args>
inline cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* cfg, void (*kern)(KArgs...), Args... args) {
  emu::launch(cfg->gridDim, cfg->blockDim, [&] { kern(static_cast<KArgs>(args)...); });
  return cudaSuccess;
}
// streams / graphs / copies as far as host code names them
typedef void* cudaGraph_t;
typedef void* cudaGraphExec_t;
constexpr int cudaStreamNonBlocking = 1, cudaStreamCaptureModeThreadLocal = 1, cudaMemcpyDeviceToDevice = 3;
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, int) { return cudaSuccess; }
inline cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamBeginCapture(cudaStream_t, int) { return 1; }      // graphs are not emulated
inline cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return 1; }
inline cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, int) { return 1; }
inline cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
inline cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
inline cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return 1; }
inline cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
inline unsigned atomicAdd(unsigned* p, unsigned v) { return std::atomic_ref<unsigned>(*p).fetch_add(v); }
inline void __threadfence() {}
inline long long clock64() { return 0; }
inline void __trap() { std::abort(); }
template <typename T> inline T __ldcg(const T* p) { return *p; }
inline float __bfloat162float(__nv_bfloat16 v) { return (float)v; }
inline unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline unsigned __ballot_sync(unsigned mask, bool pred) {
  unsigned r = 0;
  const unsigned t = emu::linear_tid(), w = t >> 5, l = t & 31;
  float* buf = emu::t_ctx->warp_buf.data() + w * 32;
  auto& bar = emu::t_ctx->group(w, mask);
  buf[l] = pred ? 1.f : 0.f;
  bar.arrive_and_wait();
  for (int i = 0; i < 32; ++i) r |= (unsigned)((mask >> i & 1) && buf[i] != 0.f) << i;
  bar.arrive_and_wait();
  return r;
}
inline float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
inline __nv_bfloat16 __ushort_as_bfloat16(unsigned short u) { __nv_bfloat16 r; r.bits = u; return r; }
#define __align__(n) alignas(n)
#define LP_WATCHDOG_CYCLES (1LL << 62)
struct int2 { int x, y; };
inline int2 make_int2(int a, int b) { return {a, b}; }

// fp64 arithmetic without contraction (the test compiles with -ffp-contract=off)
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __ddiv_rn(double a, double b) { return a / b; }

namespace lp {
typedef __nv_bfloat16 bf16;
inline char g_emu_err[512];
inline void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(g_emu_err, sizeof(g_emu_err), fmt, ap);
  va_end(ap);
}
inline void note_launch(int = 1) {}
inline void pdl_wait() {}
inline void pdl_launch_dependents() {}
inline void pdl_launch_next() {}
inline void pdl_launch_next_of_few() {}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_next(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t, cudaStream_t, Args... args) {
  emu::launch(grid, block, [&] { kern(static_cast<KArgs>(args)...); });
  return cudaSuccess;
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_attention(long long, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  return launch_next(kern, grid, block, smem, stream, args...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_ex(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int, int, Args... args) {
  return launch_next(kern, grid, block, smem, stream, args...);
}
inline int g_emu_sms = 4;      // emu_set_sm_count: rules that count CTAs per SM
inline int sm_count() { return g_emu_sms; }
inline float2 fma2(float2 a, float2 b, float2 c) { return {std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)}; }
inline float2 mul2(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }
inline uint4 ldg_once(const void* p) { return *reinterpret_cast<const uint4*>(p); }
// warp-wide 16 x 8 x 16 product: every lane's registers go round the warp, each lane sums its four outputs over k
inline void mma_bf16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  uint32_t all[6][32];
  const uint32_t mine[6] = {a0, a1, a2, a3, b0, b1};
  const unsigned w = emu::linear_tid() >> 5, l = emu::linear_tid() & 31;
  float* buf = emu::t_ctx->warp_buf.data() + w * 32;
  for (int r = 0; r < 6; ++r) {
    std::memcpy(buf + l, &mine[r], 4);
    emu::t_ctx->warp_bar[w]->arrive_and_wait();
    std::memcpy(all[r], buf, 128);
    emu::t_ctx->warp_bar[w]->arrive_and_wait();
  }
  auto half = [](uint32_t v, int hi) { const uint32_t u = hi ? v & 0xffff0000u : v << 16; float f; std::memcpy(&f, &u, 4); return f; };
  const int g = l >> 2, t = l & 3;
  for (int c = 0; c < 4; ++c) {
    const int row = g + (c >> 1) * 8, col = 2 * t + (c & 1);
    for (int k = 0; k < 16; ++k) {
      const int from = (k & 7) >> 1, up = k >> 3;
      d[c] = std::fma(half(all[(row >> 3) + 2 * up][(row & 7) * 4 + from], k & 1), half(all[4 + up][col * 4 + from], k & 1), d[c]);
    }
  }
}
inline void mma_bf16_first(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  d[0] = d[1] = d[2] = d[3] = 0.f;
  mma_bf16(d, a0, a1, a2, a3, b0, b1);
}
inline void cut3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  uint32_t* out[3] = {&hi, &mid, &lo};
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
    *out[i] = (uint32_t)p.x.bits | ((uint32_t)p.y.bits << 16);
    x -= (float)p.x;
    y -= (float)p.y;
  }
}
inline bool not_finite(float v) { return !std::isfinite(v); }
inline uint32_t smem_u32(const void* p) { return (uint32_t)(uintptr_t)p; }
#ifdef EMU_FIBERS
#define __grid_constant__
// mbarriers (an arrival count, bytes that are still to come, a phase) and bulk copies, which complete at once
struct EmuMbar { int16_t pending; uint8_t count, phase; int32_t bytes; };
static_assert(sizeof(EmuMbar) == sizeof(uint64_t));
inline EmuMbar& emu_mbar(uint64_t* b) { return *reinterpret_cast<EmuMbar*>(b); }
inline void emu_mbar_turn(EmuMbar& m) {
  ++emu::g_sched->progress;
  if (m.pending < 0) { std::fprintf(stderr, "emu: mbarrier over-arrival\n"); std::abort(); }
  if (m.pending > 0 || m.bytes != 0) return;
  m.pending = m.count;
  m.phase ^= 1;
}
inline void mbar_init(uint64_t* b, uint32_t count) { emu_mbar(b) = {(int16_t)count, (uint8_t)count, 0, 0}; }
inline void fence_barrier_init() {}
inline void mbar_arrive(uint64_t* b) { --emu_mbar(b).pending; emu_mbar_turn(emu_mbar(b)); }
inline void mbar_arrive_expect_tx(uint64_t* b, uint32_t bytes) { emu_mbar(b).bytes += (int32_t)bytes; mbar_arrive(b); }
inline void mbar_wait(uint64_t* b, uint32_t parity) { while (emu_mbar(b).phase == parity) emu::give_way(); }
inline void mbar_wait_warp(uint64_t* b, uint32_t parity) { mbar_wait(b, parity); __syncwarp(); }
inline void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
  if (((uintptr_t)src & 15) || ((uintptr_t)dst & 15) || bytes % 16) { std::fprintf(stderr, "emu: bulk copy off 16-byte boundaries\n"); std::abort(); }
  std::memcpy(dst, src, bytes);
  emu_mbar(b).bytes -= (int32_t)bytes;
  emu_mbar_turn(emu_mbar(b));
}
// tiled copies of bf16 boxes with the 128-byte swizzle: 16-byte pieces of each 128-byte line are exchanged by its number in the box
struct CUtensorMap { const uint8_t* base; uint64_t dims[4], strides[4]; uint32_t box[4]; };
inline int make_tmap_bf16_4d(CUtensorMap* m, const void* base, const uint64_t* dims, const uint64_t* strides, const uint32_t* box) {
  m->base = (const uint8_t*)base;
  for (int i = 0; i < 4; ++i) {
    m->dims[i] = dims[i];
    m->box[i] = box[i];
    m->strides[i] = i == 0 ? 2 : strides[i - 1] * 2;
    if (i > 0 && (m->strides[i] % 16 || m->strides[i] >= 1ULL << 40)) { set_error("tensor map stride"); return -1; }
  }
  return 0;
}
inline void tma_load_4d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2, int c3) {
  if ((uintptr_t)dst % 1024 || m->box[0] != 64 || c0 % 8) { std::fprintf(stderr, "emu: box off its boundary\n"); std::abort(); }
  const int64_t c[4] = {c0, c1, c2, c3};
  uint32_t line = 0;
  for (uint32_t i3 = 0; i3 < m->box[3]; ++i3)
    for (uint32_t i2 = 0; i2 < m->box[2]; ++i2)
      for (uint32_t i1 = 0; i1 < m->box[1]; ++i1, ++line)
        for (uint32_t p = 0; p < 8; ++p) {
          uint8_t* to = (uint8_t*)dst + line * 128 + ((p ^ (line & 7)) * 16);
          const bool in = c[0] + p * 8 < (int64_t)m->dims[0] && c[1] + i1 < (int64_t)m->dims[1] && c[2] + i2 < (int64_t)m->dims[2] && c[3] + i3 < (int64_t)m->dims[3];
          if (in) std::memcpy(to, m->base + (c[0] + p * 8) * 2 + (c[1] + i1) * m->strides[1] + (c[2] + i2) * m->strides[2] + (c[3] + i3) * m->strides[3], 16);
          else std::memset(to, 0, 16);
        }
  emu_mbar(bar).bytes -= (int32_t)(line * 128);
  emu_mbar_turn(emu_mbar(bar));
}
inline uint64_t read_once_policy() { return 0; }
inline void tma_load_4d_once(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2, int c3, uint64_t) { tma_load_4d(dst, m, bar, c0, c1, c2, c3); }
#endif
struct ProfScope { ProfScope(int, int, int, int, cudaStream_t) {} };
}  // namespace lp

#define LP_CHECK_CUDA(expr)                                        \
  do {                                                             \
    cudaError_t _e = (expr);                                       \
    if (_e != cudaSuccess) { lp::set_error("cuda error"); return -2; } \
  } while (0)
#define LP_REQUIRE(cond, ...)     \
  do {                            \
    if (!(cond)) {                \
      lp::set_error(__VA_ARGS__); \
      return -1;                  \
    }                             \
  } while (0)

// leopard_b200 — host utilities: error string, device query, TMA descriptor encoding.
#include "lp_host.h"
#include "../../include/leopard_b200.h"
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

namespace lp {

static thread_local char g_err[1024] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}
const char* get_error() { return g_err; }

int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
  }
  return n;
}

static int g_prefill_pdl = 1;  // default on: -2.2 % per cfg3 step (85.6 -> 83.7 ms), results unchanged
bool prefill_pdl() { return g_prefill_pdl != 0; }

// ---- launch counter / profiler ------------------------------------------------------------------------------------
static long long g_launches = 0;
void note_launch(int n) { g_launches += n; }

struct ProfRec { cudaEvent_t e0, e1; int kind, a, b, c; };
static ProfRec* g_recs = nullptr;
static int g_cap = 0, g_n = 0, g_enabled = 0;

ProfScope::ProfScope(int kind, int a, int b, int c, cudaStream_t s) : idx(-1), stream(s) {
  if (!g_enabled || g_n >= g_cap) return;
  idx = g_n++;
  g_recs[idx].kind = kind; g_recs[idx].a = a; g_recs[idx].b = b; g_recs[idx].c = c;
  cudaEventRecord(g_recs[idx].e0, stream);
}
ProfScope::~ProfScope() {
  if (idx >= 0) cudaEventRecord(g_recs[idx].e1, stream);
}

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode() {
  static PFN_encodeTiled fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_encodeTiled>(p);
  }
  return fn;
}

static int encode(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_b,
                  const cuuint32_t* box, CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_128B) {
  PFN_encodeTiled fn = get_encode();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled unavailable (no CUDA driver?)");
    return LP_ERR_CUDA;
  }
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), dims, strides_b,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed: CUresult %d (rank %d dims %llu,%llu box %u,%u stride %llu)", (int)r, rank,
              (unsigned long long)dims[0], (unsigned long long)dims[1], box[0], box[1],
              (unsigned long long)strides_b[0]);
    return LP_ERR_CUDA;
  }
  return 0;
}

int make_tmap_bf16_2d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t ld_elems,
                      uint32_t box_inner, uint32_t box_outer) {
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld_elems * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  return encode(map, base, 2, dims, strides, box);
}

int make_tmap_2d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t inner, uint64_t outer, uint64_t ld_elems,
                 uint32_t box_inner, uint32_t box_outer, int swizzle_bytes) {
  if (elem_bytes != 2) {
    set_error("make_tmap_2d: only 2-byte elements are supported");
    return LP_ERR_ARG;
  }
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld_elems * (cuuint64_t)elem_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  CUtensorMapSwizzle swz = swizzle_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                           : swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                           : swizzle_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                                 : CU_TENSOR_MAP_SWIZZLE_NONE;
  return encode(map, base, 2, dims, strides, box, swz);
}

int make_tmap_bf16_3d(CUtensorMap* map, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t ld1_elems,
                      uint64_t ld2_elems, uint32_t b0, uint32_t b1, uint32_t b2) {
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {ld1_elems * 2, ld2_elems * 2};
  cuuint32_t box[3] = {b0, b1, b2};
  return encode(map, base, 3, dims, strides, box);
}
int make_tmap_bf16_4d(CUtensorMap* map, const void* base, const uint64_t* dims, const uint64_t* strides_elems, const uint32_t* box) {
  cuuint64_t d[4] = {dims[0], dims[1], dims[2], dims[3]}, s[3] = {strides_elems[0] * 2, strides_elems[1] * 2, strides_elems[2] * 2};
  cuuint32_t b[4] = {box[0], box[1], box[2], box[3]};
  return encode(map, base, 4, d, s, b);
}

}  // namespace lp

extern "C" const char* lp_last_error(void) { return lp::get_error(); }
extern "C" int lp_set_prefill_pdl(int enable) {
  const int old = lp::g_prefill_pdl;
  lp::g_prefill_pdl = enable ? 1 : 0;
  return old;
}
extern "C" int lp_abi_version(void) { return LP_ABI_VERSION; }

extern "C" long long lp_launch_count(void) { return lp::g_launches; }

extern "C" int lp_profile_enable(int capacity) {
  using namespace lp;
  if (capacity > g_cap) {
    ProfRec* n = new ProfRec[capacity];
    for (int i = 0; i < g_cap; ++i) n[i] = g_recs[i];
    for (int i = g_cap; i < capacity; ++i) {
      if (cudaEventCreate(&n[i].e0) != cudaSuccess || cudaEventCreate(&n[i].e1) != cudaSuccess) {
        set_error("lp_profile_enable: cudaEventCreate failed");
        delete[] n;
        return LP_ERR_CUDA;
      }
    }
    delete[] g_recs;
    g_recs = n;
    g_cap = capacity;
  }
  g_n = 0;
  g_enabled = capacity > 0;
  return 0;
}

extern "C" int lp_profile_read(lp_profile_record* out, int capacity) {
  using namespace lp;
  g_enabled = 0;
  int n = g_n < capacity ? g_n : capacity;
  for (int i = 0; i < n; ++i) {
    float ms = 0.f;
    if (cudaEventSynchronize(g_recs[i].e1) != cudaSuccess || cudaEventElapsedTime(&ms, g_recs[i].e0, g_recs[i].e1) != cudaSuccess) {
      set_error("lp_profile_read: event query failed");
      return LP_ERR_CUDA;
    }
    out[i].kind = g_recs[i].kind; out[i].a = g_recs[i].a; out[i].b = g_recs[i].b; out[i].c = g_recs[i].c;
    out[i].ms = ms;
  }
  g_n = 0;
  return n;
}

// leopard_b200 — sequence mixers with 32-bit scores and state, over packed batches of requests (prefill rows or one row per request).
//
//   Rotary positions     angle = position * inv_freq[i] in fp32, accurate sincosf; two pairings: LP_ROT_HALF (i with i + dims/2) and
//                        LP_ROT_INTERLEAVED (2i with 2i + 1); both cos and sin carry a magnitude factor (frequency-rescaled tables such as
//                        YaRN's are built on the host: the kernels take the table and the factor).  Only the first `rot_dims` dimensions
//                        of a head are rotated.
//   Retention            per head S_t = decay S_(t-1) + k_t v_t^T, o_t = S_t^T q_t (no softmax, no denominator), then o / rms(o) per head
//                        and an output gate silu(g).  State [slot][head][dim][vdim] fp32, carried between steps.  Two options make
//                        it the linear ("lightning") attention of other designs: in_act = 1 applies silu to q, k and v as they
//                        are read, and finish = LP_RET_FINISH_RAW stores o itself (the norm over all heads and the gate follow
//                        in lp_rmsnorm_gated_f32).
//       prefill          chunks of 32 tokens, three kernels: (1) every chunk's own contribution sum_j decay^(len-1-j) k_j v_j^T in
//                        parallel, (2) a scan over the chunks of a request that turns them into the state at each chunk's start and
//                        stores the final state, (3) every chunk's outputs in parallel: decay^(i+1) q_i^T S_start plus the causal
//                        in-chunk part.  Any start position: the scan starts from the stored state when the request has history.
//       decode           one kernel: rotate, update the state in place, read out, normalise, gate.
//   Latent attention     keys and values are up-projections of one cached latent row c (plus one rotated key part shared by all heads).
//                        The kernels work on the cache directly (absorbed form): score = (W_uk^T q_unrot) . c + q_rot . k_rot, output =
//                        W_uv (sum_j p_j c_j); the two per-head products run as batched lp_linear calls around lp_latent_attend.
//                        Sliding window: key j is visible to query i when 0 <= i - j < window (window <= 0: all earlier keys).
//                        Cache: pages of `page_size` rows [c | k_rot] fp32, one page table row per request.  Layers may share one cache:
//                        a layer without latents of its own (dkv NULL) reads the rows another layer wrote earlier in the step.
//       lp_latent_prep   RMS-norms the latent (vector gain), rotates the shared key part and writes both to the request's pages;
//                        rotates the query's rotated part in place (without latents of its own: only that).
//       lp_latent_attend one CTA per (row, head), its warps split the visible keys: online softmax in fp32, merged at the end.
//       lp_latent_attend_tiles  prompts: tiles of (row, head) pairs share the keys they read.
#include <cuda_pipeline.h>
#include "lp_host.h"
#include "../../include/leopard_b200.h"

namespace lp {

typedef __nv_bfloat16 bf16;

constexpr int RET_CHUNK = LP_RETENTION_CHUNK;
constexpr int RET_CHUNK_THREADS = 256;      // CTA size of the two chunk kernels (their loops stride by blockDim)

// element d of one head's vector x at position pos: rotated when d < rot_dims, copied otherwise
__device__ __forceinline__ float rot_elem(const float* __restrict__ x, int d, int rot_dims, int layout, const float* __restrict__ inv_freq,
                                          float mscale, int pos) {
  if (d >= rot_dims) return x[d];
  const int half = rot_dims >> 1;
  int i, partner;
  bool first;
  if (layout == LP_ROT_INTERLEAVED) {
    i = d >> 1;
    first = (d & 1) == 0;
    partner = first ? d + 1 : d - 1;
  } else {
    first = d < half;
    i = first ? d : d - half;
    partner = first ? d + half : d - half;
  }
  const float ang = (float)pos * inv_freq[i];
  float s, c;
  sincosf(ang, &s, &c);
  s *= mscale;
  c *= mscale;
  // pair (u, v) -> (u c - v s, v c + u s)
  return first ? x[d] * c - x[partner] * s : x[d] * c + x[partner] * s;
}

struct RetArgs {
  const float* qkvg; long long ld; int q_off, k_off, v_off, g_off;
  int heads, dim, vdim;
  const float* decay;
  const float* inv_freq; int rot_dims, rot_layout; float rot_mscale;
  float k_scale, eps;
  float* state; long long slot_stride;
  void* out; long long ldo; int out_fp32;
  int in_act, finish;
};

// floats between rows of keys and queries in shared memory: rows of 16-byte pieces whose neighbours lie four banks further, or rows an odd stride apart
template <bool WIDE> __host__ __device__ inline int ret_dimp(int dim) { return WIDE ? dim + 4 : ((dim + 3) & ~3) + 1; }
// the same where the output kernel's products are matrix instructions: four 16-byte pieces of each of two rows lie in different banks
__host__ __device__ inline int ret_mm_dimp(int dim) { return dim + 16; }

__device__ __forceinline__ float ret_silu(float z) { return z / (1.0f + expf(-z)); }
// element d of one head's q or k: activation (when asked for), then rotation
__device__ __forceinline__ float ret_qk(const RetArgs& a, const float* __restrict__ x, int d, int pos) {
  if (a.in_act) return ret_silu(x[d]);      // the host admits an activation only without rotation
  return rot_elem(x, d, a.rot_dims, a.rot_layout, a.inv_freq, a.rot_mscale, pos);
}
__device__ __forceinline__ float ret_v(const RetArgs& a, float v) { return a.in_act ? ret_silu(v) : v; }

__device__ __forceinline__ float4 ret_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float ret_at(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// one chunk's keys (and queries) of a head into shared memory, rows dimp apart: a thread takes a rotation pair, whose one sine and cosine serve all it
// holds (an element a thread took an eighth of the kernels' time for them), or a dimension that is not rotated.  kw: a factor of each row's key, or null.
// MM (heads of whole RET_MM dimensions): a lane keeps its pairs from row to row, no divisions.
template <bool MM>
__device__ __forceinline__ void ret_load_keys(const RetArgs& a, int row0, int len, int pos0, int h, int dimp, const float* kw, float* ks, float* qs) {
  const int half = a.in_act ? 0 : min(a.rot_dims, a.dim) >> 1, per = a.dim - half;      // no rotation with an activation
  constexpr int BATCH = 4;      // what a batch reads is asked for before any of it is stored
  if constexpr (MM) {
    constexpr int WARPS = RET_CHUNK_THREADS / 32;
    static_assert(RET_CHUNK == BATCH * WARPS, "a warp's rows are one batch");
    const int warp = threadIdx.x >> 5;
    for (int e = threadIdx.x & 31; e < per; e += 32) {
      const bool turn = e < half;
      const int d0 = !turn ? half + e : a.rot_layout == LP_ROT_INTERLEAVED ? 2 * e : e, d1 = !turn ? d0 : a.rot_layout == LP_ROT_INTERLEAVED ? 2 * e + 1 : e + half;
      const float freq = turn ? a.inv_freq[e] : 0.f;
      float k0[BATCH], k1[BATCH], q0[BATCH], q1[BATCH];
#pragma unroll
      for (int n = 0; n < BATCH; ++n) {
        const int j = warp + n * WARPS;
        const float* base = a.qkvg + (long long)(row0 + j) * a.ld + h * a.dim;
        k0[n] = j < len ? base[a.k_off + d0] : 0.f;
        k1[n] = j < len ? base[a.k_off + d1] : 0.f;
        q0[n] = j < len && qs != nullptr ? base[a.q_off + d0] : 0.f;
        q1[n] = j < len && qs != nullptr ? base[a.q_off + d1] : 0.f;
      }
#pragma unroll
      for (int n = 0; n < BATCH; ++n) {
        const int j = warp + n * WARPS;
        if (j >= len) break;
        const float w = kw != nullptr ? kw[j] : 1.f;
        if (turn) {
          float sn, cs;
          sincosf((float)(pos0 + j) * freq, &sn, &cs);
          sn *= a.rot_mscale;
          cs *= a.rot_mscale;
          ks[j * dimp + d0] = (k0[n] * cs - k1[n] * sn) * a.k_scale * w;
          ks[j * dimp + d1] = (k1[n] * cs + k0[n] * sn) * a.k_scale * w;
          if (qs != nullptr) {
            qs[j * dimp + d0] = q0[n] * cs - q1[n] * sn;
            qs[j * dimp + d1] = q1[n] * cs + q0[n] * sn;
          }
        } else {
          ks[j * dimp + d0] = (a.in_act ? ret_silu(k0[n]) : k0[n]) * a.k_scale * w;
          if (qs != nullptr) qs[j * dimp + d0] = a.in_act ? ret_silu(q0[n]) : q0[n];
        }
      }
    }
    return;
  }
  for (int it0 = threadIdx.x; it0 < len * per; it0 += BATCH * blockDim.x) {
    float k0[BATCH], k1[BATCH], q0[BATCH], q1[BATCH];
#pragma unroll
    for (int n = 0; n < BATCH; ++n) {
      const int it = it0 + n * blockDim.x, j = it / per, e = it % per;
      if (it >= len * per) break;
      const float* base = a.qkvg + (long long)(row0 + j) * a.ld + h * a.dim;
      const int d0 = e >= half ? half + e : a.rot_layout == LP_ROT_INTERLEAVED ? 2 * e : e, d1 = e >= half ? d0 : a.rot_layout == LP_ROT_INTERLEAVED ? 2 * e + 1 : e + half;
      k0[n] = base[a.k_off + d0];
      k1[n] = base[a.k_off + d1];
      q0[n] = qs != nullptr ? base[a.q_off + d0] : 0.f;
      q1[n] = qs != nullptr ? base[a.q_off + d1] : 0.f;
    }
#pragma unroll
    for (int n = 0; n < BATCH; ++n) {
      const int it = it0 + n * blockDim.x, j = it / per, e = it % per;
      if (it >= len * per) break;
      const float w = kw != nullptr ? kw[j] : 1.f;
      if (e < half) {
        const int d0 = a.rot_layout == LP_ROT_INTERLEAVED ? 2 * e : e, d1 = a.rot_layout == LP_ROT_INTERLEAVED ? 2 * e + 1 : e + half;
        float sn, cs;
        sincosf((float)(pos0 + j) * a.inv_freq[e], &sn, &cs);
        sn *= a.rot_mscale;
        cs *= a.rot_mscale;
        ks[j * dimp + d0] = (k0[n] * cs - k1[n] * sn) * a.k_scale * w;
        ks[j * dimp + d1] = (k1[n] * cs + k0[n] * sn) * a.k_scale * w;
        if (qs != nullptr) {
          qs[j * dimp + d0] = q0[n] * cs - q1[n] * sn;
          qs[j * dimp + d1] = q1[n] * cs + q0[n] * sn;
        }
      } else {
        ks[j * dimp + half + e] = (a.in_act ? ret_silu(k0[n]) : k0[n]) * a.k_scale * w;
        if (qs != nullptr) qs[j * dimp + half + e] = a.in_act ? ret_silu(q0[n]) : q0[n];
      }
    }
  }
}
// `len` rows of vdim columns from column `off` of the projection on, rows ldd apart, copied while other work is done (the caller commits and waits);
// false: rows are not whole 16-byte pieces, nothing was copied
template <bool MM>
__device__ __forceinline__ bool ret_copy_rows(const RetArgs& a, int row0, int len, int off, float* dst, int ldd) {
  if (((a.ld | off | a.vdim | ldd) & 3) != 0 || (reinterpret_cast<uintptr_t>(a.qkvg) & 15) != 0) return false;
  const int per = a.vdim >> 2;
  if constexpr (MM) {      // a warp a row
    for (int j = threadIdx.x >> 5; j < len; j += RET_CHUNK_THREADS / 32)
      for (int c = (threadIdx.x & 31) * 4; c < a.vdim; c += 128) __pipeline_memcpy_async(dst + j * ldd + c, a.qkvg + (long long)(row0 + j) * a.ld + off + c, 16);
    return true;
  }
  for (int i = threadIdx.x; i < len * per; i += blockDim.x) {
    const int j = i / per, c = (i % per) * 4;
    __pipeline_memcpy_async(dst + j * ldd + c, a.qkvg + (long long)(row0 + j) * a.ld + off + c, 16);
  }
  return true;
}

// Heads whose keys and values both have a multiple of RET_MM dimensions take the matrix instruction for the three products of a chunk: both operands
// in three bf16 terms each (cut3), the six products of weight above 2^-26 with the small ones first, 16 terms of a sum at a time and these added in
// fp32.  The order of k within such a step is free as long as both sides agree: where a lane's four k are neighbours, it reads them at once.
// 4,096 rows of 16 heads of 128 x 128 (us, fp32 sums from shared memory and so): the chunks' states 116, 74, the outputs 237, 138; errors against
// 64 bits 1.2e-7 of the outputs for 2.3e-7.  Both are bound by instructions now (65 % of the issue slots; cutting the operands is a third of them).
constexpr int RET_MM = 128;
struct RetRows { uint32_t hi[4], mid[4], lo[4]; };      // 16 x 16: rows g and g + 8 at this lane's four k
__device__ __forceinline__ RetRows ret_cut_rows(const float4& x, const float4& y) {
  RetRows r;
  cut3(x.x, x.y, r.hi[0], r.mid[0], r.lo[0]);
  cut3(y.x, y.y, r.hi[1], r.mid[1], r.lo[1]);
  cut3(x.z, x.w, r.hi[2], r.mid[2], r.lo[2]);
  cut3(y.z, y.w, r.hi[3], r.mid[3], r.lo[3]);
  return r;
}
struct RetColumn { uint32_t hi[2], mid[2], lo[2]; };      // 16 x 8: column g at this lane's four k
__device__ __forceinline__ RetColumn ret_cut_column(float k0, float k1, float k2, float k3) {
  RetColumn r;
  cut3(k0, k1, r.hi[0], r.mid[0], r.lo[0]);
  cut3(k2, k3, r.hi[1], r.mid[1], r.lo[1]);
  return r;
}
__device__ __forceinline__ void ret_mma(float (&acc)[4], const RetRows& a, const RetColumn& b) {
  float d[4];
  mma_bf16_first(d, a.lo[0], a.lo[1], a.lo[2], a.lo[3], b.hi[0], b.hi[1]);
  mma_bf16(d, a.hi[0], a.hi[1], a.hi[2], a.hi[3], b.lo[0], b.lo[1]);
  mma_bf16(d, a.mid[0], a.mid[1], a.mid[2], a.mid[3], b.mid[0], b.mid[1]);
  mma_bf16(d, a.mid[0], a.mid[1], a.mid[2], a.mid[3], b.hi[0], b.hi[1]);
  mma_bf16(d, a.hi[0], a.hi[1], a.hi[2], a.hi[3], b.mid[0], b.mid[1]);
  mma_bf16(d, a.hi[0], a.hi[1], a.hi[2], a.hi[3], b.hi[0], b.hi[1]);
#pragma unroll
  for (int c = 0; c < 4; ++c) acc[c] += d[c];
}

// The three kernels of a prompt wait as programmatic launches do, but none lets the next one start early: its CTAs, placed beside the running ones, took a third of
// the time more than the launch gaps that they save (us a prompt of 887 rows of 4 heads of 96 x 256: early 74, so 51, plain launches 52; 5 rows of 16 heads of 128 x 128 32, 22, 23).
// (1) U[chunk][head] = sum_j decay^(len-1-j) k_j v_j^T.  4 x 4 outputs per thread (8 x 8 from 16-byte reads: 208 us for 162); a thread's four columns are vdim/4
// apart, so that the threads of a warp read consecutive shared-memory words.  MM: two CTAs an SM (three, at 80 registers, spill: 78 us for 74).
template <bool MM>
__global__ void __launch_bounds__(RET_CHUNK_THREADS, MM ? 2 : 1)
retention_chunk_state_kernel(RetArgs a, const int* __restrict__ chunk_seq, const int* __restrict__ chunk_row0, const int* __restrict__ chunk_len,
                             const int* __restrict__ seq_row0, const int* __restrict__ seq_pos0, float* __restrict__ ws) {
  pdl_wait();
  extern __shared__ float dyn_smem[];
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int s = chunk_seq[c], row0 = chunk_row0[c], len = chunk_len[c];
  const int pos0 = seq_pos0[s] + (row0 - seq_row0[s]);
  // padded rows: whole 4-tiles; MM: neighbouring rows eight banks further
  const int dimp = MM ? a.dim + 8 : ret_dimp<false>(a.dim), vdimp = MM ? a.vdim + 8 : (a.vdim + 3) & ~3;
  float* kd = dyn_smem;                   // [RET_CHUNK][dimp]
  float* vv = kd + RET_CHUNK * dimp;      // [RET_CHUNK][vdimp]
  __shared__ float power[RET_CHUNK];
  if (tid < len) power[tid] = powf(a.decay[h], (float)(len - 1 - tid));
  __syncthreads();
  const bool copied = !a.in_act && ret_copy_rows<MM>(a, row0, len, a.v_off + h * a.vdim, vv, vdimp);
  __pipeline_commit();
  for (int i = tid; !MM && i < len * (dimp - a.dim); i += blockDim.x) kd[i / (dimp - a.dim) * dimp + a.dim + i % (dimp - a.dim)] = 0.f;
  ret_load_keys<MM>(a, row0, len, pos0, h, dimp, power, kd, nullptr);
  for (int i = tid; !copied && i < len * vdimp; i += blockDim.x) {
    const int j = i / vdimp, d = i % vdimp;
    vv[i] = d < a.vdim ? ret_v(a, a.qkvg[(long long)(row0 + j) * a.ld + a.v_off + h * a.vdim + d]) : 0.f;
  }
  if constexpr (MM) {      // rows that the chunk does not have are zeros
    for (int i = len * dimp + tid; i < RET_CHUNK * dimp; i += blockDim.x) kd[i] = 0.f;
    for (int i = len * vdimp + tid; i < RET_CHUNK * vdimp; i += blockDim.x) vv[i] = 0.f;
  }
  __pipeline_wait_prior(0);
  __syncthreads();
  float* U = ws + ((long long)c * a.heads + h) * a.dim * a.vdim;
  if constexpr (MM) {      // a warp: 64 dimensions of the keys x 32 columns, whose terms it keeps
    const int lane = tid & 31, g = lane >> 2, t = lane & 3, halves = a.dim >> 6;
    bool odd = false;
    for (int tile = tid >> 5; tile < halves * (a.vdim >> 5); tile += RET_CHUNK_THREADS / 32) {
      const int x0 = tile % halves * 64, y0 = tile / halves * 32;
      RetColumn b[RET_CHUNK / 16][4];
#pragma unroll
      for (int kb = 0; kb < RET_CHUNK / 16; ++kb) {
        float4 v[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) v[n] = ret_ld4(vv + (kb * 16 + 4 * n + t) * vdimp + y0 + 4 * g);
#pragma unroll
        for (int j = 0; j < 4; ++j) b[kb][j] = ret_cut_column(ret_at(v[0], j), ret_at(v[1], j), ret_at(v[2], j), ret_at(v[3], j));
      }
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        float acc[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
        for (int kb = 0; kb < RET_CHUNK / 16; ++kb) {
          const float* k = kd + (kb * 16 + t) * dimp + x0 + 16 * i + g;
          const RetRows ka = ret_cut_rows(make_float4(k[0], k[4 * dimp], k[8 * dimp], k[12 * dimp]),
                                          make_float4(k[8], k[4 * dimp + 8], k[8 * dimp + 8], k[12 * dimp + 8]));
#pragma unroll
          for (int j = 0; j < 4; ++j) ret_mma(acc[j], ka, b[kb][j]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {      // row g or g + 8, column 2 t or 2 t + 1 of the four tiles
          float* to = U + (long long)(x0 + 16 * i + g + (e >> 1) * 8) * a.vdim + y0 + 8 * t + (e & 1) * 4;
          *reinterpret_cast<float4*>(to) = make_float4(acc[0][e], acc[1][e], acc[2][e], acc[3][e]);
#pragma unroll
          for (int j = 0; j < 4; ++j) odd |= not_finite(acc[j][e]);
        }
      }
    }
    if (!__syncthreads_or(odd)) return;      // the terms of an infinity do not add up to it: such a chunk is taken again below
  }
  const int tiles_y = (a.vdim + 3) >> 2, tiles_x = (a.dim + 3) >> 2;
  for (int tile = tid; tile < tiles_x * tiles_y; tile += blockDim.x) {
    const int x0 = (tile / tiles_y) * 4, ty = tile % tiles_y;
    float acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] = 0.f;
    for (int j = 0; j < len; ++j) {
      float k4[4], v4[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        k4[p] = kd[j * dimp + x0 + p];
        v4[p] = vv[j * vdimp + ty + p * tiles_y];
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(k4[p], v4[q], acc[p][q]);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int x = x0 + p, y = ty + q * tiles_y;
        if (x < a.dim && y < a.vdim) U[x * a.vdim + y] = acc[p][q];
      }
  }
}

// (2) V state elements of a (request, head) a thread: ws[chunk] <- state at the chunk's start; the state after the last chunk goes to the slot.  The
// chunks' own contributions are loaded SCAN_BATCH at a time, the next ones while these are added up.
constexpr int SCAN_THREADS = 256, SCAN_BATCH = 8;
template <int V> struct RetVec;
template <> struct RetVec<1> { float v[1]; };
template <> struct alignas(16) RetVec<4> { float v[4]; };
template <int V>
__global__ void __launch_bounds__(SCAN_THREADS)
retention_scan_kernel(RetArgs a, const int* __restrict__ seq_chunk0, const int* __restrict__ chunk_len, const int* __restrict__ seq_pos0,
                      const int* __restrict__ seq_slot, float* ws) {
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y;
  const long long hs = (long long)a.dim * a.vdim;
  const long long i = ((long long)blockIdx.z * SCAN_THREADS + threadIdx.x) * V;
  if (i >= hs) return;
  const int c0 = seq_chunk0[s], c1 = seq_chunk0[s + 1];
  const float dec = a.decay[h];
  const float dec_full = powf(dec, (float)RET_CHUNK);
  RetVec<V>* st = reinterpret_cast<RetVec<V>*>(a.state + (long long)seq_slot[s] * a.slot_stride + h * hs + i);
  RetVec<V> S;
  if (seq_pos0[s] == 0) {
#pragma unroll
    for (int e = 0; e < V; ++e) S.v[e] = 0.f;
  } else {
    S = *st;
  }
  const long long stride = (long long)a.heads * hs;
  float* u = ws + ((long long)c0 * a.heads + h) * hs + i;
  RetVec<V> own[SCAN_BATCH], next[SCAN_BATCH];
  auto fetch = [&](RetVec<V>* dst, const float* from, int c) {
#pragma unroll
    for (int k = 0; k < SCAN_BATCH; ++k)
      if (c + k < c1) dst[k] = *reinterpret_cast<const RetVec<V>*>(from + k * stride);
  };
  fetch(own, u, c0);
  for (int c = c0; c < c1; c += SCAN_BATCH) {
    fetch(next, u + SCAN_BATCH * stride, c + SCAN_BATCH);
#pragma unroll
    for (int k = 0; k < SCAN_BATCH; ++k) {
      if (c + k < c1) {
        const int len = chunk_len[c + k];
        const float f = len == RET_CHUNK ? dec_full : powf(dec, (float)len);
        *reinterpret_cast<RetVec<V>*>(u + k * stride) = S;
#pragma unroll
        for (int e = 0; e < V; ++e) S.v[e] = fmaf(f, S.v[e], own[k].v[e]);
      }
    }
#pragma unroll
    for (int k = 0; k < SCAN_BATCH; ++k) own[k] = next[k];
    u += SCAN_BATCH * stride;
  }
  *st = S;
}

// (3) o_i = decay^(i+1) q_i^T S_start + sum_(j<=i) decay^(i-j) (q_i . k_j) v_j; then o / rms(o) * silu(g).  The chunk's start state is
// staged in shared memory where that is small (stage_s); a state of 128 x 128 would leave one CTA an SM, and the CTAs waiting for it and for
// each other's phases took 1.23 ms (4096 tokens, 16 heads): read where it lies (L2, whole lines, eight loads in flight) three CTAs share an
// SM and it takes 0.46 ms.  4 x 4 outputs per thread.  The line is what leaves three CTAs an SM; whole prompts on both sides (us, staged up to
// 200 KB, and so): 16 heads of 128, 4096 tokens 1450, 756, 512 tokens 150, 93; 8 heads of 96 286, 203 and 62, 58; 16 of 80 355, 313 and 59, 57; 8 of
// 128 keys and 64 values 264, 188 and 60, 61.  64 x 64 is staged on both.  WIDE: the same sums in the same order from 16-byte reads,
// a quarter as many, values and gates copied in meanwhile: 0.46 -> 0.24 ms.  MM: matrix instructions, 0.14 ms; the state's terms are cut once.
template <bool WIDE, bool MM>
__global__ void __launch_bounds__(RET_CHUNK_THREADS, MM ? 3 : 1)
retention_chunk_out_kernel(RetArgs a, const int* __restrict__ chunk_seq, const int* __restrict__ chunk_row0, const int* __restrict__ chunk_len,
                           const int* __restrict__ seq_row0, const int* __restrict__ seq_pos0, const float* ws, int stage_s) {
  pdl_wait();
  extern __shared__ float dyn_smem[];
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int s = chunk_seq[c], row0 = chunk_row0[c], len = chunk_len[c];
  const int pos0 = seq_pos0[s] + (row0 - seq_row0[s]);
  const int dimp = MM ? ret_mm_dimp(a.dim) : ret_dimp<WIDE>(a.dim), vdimp = (a.vdim + 3) & ~3;
  float* qs = dyn_smem;                        // [RET_CHUNK][dimp]
  float* ks = qs + RET_CHUNK * dimp;           // [RET_CHUNK][dimp]
  float* vv = ks + RET_CHUNK * dimp;           // [RET_CHUNK][vdimp]
  float* os = vv + RET_CHUNK * vdimp;          // [RET_CHUNK][vdimp]
  float* pp = os + RET_CHUNK * vdimp;          // [RET_CHUNK][RET_CHUNK + 1]
  float* power = pp + RET_CHUNK * (RET_CHUNK + 1);   // [RET_CHUNK]: decay^(i + 1)
  float* Ss = power + RET_CHUNK;               // [dim][vdimp] when stage_s
  const float dec = a.decay[h];
  if (tid < RET_CHUNK) power[tid] = powf(dec, (float)(tid + 1));
  const bool copied = !a.in_act && ret_copy_rows<MM>(a, row0, len, a.v_off + h * a.vdim, vv, vdimp);
  __pipeline_commit();
  for (int i = len * dimp + tid; i < RET_CHUNK * dimp; i += blockDim.x) qs[i] = ks[i] = 0.f;
  if constexpr (MM)
    for (int i = len * vdimp + tid; i < RET_CHUNK * vdimp; i += blockDim.x) vv[i] = 0.f;
  ret_load_keys<MM>(a, row0, len, pos0, h, dimp, nullptr, ks, qs);
  for (int i = tid; !copied && i < RET_CHUNK * vdimp; i += blockDim.x) {
    const int j = i / vdimp, d = i % vdimp;
    vv[i] = (j < len && d < a.vdim) ? ret_v(a, a.qkvg[(long long)(row0 + j) * a.ld + a.v_off + h * a.vdim + d]) : 0.f;
  }
  const float* S = ws + ((long long)c * a.heads + h) * a.dim * a.vdim;
  if (stage_s)
    for (int i = tid; i < a.dim * vdimp; i += blockDim.x) {
      const int d = i / vdimp, y = i % vdimp;
      Ss[i] = y < a.vdim ? S[d * a.vdim + y] : 0.f;
    }
  __pipeline_wait_prior(0);
  __syncthreads();
  bool scored = false;
  if constexpr (MM) {      // in-chunk scores, a warp: 16 rows x 8 keys
    const int lane = tid & 31, g = lane >> 2, t = lane & 3, r0 = (tid >> 5 & 1) * 16, j0 = (tid >> 6) * 8;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (j0 < r0 + 16) {
      const float* q = qs + (r0 + g) * dimp + 4 * t;
      const float* k = ks + (j0 + g) * dimp + 4 * t;
#pragma unroll 2
      for (int d = 0; d < a.dim; d += 16) {
        const float4 kv = ret_ld4(k + d);
        ret_mma(acc, ret_cut_rows(ret_ld4(q + d), ret_ld4(q + 8 * dimp + d)), ret_cut_column(kv.x, kv.y, kv.z, kv.w));
      }
    }
    bool odd = false;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = r0 + g + (e >> 1) * 8, j = j0 + 2 * t + (e & 1);
      odd |= not_finite(acc[e]);
      pp[i * (RET_CHUNK + 1) + j] = (j <= i && i < len) ? acc[e] * (i == j ? 1.f : power[i - j - 1]) : 0.f;
    }
    scored = !__syncthreads_or(odd);      // the terms of an infinity do not add up to it: such scores are taken again
  }
  // in-chunk scores, 2 x 2 per thread (rows i0, i0 + 1, columns tj, tj + 16): every thread has one
  for (int tile = scored ? (RET_CHUNK / 2) * (RET_CHUNK / 2) : tid; tile < (RET_CHUNK / 2) * (RET_CHUNK / 2); tile += blockDim.x) {
    const int i0 = (tile / (RET_CHUNK / 2)) * 2, tj = tile % (RET_CHUNK / 2);
    float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    if constexpr (WIDE) {
#pragma unroll 2
      for (int d = 0; d < a.dim; d += 4) {
        const float4 qa = ret_ld4(qs + i0 * dimp + d), qb = ret_ld4(qs + (i0 + 1) * dimp + d), ka = ret_ld4(ks + tj * dimp + d),
                     kb = ret_ld4(ks + (tj + RET_CHUNK / 2) * dimp + d);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[0][0] = fmaf(ret_at(qa, e), ret_at(ka, e), acc[0][0]);
          acc[0][1] = fmaf(ret_at(qa, e), ret_at(kb, e), acc[0][1]);
          acc[1][0] = fmaf(ret_at(qb, e), ret_at(ka, e), acc[1][0]);
          acc[1][1] = fmaf(ret_at(qb, e), ret_at(kb, e), acc[1][1]);
        }
      }
    } else {
#pragma unroll 8
      for (int d = 0; d < a.dim; ++d) {
        float q2[2], k2[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          q2[p] = qs[(i0 + p) * dimp + d];
          k2[p] = ks[(tj + p * (RET_CHUNK / 2)) * dimp + d];
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int q = 0; q < 2; ++q) acc[p][q] = fmaf(q2[p], k2[q], acc[p][q]);
      }
    }
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = i0 + p, j = tj + q * (RET_CHUNK / 2);
        pp[i * (RET_CHUNK + 1) + j] = (j <= i && i < len) ? acc[p][q] * (i == j ? 1.f : power[i - j - 1]) : 0.f;
      }
  }
  __syncthreads();
  // nobody reads the keys any more: the gates come in their place while the outputs are taken
  const bool gates = WIDE && a.finish != LP_RET_FINISH_RAW && a.vdim <= dimp && ret_copy_rows<MM>(a, row0, len, a.g_off + h * a.vdim, ks, dimp);
  __pipeline_commit();
  bool taken = false;
  if constexpr (MM) {      // a warp: the chunk's 32 rows x 16 columns, so that the state is read once
    const int lane = tid & 31, g = lane >> 2, t = lane & 3;
    bool odd = false;
    for (int y0 = (tid >> 5) * 16; y0 < a.vdim; y0 += RET_CHUNK_THREADS / 2) {
      float acc[2][2][4];      // rows 16 i + .., columns 2 c + j of the 16
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
      const float* from = S + (long long)(4 * t) * a.vdim + y0 + 2 * g;
      const float* q = qs + g * dimp + 4 * t;
#pragma unroll 2
      for (int d = 0; d < a.dim; d += 16) {
        float2 s2[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) s2[n] = *reinterpret_cast<const float2*>(from + (long long)(d + n) * a.vdim);
        const RetColumn b0 = ret_cut_column(s2[0].x, s2[1].x, s2[2].x, s2[3].x), b1 = ret_cut_column(s2[0].y, s2[1].y, s2[2].y, s2[3].y);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const RetRows w = ret_cut_rows(ret_ld4(q + 16 * i * dimp + d), ret_ld4(q + (16 * i + 8) * dimp + d));
          ret_mma(acc[i][0], w, b0);
          ret_mma(acc[i][1], w, b1);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float lo = power[16 * i + g], hi = power[16 * i + g + 8];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          acc[i][j][0] *= lo;
          acc[i][j][1] *= lo;
          acc[i][j][2] *= hi;
          acc[i][j][3] *= hi;
        }
      }
#pragma unroll
      for (int kb = 0; kb < RET_CHUNK / 16; ++kb) {
        float2 v2[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) v2[n] = *reinterpret_cast<const float2*>(vv + (kb * 16 + 4 * t + n) * vdimp + y0 + 2 * g);
        const RetColumn b0 = ret_cut_column(v2[0].x, v2[1].x, v2[2].x, v2[3].x), b1 = ret_cut_column(v2[0].y, v2[1].y, v2[2].y, v2[3].y);
#pragma unroll
        for (int i = kb; i < 2; ++i) {      // the second half's keys are none of the first half's rows'
          const float* p = pp + (16 * i + g) * (RET_CHUNK + 1) + kb * 16 + 4 * t;
          const float* p8 = p + 8 * (RET_CHUNK + 1);
          const RetRows w = ret_cut_rows(make_float4(p[0], p[1], p[2], p[3]), make_float4(p8[0], p8[1], p8[2], p8[3]));
          ret_mma(acc[i][0], w, b0);
          ret_mma(acc[i][1], w, b1);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {      // columns 2 t and 2 t + 1 of both tiles
          *reinterpret_cast<float4*>(os + (16 * i + g + (e >> 1) * 8) * vdimp + y0 + 4 * t) =
              make_float4(acc[i][0][e], acc[i][1][e], acc[i][0][e + 1], acc[i][1][e + 1]);
#pragma unroll
          for (int j = 0; j < 2; ++j) odd |= not_finite(acc[i][j][e]) || not_finite(acc[i][j][e + 1]);
        }
    }
    taken = !__syncthreads_or(odd);      // as above
  }
  const int tiles_y = vdimp >> 2, tiles_i = (len + 3) >> 2;
  for (int tile = taken ? tiles_i * tiles_y : tid; tile < tiles_i * tiles_y; tile += blockDim.x) {
    const int i0 = (tile / tiles_y) * 4, ty = tile % tiles_y;
    float acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] = 0.f;
    if constexpr (WIDE) {      // four neighbouring columns a thread
      const float* from = (stage_s ? Ss : S) + ty * 4;
#pragma unroll 2
      for (int d = 0; d < a.dim; d += 4) {
        float4 q4[4], s4[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) s4[e] = ret_ld4(from + (d + e) * a.vdim);
#pragma unroll
        for (int p = 0; p < 4; ++p) q4[p] = ret_ld4(qs + (i0 + p) * dimp + d);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(ret_at(q4[p], e), ret_at(s4[e], q), acc[p][q]);
      }
    } else {
#pragma unroll 8
      for (int d = 0; d < a.dim; ++d) {
        float q4[4], s4[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          q4[p] = qs[(i0 + p) * dimp + d];
          const int y = ty + p * tiles_y;
          s4[p] = stage_s ? Ss[d * vdimp + y] : (y < a.vdim ? S[d * a.vdim + y] : 0.f);
        }
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(q4[p], s4[q], acc[p][q]);
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float sc = power[i0 + p];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] *= sc;
    }
    const int jmax = min(i0 + 3, len - 1);
    for (int j = 0; j <= jmax; ++j) {
      float p4[4], v4[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        p4[p] = pp[(i0 + p) * (RET_CHUNK + 1) + j];
        if (!WIDE) v4[p] = vv[j * vdimp + ty + p * tiles_y];
      }
      if constexpr (WIDE) {
        const float4 v = ret_ld4(vv + j * vdimp + ty * 4);
        v4[0] = v.x; v4[1] = v.y; v4[2] = v.z; v4[3] = v.w;
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(p4[p], v4[q], acc[p][q]);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) os[(i0 + p) * vdimp + (WIDE ? ty * 4 + q : ty + q * tiles_y)] = acc[p][q];
  }
  __pipeline_wait_prior(0);
  __syncthreads();
  // a warp a row: o itself (what follows it is another kernel's), or over the root mean square of the head's vdim outputs and gated
  const int warp = tid >> 5, lane = tid & 31;
  for (int i = warp; i < len; i += RET_CHUNK_THREADS / 32) {
    const long long o = (long long)(row0 + i) * a.ldo + h * a.vdim;
    float inv = 1.f;
    if (a.finish != LP_RET_FINISH_RAW) {
      float ss = 0.f;
      for (int y = lane; y < a.vdim; y += 32) ss = fmaf(os[i * vdimp + y], os[i * vdimp + y], ss);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
      inv = 1.0f / sqrtf(ss / (float)a.vdim + a.eps);
    }
#pragma unroll 4
    for (int y = lane; y < a.vdim; y += 32) {
      float v = os[i * vdimp + y];
      if (a.finish != LP_RET_FINISH_RAW) {
        const float g = gates ? ks[i * dimp + y] : a.qkvg[(long long)(row0 + i) * a.ld + a.g_off + h * a.vdim + y];
        v = v * inv * (g / (1.0f + expf(-g)));
      }
      if (a.out_fp32) reinterpret_cast<float*>(a.out)[o + y] = v;
      else reinterpret_cast<bf16*>(a.out)[o + y] = __float2bfloat16(v);
    }
  }
}

// decode: one new row per request.  Threads own V neighbouring state columns (V = 4 where rows and slots are whole 16-byte pieces), groups of them split
// the dim rows, eight of which are in flight at a time: with a column a thread and a row read after the one before was written, the chain of
// loads took 16 us (8 requests of 16 heads of 128 x 128) and 37 us (64 of 8), whose bytes take 2.6 and 10.
constexpr int RET_DEC_THREADS = 256, RET_DEC_BATCH = 8;
template <int V> __host__ __device__ inline int ret_dec_groups(int vdim) { return vdim / V >= RET_DEC_THREADS ? 1 : RET_DEC_THREADS / (vdim / V); }
template <int V>
__global__ void __launch_bounds__(RET_DEC_THREADS)
retention_decode_kernel(RetArgs a, const int* __restrict__ seq_row0, const int* __restrict__ seq_pos0, const int* __restrict__ seq_slot) {
  pdl_launch_next_of_few();
  pdl_wait();
  extern __shared__ float dyn_smem[];
  const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int row = seq_row0[s], pos = seq_pos0[s];
  float* qs = dyn_smem;            // [dim]
  float* ks = qs + a.dim;          // [dim]
  float* vv = ks + a.dim;          // [vdim]
  float* os = vv + a.vdim;         // [vdim]
  float* part = os + a.vdim;       // [groups][vdim]
  __shared__ float red[RET_DEC_THREADS / 32];
  const float* base = a.qkvg + (long long)row * a.ld;
  for (int d = tid; d < a.dim; d += blockDim.x) {
    qs[d] = ret_qk(a, base + a.q_off + h * a.dim, d, pos);
    ks[d] = ret_qk(a, base + a.k_off + h * a.dim, d, pos) * a.k_scale;
  }
  for (int y = tid; y < a.vdim; y += blockDim.x) vv[y] = ret_v(a, base[a.v_off + h * a.vdim + y]);
  __syncthreads();
  const float dec = a.decay[h];
  const bool fresh = pos == 0;
  float* st = a.state + (long long)seq_slot[s] * a.slot_stride + (long long)h * a.dim * a.vdim;
  const int groups = ret_dec_groups<V>(a.vdim);
  const int cols = a.vdim / V, g = tid / cols, per = (a.dim + groups - 1) / groups;
  if (g < groups) {
    const int d0 = g * per, d1 = min(a.dim, d0 + per);
    for (int y = tid % cols * V; y < a.vdim; y += RET_DEC_THREADS * V) {
      float acc[V], v[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        acc[k] = 0.f;
        v[k] = vv[y + k];
      }
      for (int b = d0; b < d1; b += RET_DEC_BATCH) {      // a batch of rows is read before the first of them is written
        RetVec<V> old[RET_DEC_BATCH];
#pragma unroll
        for (int i = 0; i < RET_DEC_BATCH; ++i)
          if (b + i < d1 && !fresh) old[i] = *reinterpret_cast<const RetVec<V>*>(st + (long long)(b + i) * a.vdim + y);
          else
#pragma unroll
            for (int k = 0; k < V; ++k) old[i].v[k] = 0.f;
#pragma unroll
        for (int i = 0; i < RET_DEC_BATCH; ++i) {
          if (b + i < d1) {
            const float kd = ks[b + i], qd = qs[b + i];
#pragma unroll
            for (int k = 0; k < V; ++k) {
              old[i].v[k] = fmaf(dec, old[i].v[k], kd * v[k]);
              acc[k] = fmaf(old[i].v[k], qd, acc[k]);
            }
            *reinterpret_cast<RetVec<V>*>(st + (long long)(b + i) * a.vdim + y) = old[i];
          }
        }
      }
#pragma unroll
      for (int k = 0; k < V; ++k) part[g * a.vdim + y + k] = acc[k];
    }
  }
  __syncthreads();
  float ss = 0.f;
  for (int y = tid; y < a.vdim; y += blockDim.x) {
    float acc = 0.f;
    for (int gg = 0; gg < groups; ++gg) acc += part[gg * a.vdim + y];
    os[y] = acc;
    ss = fmaf(acc, acc, ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < RET_DEC_THREADS / 32; ++w) tot += red[w];
  const float r = 1.0f / sqrtf(tot / (float)a.vdim + a.eps);
  for (int y = tid; y < a.vdim; y += blockDim.x) {
    float v = os[y];
    if (a.finish != LP_RET_FINISH_RAW) {
      const float gt = base[a.g_off + h * a.vdim + y];
      v = v * r * (gt / (1.0f + expf(-gt)));
    }
    const long long o = (long long)row * a.ldo + h * a.vdim + y;
    if (a.out_fp32) reinterpret_cast<float*>(a.out)[o] = v;
    else reinterpret_cast<bf16*>(a.out)[o] = __float2bfloat16(v);
  }
}

// ---------------------------------------------------------------------------------------------------------------------------------
// latent attention
// ---------------------------------------------------------------------------------------------------------------------------------
struct LatArgs {
  float* q; long long ldq;
  const float* dkv; long long lddkv;
  int heads, dim, rot_dim, kv_rank;
  const float* c_gain; float eps;
  const float* inv_freq; int rot_dims, rot_layout; float rot_mscale;
  float* cache; int page_size;
  const int* page_table; int max_pages;
  int window; float scale;
  const float* sink;                      // [heads] or null: exp(sink_h) joins the softmax denominator (no key, no value, not scaled)
  const float* gate; long long ldg;       // [rows, ldg] or null: head h's output is multiplied by sigmoid(gate[r, h])
};

__device__ __forceinline__ float lat_gate(const LatArgs& a, int r, int h) {
  return a.gate != nullptr ? 1.0f / (1.0f + expf(-a.gate[(long long)r * a.ldg + h])) : 1.0f;
}

__device__ __forceinline__ float* lat_cache_row(const LatArgs& a, int seq, int pos) {
  const int page = a.page_table[(long long)seq * a.max_pages + pos / a.page_size];
  return a.cache + ((long long)page * a.page_size + pos % a.page_size) * (a.kv_rank + a.rot_dim);
}

// A CTA a row; the row's sines and cosines are taken once for all heads (four a pair and head before: one row of 16 heads 7.0 us).
constexpr int LAT_PREP_THREADS = 128, LAT_PREP_WIDE = 512;      // up to two rows an SM (decoding) take wide CTAs
constexpr int LAT_PREP_PAIRS = 4096;      // rotation pairs whose sines and cosines shared memory holds; with more of them each is taken where it is used
__global__ void __launch_bounds__(LAT_PREP_WIDE)
latent_prep_kernel(LatArgs a, int R, const int* __restrict__ row_seq, const int* __restrict__ row_pos) {
  pdl_launch_next();
  pdl_wait();
  extern __shared__ float dyn_smem[];
  __shared__ float red[LAT_PREP_WIDE / 32];
  const int r = blockIdx.x, tid = threadIdx.x;
  if (r >= R) return;
  const int pos = row_pos[r], half = a.rot_dims >> 1;
  float2* s_turn = reinterpret_cast<float2*>(dyn_smem);      // [half] (cos, sin)
  const bool table = half <= LAT_PREP_PAIRS;
  auto make = [&](int i) {
    float sn, cs;
    sincosf((float)pos * a.inv_freq[i], &sn, &cs);
    return make_float2(cs * a.rot_mscale, sn * a.rot_mscale);
  };
  auto turn = [&](int i) { return table ? s_turn[i] : make(i); };
  for (int i = tid; table && i < half; i += blockDim.x) s_turn[i] = make(i);
  __syncthreads();
  if (a.dkv != nullptr) {      // the layer brings latents of its own
    const float* src = a.dkv + (long long)r * a.lddkv;
    float ss = 0.f;
    for (int c = tid; c < a.kv_rank; c += blockDim.x) ss = fmaf(src[c], src[c], ss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    float total = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) total += red[w];
    const float inv = 1.0f / sqrtf(total / (float)a.kv_rank + a.eps);
    float* dst = lat_cache_row(a, row_seq[r], pos);
    for (int c = tid; c < a.kv_rank; c += blockDim.x) dst[c] = src[c] * inv * a.c_gain[c];
    const float* x = src + a.kv_rank;
    float* y = dst + a.kv_rank;
    for (int i = tid; i < a.rot_dim - half; i += blockDim.x) {      // a pair, or a dimension that is not rotated
      if (i < half) {
        const int d0 = a.rot_layout == LP_ROT_INTERLEAVED ? 2 * i : i, d1 = a.rot_layout == LP_ROT_INTERLEAVED ? 2 * i + 1 : i + half;
        const float2 t = turn(i);
        y[d0] = x[d0] * t.x - x[d1] * t.y;
        y[d1] = x[d1] * t.x + x[d0] * t.y;
      } else {
        y[half + i] = x[half + i];
      }
    }
  }
  // the rotated part of every head's query, in place: one thread per pair
  float* q = a.q + (long long)r * a.ldq;
  const int per = a.dim + a.rot_dim;
  for (int p = tid; p < a.heads * half; p += blockDim.x) {
    float* x = q + (p / half) * per + a.dim;
    const int i = p % half;
    const int d0 = a.rot_layout == LP_ROT_INTERLEAVED ? 2 * i : i;
    const int d1 = a.rot_layout == LP_ROT_INTERLEAVED ? 2 * i + 1 : i + half;
    const float2 t = turn(i);
    const float u = x[d0] * t.x - x[d1] * t.y, v = x[d1] * t.x + x[d0] * t.y;
    x[d0] = u;
    x[d1] = v;
  }
}

// One CTA per (row, head): its W warps take every W-th visible key with an online softmax of their own, then the partial (maximum,
// denominator, weighted sum) triples are merged.  A lane holds pieces of V channels, every 32nd (NP pieces of the latent; V = 4 where cache rows are whole
// 16-byte pieces), and LAT_KEYS keys are in flight at a time: their score reductions overlap, one rescale of the running sums serves them all.
// With a channel a load and two keys in flight 8 rows of 16 heads over 150 keys took 18.5 us, 64 rows of 8 heads over 40 keys (which had a warp a row and head) 34.
constexpr int LAT_KEYS = 4;
constexpr int LAT_SPLIT_MAX_RANK = 512;      // larger latents take the per-row kernel
constexpr int LAT_MAX_RANK = 1024;
template <int V> struct LatVec;
template <> struct LatVec<1> { float v[1]; };
template <> struct alignas(16) LatVec<4> { float v[4]; };
template <int V, int NP, int W>
__global__ void __launch_bounds__(W * 32)
latent_attend_kernel(LatArgs a, int R, const int* __restrict__ row_seq, const int* __restrict__ row_pos, const float* q_abs,
                     long long ldqa, void* __restrict__ out, long long ldo, int out_fp32) {
  pdl_launch_next_of_few();
  pdl_wait();
  __align__(16) __shared__ float s_acc[W][32 * V * NP];
  __shared__ float s_mx[W], s_den[W];
  constexpr int NR = V == 4 ? 1 : NP;      // pieces of the rotated part
  const int item = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (item >= R * a.heads) return;
  const int r = item / a.heads, h = item % a.heads;
  const int seq = row_seq[r], pos = row_pos[r];
  const float* qa = q_abs + (long long)r * ldqa + (long long)h * a.kv_rank;
  const float* qr = a.q + (long long)r * a.ldq + (long long)h * (a.dim + a.rot_dim) + a.dim;
  LatVec<V> qv[NP], qrv[NR], acc[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i)
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int c = V * (lane + 32 * i) + k;
      qv[i].v[k] = c < a.kv_rank ? qa[c] : 0.f;
      acc[i].v[k] = 0.f;
    }
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int c = V * (lane + 32 * i) + k;
      qrv[i].v[k] = c < a.rot_dim ? qr[c] : 0.f;      // rot_dim <= 32 V NR (checked by the host)
    }
  const int lo = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
  // the sink is a key without a value whose score is sink_h as it stands: warp 0 starts from it
  const bool sunk = a.sink != nullptr && warp == 0;
  float mx = sunk ? a.sink[h] : -INFINITY, den = sunk ? 1.f : 0.f;
  for (int j = lo + warp; j <= pos; j += LAT_KEYS * W) {
    LatVec<V> cv[LAT_KEYS][NP];
    float sc[LAT_KEYS];
    const float* kv[LAT_KEYS];
#pragma unroll
    for (int n = 0; n < LAT_KEYS; ++n) kv[n] = lat_cache_row(a, seq, j + n * W <= pos ? j + n * W : j);
#pragma unroll
    for (int n = 0; n < LAT_KEYS; ++n) {
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const int c = V * (lane + 32 * i);
        if (c < a.kv_rank) {
          cv[n][i] = *reinterpret_cast<const LatVec<V>*>(kv[n] + c);
        } else {
#pragma unroll
          for (int k = 0; k < V; ++k) cv[n][i].v[k] = 0.f;
        }
      }
    }
#pragma unroll
    for (int n = 0; n < LAT_KEYS; ++n) {
      sc[n] = 0.f;
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int c = V * (lane + 32 * i);
        if (c < a.rot_dim) {
          const LatVec<V> kr = *reinterpret_cast<const LatVec<V>*>(kv[n] + a.kv_rank + c);
#pragma unroll
          for (int k = 0; k < V; ++k) sc[n] = fmaf(qrv[i].v[k], kr.v[k], sc[n]);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < LAT_KEYS; ++n)
#pragma unroll
      for (int i = 0; i < NP; ++i)
#pragma unroll
        for (int k = 0; k < V; ++k) sc[n] = fmaf(qv[i].v[k], cv[n][i].v[k], sc[n]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int n = 0; n < LAT_KEYS; ++n) sc[n] += __shfl_xor_sync(0xffffffffu, sc[n], o);
    float mn = mx;
#pragma unroll
    for (int n = 0; n < LAT_KEYS; ++n) {
      sc[n] = j + n * W <= pos ? sc[n] * a.scale : -INFINITY;
      mn = fmaxf(mn, sc[n]);
    }
    const float corr = expf(mx - mn);      // exp(-inf) = 0 on the first turn
    den *= corr;
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
      for (int k = 0; k < V; ++k) acc[i].v[k] *= corr;
#pragma unroll
    for (int n = 0; n < LAT_KEYS; ++n) {
      if (j + n * W > pos) break;
      const float p = expf(sc[n] - mn);
      den += p;
#pragma unroll
      for (int i = 0; i < NP; ++i)
#pragma unroll
        for (int k = 0; k < V; ++k) acc[i].v[k] = fmaf(p, cv[n][i].v[k], acc[i].v[k]);
    }
    mx = mn;
  }
#pragma unroll
  for (int i = 0; i < NP; ++i) *reinterpret_cast<LatVec<V>*>(&s_acc[warp][V * (lane + 32 * i)]) = acc[i];
  if (lane == 0) {
    s_mx[warp] = mx;
    s_den[warp] = den;
  }
  __syncthreads();
  float top = s_mx[0];
#pragma unroll
  for (int w = 1; w < W; ++w) top = fmaxf(top, s_mx[w]);
  float f[W], total = 0.f;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    f[w] = s_den[w] > 0.f ? expf(s_mx[w] - top) : 0.f;      // a warp without keys contributes nothing
    total = fmaf(s_den[w], f[w], total);
  }
  const float inv = lat_gate(a, r, h) / total;
  for (int c = threadIdx.x; c < a.kv_rank; c += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) v = fmaf(s_acc[w][c], f[w], v);
    const long long o = (long long)r * ldo + (long long)h * a.kv_rank + c;
    if (out_fp32) reinterpret_cast<float*>(out)[o] = v * inv;
    else reinterpret_cast<bf16*>(out)[o] = __float2bfloat16(v * inv);
  }
}

// Many rows (prompts): one CTA per row and group of LAT_ROW_HEADS heads, one warp per head, every warp walks all visible keys.
// The heads of a row read the same cache rows at about the same time, so the cache traffic of a row is paid once per CTA (L1), and
// neighbouring rows overlap in all but one key (L2).
// Up to LAT_SPLIT_ROWS rows latent_attend_kernel splits a row's keys over warps (us, this kernel and that one): 17 rows of 8 heads over 40 keys 37, 10; 128 over 40 38, 21, over
// 300 233, 80; 16 heads 39, 37 and 225, 164.  Beyond it that one is ahead as well (192 rows of 8 heads over 300 keys 238, 88; 512 over 40 44, 45): the line was not moved.
constexpr int LAT_ROW_HEADS = 4, LAT_SPLIT_ROWS = 128;
template <int NR>
__global__ void __launch_bounds__(LAT_ROW_HEADS * 32)
latent_attend_rows_kernel(LatArgs a, int R, const int* __restrict__ row_seq, const int* __restrict__ row_pos, const float* q_abs,
                          long long ldqa, void* __restrict__ out, long long ldo, int out_fp32) {
  pdl_launch_next_of_few();
  pdl_wait();
  const int r = blockIdx.x;
  const int h = blockIdx.y * LAT_ROW_HEADS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= R || h >= a.heads) return;
  const int seq = row_seq[r], pos = row_pos[r];
  const float* qa = q_abs + (long long)r * ldqa + (long long)h * a.kv_rank;
  const float* qr = a.q + (long long)r * a.ldq + (long long)h * (a.dim + a.rot_dim) + a.dim;
  float qv[NR], qrv[NR], acc[NR];
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int c = lane + 32 * i;
    qv[i] = c < a.kv_rank ? qa[c] : 0.f;
    qrv[i] = c < a.rot_dim ? qr[c] : 0.f;
    acc[i] = 0.f;
  }
  const int lo = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
  float mx = a.sink != nullptr ? a.sink[h] : -INFINITY, den = a.sink != nullptr ? 1.f : 0.f;
  // two keys per turn: their score reductions overlap, one rescale of the running sums serves both
  for (int j = lo; j <= pos; j += 2 * 1) {
    const bool two = j + 1 <= pos;
    const float* kv0 = lat_cache_row(a, seq, j);
    const float* kv1 = two ? lat_cache_row(a, seq, j + 1) : kv0;
    float cv0[NR], cv1[NR];
    float sc0 = 0.f, sc1 = 0.f;
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int c = lane + 32 * i;
      cv0[i] = c < a.kv_rank ? kv0[c] : 0.f;
      cv1[i] = c < a.kv_rank ? kv1[c] : 0.f;
      sc0 = fmaf(qv[i], cv0[i], sc0);
      sc1 = fmaf(qv[i], cv1[i], sc1);
      if (c < a.rot_dim) {
        sc0 = fmaf(qrv[i], kv0[a.kv_rank + c], sc0);
        sc1 = fmaf(qrv[i], kv1[a.kv_rank + c], sc1);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sc0 += __shfl_xor_sync(0xffffffffu, sc0, o);
      sc1 += __shfl_xor_sync(0xffffffffu, sc1, o);
    }
    sc0 *= a.scale;
    sc1 = two ? sc1 * a.scale : -INFINITY;
    const float mn = fmaxf(mx, fmaxf(sc0, sc1));
    const float corr = expf(mx - mn);      // exp(-inf) = 0 on the first turn
    const float p0 = expf(sc0 - mn), p1 = expf(sc1 - mn);
    den = den * corr + p0 + p1;
#pragma unroll
    for (int i = 0; i < NR; ++i) acc[i] = fmaf(p1, cv1[i], fmaf(p0, cv0[i], acc[i] * corr));
    mx = mn;
  }
  const float inv = lat_gate(a, r, h) / den;
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int c = lane + 32 * i;
    if (c < a.kv_rank) {
      const long long o = (long long)r * ldo + (long long)h * a.kv_rank + c;
      if (out_fp32) reinterpret_cast<float*>(out)[o] = acc[i] * inv;
      else reinterpret_cast<bf16*>(out)[o] = __float2bfloat16(acc[i] * inv);
    }
  }
}

// Prompts, tiled, where heads are not those that lp_latent_attend_expanded takes or requests bring a few rows each: a CTA takes LT_X = 64 (row, head) pairs of one request's chunk — all heads read the same latents, so the pairs share
// every key — and walks the union of what its rows see, LT_K = 16 keys at a time; every pair is masked by its row's own rule.  Both halves
// are register-tiled fp32 products fed from shared memory: scores 4 pairs x 2 keys a thread with two lanes splitting the channels, sums
// 8 pairs x (4 NC) latent channels a thread (NC = ceil(kv_rank / 128)).  The next tile of keys is copied in (cp.async) while this one is
// worked on.  Rows in shared memory are LD floats apart, LD = 8 mod 32, so that the 8 sixteen-byte pieces a score load of a warp touches
// lie in different banks; the padding is zero and takes part in the sums.
constexpr int LT_X = 64, LT_K = 16, LT_THREADS = 256, LT_PS = LT_X + 4, LT_MAX_NC = 4;
static int lt_ld(int width) { return (width + 23) / 32 * 32 + 8; }      // the smallest number >= width that is 8 mod 32
static size_t lt_smem_floats(int width) { return (size_t)(LT_X + 2 * LT_K) * lt_ld(width) + LT_K * LT_PS + LT_X; }

template <int NC>
__global__ void __launch_bounds__(LT_THREADS)
latent_attend_tile_kernel(LatArgs a, int ld, int n_chunks, const int* __restrict__ chunk_seq, const int* __restrict__ chunk_row0,
                          const int* __restrict__ chunk_len, int tiles_per_chunk, const int* __restrict__ row_pos,
                          const float* __restrict__ q_abs, long long ldqa, void* __restrict__ out, long long ldo, int out_fp32) {
  extern __shared__ float dyn_smem[];
  const int ck = blockIdx.x / tiles_per_chunk, v0 = (blockIdx.x % tiles_per_chunk) * LT_X;
  const int H = a.heads, C = a.kv_rank, width = a.kv_rank + a.rot_dim;
  if (ck >= n_chunks || v0 >= chunk_len[ck] * H) return;
  const int nv = min(LT_X, chunk_len[ck] * H - v0);      // pairs of this tile: pair x is row (v0 + x) / H, head (v0 + x) % H
  const int r0 = chunk_row0[ck], seq = chunk_seq[ck];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* q_s = dyn_smem;                        // [LT_X][ld]
  float* k_s = q_s + LT_X * ld;                 // [2][LT_K][ld]
  float* p_s = k_s + 2 * LT_K * ld;             // [LT_K][LT_PS] scores, then weights
  float* corr_s = p_s + LT_K * LT_PS;           // [LT_X] what the running sums are multiplied by
  for (int i = tid; i < LT_X * ld; i += LT_THREADS) {
    const int x = i / ld, d = i % ld;
    float v = 0.f;
    if (x < nv && d < width) {
      const long long r = r0 + (v0 + x) / H;
      const int h = (v0 + x) % H;
      v = d < C ? q_abs[r * ldqa + (long long)h * C + d] : a.q[r * a.ldq + (long long)h * (a.dim + a.rot_dim) + a.dim + (d - C)];
    }
    q_s[i] = v;
  }
  for (int i = tid; i < 2 * LT_K * ld; i += LT_THREADS) k_s[i] = 0.f;      // padding, and keys past the end (their weight is zero)
  const int pos_first = row_pos[r0 + v0 / H], pos_last = row_pos[r0 + (v0 + nv - 1) / H];
  const int lo = (a.window > 0 && pos_first - a.window + 1 > 0) ? pos_first - a.window + 1 : 0;
  const int n_keys = pos_last - lo + 1, pieces = width >> 2, steps = (pieces + 1) & ~1;
  auto load = [&](int t0, float* dst) {
    for (int j = warp; j < LT_K; j += LT_THREADS / 32) {
      if (t0 + j >= n_keys) break;
      const float* src = lat_cache_row(a, seq, lo + t0 + j);
      for (int p = lane; p < pieces; p += 32) __pipeline_memcpy_async(dst + j * ld + 4 * p, src + 4 * p, 16);
    }
    __pipeline_commit();
  };
  // the pair whose softmax this thread keeps, together with the three lanes beside it
  const int sx = tid >> 2, part = tid & 3;
  const int my_pos = sx < nv ? row_pos[r0 + (v0 + sx) / H] : -1;
  const int my_lo = sx < nv ? ((a.window > 0 && my_pos - a.window + 1 > 0) ? my_pos - a.window + 1 : 0) : 0x7fffffff;
  const int my_h = (v0 + sx) % H;
  float mx = a.sink != nullptr ? a.sink[my_h] : -INFINITY, den = a.sink != nullptr ? 1.f : 0.f;
  const int sl = lane & 1, x_at = (warp & 3) * 16 + ((lane >> 1) & 3), k_at = (warp >> 2) * 8 + (lane >> 3);
  float acc[8][4 * NC];
#pragma unroll
  for (int x = 0; x < 8; ++x)
#pragma unroll
    for (int i = 0; i < 4 * NC; ++i) acc[x][i] = 0.f;
  __syncthreads();
  load(0, k_s);
  for (int t0 = 0; t0 < n_keys; t0 += LT_K) {
    const float* kt = k_s + ((t0 / LT_K) & 1) * LT_K * ld;
    __pipeline_wait_prior(0);
    __syncthreads();      // the tile is here for everyone, and nobody reads the other buffer or the weights any more
    if (t0 + LT_K < n_keys) load(t0 + LT_K, k_s + ((t0 / LT_K + 1) & 1) * LT_K * ld);
    {
      float s[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = 0.f;
      const float* qp = q_s + x_at * ld + 4 * sl;
      const float* kp = kt + k_at * ld + 4 * sl;
#pragma unroll 4
      for (int g = 0; g < steps; g += 2) {
        float4 k4[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) k4[j] = *reinterpret_cast<const float4*>(kp + 4 * j * ld + 4 * g);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 q4 = *reinterpret_cast<const float4*>(qp + 4 * i * ld + 4 * g);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            s[i][j] = fmaf(q4.x, k4[j].x, s[i][j]);
            s[i][j] = fmaf(q4.y, k4[j].y, s[i][j]);
            s[i][j] = fmaf(q4.z, k4[j].z, s[i][j]);
            s[i][j] = fmaf(q4.w, k4[j].w, s[i][j]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 2; ++j) s[i][j] += __shfl_xor_sync(0xffffffffu, s[i][j], 1);
        p_s[(k_at + 4 * sl) * LT_PS + x_at + 4 * i] = sl ? s[i][1] : s[i][0];
      }
    }
    __syncthreads();
    {
      float v[LT_K / 4], top = -INFINITY;
#pragma unroll
      for (int j = 0; j < LT_K / 4; ++j) {
        const int key = part * (LT_K / 4) + j, at = lo + t0 + key;
        v[j] = (at >= my_lo && at <= my_pos) ? p_s[key * LT_PS + sx] * a.scale : -INFINITY;
        top = fmaxf(top, v[j]);
      }
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
      const float mn = fmaxf(mx, top), ref = mn == -INFINITY ? 0.f : mn;      // -inf: this pair has seen nothing yet
      const float corr = expf(mx - ref);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < LT_K / 4; ++j) {
        const float p = expf(v[j] - ref);
        p_s[(part * (LT_K / 4) + j) * LT_PS + sx] = p;
        sum += p;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      den = fmaf(den, corr, sum);
      mx = mn;
      if (part == 0) corr_s[sx] = corr;
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const float c = corr_s[warp * 8 + x];      // the same for the whole warp
      if (c != 1.f) {
#pragma unroll
        for (int i = 0; i < 4 * NC; ++i) acc[x][i] *= c;
      }
    }
    const float* wp = p_s + warp * 8;
    const float* cp = kt + 4 * lane;
#pragma unroll 2
    for (int jj = 0; jj < LT_K; ++jj) {
      const float4 w0 = *reinterpret_cast<const float4*>(wp + jj * LT_PS), w1 = *reinterpret_cast<const float4*>(wp + jj * LT_PS + 4);
      const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        if (4 * lane + 128 * i < C) {
          const float4 c4 = *reinterpret_cast<const float4*>(cp + jj * ld + 128 * i);
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            acc[x][4 * i] = fmaf(w[x], c4.x, acc[x][4 * i]);
            acc[x][4 * i + 1] = fmaf(w[x], c4.y, acc[x][4 * i + 1]);
            acc[x][4 * i + 2] = fmaf(w[x], c4.z, acc[x][4 * i + 2]);
            acc[x][4 * i + 3] = fmaf(w[x], c4.w, acc[x][4 * i + 3]);
          }
        }
      }
    }
  }
  __syncthreads();
  if (part == 0) corr_s[sx] = sx < nv ? lat_gate(a, r0 + (v0 + sx) / H, my_h) / den : 0.f;
  __syncthreads();
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    const int v = v0 + warp * 8 + x;
    if (warp * 8 + x >= nv) break;
    const float f = corr_s[warp * 8 + x];
    const long long at = (long long)(r0 + v / H) * ldo + (long long)(v % H) * C + 4 * lane;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      if (4 * lane + 128 * i < C) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (out_fp32) reinterpret_cast<float*>(out)[at + 128 * i + k] = acc[x][4 * i + k] * f;
          else reinterpret_cast<bf16*>(out)[at + 128 * i + k] = __float2bfloat16(acc[x][4 * i + k] * f);
        }
      }
    }
  }
}

// raise a kernel's dynamic shared-memory limit only when a launch needs more than any launch before it (no runtime call on the
// steady path, so the steady path can be captured into a CUDA graph)
template <typename K>
static cudaError_t ensure_smem(K kern, size_t bytes, size_t& have) {
  if (bytes <= have) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) have = bytes;
  return e;
}

static int fill_ret(RetArgs& a, const lp_retention_desc* d) {
  LP_REQUIRE(d != nullptr && d->qkvg != nullptr && d->decay != nullptr && d->state != nullptr && d->out != nullptr,
             "lp_retention: null operand");
  LP_REQUIRE(d->heads > 0 && d->dim > 0 && d->vdim > 0, "lp_retention: bad sizes heads=%d dim=%d vdim=%d", d->heads, d->dim, d->vdim);
  LP_REQUIRE(d->rot_dims >= 0 && d->rot_dims <= d->dim && d->rot_dims % 2 == 0, "lp_retention: rot_dims=%d must be even and <= dim=%d",
             d->rot_dims, d->dim);
  LP_REQUIRE(d->rot_dims == 0 || d->inv_freq != nullptr, "lp_retention: rotation without a frequency table");
  a.qkvg = d->qkvg; a.ld = d->ld; a.q_off = d->q_off; a.k_off = d->k_off; a.v_off = d->v_off; a.g_off = d->g_off;
  a.heads = d->heads; a.dim = d->dim; a.vdim = d->vdim;
  a.decay = d->decay;
  a.inv_freq = d->inv_freq; a.rot_dims = d->rot_dims; a.rot_layout = d->rot_layout; a.rot_mscale = d->rot_mscale;
  a.k_scale = d->k_scale; a.eps = d->eps;
  a.in_act = d->in_act; a.finish = d->finish;
  LP_REQUIRE(d->in_act == 0 || d->rot_dims == 0, "lp_retention: an input activation together with rotation is not supported");
  LP_REQUIRE(d->finish == LP_RET_FINISH_GATED_NORM || d->finish == LP_RET_FINISH_RAW, "lp_retention: bad finish %d", d->finish);
  a.state = d->state; a.slot_stride = d->slot_stride;
  a.out = d->out; a.ldo = d->ldo; a.out_fp32 = d->out_fp32;
  return 0;
}

static int fill_lat(LatArgs& a, const lp_latent_desc* d) {
  LP_REQUIRE(d != nullptr && d->q != nullptr && d->cache != nullptr && d->page_table != nullptr, "lp_latent: null operand");
  LP_REQUIRE(d->heads > 0 && d->dim >= 0 && d->rot_dim >= 0 && d->kv_rank > 0 && d->page_size > 0 && d->max_pages > 0,
             "lp_latent: bad sizes");
  LP_REQUIRE(d->rot_dims >= 0 && d->rot_dims <= d->rot_dim && d->rot_dims % 2 == 0, "lp_latent: rot_dims=%d must be even and <= rot_dim=%d",
             d->rot_dims, d->rot_dim);
  LP_REQUIRE(d->rot_dims == 0 || d->inv_freq != nullptr, "lp_latent: rotation without a frequency table");
  a.q = d->q; a.ldq = d->ldq; a.dkv = d->dkv; a.lddkv = d->lddkv;
  a.heads = d->heads; a.dim = d->dim; a.rot_dim = d->rot_dim; a.kv_rank = d->kv_rank;
  a.c_gain = d->c_gain; a.eps = d->eps;
  a.inv_freq = d->inv_freq; a.rot_dims = d->rot_dims; a.rot_layout = d->rot_layout; a.rot_mscale = d->rot_mscale;
  a.cache = d->cache; a.page_size = d->page_size; a.page_table = d->page_table; a.max_pages = d->max_pages;
  a.window = d->window; a.scale = d->scale;
  a.sink = d->sink; a.gate = d->gate; a.ldg = d->ldg;
  return 0;
}

}  // namespace lp

using namespace lp;

extern "C" size_t lp_retention_workspace_bytes(int n_chunks, int heads, int dim, int vdim) {
  return (size_t)n_chunks * heads * dim * vdim * sizeof(float);
}

template <bool WIDE, bool MM>
static int launch_ret_prefill(const RetArgs& a, int n_seqs, int n_chunks, const int* seq_row0, const int* seq_pos0, const int* seq_slot, const int* seq_chunk0,
                              const int* chunk_seq, const int* chunk_row0, const int* chunk_len, float* w, cudaStream_t stream) {
  static size_t have_out = 48 * 1024, have_state = 48 * 1024;
  const size_t dimp = MM ? ret_mm_dimp(a.dim) : ret_dimp<WIDE>(a.dim), vdimp = (a.vdim + 3) & ~3;
  const size_t smem1 = (size_t)RET_CHUNK * (MM ? a.dim + a.vdim + 16 : ret_dimp<false>(a.dim) + vdimp) * sizeof(float);
  size_t smem3 = ((size_t)RET_CHUNK * (2 * dimp + 2 * vdimp) + RET_CHUNK * (RET_CHUNK + 1) + RET_CHUNK) * sizeof(float);
  LP_REQUIRE(smem3 <= 200 * 1024, "lp_retention_prefill: dim=%d vdim=%d do not fit the chunk kernel's shared memory", a.dim, a.vdim);
  const int stage_s = smem3 + (size_t)a.dim * vdimp * sizeof(float) <= 64 * 1024;      // three CTAs an SM keep their operands and the chunk's start state
  if (stage_s) smem3 += (size_t)a.dim * vdimp * sizeof(float);
  LP_CHECK_CUDA(ensure_smem(retention_chunk_state_kernel<MM>, smem1, have_state));
  LP_CHECK_CUDA((ensure_smem(retention_chunk_out_kernel<WIDE, MM>, smem3, have_out)));
  LP_CHECK_CUDA(launch_next(retention_chunk_state_kernel<MM>, dim3(n_chunks, a.heads), dim3(RET_CHUNK_THREADS), smem1, stream, a, chunk_seq, chunk_row0, chunk_len, seq_row0, seq_pos0, w));
  LP_CHECK_CUDA(cudaGetLastError());
  constexpr int V = WIDE ? 4 : 1;
  LP_CHECK_CUDA(launch_next(retention_scan_kernel<V>, dim3(n_seqs, a.heads, (a.dim * a.vdim / V + SCAN_THREADS - 1) / SCAN_THREADS), dim3(SCAN_THREADS), 0, stream, 
      a, seq_chunk0, chunk_len, seq_pos0, seq_slot, w));
  LP_CHECK_CUDA(cudaGetLastError());
  LP_CHECK_CUDA((launch_next(retention_chunk_out_kernel<WIDE, MM>, dim3(n_chunks, a.heads), dim3(RET_CHUNK_THREADS), smem3, stream, a, chunk_seq, chunk_row0, chunk_len, seq_row0,
                             seq_pos0, w, stage_s)));
  LP_CHECK_CUDA(cudaGetLastError());
  note_launch(3);
  return 0;
}

extern "C" int lp_retention_prefill(const lp_retention_desc* d, int n_seqs, int n_chunks, const int* seq_row0, const int* seq_pos0,
                                    const int* seq_slot, const int* seq_chunk0, const int* chunk_seq, const int* chunk_row0,
                                    const int* chunk_len, void* ws, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  RetArgs a;
  if (int rc = fill_ret(a, d)) return rc;
  LP_REQUIRE(n_seqs >= 0 && n_chunks >= 0, "lp_retention_prefill: bad counts");
  if (n_seqs == 0 || n_chunks == 0) return 0;
  LP_REQUIRE(ws != nullptr && ws_bytes >= lp_retention_workspace_bytes(n_chunks, d->heads, d->dim, d->vdim),
             "lp_retention_prefill: workspace too small");
  float* w = reinterpret_cast<float*>(ws);
  // 16-byte pieces of the operands, the state and the workspace; the wider padding has to fit too
  const bool wide = d->dim % 8 == 0 && d->vdim % 8 == 0 && d->slot_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(d->state) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(ws) & 15) == 0 && ((size_t)RET_CHUNK * 2 * (d->dim + 4 + d->vdim) + RET_CHUNK * (RET_CHUNK + 2)) * sizeof(float) <= 200 * 1024;
  // whole 128s: every warp of both kernels has a tile; narrower heads would leave half of them without (and stay on the fp32 sums)
  const bool mm = wide && d->dim % RET_MM == 0 && d->vdim % RET_MM == 0 &&
                  ((size_t)RET_CHUNK * 2 * (ret_mm_dimp(d->dim) + d->vdim) + RET_CHUNK * (RET_CHUNK + 2)) * sizeof(float) <= 200 * 1024;
  if (mm)
    return launch_ret_prefill<true, true>(a, n_seqs, n_chunks, seq_row0, seq_pos0, seq_slot, seq_chunk0, chunk_seq, chunk_row0, chunk_len, w, stream);
  return wide ? launch_ret_prefill<true, false>(a, n_seqs, n_chunks, seq_row0, seq_pos0, seq_slot, seq_chunk0, chunk_seq, chunk_row0, chunk_len, w, stream)
              : launch_ret_prefill<false, false>(a, n_seqs, n_chunks, seq_row0, seq_pos0, seq_slot, seq_chunk0, chunk_seq, chunk_row0, chunk_len, w, stream);
}

template <int V>
static int launch_ret_decode(const RetArgs& a, int n_seqs, const int* seq_row0, const int* seq_pos0, const int* seq_slot, cudaStream_t stream) {
  static size_t have = 48 * 1024;
  const size_t smem = ((size_t)2 * a.dim + 2 * a.vdim + (size_t)ret_dec_groups<V>(a.vdim) * a.vdim) * sizeof(float);
  LP_REQUIRE(smem <= 200 * 1024, "lp_retention_decode: dim=%d vdim=%d do not fit shared memory", a.dim, a.vdim);
  LP_CHECK_CUDA(ensure_smem(retention_decode_kernel<V>, smem, have));
  // not before the launch before has ended: CTAs that are placed beside it lie on fewer SMs, whose loads then take longer (a step of 8 requests of 16 heads 1.3 % of its time;
  // 18 requests of 8 heads, launch after launch, 6.7 us, so 5.4)
  LP_CHECK_CUDA(launch_ex(retention_decode_kernel<V>, dim3(n_seqs, a.heads), dim3(RET_DEC_THREADS), smem, stream, 1, false, a, seq_row0, seq_pos0, seq_slot));
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int lp_retention_decode(const lp_retention_desc* d, int n_seqs, const int* seq_row0, const int* seq_pos0, const int* seq_slot,
                                   void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  RetArgs a;
  if (int rc = fill_ret(a, d)) return rc;
  if (n_seqs <= 0) return 0;
  const bool pieces = d->vdim % 4 == 0 && d->slot_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(d->state) & 15) == 0;
  return pieces ? launch_ret_decode<4>(a, n_seqs, seq_row0, seq_pos0, seq_slot, stream) : launch_ret_decode<1>(a, n_seqs, seq_row0, seq_pos0, seq_slot, stream);
}

extern "C" int lp_latent_prep(const lp_latent_desc* d, int R, const int* row_seq, const int* row_pos, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LatArgs a;
  if (int rc = fill_lat(a, d)) return rc;
  LP_REQUIRE((d->dkv == nullptr || d->c_gain != nullptr) && row_seq != nullptr && row_pos != nullptr, "lp_latent_prep: null operand");
  if (R <= 0) return 0;
  const size_t smem = d->rot_dims / 2 <= LAT_PREP_PAIRS ? d->rot_dims / 2 * sizeof(float2) : 0;
  LP_CHECK_CUDA(launch_next(latent_prep_kernel, dim3(R), dim3(R <= 2 * sm_count() ? LAT_PREP_WIDE : LAT_PREP_THREADS), smem, stream, a, R, row_seq, row_pos));
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int lp_latent_attend(const lp_latent_desc* d, int R, const int* row_seq, const int* row_pos, const float* q_abs, long long ldqa,
                                void* out, long long ldo, int out_fp32, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LatArgs a;
  if (int rc = fill_lat(a, d)) return rc;
  LP_REQUIRE(q_abs != nullptr && out != nullptr && row_seq != nullptr && row_pos != nullptr, "lp_latent_attend: null operand");
  LP_REQUIRE(d->kv_rank <= LAT_MAX_RANK && d->rot_dim <= LAT_MAX_RANK, "lp_latent_attend: kv_rank=%d / rot_dim=%d > %d is not instantiated",
             d->kv_rank, d->rot_dim, LAT_MAX_RANK);
  if (R <= 0) return 0;
  const long long pages = (long long)d->max_pages * d->page_size, work = (long long)R * d->heads * (d->window > 0 && d->window < pages ? d->window : pages);
  const int nr = ((d->kv_rank > d->rot_dim ? d->kv_rank : d->rot_dim) + 31) / 32;      // lanes hold both vectors strided by 32
  if (R > LAT_SPLIT_ROWS || d->kv_rank > LAT_SPLIT_MAX_RANK || d->rot_dim > LAT_SPLIT_MAX_RANK) {      // prompts: a CTA per row, a warp per head
    const dim3 grid(R, (d->heads + LAT_ROW_HEADS - 1) / LAT_ROW_HEADS);
    const int threads = (d->heads < LAT_ROW_HEADS ? d->heads : LAT_ROW_HEADS) * 32;
    if (nr <= 2) LP_CHECK_CUDA(launch_attention(work, latent_attend_rows_kernel<2>, grid, dim3(threads), 0, stream, a, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32));
    else if (nr <= 4) LP_CHECK_CUDA(launch_attention(work, latent_attend_rows_kernel<4>, grid, dim3(threads), 0, stream, a, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32));
    else if (nr <= 8) LP_CHECK_CUDA(launch_attention(work, latent_attend_rows_kernel<8>, grid, dim3(threads), 0, stream, a, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32));
    else if (nr <= 16) LP_CHECK_CUDA(launch_attention(work, latent_attend_rows_kernel<16>, grid, dim3(threads), 0, stream, a, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32));
    else LP_CHECK_CUDA(launch_attention(work, latent_attend_rows_kernel<32>, grid, dim3(threads), 0, stream, a, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32));
  } else {      // decoding: a CTA per (row, head), its warps split the keys
    const long long ctas = (long long)R * d->heads;
    const bool pieces = d->kv_rank % 4 == 0 && d->rot_dim % 4 == 0 && d->rot_dim <= 128 && (reinterpret_cast<uintptr_t>(d->cache) & 15) == 0;
#define LP_LAT(V, NP)                                                                                                                       \
  do {                                                                                                                                      \
    if (ctas <= 2LL * sm_count()) LP_CHECK_CUDA((launch_attention(work, latent_attend_kernel<V, NP, 16>, dim3((unsigned)ctas), dim3(16 * 32), 0, stream, a, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32)));    \
    else LP_CHECK_CUDA((launch_attention(work, latent_attend_kernel<V, NP, 4>, dim3((unsigned)ctas), dim3(4 * 32), 0, stream, a, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32)));     \
  } while (0)
    if (pieces) {
      const int np = (d->kv_rank + 127) / 128;
      if (np <= 1) LP_LAT(4, 1);
      else if (np <= 2) LP_LAT(4, 2);
      else LP_LAT(4, 4);
    } else {
      if (nr <= 4) LP_LAT(1, 4);
      else LP_LAT(1, 16);
    }
#undef LP_LAT
  }
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

template <int NC>
static int launch_latent_tiles(const LatArgs& a, int R, int n_chunks, const int* chunk_seq, const int* chunk_row0, const int* chunk_len,
                               const int* row_pos, const float* q_abs, long long ldqa, void* out, long long ldo, int out_fp32, cudaStream_t stream) {
  static size_t have = 48 * 1024;
  const int width = a.kv_rank + a.rot_dim;
  const size_t smem = lt_smem_floats(width) * sizeof(float);
  LP_CHECK_CUDA(ensure_smem(latent_attend_tile_kernel<NC>, smem, have));
  const int longest = R < LP_RETENTION_CHUNK ? R : LP_RETENTION_CHUNK;      // no chunk has more rows than the step or the chunk size
  const int tiles = (longest * a.heads + LT_X - 1) / LT_X;
  latent_attend_tile_kernel<NC><<<n_chunks * tiles, LT_THREADS, smem, stream>>>(a, lt_ld(width), n_chunks, chunk_seq, chunk_row0, chunk_len, tiles,
                                                                                row_pos, q_abs, ldqa, out, ldo, out_fp32);
  note_launch();
  LP_CHECK_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int lp_latent_attend_tiles(const lp_latent_desc* d, int R, const int* row_seq, const int* row_pos, int n_chunks,
                                      const int* chunk_seq, const int* chunk_row0, const int* chunk_len, const float* q_abs, long long ldqa,
                                      void* out, long long ldo, int out_fp32, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LatArgs a;
  if (int rc = fill_lat(a, d)) return rc;
  LP_REQUIRE(q_abs != nullptr && out != nullptr && row_seq != nullptr && row_pos != nullptr && chunk_seq != nullptr && chunk_row0 != nullptr &&
                 chunk_len != nullptr,
             "lp_latent_attend_tiles: null operand");
  if (R <= 0 || n_chunks <= 0) return 0;
  const int width = d->kv_rank + d->rot_dim, nc = (d->kv_rank + 127) / 128;
  // 16-byte pieces of the cache rows, all of a pair's sums in registers, both operands in shared memory; few rows are split over keys
  if (R <= LP_LATENT_SPLIT_ROWS || d->kv_rank % 4 || d->rot_dim % 4 || nc > LT_MAX_NC || lt_smem_floats(width) * sizeof(float) > 227 * 1024 ||
      (reinterpret_cast<uintptr_t>(d->cache) & 15))
    return lp_latent_attend(d, R, row_seq, row_pos, q_abs, ldqa, out, ldo, out_fp32, stream_);
  if (nc == 1) return launch_latent_tiles<1>(a, R, n_chunks, chunk_seq, chunk_row0, chunk_len, row_pos, q_abs, ldqa, out, ldo, out_fp32, stream);
  if (nc == 2) return launch_latent_tiles<2>(a, R, n_chunks, chunk_seq, chunk_row0, chunk_len, row_pos, q_abs, ldqa, out, ldo, out_fp32, stream);
  if (nc == 3) return launch_latent_tiles<3>(a, R, n_chunks, chunk_seq, chunk_row0, chunk_len, row_pos, q_abs, ldqa, out, ldo, out_fp32, stream);
  return launch_latent_tiles<4>(a, R, n_chunks, chunk_seq, chunk_row0, chunk_len, row_pos, q_abs, ldqa, out, ldo, out_fp32, stream);
}

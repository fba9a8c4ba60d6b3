// Test infrastructure: runs the kernels of leopard_b200/csrc/lp_split32.cu on the CPU under tests/emu/tc_emu.h.
#define LP_EMULATE 1
#include <atomic>
// a thread's registers as the kernels split them, and what the CTA was about when results were first taken again one by one
static thread_local int emu_registers = 0;
static std::atomic<int> emu_fewest_registers{1 << 20};
static std::atomic<long> emu_first_serial{-1};
static void emu_serial();
#include "../../leopard_b200/csrc/lp_split32.cu"

using namespace lp;

static void emu_serial() {
  for (int had = emu_fewest_registers; emu_registers < had && !emu_fewest_registers.compare_exchange_weak(had, emu_registers);) {
  }
  long none = -1;
  emu_first_serial.compare_exchange_strong(none, emu_tc::g_issued);
}
// since the last call: the fewest registers that a thread had when it took results again; MMAs that had been issued when the first one did (-1: none did), and in all
extern "C" void emu_serial_stats(int* registers, long* at_first, long* in_all) {
  *registers = emu_fewest_registers.exchange(1 << 20);
  *at_first = emu_first_serial.exchange(-1);
  *in_all = emu_tc::g_issued.exchange(0);
}

static CUtensorMap tmap3(const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t ld, uint64_t plane, uint32_t rows) {
  CUtensorMap m;
  m.base = reinterpret_cast<const uint8_t*>(base);
  m.dims[0] = d0; m.dims[1] = d1; m.dims[2] = d2;
  m.strides[0] = ld * 2; m.strides[1] = plane * 2;
  m.box[0] = 64; m.box[1] = rows; m.box[2] = 1;
  return m;
}

extern "C" void emu_split_rows(const float* src, long long ld, int M, int K, void* dst, long long ldd, long long plane) {
  emu::launch(dim3((unsigned)(((long long)M * (K / 8) + 255) / 256)), dim3(256), [&] { split_rows_kernel<false>(src, ld, M, K, (bf16*)dst, ldd, plane, Factor32{}); });
}

extern "C" void emu_gather_rows(const void* src, long long ld, int src_fp32, const int* row_of, int rows, int K, void* dst, long long plane) {
  emu::launch(dim3((unsigned)(((long long)rows * (K / 8) + 255) / 256)), dim3(256), [&] {
    if (src_fp32) gather_rows_kernel<true>(src, ld, row_of, rows, K, (bf16*)dst, plane);
    else gather_rows_kernel<false>(src, ld, row_of, rows, K, (bf16*)dst, plane);
  });
}

extern "C" void emu_gather_keys(int n_seqs, int window, int keep_first, int pool, const int* row0, const int* pos0, int n_keys, const float* cache,
                                int page_size, const int* table, int max_pages, const float* blocks, const int* block_table, int width, void* dst, long long plane) {
  Seqs32 q = {n_seqs, window, row0, pos0, 0, keep_first, pool};
  emu::launch(dim3((unsigned)(((long long)n_keys * (width / 8) + 255) / 256)), dim3(256),
              [&] { gather_keys_kernel(q, n_keys, cache, page_size, table, max_pages, blocks, block_table, max_pages, width, (bf16*)dst, plane); });
}

template <int BN, int PLANES, bool GATED>
static void run_gemm(Gemm32Args& a, int ctas, int groups, long long w_group) {
  a.n_tiles_m = (a.M + 127) / 128;
  a.n_tiles_n = (GATED ? (a.N / 2 + BN / 2 - 1) / (BN / 2) : (a.N + BN - 1) / BN);
  const CUtensorMap ta = tmap3(a.A, a.K, a.M, PLANES, a.lda, a.a_plane, 128), tw = tmap3(a.W, a.K, a.N, groups, a.ldw, w_group, GATED ? 64 : BN);
  emu::g_block_hook = [] { emu_tc::reset(); };
  emu::launch(dim3(ctas), dim3(G32_THREADS), [&] { gemm32_kernel<BN, PLANES, GATED>(ta, tw, a); });
  emu::g_block_hook = nullptr;
}

extern "C" void emu_gemm_split(const void* A, long long lda, long long a_plane, const void* W, long long ldw, void* C, long long ldc, long long c_plane,
                               int out, int M, int N, int K, const float* bias, int bn, int ctas) {
  Gemm32Args a = {};
  a.M = M; a.N = N; a.K = K; a.bias = bias; a.C = C; a.ldc = ldc; a.c_plane = c_plane; a.out = out;
  a.A = (const bf16*)A; a.lda = lda; a.a_plane = a_plane; a.W = (const bf16*)W; a.ldw = ldw;
  if (bn == 256) run_gemm<256, 3, false>(a, ctas, 1, 0);
  else run_gemm<128, 3, false>(a, ctas, 1, 0);
}

extern "C" void emu_gemm_grouped(const void* A, long long a_plane, const void* W, int groups, const int* tile_group, int n_tiles, int gated,
                                 const float* row_scale, void* C, long long c_plane, int out, int N, int K, int ctas) {
  Gemm32Args a = {};
  a.M = n_tiles * 128; a.N = N; a.K = K; a.C = C; a.ldc = gated ? N / 2 : N; a.out = out; a.c_plane = c_plane; a.w_group = (long long)N * K;
  a.A = (const bf16*)A; a.lda = K; a.a_plane = a_plane; a.W = (const bf16*)W; a.ldw = K; a.tile_group = tile_group; a.row_scale = row_scale;
  if (a_plane > 0) {
    if (gated) run_gemm<256, 3, true>(a, ctas, groups, a.w_group);
    else run_gemm<256, 3, false>(a, ctas, groups, a.w_group);
  } else {
    if (gated) run_gemm<256, 1, true>(a, ctas, groups, a.w_group);
    else run_gemm<256, 1, false>(a, ctas, groups, a.w_group);
  }
}

// q planes [3][R][heads * DQ], k and v planes [3][n_keys][heads / ratio * 128], kr planes [3][n_keys][64] or null
extern "C" void emu_attn32(const void* q, const void* k, const void* kr, const void* v, int R, int heads, int ratio, int n_seqs, int window, int chunk,
                           int keep_first, int pool, const int* row0, const int* pos0, int n_tiles, int n_keys, float scale, float softcap, int sink_one,
                           const float* sink, const float* gate, const float* out_gate, const float* v_inv_freq, int turn_half, int turn_interleaved,
                           void* table, void* out, int out_fp32) {
  const int dq = kr != nullptr ? 192 : 128;
  Attn32Args a = {};
  a.seqs = {n_seqs, window, row0, pos0, chunk, keep_first, pool};
  a.ratio = ratio; a.sink_one = sink_one; a.out_scale = 1.0f;
  // the queries again as the host function has them cut: times their factor
  const long long n = (long long)R * heads * dq;
  std::vector<float> rows(n);
  for (long long i = 0; i < n; ++i) rows[i] = s32_value((const bf16*)q + i, n);
  std::vector<bf16> scaled(3 * n);
  const Factor32 factor = scale32(scale, softcap, a.cap);
  emu::launch(dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), [&] { split_rows_kernel<true>(rows.data(), heads * dq, R, heads * dq, scaled.data(), heads * dq, n, factor); });
  q = scaled.data();
  a.sink = sink; a.gate = gate; a.ldg = heads; a.out_gate = out_gate; a.ldog = heads * 128;
  a.out = out; a.ldo = heads * 128; a.out_fp32 = out_fp32;
  a.q = (const bf16*)q; a.k = (const bf16*)k; a.kr = (const bf16*)kr; a.v = (const bf16*)v;
  a.ldq = heads * dq; a.ldk = heads / ratio * 128; a.ldkr = 64;
  a.q_plane = (long long)R * a.ldq; a.k_plane = (long long)n_keys * a.ldk; a.kr_plane = (long long)n_keys * 64;
  const CUtensorMap tq = tmap3(q, a.ldq, R, 3, a.ldq, a.q_plane, 128), tk = tmap3(k, a.ldk, n_keys, 3, a.ldk, a.k_plane, 128);
  const CUtensorMap tv = tmap3(v, a.ldk, n_keys, 3, a.ldk, a.k_plane, 64);
  const CUtensorMap tr = kr != nullptr ? tmap3(kr, 64, n_keys, 3, 64, a.kr_plane, 128) : tk;
  if (turn_half > 0) {
    emu::launch(dim3((unsigned)((R * turn_half + 255) / 256)), dim3(256), [&] { turn_table_kernel(a.seqs, R, v_inv_freq, turn_half, (float2*)table); });
    a.turn = (const float2*)table; a.turn_half = turn_half; a.turn_interleaved = turn_interleaved;
  }
  emu::g_block_hook = [] { emu_tc::reset(); };
  emu::launch(dim3(heads, n_tiles), dim3(A32_THREADS), [&] {
    if (kr != nullptr) attn32_kernel<1>(tq, tk, tr, tv, a);
    else attn32_kernel<0>(tq, tk, tr, tv, a);
  });
  emu::g_block_hook = nullptr;
}

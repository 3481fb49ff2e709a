// Pruned, fused line-FFT passes (see mlg_fft.cuh): host side -- axis tables
// and the per-pass dispatch into the instantiations of mlg_fft_pass_*.cu.
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "mlg_fft_kernels.cuh"
#include "mlg_fft_reg.cuh"
#include "mlg_fft_reg_lengths.h"

namespace mlg {

bool tma_passes_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("MLG_FFT_TMA");
    return !(e && std::strcmp(e, "0") == 0);
  }();
  return on;
}

bool register_passes_default() {
  static const bool on = std::getenv("MLG_FFT_TMA") == nullptr;
  return on;
}

bool tma_test_stall() {
  static const bool on = [] {
    const char* e = std::getenv("MLG_TEST_WAIT_TIMEOUT");
    return e && std::strcmp(e, "1") == 0;
  }();
  return on;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library)
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

int* fft_wait_word() {
  static std::mutex mu;
  static int* words[128] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!words[dev]) {
    int* w = nullptr;
    if (cudaMalloc(&w, sizeof(int)) != cudaSuccess || cudaMemset(w, 0, sizeof(int)) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    words[dev] = w;
  }
  return words[dev];
}

int fft_wait_status(int* word, cudaStream_t s) {
  if (!word) return MLG_OK;
  int h = 0;
  MLG_CUDA(cudaMemcpyAsync(&h, word, sizeof(int), cudaMemcpyDeviceToHost, s));
  MLG_CUDA(cudaStreamSynchronize(s));
  if (h == 0) return MLG_OK;
  MLG_CUDA(cudaMemsetAsync(word, 0, sizeof(int), s));
  MLG_CUDA(cudaStreamSynchronize(s));
  return fail(MLG_ERR_TIMEOUT, "a bounded wait inside a line-FFT pass ran out; results of the work since the last "
                               "check are invalid");
}

int tma_line_map(CUtensorMap* map, const void* base, int C, int dim_u, long long st_u, int len, long long st_ax,
                 int dim_v, long long st_v, int box_L, int box_rows, bool half) {
  auto enc = tensor_map_encoder();
  MLG_CHECK(enc != nullptr, "cuTensorMapEncodeTiled is not available");
  MLG_CHECK(((uintptr_t)base & 15) == 0, "TMA volume base not 16-byte aligned");
  MLG_CHECK(C >= 1 && 2 * C <= 256 && box_L >= 1 && box_L <= 256 && box_rows >= 1 && box_rows <= 256,
            "TMA box out of range");
  const cuuint64_t dims[4] = {(cuuint64_t)2 * C, (cuuint64_t)dim_u, (cuuint64_t)len, (cuuint64_t)dim_v};
  const cuuint64_t es = half ? 4 : 8;  // bytes per complex value
  const cuuint64_t strides[3] = {(cuuint64_t)st_u * es, (cuuint64_t)st_ax * es, (cuuint64_t)st_v * es};
  for (int i = 0; i < 3; ++i)
    MLG_CHECK(strides[i] % 16 == 0 && strides[i] < (1ull << 40), "TMA stride %llu not a multiple of 16 bytes",
              (unsigned long long)strides[i]);
  const cuuint32_t box[4] = {(cuuint32_t)(2 * C), (cuuint32_t)box_L, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  MLG_CHECK(!half || (4 * C) % 16 == 0, "FP16 boxes need a multiple of 4 coils");
  const CUresult r = enc(map, half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                         const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  MLG_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return MLG_OK;
}

int fft_axis_init(int N, FftAxisPlan& a) {
  a = FftAxisPlan();
  MLG_CHECK(N >= 1 && N <= 1024, "FFT length %d outside [1, 1024]", N);
  // N = N1 * N2 with N1 <= N2 <= 32, N1 as large as possible
  int best1 = 0;
  for (int n1 = 1; n1 <= 32; ++n1)
    if (N % n1 == 0 && N / n1 <= 32 && n1 <= N / n1) best1 = n1;
  if (best1 == 0) return fail(MLG_ERR_UNSUPPORTED, "FFT length %d has no factorisation N1*N2 with N1,N2 <= 32", N);
  a.N = N;
  a.N1 = best1;
  a.N2 = N / best1;
  // unrolled register transforms exist for these factor pairs (lengths 2^k
  // and 3 * 2^k from 16 to 1024); other lengths use the runtime DFT
  static const int kFast[] = {404, 408, 808, 816, 1616, 1632, 3232, 608, 812, 1216, 1624, 2432};
  a.fast = false;
  for (int f : kFast) a.fast = a.fast || f == a.N1 * 100 + a.N2;
  std::vector<float2> t(N);
  for (int j = 0; j < N; ++j) {
    const double ang = -2.0 * M_PI * (double)j / (double)N;
    t[j] = make_float2((float)std::cos(ang), (float)std::sin(ang));
  }
  switch (N) {
#define X(LEN, A, B, MAIN) \
  case LEN:                \
    a.rA = A;              \
    a.rB = B;              \
    break;
    MLG_REG_ALL(X)
#undef X
    default: break;
  }
  if (a.rA) {  // the register passes' tables: W_N^(n2 k1), conjugated for the inverse
    t.resize(3 * (size_t)N);
    for (int dir = 0; dir < 2; ++dir) {
      const int n1s = dir ? a.rB : a.rA;
      float2* u = t.data() + (size_t)(dir + 1) * N;
      for (int n2 = 0; n2 < N / n1s; ++n2)
        for (int k1 = 0; k1 < n1s; ++k1) {
          const float2 w = t[(size_t)n2 * k1];  // n2 k1 < N
          u[(size_t)n2 * n1s + k1] = make_float2(w.x, dir ? -w.y : w.y);
        }
    }
  }
  MLG_CUDA(cudaMalloc(&a.tw, sizeof(float2) * t.size()));
  MLG_CUDA(cudaMemcpy(a.tw, t.data(), sizeof(float2) * t.size(), cudaMemcpyHostToDevice));
  if (a.rA) {
    a.rtw[0] = a.tw + N;
    a.rtw[1] = a.tw + 2 * (size_t)N;
  }
  return MLG_OK;
}

void fft_axis_free(FftAxisPlan& a) {
  cudaFree(a.tw);
  a = FftAxisPlan();
}

int fft_pass_blocks(const FftAxisPlan& a, const PassDesc& d) {
  return std::max(kRegMaxBlocks, blocks_for(d, lines_per_cta(a, d.C, PassMode::kNakatshaOut)));
}

int fft_reg_group_0(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_1(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_2(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_3(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_4(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_5(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_6(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_7(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_8(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_9(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
int fft_reg_group_10(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);

// The pass's register kernel; *done stays false where there is none.
static int fft_reg_pass(const FftAxisPlan& a, PassMode mode, const PassDesc& d, int* n_partial, cudaStream_t s,
                        bool* done) {
  using Fn = int (*)(const FftAxisPlan&, PassMode, const PassDesc&, int*, cudaStream_t, bool*);
  static const Fn kGroups[] = {fft_reg_group_0, fft_reg_group_1, fft_reg_group_2, fft_reg_group_3, fft_reg_group_4, fft_reg_group_5, fft_reg_group_6, fft_reg_group_7, fft_reg_group_8, fft_reg_group_9, fft_reg_group_10};
  *done = false;
  for (Fn f : kGroups) {
    const int st = f(a, mode, d, n_partial, s, done);
    if (st != MLG_OK || *done) return st;
  }
  return MLG_OK;
}

// Passes of 96- to 192-point axes that the shared-memory kernels run faster than
// the register ones: their bundles are whole cells of 24 or 32 coils or the
// caches hold what the column pairs re-read.  us, register / shared, forward
// unless marked inv, over 3-D grids (image length in brackets):
//   unmasked y passes of at least 14 M values in and out: 128 [64] x 16 coils
//     52 / 49, 128 [80] x 8 36 / 33, x 16 69 / 60, x 32 130 / 103, 192 [96] x 12
//     108 / 100, [120] x 16 188 / 177 (below: 128 [64] x 8 24 / 28, 96 [48] x 16
//     22 / 23); exact halves at 192 with 8 or 16 coils 75 / 77, 141 / 144; inv to
//     128 points and outside the exact half, 128 [80] x 16 62 / 56, at 32 coils
//     anywhere, 128 [64] 82 / 72 (192 [120] x 24 243 / 260, 96 [48] x 24 30 / 32);
//   masked passes at 32 coils: 96 [48] 64 / 56, 128 [80] 127 / 110, inv 133 / 115
//     (inv 96 [48] 48 / 58, 192 300 / 380; 24 coils 96 [60] 56 / 56, 128 89 / 110);
//   x passes at 32 coils 128 [64] 55 / 47, [80] 99 / 70, at 24 [80] 86 / 72 (24
//     coils exact half 47 / 50, 16 coils 49 / 49);
//   inv x passes with pipelined kernels to 128 points outside the exact half: 96
//     [60] x 16 42 / 30, 128 [80] x 8 44 / 33 (192 [120] x 8 80 / 98, 12 coils 71 /
//     126, exact half 17 / 22).
// 64 points: 32 coils 15 / 18 at the most even; 256: 16 coils 284 / 315.  2-D
// passes have too few lines: 128 [80] x 16 coils 10 / 10 to 384 [240] x 16 15 / 15.
static bool shared_pass_faster(const FftAxisPlan& a, PassMode mode, const PassDesc& d) {
  const int N = a.N, C = d.C, u = d.ax == 0 ? 1 : 0, v = d.ax == 2 ? 1 : 2;
  const long long lines = (long long)d.dims[u] * d.dims[v];
  if (!a.fast || N < 96 || N > 192 || lines < 2048 || d.tma_slots < 2 || !tma_passes_enabled()) return false;
  const bool fwd = d.dir < 0;
  const bool half = fwd ? d.in_lo == N / 4 && d.in_len == N / 2 : d.out_lo == N / 4 && d.out_len == N / 2;
  if (mode == PassMode::kShannaIn) return C == 32 || (C == 24 && !half);
  if (mode == PassMode::kNakatshaOut) return !half && N <= 128 && (C == 4 || C == 8 || C == 16);
  if (fwd ? d.out_tmask != nullptr : d.in_mask != nullptr) return C == 32 && N <= 128 && (fwd || !half);
  if ((C != 8 && C != 12 && C != 16 && C != 24 && C != 32) || lines * (d.in_len + d.out_len) * C < 14000000)
    return false;
  if (fwd) return !half || N <= 128 || C == 12 || C >= 24;
  return N <= 128 && (!half || C == 32);
}

int fft_pass(const FftAxisPlan& a, PassMode mode, const PassDesc& d, int* n_partial, cudaStream_t s) {
  MLG_CHECK(a.N >= 1 && a.tw, "FFT axis not initialised");
  MLG_CHECK(d.C >= 1, "C must be >= 1");
  const int L = lines_per_cta(a, d.C, mode);
  MLG_CHECK((size_t)a.N * L * d.C * sizeof(float2) <= 200 * 1024,
            "FFT line of %d points x %d coils exceeds shared memory", a.N, d.C);
  if (d.reg && !d.dry && a.rA > 0 && mode != PassMode::kGutIn && !shared_pass_faster(a, mode, d)) {
    bool done = false;
    if (n_partial) *n_partial = 0;
    MLG_TRY(fft_reg_pass(a, mode, d, n_partial, s, &done));
    if (done) return MLG_OK;
  }
  if (n_partial) *n_partial = mode == PassMode::kNakatshaOut && d.partial ? blocks_for(d, L) : 0;
  switch (mode) {
    case PassMode::kShannaIn:
      MLG_CHECK(d.ax == 0 && d.dir < 0, "kShannaIn is a forward x pass");
      return fft_dispatch_shanna_in(a, d, L, s);
    case PassMode::kNakatshaOut:
      MLG_CHECK(d.ax == 0 && d.dir > 0, "kNakatshaOut is an inverse x pass");
      return fft_dispatch_nakatsha_out(a, d, L, s);
    case PassMode::kGutIn:
      MLG_CHECK(d.dir > 0 && d.g_rowptr && d.g_y, "kGutIn is an inverse pass over Gut");
      return fft_dispatch_gut_in(a, d, L, s);
    default:
      return d.dir < 0 ? fft_dispatch_plain_fwd(a, d, L, s) : fft_dispatch_plain_inv(a, d, L, s);
  }
}

}  // namespace mlg

// Line-FFT passes through registers: a line's values go from global memory
// straight into the registers of the first sub-transform, once through shared
// memory between the two sub-transforms, and from the registers of the second
// one straight to global memory.
//
// N = N1 * N2, both <= 32.  A CTA holds `cols` columns x G = max(N1, N2) row
// groups; thread (col, g) runs
//   A. (g < N2) rows n1 N2 + g of its column: an N1-point FFT in registers,
//      times W_N^(g k1), to shared memory;
//   C. (g < N1) the N2 values of k1 = g from shared memory: an N2-point FFT
//      -> X[g + N1 k2], stored.
//
// What bounds it and why this form.  The passes that stage whole bundles in
// shared memory (the cp.async and TMA forms in mlg_fft_kernels.cuh /
// mlg_fft_tma.cuh) move every value six times through it (copy in, read,
// write, read, write, copy out), which at 256-point lines of 16 coils held
// them to one bundle per ~2750 cycles and SM whatever the bytes: the z pass,
// with twice the lines of the y pass, took 1.7 times its time for 1.2 times
// its bytes.  Here a value crosses shared memory once (write, read), rows
// outside the stored range or the occupancy mask are never loaded or stored
// (a predicate per row, against 16-row chunks), and the loads' latency is
// covered by the other CTAs of the SM.  With the bytes moving, issue slots
// bound it next (61 % busy at one column per thread): the y and z passes give
// a thread two adjacent columns -- 16-byte accesses, addresses, predicates and
// twiddle loads shared by both, 20-25 % fewer instructions, 256-byte row
// pieces (two CTAs of 256 threads at 128 registers per SM).  That leaves the
// issue slots 40 to 50 % busy and the loads that 16 warps keep in flight as the
// bound.
//
// Measured (B200, 256^3 grid, 16 coils, masked adjoint; TMA passes -> these):
// forward x 174 -> 142 us, y 313 -> 285, z 521 -> 395, inverse z 531 -> 424,
// y 294 -> 262, x 238 -> 147 us: the y passes 5.7-6.2 TB/s of their bytes, the
// masked z passes 4.5-4.8.  192^3 x 12 coils: inverse x 213 -> 63 us (it had
// only the unpipelined kernel).  160 x 160 x 120 x 8 coils (direct-DFT passes
// before): all six passes 2.68 ms -> 0.24 ms.
//
// The y and z pass as one kernel with the intermediate kept in L2 (slabs of
// columns, a work queue) was built: DRAM traffic halved but 715 against 660
// us, bound by issue and latency (43 % of issue slots at 16 warps per SM).
//
// Columns.  The y and z passes see a plane as rows of Q = N_x * C contiguous
// values whatever the coil count (32 columns per bundle, 16 where that leaves
// SMs without work or sub-transforms are longer than 16 points, 4 where 16
// does), so odd coil counts run here too.  In the x passes the columns are the
// C coils of a line: row n of a line starts at n C, so that for a fixed n1 (or
// k2) the threads of a line touch one contiguous run.
//
// HALF: the stored input rows (forward) are exactly [N/4, 3N/4) -- twofold
// oversampling -- so half of step A's inputs are known zeros at compile time
// and its first butterfly stage vanishes; (inverse) the kept output rows are,
// so half of step C's outputs are never formed.
#pragma once

#include "mlg_fft_kernels.cuh"

namespace mlg {

struct RegPass {
  const void* in = nullptr;  // float2, or __half2 with in_half
  void* out = nullptr;
  // y / z passes: rows of Q values; bundle b = columns (b % nb_u) * COLS ...
  // of plane v = b / nb_u
  int Q = 0, nb_u = 1, planes = 1, nbundles = 0;
  long long in_v = 0, out_v = 0;      // plane strides (values)
  long long in_row = 0, out_row = 0;  // row strides (values)
  int in_lo = 0, in_len = 0, out_lo = 0, out_len = 0;
  int C = 1;
  // occupancy bits regrouped for this axis: bit j of word [line][m] = row
  // m + M j (line = x + du v); masked loads (inverse) or stores (forward)
  const uint32_t* tmask = nullptr;
  int du = 0;
  int in_half = 0, out_half = 0;
  const unsigned* h_amax = nullptr;
  int h_len = 1, h_len_out = 1;
  // x passes: `lines` lines of C columns, L per CTA; line = y + ny z
  int lines = 0, L = 1, ny = 1, par0 = 0;
  const float2* img = nullptr;
  int img_per_coil = 0;
  const float2* kfc = nullptr;
  float2* img_out = nullptr;
  float sfac = 1.f;
  double* partial = nullptr;
  unsigned* amax = nullptr;
};

// ---- register transforms of 2^a 3^b 5^c 7^d points --------------------------
// Sums and differences of complex values as packed FP32 pairs: one
// instruction each (the passes are bound by issue slots before they are bound
// by the FP32 units).
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 scale2(float c, float2 a) { return __fmul2_rn(make_float2(c, c), a); }
__device__ __forceinline__ float2 fma2(float c, float2 a, float2 b) { return __ffma2_rn(make_float2(c, c), a, b); }

constexpr int cx_odd_prime(int R) {
  for (int p = 3; p <= 7; p += 2)
    if (R % p == 0) return p;
  return 1;
}

template <int R, int DIR, bool HALF>
__device__ __forceinline__ void rfft(float2 (&r)[R]);

// R = P M, P an odd prime: r[k + M q] from the P sub-transforms b[j][k]
// (twiddles W_R^(jk) applied): cosine / sine sums over the symmetric pairs
// j, P - j.
template <int R, int P, int DIR, bool HALF>
__device__ __forceinline__ void rfft_odd(float2 (&r)[R]) {
  constexpr int M = R / P, H = (P - 1) / 2;
  float2 b[P][M];
  sfor<P>([&](auto jc) {
    constexpr int j = decltype(jc)::value;
    sfor<M>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      b[j][m] = r[P * m + j];
    });
    rfft<M, DIR, HALF>(b[j]);
    if constexpr (j > 0) {
      sfor<M>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        if constexpr (k > 0) {
          constexpr double a = cx_reduce((double)DIR * 2.0 * kPiD * (double)((j * k) % R) / (double)R);
          constexpr float wr = (float)cx_cos_red(a), wi = (float)cx_sin_red(a);
          const float2 v = b[j][k];
          b[j][k] = make_float2(wr * v.x - wi * v.y, wr * v.y + wi * v.x);
        }
      });
    }
  });
  sfor<M>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    float2 s[H], d[H], x0 = b[0][k];
    sfor<H>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      s[j] = add2(b[j + 1][k], b[P - 1 - j][k]);
      d[j] = sub2(b[j + 1][k], b[P - 1 - j][k]);
      x0 = add2(x0, s[j]);
    });
    r[k] = x0;
    sfor<H>([&](auto qc) {
      constexpr int q = decltype(qc)::value + 1;
      float2 e = b[0][k], o = make_float2(0.f, 0.f);
      sfor<H>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        constexpr double a = cx_reduce(2.0 * kPiD * (double)(((j + 1) * q) % P) / (double)P);
        constexpr float c = (float)cx_cos_red(a), sn = (float)((double)DIR * cx_sin_red(a));
        e = fma2(c, s[j], e);
        if constexpr (j == 0)
          o = scale2(sn, d[j]);
        else
          o = fma2(sn, d[j], o);
      });
      r[k + M * q] = make_float2(e.x - o.y, e.y + o.x);        // e + i o
      r[k + M * (P - q)] = make_float2(e.x + o.y, e.y - o.x);  // e - i o
    });
  });
}

// Stages LEN, 2 LEN, ... R of a radix-2 transform in bit-reversed order.
template <int R, int DIR, int LEN>
__device__ __forceinline__ void rfft_stages(float2 (&r)[R]) {
  if constexpr (LEN <= R) {
    sfor<R / LEN>([&](auto ic) {
      constexpr int I = decltype(ic)::value * LEN;
      sfor<LEN / 2>([&](auto jc) {
        constexpr int J = decltype(jc)::value;
        constexpr double ang = cx_reduce((double)DIR * 2.0 * kPiD * (double)J / (double)LEN);
        constexpr float wr = (float)cx_cos_red(ang), wi = (float)cx_sin_red(ang);
        const float2 u = r[I + J], v = r[I + J + LEN / 2];
        if constexpr (4 * J == LEN) {  // +-i: a swap and a sign
          const float2 t = DIR < 0 ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
          r[I + J] = make_float2(u.x + t.x, u.y + t.y);
          r[I + J + LEN / 2] = make_float2(u.x - t.x, u.y - t.y);
        } else {
          float2 t = v;
          if constexpr (J != 0) t = make_float2(wr * v.x - wi * v.y, wr * v.y + wi * v.x);
          r[I + J] = add2(u, t);
          r[I + J + LEN / 2] = sub2(u, t);
        }
      });
    });
    rfft_stages<R, DIR, LEN * 2>(r);
  }
}

// DIR < 0: X[k] = sum_j r[j] exp(-2 pi i jk/R); DIR > 0: inverse
// (unnormalised).  HALF (R a multiple of 4): only r[R/4 .. 3R/4) are read, the
// others are zero.
template <int R, int DIR, bool HALF>
__device__ __forceinline__ void rfft(float2 (&r)[R]) {
  static_assert(!HALF || R % 4 == 0, "HALF: a multiple of 4");
  if constexpr (R > 1 && !cx_pow2(R)) {
    constexpr int P = cx_odd_prime(R);
    static_assert(P > 1, "register FFT length must be 2^a 3^b 5^c 7^d");
    rfft_odd<R, P, DIR, HALF>(r);
  } else if constexpr (R > 1) {
    float2 t[R];
    if constexpr (HALF) {  // the first stage meets one zero in every pair
      sfor<R / 2>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        constexpr int j = bitrev(2 * i, R);  // pair (j, j + R/2), j < R/2
        if constexpr (j < R / 4) {
          t[2 * i] = r[j + R / 2];
          t[2 * i + 1] = make_float2(-r[j + R / 2].x, -r[j + R / 2].y);
        } else {
          t[2 * i] = t[2 * i + 1] = r[j];
        }
      });
    } else {
      sfor<R>([&](auto ic) { t[decltype(ic)::value] = r[bitrev(decltype(ic)::value, R)]; });
    }
    rfft_stages<R, DIR, HALF ? 4 : 2>(t);
    sfor<R>([&](auto ic) { r[decltype(ic)::value] = t[decltype(ic)::value]; });
  }
}

// ---- the two sub-transforms -----------------------------------------------------
constexpr int reg_groups(int N1, int N2) { return N1 > N2 ? N1 : N2; }

// Values between the k1 blocks in shared memory: N2 cols plus what makes k1
// -> k1 + 1 a step of `cols` modulo 16 values (128 bytes), so that step C's
// half-warps read without bank conflicts whatever the column count.
__host__ __device__ constexpr int reg_block_stride(int N2, int cols) {
  return N2 * cols + (((cols - N2 * cols) % 16) + 16) % 16;
}

// Step A's second half: the transform of the thread's VEC columns, the
// twiddles of row group n2 (T: [n2][k1]) and the writes at s[k1 * S1 + n2 *
// cols] (s already at the thread's column).
template <int N1, int DIR, bool HALF, int VEC>
__device__ __forceinline__ void reg_step_a(float2 (&r)[VEC][N1], const float2* __restrict__ T, int n2, float2* s,
                                           int S1, int cols) {
#pragma unroll
  for (int v = 0; v < VEC; ++v) rfft<N1, DIR, HALF>(r[v]);
  const float2* t = T + n2 * N1;
  if constexpr (N1 % 2 == 0) {
#pragma unroll
    for (int k = 0; k < N1; k += 2) {
      const float4 w = *reinterpret_cast<const float4*>(t + k);
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        if (k) r[v][k] = cmulf(r[v][k], make_float2(w.x, w.y));
        r[v][k + 1] = cmulf(r[v][k + 1], make_float2(w.z, w.w));
      }
    }
  } else {
#pragma unroll
    for (int k = 1; k < N1; ++k)
#pragma unroll
      for (int v = 0; v < VEC; ++v) r[v][k] = cmulf(r[v][k], t[k]);
  }
  float2* p = s + n2 * cols;
#pragma unroll
  for (int k = 0; k < N1; ++k) {
    if constexpr (VEC == 2)
      *reinterpret_cast<float4*>(p + k * S1) = make_float4(r[0][k].x, r[0][k].y, r[1][k].x, r[1][k].y);
    else
      p[k * S1] = r[0][k];
  }
}

template <int N2, int DIR, int VEC>
__device__ __forceinline__ void reg_step_c(float2 (&r)[VEC][N2], const float2* s, int S1, int k1, int cols) {
  const float2* p = s + k1 * S1;
#pragma unroll
  for (int n = 0; n < N2; ++n) {
    if constexpr (VEC == 2) {
      const float4 q = *reinterpret_cast<const float4*>(p + n * cols);
      r[0][n] = make_float2(q.x, q.y);
      r[1][n] = make_float2(q.z, q.w);
    } else {
      r[0][n] = p[n * cols];
    }
  }
#pragma unroll
  for (int v = 0; v < VEC; ++v) rfft<N2, DIR, false>(r[v]);
}

// Row n of the CTA's rows: a CTA-uniform base plus a 32-bit thread offset
// (values; the host checks the range), so that a row costs one address
// register.
template <class T>
__device__ __forceinline__ T* reg_at(T* base, unsigned off) {
  return reinterpret_cast<T*>(reinterpret_cast<char*>(const_cast<typename std::remove_const<T>::type*>(base)) +
                              off * (unsigned)sizeof(T));
}

// VEC adjacent values at row base + off (L2 only: the rows stream through).
template <int VEC>
__device__ __forceinline__ void reg_load(const float2* base, unsigned off, float2* a) {
  if constexpr (VEC == 2) {
    const float4 q = __ldcg(reinterpret_cast<const float4*>(reg_at(base, off)));
    a[0] = make_float2(q.x, q.y);
    a[1] = make_float2(q.z, q.w);
  } else {
    a[0] = __ldcg(reg_at(base, off));
  }
}

// The same of FP16 rows, unconverted: a row's conversion under the condition of
// its load waited for that load before the next went out (mixed precision, 192^3 x
// 16 coils: inverse y pass 180 -> 121 us; 120 stored rows 243 -> 168, forward z 261
// -> 206).
template <int VEC>
__device__ __forceinline__ void reg_load(const __half2* base, unsigned off, unsigned* a) {
  if constexpr (VEC == 2) {
    const uint2 w = __ldcg(reinterpret_cast<const uint2*>(reg_at(base, off)));
    a[0] = w.x;
    a[1] = w.y;
  } else {
    a[0] = __ldcg(reinterpret_cast<const unsigned*>(reg_at(base, off)));
  }
}

template <int VEC>
__device__ __forceinline__ void reg_store(float2* base, unsigned off, const float2* a) {
  if constexpr (VEC == 2)
    *reinterpret_cast<float4*>(reg_at(base, off)) = make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
  else
    *reg_at(base, off) = a[0];
}

template <int VEC>
__device__ __forceinline__ void reg_store(__half2* base, unsigned off, float hs, const float2* a) {
  __half2 h[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) h[v] = __floats2half2_rn(a[v].x * hs, a[v].y * hs);
  if constexpr (VEC == 2) {
    uint2 w;
    w.x = *reinterpret_cast<const unsigned*>(&h[0]);
    w.y = *reinterpret_cast<const unsigned*>(&h[1]);
    *reinterpret_cast<uint2*>(reg_at(base, off)) = w;
  } else {
    *reg_at(base, off) = h[0];
  }
}

// Bits j of the rows g + step j in [lo, lo + len).
template <int STEP>
__device__ __forceinline__ uint32_t reg_range_word(int g, int lo, int len) {
  const int b = max(0, (lo - g + STEP - 1) / STEP), e = (lo + len - g + STEP - 1) / STEP;
  const uint32_t below_e = e >= 32 ? ~0u : (e > 0 ? (1u << e) - 1u : 0u);
  return b >= 32 ? 0u : below_e & (~0u << b);
}

// A bundle's rows into registers: forward, the stored rows [in_lo, in_lo +
// in_len) (HALF: rows N/4 .. 3N/4, known at compile time); inverse, the rows
// whose bit is set in word.  in0: row 0 of the bundle (values; may lie before
// the stored rows), off: the thread's offset from it.
template <int N1, int N2, int DIR, bool HALF, int VEC>
__device__ __forceinline__ void reg_load_rows(float2 (&r)[VEC][N1], const RegPass& a, bool half, const void* in,
                                              long long in0, unsigned off, int g, uint32_t word, float hs) {
  if (DIR < 0 && !HALF) word = reg_range_word<N2>(g, a.in_lo, a.in_len);
  auto want = [&](int n1) {
    if (DIR < 0 && HALF) return n1 >= N1 / 4 && n1 < 3 * N1 / 4;
    return (word & (1u << n1)) != 0u;
  };
  if (half) {
    const __half2* base = reinterpret_cast<const __half2*>(in) + in0;
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) {  // (a row's bits wait in the register of its real part)
      unsigned w[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) w[v] = 0u;
      if (want(n1)) reg_load<VEC>(base + (long long)(n1 * N2) * a.in_row, off, w);
#pragma unroll
      for (int v = 0; v < VEC; ++v) r[v][n1].x = __uint_as_float(w[v]);
    }
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) {
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const unsigned w = __float_as_uint(r[v][n1].x);
        const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&w));
        r[v][n1] = make_float2(h.x * hs, h.y * hs);  // (rows that are not stored: zeros)
      }
    }
  } else {
    const float2* base = reinterpret_cast<const float2*>(in) + in0;
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) {
      float2 q[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) q[v] = make_float2(0.f, 0.f);
      if (want(n1)) reg_load<VEC>(base + (long long)(n1 * N2) * a.in_row, off, q);
#pragma unroll
      for (int v = 0; v < VEC; ++v) r[v][n1] = q[v];
    }
  }
}

// The rows of step C to memory: forward, those whose bit is set in word;
// inverse, the kept rows [out_lo, out_lo + out_len).
template <int N1, int N2, int DIR, bool HALF, int VEC>
__device__ __forceinline__ void reg_store_rows(const float2 (&r)[VEC][N2], const RegPass& a, bool half, void* out,
                                               long long out0, unsigned off, int g, uint32_t word, float hs) {
  if (DIR > 0 && !HALF) word = reg_range_word<N1>(g, a.out_lo, a.out_len);
  auto want = [&](int k2) {
    if (DIR > 0 && HALF) return k2 >= N2 / 4 && k2 < 3 * N2 / 4;
    return (word & (1u << k2)) != 0u;
  };
  if (half) {
    __half2* base = reinterpret_cast<__half2*>(out) + out0;
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      float2 q[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) q[v] = r[v][k2];
      if (want(k2)) reg_store<VEC>(base + (long long)(N1 * k2) * a.out_row, off, hs, q);
    }
  } else {
    float2* base = reinterpret_cast<float2*>(out) + out0;
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
      float2 q[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) q[v] = r[v][k2];
      if (want(k2)) reg_store<VEC>(base + (long long)(N1 * k2) * a.out_row, off, q);
    }
  }
}

// Resident threads per SM asked of the register allocator: 64 registers a
// thread for one column of up to 16-point sub-transforms, 128 for two columns
// (96 of up to 8 points) or up to 32 points.
constexpr int reg_min_blocks(int N1, int N2, int nt, int vec = 1) {
  const int g = reg_groups(N1, N2);
  const int thr = vec == 2 ? (g <= 8 ? 640 : 512) : (g <= 16 ? 1024 : (g <= 20 ? 768 : 512));
  return thr / nt < 1 ? 1 : thr / nt;
}
constexpr int reg_threads(int N1, int N2, int cols, int vec) { return cols / vec * reg_groups(N1, N2); }

constexpr size_t reg_tw_bytes(int N) { return ((size_t)N * 8 + 15) / 16 * 16; }

// ---- y / z passes ---------------------------------------------------------------
template <int N1, int N2, int DIR, int COLS, int VEC, bool HALF>
__global__ void __launch_bounds__(reg_threads(N1, N2, COLS, VEC),
                                  reg_min_blocks(N1, N2, reg_threads(N1, N2, COLS, VEC), VEC))
    reg_plain_kernel(RegPass a, const float2* __restrict__ tw) {
  constexpr int N = N1 * N2, CG = COLS / VEC, NT = reg_threads(N1, N2, COLS, VEC), S1 = reg_block_stride(N2, COLS);
  extern __shared__ __align__(16) unsigned char reg_smem[];
  float2* const T = reinterpret_cast<float2*>(reg_smem);
  float2* const s = reinterpret_cast<float2*>(reg_smem + reg_tw_bytes(N));
  const int tid = threadIdx.x, col = tid % CG * VEC, g = tid / CG;
  for (int i = tid; i < N; i += NT) T[i] = __ldg(tw + i);
  const float hs_in = a.in_half ? 1.f / half_store_scale(a.h_amax, a.h_len) : 1.f;
  const float hs_out = a.out_half ? half_store_scale(a.h_amax, a.h_len_out) : 1.f;
  // bundle (plane v, column block u), walked without divisions
  const int du = (int)(gridDim.x % a.nb_u), dv = (int)(gridDim.x / a.nb_u);
  int u = (int)(blockIdx.x % a.nb_u), v = (int)(blockIdx.x / a.nb_u);
  // this thread's occupancy word of a bundle (all rows without masks; 0 for
  // columns past the edge)
  auto row_word = [&](int uu, int vv) -> uint32_t {
    const int q = uu * COLS + col;
    if (vv >= a.planes || q >= a.Q || g >= (DIR < 0 ? N1 : N2)) return 0u;
    if (!a.tmask) return ~0u;
    return __ldg(a.tmask + ((long long)(q / a.C) + (long long)a.du * vv) * (DIR < 0 ? N1 : N2) + g);
  };
  uint32_t next_word = row_word(u, v);
  const unsigned off_in = (unsigned)g * (unsigned)a.in_row + (unsigned)col;
  const unsigned off_out = (unsigned)g * (unsigned)a.out_row + (unsigned)col;
  while (v < a.planes) {
    const bool live = u * COLS + col < a.Q;
    const long long in0 = (long long)v * a.in_v + (long long)u * COLS - (long long)a.in_lo * a.in_row;
    const long long out0 = (long long)v * a.out_v + (long long)u * COLS - (long long)a.out_lo * a.out_row;
    u += du;
    v += dv;
    if (u >= a.nb_u) {
      u -= a.nb_u;
      ++v;
    }
    const uint32_t word = next_word;
    const int any = __syncthreads_or(word != 0u);  // (also: the last bundle's reads of s are done)
    next_word = row_word(u, v);                    // in flight during this bundle
    if (DIR < 0 && !any) continue;                 // nothing of this bundle is stored
    if (any && live && g < N2) {
      float2 r[VEC][N1];
      reg_load_rows<N1, N2, DIR, HALF, VEC>(r, a, a.in_half, a.in, in0, off_in, g, word, hs_in);
      reg_step_a<N1, DIR, (DIR < 0 && HALF), VEC>(r, T, g, s + col, S1, COLS);
    }
    __syncthreads();
    if (live && g < N1) {
      float2 r[VEC][N2];
      if (any) {
        reg_step_c<N2, DIR, VEC>(r, s + col, S1, g, COLS);
      } else {  // an all-zero line
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2)
#pragma unroll
          for (int j = 0; j < VEC; ++j) r[j][k2] = make_float2(0.f, 0.f);
      }
      reg_store_rows<N1, N2, DIR, HALF, VEC>(r, a, a.out_half, a.out, out0, off_out, g, word, hs_out);
    }
  }
}

// ---- forward x pass: x .* KFC, modulation, zero-fill, transform ---------------------
// One coil per thread (two measured slower: 158 against 142 us at 256-point
// lines of 16 coils, 69 against 60 us at 192 x 12).  Without HALF the rows' loads
// go out eight at a time, conditions on the loads alone: with a row's product
// under its condition each row waited for its own loads (oversampling 1.6, 256-point
// lines of 16 coils 429 -> 290 us, 128 x 32 coils 180 -> 99, 192 x 12 167 -> 115).
// TB: launch bound, reg_x_bound for up to 16 coils, 1024 beyond.
constexpr int reg_x_bound(int N1, int N2) { return reg_groups(N1, N2) <= 16 ? 256 : 512; }

template <int N1, int N2, bool HALF, int TB>
__global__ void __launch_bounds__(TB, reg_min_blocks(N1, N2, TB))
    reg_shanna_kernel(RegPass a, const float2* __restrict__ tw) {
  constexpr int N = N1 * N2, G = reg_groups(N1, N2);
  extern __shared__ __align__(16) unsigned char reg_smem[];
  float2* const T = reinterpret_cast<float2*>(reg_smem);
  const int C = a.C, LT = G * C, S1 = reg_block_stride(N2, C);
  const int tid = threadIdx.x, l = tid / LT, w = tid - l * LT, g = w / C, c = w - g * C;
  float2* const s = reinterpret_cast<float2*>(reg_smem + reg_tw_bytes(N)) + l * (N1 * S1) + c;
  for (int i = tid; i < N; i += blockDim.x) T[i] = __ldg(tw + i);
  float amax = 0.f;
  for (int b = blockIdx.x; b < a.nbundles; b += gridDim.x) {
    const int line = b * a.L + l;
    const bool live = l < a.L && line < a.lines;
    __syncthreads();  // the last bundle's reads of s are done
    if (live && g < N2) {
      const int par = (a.par0 + line % a.ny + line / a.ny) & 1;
      const long long m0 = (long long)line * a.in_len + g - a.in_lo;
      const uint32_t word = HALF ? 0u : reg_range_word<N2>(g, a.in_lo, a.in_len);
      constexpr int LO = HALF ? N1 / 4 : 0, HI = HALF ? 3 * N1 / 4 : N1, U = HALF ? HI - LO : 8;
      float2 r[1][N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) r[0][n1] = make_float2(0.f, 0.f);
#pragma unroll
      for (int b0 = LO; b0 < HI; b0 += U) {
        float2 xv[U], kv[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
          const int n1 = b0 + q;
          xv[q] = kv[q] = make_float2(0.f, 0.f);
          if (n1 < HI && (HALF || (word & (1u << n1)))) {
            const long long m = m0 + n1 * N2;
            xv[q] = __ldg(a.img + (a.img_per_coil ? m * C + c : m));
            kv[q] = __ldg(a.kfc + m * C + c);
          }
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
          const int n1 = b0 + q;
          if (n1 < HI) {
            const float2 p = cmulf_rn(xv[q], kv[q]);
            r[0][n1] = ((n1 * N2 + g + par) & 1) ? make_float2(-p.x, -p.y) : p;
          }
        }
      }
      reg_step_a<N1, -1, HALF, 1>(r, T, g, s, S1, C);
    }
    __syncthreads();
    if (live && g < N1) {
      float2 r[1][N2];
      reg_step_c<N2, -1, 1>(r, s, S1, g, C);
      float2* o = reinterpret_cast<float2*>(a.out) + ((long long)line * N + g) * C + c;
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) {
        o[N1 * k2 * C] = r[0][k2];
        amax = fmaxf(amax, fmaxf(fabsf(r[0][k2].x), fabsf(r[0][k2].y)));
      }
    }
  }
  if (a.amax) warp_amax(a.amax, amax);  // the FP16 passes' scale (mixed precision); whole warps
}

// ---- inverse x pass: transform, crop, modulation, .* KFC_conj, coil sum -------------
// VEC coils per thread (2, even coil counts: 147 against 182 us at 256-point
// lines of 16 coils, where the larger product area of one coil per thread
// takes the L1 space the row loads need).  The products (VEC == 2: summed over the thread's coil pair) leave step C for
// a shared-memory area of their own ([pixel][C / VEC], an odd row length: no
// bank conflicts) and a thread per pixel sums them in four interleaved sums;
// |x|^2 partial sums in FP64 per CTA.  The coil maps' rows without HALF: four
// loads at a time, as in the forward pass (oversampling 1.6, 256 x 16 coils 395 ->
// 283 us, 128 x 8 58 -> 43).
template <int N1, int N2, bool HALF, int VEC, int TB>
__global__ void __launch_bounds__(TB, reg_min_blocks(N1, N2, TB, VEC))
    reg_nak_kernel(RegPass a, const float2* __restrict__ tw) {
  constexpr int N = N1 * N2, G = reg_groups(N1, N2);
  extern __shared__ __align__(16) unsigned char reg_smem[];
  __shared__ double red[32];
  float2* const T = reinterpret_cast<float2*>(reg_smem);
  const int C = a.C, CG = C / VEC, LT = G * CG, S1 = reg_block_stride(N2, C), CP = CG | 1;
  const int tid = threadIdx.x, l = tid / LT, w = tid - l * LT, g = w / CG, c = (w - g * CG) * VEC;
  float2* const s0 = reinterpret_cast<float2*>(reg_smem + reg_tw_bytes(N));
  float2* const s = s0 + l * (N1 * S1) + c;
  float2* const prod = s0 + a.L * (N1 * S1);
  for (int i = tid; i < N; i += blockDim.x) T[i] = __ldg(tw + i);
  double sq = 0.0;
  __syncthreads();
  for (int b = blockIdx.x; b < a.nbundles; b += gridDim.x) {
    const int line = b * a.L + l;
    const bool live = l < a.L && line < a.lines;
    if (live && g < N2) {  // (the last bundle's reads of s ended before its second barrier)
      const float2* p = reinterpret_cast<const float2*>(a.in) + ((long long)line * N + g) * C + c;
      float2 r[VEC][N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) {
        float2 q[VEC];
        reg_load<VEC>(p, (unsigned)(n1 * N2 * C), q);
#pragma unroll
        for (int v = 0; v < VEC; ++v) r[v][n1] = q[v];
      }
      reg_step_a<N1, 1, false, VEC>(r, T, g, s, S1, C);
    }
    __syncthreads();  // (also: the last bundle's sums are read)
    if (live && g < N1) {
      float2 r[VEC][N2];
      reg_step_c<N2, 1, VEC>(r, s, S1, g, C);
      const int par = (a.par0 + line % a.ny + line / a.ny) & 1;
      const float2* kf = a.kfc + ((long long)line * a.out_len + g - a.out_lo) * C + c;
      float2* o = prod + (l * a.out_len + g - a.out_lo) * CP + c / VEC;
      const uint32_t word = HALF ? 0u : reg_range_word<N1>(g, a.out_lo, a.out_len);
      constexpr int LO = HALF ? N2 / 4 : 0, HI = HALF ? 3 * N2 / 4 : N2, U = HALF ? HI - LO : 4;
#pragma unroll
      for (int b0 = LO; b0 < HI; b0 += U) {
        float2 kv[U][VEC];
#pragma unroll
        for (int q = 0; q < U; ++q) {
          const int k2 = b0 + q;
          if (k2 < HI && (HALF || (word & (1u << k2)))) {
            if constexpr (VEC == 2) {
              const float4 v = __ldcs(reinterpret_cast<const float4*>(kf + N1 * k2 * C));
              kv[q][0] = make_float2(v.x, v.y);
              kv[q][1] = make_float2(v.z, v.w);
            } else {
              kv[q][0] = __ldcs(kf + N1 * k2 * C);
            }
          }
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
          const int k2 = b0 + q, k = g + N1 * k2;
          if (k2 < HI && (HALF || (word & (1u << k2)))) {
            const float sg = ((k + par) & 1) ? -a.sfac : a.sfac;
            if constexpr (VEC == 2) {
              o[N1 * k2 * CP] = nak_pair_term(make_float4(r[0][k2].x, r[0][k2].y, r[1][k2].x, r[1][k2].y),
                                              make_float4(kv[q][0].x, kv[q][0].y, kv[q][1].x, kv[q][1].y), sg);
            } else {
              const float2 v = r[0][k2];
              o[N1 * k2 * CP] = cmulf_rn(make_float2(__fmul_rn(v.x, sg), __fmul_rn(v.y, sg)), kv[q][0]);
            }
          }
        }
      }
    }
    __syncthreads();
    const int npix = min(a.L, a.lines - b * a.L) * a.out_len;
    for (int o = tid; o < npix; o += blockDim.x) {
      const float2* p = prod + o * CP;
      float2 t[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) t[j] = j < CG ? p[j] : make_float2(0.f, 0.f);
      for (int k = 4; k < CG; k += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (k + j < CG) t[j] = add2(t[j], p[k + j]);
      }
      const float2 x = add2(add2(t[0], t[1]), add2(t[2], t[3]));
      a.img_out[(long long)b * a.L * a.out_len + o] = x;
      sq += (double)x.x * x.x + (double)x.y * x.y;
    }
  }
  if (a.partial) {
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
    if ((tid & 31) == 0) red[tid >> 5] = sq;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
      a.partial[blockIdx.x] = t;
    }
  }
}

// ---- host side --------------------------------------------------------------------
constexpr int kRegMaxBlocks = 2048;  // CTAs of a register pass (partial-sum slots)
constexpr size_t kRegSmemCap = 200 * 1024;

// Launches a persistent kernel over `work` bundles: at most the resident CTAs of
// the GPU.  What depends on the kernel, the CTA and the device alone is kept per
// host thread and kernel -- KERN is a template argument, every register kernel has
// the same pointer type: a cache by type was refilled (three runtime calls) on
// nearly every pass.
template <auto KERN>
static int reg_launch(const RegPass& p, const float2* tw, int threads, size_t smem, int* grid, cudaStream_t s) {
  thread_local int per_sm = 0, sms = 0, t_threads = 0, t_dev = -1;
  thread_local size_t t_smem = 0;
  int dev = 0;
  MLG_CUDA(cudaGetDevice(&dev));
  if (per_sm == 0 || t_smem != smem || t_threads != threads || t_dev != dev) {
    if (t_dev != dev) {
      MLG_CUDA(cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegSmemCap));
      MLG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    }
    per_sm = 0;
    MLG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, threads, smem));
    per_sm = std::max(1, per_sm);
    t_smem = smem;
    t_threads = threads;
    t_dev = dev;
  }
  *grid = std::max(1, std::min(std::min(p.nbundles, per_sm * sms), kRegMaxBlocks));
  KERN<<<*grid, threads, smem, s>>>(p, tw);
  MLG_LAUNCHED();
  return MLG_OK;
}

template <int N1, int N2, int DIR, int COLS, int VEC, bool HALF>
static int reg_plain_launch(RegPass& p, const float2* tw, cudaStream_t s) {
  constexpr int NT = reg_threads(N1, N2, COLS, VEC);
  const size_t smem = reg_tw_bytes(N1 * N2) + (size_t)N1 * reg_block_stride(N2, COLS) * sizeof(float2);
  p.nb_u = (p.Q + COLS - 1) / COLS;
  p.nbundles = p.nb_u * p.planes;
  int grid = 1;
  return reg_launch<reg_plain_kernel<N1, N2, DIR, COLS, VEC, HALF>>(p, tw, NT, smem, &grid, s);
}

// The geometry of a y or z pass; false where the register kernels do not
// take it.
static inline bool reg_plain_geometry(const PassDesc& d, int N, int G, RegPass& p) {
  const int v = d.ax == 2 ? 1 : 2;
  if (d.ax == 0 || d.in_stride[0] != d.C || d.out_stride[0] != d.C) return false;
  p.in = d.in;
  p.out = d.out;
  p.C = d.C;
  p.Q = d.dims[0] * d.C;
  p.planes = d.dims[v];
  p.in_v = d.in_stride[v];
  p.out_v = d.out_stride[v];
  p.in_row = d.in_stride[d.ax];
  p.out_row = d.out_stride[d.ax];
  p.in_lo = d.in_lo;
  p.in_len = d.in_len;
  p.out_lo = d.out_lo;
  p.out_len = d.out_len;
  // forward: cropped input, whole output lines; inverse: the reverse
  if (d.dir < 0 ? (d.out_lo != 0 || d.out_len != N) : (d.in_lo != 0 || d.in_len != N)) return false;
  if (d.in_mask && !d.tmask) return false;
  // 32-bit thread offsets (bytes) within a row group's rows
  if ((unsigned long long)(G + 1) * 8ull * (unsigned long long)std::max(p.in_row, p.out_row) >= (1ull << 32))
    return false;
  if (d.dir < 0 ? d.out_tmask != nullptr : d.in_mask != nullptr) {
    p.tmask = d.dir < 0 ? d.out_tmask : d.tmask;
    p.du = d.dims[0];
  }
  if (p.tmask && d.in_half && d.dir > 0) return false;  // (no such pass: the masked grid is FP32)
  p.in_half = d.in_half;
  p.out_half = d.out_half;
  p.h_amax = d.h_amax;
  p.h_len = d.h_len;
  p.h_len_out = d.in_half && d.h_len_out > 0 ? d.h_len_out : d.h_len;
  return true;
}

// Two columns per thread (16-byte accesses) need even rows and planes; an
// occupancy word then serves both columns, which must share a cell.
static inline bool reg_pairs_ok(const RegPass& p) {
  return p.Q % 2 == 0 && p.in_v % 2 == 0 && p.out_v % 2 == 0 && p.in_row % 2 == 0 && p.out_row % 2 == 0 &&
         (!p.tmask || p.C % 2 == 0);
}

// Twofold oversampling: exactly the rows [N/4, 3N/4) on the cropped side.
static inline bool reg_is_half(const RegPass& p, int dir, int N) {
  return dir < 0 ? p.in_lo == N / 4 && p.in_len == N / 2 : p.out_lo == N / 4 && p.out_len == N / 2;
}

template <int N1, int N2, int DIR, bool MAIN>
static int reg_plain_pass(const PassDesc& d, const float2* tw, cudaStream_t s, bool* done) {
  constexpr int N = N1 * N2, G = reg_groups(N1, N2);
  RegPass p;
  if (!reg_plain_geometry(d, N, G, p)) return MLG_OK;
  *done = true;
  // 32 columns, two per thread, where that leaves every SM two CTAs; else 16
  // columns (whole 128-byte rows); 4 where 16 would leave SMs without a bundle
  const long long b32 = (long long)((p.Q + 31) / 32) * p.planes, b16 = (long long)((p.Q + 15) / 16) * p.planes;
  const bool half = reg_is_half(p, DIR, N);
  if constexpr (MAIN && G <= 16) {
    if (b32 >= 2 * 148 && reg_pairs_ok(p))
      return half ? reg_plain_launch<N1, N2, DIR, 32, 2, true>(p, tw, s)
                  : reg_plain_launch<N1, N2, DIR, 32, 2, false>(p, tw, s);
  }
  if constexpr (MAIN) {
    if (half) return b16 < 148 ? reg_plain_launch<N1, N2, DIR, 4, 1, true>(p, tw, s)
                               : reg_plain_launch<N1, N2, DIR, 16, 1, true>(p, tw, s);
  }
  return b16 < 148 ? reg_plain_launch<N1, N2, DIR, 4, 1, false>(p, tw, s)
                   : reg_plain_launch<N1, N2, DIR, 16, 1, false>(p, tw, s);
}

// x passes with vec coils per thread: lines per CTA that make about 256
// threads (fewer where that would leave SMs without two bundles); false: the
// shape does not fit.
static inline bool reg_x_shape(int N1, int N2, int vec, RegPass& p, int out_len, bool sums, int* threads,
                               size_t* smem) {
  const int CG = p.C / vec, LT = reg_groups(N1, N2) * CG;
  if (LT > 1024) return false;
  const size_t line = (size_t)N1 * reg_block_stride(N2, p.C) * sizeof(float2) +
                      (sums ? (size_t)out_len * (CG | 1) * sizeof(float2) : 0);
  p.L = std::max(1, 256 / LT);
  while (p.L > 1 && ((p.lines + p.L - 1) / p.L < 2 * 148 || reg_tw_bytes(N1 * N2) + p.L * line > kRegSmemCap / 2))
    --p.L;
  *threads = (p.L * LT + 31) / 32 * 32;
  *smem = reg_tw_bytes(N1 * N2) + p.L * line;
  p.nbundles = (p.lines + p.L - 1) / p.L;
  return *smem <= kRegSmemCap;
}

template <int N1, int N2, bool MAIN>
static int reg_shanna_pass(const PassDesc& d, const float2* tw, cudaStream_t s, bool* done) {
  constexpr int N = N1 * N2;
  if (d.out_lo != 0 || d.out_len != N || d.out_half || d.out_stride[0] != d.C ||
      d.out_stride[1] != (long long)N * d.C || d.out_stride[2] != (long long)N * d.C * d.dims[1])
    return MLG_OK;
  RegPass p;
  p.out = d.out;
  p.C = d.C;
  p.in_lo = d.in_lo;
  p.in_len = d.in_len;
  p.lines = d.dims[1] * d.dims[2];
  p.ny = d.dims[1];
  p.par0 = (d.coord_off[1] + d.coord_off[2]) & 1;
  p.img = d.img;
  p.img_per_coil = d.img_per_coil;
  p.kfc = d.kfc;
  p.amax = d.out_absmax;
  int threads = 0, grid = 1;
  size_t smem = 0;
  if (!reg_x_shape(N1, N2, 1, p, 0, false, &threads, &smem)) return MLG_OK;
  constexpr int TB = reg_x_bound(N1, N2);
  *done = true;
  if constexpr (MAIN) {
    if (d.in_lo == N / 4 && d.in_len == N / 2)
      return threads <= TB ? reg_launch<reg_shanna_kernel<N1, N2, true, TB>>(p, tw, threads, smem, &grid, s)
                           : reg_launch<reg_shanna_kernel<N1, N2, true, 1024>>(p, tw, threads, smem, &grid, s);
  }
  return threads <= TB ? reg_launch<reg_shanna_kernel<N1, N2, false, TB>>(p, tw, threads, smem, &grid, s)
                       : reg_launch<reg_shanna_kernel<N1, N2, false, 1024>>(p, tw, threads, smem, &grid, s);
}

template <int N1, int N2, bool MAIN>
static int reg_nak_pass(const PassDesc& d, const float2* tw, int* n_partial, cudaStream_t s, bool* done) {
  constexpr int N = N1 * N2;
  if (d.in_lo != 0 || d.in_len != N || d.in_half || d.in_mask || d.in_stride[0] != d.C ||
      d.in_stride[1] != (long long)N * d.C || d.in_stride[2] != (long long)N * d.C * d.dims[1])
    return MLG_OK;
  RegPass p;
  p.in = d.in;
  p.C = d.C;
  p.out_lo = d.out_lo;
  p.out_len = d.out_len;
  p.lines = d.dims[1] * d.dims[2];
  p.ny = d.dims[1];
  p.par0 = (d.coord_off[1] + d.coord_off[2]) & 1;
  p.kfc = d.kfc;
  p.img_out = d.img_out;
  p.sfac = d.sfac;
  p.partial = d.partial;
  int threads = 0, grid = 1;
  size_t smem = 0;
  // two coils per thread for even coil counts and up to 16-point
  // sub-transforms (two 32-point ones would not fit the registers)
  constexpr bool kPairs = MAIN && reg_groups(N1, N2) <= 16;
  const int vec = kPairs && d.C % 2 == 0 ? 2 : 1;
  if (!reg_x_shape(N1, N2, vec, p, d.out_len, true, &threads, &smem)) return MLG_OK;
  constexpr int TB = reg_x_bound(N1, N2);
  if (threads > (vec == 2 ? 512 : 1024)) return MLG_OK;
  *done = true;
  auto run = [&](auto half, auto v) {
    constexpr bool H = decltype(half)::value;
    constexpr int V = decltype(v)::value;
    return threads <= TB
               ? reg_launch<reg_nak_kernel<N1, N2, H, V, TB>>(p, tw, threads, smem, &grid, s)
               : reg_launch<reg_nak_kernel<N1, N2, H, V, V == 2 ? 512 : 1024>>(p, tw, threads, smem, &grid, s);
  };
  using std::bool_constant;
  using std::integral_constant;
  int st;
  if constexpr (MAIN) {
    const bool half = d.out_lo == N / 4 && d.out_len == N / 2;
    if constexpr (kPairs) {
      if (vec == 2)
        st = half ? run(bool_constant<true>(), integral_constant<int, 2>())
                  : run(bool_constant<false>(), integral_constant<int, 2>());
      else
        st = half ? run(bool_constant<true>(), integral_constant<int, 1>())
                  : run(bool_constant<false>(), integral_constant<int, 1>());
    } else {
      st = half ? run(bool_constant<true>(), integral_constant<int, 1>())
                : run(bool_constant<false>(), integral_constant<int, 1>());
    }
  } else {
    st = run(bool_constant<false>(), integral_constant<int, 1>());
  }
  if (n_partial) *n_partial = d.partial ? grid : 0;
  return st;
}

// Pass `mode` over an axis of length A * B (A a multiple of 4): the forward
// splits it as N1 = A, N2 = B, the inverse as N1 = B, N2 = A, so that the
// rows that share an occupancy word are the same ones (row mod A) in both.
template <int A, int B, bool MAIN>
static int reg_dispatch(const FftAxisPlan& ax, PassMode mode, const PassDesc& d, int* n_partial, cudaStream_t s,
                        bool* done) {
  static_assert(A % 4 == 0 && A <= 32 && B <= 32, "register pass split");
  if (mode == PassMode::kShannaIn) return reg_shanna_pass<A, B, MAIN>(d, ax.rtw[0], s, done);
  if (mode == PassMode::kNakatshaOut) return reg_nak_pass<B, A, MAIN>(d, ax.rtw[1], n_partial, s, done);
  if (d.dir < 0) return reg_plain_pass<A, B, -1, MAIN>(d, ax.rtw[0], s, done);
  return reg_plain_pass<B, A, 1, MAIN>(d, ax.rtw[1], s, done);
}

}  // namespace mlg

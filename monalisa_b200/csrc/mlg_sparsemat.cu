// Sparse gridding-matrix products on the device (Gu / Gut / Gn and the
// generic bmSparseMat_vec family).
//
// The reference (bmSparseMat_cC_oBlock_omp_mex.cpp:106-260) streams the whole
// matrix once per coil and per real/imaginary part.  Here one launch covers
// every coil: a thread owns one (row, coil) output and walks the row's
// entries in stored order with explicit round-to-nearest multiply and add
// (no FMA contraction), so short rows reproduce the reference's
// floating-point result bit for bit.  Rows longer than kLongRow entries (the
// k-space centre of Gut, which every radial spoke crosses) get a whole CTA
// that splits the entries over thread groups and reduces the partial sums in
// a fixed order.
//
// Two thread mappings: coil-fastest (lanes of a warp = coils of one row;
// used when the output is coil-fastest, e.g. Gu -> k-space) and row-fastest
// (lanes = consecutive rows of one coil; used when the output is coil-major,
// e.g. Gut -> grid), so the output side is always coalesced.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "mlg_internal.cuh"

namespace mlg {

struct SpmmParams {
  const uint32_t* row_ptr;
  const int* col;
  const float* val;
  const __half* val_h;  // FP16 values in place of val when set
  int l_size;
  int nCh;
  int rows_per_block;
  const int* long_rows;
  int n_long;
  Operand in;
  Operand out;
  const float* in_row_scale;
  float out_scale;
  int normalize;
  const float* sqn_w;
  double* partial;
  int partial_long_offset;
  unsigned* absmax;
  // FP16 point-layout input (spmm_fwd_kernel, IN_H): scale from this word and length
  const unsigned* in_h_amax;
  int in_h_len;
};

__device__ __forceinline__ float abs_max4(float4 v) {
  return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}

// The block's largest value (v >= 0) into *absmax: one atomic per block, and
// none when the recorded value is already as large -- atomics on one word
// serialise, and a product has thousands of blocks.  Every thread of the
// block must call.
__device__ __forceinline__ void block_absmax(unsigned* absmax, float v) {
  __shared__ float wmax[32];
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, wmax[w]);
    const unsigned u = __float_as_uint(m);
    if (u > *reinterpret_cast<volatile const unsigned*>(absmax)) atomicMax(absmax, u);
  }
}

template <Layout L>
__device__ __forceinline__ float2 ld(const Operand& o, long long row, int c, int nCh) {
  if constexpr (L == Layout::kPointC64) {
    return __ldg(reinterpret_cast<const float2*>(o.a) + row * nCh + c);
  } else if constexpr (L == Layout::kCoilC64) {
    return __ldg(reinterpret_cast<const float2*>(o.a) + (long long)c * o.rows + row);
  } else if constexpr (L == Layout::kCoilSplit) {
    const long long i = (long long)c * o.rows + row;
    return make_float2(__ldg(reinterpret_cast<const float*>(o.a) + i), __ldg(reinterpret_cast<const float*>(o.b) + i));
  } else if constexpr (L == Layout::kPointSplit) {
    const long long i = row * nCh + c;
    return make_float2(__ldg(reinterpret_cast<const float*>(o.a) + i), __ldg(reinterpret_cast<const float*>(o.b) + i));
  } else if constexpr (L == Layout::kPointReal) {
    return make_float2(__ldg(reinterpret_cast<const float*>(o.a) + row * nCh + c), 0.f);
  } else {
    return make_float2(__ldg(reinterpret_cast<const float*>(o.a) + (long long)c * o.rows + row), 0.f);
  }
}

template <Layout L>
__device__ __forceinline__ void st(const Operand& o, long long row, int c, int nCh, float2 v) {
  if constexpr (L == Layout::kPointC64) {
    reinterpret_cast<float2*>(o.a)[row * nCh + c] = v;
  } else if constexpr (L == Layout::kCoilC64) {
    reinterpret_cast<float2*>(o.a)[(long long)c * o.rows + row] = v;
  } else if constexpr (L == Layout::kCoilSplit) {
    const long long i = (long long)c * o.rows + row;
    reinterpret_cast<float*>(o.a)[i] = v.x;
    reinterpret_cast<float*>(o.b)[i] = v.y;
  } else if constexpr (L == Layout::kPointSplit) {
    const long long i = row * nCh + c;
    reinterpret_cast<float*>(o.a)[i] = v.x;
    reinterpret_cast<float*>(o.b)[i] = v.y;
  } else if constexpr (L == Layout::kPointReal) {
    reinterpret_cast<float*>(o.a)[row * nCh + c] = v.x;
  } else {
    reinterpret_cast<float*>(o.a)[(long long)c * o.rows + row] = v.x;
  }
}

__device__ __forceinline__ float val_at(const SpmmParams& p, uint32_t k) {
  return p.val_h ? __half2float(p.val_h[k]) : __ldg(p.val + k);
}

// Accumulates entries [b, e) with stride `step` of one row for coil c.
template <Layout IN>
__device__ __forceinline__ void accumulate(const SpmmParams& p, uint32_t b, uint32_t e, uint32_t step, int c,
                                           float& ax, float& ay, float& ws) {
  const bool scale = p.in_row_scale != nullptr;
#pragma unroll 4
  for (uint32_t k = b; k < e; k += step) {
    const int j = __ldg(p.col + k);
    const float m = val_at(p, k);
    float2 v = ld<IN>(p.in, j, c, p.nCh);
    if (scale) {
      const float h = __ldg(p.in_row_scale + j);
      v.x = __fmul_rn(h, v.x);
      v.y = __fmul_rn(h, v.y);
    }
    ax = __fadd_rn(ax, __fmul_rn(m, v.x));
    ay = __fadd_rn(ay, __fmul_rn(m, v.y));
    ws = __fadd_rn(ws, m);
  }
}

template <Layout OUT>
__device__ __forceinline__ double finish(const SpmmParams& p, long long r, int c, float ax, float ay, float ws) {
  if (p.normalize) {
    // bmGridder_n2u_mex.cpp:178-191: divide by the weight sum, 1 if < 1e-5
    const float s = ws < 1e-5f ? 1.0f : ws;
    ax = __fdiv_rn(ax, s);
    ay = __fdiv_rn(ay, s);
  }
  if (p.out_scale != 1.0f) {
    ax = __fmul_rn(ax, p.out_scale);
    ay = __fmul_rn(ay, p.out_scale);
  }
  st<OUT>(p.out, r, c, p.nCh, make_float2(ax, ay));
  if (p.absmax) atomicMax(p.absmax, __float_as_uint(fmaxf(fabsf(ax), fabsf(ay))));
  if (p.partial) {
    const double w = p.sqn_w ? (double)__ldg(p.sqn_w + r) : 1.0;
    return w * ((double)ax * ax + (double)ay * ay);
  }
  return 0.0;
}

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += sh[i];
  }
  return t;
}

template <Layout IN, Layout OUT, bool ROW_FAST>
__global__ void __launch_bounds__(256) spmm_short_kernel(SpmmParams p) {
  __shared__ double sh[32];
  const long long r0 = (long long)blockIdx.x * p.rows_per_block;
  const int nrows = (int)min((long long)p.rows_per_block, (long long)p.l_size - r0);
  const int items = nrows * p.nCh;
  double sq = 0.0;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    int lr, c;
    if (ROW_FAST) {
      lr = it % nrows;
      c = it / nrows;
    } else {
      c = it % p.nCh;
      lr = it / p.nCh;
    }
    const long long r = r0 + lr;
    const uint32_t b = __ldg(p.row_ptr + r), e = __ldg(p.row_ptr + r + 1);
    if (e - b > (uint32_t)kLongRow) continue;  // owned by spmm_long_kernel
    float ax = 0.f, ay = 0.f, ws = 0.f;
    accumulate<IN>(p, b, e, 1u, c, ax, ay, ws);
    sq += finish<OUT>(p, r, c, ax, ay, ws);
  }
  if (p.partial) {
    const double t = block_sum(sq, sh);
    if (threadIdx.x == 0) p.partial[blockIdx.x] = t;
  }
}

// Long rows: one CTA per segment of at most kSegLen entries.  Thread groups
// of `cper` coils split the segment's entries (stride = number of groups);
// the group partials are summed in group order and written, per coil, to
// seg_scratch[segment][coil] = (re, im, weight sum).
template <Layout IN>
__global__ void __launch_bounds__(256) spmm_seg_kernel(SpmmParams p, const uint32_t* __restrict__ seg_lo,
                                                       const uint32_t* __restrict__ seg_hi, float3* scratch) {
  __shared__ float3 part[256];
  const uint32_t b = __ldg(seg_lo + blockIdx.x), e = __ldg(seg_hi + blockIdx.x);
  const int cper = min(p.nCh, (int)blockDim.x);   // coils per pass
  const int groups = (int)blockDim.x / cper;      // entry groups per coil
  for (int c0 = 0; c0 < p.nCh; c0 += cper) {
    const int cl = threadIdx.x % cper, g = threadIdx.x / cper;
    const int c = c0 + cl;
    float ax = 0.f, ay = 0.f, ws = 0.f;
    if (g < groups && c < p.nCh) accumulate<IN>(p, b + g, e, (uint32_t)groups, c, ax, ay, ws);
    __syncthreads();
    part[threadIdx.x] = make_float3(ax, ay, ws);
    __syncthreads();
    if ((int)threadIdx.x < cper && c0 + (int)threadIdx.x < p.nCh) {
      float sx = 0.f, sy = 0.f, sw = 0.f;
      for (int gg = 0; gg < groups; ++gg) {  // fixed order: deterministic
        const float3 q = part[gg * cper + threadIdx.x];
        sx = __fadd_rn(sx, q.x);
        sy = __fadd_rn(sy, q.y);
        sw = __fadd_rn(sw, q.z);
      }
      scratch[(long long)blockIdx.x * p.nCh + c0 + threadIdx.x] = make_float3(sx, sy, sw);
    }
  }
}

// One CTA per long row: sums its segments in segment order, then finishes
// (normalise / scale / store / FP64 partial) like the short-row kernel.
template <Layout OUT>
__global__ void __launch_bounds__(256) spmm_seg_combine_kernel(SpmmParams p, const int* __restrict__ seg0,
                                                               const float3* __restrict__ scratch) {
  __shared__ double sh[32];
  const long long r = __ldg(p.long_rows + blockIdx.x);
  const int s0 = __ldg(seg0 + blockIdx.x), s1 = __ldg(seg0 + blockIdx.x + 1);
  double sq = 0.0;
  for (int c = threadIdx.x; c < p.nCh; c += blockDim.x) {
    float sx = 0.f, sy = 0.f, sw = 0.f;
    for (int k = s0; k < s1; ++k) {
      const float3 q = scratch[(long long)k * p.nCh + c];
      sx = __fadd_rn(sx, q.x);
      sy = __fadd_rn(sy, q.y);
      sw = __fadd_rn(sw, q.z);
    }
    sq += finish<OUT>(p, r, c, sx, sy, sw);
  }
  if (p.partial) {
    const double t = block_sum(sq, sh);
    if (threadIdx.x == 0) p.partial[p.partial_long_offset + blockIdx.x] = t;
  }
}

// Rows with more than kMidRow entries inside the operators, cut into units of
// at most kUnitLen entries (Csr::heavy_units).
struct HeavyUnits {
  const int4* units = nullptr;
  const int2* multi = nullptr;
  int n = 0;                  // units = first blocks of the launch
  float* scratch = nullptr;   // partial sums of the multi-unit rows' units
  unsigned* count = nullptr;  // finished units per multi-unit row
};

__device__ __forceinline__ void fma_to(float4& a, float m, float4 v) {
  const float2 lo = __ffma2_rn(make_float2(m, m), make_float2(v.x, v.y), make_float2(a.x, a.y));
  const float2 hi = __ffma2_rn(make_float2(m, m), make_float2(v.z, v.w), make_float2(a.z, a.w));
  a = make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void fma_to(float2& a, float m, float2 v) { a = __ffma2_rn(make_float2(m, m), v, a); }
__device__ __forceinline__ float4 add_to(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ float2 add_to(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float4 scaled(float4 a, float f) {
  return make_float4(__fmul_rn(a.x, f), __fmul_rn(a.y, f), __fmul_rn(a.z, f), __fmul_rn(a.w, f));
}
__device__ __forceinline__ float2 scaled(float2 a, float f) { return make_float2(__fmul_rn(a.x, f), __fmul_rn(a.y, f)); }
__device__ __forceinline__ float abs_max4(float2 v) { return fmaxf(fabsf(v.x), fabsf(v.y)); }
__device__ __forceinline__ double sqnorm(float4 a) {
  return (double)a.x * a.x + (double)a.y * a.y + (double)a.z * a.z + (double)a.w * a.w;
}
__device__ __forceinline__ double sqnorm(float2 a) { return (double)a.x * a.x + (double)a.y * a.y; }
template <class VT>
__device__ __forceinline__ VT vzero();
template <>
__device__ __forceinline__ float4 vzero<float4>() { return make_float4(0.f, 0.f, 0.f, 0.f); }
template <>
__device__ __forceinline__ float2 vzero<float2>() { return make_float2(0.f, 0.f); }

// One heavy unit by one CTA of 256 threads (operator semantics: the row scale
// folded into the matrix value, fused multiply-adds, FP32 point layout; VT =
// float4: a coil pair per thread, float2: a coil): thread = (entry group eg,
// coil column pi), group eg takes entries eg, eg + EG, ... four at a time in
// flight, the groups' sums are added in a fixed tree.  A unit that is a whole
// row stores it; the units of a longer row leave their sums in scratch and
// the last one to finish adds them in a fixed order (deterministic).
//
// A warp per such row left a chain of up to 52 dependent gathers (60 us in
// 2-D, where nothing covers it), and the rows above 256 entries took two more
// launches (33 of 135 us on an eighth of the 4096-spoke case).
template <class VT, bool AM>
__device__ __forceinline__ void heavy_unit(const SpmmParams& p, const HeavyUnits& H, int unit) {
  __shared__ VT red[256];
  __shared__ bool last;
  const int P = p.nCh / (int)(sizeof(VT) / sizeof(float2)), EG = 256 / P;
  const int eg = threadIdx.x / P, pi = threadIdx.x - eg * P;
  const bool scale = p.in_row_scale != nullptr;
  const VT* in = reinterpret_cast<const VT*>(p.in.a);
  const int4 u = __ldg(H.units + unit);
  VT acc = vzero<VT>();
  if (eg < EG) {
    for (uint32_t k = (uint32_t)u.y + eg; k < (uint32_t)u.z; k += 4 * EG) {
      int j[4];
      float m[4];
      VT v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t kq = k + q * EG;
        const bool ok = kq < (uint32_t)u.z;
        j[q] = ok ? __ldg(p.col + kq) : -1;
        m[q] = ok ? val_at(p, kq) : 0.f;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[q] = vzero<VT>();
        if (j[q] >= 0) {
          v[q] = __ldg(in + (long long)j[q] * P + pi);
          if (scale) m[q] = __fmul_rn(m[q], __ldg(p.in_row_scale + j[q]));
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) fma_to(acc, m[q], v[q]);  // (past the end: 0 * 0)
    }
  }
  int top = 1;
  while (top < EG) top <<= 1;
  auto tree = [&](VT x) {  // the sum over the entry groups, in group 0
    red[threadIdx.x] = x;
    for (int w = top >> 1; w > 0; w >>= 1) {
      __syncthreads();
      if (eg < w && eg + w < EG) red[threadIdx.x] = add_to(red[threadIdx.x], red[threadIdx.x + w * P]);
    }
    __syncthreads();
    return red[threadIdx.x];
  };
  acc = tree(acc);
  bool store = eg == 0;
  if (u.w >= 0) {
    VT* part = reinterpret_cast<VT*>(H.scratch);
    const int2 mu = __ldg(H.multi + u.w);
    if (eg == 0) {
      part[(long long)unit * P + pi] = acc;
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      last = atomicAdd(H.count + u.w, 1u) == (unsigned)(mu.y - 1);
      if (last) H.count[u.w] = 0u;
      __threadfence();
    }
    __syncthreads();
    if (last) {
      VT sum = vzero<VT>();
      if (eg < EG)
        for (int k = eg; k < mu.y; k += EG) sum = add_to(sum, __ldcg(part + (long long)(mu.x + k) * P + pi));
      acc = tree(sum);
    } else {
      store = false;
    }
  }
  float amax = 0.f;
  if (store) {
    if (p.out_scale != 1.0f) acc = scaled(acc, p.out_scale);
    reinterpret_cast<VT*>(p.out.a)[(long long)u.x * P + pi] = acc;
    amax = abs_max4(acc);
  }
  if constexpr (AM) block_absmax(p.absmax, amax);  // every thread of the block reaches it
}

// Operator products whose input rows are scaled (the adjoint without row
// records, or of every row), point layout in and out, even nCh: a thread owns
// a (row, coil pair) output and moves 16 bytes per load and store; the row's
// column/value stream is read once per pair instead of once per coil.  `rows`
// (optional) lists the rows to compute, in that order (the matrix's ord_rows),
// and `bounds` their entry ranges; other rows are left untouched.  Entries are
// summed in stored order with the row scale folded into the matrix value and
// fused multiply-adds.  Eight 256-thread blocks per SM (32 registers, a few
// spilled bytes): the gathers are latency-bound.  HEAVY: the first heavy.n
// blocks gather the heavy units, a CTA each (heavy_unit), the others the
// listed short rows: one launch, the longest-running blocks first.
template <bool HEAVY>
__global__ void __launch_bounds__(256, 8) spmm_pair_kernel(SpmmParams p, const int* __restrict__ rows,
                                                           const uint2* __restrict__ bounds, int n_rows,
                                                           HeavyUnits heavy) {
  int bid = (int)blockIdx.x;
  if constexpr (HEAVY) {
    if (bid < heavy.n) {
      if (p.absmax)
        heavy_unit<float4, true>(p, heavy, bid);
      else
        heavy_unit<float4, false>(p, heavy, bid);
      return;
    }
    bid -= heavy.n;
  }
  const int P = p.nCh >> 1;
  const long long i0 = (long long)bid * p.rows_per_block;
  const int nr = (int)min((long long)p.rows_per_block, (long long)n_rows - i0);
  const int total = nr * P;
  const bool scale = p.in_row_scale != nullptr;
  const float4* in = reinterpret_cast<const float4*>(p.in.a);
  float amax = 0.f;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int lr = it / P, pi = it - lr * P;
    long long r;
    uint32_t b, e;
    if (rows) {  // listed rows: bounds loaded beside the row index, not after it
      r = __ldg(rows + i0 + lr);
      const uint2 be = __ldg(bounds + i0 + lr);
      b = be.x;
      e = be.y;
    } else {
      r = i0 + lr;
      b = __ldg(p.row_ptr + r);
      e = __ldg(p.row_ptr + r + 1);
    }
    if (e - b > (uint32_t)kLongRow) continue;  // segment kernels own it
    float4 acc = vzero<float4>();
#pragma unroll 4
    for (uint32_t k = b; k < e; ++k) {
      const int j = __ldg(p.col + k);
      float m = val_at(p, k);
      const float4 v = __ldg(in + (long long)j * P + pi);
      if (scale) m = __fmul_rn(m, __ldg(p.in_row_scale + j));
      fma_to(acc, m, v);
    }
    if (p.out_scale != 1.0f) acc = scaled(acc, p.out_scale);
    reinterpret_cast<float4*>(p.out.a)[r * P + pi] = acc;
    amax = fmaxf(amax, abs_max4(acc));
  }
  if (p.absmax) block_absmax(p.absmax, amax);
}

// VT values at an index of the input: FP32, or (IN_H) __half2 values times a
// power of two (the mixed-precision forward grid), 8 bytes per coil pair.
template <class VT, bool IN_H>
struct GridIn {
  using T = VT;
  static __device__ __forceinline__ VT at(const T* a, float) { return __ldg(a); }
};
template <>
struct GridIn<float4, true> {
  using T = uint2;
  static __device__ __forceinline__ float4 at(const T* a, float hin) {
    const uint2 q = __ldg(a);
    const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
    const float2 y = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
    return make_float4(x.x * hin, x.y * hin, y.x * hin, y.y * hin);
  }
};

__device__ __forceinline__ float4 mul_add_rn(float4 a, float m, float4 v) {
  return make_float4(__fadd_rn(a.x, __fmul_rn(m, v.x)), __fadd_rn(a.y, __fmul_rn(m, v.y)),
                     __fadd_rn(a.z, __fmul_rn(m, v.z)), __fadd_rn(a.w, __fmul_rn(m, v.w)));
}
__device__ __forceinline__ float2 mul_add_rn(float2 a, float m, float2 v) {
  return make_float2(__fadd_rn(a.x, __fmul_rn(m, v.x)), __fadd_rn(a.y, __fmul_rn(m, v.y)));
}

// Products of all rows without scales, point layout: the forward operator
// (CONTRACT: fused multiply-adds) and the plain complex product (separate
// round-to-nearest multiply and add: bit-identical to the reference's CPU
// products), entries in stored order; a thread per (row, coil pair; VT =
// float2: coil).  Latency-bound gathers of rows of equal length (27 entries in
// 3-D): the columns, gathers and values of kFwdBatch entries are issued as
// three groups before any is used.  Left to the compiler (unroll 4 at eight
// blocks per SM, 32 registers) the loads of a batch waited for each other; at
// six blocks (40 registers) four entries in flight take the 256^3 x 16-coil
// product from 414 to 308 us, 192^3 x 12 coils 105 -> 75, 160 x 160 x 120 x 8
// coils 62 -> 45, 512^2 x 12 coils 24 -> 19 us (3 entries at 6 blocks 316,
// 5 at 5 blocks 314, 6 at 5 339, 4 at 8 364 us).
constexpr int kFwdBatch = 4;

template <class VT, bool HV, bool IN_H, bool CONTRACT>
__global__ void __launch_bounds__(256, 6) spmm_fwd_kernel(SpmmParams p) {
  __shared__ double sh[32];
  const int P = p.nCh / (int)(sizeof(VT) / sizeof(float2));
  const long long i0 = (long long)blockIdx.x * p.rows_per_block;
  const int nr = (int)min((long long)p.rows_per_block, (long long)p.l_size - i0);
  const int total = nr * P;
  using In = GridIn<VT, IN_H>;
  const typename In::T* in = reinterpret_cast<const typename In::T*>(p.in.a);
  const float hin = IN_H ? 1.f / half_store_scale(p.in_h_amax, p.in_h_len) : 1.f;  // a power of two
  double sq = 0.0;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int lr = it / P, pi = it - lr * P;
    const long long r = i0 + lr;
    uint32_t k = __ldg(p.row_ptr + r);
    const uint32_t e = __ldg(p.row_ptr + r + 1);
    if (e - k > (uint32_t)kLongRow) continue;  // segment kernels own it
    VT acc = vzero<VT>();
    const typename In::T* const src = in + pi;
    auto add = [&](float mm, VT vv) {
      if constexpr (CONTRACT)
        fma_to(acc, mm, vv);
      else
        acc = mul_add_rn(acc, mm, vv);
    };
    for (; k + kFwdBatch <= e; k += kFwdBatch) {
      int j[kFwdBatch];
      VT v[kFwdBatch];
      float m[kFwdBatch];
#pragma unroll
      for (int q = 0; q < kFwdBatch; ++q) j[q] = __ldg(p.col + k + q);
#pragma unroll
      for (int q = 0; q < kFwdBatch; ++q) v[q] = In::at(src + (long long)j[q] * P, hin);
#pragma unroll
      for (int q = 0; q < kFwdBatch; ++q) m[q] = HV ? __half2float(p.val_h[k + q]) : __ldg(p.val + k + q);
#pragma unroll
      for (int q = 0; q < kFwdBatch; ++q) add(m[q], v[q]);
    }
    for (; k < e; ++k)
      add(HV ? __half2float(p.val_h[k]) : __ldg(p.val + k), In::at(src + (long long)__ldg(p.col + k) * P, hin));
    reinterpret_cast<VT*>(p.out.a)[r * P + pi] = acc;
    if (p.partial) {
      const double w = p.sqn_w ? (double)__ldg(p.sqn_w + r) : 1.0;
      sq += w * sqnorm(acc);
    }
  }
  if (p.partial) {
    const double t = block_sum(sq, sh);
    if (threadIdx.x == 0) p.partial[blockIdx.x] = t;
  }
}

// Short rows of an ordered non-empty product from their records (CONTRACT,
// FP32 point layout in and out): a thread per (row, coil pair; VT = float2:
// coil, for odd coil counts) reads the row's 32-byte record -- cell, count and
// up to kRecInline (column, value) pairs -- and issues every gather of the
// row at once, so such a row costs two dependent loads (record -> inputs)
// instead of three (bounds -> entry -> input), and the record stream is
// smaller than the bounds and entries it replaces.  Rows with more entries
// loop over their CSR entries.  Per coil the entries are summed in stored
// order with the same fused multiply-adds as spmm_pair_kernel: the outputs
// are identical.  With FP16 matrix values (p.val_h) the inline FP32 values are
// rounded to FP16 as they are read, which gives the values the CSR rows read
// from val_h.  The first heavy.n blocks gather the heavy units, as there.
// p.absmax (optional) is raised to the largest output component.
//
// Latency-bound gathers: the entries of longer rows go four at a time, as in
// spmm_fwd_kernel, and a brick's rows are sorted by length (csr_build_order),
// so that the rows of a warp (four at 16 coils) take one path.  MB resident
// blocks per SM: six (40 registers), eight (32, a few spilled bytes) where the
// k-space exceeds half the L2 and the gathers' latency grows (256^3 x 16
// coils, 134 MB: 499 us at eight, 531 at six; 192^3 x 12 coils, 21 MB: 99 at
// either, 512^2 x 12 coils 31 at six, 39 us at eight).  With the heavy units
// in the launch Gut went from 606 to 499, 162 to 99, 122 to 59 (160 x 160 x
// 120 x 8 coils) and 95 to 29 us.  (Measured and not kept: a warp's lanes
// loading a row's entries together and passing them by shuffles, 512 and 124
// us; two rows' records loaded before either row's gathers, 0.709 against
// 0.610 ms then.)
template <class VT, bool HV, bool AM, int MB>
__global__ void __launch_bounds__(256, MB) spmm_rec_kernel(SpmmParams p, const uint4* __restrict__ rec, int n_rows,
                                                           HeavyUnits heavy) {
  if ((int)blockIdx.x < heavy.n) {
    heavy_unit<VT, AM>(p, heavy, blockIdx.x);
    return;
  }
  const int bid = (int)blockIdx.x - heavy.n;
  const int P = p.nCh / (int)(sizeof(VT) / sizeof(float2));
  const long long i0 = (long long)bid * p.rows_per_block;
  const int nr = (int)min((long long)p.rows_per_block, (long long)n_rows - i0);
  const int total = nr * P;
  const bool scale = p.in_row_scale != nullptr;
  const VT* in = reinterpret_cast<const VT*>(p.in.a);
  float amax = 0.f;
  auto row = [&](const uint4 h0, const uint4 h1, const int pi) {
    const long long r = (int)h0.x;
    const uint32_t n = h0.y;
    VT acc = vzero<VT>();
    if (n <= (uint32_t)kRecInline) {
      const uint32_t c0 = h0.z, c1 = h1.x, c2 = h1.z;
      VT v0 = vzero<VT>(), v1 = v0, v2 = v0;
      float m0 = __uint_as_float(h0.w), m1 = __uint_as_float(h1.y), m2 = __uint_as_float(h1.w);
      if constexpr (HV) {  // FP16 matrix values: the inline FP32 values rounded alike
        m0 = __half2float(__float2half_rn(m0));
        m1 = __half2float(__float2half_rn(m1));
        m2 = __half2float(__float2half_rn(m2));
      }
      if (n > 0) v0 = __ldg(in + (long long)c0 * P + pi);
      if (n > 1) v1 = __ldg(in + (long long)c1 * P + pi);
      if (n > 2) v2 = __ldg(in + (long long)c2 * P + pi);
      if (scale) {
        if (n > 0) m0 = __fmul_rn(m0, __ldg(p.in_row_scale + c0));
        if (n > 1) m1 = __fmul_rn(m1, __ldg(p.in_row_scale + c1));
        if (n > 2) m2 = __fmul_rn(m2, __ldg(p.in_row_scale + c2));
      }
      if (n > 0) fma_to(acc, m0, v0);
      if (n > 1) fma_to(acc, m1, v1);
      if (n > 2) fma_to(acc, m2, v2);
    } else {
      constexpr int U = 4;
      const VT* const src = in + pi;
      uint32_t k = h0.z;
      const uint32_t e = k + n;
      for (; k + U <= e; k += U) {
        int j[U];
        float m[U];
        VT v[U];
#pragma unroll
        for (int q = 0; q < U; ++q) j[q] = __ldg(p.col + k + q);
#pragma unroll
        for (int q = 0; q < U; ++q) v[q] = __ldg(src + (long long)j[q] * P);
#pragma unroll
        for (int q = 0; q < U; ++q) {
          m[q] = HV ? __half2float(p.val_h[k + q]) : __ldg(p.val + k + q);
          if (scale) m[q] = __fmul_rn(m[q], __ldg(p.in_row_scale + j[q]));
        }
#pragma unroll
        for (int q = 0; q < U; ++q) fma_to(acc, m[q], v[q]);
      }
      if (k < e) {  // up to three more
        int j[U - 1];
        float m[U - 1];
        VT v[U - 1];
#pragma unroll
        for (int q = 0; q < U - 1; ++q) j[q] = k + q < e ? __ldg(p.col + k + q) : -1;
#pragma unroll
        for (int q = 0; q < U - 1; ++q) {
          v[q] = vzero<VT>();
          m[q] = 0.f;
          if (j[q] >= 0) {
            v[q] = __ldg(src + (long long)j[q] * P);
            m[q] = HV ? __half2float(p.val_h[k + q]) : __ldg(p.val + k + q);
            if (scale) m[q] = __fmul_rn(m[q], __ldg(p.in_row_scale + j[q]));
          }
        }
#pragma unroll
        for (int q = 0; q < U - 1; ++q)
          if (j[q] >= 0) fma_to(acc, m[q], v[q]);
      }
    }
    if (p.out_scale != 1.0f) acc = scaled(acc, p.out_scale);
    reinterpret_cast<VT*>(p.out.a)[r * P + pi] = acc;
    if constexpr (AM) amax = fmaxf(amax, abs_max4(acc));
  };
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int lr = it / P;
    const uint4* rp = rec + (i0 + lr) * 2;
    row(__ldg(rp), __ldg(rp + 1), it - lr * P);
  }
  if constexpr (AM) block_absmax(p.absmax, amax);
}

// Rows per block of spmm_rec_kernel: a quarter of a brick's non-empty rows or
// so (rows of neighbouring cells share samples in L1), more for the large
// k-spaces, fewer where that would leave resident blocks without work.
// Measured on 192^3 x 12, 160^2 x 120 x 8 and 512^2 x 12 coils: 64 rows 109 /
// 64 / 29, 128 rows 99 / 58 / 36, 192 rows 99 / 63 / 46 us; on 256^3 x 16: 96
// rows 521, 128 511, 192 499 us.
static int rec_rows_per_block(int n_rows, int P, bool large) {
  const int rows = std::min(large ? 192 : 128, n_rows / (148 * 24));
  return std::max(rows, (256 + P - 1) / P);
}

template <class VT, bool HV, bool AM>
static void launch_rec(const SpmmParams& p, const uint4* rec, int n_rows, const HeavyUnits& heavy, bool large,
                       cudaStream_t s) {
  SpmmParams q = p;
  q.rows_per_block = rec_rows_per_block(n_rows, p.nCh / (int)(sizeof(VT) / sizeof(float2)), large);
  const int g = heavy.n + (n_rows + q.rows_per_block - 1) / q.rows_per_block;
  if (g == 0) return;
  if (large)
    spmm_rec_kernel<VT, HV, AM, 8><<<g, 256, 0, s>>>(q, rec, n_rows, heavy);
  else
    spmm_rec_kernel<VT, HV, AM, 6><<<g, 256, 0, s>>>(q, rec, n_rows, heavy);
}

template <class VT>
static void launch_rec(const SpmmParams& p, const Csr& m, const HeavyUnits& heavy, cudaStream_t s) {
  const uint4* rec = reinterpret_cast<const uint4*>(m.ord_rec);
  const bool large = (size_t)m.r_size * p.nCh * sizeof(float2) > (64u << 20);  // half the L2
  if (p.val_h)
    p.absmax ? launch_rec<VT, true, true>(p, rec, m.ord_short, heavy, large, s)
             : launch_rec<VT, true, false>(p, rec, m.ord_short, heavy, large, s);
  else
    p.absmax ? launch_rec<VT, false, true>(p, rec, m.ord_short, heavy, large, s)
             : launch_rec<VT, false, false>(p, rec, m.ord_short, heavy, large, s);
}

// Whether a product runs as spmm_fwd_kernel: complex point layout, all rows in
// row order, no scales, no recorded maximum.
static bool use_fwd_kernel(const SpmmArgs& a) {
  return a.in.layout == Layout::kPointC64 && a.out.layout == Layout::kPointC64 && !a.normalize &&
         (a.contract || !a.half_values) && !a.nonempty_only && !a.long_only && !a.in_row_scale && a.out_scale == 1.0f && !a.absmax &&
         !(a.m->ord_rows && !a.m->ord_nonempty);
}

static void launch_fwd(const SpmmParams& p, bool contract, int grid, cudaStream_t s) {
  if (!contract) {
    p.nCh % 2 ? spmm_fwd_kernel<float2, false, false, false><<<grid, 256, 0, s>>>(p)
              : spmm_fwd_kernel<float4, false, false, false><<<grid, 256, 0, s>>>(p);
  } else if (p.nCh % 2) {
    p.val_h ? spmm_fwd_kernel<float2, true, false, true><<<grid, 256, 0, s>>>(p)
            : spmm_fwd_kernel<float2, false, false, true><<<grid, 256, 0, s>>>(p);
  } else if (p.in_h_amax) {
    p.val_h ? spmm_fwd_kernel<float4, true, true, true><<<grid, 256, 0, s>>>(p)
            : spmm_fwd_kernel<float4, false, true, true><<<grid, 256, 0, s>>>(p);
  } else {
    p.val_h ? spmm_fwd_kernel<float4, true, false, true><<<grid, 256, 0, s>>>(p)
            : spmm_fwd_kernel<float4, false, false, true><<<grid, 256, 0, s>>>(p);
  }
}

__global__ void rec_build_kernel(const int* __restrict__ rows, const uint2* __restrict__ bounds, int n,
                                 const int* __restrict__ col, const float* __restrict__ val,
                                 uint32_t* __restrict__ rec) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint2 be = bounds[i];
    const uint32_t len = be.y - be.x;
    uint32_t w[8] = {};
    w[0] = (uint32_t)rows[i];
    w[1] = len;
    if (len <= (uint32_t)kRecInline) {
      for (uint32_t k = 0; k < len; ++k) {
        w[2 + 2 * k] = (uint32_t)col[be.x + k];
        w[3 + 2 * k] = __float_as_uint(val[be.x + k]);
      }
    } else {
      w[2] = be.x;
    }
    uint4* o = reinterpret_cast<uint4*>(rec) + 2 * (size_t)i;
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// MLG_GUT_REC=0 / 1 forces the CSR rows / the records in every product;
// unset: SpmmArgs::records (the plan's variant) decides.
static int records_forced() {
  static const int v = [] {
    const char* e = std::getenv("MLG_GUT_REC");
    return e ? (std::strcmp(e, "0") == 0 ? 0 : (std::strcmp(e, "1") == 0 ? 1 : -1)) : -1;
  }();
  return v;
}

int csr_build_records(Csr& c, cudaStream_t s) {
  if (c.ord_rec || !c.ord_rows || !c.ord_nonempty || c.ord_short <= 0 || !c.val) return MLG_OK;
  MLG_CUDA(cudaMalloc(&c.ord_rec, 32 * (size_t)c.ord_short));
  const int g = std::max(1, std::min(148 * 16, (c.ord_short + 255) / 256));
  rec_build_kernel<<<g, 256, 0, s>>>(c.ord_rows, c.ord_bounds, c.ord_short, c.col, c.val, c.ord_rec);
  MLG_LAUNCHED();
  return MLG_OK;
}

// complex point layout in and out, whole coil pairs
static bool point_pairs(const SpmmArgs& a) {
  return a.in.layout == Layout::kPointC64 && a.out.layout == Layout::kPointC64 && (a.nCh % 2) == 0 && !a.normalize;
}

static bool use_pair_kernel(const SpmmArgs& a) { return point_pairs(a) && a.contract && !a.partial; }

static long long spmm_rows(const SpmmArgs& a) { return a.nonempty_only ? a.m->n_nonempty : a.m->l_size; }

// Rows per CTA of the row-per-thread-group products: a thread's share is four
// rows where there are enough of them, fewer where the CTAs would not fill
// 148 SMs x 6 (a product's few hundred CTAs of four rows each are a chain of
// dependent gathers on a part of the chip).  Gu of a 64^3 grid, 1 coil: 25 -> 12
// us, 96^3 x 4 coils 25 -> 15, 256^2 x 8 coils 12.7 -> 8.6 (8 CG steps 444 -> 392),
// 512^2 x 1 coil 12.8 -> 10.6 us; from 1.2 million (row, coil pair)s on the same.
static int rows_per_block(const SpmmArgs& a) {
  const int lanes = std::max(1, point_pairs(a) ? a.nCh / 2 : a.nCh);
  const int least = std::max(1, 256 / lanes), most = std::max(1, 1024 / lanes);
  const long long want = std::max<long long>(1, (spmm_rows(a) + 148 * 6 - 1) / (148 * 6));
  return (int)std::min<long long>(most, (want + least - 1) / least * least);
}

int spmm_partial_count(const SpmmArgs& a) {
  const int rpb = rows_per_block(a);
  return (int)((spmm_rows(a) + rpb - 1) / rpb) + a.m->n_long;
}

size_t spmm_scratch_floats(const Csr& m, int nCh) {
  return std::max(3 * (size_t)m.n_seg, 2 * (size_t)m.n_multi_units) * (size_t)nCh;
}

// Odd coil counts: the ordered non-empty product by one coil per thread.
static bool use_single_rec(const SpmmArgs& a) {
  return a.in.layout == Layout::kPointC64 && a.out.layout == Layout::kPointC64 && (a.nCh % 2) == 1 && a.nCh <= 32 &&
         a.nonempty_only && a.contract && !a.partial && !a.normalize && a.unit_count && a.m->ord_rec &&
         a.m->ord_nonempty && a.m->ord_short >= 0;
}

template <Layout IN, Layout OUT, bool ROW_FAST>
static int launch(const SpmmParams& p, const Csr& m, float3* scratch, int grid_short, cudaStream_t s) {
  if (grid_short > 0) {
    spmm_short_kernel<IN, OUT, ROW_FAST><<<grid_short, 256, 0, s>>>(p);
    MLG_LAUNCHED();
  }
  if (p.n_long > 0) {
    spmm_seg_kernel<IN><<<m.n_seg, 256, 0, s>>>(p, m.seg_lo, m.seg_hi, scratch);
    MLG_LAUNCHED();
    spmm_seg_combine_kernel<OUT><<<p.n_long, 256, 0, s>>>(p, m.long_seg0, scratch);
    MLG_LAUNCHED();
  }
  return MLG_OK;
}

static HeavyUnits heavy_of(const Csr& m, float* scratch, unsigned* count) {
  HeavyUnits h;
  h.units = m.heavy_units;
  h.multi = m.heavy_multi;
  h.n = m.n_units;
  h.scratch = scratch;
  h.count = count;
  return h;
}

int spmm(const SpmmArgs& a, cudaStream_t s) {
  const Csr& m = *a.m;
  MLG_CHECK(a.nCh >= 1, "nCh must be >= 1");
  SpmmParams p;
  p.row_ptr = m.row_ptr;
  p.col = m.col;
  p.val = m.val;
  MLG_CHECK(!a.half_values || m.val_h || m.nnz == 0, "FP16 values requested but not built");
  p.val_h = a.half_values ? m.val_h : nullptr;
  p.l_size = m.l_size;
  p.nCh = a.nCh;
  p.rows_per_block = rows_per_block(a);
  p.long_rows = m.long_rows;
  p.n_long = m.n_long;
  p.in = a.in;
  p.out = a.out;
  p.in_row_scale = a.in_row_scale;
  p.out_scale = a.out_scale;
  p.normalize = a.normalize ? 1 : 0;
  p.sqn_w = a.sqn_row_weight;
  p.partial = a.partial;
  p.absmax = a.absmax;
  p.in_h_amax = a.in_half_amax;
  p.in_h_len = a.in_half_len;
  MLG_CHECK(!a.in_half_amax || (use_fwd_kernel(a) && a.nCh % 2 == 0 && m.n_long == 0),
            "FP16 input: forward coil-pair products without long rows only");
  MLG_CHECK(!a.nonempty_only || (m.ord_rows && m.ord_nonempty && use_pair_kernel(a)) || use_single_rec(a),
            "non-empty-row products need the ordered row list and the coil-pair kernel");
  const long long nrows = spmm_rows(a);
  const int grid_all = (int)((nrows + p.rows_per_block - 1) / p.rows_per_block);
  const int grid_short = a.long_only ? 0 : grid_all;
  p.partial_long_offset = grid_all;
  MLG_CHECK(m.n_long == 0 || m.n_seg > 0, "long rows without segment tables");
  MLG_CHECK(m.n_units == 0 || (m.heavy_units && m.heavy_multi), "heavy rows without unit tables");
  DevBuf<float> own;
  float* scratch = a.seg_scratch;
  if ((m.n_long > 0 || m.n_multi_units > 0) && !scratch) {
    MLG_TRY(own.alloc(spmm_scratch_floats(m, a.nCh), s));
    scratch = own.p;
  }
  float3* sc3 = reinterpret_cast<float3*>(scratch);
  using L = Layout;
  const L i = a.in.layout, o = a.out.layout;
  if (use_single_rec(a)) {
    launch_rec<float2>(p, m, heavy_of(m, scratch, a.unit_count), s);
    MLG_LAUNCHED();
    return MLG_OK;
  }
  if (use_fwd_kernel(a) && grid_short > 0) {
    launch_fwd(p, a.contract, grid_short, s);
    MLG_LAUNCHED();
    return launch<L::kPointC64, L::kPointC64, false>(p, m, sc3, 0, s);  // long rows
  }
  if (use_pair_kernel(a)) {
    if (grid_short > 0) {
      // the matrix's processing order when it covers the requested rows
      const bool ordered = m.ord_rows && m.ord_nonempty == a.nonempty_only;
      MLG_CHECK(ordered || !a.nonempty_only, "non-empty-row products need the ordered row list");
      // operator products over a split order: the short rows by the record
      // or pair kernel, the heavy ones as units in its first blocks
      const bool split =
          ordered && a.contract && m.ord_short >= 0 && !a.partial && a.nCh / 2 <= 16 && a.unit_count != nullptr;
      const int n_pair = split ? m.ord_short : (int)nrows;
      HeavyUnits heavy;
      if (split) heavy = heavy_of(m, scratch, a.unit_count);
      const int grid_pair = split ? (n_pair + p.rows_per_block - 1) / p.rows_per_block : grid_short;
      const bool recs = records_forced() >= 0 ? records_forced() == 1 : a.records;
      if (split && m.ord_rec && recs) {
        launch_rec<float4>(p, m, heavy, s);
        MLG_LAUNCHED();
      } else if (grid_pair + heavy.n > 0) {
        const int* rows = ordered ? m.ord_rows : nullptr;
        const uint2* bounds = ordered ? m.ord_bounds : nullptr;
        if (heavy.n)
          spmm_pair_kernel<true><<<heavy.n + grid_pair, 256, 0, s>>>(p, rows, bounds, n_pair, heavy);
        else
          spmm_pair_kernel<false><<<grid_pair, 256, 0, s>>>(p, rows, bounds, n_pair, heavy);
        MLG_LAUNCHED();
      }
      if (split) return MLG_OK;  // the heavy units hold the long rows
    }
    // long rows (segment kernels) with the same element types
    return launch<L::kPointC64, L::kPointC64, false>(p, m, sc3, 0, s);
  }
  if (i == L::kCoilC64 && o == L::kPointC64) return launch<L::kCoilC64, L::kPointC64, false>(p, m, sc3, grid_short, s);
  if (i == L::kPointC64 && o == L::kCoilC64) return launch<L::kPointC64, L::kCoilC64, true>(p, m, sc3, grid_short, s);
  if (i == L::kPointC64 && o == L::kPointC64)
    return launch<L::kPointC64, L::kPointC64, false>(p, m, sc3, grid_short, s);
  if (i == L::kCoilSplit && o == L::kCoilSplit)
    return launch<L::kCoilSplit, L::kCoilSplit, true>(p, m, sc3, grid_short, s);
  if (i == L::kPointSplit && o == L::kPointSplit)
    return launch<L::kPointSplit, L::kPointSplit, false>(p, m, sc3, grid_short, s);
  if (i == L::kCoilReal && o == L::kCoilReal) return launch<L::kCoilReal, L::kCoilReal, true>(p, m, sc3, grid_short, s);
  if (i == L::kPointReal && o == L::kPointReal)
    return launch<L::kPointReal, L::kPointReal, false>(p, m, sc3, grid_short, s);
  return fail(MLG_ERR_UNSUPPORTED, "spmm: layout pair (%d,%d) not instantiated", (int)i, (int)o);
}

// ---- sign-folded copies (fftshift as a (-1)^(x+y+z) modulation) ------------
__device__ __forceinline__ float cell_sign(long long i, int imDim, int Nx, int Ny) {
  long long x = i % Nx;
  long long s = x;
  if (imDim > 1) {
    const long long q = i / Nx;
    s += q % Ny;
    if (imDim > 2) s += q / Ny;
  }
  return (s & 1) ? -1.0f : 1.0f;
}

__global__ void sign_by_col_kernel(const int* __restrict__ col, const float* __restrict__ val, float* out,
                                   long long nnz, int imDim, int Nx, int Ny, float gs) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nnz; k += (long long)gridDim.x * blockDim.x)
    out[k] = val[k] * (gs * cell_sign(col[k], imDim, Nx, Ny));
}

__global__ void sign_by_row_kernel(const uint32_t* __restrict__ row_ptr, const float* __restrict__ val, float* out,
                                   int l_size, int imDim, int Nx, int Ny, float gs) {
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < l_size; r += (long long)gridDim.x * blockDim.x) {
    const float sg = gs * cell_sign(r, imDim, Nx, Ny);
    for (uint32_t k = row_ptr[r]; k < row_ptr[r + 1]; ++k) out[k] = val[k] * sg;
  }
}

void csr_free_sign_copy(Csr& c) {
  cudaFree(c.val);
  cudaFree(c.val_h);
  cudaFree(c.ord_rec);
  c = Csr();
}

__global__ void to_half_kernel(const float* __restrict__ v, long long n, __half* __restrict__ h) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    h[i] = __float2half_rn(v[i]);
}

int csr_make_half(Csr& c, cudaStream_t s) {
  if (c.val_h || c.nnz == 0) return MLG_OK;
  MLG_CUDA(cudaMalloc(&c.val_h, sizeof(__half) * (size_t)c.nnz));
  to_half_kernel<<<(int)std::max<long long>(1, std::min<long long>(148LL * 16, (c.nnz + 255) / 256)), 256, 0, s>>>(
      c.val, c.nnz, c.val_h);
  MLG_LAUNCHED();
  return MLG_OK;
}

int csr_sign_copy(const Csr& src, bool by_row, int imDim, const int* N, float global_sign, Csr& dst,
                  cudaStream_t s) {
  dst = src;  // shares row_ptr / col / long_rows with src (not owned)
  dst.val = nullptr;
  dst.val_h = nullptr;
  dst.ord_rec = nullptr;
  MLG_CUDA(cudaMalloc(&dst.val, sizeof(float) * (size_t)std::max<long long>(1, src.nnz)));
  const int Nx = N[0], Ny = imDim > 1 ? N[1] : 1;
  if (by_row) {
    sign_by_row_kernel<<<std::max(1, std::min(65535, (src.l_size + 255) / 256)), 256, 0, s>>>(
        src.row_ptr, src.val, dst.val, src.l_size, imDim, Nx, Ny, global_sign);
  } else {
    sign_by_col_kernel<<<(int)std::max<long long>(1, std::min<long long>(65535, (src.nnz + 255) / 256)), 256, 0, s>>>(
        src.col, src.val, dst.val, src.nnz, imDim, Nx, Ny, global_sign);
  }
  MLG_LAUNCHED();
  return MLG_OK;
}

// ---- host-buffer SpMV entry points ------------------------------------------
namespace {

struct HostCall {
  cudaStream_t s = nullptr;
  Csr m;
  ~HostCall() { csr_free(m); }
};

int vec_call(int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
             const int* l_jump, int l_nJump, const float* vR, const float* vI, int nVec, float* wR,
             float* wI, Layout layout, int nBlock = 0, const int* block_length = nullptr,
             const int* l_block_start = nullptr, const long long* m_block_start = nullptr) {
  MLG_TRY(ensure_device());
  MLG_CHECK(nVec >= 1, "n_vec must be >= 1");
  const bool cplx = layout != Layout::kCoilReal && layout != Layout::kPointReal;
  MLG_CHECK(vR && wR && (!cplx || (vI && wI)), "NULL vector buffer");
  HostCall hc;
  MLG_TRY(csr_from_jump(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, hc.m, hc.s, nBlock, block_length,
                        l_block_start, m_block_start));
  const size_t nin = (size_t)r_size * nVec, nout = (size_t)l_size * nVec;
  DevBuf<float> din, dout;
  MLG_TRY(din.alloc(nin * (cplx ? 2 : 1), hc.s));
  MLG_TRY(dout.alloc(nout * (cplx ? 2 : 1), hc.s));
  MLG_CUDA(cudaMemcpyAsync(din.p, vR, nin * sizeof(float), cudaMemcpyHostToDevice, hc.s));
  if (cplx) MLG_CUDA(cudaMemcpyAsync(din.p + nin, vI, nin * sizeof(float), cudaMemcpyHostToDevice, hc.s));
  SpmmArgs a;
  a.m = &hc.m;
  a.nCh = nVec;
  a.in.layout = a.out.layout = layout;
  a.in.a = din.p;
  a.in.b = cplx ? din.p + nin : nullptr;
  a.in.rows = r_size;
  a.out.a = dout.p;
  a.out.b = cplx ? dout.p + nout : nullptr;
  a.out.rows = l_size;
  MLG_TRY(spmm(a, hc.s));
  MLG_CUDA(cudaMemcpyAsync(wR, dout.p, nout * sizeof(float), cudaMemcpyDeviceToHost, hc.s));
  if (cplx) MLG_CUDA(cudaMemcpyAsync(wI, dout.p + nout, nout * sizeof(float), cudaMemcpyDeviceToHost, hc.s));
  MLG_CUDA(cudaStreamSynchronize(hc.s));
  return MLG_OK;
}

}  // namespace
}  // namespace mlg

using namespace mlg;

extern "C" {

int mlg_sparsemat_vec_cC(int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
                         const int* l_jump, int l_nJump, const float* vReal, const float* vImag, int nVec,
                         float* wReal, float* wImag) {
  return vec_call(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, vReal, vImag, nVec, wReal, wImag,
                  Layout::kCoilSplit);
}

int mlg_sparsemat_vec_cR(int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
                         const int* l_jump, int l_nJump, const float* vReal, const float* vImag, int nVec,
                         float* wReal, float* wImag) {
  return vec_call(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, vReal, vImag, nVec, wReal, wImag,
                  Layout::kPointSplit);
}

int mlg_sparsemat_vec_rC(int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
                         const int* l_jump, int l_nJump, const float* v, int nVec, float* w) {
  return vec_call(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, v, nullptr, nVec, w, nullptr,
                  Layout::kCoilReal);
}

int mlg_sparsemat_r_nJump2index(int l_size, const int* r_nJump, long long out_length, int* out) {
  // bmSparseMat_r_nJump2index_mex.cpp:70-80.  A setup-time helper of the
  // matrix builder: runs on the host (there is no device work to amortise).
  MLG_CHECK(l_size >= 0 && (l_size == 0 || r_nJump), "r_nJump missing");
  MLG_CHECK(out || out_length == 0, "NULL output");
  long long n = 0;
  for (int i = 0; i < l_size; ++i) {
    MLG_CHECK(r_nJump[i] >= 0, "negative r_nJump");
    MLG_CHECK(n + r_nJump[i] <= out_length, "out_length %lld smaller than sum(r_nJump)", out_length);
    for (int j = 0; j < r_nJump[i]; ++j) out[n++] = i;
  }
  MLG_CHECK(n == out_length, "out_length %lld differs from sum(r_nJump)=%lld", out_length, n);
  return MLG_OK;
}

int mlg_matrix_create_blocks(int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
                             const int* l_jump, int l_nJump, int nBlock, const int* block_length,
                             const int* l_block_start, const long long* m_block_start, mlg_matrix_t* out) {
  MLG_CHECK(out, "NULL output handle");
  *out = nullptr;
  MLG_CHECK(nBlock >= 0, "nBlock must be >= 0");
  MLG_TRY(ensure_device());
  mlg_matrix_s* h = new mlg_matrix_s();
  cudaGetDevice(&h->device);
  int st = csr_from_jump(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, h->csr, nullptr, nBlock,
                         block_length, l_block_start, m_block_start);
  if (st != MLG_OK) {
    delete h;
    return st;
  }
  *out = h;
  return MLG_OK;
}

int mlg_matrix_create(int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
                      const int* l_jump, int l_nJump, mlg_matrix_t* out) {
  return mlg_matrix_create_blocks(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, 0, nullptr, nullptr,
                                  nullptr, out);
}

int mlg_sparsemat_vec(int layout, int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
                      const int* l_jump, int l_nJump, int nBlock, const int* block_length, const int* l_block_start,
                      const long long* m_block_start, const float* vR, const float* vI, int nVec, float* wR,
                      float* wI) {
  Layout L;
  switch (layout) {
    case MLG_LAYOUT_CC: L = Layout::kCoilSplit; break;
    case MLG_LAYOUT_CR: L = Layout::kPointSplit; break;
    case MLG_LAYOUT_RC: L = Layout::kCoilReal; break;
    case MLG_LAYOUT_RR: L = Layout::kPointReal; break;
    default: return fail(MLG_ERR_ARG, "unknown layout %d", layout);
  }
  MLG_CHECK(nBlock >= 0, "nBlock must be >= 0");
  return vec_call(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, vR, vI, nVec, wR, wI, L, nBlock,
                  block_length, l_block_start, m_block_start);
}

int mlg_sparsemat_vec_rR(int r_size, const int* r_jump, const int* r_nJump, const float* m_val, int l_size,
                         const int* l_jump, int l_nJump, const float* v, int nVec, float* w) {
  return vec_call(r_size, r_jump, r_nJump, m_val, l_size, l_jump, l_nJump, v, nullptr, nVec, w, nullptr,
                  Layout::kPointReal);
}

int mlg_matrix_destroy(mlg_matrix_t m) {
  if (!m) return MLG_OK;
  cudaSetDevice(m->device);
  csr_free(m->csr);
  delete m;
  return MLG_OK;
}

int mlg_matrix_info(mlg_matrix_t m, long long* nnz, int* r_size, int* l_size) {
  MLG_CHECK(m, "NULL matrix");
  if (nnz) *nnz = m->csr.nnz;
  if (r_size) *r_size = m->csr.r_size;
  if (l_size) *l_size = m->csr.l_size;
  return MLG_OK;
}

int mlg_matrix_row_stats(mlg_matrix_t m, int* nonempty_rows, int* long_rows) {
  MLG_CHECK(m, "NULL matrix");
  if (nonempty_rows) *nonempty_rows = m->csr.n_nonempty;
  if (long_rows) *long_rows = m->csr.n_long;
  return MLG_OK;
}

int mlg_matrix_download(mlg_matrix_t m, int* r_jump, int* r_nJump, float* m_val, int* l_jump, int* l_nJump_out) {
  MLG_CHECK(m && r_jump && r_nJump && m_val, "NULL argument");
  const Csr& c = m->csr;
  MLG_CUDA(cudaSetDevice(m->device));
  std::vector<uint32_t> rp((size_t)c.l_size + 1);
  std::vector<int> col((size_t)c.nnz);
  MLG_CUDA(cudaMemcpy(rp.data(), c.row_ptr, sizeof(uint32_t) * rp.size(), cudaMemcpyDeviceToHost));
  if (c.nnz) {
    MLG_CUDA(cudaMemcpy(col.data(), c.col, sizeof(int) * (size_t)c.nnz, cudaMemcpyDeviceToHost));
    MLG_CUDA(cudaMemcpy(m_val, c.val, sizeof(float) * (size_t)c.nnz, cudaMemcpyDeviceToHost));
  }
  long long prevc = 0;
  for (long long e = 0; e < c.nnz; ++e) {
    r_jump[e] = (int)(col[(size_t)e] - prevc);
    prevc = col[(size_t)e];
  }
  // l_jump != NULL: squeezed form (non-empty rows only, bmSparseMat.m:62-94)
  int n = 0;
  long long prevr = 0;
  for (int r = 0; r < c.l_size; ++r) {
    const int len = (int)(rp[(size_t)r + 1] - rp[r]);
    if (l_jump) {
      if (len == 0) continue;
      l_jump[n] = (int)(r - prevr);
      prevr = r;
    }
    r_nJump[n++] = len;
  }
  if (l_nJump_out) *l_nJump_out = n;
  return MLG_OK;
}

int mlg_matrix_spmm_dev(mlg_matrix_t m, const void* v, int nVec, void* w, void* stream) {
  MLG_CHECK(m && v && w && nVec >= 1, "invalid argument");
  MLG_CUDA(cudaSetDevice(m->device));
  PairOperand vi, wo;
  MLG_TRY(vi.in(v, (size_t)m->csr.r_size * nVec, nVec % 2 == 0, (cudaStream_t)stream));
  MLG_TRY(wo.out(w, (size_t)m->csr.l_size * nVec, nVec % 2 == 0, (cudaStream_t)stream));
  SpmmArgs a;
  a.m = &m->csr;
  a.nCh = nVec;
  a.in.layout = a.out.layout = Layout::kPointC64;
  a.in.a = vi.p;
  a.in.rows = m->csr.r_size;
  a.out.a = wo.p;
  a.out.rows = m->csr.l_size;
  MLG_TRY(spmm(a, (cudaStream_t)stream));
  return wo.finish();
}

}  // extern "C"

// hmf_dataterm.cu -- the data-term producers that precede a solve:
//
//  hmf_data_term       vtkImageDataTerm (Common/vtkRobartsCommon/vtkImageDataTerm.cxx:62-470):
//                      per voxel a constant, logistic, Gaussian or spike cost
//                      of one or two images, as a probability or an entropy,
//                      optionally normalised by the first image's range.
//  hmf_log_likelihood  vtkImageLogLikelihood (vtkImageLogLikelihood.cxx:140-250):
//                      a histogram of the image over the voxels that enough
//                      label maps mark with one label, and per voxel the
//                      negative log of its bin's frequency.
//
// Both evaluate the reference's expressions in its precision (double for the
// data term, float for the histogram) and order of operations (the library is
// built without contraction, as the reference's x86 build computes), with
// CUDA's double exp / log where the reference calls the C library's.  The data
// term is formed in float-float on the FP32 pipes first (hmf_ff.cuh) and in
// double only where that does not settle how the double result rounds to float.
// Images
// are float32 (the reference templates over VTK scalar types and writes the
// input's type; a float cost is what the solver takes).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <initializer_list>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/hmf.h"
#include "hmf_ctx.hpp"
#include "hmf_ff.cuh"

namespace hmfi {

// Scratch of one call, drawn from a memory pool of the library's own (one
// per device, keeping up to 256 MB between calls) and returned to it in
// stream order: no cudaMalloc / cudaFree per call, whose implicit device
// synchronisation would also stall the caller's other streams.
cudaMemPool_t scratch_pool() {
  static std::mutex mu;
  static std::map<int, cudaMemPool_t> pools;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  auto it = pools.find(dev);
  if (it != pools.end()) return it->second;
  cudaMemPoolProps props;
  std::memset(&props, 0, sizeof(props));
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    pool = nullptr;  // plain cudaMalloc then
  } else {
    unsigned long long keep = 256ull << 20;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  pools[dev] = pool;
  return pool;
}

}  // namespace hmfi

using namespace hmfi;
using namespace hmf;

namespace {

constexpr int kThreads = 256;

int grid_for(long long n) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long blocks = (n + kThreads - 1) / kThreads;
  return (int)std::max<long long>(1, std::min<long long>(blocks, (long long)sms * 16));
}

// Order-preserving map of a float to an unsigned int (for atomic min / max).
__device__ __forceinline__ unsigned int float_key(float f) {
  const unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float key_float(unsigned int k) {
  const unsigned int u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  std::memcpy(&f, &u, sizeof(f));
  return f;
#endif
}

// Blocks of the reductions that end in atomics on a few addresses: one set of
// atomics per block, and few blocks -- with one set per warp of 2432 blocks the
// atomics alone took 30 us of the range and 60 us of the seeds' scan.
constexpr int kReduceBlocks = 608;

// Minimum or maximum over the block, in thread 0 (every thread calls it).
template <bool MAX>
__device__ __forceinline__ unsigned block_extreme(unsigned v, unsigned* warps /* [kThreads / 32] */) {
  v = MAX ? __reduce_max_sync(0xffffffffu, v) : __reduce_min_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kThreads / 32; ++w) v = MAX ? max(v, warps[w]) : min(v, warps[w]);
  return v;
}

// mm[0] = complement of the minimum's key, mm[1] = key of the maximum, both from
// zero (NaN skipped, as vtkDataArray's range ignores it).
__global__ void range_kernel(const float* __restrict__ in, long long n, unsigned int* mm) {
  unsigned int lo = 0xffffffffu, hi = 0u;
  auto take = [&](float v) {
    if (v != v) return;
    const unsigned int k = float_key(v);
    lo = min(lo, k);
    hi = max(hi, k);
  };
  const long long stride = (long long)gridDim.x * blockDim.x, t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nq = (reinterpret_cast<uintptr_t>(in) & 15) == 0 ? n / 4 : 0;
#pragma unroll 4
  for (long long q = t; q < nq; q += stride) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(in) + q);
    take(v.x), take(v.y), take(v.z), take(v.w);
  }
  for (long long i = 4 * nq + t; i < n; i += stride) take(in[i]);
  __shared__ unsigned warps[kThreads / 32];
  lo = block_extreme<false>(lo, warps);
  hi = block_extreme<true>(hi, warps);
  if (threadIdx.x == 0) {
    atomicMax(&mm[0], ~lo);
    atomicMax(&mm[1], hi);
  }
}

struct Split3 {  // h + m + l == a double, exactly (no part under- or overflows)
  float h, m, l;
};

__host__ __device__ inline Split3 split3(double d) {
  Split3 s;
  s.h = (float)d;
  s.m = (float)(d - (double)s.h);
  s.l = (float)((d - (double)s.h) - (double)s.m);
  return s;
}
__host__ __device__ inline FFloat split2(double d) {
  FFloat s;
  s.h = (float)d;
  s.l = (float)(d - (double)s.h);
  return s;
}
// Zero, or a magnitude whose parts and products stay far from the ends of the
// float range.
__host__ __device__ inline bool ff_safe(double d) {
  const double a = d < 0.0 ? -d : d;
  return a == 0.0 || (a >= 0x1p-40 && a <= 0x1p40);
}

// Tables of the float-float exponential and logarithm, formed by the host in
// double: ln 2 in three parts of which the first two times a small integer are
// exact, exp(j / 32) for |j| <= kExpHalf, and for 64 intervals of [1, 2) a
// float near the reciprocal of the centre and minus its logarithm.
constexpr int kExpHalf = 12;
constexpr int kLogCells = 64;
struct TermTables {  // the logistic in float-float
  static constexpr bool kFast = true, kLogistic = true;
  float ln2[3];
  FFloat ln2_ff;
  FFloat exp_tab[2 * kExpHalf + 1];
  float log_inv[kLogCells];
  FFloat log_tab[kLogCells];
};

struct NoTables {  // the Gaussian's entropy in float-float
  static constexpr bool kFast = true, kLogistic = false;
};
struct InDouble {  // double throughout
  static constexpr bool kFast = false, kLogistic = false;
};

TermTables make_term_tables() {
  TermTables T;
  const double l = std::log(2.0);
  T.ln2[0] = (float)(std::floor(l * 65536.0) / 65536.0);
  T.ln2[1] = (float)(std::floor((l - T.ln2[0]) * 4294967296.0) / 4294967296.0);
  T.ln2[2] = (float)(l - (double)T.ln2[0] - (double)T.ln2[1]);
  T.ln2_ff = split2(l);
  for (int j = -kExpHalf; j <= kExpHalf; ++j) T.exp_tab[j + kExpHalf] = split2(std::exp(j / 32.0));
  for (int j = 0; j < kLogCells; ++j) {
    T.log_inv[j] = (float)(1.0 / (1.0 + (j + 0.5) / kLogCells));
    T.log_tab[j] = split2(-std::log((double)T.log_inv[j]));
  }
  return T;
}

// exp(z), |z.h| <= 33: relative error below 2^-41 + |z| 2^-46.  Reduction by n
// ln 2 and a table step of 1/32, then the series to the sixth power (the first
// two terms in float-float, the rest, below 2^-20, in float).
__device__ __forceinline__ FFloat ff_exp(FFloat z, const TermTables& T) {
  const float n = rintf(z.h * 1.44269504f);
  FFloat r = ff_sum(ff_two_sum(z.h, -(n * T.ln2[0])), ff_two_sum(z.l, -(n * T.ln2[1])));
  r = ff_sum(r, -(n * T.ln2[2]));
  const int j = max(-kExpHalf, min(kExpHalf, __float2int_rn(r.h * 32.0f)));
  r = ff_sum(r, -(float)j * 0.03125f);
  const FFloat r2 = ff_mul(r, r);
  const float x = r.h;
  const float p = (r2.h * x) * __fmaf_rn(x, __fmaf_rn(x, __fmaf_rn(x, 1.0f / 720.0f, 1.0f / 120.0f), 1.0f / 24.0f), 1.0f / 6.0f);
  FFloat u = ff_sum(r, FFloat{0.5f * r2.h, 0.5f * r2.l});
  u = ff_sum(ff_sum(u, p), 1.0f);
  u = ff_mul(u, T.exp_tab[j + kExpHalf]);
  const float scale = __int_as_float((127 + (int)n) << 23);
  return {u.h * scale, u.l * scale};
}

// log(1 + f), |f.h| <= 2^-6: the first two terms of the series in float-float.
__device__ __forceinline__ FFloat ff_log1p(FFloat f, FFloat base) {
  const FFloat f2 = ff_mul(f, f);
  const float x = f.h;
  const float p = (f2.h * x) * __fmaf_rn(x, __fmaf_rn(x, __fmaf_rn(x, __fmaf_rn(x, 1.0f / 7.0f, -1.0f / 6.0f), 0.2f), -0.25f), 1.0f / 3.0f);
  return ff_sum(ff_sum(ff_sum(base, f), FFloat{-0.5f * f2.h, -0.5f * f2.l}), p);
}

// log(a) of a float-float 1 + 2^-8 <= a < 2^100.
__device__ __forceinline__ FFloat ff_log(FFloat a, const TermTables& T) {
  const unsigned bits = __float_as_uint(a.h);
  const int k = (int)(bits >> 23) - 127;
  const float down = __int_as_float((127 - k) << 23);
  const int j = (bits >> 17) & (kLogCells - 1);
  const FFloat f = ff_sum(ff_mul(FFloat{a.h * down, a.l * down}, T.log_inv[j]), -1.0f);
  return ff_log1p(f, ff_sum(ff_mul(T.ln2_ff, (float)k), T.log_tab[j]));
}

struct TermParams {
  int op, entropy, two;
  double k1, c1, k2, c2;
  Split3 c1s, c2s;         // C1, C2
  FFloat k1s, k2s;         // Gaussian: 1/K1, 1/K2; logistic: K1, K2
  int normalize;           // 0 none, 1 by off and mul, 2 Gaussian entropy: by the range at `range`
  const unsigned int* range;
  double off, mul;
};

struct TermNorm {
  double off, mul;
  Split3 offs;
  FFloat muls;
  int fast;
};

// vtkImageDataTermExecute1 (:62-249) and vtkImageDataTermExecute2 (:255-390) in
// the reference's double arithmetic.
__device__ __noinline__ float logistic_double(const TermParams& P, float f1, float f2) {
  const double x1 = (double)f1, x2 = (double)f2;
  const double a = 1.0 + exp(-(P.k1 * (x1 - P.c1)));
  if (!P.two) return (float)(P.entropy ? log(a) : 1.0 / a);
  const double b = 1.0 + exp(-(P.k2 * (x2 - P.c2)));
  return (float)(P.entropy ? log(a * b) : 1.0 / (a * b));
}
__device__ __forceinline__ float gaussian_in_double(const TermParams& P, float f1, float f2) {
  const double x1 = (double)f1, x2 = (double)f2;
  const double q1 = (x1 - P.c1) / P.k1;
  if (!P.two) return (float)(P.entropy ? 0.5 * q1 * q1 : exp(-0.5 * q1 * q1));
  const double q2 = (x2 - P.c2) / P.k2;
  return (float)(P.entropy ? 0.5 * q1 * q1 + 0.5 * q2 * q2 : exp(-0.5 * q1 * q1 - 0.5 * (q2 * q2)));
}
__device__ __forceinline__ float norm_in_double(float o, double off, double mul) {
  return (float)(((double)o + off) * mul);
}
// The same beside the float-float path, out of line.
__device__ __noinline__ float gaussian_double(const TermParams& P, float f1, float f2) {
  return gaussian_in_double(P, f1, f2);
}
__device__ __noinline__ float norm_double(float o, double off, double mul) { return norm_in_double(o, off, mul); }

__device__ __forceinline__ bool in_range(float a, float lo, float hi) { return a >= lo && a <= hi; }

// x - c for a float x and a double c; `ok` is cleared outside the safe range
// (an exact zero is inside).
__device__ __forceinline__ FFloat ff_minus(float x, const Split3& c, bool& ok) {
  const FFloat t = ff_sum(ff_two_sum(x, -c.h), FFloat{-c.m, -c.l});
  ok = ok && ((t.h == 0.0f && t.l == 0.0f) || in_range(fabsf(t.h), 0x1p-40f, 0x1p40f));
  return t;
}

// The same result from float-float arithmetic; false where its error bound
// leaves the rounding of the double result open (or an operand is out of
// range).  Bounds, relative: the Gaussian's entropy 2^-43.2 (a difference, a
// product by the reciprocal, a square) and the double result's own 2^-50,
// tested with 2^-41; the logistic's 2^-38.6 with 2^-37: its exponential and
// logarithm, and the double result's 2^-53 / e^z from rounding 1 + e^z, which
// for an entropy keeps e^z above 2^-10.
//
// With VOTE a warp takes it together (`valid`: the lane has a voxel): where one
// of its voxels lies outside the forms' range all of them go to double at once,
// instead of after the others.  That counts in images too small to hide it: a
// logistic of 2^16 voxels of which most lie outside takes 12.3 us without, 10.3
// with it; in large images the vote costs up to a tenth.
template <bool VOTE, class Tables>
__device__ __forceinline__ bool term_fast(const TermParams& P, const Tables& T, float x1, float x2, bool valid,
                                          float& out) {
  bool ok = true;
  const FFloat t1 = ff_mul(ff_minus(x1, P.c1s, ok), P.k1s);
  FFloat t2{0.0f, 0.0f};
  if (P.two) t2 = ff_mul(ff_minus(x2, P.c2s, ok), P.k2s);
  if constexpr (Tables::kLogistic) {
    ok = ok && fabsf(t1.h) <= 32.0f && fabsf(t2.h) <= 32.0f;
    if (P.entropy) ok = ok && (P.two ? fminf(t1.h, t2.h) <= 4.8f : t1.h <= 6.9f);  // (the limits below)
  } else {
    ok = ok && (t1.h == 0.0f || in_range(fabsf(t1.h), 0x1p-30f, 0x1p30f)) &&
         (t2.h == 0.0f || in_range(fabsf(t2.h), 0x1p-30f, 0x1p30f));
  }
  if (VOTE && !__all_sync(0xffffffffu, ok || !valid)) return !valid;
  if (!valid) return true;
  if (!VOTE && !ok) return false;
  FFloat v;
  if constexpr (Tables::kLogistic) {
    const FFloat e1 = ff_exp(FFloat{-t1.h, -t1.l}, T);
    FFloat a = ff_sum(e1, 1.0f);
    if (P.two) a = ff_mul(a, ff_sum(ff_exp(FFloat{-t2.h, -t2.l}, T), 1.0f));
    if (P.entropy) {
      if (!P.two && e1.h < 0x1p-7f) {
        if (!(e1.h >= 0x1p-10f)) return false;
        v = ff_log1p(e1, FFloat{0.0f, 0.0f});
      } else {
        if (!(a.h >= 1.0f + 0x1p-7f)) return false;
        v = ff_log(a, T);
      }
    } else {
      const float r = 1.0f / a.h;
      const FFloat e = ff_sum(ff_mul(a, -r), 1.0f);  // 1 - a r
      v = ff_sum(ff_mul(e, r), r);
    }
    return ff_rounds(v, 0x1p-37f, out);
  } else {  // the Gaussian's entropy
    v = ff_mul(t1, t1);
    if (P.two) v = ff_sum(v, ff_mul(t2, t2));
    if (v.h == 0.0f) {
      out = 0.0f;
      return true;
    }
    return ff_rounds(FFloat{0.5f * v.h, 0.5f * v.l}, 0x1p-41f, out);
  }
}

template <bool VOTE, class Tables>
__device__ __forceinline__ float term_value(const TermParams& P, const Tables& T, const TermNorm& N, float x1,
                                            float x2, bool valid) {
  float o = 0.0f;
  if constexpr (!Tables::kFast) {
    o = P.op == HMF_DATA_TERM_LOGISTIC ? logistic_double(P, x1, x2) : gaussian_in_double(P, x1, x2);
    return P.normalize ? norm_in_double(o, N.off, N.mul) : o;
  } else {
    if (!term_fast<VOTE>(P, T, x1, x2, valid, o)) o = Tables::kLogistic ? logistic_double(P, x1, x2) : gaussian_double(P, x1, x2);
    if (!P.normalize) return o;
    if (N.fast) {  // (o + off) * mul
      const FFloat a = ff_sum(ff_two_sum(o, N.offs.h), FFloat{N.offs.m, N.offs.l});
      if (a.h == 0.0f && a.l == 0.0f && N.mul > 0.0) return 0.0f;
      const FFloat v = ff_mul(a, N.muls);
      float r;
      if (in_range(fabsf(a.h), 0x1p-40f, 0x1p40f) && ff_rounds(v, 0x1p-43f, r)) return r;
    }
    return norm_double(o, N.off, N.mul);
  }
}

// Normalisation of a Gaussian entropy by the image's range [R0, R1]
// (vtkImageDataTermExecute1, :187-249), in the host code's operations.
__device__ __forceinline__ void gaussian_range_norm(const TermParams& P, double R0, double R1, double& off,
                                                    double& mul) {
  const double vmax = 0.5 * ((R1 - P.c1) / P.k1) * ((R1 - P.c1) / P.k1);
  const double vmin = 0.5 * ((R0 - P.c1) / P.k1) * ((R0 - P.c1) / P.k1);
  const double mx = (vmax >= vmin) ? vmax : vmin;
  double mn = (vmax < vmin) ? vmax : vmin;
  if (P.c1 > R0 && P.c1 < R1) mn = 0.0f;
  off = -mn;
  mul = 1.0 / (mx - mn);
}

// Smallest images of the float-float forms, and of four voxels per thread in
// them (Gaussian, logistic).  Below the first, launches cost what they cost:
// us per call in double, float-float with a voxel and with four per thread,
// Gaussian entropy of 4,000 voxels 6.2, 6.0, 6.1, of 131,072 7.4, 6.1, 6.2, of
// 524,288 16.5, 7.3, 6.2; logistic entropy of 4,000 7.4, 6.0, 8.2, of 32,768 8.1,
// 6.7, 8.3, of 262,144 28.7, 10.3, 10.3, of 524,288 51.4, 14.4, 12.4; one whose
// voxels lie outside the float-float range of 16,384 7.7, 8.2, 20.6, of 262,144
// 28.7, 28.8, 32.9.
constexpr long long kTermFast[2] = {1 << 14, 1 << 15};
constexpr long long kTermQuads[2] = {1 << 18, 1 << 19};

// One voxel's result depends on it alone: bound by the arithmetic.  In double
// throughout it kept the FP64 pipe 86 % busy (256 x 256 x 192, Gaussian entropy
// normalised: 574 us); in float-float 79 us a call, of which 38 are the
// normalisation: the range's pass and every block's constants in double.  A
// logistic entropy takes 157 us of FP32 arithmetic, a Gaussian probability, in
// double still, 750.
//
// Double throughout (InDouble) is for what has no float-float form, the
// Gaussian's probability among it, and for small images.  It takes a voxel per
// thread: four in one thread wait for one another's FP64.
template <class Tables>
__global__ void __launch_bounds__(kThreads) data_term_kernel(const __grid_constant__ TermParams P,
                                                             const __grid_constant__ Tables tables,
                                                             const float* __restrict__ in1,
                                                             const float* __restrict__ in2, long long n, int quads,
                                                             float* __restrict__ out) {
  __shared__ Tables T;
  __shared__ TermNorm N;
  if constexpr (Tables::kLogistic)  // read with an index that differs from lane to lane
    for (int i = threadIdx.x; i < (int)(sizeof(Tables) / 4); i += blockDim.x)
      reinterpret_cast<float*>(&T)[i] = reinterpret_cast<const float*>(&tables)[i];
  if (threadIdx.x == 0 && P.normalize) {
    N.off = P.off;
    N.mul = P.mul;
    if (P.normalize == 2)
      gaussian_range_norm(P, (double)key_float(~P.range[0]), (double)key_float(P.range[1]), N.off, N.mul);
    if (Tables::kFast) {
      N.fast = ff_safe(N.off) && ff_safe(N.mul) && N.mul != 0.0;
      N.offs = split3(N.off);
      N.muls = split2(N.mul);
    }
  }
  if (Tables::kLogistic || P.normalize) __syncthreads();
  const long long stride = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x;
  const bool two = P.two != 0;
  const long long nq = quads ? n / 4 : 0;
  if constexpr (Tables::kFast) {
    for (long long q = first + threadIdx.x; q < nq; q += stride) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(in1) + q);
      const float4 b = two ? __ldg(reinterpret_cast<const float4*>(in2) + q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      float x1[4] = {a.x, a.y, a.z, a.w}, x2[4] = {b.x, b.y, b.z, b.w}, o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = term_value<false>(P, T, N, x1[j], x2[j], true);
      reinterpret_cast<float4*>(out)[q] = make_float4(o[0], o[1], o[2], o[3]);
    }
  }
  if constexpr (Tables::kLogistic) {  // a block's threads run the same number of turns: their warps vote
    for (long long i0 = 4 * nq + first; i0 < n; i0 += stride) {
      const long long i = i0 + threadIdx.x;
      const bool valid = i < n;
      const float o = term_value<true>(P, T, N, valid ? in1[i] : 0.0f, valid && two ? in2[i] : 0.0f, valid);
      if (valid) out[i] = o;
    }
  } else {
    for (long long i = 4 * nq + first + threadIdx.x; i < n; i += stride)
      out[i] = term_value<false>(P, T, N, in1[i], two ? in2[i] : 0.0f, true);
  }
}

// The constant and the spike operation: one of two values, formed by the host
// (without `in`: the first).
__global__ void __launch_bounds__(kThreads) term_choice_kernel(const float* __restrict__ in, float spike, float hit,
                                                               float miss, long long n, float* __restrict__ out) {
  const long long stride = (long long)gridDim.x * blockDim.x, t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nq = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 ? n / 4 : 0;
  for (long long q = t; q < nq; q += stride) {
    float4 o = make_float4(hit, hit, hit, hit);
    if (in) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(in) + q);
      o = make_float4(a.x == spike ? hit : miss, a.y == spike ? hit : miss, a.z == spike ? hit : miss,
                      a.w == spike ? hit : miss);
    }
    reinterpret_cast<float4*>(out)[q] = o;
  }
  for (long long i = 4 * nq + t; i < n; i += stride) out[i] = !in || in[i] == spike ? hit : miss;
}

struct LLParams {
  int comps, n_maps, actual_maps, label_id;
  int min_agree;  // smallest agreeing count k with (double)k >= agreement * (double)actual_maps
  float resolution;
  float inv_res;  // 1 / resolution where it divides exactly as this multiplies (a power of two), else 0
  int quads;      // image, maps and output allow 16-byte accesses
};

struct LLMaps {
  const int* map[HMF_MAX_LABEL_MAPS];
};

// A seed: enough label maps mark voxel i with the label.  The reference's
// test, (double)agree >= agreement * (double)actual_maps, is monotone in the
// integer count, so the host turns it into the threshold min_agree.
__device__ __forceinline__ bool ll_sample(const LLParams& P, const LLMaps& M, long long i) {
  int agree = 0;
  for (int k = 0; k < P.n_maps; ++k)
    if (M.map[k] && M.map[k][i] == P.label_id) ++agree;
  return agree >= P.min_agree;
}

// The seed test of four neighbouring voxels, a bit each.
__device__ __forceinline__ unsigned ll_sample4(const LLParams& P, const LLMaps& M, long long q) {
  int a0 = 0, a1 = 0, a2 = 0, a3 = 0;
#pragma unroll 4
  for (int k = 0; k < P.n_maps; ++k) {
    if (!M.map[k]) continue;
    const int4 m = __ldg(reinterpret_cast<const int4*>(M.map[k]) + q);
    a0 += m.x == P.label_id;
    a1 += m.y == P.label_id;
    a2 += m.z == P.label_id;
    a3 += m.w == P.label_id;
  }
  return (a0 >= P.min_agree ? 1u : 0u) | (a1 >= P.min_agree ? 2u : 0u) | (a2 >= P.min_agree ? 4u : 0u) |
         (a3 >= P.min_agree ? 8u : 0u);
}

// Seeds' count and range: sums: [0] samples; keys: [0..1] min, [2..3] max per
// component.  `seeds` keeps the seed bits, four voxels (a quad) to a byte and
// one byte per voxel beyond the last whole quad, so that the histogram's pass
// reads them instead of every label map again: the two passes over 4 maps of
// 256 x 256 x 192 voxels took 109 + 42 us reading one voxel at a time and
// reducing with one set of atomics per warp, and take 39 + 18 us.
__global__ void ll_scan_kernel(const LLParams P, const LLMaps M, const float* __restrict__ img, long long n,
                               unsigned long long* count, unsigned int* keys, unsigned char* __restrict__ seeds) {
  unsigned long long c = 0;
  unsigned int lo0 = 0xffffffffu, lo1 = 0xffffffffu, hi0 = 0u, hi1 = 0u;
  auto take = [&](float x0, float x1) {
    ++c;
    const unsigned int k0 = float_key(x0);
    lo0 = min(lo0, k0);
    hi0 = max(hi0, k0);
    if (P.comps == 2) {
      const unsigned int k1 = float_key(x1);
      lo1 = min(lo1, k1);
      hi1 = max(hi1, k1);
    }
  };
  const long long stride = (long long)gridDim.x * blockDim.x, t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nq = P.quads ? n / 4 : 0;
  for (long long q = t; q < nq; q += stride) {
    const unsigned bits = ll_sample4(P, M, q);
    seeds[q] = (unsigned char)bits;
    if (!bits) continue;
    const float4* src = reinterpret_cast<const float4*>(img) + q * P.comps;
    float v[8];
    const float4 a = __ldg(src);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    if (P.comps == 2) {
      const float4 b = __ldg(src + 1);
      v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (bits >> j & 1u) take(v[2 * j], v[2 * j + 1]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (bits >> j & 1u) take(v[j], 0.0f);
    }
  }
  for (long long i = 4 * nq + t; i < n; i += stride) {
    const bool on = ll_sample(P, M, i);
    seeds[nq + (i - 4 * nq)] = on;
    if (on) take(img[P.comps * i], P.comps == 2 ? img[2 * i + 1] : 0.0f);
  }
  __shared__ unsigned warps[kThreads / 32];
  __shared__ unsigned long long counts[kThreads / 32];
  for (int s = 16; s > 0; s >>= 1) c += __shfl_down_sync(0xffffffffu, c, s);
  if ((threadIdx.x & 31) == 0) counts[threadIdx.x >> 5] = c;
  lo0 = block_extreme<false>(lo0, warps);
  hi0 = block_extreme<true>(hi0, warps);
  if (P.comps == 2) {
    lo1 = block_extreme<false>(lo1, warps);
    hi1 = block_extreme<true>(hi1, warps);
  }
  if (threadIdx.x == 0) {  // (block_extreme's barriers order the counts)
    for (int w = 1; w < kThreads / 32; ++w) c += counts[w];
    if (c) atomicAdd(count, c);
    atomicMin(&keys[0], lo0);
    atomicMin(&keys[1], lo1);
    atomicMax(&keys[2], hi0);
    atomicMax(&keys[3], hi1);
  }
}

struct Hist {
  float mn0, mn1;
  int sz0, sz1;
};

__device__ __forceinline__ int ll_bin(const LLParams& P, float x, float mn) {
  return (int)(P.inv_res != 0.0f ? (x - mn) * P.inv_res : (x - mn) / P.resolution);
}

// Calls count(bin) for every seed (bins below the histogram's size: the host
// checked the seeds' range against it).
template <class Count>
__device__ __forceinline__ void ll_for_seeds(const LLParams& P, const Hist& H, const float* __restrict__ img,
                                             const unsigned char* __restrict__ seeds, long long n, Count count) {
  auto bin = [&](long long i) {
    int b = ll_bin(P, img[P.comps * i], H.mn0);
    if (P.comps == 2) b = b * H.sz1 + ll_bin(P, img[2 * i + 1], H.mn1);
    return b;
  };
  const long long stride = (long long)gridDim.x * blockDim.x, t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nq = P.quads ? n / 4 : 0;
  for (long long q = t; q < nq; q += stride) {
    const unsigned bits = seeds[q];
    if (!bits) continue;
    if (P.comps == 1) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(img) + q);
      if (bits & 1u) count(ll_bin(P, v.x, H.mn0));
      if (bits & 2u) count(ll_bin(P, v.y, H.mn0));
      if (bits & 4u) count(ll_bin(P, v.z, H.mn0));
      if (bits & 8u) count(ll_bin(P, v.w, H.mn0));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (bits >> j & 1u) count(bin(4 * q + j));
    }
  }
  for (long long i = 4 * nq + t; i < n; i += stride)
    if (seeds[nq + (i - 4 * nq)]) count(bin(i));
}

// Histograms of up to kSharedBins bins (48 KB, the default dynamic shared
// memory limit): each CTA counts its voxels in shared memory and adds its non-zero bins to the global histogram once (integer
// counts, so the totals do not depend on the order).
constexpr int kSharedBins = 12288;
constexpr int kHistBlocks = 912;  // each CTA clears and adds its own histogram once
__global__ void ll_hist_shared_kernel(const LLParams P, const Hist H, const float* __restrict__ img,
                                      const unsigned char* __restrict__ seeds, long long n, int bins,
                                      unsigned int* hist) {
  extern __shared__ unsigned int sh[];  // bins entries
  for (int b = threadIdx.x; b < bins; b += blockDim.x) sh[b] = 0u;
  __syncthreads();
  ll_for_seeds(P, H, img, seeds, n, [&](int b) { atomicAdd(&sh[b], 1u); });
  __syncthreads();
  for (int b = threadIdx.x; b < bins; b += blockDim.x) {
    const unsigned int v = sh[b];
    if (v) atomicAdd(&hist[b], v);
  }
}

// Larger histograms: global atomics.
__global__ void ll_hist_kernel(const LLParams P, const Hist H, const float* __restrict__ img,
                               const unsigned char* __restrict__ seeds, long long n, unsigned int* hist) {
  ll_for_seeds(P, H, img, seeds, n, [&](int b) { atomicAdd(&hist[b], 1u); });
}

// The cost of a voxel depends on its bin only, so it is evaluated once per
// bin: frequency hist[i] / (float)szSample + 1.0e-10 (the counts kept as the
// reference's float increments keep them: they stop growing at 2^24), cost
// -log(frequency), divided by the cost of an empty bin, -log(1.0e-10), when
// normalised.  cost[bins] is the cost of a voxel outside the histogram.
__global__ void ll_cost_kernel(const unsigned int* __restrict__ hist, int bins, unsigned long long samples,
                               int normalize, float* __restrict__ cost) {
  const double floor_cost = -log(1.0e-10);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= bins; i += gridDim.x * blockDim.x) {
    float o;
    if (i < bins) {
      const float cnt = (float)min(hist[i], 16777216u);
      const float freq = (float)((double)(cnt / (float)(int)samples) + 1.0e-10);
      o = (float)(-log((double)freq));
    } else {
      o = (float)floor_cost;
    }
    if (normalize) o = (float)((double)o / floor_cost);
    cost[i] = o;
  }
}

__global__ void ll_out_kernel(const LLParams P, const Hist H, const float* __restrict__ img,
                              const float* __restrict__ cost, int bins, long long n, float* __restrict__ out) {
  const float outside = cost[bins];
  auto look = [&](float x0, float x1) {
    const int b0 = ll_bin(P, x0, H.mn0);
    if (x0 < H.mn0 || b0 >= H.sz0) return outside;
    if (P.comps == 1) return __ldg(cost + b0);
    const int b1 = ll_bin(P, x1, H.mn1);
    return (x1 < H.mn1 || b1 >= H.sz1) ? outside : __ldg(cost + (b0 * H.sz1 + b1));
  };
  const long long stride = (long long)gridDim.x * blockDim.x, t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nq = P.quads && P.comps == 1 ? n / 4 : 0;
  for (long long q = t; q < nq; q += stride) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(img) + q);
    reinterpret_cast<float4*>(out)[q] =
        make_float4(look(v.x, 0.0f), look(v.y, 0.0f), look(v.z, 0.0f), look(v.w, 0.0f));
  }
  for (long long i = 4 * nq + t; i < n; i += stride)
    out[i] = look(img[P.comps * i], P.comps == 2 ? img[2 * i + 1] : 0.0f);
}

// Device memory of one call, returned to the pool in stream order.
struct Scratch {
  explicit Scratch(cudaStream_t s) : stream(s), pool(scratch_pool()) {}
  cudaStream_t stream;
  cudaMemPool_t pool;
  std::vector<void*> bufs;
  ~Scratch() {
    for (void* p : bufs) pool ? cudaFreeAsync(p, stream) : cudaFree(p);
  }
  template <class T>
  cudaError_t alloc(T** out, size_t count) {
    void* p = nullptr;
    cudaError_t e = pool ? cudaMallocFromPoolAsync(&p, count * sizeof(T), pool, stream)
                         : cudaMalloc(&p, count * sizeof(T));
    if (e == cudaSuccess) bufs.push_back(p);
    *out = static_cast<T*>(p);
    return e;
  }
  template <class T>
  cudaError_t bring(const T* src, size_t count, int where, const T** dst, cudaStream_t s) {
    if (where == HMF_DEVICE) {
      *dst = src;
      return cudaSuccess;
    }
    T* d = nullptr;
    cudaError_t e = alloc(&d, count);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d, src, count * sizeof(T), cudaMemcpyHostToDevice, s);
    *dst = d;
    return e;
  }
};

hmf_ctx* const kNoCtx = nullptr;

}  // namespace

extern "C" {

int hmf_data_term(int op, int entropy, int normalize, double k1, double c1, double k2, double c2, const float* in1,
                  const float* in2, long long n_voxels, float* out, int where, void* stream) {
  hmf_ctx* c = kNoCtx;
  if (!in1 || !out || n_voxels < 1) return fail(c, HMF_ERR_INVALID_ARGUMENT, "an image or the output is missing");
  if (where != HMF_HOST && where != HMF_DEVICE) return fail(c, HMF_ERR_INVALID_ARGUMENT, "bad `where`");
  if (op < HMF_DATA_TERM_CONSTANT || op > HMF_DATA_TERM_SPIKE)
    return fail(c, HMF_ERR_INVALID_ARGUMENT, "unknown data-term operation");
  if (in2 && op == HMF_DATA_TERM_SPIKE)
    return fail(c, HMF_ERR_INVALID_ARGUMENT,
                "the spike operation takes one image (the reference's two-image form writes no output)");
  if (where == HMF_DEVICE)
    for (const void* q : {(const void*)in1, (const void*)in2, (const void*)out})
      if (int rc = check_device_pointer(c, q, "data-term buffer")) return rc;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  TermParams P{};
  P.op = op;
  P.entropy = entropy != 0;
  P.two = in2 != nullptr;
  P.k1 = k1;
  P.k2 = k2;
  // constants as Execute1 / Execute2 derive them (note: Execute1's second
  // constant is C1 unless it is a logarithm; Execute2 takes logarithms for
  // the constant operation only and never normalises)
  if (!P.two) {
    const bool lg = (op == HMF_DATA_TERM_CONSTANT || op == HMF_DATA_TERM_SPIKE) && P.entropy;
    P.c1 = lg ? -std::log(c1) : c1;
    P.c2 = lg ? -std::log(c2) : c1;
  } else {
    const bool lg = op == HMF_DATA_TERM_CONSTANT && P.entropy;
    P.c1 = lg ? -std::log(c1) : c1;
    P.c2 = lg ? -std::log(c2) : c2;
  }
  Scratch sc(s);
  const float* d1 = nullptr;
  const float* d2 = nullptr;
  float* dout = out;
  cudaError_t e = sc.bring(in1, (size_t)n_voxels, where, &d1, s);
  if (e == cudaSuccess && in2) e = sc.bring(in2, (size_t)n_voxels, where, &d2, s);
  if (e == cudaSuccess && where == HMF_HOST) e = sc.alloc(&dout, (size_t)n_voxels);
  if (e != cudaSuccess) return cuda_fail(c, e, "data-term input copy");
  if (normalize && !P.two) {
    // vtkImageDataTermExecute1's normalisation (:187-249) by the first image's range
    unsigned int* mm = nullptr;
    unsigned int h[2] = {0, 0};
    // a constant's and a spike's normalisation does not depend on the range
    const bool ranged = op == HMF_DATA_TERM_GAUSSIAN || op == HMF_DATA_TERM_LOGISTIC;
    // the Gaussian entropy's needs no function of the host's library: the
    // kernel forms it from the range on the device, without a synchronisation
    const bool on_device = op == HMF_DATA_TERM_GAUSSIAN && P.entropy;
    if (ranged) {
      e = sc.alloc(&mm, 2);
      if (e == cudaSuccess) e = cudaMemsetAsync(mm, 0, 2 * sizeof(unsigned int), s);
      if (e == cudaSuccess) {
        range_kernel<<<std::min(grid_for((n_voxels + 3) / 4), kReduceBlocks), kThreads, 0, s>>>(d1, n_voxels, mm);
        e = cudaGetLastError();
      }
      if (e == cudaSuccess && !on_device) e = cudaMemcpyAsync(h, mm, sizeof(h), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess && !on_device) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return cuda_fail(c, e, "data-term range");
    }
    P.normalize = on_device ? 2 : 1;
    P.range = mm;
    const double R0 = key_float(~h[0]), R1 = key_float(h[1]);
    const double K1 = P.k1, C1 = P.c1;
    double off = 0.0, mul = 1.0 / C1;
    if (op == HMF_DATA_TERM_GAUSSIAN) {
      const double vmax = std::exp(-0.5 * ((R1 - C1) / K1) * ((R1 - C1) / K1));
      const double vmin = std::exp(-0.5 * ((R0 - C1) / K1) * ((R0 - C1) / K1));
      const double mn = std::exp(-((vmax >= vmin) ? vmax : vmin));
      double mx = std::exp(-((vmax < vmin) ? vmax : vmin));
      if (C1 > R0 && C1 < R1) mx = 1.0f;
      off = -mn;
      mul = 1.0 / (mx - mn);
    } else if (op == HMF_DATA_TERM_LOGISTIC && P.entropy) {
      const double vmax = std::log(1.0 + std::exp(-(K1 * (R1 - C1))));
      const double vmin = std::log(1.0 + std::exp(-(K1 * (R0 - C1))));
      const double mx = (vmax >= vmin) ? vmax : vmin;
      const double mn = (vmax < vmin) ? vmax : vmin;
      off = -mn;
      mul = 1.0 / (mx - mn);
    } else if (op == HMF_DATA_TERM_LOGISTIC) {
      const double vmax = 1.0 / (1.0 + std::exp(-(K1 * (R1 - C1))));
      const double vmin = 1.0 / (1.0 + std::exp(-(K1 * (R0 - C1))));
      const double mx = (vmax >= vmin) ? vmax : vmin;
      const double mn = (vmax < vmin) ? vmax : vmin;
      off = -mn;
      mul = 1.0 / (mx - mn);
    }
    P.off = off;
    P.mul = mul;
  }
  if (op == HMF_DATA_TERM_CONSTANT || op == HMF_DATA_TERM_SPIKE) {
    float value[2] = {(float)P.c1, (float)P.c2};
    if (P.normalize)
      for (float& v : value) v = (float)(((double)v + P.off) * P.mul);
    const float spike = (float)P.k1;
    if (op == HMF_DATA_TERM_SPIKE && !((double)spike == P.k1)) value[0] = value[1];  // no float equals K1
    term_choice_kernel<<<grid_for((n_voxels + 3) / 4), kThreads, 0, s>>>(op == HMF_DATA_TERM_SPIKE ? d1 : nullptr, spike,
                                                                        value[0], value[1], n_voxels, dout);
  } else {
    const bool gauss = op == HMF_DATA_TERM_GAUSSIAN;
    P.c1s = split3(P.c1);
    P.c2s = split3(P.c2);
    P.k1s = split2(gauss ? 1.0 / P.k1 : P.k1);
    P.k2s = split2(gauss ? 1.0 / P.k2 : P.k2);
    // the constants are in the float-float forms' range
    const bool fast = (!gauss || P.entropy) && ff_safe(P.c1) && ff_safe(P.k1) && P.k1 != 0.0 &&
                      (!P.two || (ff_safe(P.c2) && ff_safe(P.k2) && P.k2 != 0.0));
    const uintptr_t at = reinterpret_cast<uintptr_t>(d1) | reinterpret_cast<uintptr_t>(d2) | reinterpret_cast<uintptr_t>(dout);
    const bool in_double = !fast || n_voxels < kTermFast[gauss ? 0 : 1];
    const int quads = !in_double && n_voxels >= kTermQuads[gauss ? 0 : 1] && (at & 15) == 0;
    const int grid = grid_for(quads ? (n_voxels + 3) / 4 : n_voxels);
    if (in_double) {
      data_term_kernel<<<grid, kThreads, 0, s>>>(P, InDouble{}, d1, d2, n_voxels, 0, dout);
    } else if (gauss) {
      data_term_kernel<<<grid, kThreads, 0, s>>>(P, NoTables{}, d1, d2, n_voxels, quads, dout);
    } else {
      static const TermTables tables = make_term_tables();
      data_term_kernel<<<grid, kThreads, 0, s>>>(P, tables, d1, d2, n_voxels, quads, dout);
    }
  }
  e = cudaGetLastError();
  if (e == cudaSuccess && where == HMF_HOST) {
    e = cudaMemcpyAsync(out, dout, sizeof(float) * (size_t)n_voxels, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "data_term_kernel");
  return HMF_OK;
}

int hmf_log_likelihood(const float* image, int components, const int* const* label_maps, int n_label_maps,
                       long long n_voxels, int label_id, float resolution, double required_agreement, int normalize,
                       float* out, int where, void* stream) {
  hmf_ctx* c = kNoCtx;
  if (!image || !out || n_voxels < 1) return fail(c, HMF_ERR_INVALID_ARGUMENT, "the image or the output is missing");
  if (where != HMF_HOST && where != HMF_DEVICE) return fail(c, HMF_ERR_INVALID_ARGUMENT, "bad `where`");
  if (components != 1 && components != 2)
    return fail(c, HMF_ERR_INVALID_ARGUMENT, "the image must have one or two components");
  if (n_label_maps < 0 || n_label_maps > HMF_MAX_LABEL_MAPS || (n_label_maps && !label_maps))
    return fail(c, HMF_ERR_INVALID_ARGUMENT, "bad label-map list");
  if (!(resolution >= FLT_MIN)) return fail(c, HMF_ERR_INVALID_ARGUMENT, "histogram resolution must be positive");
  if (!(required_agreement >= 0.0 && required_agreement <= 1.0))
    return fail(c, HMF_ERR_INVALID_ARGUMENT, "required agreement must lie in [0, 1]");
  if (where == HMF_DEVICE) {
    if (int rc = check_device_pointer(c, image, "log-likelihood image")) return rc;
    if (int rc = check_device_pointer(c, out, "log-likelihood output")) return rc;
    for (int k = 0; k < n_label_maps; ++k)
      if (int rc = check_device_pointer(c, label_maps[k], "label map")) return rc;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  LLParams P{};
  P.comps = components;
  P.n_maps = n_label_maps;
  P.label_id = label_id;
  P.resolution = resolution;
  int exponent = 0;
  if (resolution <= 0x1p100f && std::frexp(resolution, &exponent) == 0.5f) P.inv_res = 1.0f / resolution;
  LLMaps M{};
  Scratch sc(s);
  const float* img = nullptr;
  float* dout = out;
  cudaError_t e = sc.bring(image, (size_t)n_voxels * components, where, &img, s);
  for (int k = 0; k < n_label_maps && e == cudaSuccess; ++k) {
    if (!label_maps[k]) continue;
    ++P.actual_maps;
    e = sc.bring(label_maps[k], (size_t)n_voxels, where, &M.map[k], s);
  }
  P.min_agree = n_label_maps + 1;  // no count qualifies
  for (int k = 0; k <= n_label_maps; ++k)
    if ((double)k >= required_agreement * (double)P.actual_maps) {
      P.min_agree = k;
      break;
    }
  if (e == cudaSuccess && where == HMF_HOST) e = sc.alloc(&dout, (size_t)n_voxels);
  unsigned long long* cnt = nullptr;
  unsigned int* keys = nullptr;
  unsigned char* seeds = nullptr;
  uintptr_t at = reinterpret_cast<uintptr_t>(img) | reinterpret_cast<uintptr_t>(dout);
  for (int k = 0; k < n_label_maps; ++k) at |= reinterpret_cast<uintptr_t>(M.map[k]);
  P.quads = (at & 15) == 0;
  const size_t n_seed_bytes = P.quads ? (size_t)(n_voxels / 4 + n_voxels % 4) : (size_t)n_voxels;
  if (e == cudaSuccess) e = sc.alloc(&seeds, n_seed_bytes);
  if (e == cudaSuccess) e = sc.alloc(&cnt, 1);
  if (e == cudaSuccess) e = sc.alloc(&keys, 4);
  if (e != cudaSuccess) return cuda_fail(c, e, "log-likelihood input copy");
  const unsigned int kinit[4] = {0xffffffffu, 0xffffffffu, 0u, 0u};
  e = cudaMemsetAsync(cnt, 0, sizeof(*cnt), s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(keys, kinit, sizeof(kinit), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    ll_scan_kernel<<<std::min(grid_for((n_voxels + 3) / 4), kReduceBlocks), kThreads, 0, s>>>(P, M, img, n_voxels, cnt, keys,
                                                                                       seeds);
    e = cudaGetLastError();
  }
  unsigned long long samples = 0;
  unsigned int hk[4] = {0, 0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&samples, cnt, sizeof(samples), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(hk, keys, sizeof(hk), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(c, e, "log-likelihood scan");
  if (samples == 0) {
    // no seed voxel: every cost 1 (std::fill_n, vtkImageLogLikelihood.cxx:193-197)
    std::vector<float> ones;
    if (where == HMF_HOST) {
      for (long long i = 0; i < n_voxels; ++i) out[i] = 1.0f;
      return HMF_OK;
    }
    ones.assign((size_t)n_voxels, 1.0f);
    e = cudaMemcpyAsync(out, ones.data(), sizeof(float) * ones.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(c, e, "log-likelihood output");
    return HMF_OK;
  }
  // min starts at FLT_MAX and max at FLT_MIN (:169-170), compared as floats
  Hist H{};
  float mn[2] = {FLT_MAX, FLT_MAX}, mx[2] = {FLT_MIN, FLT_MIN};
  for (int k = 0; k < components; ++k) {
    const float lo = key_float(hk[k]), hi = key_float(hk[2 + k]);
    mn[k] = (mn[k] < lo) ? mn[k] : lo;
    mx[k] = (mx[k] > hi) ? mx[k] : hi;
  }
  H.mn0 = mn[0];
  H.mn1 = mn[1];
  // the reference's bin counts, precedence as written: (int)(max - min/resolution) + 1
  const float s0 = mx[0] - mn[0] / resolution;
  if (!(s0 > -1.0f && s0 < 2.0e9f)) return fail(c, HMF_ERR_INVALID_ARGUMENT, "histogram size out of range");
  H.sz0 = (int)s0 + 1;
  H.sz1 = 1;
  if (components == 2) {
    const float s1 = mx[1] - mn[1] / resolution;
    if (!(s1 > -1.0f && s1 < 2.0e9f)) return fail(c, HMF_ERR_INVALID_ARGUMENT, "histogram size out of range");
    H.sz1 = (int)s1 + 1;
  }
  // the reference writes past its histogram when a seed's bin exceeds that
  // count (its bin count divides only the minimum by the resolution)
  if ((int)((mx[0] - mn[0]) / resolution) >= H.sz0 ||
      (components == 2 && (int)((mx[1] - mn[1]) / resolution) >= H.sz1))
    return fail(c, HMF_ERR_INVALID_ARGUMENT,
                "seed values span more bins than the reference's histogram holds "
                "((int)(max - min/resolution) + 1 bins): it would write past its histogram");
  const long long bins = (long long)H.sz0 * H.sz1;
  if (bins > (1LL << 28)) return fail(c, HMF_ERR_INVALID_ARGUMENT, "histogram of more than 2^28 bins");
  unsigned int* hist = nullptr;
  float* cost = nullptr;
  e = sc.alloc(&hist, (size_t)bins);
  if (e == cudaSuccess) e = sc.alloc(&cost, (size_t)bins + 1);
  if (e == cudaSuccess) e = cudaMemsetAsync(hist, 0, sizeof(unsigned int) * (size_t)bins, s);
  if (e == cudaSuccess) {
    if (bins <= kSharedBins)
      ll_hist_shared_kernel<<<std::min(grid_for((n_voxels + 3) / 4), kHistBlocks), kThreads,
                              sizeof(unsigned int) * (size_t)bins, s>>>(P, H, img, seeds, n_voxels, (int)bins, hist);
    else
      ll_hist_kernel<<<grid_for((n_voxels + 3) / 4), kThreads, 0, s>>>(P, H, img, seeds, n_voxels, hist);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    ll_cost_kernel<<<grid_for(bins + 1), kThreads, 0, s>>>(hist, (int)bins, samples, normalize != 0, cost);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    ll_out_kernel<<<grid_for(components == 1 ? (n_voxels + 3) / 4 : n_voxels), kThreads, 0, s>>>(P, H, img, cost, (int)bins, n_voxels, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && where == HMF_HOST)
    e = cudaMemcpyAsync(out, dout, sizeof(float) * (size_t)n_voxels, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // the call is synchronous
  if (e != cudaSuccess) return cuda_fail(c, e, "log-likelihood kernels");
  return HMF_OK;
}

}  // extern "C"

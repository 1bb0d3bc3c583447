// Splits the operands of an fp32 product into the fp16 parts that gemm_tcgen05_f32h2.cuh multiplies:
//   x * 2^e = hi + 2^-12 lo,
// one exponent e for 64 values of K of a row of A, or for 64 values of K of 64 columns of B, which have been multiplied by a
// power of two of each column's own, 1 or more. One pass: a CTA takes 128 rows x 64 values of K of A, or 64 values of K x 128 columns
// of B, into registers (32 KB), finds the largest magnitudes, and writes both parts where one TMA box of the product's stage
// will read them:
//   A  [panel of 128 rows][64 values of K][hi, lo][row][64 halves]
//   B  [64 columns][64 values of K][hi, lo][value of K][64 halves]
// and the factors 2^-e as [64 values of K][row, or 64 columns]. Bound by memory: 4 bytes read and 4 written per value.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "kernels/ptx_sm100.cuh"
#include "kernels/split_f32.h"

extern "C" int kcg_internal_fail(int code, const char* msg);

namespace {

constexpr int kThreads = 256, kRows = 128, kBK = 64;

struct Scale {
  float mult, inv;  // 2^e and 2^-e; e brings the largest magnitude into [2^14, 2^15)
  bool ok;          // false: outside 2^+-50 (or infinite, or NaN)
};
// from the bits of the largest magnitude
__device__ __forceinline__ Scale scale_of(uint32_t top) {
  const uint32_t e = top >> 23;  // biased
  Scale s;
  s.ok = top == 0u || (e >= 127u - 50u && e <= 127u + 50u);
  const bool use = s.ok && top != 0u;
  s.mult = use ? __uint_as_float((268u - e) << 23) : 1.f;
  s.inv = use ? __uint_as_float((e - 14u) << 23) : 1.f;
  return s;
}

// The power of two, from 1 to 2^40, that brings a value of this magnitude up to the largest of its 64 columns. (Never below 1:
// the sums that the product keeps are of the multiplied columns, and must not underflow where those of the columns do not.)
__device__ __forceinline__ float column_power(uint32_t bits, uint32_t largest) {
  const int up = bits == 0u ? 0 : min(static_cast<int>(largest >> 23) - static_cast<int>(bits >> 23), 40);
  return __uint_as_float(static_cast<uint32_t>(127 + up) << 23);
}

__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }

// Four values as hi and lo parts; true where one of them keeps less than 21 bits.
__device__ __forceinline__ bool split4(const float4& x, float mult, uint2* hi, uint2* lo) {
  const float v[4] = {x.x * mult, x.y * mult, x.z * mult, x.w * mult};
  bool lost = false;
  if (mult < 1.f)  // it may turn a value to zero, of which nothing is missed below
    lost = (v[0] == 0.f && x.x != 0.f) || (v[1] == 0.f && x.y != 0.f) || (v[2] == 0.f && x.z != 0.f) || (v[3] == 0.f && x.w != 0.f);
  uint32_t h[2], l[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const __half2 a = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    const float2 af = __half22float2(a);
    // (exact: what the rounding left has fewer bits than the value)
    const float d0 = (v[2 * i] - af.x) * 4096.f, d1 = (v[2 * i + 1] - af.y) * 4096.f;
    const __half2 b = __floats2half2_rn(d0, d1);
    const float2 bf = __half22float2(b);
    // what both parts leave out, against 2^-21 of the value: 2^-21 * 2^12
    lost |= fabsf(d0 - bf.x) > fabsf(v[2 * i]) * 0x1p-9f;
    lost |= fabsf(d1 - bf.y) > fabsf(v[2 * i + 1]) * 0x1p-9f;
    h[i] = *reinterpret_cast<const uint32_t*>(&a);
    l[i] = *reinterpret_cast<const uint32_t*>(&b);
  }
  *hi = make_uint2(h[0], h[1]);
  *lo = make_uint2(l[0], l[1]);
  return lost;
}

__global__ void __launch_bounds__(kThreads) split_f32_kernel(const kcg::SplitF32Args q) {
  kcg::griddep_launch_dependents();
  kcg::griddep_wait();  // the kernel before this one may have written the operands or still read the parts
  const int num_kb = (q.K + kBK - 1) / kBK;
  const int blocks_a = (q.M + kRows - 1) / kRows * num_kb;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool bad = false;
  // Where a value did not split, nobody will read the parts: the CTAs that come to run after that was seen leave. (Asked
  // behind the first wave or so, where it is not the whole of a small problem's time.)
  if (blockIdx.x >= 1024u && __syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile unsigned int*>(q.words) != 0u))
    return;
  if (static_cast<int>(blockIdx.x) < blocks_a) {
    const int panel = blockIdx.x / num_kb, kb = blockIdx.x % num_kb;
    // 16 threads hold a row's 64 values; eight rows per thread
    const int r0 = threadIdx.x >> 4, k4 = (threadIdx.x & 15) * 4, k = kb * kBK + k4;
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = panel * kRows + r0 + 16 * i;
      x[i] = row < q.M && k < q.K ? __ldg(reinterpret_cast<const float4*>(q.A + static_cast<size_t>(row) * q.lda + k))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    uint8_t* block = q.parts_a + (static_cast<size_t>(panel) * num_kb + kb) * (2 * kRows * 128);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t top = max(max(magnitude(x[i].x), magnitude(x[i].y)), max(magnitude(x[i].z), magnitude(x[i].w)));
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, s));
      const Scale sc = scale_of(top);
      uint2 hi, lo;
      bad |= split4(x[i], sc.mult, &hi, &lo) || !sc.ok;
      const int r = r0 + 16 * i;
      *reinterpret_cast<uint2*>(block + r * 128 + k4 * 2) = hi;
      *reinterpret_cast<uint2*>(block + (kRows + r) * 128 + k4 * 2) = lo;
      if (k4 == 0) q.scale_a[static_cast<size_t>(kb) * q.scale_lda + panel * kRows + r] = sc.inv;
    }
  } else {
    __shared__ uint4 column_top[kThreads / 32][32];
    __shared__ uint32_t chunk_top[kThreads / 32][2];
    const int b = blockIdx.x - blocks_a;
    const int cols = b / num_kb, kb = b % num_kb;
    // a warp holds 128 columns of a value of K, four per lane; eight values of K per thread
    const int n = cols * 128 + lane * 4;
    const bool there = n < q.N;  // (N is a multiple of 64: a chunk of 64 columns is there or not)
    auto load = [&](int k) {
      return k < q.K && there ? __ldg(reinterpret_cast<const float4*>(q.B + static_cast<size_t>(k) * q.ldb + n))
                              : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    const float4 sample = load(static_cast<int>(static_cast<long long>(warp) * q.K / (kThreads / 32)));
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = load(kb * kBK + warp + 8 * i);
    // each column's own power of two, from eight of its values (the same eight in every CTA): it evens out columns of
    // different size; any power would do, the exponent of the chunk follows what it leaves
    column_top[warp][lane] = make_uint4(magnitude(sample.x), magnitude(sample.y), magnitude(sample.z), magnitude(sample.w));
    __syncthreads();
    uint4 ct = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int o = 0; o < kThreads / 32; ++o) {
      const uint4 v = column_top[o][lane];
      ct = make_uint4(max(ct.x, v.x), max(ct.y, v.y), max(ct.z, v.z), max(ct.w, v.w));
    }
    uint32_t largest = max(max(ct.x, ct.y), max(ct.z, ct.w));  // of this lane's 64 columns
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, s));
    const float4 cm = make_float4(column_power(ct.x, largest), column_power(ct.y, largest), column_power(ct.z, largest),
                                  column_power(ct.w, largest));
    uint32_t top = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[i] = make_float4(x[i].x * cm.x, x[i].y * cm.y, x[i].z * cm.z, x[i].w * cm.w);
      top = max(top, max(max(magnitude(x[i].x), magnitude(x[i].y)), max(magnitude(x[i].z), magnitude(x[i].w))));
    }
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, s));
    if ((lane & 15) == 0) chunk_top[warp][lane >> 4] = top;
    __syncthreads();
#pragma unroll
    for (int o = 0; o < kThreads / 32; ++o) top = max(top, chunk_top[o][lane >> 4]);
    const Scale sc = scale_of(top);
    bad = !sc.ok;
    if (there) {
      if (kb == 0 && warp == 0)
        *reinterpret_cast<float4*>(q.columns + n) = make_float4(1.f / cm.x, 1.f / cm.y, 1.f / cm.z, 1.f / cm.w);
      if (warp == 0 && (lane & 15) == 0) q.scale_b[static_cast<size_t>(kb) * q.scale_ldb + (n >> 6)] = sc.inv;
      uint8_t* block = q.parts_b + (static_cast<size_t>(n >> 6) * num_kb + kb) * (2 * kBK * 128) + (n & 63) * 2;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint2 hi, lo;
        bad |= split4(x[i], sc.mult, &hi, &lo);
        *reinterpret_cast<uint2*>(block + (warp + 8 * i) * 128) = hi;
        *reinterpret_cast<uint2*>(block + (kBK + warp + 8 * i) * 128) = lo;
      }
    }
  }
  if (bad) *reinterpret_cast<volatile unsigned int*>(q.words) = 1u;
}

}  // namespace

// Queues the split on the current context's stream; `pdl`: it may be brought in as the kernel before it ends.
extern "C" int kcg_internal_split_f32(uint64_t stream, const kcg::SplitF32Args* q, int pdl) {
  const int num_kb = (q->K + kBK - 1) / kBK;
  const long long blocks = (static_cast<long long>((q->M + kRows - 1) / kRows) + (q->N + 127) / 128) * num_kb;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, split_f32_kernel, *q);
  if (e != cudaSuccess)
    return kcg_internal_fail(static_cast<int>(e), (std::string("operand split launch: ") + cudaGetErrorString(e)).c_str());
  return 0;  // (counted with the product that it is a part of)
}

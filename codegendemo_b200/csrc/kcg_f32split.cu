// Splits the operands of an fp32 product into the fp16 parts that gemm_tcgen05_f32h2.cuh multiplies:
//   x * 2^e = hi + 2^-12 lo,
// one exponent e for 64 values of K of a row of A, or for 64 values of K of 64 columns of B, which have been multiplied by a
// power of two of each column's own, 1 or more. One pass: a CTA takes 128 rows x 64 values of K of A, or 64 values of K x 128 columns
// of B, into registers (32 KB), finds the largest magnitudes, and writes both parts where one TMA box of the product's stage
// will read them:
//   A  [panel of 128 rows][64 values of K][hi, lo][row][64 halves]
//   B  [64 columns][64 values of K][hi, lo][value of K][64 halves]
// and the factors 2^-e as [64 values of K][row, or 64 columns]. Bound by memory: 4 bytes read and 4 written per value.
//
// A chunk (128 rows of A, or 64 columns of B, by 64 values of K) with a value so far below the largest beside it that the parts
// would keep less than 21 bits of it has such values as zeros in its parts, and a second pair, the far parts, of them alone, under
// an exponent of their own: the product multiplies the chunk once more. (A value in 10^9 of a normal distribution is one. With
// the whole product taken as 3xTF32 for it, 1024x7936x768 took 84 us, 47 without such a value.) What far parts cannot carry either -
// values outside 2^+-50, infinities, NaNs, a second pair's own far values, more chunks than there are slots - sets a flag.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "kernels/gemm_params.h"
#include "kernels/ptx_sm100.cuh"
#include "kernels/split_f32.h"

extern "C" int kcg_internal_fail(int code, const char* msg);

namespace {

constexpr int kThreads = 256, kRows = 128, kBK = kcg::H2_BK;

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

// Bit i where split4 would keep less than 21 bits of value i.
__device__ __forceinline__ uint32_t lost_of(const float4& x, float mult) {
  uint2 hi, lo;
  return (split4(make_float4(x.x, 0.f, 0.f, 0.f), mult, &hi, &lo) ? 1u : 0u) | (split4(make_float4(x.y, 0.f, 0.f, 0.f), mult, &hi, &lo) ? 2u : 0u) |
         (split4(make_float4(x.z, 0.f, 0.f, 0.f), mult, &hi, &lo) ? 4u : 0u) | (split4(make_float4(x.w, 0.f, 0.f, 0.f), mult, &hi, &lo) ? 8u : 0u);
}

// The values of x whose bit is set; the others are zero.
__device__ __forceinline__ float4 pick(const float4& x, uint32_t bits) {
  return make_float4(bits & 1u ? x.x : 0.f, bits & 2u ? x.y : 0.f, bits & 4u ? x.z : 0.f, bits & 8u ? x.w : 0.f);
}

__device__ __forceinline__ uint32_t magnitude(const float4& x) {
  return max(max(magnitude(x.x), magnitude(x.y)), max(magnitude(x.z), magnitude(x.w)));
}

// The largest of 16 threads' values (a half warp).
__device__ __forceinline__ uint32_t max_of_16(uint32_t v) {
#pragma unroll
  for (int s = 8; s > 0; s >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, s));
  return v;
}

// A slot for far parts, from 1 on; 0: they are all taken.
__device__ __forceinline__ int take_slot(const kcg::SplitF32Args& q, int taken, int slots) {
  const unsigned int n = atomicAdd(q.words + taken, 1u);
  if (n == 0u) {
    atomicOr(q.words + kcg::H2_FOUND, kcg::H2_FAR);
    q.far_scale_b[q.far_slots_b] = 0.f;
  }
  return n < static_cast<unsigned int>(slots) ? static_cast<int>(n) + 1 : 0;
}

// A factor with the chunk's slot.
__device__ __forceinline__ float with_slot(float factor, int slot) { return __uint_as_float(__float_as_uint(factor) | static_cast<uint32_t>(slot)); }

// The power of two of each of a lane's four columns n .. n + 3 (the largest of eight values of each warp's share of K): it evens out
// columns of different size; any power would do, the exponent of the chunk follows what it leaves. The same in every CTA.
struct Columns {
  uint4 top[kThreads / 32][32];
};
__device__ __forceinline__ float4 column_powers(const float4& sample, int warp, int lane, Columns* shared) {
  shared->top[warp][lane] = make_uint4(magnitude(sample.x), magnitude(sample.y), magnitude(sample.z), magnitude(sample.w));
  __syncthreads();
  uint4 ct = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int o = 0; o < kThreads / 32; ++o) {
    const uint4 v = shared->top[o][lane];
    ct = make_uint4(max(ct.x, v.x), max(ct.y, v.y), max(ct.z, v.z), max(ct.w, v.w));
  }
  const uint32_t largest = max_of_16(max(max(ct.x, ct.y), max(ct.z, ct.w)));  // of this lane's 64 columns
  return make_float4(column_power(ct.x, largest), column_power(ct.y, largest), column_power(ct.z, largest),
                     column_power(ct.w, largest));
}

// The largest of a lane's chunk of 64 columns, over all warps.
__device__ __forceinline__ uint32_t over_chunk(uint32_t v, int warp, int lane, uint32_t (*shared)[2]) {
  v = max_of_16(v);
  if ((lane & 15) == 0) shared[warp][lane >> 4] = v;
  __syncthreads();
#pragma unroll
  for (int o = 0; o < kThreads / 32; ++o) v = max(v, shared[o][lane >> 4]);
  return v;
}

__device__ __forceinline__ float4 load_a(const kcg::SplitF32Args& q, int row, int k) {
  return row < q.M && k < q.K ? __ldg(reinterpret_cast<const float4*>(q.A + static_cast<size_t>(row) * q.lda + k))
                              : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ float4 load_b(const kcg::SplitF32Args& q, int k, int n) {
  return k < q.K && n < q.N ? __ldg(reinterpret_cast<const float4*>(q.B + static_cast<size_t>(k) * q.ldb + n))
                            : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ int sample_row(const kcg::SplitF32Args& q, int warp) {
  return static_cast<int>(static_cast<long long>(warp) * q.K / (kThreads / 32));
}
__device__ __forceinline__ void store_a(uint8_t* block, int r, int k4, const uint2& hi, const uint2& lo) {
  *reinterpret_cast<uint2*>(block + r * 128 + k4 * 2) = hi;
  *reinterpret_cast<uint2*>(block + (kRows + r) * 128 + k4 * 2) = lo;
}
__device__ __forceinline__ void store_b(uint8_t* block, int k, int n, const uint2& hi, const uint2& lo) {
  *reinterpret_cast<uint2*>(block + (n & 63) * 2 + k * 128) = hi;
  *reinterpret_cast<uint2*>(block + (n & 63) * 2 + (kBK + k) * 128) = lo;
}
__device__ __forceinline__ uint8_t* parts_of_a(const kcg::SplitF32Args& q, int panel, int kb, int num_kb) {
  return q.parts_a + (static_cast<size_t>(panel) * num_kb + kb) * (2 * kRows * 128);
}
__device__ __forceinline__ uint8_t* parts_of_b(const kcg::SplitF32Args& q, int n, int kb, int num_kb) {
  return q.parts_b + (static_cast<size_t>(n >> 6) * num_kb + kb) * (2 * kBK * 128);
}

// The parts of a chunk of A again, without the values that lie far below, and its far parts. True: these cannot carry them, or all
// slots are taken. (Functions of their own, which read the operand again and take copies of the arguments: the registers are those of
// the path that every CTA goes, and its arguments stay in constant memory.)
__device__ __noinline__ bool far_parts_a(const kcg::SplitF32Args q, int panel, int kb) {
  __shared__ int slot;
  const int num_kb = (q.K + kBK - 1) / kBK;
  const int r0 = threadIdx.x >> 4, k4 = (threadIdx.x & 15) * 4;
  if (threadIdx.x == 0) slot = take_slot(q, kcg::H2_FAR_A, q.far_slots_a);
  __syncthreads();
  if (slot == 0) return true;
  uint8_t* block = parts_of_a(q, panel, kb, num_kb);
  uint8_t* far = q.far_a + static_cast<size_t>(slot - 1) * (2 * kRows * 128);
  bool bad = false;
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + 16 * i;
    const float4 x = load_a(q, panel * kRows + r, kb * kBK + k4);
    const Scale sc = scale_of(max_of_16(magnitude(x)));
    const uint32_t bits = lost_of(x, sc.mult);
    uint2 hi, lo;
    split4(pick(x, ~bits), sc.mult, &hi, &lo);
    store_a(block, r, k4, hi, lo);
    const float4 small = pick(x, bits);
    const Scale own = scale_of(max_of_16(magnitude(small)));
    bad |= split4(small, own.mult, &hi, &lo) || !own.ok;
    store_a(far, r, k4, hi, lo);
    if (k4 == 0) q.far_scale_a[(slot - 1) * kRows + r] = own.inv;
    if (r == 0 && k4 == 0) q.scale_a[static_cast<size_t>(kb) * q.scale_lda + panel * kRows] = with_slot(sc.inv, slot);
  }
  return bad;
}

// The same for the two chunks of B, of which one or both have such values.
__device__ __noinline__ bool far_parts_b(const kcg::SplitF32Args q, int cols, int kb, bool lost) {
  __shared__ Columns columns;
  __shared__ uint32_t chunk_top[2][kThreads / 32][2];
  __shared__ int slots[2];
  const int num_kb = (q.K + kBK - 1) / kBK;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = cols * 128 + lane * 4;
  const int lost0 = __syncthreads_or(lost && lane < 16), lost1 = __syncthreads_or(lost && lane >= 16);
  if (threadIdx.x < 2) slots[threadIdx.x] = (threadIdx.x == 0 ? lost0 : lost1) ? take_slot(q, kcg::H2_FAR_B, q.far_slots_b) : 0;
  const float4 cm = column_powers(load_b(q, sample_row(q, warp), n), warp, lane, &columns);
  auto load = [&](int i) {
    const float4 x = load_b(q, kb * kBK + warp + 8 * i, n);
    return make_float4(x.x * cm.x, x.y * cm.y, x.z * cm.z, x.w * cm.w);
  };
  uint32_t top = 0u;
  for (int i = 0; i < 8; ++i) top = max(top, magnitude(load(i)));
  const Scale sc = scale_of(over_chunk(top, warp, lane, chunk_top[0]));
  top = 0u;
  for (int i = 0; i < 8; ++i) {
    const float4 x = load(i);
    top = max(top, magnitude(pick(x, lost_of(x, sc.mult))));
  }
  const Scale own = scale_of(over_chunk(top, warp, lane, chunk_top[1]));
  const int slot = slots[lane >> 4];
  if ((lane < 16 ? lost0 : lost1) == 0) return false;
  if (slot == 0) return true;
  bool bad = !own.ok;
  uint8_t* block = parts_of_b(q, n, kb, num_kb);
  uint8_t* far = q.far_b + static_cast<size_t>(slot - 1) * (2 * kBK * 128);
  if (warp == 0 && (lane & 15) == 0) {
    q.far_scale_b[slot - 1] = own.inv;
    q.scale_b[static_cast<size_t>(kb) * q.scale_ldb + (n >> 6)] = with_slot(sc.inv, slot);
  }
  for (int i = 0; i < 8; ++i) {
    const float4 x = load(i);
    const uint32_t bits = lost_of(x, sc.mult);
    uint2 hi, lo;
    split4(pick(x, ~bits), sc.mult, &hi, &lo);
    store_b(block, warp + 8 * i, n, hi, lo);
    bad |= split4(pick(x, bits), own.mult, &hi, &lo);
    store_b(far, warp + 8 * i, n, hi, lo);
  }
  return bad;
}

__global__ void __launch_bounds__(kThreads) split_f32_kernel(const kcg::SplitF32Args q) {
  kcg::griddep_launch_dependents();
  kcg::griddep_wait();  // the kernel before this one may have written the operands or still read the parts
  const int num_kb = (q.K + kBK - 1) / kBK;
  const int blocks_a = (q.M + kRows - 1) / kRows * num_kb;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int* flag = q.words + kcg::H2_FLAG + blockIdx.x % kcg::H2_FLAGS * kcg::H2_LINE;
  // Where a value does not split, nobody will read the parts: the CTAs that come to run after their flag was set leave. (Asked
  // behind the first wave or so, where it is not the whole of a small problem's time.)
  if (blockIdx.x >= 1024u && __syncthreads_or(threadIdx.x == 0 && __ldcg(flag) != 0u)) return;
  bool lost = false, bad = false;
  if (static_cast<int>(blockIdx.x) < blocks_a) {
    const int panel = blockIdx.x / num_kb, kb = blockIdx.x % num_kb;
    // 16 threads hold a row's 64 values; eight rows per thread
    const int r0 = threadIdx.x >> 4, k4 = (threadIdx.x & 15) * 4;
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = load_a(q, panel * kRows + r0 + 16 * i, kb * kBK + k4);
    uint8_t* block = parts_of_a(q, panel, kb, num_kb);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const Scale sc = scale_of(max_of_16(magnitude(x[i])));
      uint2 hi, lo;
      lost |= split4(x[i], sc.mult, &hi, &lo);
      bad |= !sc.ok;
      store_a(block, r0 + 16 * i, k4, hi, lo);
      if (k4 == 0) q.scale_a[static_cast<size_t>(kb) * q.scale_lda + panel * kRows + r0 + 16 * i] = sc.inv;
    }
    if (!__syncthreads_or(lost || bad)) return;
    if (!__syncthreads_or(bad)) bad = far_parts_a(q, panel, kb);
  } else {
    __shared__ Columns columns;
    __shared__ uint32_t chunk_top[kThreads / 32][2];
    const int b = blockIdx.x - blocks_a;
    const int cols = b / num_kb, kb = b % num_kb;
    // a warp holds 128 columns of a value of K, four per lane; eight values of K per thread
    const int n = cols * 128 + lane * 4;
    const bool there = n < q.N;  // (N is a multiple of 64: a chunk of 64 columns is there or not)
    const float4 sample = load_b(q, sample_row(q, warp), n);
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = load_b(q, kb * kBK + warp + 8 * i, n);
    const float4 cm = column_powers(sample, warp, lane, &columns);
    uint32_t top = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[i] = make_float4(x[i].x * cm.x, x[i].y * cm.y, x[i].z * cm.z, x[i].w * cm.w);
      top = max(top, magnitude(x[i]));
    }
    const Scale sc = scale_of(over_chunk(top, warp, lane, chunk_top));
    bad = !sc.ok;
    if (there) {
      if (kb == 0 && warp == 0)
        *reinterpret_cast<float4*>(q.columns + n) = make_float4(1.f / cm.x, 1.f / cm.y, 1.f / cm.z, 1.f / cm.w);
      if (warp == 0 && (lane & 15) == 0) q.scale_b[static_cast<size_t>(kb) * q.scale_ldb + (n >> 6)] = sc.inv;
      uint8_t* block = parts_of_b(q, n, kb, num_kb);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint2 hi, lo;
        lost |= split4(x[i], sc.mult, &hi, &lo);
        store_b(block, warp + 8 * i, n, hi, lo);
      }
    }
    if (!__syncthreads_or(lost || bad)) return;
    if (!__syncthreads_or(bad)) bad = far_parts_b(q, cols, kb, lost);
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0 && atomicExch(flag, 1u) == 0u) atomicOr(q.words + kcg::H2_FOUND, kcg::H2_UNSPLIT);
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

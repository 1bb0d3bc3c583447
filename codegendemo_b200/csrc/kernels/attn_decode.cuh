// Fused attention for few query rows per head over a long list of keys (the step that appends one or a few tokens to a
// cache), fp16 / bf16, head dimension 64 or 128: up to 64 rows, and all calls of up to 32 (few_rows_form draws the line).
//
// What bounds it: K and V are read once, 2 * sk * d values per head, and every value meets at most 64 queries, so
// HBM does. The 256-row kernel gives a head ONE CTA, which is a serial walk over all keys with most tensor rows
// empty: 32 heads kept 32 of 148 SMs busy. Here a cluster of `splits` CTAs shares a head's keys, each CTA streams its
// range through a TMA ring (three 64-key stages of K and V at d = 128, 96 KB, two CTAs per SM: 190 KB of loads in
// flight per SM), and the partial results are joined in the cluster's shared memory: no workspace, no second launch.
//   warps 0-3  mma.sync m16n8k16 with 16 query rows each. kRowGroups = 1 (up to 16 rows): the four warps take 16 of a
//              stage's 64 keys each; 2 (up to 32): two groups of rows, 32 keys each; 4 (up to 64): all 64 keys.
//              (tcgen05 needs 128 rows: its P V chain would be the limit at one to 64 rows, mma.sync is far from one.)
//   warp 4     TMA producer
// Each warp keeps its own running maximum, sum and O rows; they meet at the end: key groups of the CTA through
// shared memory, then the CTAs of the cluster, each CTA summing one share of the output elements.
// Measured (B200, bf16, back to back from a graph), this form against the 256-row kernel: 32 heads x 1 x 8192 x 128
// 26 us = 5.2 TB/s (148 us), 128 x 1 x 8192 x 128 81 us = 6.6 TB/s, 8 x 1 x 16384 x 128 18.5 us, 32 x 32 x 8192 x 128
// 28 us. A launch costs about 4 us however short its walk.
// Waits are bounded as everywhere; the launch is ordered behind the kernel before it by griddep_wait.
#pragma once

struct AttnDecodeParams {
  CUtensorMap tmK, tmV;  // {d, rows, heads}, boxes of {64, 64, 1}, 128-byte swizzle
  const void* Q;         // heads x sq x d, contiguous
  void* O;
  int sq, sk, splits;
  float scale_log2;
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
template <bool kBf16>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  if constexpr (kBf16) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(cluster_addr)
               : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t cluster_addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(cluster_addr) : "memory");
  return v;
}

template <int kD, bool kBf16, int kRowGroups>
struct AttnDecode {
  static constexpr int BC = 64;                     // keys per stage
  static constexpr int STAGES = (kD == 128) ? 3 : 6;
  static constexpr int KEY_GROUPS = 4 / kRowGroups;
  static constexpr int WKEYS = BC / KEY_GROUPS;     // keys of a stage per warp
  static constexpr int ROWS = 16 * kRowGroups;
  static constexpr int NUM_THREADS = 160;
  static constexpr int BOX_BYTES = BC * 128;        // 64 keys x 64 values
  static constexpr int KV_BYTES = BC * kD * 2, STAGE_BYTES = 2 * KV_BYTES;
  static constexpr int RING_BYTES = STAGES * STAGE_BYTES;
  // after the walk the ring holds the warps' partial O rows, then the CTA's
  static constexpr int PART_BYTES = 4 * 16 * kD * 4, CTA_O = PART_BYTES;
  static_assert(PART_BYTES + ROWS * kD * 4 <= RING_BYTES, "the partial results must fit the ring");
  static constexpr int SMEM_BYTES = RING_BYTES + 3072;  // 1 KB alignment slack + barriers and row statistics
  using T = typename std::conditional<kBf16, __nv_bfloat16, __half>::type;

  struct Shared {
    uint64_t full[STAGES], empty[STAGES];
    volatile uint32_t abort_flag;
    uint32_t pad;
    float2 warp_ml[4][16];  // {maximum, sum} of a warp's rows
    float2 cta_ml[ROWS];    // of the CTA's rows
  };
  static_assert(sizeof(Shared) <= 2048, "barrier block exceeds its shared-memory slot");

  __device__ static __forceinline__ void report(Shared* sh, uint32_t code, uint32_t d0) {
    sh->abort_flag = 1u;
    if (atomicCAS(&g_attn_status[0], 0u, code) == 0u) {
      g_attn_status[1] = blockIdx.x;
      g_attn_status[2] = d0;
      g_attn_status[3] = 0u;
    }
  }

  // exp2(x - base) weight of a partial result whose maximum is x; a partial without a finite maximum weighs nothing
  __device__ static __forceinline__ float weight(float x, float base) { return x == -INFINITY ? 0.f : ex2(x - base); }

  __device__ static void run(const AttnDecodeParams& p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    Shared* sh = reinterpret_cast<Shared*>(smem + RING_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = static_cast<int>(cluster_cta_rank());
    const int head = static_cast<int>(blockIdx.x) / p.splits;
    const int tiles = (p.sk + BC - 1) / BC;
    // stages of this CTA: splits <= tiles, so every CTA has at least one
    const int t0 = static_cast<int>(static_cast<long long>(tiles) * rank / p.splits);
    const int t1 = static_cast<int>(static_cast<long long>(tiles) * (rank + 1) / p.splits);

    if (threadIdx.x == 0) {
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(&sh->full[s], 1);
        mbar_init(&sh->empty[s], 4);
      }
      sh->abort_flag = 0u;
      fence_mbar_init();
    }
    // K and V start towards L2 while the last CTAs of the kernel before this one end: the first ring of a long walk (32 heads x
    // 1 x 8192 x 128 27.0 -> 26.2 us), the first stage of a short one (64 x 4 x 1000 x 128 9.0 us; with the ring 9.4).
    if (threadIdx.x == 128) {
      for (int j = t0; j < t1 && j < t0 + (t1 - t0 >= 8 ? STAGES : 1); ++j)
#pragma unroll
        for (int b = 0; b < kD / 64; ++b) {
          tma_prefetch_3d(&p.tmK, b * 64, j * BC, head);
          tma_prefetch_3d(&p.tmV, b * 64, j * BC, head);
        }
    }
    __syncthreads();
    griddep_wait();

    const int q = lane >> 2, t = lane & 3;  // row and column pair of this lane in an accumulator tile
    const int rg = warp / KEY_GROUPS, kg = warp % KEY_GROUPS;
    float o[kD / 8][4];
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

    if (warp == 4) {
      if (lane == 0) {
        tma_prefetch_desc(&p.tmK);
        tma_prefetch_desc(&p.tmV);
        for (int j = t0; j < t1; ++j) {
          const int it = j - t0, s = it % STAGES;
          if (!mbar_wait(&sh->empty[s], ((it / STAGES) & 1u) ^ 1u, &sh->abort_flag)) {
            report(sh, ATTN_TIMEOUT_PRODUCER, j);
            break;
          }
          uint8_t* st = smem + s * STAGE_BYTES;
          mbar_expect_tx(&sh->full[s], STAGE_BYTES);
#pragma unroll
          for (int b = 0; b < kD / 64; ++b)
            tma_load_3d(st + b * BOX_BYTES, &p.tmK, &sh->full[s], b * 64, j * BC, head);
#pragma unroll
          for (int b = 0; b < kD / 64; ++b)
            tma_load_3d(st + KV_BYTES + b * BOX_BYTES, &p.tmV, &sh->full[s], b * 64, j * BC, head);
        }
        griddep_launch_dependents();
      }
      __syncwarp();
    } else {
      // query fragments: rows rg * 16 + {q, q + 8}, value pairs 2 t and 2 t + 8 of every 16
      uint32_t qf[kD / 16][4];
      {
        const T* Q = reinterpret_cast<const T*>(p.Q) + static_cast<size_t>(head) * p.sq * kD;
        const int r0 = rg * 16 + q, r1 = r0 + 8;
#pragma unroll
        for (int ks = 0; ks < kD / 16; ++ks)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r = (e & 1) ? r1 : r0;
            const int c = ks * 16 + 2 * t + (e >> 1) * 8;
            qf[ks][e] = r < p.sq ? *reinterpret_cast<const uint32_t*>(Q + static_cast<size_t>(r) * kD + c) : 0u;
          }
      }
#pragma unroll
      for (int n = 0; n < kD / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
      const int mat = lane >> 3, mrow = lane & 7;
      for (int j = t0; j < t1; ++j) {
        const int it = j - t0, s = it % STAGES;
        const bool got = mbar_wait(&sh->full[s], (it / STAGES) & 1u, &sh->abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) report(sh, ATTN_TIMEOUT_SOFTMAX, j);
          break;
        }
        const uint32_t kaddr = smem_u32(smem + s * STAGE_BYTES), vaddr = kaddr + KV_BYTES;
        // two accumulators per 8 keys (even and odd 16 values of d): twice as many independent chains
        float c[WKEYS / 8][4], c2[WKEYS / 8][4];
#pragma unroll
        for (int n = 0; n < WKEYS / 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) c[n][e] = c2[n][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < kD / 32; ++ks) {  // 32 values of d per load: two K steps
          const int unit = ks * 4 + mat;
#pragma unroll
          for (int n = 0; n < WKEYS / 8; ++n) {
            const int key = kg * WKEYS + n * 8 + mrow;
            uint32_t b[4];
            ldmatrix_x4(b, kaddr + key * 128 + (unit >> 3) * BOX_BYTES + (((unit & 7) ^ (key & 7)) << 4));
            mma_16816<kBf16>(c[n], qf[2 * ks][0], qf[2 * ks][1], qf[2 * ks][2], qf[2 * ks][3], b[0], b[1]);
            mma_16816<kBf16>(c2[n], qf[2 * ks + 1][0], qf[2 * ks + 1][1], qf[2 * ks + 1][2], qf[2 * ks + 1][3], b[2],
                             b[3]);
          }
        }
#pragma unroll
        for (int n = 0; n < WKEYS / 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) c[n][e] += c2[n][e];
        const int valid = p.sk - j * BC - kg * WKEYS;  // keys of this warp that exist
        if (valid < WKEYS) {
#pragma unroll
          for (int n = 0; n < WKEYS / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n * 8 + 2 * t + (e & 1) >= valid) c[n][e] = -INFINITY;
        }
        float base[2], alpha[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float mx = -INFINITY;
#pragma unroll
          for (int n = 0; n < WKEYS / 8; ++n) mx = fmaxf(mx, fmaxf(c[n][2 * h], c[n][2 * h + 1]));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
          mx = fmaxf(m[h], mx * p.scale_log2);  // (the scale is positive: checked by the host)
          base[h] = mx == -INFINITY ? 0.f : mx;
          alpha[h] = ex2(m[h] - base[h]);
          m[h] = mx;
        }
        if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
          for (int n = 0; n < kD / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[n][e] *= alpha[e >> 1];
        }
        float sum[2] = {0.f, 0.f};
#pragma unroll
        for (int n = 0; n < WKEYS / 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            c[n][e] = ex2(fmaf(c[n][e], p.scale_log2, -base[e >> 1]));
            sum[e >> 1] += c[n][e];
          }
        l[0] = l[0] * alpha[0] + sum[0];
        l[1] = l[1] * alpha[1] + sum[1];
#pragma unroll
        for (int ks = 0; ks < WKEYS / 16; ++ks) {
          const uint32_t a0 = pack_pair<kBf16>(c[2 * ks][0], c[2 * ks][1]);
          const uint32_t a1 = pack_pair<kBf16>(c[2 * ks][2], c[2 * ks][3]);
          const uint32_t a2 = pack_pair<kBf16>(c[2 * ks + 1][0], c[2 * ks + 1][1]);
          const uint32_t a3 = pack_pair<kBf16>(c[2 * ks + 1][2], c[2 * ks + 1][3]);
          const int key = kg * WKEYS + ks * 16 + (mat & 1) * 8 + mrow;
          const uint32_t vrow = vaddr + key * 128;
#pragma unroll
          for (int n = 0; n < kD / 8; n += 2) {
            const int unit = n + (mat >> 1);
            uint32_t b[4];
            ldmatrix_x4_trans(b, vrow + (unit >> 3) * BOX_BYTES + (((unit & 7) ^ (key & 7)) << 4));
            mma_16816<kBf16>(o[n], a0, a1, a2, a3, b[0], b[1]);
            mma_16816<kBf16>(o[n + 1], a0, a1, a2, a3, b[2], b[3]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->empty[s]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
      }
    }
    if (sh->abort_flag != 0u) {  // loads still in flight land before the ring is written over
      const uint64_t w0 = global_timer_ns();
      while (global_timer_ns() - w0 < 200000ull) __nanosleep(1000);
    }
    __syncthreads();
    float* part = reinterpret_cast<float*>(smem);
    if (warp < 4) {
      float* mine = part + warp * 16 * kD;
#pragma unroll
      for (int n = 0; n < kD / 8; ++n) {
        *reinterpret_cast<float2*>(mine + q * kD + n * 8 + 2 * t) = make_float2(o[n][0], o[n][1]);
        *reinterpret_cast<float2*>(mine + (q + 8) * kD + n * 8 + 2 * t) = make_float2(o[n][2], o[n][3]);
      }
      if (t == 0) {
        sh->warp_ml[warp][q] = make_float2(m[0], l[0]);
        sh->warp_ml[warp][q + 8] = make_float2(m[1], l[1]);
      }
    }
    __syncthreads();
    // the CTA's partial result: key groups joined per row
    float* cta_o = reinterpret_cast<float*>(smem + CTA_O);
    for (int i = threadIdx.x; i < ROWS * kD / 4; i += NUM_THREADS) {
      const int row = i / (kD / 4), c4 = i % (kD / 4), g = row / 16, r = row % 16;
      float base = -INFINITY;
#pragma unroll
      for (int k = 0; k < KEY_GROUPS; ++k) base = fmaxf(base, sh->warp_ml[g * KEY_GROUPS + k][r].x);
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      float sum = 0.f;
#pragma unroll
      for (int k = 0; k < KEY_GROUPS; ++k) {
        const int w = g * KEY_GROUPS + k;
        const float2 ml = sh->warp_ml[w][r];
        const float f = weight(ml.x, base);
        const float4 x = reinterpret_cast<const float4*>(part + (w * 16 + r) * kD)[c4];
        a.x = fmaf(f, x.x, a.x);
        a.y = fmaf(f, x.y, a.y);
        a.z = fmaf(f, x.z, a.z);
        a.w = fmaf(f, x.w, a.w);
        sum = fmaf(f, ml.y, sum);
      }
      reinterpret_cast<float4*>(cta_o)[i] = a;
      if (c4 == 0) sh->cta_ml[row] = make_float2(base, sum);
    }
    __syncwarp();
    cluster_sync_all();
    // this CTA's share of the output elements, joined over the cluster
    const int units = p.sq * (kD / 4);
    const int u0 = static_cast<int>(static_cast<long long>(units) * rank / p.splits);
    const int u1 = static_cast<int>(static_cast<long long>(units) * (rank + 1) / p.splits);
    const uint32_t o_addr = smem_u32(cta_o), ml_addr = smem_u32(&sh->cta_ml[0]);
    T* out = reinterpret_cast<T*>(p.O) + static_cast<size_t>(head) * p.sq * kD;
    for (int i = u0 + threadIdx.x; i < u1; i += NUM_THREADS) {
      const int row = i / (kD / 4);
      float base = -INFINITY;
      for (int k = 0; k < p.splits; ++k) base = fmaxf(base, ld_cluster_f2(map_to_cta(ml_addr + row * 8, k)).x);
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      float sum = 0.f;
#pragma unroll 4
      for (int k = 0; k < p.splits; ++k) {
        const float2 ml = ld_cluster_f2(map_to_cta(ml_addr + row * 8, k));
        const float4 x = ld_cluster_f4(map_to_cta(o_addr + i * 16, k));
        const float f = weight(ml.x, base);
        a.x = fmaf(f, x.x, a.x);
        a.y = fmaf(f, x.y, a.y);
        a.z = fmaf(f, x.z, a.z);
        a.w = fmaf(f, x.w, a.w);
        sum = fmaf(f, ml.y, sum);
      }
      const float inv = 1.f / sum;
      *reinterpret_cast<uint2*>(out + 4 * static_cast<size_t>(i)) =
          make_uint2(pack_pair<kBf16>(a.x * inv, a.y * inv), pack_pair<kBf16>(a.z * inv, a.w * inv));
    }
    __syncwarp();
    cluster_sync_all();  // the other CTAs read this one's shared memory until here
  }
};

template <int kD, bool kBf16, int kRowGroups>
__global__ void __launch_bounds__(160, 2) kcg_attention_decode_kernel(const __grid_constant__ AttnDecodeParams p) {
  AttnDecode<kD, kBf16, kRowGroups>::run(p);
}

// FlatQuant quantizer for sm_100a, right transform of size 144 .. 256 (features = M x N, M and N multiples of 16,
// 16 <= M <= 128): 28672 = 128 x 224, 32768 = 128 x 256, 24576 = 128 x 192, 20480 = 128 x 160, 18432 = 128 x 144.
//
// One persistent CTA per SM, one token at a time.  Both products are computed TRANSPOSED, because neither the rounded
// Y nor a second copy of X would fit in shared memory beside a 256 x 256 R (128 KB) and X (64 KB):
//
//   Y^T = R^T . X^T   A = R as it lies in memory (M-major), two tiles of 128 rows (the N dimension of the token),
//                     B = X rows as the TMA brings them (K-major), N = M columns, K = N
//   Z^T = Y^T . L     A = Y^T, rounded to the activation dtype, from TENSOR MEMORY: it overwrites the first half of its
//                     own float32 accumulators; B = L as it lies in memory (N-major); K = M
//
//   warp 0        TMA: 3-D tensor map (n, m, token), boxes of 64 x M, 128-byte swizzle; ONE X stage: it is free again
//                 as soon as the first product is done, so the next token's load runs under the rest of this token
//   warps 1, 2    issue the two products, tile by tile, so that the Y pass of tile 0 runs under the first product of
//                 tile 1 and the second product of tile 0 under the Y pass of tile 1; two issuers keep each other's
//                 barrier latencies off the tensor core
//   warps 4-11    Y pass: warp (tile, q) rounds lanes 32q .. 32q+31 of its tile, in place
//   warps 12-27   quantize pass: warp (tile, h, q) takes columns (rows of the token's matrix) 64h .. 64h+63 of lanes
//                 32q .. 32q+31; absmax through shared memory, scale, codes.  A lane holds one column of the token's
//                 matrix, so the eight codes of a packed word lie in eight lanes: an 8 x 8 transposition of nibbles
//                 (three shuffles) turns them round.
//
// Bound: HBM (57,344 bytes in and 14,340 out per token of 28672; 11 us for 1001 tokens).  Measured in graph replay: 29.7 us
// for 1001 bf16 tokens to packed codes, 2.4 TB/s, 112.7 us for 4000 (35.1 and 124.7 with one issuing warp and without the
// register shares); the SIMT kernel, before the only one for such widths, takes 3600 us for the former.  A token is a
// chain of load, first product, Y pass and second product; its X boxes given back one by one were measured slower (38 to
// 41 us: more barrier polls and commits in the issuing thread).
//
// Numerics are those of flatquant_sm100_n128.cu (same packed arithmetic, same rounding points; reference:
// src/quant_ops/ops/quantization/flatquant/ops.py:99-117).  Tokens with an infinity or a NaN among their transformed
// values, and tokens whose scale is zero (fp16), infinite (fp16 with a clip ratio above 1) or 2^100 and more (bf16: the
// second term of 1/s would be subnormal), take the scalar route of the SIMT kernel, code by code.
// Every mbarrier wait is bounded.
#include "flatquant_sm100_common.cuh"

namespace qo {
namespace {

using namespace ptx;
using namespace fq;

constexpr int kThreads = 896;  // 28 warps: TMA, two MMA issuers, one idle, 8 (Y pass) + 16 (quantize pass)
constexpr int kYWarp0 = 4, kQWarp0 = 12;
// Registers per thread (by warpgroup, hence the idle warp): the block is launched with 896 x 72.  With 224 KB of shared
// memory in use hardly any L1 is left, so a register spilled in the quantize pass is read back from L2.
constexpr int kRegsQuant = 88, kRegsRest = 48;
static_assert(512 * kRegsQuant + 384 * kRegsRest <= kThreads * 72, "the shares must fit the launch's registers");
constexpr int kMaxM = 128, kMaxN = 256;
constexpr int kOffX = 0;                              // four 64-column atoms of M rows
constexpr int kOffL = kOffX + 4 * kAtomBytes;         // two 64-column blocks of M rows
constexpr int kOffR = kOffL + 2 * kAtomBytes;         // four 64-column blocks of N rows
constexpr int kOffMisc = kOffR + 4 * kMaxN * 128;
constexpr int kSmemBytes = kOffMisc + 256 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");
constexpr int kTmemCols = 512;                        // first product: 2 tiles x 128 columns; second product: the same
constexpr int kColZ = 256;

struct Misc {
  uint64_t full_x, empty_x;
  uint64_t d1_full[2], y_ready[2], y_free[2], d2_full[2], d2_empty[2], set_sync;
  uint32_t tmem_base;
  uint32_t absmax_bits[3];  // bits of the token's largest |z|; a NaN among them is larger than any number
  uint32_t finite_bits[3];  // the same without the NaNs, plus one (0: every value is a NaN)
};
static_assert(sizeof(Misc) <= 256, "misc area");

// NaN-propagating |max| of packed pairs (the sign is ignored by the caller)
template <typename T> __device__ __forceinline__ uint32_t absmax_nan(uint32_t a, uint32_t b);
template <> __device__ __forceinline__ uint32_t absmax_nan<__nv_bfloat16>(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
template <> __device__ __forceinline__ uint32_t absmax_nan<__half>(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.NaN.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// Transposition inside groups of 8 lanes: lane i's nibble j becomes lane j's nibble i.
struct NibbleTurn {
  uint32_t sel4, sel2, mask1, shr1, shl1;
  __device__ __forceinline__ explicit NibbleTurn(int lane) {
    sel4 = (lane & 4) ? 0x3276u : 0x5410u;  // halves
    sel2 = (lane & 2) ? 0x3715u : 0x6240u;  // bytes
    mask1 = (lane & 1) ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
    shr1 = (lane & 1) ? 4u : 0u;
    shl1 = (lane & 1) ? 0u : 4u;
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 4), sel4);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 2), sel2);
    const uint32_t r = __shfl_xor_sync(0xffffffffu, x, 1);
    return (x & mask1) | (((r >> shr1) << shl1) & ~mask1);
  }
};
// The same for the four bytes of groups of 4 lanes.
struct ByteTurn {
  uint32_t sel2, sel1;
  __device__ __forceinline__ explicit ByteTurn(int lane) {
    sel2 = (lane & 2) ? 0x3276u : 0x5410u;
    sel1 = (lane & 1) ? 0x3715u : 0x6240u;
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 2), sel2);
    return __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 1), sel1);
  }
};

// eight codes (offset binary, a nibble each) one by one: any z and s
template <typename T>
__device__ __noinline__ uint32_t careful_word(uint32_t z0, uint32_t z1, uint32_t z2, uint32_t z3, float s) {
  const uint32_t zz[4] = {z0, z1, z2, z3};
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float z = (i & 1) ? P2<T>::hi(zz[i >> 1]) : P2<T>::lo(zz[i >> 1]);
    w |= (uint32_t)(quantize_one<T>(z, s) + 8) << (4 * i);
  }
  return w;
}

template <typename T, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
flatquant_n256_kernel(const __grid_constant__ CUtensorMap x_map, const T* __restrict__ left, const T* __restrict__ right,
                      void* __restrict__ out, void* __restrict__ scales, long long tokens, int m, int n, float clip,
                      int scale_dtype, uint32_t* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Misc* misc = reinterpret_cast<Misc*>(smem + kOffMisc);
  const uint32_t smem_base = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int feat = m * n;
  const int quads1 = (n - 128 + 31) >> 5;  // lane quadrants of tile 1 with real rows (tile 0 has four)
  const int halves = m > 64 ? 2 : 1;
  int mine = 0;  // tokens of this CTA
  if ((long long)blockIdx.x < tokens) mine = (int)((tokens - blockIdx.x + gridDim.x - 1) / gridDim.x);

  if (tid == 0) {
    mbar_init(smem_u32(&misc->full_x), 1);
    mbar_init(smem_u32(&misc->empty_x), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&misc->d1_full[i]), 1);
      mbar_init(smem_u32(&misc->y_ready[i]), i == 0 ? 4 : quads1);  // one arrival per working warp
      mbar_init(smem_u32(&misc->y_free[i]), 1);
      mbar_init(smem_u32(&misc->d2_full[i]), 1);
      mbar_init(smem_u32(&misc->d2_empty[i]), halves * (i == 0 ? 4 : quads1));
    }
    mbar_init(smem_u32(&misc->set_sync), halves * (4 + quads1));
    for (int i = 0; i < 3; ++i) misc->absmax_bits[i] = misc->finite_bits[i] = 0u;
    fence_barrier_init();
    prefetch_tensormap(&x_map);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&misc->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc->tmem_base;
  grid_dependency_wait();    // nothing below touches global memory before the kernel ahead in the stream has completed
  grid_launch_dependents();  // (after the wait: see flatquant_sm100_n128.cu)

  if (warp != 0) {
    // Both transforms as they lie in memory, 16 bytes at a time with the 128-byte XOR swizzle.  R: rows k < n in four
    // 64-column blocks, columns past n zero; L: rows k < m in two blocks, columns past m zero (never read: N = m).
    constexpr int kStagers = kThreads - 32;
    const int t1 = tid - 32;
    constexpr int kPer = 6;  // pieces requested by a thread before it stores them: the loads' latencies overlap
    for (int base = t1; base < n * 32; base += kStagers * kPer) {
      uint4 w[kPer];
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int idx = base + j * kStagers, k = idx >> 5, c = idx & 31;
        w[j] = make_uint4(0, 0, 0, 0);
        if (idx < n * 32 && 8 * c < n) w[j] = *reinterpret_cast<const uint4*>(right + k * n + 8 * c);
      }
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int idx = base + j * kStagers, k = idx >> 5, c = idx & 31;
        if (idx < n * 32) *reinterpret_cast<uint4*>(smem + kOffR + (c >> 3) * (n * 128) + k * 128 + (((c & 7) ^ (k & 7)) << 4)) = w[j];
      }
    }
    for (int idx = t1; idx < m * 16; idx += kStagers) {
      const int k = idx >> 4, c = idx & 15;
      uint4 w = make_uint4(0, 0, 0, 0);
      if (8 * c < m) w = *reinterpret_cast<const uint4*>(left + k * m + 8 * c);
      *reinterpret_cast<uint4*>(smem + kOffL + (c >> 3) * kAtomBytes + k * 128 + (((c & 7) ^ (k & 7)) << 4)) = w;
    }
    fence_proxy_async_smem();
    asm volatile("bar.sync 1, %0;" ::"n"(kStagers) : "memory");
  }

  if (warp >= kQWarp0) {
    regs_inc<kRegsQuant>();
    // ---- quantize pass -----------------------------------------------------------------------------------------------
    const int q = warp & 3, idx = (warp - kQWarp0) >> 2, tl = idx >> 1, h = idx & 1;
    const int n0 = tl * 128 + q * 32, r0 = h * 64;   // first column / first row of the token's matrix in this warp
    const int rows = min(64, m - r0);                // rows of this warp (a multiple of 16)
    const bool valid = n0 + lane < n;
    const bool first = tl == 0 && h == 0 && q == 0;
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + kColZ + tl * 128 + r0;
    const uint32_t gs = smem_u32(&misc->set_sync);
    int meets = 0;
    long long tok = blockIdx.x;
    for (int it = 0; it < (n0 < n && rows > 0 ? mine : 0); ++it, tok += gridDim.x) {
      const int buf = it % 3;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&misc->d2_full[tl]), it & 1))) { atomicCAS(status, 0u, 0xC60u + tl); break; }
      tc_fence_after();
      uint32_t zz[32];  // 64 rounded values as packed pairs; rows past the last one are zero
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        if (ch * 16 < rows) {
          uint32_t v[16];
          tmem_ld_32x32b_x16(taddr + ch * 16, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) zz[8 * ch + i] = P2<T>::cvt(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) zz[8 * ch + i] = 0u;
        }
      }
      tc_fence_before();
      mbar_arrive_warp(smem_u32(&misc->d2_empty[tl]));  // the accumulators are free again

      if (MODE == kTransform) {
        float* dst = reinterpret_cast<float*>(out) + tok * feat + (int64_t)r0 * n + n0 + lane;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (valid && 2 * i < rows) {
            dst[(2 * i) * n] = P2<T>::lo(zz[i]);
            dst[(2 * i + 1) * n] = P2<T>::hi(zz[i]);
          }
        }
        continue;
      }

      uint32_t m0 = zz[0], m1 = zz[1], m2 = zz[2], m3 = zz[3];  // four chains keep the dependent latency short
#pragma unroll
      for (int i = 4; i < 32; i += 4) {
        m0 = absmax_nan<T>(m0, zz[i]);
        m1 = absmax_nan<T>(m1, zz[i + 1]);
        m2 = absmax_nan<T>(m2, zz[i + 2]);
        m3 = absmax_nan<T>(m3, zz[i + 3]);
      }
      m0 = absmax_nan<T>(absmax_nan<T>(m0, m1), absmax_nan<T>(m2, m3));
      // bits of non-negative floats order as integers, and those of a NaN are above those of an infinity
      const uint32_t row_bits = valid ? max(__float_as_uint(fabsf(P2<T>::lo(m0))), __float_as_uint(fabsf(P2<T>::hi(m0)))) : 0u;
      const uint32_t warp_bits = __reduce_max_sync(0xffffffffu, row_bits);
      if (lane == 0) atomicMax(&misc->absmax_bits[buf], warp_bits);
      mbar_arrive_warp(gs);
      if (!__all_sync(0xffffffffu, mbar_wait(gs, meets & 1))) { atomicCAS(status, 0u, 0xC70u); break; }
      ++meets;
      const uint32_t token_bits = misc->absmax_bits[buf];
      if (first && lane == 0) misc->absmax_bits[(it + 2) % 3] = misc->finite_bits[(it + 2) % 3] = 0u;
      float amax = __uint_as_float(token_bits);
      const bool special = token_bits >= 0x7F800000u;  // the same for every warp of the token
      if (special) {
        // an infinity or a NaN in this token: the SIMT kernel's extremes skip NaNs (and start from +-3.4e38)
        float a = -1.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) a = fmaxf(a, fmaxf(fabsf(P2<T>::lo(zz[i])), fabsf(P2<T>::hi(zz[i]))));
        // (fmaxf skips a NaN; pairs of NaNs leave a at -1; rows past the last one are zeros and must not count)
        if (rows < 64) {
          a = -1.f;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (2 * i < rows) a = fmaxf(a, fmaxf(fabsf(P2<T>::lo(zz[i])), fabsf(P2<T>::hi(zz[i]))));
        }
        const uint32_t fb = __reduce_max_sync(0xffffffffu, valid && a >= 0.f ? __float_as_uint(a) + 1u : 0u);
        if (lane == 0) atomicMax(&misc->finite_bits[buf], fb);
        mbar_arrive_warp(gs);
        if (!__all_sync(0xffffffffu, mbar_wait(gs, meets & 1))) { atomicCAS(status, 0u, 0xC71u); break; }
        ++meets;
        const uint32_t tb = misc->finite_bits[buf];
        amax = tb == 0u ? 3.4e38f : __uint_as_float(tb - 1u);
      }
      const float top = rnd1<T>(amax * clip);
      const float s = fmaxf(rnd1<T>(top * 0.142857149f), DT<T>::floor_scale());  // = round(top / 7), see flatquant_sm100_n128.cu
      const float inv_s = __frcp_rn(s);
      uint32_t rhi2, rlo2;
      P2<T>::recip2(inv_s, rhi2, rlo2);
      if (first && lane == 0) store_scale(scales, tok, s, scale_dtype);
      const bool careful = special || s == 0.f || !(s < 0x1p100f);
      // a quotient can only leave [-8, 7] after rounding if some |z| / s reaches 7.5
      const bool clamp_needed = !(__uint_as_float(warp_bits) * inv_s < 7.4f);

      if (MODE == kPacked) {
        const NibbleTurn turn(lane);
        uint32_t* dst = reinterpret_cast<uint32_t*>(out) + tok * (feat / 8) + (int64_t)(r0 + (lane & 7)) * (n / 8) + n0 / 8 + (lane >> 3);
        const bool store = n0 + 8 * (lane >> 3) < n;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (8 * j >= rows) break;
          uint32_t w;
          if (careful) w = careful_word<T>(zz[4 * j], zz[4 * j + 1], zz[4 * j + 2], zz[4 * j + 3], s);
          else if (clamp_needed) w = quantize8<T, true>(&zz[4 * j], s, inv_s, rhi2, rlo2);
          else w = quantize8<T, false>(&zz[4 * j], s, inv_s, rhi2, rlo2);
          w = turn(w);
          if (store) dst[(8 * j) * (n / 8)] = w;
        }
      } else {
        const ByteTurn turn(lane);
        uint8_t* dst = reinterpret_cast<uint8_t*>(out) + tok * feat + (int64_t)(r0 + (lane & 3)) * n + n0 + 4 * (lane >> 2);
        const bool store = n0 + 4 * (lane >> 2) < n;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (8 * j >= rows) break;
          uint32_t pb, qb;
          if (careful) {
            const uint32_t w = careful_word<T>(zz[4 * j], zz[4 * j + 1], zz[4 * j + 2], zz[4 * j + 3], s);
            const uint32_t even = w & 0x0F0F0F0Fu, odd = (w >> 4) & 0x0F0F0F0Fu;
            pb = __byte_perm(even, odd, 0x5140);
            qb = __byte_perm(even, odd, 0x7362);
          } else {
            nibble_bytes_packed<T>(&zz[4 * j], s, inv_s, rhi2, rlo2, pb, qb);
          }
          pb = turn(bytes4(pb));
          qb = turn(bytes4(qb));
          if (store) {
            *reinterpret_cast<uint32_t*>(dst + (8 * j) * n) = pb;
            *reinterpret_cast<uint32_t*>(dst + (8 * j + 4) * n) = qb;
          }
        }
      }
    }
  } else {
  regs_dec<kRegsRest>();
  if (warp == 0) {
    if (lane == 0) {
      const int boxes = (n + 63) >> 6;
      long long tok = blockIdx.x;
      for (int it = 0; it < mine; ++it, tok += gridDim.x) {
        if (!mbar_wait(smem_u32(&misc->empty_x), (it & 1) ^ 1)) { atomicCAS(status, 0u, 0xC00u); break; }
        const uint32_t bar = smem_u32(&misc->full_x);
        mbar_arrive_expect_tx(bar, (uint32_t)(boxes * m * 128));
        for (int b = 0; b < boxes; ++b) tma_load_3d(smem_base + kOffX + b * kAtomBytes, &x_map, bar, b * 64, 0, (int)tok);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc1 = umma_idesc(1, Fmt<T>::id, Fmt<T>::id, 1, 0, 128, m);  // A = R^T: M-major, B = X rows: K-major
      const uint64_t desc_x = umma_smem_desc_sw128(smem_base + kOffX, 16, 1024);
      const int ks1 = n >> 4;
      bool ok = true;
      for (int it = 0; ok && it < mine; ++it) {
        const int ph = it & 1;
        for (int tl = 0; tl < 2; ++tl) {
          if (const int w = tl == 0 ? mbar_wait2(smem_u32(&misc->full_x), ph, smem_u32(&misc->y_free[0]), ph ^ 1)
                                    : (mbar_wait(smem_u32(&misc->y_free[1]), ph ^ 1) ? 0 : 3)) {
            atomicCAS(status, 0u, 0xC10u + w);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t desc_r = umma_smem_desc_sw128(smem_base + kOffR + tl * 2 * (n * 128), (uint32_t)(n * 128), 1024);
#pragma unroll 2
          for (int ks = 0; ks < ks1; ++ks)  // 16 rows of R = 2048 bytes per step; X: 32 bytes inside a 64-column atom
            mma_f16_ss(tmem + tl * 128, desc_r + (uint64_t)(ks * 128), desc_x + (uint64_t)((ks >> 2) * (kAtomBytes >> 4) + (ks & 3) * 2), idesc1, ks);
          mma_commit(smem_u32(&misc->d1_full[tl]));
        }
        if (ok) mma_commit(smem_u32(&misc->empty_x));
      }
    }
  } else if (warp == 2) {
    if (lane == 0) {
      const uint32_t idesc2 = umma_idesc(1, Fmt<T>::id, Fmt<T>::id, 0, 1, 128, m);  // A = Y^T in tensor memory, B = L: N-major
      const uint64_t desc_l = umma_smem_desc_sw128(smem_base + kOffL, kAtomBytes, 1024);
      const int ks2 = m >> 4;
      bool ok = true;
      for (int it = 0; ok && it < mine; ++it) {
        const int ph = it & 1;
        for (int tl = 0; tl < 2; ++tl) {
          if (const int w = mbar_wait2(smem_u32(&misc->y_ready[tl]), ph, smem_u32(&misc->d2_empty[tl]), ph ^ 1)) {
            atomicCAS(status, 0u, 0xC20u + 0x10u * w + tl);
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll 2
          for (int ks = 0; ks < ks2; ++ks)  // 16 values of Y^T = 8 tensor-memory columns per step
            mma_f16_ts(tmem + kColZ + tl * 128, tmem + tl * 128 + ks * 8, desc_l + (uint64_t)(ks * 128), idesc2, ks);
          mma_commit(smem_u32(&misc->y_free[tl]));
          mma_commit(smem_u32(&misc->d2_full[tl]));
        }
      }
    }
  } else if (warp >= kYWarp0) {
    // ---- Y pass: 32 lanes of one tile; every 32 float32 columns become 16 packed ones, written below what is still to read
    const int q = warp & 3, tl = (warp - kYWarp0) >> 2;
    const uint32_t base = tmem + ((uint32_t)(q * 32) << 16) + tl * 128;
    const bool works = tl * 128 + q * 32 < n;
    for (int it = 0; it < (works ? mine : 0); ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&misc->d1_full[tl]), it & 1))) { atomicCAS(status, 0u, 0xC50u + tl); break; }
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < m; c += 32) {
        uint32_t v[32], a[8], b[8];
        tmem_ld_32x32b_x32(base + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          a[i] = pack2<T>(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
          b[i] = pack2<T>(__uint_as_float(v[16 + 2 * i]), __uint_as_float(v[16 + 2 * i + 1]));
        }
        tmem_st_32x32b_x8(base + (c >> 1), a);
        if (c + 16 < m) tmem_st_32x32b_x8(base + (c >> 1) + 8, b);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive_warp(smem_u32(&misc->y_ready[tl]));
    }
  }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

template <typename T, int MODE>
int launch_one(const CUtensorMap& map, const void* left, const void* right, void* out, void* scales, int64_t tokens, int m,
               int n, float clip, int scale_dtype, uint32_t* status, cudaStream_t stream) {
  auto kern = flatquant_n256_kernel<T, MODE>;
  int dev = 0;
  QO_CUDA_TRY(cudaGetDevice(&dev));
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    QO_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    configured[dev & 63] = true;
  }
  const int sms = sm_count(dev);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tokens < sms ? tokens : sms));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  QO_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, map, reinterpret_cast<const T*>(left), reinterpret_cast<const T*>(right), out, scales,
                                 (long long)tokens, m, n, clip, scale_dtype, status));
  return check_launch("flatquant_n256_kernel");
}

template <typename T>
int launch_mode(int mode, const CUtensorMap& map, const void* left, const void* right, void* out, void* scales,
                int64_t tokens, int m, int n, float clip, int scale_dtype, uint32_t* status, cudaStream_t stream) {
  switch (mode) {
    case kInt8: return launch_one<T, kInt8>(map, left, right, out, scales, tokens, m, n, clip, scale_dtype, status, stream);
    case kPacked: return launch_one<T, kPacked>(map, left, right, out, scales, tokens, m, n, clip, scale_dtype, status, stream);
    default: return launch_one<T, kTransform>(map, left, right, out, scales, tokens, m, n, clip, scale_dtype, status, stream);
  }
}

}  // namespace

bool flatquant_sm100_n256_supported(int m, int n) { return n > 128 && n <= kMaxN && (n % 16) == 0 && m >= 16 && m <= kMaxM && (m % 16) == 0; }

int launch_flatquant_sm100_n256(int mode, const void* x_map, const void* left, const void* right, void* out, void* scales,
                                int64_t tokens, int m, int n, float clip, int in_dtype, int scale_dtype, uint32_t* status,
                                cudaStream_t stream) {
  const CUtensorMap& map = *reinterpret_cast<const CUtensorMap*>(x_map);
  if (in_dtype == QO_BF16)
    return launch_mode<__nv_bfloat16>(mode, map, left, right, out, scales, tokens, m, n, clip, scale_dtype, status, stream);
  return launch_mode<__half>(mode, map, left, right, out, scales, tokens, m, n, clip, scale_dtype, status, stream);
}

}  // namespace qo

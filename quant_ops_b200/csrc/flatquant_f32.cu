// FlatQuant quantizer for float32 activations: register-tiled SIMT kernel.
//
// float32 products stay on the FMA pipe: the tensor core has no float32 operands, and split 16-bit products would
// change the accumulation.  2 T F (M + N) operations against 5 T F bytes: at F = 4096 the FMA pipe needs 29 us for 2048
// tokens, HBM 6 us, so the kernel is built to keep the FMA pipe fed:
//
//   * a thread owns an 8 x 8 block of a token's M x N matrix through both products; per step of k it reads 8 + 8 values
//     from shared memory for 64 FMAs, all as 16-byte loads without bank conflicts (X and Y rows are padded by 16
//     bytes; a warp's threads are neighbours along N first);
//   * Y overwrites X in shared memory (every Y value is in registers when the last X value has been read), and Z never
//     leaves the registers: extremes, scale and codes come straight from the accumulators;
//   * R and L pass through shared memory in chunks of 16 rows, two buffers, cp.async: a CTA needs room for its
//     tokens' X only, so two CTAs of 256 threads share an SM and one computes while the other loads or quantizes;
//   * small matrices are batched, as many tokens per CTA as fill its threads (64 x 64: four) unless there are too few
//     tokens to give every SM two CTAs.
//
// Measured: 77.7 us for 2048 x 4096 to int8 codes in graph replay (the 29 us of multiply-adds are 37 % of that), 158 us for
// 700 x 14336; the shape-generic kernel takes 257 us for the former.  Bound by the issue slots: 71 % used while an SM is active,
// for 52 % of the FMA pipe (8192 x 4096; shared-memory reads 32 %).
//
// Every sum is one chain of fused multiply-adds in ascending k, as in flatquant_generic.cu: the results are the same
// bits (reference: src/quant_ops/ops/quantization/flatquant/ops.py:99-117).
#include "qo_internal.cuh"

namespace qo {
namespace {

constexpr int kChunk = 16;    // rows of R or L per stage
constexpr int kMaxGroup = 32; // tokens per CTA

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4_zfill(void* dst, const void* src, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(real ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// floats as unsigned integers of the same order
__device__ __forceinline__ uint32_t ordered(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k); }

// quantize_one<float> without a division for values that are not next to a rounding boundary: z * (1/s) is within
// 2^-21 of round(z / s) relative, which cannot move rint() unless the quotient is within 1e-5 of a half
// (values that large are clamped anyway).  NaNs and infinities fail the comparison and take the division.
__device__ __forceinline__ int quantize_f32(float z, float s, float inv_s, bool exact_all) {
  const float q = z * inv_s, r = rintf(q);
  if (exact_all || !(fabsf(fabsf(q - r) - 0.5f) > 1e-5f)) return quantize_one<float>(z, s);
  return (int)fminf(fmaxf(r, -8.f), 7.f);
}

// MODE 0: int8 codes, 1: packed codes, 2: transform only (float32 Z written to `codes`)
template <int MODE, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1)
flatquant_f32_kernel(const float* __restrict__ x, int64_t ldx, const float* __restrict__ left, const float* __restrict__ right,
                     void* __restrict__ codes, void* __restrict__ scales, int64_t tokens, int m, int n, int group, float clip,
                     int scale_dtype) {
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  __shared__ uint32_t ext[2][kMaxGroup];  // extremes of the CTA's tokens, as ordered integers
  const int tid = threadIdx.x;
  const int nb = n >> 3, mb = (m + 7) >> 3, m8 = mb * 8, ldy = n + 4;
  const int bpt = nb * mb;                // 8 x 8 blocks of a token = threads of a token
  const int cw = n > m8 ? n : m8;
  float* xs = smem;                       // [group][m][ldy]: X, then Y
  float* chunk = smem + (size_t)group * m * ldy;  // two buffers of kChunk rows
  const int g = tid / bpt, b = tid - g * bpt, ty = b / nb, tx = b - ty * nb;
  const bool worker = g < group;
  float* mine = xs + (size_t)(worker ? g : 0) * m * ldy;
  const int ca = 4 * tx, cb = (n >> 1) + 4 * tx;  // this thread's columns: ca .. ca + 3 and cb .. cb + 3
  const bool l_vec = (m & 7) == 0 && (reinterpret_cast<uintptr_t>(left) & 15) == 0;
  const int64_t feat = (int64_t)m * n;

  auto load_r = [&](int buf, int k0) {
    const int rows = min(kChunk, n - k0), pieces = rows * (n >> 2);
    const float* src = right + (int64_t)k0 * n;
    float* dst = chunk + buf * (kChunk * cw);
    for (int i = tid; i < pieces; i += THREADS) cp_async16(dst + 4 * i, src + 4 * i);
  };
  auto load_l = [&](int buf, int k0) {
    const int rows = min(kChunk, m - k0);
    const float* src = left + (int64_t)k0 * m;
    float* dst = chunk + buf * (kChunk * cw);
    if (l_vec) {
      const int pieces = rows * (m >> 2);
      for (int i = tid; i < pieces; i += THREADS) cp_async16(dst + 4 * i, src + 4 * i);
    } else {
      for (int i = tid; i < rows * m8; i += THREADS) {
        const int k = i / m8, r = i - k * m8;
        cp_async4_zfill(dst + i, src + (r < m ? k * m + r : 0), r < m);
      }
    }
  };

  const int64_t groups = (tokens + group - 1) / group;
  for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
    const int64_t t0 = grp * group;
    const int here = (int)min((int64_t)group, tokens - t0);
    // X: rows of n floats into rows of ldy
    {
      const int q = n >> 2, per = m * q;
      for (int i = tid; i < here * per; i += THREADS) {
        const int tk = i / per, e = i - tk * per, r = e / q, c = e - r * q;
        cp_async16(xs + ((size_t)tk * m + r) * ldy + 4 * c, x + (t0 + tk) * ldx + (int64_t)r * n + 4 * c);
      }
    }
    load_r(0, 0);
    cp_async_commit();
    if (tid < kMaxGroup) {
      ext[0][tid] = 0xFFFFFFFFu;
      ext[1][tid] = 0u;
    }
    const bool active = worker && g < here;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

    // Y = X . R: rows ty + mb i
    int buf = 0;
    for (int k0 = 0; k0 < n; k0 += kChunk, buf ^= 1) {
      cp_async_wait_all();
      __syncthreads();
      if (k0 + kChunk < n) load_r(buf ^ 1, k0 + kChunk);
      else load_l(buf ^ 1, 0);
      cp_async_commit();
      if (active) {
        const float* rc = chunk + buf * (kChunk * cw);
        const int kc = min(kChunk, n - k0);
#pragma unroll 1
        for (int k = 0; k < kc; k += 4) {
          float4 a[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(mine + min(ty + mb * i, m - 1) * ldy + k0 + k);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const float4 b0 = *reinterpret_cast<const float4*>(rc + (k + kk) * n + ca);
            const float4 b1 = *reinterpret_cast<const float4*>(rc + (k + kk) * n + cb);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float av = kk == 0 ? a[i].x : (kk == 1 ? a[i].y : (kk == 2 ? a[i].z : a[i].w));
              acc[i][0] = fmaf(av, b0.x, acc[i][0]);
              acc[i][1] = fmaf(av, b0.y, acc[i][1]);
              acc[i][2] = fmaf(av, b0.z, acc[i][2]);
              acc[i][3] = fmaf(av, b0.w, acc[i][3]);
              acc[i][4] = fmaf(av, b1.x, acc[i][4]);
              acc[i][5] = fmaf(av, b1.y, acc[i][5]);
              acc[i][6] = fmaf(av, b1.z, acc[i][6]);
              acc[i][7] = fmaf(av, b1.w, acc[i][7]);
            }
          }
        }
      }
    }
    __syncthreads();  // every X value has been read
    if (active) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = ty + mb * i;
        if (r < m) {
          *reinterpret_cast<float4*>(mine + r * ldy + ca) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
          *reinterpret_cast<float4*>(mine + r * ldy + cb) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

    // Z = L^T . Y: rows 4 ty .. 4 ty + 3 and m8 / 2 + the same
    const int ra = 4 * ty, rb = (m8 >> 1) + 4 * ty;
    for (int k0 = 0; k0 < m; k0 += kChunk, buf ^= 1) {
      cp_async_wait_all();
      __syncthreads();
      if (k0 + kChunk < m) {
        load_l(buf ^ 1, k0 + kChunk);
        cp_async_commit();
      }
      if (active) {
        const float* lc = chunk + buf * (kChunk * cw);
        const int kc = min(kChunk, m - k0);
#pragma unroll 2
        for (int k = 0; k < kc; ++k) {
          const float4 a0 = *reinterpret_cast<const float4*>(lc + k * m8 + ra), a1 = *reinterpret_cast<const float4*>(lc + k * m8 + rb);
          const float4 b0 = *reinterpret_cast<const float4*>(mine + (k0 + k) * ldy + ca), b1 = *reinterpret_cast<const float4*>(mine + (k0 + k) * ldy + cb);
          const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            acc[i][0] = fmaf(av[i], b0.x, acc[i][0]);
            acc[i][1] = fmaf(av[i], b0.y, acc[i][1]);
            acc[i][2] = fmaf(av[i], b0.z, acc[i][2]);
            acc[i][3] = fmaf(av[i], b0.w, acc[i][3]);
            acc[i][4] = fmaf(av[i], b1.x, acc[i][4]);
            acc[i][5] = fmaf(av[i], b1.y, acc[i][5]);
            acc[i][6] = fmaf(av[i], b1.z, acc[i][6]);
            acc[i][7] = fmaf(av[i], b1.w, acc[i][7]);
          }
        }
      }
    }

    const int64_t tok = t0 + g;
    if (MODE == 2) {
      if (active) {
        float* z = reinterpret_cast<float*>(codes) + tok * feat;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = (i < 4 ? ra : rb) + (i & 3);
          if (r < m) {
            *reinterpret_cast<float4*>(z + (int64_t)r * n + ca) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            *reinterpret_cast<float4*>(z + (int64_t)r * n + cb) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
          }
        }
      }
      __syncthreads();  // the next group overwrites Y
      continue;
    }
    if (active) {
      float lmin = 3.4e38f, lmax = -3.4e38f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if ((i < 4 ? ra : rb) + (i & 3) < m) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            lmin = fminf(lmin, acc[i][j]);
            lmax = fmaxf(lmax, acc[i][j]);
          }
        }
      }
      atomicMin(&ext[0][g], ordered(lmin));
      atomicMax(&ext[1][g], ordered(lmax));
    }
    __syncthreads();  // also: every Y value has been read, the next group may overwrite it
    if (active) {
      const float s = token_scale<float>(unordered(ext[0][g]), unordered(ext[1][g]), clip);
      const float inv_s = __frcp_rn(s);
      const bool exact_all = !(s < 1e37f);  // 1/s would be subnormal
      if (b == 0) store_scale(scales, tok, s, scale_dtype);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (i < 4 ? ra : rb) + (i & 3);
        if (r >= m) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int64_t at = tok * feat + (int64_t)r * n + (h ? cb : ca);
          int q[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) q[j] = quantize_f32(acc[i][4 * h + j], s, inv_s, exact_all);
          if (MODE == 1) {
            reinterpret_cast<uint16_t*>(codes)[at >> 2] =
                (uint16_t)((q[0] + 8) | ((q[1] + 8) << 4) | ((q[2] + 8) << 8) | ((q[3] + 8) << 12));
          } else {
            reinterpret_cast<char4*>(codes)[at >> 2] = make_char4((char)q[0], (char)q[1], (char)q[2], (char)q[3]);
          }
        }
      }
    }
    __syncthreads();  // the extremes are reset by the next group
  }
}

template <int MODE, int THREADS>
int launch_sized(const float* x, int64_t ldx, const float* left, const float* right, void* codes, void* scales, int64_t tokens,
                 int m, int n, float clip, int scale_dtype, cudaStream_t stream) {
  auto kern = flatquant_f32_kernel<MODE, THREADS>;
  constexpr int kSmem = THREADS == 256 ? 112 * 1024 : 200 * 1024;
  int dev = 0;
  QO_CUDA_TRY(cudaGetDevice(&dev));
  static bool configured[64] = {};
  if (!configured[dev & 63]) {
    QO_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    configured[dev & 63] = true;
  }
  const int sms = sm_count(dev), per_sm = THREADS == 256 ? 2 : 1;
  const int mb = (m + 7) / 8, bpt = mb * (n / 8), cw = n > mb * 8 ? n : mb * 8;
  const size_t token_bytes = (size_t)m * (n + 4) * 4, chunk_bytes = (size_t)2 * kChunk * cw * 4;
  // tokens per CTA: as many as fill its threads and fit, but no more than it takes to give every SM its CTAs
  int group = THREADS / bpt;
  if (group > kMaxGroup) group = kMaxGroup;
  while (group > 1 && group * token_bytes + chunk_bytes > (size_t)kSmem) --group;
  const int64_t spread = (tokens + (int64_t)sms * per_sm - 1) / ((int64_t)sms * per_sm);
  if (spread < group) group = (int)spread;
  const size_t smem = group * token_bytes + chunk_bytes;
  const int64_t groups = (tokens + group - 1) / group;
  const int grid = (int)(groups < (int64_t)sms * per_sm ? groups : (int64_t)sms * per_sm);
  kern<<<grid, THREADS, smem, stream>>>(x, ldx, left, right, codes, scales, tokens, m, n, group, clip, scale_dtype);
  return check_launch("flatquant_f32_kernel");
}

template <int THREADS>
int launch_mode(int mode, const float* x, int64_t ldx, const float* left, const float* right, void* codes, void* scales,
                int64_t tokens, int m, int n, float clip, int scale_dtype, cudaStream_t stream) {
  switch (mode) {
    case 0: return launch_sized<0, THREADS>(x, ldx, left, right, codes, scales, tokens, m, n, clip, scale_dtype, stream);
    case 1: return launch_sized<1, THREADS>(x, ldx, left, right, codes, scales, tokens, m, n, clip, scale_dtype, stream);
    default: return launch_sized<2, THREADS>(x, ldx, left, right, codes, scales, tokens, m, n, clip, scale_dtype, stream);
  }
}

}  // namespace

// rows of 16-byte pieces throughout, one thread per 8 x 8 block, and the token limit of flatquant_generic.cu (two
// buffers of M N floats in 200 KB), so that what that kernel refuses stays refused
bool flatquant_f32_supported(int64_t ldx, int m, int n, const void* x, const void* right, const void* codes) {
  return (n % 8) == 0 && (int64_t)m * n * 8 <= 200 * 1024 && ((m + 7) / 8) * (n / 8) <= 512 &&
         (size_t)m * (n + 4) * 4 + (size_t)2 * kChunk * (n > m + 7 ? n : m + 7) * 4 <= 200 * 1024 && (ldx % 4) == 0 &&
         reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(right) % 16 == 0 &&
         reinterpret_cast<uintptr_t>(codes) % 16 == 0;
}

// Small matrices of few tokens are left to the generic kernel (the same bits).  Its threads compute 8 values at a time, those
// of this kernel 64: as long as a token has no more than 256 such groups of 8 and the SM's threads are not used up, the
// shorter chains are done first.  The lines follow measurements of both kernels over the tokens an SM has at once and the
// threads they occupy (graph replay, generic / this kernel, us): 32 x 32 packed 8.7 / 12.0 for 148 tokens and 12.3 / 12.4
// for 592; 32 x 64 packed 11.6 / 14.7 for 148, 15.0 / 15.0 for 296; 64 x 32 packed 14.2 / 14.5 for 148, 17.1 / 14.4 for
// 149; 148 tokens to int8: 24 x 24 10.2 / 10.9, 32 x 32 12.2 / 11.9.  The generic kernel stores int8 codes byte by byte, and a
// tall matrix costs it more (L is read from memory, eight values a step): hence the limits by mode and M.
bool flatquant_f32_preferred(int mode, int64_t tokens, int m, int n) {
  const int groups = ((m + 7) / 8) * n;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return true; }
  const int64_t per_sm = (tokens + sm_count(dev) - 1) / sm_count(dev);
  if (groups > 256 || per_sm > 4) return true;  // more than a group per thread; more tokens than the generic kernel takes at once
  int most = 0;  // threads of an SM with work up to which the generic kernel is the faster one
  if (mode == 1) most = m <= 24 ? 768 : (m <= 32 ? 512 : (m <= 48 ? 360 : (m <= 64 ? 256 : 0)));
  else if (mode == 0) most = m <= 16 ? 768 : (m <= 24 ? 576 : 0);
  else most = m <= 8 ? 384 : 0;
  return per_sm * groups > most;
}

int launch_flatquant_f32(int mode, const void* x, int64_t ldx, const void* left, const void* right, void* codes, void* scales,
                         int64_t tokens, int m, int n, float clip, int scale_dtype, cudaStream_t stream) {
  const float* xf = reinterpret_cast<const float*>(x);
  const float* lf = reinterpret_cast<const float*>(left);
  const float* rf = reinterpret_cast<const float*>(right);
  const int bpt = ((m + 7) / 8) * (n / 8);
  const size_t one = (size_t)m * (n + 4) * 4 + (size_t)2 * kChunk * (n > m + 7 ? n : m + 7) * 4;
  if (bpt <= 256 && one <= 112 * 1024) return launch_mode<256>(mode, xf, ldx, lf, rf, codes, scales, tokens, m, n, clip, scale_dtype, stream);
  return launch_mode<512>(mode, xf, ldx, lf, rf, codes, scales, tokens, m, n, clip, scale_dtype, stream);
}

}  // namespace qo

// DeviceBackend operator set in fp32 (verse_torch/device.py:219-270; NumPy semantics of :285-335).
#include "common.cuh"
#include "gemm.cuh"
#include "gemm_f32.cuh"
#include <math_constants.h>
#include <stdint.h>

namespace {
using namespace f32_detail;

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sumf(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int THREADS>
__device__ __forceinline__ float block_reduce(float v, bool is_max, float* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = is_max ? warp_max(v) : warp_sumf(v);
  __syncthreads();
  if (lane == 0) sm[warp] = v;
  __syncthreads();
  float r = sm[0];
  for (int w = 1; w < THREADS / 32; ++w) r = is_max ? fmaxf(r, sm[w]) : r + sm[w];
  return r;
}

// softmax over the middle axis of (outer, n, inner); one block per (outer, inner) line
__global__ void __launch_bounds__(256) softmax_kernel(const float* __restrict__ x, float* __restrict__ y,
                                                      long long n, long long inner) {
  __shared__ float sm[8];
  const long long line = blockIdx.x;
  const long long base = (line / inner) * n * inner + (line % inner);
  float m = -CUDART_INF_F;
  for (long long i = threadIdx.x; i < n; i += 256) m = fmaxf(m, x[base + i * inner]);
  m = block_reduce<256>(m, true, sm);
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += 256) s += expf(x[base + i * inner] - m);
  s = block_reduce<256>(s, false, sm);
  for (long long i = threadIdx.x; i < n; i += 256) y[base + i * inner] = expf(x[base + i * inner] - m) / s;
}

// mode 0: rmsnorm  y = x / sqrt(mean(x^2) + eps) * w
// mode 1: layernorm y = (x - mean) / sqrt(var + eps) * w + b
__global__ void __launch_bounds__(256) norm_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                   const float* __restrict__ b, float* __restrict__ y,
                                                   long long cols, float eps, int mode) {
  __shared__ float sm[8];
  const float* xr = x + (long long)blockIdx.x * cols;
  float* yr = y + (long long)blockIdx.x * cols;
  float mean = 0.f;
  if (mode == 1) {
    float s = 0.f;
    for (long long i = threadIdx.x; i < cols; i += 256) s += xr[i];
    mean = block_reduce<256>(s, false, sm) / (float)cols;
  }
  float ss = 0.f;
  for (long long i = threadIdx.x; i < cols; i += 256) { float d = xr[i] - mean; ss += d * d; }
  const float var = block_reduce<256>(ss, false, sm) / (float)cols;
  const float r = sqrtf(var + eps);
  for (long long i = threadIdx.x; i < cols; i += 256) {
    float v = (xr[i] - mean) / r * w[i];
    if (mode == 1 && b) v += b[i];
    yr[i] = v;
  }
}

__global__ void rope_kernel(const float* __restrict__ x, const float* __restrict__ cs, const float* __restrict__ sn,
                            float* __restrict__ y, long long total_rows, long long T, long long D) {
  const long long half = D / 2;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total_rows * half) return;
  const long long row = i / half, j = i % half, t = row % T;
  const float x1 = x[row * D + j], x2 = x[row * D + half + j];
  const float c = cs[t * half + j], s = sn[t * half + j];
  y[row * D + j] = x1 * c - x2 * s;
  y[row * D + half + j] = x1 * s + x2 * c;
}

// ---- attention over fp32 heads ------------------------------------------------------------------------------------------
// four values of a row from element d on; elements from D on are zero
__device__ __forceinline__ float4 row4(const float* __restrict__ r, int d, int D, bool vec) {
  if (vec) return d < D ? *reinterpret_cast<const float4*>(r + d) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(d < D ? r[d] : 0.f, d + 1 < D ? r[d + 1] : 0.f, d + 2 < D ? r[d + 2] : 0.f, d + 3 < D ? r[d + 3] : 0.f);
}

// Few queries, or heads too wide for the tile kernel: a block per query row, any D.  `lpk` lanes (a power of two) share a key's
// dot product in float4 steps, so that a warp reads whole rows; scores stay in shared memory; for the values `lpk` threads
// cover a row and the block's groups of them take every (256 / lpk)-th key, summed at the end.
__global__ void __launch_bounds__(256) attention_row_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                            const float* __restrict__ v, const float* __restrict__ mask,
                                                            float* __restrict__ out, long long Tq, int Tk, int D, float scale,
                                                            int lpk, int vec) {
  extern __shared__ __align__(16) float smem[];      // Tk scores, then 256 partial float4
  __shared__ float red[8];
  float* sc = smem;
  float4* part = reinterpret_cast<float4*>(smem + ((Tk + 3) & ~3));
  const int tid = threadIdx.x;
  const long long qi = blockIdx.x, bh = blockIdx.y;
  const float* qr = q + (bh * Tq + qi) * D;
  const float* kb = k + bh * Tk * D;
  const float* vb = v + bh * Tk * D;
  const int grp = tid / lpk, li = tid % lpk, ng = 256 / lpk;
  float m = -CUDART_INF_F;
  for (int j0 = 0; j0 < Tk; j0 += ng) {              // all lanes of a warp take the same trips
    const int j = j0 + grp;
    float s = 0.f;
    if (j < Tk)
      for (int d = li * 4; d < D; d += lpk * 4) {
        const float4 a = row4(qr, d, D, vec), b = row4(kb + (long long)j * D, d, D, vec);
        s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
      }
    for (int o = lpk >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (j < Tk) {
      s *= scale;
      if (mask) s += mask[qi * Tk + j];
      if (li == 0) sc[j] = s;
      m = fmaxf(m, s);
    }
  }
  m = block_reduce<256>(m, true, red);               // its barriers also publish the scores
  float l = 0.f;
  for (int j = tid; j < Tk; j += 256) { const float e = expf(sc[j] - m); sc[j] = e; l += e; }
  l = block_reduce<256>(l, false, red);
  for (int j = tid; j < Tk; j += 256) sc[j] /= l;    // before the values: their weighted mean fits wherever they do
  __syncthreads();
  for (int d0 = 0; d0 < D; d0 += lpk * 4) {
    const int d = d0 + li * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (d < D)
      for (int j = grp; j < Tk; j += ng) {
        const float p = sc[j];
        const float4 x = row4(vb + (long long)j * D, d, D, vec);
        acc.x = fmaf(p, x.x, acc.x); acc.y = fmaf(p, x.y, acc.y); acc.z = fmaf(p, x.z, acc.z); acc.w = fmaf(p, x.w, acc.w);
      }
    part[tid] = acc;
    __syncthreads();
    for (int e = tid; e < lpk * 4; e += 256) {
      if (d0 + e < D) {
        float s = 0.f;
        for (int gi = 0; gi < ng; ++gi) s += reinterpret_cast<const float*>(part)[gi * lpk * 4 + e];
        out[(bh * Tq + qi) * D + d0 + e] = s;
      }
    }
    __syncthreads();
  }
}

// Few keys (at most a warp's lanes): a warp per query row, a lane per key, then a lane per result.  No shared memory and no barrier: the
// tile kernel's loads, soft-max and write-out take 8 to 16 us for a single tile of keys.
__global__ void __launch_bounds__(256) attention_warp_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                                                             const float* __restrict__ mask, float* __restrict__ out, long long Tq, int Tk, int D,
                                                             float scale, int vec) {
  const int lane = threadIdx.x & 31;
  const long long qi = (long long)blockIdx.x * 8 + (threadIdx.x >> 5), bh = blockIdx.y;
  if (qi >= Tq) return;
  const float* qr = q + (bh * Tq + qi) * D;
  const float* kr = k + (bh * Tk + min(lane, Tk - 1)) * D;
  const float* vb = v + bh * Tk * D;
  float s = 0.f;
  for (int d = 0; d < D; d += 4) {
    const float4 a = row4(qr, d, D, vec), b = row4(kr, d, D, vec);
    s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
  }
  s *= scale;
  if (mask && lane < Tk) s += mask[qi * Tk + lane];
  const float m = warp_max(lane < Tk ? s : -CUDART_INF_F);
  const float e = lane < Tk ? expf(s - m) : 0.f;
  const float p = e / warp_sumf(e);
  for (int d0 = 0; d0 < D; d0 += 32) {
    const int d = d0 + lane;
    float acc = 0.f;
#pragma unroll 8
    for (int j = 0; j < Tk; ++j) {
      const float w = __shfl_sync(0xffffffffu, p, j);
      if (d < D) acc = fmaf(w, vb[(long long)j * D + d], acc);
    }
    if (d < D) out[(bh * Tq + qi) * D + d] = acc;
  }
}

constexpr int64_t AT_MAX_TK = 12800;
constexpr size_t attention_row_smem(int64_t Tk) { return (size_t)((Tk + 3) & ~(int64_t)3) * sizeof(float) + 256 * sizeof(float4); }

// the power of two u with x u in [1/2, 1), for a sum x of exponentials (zero, or 1 to AT_MAX_TK); unit_of(x) / unit_of(from)
__device__ __forceinline__ unsigned exponent_of(float x) { return __float_as_uint(x) & 0x7f800000u; }
__device__ __forceinline__ float unit_of(float x) { return __uint_as_float((253u << 23) - exponent_of(x)); }
__device__ __forceinline__ float unit_ratio(float x, float from) {
  return __uint_as_float((127u << 23) + max(exponent_of(from), 64u << 23) - exponent_of(x));   // from zero: any finite value
}

// Tiles of 64 queries x 64 keys, heads of up to DM.  A warp owns 16 query rows; its 16 lanes of a row hold the row's scores of four
// keys each, so that the online soft-max needs shuffles only, and DM / 16 of its results.  Per thread 8 x 4 products of
// float4s along the head (12 shared loads for 128 FMAs) for the scores, 8 x DM / 16 along the keys for the values: the
// bound is the FMA rate over those loads.  The next keys arrive while values are summed and the values while scores are.
constexpr int AT_Q = 64, AT_K = 64;
template <int DM>
struct AttnTile {
  static constexpr int LD = DM + 4, LDP = AT_K + 4;
  static constexpr size_t SMEM = (size_t)(3 * AT_Q * LD + AT_Q * LDP) * sizeof(float);
};
template <int DM>
__global__ void __launch_bounds__(128) attention_tile_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                             const float* __restrict__ v, const float* __restrict__ mask,
                                                             float* __restrict__ out, long long Tq, int Tk, int D, float scale,
                                                             int vec) {
  constexpr int LD = AttnTile<DM>::LD, LDP = AttnTile<DM>::LDP, DC = DM / 16;
  extern __shared__ __align__(16) float smem[];
  float* sQ = smem;
  float* sK = sQ + AT_Q * LD;
  float* sV = sK + AT_K * LD;
  float* sP = sV + AT_K * LD;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ty = warp * 2 + (lane >> 4), tx = lane & 15;   // rows ty + 8 i, keys tx + 16 j
  const long long bh = blockIdx.y, q0 = (long long)blockIdx.x * AT_Q;
  const float* kb = k + bh * Tk * D;
  const float* vb = v + bh * Tk * D;
  // rows of a tile, zero beyond the last row and beyond D
  auto load = [&](float* dst, const float* src, long long r0, long long rows) {
    const unsigned base = (unsigned)__cvta_generic_to_shared(dst);
    if (vec) {
#pragma unroll 4
      for (int e = tid; e < AT_K * (DM / 4); e += 128) {
        const int r = e / (DM / 4), d = (e % (DM / 4)) * 4;
        const bool ok = r0 + r < rows && d < D;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + (r * LD + d) * 4), "l"(src + (ok ? (r0 + r) * D + d : 0)), "r"(ok ? 16 : 0));
      }
    } else {
#pragma unroll 4
      for (int e = tid; e < AT_K * DM; e += 128) {
        const int r = e / DM, d = e % DM;
        const bool ok = r0 + r < rows && d < D;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(base + (r * LD + d) * 4), "l"(src + (ok ? (r0 + r) * D + d : 0)), "r"(ok ? 4 : 0));
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  load(sQ, q + bh * Tq * D, q0, Tq);
  load(sK, kb, 0, Tk);
  float m[8], l[8];
  f32x2 o[8][DC / 2];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m[i] = -CUDART_INF_F; l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < DC / 2; ++c) o[i][c] = 0;
  }
  for (int k0 = 0; k0 < Tk; k0 += AT_K) {
    load(sV, vb, k0, Tk);
    asm volatile("cp.async.wait_group 1;");          // the keys (and the queries) are there
    __syncthreads();
    f32x2 s2[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s2[i][j] = 0;
#pragma unroll 2
    for (int d = 0; d < DM; d += 4) {
      ulonglong2 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(sQ + (ty + 8 * i) * LD + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(sK + (tx + 16 * j) * LD + d);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          fma2(s2[i][j], a[i].x, b.x);
          fma2(s2[i][j], a[i].y, b.y);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const long long row = q0 + ty + 8 * i;
      float top = m[i], s[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = k0 + tx + 16 * j;
        s[j] = sum2(s2[i][j]) * scale;
        if (mask && row < Tq && key < Tk) s[j] += mask[row * Tk + key];
        if (key >= Tk) s[j] = -CUDART_INF_F;
        top = fmaxf(top, s[j]);
      }
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
      // nothing but -inf so far: exponentials of -inf are then zero, and a row of nothing else ends without a sum
      const float at = top == -CUDART_INF_F ? 0.f : top;
      const float fade = expf(m[i] - at);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[j] = expf(s[j] - at);
        sum += s[j];
      }
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
      // weights in units of a power of two above their sum: sums of values stay within the values' range, and nothing is rounded for it
      // (32 heads x 500 x 500 x 64: 80 us, with 1 / sum instead 85, with sums that may overflow 78).  Before the first key fade is zero.
      const float all = l[i] * fade + sum, unit = unit_of(all), keep = fade * unit_ratio(all, l[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) sP[(ty + 8 * i) * LDP + tx + 16 * j] = s[j] * unit;
      l[i] = all;
      m[i] = top;
#pragma unroll
      for (int c = 0; c < DC / 2; ++c) {
        const float2 t = unpack2(o[i][c]);
        o[i][c] = pack2(t.x * keep, t.y * keep);
      }
    }
    asm volatile("cp.async.wait_group 0;");          // the values are there
    __syncthreads();                                 // and the keys' tile is free
    if (k0 + AT_K < Tk) load(sK, kb, k0 + AT_K, Tk);
    else asm volatile("cp.async.commit_group;");
#pragma unroll 2
    for (int j = 0; j < AT_K; j += 4) {
      float4 p[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) p[i] = *reinterpret_cast<const float4*>(sP + (ty + 8 * i) * LDP + j);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        f32x2 x[DC / 2];
#pragma unroll
        for (int c = 0; c < DC / 2; c += (DC < 4 ? 1 : 2)) {
          if (DC < 4) {
            x[c] = *reinterpret_cast<const f32x2*>(sV + (j + jj) * LD + tx * 2);
          } else {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(sV + (j + jj) * LD + tx * 4 + c * 32);
            x[c] = t.x; x[(c + 1) % (DC / 2)] = t.y;
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float w = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
          const f32x2 ww = pack2(w, w);
#pragma unroll
          for (int c = 0; c < DC / 2; ++c) fma2(o[i][c], ww, x[c]);
        }
      }
    }
    __syncthreads();                                 // the values' tile is free
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const long long row = q0 + ty + 8 * i;
    if (row >= Tq) continue;
    const float all = l[i] * unit_of(l[i]);
#pragma unroll
    for (int c = 0; c < DC / 2; ++c) {
      const int d = DC < 4 ? tx * 2 : tx * 4 + (c >> 1) * 64 + (c & 1) * 2;
      const float2 t = unpack2(o[i][c]);
      if (d < D) out[(bh * Tq + row) * D + d] = t.x / all;
      if (d + 1 < D) out[(bh * Tq + row) * D + d + 1] = t.y / all;
    }
  }
}

template <int DM>
int32_t launch_attention_tile(vn_ctx* ctx, const float* q, const float* k, const float* v, const float* mask, float* out, int64_t BH,
                              int64_t Tq, int64_t Tk, int D, float scale, int vec) {
  constexpr size_t smem = AttnTile<DM>::SMEM;
  VN_CUDA(ctx, cudaFuncSetAttribute(attention_tile_kernel<DM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((unsigned)ceil_div(Tq, (int64_t)AT_Q), (unsigned)BH);
  VN_LAUNCH(ctx, attention_tile_kernel<DM>, grid, 128, smem, q, k, v, mask, out, (long long)Tq, (int)Tk, D, scale, vec);
  return VN_OK;
}

}  // namespace

extern "C" {

int32_t vn_matmul(vn_ctx* ctx, const float* a, const float* b, float* c, int64_t batch, int64_t M, int64_t N,
                  int64_t K, int32_t b_broadcast) {
  VN_CHECK_CTX(ctx);
  VN_REQUIRE(ctx, a && b && c, "null pointer");
  VN_REQUIRE(ctx, batch >= 0 && M >= 0 && N >= 0 && K >= 0 && batch < 65536, "bad shape");
  if (batch * M * N == 0) return VN_OK;
  GemmArgs g;
  g.A = a; g.lda = K; g.a_stride = M * K;
  g.W = b; g.ldw = 1; g.ldw_k = N; g.w_stride = b_broadcast ? 0 : K * N;
  g.C = c; g.ldc = N; g.c_stride = M * N;
  g.M = (int)M; g.N = (int)N; g.K = (int)K; g.nseg = (int)batch;
  return launch_gemm_f32(ctx, g);
}

int32_t vn_linear(vn_ctx* ctx, const float* x, const float* w, const float* bias, float* y, int64_t M, int64_t N,
                  int64_t K) {
  VN_CHECK_CTX(ctx);
  VN_REQUIRE(ctx, x && w && y, "null pointer");
  VN_REQUIRE(ctx, M >= 0 && N >= 0 && K >= 0, "bad shape");
  if (M * N == 0) return VN_OK;
  GemmArgs g;
  g.A = x; g.lda = K; g.W = w; g.ldw = K; g.C = y; g.ldc = N; g.bias = bias;
  g.M = (int)M; g.N = (int)N; g.K = (int)K;
  return launch_gemm_f32(ctx, g);
}

int32_t vn_softmax(vn_ctx* ctx, const float* x, float* y, int64_t outer, int64_t n, int64_t inner) {
  VN_CHECK_CTX(ctx);
  VN_REQUIRE(ctx, x && y && outer >= 0 && n >= 1 && inner >= 1, "bad arguments");
  if (outer * inner == 0) return VN_OK;
  VN_REQUIRE(ctx, outer * inner < (1ll << 31), "too many lines");
  VN_LAUNCH(ctx, softmax_kernel, (unsigned)(outer * inner), 256, 0, x, y, (long long)n, (long long)inner);
  return VN_OK;
}

int32_t vn_layernorm(vn_ctx* ctx, const float* x, const float* w, const float* b, float* y, int64_t rows,
                     int64_t cols, float eps) {
  VN_CHECK_CTX(ctx);
  VN_REQUIRE(ctx, x && w && y && rows >= 0 && cols >= 1, "bad arguments");
  if (rows == 0) return VN_OK;
  VN_LAUNCH(ctx, norm_kernel, (unsigned)rows, 256, 0, x, w, b, y, (long long)cols, eps, 1);
  return VN_OK;
}

int32_t vn_rmsnorm(vn_ctx* ctx, const float* x, const float* w, float* y, int64_t rows, int64_t cols, float eps) {
  VN_CHECK_CTX(ctx);
  VN_REQUIRE(ctx, x && w && y && rows >= 0 && cols >= 1, "bad arguments");
  if (rows == 0) return VN_OK;
  VN_LAUNCH(ctx, norm_kernel, (unsigned)rows, 256, 0, x, w, (const float*)nullptr, y, (long long)cols, eps, 0);
  return VN_OK;
}

int32_t vn_rope(vn_ctx* ctx, const float* x, const float* cs, const float* sn, float* y, int64_t outer, int64_t T,
                int64_t D) {
  VN_CHECK_CTX(ctx);
  VN_REQUIRE(ctx, x && cs && sn && y && D % 2 == 0 && outer >= 0 && T >= 1, "bad arguments");
  const long long n = outer * T * (D / 2);
  if (n == 0) return VN_OK;
  VN_LAUNCH(ctx, rope_kernel, (unsigned)ceil_div(n, 256ll), 256, 0, x, cs, sn, y, (long long)(outer * T),
            (long long)T, (long long)D);
  return VN_OK;
}

int32_t vn_attention(vn_ctx* ctx, const float* q, const float* k, const float* v, const float* mask, float* out,
                     int64_t BH, int64_t Tq, int64_t Tk, int64_t D) {
  VN_CHECK_CTX(ctx);
  VN_REQUIRE(ctx, q && k && v && out && BH >= 0 && Tq >= 0 && Tk >= 1 && D >= 1, "bad arguments");
  VN_REQUIRE(ctx, BH < 65536, "too many batch*heads");
  if (BH * Tq == 0) return VN_OK;
  // one limit for every shape, whichever kernel takes it (the row kernel keeps a row of scores in shared memory, the tile kernel none)
  VN_REQUIRE(ctx, Tk <= AT_MAX_TK, "Tk %lld too long for the backend attention op", (long long)Tk);
  const int vec = D % 4 == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) == 0;
  const float scale = 1.0f / sqrtf((float)D);
  // A tile's 64 rows share the keys that are loaded; below a quarter of them a block per row is as fast and spreads over more SMs.
  // A tile of few keys is mostly fixed cost, 8 us for D of 32, 10 for 64, 16 for 128: a block per row up to 512 rows (16 x 8 keys x 64:
  // 10.3 -> 4.6 us), a warp per row beyond (64 x 64 rows, D = 16, 4 keys: 8.3 -> 4.7; 512 x 4 rows: 10.3 -> 4.6 of blocks; at 512 products a
  // row tiles are level, 64 x 128 rows x 16 keys x 32 8.3 against 12.4).
  const bool few = Tk <= 32 && D <= 128, blocks = BH * Tq <= 512;
  if (few && !blocks && (Tk <= 8 || Tk * D <= 512)) {
    dim3 grid((unsigned)ceil_div(Tq, (int64_t)8), (unsigned)BH);
    VN_LAUNCH(ctx, attention_warp_kernel, grid, 256, 0, q, k, v, mask, out, (long long)Tq, (int)Tk, (int)D, scale, vec);
    return VN_OK;
  }
  if (Tq >= 16 && D <= 128 && !(few && blocks)) {
    if (D <= 32) return launch_attention_tile<32>(ctx, q, k, v, mask, out, BH, Tq, Tk, (int)D, scale, vec);
    if (D <= 64) return launch_attention_tile<64>(ctx, q, k, v, mask, out, BH, Tq, Tk, (int)D, scale, vec);
    return launch_attention_tile<128>(ctx, q, k, v, mask, out, BH, Tq, Tk, (int)D, scale, vec);
  }
  VN_REQUIRE(ctx, Tq < (1ll << 31), "too many queries");
  int lpk = 1;
  while (lpk < 32 && lpk * 4 < D) lpk *= 2;
  const size_t smem = attention_row_smem(Tk);
  // the function's limit is shared by all contexts and threads on a device: raised once, to the longest row
  static unsigned long long attr_set = 0;
  if (smem > 48 * 1024 && !((attr_set >> (ctx->device & 63)) & 1ull)) {
    VN_CUDA(ctx, cudaFuncSetAttribute(attention_row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attention_row_smem(AT_MAX_TK)));
    attr_set |= 1ull << (ctx->device & 63);
  }
  dim3 grid((unsigned)Tq, (unsigned)BH);
  VN_LAUNCH(ctx, attention_row_kernel, grid, 256, smem, q, k, v, mask, out, (long long)Tq, (int)Tk, (int)D, scale, lpk, vec);
  return VN_OK;
}

}  // extern "C"

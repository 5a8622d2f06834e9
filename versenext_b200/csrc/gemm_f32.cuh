// fp32 GEMMs on the FMA pipes: C[M,N] = A[M,K] * W[N,K]^T with the epilogues of GemmArgs (gemm.cuh).
//
// Full fp32 arithmetic: the products are not split for the 16-bit tensor cores, whose accumulators round differently.  The
// bound is therefore 148 SMs x 128 FMA per clock (74 TFLOP/s at 1965 MHz), or HBM where few rows meet a large matrix.
#pragma once
#include "common.cuh"
#include "gemm.cuh"
#include <algorithm>

namespace f32_detail {

constexpr int BK = 16, LDT = BK + 4, STAGES = 3;   // rows of 20 floats: eight rows of 16 bytes each fall into distinct banks

__device__ __forceinline__ void cp16(unsigned dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp4(unsigned dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes));
}

// Two fp32 FMAs in one instruction: half the issue slots, and no more registers than two chains per result need.
typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ f32x2 pack2(float lo, float hi) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ float2 unpack2(f32x2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ float sum2(f32x2 v) { const float2 t = unpack2(v); return t.x + t.y; }

// one result of a GEMM at (row, n): bias, function, factors, and the store or the addition to the residual
__device__ __forceinline__ void put(const GemmArgs& g, long long c_base, long long row, int n, float v) {
  if (g.bias) v += g.bias[n];
  if (n < g.post_n) v = post_act(v, g.post, g.c_bf16);
  const long long idx = c_base + row * g.ldc + n;
  if (g.mul) v *= mul_at(g, idx);
  if (g.epi == EPI_ADD) reinterpret_cast<float*>(g.C)[idx] += v;
  else store_out<float>(g.C, idx, v, g.c_bf16);
}

// Tile kernel, any shape and stride.  Both operands lie in shared memory as [row][k] (k contiguous, as in memory), brought by
// 16-byte asynchronous copies three stages deep where `vec` says that rows start on 16 bytes, else by 4-byte ones; a
// thread reads float4s along k and multiplies TM x TN pairs of rows four k at a time, so a shared-memory load feeds TM or TN
// FMA pairs and nothing is transposed.  A thread's rows are TY apart and its columns TX apart: a warp's 4 x 8 threads read
// neighbouring rows, free of bank conflicts.  Every result is the sum of two FMA chains in ascending k (k even, k odd), whatever
// the tile.  1000 x 2752 x 1024: 317 us with scalar loads and stores of a 64 x 64 tile, 165 us now (34 TFLOP/s); 2048^3 39 TFLOP/s.
template <int BM, int BN, int TM, int TN, int MINB>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB) gemm_f32_kernel(GemmArgs g, int a_vec, int w_vec, int w_nfast) {
  constexpr int TY = BM / TM, TX = BN / TN, NT = TY * TX;
  static_assert(TY % 4 == 0 && TX % 8 == 0, "warps of 4 x 8 threads");
  extern __shared__ __align__(16) float smem[];     // STAGES x (BM + BN) x LDT, then the A rows' pointers
  const float** rows = reinterpret_cast<const float**>(smem + STAGES * (BM + BN) * LDT);
  const int z = blockIdx.z, tid = threadIdx.x;
  int row0 = 0, Mz = g.M;
  if (g.seg_cnt) { row0 = g.seg_off[z]; Mz = g.seg_cnt[z]; }
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (m0 >= Mz) return;
  const float* A = reinterpret_cast<const float*>(g.A) + (g.seg_cnt ? 0 : (long long)z * g.a_stride);
  const float* W = reinterpret_cast<const float*>(g.W) + (long long)z * g.w_stride;
  const long long c_base = g.seg_cnt ? 0 : (long long)z * g.c_stride;
  for (int r = tid; r < BM; r += NT) {
    const int m = row0 + min(m0 + r, Mz - 1);
    rows[r] = A + (long long)(g.a_rows ? g.a_rows[m] : m) * g.lda;
  }
  __syncthreads();
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem);
  const int nk = (g.K + BK - 1) / BK;

  auto load = [&](int kt) {
    const int k0 = kt * BK;
    const unsigned sA = base + (unsigned)((kt % STAGES) * (BM + BN) * LDT * 4), sW = sA + BM * LDT * 4;
    if (a_vec) {
#pragma unroll
      for (int e = tid; e < BM * (BK / 4); e += NT) {
        const int r = e / (BK / 4), k = (e % (BK / 4)) * 4;
        const bool ok = m0 + r < Mz && k0 + k < g.K;
        cp16(sA + (r * LDT + k) * 4, rows[r] + (ok ? k0 + k : 0), ok ? 16 : 0);
      }
    } else {
#pragma unroll 4
      for (int e = tid; e < BM * BK; e += NT) {
        const int r = e / BK, k = e % BK;
        const bool ok = m0 + r < Mz && k0 + k < g.K;
        cp4(sA + (r * LDT + k) * 4, rows[r] + (ok ? k0 + k : 0), ok ? 4 : 0);
      }
    }
    if (w_vec) {
#pragma unroll
      for (int e = tid; e < BN * (BK / 4); e += NT) {
        const int r = e / (BK / 4), k = (e % (BK / 4)) * 4;
        const bool ok = n0 + r < g.N && k0 + k < g.K;
        cp16(sW + (r * LDT + k) * 4, W + (ok ? (long long)(n0 + r) * g.ldw + k0 + k : 0), ok ? 16 : 0);
      }
    } else {
#pragma unroll 4
      for (int e = tid; e < BN * BK; e += NT) {
        const int r = w_nfast ? e % BN : e / BK, k = w_nfast ? e / BN : e % BK;
        const bool ok = n0 + r < g.N && k0 + k < g.K;
        cp4(sW + (r * LDT + k) * 4, W + (ok ? (long long)(n0 + r) * g.ldw + (long long)(k0 + k) * g.ldw_k : 0), ok ? 4 : 0);
      }
    }
  };

  const int warp = tid >> 5, lane = tid & 31;
  const int ty = (warp / (TX / 8)) * 4 + lane / 8, tx = (warp % (TX / 8)) * 8 + lane % 8;
  f32x2 acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load(s);
    asm volatile("cp.async.commit_group;");
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2));
    __syncthreads();
    if (kt + STAGES - 1 < nk) load(kt + STAGES - 1);
    asm volatile("cp.async.commit_group;");
    const float* sA = smem + (kt % STAGES) * (BM + BN) * LDT;
    const float* sW = sA + BM * LDT;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(sA + (ty + i * TY) * LDT + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(sW + (tx + j * TX) * LDT + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].x, w.x);
#pragma unroll
        for (int i = 0; i < TM; ++i) fma2(acc[i][j], a[i].y, w.y);
      }
    }
  }
  // The results go through shared memory: a loop over them that is not unrolled keeps the code of the epilogues small (unrolled, it
  // took 10 to 20 us a launch to fetch), and its stores are coalesced.
  static_assert(BM * (BN + 4) <= STAGES * (BM + BN) * LDT, "the tile of results fits");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) smem[(ty + i * TY) * (BN + 4) + tx + j * TX] = sum2(acc[i][j]);
  __syncthreads();
  const int pair = g.epi == EPI_SWIGLU ? 2 : 1;        // gate and up of a pair are neighbours
#pragma unroll 1
  for (int e = tid * pair; e < BM * BN; e += NT * pair) {
    const int r = e / BN, c = e % BN;
    if (m0 + r >= Mz || n0 + c + pair > g.N) continue;
    const float v = smem[r * (BN + 4) + c];
    if (pair == 2)
      store_out<float>(g.C, c_base + (long long)(row0 + m0 + r) * g.ldc + ((n0 + c) >> 1), glu(v, smem[r * (BN + 4) + c + 1], g.act, g.act_limit, g.c_bf16), g.c_bf16);
    else
      put(g, c_base, row0 + m0 + r, n0 + c, v);
  }
}

// Few rows: a warp owns NR consecutive output features and walks K in float4 steps, one 512-byte coalesced segment of every
// weight row per trip, against up to MR rows of A at a time (a few KB: they stay in L1).  With more rows the warp makes one
// pass per group of MR over the same weight rows, which it finds in L1 / L2, so DRAM still sees every weight once.  Per
// output each lane sums its k = 4 lane + 128 i terms in order (even and odd apart), then the lanes are added pair by pair; the NR x MR sums of a
// warp are spread over its lanes while they are added (a lane passes on half of what it holds at each step), so that 32 sums
// take 31 exchanges and every lane stores one of them.  NORM: every block normalises the few short rows of A into shared memory
// for itself, a launch less on a chain that is nothing but launches.  MANY: matrices of many features, bound by HBM and so by the
// weights that an SM has in flight: registers for two blocks of eight warps and more, rows addressed by 32-bit offsets.  Of few
// features every SM has a few warps anyway, and these hold as much as they can (8 x 4096 x 1024: 7.2 us, with 128 registers 16).
// 1 / 5 / 8 / 16 / 32 rows x 100,000 x 1024: 64 / 100 / 103 / 168 / 345 us, with one block of eight warps on an SM 68 / 160 / 160 / 239 / 418.
constexpr int NR = 4, NORM_MAX = 4096;
template <int MR, bool NORM, bool MANY>
__global__ void __launch_bounds__(256, !MANY ? (MR == 8 ? 1 : 2) : MR == 1 ? 4 : MR == 2 ? 3 : 2) gemm_f32_rows_kernel(GemmArgs g) {
  const int lane = threadIdx.x & 31;
  const long long n0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * NR;
  const float* A = reinterpret_cast<const float*>(g.A);
  long long lda = g.lda;
  if (NORM) {
    __shared__ __align__(16) float rows[NORM ? NORM_MAX : 4];
    for (int m = threadIdx.x >> 5; m < g.M; m += blockDim.x >> 5) {
      float ss = 0.f;
      for (int k = lane * 4; k < g.K; k += 128) {
        const float4 x = *reinterpret_cast<const float4*>(A + m * lda + k);
        ss += x.x * x.x; ss += x.y * x.y; ss += x.z * x.z; ss += x.w * x.w;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float r = sqrtf(ss / (float)g.K + g.norm_eps);
      for (int k = lane * 4; k < g.K; k += 128) {
        const float4 x = *reinterpret_cast<const float4*>(A + m * lda + k), w = *reinterpret_cast<const float4*>(g.norm + k);
        *reinterpret_cast<float4*>(rows + m * g.K + k) = make_float4(x.x / r * w.x, x.y / r * w.y, x.z / r * w.z, x.w / r * w.w);
      }
    }
    __syncthreads();
    A = rows; lda = g.K;
  }
  if (n0 >= g.N) return;
  const float* wr[NR];
#pragma unroll
  for (int j = 0; j < NR; ++j) wr[j] = reinterpret_cast<const float*>(g.W) + (n0 + j < g.N ? n0 + j : g.N - 1) * g.ldw;
  for (int m0 = 0; m0 < g.M; m0 += MR) {
    f32x2 acc[NR * MR];
#pragma unroll
    for (int i = 0; i < NR * MR; ++i) acc[i] = 0;
    int off[MANY ? MR : 1];
    if (MANY)
#pragma unroll
      for (int i = 0; i < MR; ++i) off[i] = (int)((m0 + i < g.M ? m0 + i : g.M - 1) * lda);
#pragma unroll 1
    for (int k = lane * 4; k < g.K; k += 128) {
      ulonglong2 wv[NR];
#pragma unroll
      for (int j = 0; j < NR; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(wr[j] + k);
#pragma unroll
      for (int i = 0; i < MR; ++i) {
        const int m = m0 + i < g.M ? m0 + i : g.M - 1;
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(MANY ? A + off[MANY ? i : 0] + k : A + m * lda + k);
#pragma unroll
        for (int j = 0; j < NR; ++j) {
          fma2(acc[j * MR + i], x.x, wv[j].x);
          fma2(acc[j * MR + i], x.y, wv[j].y);
        }
      }
    }
    float v[NR * MR];
#pragma unroll
    for (int i = 0; i < NR * MR; ++i) v[i] = sum2(acc[i]);
    int o = 16;
#pragma unroll
    for (int half = NR * MR / 2; half >= 1; half >>= 1, o >>= 1) {
      const bool hi = lane & o;
#pragma unroll
      for (int t = 0; t < half; ++t) {
        const float give = hi ? v[t] : v[t + half], keep = hi ? v[t + half] : v[t];
        v[t] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
#pragma unroll
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    // lane: feature lane / 8, row (lane % 8) / (8 / MR); of equal ones the first stores
    const long long n = n0 + (lane >> 3);
    const int m = m0 + (lane & 7) / (8 / MR);
    const bool mine = (lane & 7) % (8 / MR) == 0 && m < g.M && n < g.N;
    if (g.epi == EPI_SWIGLU) {
      const float up = __shfl_down_sync(0xffffffffu, v[0], 8);
      if (mine && !(n & 1) && n + 1 < g.N)
        store_out<float>(g.C, (long long)m * g.ldc + (n >> 1), glu(v[0], up, g.act, g.act_limit, g.c_bf16), g.c_bf16);
    } else if (mine) {
      put(g, 0, m, (int)n, v[0]);
    }
  }
}

template <int BM, int BN, int TM, int TN, int MINB>
inline int32_t launch_tile(vn_ctx* ctx, const GemmArgs& g, int a_vec, int w_vec, int w_nfast) {
  constexpr size_t smem = (size_t)STAGES * (BM + BN) * LDT * 4 + BM * sizeof(float*);
  static_assert(smem <= 48 * 1024, "no opt-in needed");
  dim3 grid(ceil_div(g.N, BN), ceil_div(g.M, BM), g.nseg);
  VN_LAUNCH_NAMED(ctx, g.tag ? g.tag : "gemm_f32_kernel", (gemm_f32_kernel<BM, BN, TM, TN, MINB>), grid, (BM / TM) * (BN / TN), smem, g, a_vec, w_vec, w_nfast);
  return VN_OK;
}

template <int MR>
inline int32_t launch_rows(vn_ctx* ctx, const GemmArgs& g) {
  // blocks of two warps while that leaves SMs without one, of eight where the matrix is large
  const int warps = g.N >= 8 * NR * 4 * ctx->sm_count ? 8 : 2;
  const char* name = g.tag ? g.tag : "gemm_f32_rows_kernel";
  if (g.norm) VN_LAUNCH_NAMED(ctx, name, (gemm_f32_rows_kernel<MR, true, false>), ceil_div(g.N, warps * NR), warps * 32, 0, g);
  else if (warps == 8 && g.M * g.lda < (1ll << 31)) VN_LAUNCH_NAMED(ctx, name, (gemm_f32_rows_kernel<MR, false, true>), ceil_div(g.N, warps * NR), warps * 32, 0, g);
  else VN_LAUNCH_NAMED(ctx, name, (gemm_f32_rows_kernel<MR, false, false>), ceil_div(g.N, warps * NR), warps * 32, 0, g);
  return VN_OK;
}

}  // namespace f32_detail

// GEMMs that may ask for the norm of their rows: the rows kernel's, with few short rows.  The step of 5 rows through the 64-wide
// model took 89 us with 19 launches; a norm launch is 3 us of it, the norm itself inside a GEMM of 5 x 64 values under 1 us.
inline bool gemm_f32_norm_supported(const GemmArgs& g) {
  return g.M <= 16 && (long long)g.M * g.K <= f32_detail::NORM_MAX && g.K > 0 && g.nseg == 1 && !g.seg_cnt && !g.a_rows && !g.wq && g.ldw_k == 1 &&
         (((uintptr_t)g.A | (uintptr_t)(g.lda * 4) | (uintptr_t)g.W | (uintptr_t)(g.ldw * 4) | (uintptr_t)(g.K * 4)) & 15) == 0 && ((uintptr_t)g.norm & 15) == 0;
}

inline int32_t launch_gemm_f32(vn_ctx* ctx, const GemmArgs& g) {
  using namespace f32_detail;
  if (g.M <= 0 || g.N <= 0) return VN_OK;
  if (g.norm && !gemm_f32_norm_supported(g)) return vn_fail(ctx, VN_ERR_UNSUPPORTED, "norm inside an fp32 GEMM of %d x %d", g.M, g.K);
  const bool aligned_a = (((uintptr_t)g.A | (uintptr_t)(g.lda * 4) | (uintptr_t)(g.a_stride * 4) | (uintptr_t)(g.K * 4)) & 15) == 0;
  const bool aligned_w = g.ldw_k == 1 && (((uintptr_t)g.W | (uintptr_t)(g.ldw * 4) | (uintptr_t)(g.w_stride * 4) | (uintptr_t)(g.K * 4)) & 15) == 0;
  // A warp per four features streams the weights once where few rows meet them; up to 16 rows also for narrow matrices, where the
  // tile kernel's few blocks would each walk the whole K alone.
  if (aligned_a && aligned_w && g.nseg == 1 && !g.seg_cnt && !g.a_rows && g.K > 0 && (g.M <= 16 || (g.M <= 32 && g.N >= 1024 && g.K >= 128))) {
    if (g.M == 1) return launch_rows<1>(ctx, g);
    if (g.M == 2) return launch_rows<2>(ctx, g);
    if (g.M <= 4) return launch_rows<4>(ctx, g);
    return launch_rows<8>(ctx, g);
  }
  // The tile that ends first.  Measured for K = 1024: a block alone on its SM takes 50, 35 and 26 us for tiles of 64 x 64, 32 x 64
  // and 32 x 32, and each of several resident ones adds 31.6, 17.3 and 10.8 us (the smaller a thread's part, the more
  // loads from shared memory per product).  Tiles of 8 x 8 per thread were slower everywhere (two blocks per SM).
  const long long sm = ctx->sm_count;
  auto cost = [&](int bm, int bn, double alone, double more) {
    const long long blocks = (long long)ceil_div(g.M, bm) * ceil_div(g.N, bn) * g.nseg;
    return std::max(alone, (double)((blocks + sm - 1) / sm) * more);
  };
  const double c84 = cost(64, 64, 50.0, 31.6), c44 = cost(32, 64, 35.0, 17.3), c42 = cost(32, 32, 26.0, 10.8);
  const int nfast = g.ldw_k != 1;
  // (more rows than 65,535 blocks of 32 cover take the tile of 64)
  if ((c84 <= c44 && c84 <= c42) || ceil_div(g.M, 32) > 65535) return launch_tile<64, 64, 8, 4, 4>(ctx, g, aligned_a, aligned_w, nfast);
  if (c44 <= c42) return launch_tile<32, 64, 4, 4, 5>(ctx, g, aligned_a, aligned_w, nfast);
  return launch_tile<32, 32, 4, 2, 6>(ctx, g, aligned_a, aligned_w, nfast);
}

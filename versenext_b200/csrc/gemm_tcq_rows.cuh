// Weight-only quantised linears on tcgen05, outside the split-K route of at most 256 rows (gemm_tcq.cuh): prompts, large verification
// batches, the heads of prompts' last rows, and every row count of models wider than that route takes.
//
// As in gemm_tcq.cuh the weights travel as raw bytes and become the bf16 UMMA operand inside shared memory, here always as
// the exact small integers.  A scale per output row is applied to the accumulator at the end; scales per 128 inputs (QMODE 3)
// need their groups' sums apart, so the accumulator in TMEM holds one group at a time, in two buffers, and the
// promoting warps add scale x group sum into registers (fp32, as the mma.sync kernel does: no weight is rounded) while the
// tensor cores are at the next group.
//
// CTA: 128 features x up to 128 rows, whole K; warp 0 TMA, warp 1 MMA, warps 2..7 turn the bytes into the operand, warps
// 8..11 promote (lane = feature, a register per row), the last ten write out.  One CTA per SM (a promoting thread holds 128
// sums).  A converting warp has a stage of its own and takes every S-th k block, so that it sees each phase of its barrier in turn.
// Bound by shared memory: a k block of 112 rows moves 70 KB through it (bytes in, operand out, both operands to the tensor
// cores), 560 cycles at 128 bytes each, where its MMAs take 240 and a block was seen to take 700.  448 rows, INT4 groups / INT8:
// 1024 -> 5504 28 / 26 us, -> 32,000 98 / 90 us; with mma.sync 61 us and 274 us for the groups.  Few rows leave SMs idle (no split along
// K) and are still ahead of mma.sync: 1 / 32 / 128 rows of INT4 groups, 2560 -> 3584 27 / 27 / 29 us against 34 / 37 / 60, 6848 -> 2560
// 57 / 58 / 62 against 85 / 93 / 150.
#pragma once
#include "gemm_tcq.cuh"

namespace tc_detail {

constexpr int QR_ROWS = 128, QR_CONV = 6, QR_WRITE = QR_CONV + 4, QR_THREADS = (2 + QR_WRITE) * 32;

// eight biased nibbles (value + 8, element e in bits 4e..4e+3) -> four bf16x2 words.  0x4300 | n is the bf16 128 + n.
__device__ __forceinline__ void i4x8_to_bf16_ints(unsigned x, unsigned (&o)[4]) {
  const __nv_bfloat162 off = __floats2bfloat162_rn(136.f, 136.f);
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const unsigned y = __byte_perm(x, 0u, 0x4440 + h);                       // byte h alone
    const unsigned p = ((y * 0x1001u) & 0x000f000fu) | 0x43004300u;          // its nibbles in the two halves
    const __nv_bfloat162 r = __hsub2(reinterpret_cast<const __nv_bfloat162&>(p), off);
    o[h] = reinterpret_cast<const unsigned&>(r);
  }
}

// a tile's rows from shared memory, [row][128 features] fp32, to C
template <int MODE>
__device__ __forceinline__ void qr_write(const TcArgs& g, const float* tile, int w, int lane, int n0, int row0, int cnt, bool vec) {
  const int c4 = lane * 4, n = n0 + c4;
  if (vec) {
    if (n >= g.N) return;                                                    // N % 4 == 0
    auto rows = [&](auto tag) {
      constexpr int ACT = decltype(tag)::act;
      (void)ACT;
#pragma unroll 1
      for (int r0 = w; r0 < cnt; r0 += 4 * QR_WRITE) {                         // four rows at a time: loads first, then stores
        float4 x[4];
        if (MODE == TC_ADD) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (r0 + QR_WRITE * j < cnt) x[j] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g.C) + (long long)(row0 + r0 + QR_WRITE * j) * g.ldc + n);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = r0 + QR_WRITE * j;
          if (r >= cnt) continue;
          const float4 v = *reinterpret_cast<const float4*>(tile + r * BF + c4);
          const long long at = (long long)(row0 + r) * g.ldc;
          if (MODE == TC_SWIGLU) {
            const float a = glu_of<ACT>(v.x, v.y, g.act_limit, g.c_bf16), b = glu_of<ACT>(v.z, v.w, g.act_limit, g.c_bf16);
            if (g.c_bf16) *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(g.C) + at + (n >> 1)) = __floats2bfloat162_rn(a, b);
            else *reinterpret_cast<float2*>(reinterpret_cast<float*>(g.C) + at + (n >> 1)) = make_float2(a, b);
          } else if (MODE == TC_ADD) {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(g.C) + at + n) = make_float4(x[j].x + v.x, x[j].y + v.y, x[j].z + v.z, x[j].w + v.w);
          } else if (g.c_bf16) {
            uint2 u;
            *reinterpret_cast<__nv_bfloat162*>(&u.x) = __floats2bfloat162_rn(v.x, v.y);
            *reinterpret_cast<__nv_bfloat162*>(&u.y) = __floats2bfloat162_rn(v.z, v.w);
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(g.C) + at + n) = u;
          } else {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(g.C) + at + n) = v;
          }
        }
      }
    };
    if (MODE == TC_SWIGLU) with_glu(g.act, rows);
    else rows(GluTag<GLU_SILU>());
    return;
  }
#pragma unroll 1
  for (int r = w; r < cnt; r += QR_WRITE) {
    const long long at = (long long)(row0 + r) * g.ldc;
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      if (n + i >= g.N) break;
      const float v = tile[r * BF + c4 + i];
      if (MODE == TC_SWIGLU) {
        if (!(i & 1) && n + i + 1 < g.N) store_out<float>(g.C, at + ((n + i) >> 1), glu(v, tile[r * BF + c4 + i + 1], g.act, g.act_limit, g.c_bf16), g.c_bf16);
      } else if (MODE == TC_ADD) {
        reinterpret_cast<float*>(g.C)[at + n + i] += v;
      } else {
        store_out<float>(g.C, at + n + i, v, g.c_bf16);
      }
    }
  }
}

template <int QMODE, int MODE>
__global__ void __launch_bounds__(QR_THREADS, 1)
gemm_tcq_rows_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, TcArgs g,
                     const float* __restrict__ w_scale, long long ws_stride, int stages) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ unsigned long long bar_full[8], bar_empty[8], bar_conv[8], bar_part[2], bar_free[2];
  __shared__ unsigned tmem_base_slot;
  __shared__ int s_error;
  constexpr int RAW_ROW = QMODE == 1 ? BK : BK / 2;
  constexpr unsigned RAW_BYTES = BF * RAW_ROW;
  constexpr unsigned W_BYTES = BF * BK * 2, X_BYTES = QR_ROWS * BK * 2, STAGE = W_BYTES + X_BYTES + RAW_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, z = blockIdx.z;
  const int S = stages;                                                      // at most QR_CONV
  int row0 = 0, cnt = g.M;
  pdl_trigger();
  if (g.seg_cnt) { pdl_wait(); row0 = g.seg_off[z]; cnt = g.seg_cnt[z]; }
  else { row0 = z * g.seg_rows; cnt = min(g.seg_rows, g.rows_all - row0); }
  if (cnt > QR_ROWS) cnt = QR_ROWS;
  if (cnt <= 0) return;                                                      // uniform, before any barrier or TMEM allocation
  const int cnt16 = (cnt + 15) & ~15, n0 = blockIdx.x * BF, nkb = g.K / BK;
  const int per_group = QMODE == 3 ? 2 : nkb, ngroup = (nkb + per_group - 1) / per_group;
  const int zw = g.seg_cnt ? (g.seg_w ? g.seg_w[z] : z) : 0;                 // which weight matrix
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); mbar_init(&bar_conv[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&bar_part[b], 1); mbar_init(&bar_free[b], 4); }
    s_error = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  constexpr unsigned NCOLS = 2 * QR_ROWS;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(NCOLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = tmem_base_slot;
  float acc[QR_ROWS];                                                        // promoting warps only
  bool acc_ok = true;

  if (warp == 0) {
    if (lane == 0) {
      const int w_row = (int)((long long)zw * g.w_rows_per_seg) + n0;
      const int npre = g.seg_cnt ? 0 : (nkb < S ? nkb : S);
      for (int kb = 0; kb < npre; ++kb) {                                    // weights do not depend on the kernels before
        mbar_expect_tx_only(&bar_full[kb], RAW_BYTES);
        tma_load_2d(base + (size_t)kb * STAGE + W_BYTES + X_BYTES, &tm_w, &bar_full[kb], kb * RAW_ROW, w_row);
      }
      if (!g.seg_cnt) pdl_wait();
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % S;
        unsigned char* st = base + (size_t)s * STAGE;
        if (kb < npre) {
          mbar_expect_tx(&bar_full[s], X_BYTES);
        } else {
          if (!mbar_wait(&bar_empty[s], ((kb / S) & 1) ^ 1)) { s_error = 1; break; }
          mbar_expect_tx(&bar_full[s], RAW_BYTES + X_BYTES);
          tma_load_2d(st + W_BYTES + X_BYTES, &tm_w, &bar_full[s], kb * RAW_ROW, w_row);
        }
        // always the whole box; rows beyond the segment (another's, or zeros) are not multiplied
        tma_load_2d(st + W_BYTES, &tm_x, &bar_full[s], kb * BK, row0);
      }
    }
  } else if (warp == 1) {
    // the whole warp walks the stages, one elected lane issues: 10 % faster than a loop inside `lane == 0`
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(cnt16 >> 3) << 17) | ((unsigned)(BF >> 4) << 24);
    bool ok = true;
    int s = 0;
    unsigned ph = 0;
    for (int gi = 0; gi < ngroup && ok; ++gi) {
      const int b = gi & 1;
      if (gi >= 2 && !__all_sync(0xffffffffu, mbar_wait(&bar_free[b], ((gi >> 1) & 1) ^ 1))) { s_error = 1; ok = false; break; }
      const int kb_end = min(nkb, (gi + 1) * per_group);
      for (int kb = gi * per_group; kb < kb_end; ++kb) {
        // converted implies landed; the wait on bar_full makes the TMA-written rows visible here
        if (!__all_sync(0xffffffffu, mbar_wait(&bar_conv[s], ph) && mbar_wait(&bar_full[s], ph))) { s_error = 1; ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        unsigned char* st = base + (size_t)s * STAGE;
        const unsigned long long da = umma_desc(st), db = umma_desc(st + W_BYTES);
        if (elect_one()) {
#pragma unroll
          for (int k4 = 0; k4 < BK / 16; ++k4)
            umma_bf16(tmem_base + (unsigned)(b * QR_ROWS), da + 2ull * k4, db + 2ull * k4, idesc, (kb != gi * per_group) | (k4 != 0));
          umma_commit(&bar_empty[s]);
        }
        __syncwarp();
        if (++s == S) { s = 0; ph ^= 1u; }
      }
      if (elect_one()) umma_commit(&bar_part[b]);
      __syncwarp();
    }
  } else if (warp < 2 + QR_CONV) {
    // warp 2 + s converts stage s: a barrier's phases may only be awaited one after the other.  Item i * 32 + lane covers weight
    // row item / 8, 16-byte output chunk item % 8: a warp reads 128 or 256 contiguous bytes per step and its eight-lane
    // groups write one whole swizzled row each.
    const int c = lane & 7, s = warp - 2;
    unsigned ph = 0;
    for (int kb = s; s < S && kb < nkb; kb += S, ph ^= 1u) {
      if (!__all_sync(0xffffffffu, mbar_wait(&bar_full[s], ph))) { s_error = 1; acc_ok = false; break; }
      unsigned char* st = base + (size_t)s * STAGE;
      const unsigned char* raw = st + W_BYTES + X_BYTES;
#pragma unroll 2
      for (int i0 = 0; i0 < BF * 8 / 32; i0 += 8) {
        uint2 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (QMODE == 1) v[i] = reinterpret_cast<const uint2*>(raw)[(i0 + i) * 32 + lane];
          else v[i].x = reinterpret_cast<const unsigned*>(raw)[(i0 + i) * 32 + lane];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = (i0 + i) * 4 + (lane >> 3);
          unsigned o[4];
          if (QMODE == 1) {
            i8x4_to_bf16(v[i].x ^ 0x80808080u, o[0], o[1]);
            i8x4_to_bf16(v[i].y ^ 0x80808080u, o[2], o[3]);
          } else {
            i4x8_to_bf16_ints(v[i].x ^ 0x88888888u, o);
          }
          *reinterpret_cast<uint4*>(st + r * 128 + ((c ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");           // generic writes -> tensor-core reads
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_conv[s]);
    }
    __syncwarp();
  } else {
    const int q = warp & 3, n = n0 + q * 32 + lane;
    const int groups = QMODE == 3 ? (g.K + 127) / 128 : 1;
    const float* sc = w_scale + (long long)zw * ws_stride + (long long)(n < g.N ? n : g.N - 1) * groups;
#pragma unroll
    for (int i = 0; i < QR_ROWS; ++i) acc[i] = 0.f;
    float scale = sc[0];
    for (int gi = 0; gi < ngroup; ++gi) {
      const int b = gi & 1;
      const float next = gi + 1 < ngroup ? sc[gi + 1] : 0.f;                 // on its way while this group is awaited
      if (!__all_sync(0xffffffffu, mbar_wait(&bar_part[b], (gi >> 1) & 1))) { s_error = 1; acc_ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int ch = 0; ch < QR_ROWS / 32; ++ch) {
        if (ch * 32 < cnt) {                                                 // uniform
          unsigned r[32];
          tmem_ld32(tmem_base + ((unsigned)(q * 32) << 16) + (unsigned)(b * QR_ROWS + ch * 32), r);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[ch * 32 + i] = fmaf(__uint_as_float(r[i]), scale, acc[ch * 32 + i]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_free[b]);
      scale = next;
    }
    // all MMAs are done: the stages are free.  One row of 128 features after another.
    if (acc_ok) {
      float* tile = reinterpret_cast<float*>(base);
      const int f = q * 32 + lane;
#pragma unroll
      for (int i = 0; i < QR_ROWS; ++i) tile[i * BF + f] = acc[i];
    }
  }
  if (warp >= 2) {
    if (!g.seg_cnt) pdl_wait();
    int go;
    {
      const int mine = (acc_ok && *(volatile int*)&s_error == 0) ? 1 : 0;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\t"
          "setp.ne.b32 q, %1, 0;\n\t"
          "bar.red.and.pred p, 1, 320, q;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(go) : "r"(mine) : "memory");
    }
    if (go) {
      const bool vec = g.N % 4 == 0 && g.ldc % 4 == 0 && ((uintptr_t)g.C & 15) == 0;
      qr_write<MODE>(g, reinterpret_cast<const float*>(base), warp - 2, lane, n0, row0, cnt, vec);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_error) {
    // give copies and MMAs that may still be in flight time to land before shared memory and TMEM are released
    if (threadIdx.x == 0 && g.error_flag) atomicExch(g.error_flag, 1);
    const long long t0 = clock64();
    while ((unsigned long long)(clock64() - t0) < 200000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(NCOLS) : "memory");
}

}  // namespace tc_detail

// a dense block of rows, or pieces of at most 128 rows (seg_off, seg_cnt, seg_w) each with one of n_w matrices
inline bool gemm_tcq_rows_supported(const GemmArgs& g) {
  const long long row_bytes = g.wq == 1 ? g.ldw : g.ldw / 2;
  return g.wq >= 1 && g.wq <= 3 && g.M >= 1 && g.a_rows == nullptr && g.ldw_k == 1 && g.K >= 64 && g.K % 64 == 0 && g.ldw == g.K && g.lda % 8 == 0 &&
         row_bytes % 16 == 0 && ((uintptr_t)g.A & 15) == 0 && ((uintptr_t)g.W & 15) == 0 && g.w_scale != nullptr && g.bias == nullptr && !g.post && !g.mul &&
         (g.epi == EPI_STORE || g.epi == EPI_SWIGLU || (g.epi == EPI_ADD && !g.c_bf16)) && (g.seg_cnt ? g.n_w >= 1 : g.nseg == 1) &&
         tc_detail::encode_fn() != nullptr;
}

template <int QMODE>
inline int32_t launch_gemm_tcq_rows_mode(vn_ctx* ctx, const GemmArgs& g, long long a_rows_total, int* error_flag) {
  using namespace tc_detail;
  constexpr int RAW_ROW = QMODE == 1 ? BK : BK / 2;
  const long long row_bytes = QMODE == 1 ? g.K : g.K / 2, seg_rows_w = g.seg_cnt ? g.w_stride / g.ldw : 0;
  const long long w_rows = g.seg_cnt ? (long long)(g.n_w - 1) * seg_rows_w + g.N : g.N;
  CUtensorMap tm_w, tm_x;
  if (!make_raw_map(&tm_w, g.W, w_rows, row_bytes, RAW_ROW) || !make_map(&tm_x, g.A, a_rows_total, g.K, g.lda, QR_ROWS))
    return vn_fail(ctx, VN_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  TcArgs a = {};
  a.C = g.C; a.ldc = g.ldc; a.M = g.M; a.N = g.N; a.K = g.K; a.epi = g.epi; a.c_bf16 = g.c_bf16; a.act = g.act; a.act_limit = g.act_limit;
  a.seg_off = g.seg_off; a.seg_cnt = g.seg_cnt; a.seg_w = g.seg_w; a.w_rows_per_seg = seg_rows_w; a.error_flag = error_flag;
  int nseg = g.nseg;
  if (!g.seg_cnt) {                                     // blocks of equal length
    nseg = ceil_div(g.M, QR_ROWS);
    a.seg_rows = (ceil_div(g.M, nseg) + 15) & ~15; a.rows_all = g.M;
    nseg = ceil_div(g.M, a.seg_rows);
  }
  if (nseg > 65535) return vn_fail(ctx, VN_ERR_UNSUPPORTED, "too many rows for the quantised GEMM");
  constexpr int stage = (BF + QR_ROWS) * BK * 2 + BF * RAW_ROW, most = QMODE == 1 ? 5 : 6;      // 200 or 216 KB
  static_assert(most <= QR_CONV, "a converting warp per stage");
  const int stages = std::max(2, std::min(most, g.K / BK));
  const size_t smem = (size_t)stages * stage + 1024;
  static unsigned long long attr_set = 0;
  if (!((attr_set >> (ctx->device & 63)) & 1ull)) {
    VN_CUDA(ctx, cudaFuncSetAttribute(gemm_tcq_rows_kernel<QMODE, TC_STORE>, cudaFuncAttributeMaxDynamicSharedMemorySize, most * stage + 1024));
    VN_CUDA(ctx, cudaFuncSetAttribute(gemm_tcq_rows_kernel<QMODE, TC_SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, most * stage + 1024));
    VN_CUDA(ctx, cudaFuncSetAttribute(gemm_tcq_rows_kernel<QMODE, TC_ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, most * stage + 1024));
    attr_set |= 1ull << (ctx->device & 63);
  }
  dim3 grid(ceil_div(g.N, BF), 1, nseg);
  const char* name = g.tag ? g.tag : "gemm_tcq_rows_kernel";
  if (g.epi == EPI_SWIGLU)
    VN_LAUNCH_PDL_LEVEL(ctx, 1, name, (gemm_tcq_rows_kernel<QMODE, TC_SWIGLU>), grid, QR_THREADS, smem, tm_w, tm_x, a, g.w_scale, g.ws_stride, stages);
  else if (g.epi == EPI_ADD)
    VN_LAUNCH_PDL_LEVEL(ctx, 1, name, (gemm_tcq_rows_kernel<QMODE, TC_ADD>), grid, QR_THREADS, smem, tm_w, tm_x, a, g.w_scale, g.ws_stride, stages);
  else
    VN_LAUNCH_PDL_LEVEL(ctx, 1, name, (gemm_tcq_rows_kernel<QMODE, TC_STORE>), grid, QR_THREADS, smem, tm_w, tm_x, a, g.w_scale, g.ws_stride, stages);
  return VN_OK;
}

// a_rows_total: number of valid rows behind g.A
inline int32_t launch_gemm_tcq_rows(vn_ctx* ctx, const GemmArgs& g, long long a_rows_total, int* error_flag) {
  if (g.M <= 0 || g.N <= 0) return VN_OK;
  if (g.wq == 1) return launch_gemm_tcq_rows_mode<1>(ctx, g, a_rows_total, error_flag);
  if (g.wq == 2) return launch_gemm_tcq_rows_mode<2>(ctx, g, a_rows_total, error_flag);
  return launch_gemm_tcq_rows_mode<3>(ctx, g, a_rows_total, error_flag);
}

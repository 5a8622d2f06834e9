// Dense GEMM of many rows (prompts) on pairs of SMs: tcgen05.mma with cta_group::2.
//
// The one-SM kernel of gemm_tc.cuh brings 48 KB into shared memory for 128 features x 256 rows of a k block and reads as much
// again for the MMAs: at the MMA rate 192 bytes a clock, where shared memory gives 128.  Here two CTAs of a cluster share a tile
// of 256 features x 256 rows: each loads its own 128 features and HALF of the rows, the tensor cores of both read both halves,
// and the bytes per product fall by a third.  8192 x 2048 x 8192 385 -> 227 us (1213 TFLOP/s); what TMA brings rises from 8.4 to
// 9.5 TB/s over all SMs, most of it from L2, so neither kernel is at a fixed ceiling of that path.
//
// One cluster per SM pair walks the tiles (persistent); accumulators are double buffered in TMEM (2 x 256 columns), so a tile's
// epilogue runs under the next tile's MMAs.  Per CTA: warp 0 TMA, warp 1 MMA (issued by the cluster's first CTA for both),
// warps 2..9 epilogue in two groups.  Barriers: bar_full lives in the first CTA and counts both CTAs' copies; bar_empty and
// acc_full are in each CTA, signalled by multicast commits; acc_empty is in the first CTA and counts both CTAs' epilogue warps.
// Every wait is bounded, and the CTAs of a pair leave together.
#pragma once
#include "gemm_tc.cuh"

namespace tc_detail {

constexpr int P2_STAGES = 5, P2_STAGE = 32 * 1024, P2_STAGING = 64 * 1024;   // stage: 128 features and up to 128 rows of 64 k

__device__ __forceinline__ unsigned cluster_addr(const void* p, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
// waits on a barrier that the other CTA of the pair arrives at too
__device__ __forceinline__ bool mbar_wait_pair(unsigned long long* bar, unsigned parity) {
  const long long t0 = clock64();
  const unsigned long long limit = g_wait_limit_cycles;
  for (;;) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((unsigned long long)(clock64() - t0) > limit) return false;
  }
}
__device__ __forceinline__ void mbar_arrive_at(unsigned cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// a load of one CTA of the pair that counts at a barrier of either
__device__ __forceinline__ void tma_load_pair(void* smem_dst, const CUtensorMap* tmap, unsigned cluster_bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(cluster_bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(unsigned tmem_d, unsigned long long da, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives at the same barrier of both CTAs when the MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((unsigned short)3) : "memory");
}

// Gated pairs of a 32-row chunk in 16 bits, straight from the accumulator's registers: gate and up of a pair are neighbouring lanes, so
// the even lane takes rows 0..15 and the odd one 16..31; a row's 16 results of a warp are one 32-byte sector.
__device__ __forceinline__ void pair_glu_chunk(const TcArgs& g, const unsigned (&r)[32], int ch, int q, int lane, int n0, int row0, int cnt) {
  const int n = n0 + q * 32 + (lane & ~1), odd = lane & 1, first = ch * 32 + odd * 16;
  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(g.C) + (long long)(row0 + first) * g.ldc + (n >> 1);
  const int rows = n + 1 < g.N ? cnt - first : 0;
  with_glu(g.act, [&](auto tag) {
    float v[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const float lo = __uint_as_float(r[t]), hi = __uint_as_float(r[t + 16]);
      const float other = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
      v[t] = glu_of<decltype(tag)::act>(odd ? other : lo, odd ? hi : other, g.act_limit, true);
    }
#pragma unroll
    for (int t = 0; t < 16; ++t)
      if (t < rows) dst[(long long)t * g.ldc] = __float2bfloat16_rn(v[t]);
  });
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
gemm_tc2_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_out, TcArgs g,
                int tiles_x, int tiles_total) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ unsigned long long bar_full[P2_STAGES], bar_empty[P2_STAGES], acc_full[2], acc_empty[2];
  __shared__ unsigned tmem_base_slot;
  __shared__ int s_error;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned rank = cluster_rank();
  const int cluster = blockIdx.x >> 1, n_cluster = gridDim.x >> 1;
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* stages = base + P2_STAGING;
  const int nkb = (g.K + BK - 1) / BK;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < P2_STAGES; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }     // eight warps of each CTA
    s_error = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();                                   // both CTAs' barriers are initialised, both have their columns
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = tmem_base_slot;
  pdl_wait();

  // every role of both CTAs walks the same tiles; ntok: rows of the product, both halves alike
  auto tile = [&](int id, int& z, int& n0, int& row0, int& cnt, int& ntok) {
    z = id / tiles_x;
    n0 = (id - z * tiles_x) * (2 * BF) + (int)rank * BF;
    if (g.seg_cnt) { row0 = g.seg_off[z]; cnt = g.seg_cnt[z]; }
    else { row0 = z * g.seg_rows; cnt = min(g.seg_rows, g.rows_all - row0); }
    if (cnt > 2 * BF) cnt = 2 * BF;
    ntok = (cnt + 31) & ~31;
  };

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      unsigned ph = 0;
      bool ok = true;
      for (int id = cluster; id < tiles_total && ok; id += n_cluster) {
        int z, n0, row0, cnt, ntok;
        tile(id, z, n0, row0, cnt, ntok);
        if (cnt <= 0) continue;
        const int w_row = (int)((long long)(g.seg_w ? g.seg_w[z] : z) * g.w_rows_per_seg) + n0;
        const int x_row = row0 + (int)rank * (ntok >> 1);
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait_pair(&bar_empty[s], ph ^ 1u)) { s_error = 1; ok = false; break; }
          unsigned char* st = stages + (size_t)s * P2_STAGE;
          if (rank == 0) mbar_expect_tx(&bar_full[s], 2u * P2_STAGE);       // both CTAs' boxes, always whole
          const unsigned full = cluster_addr(&bar_full[s], 0);
          tma_load_pair(st, &tm_w, full, kb * BK, w_row);
          tma_load_pair(st + BF * BK * 2, &tm_x, full, kb * BK, x_row);
          if (++s == P2_STAGES) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      int s = 0, t = 0;
      unsigned ph = 0;
      bool ok = true;
      for (int id = cluster; id < tiles_total && ok; id += n_cluster) {
        int z, n0, row0, cnt, ntok;
        tile(id, z, n0, row0, cnt, ntok);
        if (cnt <= 0) continue;
        const int buf = t & 1;
        if (!__all_sync(0xffffffffu, mbar_wait_pair(&acc_empty[buf], ((t >> 1) & 1) ^ 1))) { s_error = 1; break; }
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(ntok >> 3) << 17) | ((unsigned)(2 * BF >> 4) << 24);
        for (int kb = 0; kb < nkb; ++kb) {
          if (!__all_sync(0xffffffffu, mbar_wait_pair(&bar_full[s], ph))) { s_error = 1; ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          unsigned char* st = stages + (size_t)s * P2_STAGE;
          const unsigned long long da = umma_desc(st), db = umma_desc(st + BF * BK * 2);
          if (elect_one()) {
#pragma unroll
            for (int k4 = 0; k4 < BK / 16; ++k4)
              umma_bf16_pair(tmem_base + (unsigned)buf * 256u, da + 2ull * k4, db + 2ull * k4, idesc, (kb | k4) != 0);
            umma_commit_pair(&bar_empty[s]);
          }
          __syncwarp();
          if (++s == P2_STAGES) { s = 0; ph ^= 1u; }
        }
        if (ok && elect_one()) umma_commit_pair(&acc_full[buf]);   // an unfinished tile is nobody's: both CTAs' epilogues give up
        __syncwarp();
        ++t;
      }
    }
  } else {
    const int q = warp & 3, grp = (warp - 2) >> 2;
    const bool issuer = ((warp - 2) & 3) == 0 && lane == 0;
    const bool vec_ok = g.ldc % 4 == 0 && g.N % 4 == 0 && ((uintptr_t)g.C & 15) == 0;
    const bool swi_ok = MODE == TC_SWIGLU && g.ldc % 4 == 0 && g.N % 4 == 0 && ((uintptr_t)g.C & 7) == 0;
    int t = 0, chunk_no = 0;
    for (int id = cluster; id < tiles_total; id += n_cluster) {
      int z, n0, row0, cnt, ntok;
      tile(id, z, n0, row0, cnt, ntok);
      if (cnt <= 0) continue;
      const int buf = t & 1;
      const bool acc_ok = mbar_wait_pair(&acc_full[buf], (t >> 1) & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!acc_ok) s_error = 1;
      int go;                                           // one decision for the eight warps: their stores synchronise them
      {
        const int mine = (acc_ok && *(volatile int*)&s_error == 0) ? 1 : 0;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 q, %1, 0;\n\t"
            "bar.red.and.pred p, 1, 256, q;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(go) : "r"(mine) : "memory");
      }
      if (!go) break;
      // chunk_no counts staged chunks only: the wait before a tensor store lets the last one read on, so the next has to take the
      // other staging tile, whatever was left out in between
      const int nchunk = n0 < g.N ? (cnt + 31) >> 5 : 0;   // the pair's second CTA may have no features
      for (int ch = grp; ch < nchunk; ch += 2, ++chunk_no) {
        unsigned r[32];
        tmem_ld32(tmem_base + (unsigned)buf * 256u + ((unsigned)(q * 32) << 16) + (unsigned)(ch * 32), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (MODE == TC_SWIGLU && g.c_bf16) {
          pair_glu_chunk(g, r, ch, q, lane, n0, row0, cnt);
        } else if (MODE == TC_STORE && g.tma_out && ch * 32 + 32 <= cnt) {
          // whole chunks of fp32 rows leave as asynchronous tensor stores (a partial one would write the next segment's rows)
          float* tile_out = reinterpret_cast<float*>(base + grp * (32 * 1024) + (chunk_no & 1) * (16 * 1024));
          if (issuer) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // the store before last has read this tile
          asm volatile("bar.sync %0, 128;" ::"r"(2 + grp) : "memory");
          const int f = q * 32 + lane;
          const float bias = g.bias && n0 + f < g.N ? g.bias[n0 + f] : 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) tile_out[i * BF + f] = __uint_as_float(r[i]) + bias;
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("bar.sync %0, 128;" ::"r"(2 + grp) : "memory");
          if (issuer) {
            tma_store_3d(&tm_out, tile_out, n0, row0 + ch * 32, 0);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        } else {
          if (MODE == TC_STORE && g.tma_out) {           // the staging tiles are shared with the stores in flight
            if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            asm volatile("bar.sync %0, 128;" ::"r"(2 + grp) : "memory");
          }
          tc_epilogue_chunk<MODE>(g, r, base + grp * (32 * 1024), ch, chunk_no & 1, 2 + grp, q, lane, n0, row0, cnt, 0, vec_ok, swi_ok);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_at(cluster_addr(&acc_empty[buf], 0));
      ++t;
    }
    // the staging tiles must have been read before the CTA gives its shared memory back
    if (MODE == TC_STORE && g.tma_out && issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_error) {
    // give copies and MMAs that may still be in flight time to land before shared memory and TMEM are released
    if (threadIdx.x == 0 && g.error_flag) atomicExch(g.error_flag, 1);
    const long long t0 = clock64();
    while ((unsigned long long)(clock64() - t0) < 200000000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();                                   // nobody leaves while the other may still use its memory or barriers
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

}  // namespace tc_detail

// rows as equal segments of one matrix (seg_rows) or pieces of at most 256 rows with a matrix each (seg_off, seg_cnt, seg_w)
inline bool gemm_tc2_supported(const GemmArgs& g) {
  return (g.seg_w || (g.seg_rows > 0 && !g.seg_cnt)) && !g.a_rows && !g.mul && g.ldw_k == 1 && g.K >= 1 && g.K % 8 == 0 && g.lda % 8 == 0 && g.ldw % 8 == 0 &&
         ((uintptr_t)g.A & 15) == 0 && ((uintptr_t)g.W & 15) == 0 && (g.epi == EPI_STORE || g.epi == EPI_ADD || (g.epi == EPI_SWIGLU && !g.bias)) &&
         (!g.post || g.c_bf16) && tc_detail::encode_fn() != nullptr;
}

inline int32_t launch_gemm_tc2(vn_ctx* ctx, const GemmArgs& g, long long a_rows_total, int seg_rows, int* error_flag) {
  using namespace tc_detail;
  CUtensorMap tm_w, tm_x;
  const long long w_rows = g.seg_cnt ? (long long)(g.n_w - 1) * (g.w_stride / g.ldw) + g.N : g.N;
  if (!make_map(&tm_w, g.W, w_rows, g.K, g.ldw, BF) || !make_map(&tm_x, g.A, a_rows_total, g.K, g.lda, BF))
    return vn_fail(ctx, VN_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  TcArgs a = {};
  a.C = g.C; a.bias = g.bias; a.ldc = g.ldc; a.M = g.M; a.N = g.N; a.K = g.K; a.epi = g.epi; a.c_bf16 = g.c_bf16;
  a.act = g.act; a.act_limit = g.act_limit; a.post = g.post; a.post_n = g.post_n; a.error_flag = error_flag;
  a.seg_off = g.seg_off; a.seg_cnt = g.seg_cnt; a.seg_w = g.seg_w; a.w_rows_per_seg = g.seg_cnt ? g.w_stride / g.ldw : 0;
  long long nseg = g.nseg;
  if (!g.seg_cnt) {                                     // segments of equal length
    nseg = ceil_div(a_rows_total, (long long)seg_rows);
    a.seg_rows = (int)((ceil_div(a_rows_total, nseg) + 31) & ~31ll); a.rows_all = (int)a_rows_total;
    nseg = ceil_div(a_rows_total, (long long)a.seg_rows);
  }
  CUtensorMap tm_out = tm_x;                            // placeholder when unused
  if (g.epi == EPI_STORE && !g.c_bf16 && !g.seg_cnt && g.N >= BF && g.N % 4 == 0 && g.ldc % 4 == 0 && ((uintptr_t)g.C & 15) == 0 &&
      make_out_map(&tm_out, reinterpret_cast<const float*>(g.C), g.N, a_rows_total, 1, g.ldc, a_rows_total * g.ldc))
    a.tma_out = 1;
  const int tiles_x = ceil_div(g.N, 2 * BF);
  const long long tiles = nseg * tiles_x;
  if (tiles >= (1ll << 30)) return vn_fail(ctx, VN_ERR_UNSUPPORTED, "too many tiles");
  constexpr int smem = P2_STAGES * P2_STAGE + P2_STAGING + 1024;
  static unsigned long long attr_set = 0;
  if (!((attr_set >> (ctx->device & 63)) & 1ull)) {
    VN_CUDA(ctx, cudaFuncSetAttribute(gemm_tc2_kernel<TC_STORE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    VN_CUDA(ctx, cudaFuncSetAttribute(gemm_tc2_kernel<TC_SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    VN_CUDA(ctx, cudaFuncSetAttribute(gemm_tc2_kernel<TC_ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set |= 1ull << (ctx->device & 63);
  }
  const int grid = 2 * (int)std::min<long long>(tiles, ctx->sm_count / 2);
  const char* name = g.tag ? g.tag : "gemm_tc2_kernel";
  if (g.epi == EPI_SWIGLU) VN_LAUNCH_PDL_LEVEL(ctx, 1, name, gemm_tc2_kernel<TC_SWIGLU>, grid, TC_THREADS, smem, tm_w, tm_x, tm_out, a, tiles_x, (int)tiles);
  else if (g.epi == EPI_ADD) VN_LAUNCH_PDL_LEVEL(ctx, 1, name, gemm_tc2_kernel<TC_ADD>, grid, TC_THREADS, smem, tm_w, tm_x, tm_out, a, tiles_x, (int)tiles);
  else VN_LAUNCH_PDL_LEVEL(ctx, 1, name, gemm_tc2_kernel<TC_STORE>, grid, TC_THREADS, smem, tm_w, tm_x, tm_out, a, tiles_x, (int)tiles);
  return VN_OK;
}

// Whether the pair kernel ends before the one-SM kernel, which takes segments of g.M rows.  Both kernels' time goes in rounds over the
// SMs.  A round of the one-SM kernel with segments of 32, 64 or 128 rows takes about 0.52, 0.58 or 0.7 of one with 256 rows.  The
// pair kernel's round takes 0.9 of that of 256 rows for stores and gated pairs (its last half tile of 128 features counts whole:
// 8192 x 1152 x 1024, three rounds against two, 28 us against 19; 16384 x 5504 x 1024 gated, 20 against 19, 169 against 212),
// 0.85 where it adds to the residual, which costs the other kernel most, and 0.7 in tiles of 128 rows.  Measured over 12 widths, K
// of 64 to 2752 and 257 to 8192 rows: the kernel
// chosen here was never more than 5 % the slower one.
//  - Two rounds of pairs for stores and gated pairs, and 384 rows: 300 x 32000 x 512 stored 21.4 against 23.0 us.  From 12 tiles where it adds.
//  - K: of short products the pair kernel's start and its write-out are the longer ones (one-SM against pair, 2048 rows x 8192).  Stored in
//    32 bits, K = 128 19.3 against 22.6 us, K = 512 26.7 against 26.2; gated, K = 192 25.0 against 25.9, K = 256 25.8 against 26.0, 1024
//    38 against 36; stored in 16 bits, K = 512 29.3 against 33.6, K = 1024 38.9 against 38.8; added, 2048 x 1152, K = 192 10.0
//    against 10.9, K = 256 11.0 against 11.1, K = 512 14.1 against 12.5.
// Experts' rows: the pieces that must exist, not those that may.
inline bool gemm_tc2_pays(const vn_ctx* ctx, const GemmArgs& g, long long rows) {
  using namespace tc_detail;
  const bool add = g.epi == EPI_ADD;
  const long long sm = ctx->sm_count, pairs = sm / 2, pieces = ceil_div(rows, 256ll), tiles = ceil_div(g.N, 2 * BF) * pieces;
  if (g.K < (add || g.epi == EPI_SWIGLU ? 256 : g.c_bf16 ? 1024 : 512) || tiles < (add ? 12 : 2 * pairs) || (!add && rows <= 384)) return false;
  const double one = (double)ceil_div(ceil_div(g.N, BF) * (g.seg_cnt ? pieces : (long long)g.nseg), sm) * (g.M > 128 ? 1.0 : g.M > 64 ? 0.7 : g.M > 32 ? 0.58 : 0.52);
  const double two = 2 * tiles <= pairs ? 0.7 : (double)ceil_div(tiles, pairs) * (add ? 0.85 : 0.9);
  return two <= one;
}

// Many rows, either kernel.  Rows in tiles of 128 where those of 256 leave half of the pairs idle.
inline int32_t launch_gemm_many(vn_ctx* ctx, const GemmArgs& g, long long a_rows_total, TcPlan& plan) {
  if (gemm_tc2_supported(g) && gemm_tc2_pays(ctx, g, a_rows_total)) {
    const long long tiles = ceil_div(g.N, 2 * tc_detail::BF) * ceil_div(a_rows_total, 256ll);
    return launch_gemm_tc2(ctx, g, a_rows_total, 4 * tiles <= ctx->sm_count ? 128 : 256, plan.error_flag);
  }
  return launch_gemm_tc(ctx, g, a_rows_total, plan);
}

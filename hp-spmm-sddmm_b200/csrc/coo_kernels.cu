// FP32 COO SpMM for sm_100a: C += A * B from (row, col, val) triples in any order; zero-valued triples (the
// padding) are skipped.  Replaces the reference's LBSpMM (spmm/mm/spmm_kernel.cu:428-477, :733-768).
//
// Same machinery as the CSR product (spmm_warp.cuh): one warp per S consecutive triples, G = 32 / W lane groups
// that each gather a fragment of a row of B per step, tiles of 32 triples staged global -> shared with cp.async two
// tiles ahead, U steps of gathers in flight, an unrolled path for tiles that lie inside one row.  Row boundaries
// come from the staged row ids (one ballot per tile) instead of row_ptr; every run of equal row ids ends in one
// cross-group reduction and vector reductions into C.
#include "device_utils.cuh"
#include "hpspmm_internal.h"
#include "warp_frag.cuh"

namespace {

using namespace hpspmm;

template <int VEC, int W, int R, int U, int KS, int BT, int MINB>
__global__ void __launch_bounds__(BT, MINB)
spmm_coo_warp_kernel(int64_t nnz, int S, const int* __restrict__ row_idx, const int* __restrict__ col_idx,
                     const float* __restrict__ vals, const float* __restrict__ B, float* __restrict__ C, int ld, int off0, int cols) {
  constexpr int CW = VEC * W * R;
  constexpr int G = 32 / W;
  constexpr int T = 32;
  constexpr int BATCH = U * G;
  constexpr int STAGES = 2;
  static_assert(BATCH <= T && T % BATCH == 0, "batch must tile the staged tile");
  __shared__ int2 cv_tiles[BT / 32][STAGES][T];
  __shared__ int row_tiles[BT / 32][STAGES][T];

  chain_grid();
  const int lane = threadIdx.x & 31;
  const int g = lane / W, l = lane % W;
  const int64_t worker = ((int64_t)blockIdx.x * BT + threadIdx.x) >> 5;
  const int64_t n0 = worker * S;
  if (n0 >= nnz) return;
  const int64_t n1 = min(nnz, n0 + (int64_t)S);
  int2(*cv)[T] = cv_tiles[threadIdx.x >> 5];
  int(*rw)[T] = row_tiles[threadIdx.x >> 5];
  const int off = KS ? 0 : off0 + (int)blockIdx.y * CW;   // slabs of the columns [off0, off0 + cols)
  const int kw = KS ? CW : min(CW, cols - (int)blockIdx.y * CW);

  auto stage_tile = [&](int stage, int64_t base) {
    const int64_t j = base + lane;
    if (j < n1) {
      cp_async_4(&cv[stage][lane].x, col_idx + j);
      cp_async_4(&cv[stage][lane].y, vals + j);
      cp_async_4(&rw[stage][lane], row_idx + j);
    } else {
      cv[stage][lane] = make_int2(0, 0);   // past the chunk: column 0, value 0 (skipped)
      rw[stage][lane] = -1;
    }
    cp_async_commit();
  };
  stage_tile(0, n0);
  stage_tile(1, n0 + T);

  float acc[R][VEC];
  auto clear = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int x = 0; x < VEC; ++x) acc[r][x] = 0.f;
  };
  clear();
  const bool live_last = KS || ((R - 1) * W + l) * VEC < kw;
  const unsigned stride = (KS ? KS : ld) * 4u;
  const char* Bl = reinterpret_cast<const char*>(B + off + ((R > 1 || live_last) ? l * VEC : kw - VEC));
  const char* Bl_last = reinterpret_cast<const char*>(B + off + (live_last ? ((R - 1) * W + l) * VEC : kw - VEC));
  float* Cs = C + off;
  const int64_t ldc = KS ? KS : ld;
  int cur_row = -1;   // row of the run being accumulated

  auto gather = [&](float (&b)[R][VEC], int col) {
    const char* p = Bl + (uint64_t)(unsigned)col * stride;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (R > 1 && r == R - 1)
        gather_vec<VEC, false>(b[r], reinterpret_cast<const float*>(Bl_last + (uint64_t)(unsigned)col * stride), 0ull);
      else
        gather_vec<VEC, false>(b[r], reinterpret_cast<const float*>(p) + r * W * VEC, 0ull);
    }
  };
  auto fma = [&](float v, const float (&b)[R][VEC]) {
    if (v != 0.f)
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int x = 0; x < VEC; ++x) acc[r][x] = fmaf(v, b[r][x], acc[r][x]);
  };
  auto flush = [&]() {
    if (cur_row >= 0) {   // warp-uniform
      float* crow = Cs + (int64_t)cur_row * ldc;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool live = r < R - 1 || live_last;
        if (group_split<VEC, W>::REST == 0 && G <= 2) {
          // the groups split the sum: at K = 64 every lane adds a float2 (0.378 -> 0.365 ms on the R-MAT bench
          // graph).  With more groups many narrow reductions per row cost more than the shuffles they save
          // (K = 32: 0.233 -> 0.236 ms), so one group adds whole vectors.
          float v[group_split<VEC, W>::KEEP];
          combine_groups<VEC, W>(acc[r], v, lane);
          if (live) reduce_into(crow + r * W * VEC + group_split<VEC, W>::column(lane), v);
        } else {
          all_reduce_groups<VEC, W>(acc[r]);
          if (g == 0 && live) reduce_into(crow + (r * W + l) * VEC, acc[r]);
        }
      }
    }
    clear();
  };

  int stage = 0;
  for (int64_t base = n0; base < n1; base += T) {
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    // bit e: triple e of the tile starts a new run (its row differs from its predecessor's);
    // triples past the chunk carry row -1 and never match, which ends the last run
    const int my_row = rw[stage][lane];
    const int prev_row = lane == 0 ? cur_row : rw[stage][lane - 1];
    const unsigned bnd = __ballot_sync(0xffffffffu, my_row != prev_row);
    const int2* tile = &cv[stage][g];
    if (bnd == 0u) {
      // the whole tile continues the current run.  One batch at a time: unrolled further the compiler hoists gathers
      // until it spills (4 M triples, K = 64: 0.094 ms unrolled, 0.078 ms one batch at a time at 56 registers).
#pragma unroll(VEC == 4 ? 1 : 2)
      for (int s0 = 0; s0 < T / G; s0 += U) {
        float b[U][R][VEC];
        float v[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int2 e = tile[(s0 + i) * G];
          v[i] = __int_as_float(e.y);
          gather(b[i], e.x);
        }
#pragma unroll
        for (int i = 0; i < U; ++i) fma(v[i], b[i]);
      }
    } else {
      const int limit = (int)min((int64_t)T, n1 - base);   // triples of this tile inside the chunk
#pragma unroll 1
      for (int u0 = 0; u0 < T; u0 += BATCH) {
        if (u0 >= limit) break;
        float b[U][R][VEC];
        float v[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int2 e = tile[u0 + i * G];
          v[i] = __int_as_float(e.y);
          gather(b[i], e.x);
        }
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int lo = u0 + i * G;
          const int hi = min(lo + G, limit);
          const int mine = lo + g;
          int cur = lo;
          // warp-uniform: runs that start inside this step
          unsigned m = hi > lo ? (bnd >> lo) & (0xffffffffu >> (32 - (hi - lo))) : 0u;
          while (m) {
            const int p = lo + __ffs(m) - 1;
            m &= m - 1;
            if (mine >= cur && mine < p) fma(v[i], b[i]);
            flush();
            cur_row = rw[stage][p];
            cur = p;
          }
          if (mine >= cur && mine < hi) fma(v[i], b[i]);
        }
      }
    }
    // the last triple's row carries into the next tile's first comparison
    __syncwarp();
    stage_tile(stage, base + STAGES * T);
    stage ^= 1;
  }
  cp_async_wait<0>();
  flush();
}

struct coo_args {
  int64_t nnz;
  int S, K, off, cols;
  const int32_t *row_idx, *col_idx;
  const float *vals, *B;
  float* C;
};

template <int VEC, int W, int R, int U, int KS, int MINB>
int launch_coo(hpspmm_ctx* ctx, const coo_args& a, cudaStream_t s) {
  constexpr int BT = 64, CW = VEC * W * R;
  const int64_t workers = (a.nnz + a.S - 1) / a.S;
  const int64_t blocks = (workers + BT / 32 - 1) / (BT / 32);
  const int64_t slabs = (a.cols + CW - 1) / CW;
  if (blocks > 2147483647ll || slabs > 65535) return HPSPMM_ERR_UNSUPPORTED;
  if (!hpspmm_shape_covers(VEC, W, R, a.cols)) return HPSPMM_ERR_INVALID;
  hpspmm_launch(spmm_coo_warp_kernel<VEC, W, R, U, KS, BT, MINB>, dim3((unsigned)blocks, (unsigned)slabs), BT, 0, s,
                a.nnz, a.S, a.row_idx, a.col_idx, a.vals, a.B, a.C, a.K, a.off, a.cols);
  ctx->launches++;
  HPSPMM_CUDA_TRY(ctx, cudaGetLastError());
  return HPSPMM_OK;
}

int launch_coo_shape(hpspmm_ctx* ctx, const coo_args& a, const hpspmm_spmm_shape& sh, cudaStream_t s) {
#define GO(V, W, R, U, KS, MINB) return launch_coo<V, W, R, U, KS, MINB>(ctx, a, s)
  if (sh.VEC == 4) {
    if (a.K == 32) GO(4, 8, 1, 4, 32, 16);
    if (a.K == 64) GO(4, 16, 1, 4, 64, 18);
    if (a.K == 128) GO(4, 32, 1, 4, 128, 18);
    if (sh.W == 2) GO(4, 2, 1, 2, 0, 16);
    if (sh.W == 4) GO(4, 4, 1, 4, 0, 16);
    if (sh.W == 8) GO(4, 8, 1, 4, 0, 16);
    if (sh.W == 16 && sh.R == 3) GO(4, 16, 3, 2, 0, 16);
    if (sh.W == 16) GO(4, 16, 1, 4, 0, 16);
    if (sh.R == 1) GO(4, 32, 1, 4, 0, 16);
    if (sh.R == 2) GO(4, 32, 2, 2, 0, 16);
    if (sh.R == 3) GO(4, 32, 3, 2, 0, 12);
    GO(4, 32, 4, 1, 0, 12);
  }
  if (sh.VEC == 2) {
    if (sh.W == 2) GO(2, 2, 1, 2, 0, 16);
    if (sh.W == 4) GO(2, 4, 1, 4, 0, 16);
    if (sh.W == 8) GO(2, 8, 1, 8, 0, 16);
    if (sh.W == 16 && sh.R == 3) GO(2, 16, 3, 4, 0, 16);
    if (sh.W == 16) GO(2, 16, 1, 8, 0, 16);
    if (sh.R == 1) GO(2, 32, 1, 8, 0, 16);
    if (sh.R == 2) GO(2, 32, 2, 4, 0, 16);
    if (sh.R == 3) GO(2, 32, 3, 2, 0, 16);
    GO(2, 32, 4, 2, 0, 16);
  }
  if (sh.W == 1) GO(1, 1, 1, 1, 0, 16);
  if (sh.W == 4) GO(1, 4, 1, 4, 0, 16);
  if (sh.W == 8) GO(1, 8, 1, 8, 0, 16);
  if (sh.W == 16 && sh.R == 3) GO(1, 16, 3, 4, 0, 16);
  if (sh.W == 16) GO(1, 16, 1, 8, 0, 16);
  if (sh.R == 1) GO(1, 32, 1, 8, 0, 16);
  if (sh.R == 2) GO(1, 32, 2, 8, 0, 16);
  if (sh.R == 3) GO(1, 32, 3, 4, 0, 16);
  if (sh.R == 4) GO(1, 32, 4, 4, 0, 16);
  if (sh.R == 5) GO(1, 32, 5, 2, 0, 16);
  if (sh.R == 6) GO(1, 32, 6, 2, 0, 16);
  if (sh.R == 7) GO(1, 32, 7, 2, 0, 16);
  GO(1, 32, 8, 2, 0, 16);
#undef GO
}

}  // namespace

extern "C" int hpspmm_spmm_coo_f32(hpspmm_ctx* ctx, int64_t M, int64_t N, int64_t K, int64_t nnz_padded,
                                   const int32_t* row_idx, const int32_t* col_idx, const float* vals, const float* B,
                                   float* C, const hpspmm_opts* opts, hpspmm_stream stream) {
  HPSPMM_TRACE("hpspmm_spmm_coo_f32");
  HPSPMM_REQUIRE(ctx, ctx != nullptr, "null context");
  HPSPMM_REQUIRE(ctx, M >= 0 && N >= 0 && nnz_padded >= 0 && K >= 1, "bad size");
  if (nnz_padded == 0 || M == 0) return HPSPMM_OK;
  HPSPMM_REQUIRE(ctx, row_idx && col_idx && vals && B && C, "null operand");
  if ((K & 3) == 0 && (((uintptr_t)B & 15u) || ((uintptr_t)C & 15u))) {
    snprintf(ctx->err, sizeof(ctx->err), "dense operands must be 16-byte aligned");
    return HPSPMM_ERR_INVALID;
  }
  if (K > (1 << 20) * 16ll) return HPSPMM_ERR_UNSUPPORTED;
  hpspmm_device_guard guard(ctx->device);
  int32_t S = (opts && opts->chunk_nnz > 0) ? opts->chunk_nnz : hpspmm_coo_chunk_nnz(K, nnz_padded);
  S = (S + 31) / 32 * 32;
  coo_args a = {nnz_padded, S, (int)K, 0, 0, row_idx, col_idx, vals, B, C};
  const int VEC = hpspmm_vector_width(K, (uintptr_t)B | (uintptr_t)C);
  for (a.off = 0; a.off < a.K; a.off += a.cols) {   // every slab accumulates into its own columns
    a.cols = hpspmm_launch_cols(a.K, a.off, hpspmm_widest_slab(VEC));
    hpspmm_spmm_shape sh = hpspmm_choose_shape(VEC, a.cols, hpspmm_widest_slab(VEC), false);
    // Three vectors per lane as in the CSR product, but only from 33 vectors on: every run of equal rows is combined over
    // the groups before it goes to C, and over four groups that costs more than the idle lanes of one (1 M entries of a
    // power-law graph, K = 96: 49.0 -> 56.0 us).  With few warps the exchange is not covered either (100 K entries,
    // K = 160: 15.1 -> 16.2 us); 8 M uniform entries, K = 160: 516 -> 442 us.
    const int64_t warps = (nnz_padded + a.S - 1) / a.S;
    if (VEC == 4 && sh.R == 3 && sh.W < 32 && (sh.W == 8 || warps < (int64_t)ctx->sm_count * 24))
      sh.R = sh.W / 8, sh.W = 32;
    const int st = launch_coo_shape(ctx, a, sh, (cudaStream_t)stream);
    if (st != HPSPMM_OK) return st;
  }
  return HPSPMM_OK;
}

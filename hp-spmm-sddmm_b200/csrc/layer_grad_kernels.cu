// Both gradients of an aggregation layer in one pass over the transpose of A:
//   dH[c, :] = sum over the entries (r, c) of A of vals * dC[r, :]      (a product with the transpose)
//   dA[j]    = dot(dC[r, :], H[c, :]) for the entry j = (r, c)          (an SDDMM over A's pattern)
// The reference has neither (its driver issues single products, test/test_all.cpp:63-107).
//
// Walking the transpose by rows, every entry (c, r) needs the row dC[r, :] for both results, and H[c, :] stays in
// registers for a whole row.  So one gather per entry serves the product and the dot product, where two kernels gather
// a row each.  What is bound to the order of A's entries -- the weights that are read, the gradients that are written --
// is reached through the transpose's permutation: a 4-byte gather and a 4-byte scatter per entry, which also takes the
// place of the kernel that carried new weights into the transpose.
#include "device_utils.cuh"
#include "hpspmm_internal.h"
#include "spmm_warp.cuh"

namespace {

using namespace hpspmm;

// KS: row stride of the dense operands when it is a compile-time constant (the width is one full slab), else 0.
template <int VEC, int W, int R, int U, int KS, int BT, int MINB>
__global__ void __launch_bounds__(BT, MINB) layer_grad_kernel(const __grid_constant__ hpspmm_layer_grad_args a) {
  constexpr int CW = VEC * W * R;
  constexpr int G = 32 / W;
  constexpr int T = 32;
  constexpr int BATCH = U * G;
  constexpr int STAGES = 2;
  static_assert(T % BATCH == 0 && (U <= W || W == 1), "batch must tile the staged tile; a lane holds one total");
  static_assert(KS == 0 || KS == CW, "a fixed stride is the width of the slab");
  __shared__ int2 tiles[BT / 32][STAGES][T];
  __shared__ int perms[BT / 32][STAGES][T];
  __shared__ int meta[BT / 32][8];

  chain_grid();
  if ((int)blockIdx.x >= a.n_chunk_blocks) {
    zero_empty_rows<KS>(a.rows, a.K, a.row_ptr, a.dH, blockIdx.x - a.n_chunk_blocks, gridDim.x - a.n_chunk_blocks, BT);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int g = lane / W;
  const int l = lane % W;
  const int slot = (int)((blockIdx.x * (unsigned)BT + threadIdx.x) >> 5);
  if (slot >= a.n_chunks) return;
  int* m = meta[threadIdx.x >> 5];
  const int4 rec0 = ld_chained(a.rec + 2 * (int64_t)slot), rec1 = ld_chained(a.rec + 2 * (int64_t)slot + 1);
  int base = rec0.x, ri = rec0.y, row = rec0.z, row_end = rec0.w;
  const int n1 = rec1.z;
  if (lane == 0) m[0] = base, m[1] = rec1.x, m[2] = row, m[3] = rec1.y, m[4] = row_end;
  const int kw = KS ? KS : a.K;
  const uint64_t policy = policy_for_gathers(a.keep);
  int2(*my)[T] = tiles[threadIdx.x >> 5];
  int(*my_perm)[T] = perms[threadIdx.x >> 5];

  // Positions in A's order are fetched one tile ahead of the weights they lead to.
  auto position = [&](int j) { return j < n1 ? ld_stream(a.perm + j) : 0; };
  int pos = position(base + lane);
  auto stage_tile = [&](int stage, int base) {
    const int j = base + lane;
    if (j < n1) {
      cp_async_4(&my[stage][lane].x, a.col_idx + j);
      cp_async_4(&my[stage][lane].y, a.vals + pos);
      my_perm[stage][lane] = pos;
    } else {
      my[stage][lane] = make_int2(0, 0);   // past the chunk: row 0 of dC, weight 0
    }
    cp_async_commit();
    pos = position(j + T);
  };
  stage_tile(0, base);
  stage_tile(1, base + T);

  const bool live_last = KS || ((R - 1) * W + l) * VEC < kw;   // only the last vector of a lane can lie outside
  const unsigned stride = (unsigned)kw * 4u;
  const int o_first = (R > 1 || live_last) ? l * VEC : kw - VEC;
  const int o_last = live_last ? ((R - 1) * W + l) * VEC : kw - VEC;
  const char* Dl = reinterpret_cast<const char*>(a.dC + o_first);
  const char* Dl_last = reinterpret_cast<const char*>(a.dC + o_last);
  using Split = group_split<VEC, W>;
  const int out_col = Split::column(lane);
  char* Ol = reinterpret_cast<char*>(a.dH + out_col);

  float acc[R][VEC], x[R][VEC];   // sum of the current row of dH; fragment of the same row of H
  auto clear = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int k = 0; k < VEC; ++k) acc[r][k] = 0.f;
  };
  auto load_x = [&]() {
    const float* xr = a.H + (int64_t)row * kw;
#pragma unroll
    for (int r = 0; r < R; ++r) gather_vec<VEC, false>(x[r], xr + (R > 1 && r == R - 1 ? o_last : o_first + r * W * VEC), 0ull);
  };
  clear();
  load_x();
  auto gather = [&](float (&d)[R][VEC], int col) {
    const char* p = Dl + (uint64_t)(unsigned)col * stride;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (R > 1 && r == R - 1)
        gather_vec<VEC, true>(d[r], reinterpret_cast<const float*>(Dl_last + (uint64_t)(unsigned)col * stride), policy);
      else
        gather_vec<VEC, true>(d[r], reinterpret_cast<const float*>(p) + r * W * VEC, policy);
    }
  };
  // one entry: its weight times the row into the sum, and this lane's share of its dot product
  auto use = [&](float v, const float (&d)[R][VEC]) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int k = 0; k < VEC; ++k) {
        acc[r][k] = fmaf(v, d[r][k], acc[r][k]);
        s = (KS || r < R - 1 || live_last) ? fmaf(x[r][k], d[r][k], s) : s;   // (a lane outside the slab adds nothing)
      }
    return s;
  };
  auto store_row = [&]() {
    float* out = reinterpret_cast<float*>(Ol + (uint64_t)(unsigned)row * stride);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float v[Split::KEEP];
      combine_groups<VEC, W>(acc[r], v, lane);
      if (Split::writes(lane) && (r < R - 1 || live_last)) store_stream(out + r * W * VEC, v);
    }
  };
  auto next_row = [&]() {
    store_row();
    clear();
    ++ri;
    const int2 nx = __ldg(a.nz + ri);
    row = nx.x;
    row_end = nx.y;
    load_x();
  };

  int stage = 0;
  for (; base < n1; base += T) {
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    const int2* tile = &my[stage][g];
    const int* place = my_perm[stage];
    const bool one_row = base + T <= n1 && row_end >= base + T;
    if (!one_row) {
      // the rows of H that begin in this tile are asked for at once: a row end below then waits for the L2 cache only
      const int last_end = __ldg(&a.nz[ri + lane].y);
      if (last_end < min(base + T, n1)) {
        const float* xr = a.H + (int64_t)__ldg(&a.nz[ri + lane + 1].x) * kw;
        for (int c = 0; c < kw; c += 32) prefetch_l2(xr + c);
      }
    }
#pragma unroll 1
    for (int u0 = 0; u0 < T; u0 += BATCH) {
      const int j0 = base + u0;
      if (j0 >= n1) break;
      float d[U][R][VEC];
      float v[U], part[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int2 e = tile[u0 + i * G];
        v[i] = __int_as_float(e.y);
        gather(d[i], e.x);
      }
      if (one_row || (j0 + BATCH <= n1 && row_end >= j0 + BATCH)) {
#pragma unroll
        for (int i = 0; i < U; ++i) part[i] = use(v[i], d[i]);
      } else {
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int lo = j0 + i * G;
          const int hi = min(lo + G, n1);
          const int mine = lo + g;
          int cur = lo;
          part[i] = 0.f;
          while (row_end < hi) {   // warp-uniform: the current row ends inside this step
            if (mine >= cur && mine < row_end) part[i] = use(v[i], d[i]);
            cur = row_end;
            next_row();
          }
          if (mine >= cur && mine < hi) part[i] = use(v[i], d[i]);
        }
      }
      const float total = reduce_transposed<U, W>(part, lane);
      const int o = u0 + reduced_entry<U>(l) * G + g;   // the entry of the tile whose total this lane holds
      if (l < U && base + o < n1) a.dA[place[o]] = total;
    }
    __syncwarp();
    stage_tile(stage, base + STAGES * T);
    stage ^= 1;
  }
  cp_async_wait<0>();

  // the end of the chunk: as in spmm_warp_kernel
  const int n0 = m[0], chunk = m[1], r0 = m[2], r0_start = m[3], r0_end = m[4];
  const bool hands_on = row_end != n1;
  if (!hands_on) {
    store_row();
  } else {
    float* slot_c = a.carry + (int64_t)chunk * kw + out_col;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float v[Split::KEEP];
      combine_groups<VEC, W>(acc[r], v, lane);
      if (Split::writes(lane) && (r < R - 1 || live_last)) store_plain(slot_c + r * W * VEC, v);
    }
  }
  const bool stores_split_row = r0_start < n0 && r0_end <= n1;
  if (!hands_on && !stores_split_row) return;
  settle_split_rows<VEC, W, R>(stores_split_row, r0, r0_start, r0_end, hands_on, row,
                               row == r0 ? r0_start : __ldg(a.row_ptr + row), row_end, chunk, a.S, a.carry, a.dH,
                               a.counter, kw, kw);
}

template <int VEC, int W, int R, int U, int KS, int MINB>
int launch(hpspmm_ctx* ctx, hpspmm_layer_grad_args a, cudaStream_t s) {
  constexpr int BT = 64;
  if (!hpspmm_shape_covers(VEC, W, R, a.K) || a.K > VEC * W * R) return HPSPMM_ERR_INVALID;
  a.n_chunk_blocks = (a.n_chunks + BT / 32 - 1) / (BT / 32);
  int n_zero_blocks = (a.rows + BT - 1) / BT;
  const int cap = ctx->sm_count * 8;
  if (n_zero_blocks > cap) n_zero_blocks = cap;
  const unsigned grid = (unsigned)(a.n_chunk_blocks + n_zero_blocks);
  hpspmm_launch(layer_grad_kernel<VEC, W, R, U, KS, BT, MINB>, grid, BT, 0, s, a);
  ctx->launches++;
  HPSPMM_CUDA_TRY(ctx, cudaGetLastError());
  return HPSPMM_OK;
}

}  // namespace

// One launch covers up to 256 columns of 16- or 8-byte vectors and 128 of 4-byte ones; a wider row would need the dot
// products of several slabs added up, and two kernels then.
bool hpspmm_layer_grad_covers(int64_t K, uintptr_t addresses) {
  return K <= (hpspmm_vector_width(K, addresses) == 1 ? 128 : 256);
}

// Whether one pass is faster than the permuted weights, the product and the SDDMM by themselves.  All figures are the time
// of those three divided by the time of one pass, replayed from a graph (no launch overhead), over graphs of 4, 16 and 50
// entries per row, square.
//
// Many entries: the 4-byte accesses through the permutation are cheap as long as what they reach, 8 bytes per entry, stays
// in the L2 cache beside the rows of dC.
//   uneven rows: 8 M entries 0.99 to 1.42 at K = 2 to 256; 10 M (5/8 of the cache) in rows of 4: 0.90 to 0.97 at K <= 32,
//                1.02 to 1.19 from 47 on; in rows of 16 and more 1.00 to 1.35.  14 M in 1 M rows: 0.81, 0.83, 0.94 at K = 16, 32, 64
//   even rows:   5 M entries 0.97 to 1.54; 6 M 0.99 to 1.50, but in rows of 50 entries K = 96 to 192 0.89 to 0.98.
//                7.2 M (7/16 of the cache): what loses there has rows of dC that take between a sixth of the cache and the
//                whole of it: in rows of 4 K = 4 to 20 0.87 to 0.97, of 16 K = 20 to 47 0.91 to 0.99, of 50 K = 96 to 126
//                0.87 to 0.99; below 1.08 to 1.41, above 1.02 to 1.41.  8 M in 500 K rows: 1.03, 0.98, 0.98, 1.24 at K = 16, 32, 64, 128
// Few entries: the product and the SDDMM have builds for few chunks, which hide the ends of rows better.
//   uneven rows, 150 K / 300 K / 500 K / 700 K / 1 M / 1.5 M / 2 M entries, worst of the three graphs:
//     K = 8   0.82 / 0.84 / 0.72 / 0.81 / 0.84 / 0.94 / 1.03        K = 20  0.84 / 0.90 / 0.77 / 0.92 / 0.95 / 1.16 / 1.19
//     K = 32  0.96 / 0.98 / 0.89 / 0.98 / 1.07 / 1.23 / 1.45        K = 48  0.92 / 1.04 / 0.93 / 1.09 / 1.10 / 1.27 / 1.31
//     K = 64  1.06 / 1.17 / 1.11 / 1.06 / 1.18 / 1.50 / 1.31        K = 96  0.66 / 0.63 / 0.82 / 1.00 / 1.10 / 1.23 / 1.12
//     K = 128 0.86 / 0.89 / 1.06 / 1.33 / 1.27 / 1.24 / 1.22        K = 256 0.67 / 0.77 / 1.14 / 1.10 / 1.31 / 1.31 / 1.16
//     K = 31, 47, 127 (4-byte vectors) 0.98 to 1.44 at every size
//   even rows, 100 K / 300 K / 600 K / 700 K / 1 M: K <= 64 1.01 to 1.71 (K = 8 in rows of 4 0.94 once); K = 96 (three vectors
//     per lane) 0.97 / 0.92 / 0.91 / 1.13 / 1.30; K = 128 1.01 / 0.97 / 1.26 / 1.24 / 1.34; K = 256 0.80 / 0.93 / 1.01 / 1.33 / 1.43
//     (of these 300 K in rows of 4 and 16 1.24 and 1.18)
// A call that is not captured pays for three launches instead of one besides, and one of up to 40 M products (even
// rows, K = 256: 80 M) is over before the host has issued the next: a training step through PyTorch of 11 K to 300 K entries,
// K = 4 to 128, 88 -> 79 us, even rows, K = 256, 300 K in rows of 50 87 -> 79, and from there on as above (uneven rows, K = 96,
// 500 K entries 111 -> 120; K = 256, 300 K 116 -> 118).
bool hpspmm_layer_grad_pays(const hpspmm_ctx* ctx, int64_t M, int64_t K, int VEC, int64_t nnz, bool even, bool captured) {
  const int64_t reached = 8 * nnz, l2 = ctx->l2_bytes, rows = 4 * K * M;
  if (even) {
    if (reached > l2 * 7 / 16 || (reached > l2 * 3 / 8 && rows > l2 / 6 && rows < l2 * 5 / 4)) return false;
    if (reached > l2 * 5 / 16 && nnz >= 32 * M && VEC > 1 && K > 64 && K <= 192) return false;
  } else {
    if (reached > l2 / 2 && (reached > l2 * 5 / 8 || (K < 100 && nnz < 16 * M))) return false;
  }
  int chunks_per_sm = 0;   // of 128 entries
  if (VEC > 1 || K < 31) {
    if (even)
      chunks_per_sm = VEC < 4 || K <= 64 ? 0 : (K <= 96 || (K > 128 && K <= 192) ? 36 : (K > 192 && nnz < 32 * M ? 15 : 24));
    else if (K != 64)
      chunks_per_sm = K >= 128 ? 24 : (K >= 48 ? 36 : (K >= 32 ? 48 : (K >= 17 ? 72 : 100)));
  }
  return nnz > ctx->sm_count * 128ll * chunks_per_sm ||
         (!captured && nnz * K < (even && K > 192 ? 80000000 : 40000000));
}

// Shapes: one vector per lane and as wide a group as it takes; two and three vectors per lane, which the SDDMM prefers,
// cost the sum and the row of H twice the registers here.  4 M entries of a power-law graph / uniform, K = 64: W = 8,
// R = 2 160 / 206 us, W = 16 134 / 176; K = 128: W = 16, R = 2 227 / 377, W = 32 222 / 352.  K = 96 and 192 stay at three.
// Blocks per SM: 16 (64 registers) at K = 64 134 us, 18 138, 20 175; at K = 32 18 93, 16 95, 20 113.
int hpspmm_layer_grad_launch(hpspmm_ctx* ctx, const hpspmm_layer_grad_args& a, cudaStream_t s) {
  const uintptr_t addresses = (uintptr_t)a.dC | (uintptr_t)a.H | (uintptr_t)a.dH;
  if (!hpspmm_layer_grad_covers(a.K, addresses)) return HPSPMM_ERR_UNSUPPORTED;
  const int VEC = hpspmm_vector_width(a.K, addresses);
  const int vecs = (a.K + VEC - 1) / VEC;
#define GO(V, W, R, U, KS, MINB) return launch<V, W, R, U, KS, MINB>(ctx, a, s)
  if (VEC == 4) {
    if (vecs <= 2) GO(4, 2, 1, 2, 0, 16);
    if (vecs <= 4) GO(4, 4, 1, 4, 0, 16);
    if (a.K == 32) GO(4, 8, 1, 4, 32, 18);
    if (vecs <= 8) GO(4, 8, 1, 4, 0, 16);
    if (a.K == 64) GO(4, 16, 1, 4, 64, 16);
    if (vecs <= 16) GO(4, 16, 1, 4, 0, 16);
    if (vecs <= 24) GO(4, 8, 3, 2, 0, 14);
    if (a.K == 128) GO(4, 32, 1, 4, 128, 18);
    if (vecs <= 32) GO(4, 32, 1, 4, 0, 18);
    if (vecs <= 48) GO(4, 16, 3, 2, 0, 12);
    GO(4, 32, 2, 2, 0, 14);
  }
  if (VEC == 2) {
    if (vecs <= 2) GO(2, 2, 1, 2, 0, 16);
    if (vecs <= 4) GO(2, 4, 1, 4, 0, 16);
    if (vecs <= 8) GO(2, 8, 1, 8, 0, 16);
    if (vecs <= 16) GO(2, 8, 2, 4, 0, 16);
    if (vecs <= 24) GO(2, 8, 3, 4, 0, 16);
    if (vecs <= 32) GO(2, 16, 2, 4, 0, 16);
    if (vecs <= 48) GO(2, 16, 3, 4, 0, 14);
    if (vecs <= 64) GO(2, 16, 4, 4, 0, 12);
    if (vecs <= 96) GO(2, 32, 3, 4, 0, 14);
    GO(2, 32, 4, 4, 0, 12);
  }
  if (vecs <= 1) GO(1, 1, 1, 1, 0, 16);
  if (vecs <= 4) GO(1, 4, 1, 4, 0, 16);
  if (vecs <= 8) GO(1, 8, 1, 8, 0, 16);
  if (vecs <= 16) GO(1, 8, 2, 4, 0, 16);
  if (vecs <= 24) GO(1, 8, 3, 4, 0, 16);
  if (vecs <= 32) GO(1, 16, 2, 8, 0, 16);
  if (vecs <= 48) GO(1, 16, 3, 4, 0, 16);
  if (vecs <= 64) GO(1, 16, 4, 4, 0, 16);
  if (vecs <= 96) GO(1, 32, 3, 4, 0, 16);
  GO(1, 32, 4, 4, 0, 16);
#undef GO
}

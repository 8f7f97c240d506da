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
  const int4 rec0 = __ldg(a.rec + 2 * (int64_t)slot), rec1 = __ldg(a.rec + 2 * (int64_t)slot + 1);
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

// Whether one pass is faster than the permuted weights, the product and the SDDMM by themselves.  The 4-byte accesses
// through the permutation are cheap as long as what they reach, 8 bytes per entry, stays in the L2 cache beside the rows of
// dC: three kernels -> one in us, power-law graphs, K = 16 / 32 / 64 / 128:
//   4 M entries, 250 K rows   118 -> 85 / 131 -> 93 / 180 -> 134 / 280 -> 222     (update of the weights 21, product 79, SDDMM 76 at K = 64)
//   10 M, 600 K               257 -> 243 / 278 -> 274 / 410 -> 383 / 710 -> 659
//   14 M, 1 M                 382 -> 471 / 398 -> 480 / 588 -> 624
// and with uniform columns, where hardly a row of dC is found in the cache, it ends earlier:
//   6 M, 350 K                170 -> 129 / 212 -> 186 / 335 -> 304 / 722 -> 623
//   8 M, 500 K                240 -> 234 / 302 -> 308 / 501 -> 511 / 1098 -> 888
bool hpspmm_layer_grad_pays(const hpspmm_ctx* ctx, int64_t nnz, bool even) {
  return 8 * nnz <= (even ? ctx->l2_bytes * 7 / 16 : ctx->l2_bytes * 5 / 8);
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

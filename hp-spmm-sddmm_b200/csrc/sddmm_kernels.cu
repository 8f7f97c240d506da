// FP32 SDDMM over a CSR pattern for sm_100a: out[j] = dot(X[row(j), :], Y[col[j], :]).
//
// The reference names SDDMM but ships no code for it (only the unused ResInfo::sddmm_*
// fields, include/spmm/mm/spmm_common.h:130-135).  The kernels reuse the nnz-balanced chunk
// table of the SpMM (one warp per chunk); A's values are not multiplied in.
#include "device_utils.cuh"
#include "hpspmm_internal.h"
#include "warp_frag.cuh"

namespace {

using namespace hpspmm;

// ---- warp kernel: one warp per chunk, G = 32/W interleaved lane groups (warp_frag.cuh) -----------
// Same shape as the SpMM warp kernel: (col) tiles of 32 entries staged in shared memory with
// asynchronous copies; in every step group g takes entry G*s+g and gathers its fragment of that
// row of Y, U steps at a time.  The fragment of the current row of X stays in registers; row
// changes are warp-uniform.  The U partial dot products of a batch are reduced across the W lanes
// of each group with a transposing butterfly (4 shuffles for 4 results at W = 8).

// KS: row stride of X and Y when it is a compile-time constant, else 0.  The slab is columns [off0, off0 + cols) of
// X and Y; add: add to what an earlier slab wrote.
// The kernel walks the list nz of the rows that hold entries and never looks at an empty row.
// SERIAL: a row end waits for the next row's fragment of X.  With many chunks per SM other warps cover that, and the
// path needs no registers beyond the gathers' (16 M entries, 64 columns: 0.327 ms against 0.366).  With few chunks the
// waits add up instead -- a chunk of very short rows waits once per row -- so there all row bounds of a tile come from
// one load and the entries of a batch gather their own rows of X (70 K entries of a power-law graph in chunks of 64,
// 64 columns: 8.6 us against 12.6).
template <int VEC, int W, int R, int U, int KS, bool HINT, int BT, int MINB, bool SERIAL>
__global__ void __launch_bounds__(BT, MINB)
sddmm_warp_kernel(int n_chunks, int ld, int off0, int cols, int add, int keep_y, const int* __restrict__ col_idx,
                  const float* __restrict__ X, const float* __restrict__ Y, float* __restrict__ out,
                  const int4* __restrict__ rec, const int2* __restrict__ nz) {
  constexpr int CW = VEC * W * R;
  constexpr int G = 32 / W;
  constexpr int T = 32;
  constexpr int BATCH = U * G;
  constexpr int STAGES = 2;
  static_assert(T % BATCH == 0 && (U <= W || W == 1), "batch must tile the staged tile; a lane holds one total");
  __shared__ int tiles[BT / 32][STAGES][T];

  chain_grid();
  const int lane = threadIdx.x & 31;
  const int g = lane / W;
  const int l = lane % W;
  const int slot = (int)((blockIdx.x * (unsigned)BT + threadIdx.x) >> 5);
  if (slot >= n_chunks) return;
  // (a compile-time policy and no `add` where the width is one full slab: 0.324 -> 0.301 ms at K = 64, 0.577 -> 0.528 at
  // K = 128, R-MAT scale 20; both are live through the loop otherwise)
  const uint64_t policy = HINT ? (KS ? policy_evict_last() : policy_for_gathers(keep_y)) : 0ull;
  int(*my)[T] = tiles[threadIdx.x >> 5];

  const int4 p = ld_chained(rec + 2 * (int64_t)slot);
  const int n0 = p.x;
  int ri = p.y, row = p.z, row_end = p.w;
  const int n1 = ld_chained(&rec[2 * (int64_t)slot + 1].z);

  auto stage_tile = [&](int stage, int base) {
    const int j = base + lane;
    if (j < n1)
      cp_async_4(&my[stage][lane], col_idx + j);
    else
      my[stage][lane] = 0;   // past the chunk: column 0 (a valid row of Y), result discarded
    cp_async_commit();
  };
  stage_tile(0, n0);
  stage_tile(1, n0 + T);

  // a lane beyond the slab's width works on the slab's last vector with an x of zero
  const int kw = KS ? CW : cols;
  const bool live_last = KS || ((R - 1) * W + l) * VEC < kw;
  const unsigned stride = (KS ? KS : ld) * 4u;
  const int o_first = off0 + ((R > 1 || live_last) ? l * VEC : kw - VEC);
  const int o_last = off0 + (live_last ? ((R - 1) * W + l) * VEC : kw - VEC);
  const char* Yl = reinterpret_cast<const char*>(Y + o_first);
  const char* Yl_last = reinterpret_cast<const char*>(Y + o_last);
  float x[R][VEC];
  auto load_x = [&](float (&x)[R][VEC], int row) {
    const float* xr = X + (int64_t)row * (KS ? KS : ld);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      gather_vec<VEC, false>(x[r], xr + (R > 1 && r == R - 1 ? o_last : o_first + r * W * VEC), 0ull);
      if (r == R - 1 && !live_last)
#pragma unroll
        for (int k = 0; k < VEC; ++k) x[r][k] = 0.f;
    }
  };
  bool have_x = SERIAL;   // x holds the fragment of the current row
  if (SERIAL) load_x(x, row);
  auto gather = [&](float (&y)[R][VEC], int col) {
    const char* q = Yl + (uint64_t)(unsigned)col * stride;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (R > 1 && r == R - 1)
        gather_vec<VEC, HINT>(y[r], reinterpret_cast<const float*>(Yl_last + (uint64_t)(unsigned)col * stride), policy);
      else
        gather_vec<VEC, HINT>(y[r], reinterpret_cast<const float*>(q) + r * W * VEC, policy);
    }
  };
  auto dot = [&](const float (&x)[R][VEC], const float (&y)[R][VEC]) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int k = 0; k < VEC; ++k)
        // (0 * inf of a lane outside the slab must not reach the sum)
        s = (KS || r < R - 1 || live_last) ? fmaf(x[r][k], y[r][k], s) : s;
    return s;
  };
  // reduce the U partial dot products of a batch over the W lanes of each group and store the U * G results
  auto finish_batch = [&](float (&part)[U], int j0) {
    const float total = reduce_transposed<U, W>(part, lane);
    const int j = j0 + reduced_entry<U>(l) * G + g;
    if (l < U && j < n1) out[j] = (KS == 0 && add) ? out[j] + total : total;
  };

  int stage = 0;
  for (int base = n0; base < n1; base += T) {
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    const int* tile = &my[stage][g];
    if (base + T <= n1 && row_end >= base + T) {
      // Fast tile: all 32 entries belong to the current row.  Fully unrolled, every shared-memory offset a
      // compile-time constant, no tests between gathers (two thirds of the tiles of a power-law graph).
      if (!SERIAL && !have_x) load_x(x, row);
      have_x = true;
#pragma unroll
      for (int u0 = 0; u0 < T; u0 += BATCH) {
        float y[U][R][VEC];
#pragma unroll
        for (int i = 0; i < U; ++i) gather(y[i], tile[u0 + i * G]);
        float part[U];
#pragma unroll
        for (int i = 0; i < U; ++i) part[i] = dot(x, y[i]);
        finish_batch(part, base + u0);
      }
    } else if (SERIAL) {
      {
        // The rows of X that begin in this tile are asked for at once, a lane a row: a row end below then waits for the
        // L2 cache and not for DRAM.  8 M entries of a power-law graph, K = 32: 0.102 -> 0.096 ms; 3 M, K = 64: 0.082 ->
        // 0.061 ms, where the chunk with the most rows decides.
        const int last_end = __ldg(&nz[ri + lane].y);          // the row before the one this lane asks for
        if (last_end < min(base + T, n1)) {
          const float* xr = X + (int64_t)__ldg(&nz[ri + lane + 1].x) * (KS ? KS : ld) + off0;
          for (int c = 0; c < kw; c += 32) prefetch_l2(xr + c);
        }
      }
#pragma unroll 1
      for (int u0 = 0; u0 < T; u0 += BATCH) {
        const int j0 = base + u0;
        if (j0 >= n1) break;
        float y[U][R][VEC];
#pragma unroll
        for (int i = 0; i < U; ++i) gather(y[i], tile[u0 + i * G]);
        float part[U];
        if (row_end >= j0 + BATCH) {
#pragma unroll
          for (int i = 0; i < U; ++i) part[i] = dot(x, y[i]);
        } else {
#pragma unroll
          for (int i = 0; i < U; ++i) {
            const int lo = j0 + i * G;
            const int hi = min(lo + G, n1);
            const int mine = lo + g;
            int cur = lo;
            part[i] = 0.f;
            while (row_end < hi) {   // warp-uniform: the current row ends inside this step
              if (mine >= cur && mine < row_end) part[i] = dot(x, y[i]);
              cur = row_end;
              ++ri;
              const int2 nx = __ldg(nz + ri);
              row = nx.x;
              row_end = nx.y;
              load_x(x, row);
            }
            if (mine >= cur) part[i] = dot(x, y[i]);
          }
        }
        finish_batch(part, j0);
      }
    } else {
      // Rows end inside this tile (or just before it).  Lane i holds the i-th row from the tile's first one on; bit p
      // of `starts` (p > 0) says that entry p of the tile opens a new row.  In a batch that holds several row starts every
      // entry gathers the fragment of its own row of X beside that of Y (neighbours share rows and hit the same lines):
      // waiting for the next row's fragment at each row end cost a memory latency per row.
      if (row_end == base) {                 // the current row ended with the previous tile
        ++ri;
        have_x = false;
      }
      const int2 mine_nz = __ldg(nz + ri + lane);
      const int limit = min(T, n1 - base);   // entries of this tile inside the chunk
      const unsigned p = (unsigned)(mine_nz.y - base);
      const unsigned starts = __reduce_or_sync(0xffffffffu, p < (unsigned)limit ? 1u << p : 0u);
      int passed = 0;                        // row starts before the batch
#pragma unroll 1
      for (int u0 = 0; u0 < limit; u0 += BATCH) {
        float y[U][R][VEC];
        float part[U];
#pragma unroll
        for (int i = 0; i < U; ++i) gather(y[i], tile[u0 + i * G]);
        const unsigned here = BATCH == 32 ? starts : (starts >> u0) & ((1u << (BATCH & 31)) - 1u);
        const int n_here = __popc(here);     // all of this is warp-uniform
        if (n_here <= 1) {
          // one row, or the end of one and the start of the next: the fragments of both travel with the gathers
          if (!have_x) load_x(x, __shfl_sync(0xffffffffu, mine_nz.x, passed));
          have_x = true;
          if (n_here == 0) {
#pragma unroll
            for (int i = 0; i < U; ++i) part[i] = dot(x, y[i]);
          } else {
            float x2[R][VEC];
            load_x(x2, __shfl_sync(0xffffffffu, mine_nz.x, passed + 1));
            const int first = __ffs(here) - 1 - g;   // entry i * G of this group lies in the next row from here on
#pragma unroll
            for (int i = 0; i < U; ++i) {
              float xi[R][VEC];
#pragma unroll
              for (int r = 0; r < R; ++r)
#pragma unroll
                for (int k = 0; k < VEC; ++k) xi[r][k] = i * G >= first ? x2[r][k] : x[r][k];
              part[i] = dot(xi, y[i]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int k = 0; k < VEC; ++k) x[r][k] = x2[r][k];
          }
        } else {
          constexpr int H = U >= 2 ? U / 2 : 1;
#pragma unroll
          for (int i0 = 0; i0 < U; i0 += H) {
            float xs[H][R][VEC];
#pragma unroll
            for (int i = 0; i < H; ++i) {
              const int q = (i0 + i) * G + g;   // entry u0 + q of the tile
              load_x(xs[i], __shfl_sync(0xffffffffu, mine_nz.x, passed + __popc(here & (0xffffffffu >> (31 - q)))));
            }
#pragma unroll
            for (int i = 0; i < H; ++i) part[i0 + i] = dot(xs[i], y[i0 + i]);
          }
          have_x = false;
        }
        passed += n_here;
        finish_batch(part, base + u0);
      }
      ri += passed;
      row = __shfl_sync(0xffffffffu, mine_nz.x, passed);
      row_end = __shfl_sync(0xffffffffu, mine_nz.y, passed);
    }
    __syncwarp();
    stage_tile(stage, base + STAGES * T);
    stage ^= 1;
  }
  cp_async_wait<0>();
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct sddmm_args {
  int n_chunks, K, off, cols, keep_y;
  bool few;         // at most one wave of chunks
  bool waves;       // four waves of chunks and more
  bool long_rows;   // rows are long enough that waiting for each row of X costs little
  const int32_t* col_idx;
  const float *X, *Y;
  float* out;
  const int4* rec;
  const int2* nz;
};

// one slab of the width: the first writes the partial dot products, the others add theirs
template <int VEC, int W, int R, int U, int KS, bool HINT, int MINB, bool SERIAL>
int launch_sddmm(hpspmm_ctx* ctx, const sddmm_args& a, cudaStream_t s) {
  constexpr int BT = 64;
  const unsigned grid = (unsigned)((a.n_chunks + BT / 32 - 1) / (BT / 32));
  if (a.cols > VEC * W * R || !hpspmm_shape_covers(VEC, W, R, a.cols)) return HPSPMM_ERR_INVALID;
  hpspmm_launch(sddmm_warp_kernel<VEC, W, R, U, KS, HINT, BT, MINB, SERIAL>, grid, BT, 0, s, a.n_chunks, a.K, a.off,
                a.cols, a.off > 0 ? 1 : 0, a.keep_y, a.col_idx, a.X, a.Y, a.out, a.rec, a.nz);
  ctx->launches++;
  HPSPMM_CUDA_TRY(ctx, cudaGetLastError());
  return HPSPMM_OK;
}

// Shapes.  With many chunks the shared-memory and shuffle pipe
// that also carries the gathers decides, and narrow groups with several vectors per lane use it less: W = 8 instead of 16
// halves the broadcast reads of an entry and the exchanges of its sum, and R = 3 leaves fewer lanes idle than the next
// power of two.  R-MAT scale 20, 16 M entries, before -> after in us:
//   K = 48 360 -> 309, 64 294 -> 281, 96 606 -> 424, 100 617 -> 515, 128 521 -> 490, 160 1055 -> 743, 192 1083 -> 792,
//   256 1187 -> 1029; uniform columns, K = 64 551 -> 520, 96 984 -> 882, 160 1794 -> 1564
//   2-float vectors: K = 46 407 -> 321, 62 419 -> 363, 126 694 -> 577; 4-byte: K = 13 205 -> 193, 23 306 -> 253, 31 310 -> 279
// K = 32 stays at W = 8, R = 1 (185 us; 193 to 218 with other shapes).  16 blocks per SM (64 registers) where two or three
// vectors per lane are in flight; 20 (48 registers) at K = 32: 193 against 204 us at 18.
// With few chunks (lat) a chunk's chain of batches decides, and several groups make it shorter: a batch holds U entries
// of each, and every load of its rows of X is waited for once.  There registers are plenty, so more of it is in flight.
// Power-law graph of 300 K entries / uniform columns, 300 K / power-law, 1 M: K = 96 29.1 -> 14.8 / 23.0 -> 14.8 / 44.8 ->
// 34.9 us, K = 128 29.1 -> 18.8 / 27.1 -> 19.4 us, K = 160 49.7 -> 22.0 / 45.6 -> 24.8 / 77.4 -> 58.5 us, K = 256 50.8 ->
// 25.1 / 48.7 -> 41.4 / 80.6 -> 76.9 us, K = 126 29.2 -> 18.9 / 25.1 -> 19.6 us, K = 23, 1 M 25.1 -> 20.9 us.  Shapes that
// lose with more than one wave of chunks (1 M uniform entries, K = 128: 55 against 60 us) end there (few), those that lose
// on short rows (500 K entries in 100 K rows, K = 128: 42 against 49 us) want long ones; at 9 to 16 vectors and at K = 62 and 63 a wide group stays ahead.
// Which of them are SERIAL: 16-byte vectors fill the registers that the other path needs (K = 96 424 against 477 us); with
// narrower vectors it costs more than it saves except where noted by the shape.  Where rows are short the waits do not
// pay (uniform rows of 4 entries, K = 100: 176 against 159 us; of 8: 130 against 119; of 12: 110 against 105, but K = 96 92
// against 103 and K = 160 158 against 185): rows_are_long.  K = 32, 64 and 128 take SERIAL at any row length; on short rows
// that is compared with the kernel before it only (4 M uniform entries in rows of 4: K = 32 164 -> 134 us, 64 234 ->
// 193, 128 401 -> 398).  Where the gain is small it also takes enough chunks to cover the waits (12,500 chunks: K = 48 38.9 against 41.4 us, K = 62 45.7
// against 55.1; 31,000: 105 against 97 and 110 against 97).
int launch_sddmm_shape(hpspmm_ctx* ctx, const sddmm_args& a, const hpspmm_spmm_shape& sh, cudaStream_t s) {
#define GO(V, W, R, U, KS, H, MINB) return launch_sddmm<V, W, R, U, KS, H, MINB, false>(ctx, a, s)
#define GO_SERIAL(V, W, R, U, KS, H, MINB) return launch_sddmm<V, W, R, U, KS, H, MINB, true>(ctx, a, s)
  if (sh.VEC == 4) {
    const int vecs = a.cols / 4;
    if (sh.lat) {
      if (a.few && vecs > 16 && vecs <= 24) GO(4, 8, 3, 4, 0, true, 8);
      if (vecs > 16 && vecs <= 24) GO(4, 8, 3, 2, 0, true, 10);
      if (a.few && a.long_rows && vecs > 24 && vecs <= 32) GO(4, 8, 4, 2, 0, true, 8);
      if (vecs > 32 && vecs <= 48) GO(4, 16, 3, 4, 0, true, 8);
      if (a.long_rows && vecs > 48 && vecs <= 64) GO(4, 16, 4, 4, 0, true, 6);
    } else if (a.K == 32) {
      if (sh.hint) GO_SERIAL(4, 8, 1, 4, 32, true, 20); else GO_SERIAL(4, 8, 1, 4, 32, false, 20);
    } else if (a.K == 64) {
      if (sh.hint) GO_SERIAL(4, 8, 2, 4, 64, true, 16); else GO_SERIAL(4, 8, 2, 4, 64, false, 16);
    } else if (a.K == 128) {
      if (sh.hint) GO_SERIAL(4, 16, 2, 4, 128, true, 16); else GO_SERIAL(4, 16, 2, 4, 128, false, 16);
    } else if (a.long_rows && vecs > 8 && vecs <= 64) {
      if (vecs <= 16) {
        if (a.waves) GO_SERIAL(4, 8, 2, 4, 0, true, 16); else GO(4, 16, 1, 4, 0, true, 16);
      }
      if (vecs <= 24) GO_SERIAL(4, 8, 3, 2, 0, true, 16);
      if (vecs <= 32) GO_SERIAL(4, 16, 2, 4, 0, true, 16);
      if (vecs <= 48) GO_SERIAL(4, 16, 3, 2, 0, true, 16);
      GO_SERIAL(4, 16, 4, 2, 0, true, 14);
    }
    if (sh.W == 2) GO(4, 2, 1, 2, 0, true, 16);
    if (sh.W == 4) GO(4, 4, 1, 4, 0, true, 16);
    if (sh.W == 8) GO(4, 8, 1, 4, 0, true, 16);
    if (sh.W == 16) GO(4, 16, 1, 4, 0, true, 16);
    if (sh.R == 1) GO(4, 32, 1, 4, 0, true, 18);
    if (sh.R == 2) GO(4, 32, 2, 2, 0, true, 18);
    if (sh.R == 3) GO(4, 32, 3, 2, 0, true, 12);
    GO(4, 32, 4, 2, 0, true, 10);
  }
  if (sh.VEC == 2) {
    const int vecs = (a.cols + 1) / 2;
    if (a.few && vecs > 16 && vecs <= 24) GO(2, 8, 3, 4, 0, true, 8);
    if (a.few && a.long_rows && vecs > 48 && vecs <= 64) GO(2, 16, 4, 4, 0, true, 6);
    if (!sh.lat && vecs > 16 && vecs <= 24) GO(2, 8, 3, 4, 0, true, 16);
    if (!sh.lat && a.long_rows && a.waves && vecs > 24 && vecs <= 32) GO_SERIAL(2, 16, 2, 8, 0, true, 16);
    if (!sh.lat && a.long_rows && vecs > 48 && vecs <= 64) GO_SERIAL(2, 16, 4, 4, 0, true, 16);
    if (sh.W == 2) GO(2, 2, 1, 2, 0, true, 16);
    if (sh.W == 4) GO(2, 4, 1, 4, 0, true, 16);
    if (sh.W == 8) GO(2, 8, 1, 8, 0, true, 16);
    if (sh.W == 16 && sh.R == 3) GO(2, 16, 3, 4, 0, true, 14);
    if (sh.W == 16) GO(2, 16, 1, 8, 0, true, 16);
    if (sh.R == 1) GO(2, 32, 1, 8, 0, true, 16);
    if (sh.R == 2) GO(2, 32, 2, 4, 0, true, 16);
    if (sh.R == 3) GO(2, 32, 3, 4, 0, true, 14);
    GO(2, 32, 4, 4, 0, true, 12);
  }
  if (sh.lat && a.cols > 16 && a.cols <= 24) GO(1, 8, 3, 4, 0, true, 8);
  if (!sh.lat) {
    if (a.cols > 8 && a.cols <= 16) GO(1, 8, 2, 4, 0, true, 18);
    if (a.cols > 16 && a.cols <= 24) GO(1, 8, 3, 4, 0, true, 18);
    if (a.cols > 24 && a.cols <= 32) GO(1, 16, 2, 8, 0, true, 16);
    if (a.cols > 48 && a.cols <= 64) GO(1, 16, 4, 4, 0, true, 16);
  }
  if (sh.W == 1) GO(1, 1, 1, 1, 0, true, 16);
  if (sh.W == 4) GO(1, 4, 1, 4, 0, true, 16);
  if (sh.W == 8) GO(1, 8, 1, 8, 0, true, 16);
  if (sh.W == 16 && sh.R == 3) GO(1, 16, 3, 4, 0, true, 18);
  if (sh.W == 16) GO(1, 16, 1, 8, 0, true, 16);
  if (sh.R == 1) GO(1, 32, 1, 8, 0, true, 16);
  if (sh.R == 2) GO(1, 32, 2, 8, 0, true, 16);
  if (sh.R == 3) GO(1, 32, 3, 4, 0, true, 16);
  if (sh.R == 4) GO(1, 32, 4, 4, 0, true, 16);
  if (sh.R == 5) GO(1, 32, 5, 4, 0, true, 14);
  if (sh.R == 6) GO(1, 32, 6, 4, 0, true, 14);
  if (sh.R == 7) GO(1, 32, 7, 4, 0, true, 12);
  GO(1, 32, 8, 4, 0, true, 12);
#undef GO
#undef GO_SERIAL
}

// Whether the rows are long enough on average for the SERIAL shapes.  At 129 to 160 columns they pay early (uniform rows of
// 9 entries, K = 160: 435 -> 401 us; of 5 about level; of 4: 519 -> 534).  Without a plan nothing tells a skewed matrix, most
// of whose entries lie in long rows whatever the average, so there the line lies where a uniform one loses little:
//   power-law, 4 M entries in 1 M rows: K = 96 273 -> 233, 160 420 -> 333, 192 451 -> 356 us
//   uniform, the same sizes:            K = 96 322 -> 331, 160 544 -> 554, 192 609 -> 643 us; rows of 8, K = 160 224 -> 200 us
bool rows_are_long(int VEC, int64_t M, int64_t K, int64_t nnz, bool has_plan) {
  if (VEC == 4) {
    if (!has_plan && ((K > 64 && K <= 96) || (K > 128 && K <= 192))) return nnz >= 4 * M;
    if (K > 128 && K <= 160) return nnz >= 5 * M;
  }
  return nnz >= 10 * M;
}

// Widest slab of the SDDMM's columns.  289 to 512 columns in one pass are three or four vectors of 32 lanes with one or two
// entries in flight; two passes of at most 256 columns run the shapes of 16 lanes, and the second adds its part.  A short
// rest is a cheap second pass on any graph; a long one pays on rows of even length only, once there are enough chunks or
// Y is too large for the L2 cache anyway.  One pass -> two in us:
//   K = 288: uniform, 1 M entries 137 -> 127, 2.5 M 322 -> 304, 4 M 671 -> 600;  power-law, 4 M 411 -> 329
//   K = 384: uniform, 2 M 416 -> 391, 4 M in 100 K rows 612 -> 484;  power-law, 4 M without a plan +10 %
//   K = 448: uniform, 2.5 M 515 -> 463, 4 M 1005 -> 896, but 1.5 M, whose Y fits the cache, 210 -> 220
//   K = 512: uniform, 2 M 566 -> 513, 4 M 1123 -> 998
int widest_sddmm_slab(const hpspmm_ctx* ctx, int VEC, int64_t N, int64_t K, int64_t n_chunks, bool even) {
  if (VEC == 4 && K > 256 && K <= 512) {
    if (K <= 288 && n_chunks > ctx->sm_count * 48ll) return 256;
    const bool many = n_chunks > ctx->sm_count * 80ll;
    const bool large = n_chunks > ctx->sm_count * 48ll && 4 * N * K > ctx->l2_bytes;
    if (K >= 320 && even && (many || large)) return 256;
  }
  return hpspmm_widest_slab(VEC);
}

// Up to about two waves of resident warps (80 chunks per SM) a call takes the shapes for few chunks -- except that at 32,
// 64 and 128 columns the SERIAL kernel of a fixed width is ahead from some number of chunks on.  With rows of even length
// no chunk has many more row ends to wait at than the others; a power-law graph (even: false, also where there is no plan
// to tell) needs more chunks to cover its worst one.  Uniform rows, shapes for few chunks -> SERIAL in us:
//   K = 32:  300 K entries 8.3 -> 8.3, 600 K 14.4 -> 12.4, 1.3 M 24.7 -> 20.7, 1.5 M 20.9 -> 17.7; rows of 4 or 5 entries
//            lose (400 K 13.8 -> 15.3, 1 M 23.2 -> 27.6), as does a power-law graph at any size (1.5 M 20.6 -> 23.7)
//   K = 64:  150 K 10.3 -> 8.3, 1.3 M 37.0 -> 30.8, 1.5 M 32.9 -> 26.7; 67.6 K 8.3 -> 8.3; power-law, 1 M 26.7 -> 28.8
//   K = 128: 400 K 24.7 -> 20.6, 1 M 49.6 -> 43.0, 1.5 M 59.5 -> 49.2, 3 M 135 -> 109; 300 K 16.3 -> 18.5;
//            power-law, 1 M 43.5 -> 40.9, 3 M 120 -> 94, but 600 K 26.7 -> 36.9
bool serial_when_few(int64_t K, int64_t n_chunks, bool long_rows, bool even, int sm_count) {
  if (K == 32) return even && long_rows && n_chunks > sm_count * 30;
  if (K == 64) return even && n_chunks > sm_count * 12;
  if (K == 128) return n_chunks > sm_count * (even ? 20 : 48);
  return false;
}

}  // namespace

extern "C" int hpspmm_sddmm_csr_f32(hpspmm_ctx* ctx, const hpspmm_plan* plan, int64_t M, int64_t N,
                                    int64_t K, int64_t nnz, const int32_t* row_ptr,
                                    const int32_t* col_idx, const float* X, const float* Y,
                                    float* out_vals, const hpspmm_opts* opts,
                                    hpspmm_stream stream) {
  HPSPMM_TRACE("hpspmm_sddmm_csr_f32");
  HPSPMM_REQUIRE(ctx, ctx != nullptr, "null context");
  HPSPMM_REQUIRE(ctx, M >= 0 && N >= 0 && nnz >= 0, "negative size");
  HPSPMM_REQUIRE(ctx, K >= 1, "K must be >= 1");
  if (M > 2147483646ll || N > 2147483647ll || nnz > 2147483647ll - 4096 || K > (1 << 20)) {
    snprintf(ctx->err, sizeof(ctx->err), "sizes beyond 32-bit CSR indices");
    return HPSPMM_ERR_UNSUPPORTED;
  }
  if (nnz == 0 || M == 0) return HPSPMM_OK;
  HPSPMM_REQUIRE(ctx, row_ptr && col_idx && X && Y && out_vals, "null operand");
  if ((K & 3) == 0 && (((uintptr_t)X & 15u) || ((uintptr_t)Y & 15u))) {
    snprintf(ctx->err, sizeof(ctx->err), "dense operands must be 16-byte aligned");
    return HPSPMM_ERR_INVALID;
  }
  hpspmm_device_guard guard(ctx->device);
  cudaStream_t s = (cudaStream_t)stream;
  const int hint_mode = opts ? opts->b_l2_hint : 0;
  const bool hint = hint_mode == 2 || (hint_mode == 0 && K >= 64);
  sddmm_args a = {0, (int)K, 0, 0, hint ? 1 : 0, false, false, false, col_idx, X, Y, out_vals, nullptr, nullptr};
  const int VEC = hpspmm_vector_width(K, (uintptr_t)X | (uintptr_t)Y);
  a.long_rows = rows_are_long(VEC, M, K, nnz, plan != nullptr);
  bool even = false;   // rows are known to be of even length
  if (plan) {
    HPSPMM_REQUIRE(ctx, plan->M == M && plan->nnz == nnz, "plan built for another matrix");
    HPSPMM_REQUIRE(ctx, plan->device == ctx->device, "plan built on another device");
    a.n_chunks = (int)plan->n_chunks;
    // The average says nothing about a skewed matrix, most of whose entries lie in long rows; there many rows are split.
    // (power-law graph of 1 M rows, 5 M entries, K = 96: serial 175 us, mask 230 us)
    even = hpspmm_even_rows(plan);
    a.long_rows = a.long_rows || !even;
    a.rec = plan->rec;
    a.nz = plan->nz;
  } else {
    int32_t S = (opts && opts->chunk_nnz > 0) ? opts->chunk_nnz : hpspmm_default_chunk_nnz(K, nnz);
    S = (S + 31) / 32 * 32;
    const int64_t n_chunks = (nnz + S - 1) / S;
    const size_t b_tiles = align_up((size_t)hpspmm_row_tile_ints(M) * 4, 256);
    const size_t b_rec = align_up((size_t)n_chunks * 32, 256);
    int st = hpspmm_ensure_scratch(ctx, b_tiles + b_rec + hpspmm_nz_bytes(M));
    if (st != HPSPMM_OK) return st;
    char* base = (char*)ctx->scratch;
    int4* rec = (int4*)(base + b_tiles);
    int2* nz = (int2*)(base + b_tiles + b_rec);
    st = hpspmm_build_structure(ctx, M, nnz, row_ptr, S, n_chunks, nz, rec, (int32_t*)base,
                                hpspmm_structure_tables{}, s);
    if (st != HPSPMM_OK) return st;
    a.n_chunks = (int)n_chunks;
    a.rec = rec;
    a.nz = nz;
  }
  a.few = a.n_chunks <= ctx->sm_count * 32;
  a.waves = a.n_chunks > ctx->sm_count * 160;
  const int widest = widest_sddmm_slab(ctx, VEC, N, K, a.n_chunks, even);
  for (a.off = 0; a.off < a.K; a.off += a.cols) {
    a.cols = a.K - a.off < widest ? a.K - a.off : widest;
    hpspmm_spmm_shape sh = hpspmm_choose_shape(VEC, a.cols, widest, hint);
    sh.lat = a.n_chunks <= ctx->sm_count * 80 && !serial_when_few(K, a.n_chunks, nnz >= 10 * M, even, ctx->sm_count);
    if (sh.VEC == 4 && sh.R == 3 && sh.W < 32) sh.R = sh.W / 8, sh.W = 32;
    const int st = launch_sddmm_shape(ctx, a, sh, s);
    if (st != HPSPMM_OK) return st;
  }
  return HPSPMM_OK;
}

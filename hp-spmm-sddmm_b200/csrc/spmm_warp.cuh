// The nnz-balanced warp kernel of the CSR product, for every width.
//
// One warp owns one chunk of the entry axis.  It stages (col, val) tiles of 32 entries in shared memory with
// asynchronous copies, two tiles ahead of their use; in every step group g of the warp takes entry G*s+g of the
// tile, reads its (col, val) pair as one shared-memory broadcast and gathers its fragment of that row of B
// (warp_frag.cuh), U steps of gathers being in flight before the first FMA.  Row ends are warp-uniform, so groups
// never diverge.  A finished row is combined across the groups and stored once.
//
// A chunk that ends inside a heavy row leaves its partial sum in a carry slot; the pieces of a split row settle it
// among themselves (settle_split_rows).  The order of all additions is fixed by the chunking and the shape, so
// results are bit-reproducible from run to run.
#pragma once
#include "device_utils.cuh"
#include "hpspmm_internal.h"
#include "warp_frag.cuh"

namespace hpspmm {

// Writes zeros into the rows that hold no entries: extra blocks of the product's grid walk all rows, 32 at a time,
// the bounds of the next 32 in flight while the current ones are stored.  KS: the width when it is a compile-time
// constant (one store instruction then covers 32 * 4 / KS rows), else 0.
template <int KS>
__device__ __forceinline__ void zero_empty_rows(int M, int K, const int* __restrict__ row_ptr, float* __restrict__ C,
                                                int zero_block, int n_zero_blocks, int block_threads) {
  const int lane = threadIdx.x & 31;
  const int warps_per_block = block_threads / 32;
  const int64_t stride = (int64_t)n_zero_blocks * warps_per_block * 32;
  int64_t r0 = ((int64_t)zero_block * warps_per_block + (threadIdx.x >> 5)) * 32;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto is_empty = [&](int64_t r) {
    if (r >= M) return false;
    const int s = ld_chained(row_ptr + r), e = ld_chained(row_ptr + r + 1);
    return s == e;
  };
  bool next = is_empty(r0 + lane);
  for (; r0 < M; r0 += stride) {
    unsigned m = __ballot_sync(0xffffffffu, next);
    next = is_empty(r0 + stride + lane);
    if (KS == 32 || KS == 64 || KS == 128) {
      constexpr int W = KS >= 4 ? KS / 4 : 1;
      float* c = C + r0 * KS + lane * 4;   // lane / W = row of the store, lane % W = its column
      m >>= lane / W;
#pragma unroll 4
      for (int q = 0; q < W; ++q)
        if ((m >> (q * (32 / W))) & 1u) st_stream(c + q * 128, zero);
    } else {
      while (m) {
        const int b = __ffs(m) - 1;
        m &= m - 1;
        float* crow = C + (r0 + b) * K;
        if ((K & 3) == 0) {
          for (int c = lane * 4; c < K; c += 128) st_stream(crow + c, zero);
        } else {
          for (int c = lane; c < K; c += 32) crow[c] = 0.f;
        }
      }
    }
  }
}

// The row that holds entry t, i.e. the last r in [lo, hi) with row_ptr[r] <= t, given that row_ptr[lo] <= t.  The
// whole warp searches: 32 probes a round, so a million rows take four rounds of one load.
__device__ __forceinline__ int find_row(const int* __restrict__ row_ptr, int lo, int hi, int t) {
  const int lane = threadIdx.x & 31;
  while (hi - lo > 1) {
    const int step = (int)(((unsigned)(hi - lo) + 31u) >> 5);
    const int64_t r = lo + (int64_t)lane * step;
    const unsigned m = __ballot_sync(0xffffffffu, r < hi && ld_chained(row_ptr + r) <= t);
    lo += (__popc(m | 1u) - 1) * step;   // lane 0 probes lo itself
    hi = step < hi - lo ? lo + step : hi;
  }
  return lo;
}

// The next row that holds entries after `row`, whose end is `row_end` (< nnz): (row, end).  The warp looks at 32 rows
// at once and searches when all of them are empty.
__device__ __forceinline__ int2 next_filled_row(const int* __restrict__ row_ptr, int M, int row, int row_end) {
  const int lane = threadIdx.x & 31;
  const int r = row + 1 + lane;   // candidate
  const int e = __ldg(row_ptr + (r + 1 < M ? r + 1 : M));
  const unsigned m = __ballot_sync(0xffffffffu, e > row_end);
  if (m) {
    const int b = __ffs(m) - 1;
    return make_int2(row + 1 + b, __shfl_sync(0xffffffffu, e, b));
  }
  const int f = find_row(row_ptr, row + 32, M, row_end);
  return make_int2(f, __ldg(row_ptr + f + 1));
}

// Adds up the split rows that a chunk has a piece of: row r0, whose last piece the chunk has stored (`stored`), and row
// r1, whose partial sum it has left in its carry slot (`handed_on`).
//
// A row longer than S is cut at multiples of S only, so its pieces are the chunks first = row_ptr[r] / S .. last =
// (row_ptr[r+1] - 1) / S: all but the last hand a carry on, the last stores the row.  A piece bumps a counter when its
// own part is visible device-wide, and whoever bumps it last adds the carries up: nobody waits, and the order of the
// additions does not depend on who that is.  Up to kCarryGroup carries meet at one counter (counter[first]) and are
// added to the stored row.  More meet in groups: the last of a group (counter[first + 16 q]) leaves the group's sum in
// the group's first slot, and the groups and the stored row meet at counter[first + 1].  A row of 40,000 entries has 250
// carries; added by one warp they were a chain of 16 memory round trips at the end of the launch.
// Both rows are announced by one instruction (lane 0 and lane 1), so a chunk that has a piece of two rows pays for one
// release and one round trip.  Power-law graphs, one row at a time and all carries by one warp -> this: 4 M entries,
// K = 64 79.3 -> 76.5 us, K = 128 132.6 -> 126.5 us; 16 M entries, K = 64 291.9 -> 283.4 us, K = 128 517 -> 505 us.
// `C`, `carry` and `counter` are those of the slab: ld is the row stride of C and of the carry slots, kw the width.
constexpr int kCarryGroup = 16;

// sum of slots 0, step, 2 * step, .. of n, the lane groups taking them in turn; every lane gets the total
template <int VEC, int W>
__device__ __forceinline__ void sum_carries(float (&sum)[VEC], const float* src, int n, int64_t step) {
  constexpr int G = 32 / W;
  constexpr int BATCH = kCarryGroup / G < 1 ? 1 : (kCarryGroup / G > 8 ? 8 : kCarryGroup / G);   // loads in flight
  const int g = (threadIdx.x & 31) / W;
#pragma unroll
  for (int x = 0; x < VEC; ++x) sum[x] = 0.f;
#pragma unroll 1
  for (int i = g; i < n; i += BATCH * G) {
    float v[BATCH][VEC];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
#pragma unroll
      for (int x = 0; x < VEC; ++x) v[u][x] = 0.f;
      if (i + u * G < n) load_l2(v[u], src + (int64_t)(i + u * G) * step);
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
#pragma unroll
      for (int x = 0; x < VEC; ++x) sum[x] += v[u][x];
  }
  all_reduce_groups<VEC, W>(sum);
}

template <int VEC, int W, int R>
__device__ __forceinline__ void settle_split_rows(bool stored, int r0, int r0_start, int r0_end, bool handed_on, int r1,
                                                  int r1_start, int r1_end, int chunk, int S, float* __restrict__ carry,
                                                  float* __restrict__ C, int* __restrict__ counter, int ld, int kw) {
  const int lane = threadIdx.x & 31;
  const int g = lane / W, l = lane % W;
  const int my_row = lane == 0 ? r0 : r1;
  const int my_first = (lane == 0 ? r0_start : r1_start) / S;
  const int my_len = ((lane == 0 ? r0_end : r1_end) - 1) / S - my_first;   // carries of the row
  const int my_group = (chunk - my_first) / kCarryGroup * kCarryGroup;      // first carry of this piece's group
  __syncwarp();   // every lane's part is written before lanes 0 and 1 announce it
  bool complete = false;
  if (lane == 0 ? stored : (lane == 1 && handed_on)) {
    int at = my_first, others = my_len;
    if (my_len > kCarryGroup) {
      at += lane == 0 ? 1 : my_group;
      others = lane == 0 ? (my_len + kCarryGroup - 1) / kCarryGroup : min(kCarryGroup, my_len - my_group) - 1;
    }
    complete = atomic_add_release(counter + at, 1) == others;
  }
  const unsigned todo = __ballot_sync(0xffffffffu, complete);
  if (todo == 0) return;
  __threadfence();
  const int64_t K = ld;
#pragma unroll 1
  for (int t = 0; t < 2; ++t) {
    if (!((todo >> t) & 1u)) continue;
    const int row = __shfl_sync(0xffffffffu, my_row, t), first = __shfl_sync(0xffffffffu, my_first, t);
    const int len = __shfl_sync(0xffffffffu, my_len, t), group = __shfl_sync(0xffffffffu, my_group, t);
    const bool grouped = len > kCarryGroup;
    const int n_groups = (len + kCarryGroup - 1) / kCarryGroup;
    const int at = first + (grouped ? 1 : 0);
    if (grouped && t == 1) {
      // the group is complete: its sum replaces its first carry
      float* slot = carry + (int64_t)(first + group) * K;
#pragma unroll 1
      for (int rr = 0; rr < R; ++rr) {
        const int col = (rr * W + l) * VEC;
        const bool live = col < kw;
        float sum[VEC];
        sum_carries<VEC, W>(sum, slot + (live ? col : 0), min(kCarryGroup, len - group), K);
        if (g == 0 && live) store_plain(slot + col, sum);
      }
      __syncwarp();
      bool all = false;
      if (lane == 0) {
        counter[first + group] = 0;
        all = atomic_add_release(counter + at, 1) == n_groups;
      }
      if (!__shfl_sync(0xffffffffu, (int)all, 0)) continue;
      __threadfence();
    }
#pragma unroll 1
    for (int rr = 0; rr < R; ++rr) {
      const int col = (rr * W + l) * VEC;
      const bool live = col < kw;
      float sum[VEC];
      sum_carries<VEC, W>(sum, carry + (int64_t)first * K + (live ? col : 0), grouped ? n_groups : len,
                          grouped ? K * kCarryGroup : K);
      if (g == 0 && live) {
        float* out = C + (int64_t)row * K + col;
        float o[VEC];
        load_l2(o, out);
#pragma unroll
        for (int x = 0; x < VEC; ++x) o[x] += sum[x];
        store_stream(out, o);
      }
    }
    if (lane == 0) counter[at] = 0;   // ready for the next launch
  }
}

// KS: row stride of B and C when it is a compile-time constant (the whole width is one full slab), else 0.
// LIST: the rows that hold entries are listed (a.nz, with records a.rec).  Without the list a warp finds the bounds
// of its chunk by searching row_ptr and steps from row to row along row_ptr: for calls without a plan whose matrix is
// so small that the two launches that build the list would cost more than the searches, and for the allocation-free
// entry point, whose scratch has no room for it.
template <int VEC, int W, int R, int U, int KS, int BT, int MINB, bool HINT, bool LIST>
__global__ void __launch_bounds__(BT, MINB) spmm_warp_kernel(const __grid_constant__ hpspmm_spmm_args a) {
  constexpr int CW = VEC * W * R;   // columns a warp covers
  constexpr int G = 32 / W;         // lane groups = entries gathered per step
  constexpr int T = 32;             // entries per staged tile
  constexpr int BATCH = U * G;      // entries per batch of gathers
  constexpr int STAGES = 2;
  static_assert(BATCH <= T && T % BATCH == 0, "batch must tile the staged tile");
  static_assert(KS == 0 || KS == CW, "a fixed stride is the width of the slab");
  __shared__ int2 tiles[BT / 32][STAGES][T];
  __shared__ int meta[BT / 32][8];

  chain_grid();
  if ((int)blockIdx.x >= a.n_chunk_blocks) {
    if (blockIdx.y == 0 && a.slab0 == 0 && a.off == 0) {
      if (!LIST)
        for (int i = ((int)blockIdx.x - a.n_chunk_blocks) * BT + (int)threadIdx.x; i < a.n_clear;
             i += ((int)gridDim.x - a.n_chunk_blocks) * BT)
          a.clear[i] = 0;
      zero_empty_rows<KS>(a.M, a.K, a.row_ptr, a.C, blockIdx.x - a.n_chunk_blocks, gridDim.x - a.n_chunk_blocks, BT);
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  const int g = lane / W;   // group
  const int l = lane % W;   // position inside the group
  int n1, row, row_end, ri, base;
  {
    const int slot = (int)((blockIdx.x * (unsigned)BT + threadIdx.x) >> 5);
    if (slot >= a.n_chunks) return;
    int* m = meta[threadIdx.x >> 5];   // what the tail of the kernel needs of the chunk waits in shared memory
    if (LIST) {
      const int4 p = ld_chained(a.rec + 2 * (int64_t)slot), q = ld_chained(a.rec + 2 * (int64_t)slot + 1);
      base = p.x, ri = p.y, row = p.z, row_end = p.w;
      n1 = q.z;
      if (lane == 0) m[0] = base, m[1] = q.x, m[2] = row, m[3] = q.y, m[4] = row_end;
    } else {
      // chunk `slot` begins at the start of the row that holds entry slot * S, or at that entry if the row is longer
      // than S; it ends where the next one begins
      ri = 0;
      const int t0 = slot * a.S, t1 = t0 + a.S;
      row = find_row(a.row_ptr, 0, a.M, t0);
      const int rs = __ldg(a.row_ptr + row);
      row_end = __ldg(a.row_ptr + row + 1);
      base = slot == 0 ? 0 : (row_end - rs <= a.S ? rs : t0);
      if (slot + 1 < a.n_chunks) {
        n1 = t1;
        if (row_end <= t1) {   // (a row that reaches from t0 over t1 is longer than S and is cut there)
          const int r1 = find_row(a.row_ptr, row + 1, a.M, t1);
          const int s1 = __ldg(a.row_ptr + r1), e1 = __ldg(a.row_ptr + r1 + 1);
          if (e1 - s1 <= a.S) n1 = s1;
        }
      } else {
        n1 = ld_chained(a.row_ptr + a.M);
      }
      if (lane == 0) m[0] = base, m[1] = slot, m[2] = row, m[3] = rs, m[4] = row_end;
    }
  }
  const int off = KS ? 0 : a.off + (a.slab0 + (int)blockIdx.y) * CW;
  const int kw = KS ? CW : min(CW, a.cols - (a.slab0 + (int)blockIdx.y) * CW);
  const uint64_t policy = HINT ? (KS ? policy_evict_last() : policy_for_gathers(a.keep_b)) : 0ull;
  int2(*my)[T] = tiles[threadIdx.x >> 5];

  // The row after the current one is fetched while the current one is summed, where the registers allow it (R-MAT
  // scale 18, 64 columns: 0.1009 against 0.1032 ms; scale 20, 128 columns: 0.587 against 0.556 ms, so not there).
  constexpr bool AHEAD = W <= 16;
  int2 next = make_int2(0, 0);
  if (LIST && AHEAD) next = __ldg(a.nz + ri + 1);
  if (!LIST) next.y = __ldg(a.row_ptr + (row + 2 < a.M ? row + 2 : a.M));

  auto stage_tile = [&](int stage, int base) {
    const int j = base + lane;
    if (j < n1) {
      cp_async_4(&my[stage][lane].x, a.col_idx + j);
      cp_async_4(&my[stage][lane].y, a.vals + j);
    } else {
      my[stage][lane] = make_int2(0, 0);   // past the chunk: column 0, value 0
    }
    cp_async_commit();
  };
  stage_tile(0, base);
  stage_tile(1, base + T);

  float acc[R][VEC];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int x = 0; x < VEC; ++x) acc[r][x] = 0.f;
  const bool live_last = KS || ((R - 1) * W + l) * VEC < kw;   // only the last vector of a lane can lie outside
  const unsigned stride = (KS ? KS : a.K) * 4u;                // bytes
  const char* Bl = reinterpret_cast<const char*>(a.B + off + ((R > 1 || live_last) ? l * VEC : kw - VEC));
  const char* Bl_last = reinterpret_cast<const char*>(a.B + off + (live_last ? ((R - 1) * W + l) * VEC : kw - VEC));
  using Split = group_split<VEC, W>;
  const int out_col = Split::column(lane);   // where this lane's share of a finished row goes
  char* Cl = reinterpret_cast<char*>(a.C + off + out_col);

  auto gather = [&](float (&b)[R][VEC], int col) {
    const char* p = Bl + (uint64_t)(unsigned)col * stride;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (R > 1 && r == R - 1)
        gather_vec<VEC, HINT>(b[r], reinterpret_cast<const float*>(Bl_last + (uint64_t)(unsigned)col * stride), policy);
      else
        gather_vec<VEC, HINT>(b[r], reinterpret_cast<const float*>(p) + r * W * VEC, policy);
    }
  };
  auto fma = [&](float v, const float (&b)[R][VEC]) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int x = 0; x < VEC; ++x) acc[r][x] = fmaf(v, b[r][x], acc[r][x]);
  };
  auto store_row = [&]() {
    float* crow = reinterpret_cast<float*>(Cl + (uint64_t)(unsigned)row * stride);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float v[Split::KEEP];
      combine_groups<VEC, W>(acc[r], v, lane);
      if (Split::writes(lane) && (r < R - 1 || live_last)) store_stream(crow + r * W * VEC, v);
    }
  };
  // the row is complete: store it, start the next row that holds entries
  auto finish_row = [&]() {
    store_row();
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int x = 0; x < VEC; ++x) acc[r][x] = 0.f;
    if (LIST) {
      ++ri;
      if (!AHEAD) next = __ldg(a.nz + ri);
      row = next.x;
      row_end = next.y;
      if (AHEAD) next = __ldg(a.nz + ri + 1);
    } else {
      // next.y: the end of the row below, fetched ahead; the rows below it are looked at when that one is empty
      if (next.y > row_end) {
        ++row;
        row_end = next.y;
      } else {
        const int2 f = next_filled_row(a.row_ptr, a.M, row, row_end);
        row = f.x;
        row_end = f.y;
      }
      next.y = __ldg(a.row_ptr + (row + 2 < a.M ? row + 2 : a.M));
    }
  };

  int stage = 0;
  for (; base < n1; base += T) {
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    const int2* tile = &my[stage][g];
    if (base + T <= n1 && row_end >= base + T) {
      // Fast tile: all 32 entries belong to the current row: no tests between gathers.  Not unrolled all the way:
      // the compiler then hoists gathers of later batches over the FMAs of earlier ones until it has to spill (K = 128
      // at 48 registers, R-MAT scale 20: 0.700 ms fully unrolled, 0.576 ms two batches at a time, 0.582 ms one).
#pragma unroll(W == 32 ? 2 : 1)
      for (int s0 = 0; s0 < T / G; s0 += U) {
        float b[U][R][VEC];
        float v[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int2 e = tile[(s0 + i) * G];   // one broadcast per group
          v[i] = __int_as_float(e.y);
          gather(b[i], e.x);
        }
#pragma unroll
        for (int i = 0; i < U; ++i) fma(v[i], b[i]);
      }
    } else {
#pragma unroll 1
      for (int u0 = 0; u0 < T; u0 += BATCH) {
        const int j0 = base + u0;
        if (j0 >= n1) break;
        float b[U][R][VEC];
        float v[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int2 e = tile[u0 + i * G];
          v[i] = __int_as_float(e.y);
          gather(b[i], e.x);
        }
        if (j0 + BATCH <= n1 && row_end >= j0 + BATCH) {
#pragma unroll
          for (int i = 0; i < U; ++i) fma(v[i], b[i]);
        } else {
#pragma unroll
          for (int i = 0; i < U; ++i) {
            const int lo = j0 + i * G;
            const int hi = min(lo + G, n1);
            const int mine = lo + g;
            int cur = lo;
            while (row_end < hi) {   // warp-uniform: the current row ends inside this step
              if (mine >= cur && mine < row_end) fma(v[i], b[i]);
              cur = row_end;
              finish_row();
            }
            if (mine >= cur && mine < hi) fma(v[i], b[i]);
          }
        }
      }
    }
    __syncwarp();
    stage_tile(stage, base + STAGES * T);
    stage ^= 1;
  }
  cp_async_wait<0>();

  const int* m = meta[threadIdx.x >> 5];
  const int n0 = m[0], chunk = m[1], r0 = m[2], r0_start = m[3], r0_end = m[4];
  const bool hands_on = row_end != n1;   // the chunk ends inside `row`
  const int64_t ldc = KS ? KS : a.K;
  float* carry = a.carry + off;
  if (!hands_on) {
    store_row();
  } else {
    float* slot_c = carry + (int64_t)chunk * ldc + out_col;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float v[Split::KEEP];
      combine_groups<VEC, W>(acc[r], v, lane);
      if (Split::writes(lane) && (r < R - 1 || live_last)) store_plain(slot_c + r * W * VEC, v);
    }
  }
  // the pieces of a split row settle it among themselves
  const bool stores_split_row = r0_start < n0 && r0_end <= n1;   // began in an earlier chunk, ends here
  if (!hands_on && !stores_split_row) return;
  int* counter = KS ? a.counter : a.counter + (int64_t)blockIdx.y * a.n_chunks;
  settle_split_rows<VEC, W, R>(stores_split_row, r0, r0_start, r0_end, hands_on, row,
                               row == r0 ? r0_start : __ldg(a.row_ptr + row), row_end, chunk, a.S, carry, a.C + off,
                               counter, (int)ldc, kw);
}

// Launches one shape.  Slabs of the width run as blockIdx.y, each with counters of its own; where the counters are
// shared (shared_counters: the fixed scratch has room for one set) they run one after the other.
template <int VEC, int W, int R, int U, int KS, int MINB, bool HINT, int BT = 64>
int launch_spmm_shape(hpspmm_ctx* ctx, hpspmm_spmm_args a, bool shared_counters, cudaStream_t stream) {
  constexpr int CW = VEC * W * R;
  constexpr int per_block = BT / 32;
  a.n_chunk_blocks = (a.n_chunks + per_block - 1) / per_block;
  int n_zero_blocks = (a.M + BT - 1) / BT;
  const int cap = ctx->sm_count * 8;
  if (n_zero_blocks > cap) n_zero_blocks = cap;
  const int slabs = (a.cols + CW - 1) / CW;
  const int64_t grid = (int64_t)a.n_chunk_blocks + n_zero_blocks;
  if (grid == 0) return HPSPMM_OK;
  if (!hpspmm_shape_covers(VEC, W, R, a.cols)) return HPSPMM_ERR_INVALID;
  const int step = shared_counters ? 1 : 65535;
  for (int s = 0; s < slabs; s += step) {
    a.slab0 = s;
    const int ny = slabs - s < step ? slabs - s : step;
    const dim3 g((unsigned)grid, (unsigned)ny);
    if (a.nz != nullptr)
      hpspmm_launch(spmm_warp_kernel<VEC, W, R, U, KS, BT, MINB, HINT, true>, g, BT, 0, stream, a);
    else   // (a runtime stride serves every width)
      hpspmm_launch(spmm_warp_kernel<VEC, W, R, U, 0, BT, (MINB < 16 ? MINB : 16), true, false>, g, BT, 0, stream, a);
    ctx->launches++;
  }
  HPSPMM_CUDA_TRY(ctx, cudaGetLastError());
  return HPSPMM_OK;
}

}  // namespace hpspmm
